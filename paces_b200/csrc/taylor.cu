// Truncated-Taylor exp(-i dt H) psi as one persistent cooperative kernel.
//
// Reference (paces/core/time_evolution.py:482-512, _simple_taylor): term_{j+1} =
// (-i dt/(j+1)) H term_j, res += term_{j+1}, stop when (|term_j|_inf + |term_{j+1}|_inf) /
// |res|_inf <= tol, at most m_star terms; one host sync per term in the reference.
//
// B200 design: every term is one grid-stride sweep over the rows (neighbour-table SpMV,
// term write, res update and the two inf-norms fused), separated by a bounded grid
// barrier; every block reduces the per-block maxima itself and takes the same stop
// decision, so the whole series runs in one launch with no host round trip.  The
// neighbour indices of consecutive rows are monotone (images of a sorted block are
// sorted), so the four gathers stream through L2.  complex128 rounds every operation
// like the reference; complex64 uses fp32 FMA with fp64 stop arithmetic.
//
// Two row schedules (a tuning choice; the results are identical because every row's
// arithmetic is the same and the maxima are exact):
//  * direct: grid-stride, two rows per thread per pass, all loads from global memory;
//  * bulk:   each block owns 512-row chunks.  When no block owns more than two, they stay in
//            shared memory for the whole series: a sweep then only gathers, stores the new
//            term and updates the sum on chip (S up to 1024 rows per block of the wave).
//            Otherwise the chunks stream: while a block computes one, one thread has the
//            next chunk's neighbour rows, metadata and own elements brought into the other
//            half of a shared-memory double buffer by bulk TMA copies (cp.async.bulk,
//            completion on an mbarrier), so the streaming reads are in flight while the
//            gathers of the current chunk wait on L2.
//
// The streamed sum lags: a sweep that starts with the sum up to date writes its term only,
// and the next one adds both terms in the order of the series (the row's own element of the
// source is the last term, and it is loaded for H's diagonal anyway).  Per pair of sweeps the
// sum is read and written once instead of twice.  The stop test needs the sum's inf-norm; in
// a sweep that left the sum alone it is known to lie within the new term's norm of the last
// exact one, which settles the test unless the series may end here -- then an extra pass adds
// the term and measures the norm.  Terms, sums, norms and decisions are the ones of a series
// that updates the sum in every sweep, bit for bit.
#include "grid.cuh"
#include "hrow.cuh"
#include "kernels.cuh"
#include "tc.cuh"

namespace paces {

namespace {

constexpr int kTThreads = 256;
constexpr int kTWarps = kTThreads / 32;

// Largest of a warp's non-negative values (their bit patterns order like the values).
__device__ __forceinline__ float warp_max(float v) {
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v)));
}
__device__ __forceinline__ double warp_max(double v) {
    const unsigned hi = unsigned(__double2hiint(v)), lo = unsigned(__double2loint(v));
    const unsigned h = __reduce_max_sync(0xffffffffu, hi);
    return __hiloint2double(int(h), int(__reduce_max_sync(0xffffffffu, hi == h ? lo : 0u)));
}

// A sweep's maxima over the grid: |term|^2, |res|^2, |v|^2 (first sweep) and a non-finite flag.
template <typename R>
struct SweepMax {
    R term, res, v;
    bool bad;
};

// Fold the block's maxima into g[0..3] (fp64 bit patterns; atomicMax is exact and order-free),
// pass the grid barrier and read the grid's maxima into fin[0..3] (shared).  false on a timeout.
template <typename R>
__device__ bool grid_max(const SweepMax<R>& mx, unsigned long long* g, double (*red)[kTWarps], double* fin,
                         const TaylorWs& ws, unsigned& gen, int* status) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const R a = warp_max(mx.term), b = warp_max(mx.res), c = warp_max(mx.v);
    const bool bad = __any_sync(0xffffffffu, mx.bad);
    if (lane == 0) {
        red[0][wid] = double(a);
        red[1][wid] = double(b);
        red[2][wid] = double(c);
        red[3][wid] = bad ? 1.0 : 0.0;
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        double r = 0.0;
        for (int w = 0; w < kTWarps; ++w) r = fmax(r, red[threadIdx.x][w]);
        if (r > 0.0) atomicMax(g + threadIdx.x, static_cast<unsigned long long>(__double_as_longlong(r)));
    }
    if (!grid_barrier(ws.barrier, gridDim.x, gen, status, ws.wait_ns, int(blockIdx.x) == ws.skip_block)) return false;
    if (threadIdx.x < 4) fin[threadIdx.x] = __longlong_as_double((long long)__ldcg(g + threadIdx.x));
    __syncthreads();
    return true;
}

constexpr int kChunk = 2 * kTThreads;  // rows per block pass of the bulk schedule
template <bool C64>
constexpr uint32_t chunk_bytes() {  // neighbour rows, metadata, result, own term element
    return uint32_t(kChunk) * (16 + 4 + 2 * (C64 ? 8 : 16));
}

// XHOP: a lattice with several hopping channels (the channel loop of h_row_*_x).
template <bool C64, bool BULK, bool XHOP>
__global__ void __launch_bounds__(kTThreads, C64 ? 4 : 3)
taylor_kernel(ModelDev m, const int* __restrict__ blk, const int* __restrict__ nbr, int64_t cap,
              const uint32_t* __restrict__ meta, const void* v_in, void* res_out, TaylorWs ws,
              double dt, int m_star, double tol, TaylorOut out, int* status) {
    using C = typename std::conditional<C64, float2, double2>::type;
    using R = typename std::conditional<C64, float, double>::type;
    extern __shared__ __align__(128) unsigned char t_smem[];  // bulk: 2 x chunk_bytes
    __shared__ R s_sq[260];
    __shared__ double s_red[4][kTWarps];
    __shared__ double s_fin[4];
    __shared__ __align__(8) uint64_t s_mbar[2];
    __shared__ int s_abort;
    for (int k = threadIdx.x; k < 260; k += kTThreads) s_sq[k] = R(__dmul_rn(sqrt(double(k)), m.g));
    if constexpr (BULK) {
        if (threadIdx.x == 0) {
            tc::mbar_init(tc::smem_addr(&s_mbar[0]), 1);
            tc::mbar_init(tc::smem_addr(&s_mbar[1]), 1);
            s_abort = 0;
        }
    }
    __syncthreads();
    uint32_t parity = 0;    // bulk: phase parity of each buffer's mbarrier (bit b)
    uint32_t pending = 0;   // bulk, thread 0: buffers with copies issued and not yet consumed

    const int64_t S = blk[m.L];
    unsigned gen = 0;
    const C* v = reinterpret_cast<const C*>(v_in);
    C* res = reinterpret_cast<C*>(res_out);
    C* ta = reinterpret_cast<C*>(ws.ta);
    C* tb = reinterpret_cast<C*>(ws.tb);
    const R J = R(m.J);
    double c1 = 0.0, c1c2 = 0.0, ratio = 0.0;
    int conv = 0, fin_j = 0;

    // bulk: the chunks this block owns (c, c + grid, ..); with at most two they stay in the two
    // buffers for the whole series, otherwise they stream through them
    const int64_t nch = (S + kChunk - 1) / kChunk;
    const bool resident = BULK && nch <= 2 * int64_t(gridDim.x);
    // bulk, streaming: the sum lags one term behind (see the head of this file)
    bool lag = false;
    const C* rbase = v;      // where the sum without the lagging term is
    double rnorm = 0.0;      // its inf-norm
    unsigned sweep = 0;      // barriers passed with maxima: the maxima's buffers rotate
    auto maxima = [&](unsigned s) { return ws.maxima + (s % 3) * 4; };
    // after sweep s's barrier: clear the buffer that sweep s + 2 folds into
    auto next_sweep = [&]() {
        if (blockIdx.x == 0 && threadIdx.x < 4) maxima(sweep + 2)[threadIdx.x] = 0ull;
        ++sweep;
    };
    constexpr uint32_t kCB = chunk_bytes<C64>();
    constexpr uint32_t kOffMeta = kChunk * 16, kOffRin = kOffMeta + kChunk * 4,
                       kOffSelf = kOffRin + kChunk * sizeof(C);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // chunk rows of this thread when a warp holds one 64-row group (the first sweep's diagnostics)
    const int g0 = kDiagGroup * wid + lane, g1 = g0 + 32;
    if constexpr (BULK) {
        if (resident) {
            for (int k = 0; k < 2; ++k) {
                const int64_t r0 = (blockIdx.x + int64_t(k) * gridDim.x) * kChunk;
                unsigned char* base = t_smem + k * kCB;
                for (int t = threadIdx.x; t < kChunk && r0 + t < S; t += kTThreads) {
                    reinterpret_cast<int4*>(base)[t] = load_nbr(nbr, r0 + t);
                    reinterpret_cast<uint32_t*>(base + kOffMeta)[t] = __ldg(meta + r0 + t);
                    const C z = v[r0 + t];
                    reinterpret_cast<C*>(base + kOffRin)[t] = z;
                    reinterpret_cast<C*>(base + kOffSelf)[t] = z;
                }
            }
            __syncthreads();
        }
    }

    for (int j = 0; j < m_star; ++j) {
        const C* src = j == 0 ? v : ((j & 1) ? ta : tb);
        C* dst = (j & 1) ? tb : ta;
        const double cd = dt / double(j + 1);
        const R c = R(cd);
        SweepMax<R> mx{R(0), R(0), R(0), false};
        auto sq_abs = [](const C& z) -> R {
            if constexpr (C64) return fmaf(z.x, z.x, __fmul_rn(z.y, z.y));
            else return fma(z.x, z.x, __dmul_rn(z.y, z.y));
        };
        auto finite = [](const C& z) { return isfinite(z.x) && isfinite(z.y); };
        auto add = [](const C& a, const C& t) -> C {
            if constexpr (C64) return make_float2(__fadd_rn(a.x, t.x), __fadd_rn(a.y, t.y));
            else return make_double2(__dadd_rn(a.x, t.x), __dadd_rn(a.y, t.y));
        };
        // the new term from y = H src: separate roundings (no contraction into an FMA), so that
        // every kernel and schedule that runs these rows -- direct, bulk, batched -- rounds alike
        auto term = [&](const C& y) -> C {
            C t;
            if constexpr (C64) t = make_float2(__fmul_rn(c, y.y), -__fmul_rn(c, y.x));
            else t = make_double2(__dmul_rn(cd, y.y), -__dmul_rn(cd, y.x));
            mx.term = fmax(mx.term, sq_abs(t));
            return t;
        };
        auto sum_to = [&](const C& a, const C& t) -> C {  // a + t, the new sum
            const C rr = add(a, t);
            mx.res = fmax(mx.res, sq_abs(rr));
            mx.bad |= !finite(rr);
            return rr;
        };
        auto hrow = [&](int64_t r) -> C {
            const uint32_t mm = __ldg(meta + r);
            if constexpr (XHOP) {
                if constexpr (C64) return h_row_c64_x(m, s_sq, r, load_nbr(nbr, r), mm, __ldcg(src + r), src);
                else return h_row_c128_x(m, s_sq, r, load_nbr(nbr, r), mm, __ldcg(src + r), src);
            } else {
                if constexpr (C64) return h_row_c64(m, s_sq, J, r, nbr, mm, src);
                else return h_row_c128(m, s_sq, r, nbr, mm, src);
            }
        };
        // one row of a chunk whose neighbour row, metadata and own element are in shared memory
        auto crow = [&](int64_t r, const int4& nb, uint32_t mm, const C& own) -> C {
            if constexpr (XHOP) {
                if constexpr (C64) return h_row_c64_x(m, s_sq, r, nb, mm, own, src);
                else return h_row_c128_x(m, s_sq, r, nb, mm, own, src);
            } else if constexpr (C64) {
                return h_row_c64_nb(m, s_sq, J, r, nb, mm, own, src);
            } else {
                return h_row_c128_nb(m, s_sq, r, nb, mm, own, src);
            }
        };
        const bool diag = j == 0 && ws.diag != nullptr;  // first sweep: fold the input's diagnostics
        bool exact = true;  // this sweep brings the sum and its norm up to date
        if constexpr (!BULK) {
            const C* rin = j == 0 ? v : res;
            auto finish = [&](int64_t r, const C& y, const C& a) {
                const C t = term(y);
                if (j == 0) mx.v = fmax(mx.v, sq_abs(a));
                res[r] = sum_to(a, t);
                dst[r] = t;
            };
            // two rows per thread per pass: all loads of both rows precede the stores
            const int64_t stride = int64_t(gridDim.x) * kTThreads;
            if (!diag) {
                int64_t r = int64_t(blockIdx.x) * kTThreads + threadIdx.x;
                for (; r + stride < S; r += 2 * stride) {
                    const C y0 = hrow(r), y1 = hrow(r + stride);
                    const C a0 = rin[r], a1 = rin[r + stride];
                    finish(r, y0, a0);
                    finish(r + stride, y1, a1);
                }
                if (r < S) finish(r, hrow(r), rin[r]);
            } else {
                // every row once, in 64-row units per warp (rows u + lane and u + 32 + lane, a
                // warp-uniform loop), so that each warp folds its 64-row groups
                const int64_t ustride = int64_t(gridDim.x) * kTWarps * kDiagGroup;
                for (int64_t ub = (int64_t(blockIdx.x) * kTWarps + wid) * kDiagGroup; ub < S; ub += ustride) {
                    const int64_t r0 = ub + lane, r1 = ub + 32 + lane;
                    const bool v0 = r0 < S, v1 = r1 < S;
                    C y0{}, y1{}, a0{}, a1{};
                    if (v0) {
                        y0 = hrow(r0);
                        a0 = rin[r0];
                    }
                    if (v1) {
                        y1 = hrow(r1);
                        a1 = rin[r1];
                    }
                    if (v0) finish(r0, y0, a0);
                    if (v1) finish(r1, y1, a1);
                    diag_group(ws.diag, ub / kDiagGroup, v0, a0, y0, v1, a1, y1);
                }
            }
        } else if (resident) {
            for (int k = 0; k < 2; ++k) {
                const int64_t ch = blockIdx.x + int64_t(k) * gridDim.x;
                const int64_t r0 = ch * kChunk;
                if (r0 + kDiagGroup * wid >= S) break;  // no row of this warp's group
                unsigned char* base = t_smem + k * kCB;
                const int4* snb = reinterpret_cast<const int4*>(base);
                const uint32_t* smeta = reinterpret_cast<const uint32_t*>(base + kOffMeta);
                C* sres = reinterpret_cast<C*>(base + kOffRin);
                C* sself = reinterpret_cast<C*>(base + kOffSelf);
                const bool v0 = r0 + g0 < S, v1 = r0 + g1 < S;
                C y0{}, y1{};
                if (v0) y0 = crow(r0 + g0, snb[g0], smeta[g0], sself[g0]);
                if (v1) y1 = crow(r0 + g1, snb[g1], smeta[g1], sself[g1]);
                if (diag) {
                    const C z{};
                    diag_group(ws.diag, r0 / kDiagGroup + wid, v0, v0 ? sself[g0] : z, y0, v1, v1 ? sself[g1] : z, y1);
                }
                auto finish = [&](int g, const C& y) {
                    const C t = term(y);
                    const C a = sres[g];
                    if (j == 0) mx.v = fmax(mx.v, sq_abs(a));
                    sres[g] = sum_to(a, t);
                    sself[g] = t;
                    dst[r0 + g] = t;
                };
                if (v0) finish(g0, y0);
                if (v1) finish(g1, y1);
            }
        } else {
            exact = lag;
            auto full = [&](int64_t ch) { return (ch + 1) * kChunk <= S; };
            auto issue = [&](int64_t ch, int b) {  // thread 0
                const int64_t r0 = ch * kChunk;
                const uint32_t base = tc::smem_addr(t_smem + b * kCB);
                const uint32_t mb = tc::smem_addr(&s_mbar[b]);
                tc::mbar_expect_tx(mb, lag ? kCB : kCB - kChunk * uint32_t(sizeof(C)));
                tc::bulk_g2s(base, nbr + r0 * 4, kChunk * 16, mb);
                tc::bulk_g2s(base + kOffMeta, meta + r0, kChunk * 4, mb);
                if (lag) tc::bulk_g2s(base + kOffRin, rbase + r0, kChunk * sizeof(C), mb);
                tc::bulk_g2s(base + kOffSelf, src + r0, kChunk * sizeof(C), mb);
                pending |= 1u << b;
            };
            // row r: its new term and, when the sum lags, the sum with the last term and this one
            auto finish = [&](int64_t r, const C& y, const C& own, const C& a) {
                const C t = term(y);
                if (lag) {
                    const C prev = add(a, own);
                    mx.bad |= !finite(prev);
                    res[r] = sum_to(prev, t);
                } else {
                    mx.bad |= !finite(t);
                    if (j == 0) {
                        mx.bad |= !finite(own);
                        mx.v = fmax(mx.v, sq_abs(own));
                    }
                }
                dst[r] = t;
            };
            int64_t ch = blockIdx.x;
            if (threadIdx.x == 0 && ch < nch) {
                // the previous term's stores (every block's, ordered by the grid barrier) before
                // this term's bulk reads of them
                tc::fence_proxy_async_global();
                if (full(ch)) issue(ch, 0);
            }
            for (int k = 0; ch < nch; ch += gridDim.x, ++k) {
                const int b = k & 1;
                const int64_t cn = ch + gridDim.x;
                if (threadIdx.x == 0 && cn < nch && full(cn)) issue(cn, b ^ 1);
                const int64_t r0 = ch * kChunk;
                const int t0 = diag ? g0 : threadIdx.x;
                const int t1 = diag ? g1 : threadIdx.x + kTThreads;
                if (full(ch)) {
                    if (!tc::mbar_wait(tc::smem_addr(&s_mbar[b]), (parity >> b) & 1u)) s_abort = 1;
                    parity ^= 1u << b;
                    if (threadIdx.x == 0) pending &= ~(1u << b);
                    const unsigned char* base = t_smem + b * kCB;
                    const int4* snb = reinterpret_cast<const int4*>(base);
                    const uint32_t* smeta = reinterpret_cast<const uint32_t*>(base + kOffMeta);
                    const C* srin = reinterpret_cast<const C*>(base + kOffRin);
                    const C* sself = reinterpret_cast<const C*>(base + kOffSelf);
                    const C y0 = crow(r0 + t0, snb[t0], smeta[t0], sself[t0]);
                    const C y1 = crow(r0 + t1, snb[t1], smeta[t1], sself[t1]);
                    const C z{};
                    finish(r0 + t0, y0, sself[t0], lag ? srin[t0] : z);
                    finish(r0 + t1, y1, sself[t1], lag ? srin[t1] : z);
                    if (diag) diag_group(ws.diag, r0 / kDiagGroup + wid, true, sself[t0], y0, true, sself[t1], y1);
                } else {
                    // the last, partial chunk: direct loads
                    const bool v0 = r0 + t0 < S, v1 = r0 + t1 < S;
                    C y0{}, y1{}, a0{}, a1{};
                    const C z{};
                    if (v0) {
                        y0 = hrow(r0 + t0);
                        a0 = __ldcg(src + r0 + t0);
                        finish(r0 + t0, y0, a0, lag ? rbase[r0 + t0] : z);
                    }
                    if (v1) {
                        y1 = hrow(r0 + t1);
                        a1 = __ldcg(src + r0 + t1);
                        finish(r0 + t1, y1, a1, lag ? rbase[r0 + t1] : z);
                    }
                    if (diag && r0 + kDiagGroup * wid < S)  // groups with at least one row (warp-uniform)
                        diag_group(ws.diag, r0 / kDiagGroup + wid, v0, a0, y0, v1, a1, y1);
                }
                __syncthreads();  // the buffer is free for the copy issued next iteration
                if (s_abort) break;
            }
            if (s_abort) {
                // a copy that never completed: wait (bounded) for what is still in flight
                if (threadIdx.x == 0)
                    for (int bb = 0; bb < 2; ++bb)
                        if (pending & (1u << bb)) tc::mbar_wait(tc::smem_addr(&s_mbar[bb]), (parity >> bb) & 1u);
                if (threadIdx.x == 0) raise_status(status, PACES_ERR_TIMEOUT);
                fin_j = j;
                break;
            }
        }
        fin_j = j;
        if (!grid_max(mx, maxima(sweep), s_red, s_fin, ws, gen, status)) break;
        next_sweep();
        if (s_fin[3] != 0.0) {
            if (blockIdx.x == 0 && threadIdx.x == 0) raise_status(status, PACES_ERR_NONFINITE);
            break;
        }
        // the maxima are of |z|^2; one square root per term gives the inf-norms
        if (j == 0) c1 = sqrt(s_fin[2]);
        const double c2 = sqrt(s_fin[0]);
        c1c2 = c1 + c2;
        if (exact) {
            if (lag) rbase = res;
            lag = false;
            rnorm = sqrt(s_fin[1]);
        } else {
            if (j == 0) rnorm = c1;
            lag = true;
            // the sum's norm lies in rnorm -+ c2 (to a few roundings): only a ratio that may end
            // the series, or the series' last, needs it exactly
            if (j == m_star - 1 || c1c2 <= tol * (rnorm + c2) * 1.00001) {
                mx = SweepMax<R>{R(0), R(0), R(0), false};
                for (int64_t ch = blockIdx.x; ch < nch; ch += gridDim.x) {
                    const int64_t r0 = ch * kChunk + threadIdx.x, r1 = r0 + kTThreads;
                    C a0{}, a1{}, b0{}, b1{};
                    if (r0 < S) {
                        a0 = __ldcg(rbase + r0);
                        b0 = __ldcg(dst + r0);
                    }
                    if (r1 < S) {
                        a1 = __ldcg(rbase + r1);
                        b1 = __ldcg(dst + r1);
                    }
                    if (r0 < S) res[r0] = sum_to(a0, b0);
                    if (r1 < S) res[r1] = sum_to(a1, b1);
                }
                if (!grid_max(mx, maxima(sweep), s_red, s_fin, ws, gen, status)) break;
                next_sweep();
                if (s_fin[3] != 0.0) {
                    if (blockIdx.x == 0 && threadIdx.x == 0) raise_status(status, PACES_ERR_NONFINITE);
                    break;
                }
                exact = true;
                rbase = res;
                lag = false;
                rnorm = sqrt(s_fin[1]);
            }
        }
        if (exact) {
            ratio = c1c2 / rnorm;
            if (ratio <= tol) {
                conv = 1;
                break;
            }
        }
        c1 = c2;
    }
    if constexpr (BULK) {
        if (resident) {
            // the sum out of shared memory (each thread its own rows)
            for (int k = 0; k < 2; ++k) {
                const int64_t r0 = (blockIdx.x + int64_t(k) * gridDim.x) * kChunk;
                const C* sres = reinterpret_cast<const C*>(t_smem + k * kCB + kOffRin);
                if (r0 + g0 < S) res[r0 + g0] = sres[g0];
                if (r0 + g1 < S) res[r0 + g1] = sres[g1];
            }
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (out.converged) *out.converged = conv;
        if (out.final_m) *out.final_m = fin_j;
        if (out.c1_plus_c2) *out.c1_plus_c2 = c1c2;
        if (out.term_ratio) *out.term_ratio = ratio;
    }
}

template <bool C64, bool BULK>
size_t dyn_smem() {
    return BULK ? size_t(2) * chunk_bytes<C64>() : 0;
}

template <bool C64, bool BULK, bool XHOP>
int occupancy() {
    static int cached = 0;  // per process: the kernels' resources do not change
    if (cached) return cached;
    auto kfn = taylor_kernel<C64, BULK, XHOP>;
    if (BULK) cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(dyn_smem<C64, BULK>()));
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, kTThreads, dyn_smem<C64, BULK>());
    cached = per_sm < 1 ? 1 : (per_sm > 8 ? 8 : per_sm);
    return cached;
}

template <bool C64>
int occupancy_any(int variant, bool xhop) {
    if (xhop) return variant == 1 ? occupancy<C64, true, true>() : occupancy<C64, false, true>();
    return variant == 1 ? occupancy<C64, true, false>() : occupancy<C64, false, false>();
}

template <bool C64, bool BULK, bool XHOP>
cudaError_t launch_one(const cudaLaunchConfig_t& cfg, const ModelDev& m, const int* blk, const int* nbr, int64_t cap,
                       const uint32_t* meta, const void* v_in, void* res, const TaylorWs& ws, double dt, int m_star,
                       double tol, const TaylorOut& out, int* status) {
    if (BULK) {  // the attribute belongs to the current device: set it on every launch
        const cudaError_t a = cudaFuncSetAttribute(taylor_kernel<C64, BULK, XHOP>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   int(dyn_smem<C64, BULK>()));
        if (a != cudaSuccess) return a;
    }
    return cudaLaunchKernelEx(&cfg, taylor_kernel<C64, BULK, XHOP>, m, blk, nbr, cap, meta, v_in, res, ws, dt, m_star,
                              tol, out, status);
}

}  // namespace

int taylor_max_grid(bool c64, int num_sms) {
    int best = 0;
    for (int v = 0; v < 2; ++v)
        for (int x = 0; x < 2; ++x) {
            const int o = c64 ? occupancy_any<true>(v, x != 0) : occupancy_any<false>(v, x != 0);
            best = o > best ? o : best;
        }
    return num_sms * best;
}

int launch_taylor(bool c64, const ModelDev& m, const int* blk, const int* nbr, int64_t nbr_cap,
                  const uint32_t* meta, const void* v_in, void* res, double dt, int m_star,
                  double tol, const TaylorWs& ws, const TaylorOut& out, int* status, int num_sms,
                  int blocks_per_sm, int variant, cudaStream_t st) {
    if (m_star < 1 || variant < 0 || variant > 1) return PACES_ERR_BADARG;
    if (m.nhop > 1 && !m.xnbr) return PACES_ERR_BADARG;
    if (cudaMemsetAsync(ws.barrier, 0, kTaylorBarrierBytes, st) != cudaSuccess) return PACES_ERR_CUDA;
    const bool xhop = m.nhop > 1;
    const int occ = c64 ? occupancy_any<true>(variant, xhop) : occupancy_any<false>(variant, xhop);
    // a wave of blocks, or one block per 1024 rows of room in a small problem (fewer blocks at the
    // grid barriers, and at most two chunks each; the results do not depend on the grid)
    const int grid = grid_for(nbr_cap, 2 * kChunk, num_sms * (blocks_per_sm > 0 && blocks_per_sm < occ ? blocks_per_sm : occ));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kTThreads);
    cfg.dynamicSmemBytes = variant == 1 ? (c64 ? dyn_smem<true, true>() : dyn_smem<false, true>()) : 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int64_t cap = nbr_cap;
    cudaError_t e;
#define PACES_TAYLOR_ONE(C, B, X) launch_one<C, B, X>(cfg, m, blk, nbr, cap, meta, v_in, res, ws, dt, m_star, tol, out, status)
    if (c64) {
        if (xhop) e = variant == 1 ? PACES_TAYLOR_ONE(true, true, true) : PACES_TAYLOR_ONE(true, false, true);
        else e = variant == 1 ? PACES_TAYLOR_ONE(true, true, false) : PACES_TAYLOR_ONE(true, false, false);
    } else {
        if (xhop) e = variant == 1 ? PACES_TAYLOR_ONE(false, true, true) : PACES_TAYLOR_ONE(false, false, true);
        else e = variant == 1 ? PACES_TAYLOR_ONE(false, true, false) : PACES_TAYLOR_ONE(false, false, false);
    }
#undef PACES_TAYLOR_ONE
    return e == cudaSuccess ? PACES_OK : PACES_ERR_CUDA;
}

}  // namespace paces
