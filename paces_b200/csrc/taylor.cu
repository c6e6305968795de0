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
//  * direct: grid-stride, two rows per thread per pass, the sum updated in every sweep;
//  * stream: a warp takes 64-row units, two rows per lane, and loads the next unit's
//            neighbour rows, metadata, own elements and sums into registers while this
//            unit's gathers are waited for.  Loads in flight per thread are what the sweep
//            lives on: two rows per lane and 80 / 128 registers (three / two blocks per SM)
//            measured faster than one row and more blocks (complex64, 15.2M rows, 10 sweeps:
//            1.15 ms; one row at four blocks 1.27, five blocks 1.35), than chunks copied to
//            shared memory by bulk TMA copies (1.36), and than neighbours packed to 16-bit
//            offsets (1.29: fewer bytes, more instructions before a gather).  Shared memory
//            taken for chunks of small problems costs the L1 that holds the loads in flight
//            (73 KB a block: 1.18; keeping whole small problems there gained nothing).
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
#include "taylor_row.cuh"

namespace paces {

namespace {

constexpr int kTThreads = kStreamThreads;
constexpr int kTWarps = kTThreads / 32;

// GEO: 0 the chain, otherwise the dimensions of a lattice with several hopping channels (h_row_*_geo).
template <bool C64, bool STREAM, int GEO>
__global__ void __launch_bounds__(kTThreads, STREAM ? (C64 ? 3 : 2) : (C64 ? 4 : 3))
taylor_kernel(ModelDev m, const int* __restrict__ blk, const int* __restrict__ nbr,
              const uint32_t* __restrict__ meta, const void* v_in, void* res_out, TaylorWs ws,
              double dt, int m_star, double tol, TaylorOut out, int* status) {
    using C = typename std::conditional<C64, float2, double2>::type;
    using R = typename std::conditional<C64, float, double>::type;
    __shared__ R s_sq[260];
    __shared__ double s_red[4][kTWarps];
    __shared__ double s_fin[5];
    __shared__ FirstUnit s_fu;
    for (int k = threadIdx.x; k < 260; k += kTThreads) s_sq[k] = R(__dmul_rn(sqrt(double(k)), m.g));
    __syncthreads();

    const int64_t S = blk[m.L];
    unsigned gen = 0;
    const C* v = reinterpret_cast<const C*>(v_in);
    C* res = reinterpret_cast<C*>(res_out);
    C* ta = reinterpret_cast<C*>(ws.ta);
    C* tb = reinterpret_cast<C*>(ws.tb);
    double c1 = 0.0, c1c2 = 0.0, ratio = 0.0;
    int conv = 0, fin_j = 0;

    // streaming: the sum lags one term behind (see the head of this file)
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
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // streaming: the warp's first unit and the rows from one of its units to the next
    const uint32_t first = (blockIdx.x * uint32_t(kTWarps) + wid) * uint32_t(kDiagGroup);
    const uint32_t step = gridDim.x * uint32_t(kTWarps * kDiagGroup);

    for (int j = 0; j < m_star; ++j) {
        const C* src = j == 0 ? v : ((j & 1) ? ta : tb);
        C* dst = (j & 1) ? tb : ta;
        const double cd = dt / double(j + 1);
        const R c = R(cd);
        SweepMax<R> mx{R(0), R(0), R(0), R(0)};
        auto hrow = [&](int64_t r) -> C {
            return any_row<GEO>(m, s_sq, r, load_nbr(nbr, r), __ldg(meta + r), __ldcg(src + r), src);
        };
        // the row's new term; the sum with it
        auto finish = [&](const C& y, const C& a, C& t) -> C {
            t = term_of(c, y);
            const C rr = add_c(a, t);
            mx.term = fmax(mx.term, sq_abs(t));
            mx.res = fmax(mx.res, sq_abs(rr));
            if (j == 0) mx.v = fmax(mx.v, sq_abs(a));
            note(mx.nan, rr);
            return rr;
        };
        const bool diag = j == 0 && ws.diag != nullptr;  // first sweep: fold the input's diagnostics
        bool exact = true;  // this sweep brings the sum and its norm up to date
        if constexpr (!STREAM) {
            const C* rin = j == 0 ? v : res;
            auto store = [&](int64_t r, const C& y, const C& a) {
                C t;
                res[r] = finish(y, a, t);
                dst[r] = t;
            };
            // two rows per thread per pass: all loads of both rows precede the stores
            const int64_t stride = int64_t(gridDim.x) * kTThreads;
            if (!diag) {
                int64_t r = int64_t(blockIdx.x) * kTThreads + threadIdx.x;
                for (; r + stride < S; r += 2 * stride) {
                    const C y0 = hrow(r), y1 = hrow(r + stride);
                    const C a0 = rin[r], a1 = rin[r + stride];
                    store(r, y0, a0);
                    store(r + stride, y1, a1);
                }
                if (r < S) store(r, hrow(r), rin[r]);
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
                    if (v0) store(r0, y0, a0);
                    if (v1) store(r1, y1, a1);
                    diag_group(ws.diag, ub / kDiagGroup, v0, a0, y0, v1, a1, y1);
                }
            }
        } else {
            exact = lag;
            if (j == 0) {
                if (ws.diag) mx = stream_rows<C64, GEO, SW_FIRST_DIAG, true>(m, s_sq, nbr, meta, src, src, dst, res, R(cd), first, step, uint32_t(S), uint32_t(S), ws.diag, &s_fu);
                else mx = stream_rows<C64, GEO, SW_FIRST, true>(m, s_sq, nbr, meta, src, src, dst, res, R(cd), first, step, uint32_t(S), uint32_t(S), nullptr, &s_fu);
            } else if (lag) {
                mx = stream_rows<C64, GEO, SW_SUM, true>(m, s_sq, nbr, meta, src, rbase, dst, res, R(cd), first, step, uint32_t(S), uint32_t(S), nullptr, &s_fu);
            } else {
                mx = stream_rows<C64, GEO, SW_TERM, true>(m, s_sq, nbr, meta, src, src, dst, res, R(cd), first, step, uint32_t(S), uint32_t(S), nullptr, &s_fu);
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
            // only a ratio that may end the series, or the series' last, needs the sum's exact norm
            if (j == m_star - 1 || may_end(c1c2, tol, rnorm, c2)) {
                mx = SweepMax<R>{R(0), R(0), R(0), R(0)};
                const int64_t stride = int64_t(gridDim.x) * kTThreads;
#pragma unroll 2
                for (int64_t r = int64_t(blockIdx.x) * kTThreads + threadIdx.x; r < S; r += stride) {
                    const C rr = add_c(__ldcg(rbase + r), __ldcg(dst + r));
                    mx.res = fmax(mx.res, sq_abs(rr));
                    note(mx.nan, rr);
                    res[r] = rr;
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
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (out.converged) *out.converged = conv;
        if (out.final_m) *out.final_m = fin_j;
        if (out.c1_plus_c2) *out.c1_plus_c2 = c1c2;
        if (out.term_ratio) *out.term_ratio = ratio;
    }
}

template <bool C64, bool STREAM, int GEO>
int occupancy() {
    static int cached = 0;  // per process: the kernels' resources do not change
    if (cached) return cached;
    auto kfn = taylor_kernel<C64, STREAM, GEO>;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, kTThreads, 0);
    cached = per_sm < 1 ? 1 : (per_sm > 8 ? 8 : per_sm);
    return cached;
}

// Blocks per SM of the instance for a schedule and a lattice (geo 0: the chain).
template <bool C64, bool STREAM>
int occupancy_geo(int geo) {
    return geo == 0 ? occupancy<C64, STREAM, 0>() : (geo == 1 ? occupancy<C64, STREAM, 1>()
                                                  : (geo == 2 ? occupancy<C64, STREAM, 2>() : occupancy<C64, STREAM, 3>()));
}
int occupancy_any(bool c64, int variant, int geo) {
    if (c64) return variant == 1 ? occupancy_geo<true, true>(geo) : occupancy_geo<true, false>(geo);
    return variant == 1 ? occupancy_geo<false, true>(geo) : occupancy_geo<false, false>(geo);
}

template <bool C64, bool STREAM, int GEO>
cudaError_t launch_one(const cudaLaunchConfig_t& cfg, const ModelDev& m, const int* blk, const int* nbr,
                       const uint32_t* meta, const void* v_in, void* res, const TaylorWs& ws, double dt, int m_star,
                       double tol, const TaylorOut& out, int* status) {
    return cudaLaunchKernelEx(&cfg, taylor_kernel<C64, STREAM, GEO>, m, blk, nbr, meta, v_in, res, ws, dt, m_star,
                              tol, out, status);
}

}  // namespace

int taylor_max_grid(bool c64, int num_sms) {
    int best = 0;
    for (int v = 0; v < 2; ++v)
        for (int geo = 0; geo <= 3; ++geo) {
            const int o = occupancy_any(c64, v, geo);
            best = o > best ? o : best;
        }
    return num_sms * best;
}

int launch_taylor(bool c64, const ModelDev& m, const int* blk, const int* nbr, int64_t nbr_cap,
                  const uint32_t* meta, const void* v_in, void* res, double dt, int m_star,
                  double tol, const TaylorWs& ws, const TaylorOut& out, int* status, int num_sms,
                  int blocks_per_sm, int variant, cudaStream_t st, bool cleared) {
    if (m_star < 1 || variant < 0 || variant > 1) return PACES_ERR_BADARG;
    if (m.nhop > 1 && !m.xnbr) return PACES_ERR_BADARG;
    if (!cleared && cudaMemsetAsync(ws.barrier, 0, kTaylorBarrierBytes, st) != cudaSuccess) return PACES_ERR_CUDA;
    const int geo = m.nhop > 1 ? m.hop_n[0] >> 1 : 0;
    const int occ = occupancy_any(c64, variant, geo);
    // a wave of blocks, or one block per 512 rows of room in a small problem (fewer blocks at the
    // grid barriers; the results do not depend on the grid)
    const int grid = grid_for(nbr_cap, kTThreads * 2, num_sms * (blocks_per_sm > 0 && blocks_per_sm < occ ? blocks_per_sm : occ));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kTThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e;
#define PACES_TAYLOR_ONE(C, B, G) \
    launch_one<C, B, G>(cfg, m, blk, nbr, meta, v_in, res, ws, dt, m_star, tol, out, status)
#define PACES_TAYLOR_GEO(C, B)                                             \
    (geo == 0 ? PACES_TAYLOR_ONE(C, B, 0)                                  \
              : (geo == 1 ? PACES_TAYLOR_ONE(C, B, 1)                      \
                          : (geo == 2 ? PACES_TAYLOR_ONE(C, B, 2) : PACES_TAYLOR_ONE(C, B, 3))))
    if (c64) e = variant == 1 ? PACES_TAYLOR_GEO(true, true) : PACES_TAYLOR_GEO(true, false);
    else e = variant == 1 ? PACES_TAYLOR_GEO(false, true) : PACES_TAYLOR_GEO(false, false);
#undef PACES_TAYLOR_GEO
#undef PACES_TAYLOR_ONE
    return e == cudaSuccess ? PACES_OK : PACES_ERR_CUDA;
}

}  // namespace paces
