// Krylov (Lanczos) exp(-i dt H) psi as one persistent cooperative kernel.
//
// Reference: _lanczos (paces/core/time_evolution.py:515-549), selected by
// ExpmParams.lanczos_order = m > 0 (:577-578).  From q_0 = psi / |psi| the plain Lanczos
// recurrence (no re-orthogonalisation) builds m+1 vectors:
//   w = H q_i - beta_i q_{i-1},  alpha_i = vdot(w, q_i) (complex),  w -= alpha_i q_i,
//   beta_{i+1} = |w|  (stop when beta < 1e-15),  q_{i+1} = w / beta_{i+1};
// the (m+1)^2 tridiagonal T = tridiag(beta, alpha, beta) is exponentiated densely
// (scipy/cupyx expm) and psi(t + dt) = |psi| V exp(-i dt T) e_0.  The diagnostics are the
// reference's placeholder [False, 0, 0, 0].  The reference makes one host round trip per
// vector (norms, vdot) and a dense expm on the device.
//
// B200 design: the whole recurrence is one launch.  Per Krylov vector two grid-stride
// sweeps, each closed by a bounded grid barrier:
//   A_i  q_i = s_i / beta_i and (H q_i)_r = (H s_i)_r / beta_i from the unnormalised column s_i
//        (s_0 = psi; gathered through the neighbour table, as in the Taylor kernel), stores
//        w = H q_i - beta_i q_{i-1} as column i + 1; partial vdot(w, q_i);
//   B_i  w -= alpha_i q_i in place, which makes it s_{i+1}; partial |w|^2.
// The columns stay unnormalised: q_i = s_i (1 / beta_i) is one rounding of what is read anyway,
// and storing it as well cost a vector written per A sweep.  A warp takes rows in units of 64, two
// per lane, and the next unit's loads are under way while this unit's gathers wait on L2.
// (A sweep that stored q_i and w, rows a grid stride apart, loads of the next row only after
// this one's gathers: 337 us for 13 vectors of 825K complex128 rows; 270 now, with the sums and the
// small exponential below.)
// The partial sums are fp64 (complex64 vectors too) and every block adds the per-block
// partials in the same order, so all blocks hold bit-identical alpha and beta and take the
// same stop decision.  After the recurrence every block computes the first column of
// exp(-i dt T) itself in fp64 (below), and a last sweep forms |psi| sum_i c_i q_i.
//
// The small exponential: x = exp(A) e_0 for A = -i dt T by the truncated Taylor series with
// s sub-steps, x <- sum_j (A/s)^j x / j!, s = ceil(|A|_1) so every sub-step has |A/s|_1 <= 1
// -- the stepping of Al-Mohy and Higham, "Computing the action of the matrix exponential"
// (SIAM J. Sci. Comput. 33, 2011), with the stop test of the plain Taylor path (two
// consecutive terms below 2^-53 of the sum in the inf-norm).  T is tridiagonal, so each
// term costs O(m); one warp computes it, two rows per lane.
#include "grid.cuh"
#include "kernels.cuh"
#include "taylor_row.cuh"

namespace paces {

namespace {

constexpr int kLThreads = 256;
constexpr int kLWarps = kLThreads / 32;
constexpr int kKrylovMax = kMaxLanczosOrder + 1;  // vectors
static_assert(kKrylovMax <= 64, "the small exponential holds two rows per lane of one warp");

// Grid-wide sum of NV doubles: the warps' sums through shared memory, then one warp alone adds
// them, publishes the block's partial in ws.partials[parity], passes the barrier and adds all
// blocks' partials -- in the same order in every block, so the sums agree in every bit.  The
// result is in fin[0..NV) for every thread; false when the barrier timed out.  (With the partials
// added by the whole block, two more block barriers a sum: 9 us more of a launch of 12 vectors.)
template <int NV>
__device__ bool grid_sum(double v[NV], const LanczosWs& ws, int parity, unsigned& gen, int* status,
                         double (*red)[kLWarps], double* fin) {
    __shared__ int s_ok;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    auto warp_sum = [](double x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return x;
    };
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const double x = warp_sum(v[k]);
        if (lane == 0) red[k][wid] = x;
    }
    __syncthreads();
    if (wid == 0) {
        double* part = ws.partials + size_t(parity) * ws.max_grid * 4;
        const unsigned nblocks = gridDim.x;
        if (lane < NV) {
            double r = 0.0;
            for (int w = 0; w < kLWarps; ++w) r += red[lane][w];
            part[size_t(blockIdx.x) * 4 + lane] = r;
        }
        __syncwarp();
        const bool ok = grid_barrier_warp(ws.barrier, nblocks, gen, status, ws.wait_ns, int(blockIdx.x) == ws.skip_block);
        if (ok) {
            double g[NV];
#pragma unroll
            for (int k = 0; k < NV; ++k) g[k] = 0.0;
            constexpr int kFly = 10;  // blocks per lane and round, their loads in flight together
            for (unsigned b0 = lane; b0 < nblocks; b0 += 32 * kFly) {
                double x[kFly][NV];
#pragma unroll
                for (int u = 0; u < kFly; ++u) {
                    const unsigned b = b0 + 32 * u;
#pragma unroll
                    for (int k = 0; k < NV; ++k) x[u][k] = b < nblocks ? __ldcg(part + size_t(b) * 4 + k) : 0.0;
                }
#pragma unroll
                for (int u = 0; u < kFly; ++u) {
#pragma unroll
                    for (int k = 0; k < NV; ++k) g[k] += x[u][k];
                }
            }
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const double x = warp_sum(g[k]);
                if (lane == 0) fin[k] = x;
            }
        }
        if (lane == 0) s_ok = ok ? 1 : 0;
    }
    ++gen;
    __syncthreads();
    return s_ok != 0;
}

// First column of exp(-i dt T), T = tridiag(beta[1..k-1], alpha[0..k-1], beta[1..k-1]),
// into (lre, lim); warp 0 of the block, fp64.  A chain of short dependent steps on one warp: rows
// l and l + 32 live in lane l's registers, a step's neighbours come by shuffles, the norms from
// the squares.  (Rows in shared memory and hypot took 60K cycles for 13 vectors, 32 us of a
// launch; now 23K.)
__device__ void small_expm_col0(int k, double dt, const double* are, const double* aim, const double* beta,
                                double* lre, double* lim) {
    const int lane = threadIdx.x;  // warp 0 only
    double ar[2], ai[2], lo[2], hi[2], xr[2], xi[2];  // alpha, the couplings to r - 1 and r + 1, the sum
    double a1 = 0.0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = lane + 32 * h;
        const bool in = r < k;
        ar[h] = in ? are[r] : 0.0;
        ai[h] = in ? aim[r] : 0.0;
        lo[h] = in && r >= 1 ? beta[r] : 0.0;
        hi[h] = in && r + 1 < k ? beta[r + 1] : 0.0;
        xr[h] = r == 0 ? 1.0 : 0.0;
        xi[h] = 0.0;
        a1 = fmax(a1, dt * (hypot(ar[h], ai[h]) + lo[h] + hi[h]));
    }
    a1 = warp_max(a1);
    const int s = a1 > 1.0 ? int(ceil(a1)) : 1;
    // from the squares: a term so small that its square underflows is far below the stop test's
    // tolerance, and sums stay near one
    auto norm2 = [&](const double* vr, const double* vi) {
        return warp_max(fmax(fma(vr[0], vr[0], vi[0] * vi[0]), fma(vr[1], vr[1], vi[1] * vi[1])));
    };
    // element r - 1 or r + 1 of a vector held two per lane
    auto below_of = [&](const double* v, double* o) {
        const double e = __shfl_sync(0xffffffffu, v[0], 31);
        o[0] = __shfl_up_sync(0xffffffffu, v[0], 1);
        o[1] = __shfl_up_sync(0xffffffffu, v[1], 1);
        if (lane == 0) o[1] = e;
    };
    auto above_of = [&](const double* v, double* o) {
        const double e = __shfl_sync(0xffffffffu, v[1], 0);
        o[0] = __shfl_down_sync(0xffffffffu, v[0], 1);
        o[1] = __shfl_down_sync(0xffffffffu, v[1], 1);
        if (lane == 31) o[0] = e;
    };
    double coef[3];  // dt / (s j) for j = lane + 1, + 33, + 65
#pragma unroll
    for (int q = 0; q < 3; ++q) coef[q] = dt / (double(s) * double(lane + 1 + 32 * q));
    for (int step = 0; step < s; ++step) {
        double tr[2] = {xr[0], xr[1]}, ti[2] = {xi[0], xi[1]};
        double c1 = sqrt(norm2(tr, ti));
        for (int j = 1; j <= 80; ++j) {
            const int q = (j - 1) >> 5;
            const double c = __shfl_sync(0xffffffffu, q == 0 ? coef[0] : (q == 1 ? coef[1] : coef[2]), (j - 1) & 31);
            // new term = -i c T term
            double dr[2], di[2], ur[2], ui[2];
            below_of(tr, dr);
            below_of(ti, di);
            above_of(tr, ur);
            above_of(ti, ui);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const double yr = ar[h] * tr[h] - ai[h] * ti[h] + lo[h] * dr[h] + hi[h] * ur[h];
                const double yi = ar[h] * ti[h] + ai[h] * tr[h] + lo[h] * di[h] + hi[h] * ui[h];
                tr[h] = c * yi;
                ti[h] = -c * yr;
                xr[h] += tr[h];
                xi[h] += ti[h];
            }
            const double c2 = sqrt(norm2(tr, ti)), f = sqrt(norm2(xr, xi));
            if (c1 + c2 <= 1.1102230246251565e-16 * f) break;
            c1 = c2;
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (lane + 32 * h < k) {
            lre[lane + 32 * h] = xr[h];
            lim[lane + 32 * h] = xi[h];
        }
    }
}

template <bool C64, bool XHOP>
__global__ void __launch_bounds__(kLThreads, C64 ? 3 : 2)
lanczos_kernel(ModelDev m, const int* __restrict__ blk, const int* __restrict__ nbr, const uint32_t* __restrict__ meta,
               const void* v_in, void* res_out, LanczosWs ws, double dt, int order, TaylorOut out, int* status) {
    using C = typename std::conditional<C64, float2, double2>::type;
    using R = typename std::conditional<C64, float, double>::type;
    __shared__ R s_sq[260];
    __shared__ double s_red[4][kLWarps];
    __shared__ double s_fin[4];
    __shared__ double s_are[kKrylovMax], s_aim[kKrylovMax], s_beta[kKrylovMax + 1];
    __shared__ R s_rb[kKrylovMax];  // 1 / the norm of column i
    __shared__ double s_lre[kKrylovMax], s_lim[kKrylovMax];
    for (int k = threadIdx.x; k < 260; k += kLThreads) s_sq[k] = R(__dmul_rn(sqrt(double(k)), m.g));
    for (int k = threadIdx.x; k <= kKrylovMax; k += kLThreads) s_beta[k] = 0.0;
    __syncthreads();

    const int64_t S = blk[m.L];
    const int64_t cap = ws.cap;
    // this warp's units of 64 rows, lane l their rows l and l + 32
    const int64_t step = int64_t(gridDim.x) * kLWarps * 64;
    const int64_t r0 = (int64_t(blockIdx.x) * kLWarps + (threadIdx.x >> 5)) * 64 + (threadIdx.x & 31);
    const C* v = reinterpret_cast<const C*>(v_in);
    C* res = reinterpret_cast<C*>(res_out);
    C* U = reinterpret_cast<C*>(ws.u);
    auto column = [&](int i) -> const C* { return i == 0 ? v : U + int64_t(i - 1) * cap; };
    const R J = R(m.J);
    unsigned gen = 0;
    int parity = 0;
    bool ok = true;
    auto scaled = [](const C& x, R b) -> C {  // q from its column
        C q;
        if constexpr (C64) q = make_float2(__fmul_rn(x.x, b), __fmul_rn(x.y, b));
        else q = make_double2(__dmul_rn(x.x, b), __dmul_rn(x.y, b));
        return q;
    };

    // |psi|
    double nv[1] = {0.0};
    for (int64_t r = r0; r < S; r += step) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (r + 32 * u >= S) continue;
            const C x = v[r + 32 * u];
            nv[0] += double(x.x) * double(x.x) + double(x.y) * double(x.y);
        }
    }
    ok = grid_sum<1>(nv, ws, parity, gen, status, s_red, s_fin);
    parity ^= 1;
    const double nrm = sqrt(s_fin[0]);
    if (ok && !(nrm > 0.0 && nrm <= 1.7976931348623157e308)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) raise_status(status, PACES_ERR_NONFINITE);
        ok = false;
    }
    int k = 0;             // Krylov vectors built
    double beta = nrm;     // norm of the column of the next A sweep
    R rp = R(0);           // 1 / the norm of the column before it
    for (int i = 0; ok && i <= order; ++i) {
        // A_i
        const C* src = column(i);
        const C* sp = i > 0 ? column(i - 1) : nullptr;
        C* w = i < order ? U + int64_t(i) * cap : nullptr;  // the last vector has no successor
        const R bi = R(i > 0 ? s_beta[i] : 0.0);
        const R rb = R(1.0 / beta);
        double pa[2] = {0.0, 0.0};
        struct Row {
            int4 nb;
            uint32_t mm;
            C own, prev;
        };
        auto fetch = [&](int64_t r, Row& x) {
            if (r >= S) return;
            x.nb = load_nbr(nbr, r);
            x.mm = __ldg(meta + r);
            x.own = __ldcg(src + r);
            if (sp) x.prev = __ldcg(sp + r);
        };
        auto h_row = [&](int64_t r, const Row& x) -> C {
            if constexpr (XHOP) {
                if constexpr (C64) return h_row_c64_x(m, s_sq, r, x.nb, x.mm, x.own, src);
                else return h_row_c128_x(m, s_sq, r, x.nb, x.mm, x.own, src);
            } else {
                if constexpr (C64) return h_row_c64_nb(m, s_sq, J, r, x.nb, x.mm, x.own, src);
                else return h_row_c128_nb(m, s_sq, r, x.nb, x.mm, x.own, src);
            }
        };
        // w_r = (H s)_r / beta - beta_i q_{i-1,r}; the vdot partial
        auto finish_row = [&](int64_t r, const C& y, const Row& x) {
            const C q = scaled(x.own, rb), p = scaled(x.prev, rp);
            C wr = scaled(y, rb);
            if constexpr (C64) {
                wr.x = fmaf(-bi, p.x, wr.x);
                wr.y = fmaf(-bi, p.y, wr.y);
            } else {
                wr = make_double2(__dsub_rn(wr.x, __dmul_rn(bi, p.x)), __dsub_rn(wr.y, __dmul_rn(bi, p.y)));
            }
            if (w) w[r] = wr;
            // vdot(w, q) = sum conj(w) q
            pa[0] += double(wr.x) * double(q.x) + double(wr.y) * double(q.y);
            pa[1] += double(wr.x) * double(q.y) - double(wr.y) * double(q.x);
        };
        {
            Row w0{}, w1{};
            fetch(r0, w0);
            fetch(r0 + 32, w1);
            for (int64_t r = r0; r < S; r += step) {
                Row n0{}, n1{};
                fetch(r + step, n0);
                fetch(r + step + 32, n1);
                if (r + 32 < S) {
                    const C y0 = h_row(r, w0), y1 = h_row(r + 32, w1);
                    finish_row(r, y0, w0);
                    finish_row(r + 32, y1, w1);
                } else {
                    finish_row(r, h_row(r, w0), w0);
                }
                w0 = n0;
                w1 = n1;
            }
        }
        if (!grid_sum<2>(pa, ws, parity, gen, status, s_red, s_fin)) {
            ok = false;
            break;
        }
        parity ^= 1;
        const double are = s_fin[0], aim = s_fin[1];
        if (!(isfinite(are) && isfinite(aim))) {
            if (blockIdx.x == 0 && threadIdx.x == 0) raise_status(status, PACES_ERR_NONFINITE);
            ok = false;
            break;
        }
        if (threadIdx.x == 0) {
            s_are[i] = are;
            s_aim[i] = aim;
            s_rb[i] = rb;
        }
        k = i + 1;
        if (i == order) break;
        // B_i
        double pb[1] = {0.0};
        auto axpy_row = [&](int64_t r, const C& x, C wr) {
            const C q = scaled(x, rb);
            if constexpr (C64) {
                const float ar = float(are), ai = float(aim);
                wr.x -= ar * q.x - ai * q.y;
                wr.y -= ar * q.y + ai * q.x;
            } else {
                const double px = __dsub_rn(__dmul_rn(are, q.x), __dmul_rn(aim, q.y));
                const double py = __dadd_rn(__dmul_rn(are, q.y), __dmul_rn(aim, q.x));
                wr = make_double2(__dsub_rn(wr.x, px), __dsub_rn(wr.y, py));
            }
            w[r] = wr;
            pb[0] += double(wr.x) * double(wr.x) + double(wr.y) * double(wr.y);
        };
        {
            auto get = [&](int64_t r, C& x, C& wr) {
                if (r >= S) return;
                x = __ldcg(src + r);
                wr = __ldcg(w + r);
            };
            C x0{}, x1{}, w0{}, w1{};
            get(r0, x0, w0);
            get(r0 + 32, x1, w1);
            for (int64_t r = r0; r < S; r += step) {
                C nx0{}, nx1{}, nw0{}, nw1{};
                get(r + step, nx0, nw0);
                get(r + step + 32, nx1, nw1);
                axpy_row(r, x0, w0);
                if (r + 32 < S) axpy_row(r + 32, x1, w1);
                x0 = nx0;
                x1 = nx1;
                w0 = nw0;
                w1 = nw1;
            }
        }
        if (!grid_sum<1>(pb, ws, parity, gen, status, s_red, s_fin)) {
            ok = false;
            break;
        }
        parity ^= 1;
        const double bnext = sqrt(s_fin[0]);
        if (!(bnext <= 1.7976931348623157e308)) {
            if (blockIdx.x == 0 && threadIdx.x == 0) raise_status(status, PACES_ERR_NONFINITE);
            ok = false;
            break;
        }
        if (bnext < 1e-15) break;  // the Krylov space is invariant: k vectors
        if (threadIdx.x == 0) s_beta[i + 1] = bnext;
        __syncthreads();
        rp = rb;
        beta = bnext;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (out.converged) *out.converged = 0;
        if (out.final_m) *out.final_m = 0;
        if (out.c1_plus_c2) *out.c1_plus_c2 = 0.0;
        if (out.term_ratio) *out.term_ratio = 0.0;
    }
    if (!ok) return;
    __syncthreads();
    if (threadIdx.x < 32) small_expm_col0(k, dt, s_are, s_aim, s_beta, s_lre, s_lim);
    __syncthreads();
    // psi(t + dt) = |psi| sum_i c_i q_i
    bool finite = true;
    for (int64_t r = r0; r < S; r += step) {
        constexpr int kCols = 4;  // of both rows' columns, loads in flight together
        const bool two = r + 32 < S;
        double fr[2] = {0.0, 0.0}, fi[2] = {0.0, 0.0};
        for (int i0 = 0; i0 < k; i0 += kCols) {
            C x[kCols][2];
#pragma unroll
            for (int u = 0; u < kCols; ++u) {
                if (i0 + u >= k) continue;
                const C* col = column(i0 + u);
                x[u][0] = __ldcg(col + r);
                if (two) x[u][1] = __ldcg(col + r + 32);
            }
#pragma unroll
            for (int u = 0; u < kCols; ++u) {
                if (i0 + u >= k) continue;
                const int i = i0 + u;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const C q = scaled(x[u][h], s_rb[i]);
                    fr[h] += s_lre[i] * double(q.x) - s_lim[i] * double(q.y);
                    fi[h] += s_lre[i] * double(q.y) + s_lim[i] * double(q.x);
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (h == 1 && !two) continue;
            const double re = fr[h] * nrm, im = fi[h] * nrm;
            if (!(isfinite(re) && isfinite(im))) finite = false;
            if constexpr (C64) res[r + 32 * h] = make_float2(float(re), float(im));
            else res[r + 32 * h] = make_double2(re, im);
        }
    }
    if (!finite) raise_status(status, PACES_ERR_NONFINITE);
}

template <bool C64, bool XHOP>
int lanczos_occupancy() {
    static int cached = 0;  // per process: the kernel's resources do not change
    if (cached) return cached;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lanczos_kernel<C64, XHOP>, kLThreads, 0);
    cached = per_sm < 1 ? 1 : (per_sm > 8 ? 8 : per_sm);
    return cached;
}

}  // namespace

int lanczos_max_grid(int num_sms) {
    int best = lanczos_occupancy<true, false>();
    const int o[3] = {lanczos_occupancy<true, true>(), lanczos_occupancy<false, false>(),
                      lanczos_occupancy<false, true>()};
    for (int x : o) best = x > best ? x : best;
    return num_sms * best;
}

int launch_lanczos(bool c64, const ModelDev& m, const int* blk, const int* nbr, const uint32_t* meta,
                   const void* v_in, void* res, double dt, int order, const LanczosWs& ws, const TaylorOut& out,
                   int* status, int num_sms, cudaStream_t st) {
    if (order < 1 || order > kMaxLanczosOrder) return PACES_ERR_BADARG;
    if (m.nhop > 1 && !m.xnbr) return PACES_ERR_BADARG;
    if (cudaMemsetAsync(ws.barrier, 0, 2 * sizeof(unsigned), st) != cudaSuccess) return PACES_ERR_CUDA;
    const bool xhop = m.nhop > 1;
    const int occ = c64 ? (xhop ? lanczos_occupancy<true, true>() : lanczos_occupancy<true, false>())
                        : (xhop ? lanczos_occupancy<false, true>() : lanczos_occupancy<false, false>());
    // a fixed wave: the fp64 partial sums (and so alpha, beta) do not depend on buffer sizes
    int grid = num_sms * occ;
    if (grid > ws.max_grid) grid = ws.max_grid;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kLThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e;
    if (c64) {
        e = xhop ? cudaLaunchKernelEx(&cfg, lanczos_kernel<true, true>, m, blk, nbr, meta, v_in, res, ws, dt, order, out, status)
                 : cudaLaunchKernelEx(&cfg, lanczos_kernel<true, false>, m, blk, nbr, meta, v_in, res, ws, dt, order, out, status);
    } else {
        e = xhop ? cudaLaunchKernelEx(&cfg, lanczos_kernel<false, true>, m, blk, nbr, meta, v_in, res, ws, dt, order, out, status)
                 : cudaLaunchKernelEx(&cfg, lanczos_kernel<false, false>, m, blk, nbr, meta, v_in, res, ws, dt, order, out, status);
    }
    return e == cudaSuccess ? PACES_OK : PACES_ERR_CUDA;
}

}  // namespace paces
