// Batched truncated-Taylor series: many independent trajectories (each its own basis, H,
// dt, model constants and stop test) advance through exp(-i dt H) psi in ONE persistent
// cooperative launch.
//
// Reference: _simple_taylor (paces/core/time_evolution.py:482-512) with total_ham
// (:382-400), run once per trajectory; the reference has no batching.
//
// Design.  The rows of all trajectories form one index space (trajectory t owns rows
// [off[t], off[t] + rows_t), computed on the device from every basis' blk[L] rounded up to a
// multiple of the 64-row unit, so the host never reads a size and no unit straddles two
// trajectories).  Each sweep goes over the units of the trajectories still running, every warp
// an equal, consecutive share of them, streamed as by the single-trajectory kernel
// (stream_rows).  Consecutive units mostly belong to one trajectory, so its pointers and
// constants are read once per share: with units dealt out one at a time, each unit's set-up
// through the parameters made a row cost 288 instructions per warp.  A trajectory's sum lags as there: a sweep either leaves it
// alone (TERM), adds the last term and the new one (SUM), or only adds the last term and
// measures the sum's norm (FIX) where the stop test needs it; every trajectory has its own
// term index and kind of sweep.  A warp folds the maxima of |term|^2, |res|^2, |v|^2 and a
// non-finite mark of a trajectory's part of its share into shared memory.  Rows 64 u + l and 64 u + 32 + l of a trajectory sit on lane l
// of its unit, as in the single-trajectory kernel's 64-row groups, so the first sweep folds
// the input's diagnostics (diag_group) exactly as that kernel does.  Blocks then fold into
// per-trajectory global maxima with atomicMax on the fp64 bit patterns (non-negative doubles
// order like their bits), which is exact and order-independent, so each trajectory's stop
// decision -- taken by every block from the same global maxima -- and its arithmetic are
// bit-identical to the single-trajectory kernel.  Three rotating maxima buffers let block 0
// clear the one for sweep s+2 after barrier s without racing the writers of sweep s+1.  A
// trajectory that converges, overflows or reaches its m_star leaves the sweep; the launch ends
// when none is left.
#include "grid.cuh"
#include "hrow.cuh"
#include "kernels.cuh"
#include "taylor_row.cuh"

namespace paces {

namespace {

constexpr int kBThreads = kStreamThreads;
constexpr int kBWarps = kBThreads / 32;
constexpr int kUnit = 64;

__device__ __forceinline__ unsigned long long dbits(double x) {
    return static_cast<unsigned long long>(__double_as_longlong(x));
}

enum BatchSweep : int { BS_TERM = 0, BS_SUM = 1, BS_FIX = 2 };

template <bool C64>
__global__ void __launch_bounds__(kBThreads, C64 ? 3 : 2)
taylor_batch_kernel(const __grid_constant__ TaylorBatch bt, TaylorBatchWs ws) {
    using C = typename std::conditional<C64, float2, double2>::type;
    using R = typename std::conditional<C64, float, double>::type;
    __shared__ long long s_unit[kMaxBatch + 1];  // first unit of each running trajectory
    __shared__ long long s_rows[kMaxBatch];
    __shared__ unsigned long long s_max[kMaxBatch][4];
    __shared__ double s_c1[kMaxBatch], s_c2[kMaxBatch], s_c1c2[kMaxBatch], s_ratio[kMaxBatch], s_cd[kMaxBatch],
        s_rnorm[kMaxBatch];
    __shared__ int s_j[kMaxBatch];
    __shared__ uint8_t s_kind[kMaxBatch], s_written[kMaxBatch];  // sweep kind; the sum is in res (else: the input)
    __shared__ uint8_t s_active[kMaxBatch];
    __shared__ int s_left;

    const int n = bt.n;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int i = tid; i < n; i += kBThreads) {
        const TaylorItem& I = bt.items[i];
        s_rows[i] = I.blk[I.L];
        s_active[i] = 1;
        s_c1[i] = s_c2[i] = s_c1c2[i] = s_ratio[i] = s_rnorm[i] = 0.0;
        s_j[i] = 0;
        s_cd[i] = I.dt;
        s_kind[i] = BS_TERM;
        s_written[i] = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) s_max[i][k] = 0ull;
    }
    __syncthreads();
    const long long gwarp = (long long)blockIdx.x * kBWarps + wid;
    const long long nwarps = (long long)gridDim.x * kBWarps;
    const unsigned nblocks = gridDim.x;
    unsigned gen = 0;

    auto emit = [&](int i, int conv) {
        const TaylorOut& o = bt.items[i].out;
        if (o.converged) *o.converged = conv;
        if (o.final_m) *o.final_m = s_j[i];
        if (o.c1_plus_c2) *o.c1_plus_c2 = s_c1c2[i];
        if (o.term_ratio) *o.term_ratio = s_ratio[i];
    };

    auto source = [&](const TaylorItem& I, int j) {  // of term j; the destination of term j - 1
        return reinterpret_cast<const C*>(j == 0 ? I.v_in : ((j & 1) ? I.ta : I.tb));
    };

    for (unsigned sweep = 0;; ++sweep) {
        // units of the running trajectories, in trajectory order
        if (wid == 0) {
            long long before = 0;
            for (int i0 = 0; i0 < n; i0 += 32) {
                const int i = i0 + lane;
                const long long own = i < n && s_active[i] ? (s_rows[i] + kUnit - 1) / kUnit : 0;
                long long incl = own;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const long long v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                if (i < n) s_unit[i] = before + incl - own;
                before += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) s_unit[n] = before;
        }
        __syncthreads();
        const long long units = s_unit[n];
        long long u = units * gwarp / nwarps;
        const long long u1 = units * (gwarp + 1) / nwarps;
        for (int it = 0; u < u1; ++it) {
            if (s_unit[it + 1] <= u) continue;
            const long long seg = min(u1, s_unit[it + 1]);  // this trajectory's part of the share
            const TaylorItem& I = bt.items[it];
            const int kind = s_kind[it], j = s_j[it];
            const uint32_t first = uint32_t(u - s_unit[it]) * kUnit, end = uint32_t(seg - s_unit[it]) * kUnit;
            const uint32_t nr = uint32_t(s_rows[it]);
            const R* sq;
            if constexpr (C64) sq = I.sqf;
            else sq = I.sq;
            const C* src = source(I, j);
            const C* rbase = reinterpret_cast<const C*>(s_written[it] ? I.res : I.v_in);
            C* dst = reinterpret_cast<C*>((j & 1) ? I.tb : I.ta);
            C* res = reinterpret_cast<C*>(I.res);
            const R c = R(s_cd[it]);
            SweepMax<R> mx{R(0), R(0), R(0), R(0)};
            if (kind == BS_FIX) {
                for (uint32_t r = first + lane; r < min(end, nr); r += 32u) {
                    const C rr = add_c(__ldcg(rbase + r), __ldcg(dst + r));
                    mx.res = fmax(mx.res, sq_abs(rr));
                    note(mx.nan, rr);
                    res[r] = rr;
                }
            } else if (kind == BS_SUM) {
                mx = stream_rows<C64, 0, SW_SUM, false>(I, sq, I.nbr, I.meta, src, rbase, dst, res, c, first, kUnit, end, nr,
                                                        nullptr, nullptr);
            } else if (j > 0) {
                mx = stream_rows<C64, 0, SW_TERM, false>(I, sq, I.nbr, I.meta, src, src, dst, res, c, first, kUnit, end, nr,
                                                         nullptr, nullptr);
            } else if (I.diag) {
                mx = stream_rows<C64, 0, SW_FIRST_DIAG, false>(I, sq, I.nbr, I.meta, src, src, dst, res, c, first, kUnit, end,
                                                               nr, I.diag, nullptr);
            } else {
                mx = stream_rows<C64, 0, SW_FIRST, false>(I, sq, I.nbr, I.meta, src, src, dst, res, c, first, kUnit, end, nr,
                                                          nullptr, nullptr);
            }
            const double m4[4] = {double(warp_max(mx.term)), double(warp_max(mx.res)), double(warp_max(mx.v)),
                                  __any_sync(0xffffffffu, mx.nan != R(0)) ? 1.0 : 0.0};
            if (lane == 0) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (m4[k] > 0.0) atomicMax(&s_max[it][k], dbits(m4[k]));
            }
            u = seg;
        }
        __syncthreads();
        unsigned long long* gmax = ws.maxima + size_t(sweep % 3) * kMaxBatch * 4;
        for (int e = tid; e < n * 4; e += kBThreads) {
            const unsigned long long v = s_max[e >> 2][e & 3];
            if (v) atomicMax(&gmax[e], v);
            s_max[e >> 2][e & 3] = 0ull;
        }
        if (!grid_barrier(ws.barrier, nblocks, gen, nullptr, ws.wait_ns, int(blockIdx.x) == ws.skip_block)) {
            for (int i = tid; i < n; i += kBThreads) {
                if (!s_active[i]) continue;
                raise_status(bt.items[i].status, PACES_ERR_TIMEOUT);
                if (blockIdx.x == 0) emit(i, 0);
                s_active[i] = 0;
            }
            break;
        }
        // every block takes the same per-trajectory decisions from the same maxima
        for (int i = tid; i < n; i += kBThreads) {
            if (!s_active[i]) continue;
            double g4[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) g4[k] = __longlong_as_double((long long)__ldcg(&gmax[i * 4 + k]));
            const TaylorItem& I = bt.items[i];
            if (g4[3] != 0.0) {
                if (blockIdx.x == 0) {
                    raise_status(I.status, PACES_ERR_NONFINITE);
                    emit(i, 0);
                }
                s_active[i] = 0;
                continue;
            }
            const int kind = s_kind[i], j = s_j[i];
            if (kind != BS_FIX) {
                if (j == 0) s_c1[i] = s_rnorm[i] = sqrt(g4[2]);
                s_c2[i] = sqrt(g4[0]);
                s_c1c2[i] = s_c1[i] + s_c2[i];
            }
            if (kind == BS_TERM) {
                if (j == I.m_star - 1 || may_end(s_c1c2[i], I.tol, s_rnorm[i], s_c2[i])) {
                    s_kind[i] = BS_FIX;
                    continue;
                }
                s_kind[i] = BS_SUM;
            } else {
                s_written[i] = 1;
                s_rnorm[i] = sqrt(g4[1]);
                s_ratio[i] = s_c1c2[i] / s_rnorm[i];
                if (s_ratio[i] <= I.tol || j == I.m_star - 1) {
                    if (blockIdx.x == 0) emit(i, s_ratio[i] <= I.tol ? 1 : 0);
                    s_active[i] = 0;
                    continue;
                }
                s_kind[i] = BS_TERM;
            }
            s_c1[i] = s_c2[i];
            s_j[i] = j + 1;
            s_cd[i] = I.dt / double(j + 2);
        }
        if (blockIdx.x == 0) {
            unsigned long long* clr = ws.maxima + size_t((sweep + 2) % 3) * kMaxBatch * 4;
            for (int e = tid; e < n * 4; e += kBThreads) clr[e] = 0ull;
        }
        if (tid == 0) s_left = 0;
        __syncthreads();
        for (int i = tid; i < n; i += kBThreads)
            if (s_active[i]) atomicAdd(&s_left, 1);
        __syncthreads();
        if (s_left == 0) break;
    }
}

template <bool C64>
int batch_occupancy() {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, taylor_batch_kernel<C64>, kBThreads, 0);
    return per_sm < 1 ? 1 : (per_sm > 8 ? 8 : per_sm);
}

}  // namespace

int taylor_batch_max_grid(bool c64, int num_sms) {
    return num_sms * (c64 ? batch_occupancy<true>() : batch_occupancy<false>());
}

int launch_taylor_batch(bool c64, const TaylorBatch& bt, const TaylorBatchWs& ws, int num_sms, int blocks_per_sm,
                        cudaStream_t st) {
    if (bt.n < 1 || bt.n > kMaxBatch || bt.max_m_star < 1) return PACES_ERR_BADARG;
    if (cudaMemsetAsync(ws.barrier, 0, kTaylorBatchWsBytes, st) != cudaSuccess) return PACES_ERR_CUDA;
    cudaLaunchConfig_t cfg = {};
    const int occ = c64 ? batch_occupancy<true>() : batch_occupancy<false>();
    cfg.gridDim = dim3(num_sms * (blocks_per_sm > 0 && blocks_per_sm < occ ? blocks_per_sm : occ));
    cfg.blockDim = dim3(kBThreads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = c64 ? cudaLaunchKernelEx(&cfg, taylor_batch_kernel<true>, bt, ws)
                        : cudaLaunchKernelEx(&cfg, taylor_batch_kernel<false>, bt, ws);
    return e == cudaSuccess ? PACES_OK : PACES_ERR_CUDA;
}

}  // namespace paces
