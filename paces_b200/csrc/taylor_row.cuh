// Row arithmetic and maxima shared by the Taylor kernels (single, batched).
#pragma once

#include "grid.cuh"
#include "hrow.cuh"
#include "kernels.cuh"

namespace paces {

constexpr int kStreamThreads = 256;  // threads per block of the kernels that stream rows
constexpr int kStreamWarps = kStreamThreads / 32;

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
    R nan;  // 0, or a NaN once an element was not finite
};

// Fold the block's maxima into g[0..3] (fp64 bit patterns; atomicMax is exact and order-free),
// pass the grid barrier and read the grid's maxima into fin[0..3] (shared; fin[4] is the
// barrier's success).  false on a timeout.
template <typename R>
__device__ __forceinline__ bool grid_max(const SweepMax<R>& mx, unsigned long long* g, double (*red)[kStreamWarps], double* fin,
                         const TaylorWs& ws, unsigned& gen, int* status) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const R a = warp_max(mx.term), b = warp_max(mx.res), c = warp_max(mx.v);
    const bool bad = __any_sync(0xffffffffu, mx.nan != R(0));
    if (lane == 0) {
        red[0][wid] = double(a);
        red[1][wid] = double(b);
        red[2][wid] = double(c);
        red[3][wid] = bad ? 1.0 : 0.0;
    }
    __syncthreads();
    if (wid == 0) {
        double r = 0.0;
        if (lane < 4)
            for (int w = 0; w < kStreamWarps; ++w) r = fmax(r, red[lane][w]);
        if (r > 0.0) atomicMax(g + lane, static_cast<unsigned long long>(__double_as_longlong(r)));
        __syncwarp();
        const bool ok = grid_barrier_warp(ws.barrier, gridDim.x, gen, status, ws.wait_ns, int(blockIdx.x) == ws.skip_block);
        if (lane < 4) fin[lane] = __longlong_as_double((long long)__ldcg(g + lane));
        if (lane == 4) fin[4] = ok ? 1.0 : 0.0;
    }
    ++gen;
    __syncthreads();
    return fin[4] != 0.0;
}

// Separate roundings (no contraction into an FMA), so
// that every kernel and schedule that runs these rows -- direct, streamed, batched -- rounds alike.
__device__ __forceinline__ float sq_abs(const float2& z) { return fmaf(z.x, z.x, __fmul_rn(z.y, z.y)); }
__device__ __forceinline__ double sq_abs(const double2& z) { return fma(z.x, z.x, __dmul_rn(z.y, z.y)); }
__device__ __forceinline__ float2 add_c(const float2& a, const float2& t) {
    return make_float2(__fadd_rn(a.x, t.x), __fadd_rn(a.y, t.y));
}
__device__ __forceinline__ double2 add_c(const double2& a, const double2& t) {
    return make_double2(__dadd_rn(a.x, t.x), __dadd_rn(a.y, t.y));
}
__device__ __forceinline__ float2 term_of(float c, const float2& y) {  // -i c y
    return make_float2(__fmul_rn(c, y.y), -__fmul_rn(c, y.x));
}
__device__ __forceinline__ double2 term_of(double c, const double2& y) {
    return make_double2(__dmul_rn(c, y.y), -__dmul_rn(c, y.x));
}
// 0 * z is a NaN exactly when z is not finite, and a NaN stays in the sum
__device__ __forceinline__ void note(float& nan, const float2& z) { nan = fmaf(z.x, 0.f, fmaf(z.y, 0.f, nan)); }
__device__ __forceinline__ void note(double& nan, const double2& z) { nan = fma(z.x, 0.0, fma(z.y, 0.0, nan)); }

template <int GEO, class P>
__device__ __forceinline__ float2 any_row(const P& m, const float* sq, int64_t r, const int4& nb, uint32_t mm,
                                          const float2& own, const float2* src) {
    if constexpr (GEO > 0) return h_row_c64_geo<GEO>(m, sq, r, nb, mm, own, src);
    else return h_row_c64_nb(m, sq, float(m.J), r, nb, mm, own, src);
}
template <int GEO, class P>
__device__ __forceinline__ double2 any_row(const P& m, const double* sq, int64_t r, const int4& nb, uint32_t mm,
                                           const double2& own, const double2* src) {
    if constexpr (GEO > 0) return h_row_c128_geo<GEO>(m, sq, r, nb, mm, own, src);
    else return h_row_c128_nb(m, sq, r, nb, mm, own, src);
}

// What a streaming sweep does beside its new term: SUM adds the last term and the new one to
// the sum; FIRST also takes the input's norm; FIRST_DIAG folds its diagnostics as well.
enum SweepKind : int { SW_TERM = 0, SW_SUM = 1, SW_FIRST = 2, SW_FIRST_DIAG = 3 };

// The neighbour rows and metadata of every warp's first unit, kept from the first sweep: a
// sweep's first gathers then start with the sweep.
struct FirstUnit {
    int4 nb[2 * kStreamThreads];
    uint32_t mm[2 * kStreamThreads];
};

// A warp's share of a sweep: 64-row units first, first + step, .. below `end` of a trajectory of
// `n` rows, two rows per lane; the next unit's neighbours, metadata, own elements and sums are
// on their way to registers while this unit's gathers wait on L2.  KEEP: the first unit's
// neighbours stay in `fu` from the FIRST sweep on.
template <bool C64, int GEO, int KIND, bool KEEP, class P, typename C = typename std::conditional<C64, float2, double2>::type,
          typename R = typename std::conditional<C64, float, double>::type>
__device__ __forceinline__ SweepMax<R> stream_rows(const P& m, const R* sq, const int* __restrict__ nbr,
                                                   const uint32_t* __restrict__ meta, const C* src, const C* rbase,
                                                   C* dst, C* res, R c, uint32_t first, uint32_t step, uint32_t end,
                                                   uint32_t n, double* diag, FirstUnit* fu) {
    constexpr bool kSum = KIND == SW_SUM, kFirst = KIND >= SW_FIRST, kDiag = KIND == SW_FIRST_DIAG;
    SweepMax<R> mx{R(0), R(0), R(0), R(0)};
    const uint32_t lane = threadIdx.x & 31u;
    struct Row {
        int4 nb;
        uint32_t mm;
        C own, a;
    };
    auto fetch = [&](uint32_t r, Row& w) {
        w.nb = ldcs_nbr(nbr, r);
        w.mm = __ldcs(meta + r);
        w.own = __ldcg(src + r);
        if constexpr (kSum) w.a = __ldcg(rbase + r);
    };
    auto finish = [&](uint32_t r, const C& y, const Row& w) {
        const C t = term_of(c, y);
        mx.term = fmax(mx.term, sq_abs(t));
        if constexpr (kSum) {
            const C prev = add_c(w.a, w.own), rr = add_c(prev, t);
            note(mx.nan, prev);
            note(mx.nan, rr);
            mx.res = fmax(mx.res, sq_abs(rr));
            res[r] = rr;
        } else {
            note(mx.nan, t);
            if constexpr (kFirst) {
                note(mx.nan, w.own);
                mx.v = fmax(mx.v, sq_abs(w.own));
            }
        }
        dst[r] = t;
    };
    uint32_t ub = first;  // the warp's unit
    Row w0{}, w1{};
    auto fetch_first = [&](uint32_t r, Row& w, uint32_t at) {  // a slot is its thread's own
        if (r >= n) return;
        if constexpr (!KEEP) {
            fetch(r, w);
        } else if constexpr (kFirst) {
            fetch(r, w);
            fu->nb[at] = w.nb;
            fu->mm[at] = w.mm;
        } else {
            w.nb = fu->nb[at];
            w.mm = fu->mm[at];
            w.own = __ldcg(src + r);
            if constexpr (kSum) w.a = __ldcg(rbase + r);
        }
    };
    if (ub < end) {
        fetch_first(ub + lane, w0, threadIdx.x);
        fetch_first(ub + lane + 32u, w1, threadIdx.x + kStreamThreads);
    }
    for (; ub < end; ub += step) {
        const uint32_t r0 = ub + lane, r1 = r0 + 32u;
        Row n0{}, n1{};
        if (ub + step < end) {
            if (r0 + step < n) fetch(r0 + step, n0);
            if (r1 + step < n) fetch(r1 + step, n1);
        }
        C y0{}, y1{};
        const bool v0 = r0 < n, v1 = r1 < n;
        if (v1) {  // then v0 too
            y0 = any_row<GEO>(m, sq, r0, w0.nb, w0.mm, w0.own, src);
            y1 = any_row<GEO>(m, sq, r1, w1.nb, w1.mm, w1.own, src);
            finish(r0, y0, w0);
            finish(r1, y1, w1);
        } else if (v0) {
            y0 = any_row<GEO>(m, sq, r0, w0.nb, w0.mm, w0.own, src);
            finish(r0, y0, w0);
        }
        if constexpr (kDiag) diag_group(diag, ub / kDiagGroup, v0, w0.own, y0, v1, w1.own, y1);
        w0 = n0;
        w1 = n1;
    }
    return mx;
}

// A ratio (term norms over the sum's norm) that may end the series, from a bound on the sum's
// norm: it lies within the last term's norm c2 of its last exact value (to a few roundings).
__device__ __forceinline__ bool may_end(double c1c2, double tol, double rnorm, double c2) {
    return c1c2 <= tol * (rnorm + c2) * 1.00001;
}

}  // namespace paces
