// One row of H applied to a vector, from the neighbour table (one int4 per row: left,
// right, one phonon less, one phonon more; -1 = absent) and the row metadata.
//
// Reference: total_ham (paces/core/time_evolution.py:382-400) computes
//   diag * v + hopping_csr.dot(v) + vib_coupling_csr.dot(v)
// with CSR rows summed in increasing column order and float64 matrix elements
// J (hopping, paces/models/holstein.py:205-206) and g*sqrt(n) (vibronic coupling,
// holstein.py:271-274).  The complex128 form below keeps exactly that grouping and
// rounds every product and sum separately (no fused multiply-add), so it reproduces
// the reference arithmetic row by row.
//
// The rows are branch-free, so the five loads of a row -- and of several rows handled by one
// thread -- are in flight together.  An absent neighbour is a load left out by its predicate
// (see `neighbour`); complex64 chains and couplings re-read the row's own element instead,
// already in flight, under a zero coefficient.
#pragma once

#include "common.cuh"

namespace paces {

// Diagonal element from the row metadata (paces/models/holstein.py:280-287).  `P` is the
// model (ModelDev) or a batched trajectory's parameters: any type with eps_sys,
// hbar_omega, delta_eps, has_site_eps, site_eps[] and J.
template <class P>
__device__ __forceinline__ double diag_value(const P& m, uint32_t meta) {
    const int pos = int(meta & 0xffu);
    const uint32_t ntot = meta >> 16;
    double d = __dadd_rn(m.eps_sys, __dmul_rn(m.hbar_omega, double(ntot)));
    if (m.delta_eps != 0.0) d = __dadd_rn(d, __dmul_rn(m.delta_eps, double(pos)));
    if (m.has_site_eps) d = __dadd_rn(d, m.site_eps[pos]);
    return d;
}

__device__ __forceinline__ int4 load_nbr(const int* __restrict__ nbr, int64_t r) {
    return __ldg(reinterpret_cast<const int4*>(nbr) + r);
}

// x[idx], or zero for an absent neighbour (idx < 0).  A coefficient of zero would not do: times an
// infinite element of the row itself it is a NaN where the row's sum is infinite.
template <class C>
__device__ __forceinline__ C neighbour(const C* __restrict__ x, int idx) {
    C v{};
    if (idx >= 0) v = __ldcg(x + idx);
    return v;
}

// The same, read once per sweep of a table larger than L2: not kept in the caches.
__device__ __forceinline__ int4 ldcs_nbr(const int* __restrict__ nbr, int64_t r) {
    return __ldcs(reinterpret_cast<const int4*>(nbr) + r);
}

// y = (H x)[r] in complex128 from the row's neighbour entry nb and its own element xr.
// sq[k] = sqrt(k) * g.
template <class P>
__device__ __forceinline__ double2 h_row_c128_nb(const P& m, const double* sq, int64_t r, int4 nb, uint32_t meta,
                                                 double2 xr, const double2* __restrict__ x) {
    const int n = int((meta >> 8) & 0xffu);
    const double2 xa = neighbour(x, nb.x), xb = neighbour(x, nb.y);
    const double2 xd = neighbour(x, nb.z), xu = neighbour(x, nb.w);
    const double d = diag_value(m, meta);
    // the CSR row sums hop and coupling pairs by themselves; a two-term sum does not depend on
    // the column order, and an absent neighbour's zero product leaves the sum as it is
    const double cd = sq[n], cu = sq[n + 1];
    const double hx = __dadd_rn(__dmul_rn(m.J, xa.x), __dmul_rn(m.J, xb.x));
    const double hy = __dadd_rn(__dmul_rn(m.J, xa.y), __dmul_rn(m.J, xb.y));
    const double vx = __dadd_rn(__dmul_rn(cd, xd.x), __dmul_rn(cu, xu.x));
    const double vy = __dadd_rn(__dmul_rn(cd, xd.y), __dmul_rn(cu, xu.y));
    return make_double2(__dadd_rn(__dadd_rn(__dmul_rn(d, xr.x), hx), vx), __dadd_rn(__dadd_rn(__dmul_rn(d, xr.y), hy), vy));
}

// y = (H x)[r] in complex64 with fp32 accumulation.  sq[k] = float(sqrt(k) * g).
template <class P>
__device__ __forceinline__ float2 h_row_c64_nb(const P& m, const float* sq, float J, int64_t r, int4 nb,
                                               uint32_t meta, float2 xr, const float2* __restrict__ x) {
    const int n = int((meta >> 8) & 0xffu);
    const float2 xa = __ldcg(x + (nb.x >= 0 ? nb.x : r));
    const float2 xb = __ldcg(x + (nb.y >= 0 ? nb.y : r));
    const float2 xd = __ldcg(x + (nb.z >= 0 ? nb.z : r));
    const float2 xu = __ldcg(x + (nb.w >= 0 ? nb.w : r));
    const float d = float(diag_value(m, meta));
    const float ja = nb.x >= 0 ? J : 0.f, jb = nb.y >= 0 ? J : 0.f;
    const float cd = nb.z >= 0 ? sq[n] : 0.f, cu = nb.w >= 0 ? sq[n + 1] : 0.f;
    float2 y = make_float2(__fmul_rn(d, xr.x), __fmul_rn(d, xr.y));
    y.x = fmaf(ja, xa.x, y.x);
    y.y = fmaf(ja, xa.y, y.y);
    y.x = fmaf(jb, xb.x, y.x);
    y.y = fmaf(jb, xb.y, y.y);
    y.x = fmaf(cd, xd.x, y.x);
    y.y = fmaf(cd, xd.y, y.y);
    y.x = fmaf(cu, xu.x, y.x);
    y.y = fmaf(cu, xu.y, y.y);
    return y;
}

// ---- lattices with several hopping channels (ModelDev::nhop > 1) ---------------------------
// The reference sums H x term by term -- diag * x, then the "hopping" CSR row, then the
// "hopping2" row, then the vibronic row (paces/core/time_evolution.py:382-400, the terms in
// the order of use_terms) -- and each CSR row in increasing column order, which for open
// boundaries is increasing exciton position (hop_ord).  Channel 0 lives in the int4 row
// (left = lower, right = upper), channels 1.. in m.xnbr.

__device__ __forceinline__ int hop_index(const ModelDev& m, int64_t r, int4 nb, int code) {
    const int ch = code >> 1, up = code & 1;
    if (ch == 0) return up ? nb.y : nb.x;
    const int2 e = __ldg(m.xnbr + int64_t(ch - 1) * m.xcap + r);
    return up ? e.y : e.x;
}
//
// GEO is the number of lattice dimensions: a term has one channel per dimension.  A term's
// indices are read and its gathers issued before its sum, an absent neighbour being zero (which
// leaves the sum as it is); the sum visits the lower neighbours from the largest distance and
// the upper ones from the smallest, the column order.  With the channels a runtime loop the gathers waited for one another (866K
// rows of a square lattice with both terms, complex128: 41 us a Taylor sweep, now 20); three
// dimensions unrolled for every model spilled (47 us).
template <int GEO>
__device__ __forceinline__ void load_hops(const ModelDev& m, int t, int64_t r, int4 nb, int (&lo)[GEO], int (&up)[GEO]) {
#pragma unroll
    for (int d = 0; d < GEO; ++d) {
        if (t == 0 && d == 0) {
            lo[d] = nb.x;
            up[d] = nb.y;
        } else {
            const int2 e = __ldg(m.xnbr + int64_t(t * GEO + d - 1) * m.xcap + r);
            lo[d] = e.x;
            up[d] = e.y;
        }
    }
}

template <int GEO>
__device__ __forceinline__ double2 h_row_c128_geo(const ModelDev& m, const double* sq, int64_t r, int4 nb, uint32_t meta,
                                                  double2 xr, const double2* __restrict__ x) {
    const int n = int((meta >> 8) & 0xffu);
    const double2 xd = neighbour(x, nb.z), xu = neighbour(x, nb.w);
    const double d = diag_value(m, meta);
    double2 y = make_double2(__dmul_rn(d, xr.x), __dmul_rn(d, xr.y));
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        if (t == 1 && m.nhop == GEO) break;  // no second hopping term
        const double Jt = t == 0 ? m.J : m.J2;
        int lo[GEO], up[GEO];
        load_hops<GEO>(m, t, r, nb, lo, up);
        double2 vl[GEO], vu[GEO];
#pragma unroll
        for (int k = 0; k < GEO; ++k) {
            vl[k] = neighbour(x, lo[k]);
            vu[k] = neighbour(x, up[k]);
        }
        double2 hs = make_double2(0.0, 0.0);
        auto add = [&](const double2& v) {
            hs = make_double2(__dadd_rn(hs.x, __dmul_rn(Jt, v.x)), __dadd_rn(hs.y, __dmul_rn(Jt, v.y)));
        };
#pragma unroll
        for (int k = GEO - 1; k >= 0; --k) add(vl[k]);
#pragma unroll
        for (int k = 0; k < GEO; ++k) add(vu[k]);
        y = make_double2(__dadd_rn(y.x, hs.x), __dadd_rn(y.y, hs.y));
    }
    const double cd = sq[n], cu = sq[n + 1];
    const double vx = __dadd_rn(__dmul_rn(cd, xd.x), __dmul_rn(cu, xu.x));
    const double vy = __dadd_rn(__dmul_rn(cd, xd.y), __dmul_rn(cu, xu.y));
    return make_double2(__dadd_rn(y.x, vx), __dadd_rn(y.y, vy));
}

template <int GEO>
__device__ __forceinline__ float2 h_row_c64_geo(const ModelDev& m, const float* sq, int64_t r, int4 nb, uint32_t meta,
                                                float2 xr, const float2* __restrict__ x) {
    const int n = int((meta >> 8) & 0xffu);
    const float2 xd = __ldcg(x + (nb.z >= 0 ? nb.z : r));
    const float2 xu = __ldcg(x + (nb.w >= 0 ? nb.w : r));
    const float d = float(diag_value(m, meta));
    float2 y = make_float2(__fmul_rn(d, xr.x), __fmul_rn(d, xr.y));
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        if (t == 1 && m.nhop == GEO) break;
        const float Jt = float(t == 0 ? m.J : m.J2);
        int lo[GEO], up[GEO];
        load_hops<GEO>(m, t, r, nb, lo, up);
        float2 vl[GEO], vu[GEO];
#pragma unroll
        for (int k = 0; k < GEO; ++k) {
            vl[k] = neighbour(x, lo[k]);
            vu[k] = neighbour(x, up[k]);
        }
        auto add = [&](const float2& v) {
            y.x = fmaf(Jt, v.x, y.x);
            y.y = fmaf(Jt, v.y, y.y);
        };
#pragma unroll
        for (int k = GEO - 1; k >= 0; --k) add(vl[k]);
#pragma unroll
        for (int k = 0; k < GEO; ++k) add(vu[k]);
    }
    const float cd = nb.z >= 0 ? sq[n] : 0.f, cu = nb.w >= 0 ? sq[n + 1] : 0.f;
    y.x = fmaf(cd, xd.x, y.x);
    y.y = fmaf(cd, xd.y, y.y);
    y.x = fmaf(cu, xu.x, y.x);
    y.y = fmaf(cu, xu.y, y.y);
    return y;
}

// The same for kernels that are not compiled per dimension count.
__device__ __forceinline__ double2 h_row_c128_x(const ModelDev& m, const double* sq, int64_t r, int4 nb, uint32_t meta,
                                                double2 xr, const double2* __restrict__ x) {
    const int geo = m.hop_n[0] >> 1;
    if (geo == 1) return h_row_c128_geo<1>(m, sq, r, nb, meta, xr, x);
    if (geo == 2) return h_row_c128_geo<2>(m, sq, r, nb, meta, xr, x);
    return h_row_c128_geo<3>(m, sq, r, nb, meta, xr, x);
}
__device__ __forceinline__ float2 h_row_c64_x(const ModelDev& m, const float* sq, int64_t r, int4 nb, uint32_t meta,
                                              float2 xr, const float2* __restrict__ x) {
    const int geo = m.hop_n[0] >> 1;
    if (geo == 1) return h_row_c64_geo<1>(m, sq, r, nb, meta, xr, x);
    if (geo == 2) return h_row_c64_geo<2>(m, sq, r, nb, meta, xr, x);
    return h_row_c64_geo<3>(m, sq, r, nb, meta, xr, x);
}

// One row of H x for either model: the chain's fixed form, or the channel loop.
__device__ __forceinline__ double2 h_row_c128_any(const ModelDev& m, const double* sq, int64_t r, int4 nb,
                                                  uint32_t meta, double2 xr, const double2* __restrict__ x) {
    return m.nhop > 1 ? h_row_c128_x(m, sq, r, nb, meta, xr, x) : h_row_c128_nb(m, sq, r, nb, meta, xr, x);
}
__device__ __forceinline__ float2 h_row_c64_any(const ModelDev& m, const float* sq, float J, int64_t r, int4 nb,
                                                uint32_t meta, float2 xr, const float2* __restrict__ x) {
    return m.nhop > 1 ? h_row_c64_x(m, sq, r, nb, meta, xr, x) : h_row_c64_nb(m, sq, J, r, nb, meta, xr, x);
}

// H 1 of one row: diag + the row sums term by term (total_ham_ones,
// paces/core/time_evolution.py:403-420), in the order h_row_c128_x sums H x.
__device__ __forceinline__ double h_ones_row_any(const ModelDev& m, const double* sq, int64_t r, int4 nb,
                                                 uint32_t meta) {
    const int n = int((meta >> 8) & 0xffu);
    double h = diag_value(m, meta);
    if (m.nhop > 1) {
        for (int t = 0; t < 2; ++t) {
            const double Jt = t == 0 ? m.J : m.J2;
            double hs = 0.0;
            bool any = false;
            for (int e = 0; e < m.hop_n[t]; ++e) {
                if (hop_index(m, r, nb, m.hop_ord[t][e]) < 0) continue;
                hs = any ? __dadd_rn(hs, Jt) : Jt;
                any = true;
            }
            if (any) h = __dadd_rn(h, hs);
        }
    } else {
        const bool ha = nb.x >= 0, hb = nb.y >= 0;
        if (ha || hb) h = __dadd_rn(h, (ha && hb) ? __dadd_rn(m.J, m.J) : m.J);
    }
    const bool hd = nb.z >= 0, hu = nb.w >= 0;
    const double cd = sq[n], cu = sq[n + 1];
    if (hd || hu) h = __dadd_rn(h, (hd && hu) ? __dadd_rn(cd, cu) : (hd ? cd : cu));
    return h;
}

}  // namespace paces
