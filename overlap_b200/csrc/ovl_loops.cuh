// The closed link loops of one quadrant of a lattice plane, for either colour
// count: the plaquette and the two 2 x 1 rectangles with the site at a corner,
// which the improved E.B (ovl_gauge.cu, ovl_su3.cu) sums over the quadrants.
#pragma once

#include "ovl_su3.cuh"

namespace ovl {

// Offset of the site index when coordinate c (of extent n, index stride
// `stride`) moves by k, periodic; any n >= 1.
__device__ __forceinline__ int wrap_offset(int c, int n, int stride, int k) {
    int w = c + k;
    while (w >= n) w -= n;
    while (w < 0) w += n;
    return (w - c) * stride;
}

// Extent and index stride of direction d, and the site's coordinate along it.
__device__ __forceinline__ int extent_of(const Lattice &L, int d) { return d == 0 ? L.N0 : (d == 1 ? L.N1 : L.N2); }
__device__ __forceinline__ int stride_of(const Lattice &L, int d) { return d == 0 ? 1 : (d == 1 ? L.N0 : L.N0 * L.N1); }

struct Su2Ops {
    using M = quat;
    static __device__ __forceinline__ M load(const double *__restrict__ U, int s, int mu) { return load_link(U, s, mu); }
    static __device__ __forceinline__ M dag(const M &a) { return qdag(a); }
    static __device__ __forceinline__ M mul(const M &a, const M &b) { return qmul(a, b); }
    static __device__ __forceinline__ M one() { return {0.0, 0.0, 0.0, 1.0}; }
};
struct Su3Ops {
    using M = cmat3<double>;
    static __device__ __forceinline__ M load(const double *__restrict__ U, int s, int mu) { return load_su3(U, s, mu); }
    static __device__ __forceinline__ M dag(const M &a) { return m3_dag(a); }
    static __device__ __forceinline__ M mul(const M &a, const M &b) { return m3_mul(a, b); }
    static __device__ __forceinline__ M one() { return m3_unit<double>(); }
};

// Quadrant q of the plane (mu, nu) at `site` (coordinates c): counter-clockwise
// from the site its sides start along d1 (sign s1) and turn along d2 (sign s2).
struct Quadrant {
    int site, d1, d2, s1, s2;
    int o1[3], o2[3];  // offsets of 0, 1, 2 steps along (d1, s1) and (d2, s2)

    __device__ __forceinline__ Quadrant(const Lattice &L, int site_, const int (&c)[3], int mu, int nu, int q)
        : site(site_) {
        const bool swap = q & 1;  // quadrants (+,+), (-,+), (-,-), (+,-) of (mu, nu)
        d1 = swap ? nu : mu;
        d2 = swap ? mu : nu;
        s1 = q < 2 ? 1 : -1;
        s2 = (q == 0 || q == 3) ? 1 : -1;
        const int c1 = d1 == 0 ? c[0] : (d1 == 1 ? c[1] : c[2]), c2 = d2 == 0 ? c[0] : (d2 == 1 ? c[1] : c[2]);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            o1[k] = wrap_offset(c1, extent_of(L, d1), stride_of(L, d1), s1 * k);
            o2[k] = wrap_offset(c2, extent_of(L, d2), stride_of(L, d2), s2 * k);
        }
    }
    // The link that leads from the point (i, j) one step along d1 / d2.
    template <class OPS> __device__ __forceinline__ typename OPS::M a(const double *__restrict__ U, int i, int j) const {
        const typename OPS::M u = OPS::load(U, site + (s1 > 0 ? o1[i] : o1[i + 1]) + o2[j], d1);
        return s1 > 0 ? u : OPS::dag(u);
    }
    template <class OPS> __device__ __forceinline__ typename OPS::M b(const double *__restrict__ U, int i, int j) const {
        const typename OPS::M u = OPS::load(U, site + o1[i] + (s2 > 0 ? o2[j] : o2[j + 1]), d2);
        return s2 > 0 ? u : OPS::dag(u);
    }
    // visit(loop, coefficient) for the plaquette (5/12) and the two rectangles
    // (-1/24): 10 links loaded and 11 products, the common sides shared.
    template <class OPS, class Visit> __device__ __forceinline__ void loops(const double *__restrict__ U, Visit &&visit) const {
        using M = typename OPS::M;
        const M a00 = a<OPS>(U, 0, 0), b00 = b<OPS>(U, 0, 0);
        const M x = OPS::mul(a00, b<OPS>(U, 1, 0)), y = OPS::mul(b00, a<OPS>(U, 0, 1));
        visit(OPS::mul(x, OPS::dag(y)), 5.0 / 12.0);
        visit(OPS::mul(OPS::mul(OPS::mul(a00, a<OPS>(U, 1, 0)), b<OPS>(U, 2, 0)), OPS::dag(OPS::mul(y, a<OPS>(U, 1, 1)))),
              -1.0 / 24.0);
        visit(OPS::mul(OPS::mul(x, b<OPS>(U, 1, 1)), OPS::dag(OPS::mul(OPS::mul(b00, b<OPS>(U, 0, 1)), a<OPS>(U, 0, 2)))),
              -1.0 / 24.0);
    }
};

// Plaquette q of the staple force of link l = 3 site + mu (Dynamics.cpp:145-197),
// starting with U_mu(x): q >> 1 picks the transverse direction nu, q & 1 the
// side: x -> x+mu -> x+mu+nu -> x+nu, or the same towards -nu.
template <class OPS>
__device__ __forceinline__ typename OPS::M staple_plaquette(const double *__restrict__ U, const Lattice &L, int l, int q) {
    const int site = l / 3, mu = l % 3, nu = (mu + 1 + (q >> 1)) % 3;
    int c[3];
    site_coords(L, site, c[0], c[1], c[2]);
    const int cm = mu == 0 ? c[0] : (mu == 1 ? c[1] : c[2]), cn = nu == 0 ? c[0] : (nu == 1 ? c[1] : c[2]);
    const int om = wrap_offset(cm, extent_of(L, mu), stride_of(L, mu), 1);
    const int on = wrap_offset(cn, extent_of(L, nu), stride_of(L, nu), (q & 1) ? -1 : 1);
    const typename OPS::M u0 = OPS::load(U, site, mu), u2 = OPS::load(U, site + on, mu);
    if (q & 1) {
        const typename OPS::M u1 = OPS::load(U, site + om + on, nu), u3 = OPS::load(U, site + on, nu);
        return OPS::mul(OPS::mul(OPS::mul(u0, OPS::dag(u1)), OPS::dag(u2)), u3);
    }
    const typename OPS::M u1 = OPS::load(U, site + om, nu), u3 = OPS::load(U, site, nu);
    return OPS::mul(OPS::mul(u0, u1), OPS::mul(OPS::dag(u2), OPS::dag(u3)));
}

// The improved electric field (ChernSimonsOperators.cpp:379-401) is the sum of
// -1/12, 7/12, 7/12, -1/12 of E_mu at x+mu, x, x-mu, x-2mu transported to x.
// Term q (0: x, 1: x+mu, 2: x-mu, 3: x-2mu): its site, transporter and weight.
template <class OPS>
__device__ __forceinline__ void improved_e_term(const double *__restrict__ U, const Lattice &L, int site, const int (&c)[3],
                                                int mu, int q, int &es, typename OPS::M &V, double &weight) {
    const int cm = mu == 0 ? c[0] : (mu == 1 ? c[1] : c[2]), n = extent_of(L, mu), st = stride_of(L, mu);
    const int sm = site + wrap_offset(cm, n, st, -1);
    es = site;
    V = OPS::one();
    weight = (q == 0 || q == 2) ? 7.0 / 12.0 : -1.0 / 12.0;
    if (q == 1) {
        es = site + wrap_offset(cm, n, st, 1);
        V = OPS::load(U, site, mu);
    } else if (q >= 2) {
        es = sm;
        V = OPS::dag(OPS::load(U, sm, mu));
        if (q == 3) {
            es = site + wrap_offset(cm, n, st, -2);
            V = OPS::mul(V, OPS::dag(OPS::load(U, es, mu)));
        }
    }
}

// Sum over the four lanes of a quadrant group (lanes 4 g .. 4 g + 3).
__device__ __forceinline__ double quad_sum(double v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

}  // namespace ovl
