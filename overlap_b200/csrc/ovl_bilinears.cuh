// Building blocks of the kernels that sum FP64 bilinears of the modes over the
// mode batch (currents, charges, the fermions' colour force), for two and three
// colours and every mode storage.
#pragma once

#include "ovl_fp40.cuh"
#include "ovl_stencil.cuh"
#include "ovl_su3.cuh"

namespace ovl {

// One site's spinor of the lane's mode as loaded: get(k) hands out component
// k = 4 colour + spin as complex double.  Holding the raw words lets the loads
// of the next neighbour be in flight while the current one is multiplied.
template <int NC, class SRC> struct SiteRaw;

template <int NC, typename T> struct SiteRaw<NC, SrcPlain<T>> {
    cpx<T> v[4 * NC];
    __device__ __forceinline__ void load(const SrcPlain<T> &f, int V, int mb, int site, int lane) {
        const cpx<T> *p = f.p + (((size_t)mb * V + site) * (4 * NC)) * kModeBlock + lane;
#pragma unroll
        for (int k = 0; k < 4 * NC; k++) v[k] = ld(p + k * kModeBlock);
    }
    __device__ __forceinline__ cpx<double> get(int k) const { return mk<double>((double)v[k].re, (double)v[k].im); }
};

// 40-bit storage: the extension bytes of the site in one 16-byte load.
template <> struct SiteRaw<2, Src40> {
    uint2 h[kComp];
    uint4 l;
    __device__ __forceinline__ void load(const Src40 &f, int V, int mb, int site, int lane) {
        const size_t base = field_index(V, mb, site, 0, lane);
#pragma unroll
        for (int k = 0; k < kComp; k++) h[k] = __ldg(f.hi + base + k * kModeBlock);
        l = __ldg(reinterpret_cast<const uint4 *>(f.lo) + ((size_t)mb * V + site) * kModeBlock + lane);
    }
    __device__ __forceinline__ unsigned low(int b) const {
        const unsigned w = b < 4 ? l.x : b < 8 ? l.y : b < 12 ? l.z : l.w;
        return __byte_perm(w, 0u, 0x0444u | ((unsigned)(b & 3) << 12));
    }
    __device__ __forceinline__ cpx<double> get(int k) const {
        return mk<double>(__hiloint2double((int)h[k].x, (int)low(2 * k)), __hiloint2double((int)h[k].y, (int)low(2 * k + 1)));
    }
};

// The dressed FP64 links of SITES consecutive sites, [site][mu][NC i + j], built
// once per CTA in shared memory (broadcast reads in the mode loop, no registers
// held over it).  Every thread of the CTA calls it: it holds a barrier.
template <int NC, int SITES>
__device__ __forceinline__ void fill_bilinear_links(const double *__restrict__ U, const double *__restrict__ u1,
                                                    const Lattice &L, int site0, double2 (*tab)[3][NC * NC]) {
    const int t = threadIdx.y * kModeBlock + threadIdx.x;
    if (t < 3 * SITES) {
        const int s = site0 + t / 3, mu = t % 3;
        if (s < L.V) {
            double2 *o = tab[t / 3][mu];
            if constexpr (NC == 2) {
                const cmat2<double> M = dressed_link<double>(U, reinterpret_cast<const double2 *>(u1), s, mu, L.N0 * L.N1);
                o[0] = make_double2(M.m00.re, M.m00.im);
                o[1] = make_double2(M.m01.re, M.m01.im);
                o[2] = make_double2(M.m10.re, M.m10.im);
                o[3] = make_double2(M.m11.re, M.m11.im);
            } else {
                const cmat3<double> M = u1 ? Links3<false, true>{U, u1, L.N0 * L.N1}.template get<double>(s, mu)
                                           : Links3<false, false>{U, nullptr, L.N0 * L.N1}.template get<double>(s, mu);
                for (int i = 0; i < 3; i++)
                    for (int j = 0; j < 3; j++) o[3 * i + j] = make_double2(M.m[i][j].re, M.m[i][j].im);
            }
        }
    }
    __syncthreads();
}

// chi_c = sum_j M_cj h_j of one spin component.
template <int NC>
__device__ __forceinline__ void link_times(const double2 *__restrict__ M, const cpx<double> (&h)[NC], cpx<double> (&chi)[NC]) {
#pragma unroll
    for (int c = 0; c < NC; c++) {
        double re = 0.0, im = 0.0;
#pragma unroll
        for (int j = NC - 1; j >= 0; j--) {
            const double2 m = M[NC * c + j];
            re = j == NC - 1 ? m.x * h[j].re : fma(m.x, h[j].re, re);
            im = j == NC - 1 ? m.x * h[j].im : fma(m.x, h[j].im, im);
            re = fma(-m.y, h[j].im, re);
            im = fma(m.y, h[j].re, im);
        }
        chi[c] = mk<double>(re, im);
    }
}

// v += the real (IM: imaginary) part of conj(f) i^ph h.
template <bool IM> __device__ __forceinline__ void add_part(double &v, int ph, const cpx<double> &f, const cpx<double> &h) {
    // Re: ph 0 f.re h.re + f.im h.im; 1 f.im h.re - f.re h.im; 2, 3 their negatives.  Im(z) = Re(-i z): ph + 3
    switch ((IM ? ph + 3 : ph) & 3) {
        case 0: v = fma(f.re, h.re, fma(f.im, h.im, v)); break;
        case 1: v = fma(f.im, h.re, fma(-f.re, h.im, v)); break;
        case 2: v = fma(-f.re, h.re, fma(-f.im, h.im, v)); break;
        default: v = fma(-f.im, h.re, fma(f.re, h.im, v)); break;
    }
}

// Sums the 16 values over the warp's 32 lanes: lanes 2 i and 2 i + 1 return the
// total of v[i].  Each step exchanges half of the values still held (16 shuffles
// instead of 80), every sum over the same balanced tree of lanes.
__device__ __forceinline__ double warp_sum16(double (&v)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int n = 8, off = 16; n >= 1; n >>= 1, off >>= 1) {
        const bool up = lane & off;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const double send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// The same for 32 values: lane i returns the total of v[i] (31 shuffles for 160).
__device__ __forceinline__ double warp_sum32(double (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int n = 16; n >= 1; n >>= 1) {
        const bool up = lane & n;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const double send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, n);
        }
    }
    return v[0];
}

// The colour force's link-independent bilinears of one hop direction,
// C_ij += psi_i^+ g0 (1 - G_mu) psi'_j with psi' the neighbour.  1 - G_mu = 1 + i
// g_mu is twice a rank-2 projector: (1 + i g_mu) psi' is rebuilt from its two
// upper spin components h0, h1 (the forward projection of hop()), so that
// psi^+ g0 (1 + i g_mu) psi' = q0^+ h0 + q1^+ h1 with q0, q1 the backward projection
// of psi: two dot products per colour pair instead of the eight terms of two
// full spinor bilinears.  f carries the vacuum weight.
template <int NC, int MU, class RAW>
__device__ __forceinline__ void add_colour_pairs(const cpx<double> (&f)[NC][kSpin], const RAW &raw, double *acc) {
    cpx<double> h0[NC], h1[NC];
#pragma unroll
    for (int j = 0; j < NC; j++) {
        const cpx<double> p0 = raw.get(kSpin * j), p1 = raw.get(kSpin * j + 1), p2 = raw.get(kSpin * j + 2),
                          p3 = raw.get(kSpin * j + 3);
        h0[j] = MU == 0 ? p0 + times_i(p3) : (MU == 1 ? p0 + p3 : p0 + times_i(p2));
        h1[j] = MU == 0 ? p1 + times_i(p2) : (MU == 1 ? p1 - p2 : p1 - times_i(p3));
    }
#pragma unroll
    for (int i = 0; i < NC; i++) {
        const cpx<double> *p = f[i];
        const cpx<double> q0 = MU == 0 ? p[0] - times_i(p[3]) : (MU == 1 ? p[0] - p[3] : p[0] - times_i(p[2]));
        const cpx<double> q1 = MU == 0 ? p[1] - times_i(p[2]) : (MU == 1 ? p[1] + p[2] : p[1] + times_i(p[3]));
#pragma unroll
        for (int j = 0; j < NC; j++) {
            double *a = acc + 2 * (NC * i + j);
            add_part<false>(a[0], 0, q0, h0[j]);
            add_part<false>(a[0], 0, q1, h1[j]);
            add_part<true>(a[1], 0, q0, h0[j]);
            add_part<true>(a[1], 0, q1, h1[j]);
        }
    }
}

// Vacuum weight of a mode: +-1 by the parity of its global index, 0 for padding.
__device__ __forceinline__ double vacuum_weight(int mode, int n_modes, int first_mode) {
    return mode >= n_modes ? 0.0 : (((first_mode + mode) & 1) == 0 ? 1.0 : -1.0);
}

// A per-thread running sum, compensated or plain.
template <bool COMP> struct RunSum {
    CompSum s;
    __device__ __forceinline__ void add(double x) { s.add(x); }
    __device__ __forceinline__ double value() const { return s.value(); }
};
template <> struct RunSum<false> {
    double s = 0.0;
    __device__ __forceinline__ void add(double x) { s += x; }
    __device__ __forceinline__ double value() const { return s; }
};

}  // namespace ovl
