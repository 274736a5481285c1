// The whole Chebyshev overlap operator of a few modes on chip: a thread-block
// cluster holds every site of the lattice for its modes, so that the series
// reads phi from memory once and writes the result once.  Kernel by kernel
// (ovl_chebyshev.cu, ovl_su3.cu) a term moves seven fields through memory; here
// it moves none, and what bounds it is the shared memory the stencil reads its
// neighbours from, with the FP32 arithmetic close behind.
//
// The CTAs of a cluster own consecutive z planes.  A thread owns one site of two
// FP32 modes (two colours) or of one mode (three colours, FP64).  The Clenshaw
// vector b_{k+1} and w = D b_{k+1} are in shared memory (the fields neighbours
// read), b_{k+2} in registers; phi is in shared memory where a two-colour lattice
// fits one CTA, otherwise laid out once, coalesced, in a field of scratch and read
// from L2.  The x and y neighbours are the CTA's own.  A CTA's outer planes are
// projected where they are made, and the half spinors (the backward hop's already
// multiplied by its link) are written into the next CTA's shared memory.  A term
// is two phases, each ending in a barrier of the cluster that is waited for only
// where the half spinors are read.
// One overlap step, through memory and here: 8^3, two colours, 4096 FP32 modes,
// degree 64: 23.7 and 10.1 ms (one CTA; L1 data pipe 92 % busy); 12^3, three
// colours, 1536 FP32 modes, degree 96: 71.0 and 58.3 ms (six CTAs; 65.0 ms reading
// whole spinors from the other CTAs, 53.0 ms if nothing had to come from them).
#pragma once

#include <algorithm>
#include <cmath>
#include <type_traits>

#include <cooperative_groups.h>

#include "ovl_internal.h"
#include "ovl_rules.h"
#include "ovl_stencil.cuh"
#include "ovl_su3.cuh"

namespace ovl {

// What a thread works on: two FP32 modes with the paired FP32 instructions, one
// FP32 mode, or one FP64 mode.
template <typename T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };
struct LanePair {
    using T = float;
    using V = float2;
    using Slot = float4;
    static constexpr int kModes = 2;
};
template <typename S> struct LaneOne {
    using T = S;
    using V = S;
    using Slot = typename Vec2<S>::type;
    static constexpr int kModes = 1;
};

template <typename V, typename T> __device__ __forceinline__ V vsplat(T a) {
    if constexpr (std::is_same<V, float2>::value) return make_float2(a, a);
    else return a;
}
template <typename V> __device__ __forceinline__ V vfma(V a, V b, V c) {
    if constexpr (std::is_same<V, float2>::value) return __ffma2_rn(a, b, c);
    else return fma(a, b, c);
}
template <typename V> __device__ __forceinline__ V vmul(V a, V b) {
    if constexpr (std::is_same<V, float2>::value) return __fmul2_rn(a, b);
    else return a * b;
}
template <typename V> __device__ __forceinline__ V vadd(V a, V b) {
    if constexpr (std::is_same<V, float2>::value) return __fadd2_rn(a, b);
    else return a + b;
}
template <typename V> __device__ __forceinline__ V vsub(V a, V b) {  // pairs: -b is exact, rounded once
    if constexpr (std::is_same<V, float2>::value) return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
    else return a - b;
}
template <typename V> __device__ __forceinline__ V vneg(V a) {
    if constexpr (std::is_same<V, float2>::value) return __fmul2_rn(a, make_float2(-1.0f, -1.0f));
    else return -a;
}

// x, computed with where it is used: without this the addresses that follow from
// it, one per component, are kept in registers through the whole series.
__device__ __forceinline__ int res_here(int x) {
    asm volatile("" : "+r"(x));
    return x;
}
template <typename P> __device__ __forceinline__ P *res_here(P *x) {
    asm volatile("" : "+l"(x));
    return x;
}

template <typename V> struct vcpx { V re, im; };

// A slot in shared memory holds (re a, re b, im a, im b) or (re, im); in memory
// the modes are (re a, im a, re b, im b).
__device__ __forceinline__ vcpx<float2> slot_get(const float4 &s) { return {make_float2(s.x, s.y), make_float2(s.z, s.w)}; }
__device__ __forceinline__ vcpx<float> slot_get(const float2 &s) { return {s.x, s.y}; }
__device__ __forceinline__ vcpx<double> slot_get(const double2 &s) { return {s.x, s.y}; }
__device__ __forceinline__ float4 slot_put(const vcpx<float2> &v) { return make_float4(v.re.x, v.re.y, v.im.x, v.im.y); }
__device__ __forceinline__ float2 slot_put(const vcpx<float> &v) { return make_float2(v.re, v.im); }
__device__ __forceinline__ double2 slot_put(const vcpx<double> &v) { return make_double2(v.re, v.im); }
__device__ __forceinline__ vcpx<float2> slot_load(const float4 *p) {
    const float4 s = *p;
    return {make_float2(s.x, s.z), make_float2(s.y, s.w)};
}
__device__ __forceinline__ vcpx<float> slot_load(const float2 *p) { return slot_get(*p); }
__device__ __forceinline__ vcpx<double> slot_load(const double2 *p) { return slot_get(*p); }
__device__ __forceinline__ void slot_store(float4 *p, const vcpx<float2> &v) {
    *p = make_float4(v.re.x, v.im.x, v.re.y, v.im.y);
}
__device__ __forceinline__ void slot_store(float2 *p, const vcpx<float> &v) { *p = slot_put(v); }
__device__ __forceinline__ void slot_store(double2 *p, const vcpx<double> &v) { *p = slot_put(v); }

// A link in shared memory.  Two colours: the first row of the SU(2) matrix; the
// U(1) phase is multiplied on at use.  Three colours: the 3x3 matrix with its
// phase, by columns.  The sizes keep the lanes' records in different banks.
template <int NC> constexpr int kResLinkReals = NC == 2 ? 4 : 18;

// Element (i, j) of the link in direction MU at `rec`.  Three colours read it where
// it is used: the whole matrix would take 18 registers.
template <int NC, typename T, bool U1, int MU> struct ResMat {
    const T *rec;
    __device__ __forceinline__ ResMat(const T *r, const cpx<T> *) : rec(r) {}
    __device__ __forceinline__ cpx<T> operator()(int i, int j) const {
        const typename Vec2<T>::type w = reinterpret_cast<const typename Vec2<T>::type *>(rec)[i + 3 * j];
        return mk<T>(w.x, w.y);
    }
};
template <typename T, bool U1, int MU> struct ResMat<2, T, U1, MU> {
    cpx<T> m[2][2];
    __device__ __forceinline__ ResMat(const T *r, const cpx<T> *phase) {
        T f[4];
#pragma unroll
        for (int k = 0; k < 4; k += 16 / sizeof(T)) {
            using Word = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
            const Word w = *reinterpret_cast<const Word *>(r + k);
            f[k] = w.x;
            f[k + 1] = w.y;
            if constexpr (sizeof(T) == 4) {
                f[k + 2] = w.z;
                f[k + 3] = w.w;
            }
        }
        m[0][0] = mk<T>(f[0], f[1]);
        m[0][1] = mk<T>(f[2], f[3]);
        m[1][0] = mk<T>(-f[2], f[3]);
        m[1][1] = mk<T>(f[0], -f[1]);
        if constexpr (U1 && MU < 2) {
            const cpx<T> p = phase[MU];
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) m[i][j] = p * m[i][j];
        }
    }
    __device__ __forceinline__ cpx<T> operator()(int i, int j) const { return m[i][j]; }
};

// The hops acc -= (1 - G_mu) U phi (forward) and (1 + G_mu) U^+ phi (backward) by
// halves, the projections of hop() in ovl_stencil.cuh: half h projects spin h and
// its partner to v = p_h + g p_partner, g = s i in x and z and s in y, where s is
// +1 forward and -1 backward, and turned for h = 1 in y and z; the product k is
// taken from spin h, and g^* k from the partner.
template <int MU> __device__ __forceinline__ constexpr int res_partner(int h) { return MU == 2 ? h + 2 : 3 - h; }

template <int MU, bool FWD, int NC, typename V, class Load>
__device__ __forceinline__ void res_project(int h, const Load &load, vcpx<V> (&v)[NC]) {
    const bool plus = FWD != (h == 1 && MU != 0);
#pragma unroll
    for (int c = 0; c < NC; c++) {
        const vcpx<V> p = load(c, h), q = load(c, res_partner<MU>(h));
        if (MU == 1) {
            v[c].re = plus ? vadd(p.re, q.re) : vsub(p.re, q.re);
            v[c].im = plus ? vadd(p.im, q.im) : vsub(p.im, q.im);
        } else {
            v[c].re = plus ? vsub(p.re, q.im) : vadd(p.re, q.im);
            v[c].im = plus ? vadd(p.im, q.re) : vsub(p.im, q.re);
        }
    }
}

// Colour i of M v (forward) or M^+ v (backward), for both halves
template <bool FWD, int NC, class MAT, typename V>
__device__ __forceinline__ void res_row(int i, const MAT &M, const vcpx<V> (&v)[2][NC], vcpx<V> (&k)[2]) {
#pragma unroll
    for (int j = 0; j < NC; j++) {
        const auto m = FWD ? M(i, j) : M(j, i);
        const V a = vsplat<V>(m.re), b = vsplat<V>(FWD ? m.im : -m.im), nb = vsplat<V>(FWD ? -m.im : m.im);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const vcpx<V> &x = v[h][j];
            k[h].re = vfma(nb, x.im, j == 0 ? vmul(a, x.re) : vfma(a, x.re, k[h].re));
            k[h].im = vfma(b, x.re, j == 0 ? vmul(a, x.im) : vfma(a, x.im, k[h].im));
        }
    }
}

// Colour c of half h out of the accumulator
template <int MU, bool FWD, typename V>
__device__ __forceinline__ void res_take(int h, const vcpx<V> &k, vcpx<V> (&acc)[kSpin]) {
    const bool plus = FWD != (h == 1 && MU != 0);
    vcpx<V> &x = acc[h], &y = acc[res_partner<MU>(h)];
    x.re = vsub(x.re, k.re);
    x.im = vsub(x.im, k.im);
    if (MU == 1) {
        y.re = plus ? vsub(y.re, k.re) : vadd(y.re, k.re);
        y.im = plus ? vsub(y.im, k.im) : vadd(y.im, k.im);
    } else {
        y.re = plus ? vsub(y.re, k.im) : vadd(y.re, k.im);
        y.im = plus ? vadd(y.im, k.re) : vsub(y.im, k.re);
    }
}

template <int MU, bool FWD, int NC, class MAT, typename V>
__device__ __forceinline__ void res_apply(vcpx<V> (&acc)[NC][kSpin], const MAT &M, const vcpx<V> (&v)[2][NC]) {
#pragma unroll
    for (int i = 0; i < NC; i++) {
        vcpx<V> k[2];
        res_row<FWD, NC>(i, M, v, k);
        res_take<MU, FWD>(0, k[0], acc[i]);
        res_take<MU, FWD>(1, k[1], acc[i]);
    }
}

template <int MU, bool FWD, int NC, class MAT, typename V, class Load>
__device__ __forceinline__ void res_hop(vcpx<V> (&acc)[NC][kSpin], const MAT &M, const Load &load) {
    vcpx<V> v[2][NC];
    res_project<MU, FWD, NC>(0, load, v[0]);
    res_project<MU, FWD, NC>(1, load, v[1]);
    res_apply<MU, FWD, NC>(acc, M, v);
}

template <typename T> struct ResidentArgs {
    const void *U, *u1;            // links as HopConfig and Su3Links hold them for T
    const cpx<T> *phi;
    cpx<T> *dst, *scratch;         // scratch: one field, phi as [slot][component][site]
    Lattice L;
    ResidentShape sh;
    int slots;                     // of all modes
    int K, accumulate;
    T amass, a, beta, mdw, cp, cm, dt;
    T c[kMaxChebDegree + 1];       // c_k lambda_max^-1/2, c_0 halved
};

template <int NC, class LN> struct ResidentLayout {
    using T = typename LN::T;
    static constexpr int kComps = NC * kSpin, kHalf = 2 * NC;
    // phi of two colours has room in shared memory where there are no half spinors
    static constexpr bool phi_shared(bool cluster) { return NC == 2 && !cluster; }
    // bytes with CAP threads per CTA: b, w and phi; half spinors of the two outer
    // planes of either; the links of the CTA's sites; the U(1) phases of a plane
    static size_t bytes(int cap, const ResidentShape &sh, int n01) {
        return sizeof(typename LN::Slot) * ((size_t)kComps * (phi_shared(sh.ranks > 1) ? 3 : 2) * cap + (sh.ranks > 1 ? (size_t)4 * kHalf * n01 * sh.groups : 0)) +
               sizeof(T) * kResLinkReals<NC> * (size_t)3 * n01 * sh.planes +
               (NC == 2 ? 2 * sizeof(cpx<T>) * (size_t)n01 : 0);
    }
};

template <int NC, class LN, bool U1, bool CLUSTER, int CAP>
__global__ void __launch_bounds__(CAP, 1)
    resident_cheb_kernel(const __grid_constant__ ResidentArgs<typename LN::T> A) {
    using T = typename LN::T;
    using V = typename LN::V;
    using Slot = typename LN::Slot;
    constexpr int C = NC * kSpin, R = kResLinkReals<NC>, H = 2 * NC;
    extern __shared__ __align__(16) unsigned char res_smem[];
    Slot *buf = reinterpret_cast<Slot *>(res_smem);  // [b, w, phi if it is here][component][CAP]
    const Lattice &L = A.L;
    const int n01 = L.N0 * L.N1, S = n01 * A.sh.planes, NH = n01 * A.sh.groups;
    constexpr bool kPhiShared = ResidentLayout<NC, LN>::phi_shared(CLUSTER);
    // [b, w][from below, from above][half spinor][NH]
    Slot *halo = buf + (size_t)(kPhiShared ? 3 : 2) * C * CAP;
    T *links = reinterpret_cast<T *>(halo + (CLUSTER ? (size_t)4 * H * NH : 0));
    cpx<T> *phases = reinterpret_cast<cpx<T> *>(links + (size_t)R * 3 * S);

    const int rank = CLUSTER ? blockIdx.x % A.sh.ranks : 0, first = (blockIdx.x / A.sh.ranks) * A.sh.groups;
    const int z0 = rank * A.sh.planes, nz = min(A.sh.planes, L.N2 - z0);
    // the modes of a site are neighbouring threads: one read of a link serves them
    const int G = A.sh.groups, s = threadIdx.x / G, g = threadIdx.x - s * G, slot = first + g;
    const bool live = s < nz * n01 && slot < A.slots;

    for (int i = threadIdx.x; i < 3 * nz * n01; i += blockDim.x) {
        const int site = z0 * n01 + i / 3, mu = i % 3;
        T *r = links + (size_t)R * i;
        if constexpr (NC == 2) {
            cmat2<T> M;
            if constexpr (sizeof(T) == 4)
                M = LinksF32<false>{reinterpret_cast<const float4 *>(A.U), nullptr, n01}.template get<T>(site, mu);
            else
                M = LinksF64<false>{reinterpret_cast<const double *>(A.U), nullptr, n01}.template get<T>(site, mu);
            r[0] = M.m00.re;
            r[1] = M.m00.im;
            r[2] = M.m01.re;
            r[3] = M.m01.im;
        } else {
            const cmat3<T> M = Links3<sizeof(T) == 4, U1>{A.U, A.u1, n01}.template get<T>(site, mu);
#pragma unroll
            for (int c = 0; c < 9; c++) {
                r[2 * c] = M.m[c % 3][c / 3].re;
                r[2 * c + 1] = M.m[c % 3][c / 3].im;
            }
        }
    }
    if constexpr (NC == 2 && U1)
        for (int i = threadIdx.x; i < 2 * n01; i += blockDim.x) phases[i] = reinterpret_cast<const cpx<T> *>(A.u1)[i];

    // the neighbours' slots and links
    const int p = s % n01, z = s / n01, x = p % L.N0, y = p / L.N0, me = threadIdx.x;
    const int dxp = x + 1 == L.N0 ? 1 - L.N0 : 1, dxm = x == 0 ? L.N0 - 1 : -1;
    const int dyp = y + 1 == L.N1 ? L.N0 - n01 : L.N0, dym = y == 0 ? n01 - L.N0 : -L.N0;
    const bool top = z + 1 == nz, bottom = z == 0;
    const int dzp = top ? n01 - nz * n01 : n01, dzm = bottom ? (nz - 1) * n01 : -n01;  // own planes only
    const T *lk = links + (size_t)R * 3 * s;
    const cpx<T> *ph = phases + 2 * p;
    Slot *edge = halo + p * G + g;

    // A phase ends in arrive(): the CTA's own threads meet, and the cluster's
    // barrier is only waited for (wait()) where the next phase turns to the half
    // spinors of the other CTAs.
    auto arrive = [&] {
        if constexpr (CLUSTER) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        __syncthreads();
    };
    auto wait = [&] {
        if constexpr (CLUSTER) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    };
    // acc = amass f - hops of field `which` (b: 0, w: 1) around the site, from the CTA's own sites
    auto stencil = [&](int which, vcpx<V> (&acc)[NC][kSpin]) {
        const Slot *f = buf + (size_t)which * C * CAP + me;
        const V m = vsplat<V>(A.amass);
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int a = 0; a < kSpin; a++) {
                const vcpx<V> v = slot_get(f[(c * kSpin + a) * CAP]);
                acc[c][a] = {vmul(m, v.re), vmul(m, v.im)};
            }
        auto at = [](const Slot *q) { return [q](int c, int a) { return slot_get(q[(c * kSpin + a) * CAP]); }; };
        res_hop<0, true, NC>(acc, ResMat<NC, T, U1, 0>(lk, ph), at(f + G * dxp));
        res_hop<0, false, NC>(acc, ResMat<NC, T, U1, 0>(lk + 3 * R * dxm, ph + 2 * dxm), at(f + G * dxm));
        res_hop<1, true, NC>(acc, ResMat<NC, T, U1, 1>(lk + R, ph), at(f + G * dyp));
        res_hop<1, false, NC>(acc, ResMat<NC, T, U1, 1>(lk + 3 * R * dym + R, ph + 2 * dym), at(f + G * dym));
        if (!CLUSTER || !top) res_hop<2, true, NC>(acc, ResMat<NC, T, U1, 2>(lk + 2 * R, ph), at(f + G * dzp));
        if (!CLUSTER || !bottom)
            res_hop<2, false, NC>(acc, ResMat<NC, T, U1, 2>(lk + 3 * R * dzm + 2 * R, ph), at(f + G * dzm));
    };
    // the hops of the outer planes, from the half spinors the other CTAs wrote
    auto outer = [&](int which, vcpx<V> (&acc)[NC][kSpin]) {
        if constexpr (CLUSTER) {
            const int nh = res_here(NH);
            const Slot *e = edge + which * 2 * H * nh;
            if (top) {
                vcpx<V> v[2][NC];
#pragma unroll
                for (int k = 0; k < H; k++) v[k / NC][k % NC] = slot_get(e[(H + k) * nh]);
                res_apply<2, true, NC>(acc, ResMat<NC, T, U1, 2>(lk + 2 * R, ph), v);
            }
            if (bottom) {
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    res_take<2, false>(0, slot_get(e[c * nh]), acc[c]);
                    res_take<2, false>(1, slot_get(e[(NC + c) * nh]), acc[c]);
                }
            }
        }
    };
    // v becomes field `which` at the site, and at the outer planes' neighbours
    auto publish = [&](int which, const vcpx<V> (&v)[NC][kSpin]) {
        Slot *f = buf + (size_t)which * C * CAP + me;
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int a = 0; a < kSpin; a++) f[(c * kSpin + a) * CAP] = slot_put(v[c][a]);
        if constexpr (CLUSTER) {
            auto cl = cooperative_groups::this_cluster();
            auto own = [&](int c, int a) { return v[c][a]; };
            const int nh = res_here(NH);
            Slot *e = edge + which * 2 * H * nh;
            if (top) {
                Slot *to = cl.map_shared_rank(e, rank + 1 == A.sh.ranks ? 0 : rank + 1);
                const ResMat<NC, T, U1, 2> M(lk + 2 * R, ph);
                vcpx<V> u[2][NC];
                res_project<2, false, NC>(0, own, u[0]);
                res_project<2, false, NC>(1, own, u[1]);
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    vcpx<V> k[2];
                    res_row<false, NC>(c, M, u, k);
                    to[c * nh] = slot_put(k[0]);
                    to[(NC + c) * nh] = slot_put(k[1]);
                }
            }
            if (bottom) {
                Slot *to = cl.map_shared_rank(e + H * nh, rank == 0 ? A.sh.ranks - 1 : rank - 1);
                vcpx<V> u[2][NC];
                res_project<2, true, NC>(0, own, u[0]);
                res_project<2, true, NC>(1, own, u[1]);
#pragma unroll
                for (int k = 0; k < H; k++) to[k * nh] = slot_put(u[k / NC][k % NC]);
            }
        }
    };
    // -i g0 / 2 of a component: spins 0, 1 times -i/2, spins 2, 3 times +i/2
    auto finish = [](const vcpx<V> &v, int a) {
        const V hp = vsplat<V>((T)(a < 2 ? 0.5 : -0.5)), hm = vsplat<V>((T)(a < 2 ? -0.5 : 0.5));
        return vcpx<V>{vmul(hp, v.im), vmul(hm, v.re)};
    };

    const int mode = slot * LN::kModes;
    const size_t base = (((size_t)(mode / kModeBlock) * L.V + z0 * n01 + s) * C * kModeBlock + mode % kModeBlock) /
                        LN::kModes;
    constexpr int kCompStride = kModeBlock / LN::kModes;
    const int ng = min(G, A.slots - first);  // modes of this cluster
    const size_t phi_stride = (size_t)L.V * ng;
    Slot *phi = kPhiShared ? buf + (size_t)2 * C * CAP + me
                           : reinterpret_cast<Slot *>(A.scratch) + (size_t)first * C * L.V + (z0 * n01 + s) * ng + g;
    // component by component in order
    auto phi_at = [&](const Slot *&q, int comp) {
        if constexpr (kPhiShared) return slot_get(phi[comp * CAP]);
        const Slot w = __ldcg(q);
        q += phi_stride;
        return slot_get(w);
    };
    arrive();  // the links are laid out, and the whole cluster runs
    wait();
    // b_K = c_K phi, b_{K+1} = 0
    vcpx<V> acc[NC][kSpin], b2[NC][kSpin];
#pragma unroll
    for (int c = 0; c < NC; c++)
#pragma unroll
        for (int a = 0; a < kSpin; a++) b2[c][a] = {vsplat<V>((T)0), vsplat<V>((T)0)};
    if (live) {
        const V cK = vsplat<V>(A.K & 2 ? -A.c[A.K] : A.c[A.K]);  // signed as below
        const Slot *in = reinterpret_cast<const Slot *>(A.phi) + base;
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int a = 0; a < kSpin; a++) {
                const int comp = c * kSpin + a;
                const vcpx<V> f = slot_load(in + comp * kCompStride);
                if constexpr (kPhiShared) phi[comp * CAP] = slot_put(f);
                else __stcg(phi + comp * phi_stride, slot_put(f));
                acc[c][a] = {vmul(cK, f.re), vmul(cK, f.im)};
            }
        publish(0, acc);
    }
    arrive();
    for (int k = A.K - 1; k >= 0; k--) {
        if (live) stencil(0, acc);
        wait();
        if (live) {
            outer(0, acc);
#pragma unroll
            for (int c = 0; c < NC; c++)
#pragma unroll
                for (int a = 0; a < kSpin; a++) acc[c][a] = finish(acc[c][a], a);
            publish(1, acc);
        }
        arrive();
        if (live) stencil(1, acc);
        wait();
        if (live) {
            outer(1, acc);
            // b_k = factor (a (-D w) + beta b_{k+1}) - b_{k+2} + c_k phi, three roundings.
            // The fields hold s_k b_k with s = +, +, -, -, ... from k = 0, so that
            // b_{k+2} is added and every sign is in a coefficient.
            const Slot *q = res_here(phi);
            const T factor = (T)(k & 1 ? -2 : k > 0 ? 2 : 1);
            const V fa = vsplat<V>(-factor * A.a), fb = vsplat<V>(factor * A.beta), ck = vsplat<V>(k & 2 ? -A.c[k] : A.c[k]);
#pragma unroll
            for (int c = 0; c < NC; c++)
#pragma unroll
                for (int a = 0; a < kSpin; a++) {
                    const vcpx<V> d = finish(acc[c][a], a), v1 = slot_get(buf[(size_t)(c * kSpin + a) * CAP + me]),
                                  f = phi_at(q, c * kSpin + a);
                    acc[c][a].re = vfma(fa, d.re, vfma(fb, v1.re, vfma(ck, f.re, b2[c][a].re)));
                    acc[c][a].im = vfma(fa, d.im, vfma(fb, v1.im, vfma(ck, f.im, b2[c][a].im)));
                    b2[c][a] = v1;
                }
            publish(0, acc);
        }
        arrive();
    }
    // chi = b_0; the overlap combination M [-i g0 (1 + m/2) phi + (1 - m/2) D chi].
    // After this wait nothing reaches another CTA's shared memory, so a CTA may
    // leave when it is done.
    if (live) stencil(0, acc);
    wait();
    if (live) {
        outer(0, acc);
        const Slot *in = phi;
        Slot *out = reinterpret_cast<Slot *>(A.dst) + base;
        const V mdw = vsplat<V>(A.mdw), cm = vsplat<V>(A.cm), dt = vsplat<V>(A.dt);
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int a = 0; a < kSpin; a++) {
                const vcpx<V> d = finish(acc[c][a], a), f = phi_at(in, c * kSpin + a);
                const V cr = vsplat<V>(a < 2 ? A.cp : -A.cp), ci = vsplat<V>(a < 2 ? -A.cp : A.cp);
                vcpx<V> o;
                o.re = vmul(mdw, vfma(cm, d.re, vmul(cr, f.im)));
                o.im = vmul(mdw, vfma(cm, d.im, vmul(ci, f.re)));
                Slot *q = out + (c * kSpin + a) * kCompStride;
                if (A.accumulate) {
                    const vcpx<V> v = slot_load(q);
                    o.re = vfma(dt, o.re, v.re);
                    o.im = vfma(dt, o.im, v.im);
                }
                slot_store(q, o);
            }
    }
}

// What a kernel is built for: the work of a thread and the threads per CTA, one CTA per SM.
template <class LN, int CAP> struct ResidentCap {
    using Lane = LN;
    static constexpr int kCap = CAP;
};

// Whole warps (capacities are multiples of 32).
inline int resident_threads(int n) { return (n + 31) / 32 * 32; }

// Offers capacity number `index` to the plan: the shape of the least time
// (resident_choose, ovl_rules.h), if it is less than the plan's so far, which
// starts at the time through memory.
// Per application at degree 24, through memory / here (us): 8^3, two colours, FP32,
// 32, 256, 1024 and 4096 modes 306/100, 406/158, 1250/590 and 4220/2160; 5^3 x 64
// 305/58 (one set of modes in each of 32 CTAs; 147 with four in each of 8);
// 12 x 11 x 10 x 2048 5440 through memory, which is taken, 6240 here; 8^3, three
// colours, FP64, 1024: 3500/2810 with two sets on 4 CTAs of 2 planes, 3760 with one on
// 3 of 3.
// Over 597 calls (51 pairs of lattice and storage, 32 to 4096 modes, degrees 24 and
// 96) the choice takes 0.5 to 2 % (geometric mean) more than the best of all shapes
// and memory, 18 calls over 3 % more than memory, none over 13 %.  A plan for the
// largest throughput whatever the number of modes took 12 to 17 % more than this one,
// 45 calls over 2 % and up to 23 % more than memory.  The 224 threads of three colours
// in FP64 hold planes of 110 to 112 sites in pairs or two sets of modes, which 256 do
// not: 8 x 14 x 6 x 4096 at degree 96 58.2 ms, 76.0 through memory.
template <int NC, bool U1, class Cap>
static void resident_offer(const Lattice &L, int index, int modes, int degree, ResidentPlan &pl) {
    using Lane = typename Cap::Lane;
    const int n01 = L.N0 * L.N1;
    const ResidentCall call{NC, sizeof(typename Lane::T) == 8, L.N0, L.N1, L.N2, modes / Lane::kModes, degree};
    const void *kernels[2] = {(const void *)resident_cheb_kernel<NC, Lane, U1, false, Cap::kCap>,
                              (const void *)resident_cheb_kernel<NC, Lane, U1, true, Cap::kCap>};
    int dev = 0, optin = 0;
    bool able = cudaGetDevice(&dev) == cudaSuccess &&
                cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess;
    for (const void *fn : kernels)
        able = able && cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin) == cudaSuccess;
    if (!able) {
        cudaGetLastError();
        return;
    }
    auto fits = [&](const ResidentShape &sh) {
        const size_t smem = ResidentLayout<NC, Lane>::bytes(Cap::kCap, sh, n01);
        if (smem > (size_t)optin) return 0;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = sh.ranks;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(sh.ranks);
        cfg.blockDim = dim3(resident_threads(n01 * sh.planes * sh.groups));
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernels[sh.ranks > 1], &cfg) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return clusters;
    };
    if (!resident_choose(call, Cap::kCap, current_sm_count(), fits, pl.sh, pl.us)) return;
    pl.ok = true;
    pl.kernel = index;
    pl.smem = ResidentLayout<NC, Lane>::bytes(Cap::kCap, pl.sh, n01);
}

template <int NC, bool U1, class Cap>
static cudaError_t resident_launch(const ResidentPlan &pl, const ResidentArgs<typename Cap::Lane::T> &a, cudaStream_t stream) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = pl.sh.ranks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.sh.ranks * ((a.slots + pl.sh.groups - 1) / pl.sh.groups));
    cfg.blockDim = dim3(resident_threads(a.L.N0 * a.L.N1 * pl.sh.planes * pl.sh.groups));
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (pl.sh.ranks > 1) return cudaLaunchKernelEx(&cfg, resident_cheb_kernel<NC, typename Cap::Lane, U1, true, Cap::kCap>, a);
    return cudaLaunchKernelEx(&cfg, resident_cheb_kernel<NC, typename Cap::Lane, U1, false, Cap::kCap>, a);
}

template <class... Caps> struct ResidentCaps {};

// The plan for n_mb mode blocks and a series of this degree with one of the
// capacities.  It is the context's: it holds sizes only, and is made again when they
// change.  Whether there is one.
template <int NC, typename T, bool U1, class... Caps>
static bool resident_plan(ResidentCaps<Caps...>, ResidentPlan &pl, const Lattice &L, int n_mb, int degree) {
    const int modes = n_mb * kModeBlock;
    if (pl.modes != modes || pl.degree != degree || pl.u1 != U1) {
        pl = ResidentPlan{};
        pl.modes = modes;
        pl.degree = degree;
        pl.u1 = U1;
        const ResidentCall call{NC, sizeof(T) == 8, L.N0, L.N1, L.N2, modes, degree};
        pl.us = through_memory_us(call, sizeof(cpx<T>) * NC * kSpin * (double)L.V * modes);
        int i = 0;
        (resident_offer<NC, U1, Caps>(L, i++, modes, degree, pl), ...);
    }
    return pl.ok;
}

// The operator on chip, if there is a plan for it.
template <int NC, typename T, bool U1, class... Caps>
static bool resident_apply(ResidentCaps<Caps...> caps, ResidentPlan &pl, const void *U, const void *u1, const void *src,
                           void *dst, const Lattice &L, int n_mb, void *scratch, const double *coeff, int K, double eps,
                           double lambda_max, double amass, double mdw, double mf, double dt, bool accumulate,
                           cudaStream_t stream, uint64_t *launches) {
    const int modes = n_mb * kModeBlock;
    if (!resident_plan<NC, T, U1>(caps, pl, L, n_mb, K)) return false;
    ResidentArgs<T> a;
    a.U = U;
    a.u1 = u1;
    a.phi = reinterpret_cast<const cpx<T> *>(src);
    a.dst = reinterpret_cast<cpx<T> *>(dst);
    a.scratch = reinterpret_cast<cpx<T> *>(scratch);
    a.L = L;
    a.sh = pl.sh;
    a.K = K;
    a.accumulate = accumulate ? 1 : 0;
    a.amass = (T)amass;
    a.a = (T)(2.0 / ((1.0 - eps) * lambda_max));
    a.beta = (T)(-(1.0 + eps) / (1.0 - eps));
    a.mdw = (T)mdw;
    a.cp = (T)(1.0 + 0.5 * mf);
    a.cm = (T)(1.0 - 0.5 * mf);
    a.dt = (T)dt;
    const double scale = 1.0 / std::sqrt(lambda_max);
    for (int k = 0; k <= K; k++) a.c[k] = (T)((k > 0 ? coeff[k] : 0.5 * coeff[0]) * scale);
    int i = 0;
    ((pl.kernel == i++ ? (a.slots = modes / Caps::Lane::kModes, (void)resident_launch<NC, U1, Caps>(pl, a, stream)) : (void)0),
     ...);
    if (launches) *launches += 1;
    return true;
}

}  // namespace ovl
