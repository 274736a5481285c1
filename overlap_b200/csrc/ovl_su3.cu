// Three-colour kernels: the Wilson leapfrog half step (plain and fused), the
// link update, the Chebyshev overlap operator, the charges, the improved E.B,
// the geodesic interpolation of Delta N_CS and the bulk observables, for
// 12-component modes and SU(3) links (layouts in ovl_su3.cuh).  Each follows
// the two-colour kernel of the same job (ovl_wilson.cu, ovl_chebyshev.cu,
// ovl_modes.cu, ovl_gauge.cu) with 3x3 links; the reference routines are
// cited there.
#include <algorithm>
#include <cmath>

#include "ovl_bilinears.cuh"
#include "ovl_internal.h"
#include "ovl_loops.cuh"
#include "ovl_resident.cuh"
#include "ovl_su3.cuh"
#include "ovl_su3_packed.cuh"

namespace ovl {

// ------------------------------------------------------------ hop kernel --
// MODE 0: out = D src; MODE 1: out += dt D src (the fused half step).
// CTAs per SM the register allocation must allow: FP32 6 (85 registers; 64 for 8 spill).
template <typename T> struct Occ3 { static constexpr int kMinBlocks = sizeof(T) == 4 ? 6 : 1; };

template <typename T, int MODE, class LK>
__global__ void __launch_bounds__(kModeBlock *kSites3, Occ3<T>::kMinBlocks)
    su3_wilson_kernel(LK lk, const cpx<T> *__restrict__ src, cpx<T> *__restrict__ out, Lattice L, int mb0, T amass,
                      T dt) {
    const int lane = threadIdx.x;
    const int site = blockIdx.x * kSites3 + threadIdx.y;
    const int mb = mb0 + blockIdx.y;
    if (site >= L.V) return;
    Spinor3<T> acc;
    wilson_site3(lk, src, L, site, mb, lane, amass, acc);
    cpx<T> *o = out + field_index3(L.V, MODE == 1 ? mb : blockIdx.y, site, 0, lane);
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int a = 0; a < kSpin; a++) {
            const cpx<T> v = acc.c[c][a];
            const cpx<T> d = (T)0.5 * (a < 2 ? times_mi(v) : times_i(v));  // -i gamma_0 / 2
            cpx<T> *p = o + (c * kSpin + a) * kModeBlock;
            if (MODE == 1) {
                const cpx<T> w = ld(p);
                st(p, w + dt * d);
            } else {
                st(p, d);
            }
        }
}

template <typename T, int MODE, bool F32, bool U1>
static void hop3_launch(const Su3Links &lk, const void *src, void *dst, const Lattice &L, int mb0, int n_mb, double amass,
                        double dt, cudaStream_t s) {
    const dim3 block(kModeBlock, kSites3), grid((L.V + kSites3 - 1) / kSites3, n_mb);
    Links3<F32, U1> links{F32 ? (const void *)lk.U32 : (const void *)lk.U, F32 ? (const void *)lk.u1_32 : (const void *)lk.u1,
                          L.N0 * L.N1};
    su3_wilson_kernel<T, MODE, Links3<F32, U1>><<<grid, block, 0, s>>>(
        links, reinterpret_cast<const cpx<T> *>(src), reinterpret_cast<cpx<T> *>(dst), L, mb0, (T)amass, (T)dt);
}

// The packed-pair stencil (variant 3, FP32): CTAs of kPk3Warps warps (2
// kPk3Warps sites) running kPk3Blocks mode blocks each on one set of link
// records.  MODE 0: dst = D src, 1: dst += dt D src, 2: the Clenshaw term.
constexpr int kPk3Warps = 4, kPk3Sites = 2 * kPk3Warps, kPk3Blocks = 8, kPk3MinBlocks = 3;

template <int MODE, bool U1>
__global__ void __launch_bounds__(kModeBlock *kPk3Warps, kPk3MinBlocks)
    su3_packed_kernel(const float4 *__restrict__ U32, const float2 *__restrict__ u1, const float4 *__restrict__ src,
                      float4 *__restrict__ dst, Lattice L, int n_mb, float amass, float hdt, const ClenshawArgs cl) {
    __shared__ float4 rec[kPk3Sites][6][kPk3RecVec];
    const int mb0 = blockIdx.y * kPk3Blocks;
    packed_tile3<MODE, U1, kPk3Warps>(rec, U32, u1, src, dst, L, blockIdx.x * kPk3Sites, mb0,
                                      min(n_mb, mb0 + kPk3Blocks), amass, hdt, cl);
}

template <int MODE>
static void packed3_launch(const Su3Links &lk, const void *src, void *dst, const Lattice &L, int n_mb, double amass,
                           double dt, const ClenshawArgs &cl, cudaStream_t s) {
    const dim3 block(kModeBlock, kPk3Warps), grid((L.V + kPk3Sites - 1) / kPk3Sites, (n_mb + kPk3Blocks - 1) / kPk3Blocks);
    const float4 *U = reinterpret_cast<const float4 *>(lk.U32);
    const float4 *a = reinterpret_cast<const float4 *>(src);
    float4 *d = reinterpret_cast<float4 *>(dst);
    const float am = (float)amass, h = (float)(0.5 * dt);
    if (lk.u1_32)
        su3_packed_kernel<MODE, true><<<grid, block, 0, s>>>(U, reinterpret_cast<const float2 *>(lk.u1_32), a, d, L,
                                                             n_mb, am, h, cl);
    else
        su3_packed_kernel<MODE, false><<<grid, block, 0, s>>>(U, nullptr, a, d, L, n_mb, am, h, cl);
}

static bool packed3(const Su3Links &lk, size_t elem) { return elem == 4 && lk.variant == kPackedVariant && lk.U32; }

template <typename T>
void su3_launch_hop(const Su3Links &lk, const void *src, void *dst, const Lattice &L, int mb0, int n_mb, double amass,
                    double dt, bool accumulate, cudaStream_t s) {
    constexpr bool F32 = sizeof(T) == 4;
    if (packed3(lk, sizeof(T))) {
        const size_t off = field_index3(L.V, mb0, 0, 0, 0);
        const cpx<T> *a = reinterpret_cast<const cpx<T> *>(src) + off;
        cpx<T> *d = reinterpret_cast<cpx<T> *>(dst) + (accumulate ? off : 0);
        if (accumulate) packed3_launch<1>(lk, a, d, L, n_mb, amass, dt, ClenshawArgs{}, s);
        else packed3_launch<0>(lk, a, d, L, n_mb, amass, 0.0, ClenshawArgs{}, s);
        return;
    }
    const bool u1 = F32 ? lk.u1_32 != nullptr : lk.u1 != nullptr;
    if (accumulate) {
        if (u1) hop3_launch<T, 1, F32, true>(lk, src, dst, L, mb0, n_mb, amass, dt, s);
        else hop3_launch<T, 1, F32, false>(lk, src, dst, L, mb0, n_mb, amass, dt, s);
    } else {
        if (u1) hop3_launch<T, 0, F32, true>(lk, src, dst, L, mb0, n_mb, amass, dt, s);
        else hop3_launch<T, 0, F32, false>(lk, src, dst, L, mb0, n_mb, amass, dt, s);
    }
}

// ----------------------------------------------------------- link update --
// U <- exp(i cU t^a E^a) U (Dynamics.cpp:97-138, cU = -dt_step), optionally
// projected back onto SU(3), with the FP32 copy kept.
__global__ void su3_links_kernel(double *U, const double *__restrict__ E, int n_links, double c, float *U32, int reunit) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= n_links) return;
    const int site = l / 3, mu = l % 3;
    double e[8];
#pragma unroll
    for (int a = 0; a < 8; a++) e[a] = E[8 * (size_t)l + a];
    cmat3<double> u = m3_mul(su3_exp(c, e), load_su3(U, site, mu));
    if (reunit) u = su3_reunitarize(u);
    store_su3(U, site, mu, u);
    if (U32) {
        float2 *p = reinterpret_cast<float2 *>(U32 + (size_t)kLink32Floats * l);
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
            for (int j = 0; j < 3; j++) p[i + 3 * j] = float2{(float)u.m[i][j].re, (float)u.m[i][j].im};
        p[9] = float2{0.0f, 0.0f};
    }
}

void su3_launch_update_links(double *U, const double *E, const Lattice &L, double dt_step, float *U32, bool reunit,
                             cudaStream_t s) {
    const int n = 3 * L.V;
    su3_links_kernel<<<(n + 127) / 128, 128, 0, s>>>(U, E, n, -dt_step, U32, reunit ? 1 : 0);
}

// --------------------------------------------------------- Chebyshev sign --
// One Clenshaw term b_out = factor (a (-D w) + beta b1) - s2 b2 + ck phi, -D w
// the stencil applied to w = D b1 (ovl_chebyshev.cu, three colours).
template <typename T, class LK>
__global__ void __launch_bounds__(kModeBlock *kSites3, Occ3<T>::kMinBlocks)
    su3_clenshaw_kernel(LK lk, const cpx<T> *__restrict__ w, const cpx<T> *__restrict__ b1,
                        const cpx<T> *__restrict__ b2, const cpx<T> *__restrict__ phi, cpx<T> *__restrict__ bout,
                        Lattice L, T amass, T a, T beta, T factor, T s2, T ck) {
    const int lane = threadIdx.x;
    const int site = blockIdx.x * kSites3 + threadIdx.y;
    const int mb = blockIdx.y;
    if (site >= L.V) return;
    Spinor3<T> acc;
    wilson_site3(lk, w, L, site, mb, lane, amass, acc);
    const size_t base = field_index3(L.V, mb, site, 0, lane);
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int s = 0; s < kSpin; s++) {
            const size_t i = base + (c * kSpin + s) * kModeBlock;
            const cpx<T> v = acc.c[c][s];
            const cpx<T> dw = (T)0.5 * (s < 2 ? times_mi(v) : times_i(v));
            const cpx<T> v1 = ld(b1 + i), v2 = ld(b2 + i), f = ld(phi + i);
            const cpx<T> tx = mk<T>(-a * dw.re + beta * v1.re, -a * dw.im + beta * v1.im);
            st(bout + i, mk<T>(factor * tx.re - s2 * v2.re + ck * f.re, factor * tx.im - s2 * v2.im + ck * f.im));
        }
}

// out = M [ -i g0 (1 + m/2) phi + (1 - m/2) dchi ];  dst = out or dst += dt out
template <typename T>
__global__ void su3_overlap_finish_kernel(const cpx<T> *__restrict__ phi, const cpx<T> *__restrict__ dchi, cpx<T> *dst,
                                          size_t n, T mdw, T mf, T dt, int accumulate) {
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int spin = (int)((e / kModeBlock) % kSpin);
        const cpx<T> f = ld(phi + e), d = ld(dchi + e);
        const T cp = (T)1 + (T)0.5 * mf, cm = (T)1 - (T)0.5 * mf;
        const cpx<T> g = spin < 2 ? mk<T>(cp * f.im, -cp * f.re) : mk<T>(-cp * f.im, cp * f.re);
        const cpx<T> o = mk<T>(mdw * (g.re + cm * d.re), mdw * (g.im + cm * d.im));
        if (accumulate) {
            const cpx<T> v = ld(dst + e);
            st(dst + e, mk<T>(v.re + dt * o.re, v.im + dt * o.im));
        } else {
            st(dst + e, o);
        }
    }
}

template <typename T>
using Caps3 = ResidentCaps<ResidentCap<LaneOne<T>, sizeof(T) == 4 ? 512 : 256>, ResidentCap<LaneOne<T>, sizeof(T) == 4 ? 576 : 224>>;

template <typename T>
bool su3_chebyshev_on_chip(ChebyshevWork &w, const Su3Links &lk, const Lattice &L, int n_mb, int degree) {
    const bool u1 = sizeof(T) == 4 ? lk.u1_32 != nullptr : lk.u1 != nullptr;
    return u1 ? resident_plan<3, T, true>(Caps3<T>{}, w.resident, L, n_mb, degree)
              : resident_plan<3, T, false>(Caps3<T>{}, w.resident, L, n_mb, degree);
}
template bool su3_chebyshev_on_chip<float>(ChebyshevWork &, const Su3Links &, const Lattice &, int, int);

template <typename T, bool F32, bool U1>
static void cheb3(ChebyshevWork &w, const Su3Links &lk, const void *src, void *dst, const Lattice &L, int n_mb,
                  const double *coeff, int K, double eps, double lambda_max, double amass, double mdw, double mf,
                  double dt, bool accumulate, int sm_count, cudaStream_t stream, uint64_t *launches) {
    if (!w.through_memory &&
        resident_apply<3, T, U1>(
            Caps3<T>{}, w.resident, F32 ? (const void *)lk.U32 : (const void *)lk.U, F32 ? (const void *)lk.u1_32 : (const void *)lk.u1,
            src, dst, L, n_mb, w.b0, coeff, K, eps, lambda_max, amass, mdw, mf, dt, accumulate, stream, launches))
        return;
    const size_t n = (size_t)n_mb * L.V * kComp3 * kModeBlock;
    const dim3 block(kModeBlock, kSites3), grid((L.V + kSites3 - 1) / kSites3, n_mb);
    Links3<F32, U1> links{F32 ? (const void *)lk.U32 : (const void *)lk.U, F32 ? (const void *)lk.u1_32 : (const void *)lk.u1,
                          L.N0 * L.N1};
    const cpx<T> *phi = reinterpret_cast<const cpx<T> *>(src);
    cpx<T> *b[3] = {reinterpret_cast<cpx<T> *>(w.b0), reinterpret_cast<cpx<T> *>(w.b1), reinterpret_cast<cpx<T> *>(w.b2)};
    cpx<T> *tmp = reinterpret_cast<cpx<T> *>(w.w);
    const double scale = 1.0 / std::sqrt(lambda_max);
    const T a = (T)(2.0 / ((1.0 - eps) * lambda_max)), beta = (T)(-(1.0 + eps) / (1.0 - eps)), am = (T)amass;
    int i1 = 1, i2 = 2, io = 0;
    uint64_t nl = 0;
    // variant 3 (FP32): the D passes in the packed stencil, and the overlap
    // combination fused into the last one
    const bool pk = packed3(lk, sizeof(T));
    // b_K = c_K phi is not formed (cheb_run, ovl_chebyshev.cu)
    const T cK = (T)(coeff[K] * scale);
    for (int k = K - 1; k >= 0; k--) {
        const cpx<T> *b1 = k == K - 1 ? phi : b[i1], *b2 = k >= K - 2 ? phi : b[i2];
        const T s1 = k == K - 1 ? cK : (T)1, s2 = k == K - 1 ? (T)0 : (k == K - 2 ? cK : (T)1);
        const T factor = s1 * (T)(k > 0 ? 2 : 1), ck = (T)((k > 0 ? coeff[k] : 0.5 * coeff[0]) * scale);
        if (pk) packed3_launch<0>(lk, b1, tmp, L, n_mb, amass, 0.0, ClenshawArgs{}, stream);
        else su3_wilson_kernel<T, 0, Links3<F32, U1>><<<grid, block, 0, stream>>>(links, b1, tmp, L, 0, am, (T)0);
        su3_clenshaw_kernel<T, Links3<F32, U1>><<<grid, block, 0, stream>>>(links, tmp, b1, b2, phi, b[io], L, am, a, beta,
                                                                            factor, s2, ck);
        nl += 2;
        const int t = i2;
        i2 = i1;
        i1 = io;
        io = t;
    }
    // chi = b[i1]; D chi, then the overlap combination (one pass of the
    // packed stencil with the combination in its epilogue)
    if (pk) {
        ClenshawArgs cl{};
        cl.phi = reinterpret_cast<const float4 *>(phi);
        cl.mdw = (float)mdw;
        cl.cp = (float)(1.0 + 0.5 * mf);
        cl.cm = (float)(1.0 - 0.5 * mf);
        cl.dt = (float)dt;
        cl.accumulate = accumulate ? 1 : 0;
        packed3_launch<3>(lk, b[i1], dst, L, n_mb, amass, 0.0, cl, stream);
        nl += 1;
        if (launches) *launches += nl;
        return;
    }
    su3_wilson_kernel<T, 0, Links3<F32, U1>><<<grid, block, 0, stream>>>(links, b[i1], tmp, L, 0, am, (T)0);
    const size_t blocks = (n + 255) / 256, cap = (size_t)sm_count * 16;
    su3_overlap_finish_kernel<T><<<(int)std::min(blocks, cap), 256, 0, stream>>>(
        phi, tmp, reinterpret_cast<cpx<T> *>(dst), n, (T)mdw, (T)mf, (T)dt, accumulate ? 1 : 0);
    nl += 2;
    if (launches) *launches += nl;
}

template <typename T>
void su3_chebyshev_apply(ChebyshevWork &w, const Su3Links &lk, const void *src, void *dst, const Lattice &L, int n_mb,
                         const double *coeff, int K, double eps, double lambda_max, double amass, double mdw, double mf,
                         double dt, bool accumulate, int sm_count, cudaStream_t stream, uint64_t *launches) {
    constexpr bool F32 = sizeof(T) == 4;
    const bool u1 = F32 ? lk.u1_32 != nullptr : lk.u1 != nullptr;
    if (u1)
        cheb3<T, F32, true>(w, lk, src, dst, L, n_mb, coeff, K, eps, lambda_max, amass, mdw, mf, dt, accumulate, sm_count,
                            stream, launches);
    else
        cheb3<T, F32, false>(w, lk, src, dst, L, n_mb, coeff, K, eps, lambda_max, amass, mdw, mf, dt, accumulate, sm_count,
                             stream, launches);
}

// Sums `n` partial rows of `nv` values in a fixed order (one CTA: a strided
// sum per thread, then a tree), scaled.
template <int NV>
__global__ void su3_sum_rows_kernel(const double *__restrict__ partial, int n, double scale, double *__restrict__ out) {
    partial += (size_t)blockIdx.x * n * NV;  // one CTA per result
    out += blockIdx.x * NV;
    __shared__ double sh[256][NV];
    CompSum t[NV];
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        for (int k = 0; k < NV; k++) t[k].add(partial[(size_t)i * NV + k]);
    for (int k = 0; k < NV; k++) sh[threadIdx.x][k] = t[k].value();
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w)
            for (int k = 0; k < NV; k++) sh[threadIdx.x][k] += sh[threadIdx.x + w][k];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int k = 0; k < NV; k++) out[k] = scale * sh[0][k];
}

// V (t^b e^b) V^+ as components: the adjoint transport R(V) e, R_ab = 2 tr(t^a V t^b V^+).
__device__ inline void su3_transport(const cmat3<double> &V, const double *e, double *out) {
    const cmat3<double> A = su3_form(e);
    su3_components(m3_mul(m3_mul(V, A), m3_dag(V)), out);
}

constexpr int kReduce3Threads = 128;

__device__ inline double block_sum(double v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[w];
    __syncthreads();
    return t;
}

// Improved E.B (ChernSimonsOperators.cpp:128-439): four lanes per (site,
// direction), lane q with quadrant q of B_mu and term q of E_mu, as
// ncsdot_kernel of ovl_gauge.cu; blockIdx.y: the link field.
struct NcsSets3 {
    const double *U[3];
};

__global__ void __launch_bounds__(kReduce3Threads)
    su3_ncsdot_kernel(const NcsSets3 sets, const double *__restrict__ E, Lattice L, double *__restrict__ partial) {
    __shared__ double sh[32];
    const double *__restrict__ U = sets.U[blockIdx.y];
    CompSum sum;
    const long long items = 12LL * L.V, stride = (long long)gridDim.x * kReduce3Threads;
    for (long long t0 = (long long)blockIdx.x * kReduce3Threads + (threadIdx.x & ~31); t0 < items; t0 += stride) {
        const long long t = t0 + (threadIdx.x & 31);
        const bool live = t < items;  // padded lanes repeat site 0: the shuffles need the whole warp
        const int q = (int)(t & 3), sd = live ? (int)(t >> 2) : 0;
        const int s = sd / 3, mu = sd % 3;
        int c[3];
        site_coords(L, s, c[0], c[1], c[2]);
        double e[8], b[8];
        {
            int es;
            cmat3<double> V;
            double w;
            improved_e_term<Su3Ops>(U, L, s, c, mu, q, es, V, w);
            su3_transport(V, E + 8 * (mu + 3 * (size_t)es), e);
#pragma unroll
            for (int a = 0; a < 8; a++) e[a] *= w;
        }
#pragma unroll
        for (int a = 0; a < 8; a++) b[a] = 0.0;
        const Quadrant quad(L, s, c, mu == 2 ? 0 : mu + 1, mu == 0 ? 2 : mu - 1, q);
        quad.loops<Su3Ops>(U, [&](const cmat3<double> &p, double f) {
            double g[8];
            su3_retr_ita(p, g);
#pragma unroll
            for (int a = 0; a < 8; a++) b[a] += f * g[a];
        });
        double eb = 0.0;
#pragma unroll
        for (int a = 0; a < 8; a++) eb += quad_sum(e[a]) * (2.0 * quad_sum(b[a]));
        if (live && q == 0) sum.add(eb);
    }
    const double tot = block_sum(sum.value(), sh);
    if (threadIdx.x == 0) partial[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = tot;
}

size_t su3_reduce_partial_doubles(const Lattice &L) {
    return (size_t)std::max(11 * ((L.V + kReduce3Threads - 1) / kReduce3Threads), 1);
}

// partial holds ncsdot_partial_doubles
static void su3_ncsdot_sets(const NcsSets3 &sets, int n, const double *E, const Lattice &L, double *partial,
                            double *out, cudaStream_t s) {
    const int nb = ncsdot_blocks(L);
    su3_ncsdot_kernel<<<dim3(nb, n), kReduce3Threads, 0, s>>>(sets, E, L, partial);
    su3_sum_rows_kernel<1><<<n, 256, 0, s>>>(partial, nb, 0.125 / (M_PI * M_PI), out);
}

void su3_launch_ncsdot(const double *U, const double *E, const Lattice &L, double *partial, double *out, cudaStream_t s) {
    su3_ncsdot_sets(NcsSets3{{U, U, U}}, 1, E, L, partial, out, s);
}

void su3_launch_ncsdot3(const double *U0, const double *U1, const double *U2, const double *E, const Lattice &L,
                        double *partial, double *out3, cudaStream_t s) {
    su3_ncsdot_sets(NcsSets3{{U0, U1, U2}}, 3, E, L, partial, out3, s);
}

// ---------------------------------------------------- geodesic interpolation --
// Eigensystem of a hermitian 3x3 matrix by cyclic Jacobi rotations (each
// rotation diag(1, e^{-i phi}) R(theta) on a pair (p, q), a_pq = r e^{i phi},
// tan 2 theta = 2 r / (a_qq - a_pp)); columns of Vec are the eigenvectors.
__device__ inline void herm3_eigen(cmat3<double> A, cmat3<double> &Vec) {
    Vec = m3_unit<double>();
    for (int sweep = 0; sweep < 32; sweep++) {
        double off = 0.0, diag = 0.0;
        for (int i = 0; i < 3; i++) {
            diag += A.m[i][i].re * A.m[i][i].re;
            for (int j = i + 1; j < 3; j++) off += A.m[i][j].re * A.m[i][j].re + A.m[i][j].im * A.m[i][j].im;
        }
        if (off <= 1e-34 * diag || off < 1e-300) break;
        for (int p = 0; p < 2; p++)
            for (int q = p + 1; q < 3; q++) {
                const double r = sqrt(A.m[p][q].re * A.m[p][q].re + A.m[p][q].im * A.m[p][q].im);
                if (r == 0.0) continue;
                const cpx<double> phc = mk<double>(A.m[p][q].re / r, -A.m[p][q].im / r);  // e^{-i phi}
                const double th = 0.5 * atan2(2.0 * r, A.m[q][q].re - A.m[p][p].re);
                double sn, cs;
                sincos(th, &sn, &cs);
                cmat3<double> J = m3_unit<double>();
                J.m[p][p] = mk<double>(cs, 0.0);
                J.m[p][q] = mk<double>(sn, 0.0);
                J.m[q][p] = -sn * phc;
                J.m[q][q] = cs * phc;
                A = m3_mul(m3_dag(J), m3_mul(A, J));
                Vec = m3_mul(Vec, J);
            }
    }
}

// A^a with exp(-i A^a t^a) = W (MatrixILog with C = -1,
// SU3/AlgebraOperations.cpp:186-234), through the eigenvectors of the hermitian
// H = (W + W^+)/2 + (W - W^+)/2i, which are W's while no two of its
// eigenphases add up to pi/2 (nearby links); phases made to sum to zero.
__device__ inline void su3_log(const cmat3<double> &W, double *out) {
    const cmat3<double> Wd = m3_dag(W);
    cmat3<double> H, Vec;
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++) {
            const cpx<double> s = W.m[i][j] + Wd.m[i][j], d = W.m[i][j] - Wd.m[i][j];
            H.m[i][j] = mk<double>(0.5 * s.re - 0.5 * d.im, 0.5 * s.im + 0.5 * d.re);  // s/2 - i d/2
        }
    herm3_eigen(H, Vec);
    double th[3], sum = 0.0;
    for (int j = 0; j < 3; j++) {
        cpx<double> e = mk<double>(0.0, 0.0);
        for (int i = 0; i < 3; i++)
            for (int k = 0; k < 3; k++) e = e + conj(Vec.m[i][j]) * W.m[i][k] * Vec.m[k][j];
        th[j] = atan2(e.im, e.re);
        sum += th[j];
    }
    if (fabs(sum) > M_PI) {
        int big = 0;
        for (int j = 1; j < 3; j++)
            if (fabs(th[j]) > fabs(th[big])) big = j;
        th[big] -= sum > 0 ? 2.0 * M_PI : -2.0 * M_PI;
        sum = th[0] + th[1] + th[2];
    }
    cmat3<double> G;  // -sum_j theta_j v_j v_j^+ = A^a t^a
    for (int i = 0; i < 3; i++)
        for (int k = 0; k < 3; k++) {
            cpx<double> t = mk<double>(0.0, 0.0);
            for (int j = 0; j < 3; j++) t = t + (th[j] - sum / 3.0) * (Vec.m[i][j] * conj(Vec.m[k][j]));
            G.m[i][k] = mk<double>(-t.re, -t.im);
        }
    su3_components(G, out);
}

// GeodesicInterpolation (SUNc/AdvancedOperations.cpp:432-443) for three
// colours: E_mid = A with exp(-i A t) = U_new U_old^+, U_mid = exp(-i c A t) U_old.
__global__ void su3_geodesic_kernel(const double *__restrict__ Uold, const double *__restrict__ Unew, double c,
                                    double *Umid, double *Emid, int n_links) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= n_links) return;
    const int site = l / 3, mu = l % 3;
    const cmat3<double> uo = load_su3(Uold, site, mu);
    double e[8];
    su3_log(m3_mul(load_su3(Unew, site, mu), m3_dag(uo)), e);
    for (int a = 0; a < 8; a++) Emid[8 * (size_t)l + a] = e[a];
    store_su3(Umid, site, mu, m3_mul(su3_exp(-c, e), uo));
}

void su3_launch_geodesic(const double *Uold, const double *Unew, double c, double *Umid, double *Emid, const Lattice &L,
                         cudaStream_t s) {
    const int n = 3 * L.V;
    su3_geodesic_kernel<<<(n + 127) / 128, 128, 0, s>>>(Uold, Unew, c, Umid, Emid, n);
}

// ------------------------------------------------------------ staple force --
// E^a_mu(x) += -2 dt sum_{nu != mu} [Re tr(i t^a U_{mu,nu}) + Re tr(i t^a U_{mu,-nu})]
// (Dynamics.cpp:145-197; update_efield_kernel of ovl_gauge.cu for three colours).
// Four lanes per link, a plaquette each (update_efield_kernel of ovl_gauge.cu).
__global__ void su3_efield_kernel(const double *__restrict__ U, double *E, Lattice L, double gamma) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, q = t & 3;
    const bool live = t < 12 * L.V;  // padded lanes repeat link 0: the shuffles need the whole warp
    const int l = live ? t >> 2 : 0;
    double f[8];
    su3_retr_ita(staple_plaquette<Su3Ops>(U, L, l, q), f);
#pragma unroll
    for (int k = 0; k < 8; k++) f[k] = quad_sum(f[k]);
    if (!live) return;
#pragma unroll
    for (int k = 0; k < 8; k++)
        if ((k & 3) == q) E[8 * (size_t)l + k] += gamma * f[k];
}

// The force of every link reads the links only, so one pass updates E in place.
void su3_launch_update_efield(const double *U, double *E, const Lattice &L, double dt_step, cudaStream_t s) {
    su3_efield_kernel<<<(12 * L.V + 127) / 128, 128, 0, s>>>(U, E, L, -2.0 * dt_step);
}

// ------------------------------------------------------ Gauss restoration --
// GaussLawRestoration (GAUSSLAWFIXING/GaussRestore.cpp:13-168) for three
// colours: G^a(x) = sum_mu E_mu(x) - R(U_mu(x-mu)^+) E_mu(x-mu) into G (8 per
// site), CTA partial sums of G^2 and signed maxima (from 0).
__global__ void __launch_bounds__(kReduce3Threads)
    su3_gauss_violation_kernel(const double *__restrict__ U, const double *__restrict__ E, Lattice L, double *G,
                               double *partial) {
    __shared__ double sh[32];
    double sum = 0.0, mx = 0.0;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < L.V) {
        int x, y, z;
        site_coords(L, s, x, y, z);
        double g[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int mu = 0; mu < 3; mu++) {
            int c[3] = {x, y, z};
            c[mu] -= 1;
            const int sm = site_index(L, c[0], c[1], c[2]);
            double t[8];
            su3_transport(m3_dag(load_su3(U, sm, mu)), E + 8 * (mu + 3 * sm), t);
            for (int a = 0; a < 8; a++) g[a] += E[a + 8 * (mu + 3 * s)] - t[a];
        }
        for (int a = 0; a < 8; a++) {
            G[a + 8 * (size_t)s] = g[a];
            sum += g[a] * g[a];
            mx = fmax(mx, g[a]);
        }
    }
    const double tsum = block_sum(sum, sh);
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) m = fmax(m, sh[w]);
        partial[2 * blockIdx.x] = tsum;
        partial[2 * blockIdx.x + 1] = m;
    }
}

__global__ void su3_gauss_finish_kernel(const double *__restrict__ partial, int n, double *out2) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double sum = 0.0, mx = 0.0;
    for (int i = 0; i < n; i++) {
        sum += partial[2 * i];
        mx = fmax(mx, partial[2 * i + 1]);
    }
    out2[0] = sum;
    out2[1] = mx;
}

// E_mu(x) -= gamma (G(x) - R(U_mu(x)) G(x + mu))   (GaussRestore.cpp:72-118)
__global__ void su3_gauss_update_kernel(const double *__restrict__ U, const double *__restrict__ G,
                                        double *__restrict__ E, Lattice L, double gamma) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * L.V) return;
    const int s = t / 3, mu = t % 3;
    int x, y, z;
    site_coords(L, s, x, y, z);
    int c[3] = {x, y, z};
    c[mu] += 1;
    const int sp = site_index(L, c[0], c[1], c[2]);
    double up[8];
    su3_transport(load_su3(U, s, mu), G + 8 * (size_t)sp, up);
    for (int a = 0; a < 8; a++) E[a + 8 * (size_t)t] -= gamma * (G[a + 8 * (size_t)s] - up[a]);
}

void su3_launch_gauss_violation(const double *U, const double *E, const Lattice &L, double *G, double *partial,
                                double *out2, cudaStream_t s) {
    const int nb = (L.V + kReduce3Threads - 1) / kReduce3Threads;
    su3_gauss_violation_kernel<<<nb, kReduce3Threads, 0, s>>>(U, E, L, G, partial);
    su3_gauss_finish_kernel<<<1, 32, 0, s>>>(partial, nb, out2);
}

void su3_launch_gauss_update(const double *U, const double *G, double *E, const Lattice &L, double gamma,
                             cudaStream_t s) {
    const int n = 3 * L.V;
    su3_gauss_update_kernel<<<(n + 127) / 128, 128, 0, s>>>(U, G, E, L, gamma);
}

// ------------------------------------------------------------ back-reaction --
// The fermion force on E for three colours (ovl_force.cu with 3x3 links and
// t^a = lambda^a / 2): per site and mu the link-independent colour bilinears
//   C_ij = sum_m w_m sum_ab conj(psi_ia(x)) [g0 (1 - G_mu)]_ab psi_jb(x+mu),
// then dH_F/dtheta^a = (1/2V) Im tr(t^a Q), Q = M C^T, M the dressed link.
constexpr int kForce3PerSite = 3 * 18;  // mu, (i, j), (re, im)

// One direction mu per blockIdx.z: the 18 sums of one mu beside the spinor fit
// the registers, the 54 of all three do not.
template <typename T, int MU>
__device__ __forceinline__ void su3_force_modes(const SrcPlain<T> &psi, const Lattice &L, int n_mb, int n_modes,
                                                int first_mode, int site, double *__restrict__ partial) {
    const int lane = threadIdx.x, g = blockIdx.y, groups = gridDim.y;
    const Nbrs n = neighbours(L, site);
    const int nb = MU == 0 ? n.xp : (MU == 1 ? n.yp : n.zp);
    double acc[32];  // 18 used
#pragma unroll
    for (int k = 0; k < 32; k++) acc[k] = 0.0;
    for (int mb = g; mb < n_mb; mb += groups) {
        const double w = vacuum_weight(mb * kModeBlock + lane, n_modes, first_mode);
        SiteRaw<3, SrcPlain<T>> raw;
        raw.load(psi, L.V, mb, site, lane);
        cpx<double> f[3][kSpin];
#pragma unroll
        for (int k = 0; k < kComp3; k++) f[k / kSpin][k % kSpin] = w * raw.get(k);
        raw.load(psi, L.V, mb, nb, lane);
        add_colour_pairs<3, MU>(f, raw, acc);
    }
    const double total = warp_sum32(acc);
    if (lane < 18) partial[((size_t)g * L.V + site) * kForce3PerSite + 18 * MU + lane] = total;
}

template <typename T>
__global__ void __launch_bounds__(kModeBlock *kSites3, 3)
    su3_force_modes_kernel(SrcPlain<T> psi, Lattice L, int n_mb, int n_modes, int first_mode,
                           double *__restrict__ partial) {
    const int site = blockIdx.x * kSites3 + threadIdx.y;
    if (site >= L.V) return;  // whole warps exit together
    if (blockIdx.z == 0) su3_force_modes<T, 0>(psi, L, n_mb, n_modes, first_mode, site, partial);
    else if (blockIdx.z == 1) su3_force_modes<T, 1>(psi, L, n_mb, n_modes, first_mode, site, partial);
    else su3_force_modes<T, 2>(psi, L, n_mb, n_modes, first_mode, site, partial);
}

// One warp per (site, mu): lane k < 18 sums C's value k over the groups, every
// lane contracts C with the dressed link, and lane a < 8 writes.  out != null:
// out[a + 8 (mu + 3 site)] = dH_F/dtheta^a; otherwise
// E[a + 8 (mu + 3 site)] += coef dH_F/dtheta^a.
template <bool U1>
__global__ void su3_force_finish_kernel(const double *__restrict__ partial, int groups, const double *__restrict__ U,
                                        const double *__restrict__ u1, Lattice L, double *__restrict__ out,
                                        double *__restrict__ E, double coef) {
    const int t = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (t >= 3 * L.V) return;  // whole warps exit together
    const int site = t / 3, mu = t % 3;
    double v = 0.0;
    if (lane < 18)
        for (int g = 0; g < groups; g++) v += partial[((size_t)g * L.V + site) * kForce3PerSite + 18 * mu + lane];
    cmat3<double> C;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++)
            C.m[i][j] = mk<double>(__shfl_sync(0xffffffffu, v, 2 * (3 * i + j)), __shfl_sync(0xffffffffu, v, 2 * (3 * i + j) + 1));
    const Links3<false, U1> lk{U, u1, L.N0 * L.N1};
    const cmat3<double> M = lk.template get<double>(site, mu);
    cmat3<double> Q;  // M C^T
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
        for (int i = 0; i < 3; i++) Q.m[k][i] = M.m[k][0] * C.m[i][0] + M.m[k][1] * C.m[i][1] + M.m[k][2] * C.m[i][2];
    if (lane >= 8) return;
    // Im tr(t^a Q) per generator (t^a = lambda^a / 2)
    const double r3 = 0.57735026918962576451;
    double f[8];
    f[0] = 0.5 * (Q.m[1][0].im + Q.m[0][1].im);
    f[1] = 0.5 * (Q.m[0][1].re - Q.m[1][0].re);  // Im((-i Q10 + i Q01)/2)
    f[2] = 0.5 * (Q.m[0][0].im - Q.m[1][1].im);
    f[3] = 0.5 * (Q.m[2][0].im + Q.m[0][2].im);
    f[4] = 0.5 * (Q.m[0][2].re - Q.m[2][0].re);
    f[5] = 0.5 * (Q.m[2][1].im + Q.m[1][2].im);
    f[6] = 0.5 * (Q.m[1][2].re - Q.m[2][1].re);
    f[7] = 0.5 * r3 * (Q.m[0][0].im + Q.m[1][1].im - 2.0 * Q.m[2][2].im);
    double fa = f[0];
#pragma unroll
    for (int a = 1; a < 8; a++) fa = lane == a ? f[a] : fa;
    fa *= 1.0 / (2.0 * L.V);
    const size_t o = 8 * (size_t)t + lane;
    if (out) out[o] = fa;
    else E[o] += coef * fa;
}

int su3_force_groups(int n_mb) { return n_mb < 16 ? n_mb : 16; }

size_t su3_force_partial_doubles(const Lattice &L, int n_mb) {
    return (size_t)su3_force_groups(n_mb) * L.V * kForce3PerSite;
}

template <typename T>
void su3_launch_color_force(const double *U, const double *u1, const void *psi, const Lattice &L, int n_mb, int n_modes,
                            int first_mode, double *partial, double *out, double *E, double coef, cudaStream_t s) {
    const int groups = su3_force_groups(n_mb);
    const dim3 block(kModeBlock, kSites3), grid((L.V + kSites3 - 1) / kSites3, groups, 3);
    su3_force_modes_kernel<T><<<grid, block, 0, s>>>(SrcPlain<T>{reinterpret_cast<const cpx<T> *>(psi)}, L, n_mb, n_modes,
                                                     first_mode, partial);
    const int n = (3 * L.V + 3) / 4;  // four links (warps) per CTA
    if (u1) su3_force_finish_kernel<true><<<n, 128, 0, s>>>(partial, groups, U, u1, L, out, E, coef);
    else su3_force_finish_kernel<false><<<n, 128, 0, s>>>(partial, groups, U, u1, L, out, E, coef);
}

// sum_m w_m Re <psi_m, i (D psi)_m> / 2V from psi and D psi (ovl_force.cu's
// energy reduction for 12-component modes): CTA partial sums, one CTA adds them.
template <typename T>
__global__ void __launch_bounds__(256)
    su3_energy_partial_kernel(const cpx<T> *__restrict__ psi, const cpx<T> *__restrict__ dpsi, size_t n, int V,
                              int n_modes, int first_mode, double *__restrict__ partial) {
    __shared__ double sh[32];
    const size_t per_mb = (size_t)V * kComp3 * kModeBlock;
    CompSum acc;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int mode = (int)(e / per_mb) * kModeBlock + (int)(e % kModeBlock);
        if (mode >= n_modes) continue;
        const cpx<T> a = ld(psi + e), d = ld(dpsi + e);
        const double im = (double)a.re * (double)d.im - (double)a.im * (double)d.re;  // Im conj(a) d
        acc.add((((first_mode + mode) & 1) == 0) ? -im : im);
    }
    const double t = block_sum(acc.value(), sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = t;
}

template <typename T>
void su3_launch_fermion_energy(const void *psi, const void *dpsi, const Lattice &L, int n_mb, int n_modes,
                               int first_mode, double *partial, double *out, cudaStream_t s) {
    const size_t n = (size_t)n_mb * L.V * kComp3 * kModeBlock;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 1024);
    su3_energy_partial_kernel<T><<<blocks, 256, 0, s>>>(reinterpret_cast<const cpx<T> *>(psi),
                                                         reinterpret_cast<const cpx<T> *>(dpsi), n, L.V, n_modes,
                                                         first_mode, partial);
    su3_sum_rows_kernel<1><<<1, 256, 0, s>>>(partial, blocks, 1.0 / (2.0 * L.V), out);
}

// ------------------------------------------------------------ FP32 links --
// n = padded floats: link l's 18 doubles into floats [20 l, 20 l + 18), zeros after.
__global__ void su3_links_f32_kernel(const double *__restrict__ U, float *U32, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t l = i / kLink32Floats, k = i % kLink32Floats;
        U32[i] = k < 18 ? (float)U[18 * l + k] : 0.0f;
    }
}

void su3_launch_links_to_f32(const double *U, float *U32, const Lattice &L, cudaStream_t s) {
    const size_t n = (size_t)kLink32Floats * 3 * L.V;
    su3_links_f32_kernel<<<(int)std::min<size_t>((n + 255) / 256, 65535), 256, 0, s>>>(U, U32, n);
}

#define OVL_SU3_INSTANTIATE(T)                                                                                           \
    template void su3_launch_hop<T>(const Su3Links &, const void *, void *, const Lattice &, int, int, double, double,   \
                                    bool, cudaStream_t);                                                                \
    template void su3_chebyshev_apply<T>(ChebyshevWork &, const Su3Links &, const void *, void *, const Lattice &, int, \
                                         const double *, int, double, double, double, double, double, double, bool, int, \
                                         cudaStream_t, uint64_t *);                                                      \
    template void su3_launch_color_force<T>(const double *, const double *, const void *, const Lattice &, int, int,    \
                                            int, double *, double *, double *, double, cudaStream_t);                   \
    template void su3_launch_fermion_energy<T>(const void *, const void *, const Lattice &, int, int, int, double *,    \
                                               double *, cudaStream_t);
OVL_SU3_INSTANTIATE(double)
OVL_SU3_INSTANTIATE(float)

}  // namespace ovl
