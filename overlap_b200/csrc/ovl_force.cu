// Fermion back-reaction on the electric field, and the fermion energy.
//
// An extension without reference counterpart: the reference evolves the modes
// in a fixed gauge background (FERMIONS/WILSON/Update.cpp:48-79 moves the links
// with a constant E and never changes E).  With the links parametrised as
// U_mu(x) -> exp(i theta^a t^a) U_mu(x), t^a = sigma^a / 2, and the fermion energy
//   H_F = (1/2V) sum_m w_m Re <psi_m, h_W psi_m>,   h_W = i D,
// the only terms of h_W that contain U_mu(x) are the hops between x and x+mu,
// and
//   dH_F/dtheta^a_mu(x) = -(1/2V) sum_m w_m Re[psi(x)^+ g0 (1 - G_mu) i t^a U_mu(x) psi(x+mu)]
// with G_mu = -i gamma_mu.  The colour structure separates: per site and mu,
//   C_ij = sum_m w_m sum_ab conj(psi_ia(x)) [g0 (1 - G_mu)]_ab psi_jb(x+mu)
// is link-independent (one pass over the modes, like the currents), and
//   dH_F/dtheta^a = -(1/2V) Re sum_ij (i t^a M)_ij C_ij = (1/4V) Im sum_ij (sigma^a M)_ij C_ij
// with M the (U(1)-dressed) link.  The link update U <- exp(-i dt E^a t^a) U of
// the reference makes d theta / dt = -E, so dE/dt = dH/dtheta conserves
// H_gauge + g^2 H_F.
#include "ovl_bilinears.cuh"
#include "ovl_device.cuh"
#include "ovl_fp40.cuh"
#include "ovl_internal.h"

namespace ovl {

constexpr int kForceSites = 4;

// partial[(g V + site) kForcePerSite + 8 mu + 2 (2 i + j) + {re, im}] = C_ij of
// mode-block group g (a warp is one site, its lanes the 32 modes of a block).
// Four coupled steps at 8^3, 1024 FP64 modes: 645 us with the eight-term
// bilinears and one thread per link in the finish and the staple force, 539 us so.
template <class SRC>
__global__ void __launch_bounds__(kModeBlock *kForceSites, 3)
    color_force_modes_kernel(SRC psi, Lattice L, int n_mb, int n_modes, int first_mode, int groups,
                             double *__restrict__ partial) {
    const int lane = threadIdx.x;
    const int site = blockIdx.x * kForceSites + threadIdx.y;
    const int g = blockIdx.y;
    if (site >= L.V) return;  // whole warps exit together
    const Nbrs nb = neighbours(L, site);
    double acc[32];  // kForcePerSite used
#pragma unroll
    for (int k = 0; k < 32; k++) acc[k] = 0.0;
    for (int mb = g; mb < n_mb; mb += groups) {
        const double w = vacuum_weight(mb * kModeBlock + lane, n_modes, first_mode);
        SiteRaw<2, SRC> raw;
        raw.load(psi, L.V, mb, site, lane);
        cpx<double> f[kColours][kSpin];
#pragma unroll
        for (int k = 0; k < kComp; k++) f[k / kSpin][k % kSpin] = w * raw.get(k);
        raw.load(psi, L.V, mb, nb.xp, lane);
        add_colour_pairs<2, 0>(f, raw, acc);
        raw.load(psi, L.V, mb, nb.yp, lane);
        add_colour_pairs<2, 1>(f, raw, acc + 8);
        raw.load(psi, L.V, mb, nb.zp, lane);
        add_colour_pairs<2, 2>(f, raw, acc + 16);
    }
    const double total = warp_sum32(acc);
    if (lane < kForcePerSite) partial[((size_t)g * L.V + site) * kForcePerSite + lane] = total;
}

// One warp per (site, mu): lane k + 8 s sums C's value k over the groups s, s + 4,
// ..., then every lane contracts C with the dressed link and lane a < 3 writes
// dH_F/dtheta^a: out[a + 3 (mu + 3 site)] when out is set, otherwise
// E[a + 3 (mu + 3 site)] += coef dH_F/dtheta^a.
__global__ void color_force_finish_kernel(const double *__restrict__ partial, int groups, const double *__restrict__ U,
                                          const double2 *__restrict__ u1, Lattice L, double *__restrict__ out,
                                          double *__restrict__ E, double coef) {
    const int t = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (t >= 3 * L.V) return;  // whole warps exit together
    const int site = t / 3, mu = t % 3;
    double v = 0.0;
    for (int g = lane >> 3; g < groups; g += 4)
        v += partial[((size_t)g * L.V + site) * kForcePerSite + 8 * mu + (lane & 7)];
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    double c[8];
#pragma unroll
    for (int k = 0; k < 8; k++) c[k] = __shfl_sync(0xffffffffu, v, k);
    const cpx<double> C00 = mk<double>(c[0], c[1]), C01 = mk<double>(c[2], c[3]);
    const cpx<double> C10 = mk<double>(c[4], c[5]), C11 = mk<double>(c[6], c[7]);
    const cmat2<double> M = dressed_link<double>(U, u1, site, mu, L.N0 * L.N1);
    // S_a = sum_ij (sigma^a M)_ij C_ij
    const cpx<double> m1c0 = M.m10 * C00 + M.m11 * C01;  // sum_j M_1j C_0j
    const cpx<double> m0c1 = M.m00 * C10 + M.m01 * C11;  // sum_j M_0j C_1j
    const cpx<double> m0c0 = M.m00 * C00 + M.m01 * C01;
    const cpx<double> m1c1 = M.m10 * C10 + M.m11 * C11;
    if (lane >= 3) return;
    const double sx = m1c0.im + m0c1.im;
    const double sy = -m1c0.re + m0c1.re;  // Im(-i m1c0 + i m0c1)
    const double sz = m0c0.im - m1c1.im;
    const double f = 1.0 / (4.0 * L.V) * (lane == 0 ? sx : (lane == 1 ? sy : sz));
    const size_t o = 3 * (size_t)t + lane;
    if (out) out[o] = f;
    else E[o] += coef * f;
}

int force_groups(int n_mb) { return n_mb < 16 ? n_mb : 16; }

size_t force_partial_doubles(const Lattice &L, int n_mb) { return (size_t)force_groups(n_mb) * L.V * kForcePerSite; }

template <class SRC>
static void color_force_from(const SRC &src, const double *U, const double *u1, const Lattice &L, int n_mb,
                             int n_modes, int first_mode, double *partial, double *out, double *E, double coef,
                             cudaStream_t stream) {
    const int groups = force_groups(n_mb);
    const dim3 block(kModeBlock, kForceSites), grid((L.V + kForceSites - 1) / kForceSites, groups);
    color_force_modes_kernel<SRC><<<grid, block, 0, stream>>>(src, L, n_mb, n_modes, first_mode, groups, partial);
    const int links_per_cta = 8;  // a warp each
    color_force_finish_kernel<<<(3 * L.V + links_per_cta - 1) / links_per_cta, 32 * links_per_cta, 0, stream>>>(
        partial, groups, U, reinterpret_cast<const double2 *>(u1), L, out, E, coef);
}

template <typename T>
void launch_color_force(const double *U, const double *u1, const void *psi, const Lattice &L, int n_mb, int n_modes,
                        int first_mode, double *partial, double *out, double *E, double coef, cudaStream_t stream) {
    color_force_from(SrcPlain<T>{reinterpret_cast<const cpx<T> *>(psi)}, U, u1, L, n_mb, n_modes, first_mode, partial,
                     out, E, coef, stream);
}

void launch_color_force40(const double *U, const double *u1, const void *hi, const void *lo, const Lattice &L, int n_mb,
                          int n_modes, int first_mode, double *partial, double *out, double *E, double coef,
                          cudaStream_t stream) {
    color_force_from(Src40{reinterpret_cast<const uint2 *>(hi), reinterpret_cast<const unsigned char *>(lo)}, U, u1, L, n_mb,
                     n_modes, first_mode, partial, out, E, coef, stream);
}

template void launch_color_force<float>(const double *, const double *, const void *, const Lattice &, int, int, int,
                                        double *, double *, double *, double, cudaStream_t);
template void launch_color_force<double>(const double *, const double *, const void *, const Lattice &, int, int, int,
                                         double *, double *, double *, double, cudaStream_t);

// ------------------------------------------------------------ fermion energy --
// sum_m w_m Re <psi_m, i (D psi)_m> = -sum_m w_m Im <psi_m, (D psi)_m>: per CTA
// partial sums over a fixed grid, then one CTA adds them in order and scales
// by 1/(2V).  Element e of the mode-block layout belongs to mode
// 32 (e / (32 kComp V)) + e % 32.
constexpr int kEnergyThreads = 256;
constexpr int kEnergyBlocks = 1024;

template <class SRC>
__global__ void __launch_bounds__(kEnergyThreads)
    energy_partial_kernel(SRC psi, SRC dpsi, size_t n, int V, int n_modes, int first_mode, double *__restrict__ partial) {
    __shared__ double sh[kEnergyThreads];
    const size_t per_mb = (size_t)V * kComp * kModeBlock;
    CompSum acc;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int mode = (int)(e / per_mb) * kModeBlock + (int)(e % kModeBlock);
        if (mode >= n_modes) continue;
        const cpx<double> a = psi(e), d = dpsi(e);
        const double im = a.re * d.im - a.im * d.re;  // Im conj(a) d
        acc.add((((first_mode + mode) & 1) == 0) ? -im : im);
    }
    sh[threadIdx.x] = acc.value();
    __syncthreads();
    for (int s = kEnergyThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = sh[0];
}

__global__ void __launch_bounds__(kEnergyThreads)
    energy_finish_kernel(const double *__restrict__ partial, int blocks, double scale, double *__restrict__ out) {
    __shared__ double sh[kEnergyThreads];
    CompSum acc;
    for (int b = threadIdx.x; b < blocks; b += kEnergyThreads) acc.add(partial[b]);
    sh[threadIdx.x] = acc.value();
    __syncthreads();
    for (int s = kEnergyThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = scale * sh[0];
}

size_t energy_partial_doubles() { return kEnergyBlocks; }

template <class SRC>
static void energy_from(const SRC &psi, const SRC &dpsi, const Lattice &L, int n_mb, int n_modes, int first_mode,
                        double *partial, double *out, cudaStream_t stream) {
    const size_t n = (size_t)n_mb * L.V * kComp * kModeBlock;
    const size_t want = (n + kEnergyThreads - 1) / kEnergyThreads;
    const int blocks = (int)(want < (size_t)kEnergyBlocks ? want : (size_t)kEnergyBlocks);
    energy_partial_kernel<SRC><<<blocks, kEnergyThreads, 0, stream>>>(psi, dpsi, n, L.V, n_modes, first_mode, partial);
    energy_finish_kernel<<<1, kEnergyThreads, 0, stream>>>(partial, blocks, 1.0 / (2.0 * L.V), out);
}

template <typename T>
void launch_fermion_energy(const void *psi, const void *dpsi, const Lattice &L, int n_mb, int n_modes, int first_mode,
                           double *partial, double *out, cudaStream_t stream) {
    energy_from(SrcPlain<T>{reinterpret_cast<const cpx<T> *>(psi)}, SrcPlain<T>{reinterpret_cast<const cpx<T> *>(dpsi)},
                L, n_mb, n_modes, first_mode, partial, out, stream);
}

void launch_fermion_energy40(const void *hi, const void *lo, const void *dhi, const void *dlo, const Lattice &L,
                             int n_mb, int n_modes, int first_mode, double *partial, double *out, cudaStream_t stream) {
    energy_from(Src40{reinterpret_cast<const uint2 *>(hi), reinterpret_cast<const unsigned char *>(lo)},
                Src40{reinterpret_cast<const uint2 *>(dhi), reinterpret_cast<const unsigned char *>(dlo)}, L, n_mb, n_modes,
                first_mode, partial, out, stream);
}

template void launch_fermion_energy<float>(const void *, const void *, const Lattice &, int, int, int, double *,
                                           double *, cudaStream_t);
template void launch_fermion_energy<double>(const void *, const void *, const Lattice &, int, int, int, double *,
                                            double *, cudaStream_t);

}  // namespace ovl
