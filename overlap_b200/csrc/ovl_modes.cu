// Kernels over the mode batch other than the Wilson operator: the fermion
// currents and their lattice sums, layout conversion between the reference's
// per-mode arrays and the mode-block layout, and free plane-wave modes.

#include "ovl_bilinears.cuh"
#include "ovl_device.cuh"
#include "ovl_fp40.cuh"
#include "ovl_internal.h"

namespace ovl {

// ---------------------------------------------------------------- currents --
// Fermions::Observables::ComputeCurrents, Wilson (FERMIONS/WILSON/Currents.cpp:7-309).
// For each mode (vacuum weight w = +1 even / -1 odd global index,
// FermionField.cpp:109-122) and site, with chi_mu = U_mu(x) psi(x+mu) and
// chib_mu = U_mu(x-mu)^+ psi(x-mu):
//   jV^0 = psi^+ psi              jA^0 = psi^+ g5 psi
//   jV^mu = Re psi^+ g0 g_mu chi   jA^mu = Re psi^+ g0 g_mu g5 chi
//   jVw^mu = Re psi^+ (-i r g0) chi, jAw^mu = Re psi^+ (-i r g0 g5) chi
//   PS = Re psi^+ (i g0 g5) psi
//   WA = Re[-6 psi^+ (-i r g0 g5) psi + sum_mu psi^+ (-i r g0 g5) (chi_mu + chib_mu)]
// summed over colours and modes, times 1/(2V) (Currents.cpp:289).
// Output per site: jV[4] jA[4] jVw[4] jAw[4] PS WA (jVw^0 = jAw^0 = 0).
//
// The backward term of WA is not evaluated on the modes: Gamma = -i r g0 g5 is
// hermitian, so psi^+(x) Gamma U_mu(x-mu)^+ psi(x-mu) is the complex conjugate
// of the forward term of the site x-mu, and its real part is jAw^mu(x-mu); the
// finishing kernel adds it per site.  That leaves four spinor reads and 128
// FP64 multiply-adds per hop and mode (two colours) of the seven reads and 208.
// What bounds the kernel is FP64 arithmetic (and, for FP32 modes, the FP32 to
// FP64 conversions beside it): the links sit in shared memory instead of
// registers, and a neighbour is converted as a whole so that the next one's
// loads are in flight while it is used.  ovl_currents at 16^3, 4096 FP32 modes:
// 1715 us with the seven reads (254 registers, 8 warps per SM), 924 us with four
// reads at 128 registers (16 warps) without the loads in flight, 845 us so (168
// registers, 12 warps), 913 us so squeezed into 128 registers.
constexpr int kCurrentVals = 16;  // partial sums per site and group: jV0, jA0, PS, then jV, jA, jVw, jAw by mu; one spare

// Slot k of the per-site output is partial value kCurrentSlot[k] (-1: zero, -2: WA).
__constant__ int kCurrentSlot[kCurrentsPerSite] = {0, 3, 4, 5, 1, 6, 7, 8, -1, 9, 10, 11, -1, 12, 13, 14, 2, -2};

constexpr int kCurrentSites = 4;  // per CTA, a warp each

template <int NC, class SRC>
__global__ void __launch_bounds__(kModeBlock *kCurrentSites, NC == 2 ? 3 : 2)
    currents_kernel(const double *__restrict__ U, const double *__restrict__ u1, SRC psi, Lattice L, int n_mb,
                    int n_modes, int first_mode, int groups, double r, double *__restrict__ partial) {
    constexpr int S = kCurrentSites;
    constexpr mono G05 = mono_mul(kGamma0, kGamma5);
    constexpr mono GV[3] = {mono_mul(kGamma0, kGammaX), mono_mul(kGamma0, kGammaY), mono_mul(kGamma0, kGammaZ)};
    constexpr mono GA[3] = {mono_mul(GV[0], kGamma5), mono_mul(GV[1], kGamma5), mono_mul(GV[2], kGamma5)};
    __shared__ double2 tab[S][3][NC * NC];
    const int site0 = blockIdx.x * S;
    fill_bilinear_links<NC, S>(U, u1, L, site0, tab);
    const int lane = threadIdx.x, site = site0 + threadIdx.y, g = blockIdx.y, V = L.V;
    if (site >= V) return;  // whole warps exit together: a warp is one site
    const Nbrs nb = neighbours(L, site);
    RunSum<NC == 3> acc[kCurrentVals - 1];
    for (int mb = g; mb < n_mb; mb += groups) {
        const double w = vacuum_weight(mb * kModeBlock + lane, n_modes, first_mode);
        SiteRaw<NC, SRC> raw;
        raw.load(psi, V, mb, site, lane);
        cpx<double> f[NC][kSpin];
#pragma unroll
        for (int k = 0; k < 4 * NC; k++) f[k / kSpin][k % kSpin] = raw.get(k);
        raw.load(psi, V, mb, nb.xp, lane);
        {
            // psi^+ psi, psi^+ g5 psi = 2 Re z, psi^+ (i g0 g5) psi = -2 Im z with z = conj(psi_0) psi_2 + conj(psi_1) psi_3
            double nv = 0.0, zr = 0.0, zi = 0.0;
#pragma unroll
            for (int c = 0; c < NC; c++) {
#pragma unroll
                for (int a = 0; a < kSpin; a++) add_part<false>(nv, 0, f[c][a], f[c][a]);
#pragma unroll
                for (int a = 0; a < 2; a++) {
                    add_part<false>(zr, 0, f[c][a], f[c][a + 2]);
                    add_part<true>(zi, 0, f[c][a], f[c][a + 2]);
                }
            }
            acc[0].add(w * nv);
            acc[1].add(w * (2.0 * zr));
            acc[2].add(w * (-2.0 * zi));
        }
#pragma unroll
        for (int mu = 0; mu < 3; mu++) {
            // the neighbour in FP64, and the next one's loads in flight while it is used
            cpx<double> nbr[4 * NC];
#pragma unroll
            for (int k = 0; k < 4 * NC; k++) nbr[k] = raw.get(k);
            if (mu == 0) raw.load(psi, V, mb, nb.yp, lane);
            if (mu == 1) raw.load(psi, V, mb, nb.zp, lane);
            double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int b = 0; b < kSpin; b++) {  // chi = U_mu(x) psi(x+mu), one spin component at a time
                cpx<double> h[NC], chi[NC];
#pragma unroll
                for (int j = 0; j < NC; j++) h[j] = nbr[kSpin * j + b];
                link_times<NC>(tab[threadIdx.y][mu], h, chi);
                // component b meets the row a with perm[a] = b; the permutations are involutions
                const mono Gs[4] = {GV[mu], GA[mu], kGamma0, G05};
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int a = Gs[k].perm[b];
#pragma unroll
                    for (int c = 0; c < NC; c++) {
                        if (k < 2) add_part<false>(v[k], Gs[k].ph[a], f[c][a], chi[c]);
                        else add_part<true>(v[k], Gs[k].ph[a], f[c][a], chi[c]);
                    }
                }
            }
            acc[3 + mu].add(w * v[0]);
            acc[6 + mu].add(w * v[1]);
            acc[9 + mu].add(w * (r * v[2]));
            acc[12 + mu].add(w * (r * v[3]));
        }
    }
    // the 32 modes of the warp, fixed order
    double t[kCurrentVals];
#pragma unroll
    for (int k = 0; k < kCurrentVals - 1; k++) t[k] = acc[k].value();
    t[kCurrentVals - 1] = 0.0;
    const double total = warp_sum16(t);
    if ((lane & 1) == 0) partial[((size_t)g * V + site) * kCurrentVals + (lane >> 1)] = total;
}

// The groups' sums per site and output slot, with WA from the site's and its
// backward neighbours' jAw.
__global__ void wilson_currents_finish_kernel(const double *__restrict__ partial, int groups, Lattice L, double r,
                                              double scale, double *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= L.V * kCurrentsPerSite) return;
    const int site = i / kCurrentsPerSite, slot = kCurrentSlot[i % kCurrentsPerSite];
    auto total = [&](int s, int k) {
        double t = 0.0;
        for (int g = 0; g < groups; g++) t += partial[((size_t)g * L.V + s) * kCurrentVals + k];
        return t;
    };
    double t = 0.0;
    if (slot >= 0) {
        t = total(site, slot);
    } else if (slot == -2) {
        // -6 Re psi^+ (-i r g0 g5) psi = 6 r PS
        const Nbrs n = neighbours(L, site);
        t = 6.0 * r * total(site, 2);
        const int back[3] = {n.xm, n.ym, n.zm};
        for (int mu = 0; mu < 3; mu++) t += total(site, 12 + mu) + total(back[mu], 12 + mu);
    }
    out[i] = scale * t;
}

// Sums the groups of a per-site array written slot by slot (overlap currents).
__global__ void currents_finish_kernel(const double *__restrict__ partial, int groups, int V, double scale,
                                       double *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = V * kCurrentsPerSite;
    if (i >= n) return;
    double t = 0.0;
    for (int g = 0; g < groups; g++) t += partial[(size_t)g * n + i];
    out[i] = scale * t;
}

int currents_groups(int n_mb) { return n_mb < 16 ? n_mb : 16; }

void launch_currents_finish(const double *partial, int groups, const Lattice &L, double *per_site, cudaStream_t stream) {
    const int n = L.V * kCurrentsPerSite;
    currents_finish_kernel<<<(n + 255) / 256, 256, 0, stream>>>(partial, groups, L.V, 1.0 / (2.0 * L.V), per_site);
}

size_t currents_partial_doubles(const Lattice &L, int n_mb) {
    return (size_t)currents_groups(n_mb) * L.V * kCurrentsPerSite;
}

template <int NC, class SRC>
static void currents_from(const SRC &src, const double *U, const double *u1, const Lattice &L, int n_mb, int n_modes,
                          int first_mode, double r_wilson, double *partial, double *per_site, cudaStream_t stream) {
    constexpr int S = kCurrentSites;
    const int groups = currents_groups(n_mb);
    currents_kernel<NC, SRC><<<dim3((L.V + S - 1) / S, groups), dim3(kModeBlock, S), 0, stream>>>(
        U, u1, src, L, n_mb, n_modes, first_mode, groups, r_wilson, partial);
    const int n = L.V * kCurrentsPerSite;
    wilson_currents_finish_kernel<<<(n + 127) / 128, 128, 0, stream>>>(partial, groups, L, r_wilson, 1.0 / (2.0 * L.V),
                                                                       per_site);
}

template <typename T>
void launch_currents(const double *U, const double *u1, const void *psi, const Lattice &L, int n_mb, int n_modes,
                     int first_mode, double r_wilson, double *partial, double *per_site, cudaStream_t stream) {
    currents_from<2>(SrcPlain<T>{reinterpret_cast<const cpx<T> *>(psi)}, U, u1, L, n_mb, n_modes, first_mode, r_wilson,
                     partial, per_site, stream);
}

template <typename T>
void su3_launch_currents(const double *U, const double *u1, const void *psi, const Lattice &L, int n_mb, int n_modes,
                         int first_mode, double r_wilson, double *partial, double *per_site, cudaStream_t stream) {
    currents_from<3>(SrcPlain<T>{reinterpret_cast<const cpx<T> *>(psi)}, U, u1, L, n_mb, n_modes, first_mode, r_wilson,
                     partial, per_site, stream);
}

void launch_currents40(const double *U, const double *u1, const void *hi, const void *lo, const Lattice &L, int n_mb,
                       int n_modes, int first_mode, double r_wilson, double *partial, double *per_site,
                       cudaStream_t stream) {
    currents_from<2>(Src40{reinterpret_cast<const uint2 *>(hi), reinterpret_cast<const unsigned char *>(lo)}, U, u1, L, n_mb,
                     n_modes, first_mode, r_wilson, partial, per_site, stream);
}

// ----------------------------------------------------------------- charges --
// The lattice sums of the current densities without the per-site maps:
//   N_V = sum psi^+ psi,  N_5 = sum psi^+ g5 psi = 2 Re z,  PS = -2 Im z,
//   z = sum_c conj(psi_0) psi_2 + conj(psi_1) psi_3,
//   WA  = -12 r Im z + 2 r sum_mu Im psi^+(x) g0 g5 U_mu(x) psi(x+mu).
// For the WA sum the backward hop of Currents.cpp:273-283 is not evaluated:
// with Gamma = -i r g0 g5 hermitian, shifting x -> x+mu turns
// sum_x psi^+(x) Gamma U_mu(x-mu)^+ psi(x-mu) into the complex conjugate of the
// forward sum, whose real part is the same.  Each thread evaluates its mode
// and site in double whatever the mode precision (each of the ~1e8 terms of a
// lattice sum then carries a 1e-16 rounding error); partial sums per CTA are
// added in a fixed order.
// The links are read from shared memory and a hop is taken one spin component
// at a time, so that a thread fits 128 registers and four CTAs share an SM
// (with the three link matrices in registers: 168, one CTA of 8 warps).
// An observation (charges, Delta N_CS, bulk) at 12^3, 4096 FP32 modes: 466 us
// with the link matrices in registers, 318 us so.
constexpr int kChargeVals = 4;
constexpr int kChargeSites = 4;

template <int NC, class SRC>
__global__ void __launch_bounds__(kModeBlock *kChargeSites, NC == 2 ? 4 : 3)
    charges_kernel(const double *__restrict__ U, const double *__restrict__ u1, SRC psi, Lattice L, int n_mb,
                   int n_modes, int first_mode, int groups, double r, double *__restrict__ partial) {
    __shared__ double sh[kChargeSites][kChargeVals];
    __shared__ double2 tab[kChargeSites][3][NC * NC];
    const int site0 = blockIdx.x * kChargeSites;
    fill_bilinear_links<NC, kChargeSites>(U, u1, L, site0, tab);
    const int lane = threadIdx.x, site = site0 + threadIdx.y, g = blockIdx.y, V = L.V;
    CompSum sum[kChargeVals];
    if (site < V) {
        const Nbrs nb = neighbours(L, site);
        for (int mb = g; mb < n_mb; mb += groups) {
            const double w = vacuum_weight(mb * kModeBlock + lane, n_modes, first_mode);
            SiteRaw<NC, SRC> raw;
            raw.load(psi, V, mb, site, lane);
            cpx<double> f[NC][kSpin];
#pragma unroll
            for (int k = 0; k < 4 * NC; k++) f[k / kSpin][k % kSpin] = raw.get(k);
            raw.load(psi, V, mb, nb.xp, lane);
            double nv = 0.0, zr = 0.0, zi = 0.0, hop = 0.0;
#pragma unroll
            for (int c = 0; c < NC; c++) {
#pragma unroll
                for (int a = 0; a < kSpin; a++) add_part<false>(nv, 0, f[c][a], f[c][a]);
#pragma unroll
                for (int a = 0; a < 2; a++) {
                    add_part<false>(zr, 0, f[c][a], f[c][a + 2]);
                    add_part<true>(zi, 0, f[c][a], f[c][a + 2]);
                }
            }
#pragma unroll
            for (int mu = 0; mu < 3; mu++) {
#pragma unroll
                for (int b = 0; b < kSpin; b++) {
                    cpx<double> h[NC], chi[NC];
#pragma unroll
                    for (int j = 0; j < NC; j++) h[j] = raw.get(kSpin * j + b);
                    link_times<NC>(tab[threadIdx.y][mu], h, chi);
                    // Im of f0* chi2 + f1* chi3 - f2* chi0 - f3* chi1
#pragma unroll
                    for (int c = 0; c < NC; c++) add_part<true>(hop, b < 2 ? 2 : 0, f[c][b ^ 2], chi[c]);
                }
                if (mu == 0) raw.load(psi, V, mb, nb.yp, lane);
                if (mu == 1) raw.load(psi, V, mb, nb.zp, lane);
            }
            sum[0].add(w * nv);
            sum[1].add(w * 2.0 * zr);
            sum[2].add(w * -2.0 * zi);
            sum[3].add(w * (r * (-12.0 * zi + 2.0 * hop)));
        }
    }
    double acc[kChargeVals];
#pragma unroll
    for (int k = 0; k < kChargeVals; k++) acc[k] = sum[k].value();
#pragma unroll
    for (int k = 0; k < kChargeVals; k++) {
        double t = acc[k];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        acc[k] = t;
    }
    if (lane == 0)
        for (int k = 0; k < kChargeVals; k++) sh[threadIdx.y][k] = acc[k];
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        double *p = partial + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * kChargeVals;
        for (int k = 0; k < kChargeVals; k++) {
            double t = 0.0;
            for (int j = 0; j < kChargeSites; j++) t += sh[j][k];
            p[k] = t;
        }
    }
}

__global__ void __launch_bounds__(1024) charges_finish_kernel(const double *__restrict__ partial, int n, double scale,
                                                              double *__restrict__ out4) {
    // one thread per row and value (the four values of a row are one 32-byte sector), then a fixed tree
    __shared__ double sh[1024];
    CompSum t;
    const int k = threadIdx.x % kChargeVals;
    for (int i = threadIdx.x / kChargeVals; i < n; i += 1024 / kChargeVals) t.add(partial[(size_t)i * kChargeVals + k]);
    sh[threadIdx.x] = t.value();
    __syncthreads();
    for (int stride = 512; stride >= kChargeVals; stride >>= 1) {
        if ((int)threadIdx.x < stride) sh[threadIdx.x] += sh[threadIdx.x + stride];
        __syncthreads();
    }
    if (threadIdx.x < kChargeVals) out4[threadIdx.x] = scale * sh[threadIdx.x];
}

size_t charges_partial_doubles(const Lattice &L, int n_mb) {
    return (size_t)currents_groups(n_mb) * ((L.V + kChargeSites - 1) / kChargeSites) * kChargeVals;
}

template <int NC, class SRC>
static void charges_from(const SRC &src, const double *U, const double *u1, const Lattice &L, int n_mb, int n_modes,
                         int first_mode, double r, double *partial, double *out4, cudaStream_t stream) {
    const int groups = currents_groups(n_mb);
    const dim3 block(kModeBlock, kChargeSites), grid((L.V + kChargeSites - 1) / kChargeSites, groups);
    charges_kernel<NC, SRC><<<grid, block, 0, stream>>>(U, u1, src, L, n_mb, n_modes, first_mode, groups, r, partial);
    charges_finish_kernel<<<1, 1024, 0, stream>>>(partial, (int)(grid.x * grid.y), 1.0 / (2.0 * L.V), out4);
}

template <typename T>
void launch_charges(const double *U, const double *u1, const void *psi, const Lattice &L, int n_mb, int n_modes,
                    int first_mode, double r_wilson, double *partial, double *out4, cudaStream_t stream) {
    // the arithmetic precision of r as before: the FP32 path rounds it to float
    charges_from<2>(SrcPlain<T>{reinterpret_cast<const cpx<T> *>(psi)}, U, u1, L, n_mb, n_modes, first_mode,
                    (double)(T)r_wilson, partial, out4, stream);
}

template <typename T>
void su3_launch_charges(const double *U, const double *u1, const void *psi, const Lattice &L, int n_mb, int n_modes,
                        int first_mode, double r_wilson, double *partial, double *out4, cudaStream_t stream) {
    charges_from<3>(SrcPlain<T>{reinterpret_cast<const cpx<T> *>(psi)}, U, u1, L, n_mb, n_modes, first_mode, r_wilson,
                    partial, out4, stream);
}

void launch_charges40(const double *U, const double *u1, const void *hi, const void *lo, const Lattice &L, int n_mb,
                      int n_modes, int first_mode, double r_wilson, double *partial, double *out4, cudaStream_t stream) {
    charges_from<2>(Src40{reinterpret_cast<const uint2 *>(hi), reinterpret_cast<const unsigned char *>(lo)}, U, u1, L, n_mb,
                    n_modes, first_mode, r_wilson, partial, out4, stream);
}

// Lattice sums of jV^0, jA^0, PS, WA from the per-site array, fixed order.
__global__ void site_sums_kernel(const double *__restrict__ per_site, int V, double *__restrict__ out4) {
    __shared__ double sh[4][256];
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (int s = threadIdx.x; s < V; s += blockDim.x) {
        const double *p = per_site + (size_t)s * kCurrentsPerSite;
        t[0] += p[0];
        t[1] += p[4];
        t[2] += p[16];
        t[3] += p[17];
    }
    for (int k = 0; k < 4; k++) sh[k][threadIdx.x] = t[k];
    __syncthreads();
    for (int stride = blockDim.x / 2; stride > 0; stride >>= 1) {
        if ((int)threadIdx.x < stride)
            for (int k = 0; k < 4; k++) sh[k][threadIdx.x] += sh[k][threadIdx.x + stride];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        for (int k = 0; k < 4; k++) out4[k] = sh[k][0];
}

void launch_site_sums(const double *per_site, const Lattice &L, double * /*partial*/, double *out4, cudaStream_t stream) {
    site_sums_kernel<<<1, 256, 0, stream>>>(per_site, L.V, out4);
}

// ---------------------------------------------------------- layout change --
// ncomp complex components per mode and site: 8 (two colours) or 12 (three).
__device__ __forceinline__ size_t block_index(int V, int ncomp, int m, int site, int comp) {
    return (((size_t)(m / kModeBlock) * V + site) * ncomp + comp) * kModeBlock + m % kModeBlock;
}

template <typename T>
__global__ void ref_to_blocks_kernel(const double2 *__restrict__ ref, cpx<T> *__restrict__ blocks, int V, int m0,
                                     int count, unsigned char *__restrict__ lo, int ncomp) {
    const size_t n = (size_t)count * V * ncomp;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int comp = (int)(i % ncomp);
        const size_t ms = i / ncomp;
        const int site = (int)(ms % V);
        const int m = m0 + (int)(ms / V);
        const double2 v = ref[i];
        const size_t j = block_index(V, ncomp, m, site, comp);
        if (lo) store40(reinterpret_cast<uint2 *>(blocks), lo, j, v.x, v.y);  // 40-bit storage
        else st(blocks + j, mk<T>((T)v.x, (T)v.y));
    }
}

template <typename T>
__global__ void blocks_to_ref_kernel(const cpx<T> *__restrict__ blocks, double2 *__restrict__ ref, int V, int m0,
                                     int count, const unsigned char *__restrict__ lo, int ncomp) {
    const size_t n = (size_t)count * V * ncomp;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int comp = (int)(i % ncomp);
        const size_t ms = i / ncomp;
        const int site = (int)(ms % V);
        const int m = m0 + (int)(ms / V);
        const size_t j = block_index(V, ncomp, m, site, comp);
        if (lo) {  // 40-bit storage
            const cpx<double> v = Src40{reinterpret_cast<const uint2 *>(blocks), lo}(j);
            ref[i] = double2{v.re, v.im};
        } else {
            const cpx<T> v = blocks[j];
            ref[i] = double2{(double)v.re, (double)v.im};
        }
    }
}

static int grid_for(size_t n) {
    size_t b = (n + 255) / 256;
    return (int)(b < 65535 ? b : 65535);
}

template <typename T>
void launch_ref_to_blocks(const double *ref, void *blocks, const Lattice &L, int m0, int count, cudaStream_t stream,
                          void *lo, int nc) {
    const size_t n = (size_t)count * L.V * nc * kSpin;
    if (n == 0) return;
    ref_to_blocks_kernel<T><<<grid_for(n), 256, 0, stream>>>(reinterpret_cast<const double2 *>(ref),
                                                             reinterpret_cast<cpx<T> *>(blocks), L.V, m0, count,
                                                             reinterpret_cast<unsigned char *>(lo), nc * kSpin);
}

template <typename T>
void launch_blocks_to_ref(const void *blocks, double *ref, const Lattice &L, int m0, int count, cudaStream_t stream,
                          const void *lo, int nc) {
    const size_t n = (size_t)count * L.V * nc * kSpin;
    if (n == 0) return;
    blocks_to_ref_kernel<T><<<grid_for(n), 256, 0, stream>>>(reinterpret_cast<const cpx<T> *>(blocks),
                                                             reinterpret_cast<double2 *>(ref), L.V, m0, count,
                                                             reinterpret_cast<const unsigned char *>(lo), nc * kSpin);
}

// ------------------------------------------------------------ plane waves --
// InitialConditions::SetFreeFermions with GetWilsonDiracSpinor / GetWilsonPhase
// (SetFreeFermions.cpp:3-56, FermionField.cpp:145-328), or for overlap
// fermions GetOverlapDiracSpinor / GetOverlapPhase (FermionField.cpp:331-528):
// the same helicity spinors of the momentum p and mass meff, which for the
// overlap operator are p = M hp / s and meff = M (1 + hp5 / s) with
// hp = sin(2 pi n / N), hp5 = 3 - M - sum cos(2 pi n / N), s = |(hp, hp5)|.
// Mode index
// particle + 2(colour + Nc(spin + 2(px + N0(py + N1 pz)))); particles
// exp(+i p.x) with frequency +w, antiparticles exp(-i p.x) with -w; psimid =
// psi exp(-i w dt / 2).
struct FreeMode { double u[8]; double omega; int colour, k0, k1, k2, particle, bad; };

__device__ FreeMode free_mode(const Lattice &L, int g, double r, double m, int nc, int overlap, double mdw) {
    FreeMode fm;
    const int N[3] = {L.N0, L.N1, L.N2};
    fm.particle = g % 2; g /= 2;
    fm.colour = g % nc; g /= nc;
    const int spin = g % 2; g /= 2;
    int k[3];
    k[0] = g % N[0]; g /= N[0];
    k[1] = g % N[1]; g /= N[1];
    k[2] = g % N[2];
    fm.k0 = k[0]; fm.k1 = k[1]; fm.k2 = k[2];
    double pp[3], meff = m, p2 = 0.0;
    if (overlap) {
        double hp5 = 3.0 - mdw, s2 = 0.0;
        for (int i = 0; i < 3; i++) {
            const int n = fm.particle == 0 ? k[i] : N[i] - k[i];
            pp[i] = sin(2.0 * M_PI * n / (double)N[i]);
            hp5 -= cos(2.0 * M_PI * n / (double)N[i]);
            s2 += pp[i] * pp[i];
        }
        const double sabs = sqrt(s2 + hp5 * hp5);
        for (int i = 0; i < 3; i++) {
            pp[i] = mdw * pp[i] / sabs;
            p2 += pp[i] * pp[i];
        }
        meff = mdw * (1.0 + hp5 / sabs);
    } else {
        for (int i = 0; i < 3; i++) {
            const int n = fm.particle == 0 ? k[i] : N[i] - k[i];
            pp[i] = sin(2.0 * M_PI * n / (double)N[i]);
            const double h = sin(M_PI * n / (double)N[i]);
            meff += 2.0 * r * h * h;
            p2 += pp[i] * pp[i];
        }
    }
    const double pabs = sqrt(p2);
    const double w = sqrt(p2 + meff * meff);
    const double omega = fm.particle == 0 ? w : -w;
    fm.omega = omega;
    // the axis cases test k == 0 or k == N/2 in integer division (FermionField.cpp:188,229):
    // for odd N the index (N-1)/2 takes them too, and its spinor fails the eigen check
    bool edge[3];
    for (int i = 0; i < 3; i++) edge[i] = (k[i] == 0 || k[i] == N[i] / 2);
    cpx<double> phi0, phi1;
    double hel;
    if (edge[0] && edge[1]) {
        phi0 = mk<double>(spin == 0 ? 1.0 : 0.0, 0.0);
        phi1 = mk<double>(spin == 0 ? 0.0 : 1.0, 0.0);
        hel = (spin == 0 ? 1.0 : -1.0) * pp[2] / fabs(pp[2]);
        if (edge[2]) hel = 0.0;
    } else {
        hel = spin == 0 ? 1.0 : -1.0;
        // q = -(pz - hel |p|) / (px - i py)
        const double nr = -(pp[2] - hel * pabs);
        const double den = pp[0] * pp[0] + pp[1] * pp[1];
        const cpx<double> q = mk<double>(nr * pp[0] / den, nr * pp[1] / den);
        const double d = sqrt(1.0 + q.re * q.re + q.im * q.im);
        phi0 = mk<double>(1.0 / d, 0.0);
        phi1 = mk<double>(q.re / d, q.im / d);
    }
    cpx<double> u[4];
    if (edge[0] && edge[1] && edge[2]) {
        const bool upper = (fm.particle == 0) == (meff >= 0.0);
        const cpx<double> zero = mk<double>(0.0, 0.0);
        u[0] = upper ? phi0 : zero;
        u[1] = upper ? phi1 : zero;
        u[2] = upper ? zero : phi0;
        u[3] = upper ? zero : phi1;
    } else {
        const double norm = sqrt(2.0 * omega * (omega - meff) / p2);
        const double lower = hel * (omega - meff) / pabs;
        u[0] = (1.0 / norm) * phi0;
        u[1] = (1.0 / norm) * phi1;
        u[2] = (lower / norm) * phi0;
        u[3] = (lower / norm) * phi1;
    }
    // eigen-residual |w u - H u| and |u|^2 - 1 with H = g0 (meff + p.gamma) (FermionField.cpp:270-312)
    constexpr mono G0 = kGamma0;
    constexpr mono GX0 = mono_mul(kGamma0, kGammaX), GY0 = mono_mul(kGamma0, kGammaY), GZ0 = mono_mul(kGamma0, kGammaZ);
    bool bad = false;
    double n2 = 0.0;
#pragma unroll
    for (int a = 0; a < 4; a++) {
        cpx<double> hu = (G0.ph[a] == 0 ? meff : -meff) * u[G0.perm[a]];
        hu = hu + pp[0] * iphase(GX0.ph[a], u[GX0.perm[a]]) + pp[1] * iphase(GY0.ph[a], u[GY0.perm[a]]) +
             pp[2] * iphase(GZ0.ph[a], u[GZ0.perm[a]]);
        const cpx<double> dlt = omega * u[a] - hu;
        if (sqrt(dlt.re * dlt.re + dlt.im * dlt.im) > 1e-6) bad = true;
        n2 += u[a].re * u[a].re + u[a].im * u[a].im;
    }
    if (fabs(n2 - 1.0) > 1e-6) bad = true;
    fm.bad = bad ? 1 : 0;
    for (int a = 0; a < 4; a++) { fm.u[2 * a] = u[a].re; fm.u[2 * a + 1] = u[a].im; }
    return fm;
}

__global__ void free_modes_kernel(FreeMode *info, int n_modes, int first_mode, Lattice L, double r, double m, int *bad,
                                  int nc, int overlap, double mdw) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_modes) return;
    FreeMode fm = free_mode(L, first_mode + i, r, m, nc, overlap, mdw);
    info[i] = fm;
    if (fm.bad) atomicAdd(bad, 1);
}

template <typename T>
__global__ void free_fill_kernel(const FreeMode *__restrict__ info, cpx<T> *psi, cpx<T> *psimid, Lattice L, int n_modes,
                                 int n_mb, double dt, unsigned char *lo_psi, unsigned char *lo_mid, int nc) {
    const int lane = threadIdx.x;
    const int site = blockIdx.x * blockDim.y + threadIdx.y;
    const int mb = blockIdx.y;
    if (site >= L.V) return;
    const int m = mb * kModeBlock + lane;
    int x, y, z;
    site_coords(L, site, x, y, z);
    cpx<double> u[4] = {mk<double>(0, 0), mk<double>(0, 0), mk<double>(0, 0), mk<double>(0, 0)};
    cpx<double> phase = mk<double>(0, 0), half = mk<double>(1, 0);
    int colour = -1;
    if (m < n_modes) {
        const FreeMode fm = info[m];
        for (int a = 0; a < 4; a++) u[a] = mk<double>(fm.u[2 * a], fm.u[2 * a + 1]);
        const double arg = (fm.k0 * x) / (double)L.N0 + (fm.k1 * y) / (double)L.N1 + (fm.k2 * z) / (double)L.N2;
        double sn, cs;
        sincos((fm.particle == 0 ? 2.0 : -2.0) * M_PI * arg, &sn, &cs);
        phase = mk<double>(cs, sn);
        sincos(-0.5 * fm.omega * dt, &sn, &cs);
        half = mk<double>(cs, sn);
        colour = fm.colour;
    }
    for (int c = 0; c < nc; c++)
        for (int a = 0; a < kSpin; a++) {
            cpx<double> v = c == colour ? phase * u[a] : mk<double>(0, 0);
            cpx<double> vm = c == colour ? v * half : mk<double>(0, 0);
            const size_t idx = block_index(L.V, nc * kSpin, m, site, c * kSpin + a);
            if (lo_psi) {  // 40-bit storage
                store40(reinterpret_cast<uint2 *>(psi), lo_psi, idx, v.re, v.im);
                store40(reinterpret_cast<uint2 *>(psimid), lo_mid, idx, vm.re, vm.im);
            } else {
                st(psi + idx, mk<T>((T)v.re, (T)v.im));
                st(psimid + idx, mk<T>((T)vm.re, (T)vm.im));
            }
        }
}

template <typename T>
void launch_free_fermions(void *psi, void *psimid, const Lattice &L, int n_modes, int n_mb, int first_mode,
                          double r_wilson, double m_fermion, double dt, int *bad, cudaStream_t stream, void *lo_psi,
                          void *lo_mid, int nc, bool overlap, double m_dw) {
    FreeMode *info = nullptr;
    cudaMallocAsync(&info, sizeof(FreeMode) * (size_t)n_modes, stream);
    cudaMemsetAsync(bad, 0, sizeof(int), stream);
    free_modes_kernel<<<(n_modes + 127) / 128, 128, 0, stream>>>(info, n_modes, first_mode, L, r_wilson, m_fermion, bad,
                                                                 nc, overlap ? 1 : 0, m_dw);
    dim3 block(kModeBlock, kSitesPerCta);
    dim3 grid((L.V + kSitesPerCta - 1) / kSitesPerCta, n_mb);
    free_fill_kernel<T><<<grid, block, 0, stream>>>(info, reinterpret_cast<cpx<T> *>(psi), reinterpret_cast<cpx<T> *>(psimid),
                                                    L, n_modes, n_mb, dt, reinterpret_cast<unsigned char *>(lo_psi),
                                                    reinterpret_cast<unsigned char *>(lo_mid), nc);
    cudaFreeAsync(info, stream);
}

#define OVL_INSTANTIATE(T)                                                                                          \
    template void launch_charges<T>(const double *, const double *, const void *, const Lattice &, int, int, int,     \
                                    double, double *, double *, cudaStream_t);                                      \
    template void launch_currents<T>(const double *, const double *, const void *, const Lattice &, int, int, int,   \
                                     double, double *, double *, cudaStream_t);                                     \
    template void su3_launch_charges<T>(const double *, const double *, const void *, const Lattice &, int, int, int, \
                                        double, double *, double *, cudaStream_t);                                  \
    template void su3_launch_currents<T>(const double *, const double *, const void *, const Lattice &, int, int,    \
                                         int, double, double *, double *, cudaStream_t);                            \
    template void launch_ref_to_blocks<T>(const double *, void *, const Lattice &, int, int, cudaStream_t, void *,    \
                                          int);                                                                     \
    template void launch_blocks_to_ref<T>(const void *, double *, const Lattice &, int, int, cudaStream_t,          \
                                          const void *, int);                                                       \
    template void launch_free_fermions<T>(void *, void *, const Lattice &, int, int, int, double, double, double,    \
                                          int *, cudaStream_t, void *, void *, int, bool, double);
OVL_INSTANTIATE(double)
OVL_INSTANTIATE(float)

}  // namespace ovl
