// Overlap evolution operator -i h_ov on the mode batch (FP64 parity form).
//
// Reference: OverlapOperator::Compute (FERMIONS/OVERLAP/OPERATOR/OverlapOperator.cpp:25-65)
// -> OverlapU (OverlapU.cpp:152-208) -> Zolotrr (OverlapU.cpp:5-149):
//   chi = sum_k b_k (h_W^2 + d_k)^-1 phi        (multi-shift CG, 25 shifts)
//   out = M [ -i g0 (1 + m/2) phi + (1 - m/2) D chi ],   D = -i h_W,  h_W^2 = -D^2.
// The reference runs the multi-shift CG once per mode; here every mode of the
// batch runs it in lockstep.  Each mode keeps its own CG scalars and stops on
// its own test (rnorm > cgerr * bnorm, at most nitcgm iterations, OverlapU.cpp:56,113)
// through a per-mode `active` mask, so every mode takes exactly the iterations
// the reference would.  The scalar recurrences keep the reference's order of
// operations (OverlapU.cpp:71-110).  Dot products are per mode, two-stage with
// a fixed order.

#include <algorithm>
#include <type_traits>
#include <vector>

#include "ovl_device.cuh"
#include "ovl_internal.h"
#include "ovl_stencil.cuh"

namespace ovl {

static int elem_grid(size_t n, int sm_count) {
    size_t b = (n + 255) / 256;
    size_t cap = (size_t)sm_count * 16;
    return (int)(b < cap ? (b > 0 ? b : 1) : cap);
}

// ---------------------------------------------------------- vector kernels --
// The vector kernels put a mode on a lane: a warp walks the rows (site,
// component) of one mode block, 512 contiguous bytes each, so the CG scalars
// of its 32 modes are read once per thread.  Grid (mode blocks, chunks of
// rows), CTAs of kCgWarps warps.
constexpr int kCgWarps = 8;

// The sum of v over the CTA's warps, per lane, in a fixed order; warp 0 writes
// it to part[chunk][mode].
__device__ __forceinline__ void cg_partial(double v, double *__restrict__ part, int chunk, int m, int modes_padded) {
    __shared__ double sh[kCgWarps][kModeBlock];
    __syncthreads();  // sh is reused by the CTA's next mode block
    sh[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.y == 0) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < kCgWarps; w++) t += sh[w][threadIdx.x];
        part[(size_t)chunk * modes_padded + m] = t;
    }
}

// r = phi, p_k = phi, chi = 0 and the partial sums of |phi|^2.
__global__ void __launch_bounds__(kModeBlock *kCgWarps)
    mscg_init_vectors_kernel(const cpx<double> *__restrict__ phi, cpx<double> *__restrict__ r, cpx<double> *__restrict__ p,
                             cpx<double> *__restrict__ chi, int V, size_t n, int npoles, double *__restrict__ part,
                             int modes_padded) {
    const int lane = threadIdx.x, mb = blockIdx.x, rows = V * kComp;
    const size_t base = (size_t)mb * rows * kModeBlock + lane;
    double t = 0.0;
    for (int j = blockIdx.y * kCgWarps + threadIdx.y; j < rows; j += gridDim.y * kCgWarps) {
        const size_t e = base + (size_t)j * kModeBlock;
        const cpx<double> v = ld(phi + e);
        st(r + e, v);
        st(chi + e, mk<double>(0.0, 0.0));
        for (int k = 0; k < npoles; k++) st(p + (size_t)k * n + e, v);
        t += v.re * v.re + v.im * v.im;
    }
    cg_partial(t, part, blockIdx.y, mb * kModeBlock + lane, modes_padded);
}

// q = -D t + d0 p0 with t = D p0 (h_W^2 = -D^2, WilsonUU, RitzSolver.cpp:49-89)
// and the partial sums of <p0, q>, one chunk per CTA row of sites.  TABLE: the
// CTA runs mblk mode blocks on its sites' links gathered once (fill_link_table).
template <class LK, bool TABLE>
__global__ void __launch_bounds__(kModeBlock *kSitesPerCta, 2)
    cg_square_kernel(LK lk, const cpx<double> *__restrict__ t, const cpx<double> *__restrict__ p0,
                     cpx<double> *__restrict__ q, Lattice L, double amass, double d0, int n_mb, int mblk,
                     double *__restrict__ part, int modes_padded) {
    static_assert(kCgWarps == kSitesPerCta, "cg_partial sums the CTA's warps");
    const int lane = threadIdx.x, site0 = blockIdx.x * kSitesPerCta, site = site0 + threadIdx.y;
    const bool live = site < L.V;
    auto block = [&](const auto &links, int mb) {
        double sum = 0.0;
        if (live) {
            Spinor<double> acc;
            wilson_site_lk(links, t, L, site, mb, lane, amass, acc);
            const size_t base = field_index(L.V, mb, site, 0, lane);
#pragma unroll
            for (int c = 0; c < kColours; c++)
#pragma unroll
                for (int a = 0; a < kSpin; a++) {
                    const size_t i = base + (c * kSpin + a) * kModeBlock;
                    const cpx<double> d = finish_component(acc.c[c][a], a), b = ld(p0 + i);
                    const cpx<double> v = mk<double>(-d.re + b.re * d0, -d.im + b.im * d0);
                    st(q + i, v);
                    sum += b.re * v.re + b.im * v.im;
                }
        }
        cg_partial(sum, part, blockIdx.x, mb * kModeBlock + lane, modes_padded);
    };
    if constexpr (TABLE) {
        __shared__ cmat2<double> tab[kSitesPerCta][6];
        fill_link_table<kSitesPerCta>(lk, L, [&](int j) { return site0 + j < L.V ? site0 + j : -1; }, tab);
        const LinksTable lt{tab[threadIdx.y], site};
        const int mb0 = blockIdx.y * mblk, mb1 = min(n_mb, mb0 + mblk);
        for (int mb = mb0; mb < mb1; mb++) block(lt, mb);
    } else {
        block(lk, (int)blockIdx.y);
    }
}

static void launch_cg_square(const double *U, const double *u1, const void *t, const void *p0, void *q, const Lattice &L,
                             int n_mb, double amass, double d0, double *part, int modes_padded, cudaStream_t stream) {
    const cpx<double> *ts = reinterpret_cast<const cpx<double> *>(t), *ps = reinterpret_cast<const cpx<double> *>(p0);
    cpx<double> *qs = reinterpret_cast<cpx<double> *>(q);
    const int gx = cg_square_chunks(L), m = link_blocks(gx, n_mb, current_sm_count());
    const dim3 block(kModeBlock, kSitesPerCta), grid(gx, (n_mb + m - 1) / m);
    auto go = [&](const auto &lk) {
        using LK = std::decay_t<decltype(lk)>;
        if (m > 1)
            cg_square_kernel<LK, true><<<grid, block, 0, stream>>>(lk, ts, ps, qs, L, amass, d0, n_mb, m, part, modes_padded);
        else
            cg_square_kernel<LK, false><<<grid, block, 0, stream>>>(lk, ts, ps, qs, L, amass, d0, n_mb, 1, part, modes_padded);
    };
    if (u1) go(LinksF64<true>{U, reinterpret_cast<const double2 *>(u1), L.N0 * L.N1});
    else go(LinksF64<false>{U, nullptr, L.N0 * L.N1});
}

// r -= beta0 q for active modes, and the partial sums of |r|^2.
__global__ void __launch_bounds__(kModeBlock *kCgWarps)
    residual_kernel(cpx<double> *r, const cpx<double> *__restrict__ q, const double *__restrict__ beta0,
                    const int *__restrict__ active, int V, double *__restrict__ part, int modes_padded) {
    const int lane = threadIdx.x, mb = blockIdx.x, rows = V * kComp, m = mb * kModeBlock + lane;
    const size_t base = (size_t)mb * rows * kModeBlock + lane;
    const bool act = active[m] != 0;
    const double b = act ? beta0[m] : 0.0;
    double t = 0.0;
    if (act)
        for (int j = blockIdx.y * kCgWarps + threadIdx.y; j < rows; j += gridDim.y * kCgWarps) {
            const size_t e = base + (size_t)j * kModeBlock;
            const cpx<double> a = r[e], y = ld(q + e);
            const cpx<double> v = mk<double>(a.re - b * y.re, a.im - b * y.im);
            st(r + e, v);
            t += v.re * v.re + v.im * v.im;
        }
    cg_partial(t, part, blockIdx.y, m, modes_padded);
}

// For active modes and their unfinished shifts k < kact: chi += b_k beta_k p_k
// (the step x_k += beta_k p_k of OverlapU.cpp:95-108 and the combination
// chi = sum_k b_k x_k of :129-133 in one), then p_k = p_k alpha_k + r g_k.
// Only the combination of the shifted solutions is wanted, so the 25 x_k are
// not kept: per iteration the kernel moves 2 kact + 3 fields instead of 4 x 25 + 1
// and the work space is half as large.  A thread holds kShiftRows rows so that
// the scalars of a shift are read once for all of them.
// One overlap leapfrog step at 8^3, 256 modes, 25 poles: 125 ms with the x_k,
// separate dot products and a host wait per iteration, 91 ms with this CG (the
// rest are the Ritz solves).
constexpr int kShiftRows = 4;

__global__ void __launch_bounds__(kModeBlock *kCgWarps)
    shift_update_kernel(cpx<double> *__restrict__ chi, cpx<double> *__restrict__ p, const cpx<double> *__restrict__ r,
                        const double *__restrict__ beta, const double *__restrict__ alpha, const double *__restrict__ g,
                        const double *__restrict__ bz, const int *__restrict__ active, const int *__restrict__ kact,
                        int V, size_t n, int modes_padded) {
    const int lane = threadIdx.x, mb = blockIdx.x, rows = V * kComp, m = mb * kModeBlock + lane;
    if (!active[m]) return;
    const int nk = kact[m];
    const size_t base = (size_t)mb * rows * kModeBlock + lane;
    const int step = gridDim.y * kCgWarps;
    for (int j0 = blockIdx.y * kCgWarps + threadIdx.y; j0 < rows; j0 += step * kShiftRows) {
        cpx<double> rv[kShiftRows], x[kShiftRows];
        size_t e[kShiftRows];
#pragma unroll
        for (int u = 0; u < kShiftRows; u++) {
            const int j = j0 + u * step;
            e[u] = base + (size_t)min(j, rows - 1) * kModeBlock;
            rv[u] = ld(r + e[u]);
            x[u] = chi[e[u]];
        }
        for (int k = 0; k < nk; k++) {
            const size_t s = (size_t)k * modes_padded + m;
            const double cb = bz[k] * beta[s], ak = alpha[s], gk = g[s];
            cpx<double> *pk = p + (size_t)k * n;
            cpx<double> pv[kShiftRows];
#pragma unroll
            for (int u = 0; u < kShiftRows; u++) pv[u] = pk[e[u]];
#pragma unroll
            for (int u = 0; u < kShiftRows; u++) {
                x[u] = mk<double>(x[u].re + cb * pv[u].re, x[u].im + cb * pv[u].im);
                if (j0 + u * step < rows)
                    st(pk + e[u], mk<double>(pv[u].re * ak + rv[u].re * gk, pv[u].im * ak + rv[u].im * gk));
            }
        }
#pragma unroll
        for (int u = 0; u < kShiftRows; u++)
            if (j0 + u * step < rows) st(chi + e[u], x[u]);
    }
}

// out = M [ -i g0 (1 + m/2) phi + (1 - m/2) Dchi ]  (OverlapU.cpp:188-202); dst = out or dst += dt out
__global__ void overlap_finish_kernel(const cpx<double> *__restrict__ phi, const cpx<double> *__restrict__ dchi,
                                      cpx<double> *dst, size_t n, double mdw, double mf, double dt, int accumulate) {
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int spin = (int)((e / kModeBlock) % kComp) % kSpin;
        const cpx<double> f = ld(phi + e), d = ld(dchi + e);
        const double cp = 1.0 + 0.5 * mf, cm = 1.0 - 0.5 * mf;
        // -i g0: spins 0,1 -> -i, spins 2,3 -> +i
        const cpx<double> a = spin < 2 ? mk<double>(cp * f.im, -cp * f.re) : mk<double>(-cp * f.im, cp * f.re);
        const cpx<double> o = mk<double>(mdw * (a.re + cm * d.re), mdw * (a.im + cm * d.im));
        if (accumulate) {
            const cpx<double> v = ld(dst + e);
            st(dst + e, mk<double>(v.re + dt * o.re, v.im + dt * o.im));
        } else {
            st(dst + e, o);
        }
    }
}

// ---------------------------------------------------------- scalar kernels --
// One CTA of 32 x kCgWarps threads per mode block: the chunks' partial sums of
// the dot product are added (in a fixed order), then the shifts of a mode are
// shared out over the CTA's warps.  One thread per mode walking the chunks and
// the 25 shifts alone took 16-20 us per launch, all of it load latency.
struct CgScalars {
    double *rnorm, *bnorm, *betam;
    double *alpha, *beta, *z, *g;  // [npoles][modes_padded]
    int *active, *next, *iters;    // active this iteration / after it
    int *kact, *knext;             // unfinished shifts of a mode, k < kact: this iteration / after it
    int *count;                    // number of modes active after the update
};

__device__ __forceinline__ double cg_total(const double *__restrict__ part, int chunks, int m, int modes_padded) {
    __shared__ double sh[kCgWarps][kModeBlock];
    double t = 0.0;
    for (int c = threadIdx.y; c < chunks; c += kCgWarps) t += part[(size_t)c * modes_padded + m];
    sh[threadIdx.y][threadIdx.x] = t;
    __syncthreads();
    t = 0.0;
#pragma unroll
    for (int w = 0; w < kCgWarps; w++) t += sh[w][threadIdx.x];
    return t;
}

// rnorm = |phi|^2, bnorm = sqrt(rnorm), betam = 1, alpha_0 = 0, z_k = g_k = 1 (OverlapU.cpp:39-54)
__global__ void __launch_bounds__(kModeBlock *kCgWarps)
    cg_init_scalars_kernel(CgScalars s, const double *__restrict__ part, int chunks, int n_modes, int modes_padded,
                           int npoles, double cgerr) {
    const int m = blockIdx.x * kModeBlock + threadIdx.x;
    const double rn = cg_total(part, chunks, m, modes_padded);
    for (int k = threadIdx.y; k < npoles; k += kCgWarps) {
        const size_t i = (size_t)k * modes_padded + m;
        s.alpha[i] = 0.0;
        s.z[i] = 1.0;
        s.g[i] = 1.0;
        s.beta[i] = 0.0;
    }
    if (threadIdx.y != 0) return;
    s.rnorm[m] = rn;
    s.bnorm[m] = sqrt(rn);
    s.betam[m] = 1.0;
    s.iters[m] = 0;
    s.kact[m] = npoles;
    s.knext[m] = npoles;
    const int act = (m < n_modes) && (rn > cgerr * sqrt(rn));
    s.active[m] = act;
    s.next[m] = act;
    if (act) atomicAdd(s.count, 1);
}

// beta_0 = rnorm / <p0, q>; for k >= 1: z_k, beta_k from the previous alpha_0,
// z_k, betam (OverlapU.cpp:71-88).  Clears this iteration's count.
__global__ void __launch_bounds__(kModeBlock *kCgWarps)
    cg_scalars_beta_kernel(CgScalars s, const double *__restrict__ part, int chunks, const double *__restrict__ dz,
                           int modes_padded) {
    const int m = blockIdx.x * kModeBlock + threadIdx.x;
    const double pap = cg_total(part, chunks, m, modes_padded);
    if (blockIdx.x == 0 && threadIdx.x == 0 && threadIdx.y == 0) *s.count = 0;
    if (!s.active[m]) return;
    const double b0 = s.rnorm[m] / pap, a0 = s.alpha[m], bm = s.betam[m];
    const int nk = s.kact[m];
    for (int k = threadIdx.y; k < nk; k += kCgWarps) {
        const size_t i = (size_t)k * modes_padded + m;
        if (k == 0) {
            s.beta[i] = b0;
            continue;
        }
        const double dr = b0 * a0 * (1.0 - s.z[i]) + bm * (1.0 + (dz[k] - dz[0]) * b0);
        s.z[i] = bm / dr;
        s.beta[i] = b0 * s.z[i];
    }
}

// alpha_0 = |r|^2 / rnorm, rnorm = |r|^2; per shift alpha_k and g_k as the
// shift loop of OverlapU.cpp:95-106 computes them (alpha_0 is rewritten at
// k = 0 before the other shifts read it); betam = beta_0; iteration count and
// the stopping test (OverlapU.cpp:56, 110-117).
//
// Finished shifts: g_k r is the residual of the shifted system k, so what its
// further steps could still add to chi is at most b_k |g_k r| / (lambda_min +
// d_k).  sum_k b_k / (lambda + d_k) approximates lambda^(-1/2), every term is
// positive, and |chi| >= |phi| lambda_max^(-1/2): relative to chi that is at
// most sqrt(lambda_max / lambda_min) |g_k r| / |phi|.  A shift is left alone
// once |g_k r| <= kShiftDone |phi| = 1e-20 |phi|, which bounds it by 1e-18 at a
// condition number of 1e4, below the rounding of chi.  Poles come in
// ascending order and the larger ones finish first; kact is the last
// unfinished one + 1 and never grows; the step that finishes a shift is still
// applied (knext is the next iteration's kact).
constexpr double kShiftDone = 1e-20;

__global__ void __launch_bounds__(kModeBlock *kCgWarps)
    cg_scalars_alpha_kernel(CgScalars s, const double *__restrict__ part, int chunks, int modes_padded, double cgerr,
                            int max_iter) {
    __shared__ int last[kCgWarps][kModeBlock];
    const int m = blockIdx.x * kModeBlock + threadIdx.x;
    const double rr = cg_total(part, chunks, m, modes_padded);
    const bool active = s.active[m] != 0;
    int unfinished = 0;
    double b0 = 0.0;
    if (active) {
        const int nk = s.kact[m];
        const double bnorm = s.bnorm[m], a00 = rr / s.rnorm[m];
        b0 = s.beta[m];
        const double a0 = a00 * s.z[m] * s.beta[m] / b0;  // shift 0
        for (int k = threadIdx.y; k < nk; k += kCgWarps) {
            const size_t i = (size_t)k * modes_padded + m;
            const double zk = s.z[i], gk = s.g[i] * zk;
            s.alpha[i] = k == 0 ? a0 : a0 * zk * s.beta[i] / b0;
            s.g[i] = gk;
            // bnorm = |phi|; compared as squares
            if (gk * gk * rr > kShiftDone * kShiftDone * bnorm * bnorm) unfinished = k + 1;
        }
    }
    last[threadIdx.y][threadIdx.x] = unfinished;
    __syncthreads();  // every warp has read rnorm, z, beta of shift 0 and kact
    if (threadIdx.y != 0) return;
    if (!active) {
        s.next[m] = 0;
        return;
    }
    for (int w = 1; w < kCgWarps; w++) unfinished = max(unfinished, last[w][threadIdx.x]);
    s.knext[m] = max(1, unfinished);  // shift 0 carries the iteration
    s.rnorm[m] = rr;
    s.betam[m] = b0;
    const int it = s.iters[m] + 1;
    s.iters[m] = it;
    const int act = (it < max_iter) && (rr > cgerr * s.bnorm[m]);
    s.next[m] = act;
    if (act) atomicAdd(s.count, 1);
}

// --------------------------------------------------------- overlap currents --
// Fermions::Observables::ComputeCurrents, overlap (FERMIONS/OVERLAP/OverlapCurrents.cpp:35-212):
// local bilinears only, with O = -i h_ov psi:
//   jV^mu = Re[psi^+ g0 g_mu psi + psi^+ (-i/2) g0 g_mu g0 O]
//   jA^mu = Re[psi^+ g0 g_mu g5 psi + psi^+ (-i/2) g0 g_mu g5 g0 O]      (g_0 for mu = 0)
// weighted by the vacuum sign and summed over colours and modes; per site the
// output slots are those of the Wilson currents (jV, jA; the rest zero).
// Modes of precision T and NC colours; the bilinears in FP64.
template <typename T, int NC>
__global__ void __launch_bounds__(kModeBlock *kSitesPerCta)
    overlap_currents_kernel(const cpx<T> *__restrict__ psi, const cpx<T> *__restrict__ opsi, Lattice L,
                            int n_mb, int n_modes, int first_mode, int groups, double *__restrict__ partial) {
    constexpr mono GV[4] = {mono_mul(kGamma0, kGamma0), mono_mul(kGamma0, kGammaX), mono_mul(kGamma0, kGammaY),
                            mono_mul(kGamma0, kGammaZ)};
    constexpr mono GA[4] = {mono_mul(GV[0], kGamma5), mono_mul(GV[1], kGamma5), mono_mul(GV[2], kGamma5),
                            mono_mul(GV[3], kGamma5)};
    constexpr mono GV2[4] = {mono_mul(GV[0], kGamma0), mono_mul(GV[1], kGamma0), mono_mul(GV[2], kGamma0),
                             mono_mul(GV[3], kGamma0)};
    constexpr mono GA2[4] = {mono_mul(GA[0], kGamma0), mono_mul(GA[1], kGamma0), mono_mul(GA[2], kGamma0),
                             mono_mul(GA[3], kGamma0)};
    const int lane = threadIdx.x;
    const int site = blockIdx.x * kSitesPerCta + threadIdx.y;
    const int g = blockIdx.y;
    if (site >= L.V) return;
    CompSum sum[8];
    for (int mb = g; mb < n_mb; mb += groups) {
        const int mode = mb * kModeBlock + lane;
        const double w = mode >= n_modes ? 0.0 : (((first_mode + mode) & 1) == 0 ? 1.0 : -1.0);
        cpx<double> f[NC][kSpin], o[NC][kSpin];
        const size_t base = (((size_t)mb * L.V + site) * (NC * kSpin)) * kModeBlock + lane;
#pragma unroll
        for (int c = 0; c < NC; c++)
#pragma unroll
            for (int a = 0; a < kSpin; a++) {
                const cpx<T> x = ld(psi + base + (c * kSpin + a) * kModeBlock);
                const cpx<T> y = ld(opsi + base + (c * kSpin + a) * kModeBlock);
                f[c][a] = mk<double>((double)x.re, (double)x.im);
                o[c][a] = mk<double>((double)y.re, (double)y.im);
            }
#pragma unroll
        for (int mu = 0; mu < 4; mu++) {
            cpx<double> v1 = mk<double>(0, 0), v2 = mk<double>(0, 0), a1 = mk<double>(0, 0), a2 = mk<double>(0, 0);
#pragma unroll
            for (int c = 0; c < NC; c++) {
                v1 = v1 + bilinear<double>(GV[mu], f[c], f[c]);
                v2 = v2 + bilinear<double>(GV2[mu], f[c], o[c]);
                a1 = a1 + bilinear<double>(GA[mu], f[c], f[c]);
                a2 = a2 + bilinear<double>(GA2[mu], f[c], o[c]);
            }
            // Re(z1 + (-i/2) z2) = Re z1 + Im z2 / 2
            sum[mu].add(w * (v1.re + 0.5 * v2.im));
            sum[4 + mu].add(w * (a1.re + 0.5 * a2.im));
        }
    }
    double acc[8];
#pragma unroll
    for (int k = 0; k < 8; k++) acc[k] = sum[k].value();
#pragma unroll
    for (int k = 0; k < 8; k++) {
        double t = acc[k];
        for (int off = 16; off > 0; off >>= 1) t += __shfl_down_sync(0xffffffffu, t, off);
        acc[k] = t;
    }
    if (lane == 0) {
        double *p = partial + ((size_t)g * L.V + site) * kCurrentsPerSite;
        for (int k = 0; k < kCurrentsPerSite; k++) p[k] = k < 8 ? acc[k] : 0.0;
    }
}

template <typename T, int NC>
static void overlap_currents_t(const void *psi, const void *opsi, const Lattice &L, int n_mb, int n_modes,
                               int first_mode, int groups, double *partial, cudaStream_t stream) {
    dim3 block(kModeBlock, kSitesPerCta);
    dim3 grid((L.V + kSitesPerCta - 1) / kSitesPerCta, groups);
    overlap_currents_kernel<T, NC><<<grid, block, 0, stream>>>(reinterpret_cast<const cpx<T> *>(psi),
                                                               reinterpret_cast<const cpx<T> *>(opsi), L, n_mb, n_modes,
                                                               first_mode, groups, partial);
}

void launch_overlap_currents(const void *psi, const void *opsi, const Lattice &L, int n_mb, int n_modes,
                             int first_mode, double *partial, double *per_site, cudaStream_t stream, bool fp32, int nc) {
    const int groups = currents_groups(n_mb);
    if (nc == 3) {
        if (fp32) overlap_currents_t<float, 3>(psi, opsi, L, n_mb, n_modes, first_mode, groups, partial, stream);
        else overlap_currents_t<double, 3>(psi, opsi, L, n_mb, n_modes, first_mode, groups, partial, stream);
    } else {
        if (fp32) overlap_currents_t<float, 2>(psi, opsi, L, n_mb, n_modes, first_mode, groups, partial, stream);
        else overlap_currents_t<double, 2>(psi, opsi, L, n_mb, n_modes, first_mode, groups, partial, stream);
    }
    launch_currents_finish(partial, groups, L, per_site, stream);
}

// ------------------------------------------------------------------ driver --
int cg_square_chunks(const Lattice &L) { return (L.V + kSitesPerCta - 1) / kSitesPerCta; }

// Chunks of rows of the vector kernels: at least four CTAs per SM where the
// rows allow it, at most kDotChunks.
static int cg_chunks(const Lattice &L, int n_mb, int sm_count) {
    const int most = std::min(kDotChunks, (L.V * kComp + kCgWarps * kShiftRows - 1) / (kCgWarps * kShiftRows));
    return std::max(1, std::min(most, (8 * sm_count + n_mb - 1) / n_mb));
}

size_t cg_partial_chunks(const Lattice &L) { return (size_t)std::max(kDotChunks, cg_square_chunks(L)); }

void overlap_apply(OverlapWork &w, const double *U, const double *u1, const void *src, void *dst, const Lattice &L, int n_mb,
                   int n_modes, const OverlapCoeffs &co, double amass, double mdw, double mf, double dt,
                   bool accumulate, int sm_count, cudaStream_t stream, OverlapStats *stats) {
    const size_t n = (size_t)n_mb * L.V * kComp * kModeBlock;
    const int mp = n_mb * kModeBlock;
    const int np = co.npoles;
    const int grid = elem_grid(n, sm_count);
    const cpx<double> *phi = reinterpret_cast<const cpx<double> *>(src);
    cpx<double> *r = reinterpret_cast<cpx<double> *>(w.r), *q = reinterpret_cast<cpx<double> *>(w.q);
    cpx<double> *t = reinterpret_cast<cpx<double> *>(w.t);
    cpx<double> *chi = reinterpret_cast<cpx<double> *>(w.x), *p = reinterpret_cast<cpx<double> *>(w.p);
    CgScalars s{w.rnorm, w.bnorm, w.betam, w.alpha, w.beta, w.z, w.g, w.active, w.next, w.iters, w.kact, w.knext, w.count};
    cudaMemcpyAsync(w.dz, co.d, sizeof(double) * np, cudaMemcpyHostToDevice, stream);
    cudaMemcpyAsync(w.bz, co.b, sizeof(double) * np, cudaMemcpyHostToDevice, stream);

    const int chunks = cg_chunks(L, n_mb, sm_count), sq_chunks = cg_square_chunks(L);
    const dim3 vblock(kModeBlock, kCgWarps), vgrid(n_mb, chunks);
    mscg_init_vectors_kernel<<<vgrid, vblock, 0, stream>>>(phi, r, p, chi, L.V, n, np, w.part, mp);
    cudaMemsetAsync(w.count, 0, sizeof(int) * 2, stream);
    cg_init_scalars_kernel<<<n_mb, vblock, 0, stream>>>(s, w.part, chunks, n_modes, mp, np, co.cg_tol);
    int launches = 2;
    // The count of modes still active is read back one iteration late, while
    // the next iteration is already queued: the GPU does not wait for the host,
    // and the one iteration queued past the end finds no active mode (two
    // stencil passes, no vector changes).
    auto read_count = [&](int slot) {
        cudaMemcpyAsync(w.host_count + slot, w.count + slot, sizeof(int), cudaMemcpyDeviceToHost, stream);
        cudaEventRecord(w.counted[slot], stream);
    };
    auto counted = [&](int slot) {
        cudaEventSynchronize(w.counted[slot]);
        return w.host_count[slot];
    };
    read_count(0);
    int iterations = 0;
    for (int it = 0;; it++) {
        // q = h_W^2 p0 + d0 p0 = -D(D p0) + d0 p0
        s.count = w.count + ((it + 1) & 1);
        launch_wilson<double>(U, u1, p, w.t, L, 0, n_mb, amass, 0.0, false, stream);
        launch_cg_square(U, u1, w.t, p, q, L, n_mb, amass, co.d[0], w.part, mp, stream);
        cg_scalars_beta_kernel<<<n_mb, vblock, 0, stream>>>(s, w.part, sq_chunks, w.dz, mp);
        residual_kernel<<<vgrid, vblock, 0, stream>>>(r, q, w.beta, s.active, L.V, w.part, mp);
        cg_scalars_alpha_kernel<<<n_mb, vblock, 0, stream>>>(s, w.part, chunks, mp, co.cg_tol, co.cg_max_iter);
        shift_update_kernel<<<vgrid, vblock, 0, stream>>>(chi, p, r, w.beta, w.alpha, w.g, w.bz, s.active, s.kact, L.V, n,
                                                          mp);
        launches += 6;
        std::swap(s.active, s.next);
        std::swap(s.kact, s.knext);
        read_count((it + 1) & 1);
        if (counted(it & 1) == 0) break;  // no mode was active before this iteration
        iterations++;
        if (iterations > co.cg_max_iter + 1) break;  // every mode stops by then
    }
    launch_wilson<double>(U, u1, chi, w.t, L, 0, n_mb, amass, 0.0, false, stream);
    overlap_finish_kernel<<<grid, 256, 0, stream>>>(phi, t, reinterpret_cast<cpx<double> *>(dst), n, mdw, mf, dt,
                                                    accumulate ? 1 : 0);
    launches += 2;
    if (stats) {
        stats->launches += launches;
        stats->iterations = iterations;
        int mx = 0;
        std::vector<int> it(mp);
        cudaMemcpyAsync(it.data(), w.iters, sizeof(int) * mp, cudaMemcpyDeviceToHost, stream);
        cudaStreamSynchronize(stream);
        int capped = 0;
        for (int m = 0; m < n_modes; m++) {
            mx = std::max(mx, it[m]);
            if (it[m] >= co.cg_max_iter) capped++;
        }
        stats->max_mode_iterations = mx;
        stats->not_converged = capped;
    }
}

}  // namespace ovl
