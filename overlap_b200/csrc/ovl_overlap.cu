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
constexpr int kCgWarps = 8, kCgRows = 2;

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

// r = p0 = p_k = phi, chi = 0 and the partial sums of |phi|^2.
__global__ void __launch_bounds__(kModeBlock *kCgWarps)
    mscg_init_vectors_kernel(const cpx<double> *__restrict__ phi, cpx<double> *__restrict__ r, cpx<double> *__restrict__ p0,
                             cpx<double> *__restrict__ p, cpx<double> *__restrict__ chi, int V, size_t n, int npoles,
                             double *__restrict__ part, int modes_padded) {
    const int lane = threadIdx.x, mb = blockIdx.x, rows = V * kComp;
    const size_t base = (size_t)mb * rows * kModeBlock + lane;
    double t = 0.0;
    for (int j = blockIdx.y * kCgWarps + threadIdx.y; j < rows; j += gridDim.y * kCgWarps) {
        const size_t e = base + (size_t)j * kModeBlock;
        const cpx<double> v = ld(phi + e);
        st(r + e, v);
        st(p0 + e, v);
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

// The sum of a mode's partial sums over the chunks, in a fixed order; every
// thread of the CTA (32 modes x kCgWarps) gets its mode's.
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

// Sums the chunks' partial sums down to kDotChunks chunks (lattices of many
// site CTAs, so that the kernels that read them add few).
__global__ void __launch_bounds__(kModeBlock *kCgWarps)
    cg_fold_kernel(const double *__restrict__ part, int chunks, double *__restrict__ out, int modes_padded) {
    const int m = blockIdx.x * kModeBlock + threadIdx.x;
    for (int o = blockIdx.y * kCgWarps + threadIdx.y; o < kDotChunks; o += gridDim.y * kCgWarps) {
        const int c0 = (int)((long long)chunks * o / kDotChunks), c1 = (int)((long long)chunks * (o + 1) / kDotChunks);
        double t = 0.0;
        for (int c = c0; c < c1; c++) t += part[(size_t)c * modes_padded + m];
        out[(size_t)o * modes_padded + m] = t;
    }
}

// ---------------------------------------------------------- CG scalars --
// The CG of the smallest shift runs iteration by iteration; the other shifts'
// vectors only follow it (x_k += beta_k p_k, p_k = alpha_k p_k + g_k r), so they
// are brought up to date once per kCgBatch iterations from the residuals and
// the scalars of those iterations: their 2 x 25 fields are moved once per
// batch.  Slot j of a batch: its residual r[j] and its scalars.
constexpr int kCgBatch = kCgBatchSlots;

struct CgScalars {
    double *rnorm[2];              // |r|^2 before / after an iteration, by its parity
    double *bnorm, *betam, *alpha0, *beta0;
    double *z, *g;                 // [npoles][modes_padded]
    double *cb, *al, *gg;          // [kCgBatch][npoles][modes_padded]: b_k beta_k, alpha_k, g_k of a slot
    int *active, *next, *iters;    // active this iteration / after it
    int *kact, *knext;             // unfinished shifts of a mode, k < kact: in this batch / by the last iteration
    int *steps;                    // iterations of this batch that a mode took part in
    int *count;                    // number of modes active after the iteration
};

// rnorm = |phi|^2, bnorm = sqrt(rnorm), betam = 1, alpha_0 = 0, z_k = g_k = 1 (OverlapU.cpp:39-54)
__global__ void __launch_bounds__(kModeBlock *kCgWarps)
    cg_init_scalars_kernel(CgScalars s, const double *__restrict__ part, int chunks, int n_modes, int modes_padded,
                           int npoles, double cgerr) {
    const int m = blockIdx.x * kModeBlock + threadIdx.x;
    const double rn = cg_total(part, chunks, m, modes_padded);
    for (int k = threadIdx.y; k < npoles; k += kCgWarps) {
        const size_t i = (size_t)k * modes_padded + m;
        s.z[i] = 1.0;
        s.g[i] = 1.0;
    }
    if (threadIdx.y != 0) return;
    s.rnorm[0][m] = rn;
    s.bnorm[m] = sqrt(rn);
    s.betam[m] = 1.0;
    s.alpha0[m] = 0.0;
    s.iters[m] = 0;
    s.kact[m] = npoles;
    s.knext[m] = npoles;
    s.steps[m] = 0;
    const int act = (m < n_modes) && (rn > cgerr * sqrt(rn));
    s.active[m] = act;
    s.next[m] = act;
    if (act) atomicAdd(s.count, 1);
}

// beta_0 = rnorm / <p0, q> (OverlapU.cpp:71-75) from the partial sums of <p0, q>,
// rout = rin - beta_0 q for active modes, and the partial sums of |rout|^2.
// INPLACE: rin is rout (a batch of one iteration).  Clears this iteration's count.
template <bool INPLACE>
__global__ void __launch_bounds__(kModeBlock *kCgWarps)
    residual_kernel(CgScalars s, int parity, const double *__restrict__ pap_part, int pap_chunks,
                    const cpx<double> *__restrict__ rin, cpx<double> *__restrict__ rout, const cpx<double> *__restrict__ q,
                    int V, double *__restrict__ part, int modes_padded) {
    const int lane = threadIdx.x, mb = blockIdx.x, rows = V * kComp, m = mb * kModeBlock + lane;
    const double pap = cg_total(pap_part, pap_chunks, m, modes_padded);
    const size_t base = (size_t)mb * rows * kModeBlock + lane;
    const bool act = s.active[m] != 0;
    const double b = act ? s.rnorm[parity][m] / pap : 0.0;
    if (blockIdx.y == 0 && threadIdx.y == 0) {
        s.beta0[m] = b;
        if (m == 0) *s.count = 0;
    }
    double t = 0.0;
    if (act)
        for (int j = blockIdx.y * kCgWarps + threadIdx.y; j < rows; j += gridDim.y * kCgWarps) {
            const size_t e = base + (size_t)j * kModeBlock;
            const cpx<double> a = INPLACE ? rout[e] : ld(rin + e), y = ld(q + e);
            const cpx<double> v = mk<double>(a.re - b * y.re, a.im - b * y.im);
            st(rout + e, v);
            t += v.re * v.re + v.im * v.im;
        }
    cg_partial(t, part, blockIdx.y, m, modes_padded);
}

// Finished shifts: g_k r is the residual of the shifted system k, so what its
// further steps could still add to chi is at most b_k |g_k r| / (lambda_min +
// d_k).  sum_k b_k / (lambda + d_k) approximates lambda^(-1/2), every term is
// positive, and |chi| >= |phi| lambda_max^(-1/2): relative to chi that is at
// most sqrt(lambda_max / lambda_min) |g_k r| / |phi|.  A shift is left alone
// once |g_k r| <= kShiftDone |phi| = 1e-20 |phi|, which bounds it by 1e-18 at a
// condition number of 1e4, below the rounding of chi.  Poles come in
// ascending order and the larger ones finish first; kact is the last
// unfinished one + 1 and never grows.
constexpr double kShiftDone = 1e-20;

// The end of an iteration (slot j of its batch).  CTAs with blockIdx.y > 0:
// alpha_0 = |r|^2 / rnorm and p0 = alpha_0 p0 + r for active modes.  The CTA
// with blockIdx.y = 0: the iteration's scalars of every unfinished shift, shared
// out over its warps -- z_k, beta_k from the previous alpha_0, z_k, betam
// (OverlapU.cpp:71-88), alpha_k and g_k as the shift loop of :95-106 computes
// them (alpha_0 is rewritten at k = 0 before the other shifts read it) -- then
// betam = beta_0, the iteration count and the stopping test (:56, 110-117).
// keep (or null): receives p0 of before the step, the direction that a single
// shift's update needs after it.
__global__ void __launch_bounds__(kModeBlock *kCgWarps)
    cg_advance_kernel(CgScalars s, int parity, int slot, const double *__restrict__ part, int chunks,
                      const double *__restrict__ dz, const double *__restrict__ bz, int npoles, double cgerr, int max_iter,
                      cpx<double> *__restrict__ p0, const cpx<double> *__restrict__ r, cpx<double> *__restrict__ keep,
                      int V, int modes_padded) {
    const int lane = threadIdx.x, mb = blockIdx.x, m = mb * kModeBlock + lane;
    const double rr = cg_total(part, chunks, m, modes_padded);
    const bool active = s.active[m] != 0;
    const double b0 = s.beta0[m];
    // z_0 = 1 and beta_0 = b0, in the reference's order of operations
    const double a0 = active ? rr / s.rnorm[parity][m] * 1.0 * b0 / b0 : 0.0;
    if (blockIdx.y > 0) {
        if (!active) return;
        const int rows = V * kComp;
        const size_t base = (size_t)mb * rows * kModeBlock + lane;
        for (int j = (blockIdx.y - 1) * kCgWarps + threadIdx.y; j < rows; j += (gridDim.y - 1) * kCgWarps) {
            const size_t e = base + (size_t)j * kModeBlock;
            const cpx<double> pv = p0[e], rv = ld(r + e);
            if (keep) st(keep + e, pv);
            st(p0 + e, mk<double>(pv.re * a0 + rv.re, pv.im * a0 + rv.im));
        }
        return;
    }
    __shared__ int last[kCgWarps][kModeBlock];
    const int nk = slot == 0 ? s.knext[m] : s.kact[m];
    int unfinished = 0;
    if (active) {
        const double ap = s.alpha0[m], bm = s.betam[m], bnorm = s.bnorm[m];
        for (int k = threadIdx.y; k < nk; k += kCgWarps) {
            const size_t i = (size_t)k * modes_padded + m, o = (size_t)slot * npoles * modes_padded + i;
            double zk = 1.0, bk = b0, ak = a0;
            if (k > 0) {
                const double dr = b0 * ap * (1.0 - s.z[i]) + bm * (1.0 + (dz[k] - dz[0]) * b0);
                zk = bm / dr;
                bk = b0 * zk;
                ak = a0 * zk * bk / b0;
                s.z[i] = zk;
            }
            const double gk = s.g[i] * zk;
            s.g[i] = gk;
            s.cb[o] = bz[k] * bk;
            s.al[o] = ak;
            s.gg[o] = gk;
            // bnorm = |phi|; compared as squares
            if (gk * gk * rr > kShiftDone * kShiftDone * bnorm * bnorm) unfinished = k + 1;
        }
    }
    last[threadIdx.y][lane] = unfinished;
    __syncthreads();  // every warp has read kact, knext, alpha0 and betam
    if (threadIdx.y != 0) return;
    if (slot == 0) {
        s.kact[m] = nk;
        s.steps[m] = 0;
    }
    if (!active) {
        s.next[m] = 0;
        return;
    }
    for (int w = 1; w < kCgWarps; w++) unfinished = max(unfinished, last[w][lane]);
    s.knext[m] = unfinished;
    s.steps[m] = slot + 1;
    s.rnorm[parity ^ 1][m] = rr;
    s.betam[m] = b0;
    s.alpha0[m] = a0;
    const int it = s.iters[m] + 1;
    s.iters[m] = it;
    const int act = (it < max_iter) && (rr > cgerr * s.bnorm[m]);
    s.next[m] = act;
    if (act) atomicAdd(s.count, 1);
}

// Brings the unfinished shifts of a batch up to date: for each of the mode's
// iterations of the batch chi += b_k beta_k p_k (the step x_k += beta_k p_k of
// OverlapU.cpp:95-108 and the combination chi = sum_k b_k x_k of :129-133 in
// one), then p_k = p_k alpha_k + r g_k.  Only the combination of the shifted
// solutions is wanted, so the 25 x_k are not kept; per batch the kernel moves
// 2 kact fields, the residuals of the batch and chi (HBM bound), against 4 x 25 + 1
// fields per iteration for separate x_k and p_k.
// The scalars of the batch, three per shift and iteration and mode, are staged in
// shared memory once per CTA, for kShiftStage shifts at a time; left to L1 they are
// more than it holds, and their reads from L2 as long as those of the fields.
// One overlap leapfrog step with its two pairs of bounds at 8^3, 256 modes:
// 50 ms with the shifts updated in every iteration, 42.9 ms in batches of eight;
// then, the Ritz solver made faster, 27.3 ms with the scalars left to L1 (508 us
// per batch, 1.9 TB/s) and 20.1 ms with them staged (147 us, 6.6 TB/s; 160 us with
// 12 warps, 188 us with 16 warps of one row each).
constexpr int kShiftRows = 2, kShiftWarps = 16, kShiftStage = 32;

inline size_t shift_smem(int npoles) {
    return sizeof(double) * 3 * kCgBatch * kModeBlock * (size_t)std::min(npoles, kShiftStage);
}

__global__ void __launch_bounds__(kModeBlock *kShiftWarps, 1)
    shift_update_kernel(CgScalars s, cpx<double> *__restrict__ chi, cpx<double> *__restrict__ p,
                        const cpx<double> *__restrict__ r, int V, size_t n, int npoles, int modes_padded) {
    extern __shared__ double shift_sc[];  // [shift of the stage][iteration][b beta, alpha, g][mode]
    const int lane = threadIdx.x, mb = blockIdx.x, rows = V * kComp, m = mb * kModeBlock + lane;
    const int nj = s.steps[m], nk = nj == 0 ? 0 : s.kact[m];
    if (!__syncthreads_or(nk)) return;
    const size_t base = (size_t)mb * rows * kModeBlock + lane;
    const int step = gridDim.y * kShiftWarps;
    for (int k0 = 0; k0 < npoles; k0 += kShiftStage) {
        const int staged = min(kShiftStage, npoles - k0), k1 = min(nk, k0 + staged);
        if (k0) __syncthreads();
        for (int i = threadIdx.y; i < staged * kCgBatch; i += kShiftWarps) {
            const int k = i / kCgBatch, j = i % kCgBatch;
            const size_t o = ((size_t)j * npoles + k0 + k) * modes_padded + m;
            double *d = shift_sc + 3 * i * kModeBlock + lane;
            d[0] = s.cb[o];
            d[kModeBlock] = s.al[o];
            d[2 * kModeBlock] = s.gg[o];
        }
        __syncthreads();
        if (k1 <= k0) continue;
        for (int j0 = blockIdx.y * kShiftWarps + threadIdx.y; j0 < rows; j0 += step * kShiftRows) {
            cpx<double> rv[kCgBatch][kShiftRows], x[kShiftRows], next[kShiftRows];
            size_t e[kShiftRows];
#pragma unroll
            for (int u = 0; u < kShiftRows; u++) {
                e[u] = base + (size_t)min(j0 + u * step, rows - 1) * kModeBlock;
                x[u] = chi[e[u]];
                next[u] = p[(size_t)k0 * n + e[u]];
            }
#pragma unroll
            for (int j = 0; j < kCgBatch; j++)
#pragma unroll
                for (int u = 0; u < kShiftRows; u++)
                    rv[j][u] = j < nj ? ld(r + (size_t)j * n + e[u]) : mk<double>(0.0, 0.0);
            for (int k = k0; k < k1; k++) {
                cpx<double> *pk = p + (size_t)k * n;
                cpx<double> pv[kShiftRows];
#pragma unroll
                for (int u = 0; u < kShiftRows; u++) {
                    pv[u] = next[u];
                    if (k + 1 < k1) next[u] = pk[n + e[u]];  // in flight while this shift is brought up to date
                }
                const double *sc = shift_sc + 3 * (k - k0) * kCgBatch * kModeBlock + lane;
#pragma unroll
                for (int j = 0; j < kCgBatch; j++) {
                    if (j < nj) {
                        const double cb = sc[3 * j * kModeBlock], ak = sc[(3 * j + 1) * kModeBlock],
                                     gk = sc[(3 * j + 2) * kModeBlock];
#pragma unroll
                        for (int u = 0; u < kShiftRows; u++) {
                            x[u] = mk<double>(x[u].re + cb * pv[u].re, x[u].im + cb * pv[u].im);
                            pv[u] = mk<double>(pv[u].re * ak + rv[j][u].re * gk, pv[u].im * ak + rv[j][u].im * gk);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < kShiftRows; u++)
                    if (j0 + u * step < rows) st(pk + e[u], pv[u]);
            }
#pragma unroll
            for (int u = 0; u < kShiftRows; u++)
                if (j0 + u * step < rows) st(chi + e[u], x[u]);
        }
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
    const int most = std::min(kDotChunks, (L.V * kComp + kCgWarps * kCgRows - 1) / (kCgWarps * kCgRows));
    return std::max(1, std::min(most, (8 * sm_count + n_mb - 1) / n_mb));
}

// chunks of |r|^2, of <p0, q>, and of the latter folded
size_t cg_partial_chunks(const Lattice &L) { return (size_t)2 * kDotChunks + cg_square_chunks(L); }

void overlap_apply(OverlapWork &w, const double *U, const double *u1, const void *src, void *dst, const Lattice &L, int n_mb,
                   int n_modes, const OverlapCoeffs &co, double amass, double mdw, double mf, double dt,
                   bool accumulate, int sm_count, cudaStream_t stream, OverlapStats *stats) {
    const size_t n = (size_t)n_mb * L.V * kComp * kModeBlock;
    const int mp = n_mb * kModeBlock;
    const int np = co.npoles;
    const int grid = elem_grid(n, sm_count);
    const cpx<double> *phi = reinterpret_cast<const cpx<double> *>(src);
    cpx<double> *r = reinterpret_cast<cpx<double> *>(w.r), *q = reinterpret_cast<cpx<double> *>(w.q);
    cpx<double> *t = reinterpret_cast<cpx<double> *>(w.t), *p0 = reinterpret_cast<cpx<double> *>(w.p0);
    cpx<double> *chi = reinterpret_cast<cpx<double> *>(w.x);
    // One pole: its direction at the start of a batch of one is p0 before the
    // step, kept in t, which is free between two applications of D.
    cpx<double> *const keep = np == 1 ? t : nullptr, *const p = np == 1 ? t : reinterpret_cast<cpx<double> *>(w.p);
    const int slots = cg_batch_slots(np);
    CgScalars s;
    const size_t pm = (size_t)np * mp;
    s.rnorm[0] = w.scalars;
    s.rnorm[1] = w.scalars + mp;
    s.bnorm = w.scalars + 2 * mp;
    s.betam = w.scalars + 3 * mp;
    s.alpha0 = w.scalars + 4 * mp;
    s.beta0 = w.scalars + 5 * mp;
    s.z = w.shifts;
    s.g = w.shifts + pm;
    s.cb = w.shifts + 2 * pm;
    s.al = s.cb + kCgBatch * pm;
    s.gg = s.al + kCgBatch * pm;
    s.active = w.flags;
    s.next = w.flags + mp;
    s.iters = w.flags + 2 * mp;
    s.kact = w.flags + 3 * mp;
    s.knext = w.flags + 4 * mp;
    s.steps = w.flags + 5 * mp;
    s.count = w.flags + 6 * mp;
    int *const count = s.count;
    cudaMemcpyAsync(w.dz, co.d, sizeof(double) * np, cudaMemcpyHostToDevice, stream);
    cudaMemcpyAsync(w.bz, co.b, sizeof(double) * np, cudaMemcpyHostToDevice, stream);

    const int chunks = cg_chunks(L, n_mb, sm_count), sq_chunks = cg_square_chunks(L);
    const bool fold = sq_chunks > 2 * kDotChunks;
    double *const rr_part = w.part, *const pap_part = rr_part + (size_t)kDotChunks * mp;
    double *const pap_fold = pap_part + (size_t)sq_chunks * mp;
    const dim3 vblock(kModeBlock, kCgWarps), vgrid(n_mb, chunks);
    // the residual of slot j is r[j]; the iteration of slot 0 starts from the last slot
    mscg_init_vectors_kernel<<<vgrid, vblock, 0, stream>>>(phi, r + (size_t)(slots - 1) * n, p0, p, chi, L.V, n, np, rr_part,
                                                           mp);
    cudaMemsetAsync(count, 0, sizeof(int) * 2, stream);
    cg_init_scalars_kernel<<<n_mb, vblock, 0, stream>>>(s, rr_part, chunks, n_modes, mp, np, co.cg_tol);
    int launches = 2;
    // The count of modes still active is read back one iteration late, while
    // the next iteration is already queued: the GPU does not wait for the host,
    // and the one iteration queued past the end finds no active mode (two
    // stencil passes, no vector changes).
    auto read_count = [&](int slot) {
        cudaMemcpyAsync(w.host_count + slot, count + slot, sizeof(int), cudaMemcpyDeviceToHost, stream);
        cudaEventRecord(w.counted[slot], stream);
    };
    auto counted = [&](int slot) {
        cudaEventSynchronize(w.counted[slot]);
        return w.host_count[slot];
    };
    // a CTA per SM and one wave of them, or four CTAs per mode block where there are more blocks than SMs
    const int shift_ctas = std::max(1, std::min(n_mb > sm_count ? 4 : sm_count / n_mb,
                                                (L.V * kComp + kShiftWarps * kShiftRows - 1) / (kShiftWarps * kShiftRows)));
    cudaFuncSetAttribute(shift_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shift_smem(kShiftStage));
    auto update_shifts = [&]() {
        shift_update_kernel<<<dim3(n_mb, shift_ctas), dim3(kModeBlock, kShiftWarps), shift_smem(np), stream>>>(s, chi, p, r, L.V,
                                                                                                          n, np, mp);
        launches++;
    };
    read_count(0);
    int iterations = 0;
    for (int it = 0;; it++) {
        const int slot = it % slots, par = it & 1;
        cpx<double> *rin = r + (size_t)((slot + slots - 1) % slots) * n, *rout = r + (size_t)slot * n;
        // q = h_W^2 p0 + d0 p0 = -D(D p0) + d0 p0
        s.count = count + (par ^ 1);
        launch_wilson<double>(U, u1, p0, w.t, L, 0, n_mb, amass, 0.0, false, stream);
        launch_cg_square(U, u1, w.t, p0, q, L, n_mb, amass, co.d[0], pap_part, mp, stream);
        if (fold) cg_fold_kernel<<<dim3(n_mb, kDotChunks / kCgWarps), vblock, 0, stream>>>(pap_part, sq_chunks, pap_fold, mp);
        (slots > 1 ? residual_kernel<false> : residual_kernel<true>)<<<vgrid, vblock, 0, stream>>>(
            s, par, fold ? pap_fold : pap_part, fold ? kDotChunks : sq_chunks, rin, rout, q, L.V, rr_part, mp);
        cg_advance_kernel<<<dim3(n_mb, chunks + 1), vblock, 0, stream>>>(s, par, slot, rr_part, chunks, w.dz, w.bz, np,
                                                                         co.cg_tol, co.cg_max_iter, p0, rout, keep, L.V, mp);
        launches += fold ? 5 : 4;
        std::swap(s.active, s.next);
        read_count(par ^ 1);
        const bool over = counted(par) == 0;  // no mode was active before this iteration
        if (!over) iterations++;
        const bool stop = over || iterations > co.cg_max_iter + 1;  // every mode stops by then
        if (slot == slots - 1 || (stop && slot > 0)) update_shifts();
        if (stop) break;
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
        cudaMemcpyAsync(it.data(), s.iters, sizeof(int) * mp, cudaMemcpyDeviceToHost, stream);
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
