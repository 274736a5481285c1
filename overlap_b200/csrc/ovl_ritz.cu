// Extreme eigenvalues of h_W^2 for the overlap operator's spectral bounds:
// OverlapOperations::RitzSolver with one eigenvalue
// (FERMIONS/OVERLAP/OPERATOR/RitzSolver.cpp:91-292), called twice per bound
// computation by Dynamics::Fermions::ComputeRitzEigenvalues
// (FERMIONS/OVERLAP/OverlapUpdate.cpp:61-97): sign = +1 gives the smallest
// eigenvalue, sign = -1 the largest (negated).  The iteration is a
// conjugate-gradient minimisation of the Rayleigh quotient of sign * A,
// A = -D^2 = h_W^2: per step a rotation of x in the plane of (x, p) chosen from
// 2x2 Rayleigh-Ritz, and a new search direction p = g + beta (p - x <x, p>).
//
// Both problems run together, one per blockIdx.y, on vectors in a compact
// layout [problem][site][colour * 4 + spin] (double2): one thread per site;
// NCOMP = 4 Nc components per site (two or three colours).
// Each step is a fixed sequence of kernels; every dot product is reduced per
// CTA into a partial buffer and the next kernel adds the partials in a fixed
// order (every CTA computes bit-identical scalars, so all take the same
// decisions).  Scalars that outlive a kernel sit in RitzScalars; each field is
// written (by CTA 0) in exactly one kernel of a step and read only by later
// kernels.  The partial buffers alternate between two slots so that no kernel
// reads the slot it writes.  A problem that has stopped skips all work.
#include <algorithm>
#include <cmath>

#include <cooperative_groups.h>

#include "ovl_internal.h"
#include "ovl_stencil.cuh"
#include "ovl_su3.cuh"

namespace ovl {

constexpr int kRitzThreads = 128;
constexpr int kRitzParts = 4;  // doubles per CTA partial

struct RitzScalars {
    double xy_re, xy_im;    // Rayleigh quotient <x, y> (restart, residual)
    double oxy_re, oxy_im;  // its value before the rotation (rotate)
    double pnorm;           // |p| before normalisation (normp)
    double gnormim;         // |g|^2 of the previous step (normp)
    double gnorm;           // |g|^2 of this step (direction)
    int ittot;              // steps taken (rotate)
    int done;               // stopped (direction; host at start)
};

struct RitzArgs {
    int nblocks;            // CTAs per problem
    double sign[2];         // problem 0: +1 (lambda_min), problem 1: -1 (-lambda_max)
    double delitr;          // NormRatio
    int max_iter;           // MaximumIterations
};

__device__ __forceinline__ double2 ld2(const double2 *p) { return __ldg(p); }

template <typename T>
__device__ __forceinline__ void load_compact(const double2 *__restrict__ v, int site, Spinor<T> &s) {
    const double2 *p = v + (size_t)site * kComp;
#pragma unroll
    for (int c = 0; c < kColours; c++)
#pragma unroll
        for (int a = 0; a < kSpin; a++) {
            const double2 t = ld2(p + c * kSpin + a);
            s.c[c][a] = mk<T>(t.x, t.y);
        }
}

// Block-wide sum of up to kRitzParts values in a fixed order; thread 0 writes
// them to part[k].
__device__ __forceinline__ void block_partials(double (&v)[kRitzParts], int nv, double *part) {
    __shared__ double sh[kRitzThreads / 32][kRitzParts];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = 0; k < nv; k++) {
        double t = v[k];
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) sh[warp][k] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 0; k < nv; k++) {
            double t = 0.0;
            for (int w = 0; w < kRitzThreads / 32; w++) t += sh[w][k];
            part[k] = t;
        }
    }
}

// Sums the nblocks partials of a problem (k = 0..nv-1) in a fixed order; every
// thread of the CTA gets the same values.
__device__ __forceinline__ void reduce_partials(const double *__restrict__ part, int nblocks, int nv,
                                                double (&out)[kRitzParts]) {
    __shared__ double sh[kRitzParts];
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        for (int k = 0; k < nv; k++) {
            double t = 0.0;
            for (int b = lane; b < nblocks; b += 32) t += part[(size_t)b * kRitzParts + k];
            for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
            if (lane == 0) sh[k] = t;
        }
    }
    __syncthreads();
    for (int k = 0; k < nv; k++) out[k] = sh[k];
    __syncthreads();
}

// Whether a problem has stopped, read once per CTA (thread 0) and shared, so
// that the whole CTA takes the same branch even while CTA 0 of the direction
// kernel sets the flag.
__device__ __forceinline__ bool ritz_stopped(const RitzScalars *st, int prob) {
    __shared__ int flag;
    if (threadIdx.x == 0) flag = *reinterpret_cast<const volatile int *>(&st[prob].done);
    __syncthreads();
    return flag != 0;
}

__device__ __forceinline__ double *part_of(double *base, int slot, int prob, int nblocks) {
    return base + ((size_t)slot * 2 + prob) * nblocks * kRitzParts;
}

// <a, b> = sum conj(a) b over the NCOMP components of one site
template <int NCOMP>
__device__ __forceinline__ void site_dot(const double2 *a, const double2 *b, double &re, double &im) {
#pragma unroll
    for (int k = 0; k < NCOMP; k++) {
        const double2 u = a[k], w = b[k];
        re += u.x * w.x + u.y * w.y;
        im += u.x * w.y - u.y * w.x;
    }
}

// x = start for both problems; partial |x|^2 -> slot 0
template <int NCOMP>
__global__ void __launch_bounds__(kRitzThreads)
    ritz_start_kernel(const double2 *__restrict__ start, double2 *x, int V, RitzArgs a, double *part) {
    const int prob = blockIdx.y, site = blockIdx.x * kRitzThreads + threadIdx.x;
    double v[kRitzParts] = {0.0, 0.0, 0.0, 0.0};
    if (site < V) {
        double2 *xs = x + ((size_t)prob * V + site) * NCOMP;
#pragma unroll
        for (int k = 0; k < NCOMP; k++) {
            const double2 s = start[(size_t)site * NCOMP + k];
            xs[k] = s;
            v[0] += s.x * s.x + s.y * s.y;
        }
    }
    block_partials(v, 1, part_of(part, 0, prob, a.nblocks) + (size_t)blockIdx.x * kRitzParts);
}

// x /= |x| (slot 0)
template <int NCOMP>
__global__ void __launch_bounds__(kRitzThreads)
    ritz_scale_x_kernel(double2 *x, int V, RitzArgs a, double *part) {
    const int prob = blockIdx.y, site = blockIdx.x * kRitzThreads + threadIdx.x;
    double r[kRitzParts];
    reduce_partials(part_of(part, 0, prob, a.nblocks), a.nblocks, 1, r);
    const double s = 1.0 / sqrt(r[0]);
    if (site < V) {
        double2 *xs = x + ((size_t)prob * V + site) * NCOMP;
#pragma unroll
        for (int k = 0; k < NCOMP; k++) xs[k] = make_double2(xs[k].x * s, xs[k].y * s);
    }
}

// SECOND = false: dst = D src.  SECOND = true: dst = -sign D src (= sign A v
// when src = D v) and partials <da, dst> (k = 0, 1) and <db, dst> (k = 2, 3,
// when db is set) -> slot 0.  NC colours: the two-colour stencil of
// ovl_stencil.cuh or the three-colour one of ovl_su3.cuh on the compact layout.
template <int NC, bool U1, bool SECOND, class LK>
__global__ void __launch_bounds__(kRitzThreads)
    ritz_apply_kernel(LK lk, const double2 *__restrict__ src, double2 *__restrict__ dst,
                      const double2 *__restrict__ da, const double2 *__restrict__ db, Lattice L, double amass,
                      const RitzScalars *__restrict__ st, RitzArgs a, double *part) {
    constexpr int NCOMP = 4 * NC;
    const int prob = blockIdx.y, site = blockIdx.x * kRitzThreads + threadIdx.x;
    if (ritz_stopped(st, prob)) return;
    const int V = L.V;
    const size_t off = (size_t)prob * V;
    double v[kRitzParts] = {0.0, 0.0, 0.0, 0.0};
    if (site < V) {
        const double2 *s = src + off * NCOMP;
        const Nbrs n = neighbours(L, site);
        const double scale = SECOND ? -a.sign[prob] : 1.0;
        double2 o[NCOMP];
        if constexpr (NC == 2) {
            Spinor<double> acc, f;
            load_compact(s, site, f);
#pragma unroll
            for (int c = 0; c < kColours; c++)
#pragma unroll
                for (int s2 = 0; s2 < kSpin; s2++) acc.c[c][s2] = amass * f.c[c][s2];
            load_compact(s, n.xp, f);
            hop<double, 0, true>(acc, f, lk.template get<double>(site, 0));
            load_compact(s, n.xm, f);
            hop<double, 0, false>(acc, f, lk.template get<double>(n.xm, 0));
            load_compact(s, n.yp, f);
            hop<double, 1, true>(acc, f, lk.template get<double>(site, 1));
            load_compact(s, n.ym, f);
            hop<double, 1, false>(acc, f, lk.template get<double>(n.ym, 1));
            load_compact(s, n.zp, f);
            hop<double, 2, true>(acc, f, lk.template get<double>(site, 2));
            load_compact(s, n.zm, f);
            hop<double, 2, false>(acc, f, lk.template get<double>(n.zm, 2));
#pragma unroll
            for (int c = 0; c < kColours; c++)
#pragma unroll
                for (int s2 = 0; s2 < kSpin; s2++) {
                    const cpx<double> r = finish_component(acc.c[c][s2], s2);
                    o[c * kSpin + s2] = make_double2(scale * r.re, scale * r.im);
                }
        } else {
            const cpx<double> *f = reinterpret_cast<const cpx<double> *>(s);
            Spinor3<double> acc;
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int s2 = 0; s2 < kSpin; s2++) acc.c[c][s2] = amass * ld(f + (size_t)site * NCOMP + c * kSpin + s2);
            hop3<double, 0, true, false, 1>(acc, f + (size_t)n.xp * NCOMP, lk.template get<double>(site, 0));
            hop3<double, 0, false, false, 1>(acc, f + (size_t)n.xm * NCOMP, lk.template get<double>(n.xm, 0));
            hop3<double, 1, true, false, 1>(acc, f + (size_t)n.yp * NCOMP, lk.template get<double>(site, 1));
            hop3<double, 1, false, false, 1>(acc, f + (size_t)n.ym * NCOMP, lk.template get<double>(n.ym, 1));
            hop3<double, 2, true, false, 1>(acc, f + (size_t)n.zp * NCOMP, lk.template get<double>(site, 2));
            hop3<double, 2, false, false, 1>(acc, f + (size_t)n.zm * NCOMP, lk.template get<double>(n.zm, 2));
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int s2 = 0; s2 < kSpin; s2++) {
                    const cpx<double> r = finish_component(acc.c[c][s2], s2);
                    o[c * kSpin + s2] = make_double2(scale * r.re, scale * r.im);
                }
        }
        double2 *d = dst + (off + site) * NCOMP;
#pragma unroll
        for (int k = 0; k < NCOMP; k++) d[k] = o[k];
        if (SECOND) {
            site_dot<NCOMP>(da + (off + site) * NCOMP, o, v[0], v[1]);
            if (db) site_dot<NCOMP>(db + (off + site) * NCOMP, o, v[2], v[3]);
        }
    }
    if (SECOND) block_partials(v, 4, part_of(part, 0, prob, a.nblocks) + (size_t)blockIdx.x * kRitzParts);
}

// Restart (RitzSolver.cpp:138-166): xy = <x, y>; g = p = y - xy x; |g|^2 -> slot 1.
template <int NCOMP>
__global__ void __launch_bounds__(kRitzThreads)
    ritz_restart_kernel(const double2 *__restrict__ x, const double2 *__restrict__ y, double2 *__restrict__ g,
                        double2 *__restrict__ praw, int V, RitzScalars *st, RitzArgs a, double *part) {
    const int prob = blockIdx.y, site = blockIdx.x * kRitzThreads + threadIdx.x;
    if (ritz_stopped(st, prob)) return;
    double r[kRitzParts];
    reduce_partials(part_of(part, 0, prob, a.nblocks), a.nblocks, 2, r);
    const double xr = r[0], xi = r[1];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st[prob].xy_re = xr;
        st[prob].xy_im = xi;
    }
    double v[kRitzParts] = {0.0, 0.0, 0.0, 0.0};
    if (site < V) {
        const size_t o = ((size_t)prob * V + site) * NCOMP;
#pragma unroll
        for (int k = 0; k < NCOMP; k++) {
            const double2 xv = x[o + k], yv = y[o + k];
            const double2 gv = make_double2(yv.x - (xr * xv.x - xi * xv.y), yv.y - (xr * xv.y + xi * xv.x));
            g[o + k] = gv;
            praw[o + k] = gv;
            v[0] += gv.x * gv.x + gv.y * gv.y;
        }
    }
    block_partials(v, 1, part_of(part, 1, prob, a.nblocks) + (size_t)blockIdx.x * kRitzParts);
}

// p = praw / |praw| (slot 1); pnorm; gnormim = |praw|^2 on a restart (p = g
// there), else the gnorm of this step.
template <int NCOMP>
__global__ void __launch_bounds__(kRitzThreads)
    ritz_normp_kernel(const double2 *__restrict__ praw, double2 *__restrict__ p, int V, int restart, RitzScalars *st,
                      RitzArgs a, const double *part) {
    const int prob = blockIdx.y, site = blockIdx.x * kRitzThreads + threadIdx.x;
    if (ritz_stopped(st, prob)) return;
    double r[kRitzParts];
    reduce_partials(part_of(const_cast<double *>(part), 1, prob, a.nblocks), a.nblocks, 1, r);
    const double pn = sqrt(r[0]);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st[prob].pnorm = pn;
        st[prob].gnormim = restart ? r[0] : st[prob].gnorm;
    }
    if (site < V) {
        const size_t o = ((size_t)prob * V + site) * NCOMP;
#pragma unroll
        for (int k = 0; k < NCOMP; k++) p[o + k] = make_double2(praw[o + k].x / pn, praw[o + k].y / pn);
    }
}

// cos and sin of the rotation of x in the (x, p) plane from amb = Re(xy - Re
// <p, z>) and ccc = Re <x, z> (RitzSolver.cpp:176-222).
__device__ __forceinline__ void ritz_rotation(double amb, double ccc, double &ct, double &sn) {
    const double cox = 2.0 * ccc / amb;
    const double sig1 = -copysign(1.0, amb);
    const double sig2 = copysign(1.0, cox) * sig1;
    const double c2 = cox * cox;
    if (c2 <= 1.0e-3) {
        // the reference's series for the rotation, constants as there (:197-200)
        const double sqp = 1.0 - 0.125 * c2 + 0.0859375 * c2 * c2 - 0.0673828125 * c2 * c2 * c2 +
                           0.0562439 * c2 * c2 * c2 * c2 + 0.0487 * c2 * c2 * c2 * c2 * c2;
        const double sqm = 0.5 * sig1 * sig2 * cox *
                           (1.0 - 0.375 * c2 + 0.2421875 * c2 * c2 - 0.182617875 * c2 * c2 * c2 +
                            0.1482849 * c2 * c2 * c2 * c2 - 0.12575 * c2 * c2 * c2 * c2 * c2 +
                            0.1097 * c2 * c2 * c2 * c2 * c2 * c2);
        if (sig1 < 0.0) {
            ct = sqm;
            sn = sig2 * sqp;
        } else {
            ct = sqp;
            sn = sig2 * sqm;
        }
    } else {
        const double sox = sig1 / sqrt(1.0 + c2);
        ct = sqrt((1.0 + sox) * 0.5);
        sn = sqrt((1.0 - sox) * 0.5) * sig2;
    }
}

// The rotation of x in the (x, p) plane (RitzSolver.cpp:176-222), from slot 0:
// pz = Re <p, z>, xz = Re <x, z>.  Then <x, x>, <x, y> -> slot 1.
template <int NCOMP>
__global__ void __launch_bounds__(kRitzThreads)
    ritz_rotate_kernel(double2 *x, double2 *y, const double2 *__restrict__ p, const double2 *__restrict__ z, int V,
                       RitzScalars *st, RitzArgs a, double *part) {
    const int prob = blockIdx.y, site = blockIdx.x * kRitzThreads + threadIdx.x;
    if (ritz_stopped(st, prob)) return;
    double r[kRitzParts];
    reduce_partials(part_of(part, 0, prob, a.nblocks), a.nblocks, 4, r);
    const double pz = r[0], ccc = r[2];
    const double xy_re = st[prob].xy_re, xy_im = st[prob].xy_im;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st[prob].oxy_re = xy_re;
        st[prob].oxy_im = xy_im;
        st[prob].ittot += 1;
    }
    double ct, sn;
    ritz_rotation(xy_re - pz, ccc, ct, sn);
    double v[kRitzParts] = {0.0, 0.0, 0.0, 0.0};
    if (site < V) {
        const size_t o = ((size_t)prob * V + site) * NCOMP;
        double2 xn[NCOMP], yn[NCOMP];
#pragma unroll
        for (int k = 0; k < NCOMP; k++) {
            const double2 xv = x[o + k], pv = p[o + k], yv = y[o + k], zv = z[o + k];
            xn[k] = make_double2(xv.x * ct + pv.x * sn, xv.y * ct + pv.y * sn);
            yn[k] = make_double2(yv.x * ct + zv.x * sn, yv.y * ct + zv.y * sn);
            x[o + k] = xn[k];
            y[o + k] = yn[k];
        }
        double im0 = 0.0;
        site_dot<NCOMP>(xn, xn, v[0], im0);
        site_dot<NCOMP>(xn, yn, v[1], v[2]);
    }
    block_partials(v, 3, part_of(part, 1, prob, a.nblocks) + (size_t)blockIdx.x * kRitzParts);
}

// x normalised, xy = <x, y> / |x|, g = y - xy x (RitzSolver.cpp:224-243), from
// slot 1.  Then |g|^2, <x, p> -> slot 0.
template <int NCOMP>
__global__ void __launch_bounds__(kRitzThreads)
    ritz_residual_kernel(double2 *x, const double2 *__restrict__ y, double2 *__restrict__ g,
                         const double2 *__restrict__ p, int V, RitzScalars *st, RitzArgs a, double *part) {
    const int prob = blockIdx.y, site = blockIdx.x * kRitzThreads + threadIdx.x;
    if (ritz_stopped(st, prob)) return;
    double r[kRitzParts];
    reduce_partials(part_of(part, 1, prob, a.nblocks), a.nblocks, 3, r);
    const double xnorm = 1.0 / sqrt(r[0]);
    const double xr = r[1] * xnorm, xi = r[2] * xnorm;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st[prob].xy_re = xr;
        st[prob].xy_im = xi;
    }
    double v[kRitzParts] = {0.0, 0.0, 0.0, 0.0};
    if (site < V) {
        const size_t o = ((size_t)prob * V + site) * NCOMP;
        double2 xn[NCOMP], gn[NCOMP];
#pragma unroll
        for (int k = 0; k < NCOMP; k++) {
            const double2 xv = x[o + k], yv = y[o + k];
            xn[k] = make_double2(xv.x * xnorm, xv.y * xnorm);
            gn[k] = make_double2(yv.x - (xr * xn[k].x - xi * xn[k].y), yv.y - (xr * xn[k].y + xi * xn[k].x));
            x[o + k] = xn[k];
            g[o + k] = gn[k];
        }
        double im0 = 0.0;
        site_dot<NCOMP>(gn, gn, v[0], im0);
        site_dot<NCOMP>(xn, p + o, v[1], v[2]);
    }
    block_partials(v, 3, part_of(part, 0, prob, a.nblocks) + (size_t)blockIdx.x * kRitzParts);
}

// Stopping tests and the new search direction (RitzSolver.cpp:245-284), from
// slot 0: gnorm = |g|^2, xp = <x, p>.  praw = g + beta (p - x xp); |praw|^2 -> slot 1.
template <int NCOMP>
__global__ void __launch_bounds__(kRitzThreads)
    ritz_direction_kernel(const double2 *__restrict__ x, const double2 *__restrict__ g, const double2 *__restrict__ p,
                          double2 *__restrict__ praw, int V, RitzScalars *st, RitzArgs a, double *part) {
    const int prob = blockIdx.y, site = blockIdx.x * kRitzThreads + threadIdx.x;
    if (ritz_stopped(st, prob)) return;
    double r[kRitzParts];
    reduce_partials(part_of(part, 0, prob, a.nblocks), a.nblocks, 3, r);
    const double gnorm = r[0], xpr = r[1], xpi = r[2];
    // fields not written by this kernel (gnorm and done are: CTA 0 below)
    const double xy_re = st[prob].xy_re, oxy_re = st[prob].oxy_re;
    const double gnormim = st[prob].gnormim, pnorm = st[prob].pnorm;
    const int ittot = st[prob].ittot;
    bool stop = xy_re > oxy_re || gnorm < a.delitr * a.sign[prob] * xy_re;
    const double beta = gnorm / gnormim * pnorm;
    double v[kRitzParts] = {0.0, 0.0, 0.0, 0.0};
    if (!stop && site < V) {
        const size_t o = ((size_t)prob * V + site) * NCOMP;
#pragma unroll
        for (int k = 0; k < NCOMP; k++) {
            const double2 xv = x[o + k], gv = g[o + k], pv = p[o + k];
            const double2 xxp = make_double2(xv.x * xpr - xv.y * xpi, xv.x * xpi + xv.y * xpr);
            const double2 pn = make_double2(gv.x + beta * (pv.x - xxp.x), gv.y + beta * (pv.y - xxp.y));
            praw[o + k] = pn;
            v[0] += pn.x * pn.x + pn.y * pn.y;
        }
    }
    if (!stop && ittot >= a.max_iter) stop = true;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st[prob].gnorm = gnorm;
        if (stop) st[prob].done = 1;
    }
    block_partials(v, 1, part_of(part, 1, prob, a.nblocks) + (size_t)blockIdx.x * kRitzParts);
}

// ------------------------------------------------- one launch per solve --
// The whole two-colour iteration in one launch.  The kernels above take a step
// in six launches of a few CTAs each, and at the sizes of the spectral bounds a
// launch is all latency (8^3: 37 us per step, 6.3 us per kernel).  Here two
// threads own a site, half h the spins h and 3 - h of both colours, and keep x,
// y = A x, p, z = A p and g of it in registers for the whole solve; only the
// vectors the stencil reads from neighbours (v: the raw direction, or x at a
// restart; t = D p) are exchanged.  A step is five phases, each ending in a
// barrier of the problem's CTAs that also delivers the phase's sums: t = D p;
// z = -s D t; the rotation; the residual; the new direction (normalised on the
// way into the next step).  The arithmetic is that of the kernels above, except
// that D is applied to the raw direction and its result scaled.
//
// Two ways to exchange and to meet:
//   RitzCluster  a problem is one thread-block cluster: v and t in distributed
//                shared memory, the hardware's cluster barrier (up to
//                16 CTAs x 128 sites)
//   RitzGrid     a cooperative launch: v and t in global memory, a counter per
//                problem.  The CTAs wait for one another, so all are resident
//                and every wait is bounded (1 s of %globaltimer): on expiry the
//                error word is set, every CTA leaves at its next wait, and the
//                host solves again with the kernels above, which wait for
//                nothing (the second also passes while the GPU runs another
//                process's work, so an expired wait is not yet a failed solve).
// One overlap leapfrog step with its two pairs of bounds at 8^3, 256 modes:
// 91 ms with six launches per Ritz step, 50 ms with the cooperative launch; then,
// the CG made faster, 42.9 ms with the cooperative launch and 30.8 ms with
// clusters (8 CTAs of 64 sites per problem).
constexpr int kRitzTabStride = 50;  // doubles per site of the link table: 6 x 8 and 2 to spread the banks
constexpr int kRitzGridSites = 32;  // sites per CTA of the cooperative launch

struct RitzOne {
    const double2 *start;  // [V][8]
    RitzScalars *st;
    double amass, delitr;
    int max_iter, nrestart;
    int sites;             // per CTA
    // RitzGrid
    double2 *v, *t;        // [problem][8][V]
    double *part;          // [2 slots][problem][CTAs][kRitzParts]
    int *count, *err;      // arrivals per problem; error word
};

using RitzHalf = cpx<double>[2][2];  // [colour][upper, lower component of the half]

// Component (colour c, upper 0 / lower 1) of half h: spin h or 3 - h.
__device__ __forceinline__ int ritz_comp(int c, int lower, int h) { return c * kSpin + (lower ? 3 - h : h); }

// The warps' sums of nv values in sh (lane 0 of each writes); a barrier of the
// CTA has to follow before they are read.
template <int WARPS>
__device__ __forceinline__ void ritz_warp_sums(int nv, const double (&v)[kRitzParts], double (*sh)[kRitzParts]) {
    for (int k = 0; k < nv; k++) {
        double t = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5][k] = t;
    }
}

// One thread waits for the count, polling without a pause (the phases are a
// few hundred nanoseconds apart); bounded as wait_count.
__device__ __forceinline__ bool ritz_wait(const int *counter, int target, int *err) {
    if (ld_acquire(counter) >= target) return true;
    const unsigned long long t0 = global_ns();
    for (long long polls = 1; ld_acquire(counter) < target; polls++) {
        if ((polls & 255) == 0 &&
            (polls > kWaitPolls || (long long)(global_ns() - t0) > kWaitNs || *(volatile int *)err)) {
            atomicExch(err, 1);
            return false;
        }
    }
    return true;
}

struct RitzGrid {
    double2 *vec[2];  // v, t of this problem
    int V, site, nb[6];
    bool live;
    double *part;     // this problem's partials of slot 0; slot 1 at + slot_stride
    size_t slot_stride;
    int *count, *err;
    int nblocks, phase;
    static constexpr int kWarps = 2 * kRitzGridSites / 32;

    __device__ __forceinline__ RitzGrid(const RitzOne &a, const Lattice &L, int site_, bool live_, const int (&n)[6])
        : V(L.V), site(site_), live(live_) {
        const int prob = blockIdx.y;
        vec[0] = a.v + (size_t)prob * kComp * V;
        vec[1] = a.t + (size_t)prob * kComp * V;
        for (int d = 0; d < 6; d++) nb[d] = n[d];
        nblocks = gridDim.x;
        slot_stride = (size_t)2 * gridDim.x * kRitzParts;
        part = a.part + (size_t)prob * gridDim.x * kRitzParts;
        count = a.count + prob;
        err = a.err;
        phase = 0;
    }
    __device__ __forceinline__ void put(int which, int comp, double re, double im) {
        if (live) __stcg(vec[which] + (size_t)comp * V + site, make_double2(re, im));
    }
    __device__ __forceinline__ cpx<double> get(int which, int dir, int comp) const {
        const double2 u = __ldcg(vec[which] + (size_t)comp * V + nb[dir]);
        return mk<double>(u.x, u.y);
    }
    // Sums nv values over the problem's CTAs (in the order of the CTAs; every
    // thread gets the same totals) behind a barrier of them: what the CTAs wrote
    // before it is visible after it.  False when a wait ran out.
    __device__ __forceinline__ bool sum(int nv, const double (&v)[kRitzParts], double (&out)[kRitzParts]) {
        __shared__ double sh[kWarps][kRitzParts], tot[kRitzParts];
        __shared__ int ok;
        const int lane = threadIdx.x & 31;
        ritz_warp_sums<kWarps>(nv, v, sh);
        __syncthreads();
        double *slot = part + (phase & 1) * slot_stride;
        phase++;
        if (threadIdx.x == 0) {
            for (int k = 0; k < nv; k++) {
                double t = 0.0;
                for (int w = 0; w < kWarps; w++) t += sh[w][k];
                __stcg(slot + (size_t)blockIdx.x * kRitzParts + k, t);
            }
            red_release_add(count, 1);
            ok = ritz_wait(count, nblocks * phase, err) ? 1 : 0;
        }
        __syncthreads();
        if (!ok) return false;
        if (nv > 0) {
            if (threadIdx.x < 32) {
                double t[kRitzParts] = {0.0, 0.0, 0.0, 0.0};
                for (int i = lane; i < nblocks; i += 32)
                    for (int k = 0; k < nv; k++) t[k] += __ldcg(slot + (size_t)i * kRitzParts + k);
                for (int k = 0; k < nv; k++) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
                    if (lane == 0) tot[k] = t[k];
                }
            }
            __syncthreads();
            for (int k = 0; k < nv; k++) out[k] = tot[k];
        }
        __syncthreads();  // sh, tot and ok are reused by the next phase
        return true;
    }
    __device__ __forceinline__ void finish() {}
};

// The cluster's CTAs hold `sites` consecutive sites each; dynamic shared memory:
// v [8][sites], t [8][sites], then the link table.
constexpr int kRitzClusterMax = 16;                                 // CTAs per cluster, at most
constexpr int kRitzClusterThreads = 256;                            // at most: 255 registers a thread
constexpr size_t ritz_cluster_smem(int sites) {
    return (sizeof(double2) * 2 * kComp + sizeof(double) * kRitzTabStride) * (size_t)sites;
}

struct RitzCluster {
    double2 *own;      // v of this CTA's sites, at this thread's site
    double2 *at[6];    // v of the neighbours (distributed shared memory)
    int sites, nranks, phase;
    static constexpr int kWarps = kRitzClusterThreads / 32;

    __device__ __forceinline__ RitzCluster(const RitzOne &a, double2 *smem, int sl, const int (&n)[6])
        : own(smem + sl), sites(a.sites), phase(0) {
        cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        nranks = (int)cl.num_blocks();
        for (int d = 0; d < 6; d++) at[d] = cl.map_shared_rank(smem, n[d] / sites) + n[d] % sites;
        cl.sync();  // every CTA has started before its memory is written
    }
    __device__ __forceinline__ void put(int which, int comp, double re, double im) {
        own[(size_t)(which * kComp + comp) * sites] = make_double2(re, im);
    }
    __device__ __forceinline__ cpx<double> get(int which, int dir, int comp) const {
        const double2 u = at[dir][(size_t)(which * kComp + comp) * sites];
        return mk<double>(u.x, u.y);
    }
    __device__ __forceinline__ bool sum(int nv, const double (&v)[kRitzParts], double (&out)[kRitzParts]) {
        __shared__ double sh[kWarps][kRitzParts], all[2][kRitzClusterMax][kRitzParts];
        cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
        const int par = phase & 1;
        phase++;
        if (nv > 0) {
            ritz_warp_sums<kWarps>(nv, v, sh);
            __syncthreads();
            // this CTA's sums into every CTA's table
            for (int i = threadIdx.x; i < nranks * nv; i += blockDim.x) {
                const int k = i % nv;
                double t = 0.0;
                for (int w = 0; w < (int)blockDim.x / 32; w++) t += sh[w][k];
                cl.map_shared_rank(&all[0][0][0], i / nv)[(par * kRitzClusterMax + (int)cl.block_rank()) * kRitzParts + k] = t;
            }
        }
        cl.sync();
        for (int k = 0; k < nv; k++) {
            double t = 0.0;
            for (int r = 0; r < nranks; r++) t += all[par][r][k];
            out[k] = t;
        }
        return true;
    }
    __device__ __forceinline__ void finish() { cooperative_groups::this_cluster().sync(); }  // no CTA leaves while its memory is read
};

// The half spinor of D w at the thread's site: own[c][0] spin h, own[c][1]
// spin 3 - h of w there; the neighbours' components through x (vector `which`).
// The projections and reconstruction of hop() (ovl_stencil.cuh), half by half:
// h0 and its products belong to half 0, h1 to half 1; in the z hops the lower
// component rebuilt from one half's product belongs to the other half.
template <class X>
__device__ __forceinline__ void ritz_half_d(const X &x, int which, const double *tab, int h, double amass,
                                            const RitzHalf &own, RitzHalf &out) {
    const double sg = h ? -1.0 : 1.0;
    RitzHalf acc;
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
        for (int k = 0; k < 2; k++) acc[c][k] = amass * own[c][k];
    auto link = [&](int dir) {
        const double2 *q = reinterpret_cast<const double2 *>(tab + 8 * dir);
        const double2 a = q[0], b = q[1], c = q[2], d = q[3];
        return cmat2<double>{{a.x, a.y}, {b.x, b.y}, {c.x, c.y}, {d.x, d.y}};
    };
#pragma unroll
    for (int dir = 0; dir < 6; dir++) {  // +x, +y, +z, -x, -y, -z as in the link table
        const int mu = dir % 3;
        const bool fwd = dir < 3;
        const double s = fwd ? 1.0 : -1.0;
        cpx<double> hh[2], k[2];
#pragma unroll
        for (int c = 0; c < 2; c++) {
            const cpx<double> up = x.get(which, dir, c * kSpin + h);
            const cpx<double> lo = x.get(which, dir, c * kSpin + (mu == 2 ? 2 + h : 3 - h));
            if (mu == 0) hh[c] = mk<double>(fma(-s, lo.im, up.re), fma(s, lo.re, up.im));              // p_h +- i p_{3-h}
            else if (mu == 1) hh[c] = mk<double>(fma(s * sg, lo.re, up.re), fma(s * sg, lo.im, up.im));  // p_h +- sg p_{3-h}
            else hh[c] = mk<double>(fma(-s * sg, lo.im, up.re), fma(s * sg, lo.re, up.im));            // p_h +- sg i p_{2+h}
        }
        const cmat2<double> M = link(dir);
        if (fwd) mul(M, hh[0], hh[1], k[0], k[1]);
        else mul_dag(M, hh[0], hh[1], k[0], k[1]);
#pragma unroll
        for (int c = 0; c < 2; c++) {
            acc[c][0] = acc[c][0] - k[c];
            if (mu == 0) {  // lower -= -+ i k
                acc[c][1] = acc[c][1] - s * times_mi(k[c]);
            } else if (mu == 1) {  // lower -= +- sg k
                acc[c][1] = acc[c][1] - (s * sg) * k[c];
            } else {  // the other half's product: lower -= +- sg i k'
                const cpx<double> o = mk<double>(__shfl_xor_sync(0xffffffffu, k[c].re, 1), __shfl_xor_sync(0xffffffffu, k[c].im, 1));
                acc[c][1] = acc[c][1] - (s * sg) * times_i(o);
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 2; c++) {  // -i gamma_0 / 2
        out[c][0] = 0.5 * times_mi(acc[c][0]);
        out[c][1] = 0.5 * times_i(acc[c][1]);
    }
}

// The CTA's link table: the six dressed links of each of its sites' hops.
template <bool U1>
__device__ __forceinline__ void ritz_fill_links(const LinksF64<U1> &lk, const Lattice &L, int site0, int sites, double *tab) {
    for (int i = threadIdx.x; i < sites * 6; i += blockDim.x) {
        const int s = site0 + i / 6, dir = i % 6, mu = dir % 3;
        if (s >= L.V) continue;
        int ls = s;
        if (dir >= 3) {
            const Nbrs n = neighbours(L, s);
            ls = mu == 0 ? n.xm : (mu == 1 ? n.ym : n.zm);
        }
        const cmat2<double> M = lk.template get<double>(ls, mu);
        double2 *o = reinterpret_cast<double2 *>(tab + (i / 6) * kRitzTabStride + 8 * dir);
        o[0] = make_double2(M.m00.re, M.m00.im);
        o[1] = make_double2(M.m01.re, M.m01.im);
        o[2] = make_double2(M.m10.re, M.m10.im);
        o[3] = make_double2(M.m11.re, M.m11.im);
    }
    __syncthreads();
}

// The iteration; x exchanges and sums.  A padded pair (live false) computes on
// some site and adds nothing.
template <class X>
__device__ __forceinline__ void ritz_solve(X &ex, const RitzOne &a, const double *tab, int site, int h, bool live) {
    const int prob = blockIdx.y;
    const double sign = prob == 0 ? 1.0 : -1.0;
    auto store = [&](int which, const RitzHalf &f) {
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
            for (int k = 0; k < 2; k++) ex.put(which, ritz_comp(c, k, h), f[c][k].re, f[c][k].im);
    };
    auto dot = [&](const RitzHalf &u, const RitzHalf &w, double &re, double &im) {
        if (!live) return;
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
            for (int k = 0; k < 2; k++) {
                re += u[c][k].re * w[c][k].re + u[c][k].im * w[c][k].im;
                im += u[c][k].re * w[c][k].im - u[c][k].im * w[c][k].re;
            }
    };
#define OVL_RITZ_EACH for (int c = 0; c < 2; c++) for (int k = 0; k < 2; k++)
    RitzHalf x, y, p, z, g, raw;
    double s[kRitzParts], r[kRitzParts];
    auto clear = [&]() { s[0] = s[1] = s[2] = s[3] = 0.0; };
    // x = start / |start|
#pragma unroll
    OVL_RITZ_EACH {
        const double2 u = a.start[(size_t)site * kComp + ritz_comp(c, k, h)];
        x[c][k] = mk<double>(u.x, u.y);
        y[c][k] = p[c][k] = z[c][k] = g[c][k] = raw[c][k] = mk<double>(0.0, 0.0);
    }
    clear();
    dot(x, x, s[0], s[3]);
    if (!ex.sum(1, s, r)) return;
    {
        const double inv = 1.0 / sqrt(r[0]);
#pragma unroll
        OVL_RITZ_EACH x[c][k] = inv * x[c][k];
    }
    double xy_re = 0.0, xy_im = 0.0, gnorm = 0.0, raw2 = 0.0;
    int ittot = 0;
    bool stop = false;
    while (!stop) {
        // restart (RitzSolver.cpp:138-166): y = s A x, xy = <x, y>, g = raw direction = y - xy x
        store(0, x);
        if (!ex.sum(0, s, r)) return;
        RitzHalf w;
        ritz_half_d(ex, 0, tab, h, a.amass, x, w);
        store(1, w);
        if (!ex.sum(0, s, r)) return;
        ritz_half_d(ex, 1, tab, h, a.amass, w, y);
#pragma unroll
        OVL_RITZ_EACH y[c][k] = (-sign) * y[c][k];
        clear();
        dot(x, y, s[0], s[1]);
        if (!ex.sum(2, s, r)) return;
        xy_re = r[0];
        xy_im = r[1];
        clear();
#pragma unroll
        OVL_RITZ_EACH {
            g[c][k] = mk<double>(y[c][k].re - (xy_re * x[c][k].re - xy_im * x[c][k].im),
                                 y[c][k].im - (xy_re * x[c][k].im + xy_im * x[c][k].re));
            raw[c][k] = g[c][k];
        }
        dot(g, g, s[0], s[3]);
        store(0, raw);
        if (!ex.sum(1, s, r)) return;
        raw2 = r[0];
        double gnormim = raw2;
        for (int itt = 1; itt <= a.nrestart && !stop; itt++) {
            // p = raw / |raw|; t = D p
            const double pnorm = sqrt(raw2), inv = 1.0 / pnorm;
#pragma unroll
            OVL_RITZ_EACH p[c][k] = mk<double>(raw[c][k].re / pnorm, raw[c][k].im / pnorm);
            ritz_half_d(ex, 0, tab, h, a.amass, raw, w);
#pragma unroll
            OVL_RITZ_EACH w[c][k] = inv * w[c][k];
            store(1, w);
            if (!ex.sum(0, s, r)) return;
            // z = s A p; <p, z>, <x, z>
            ritz_half_d(ex, 1, tab, h, a.amass, w, z);
#pragma unroll
            OVL_RITZ_EACH z[c][k] = (-sign) * z[c][k];
            clear();
            dot(p, z, s[0], s[1]);
            dot(x, z, s[2], s[3]);
            if (!ex.sum(4, s, r)) return;
            // the rotation in the (x, p) plane (RitzSolver.cpp:176-222)
            const double oxy_re = xy_re;
            double ct, sn;
            ritz_rotation(xy_re - r[0], r[2], ct, sn);
            ittot++;
#pragma unroll
            OVL_RITZ_EACH {
                x[c][k] = mk<double>(x[c][k].re * ct + p[c][k].re * sn, x[c][k].im * ct + p[c][k].im * sn);
                y[c][k] = mk<double>(y[c][k].re * ct + z[c][k].re * sn, y[c][k].im * ct + z[c][k].im * sn);
            }
            clear();
            dot(x, x, s[0], s[3]);
            dot(x, y, s[1], s[2]);
            if (!ex.sum(3, s, r)) return;
            // x normalised, xy, g (RitzSolver.cpp:224-243)
            const double xnorm = 1.0 / sqrt(r[0]);
            xy_re = r[1] * xnorm;
            xy_im = r[2] * xnorm;
            clear();
#pragma unroll
            OVL_RITZ_EACH {
                x[c][k] = xnorm * x[c][k];
                g[c][k] = mk<double>(y[c][k].re - (xy_re * x[c][k].re - xy_im * x[c][k].im),
                                     y[c][k].im - (xy_re * x[c][k].im + xy_im * x[c][k].re));
            }
            dot(g, g, s[0], s[3]);
            s[3] = 0.0;
            dot(x, p, s[1], s[2]);
            if (!ex.sum(3, s, r)) return;
            // stopping tests and the new direction (RitzSolver.cpp:245-284)
            gnorm = r[0];
            const double xpr = r[1], xpi = r[2];
            stop = xy_re > oxy_re || gnorm < a.delitr * sign * xy_re || ittot >= a.max_iter;
            if (stop) break;
            const double beta = gnorm / gnormim * pnorm;
            clear();
#pragma unroll
            OVL_RITZ_EACH {
                const cpx<double> xxp = mk<double>(x[c][k].re * xpr - x[c][k].im * xpi, x[c][k].re * xpi + x[c][k].im * xpr);
                raw[c][k] = mk<double>(g[c][k].re + beta * (p[c][k].re - xxp.re), g[c][k].im + beta * (p[c][k].im - xxp.im));
            }
            dot(raw, raw, s[0], s[3]);
            store(0, raw);
            if (!ex.sum(1, s, r)) return;
            raw2 = r[0];
            gnormim = gnorm;
        }
    }
#undef OVL_RITZ_EACH
    ex.finish();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.st[prob].xy_re = xy_re;
        a.st[prob].xy_im = xy_im;
        a.st[prob].ittot = ittot;
        a.st[prob].done = 1;
    }
}

template <bool U1>
__global__ void __launch_bounds__(2 * kRitzGridSites) ritz_grid_kernel(LinksF64<U1> lk, Lattice L, RitzOne a) {
    __shared__ double tab[kRitzGridSites * kRitzTabStride];
    const int sl = threadIdx.x >> 1, h = threadIdx.x & 1, want = blockIdx.x * kRitzGridSites + sl;
    const bool live = want < L.V;
    const int site = live ? want : 0;  // a padded pair repeats site 0
    ritz_fill_links(lk, L, blockIdx.x * kRitzGridSites, kRitzGridSites, tab);
    const Nbrs n = neighbours(L, site);
    const int nb[6] = {n.xp, n.yp, n.zp, n.xm, n.ym, n.zm};
    RitzGrid ex(a, L, site, live, nb);
    ritz_solve(ex, a, tab + (live ? sl : 0) * kRitzTabStride, site, h, live);
}

template <bool U1>
__global__ void __launch_bounds__(kRitzClusterThreads) ritz_cluster_kernel(LinksF64<U1> lk, Lattice L, RitzOne a) {
    extern __shared__ double2 smem[];
    double *tab = reinterpret_cast<double *>(smem + (size_t)2 * kComp * a.sites);
    const int sl = threadIdx.x >> 1, h = threadIdx.x & 1, want = blockIdx.x * a.sites + sl;
    const bool live = want < L.V;
    const int site = live ? want : 0;  // a padded pair computes on site 0's neighbours and stores to its own slot
    for (int i = threadIdx.x; i < a.sites * kRitzTabStride; i += blockDim.x) tab[i] = 0.0;  // no link for padded sites
    __syncthreads();
    ritz_fill_links(lk, L, blockIdx.x * a.sites, a.sites, tab);
    const Nbrs n = neighbours(L, site);
    const int nb[6] = {n.xp, n.yp, n.zp, n.xm, n.ym, n.zm};
    RitzCluster ex(a, smem, sl, nb);
    ritz_solve(ex, a, tab + sl * kRitzTabStride, site, h, live);
}

// Start vector with the reference's distribution (Re, Im uniform in [0, 1),
// OverlapUpdate.cpp:69-84) from a counter-based generator: SplitMix64
// (Steele, Lea and Flood, "Fast splittable pseudorandom number generators",
// OOPSLA 2014) of (seed, call, index); the top 53 bits give the uniform.
__device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

__global__ void ritz_random_start_kernel(double2 *start, size_t n, uint64_t seed, uint64_t call) {
    const uint64_t key = splitmix64(seed ^ splitmix64(call));
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const uint64_t a = splitmix64(key + 2 * i), b = splitmix64(key + 2 * i + 1);
        start[i] = make_double2((double)(a >> 11) * 0x1.0p-53, (double)(b >> 11) * 0x1.0p-53);
    }
}

// ---------------------------------------------------------------- host side --

// The iteration between two reads of the stop flags (kRitzPoll steps, with or
// without the restart that opens a cycle of nrestart steps) captured once as
// CUDA graphs and replayed; recaptured when an argument they bake in changes.
constexpr int kRitzPoll = 25;

struct RitzGraphs {
    cudaGraphExec_t restart = nullptr, plain = nullptr;
    const double *U = nullptr, *u1 = nullptr;
    int N[3] = {0, 0, 0};
    double amass = 0.0, delitr = 0.0;
    int max_iter = 0;
    bool failed = false;  // capture not possible on this stream: step the loop instead
    void release() {
        if (restart) cudaGraphExecDestroy(restart);
        if (plain) cudaGraphExecDestroy(plain);
        restart = plain = nullptr;
    }
};

// How a lattice of V sites is solved: by clusters of `ranks` CTAs of `sites`
// sites (ranks > 0), by the cooperative launch (grid), or kernel by kernel.
struct RitzPlan {
    int ranks = 0, sites = 0;
    size_t smem = 0;
    bool grid = false;
};

struct RitzWork {
    double2 *x = nullptr, *y = nullptr, *z = nullptr, *t = nullptr, *p = nullptr, *praw = nullptr, *g = nullptr;
    double2 *start = nullptr;
    double *part = nullptr;
    int *count = nullptr;         // one-launch solve: arrivals of the two problems, error word
    RitzScalars *st = nullptr;
    RitzScalars *host = nullptr;  // pinned, two and the error word
    int V = 0;
    int nc = 2;  // colours: vectors of 4 nc components per site
    RitzGraphs graphs;
    RitzPlan plan[2];             // without and with a U(1) background
    bool planned[2] = {false, false};
};

void *ritz_create(int V, int nc) {
    RitzWork *w = new RitzWork;
    w->V = V;
    w->nc = nc;
    const size_t vec = sizeof(double2) * 4 * nc * (size_t)V * 2;
    // partials of the kernel-by-kernel iteration or of the cooperative solve (smaller CTAs)
    const int nblocks = (V + kRitzGridSites - 1) / kRitzGridSites;
    double2 **bufs[] = {&w->x, &w->y, &w->z, &w->t, &w->p, &w->praw, &w->g};
    bool ok = true;
    for (double2 **b : bufs) ok = ok && cudaMalloc(b, vec) == cudaSuccess;
    ok = ok && cudaMalloc(&w->start, vec / 2) == cudaSuccess;
    ok = ok && cudaMalloc(&w->part, sizeof(double) * 4 * nblocks * kRitzParts) == cudaSuccess;
    ok = ok && cudaMalloc(&w->count, sizeof(int) * 3) == cudaSuccess;
    ok = ok && cudaMalloc(&w->st, 2 * sizeof(RitzScalars)) == cudaSuccess;
    ok = ok && cudaMallocHost(&w->host, 3 * sizeof(RitzScalars)) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        ritz_destroy(w);
        return nullptr;
    }
    return w;
}

void ritz_destroy(void *work) {
    RitzWork *w = static_cast<RitzWork *>(work);
    if (!w) return;
    void *bufs[] = {w->x, w->y, w->z, w->t, w->p, w->praw, w->g, w->start, w->part, w->count, w->st};
    for (void *b : bufs)
        if (b) cudaFree(b);
    if (w->host) cudaFreeHost(w->host);
    w->graphs.release();
    delete w;
}

double2 *ritz_start_buffer(void *work) { return static_cast<RitzWork *>(work)->start; }

void launch_ritz_random_start(void *work, uint64_t seed, uint64_t call, cudaStream_t stream) {
    RitzWork &w = *static_cast<RitzWork *>(work);
    const size_t n = (size_t)w.V * 4 * w.nc;
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 1024);
    ritz_random_start_kernel<<<blocks, 256, 0, stream>>>(w.start, n, seed, call);
}

template <int NC, bool U1>
static void launch_apply(const RitzWork &w, const double *U, const double *u1, const Lattice &L, double amass,
                         const double2 *src, double2 *dst, const double2 *da, const double2 *db, bool second,
                         const RitzArgs &a, dim3 grid, cudaStream_t stream) {
    if constexpr (NC == 2) {
        LinksF64<U1> lk{U, reinterpret_cast<const double2 *>(u1), L.N0 * L.N1};
        if (second)
            ritz_apply_kernel<2, U1, true><<<grid, kRitzThreads, 0, stream>>>(lk, src, dst, da, db, L, amass, w.st, a,
                                                                             w.part);
        else
            ritz_apply_kernel<2, U1, false><<<grid, kRitzThreads, 0, stream>>>(lk, src, dst, da, db, L, amass, w.st, a,
                                                                              w.part);
    } else {
        Links3<false, U1> lk{U, u1, L.N0 * L.N1};
        if (second)
            ritz_apply_kernel<3, U1, true><<<grid, kRitzThreads, 0, stream>>>(lk, src, dst, da, db, L, amass, w.st, a,
                                                                             w.part);
        else
            ritz_apply_kernel<3, U1, false><<<grid, kRitzThreads, 0, stream>>>(lk, src, dst, da, db, L, amass, w.st, a,
                                                                              w.part);
    }
}

template <int NC>
static cudaError_t ritz_run_nc(RitzWork &w, const double *U, const double *u1, const Lattice &L, double amass,
                               int max_iter, int nrestart, double delitr, double out[2], int iters[2],
                               cudaStream_t stream, uint64_t *launches) {
    constexpr int NCOMP = 4 * NC;
    const int V = L.V;
    RitzArgs a;
    a.nblocks = (V + kRitzThreads - 1) / kRitzThreads;
    a.sign[0] = 1.0;
    a.sign[1] = -1.0;
    a.delitr = delitr;
    a.max_iter = max_iter;
    const dim3 grid(a.nblocks, 2);
    uint64_t nl = 0;
    cudaError_t e = cudaMemsetAsync(w.st, 0, 2 * sizeof(RitzScalars), stream);
    if (e != cudaSuccess) return e;
    auto apply = [&](const double2 *src, double2 *dst, const double2 *da, const double2 *db, bool second) {
        if (u1) launch_apply<NC, true>(w, U, u1, L, amass, src, dst, da, db, second, a, grid, stream);
        else launch_apply<NC, false>(w, U, u1, L, amass, src, dst, da, db, second, a, grid, stream);
        nl++;
    };
    ritz_start_kernel<NCOMP><<<grid, kRitzThreads, 0, stream>>>(w.start, w.x, V, a, w.part);
    ritz_scale_x_kernel<NCOMP><<<grid, kRitzThreads, 0, stream>>>(w.x, V, a, w.part);
    nl += 2;
    // restart: y = sign A x, xy, g = p = y - xy x
    auto restart_seq = [&]() {
        apply(w.x, w.t, nullptr, nullptr, false);
        apply(w.t, w.y, w.x, nullptr, true);
        ritz_restart_kernel<NCOMP><<<grid, kRitzThreads, 0, stream>>>(w.x, w.y, w.g, w.praw, V, w.st, a, w.part);
        ritz_normp_kernel<NCOMP><<<grid, kRitzThreads, 0, stream>>>(w.praw, w.p, V, 1, w.st, a, w.part);
        nl += 2;
    };
    auto step_seq = [&]() {
        apply(w.p, w.t, nullptr, nullptr, false);
        apply(w.t, w.z, w.p, w.x, true);
        ritz_rotate_kernel<NCOMP><<<grid, kRitzThreads, 0, stream>>>(w.x, w.y, w.p, w.z, V, w.st, a, w.part);
        ritz_residual_kernel<NCOMP><<<grid, kRitzThreads, 0, stream>>>(w.x, w.y, w.g, w.p, V, w.st, a, w.part);
        ritz_direction_kernel<NCOMP><<<grid, kRitzThreads, 0, stream>>>(w.x, w.g, w.p, w.praw, V, w.st, a, w.part);
        ritz_normp_kernel<NCOMP><<<grid, kRitzThreads, 0, stream>>>(w.praw, w.p, V, 0, w.st, a, w.part);
        nl += 4;
    };
    auto poll = [&](bool &finished, int step) -> cudaError_t {
        cudaError_t r;
        if ((r = cudaGetLastError()) != cudaSuccess) return r;
        if ((r = cudaMemcpyAsync(w.host, w.st, 2 * sizeof(RitzScalars), cudaMemcpyDeviceToHost, stream)) !=
            cudaSuccess)
            return r;
        if ((r = cudaStreamSynchronize(stream)) != cudaSuccess) return r;
        finished = (w.host[0].done && w.host[1].done) || step >= max_iter;
        return cudaSuccess;
    };
    // The graphs replace the loop below when the restart cycle and the step
    // limit are whole numbers of poll intervals: the same kernels in the same
    // order, so the same results.
    RitzGraphs &gr = w.graphs;
    bool graphs = !gr.failed && nrestart % kRitzPoll == 0 && max_iter % kRitzPoll == 0;
    if (graphs && !(gr.restart && gr.U == U && gr.u1 == u1 && gr.N[0] == L.N0 && gr.N[1] == L.N1 && gr.N[2] == L.N2 &&
                    gr.amass == amass && gr.delitr == delitr && gr.max_iter == max_iter)) {
        gr.release();
        auto capture = [&](bool with_restart, cudaGraphExec_t &exec) {
            if (cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return false;
            const uint64_t nl0 = nl;
            if (with_restart) restart_seq();
            for (int i = 0; i < kRitzPoll; i++) step_seq();
            nl = nl0;  // counted when replayed
            cudaGraph_t g = nullptr;
            if (cudaStreamEndCapture(stream, &g) != cudaSuccess || !g) return false;
            const bool ok = cudaGraphInstantiate(&exec, g, 0) == cudaSuccess;
            cudaGraphDestroy(g);
            return ok;
        };
        if (capture(true, gr.restart) && capture(false, gr.plain)) {
            gr.U = U;
            gr.u1 = u1;
            gr.N[0] = L.N0;
            gr.N[1] = L.N1;
            gr.N[2] = L.N2;
            gr.amass = amass;
            gr.delitr = delitr;
            gr.max_iter = max_iter;
        } else {
            cudaGetLastError();
            gr.release();
            gr.failed = true;
            graphs = false;
        }
    }
    int step = 0;
    bool finished = false;
    if (graphs) {
        // one graph per poll interval, the restart one opening each cycle
        while (!finished) {
            const bool restart = step % nrestart == 0;
            if ((e = cudaGraphLaunch(restart ? gr.restart : gr.plain, stream)) != cudaSuccess) return e;
            nl += (restart ? 4 : 0) + 6 * kRitzPoll;
            step += kRitzPoll;
            if ((e = poll(finished, step)) != cudaSuccess) return e;
        }
    } else {
        // Host loop: restarts every nrestart steps; the done flags are read back
        // every kRitzPoll steps (both problems step in lockstep until they stop).
        while (!finished) {
            restart_seq();
            for (int itt = 1; itt <= nrestart; itt++) {
                step_seq();
                step++;
                if (step % kRitzPoll == 0 || itt == nrestart || step >= max_iter) {
                    if ((e = poll(finished, step)) != cudaSuccess) return e;
                    if (finished) break;
                }
            }
        }
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(w.host, w.st, 2 * sizeof(RitzScalars), cudaMemcpyDeviceToHost, stream)) != cudaSuccess)
        return e;
    if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return e;
    for (int k = 0; k < 2; k++) {
        out[k] = w.host[k].xy_re;
        if (iters) iters[k] = w.host[k].ittot;
    }
    if (launches) *launches += nl;
    return cudaSuccess;
}

template <bool U1> static RitzPlan ritz_plan(int V) {
    RitzPlan pl;
    int dev = 0, sms = 0, coop = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess) {
        cudaGetLastError();
        return pl;
    }
    // eight CTAs are the portable cluster size; sixteen halve the sites of a CTA
    // where the GPU takes them
    for (int ranks = 8; ranks <= kRitzClusterMax; ranks *= 2) {
        const int sites = (((V + ranks - 1) / ranks + 15) / 16) * 16;  // whole warps of two threads per site
        if (2 * sites > kRitzClusterThreads) continue;
        const size_t smem = ritz_cluster_smem(sites);
        // the attribute belongs to the kernel, not to this solve: always the largest
        if (cudaFuncSetAttribute(ritz_cluster_kernel<U1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)ritz_cluster_smem(kRitzClusterThreads / 2)) != cudaSuccess ||
            (ranks > 8 && cudaFuncSetAttribute(ritz_cluster_kernel<U1>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                              cudaSuccess)) {
            cudaGetLastError();
            continue;
        }
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = ranks;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(ranks, 2);
        cfg.blockDim = dim3(2 * sites);
        cfg.dynamicSmemBytes = smem;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, ritz_cluster_kernel<U1>, &cfg) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        if (clusters < 1) continue;
        pl.ranks = ranks;
        pl.sites = sites;
        pl.smem = smem;
        return pl;
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ritz_grid_kernel<U1>, 2 * kRitzGridSites, 0) != cudaSuccess) {
        cudaGetLastError();
        return pl;
    }
    pl.grid = coop && 2LL * ((V + kRitzGridSites - 1) / kRitzGridSites) <= (long long)sms * per_sm;
    return pl;
}

// stall: the arrival counters start where no phase's count reaches (the bounded
// waits of the cooperative launch then run out).
template <bool U1>
static cudaError_t ritz_run_one(RitzWork &w, const RitzPlan &pl, const double *U, const double *u1, const Lattice &L,
                                double amass, int max_iter, int nrestart, double delitr, double out[2], int iters[2],
                                cudaStream_t stream, uint64_t *launches, bool stall) {
    RitzOne a;
    a.start = w.start;
    a.st = w.st;
    a.amass = amass;
    a.delitr = delitr;
    a.max_iter = max_iter;
    a.nrestart = nrestart;
    a.sites = pl.ranks ? pl.sites : kRitzGridSites;
    a.v = w.praw;
    a.t = w.t;
    a.part = w.part;
    a.count = w.count;
    a.err = w.count + 2;
    LinksF64<U1> lk{U, reinterpret_cast<const double2 *>(u1), L.N0 * L.N1};
    Lattice lat = L;
    cudaError_t e = cudaMemsetAsync(w.count, 0, sizeof(int) * 3, stream);
    if (e == cudaSuccess && stall) e = cudaMemsetAsync(w.count, 0x80, sizeof(int) * 2, stream);  // -2.1e9
    if (e != cudaSuccess) return e;
    if (pl.ranks) {
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = pl.ranks;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(pl.ranks, 2);
        cfg.blockDim = dim3(2 * pl.sites);
        cfg.dynamicSmemBytes = pl.smem;
        cfg.stream = stream;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, ritz_cluster_kernel<U1>, lk, lat, a);
    } else {
        void *args[] = {&lk, &lat, &a};
        const dim3 grid((L.V + kRitzGridSites - 1) / kRitzGridSites, 2);
        e = cudaLaunchCooperativeKernel(ritz_grid_kernel<U1>, grid, dim3(2 * kRitzGridSites), args, 0, stream);
    }
    if (e != cudaSuccess) return e;
    if (launches) *launches += 1;
    int *err = reinterpret_cast<int *>(w.host + 2);
    if ((e = cudaMemcpyAsync(w.host, w.st, 2 * sizeof(RitzScalars), cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
        (e = cudaMemcpyAsync(err, a.err, sizeof(int), cudaMemcpyDeviceToHost, stream)) != cudaSuccess ||
        (e = cudaStreamSynchronize(stream)) != cudaSuccess)
        return e;
    if (*err) return cudaErrorLaunchTimeout;  // a wait between the CTAs ran out
    for (int k = 0; k < 2; k++) {
        out[k] = w.host[k].xy_re;
        if (iters) iters[k] = w.host[k].ittot;
    }
    return cudaSuccess;
}

// Runs both Ritz problems from the start vector already in the start buffer
// (compact [V][4 nc] double2; links of the work space's colour count).  out:
// {lambda_min, -lambda_max as returned by the sign = -1 problem}; iters: steps
// per problem.  Returns a CUDA error or cudaSuccess; *launches counts kernels.
cudaError_t ritz_run(void *work, const double *U, const double *u1, const Lattice &L, double amass, int max_iter,
                     int nrestart, double delitr, double out[2], int iters[2], cudaStream_t stream,
                     uint64_t *launches, bool stall, bool *expired) {
    RitzWork &w = *static_cast<RitzWork *>(work);
    if (stall && w.nc == 3) return cudaErrorNotSupported;
    if (w.nc == 3)
        return ritz_run_nc<3>(w, U, u1, L, amass, max_iter, nrestart, delitr, out, iters, stream, launches);
    const int b = u1 ? 1 : 0;
    if (!w.planned[b]) {  // the work space belongs to one lattice size and device
        w.plan[b] = u1 ? ritz_plan<true>(L.V) : ritz_plan<false>(L.V);
        w.planned[b] = true;
    }
    RitzPlan &pl = w.plan[b];
    if (stall && !pl.grid) return cudaErrorNotSupported;
    if (pl.ranks || pl.grid) {
        const cudaError_t e =
            u1 ? ritz_run_one<true>(w, pl, U, u1, L, amass, max_iter, nrestart, delitr, out, iters, stream, launches, stall)
               : ritz_run_one<false>(w, pl, U, u1, L, amass, max_iter, nrestart, delitr, out, iters, stream, launches, stall);
        if (expired) *expired = e == cudaErrorLaunchTimeout;
        if (e == cudaSuccess) return e;
        // The launch was refused or a wait ran out: from here on kernel by kernel
        // (an error of the device itself shows up there again).
        cudaGetLastError();
        if (!stall) pl = RitzPlan{};
    }
    return ritz_run_nc<2>(w, U, u1, L, amass, max_iter, nrestart, delitr, out, iters, stream, launches);
}

}  // namespace ovl
