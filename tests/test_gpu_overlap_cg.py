"""The batched multi-shift CG of the Zolotarev overlap operator at the edges of
its batches: the shifted vectors are brought up to date every eight iterations,
so iteration limits just below, at and above multiples of eight, and modes that
stop at different iterations, are compared with the reference's loop
(FERMIONS/OVERLAP/OPERATOR/OverlapU.cpp:5-149) restated in numpy on the dense
operator."""
import ctypes as C

import numpy as np
import pytest

from _helpers import oracle_params, random_modes
from _oracle import oracle, ptr
from overlap_b200 import Context
from overlap_b200.api import zolotarev
from overlap_b200.inputs import random_links, volume

pytestmark = pytest.mark.gpu

M, MDW = 0.1, 1.4


def dense_d(N, U):
    """D = -i h_W as a matrix: column j is D applied to the j-th unit vector."""
    p = oracle_params(N, m=M, mdw=MDW)
    n = 8 * volume(N)
    D = np.zeros((n, n), np.complex128)
    for j in range(n):
        e, out = np.zeros(n, np.complex128), np.zeros(n, np.complex128)
        e[j] = 1.0
        oracle().orc_wilson_apply(C.byref(p), ptr(U), ptr(e.view(np.float64)), ptr(out.view(np.float64)))
        D[:, j] = out
    return D


def overlap_u(D, phi, b, d, cgerr, max_iter):
    """-i h_ov phi of one mode, OverlapU.cpp's recurrences."""
    np_ = len(b)
    r, p, x = phi.copy(), [phi.copy() for _ in b], [np.zeros_like(phi) for _ in b]
    rnorm = np.vdot(phi, phi).real
    bnorm, betam, alpha0 = np.sqrt(rnorm), 1.0, 0.0
    z, g, it = np.ones(np_), np.ones(np_), 0
    while rnorm > cgerr * bnorm and it < max_iter:
        q = -(D @ (D @ p[0])) + d[0] * p[0]
        beta = np.empty(np_)
        beta[0] = rnorm / np.vdot(p[0], q).real
        for k in range(1, np_):
            z[k] = betam / (beta[0] * alpha0 * (1.0 - z[k]) + betam * (1.0 + (d[k] - d[0]) * beta[0]))
            beta[k] = beta[0] * z[k]
        r = r - beta[0] * q
        rr = np.vdot(r, r).real
        alpha0 = rr / rnorm
        rnorm = rr
        for k in range(np_):
            g[k] *= z[k]
            x[k] = x[k] + beta[k] * p[k]
            p[k] = p[k] * (alpha0 * z[k] * beta[k] / beta[0]) + r * g[k]
        betam = beta[0]
        it += 1
    chi = sum(bk * xk for bk, xk in zip(b, x))
    g0 = np.tile(np.array([-1j, -1j, 1j, 1j]), len(phi) // 4)  # -i gamma_0
    return MDW * ((1.0 + 0.5 * M) * g0 * phi + (1.0 - 0.5 * M) * (D @ chi)), it


# 25 poles are the reference's; the scalars of more than 32 are staged in two parts
@pytest.mark.parametrize("max_iter,poles", [(1, 25), (7, 25), (8, 25), (9, 25), (16, 25), (1000, 25), (17, 33)])
def test_cg_batches_match_the_reference_loop(max_iter, poles):
    N = (3, 4, 3)
    U = random_links(N, 0.5, 11)
    D = dense_d(N, U)
    lam = np.linalg.eigvalsh(-(D @ D))
    lo, hi = 0.95 * lam[0], 1.05 * lam[-1]
    b, d, _ = zolotarev(lo, hi, npoles=poles)
    phi = random_modes(35, N, 12)  # two mode blocks, the second mostly padding
    # modes of very different norm: the test |r|^2 > 1e-16 |phi| stops them at different iterations
    phi *= 10.0 ** np.linspace(-7, 3, 35)[:, None, None, None]
    with Context(N=N, n_modes=35, fermion="overlap", precision="fp64", m_fermion=M, m_dw=MDW, cg_max_iter=max_iter,
                 zolo_poles=poles) as ctx:
        ctx.set_links(U)
        ctx.set_spectral_bounds([(lo, hi)])
        out = ctx.apply(phi)
        stats = ctx.solver_stats()
    its = []
    for m in range(35):
        want, it = overlap_u(D, phi[m].ravel(), b, d, 1e-16, max_iter)
        its.append(it)
        # the rounding of a CG of a few steps at condition numbers below 1e2
        tol = 1e-11 * np.max(np.abs(want))
        if it < max_iter:
            # Stopped by its test, a run is known to its residual r only: shift k's residual is g_k r
            # with 0 <= g_k <= 1, so D chi is off by sum_k b_k D (h^2 + d_k)^-1 g_k r, where
            # sqrt(l) b_k / (l + d_k) > 0 sum to 1 at each eigenvalue l of h^2.  That is |r| at most,
            # |r|^2 <= 1e-16 |phi|, on either side (the loop above differs from itself by 1.6e-11 at
            # mode 24 when D's columns are only summed in another order).
            tol += 2 * MDW * (1.0 - 0.5 * M) * np.sqrt(1e-16 * np.linalg.norm(phi[m]))
        assert np.max(np.abs(out[m].ravel() - want)) < tol, (m, it)
    # a mode's last iterations sit at round-off, so its count may differ by one
    assert abs(stats["max_mode_iterations"] - max(its)) <= 1
    if max_iter == 1000:
        assert len(set(its)) > 3 and stats["not_converged"] == 0


# Few poles: batches of one (1 and 2 poles; with one its direction shares a temporary), 2, 3 and 7 iterations
@pytest.mark.parametrize("poles,max_iter", [(1, 1), (1, 1000), (2, 5), (2, 1000), (3, 3), (3, 1000), (4, 7), (8, 15)])
def test_cg_with_few_poles_matches_the_reference_loop(poles, max_iter):
    N = (3, 4, 3)
    U = random_links(N, 0.5, 11)
    D = dense_d(N, U)
    lam = np.linalg.eigvalsh(-(D @ D))
    lo, hi = 0.95 * lam[0], 1.05 * lam[-1]
    b, d, _ = zolotarev(lo, hi, npoles=poles)
    phi = random_modes(35, N, 12)
    phi *= 10.0 ** np.linspace(-7, 3, 35)[:, None, None, None]
    with Context(N=N, n_modes=35, fermion="overlap", precision="fp64", m_fermion=M, m_dw=MDW, cg_max_iter=max_iter,
                 zolo_poles=poles) as ctx:
        ctx.set_links(U)
        ctx.set_spectral_bounds([(lo, hi)])
        out = ctx.apply(phi)
    # sum_k sqrt(l) b_k / (l + d_k) at the eigenvalues l: 1 for many poles, at most this for few
    sign = max(np.sum(np.sqrt(l) * b / (l + d)) for l in lam)
    for m in range(35):
        want, it = overlap_u(D, phi[m].ravel(), b, d, 1e-16, max_iter)
        tol = 1e-11 * np.max(np.abs(want))
        if it < max_iter:  # the bound of the test above
            tol += 2 * MDW * (1.0 - 0.5 * M) * sign * np.sqrt(1e-16 * np.linalg.norm(phi[m]))
        assert np.max(np.abs(out[m].ravel() - want)) < tol, (m, it)


@pytest.mark.parametrize("poles", [1, 2, 4, 9, 25])
def test_cg_workspace_fields(poles):
    """The work space of a Zolotarev context takes no more fields than the five
    vectors and the two per pole of separate x_k and p_k: 3 + 2 poles."""
    import torch

    N, modes = (16, 16, 16), 64
    kw = dict(N=N, n_modes=modes, precision="fp64", m_fermion=M, m_dw=MDW)

    def taken(**more):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        with Context(**kw, **more) as ctx:
            ctx.synchronize()
            return before - torch.cuda.mem_get_info()[0]

    taken(), taken(fermion="overlap", zolo_poles=poles)  # what the first of either loads
    field = volume(N) * 8 * 16 * modes
    extra = taken(fermion="overlap", zolo_poles=poles) - taken()
    # the scalars, the dot products' partial sums (one double per mode and 8 sites, and 128) and
    # what allocations round up to stay below a field
    assert extra < (3 + 2 * poles + 1) * field
