"""The Chebyshev overlap operator with a lattice's modes held on chip by a
thread-block cluster: lattices that need one CTA and several, z planes that do
not divide among the CTAs, several sets of modes per cluster with the last
cluster partly filled, and lattices just beyond what fits (the kernels that go
through memory), against the FP64 oracle."""
import ctypes as C

import numpy as np
import pytest

from _helpers import oracle_params, rel_err
from _oracle import oracle, ptr
from overlap_b200 import Context
from overlap_b200.inputs import (embed_su2_efield, embed_su2_links, random_efield, random_efield_su3, random_links,
                                 random_links_su3, u1_flux, volume)

pytestmark = pytest.mark.gpu

K, EPS, M, MDW, DT = 6, 0.02, 0.05, 1.0, 0.05
MODES, CHECKED = 33, [0, 17, 32]  # two mode blocks, the second one mode and padding


def f64(a):
    return np.ascontiguousarray(a).view(np.float64)


# (nc, precision, N): two colours on one CTA below and at its 512 sites; 2, 5 and 8
# CTAs, even and uneven; a plane over 512 sites and z too long for 8 CTAs (through
# memory).  Three colours alike, with 512 and 576 threads, FP64 with 256 and 224.
SHAPES = [(2, "fp32", N) for N in ((3, 3, 3), (5, 7, 3), (8, 8, 8), (7, 6, 13), (12, 11, 10), (16, 16, 16), (16, 16, 17),
                                   (23, 23, 3))]
SHAPES += [(2, "fp64", N) for N in ((3, 3, 3), (8, 6, 8), (9, 10, 8), (11, 4, 13), (16, 16, 8))]
SHAPES += [(3, "fp32", N) for N in ((3, 3, 3), (8, 8, 8), (9, 5, 11), (10, 10, 10), (6, 10, 15), (12, 12, 12),
                                    (13, 13, 9), (12, 12, 17))]
SHAPES += [(3, "fp64", N) for N in ((3, 3, 3), (6, 6, 6), (8, 8, 8), (8, 8, 5), (10, 10, 11), (16, 16, 3))]


@pytest.mark.parametrize("u1", [False, True])
@pytest.mark.parametrize("nc,precision,N", SHAPES)
def test_resident_chebyshev_matches_the_oracle(nc, precision, N, u1):
    U, E = (random_links_su3(N, 0.6, 61), random_efield_su3(N, 0.3, 62)) if nc == 3 else (random_links(N, 0.6, 61),
                                                                                          random_efield(N, 0.3, 62))
    U3, E3 = (U.copy(), E) if nc == 3 else (embed_su2_links(U).copy(), embed_su2_efield(E))
    rng = np.random.default_rng(63)
    shape = (2, MODES, volume(N), nc, 4)
    psi, mid = rng.normal(size=shape) + 1j * rng.normal(size=shape)

    def embed(q):
        out = np.zeros(q.shape[:2] + (3, 4), complex)
        out[:, :, :nc, :] = q
        return out

    ph = np.ascontiguousarray(u1_flux(N, 2)) if u1 else None
    p = oracle_params(N, m=M, mdw=MDW, dt=DT)
    lmax = (0.5 * abs(6 + 2 * M - 2 * MDW) + 3.0) ** 2  # the context's default bound on h_W^2
    src, o_psi, o_mid = embed(psi[CHECKED]), embed(psi[CHECKED]), embed(mid[CHECKED])
    want = np.zeros_like(src)
    t = C.c_int(0)
    if u1:
        oracle().orc_set_u1(ptr(f64(ph)))
    try:
        for k in range(len(CHECKED)):
            oracle().orc3_overlap_apply(C.byref(p), ptr(f64(U3)), ptr(f64(src[k])), ptr(f64(want[k])), K, EPS, lmax)
        oracle().orc3_overlap_leapfrog(C.byref(p), ptr(f64(U3)), ptr(f64(E3)), ptr(f64(o_psi)), ptr(f64(o_mid)),
                                       len(CHECKED), C.byref(t), 1, K, EPS, lmax)
    finally:
        oracle().orc_set_u1(None)
    with Context(N=N, n_modes=MODES, n_colours=nc, fermion="overlap", sign_method="chebyshev", cheb_degree=K, cheb_eps=EPS,
                 m_fermion=M, m_dw=MDW, dt=DT, precision=precision, form="fused") as ctx:
        ctx.set_links(U)
        ctx.set_efield(E)
        if u1:
            ctx.set_u1(ph)
        got = ctx.apply(psi)
        ctx.set_modes(psi, mid)
        ctx.step(1)
        g_psi, g_mid = ctx.get_modes()
    # a term rounds its stencil, sums of some 16 products, and Clenshaw's recurrence
    # carries that on at most k + 1 times: 16 u (1 + ... + K + 1), twice that for both sides
    tol = 16 * (K + 1) * (K + 2) * (2.0 ** -24 if precision == "fp32" else 2.0 ** -53)
    assert rel_err(got[CHECKED], want[:, :, :nc, :]) < tol
    assert rel_err(g_psi[CHECKED], o_psi[:, :, :nc, :]) < tol
    assert rel_err(g_mid[CHECKED], o_mid[:, :, :nc, :]) < tol
