"""The Chebyshev overlap operator with a lattice's modes held on chip by a
thread-block cluster: lattices that need one CTA and several, z planes that do
not divide among the CTAs, several sets of modes per cluster with the last
cluster partly filled, and lattices that go through memory (beyond what fits,
or faster there), against the FP64 oracle.  Both routes compute the same
operator, so every case states its route and the launches tell it."""
import ctypes as C

import numpy as np
import pytest

from _helpers import oracle_params, rel_err
from _oracle import oracle, ptr
from overlap_b200 import Context
from overlap_b200.inputs import (embed_su2_efield, embed_su2_links, random_efield, random_efield_su3, random_links,
                                 random_links_su3, u1_flux, volume)

pytestmark = pytest.mark.gpu

EPS, M, MDW, DT = 0.02, 0.05, 1.0, 0.05


def f64(a):
    return np.ascontiguousarray(a).view(np.float64)


# (nc, precision, N, modes, degree, on chip).  33 modes: two mode blocks, the second
# one mode and padding.  Two colours on one CTA below and at its 512 sites; 2 to 8
# CTAs, even and uneven, with one set of modes and several; a plane over 512 sites
# and z too long for 8 CTAs (through memory).  Three colours alike, with 512 and 576
# threads, FP64 with 256 and 224.
SHAPES = [(2, "fp32", N, 33, 6, on) for N, on in (((3, 3, 3), True), ((5, 7, 3), True), ((8, 8, 8), True), ((7, 6, 13), True),
                                                  ((12, 11, 10), True), ((16, 16, 16), False), ((16, 16, 17), False),
                                                  ((23, 23, 3), False))]
SHAPES += [(2, "fp32", N, m, k, True) for N, m, k in (((3, 3, 3), 385, 6), ((5, 7, 3), 1025, 6), ((8, 8, 8), 257, 6),
                                                      ((8, 8, 8), 97, 6), ((7, 6, 13), 97, 12), ((7, 6, 13), 130, 6),
                                                      ((7, 6, 13), 385, 6), ((16, 16, 16), 65, 24))]
SHAPES += [(2, "fp64", N, 33, 6, on) for N, on in (((3, 3, 3), True), ((8, 6, 8), True), ((9, 10, 8), True),
                                                   ((11, 4, 13), True), ((16, 16, 8), False))]
SHAPES += [(2, "fp64", N, m, k, True) for N, m, k in (((3, 3, 3), 1025, 6), ((8, 6, 8), 97, 6), ((8, 6, 8), 130, 6),
                                                      ((11, 4, 13), 65, 12), ((16, 16, 8), 33, 24))]
SHAPES += [(3, "fp32", N, 33, 6, on) for N, on in (((3, 3, 3), True), ((8, 8, 8), True), ((9, 5, 11), True),
                                                   ((10, 10, 10), True), ((6, 10, 15), True), ((12, 12, 12), False),
                                                   ((13, 13, 9), False), ((12, 12, 17), False))]
SHAPES += [(3, "fp32", N, m, k, True) for N, m, k in (((3, 3, 3), 513, 6), ((8, 8, 8), 97, 6), ((9, 5, 11), 97, 6),
                                                      ((9, 5, 11), 65, 12), ((12, 12, 12), 97, 24))]
SHAPES += [(3, "fp64", N, 33, 6, on) for N, on in (((3, 3, 3), True), ((6, 6, 6), True), ((8, 8, 8), True), ((8, 8, 5), True),
                                                   ((10, 10, 11), False), ((16, 16, 3), False), ((8, 14, 4), True))]
SHAPES += [(3, "fp64", N, m, k, True) for N, m, k in (((3, 3, 3), 385, 6), ((6, 6, 6), 97, 6), ((8, 14, 4), 161, 24))]
# the first terms of the series read phi in place of b_K: degrees with one, two and three terms
SHAPES += [(nc, precision, N, 33, k, on) for k in (1, 2, 3) for nc in (2, 3) for precision in ("fp32", "fp64")
           for N, on in (((4, 4, 4), True), ((25, 24, 3), False))]


@pytest.mark.parametrize("u1", [False, True])
@pytest.mark.parametrize("nc,precision,N,modes,degree,on_chip", SHAPES)
def test_resident_chebyshev_matches_the_oracle(nc, precision, N, modes, degree, on_chip, u1):
    K, checked = degree, [0, modes // 2, modes - 1]
    U, E = (random_links_su3(N, 0.6, 61), random_efield_su3(N, 0.3, 62)) if nc == 3 else (random_links(N, 0.6, 61),
                                                                                          random_efield(N, 0.3, 62))
    U3, E3 = (U.copy(), E) if nc == 3 else (embed_su2_links(U).copy(), embed_su2_efield(E))
    rng = np.random.default_rng(63)
    shape = (2, modes, volume(N), nc, 4)
    psi, mid = rng.normal(size=shape) + 1j * rng.normal(size=shape)

    def embed(q):
        out = np.zeros(q.shape[:2] + (3, 4), complex)
        out[:, :, :nc, :] = q
        return out

    ph = np.ascontiguousarray(u1_flux(N, 2)) if u1 else None
    p = oracle_params(N, m=M, mdw=MDW, dt=DT)
    lmax = (0.5 * abs(6 + 2 * M - 2 * MDW) + 3.0) ** 2  # the context's default bound on h_W^2
    src, o_psi, o_mid = embed(psi[checked]), embed(psi[checked]), embed(mid[checked])
    want = np.zeros_like(src)
    t = C.c_int(0)
    if u1:
        oracle().orc_set_u1(ptr(f64(ph)))
    try:
        for k in range(len(checked)):
            oracle().orc3_overlap_apply(C.byref(p), ptr(f64(U3)), ptr(f64(src[k])), ptr(f64(want[k])), K, EPS, lmax)
        oracle().orc3_overlap_leapfrog(C.byref(p), ptr(f64(U3)), ptr(f64(E3)), ptr(f64(o_psi)), ptr(f64(o_mid)),
                                       len(checked), C.byref(t), 1, K, EPS, lmax)
    finally:
        oracle().orc_set_u1(None)
    with Context(N=N, n_modes=modes, n_colours=nc, fermion="overlap", sign_method="chebyshev", cheb_degree=K, cheb_eps=EPS,
                 m_fermion=M, m_dw=MDW, dt=DT, precision=precision, form="fused") as ctx:
        ctx.set_links(U)
        ctx.set_efield(E)
        if u1:
            ctx.set_u1(ph)
        before = ctx.launch_count
        got = ctx.apply(psi)
        launches = ctx.launch_count - before
        ctx.set_modes(psi, mid)
        ctx.step(1)
        g_psi, g_mid = ctx.get_modes()
    # the layout on the way in and out, and the operator: one launch, or two a term and the end
    assert launches == 3 if on_chip else launches >= 2 + 2 * K + 1, launches
    # a term rounds its stencil, sums of some 16 products, and Clenshaw's recurrence
    # carries that on at most k + 1 times: 16 u (1 + ... + K + 1), twice that for both sides
    tol = 16 * (K + 1) * (K + 2) * (2.0 ** -24 if precision == "fp32" else 2.0 ** -53)
    assert rel_err(got[checked], want[:, :, :nc, :]) < tol
    assert rel_err(g_psi[checked], o_psi[:, :, :nc, :]) < tol
    assert rel_err(g_mid[checked], o_mid[:, :, :nc, :]) < tol
