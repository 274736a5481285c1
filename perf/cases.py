"""Performance cases of the framework: what a program that evolves fermion modes in a gauge background calls.

Five kinds of pass, each through the public host API (overlap_b200.Context, overlap_b200.Ensemble):

  step      leapfrog steps of the mode batch (plain or fused form, FP64 / FP32 / 40-bit modes, two or three
            colours, with or without the U(1) background), optionally with the charges summed inside the last
            step, with the currents read after it, or with the coupled gauge evolution (staple force and the
            fermions' back-reaction on E)
  overlap   leapfrog steps of overlap fermions (Zolotarev multi-shift CG with Ritz bounds, or the Chebyshev series)
  currents  the per-site current densities of the modes
  observe   one observation of a trajectory: charges, change of N_CS along the path, bulk observables
  ensemble  steps of several trajectories of mixed lattice size batched together

Inputs: random SU(2) / SU(3) links and electric fields of the spread the configurations use, and Gaussian random
modes with |psi(x)|^2 = 1 (the normalisation of the plane waves and of the Z2 noise) whose half-step partner is
close to them; all from the seed, the modes made on the GPU.  exact() evaluates the same operators in complex128
with torch, written from their definitions.
"""
import math

import numpy as np
import torch

from overlap_b200 import Context, Ensemble, Params
from overlap_b200.inputs import random_efield, random_efield_su3, random_links, random_links_su3, u1_flux

R_WILSON = 1.0
LANES = 32  # modes per block of the mode layout [mode / 32][site][colour * 4 + spin][mode % 32]


# ------------------------------------------------------------------ cases --
def listed():
    step = dict(kind="step", nc=2, precision="fp64", form="fused", flux=0, m=0.05, dt=0.05, steps=1, observe=False,
                currents=False, coupled=0.0, variant=-1)
    overlap = dict(kind="overlap", nc=2, precision="fp32", m=0.05, mdw=1.4, dt=0.02, steps=1, variant=-1)
    return [
        # the smallest call: one step of a thin slice of modes with its charges, as a monitor or a test runs it
        dict(step, name="step_small_observe", n0=8, n1=8, n2=8, modes=128, precision="fp32", observe=True),
        # the plain two-phase FP64 form on the complete basis of 8^3 (the parity configuration)
        dict(step, name="step_fp64_plain_8", n0=8, n1=8, n2=8, modes=4096, form="plain", m=0.1),
        # FP64 production form on a lattice of unequal, odd extents, a mode count that does not fill its blocks
        dict(step, name="step_fp64_ragged", n0=10, n1=13, n2=9, modes=1501, flux=2),
        # the headline: FP32 modes on 16^3 with the U(1) flux, half of the complete basis, the packed kernel
        dict(step, name="step_fp32_16_flux", n0=16, n1=16, n2=16, modes=16384, precision="fp32", flux=4, variant=3),
        # 40-bit modes, evolved between two observation points and then measured
        dict(step, name="step_fp40_12_currents", n0=12, n1=12, n2=12, modes=1000, precision="fp40", flux=2, steps=4,
             currents=True),
        # the coupled evolution: staple force and fermion force on E in every step
        dict(step, name="step_coupled_fp64_8", n0=8, n1=8, n2=8, modes=1024, steps=4, coupled=0.25),
        # overlap fermions, three colours, 12^3, degree 96 (a slice of the complete basis of 20736)
        dict(overlap, name="overlap_su3_cheb_12", nc=3, n0=12, n1=12, n2=12, modes=1536, sign="chebyshev", degree=96,
             variant=3),
        # an overlap request as the server admits them: two colours, degree 64
        dict(overlap, name="overlap_su2_cheb_8", n0=8, n1=8, n2=8, modes=4096, sign="chebyshev", degree=64),
        # the reference's own overlap form: 25 poles, FP64, spectral bounds from the Ritz solver in every half step
        dict(overlap, name="overlap_zolotarev_8", n0=8, n1=8, n2=8, modes=256, precision="fp64", sign="zolotarev",
             degree=0),
        # current densities of a large batch
        dict(kind="currents", name="currents_fp32_16", nc=2, n0=16, n1=16, n2=16, modes=4096, precision="fp32", flux=4),
        # one observation of a running trajectory
        dict(kind="observe", name="observe_fp32_12", nc=2, n0=12, n1=12, n2=12, modes=4096, precision="fp32", flux=0),
        # mixed lattices stepped together, 1024 modes each
        dict(kind="ensemble", name="ensemble_mixed", nc=2, sizes="8,10,12,16", copies=3, modes=1024, precision="fp32",
             flux=4, steps=2),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "overlap", "overlap", "currents", "observe", "ensemble"])
    n = [_log(rng, 5, 16) for _ in range(3)]
    n0, n1, n2 = n if rng.random() < 0.5 else (n[0],) * 3
    nc = 3 if rng.random() < 0.25 else 2
    V = n0 * n1 * n2
    case = dict(kind=kind, nc=nc, n0=n0, n1=n1, n2=n2)
    if kind == "step":
        precision = rng.choice(["fp64", "fp32", "fp32"] + ([] if nc == 3 else ["fp40"]))
        steps = rng.choice([1, 2, 4])
        most = 1024 if precision == "fp40" else max(64, min(16384, int(1e8 / (V * nc * steps * (2 if precision == "fp64" else 1)))))
        coupled = 0.25 if precision != "fp40" and rng.random() < 0.2 else 0.0
        observe = precision != "fp40" and not coupled and rng.random() < 0.3
        case.update(precision=precision, modes=_log(rng, 32, most), flux=rng.choice([0, 2, 4]), dt=0.05,
                    form="plain" if precision == "fp64" and rng.random() < 0.3 else "fused", m=rng.choice([0.05, 0.1]),
                    steps=steps, observe=observe, currents=precision == "fp40", coupled=coupled,
                    variant=3 if precision == "fp32" and rng.random() < 0.5 else -1)
    elif kind == "overlap":
        sign = "chebyshev" if nc == 3 or rng.random() < 0.7 else "zolotarev"
        if sign == "zolotarev":
            n0, n1, n2 = (min(8, v) for v in (n0, n1, n2))
            case.update(n0=n0, n1=n1, n2=n2)
            most = max(32, int(1.2e5 / (n0 * n1 * n2)))
        else:
            most = max(64, min(4096, int(2.5e6 / V)))
        fp64 = sign == "zolotarev" or rng.random() < 0.2
        if fp64 and sign == "chebyshev":
            most = max(64, most // 2)
        case.update(sign=sign, modes=_log(rng, 32, most), degree=0 if sign == "zolotarev" else rng.choice([48, 64, 96]),
                    precision="fp64" if fp64 else "fp32", m=0.05, mdw=1.4, dt=0.02, steps=1,
                    variant=3 if nc == 3 and not fp64 else -1)
    elif kind in ("currents", "observe"):
        case.update(precision=rng.choice(["fp64", "fp32", "fp32"]), modes=_log(rng, 32, max(64, min(8192, int(1.6e7 / V)))),
                    flux=rng.choice([0, 4]))
    else:
        sizes = sorted(_log(rng, 5, 16) for _ in range(rng.choice([2, 3, 4])))
        case = dict(kind=kind, nc=nc, sizes=",".join(map(str, sizes)), copies=rng.choice([1, 2, 3]),
                    modes=_log(rng, 64, 1024), precision=rng.choice(["fp64", "fp32", "fp32"]), flux=rng.choice([0, 4]),
                    steps=rng.choice([1, 2, 4]))
    return case


def _dims(case):
    return int(case["n0"]), int(case["n1"]), int(case["n2"])


# ----------------------------------------------------------------- inputs --
def _gauge(case, N, seed):
    """(links, E) in the host layouts, and the U(1) phases or None."""
    overlap = case["kind"] == "overlap"
    sigma_e = 0.02 if overlap else 0.1
    if case["nc"] == 3:
        U, E = random_links_su3(N, 0.3, seed), random_efield_su3(N, sigma_e, seed + 1)
    else:
        U, E = random_links(N, 0.3, seed), random_efield(N, sigma_e, seed + 1)
    return U, E, u1_flux(N, case["flux"]) if case.get("flux") else None


def _random_modes(blocks, V, comp, modes, dtype, seed, out=None):
    """(psi, psimid) as real tensors [blocks, V, comp, 32, 2] on the GPU, zero beyond `modes`; into `out` when given."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    psi, mid = out if out is not None else (torch.empty(blocks, V, comp, LANES, 2, dtype=dtype, device="cuda") for _ in range(2))
    scale = 1.0 / math.sqrt(2.0 * comp)
    psi.normal_(0.0, scale, generator=g)
    mid.normal_(0.0, 0.05 * scale, generator=g)
    mid += psi
    if modes < blocks * LANES:
        for f in (psi, mid):
            f[-1, :, :, modes - blocks * LANES:] = 0
    return psi, mid


class _DeviceArray:
    """A device buffer of `owner` as an array that torch can share; a tensor made of it keeps the owner."""

    def __init__(self, owner, pointer, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": tuple(shape), "typestr": typestr, "version": 3,
                                         "strides": None}


def _field_views(ctx, precision, blocks, V, comp):
    """The context's mode fields, shared: real pairs [blocks, V, comp, 32, 2] (40-bit modes: the high words)."""
    psi, mid, nbytes = ctx.device_modes()
    kind, size = {"fp64": ("<f8", 8), "fp32": ("<f4", 4), "fp40": ("<i4", 4)}[precision]
    shape = (blocks, V, comp, LANES, 2)
    assert nbytes == math.prod(shape) * size
    return [torch.as_tensor(_DeviceArray(ctx, p, shape, kind), device="cuda") for p in (psi, mid)]


def _params(case, N):
    p = dict(N=N, n_colours=case["nc"], n_modes=case["modes"], precision=case["precision"], t_sphaleron=1e9,
             r_wilson=R_WILSON, form="fused", m_dw=0.0)
    if case["kind"] == "overlap":
        p.update(fermion="overlap", sign_method=case["sign"], m_fermion=case["m"], m_dw=case["mdw"], dt=case["dt"],
                 hop_variant=case["variant"])
        if case["sign"] == "chebyshev":
            p.update(cheb_degree=case["degree"], cheb_eps=0.01)
        else:
            p.update(ritz_auto=True)
    elif case["kind"] == "step":
        p.update(form=case["form"], m_fermion=case["m"], dt=case["dt"], hop_variant=case["variant"],
                 gauge_force=bool(case["coupled"]), backreaction=case["coupled"])
    else:
        p.update(m_fermion=0.05, dt=0.05)
    return p


def _fill(ctx, case, N, seed):
    U, E, u1 = _gauge(case, N, seed)
    ctx.set_links(U)
    ctx.set_efield(E)
    if u1 is not None:
        ctx.set_u1(u1)
    V, comp, modes = math.prod(N), 4 * case["nc"], case["modes"]
    blocks = -(-modes // LANES)
    views = _field_views(ctx, case["precision"], blocks, V, comp)
    if case["precision"] == "fp40":  # modes enter through the host in 40-bit storage
        fields = _random_modes(blocks, V, comp, modes, torch.float32, seed)
        host = [_to_host_layout(f, modes, case["nc"]) for f in fields]
        ctx.set_modes(*host)
    else:
        ctx.synchronize()
        _random_modes(blocks, V, comp, modes, torch.float64 if case["precision"] == "fp64" else torch.float32, seed, views)
        torch.cuda.synchronize()
    return views


def _to_host_layout(f, modes, nc):
    """[blocks, V, comp, 32, 2] -> complex128 [modes, V, nc, 4] on the host."""
    b, V, comp = f.shape[:3]
    z = torch.view_as_complex(f.double()).permute(0, 3, 1, 2).reshape(b * LANES, V, nc, 4)[:modes]
    return np.ascontiguousarray(z.cpu().numpy())


def prepare(case, seed):
    if case["kind"] == "ensemble":
        sizes = [int(n) for n in case["sizes"].split(",")] * case["copies"]
        ens = Ensemble([Params(**_params(case, (n, n, n))) for n in sizes])
        views = [_fill(ens[i], case, (n, n, n), seed + 101 * i) for i, n in enumerate(sizes)]
        ens.synchronize()
        return {"case": case, "ens": ens, "out": {"psi": [v[0] for v in views], "mid": [v[1] for v in views]}}
    N = _dims(case)
    ctx = Context(Params(**_params(case, N)))
    views = _fill(ctx, case, N, seed)
    if case["kind"] == "step" and case["variant"] < 0:
        ctx.autotune()  # a program tunes once per context; otherwise its first step does
    if case["kind"] == "observe":
        ctx.ncs_update()  # the path of N_CS starts here
    ctx.synchronize()
    return {"case": case, "ctx": ctx, "out": {"psi": views[0], "mid": views[1]}}


# -------------------------------------------------------------------- run --
def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        state["ens"].step(case["steps"])
        return state["out"]
    ctx = state["ctx"]
    if case["kind"] == "currents":
        return ctx.currents()
    if case["kind"] == "observe":
        ctx.update_links(0.05)  # the links have moved since the last observation
        c, bulk = ctx.charges(), ctx.bulk()
        return {"charges": np.array([c["NV"], c["N5"], c["PS"], c["WA"]]), "ncs": np.array([ctx.ncs_update()[0]]),
                "bulk": np.array([bulk[k] for k in BULK])}
    out = dict(state["out"])
    if case["kind"] == "step" and case["observe"]:
        c = ctx.step_observe(case["steps"])
        out["charges"] = np.array([c["NV"], c["N5"], c["PS"]])
        return out
    ctx.step(case["steps"])
    if case["kind"] == "step" and case["currents"]:
        out["currents"] = ctx.currents()
    if case["kind"] == "step" and case["coupled"]:
        out["E"], out["links"] = ctx.get_efield(), ctx.get_links()
    return out


# The bulk observables that are not rounding noise (the unitarity violation is) or a maximum over sites.
BULK = ("T00", "TXX", "TYY", "TZZ", "electric", "magnetic", "gauss_avg")


# ------------------------------------------------------------------- work --
def _hop_flops(nc):
    """One application of D per mode and site: six hops of (projection, two colour vectors times the link, sum)."""
    return 6 * (16 * nc * nc + 8 * nc) + 16 * nc


def work(case):
    if case["kind"] == "ensemble":
        one = [work(dict(kind="step", nc=case["nc"], n0=int(n), n1=int(n), n2=int(n), modes=case["modes"],
                         precision=case["precision"], steps=case["steps"], coupled=0.0, currents=False))
               for n in case["sizes"].split(",")]
        return {k: case["copies"] * sum(w[k] for w in one) for k in ("bytes", "flops")}
    nc, V, modes = case["nc"], math.prod(_dims(case)), case["modes"]
    element = 4 * nc * {"fp64": 16, "fp32": 8, "fp40": 10}[case["precision"]]  # bytes of one mode at one site
    field = modes * V * element
    gauge = 3 * V * 8 * ((18 + 8) if nc == 3 else (4 + 3))
    currents = 18 * 8 * V
    if case["kind"] == "step":
        # both fields read and written once per step; the links and E once
        n, flops = case["steps"], 2 * (_hop_flops(nc) + 16 * nc) * modes * V
        if case["coupled"]:
            flops += 3 * 64 * nc * nc * modes * V
        extra = currents if case["currents"] else 0
        return {"bytes": n * (4 * field + gauge) + extra, "flops": n * flops}
    if case["kind"] == "overlap":
        if case["sign"] == "chebyshev":
            # per half step: every Clenshaw vector written once and read once, phi read, the destination updated
            K = case["degree"]
            return {"bytes": 2 * case["steps"] * (3 * K + 6) * field,
                    "flops": 2 * case["steps"] * ((2 * K + 1) * _hop_flops(nc) + K * 48 * nc) * modes * V}
        # per half step and CG iteration (about 100 on these fields): two applications of D, 25 search directions
        # read and written, the residual
        its, poles = 100, 25
        return {"bytes": 2 * its * (2 * poles + 6) * field, "flops": 2 * its * (2 * _hop_flops(nc) + poles * 48 * nc) * modes * V}
    if case["kind"] == "currents":
        return {"bytes": field + gauge + currents, "flops": modes * V * (6 * 32 * nc * nc + 20 * 32 * nc)}
    return {"bytes": field + 4 * gauge, "flops": modes * V * (3 * 32 * nc * nc + 8 * 32 * nc)}


def tolerance(case):
    """About four times what exact() shows (a 2-norm error of 3e-8 per FP32 step, 1e-16 per FP64 step)."""
    precision = case["precision"]
    if case["kind"] == "overlap":
        if case["sign"] == "zolotarev":  # the CG stops at |r|^2 = 1e-16 |phi|, the Ritz bounds agree to 1e-12
            return {"rel": 2e-10, "max": 2e-8}
        return {"rel": 2e-7, "max": 1e-5} if precision == "fp32" else {"rel": 1e-14, "max": 1e-12}
    if case["kind"] in ("currents", "observe"):
        # FP64 sums of the stored modes; the vacuum weights make the sums small against their terms
        return {"rel": 5e-14, "max": 5e-12}
    if precision == "fp32":
        # the charges are vacuum-subtracted sums of FP32 modes
        return {"rel": 2e-6, "max": 1e-4} if case.get("observe") else {"rel": 5e-7, "max": 2e-5}
    if precision == "fp40":
        # currents of modes rounded to 2^-29 in every half step; the high words of the 40-bit numbers
        return {"rel": 2e-8, "max": 2e-6, "differ": 1e-3}
    return {"rel": 1e-14, "max": 1e-12}


# ------------------------------------------------------------------ exact --
# The operators in complex128.  Fields are [block, z, y, x, colour, spin, lane], links [z, y, x, mu, i, j].
# Dirac matrices as (permutation, power of i): (G psi)_a = i^ph[a] psi_perm[a].
G0 = ((0, 1, 2, 3), (0, 0, 2, 2))
GX = ((3, 2, 1, 0), (0, 0, 2, 2))
GY = ((3, 2, 1, 0), (3, 1, 1, 3))
GZ = ((2, 3, 0, 1), (0, 2, 2, 0))
G5 = ((2, 3, 0, 1), (0, 0, 0, 0))
GAMMA = (GX, GY, GZ)
PLANES = ((1, 2), (2, 0), (0, 1))


def _times(G, f, dim=5):
    perm, ph = G
    c = torch.tensor([1j ** p for p in ph], dtype=torch.complex128, device=f.device)
    return f.index_select(dim, torch.tensor(perm, device=f.device)) * c.view(-1, *([1] * (f.dim() - dim - 1)))


def _product(A, B):
    return tuple(B[0][A[0][a]] for a in range(4)), tuple((A[1][a] + B[1][A[0][a]]) % 4 for a in range(4))


def _shift(f, mu, n, first):
    """f(x + n mu); `first` is the dimension of z."""
    return torch.roll(f, -n, dims=first + 2 - mu)


def _link(M, f):
    """M(x) f(x): colour matrices [z, y, x, i, j] on fields."""
    nc = M.shape[-1]
    rows = [sum(M[..., i, j, None, None] * f[..., j, :, :] for j in range(nc)) for i in range(nc)]
    return torch.stack(rows, dim=4)


def _dag(M):
    return M.conj().transpose(-1, -2)


class _Exact:
    """Gauge fields of one trajectory and the operators on them, in 64 bits."""

    def __init__(self, case, N, seed, dt, m, mdw):
        self.nc, self.N, self.dt, self.m, self.mdw = case["nc"], N, dt, m, mdw
        U, E, u1 = _gauge(case, N, seed)
        shape = (N[2], N[1], N[0], 3)
        dev = "cuda"
        if self.nc == 3:
            U = torch.from_numpy(U).to(dev).view(*shape, 3, 3).transpose(-1, -2).contiguous()
        else:
            q = torch.from_numpy(U).to(dev).view(*shape, 4)
            rows = [torch.complex(q[..., 3], q[..., 2]), torch.complex(q[..., 1], q[..., 0]),
                    torch.complex(-q[..., 1], q[..., 0]), torch.complex(q[..., 3], -q[..., 2])]
            U = torch.stack(rows, -1).view(*shape, 2, 2)
        self.U, self.E = U, torch.from_numpy(E).to(dev).view(*shape, -1)
        self.phase = torch.ones(shape, dtype=torch.complex128, device=dev)
        if u1 is not None:
            self.phase[..., :2] = torch.from_numpy(u1).to(dev)[None]
        self.gen = _generators(self.nc).to(dev)
        self.amass = 6 * R_WILSON + 2 * m - 2 * mdw

    def algebra(self, E):
        return torch.einsum("...a,aij->...ij", E.to(torch.complex128), self.gen)

    def move_links(self, dt):
        self.U = torch.linalg.matrix_exp(-1j * dt * self.algebra(self.E)) @ self.U

    def dressed(self):
        return self.U * self.phase[..., None, None]

    def D(self, f):
        W, out = self.dressed(), self.amass * f
        for mu in range(3):
            fw = _link(W[..., mu, :, :], _shift(f, mu, 1, 1))
            bw = _shift(_link(_dag(W[..., mu, :, :]), f), mu, -1, 1)
            out = out - (fw + bw) - 1j * _times(GAMMA[mu], fw - bw)  # (1 - G) = 1 + i gamma, (1 + G) = 1 - i gamma
        return -0.5j * _times(G0, out)

    # ------------------------------------------------------------ overlap --
    def overlap(self, f, K, eps, lam, coeff):
        """-i h_ov f with chi = lam^(-1/2) sum c_k T_k(t(h^2 / lam)) f."""
        a, beta, s = 2 / ((1 - eps) * lam), -(1 + eps) / (1 - eps), 1 / math.sqrt(lam)
        b1 = b2 = None
        for k in range(K, -1, -1):
            new = ((coeff[k] if k else 0.5 * coeff[0]) * s) * f
            if b1 is not None:
                new += (2 if k else 1) * (-a * self.D(self.D(b1)) + beta * b1)
            if b2 is not None:
                new -= b2
            b1, b2 = new, b1
        return self.mdw * ((1 + 0.5 * self.m) * -1j * _times(G0, f) + (1 - 0.5 * self.m) * self.D(b1))

    # -------------------------------------------------------- observables --
    def currents(self, f, w):
        """The 18 densities per site of modes f with vacuum weights w[block, lane], summed over the modes."""
        V2 = 1.0 / (2 * math.prod(self.N))
        W, r = self.dressed(), R_WILSON
        wl = w[:, None, None, None, None, None, :]

        def bil(G, h):
            return (wl * f.conj() * _times(G, h)).sum(dim=(0, 4, 5, 6))

        G05, one = _product(G0, G5), ((0, 1, 2, 3), (0, 0, 0, 0))
        j = torch.zeros(*f.shape[1:4], 18, dtype=torch.float64, device=f.device)
        b05 = bil(G05, f).imag
        j[..., 0], j[..., 4], j[..., 16], j[..., 17] = bil(one, f).real, bil(G5, f).real, -b05, -6 * r * b05
        for mu in range(3):
            chi = _link(W[..., mu, :, :], _shift(f, mu, 1, 1))
            GV = _product(G0, GAMMA[mu])
            j[..., 1 + mu], j[..., 5 + mu] = bil(GV, chi).real, bil(_product(GV, G5), chi).real
            j[..., 9 + mu], j[..., 13 + mu] = r * bil(G0, chi).imag, r * bil(G05, chi).imag
            back = _shift(_link(_dag(W[..., mu, :, :]), f), mu, -1, 1)
            j[..., 17] += j[..., 13 + mu] + r * bil(G05, back).imag
        return V2 * j

    def fermion_force(self, f, w):
        """dH_F / dtheta^a_mu(x)."""
        wl, W, out = w[:, None, None, None, None, None, :], self.dressed(), []
        for mu in range(3):
            h = _shift(f, mu, 1, 1)
            h = _times(G0, h + 1j * _times(GAMMA[mu], h))
            C = torch.stack([torch.stack([((wl[..., 0, :, :] * f[..., i, :, :].conj()) * h[..., k, :, :]).sum(dim=(0, 4, 5))
                                          for k in range(self.nc)], -1) for i in range(self.nc)], -2)
            out.append(torch.einsum("aij,zyxjk,zyxik->zyxa", 1j * self.gen, W[..., mu, :, :], C).real)
        return torch.stack(out, 3) * (-1.0 / (2 * math.prod(self.N)))

    # Wilson loops as products of links along a path, based at x.
    def path(self, U, steps):
        n, acc = [0, 0, 0], None
        for mu, s in steps:
            if s < 0:
                n[mu] -= 1
            u = U[..., mu, :, :]
            for nu in range(3):
                u = _shift(u, nu, n[nu], 0)
            u = u if s > 0 else _dag(u)
            acc = u if acc is None else acc @ u
            if s > 0:
                n[mu] += 1
        return acc

    def loop(self, U, mu, nu, smu, snu, lmu, lnu):
        sides = [[(mu, 1)] * lmu, [(nu, 1)] * lnu, [(mu, -1)] * lmu, [(nu, -1)] * lnu]
        start = {(1, 1): 0, (-1, 1): 1, (-1, -1): 2, (1, -1): 3}[(smu, snu)]
        return self.path(U, sum((sides[(start + k) % 4] for k in range(4)), []))

    def re_tr_it(self, M):
        return (1j * torch.einsum("aij,...ji->...a", self.gen, M)).real

    def staple_force(self):
        out = []
        for mu in range(3):
            f = 0
            for nu in range(3):
                if nu != mu:
                    f = f + self.re_tr_it(self.path(self.U, [(mu, 1), (nu, 1), (mu, -1), (nu, -1)]))
                    f = f + self.re_tr_it(self.path(self.U, [(mu, 1), (nu, -1), (mu, -1), (nu, 1)]))
            out.append(-2 * f)
        return torch.stack(out, 3)

    def components(self, H):
        return 2 * torch.einsum("aij,...ji->...a", self.gen, H).real

    def ncsdot(self, U, E):
        total, EM = 0.0, self.algebra(E)
        for mu in range(3):
            u, e = U[..., mu, :, :], EM[..., mu, :, :]
            um = _dag(_shift(u, mu, -1, 0))
            umm = um @ _dag(_shift(u, mu, -2, 0))
            h = 7 / 12 * e - 1 / 12 * (u @ _shift(e, mu, 1, 0) @ _dag(u)) + 7 / 12 * (um @ _shift(e, mu, -1, 0) @ _dag(um))
            h = h - 1 / 12 * (umm @ _shift(e, mu, -2, 0) @ _dag(umm))
            avg = 0
            for s in ((1, 1), (-1, 1), (-1, -1), (1, -1)):
                p = PLANES[mu] + s
                avg = avg + 5 / 12 * self.loop(U, *p, 1, 1) - 1 / 24 * (self.loop(U, *p, 2, 1) + self.loop(U, *p, 1, 2))
            total += float((self.components(h) * 2 * self.re_tr_it(avg)).sum())
        return total / (8 * math.pi ** 2)

    def bulk(self):
        V = math.prod(self.N)
        e2 = [float((self.E[..., mu, :] ** 2).sum()) / V for mu in range(3)]
        b2 = [float(4 * (self.nc - self.loop(self.U, *PLANES[k], 1, 1, 1, 1).diagonal(dim1=-2, dim2=-1).sum(-1).real).sum()) / V
              for k in range(3)]
        g, EM = 0, self.algebra(self.E)
        for mu in range(3):
            u, e = _shift(self.U[..., mu, :, :], mu, -1, 0), _shift(EM[..., mu, :, :], mu, -1, 0)
            g = g + self.E[..., mu, :] - self.components(_dag(u) @ e @ u)
        t = [0.5 * (sum(e2) + sum(b2)) - (e2[k] + b2[k]) for k in range(3)]
        return np.array([0.5 * (sum(e2) + sum(b2)), *t, 0.5 * sum(e2), 0.5 * sum(b2),
                         math.sqrt(float((g ** 2).sum()) / ((3 if self.nc == 2 else 8) * V))])


def _generators(nc):
    if nc == 2:
        s = [[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]]
        return 0.5 * torch.tensor(s, dtype=torch.complex128)
    t = torch.zeros(8, 3, 3, dtype=torch.complex128)
    for a, (i, j) in zip((0, 3, 5), ((0, 1), (0, 2), (1, 2))):
        t[a, i, j] = t[a, j, i] = 0.5
        t[a + 1, i, j], t[a + 1, j, i] = -0.5j, 0.5j
    t[2, 0, 0], t[2, 1, 1] = 0.5, -0.5
    t[7] = torch.diag(torch.tensor([1, 1, -2], dtype=torch.complex128)) / (2 * math.sqrt(3))
    return t


def _inverse_sqrt_series(K, eps):
    """Chebyshev coefficients of x^(-1/2) on [eps, 1], by Gauss quadrature."""
    M = max(4 * K, 256)
    th = math.pi * (np.arange(M) + 0.5) / M
    f = 1 / np.sqrt(0.5 * (1 + eps) + 0.5 * (1 - eps) * np.cos(th))
    return [2 * float((f * np.cos(k * th)).sum()) / M for k in range(K + 1)]


def _weights(modes, blocks):
    m = torch.arange(blocks * LANES, device="cuda")
    w = torch.where(m % 2 == 0, 1.0, -1.0).double()
    return torch.where(m < modes, w, torch.zeros_like(w)).view(blocks, LANES)


def _as_field(f, N, nc):
    return torch.view_as_complex(f.double()).view(f.shape[0], N[2], N[1], N[0], nc, 4, LANES)


def _as_output(f, N, nc):
    return torch.view_as_real(f.reshape(f.shape[0], math.prod(N), 4 * nc, LANES))


def _by_blocks(f, chunk):
    return [slice(i, min(i + chunk, f.shape[0])) for i in range(0, f.shape[0], chunk)]


def _named(j):
    j = j.reshape(-1, 18).cpu().numpy()
    return {"jV": j[:, 0:4], "jA": j[:, 4:8], "jVw": np.concatenate([0 * j[:, :1], j[:, 9:12]], 1),
            "jAw": np.concatenate([0 * j[:, :1], j[:, 13:16]], 1), "PS": j[:, 16], "WA": j[:, 17]}


def exact(case, seed):
    if case["kind"] == "ensemble":
        sizes = [int(n) for n in case["sizes"].split(",")] * case["copies"]
        one = [_exact_one(dict(case, kind="step", m=0.05, dt=0.05, coupled=0.0, observe=False, currents=False, n0=n, n1=n,
                               n2=n), seed + 101 * i) for i, n in enumerate(sizes)]
        return {k: [o[k] for o in one] for k in ("psi", "mid")}
    return _exact_one(case, seed)


def _exact_one(case, seed):
    N, nc, modes = _dims(case), case["nc"], case["modes"]
    V, comp, blocks = math.prod(N), 4 * nc, -(-modes // LANES)
    x = _Exact(case, N, seed, case.get("dt", 0.05), case.get("m", 0.05), case.get("mdw", 0.0))
    w = _weights(modes, blocks)
    dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
    psi, mid = _random_modes(blocks, V, comp, modes, dtype, seed)
    chunk = max(1, int(1.2e8 / (V * comp * LANES)))  # about 2 GB of complex128 at a time
    if case["kind"] in ("currents", "observe"):
        if case["kind"] == "observe":
            old = x.U
            x.move_links(0.05)
        j = sum(x.currents(_as_field(psi[s], N, nc), w[s]) for s in _by_blocks(psi, chunk))
        if case["kind"] == "currents":
            return _named(j)
        # the path from the old links to the new: exp(-i A) = U_new U_old^+ is the motion itself
        A, half = 0.05 * x.E, torch.linalg.matrix_exp(-0.5j * x.algebra(0.05 * x.E)) @ old
        ncs = (4 * x.ncsdot(half, A) + x.ncsdot(old, A) + x.ncsdot(x.U, A)) / 6
        tot = j.sum(dim=(0, 1, 2))
        return {"charges": np.array([float(tot[k]) for k in (0, 4, 16, 17)]), "ncs": np.array([ncs]), "bulk": x.bulk()}
    if case["kind"] == "overlap":
        lam = (0.5 * abs(x.amass) + 3.0) ** 2
        K, eps = (case["degree"], 0.01) if case["sign"] == "chebyshev" else (900, 1.5e-4)
        coeff = _inverse_sqrt_series(K, eps)

        def rate(f):
            return x.overlap(f, K, eps, lam, coeff)
        if K * V * modes * comp > 4e9:
            return None
    else:
        rate = x.D
    # the whole step block by block needs the links of both half steps; they move without the modes unless coupled
    for _ in range(case["steps"]):
        for half, (dst, src) in enumerate(((psi, mid), (mid, psi))):
            if dst.dtype == torch.float32:  # from here on in 64 bits
                psi, mid = psi.double(), mid.double()
                dst, src = ((psi, mid), (mid, psi))[half]
            for s in _by_blocks(src, chunk):
                dst[s] += x.dt * _as_output(rate(_as_field(src[s], N, nc)), N, nc)
            x.move_links(0.5 * x.dt)
        if case.get("coupled"):
            force = x.staple_force()
            ferm = sum(x.fermion_force(_as_field(psi[s], N, nc), w[s]) for s in _by_blocks(psi, chunk))
            x.E = x.E + x.dt * force + x.dt * case["coupled"] * ferm
    out = {"psi": psi, "mid": mid}
    if case.get("observe") or case.get("currents"):
        j = sum(x.currents(_as_field(psi[s], N, nc), w[s]) for s in _by_blocks(psi, chunk))
        if case.get("observe"):
            tot = j.sum(dim=(0, 1, 2))
            out["charges"] = np.array([float(tot[k]) for k in (0, 4, 16)])
        else:
            out = {"psi": None, "mid": None, "currents": _named(j)}
    if case.get("coupled"):
        U = x.U
        out["E"] = x.E.reshape(V, 3, -1)
        if nc == 3:
            out["links"] = torch.view_as_real(U.transpose(-1, -2).reshape(V, 3, 9).contiguous())
        else:
            q = torch.stack([U[..., 0, 1].imag, U[..., 0, 1].real, U[..., 0, 0].imag, U[..., 0, 0].real], -1)
            out["links"] = q.reshape(V, 3, 4)
    return out
