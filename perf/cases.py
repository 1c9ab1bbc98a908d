"""What the framework is measured on: the calls its users make, over their real range.

A case is a dict of plain values; `prepare` makes what a program holds before
the call (planet, plans, model, seeded state on the GPU), `run` is one call
through the public entry points, `exact` the same result from plain torch in
64 bits.  Kinds:

  bve        one member (or a few) of the barotropic model, `model.rk4`
  swe        shallow water, `model.rk4` with its default state checks
  ensemble   uneven BVE ensemble: one captured RK4 step, replayed
  grad       gradient of a final-geopotential misfit through checkpointed
             RK4 steps (the hand-written adjoints behind torch.autograd)
  pe         primitive equations: one tendency (steps = 0) or RK4 steps
  transform  synthesis and analysis of a batch of fields on a point set
"""
import math

import numpy as np
import torch

import aeolus_gb300 as ae
from aeolus_gb300 import _lib
from aeolus_gb300.adjoint import swe_rk4_checkpointed, weighted_phi_misfit
from aeolus_gb300.barotropic import BarotropicVorticity
from aeolus_gb300.ensemble import BarotropicEnsemble
from aeolus_gb300.primitive_equations import PrimitiveEquationsModel, SigmaGrid
from aeolus_gb300.shallow_water import ShallowWaterModel

RADIUS = 6.371e6      # m
OMEGA = 7.292e-5      # 1/s
GRAVITY = 9.80616     # m/s^2
GH0 = 2.94e4          # m^2/s^2, Williamson-2
R_DRY, CP_DRY = 287.04, 1004.64
ENSEMBLE = ((42, 64, 128), (63, 96, 192), (85, 128, 256), (106, 160, 320), (127, 192, 384))


def listed():
    return [
        # the reference's own default run: BVE on the icosahedral grid of
        # resolution 4, products on the resolution-5 co-grid, one step per call
        {"name": "bve_geodesic4_l20", "kind": "bve", "grid": "geodesic", "res": 4, "lmax": 20, "members": 1,
         "split": False, "steps": 1},
        # the small interactive run: 32 x 64, l_max 21, one step per call
        # (a run layer reads diagnostics between steps)
        {"name": "bve_gauss_l21", "kind": "bve", "grid": "gauss", "nlat": 32, "nlon": 64, "lmax": 21, "members": 1,
         "split": False, "steps": 1},
        # one shallow-water run at medium resolution in FP64, one checked step
        # per call as the run layer makes it
        {"name": "swe_l85_fp64", "kind": "swe", "grid": "gauss", "nlat": 128, "nlon": 256, "lmax": 85, "members": 1,
         "split": False, "steps": 1},
        # the same run in split precision, ten steps per call
        {"name": "swe_l85_split", "kind": "swe", "grid": "gauss", "nlat": 128, "nlon": 256, "lmax": 85, "members": 1,
         "split": True, "steps": 10},
        # a state grid that just resolves l_max 63: its 3/2-rule product grid
        # is 95 x 190, an odd row count and a row length with a factor 19
        {"name": "swe_l63_ragged_fp64", "kind": "swe", "grid": "gauss", "nlat": 64, "nlon": 128, "lmax": 63,
         "members": 3, "split": False, "steps": 1},
        # a batch in plain FP64, the accuracy reference of the split runs
        {"name": "swe_l127_fp64_m8", "kind": "swe", "grid": "gauss", "nlat": 192, "nlon": 384, "lmax": 127,
         "members": 8, "split": False, "steps": 1},
        # the benchmark's workload: 64 members in split precision
        {"name": "swe_l127_split_m64", "kind": "swe", "grid": "gauss", "nlat": 192, "nlon": 384, "lmax": 127,
         "members": 64, "split": True, "steps": 1},
        # 256 members of uneven l_max, one captured step replayed
        {"name": "ensemble_256_split", "kind": "ensemble", "members": 256, "groups": 5, "split": True, "steps": 1},
        # 8 gradients at once through 8 steps with checkpoints every 4 (data assimilation)
        {"name": "grad_l127_split_m8", "kind": "grad", "nlat": 192, "nlon": 384, "lmax": 127, "members": 8,
         "split": True, "steps": 8, "every": 4},
        # primitive equations: a small FP64 run's step, and the large batched
        # split-precision tendency
        {"name": "pe_l42_k8_fp64", "kind": "pe", "nlat": 64, "nlon": 128, "lmax": 42, "levels": 8, "members": 1,
         "split": False, "steps": 1},
        {"name": "pe_l127_k20_split_m4", "kind": "pe", "nlat": 192, "nlon": 384, "lmax": 127, "levels": 20,
         "members": 4, "split": True, "steps": 0},
        # dense transforms on 40,962 icosahedral points, 64 fields at l_max 127
        {"name": "geodesic6_l127_f64_split", "kind": "transform", "res": 6, "lmax": 127, "fields": 64,
         "split": True},
    ]


# ------------------------------------------------------------------ drawing
def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _gauss_size(rng, lo=12, hi=127):
    """l_max and a state grid: either just resolving (its product grid is the
    ragged 3/2-rule one) or the 3/2-rule grid itself with rounded-up rows."""
    lmax = _log_int(rng, lo, hi)
    if rng.random() < 0.4:
        nlat, nlon = lmax + 1 + rng.randint(0, 2), 2 * lmax + 1 + rng.randint(0, 3)
    else:
        nlat, nlon = -(-(3 * lmax // 2 + 1) // 16) * 16, -(-(3 * lmax + 1) // 32) * 32
    return lmax, min(nlat, 192), nlon


def draw(rng):
    top = {c["kind"]: max(_cost(work(d)) for d in listed() if d["kind"] == c["kind"]) for c in listed()}
    kind = rng.choice(("bve", "bve", "swe", "swe", "swe", "swe", "ensemble", "grad", "pe", "pe", "transform"))
    while True:
        split = rng.random() < 0.5
        if kind in ("bve", "swe"):
            lmax, nlat, nlon = _gauss_size(rng)
            c = {"kind": kind, "grid": "gauss", "nlat": nlat, "nlon": nlon, "lmax": lmax,
                 "members": _log_int(rng, 1, 64 if split else 8), "split": split, "steps": rng.choice((1, 1, 2, 10))}
            if kind == "bve" and rng.random() < 0.4:
                res = rng.randint(2, 4)
                c = {"kind": kind, "grid": "geodesic", "res": res, "lmax": rng.randint(5, (8, 15, 30)[res - 2]),
                     "members": _log_int(rng, 1, 6), "split": split, "steps": 1}
            limit = top["swe"]
        elif kind == "ensemble":
            c = {"kind": kind, "members": _log_int(rng, 9, 256), "groups": rng.randint(2, 5), "split": split, "steps": 1}
            limit = top[kind]
        elif kind == "grad":
            lmax, nlat, nlon = _gauss_size(rng, 20)
            c = {"kind": kind, "nlat": nlat, "nlon": nlon, "lmax": lmax, "members": _log_int(rng, 1, 8),
                 "split": split, "steps": rng.randint(2, 8), "every": rng.randint(1, 4)}
            limit = top[kind] / (1 if split else 4)
        elif kind == "pe":
            lmax, nlat, nlon = _gauss_size(rng, 12, 126)
            c = {"kind": kind, "nlat": nlat, "nlon": nlon, "lmax": lmax, "levels": rng.randint(3, 30),
                 "members": _log_int(rng, 1, 4), "split": split, "steps": rng.choice((0, 0, 1))}
            limit = top[kind] / (1 if split else 4)
        else:
            res = rng.randint(3, 6)
            c = {"kind": kind, "res": res, "lmax": _log_int(rng, 8, (15, 30, 60, 127)[res - 3]),
                 "fields": _log_int(rng, 1, 64), "split": split}
            limit = top[kind] / (1 if split else 16)
        if "nlat" in c and c["split"] and max((3 * c["lmax"]) // 2 + 1, c["nlat"]) > 192:
            continue  # split precision takes up to 192 rows
        if _cost(work(c)) <= limit:
            return c


# ------------------------------------------------------------------- inputs
def _spectra(g, shape, lmax, slope, amp=1.0, monopole=False):
    """Coefficients of real fields ~ N(0,1) (l+1)^slope amp, [*shape, L+1, L+1]."""
    n = lmax + 1
    a = torch.randn(tuple(shape) + (n, n), dtype=torch.complex128, device="cuda", generator=g) * math.sqrt(2.0)
    a = a * (amp * (torch.arange(n, device="cuda", dtype=torch.float64) + 1.0) ** slope)[:, None]
    a[..., 0] = a[..., 0].real.to(torch.complex128)
    if not monopole:
        a[..., 0, :] = 0.0
    return a.tril()


def _rms(a):
    p = a.abs() ** 2
    return torch.sqrt((2.0 * p.sum((-2, -1)) - p[..., 0].sum(-1)) / (4.0 * math.pi))


def _williamson2(lmax):
    u0 = 2.0 * math.pi * RADIUS / (12.0 * 86400.0)
    c = RADIUS * OMEGA * u0 + 0.5 * u0 * u0
    s = torch.zeros((3, lmax + 1, lmax + 1), dtype=torch.complex128, device="cuda")
    s[0, 1, 0] = (2.0 * u0 / RADIUS) * math.sqrt(4.0 * math.pi / 3.0)
    s[2, 2, 0] = -(4.0 * c / 3.0) * math.sqrt(math.pi / 5.0)
    return s, (GH0 - c / 3.0) / GRAVITY


def _swe_states(lmax, members, seed):
    """Williamson-2 plus a 1 % seeded perturbation of every field, per member."""
    g = torch.Generator("cuda").manual_seed(seed)
    base, depth = _williamson2(lmax)
    p = _spectra(g, (members, 3), lmax, -2.0)
    ref = _rms(base)
    ref = torch.stack((ref[0], ref[0], ref[2]))
    return base + p * (0.01 * ref / _rms(p))[..., None, None], depth


def _bve_states(lmax, members, seed):
    return _spectra(torch.Generator("cuda").manual_seed(seed), (members,), lmax, -1.5, 1e-5)


def _pe_states(lmax, levels, members, seed):
    """Isothermal rest (260 K, 1013 hPa) plus band-limited perturbations of every field."""
    g = torch.Generator("cuda").manual_seed(seed)
    n, K, cut = lmax + 1, levels, (2 * lmax) // 3
    a = torch.randn((members, 3 * K + 1, n, n), dtype=torch.complex128, device="cuda", generator=g) * math.sqrt(2.0)
    a[..., 0] = a[..., 0].real.to(torch.complex128)
    a = a.tril()
    a[..., cut + 1:, :] = 0.0
    a[:, :2 * K] *= 2e-6
    a[:, 2 * K:3 * K] *= 0.5
    a[:, 3 * K] *= 1e-3
    a[:, :2 * K, 0, 0] = 0.0
    a[:, 3 * K, 0, 0] = 0.0
    mono = math.sqrt(4.0 * math.pi)
    a[:, 2 * K:3 * K, 0, 0] += 260.0 * mono
    a[:, 3 * K, 0, 0] += math.log(101325.0) * mono
    return a


def _time_step(lmax):
    return 240.0 * 127.0 / max(lmax, 21)


def _planet(case):
    if case.get("grid") == "geodesic":
        planet = ae.make_planet("geodesic", resolution=case["res"], l_max=case["lmax"])
    else:
        planet = ae.make_planet("latlon", nlat=case["nlat"], nlon=case["nlon"], l_max=case["lmax"])
    if case["split"]:
        planet.so._product_space.sh.plan.set_precision(_lib.PREC_SPLIT_BF16)
    return planet


def _groups(case):
    """(l_max, nlat, nlon, members) of the uneven ensemble's groups."""
    n, total = case["groups"], case["members"]
    return [ENSEMBLE[g] + (total // n + (1 if g < total % n else 0),) for g in range(n)]


def prepare(case, seed):
    kind, L = case["kind"], case.get("lmax", 0)
    s = {"case": case, "dt": _time_step(L)}
    if kind == "bve":
        s["model"] = BarotropicVorticity(_planet(case), viscosity=1e5)
        s["y"] = _bve_states(L, case["members"], seed)
    elif kind == "swe":
        s["y"], depth = _swe_states(L, case["members"], seed)
        s["model"] = ShallowWaterModel(_planet(case), gravity=GRAVITY, mean_depth=depth)
    elif kind == "ensemble":
        models, states = [], []
        for g, (L, nlat, nlon, b) in enumerate(_groups(case)):
            models.append(BarotropicVorticity(_planet({"nlat": nlat, "nlon": nlon, "lmax": L, "split": case["split"]}),
                                              viscosity=1e5))
            states.append(_bve_states(L, b, 1000 * seed + g))
        s["dt"] = 60.0  # stays stable over any number of replays
        s["ens"] = BarotropicEnsemble(models, [x.shape[0] for x in states])
        s["y"] = states
        s["ens"].capture(states, s["dt"])
    elif kind == "grad":
        s["y"], depth = _swe_states(L, case["members"], 2 * seed)
        s["model"] = ShallowWaterModel(_planet(case), gravity=GRAVITY, mean_depth=depth)
        other, _ = _swe_states(L, case["members"], 2 * seed + 1)
        s["target"] = s["model"].sh.inv_transform(other[:, 2])
    elif kind == "pe":
        s["model"] = PrimitiveEquationsModel(_planet(case), SigmaGrid.uniform(case["levels"]))
        s["y"] = _pe_states(L, case["levels"], case["members"], seed)
        s["dt"] = 60.0
    else:
        planet = ae.make_planet("geodesic", resolution=case["res"], l_max=L, product_quadrature="coarse")
        if case["split"]:
            planet.sh.plan.set_precision(_lib.PREC_SPLIT_BF16)
        s["sh"] = planet.sh
        g = torch.Generator("cuda").manual_seed(seed)
        s["a"] = _spectra(g, (case["fields"],), L, -1.5, monopole=True)
        s["f"] = torch.randn((case["fields"], planet.sh.n_points), dtype=torch.float64, device="cuda", generator=g)
    return s


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind in ("bve", "swe"):
        return s["model"].rk4(s["y"], s["dt"], c["steps"])
    if kind == "ensemble":
        s["ens"].replay(c["steps"])
        return s["y"]
    if kind == "grad":
        y = s["y"].clone().requires_grad_(True)
        m = s["model"]
        loss = weighted_phi_misfit(m, swe_rk4_checkpointed(m, y, s["dt"], c["steps"], c["every"]), s["target"])
        (grad,) = torch.autograd.grad(loss.sum(), y)
        return {"grad": grad, "loss": loss.detach()}
    if kind == "pe":
        m = s["model"]
        return m.rk4(s["y"], s["dt"], c["steps"]) if c["steps"] else m.tendency(s["y"])
    return {"grid": s["sh"].inv_transform(s["a"]), "coeffs": s["sh"].transform(s["f"])}


# --------------------------------------------------------------------- work
def _fine(c):
    if c.get("grid") == "geodesic":
        return None
    return max((3 * c["lmax"]) // 2 + 1, c["nlat"]), max(3 * c["lmax"] + 1, c["nlon"])


def _gauss_flops(nlat, nlon, lmax):
    """One real field: hemisphere-folded Legendre sums and the row FFTs."""
    return nlat * (lmax + 1.0) * (lmax + 2.0) + 2.5 * nlat * nlon * math.log2(nlon)


def _dense(npts, lmax):
    """(flops of one field, bytes of the FP64 basis) of one dense product."""
    return 2.0 * npts * (lmax + 1.0) ** 2, 8.0 * npts * (lmax + 1.0) ** 2


def _points(res):
    return 10 * 4 ** res + 2


def work(case):
    k, L = case["kind"], case.get("lmax", 0)
    tri = 16.0 * (L + 1) ** 2  # one dense spectrum
    if k == "transform":
        fl, by = _dense(_points(case["res"]), L)
        nf = case["fields"]
        return {"bytes": 2 * by + 2 * nf * (tri + 8.0 * _points(case["res"])), "flops": 2 * nf * fl}
    if k == "ensemble":
        by = fl = 0.0
        for L, nlat, nlon, b in _groups(case):
            by += 2 * 16.0 * (L + 1) ** 2 * b
            fl += 4 * 5 * b * _gauss_flops(nlat, nlon, L)
        return {"bytes": by * case["steps"], "flops": fl * case["steps"]}
    B = case["members"]
    if case.get("grid") == "geodesic":
        fl, by = _dense(_points(case["res"] + 1), L)
        n = 4 * case["steps"]
        return {"bytes": 2.0 * n * by + 2 * B * tri, "flops": n * 5 * B * fl}
    one = _gauss_flops(*_fine(case), L)
    table = 8.0 * _fine(case)[0] * (L + 1.0) * (L + 2.0) / 4
    if k == "pe":
        K, n = case["levels"], max(1, 4 * case["steps"])
        fields = (8 * K + 2) + (4 * K + 1) + 2 * K
        return {"bytes": n * 2 * table + 2 * B * (3 * K + 1) * tri, "flops": n * B * fields * one}
    n = 4 * case["steps"]
    if k == "grad":  # forward, segment recomputation, stage recomputation and four VJPs per step
        n = case["steps"] * (4 + 4 + 3)
        fl = (n * 11 + case["steps"] * 4 * 20) * one
        return {"bytes": 2 * B * 3 * tri + 2 * table, "flops": B * fl}
    nf = 3 if k == "swe" else 1
    return {"bytes": 2 * table + 2 * B * nf * tri, "flops": n * B * (11 if k == "swe" else 5) * one}


def _cost(w):
    return max(w["bytes"], w["flops"] / 50)


# ------------------------------------------------- the same in plain 64 bits
_CACHE = {}


def _legendre_table(x, s, L):
    """Normalised P_lm(x) e^0 with the Condon-Shortley sign, [points, L+1 (l), L+1 (m)]."""
    p = torch.zeros((L + 1, L + 1) + x.shape, dtype=torch.float64, device=x.device)
    pmm = torch.full_like(x, math.sqrt(1.0 / (4.0 * math.pi)))
    for m in range(L + 1):
        if m:
            pmm = -math.sqrt((2.0 * m + 1.0) / (2.0 * m)) * s * pmm
        p[m, m] = pmm
    m = torch.arange(L + 1, dtype=torch.float64, device=x.device)
    for l in range(1, L + 1):
        mm = m[:l]
        a = torch.sqrt((4.0 * l * l - 1.0) / (l * l - mm * mm))[:, None]
        b = torch.sqrt(((l - 1.0) ** 2 - mm * mm).clamp(min=0.0) / (4.0 * (l - 1.0) ** 2 - 1.0))[:, None]
        p[l, :l] = a * (x * p[l - 1, :l] - (b * p[l - 2, :l] if l > 1 else 0.0))
    return p


def _gauss_nodes(n):
    """cos(colatitude) north to south and weights (sum 2), Newton in extended precision."""
    t = np.longdouble
    k = np.arange(n, dtype=t)
    th = (k + t(0.75)) / (t(n) + t(0.5)) * np.arccos(t(-1.0))
    x = np.cos(th)
    for _ in range(12):
        p0, p1 = np.ones_like(x), x
        for l in range(2, n + 1):
            p0, p1 = p1, ((2 * l - 1) * x * p1 - (l - 1) * p0) / t(l)
        d = n * (x * p1 - p0) / (x * x - 1)
        x = x - p1 / d
    w = 2 / ((1 - x * x) * d * d)
    return x.astype(np.float64), np.sqrt((1 - x) * (1 + x)).astype(np.float64), w.astype(np.float64)


class _Space:
    """Transforms of one sampling; the dealiased products live here."""

    def _metric(self, L):
        self.L = L
        n = L + 1
        l = torch.arange(n, dtype=torch.float64, device="cuda")[:, None]
        m = torch.arange(n, dtype=torch.float64, device="cuda")[None, :]
        ok = m <= l
        cp = torch.where(ok, l * torch.sqrt(((l + 1) ** 2 - m ** 2).clamp(min=0) / ((2 * l + 1) * (2 * l + 3))), 0.0)
        cm = torch.where(ok, -(l + 1) * torch.sqrt((l ** 2 - m ** 2).clamp(min=0) / ((2 * l - 1) * (2 * l + 1)).clamp(min=1)), 0.0)
        cm[0] = 0.0
        self.cp_true = cp
        self.cp, self.cm = cp.clone(), cm
        self.cp[L] = 0.0
        self.lap = (-l * (l + 1.0) / RADIUS ** 2)
        self.ilap = torch.zeros_like(self.lap)
        self.ilap[1:] = 1.0 / self.lap[1:]
        self.im = 1j * m / RADIUS
        cut = (2 * L) // 3
        self.keep = ((l <= cut) & (m <= cut)).to(torch.float64)

    def lam(self, a):
        return self.synth(self.im * a)

    def snt(self, a):
        z = torch.zeros_like(a[..., :1, :])
        up = torch.cat((z, (self.cp * a)[..., :-1, :]), -2)
        return self.synth((up + torch.cat(((self.cm * a)[..., 1:, :], z), -2)) / RADIUS)

    def cut(self, a):
        return a * self.keep


class _Gauss(_Space):
    def __init__(self, nlat, nlon, L):
        self._metric(L)
        x, s, w = (torch.from_numpy(v).cuda() for v in _gauss_nodes(nlat))
        self.P = _legendre_table(x, s, L).permute(1, 2, 0).contiguous()  # [m, j, l]
        k = torch.arange(nlon, device="cuda")[:, None] * torch.arange(L + 1, device="cuda")[None, :] % nlon
        ang = k.to(torch.float64) * (2.0 * math.pi / nlon)
        self.c, self.s = torch.cos(ang), torch.sin(ang)
        self.w = w * (2.0 * math.pi / nlon)
        self.shape = (nlat, nlon)
        self.cos = s.clamp(min=1e-8).repeat_interleave(nlon)
        self.weights = self.w.repeat_interleave(nlon)

    def synth(self, a):
        lead = a.shape[:-2]
        v = torch.view_as_real(a.reshape((-1,) + a.shape[-2:]).permute(2, 1, 0).contiguous())  # [m, l, b, 2]
        f = torch.bmm(self.P, v.reshape(v.shape[0], v.shape[1], -1))          # [m, j, b*2]
        f = f.reshape(f.shape[0], f.shape[1], -1, 2).permute(2, 1, 0, 3)                        # [b, j, m, 2]
        two = torch.full((self.L + 1,), 2.0, dtype=torch.float64, device="cuda")
        two[0] = 1.0
        g = (f[..., 0] * two) @ self.c.T - (f[..., 1] * two) @ self.s.T
        return g.reshape(lead + (-1,))

    def anal(self, g):
        lead = g.shape[:-1]
        x = g.reshape((-1,) + self.shape) * self.w[:, None]
        f = torch.stack((x @ self.c, -(x @ self.s)), -1).permute(2, 1, 0, 3).contiguous()       # [m, j, b, 2]
        a = torch.bmm(self.P.transpose(1, 2), f.reshape(f.shape[0], f.shape[1], -1))            # [m, l, b*2]
        a = torch.view_as_complex(a.reshape(a.shape[0], a.shape[1], -1, 2).contiguous()).permute(2, 1, 0)
        return a.reshape(lead + a.shape[1:])


class _Points(_Space):
    """Dense products on given points (latitudes, longitudes, weights are inputs)."""

    def __init__(self, lat, lon, w, L):
        self._metric(L)
        self.tri = torch.tril_indices(L + 1, L + 1, device="cuda")
        self.lat, self.lon, self.weights = lat, lon, w
        self.cos = torch.cos(lat).clamp(min=1e-8)

    def _blocks(self):
        l, m = self.tri
        for i in range(0, self.lat.numel(), 8192):
            la, lo = self.lat[i:i + 8192], self.lon[i:i + 8192]
            p = _legendre_table(torch.sin(la), torch.cos(la), self.L)[l, m]
            e = lo[None, :] * m[:, None].to(torch.float64)
            yield slice(i, i + la.numel()), p * torch.cos(e), p * torch.sin(e)

    def synth(self, a):
        lead = a.shape[:-2]
        v = a.reshape((-1,) + a.shape[-2:])[:, self.tri[0], self.tri[1]]
        v = v * torch.where(self.tri[1] > 0, 2.0, 1.0)
        out = [v.real @ c - v.imag @ s for _, c, s in self._blocks()]
        return torch.cat(out, -1).reshape(lead + (-1,))

    def anal(self, g):
        lead = g.shape[:-1]
        x = (g * self.weights).reshape(-1, g.shape[-1])
        v = 0.0
        for i, c, s in self._blocks():
            v = v + torch.complex(x[:, i] @ c.T, -(x[:, i] @ s.T))
        a = torch.zeros((x.shape[0], self.L + 1, self.L + 1), dtype=torch.complex128, device="cuda")
        a[:, self.tri[0], self.tri[1]] = v
        return a.reshape(lead + a.shape[1:])


def _space(key, make):
    if key not in _CACHE:
        if len(_CACHE) > 6:
            _CACHE.clear()
        _CACHE[key] = make()
    return _CACHE[key]


def _gauss(nlat, nlon, L):
    return _space((nlat, nlon, L), lambda: _Gauss(nlat, nlon, L))


def _product_space(case):
    if case.get("grid") == "geodesic":
        # the co-grid's points and cell weights are inputs of the transform
        sh = _planet(case).so.backend.product_space("fine").sh
        return _Points(sh.latitudes, sh.longitudes, sh.weights, case["lmax"])
    return _gauss(*_fine(case), case["lmax"])


def _f_lm(L):
    f = torch.zeros((L + 1, L + 1), dtype=torch.complex128, device="cuda")
    f[1, 0] = 2.0 * OMEGA * math.sqrt(4.0 * math.pi / 3.0)
    return f


def _bve_rhs(sp, z):
    psi, eta = sp.ilap * z, z + _f_lm(sp.L)
    j = (sp.snt(psi) * sp.lam(eta) - sp.lam(psi) * sp.snt(eta)) / sp.cos ** 2
    k = -sp.cut(sp.anal(j)) + 1e5 * sp.lap * z
    k[..., 0, :] = 0.0
    return k


def _swe_rhs(sp, y, phi0):
    z, d, ph = y.unbind(-3)
    psi, chi, eta = sp.ilap * z, sp.ilap * d, z + _f_lm(sp.L)
    u, v = (sp.snt(psi) + sp.lam(chi)) / sp.cos, (sp.lam(psi) - sp.snt(chi)) / sp.cos
    el, es, pl, ps = sp.lam(eta), sp.snt(eta), sp.lam(ph), sp.snt(ph)
    eg, zg, dg, pg = sp.synth(eta), sp.synth(z), sp.synth(d), sp.synth(ph)
    a = sp.cut(sp.anal(torch.stack((-((u * el - v * es) / sp.cos + eg * dg), eg * zg + (v * el + u * es) / sp.cos,
                                    0.5 * (u * u + v * v), -((u * pl - v * ps) / sp.cos + pg * dg)), -2)))
    k = torch.stack((a[..., 0, :, :], a[..., 1, :, :] - sp.lap * (a[..., 2, :, :] + ph), a[..., 3, :, :] - phi0 * d), -3)
    row = torch.ones((sp.L + 1, 1), dtype=torch.float64, device="cuda")
    row[0] = 0.0
    return k * row


def _pe_rhs(sp, ext, y, K):
    z, d, t, lp = y[..., :K, :, :], y[..., K:2 * K, :, :], y[..., 2 * K:3 * K, :, :], y[..., 3 * K, :, :]
    s = [k / K for k in range(K + 1)]
    ds = [s[k + 1] - s[k] for k in range(K)]
    beta = [0.0] + [math.log(s[k + 1] / s[k]) for k in range(1, K)]
    alpha = [math.log(2.0)] + [1.0 - (s[k] / ds[k]) * beta[k] for k in range(1, K)]
    psi, chi, eta = sp.ilap * z, sp.ilap * d, z + _f_lm(sp.L)
    u, v = (sp.snt(psi) + sp.lam(chi)) / sp.cos, (sp.lam(psi) - sp.snt(chi)) / sp.cos
    ll, ls = sp.lam(lp)[..., None, :], sp.snt(lp)[..., None, :]
    zg, dg, tg, eg = sp.synth(z), sp.synth(d), sp.synth(t), sp.synth(eta)
    A = (u * ll - v * ls) / sp.cos
    G = dg + A
    dsv = torch.tensor(ds, dtype=torch.float64, device="cuda")[:, None]
    part = torch.cumsum(dsv * G, -2)
    total = part[..., -1:, :]
    zero = torch.zeros_like(total)
    sd = torch.cat([zero] + [s[k] * total - part[..., k - 1:k, :] for k in range(1, K)] + [zero], -2)
    before = torch.cat((zero, part[..., :-1, :]), -2)
    bd = torch.tensor([beta[k] / ds[k] for k in range(K)], dtype=torch.float64, device="cuda")[:, None]
    al = torch.tensor(alpha, dtype=torch.float64, device="cuda")[:, None]
    wp = A - bd * before - al * G

    def vadv(x):
        dx = x[..., 1:, :] - x[..., :-1, :]
        f = sd[..., 1:-1, :] * dx
        return (torch.cat((f, zero), -2) + torch.cat((zero, f), -2)) / (2.0 * dsv)

    kappa = R_DRY / CP_DRY
    td = sp.cut(sp.anal(-(u * sp.lam(t) - v * sp.snt(t)) / sp.cos - vadv(tg) + kappa * tg * wp))
    lpd = sp.cut(sp.anal(-total[..., 0, :]))
    el, es = sp.lam(eta), sp.snt(eta)
    zd = sp.cut(sp.anal(-((u * el - v * es) / sp.cos + eg * dg)))
    dd = sp.cut(sp.anal(eg * zg + (v * el + u * es) / sp.cos))
    ke = sp.cut(sp.anal(0.5 * (u * u + v * v)))
    n = sp.L + 1
    a = ext.anal((vadv(u) + R_DRY * tg * ll / sp.cos) / sp.cos)
    b = ext.anal((vadv(v) - R_DRY * tg * ls / sp.cos) / sp.cos)

    def snt_t(c):
        o = sp.cp_true * c[..., 1:n + 1, :n]
        z0 = torch.zeros_like(o[..., :1, :])
        return (o + torch.cat((z0, sp.cm[1:] * c[..., :n - 1, :n]), -2)) / RADIUS

    div, curl = sp.im * a[..., :n, :n] + snt_t(b), sp.im * b[..., :n, :n] - snt_t(a)
    below, phi = torch.zeros_like(t[..., 0, :, :]), [None] * K
    for k in range(K - 1, -1, -1):
        phi[k] = below + R_DRY * alpha[k] * t[..., k, :, :]
        below = below + R_DRY * beta[k] * t[..., k, :, :]
    zd = sp.cut(zd - curl)
    dd = sp.cut(dd - div) - sp.lap * (ke + torch.stack(phi, -3))
    zd[..., 0, :] = 0.0
    dd[..., 0, :] = 0.0
    return torch.cat((zd, dd, td, lpd[..., None, :, :]), -3)


def _rk4(rhs, y, dt, steps):
    for _ in range(steps):
        k1 = rhs(y)
        k2 = rhs(y + 0.5 * dt * k1)
        k3 = rhs(y + 0.5 * dt * k2)
        k4 = rhs(y + dt * k3)
        y = y + (dt / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
    return y


def exact(case, seed):
    kind, L = case["kind"], case.get("lmax", 0)
    dt = _time_step(L)
    if kind == "bve":
        sp = _product_space(case)
        return _rk4(lambda y: _bve_rhs(sp, y), _bve_states(L, case["members"], seed), dt, case["steps"])
    if kind == "ensemble":
        out = []
        for g, (L, nlat, nlon, b) in enumerate(_groups(case)):
            sp = _gauss(nlat, nlon, L)
            out.append(_rk4(lambda y: _bve_rhs(sp, y), _bve_states(L, b, 1000 * seed + g), 60.0, case["steps"]))
        return out
    if kind == "swe":
        y, depth = _swe_states(L, case["members"], seed)
        sp = _product_space(case)
        # a few members at a time: the grid fields of all stages fit easily
        return torch.cat([_rk4(lambda x: _swe_rhs(sp, x, GRAVITY * depth), p, dt, case["steps"]) for p in y.split(16)])
    if kind == "grad":
        y, depth = _swe_states(L, case["members"], 2 * seed)
        other, _ = _swe_states(L, case["members"], 2 * seed + 1)
        sp, st = _product_space(case), _gauss(case["nlat"], case["nlon"], L)
        target = st.synth(other[:, 2])
        grads, losses = [], []
        for p, t in zip(y.split(1), target.split(1)):
            p = p.clone().requires_grad_(True)
            end = _rk4(lambda x: _swe_rhs(sp, x, GRAVITY * depth), p, dt, case["steps"])
            loss = ((st.synth(end[:, 2]) - t) ** 2 * st.weights).sum(-1)
            grads.append(torch.autograd.grad(loss.sum(), p)[0].tril())
            losses.append(loss.detach())
        return {"grad": torch.cat(grads), "loss": torch.cat(losses)}
    if kind == "pe":
        K = case["levels"]
        sp, ext = _product_space(case), _gauss(*_fine(case), L + 1)
        outs = []
        for p in _pe_states(L, K, case["members"], seed).split(1):
            rhs = lambda x: _pe_rhs(sp, ext, x, K)  # noqa: E731
            outs.append(_rk4(rhs, p, 60.0, case["steps"]) if case["steps"] else rhs(p))
        return torch.cat(outs)
    s = prepare(dict(case, split=False), seed)
    sp = _Points(s["sh"].latitudes, s["sh"].longitudes, s["sh"].weights, L)
    return {"grid": sp.synth(s["a"]), "coeffs": sp.anal(s["f"])}
