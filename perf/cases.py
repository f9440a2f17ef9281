"""Performance cases: what a user of gbflow has it do, through its public entry points.

Every case is a stretch of a simulation: a state in hand (a DNAPL plume in a
water-saturated grid, pressure off hydrostatic), some time steps, the new
pressure and saturation read back. `run` starts from the same state each time,
so a pass is upload + steps + read-back, as between two outputs of a run.

listed(), draw(rng): the cases; prepare(case, seed): inputs and the grid
object a program keeps; run(state): one pass; work(case): the bytes and
operations it cannot do without; exact(case, seed): the same steps in plain
64-bit torch (increments and log1p/expm1 forms, so that nothing cancels).
"""
import ctypes
import math
import types
from importlib import import_module

import numpy as np
import torch

from __graft_entry__ import load_package

PKG = load_package()
abi = PKG.abi
wl = import_module(PKG.__name__ + ".workloads")
Domain = import_module(PKG.__name__ + ".domain").Domain
Ensemble = import_module(PKG.__name__ + ".ensemble").Ensemble
dropin = import_module(PKG.__name__ + ".dropin")

PRECISION = {"f64": abi.GBF_PREC_F64, "split": abi.GBF_PREC_SPLIT, "split_df": abi.GBF_PREC_SPLIT_DF,
             "split_defect": abi.GBF_PREC_SPLIT_DEFECT}


def listed():
    return [
        # The reference driver's own grid through its five calls, one kernel each (the drop-in's default
        # mode): the smallest calls, bound by launches and latency.
        {"name": "dropin_eager_15", "kind": "dropin", "mode": 0, "nx": 15, "ny": 15, "nz": 15, "steps": 16,
         "fields": False, "patch": True, "ini": True},
        # The same mode on a laboratory-tank grid with two media, ragged sides.
        {"name": "dropin_eager_100x84x61", "kind": "dropin", "mode": 0, "nx": 100, "ny": 84, "nz": 61, "steps": 8,
         "fields": False, "patch": True, "ini": True},
        # The five calls as one fused FP64 step (GBF_DROPIN_MODE=1).
        {"name": "dropin_fused_128x112x120", "kind": "dropin", "mode": 1, "nx": 128, "ny": 112, "nz": 120,
         "steps": 8, "fields": False, "patch": True, "ini": True},
        # The five calls in split mode on the benchmark's drop-in grid: 16.8M cells, media table.
        {"name": "dropin_split_256", "kind": "dropin", "mode": 2, "nx": 256, "ny": 256, "nz": 256, "steps": 20,
         "fields": False, "patch": True, "ini": False},
        # Config 0 (40^3, homogeneous) in the default precision: a small grid's step latency.
        {"name": "domain_f64_config0_40", "kind": "domain", "prec": "f64", "nx": 40, "ny": 40, "nz": 40, "steps": 40,
         "fields": False, "patch": False, "ini": False},
        # Config 1 (256^3, heterogeneous K and porosity) in the default precision.
        {"name": "domain_f64_config1_256", "kind": "domain", "prec": "f64", "nx": 256, "ny": 256, "nz": 256,
         "steps": 4, "fields": True, "patch": False, "ini": False},
        # Config 1 in the split form, every step's phase masses kept.
        {"name": "domain_split_config1_256", "kind": "domain", "prec": "split", "nx": 256, "ny": 256, "nz": 256,
         "steps": 30, "fields": True, "patch": False, "ini": False},
        # Config 2, the largest single grid (67M cells).
        {"name": "domain_split_config2_512", "kind": "domain", "prec": "split", "nx": 512, "ny": 512, "nz": 256,
         "steps": 20, "fields": True, "patch": False, "ini": False},
        # A grid whose sides fit no tile (measured fields come in such sizes).
        {"name": "domain_split_odd_151x97x83", "kind": "domain", "prec": "split", "nx": 151, "ny": 97, "nz": 83,
         "steps": 40, "fields": True, "patch": False, "ini": False},
        # A slice of config 4's Monte-Carlo ensemble (24 of its 256 realizations), state resident.
        {"name": "ensemble_split_config4_24", "kind": "ensemble", "prec": "split", "members": 24, "config": 4,
         "steps": 16, "host": False},
        # A few realizations in plain FP64 (the accuracy baseline of an ensemble study).
        {"name": "ensemble_f64_config3_4", "kind": "ensemble", "prec": "f64", "members": 4, "config": 3, "steps": 2,
         "host": False},
        # Host-resident ensemble: upload, one step, download in one pipelined call (the benchmark's end-to-end path).
        {"name": "ensemble_host_config3_16", "kind": "ensemble", "prec": "split", "members": 16, "config": 3,
         "steps": 1, "host": True},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["dropin", "domain", "domain", "ensemble"])
    if kind == "ensemble":
        prec = rng.choice(["f64", "split", "split", "split_df", "split_defect"])
        return {"kind": "ensemble", "prec": prec, "members": size(2, 8 if prec == "f64" else 32),
                "config": rng.choice([3, 4]), "steps": rng.randint(1, 3), "host": rng.random() < 0.3}
    if kind == "dropin":
        mode = rng.choice([0, 1, 2])
        hi = (96, 160, 256)[mode]
        return {"kind": "dropin", "mode": mode, "nx": size(11, hi), "ny": size(11, hi), "nz": size(11, hi),
                "steps": rng.randint(4, 16), "fields": False, "patch": True, "ini": rng.random() < 0.7}
    prec = rng.choice(["f64", "split", "split", "split_df", "split_defect"])
    hi = 160 if prec == "f64" else 320
    return {"kind": "domain", "prec": prec, "nx": size(13, hi), "ny": size(13, hi), "nz": size(13, hi),
            "steps": rng.randint(4, 16), "fields": rng.random() < 0.7, "patch": rng.random() < 0.3,
            "ini": rng.random() < 0.3}


# ------------------------------------------------------------------ inputs


def _smooth(gen, shape, corr=8):
    """A smooth field of zero mean and unit variance: noise every `corr` cells, interpolated."""
    coarse = [max(3, n // corr + 2) for n in shape]
    a = torch.randn([1, 1] + coarse, generator=gen, device="cuda", dtype=torch.float32)
    a = torch.nn.functional.interpolate(a, size=list(shape), mode="trilinear", align_corners=True)[0, 0]
    return (a - a.mean()) / a.std()


def _dt(m, K, phi, media, safety=0.5):
    """Half the explicit scheme's pressure-diffusion bound (what gbf_stable_dt gives a program)."""
    worst = 0.0
    for md in (0, 1):
        swr, lam = m.S_wr[md], m.lam[md]
        cap = min(m.S2_gr, 1 - swr) if m.source_mode == abi.GBF_SOURCE_DIRICHLET_PATCH else 1 - swr
        s = np.linspace(0.0, cap, 257)
        se = np.maximum(0.0, (1 - s - swr) / (1 - swr))
        kr1 = se ** ((2 + 3 * lam) / lam)
        kr2 = (1 - se) ** 2 * (1 - se ** ((2 + lam) / lam))
        ratio = float(((kr1 / m.mu1 + kr2 / m.mu2) / ((1 - s) * m.beta1 + s * m.beta2)).max())
        if K is not None:
            worst = max(worst, ratio * float((K / phi).max()) if md == 0 else 0.0)
        elif md == 0 or media is not None:
            worst = max(worst, ratio * m.K[md] / m.m[md])
    return safety / (2 * worst * (1 / m.h1 ** 2 + m.kv / m.h2 ** 2 + 1 / m.h3 ** 2))


def _grid(n, seed, *, fields, patch, ini, sigma=1.0, rate=5e-3, rate_cells=4, length=10.0, lam=2.7, P_d=755.0,
          kv=1.0, dropin_physics=False):
    """One grid's model, cell fields and state on the GPU, from the seed alone."""
    nx, ny, nz = n
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if patch or dropin_physics:  # the reference's rules: Dirichlet patch at the top centre, its boundary copies
        m = abi.reference_model(nx, ny, nz, 1.0)
        m.source = min(3, (min(nx, nz) - 3) // 2)
        if not ini:
            m.h1 = m.h2 = m.h3 = length / max(n)
    else:  # mass-rate injection at the top centre, hydrostatic sides, no-flow bottom
        m = wl.base_model(n, length, rate, min(rate_cells, nx - 2, nz - 2), lam=lam, P_d=P_d, kv=kv)
        m.h1 = m.h2 = m.h3 = length / max(n)
    if ini:
        m.beta1, m.beta2 = 1e-4, 1e-8
    elif patch or dropin_physics:
        m.beta1 = m.beta2 = 1e-9
    if not dropin_physics:
        m.newton_tol = 1e-11
    K = phi = media = None
    shape = (nz, ny, nx)
    if fields:
        K = (6.64e-11 * torch.exp(sigma * _smooth(gen, shape))).float()
        phi = (0.35 + 0.05 * (2 * torch.rand(shape, generator=gen, device="cuda") - 1)).float()
    elif patch or dropin_physics:
        media = (_smooth(gen, shape) > 0.8).to(torch.int32)
    m.dt = _dt(m, K, phi, media)
    # the plume: below the top centre, S up to about 0.35, exactly 0 outside
    z, y, x = (torch.linspace(-1, 1, k, device="cuda", dtype=torch.float64) for k in shape)
    r2 = (x[None, None, :] / 0.45) ** 2 + ((y[None, :, None] + 0.7) / 0.8) ** 2 + (z[:, None, None] / 0.45) ** 2
    S = (0.35 * (torch.exp(-r2) - 0.1).clamp(min=0.0) * (1 + 0.1 * _smooth(gen, shape).double()).clamp(0.6, 1.4))
    j = torch.arange(ny, device="cuda", dtype=torch.float64)[None, :, None]
    P = m.P_atm + j * (m.ro01 * m.g * m.h2) + 50.0 * _smooth(gen, shape).double() + 200.0 * torch.exp(-r2)
    return types.SimpleNamespace(m=m, K=K, phi=phi, media=media, P=P.contiguous(), S=S.contiguous())


def _member_grids(case, seed):
    specs = (wl.config3_specs if case["config"] == 3 else wl.config4_specs)(case["members"])
    for q, s in enumerate(specs):
        e = s["edge"]
        yield _grid((e, e, e), seed * 1000 + q, fields=True, patch=False, ini=False, sigma=min(s["sigma_lnK"], 1.5),
                    rate=s["rate"], length=e / 32.0, lam=s.get("lambda", 2.7), P_d=s.get("P_d", 755.0),
                    kv=s.get("kv", 1.0))


def _case_grid(case, seed):
    return _grid((case["nx"], case["ny"], case["nz"]), seed, fields=case["fields"], patch=case["patch"],
                 ini=case["ini"], dropin_physics=case["kind"] == "dropin")


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _host(t):
    return None if t is None else t.cpu().numpy()


# ------------------------------------------------------------------ states


class _DomainState:
    """A gbf_domain between two outputs of a run; P, S start on the device and end in pinned host arrays."""

    def __init__(self, case, seed):
        g = _case_grid(case, seed)
        self.steps, self.P, self.S = case["steps"], g.P, g.S
        self.dom = Domain(g.m, _host(g.media), _host(g.K), _host(g.phi), precision=PRECISION[case["prec"]])
        self.dom.set_outputs(abi.GBF_OUT_MASS, self.steps)
        self.out = [_pinned(g.m.ncells).reshape(g.m.shape) for _ in range(2)]

    def run(self):
        d = self.dom
        d.upload_device(self.P.data_ptr(), self.S.data_ptr())
        d.step(self.steps)
        return {"P1": d.download("P1", self.out[0]), "S2": d.download("S2", self.out[1]),
                "masses": d.mass_history(self.steps)}


class _EnsembleState:
    """A gbf_ensemble: resident (state packed on the device) or host-resident (pinned host arrays)."""

    def __init__(self, case, seed):
        self.steps, self.host = case["steps"], case["host"]
        P, S, members = [], [], []
        for g in _member_grids(case, seed):
            P.append(g.P.reshape(-1))
            S.append(g.S.reshape(-1))
            members.append(types.SimpleNamespace(model=g.m, K=_host(g.K), phi=_host(g.phi)))
        self.P, self.S = torch.cat(P), torch.cat(S)
        self.ens = Ensemble(members, precision=PRECISION[case["prec"]])
        if case["prec"] != "f64":
            self.ens.set_tuning(5 if case["config"] == 4 else 4)  # the shapes the autotuner picks on these ensembles
        if self.host:
            self.hin = [_pinned(t.numel()) for t in (self.P, self.S)]
            for h, t in zip(self.hin, (self.P, self.S)):
                torch.from_numpy(h).copy_(t)
            self.out = [_pinned(self.P.numel()) for _ in range(2)]
        else:
            self.ens.set_outputs(abi.GBF_OUT_MASS, self.steps)
            self.out = [torch.empty_like(self.P) for _ in range(2)]

    def run(self):
        e = self.ens
        if self.host:
            e.advance_host(self.hin[0], self.hin[1], self.steps, self.out[0], self.out[1])
            return {"P1": self.out[0], "S2": self.out[1]}
        abi.check(e.lib.gbf_ensemble_upload_all(e.h, self.P.data_ptr(), self.S.data_ptr()))
        e.step(self.steps)
        abi.check(e.lib.gbf_ensemble_download_all(e.h, self.out[0].data_ptr(), self.out[1].data_ptr()))
        return {"P1": self.out[0], "S2": self.out[1], "masses": e.mass_history(self.steps)}


class _DropinState:
    """The reference's host function set, driven as its main program drives it."""

    def __init__(self, case, seed):
        g = _case_grid(case, seed)
        self.mode, self.steps, self.nx, self.dt = case["mode"], case["steps"], g.m.nx, g.m.dt
        self.di = dropin.DropIn()
        self.di.set_mode(self.mode)
        self.c = dropin.consts_from_model(g.m)
        self.H, self.D, self.buf = dropin.PtrArrays(), dropin.PtrArrays(), ctypes.c_void_p()
        self.di.f["device_memory_alloc"](ctypes.byref(self.D), ctypes.byref(self.buf), self.nx + 3, self.c)
        media = _host(g.media)
        self.di.f["load_data_to_device_int"](media.ctypes.data, self.D.media, self.nx, self.c)
        self.ins = [_pinned(g.m.ncells).reshape(g.m.shape) for _ in range(2)]
        for h, t in zip(self.ins, (g.P, g.S)):
            torch.from_numpy(h).copy_(t)
        self.out = [_pinned(g.m.ncells).reshape(g.m.shape) for _ in range(2)]

    def run(self):
        di, c = self.di, self.c
        di.set_mode(self.mode)
        di.f["load_data_to_device"](self.ins[0].ctypes.data, self.D.P1, self.nx, c)
        di.f["load_data_to_device"](self.ins[1].ctypes.data, self.D.S2, self.nx, c)
        for s in range(1, self.steps + 1):
            di.time_step(self.H, self.D, c, s * self.dt)
        di.f["load_data_to_host"](self.out[0].ctypes.data, self.D.P1, self.nx, c)
        di.f["load_data_to_host"](self.out[1].ctypes.data, self.D.S2, self.nx, c)
        return {"P1": self.out[0], "S2": self.out[1]}

    def __del__(self):
        if getattr(self, "buf", None):
            self.di.f["device_memory_free"](self.D, self.buf)


def prepare(case, seed):
    return {"domain": _DomainState, "ensemble": _EnsembleState, "dropin": _DropinState}[case["kind"]](case, seed)


def run(state):
    return state.run()


# -------------------------------------------------------------------- work


def _cells(case):
    if case["kind"] == "ensemble":
        specs = (wl.config3_specs if case["config"] == 3 else wl.config4_specs)(case["members"])
        return sum(wl.spec_cells(s) for s in specs), sum((s["edge"] - 2) ** 3 for s in specs)
    n = (case["nx"], case["ny"], case["nz"])
    return math.prod(n), math.prod(k - 2 for k in n)


def work(case):
    """Per pass: the state in and out in FP64 (16 + 16 bytes a cell), and per step the state, the phase masses
    (where the form keeps them) and the cell fields read once, the new state and masses written once. About
    150 operations a cell and step: mobilities, six upwinded faces of two phases, mass update, Newton."""
    cells, inner = _cells(case)
    form = {0: "f64", 1: "f64", 2: "split"}[case["mode"]] if case["kind"] == "dropin" else case["prec"]
    step = {"f64": 32, "split": 48, "split_df": 48, "split_defect": 32}[form]
    step += 4 if case["kind"] == "dropin" else 8
    return {"bytes": 32.0 * cells + float(step) * inner * case["steps"], "flops": 150.0 * inner * case["steps"]}


# ------------------------------------------------------------------- exact


def _exact_grid(g, steps):
    """The time steps in 64 bits, increments kept apart from what they are added to: (P, S, masses per step)."""
    m, P, S = g.m, g.P.clone(), g.S.clone()
    nz, ny, nx = P.shape

    def table(v):  # a media-table value per cell
        if g.media is None:
            return v[0]
        return torch.tensor(v, dtype=torch.float64, device="cuda")[g.media.long()]

    K = g.K.double() if g.K is not None else table(list(m.K))
    phi = g.phi.double() if g.phi is not None else table(list(m.m))
    swr, lam, pd = table(list(m.S_wr)), table(list(m.lam)), table(list(m.P_d))
    inner = (slice(1, -1),) * 3
    at = lambda v: v[inner] if isinstance(v, torch.Tensor) else v  # noqa: E731
    hydro = m.bc_mode == abi.GBF_BC_HYDROSTATIC_SIDES
    V = m.h1 * m.h2 * m.h3
    masses = []
    for _ in range(steps):
        om = S / (1 - swr)  # 1 - S_e
        ln = torch.log1p(-om)
        ro1, ro2 = m.ro01 * (1 + m.beta1 * (P - m.P_atm)), m.ro02 * (1 + m.beta2 * (P - m.P_atm))
        L1 = K * torch.exp((2 + 3 * lam) / lam * ln) / m.mu1 * ro1
        L2 = K * om * om * -torch.expm1((2 + lam) / lam * ln) / m.mu2 * ro2
        del om
        c = inner
        f = [0.0, 0.0]
        for axis, h, w in ((2, m.h1, 1.0), (1, m.h2, m.kv), (0, m.h3, 1.0)):
            lo, hi = list(inner), list(inner)
            lo[axis], hi[axis] = slice(0, -2), slice(2, None)
            lo, hi = tuple(lo), tuple(hi)
            x1, x2 = (P[lo] - P[c]) / h, (P[c] - P[hi]) / h
            for a, (L, ro) in enumerate(((L1, ro1), (L2, ro2))):
                y1, y2 = x1, x2
                if axis == 1:
                    y1, y2 = x1 + ro[c] * m.g, x2 + ro[c] * m.g
                    if hydro:
                        y2[:, -1, :] = 0.0
                out = y2 * torch.where(y2 >= 0, L[c], L[hi])
                f[a] = f[a] + w * (out - y1 * torch.where(y1 >= 0, L[lo], L[c])) / h
                del out, y1, y2
        del x1, x2, L1, L2
        r1, r2 = m.dt / at(phi) * f[0], m.dt / at(phi) * f[1]
        if m.source_mode == abi.GBF_SOURCE_RATE:
            n, i0, k0 = m.rate_cells, nx // 2 - m.rate_cells // 2, nz // 2 - m.rate_cells // 2
            lo_k, hi_k, lo_i, hi_i = max(k0, 1), min(k0 + n, nz - 1), max(i0, 1), min(i0 + n, nx - 1)
            ph = at(phi)[lo_k - 1:hi_k - 1, 0, lo_i - 1:hi_i - 1] if isinstance(phi, torch.Tensor) else phi
            r2[lo_k - 1:hi_k - 1, 0, lo_i - 1:hi_i - 1] -= m.dt / ph * (m.rate / (n * n) / V)
        Pc, Sc = P[c], S[c]
        masses.append(torch.stack([((ro1[c] * (1 - Sc) - r1) * at(phi)).sum() * V,
                                   ((ro2[c] * Sc - r2) * at(phi)).sum() * V]))
        lamc, swrc = at(lam), at(swr)
        Se, lnc = 1 - Sc / (1 - swrc), ln[c]
        Pk = at(pd) * torch.exp(-lnc / lamc)
        r2 = r2 + m.ro02 * m.beta2 * Pk * Sc  # the targets take ro2 at P2 = P1, the Newton at P1 + P_k
        a, b = 1 + m.beta1 * (Pc - m.P_atm), 1 + m.beta2 * (Pc - m.P_atm + Pk)
        dp, ds = torch.zeros_like(r1), torch.zeros_like(r1)
        for _ in range(4):
            dPk = Pk * torch.expm1(-torch.log1p(-ds / ((1 - swrc) * Se)) / lamc)
            Sn = Sc + ds
            G1 = r1 + m.ro01 * (m.beta1 * dp * (1 - Sn) - a * ds)
            G2 = r2 + m.ro02 * (m.beta2 * (dp + dPk) * Sn + b * ds)
            slope = (Pk + dPk) / (lamc * ((1 - swrc) - Sn))
            J11, J12 = m.ro01 * m.beta1 * (1 - Sn), -m.ro01 * (a + m.beta1 * dp)
            J21, J22 = m.ro02 * m.beta2 * Sn, m.ro02 * (b + m.beta2 * (dp + dPk + slope * Sn))
            det = J11 * J22 - J12 * J21
            dp, ds = dp - (J22 * G1 - J12 * G2) / det, ds - (J11 * G2 - J21 * G1) / det
        # boundary cells in the sweep's order: what it has passed is new, what comes later is old
        Pn, Sn = P.clone(), S.clone()
        Pn[c], Sn[c] = Pc + dp, Sc + ds
        ii = slice(1, -1)
        for N, old in ((Sn, S), (Pn, P)):
            top = 0.0 if N is Sn else m.P_atm
            N[0, ii, ii], N[-1, ii, ii] = N[1, ii, ii], N[-2, ii, ii]
            if N is Pn and hydro:
                hs = (m.P_atm + torch.arange(ny, device="cuda", dtype=torch.float64) * (m.ro01 * m.g * m.h2))[:, None]
                N[0], N[-1] = hs, hs
            N[ii, 0, ii] = top
            if N is Sn and m.source_mode == abi.GBF_SOURCE_DIRICHLET_PATCH:
                lo_i, hi_i = max(nx // 2 - m.source, 1), min(nx // 2 + m.source + 1, nx - 1)
                lo_k, hi_k = max(nz // 2 - m.source, 1), min(nz // 2 + m.source + 1, nz - 1)
                N[lo_k:hi_k, 0, lo_i:hi_i] = m.S2_gr
            if N is Sn:
                N[0, 0, ii], N[-1, 0, ii] = old[1, 0, ii], N[-2, 0, ii]
            elif not hydro:
                N[0, 0, ii], N[-1, 0, ii] = top, top
            rows = slice(1, -1) if (N is Pn and hydro) else slice(None)
            add = m.ro01 * (1 + m.beta1 * (P[0, 1, ii] - m.P_atm)) * m.g * m.h2 if N is Pn else 0.0
            N[rows, -1, ii] = N[rows, -2, ii] + add
            if N is Pn and hydro:
                N[:, :, 0], N[:, :, -1] = hs[:, 0], hs[:, 0]
            else:
                first = old[:, :, 1].clone()
                first[ii, ii] = N[ii, ii, 1]
                N[:, :, -1] = N[:, :, -2]
                N[:, :, 0] = first
        P, S = Pn, Sn
    return P, S, torch.stack(masses)


def exact(case, seed):
    if case["kind"] == "ensemble":
        parts = [_exact_grid(g, case["steps"]) for g in _member_grids(case, seed)]
        out = {"P1": torch.cat([p[0].reshape(-1) for p in parts]), "S2": torch.cat([p[1].reshape(-1) for p in parts])}
        if not case["host"]:
            out["masses"] = torch.stack([p[2] for p in parts], dim=1)
        return out
    P, S, masses = _exact_grid(_case_grid(case, seed), case["steps"])
    return {"P1": P, "S2": S} if case["kind"] == "dropin" else {"P1": P, "S2": S, "masses": masses}
