"""What the framework is timed on: mechanical steps of one volume, batches of
volumes, the calibration gradient, the local solve on device arrays and the
phase-field relaxation, each through its public entry point.

A case is a dict of plain values.  `prepare` makes what a user's program holds
before the call (inputs from the seed, an uploaded volume), `run` is one call,
`exact` is the same result in 64-bit torch without the framework's code.

Fields that a volume keeps in FP32 (the mixed modes) are returned in FP32, the
type they are held in; FP64 runs return FP64.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "m-themes_gb300"))

from mth import Batch, Solver, capi, synth  # noqa: E402

PRECISION = {"fp64": capi.MTH_FP64, "mixed": capi.MTH_MIXED, "fast": capi.MTH_MIXED_FAST,
             "root64": capi.MTH_MIXED_ROOT64}
EDGES = [8, 12, 16, 18, 24, 32, 36, 48, 54, 64, 72, 96, 108, 128]   # even, 2^a 3^b
MOST_VOXEL_ITERATIONS = 128 ** 3 * 100   # of a mixed step: the cost of the largest listed case


# ------------------------------------------------------------------ the cases
def _step(name, dims, grains, precision, iters, **kw):
    c = {"name": name, "kind": "step", "nx": dims[0], "ny": dims[1], "nz": dims[2], "grains": grains, "pores": 0,
         "precision": precision, "iters": iters, "nrs": 10.0, "law": "power", "drx": False, "warm": 0,
         "fields": "sig,crss"}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: a unit-cell study of a few grains, where launches and the end of the step count
        _step("step_16_fp64", (16, 16, 16), 6, "fp64", 10, warm=2),
        # a small polycrystal in full precision, 100 Green iterations a step, texture and hardening in force
        _step("step_32_fp64", (32, 32, 32), 64, "fp64", 100, warm=2),
        # the benchmark volume: 512 grains with pores, mixed precision, the stress field read after the step
        _step("step_128_mixed", (128, 128, 128), 512, "mixed", 100, pores=40, fields="sig"),
        # the same volume in full precision, ten iterations (a restart that polishes a mixed solution)
        _step("step_128_fp64", (128, 128, 128), 512, "fp64", 10, pores=40, fields="sig"),
        # a rolled-sheet volume with unequal edges that are no powers of two, a rate exponent of 15
        _step("step_ragged_mixed", (72, 54, 108), 150, "mixed", 100, pores=6, nrs=15.0, warm=2),
        # a volume of a parameter study run in the fastest mode, an exponent that is no whole number
        _step("step_64_fast", (64, 64, 64), 128, "fast", 100, nrs=12.5, warm=2),
        # dislocation-density law (the reference's shipped one)
        _step("step_dd_96", (96, 96, 96), 216, "mixed", 100, law="dd", pores=17, fields="sig,rho_ssd"),
        # recrystallising volume in full precision: nucleation, phase field and mechanics in one step
        _step("step_drx_48_fp64", (48, 48, 48), 64, "fp64", 20, drx=True, warm=2, fields="sig,grain"),
        # one gradient of a calibration loop: forward run and adjoint of a tension curve
        {"name": "gradient_64", "kind": "gradient", "n": 64, "grains": 256, "steps": 4, "every": 2,
         "precision": "mixed", "iters": 100},
        # a batch of small volumes of several sizes and materials stepped together
        {"name": "batch_12", "kind": "batch", "n32": 4, "n48": 4, "n64": 4, "precision": "mixed", "iters": 100},
        # the local solve called by a host code on its own device arrays, an odd number of points
        {"name": "local_100003", "kind": "local", "n": 100003, "nrs": 10.0},
        # phase-field relaxation of a partly recrystallised volume on arrays, ten substeps
        {"name": "phase_field_128", "kind": "phase_field", "nx": 128, "ny": 128, "nz": 128, "grains": 1000,
         "nuclei": 200, "substeps": 10, "precision": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["dd", "drx", "gradient", "batch", "local", "phase_field"])
    if kind in ("step", "dd", "drx"):
        precision = "mixed" if kind == "dd" else "fp64" if kind == "drx" else rng.choice(
            ["fp64", "fp64", "mixed", "mixed", "mixed", "fast", "root64"])
        iters = rng.randint(8, 100)
        most = MOST_VOXEL_ITERATIONS / 2 / iters / (18 if precision == "fp64" else 1)
        side = max(8.0, min(128.0, most ** (1.0 / 3.0)))
        target = math.exp(rng.uniform(math.log(8.0), math.log(side)))
        dims = []
        for _ in range(3):
            e = min(EDGES, key=lambda x: abs(math.log(x / (target * rng.uniform(0.7, 1.4)))))
            dims.append(e)
        while dims[0] * dims[1] * dims[2] > max(most, 512):
            k = dims.index(max(dims))
            dims[k] = EDGES[max(0, EDGES.index(dims[k]) - 1)]
        v = dims[0] * dims[1] * dims[2]
        grains = max(2, min(600, int(v / rng.choice([500, 2000, 4096]))))
        pores = 0 if kind == "drx" or min(dims) < 16 else rng.choice([0, 0, max(1, v // 60000)])
        c = _step("", tuple(dims), grains, precision, iters, pores=pores,
                  nrs=rng.choice([8.0, 10.0, 10.0, 15.0, 20.0, 12.5]), warm=1 if kind == "dd" else 2)
        if kind == "dd":
            c.update(law="dd", fields="sig,rho_ssd", nrs=10.0)
        if kind == "drx":
            c.update(drx=True, fields="sig,grain", nrs=10.0)
        del c["name"]
        return c
    if kind == "gradient":
        n = rng.choice([16, 24, 32, 36, 48, 64])
        steps = rng.randint(2, 4)
        return {"kind": "gradient", "n": n, "grains": max(4, n ** 3 // 2000), "steps": steps,
                "every": rng.randint(1, steps), "precision": "mixed", "iters": rng.randint(40, 100)}
    if kind == "batch":
        return {"kind": "batch", "n32": rng.randint(1, 6), "n48": rng.randint(0, 5), "n64": rng.randint(0, 4),
                "precision": "mixed", "iters": rng.randint(20, 100)}
    if kind == "local":
        return {"kind": "local", "n": _log_int(rng, 300, 1 << 20), "nrs": rng.choice([8.0, 10.0, 15.0, 20.0, 12.5])}
    dims = [_log_int(rng, 20, 128) for _ in range(3)]
    v = dims[0] * dims[1] * dims[2]
    return {"kind": "phase_field", "nx": dims[0], "ny": dims[1], "nz": dims[2], "grains": max(2, v // 2000),
            "nuclei": max(1, v // 10000), "substeps": rng.randint(2, 10), "precision": rng.choice(["mixed", "fp64"])}


# ------------------------------------------------------------- the inputs
def _grain_map(dims, seeds):
    """Periodic Voronoi cells on the GPU: the 0-based nearest seed of every voxel centre, (nx, ny, nz)."""
    s = torch.as_tensor(seeds, device="cuda", dtype=torch.float32)
    d2 = []
    for a in range(3):
        x = torch.arange(dims[a], device="cuda", dtype=torch.float32) + 0.5
        d = (x[:, None] - s[None, :, a]).abs()
        d2.append(torch.minimum(d, dims[a] - d) ** 2)
    out = torch.empty(dims, device="cuda", dtype=torch.int64)
    for i in range(dims[0]):
        out[i] = (d2[0][i] + d2[1][:, None, :] + d2[2][None, :, :]).argmin(dim=2)
    return out


def _balls(dims, centres, radius):
    """Index of the last ball that covers each voxel (periodic), -1 where none does."""
    out = torch.full(dims, -1, device="cuda", dtype=torch.int64)
    ax = [torch.arange(n, device="cuda", dtype=torch.float32) + 0.5 for n in dims]
    for k, c in enumerate(centres):
        d = []
        for a in range(3):
            t = (ax[a] - float(c[a])).abs()
            d.append(torch.minimum(t, dims[a] - t) ** 2)
        out[(d[0][:, None, None] + d[1][None, :, None] + d[2][None, None, :]) <= radius * radius] = k
    return out


def _microstructure(dims, grains, pores, seed):
    """(grain, phase, Euler angles) as the host arrays that an upload takes, and the grain map on the GPU."""
    rng = np.random.default_rng(seed)
    g = _grain_map(dims, rng.random((grains, 3)) * np.asarray(dims))
    euler = np.concatenate([synth.uniform_orientations(grains, rng), np.zeros((1, 3))])
    if pores:
        g[_balls(dims, rng.random((pores, 3)) * np.asarray(dims), 3) >= 0] = grains
    flat = g.reshape(-1)
    ang = torch.as_tensor(euler, device="cuda")[flat]
    return ((flat + 1).to(torch.int32).cpu().numpy(), (1 + (flat == grains)).to(torch.int32).cpu().numpy(),
            ang.cpu().numpy(), euler, flat)


def _dims(case):
    return (case["nx"], case["ny"], case["nz"])


def _config(case, dims, material=None):
    drx = None
    load = (-0.5, -0.5, 1.0, 0.0, 0.0, 0.0)
    if case.get("drx"):
        drx = synth.Drx(rho_k=40000.0, nucleation_prob=2e-3)
        load = (0.5, 0.5, -1.0, 0.0, 0.0, 0.0)
    return synth.Config(cell_dim=dims, n_grains=case.get("grains", 1), n_pores=case.get("pores", 0),
                        material=material or synth.Material(nrs=case.get("nrs", 10.0)), iter_max=case["iters"],
                        velgrad_bc=load, drx=drx, dd=synth.DD() if case.get("law") == "dd" else None)


def _batch_members(case, seed):
    """Grid edge, grains and material of each member, spread as in a parameter study."""
    rng = np.random.default_rng(seed)
    out = []
    for edge in [32] * case["n32"] + [48] * case["n48"] + [64] * case["n64"]:
        tau0 = float(rng.uniform(12.0, 20.0))
        out.append((edge, int(rng.integers(32, 257)),
                    synth.Material(tau0f=tau0, tau0b=tau0, nrs=float(rng.choice([8.0, 10.0, 15.0, 20.0])))))
    return out


def _local_inputs(case, seed):
    """Points of a polycrystal under load, in the six-component basis of the C interface."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    ang = torch.as_tensor(synth.uniform_orientations(n, rng), device="cuda")
    rot = _rotation(ang)
    lam = torch.as_tensor(rng.normal(0.0, 20.0, (n, 6)), device="cuda")
    crss = torch.as_tensor(rng.uniform(14.0, 30.0, (n, 12)), device="cuda")
    epsp = torch.as_tensor(rng.normal(0.0, 2e-3, (n, 6)), device="cuda")
    epsp[:, 5] = 0.0
    mean = _mean_stiffness()
    strain = epsp + lam @ torch.linalg.inv(mean) + torch.as_tensor(rng.normal(0.0, 3e-4, (n, 6)), device="cuda")
    return {"lam": lam, "epsp": epsp, "strain": strain, "rot": rot.reshape(n, 9).contiguous(), "crss": crss,
            "c066": mean}


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        dims = _dims(case)
        g, p, e, _, _ = _microstructure(dims, case["grains"], case["pores"], seed)
        cfg = _config(case, dims)
        s = Solver(capi.params_from_config(cfg, precision=PRECISION[case["precision"]]), g, p, e)
        for _ in range(case["warm"]):
            s.step()
        nv = s.nv
        st = {"kind": kind, "solver": s, "out": {}, "mixed": case["precision"] != "fp64"}
        for f in case["fields"].split(","):
            k = capi.FIELD_NCOMP[capi.FIELD[f]]
            host = torch.empty((nv, k), dtype=torch.float64, pin_memory=True)
            held = torch.int32 if f == "grain" else torch.float32 if st["mixed"] else None
            st["out"][f] = (host, torch.zeros((nv, k), dtype=held) if held is not None else None)
        return st
    if kind == "batch":
        par, ms = [], []
        for i, (edge, grains, mat) in enumerate(_batch_members(case, seed)):
            dims = (edge, edge, edge)
            cfg = _config(dict(case, grains=grains), dims, mat)
            par.append(capi.params_from_config(cfg, precision=PRECISION[case["precision"]]))
            ms.append(_microstructure(dims, grains, 0, seed * 1000 + i)[:3])
        b = Batch(par, ms)
        return {"kind": kind, "batch": b, "mixed": case["precision"] != "fp64",
                "out": [(torch.empty((v, 9), dtype=torch.float64, pin_memory=True),
                         torch.zeros((v, 9), dtype=torch.float32)) for v in b.nv]}
    if kind == "gradient":
        dims = (case["n"],) * 3
        cfg = _config(case, dims, synth.Material())
        return {"kind": kind, "par": capi.params_from_config(cfg, precision=PRECISION[case["precision"]]),
                "ms": _microstructure(dims, case["grains"], 0, seed)[:3], "every": case["every"],
                "mixed": case["precision"] != "fp64", "target": _target_curve(case["steps"])}
    if kind == "local":
        st = _local_inputs(case, seed)
        n = case["n"]
        st.update(kind=kind, n=n, sig=torch.empty_like(st["lam"]), edot=torch.empty_like(st["lam"]),
                  err=torch.empty((n, 2), dtype=torch.float64, device="cuda"),
                  c066_host=np.ascontiguousarray(st["c066"].cpu().numpy()),
                  par=capi.params_from_config(synth.Config(material=synth.Material(nrs=case["nrs"]))))
        return st
    dims = _dims(case)
    rng = np.random.default_rng(seed)
    g = _grain_map(dims, rng.random((case["grains"], 3)) * np.asarray(dims)) + 1
    stored = torch.as_tensor(rng.uniform(200.0, 900.0, case["grains"] + 1), device="cuda")[g]
    stored = stored * torch.as_tensor(rng.uniform(0.9, 1.1, dims), device="cuda")
    ball = _balls(dims, rng.random((case["nuclei"], 3)) * np.asarray(dims), 3.0)
    g = torch.where(ball >= 0, case["grains"] + 1 + ball, g)
    stored[ball >= 0] = 1.0
    drx = synth.Drx()
    par = capi.params_from_config(synth.Config(cell_dim=dims, drx=drx), precision=PRECISION[case["precision"]])
    ids = case["grains"] + case["nuclei"]
    return {"kind": kind, "par": par, "dims": (ctypes.c_int * 3)(*dims), "init": case["grains"], "ids": ids,
            "substeps": case["substeps"], "grain": g.reshape(-1).to(torch.int32).cpu().numpy(),
            "rho": stored.reshape(-1).cpu().numpy(), "table": np.zeros(ids), "out": np.zeros(g.numel(), np.int32),
            "mixed": case["precision"] != "fp64"}


def _target_curve(steps):
    """Measured axial stress of the calibration loop [MPa]."""
    return np.array([60.0 + 12.0 * math.sqrt(1.0 + i) for i in range(steps)])


# ------------------------------------------------------------------- a call
def _as_held(x, mixed):
    return np.asarray(x, dtype=np.float32 if mixed else np.float64)


def _report(r, mixed):
    return {k: _as_held(r[k], mixed) for k in ("sig_avg", "disgrad_avg", "eps_avg", "edot_avg")}


def _dptr(t):
    return ctypes.cast(ctypes.c_void_p(t.data_ptr()), ctypes.POINTER(ctypes.c_double))


def run(st):
    kind = st["kind"]
    lib = capi.load()
    if kind == "step":
        s = st["solver"]
        r = s.step()
        out = _report(r, st["mixed"])
        out["iterations"] = r["iterations"]
        out["new_grains"] = r["n_new_grains"]
        for f, (host, held) in st["out"].items():
            capi.check(lib, lib.mth_download_field(s.ctx, capi.FIELD[f], _dptr(host), host.numel()))
            out[f] = host if held is None else held.copy_(host)
        return out
    if kind == "batch":
        b = st["batch"]
        out = {}
        for i, r in enumerate(b.step()):
            host, held = st["out"][i]
            capi.check(lib, lib.mth_batch_download_field(b.b, i, capi.FIELD["sig"], _dptr(host), host.numel()))
            out["member%02d" % i] = {"sig_avg": _as_held(r["sig_avg"], st["mixed"]),
                                     "sig": held.copy_(host) if st["mixed"] else host}
        return out
    if kind == "gradient":
        with Solver(st["par"], *st["ms"]) as s:
            j, grad, s33, _ = s.adjoint(st["target"], checkpoint_every=st["every"])
        m = st["mixed"]
        return {"misfit": _as_held([j], m), "grad": _as_held(grad, m), "s33": _as_held(s33, m)}
    if kind == "local":
        st["sig"].copy_(st["lam"])
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        it = ctypes.c_longlong(0)
        capi.check(lib, lib.mth_local_solve_noalloc(
            ctypes.byref(st["par"]), capi._dptr(st["c066_host"]), st["n"], _ptr(st["sig"]), _ptr(st["epsp"]),
            _ptr(st["strain"]), _ptr(st["rot"]), _ptr(st["crss"]), _ptr(st["edot"]), _ptr(st["err"]),
            ctypes.byref(it), stream))
        return {"sig": st["sig"], "edot": st["edot"], "err": st["err"]}
    table = st["table"].copy()
    capi.check(lib, lib.mth_pf_relax(ctypes.byref(st["par"]), st["dims"], capi._iptr(st["grain"]),
                                     capi._dptr(st["rho"]), st["substeps"], st["init"], capi._dptr(table), st["ids"],
                                     capi._iptr(st["out"]), None, None, None))
    return {"grain": st["out"], "table": _as_held(table, st["mixed"])}


# ------------------------------------------------------- what it cannot do without
def _step_work(voxels, iters, width):
    """Bytes: the volume's state in and out once.  Operations of the Green iterations: per voxel the six
    real transforms both ways and, in the local solve, three evaluations of 12 slip systems with their
    Hessian and two 5x5 solves."""
    planes_in, planes_out = 6 * 4 + 9 + 12 + 1, 6 * 4 + 9 + 12 + 1
    fft = 12 * 2.5 * math.log2(max(2, voxels))
    newton = 3 * 12 * 70 + 2 * 130 + 600
    return {"bytes": voxels * width * (planes_in + planes_out), "flops": iters * voxels * (fft + newton)}


def work(case):
    kind = case["kind"]
    if kind == "step":
        v = case["nx"] * case["ny"] * case["nz"]
        return _step_work(v, case["iters"], 8 if case["precision"] == "fp64" else 4)
    if kind == "batch":
        v = sum(case["n%d" % e] * e ** 3 for e in (32, 48, 64))
        return _step_work(v, case["iters"], 4)
    if kind == "gradient":
        w = _step_work(case["n"] ** 3, case["iters"] * case["steps"], 4)
        return {"bytes": 2 * w["bytes"], "flops": 2 * w["flops"]}
    if kind == "local":
        return {"bytes": 8.0 * case["n"] * (6 + 6 + 6 + 9 + 12 + 6 + 6 + 2),
                "flops": case["n"] * (4 * 12 * 70 + 3 * 130 + 600)}
    v = case["nx"] * case["ny"] * case["nz"]
    # grain ids and energies in, ids out; the boundary layer (about a third of the voxels) relaxes
    # about three order parameters of 40 operations a substep
    return {"bytes": v * (4 + 8 + 4), "flops": case["substeps"] * v / 3 * 3 * 40}


# --------------------------------------------------------------- in 64 bits
# The Lebensohn-Tome basis of symmetric tensors, as the C interface documents it.
def _basis():
    r2, r3, r6 = math.sqrt(0.5), math.sqrt(1.0 / 3.0), math.sqrt(1.0 / 6.0)
    b = torch.zeros((6, 3, 3), dtype=torch.float64)
    b[0, 0, 0], b[0, 1, 1] = -r2, r2
    b[1, 0, 0], b[1, 1, 1], b[1, 2, 2] = -r6, -r6, 2 * r6
    b[2, 1, 2] = b[2, 2, 1] = r2
    b[3, 0, 2] = b[3, 2, 0] = r2
    b[4, 0, 1] = b[4, 1, 0] = r2
    b[5, 0, 0] = b[5, 1, 1] = b[5, 2, 2] = r3
    return b.cuda()


def _rotation(angles):
    """Crystal-to-sample matrices of Bunge angles in degrees."""
    a = angles * (3.14159265359 / 180.0)
    c1, s1, c, s, c2, s2 = (f(a[:, k]) for k in (0, 1, 2) for f in (torch.cos, torch.sin))
    rows = [c1 * c2 - s1 * s2 * c, s1 * c2 + c1 * s2 * c, s2 * s,
            -c1 * s2 - s1 * c2 * c, -s1 * s2 + c1 * c2 * c, c2 * s,
            s1 * s, -c1 * s, c]
    return torch.stack(rows, dim=1).reshape(-1, 3, 3).transpose(1, 2).contiguous()


def _q(rot, b):
    """(n, 5, 5): deviatoric components from sample to crystal axes."""
    m = torch.einsum("nai,jab,nbk->njik", rot, b[:5], rot)
    return torch.einsum("iab,njab->nij", b[:5], m)


def _cubic(m):
    return torch.tensor([m.c11 - m.c12] * 2 + [2 * m.c44] * 3 + [m.c11 + 2 * m.c12], dtype=torch.float64).cuda()


def _mean_stiffness(material=None):
    """Average of the cubic stiffness over all orientations."""
    ev = _cubic(material or synth.Material())
    mean = (2 * ev[0] + 3 * ev[2]) / 5
    return torch.diag(torch.stack([mean] * 5 + [ev[5]]))


def _schmid(b):
    n = torch.tensor([s[0] for s in synth.FCC_SLIP], dtype=torch.float64).cuda() / math.sqrt(3.0)
    d = torch.tensor([s[1] for s in synth.FCC_SLIP], dtype=torch.float64).cuda() / math.sqrt(2.0)
    t = 0.5 * (n[:, :, None] * d[:, None, :] + d[:, :, None] * n[:, None, :])
    return torch.einsum("sab,iab->si", t, b[:5]), n, d


class _Power:
    """Power law: shear rates, their slopes and the potential at resolved shear stresses."""

    def __init__(self, material, crss):
        self.n, self.g0, self.tau = material.nrs, material.gamd0, crss

    def rates(self, rss, at=None):
        tau = self.tau if at is None else self.tau[at]
        r = (rss / tau).abs()
        p = r ** (self.n - 1.0)
        g = self.g0 * p * r
        return g * rss.sign(), self.g0 * self.n * p / tau, g * rss.abs() / (self.n + 1.0)


class _Sinh:
    """Dislocation-density law: thermally activated slip above the passing stress."""

    def __init__(self, tp, td, g0):
        self.tp, self.td, self.g0 = tp, td, g0

    def rates(self, rss, at=None):
        tp, td, g0 = (self.tp, self.td, self.g0) if at is None else (self.tp[at], self.td[at], self.g0[at])
        t = (rss.abs() - tp).clamp_min(0.0) / td
        on = (rss.abs() > tp).to(rss.dtype)
        return (g0 * torch.sinh(t) * rss.sign() * on, g0 * torch.cosh(t) / td * on,
                2.0 * g0 * td * torch.sinh(0.5 * t) ** 2 * on)


_PAIRS = [(i, j) for i in range(5) for j in range(i, 5)]


def _solve5(h, g):
    """Solutions of packed symmetric positive definite 5x5 systems, column by column."""
    idx = {}
    for k, (i, j) in enumerate(_PAIRS):
        idx[i, j] = idx[j, i] = k
    low, d = {}, []
    for j in range(5):
        a = h[:, idx[j, j]]
        for k in range(j):
            a = a - low[j, k] ** 2 * d[k]
        d.append(a)
        for i in range(j + 1, 5):
            a = h[:, idx[i, j]]
            for k in range(j):
                a = a - low[i, k] * low[j, k] * d[k]
            low[i, j] = a / d[j]
    y = []
    for i in range(5):
        a = g[:, i]
        for k in range(i):
            a = a - low[i, k] * y[k]
        y.append(a)
    x = [None] * 5
    for i in range(4, -1, -1):
        a = y[i] / d[i]
        for k in range(i + 1, 5):
            a = a - low[k, i] * x[k]
        x[i] = a
    return torch.stack(x, dim=1)


def _newton(lam, strain, epsp, q, sdev, shh, s0, law, dt, schmid):
    """Stress and plastic rate with S0 (sig - lam) + S sig + epsp + dt edot(sig) = strain, by a damped Newton
    method in crystal axes.  sdev: (n, 5, 5) sample compliance; s0: (6, 6)."""
    k = q @ (s0[:5, :5] + sdev) @ q.transpose(1, 2)
    kp = torch.stack([k[:, i, j] for i, j in _PAIRS], dim=1)
    mm = torch.stack([schmid[:, i] * schmid[:, j] for i, j in _PAIRS], dim=1)
    rhs = (q @ (lam[:, :5] @ s0[:5, :5] + strain[:, :5] - epsp[:, :5])[:, :, None])[:, :, 0]
    x = (q @ lam[:, :5, None])[:, :, 0]
    act = torch.arange(x.shape[0], device=x.device)
    scale = lam.norm(dim=1) + 1e-6

    def phi(y, at):
        kx = (k[at] @ y[:, :, None])[:, :, 0]
        _, _, psi = law.rates(y @ schmid.T, at)
        return (y * (0.5 * kx - rhs[at])).sum(1) + dt * psi.sum(1)

    for _ in range(100):
        y = x[act]
        g, w, psi = law.rates(y @ schmid.T, act)
        kx = (k[act] @ y[:, :, None])[:, :, 0]
        res = kx - rhs[act] + dt * (g @ schmid)
        p = -_solve5(kp[act] + dt * (w @ mm), res)
        size = p.norm(dim=1)
        big = (size > 1e-4 * scale[act]).nonzero()[:, 0]
        if big.numel():
            f0 = ((y * (0.5 * kx - rhs[act])).sum(1) + dt * psi.sum(1))[big]
            slope = (res * p).sum(1)[big]
            a = torch.ones_like(f0)
            for _ in range(40):
                f = phi(y[big] + a[:, None] * p[big], act[big])
                bad = ~(f <= f0 + 1e-4 * a * slope)
                if not bool(bad.any()):
                    break
                a = torch.where(bad, 0.5 * a, a)
            p[big] = p[big] * a[:, None]
        x[act] = y + p
        act = act[p.norm(dim=1) > 1e-13 * scale[act]]
        if act.numel() == 0:
            break
    g, _, _ = law.rates(x @ schmid.T)
    sig = torch.empty_like(lam)
    sig[:, :5] = (q.transpose(1, 2) @ x[:, :, None])[:, :, 0]
    sig[:, 5] = (s0[5, 5] * lam[:, 5] + strain[:, 5] - epsp[:, 5]) / (s0[5, 5] + shh)
    edot = torch.zeros_like(lam)
    edot[:, :5] = (q.transpose(1, 2) @ (g @ schmid)[:, :, None])[:, :, 0]
    return sig, edot, g


class _Volume:
    """One volume in 64 bits: the Green iterations and end-of-step updates in plain torch."""

    def __init__(self, dims, flat, euler, grains, material, iters, dd=None):
        self.dims, self.m, self.iters, self.dd = dims, material, iters, dd
        b = self.b = _basis()
        self.schmid, self.sn, self.sb = _schmid(b)
        self.dt, self.err = 1e-3, 1e-5
        # axial rate 1/s along 33; 11 and 22 are stress controlled
        self.udot = torch.diag(torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64)).cuda()
        self.nv = flat.numel()
        self.solid = (flat < grains).nonzero()[:, 0]
        ang = torch.as_tensor(euler, device="cuda")[flat[self.solid]]
        self.rot = _rotation(ang)
        ev = _cubic(material)
        # stiffness and compliance in sample axes, of the initial orientations
        per = _q(_rotation(torch.as_tensor(euler[:grains], device="cuda")), b)
        cg = per.transpose(1, 2) @ (ev[:5, None] * per)
        sg = per.transpose(1, 2) @ (per / ev[:5, None])
        cls = flat[self.solid]
        count = torch.bincount(cls, minlength=grains).to(torch.float64)
        c0 = torch.zeros((6, 6), dtype=torch.float64).cuda()
        c0[:5, :5] = (count[:, None, None] * cg).sum(0) / self.nv
        c0[5, 5] = ev[5] * self.solid.numel() / self.nv
        self.s0 = torch.linalg.inv(c0)
        self.sdev, self.shh = sg[cls], float(1.0 / ev[5])
        self.c4 = torch.einsum("ij,iab,jcd->abcd", c0, b, b)
        self.s4 = torch.einsum("ij,iab,jcd->abcd", self.s0, b, b)
        n = self.solid.numel()
        d6 = torch.einsum("ab,iab->i", self.udot * self.dt, b)
        self.sig = torch.zeros((self.nv, 6), dtype=torch.float64).cuda()
        self.sig[self.solid, :5] = cg[cls] @ d6[:5]
        self.sig[self.solid, 5] = ev[5] * d6[5]
        self.strain = torch.zeros_like(self.sig)
        self.epsp = torch.zeros((n, 6), dtype=torch.float64).cuda()
        self.crss = torch.full((n, 12), material.tau0f, dtype=torch.float64).cuda()
        self.gam = torch.zeros(n, dtype=torch.float64).cuda()
        if dd is not None:
            self.rho = torch.full((n, 12), dd.rho_ssd0, dtype=torch.float64).cuda()
        self.avg = self.udot * self.dt
        dev = self.udot - torch.eye(3).cuda() * self.udot.trace() / 3
        self.evm = float(torch.sqrt(2.0 / 3.0 * (dev * dev).sum()) * self.dt)
        self.step_no = 0
        # Green operator: wave vectors (the Nyquist index counts as -1/2) and Omega = (n C0 n)^-1
        f = []
        for a in dims:
            k = torch.arange(a, dtype=torch.float64).cuda()
            f.append(torch.where(2 * k >= a, k - a, k) / a)
        kv = torch.stack(torch.meshgrid(*f, indexing="ij"), dim=-1).reshape(-1, 3)
        kv[0] = 1.0
        self.kn = kv / kv.norm(dim=1, keepdim=True)
        ac = torch.einsum("abcd,nb,nd->nac", self.c4, self.kn, self.kn)
        cof = torch.cross(ac[:, [1, 2, 0]], ac[:, [2, 0, 1]], dim=2)
        self.om = cof / (ac[:, 0] * cof[:, 0]).sum(1)[:, None, None]
        self.om[0] = 0.0

    def transform(self, x, inverse=False):
        f = torch.fft.ifftn if inverse else torch.fft.fftn
        return f(x.reshape(self.dims), dim=(0, 1, 2)).reshape(-1)

    def green(self, spin):
        """Strain increment of the polarised stress; its antisymmetric part is added to spin."""
        t = torch.einsum("ni,iab->nab", self.sig, self.b)
        h = {(i, j): self.transform(t[:, i, j]) for i in range(3) for j in range(i, 3)}
        tn = torch.stack([sum(h[min(i, j), max(i, j)] * self.kn[:, j] for j in range(3)) for i in range(3)], dim=1)
        v = -(self.om.to(tn.dtype) @ tn[:, :, None])[:, :, 0]
        d = lambda i, j: v[:, i] * self.kn[:, j]   # noqa: E731
        for c in range(6):
            w = sum(float(self.b[c, i, j]) * d(i, j) for i in range(3) for j in range(3) if self.b[c, i, j] != 0)
            self.strain[:, c] += self.transform(w, inverse=True).real
        for c, (i, j) in enumerate(((2, 1), (0, 2), (1, 0))):
            spin[c] += 0.5 * (d(i, j) - d(j, i))

    def von_mises(self, t):
        s = 0.5 * (t + t.T)
        s = s - torch.eye(3).cuda() * t.trace() / 3
        return float(torch.sqrt(2.0 / 3.0 * (s * s).sum()))

    def law(self):
        if self.dd is None:
            return _Power(self.m, self.crss)
        k, d = self.dd_constants(), self.dd
        rf, rp = self.rho @ k["f"].T, self.rho @ k["p"].T
        rm = k["rm"] * torch.sqrt(rp * rf)
        self.forest = (rf, rm)
        return _Sinh(k["tp"] * torch.sqrt((rp + rm).abs()), 1000.0 + k["tcut"] * torch.sqrt(rf),
                     k["g0"] * rm / torch.sqrt(rf))

    def dd_constants(self):
        d, m = self.dd, self.m
        b = d.a0 / math.sqrt(2.0)
        mu = 0.1 * (m.c11 - m.c12 + 3 * m.c44) + 0.5 * (5 * (m.c11 - m.c12) * m.c44) / (4 * m.c44 + 3 * (m.c11 - m.c12))
        kt = d.T * 1.380658e-23 / 1.60217733e-19
        ev = 0.62415063631
        c = d.c
        n, s = self.sn, self.sb
        chi = torch.empty((12, 12), dtype=torch.float64)
        for i in range(12):
            for j in range(12):
                nn, bb = float(n[i] @ n[j]), float(s[i] @ s[j])
                if i == j:
                    x = d.chi[0]
                elif abs(abs(nn) - 1) < 1e-6:
                    x = d.chi[1]
                elif abs(abs(bb) - 1) < 1e-6:
                    x = d.chi[2]
                elif abs(bb) < 1e-6:
                    x = d.chi[4]
                else:
                    q = s[i] - math.copysign(1.0, bb) * s[j]
                    x = d.chi[3] if min(abs(float(q @ n[i])), abs(float(q @ n[j]))) < 1e-6 else d.chi[5]
                chi[i, j] = x
        cs = (n @ torch.linalg.cross(n, s).T).abs()
        ss = (1 - cs * cs).abs().sqrt()
        chi = chi.cuda()
        return {"f": chi * cs, "p": chi * ss, "rm": 2 * kt / c[0] / c[1] / c[2] / mu / b ** 3 * 160.2177,
                "tp": c[0] * mu * b * 1e-3, "tcut": kt / ev / c[1] / c[2] / b / b * 0.1,
                "g0": 1e-3 * 1e10 * c[1] * b * math.exp(-d.q_slip * ev / kt),
                "dip": math.sqrt(3.0) * mu * b / 16 / math.pi / (1 - d.nu), "ann": c[6] * 1.6e3,
                "clb": 4e12 * d.d0 / b, "clb_h": b ** 3 * 100 / (1.38 * d.T), "clb_0": -1 - d.q_bulk * ev / kt}

    def step(self):
        b, dt = self.b, self.dt
        law = self.law()
        q = _q(self.rot, b)
        spin = torch.zeros((3, self.nv), dtype=torch.complex128).cuda()
        ddg = torch.zeros((3, 3), dtype=torch.float64).cuda()
        acum, applied = ddg.clone(), ddg.clone()
        for it in range(1, self.iters + 1):
            u = ddg + (self.udot * dt if it == 1 else 0.0)
            applied += ddg
            self.green(spin)
            self.strain += torch.einsum("ab,iab->i", u, b)
            lam, eps = self.sig[self.solid], self.strain[self.solid]
            sig, edot, gdot = _newton(lam, eps, self.epsp, q, self.sdev, self.shh, self.s0, law, dt, self.schmid)
            self.sig[self.solid] = sig
            tot = self.epsp + dt * edot - eps
            tot[:, :5] += (self.sdev @ sig[:, :5, None])[:, :, 0]
            tot[:, 5] += self.shh * sig[:, 5]
            err_s = float((sig - lam).norm(dim=1).sum() / self.nv)
            err_e = float(tot.norm(dim=1).sum() / self.nv)
            mean = torch.einsum("i,iab->ab", sig.sum(0) / self.nv, b)
            mean1 = torch.einsum("i,iab->ab", sig.sum(0) / self.solid.numel(), b)
            ddg = torch.zeros_like(ddg)
            for a in (0, 1):   # axial components 11 and 22 are stress free
                ddg[a, a] = -(self.s4[a, a, 0, 0] * mean[0, 0] + self.s4[a, a, 1, 1] * mean[1, 1])
            acum += ddg
            dev = mean - torch.eye(3).cuda() * mean.trace() / 3
            off = (dev[1, 1] + dev[2, 2] + mean1[0, 0]) / 3
            svm = float(torch.sqrt(1.5 * ((dev - torch.eye(3).cuda() * off) ** 2).sum()))
            err_e = 0.0 if abs(self.evm) < 1e-5 else err_e / self.evm
            if max(err_s / svm, err_e) <= self.err:
                break
        actual = self.avg + acum
        self.evm = self.von_mises(actual)
        self.epsp = self.epsp + dt * edot
        out = {"sig_avg": mean, "disgrad_avg": actual, "iterations": it,
               "eps_avg": torch.einsum("i,iab->ab", self.epsp.sum(0) / self.nv, b),
               "edot_avg": torch.einsum("i,iab->ab", edot.sum(0) / self.nv, b)}
        if self.dd is not None:
            k, d = self.dd_constants(), self.dd
            rf, rm = self.forest
            rss = (q @ sig[:, :5, None])[:, :, 0] @ self.schmid.T
            dip = k["dip"] / (rss.abs() + 5e-3)
            climb = torch.exp(((sig[:, 0] + sig[:, 1] + sig[:, 2]) / 3).abs() * k["clb_h"] + k["clb_0"])[:, None]
            grow = gdot.abs() * (d.c[3] * rf.sqrt() + d.c[5] * dip * rm - d.c[4] * self.rho)
            self.rho = self.rho + dt * (grow - k["ann"] * self.rho ** 2 - k["clb"] * dip * self.rho ** 2 * climb)
        if self.step_no > 1:
            self.turn(gdot, spin, applied)
        if self.dd is None:
            self.harden(gdot)
        self.avg = actual + self.udot * dt
        self.step_no += 1
        return out

    def turn(self, gdot, spin, applied):
        """Lattice rotation: local spin plus the uniform part, less the plastic spin."""
        loc = torch.stack([self.transform(s, inverse=True).real[self.solid] for s in spin], dim=1)
        au = 0.5 * (applied - applied.T)
        c = gdot @ torch.linalg.cross(self.sb, self.sn)
        slip = -0.5 * (self.rot @ c[:, :, None])[:, :, 0]
        w = torch.stack([au[2, 1], au[0, 2], au[1, 0]]) + loc - slip * self.dt
        wn = w.norm(dim=1, keepdim=True)
        wt = torch.tan(wn / 2)
        w = w * wt / torch.where(wn < 1e-6, torch.ones_like(wn), wn)
        o = torch.zeros((w.shape[0], 3, 3), dtype=torch.float64).cuda()
        o[:, 0, 1], o[:, 0, 2], o[:, 1, 2] = -w[:, 2], w[:, 1], -w[:, 0]
        o = o - o.transpose(1, 2)
        self.rot = (torch.eye(3).cuda() + 2 * (o + o @ o) / (1 + wt[:, :, None] ** 2)) @ self.rot

    def harden(self, gdot):
        m, dg = self.m, gdot.abs().sum(1) * self.dt
        fact = abs(m.thet0 / m.tau1)
        e0, em1 = torch.exp(-self.gam * fact), torch.expm1(-dg * fact)
        voce = (m.thet1 * dg - (fact * m.tau1 - m.thet1) / fact * e0 * em1 -
                m.thet1 / fact * e0 * (em1 * (self.gam * fact + 1) + (em1 + 1) * dg * fact))
        self.crss = self.crss + torch.where(dg > 0, voce, torch.zeros_like(voce))[:, None]
        self.gam = self.gam + dg

    def field(self, name):
        out = torch.zeros((self.nv, 12), dtype=torch.float64).cuda()
        if name == "sig":
            return torch.einsum("ni,iab->nab", self.sig, self.b).reshape(-1, 9)
        if name == "crss":
            out[self.solid] = self.crss
            return out
        out[:] = self.dd.rho_ssd0
        out[self.solid] = self.rho
        return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "step" and not case["drx"]:
        dims = _dims(case)
        _, _, _, euler, flat = _microstructure(dims, case["grains"], case["pores"], seed)
        v = _Volume(dims, flat, euler, case["grains"], synth.Material(nrs=case["nrs"]), case["iters"],
                    synth.DD() if case["law"] == "dd" else None)
        for _ in range(case["warm"] + 1):
            out = v.step()
        out["new_grains"] = 0
        for f in case["fields"].split(","):
            out[f] = v.field(f)
        return out
    if kind == "batch":
        out = {}
        for i, (edge, grains, mat) in enumerate(_batch_members(case, seed)):
            _, _, _, euler, flat = _microstructure((edge,) * 3, grains, 0, seed * 1000 + i)
            v = _Volume((edge,) * 3, flat, euler, grains, mat, case["iters"])
            out["member%02d" % i] = {"sig_avg": v.step()["sig_avg"], "sig": v.field("sig")}
        return out
    if kind == "gradient":
        # the gradient is that of the converged fixed point: no short 64-bit formula gives it
        dims = (case["n"],) * 3
        _, _, _, euler, flat = _microstructure(dims, case["grains"], 0, seed)
        v = _Volume(dims, flat, euler, case["grains"], synth.Material(), case["iters"])
        s33 = np.array([float(v.step()["sig_avg"][2, 2]) for _ in range(case["steps"])])
        return {"misfit": np.array([((s33 - _target_curve(case["steps"])) ** 2).sum()]), "grad": None, "s33": s33}
    if kind == "local":
        x = _local_inputs(case, seed)
        b = _basis()
        mat = synth.Material(nrs=case["nrs"])
        q = _q(x["rot"].reshape(-1, 3, 3), b)
        ev = _cubic(mat)
        sdev = q.transpose(1, 2) @ (q / ev[:5, None])
        schmid, _, _ = _schmid(b)
        sig, edot, _ = _newton(x["lam"], x["strain"], x["epsp"], q, sdev, float(1 / ev[5]),
                               torch.linalg.inv(x["c066"]), _Power(mat, x["crss"]), 1e-3, schmid)
        tot = x["epsp"] + 1e-3 * edot - x["strain"]
        tot[:, :5] += (sdev @ sig[:, :5, None])[:, :, 0]
        tot[:, 5] += sig[:, 5] / ev[5]
        return {"sig": sig, "edot": edot, "err": torch.stack([(sig - x["lam"]).norm(dim=1), tot.norm(dim=1)], dim=1)}
    return None   # a sweep whose every voxel waits for the one before it (recrystallisation)
