"""The local-solve kernels over every form their dispatch tells apart: block
sizes (32, 64 and 128 threads with ragged last blocks), whole, half and other
rate exponents, equal and unequal forward/backward CRSS, fewer than twelve
systems, and iteration caps that keep every pass in FP64.  The FP64 kernels are
held to the oracle as in test_gpu_parity.py (both solve to 1e-10 |lambda|); the
mixed modes to their stated 1e-4.  The oracle keeps the reference's pow of a
negative base, NaN for an exponent that is no whole number; there the reference
is the iteration with every pass in FP64 (which a cap below 50 selects)."""
import numpy as np
import pytest

from helpers import rel, rel_l2, run_oracle
from mth import Solver, capi, local_solve, synth

pytestmark = pytest.mark.gpu


def _against_oracle(n, nrs=10.0, off=0.0, itmax=0, nsys=12, seed=11):
    import pyoracle
    from test_oracle_cpu import random_states
    cfg = synth.Config(cell_dim=(8, 8, 8), n_grains=4)
    p = capi.params_from_config(cfg)
    o = pyoracle.Oracle(p, *synth.microstructure(cfg), nthreads=2)
    c066 = o.c066()
    p.phase[0].nrs = nrs
    p.phase[0].tau0b = p.phase[0].tau0f + off
    p.phase[0].nsys = nsys
    st = random_states(n, np.random.default_rng(seed), cfg)
    if nrs == int(nrs):
        so, eo, erro, _ = pyoracle.local_solve(p, c066, *st)
    else:
        p.newton_itmax = 49
        so, eo, erro, _ = local_solve(p, c066, *st)
    p.newton_itmax = itmax   # the oracle's undamped start takes up to 500
    sg, eg, errg, it = local_solve(p, c066, *st)
    assert it > 0
    assert rel(sg, so) < 1e-8
    assert rel(eg, eo) < 1e-6
    assert rel(errg[:, 0], erro[:, 0]) < 1e-6


@pytest.mark.parametrize("n", [1, 31, 33, 129, 19487, 38977])
def test_point_counts(n):
    _against_oracle(n)


@pytest.mark.parametrize("nrs", [1.0, 2.0, 1.5, 8.0, 12.5, 11.3, 20.0])
@pytest.mark.parametrize("off", [0.0, 3.0])
def test_exponents_and_backward_crss(nrs, off):
    _against_oracle(257, nrs=nrs, off=off)


@pytest.mark.parametrize("kw", [dict(itmax=40), dict(nsys=5), dict(nsys=5, off=-2.0)])
def test_caps_and_fewer_systems(kw):
    _against_oracle(65, **kw)


def test_zero_start():
    """lambda = 0 (a voxel after a recrystallisation reset): the tolerance is then
    relative to the stress itself."""
    import pyoracle
    from test_oracle_cpu import random_states
    cfg = synth.Config(cell_dim=(8, 8, 8), n_grains=4)
    p = capi.params_from_config(cfg)
    c066 = pyoracle.Oracle(p, *synth.microstructure(cfg), nthreads=2).c066()
    st = list(random_states(40, np.random.default_rng(5), cfg))
    st[0] = np.zeros_like(st[0])
    full = capi.params_from_config(cfg, newton_itmax=49)     # every pass in FP64
    s0, e0, _, _ = local_solve(full, c066, *st)
    s1, e1, _, _ = local_solve(p, c066, *st)
    assert rel(s1, s0) < 1e-9 and rel(e1, e0) < 1e-8         # a step of 1e-10, amplified by n = 10


@pytest.mark.parametrize("precision", [capi.MTH_MIXED, capi.MTH_MIXED_FAST, capi.MTH_MIXED_ROOT64, capi.MTH_FP64])
@pytest.mark.parametrize("nrs,tau0b", [(10.0, 16.0), (12.5, 16.0), (11.3, 16.0), (10.0, 18.0)])
def test_volume_forms(precision, nrs, tau0b):
    cfg = synth.Config(cell_dim=(16, 8, 12), n_grains=5, n_pores=1, pore_radius=2, n_steps=3, seed=53, iter_max=10,
                       material=synth.Material(nrs=nrs, tau0b=tau0b))
    g, p, e = synth.microstructure(cfg)
    if nrs == int(nrs):
        o, ro = run_oracle(cfg)
    else:
        o = Solver(capi.params_from_config(cfg, newton_itmax=49), g, p, e)
        ro = [o.step() for _ in range(cfg.n_steps)]
    with Solver(capi.params_from_config(cfg, precision=precision), g, p, e) as s:
        tol = 1e-6 if precision == capi.MTH_FP64 else 1e-4
        for b in ro:
            a = s.step()
            assert rel(a["sig_avg"], b["sig_avg"]) < tol
            assert a["newton_failed"] == 0
        assert rel_l2(s.field("sig"), o.field("sig")) < tol
    o.close()


@pytest.mark.parametrize("precision", [capi.MTH_MIXED, capi.MTH_MIXED_FAST, capi.MTH_MIXED_ROOT64])
def test_steep_first_step_recovers(precision):
    """n = 20 at a low CRSS: in the first iteration the Newton steps of some voxels are too
    long to square in FP32; the line search brings them back and no NaN leaves the solve."""
    cfg = synth.Config(cell_dim=(64, 64, 64), n_grains=160, n_steps=2, seed=3, iter_max=60,
                       material=synth.Material(nrs=20.0, tau0f=12.0, tau0b=12.0))
    g, p, e = synth.microstructure(cfg)
    with Solver(capi.params_from_config(cfg, precision=precision), g, p, e) as s:
        r = [s.step() for _ in range(2)]
        assert np.all(np.isfinite(s.field("sig"))) and r[1]["newton_failed"] == 0


@pytest.mark.parametrize("nrs", [2.0, 5.5, 10.0, 20.0, 40.5])
def test_fp64_mode_is_the_all_fp64_iteration(nrs):
    """The first of the FP64 mode's last steps takes its rates in pairs of FP32 numbers (whole
    and half exponents); the converged fields are those of the iteration in FP64 throughout
    (newton_itmax below 50).  Both end with an error far below the tolerance's 1e-10."""
    cfg = synth.Config(cell_dim=(16, 12, 8), n_grains=6, n_steps=2, seed=19, iter_max=8,
                       material=synth.Material(nrs=nrs))
    g, p, e = synth.microstructure(cfg)
    out = []
    for kw in ({}, {"newton_itmax": 49}):
        with Solver(capi.params_from_config(cfg, precision=capi.MTH_FP64, **kw), g, p, e) as s:
            for _ in range(cfg.n_steps):
                s.step()
            out.append((s.field("sig"), s.field("edot"), s.field("crss")))
    for a, b, tol in zip(*out, (1e-12, 1e-11, 1e-12)):   # edot: amplified by n
        assert rel_l2(a, b) < tol
