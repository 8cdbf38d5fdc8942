"""CRSS at or below zero in a local solve, forward or backward (softening laws;
a backward CRSS below the forward one).  Such a solve has no positive definite
system to rely on: no kernel may treat the system as one that does not slip or
take a reciprocal of another sign."""
import numpy as np
import pytest

from mth import Solver, capi, local_solve, synth

pytestmark = pytest.mark.gpu


def _softening(thet, precision):
    cfg = synth.Config(cell_dim=(16, 8, 12), n_grains=5, n_steps=3, seed=53, iter_max=10,
                       material=synth.Material(thet0=thet, thet1=thet, tau1=0.0))
    return Solver(capi.params_from_config(cfg, precision=precision), *synth.microstructure(cfg))


@pytest.mark.parametrize("precision", [capi.MTH_MIXED, capi.MTH_MIXED_FAST, capi.MTH_MIXED_ROOT64])
def test_softened_system_is_reported(precision):
    """The report shows a step whose solves meet a CRSS below zero: failed solves, or the error
    on a field that is not finite where the whole volume softened."""
    with _softening(-2000.0, precision) as s:
        assert s.step()["newton_failed"] == 0 and s.step()["newton_failed"] == 0
        crss = np.asarray(s.field("crss"))
        assert (crss < 0).any() and (crss > 0).any()
        assert s.step()["newton_failed"] > 0
    with _softening(-6000.0, precision) as s:
        s.step()
        with pytest.raises(capi.MthError):
            s.step()


@pytest.mark.parametrize("off", [-4.0, -12.0])
def test_array_points_below_the_backward_offset(off):
    """Points whose CRSS lies below tau0f - tau0b: the result is the iteration's with every
    pass in FP64 (a cap below 50 selects it)."""
    import pyoracle
    from test_oracle_cpu import random_states
    cfg = synth.Config(cell_dim=(8, 8, 8), n_grains=4)
    p = capi.params_from_config(cfg)
    c066 = pyoracle.Oracle(p, *synth.microstructure(cfg), nthreads=2).c066()
    p.phase[0].tau0b = p.phase[0].tau0f + off
    st = [np.array(x) for x in random_states(65, np.random.default_rng(11), cfg)]
    st[4][::3] *= 0.1
    assert (st[4] + off < 0).any() and (st[4] + off > 0).any()
    p.newton_itmax = 49
    full = local_solve(p, c066, *st)
    p.newton_itmax = 0
    got = local_solve(p, c066, *st)
    for a, b in zip(got[:2], full[:2]):
        assert np.abs(a - b).max() <= 1e-8 * np.abs(b).max()   # both solve to 1e-10 |lambda|
