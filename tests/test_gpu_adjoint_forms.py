"""The adjoint on grids whose projections take the tile passes on every axis,
on z alone and on none, with whole, half and other exponents, against central
differences (bound 1e-3, relative step 1e-4, as on the cubic grid), and the
end of its conjugate-gradient solve at the iteration limit."""
import dataclasses

import numpy as np
import pytest

from mth import MthError, Solver, capi, synth

pytestmark = pytest.mark.gpu


def _cfg(dims, mat, **kw):
    return synth.Config(cell_dim=dims, n_grains=4, n_steps=2, seed=41, material=mat, err=1e-10, iter_max=2500, **kw)


def _curve(cfg):
    with Solver(capi.params_from_config(cfg, precision=capi.MTH_FP64), *synth.microstructure(cfg)) as s:
        return np.array([s.step()["sig_avg"][2][2] for _ in range(cfg.n_steps)])


@pytest.mark.parametrize("dims,nrs", [((18, 8, 24), 10.0), ((12, 8, 18), 10.5), ((8, 16, 6), 10.3)])
def test_gradient_matches_central_differences(dims, nrs):
    base = dataclasses.replace(synth.Material(), nrs=nrs)
    tgt = 0.9 * _curve(_cfg(dims, base))
    cfg = _cfg(dims, base)
    with Solver(capi.params_from_config(cfg, precision=capi.MTH_FP64), *synth.microstructure(cfg)) as s:
        _, grad, _, info = s.adjoint(tgt, checkpoint_every=2)
    assert info["cg_iterations"] > 0
    vals = synth.calibration_values(base)
    for k in (0, 4):
        h = 1e-4 * vals[k]
        jp, jm = (np.sum((_curve(_cfg(dims, synth.perturb_material(base, k, d))) - tgt) ** 2) for d in (h, -h))
        fd = (jp - jm) / (2 * h)
        assert abs(grad[k] - fd) <= 1e-3 * abs(fd), (k, grad[k], fd)


@pytest.mark.parametrize("precision", [capi.MTH_FP64, capi.MTH_MIXED])
def test_iteration_limit_is_an_error(precision):
    cfg = _cfg((18, 8, 24), synth.Material())
    with Solver(capi.params_from_config(cfg, precision=precision), *synth.microstructure(cfg)) as s:
        with pytest.raises(MthError, match="CG did not reach"):
            s.adjoint(np.zeros(2), checkpoint_every=2, cg_itmax=1)
