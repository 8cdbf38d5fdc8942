"""Long first Newton steps in the FP32 modes (n = 20 at a CRSS of 12 MPa): the
rounding of the FP32 Hessian decides which solves find a pivot that is not
positive; those keep their iterate and are counted in newton_failed, and the
volume's later iterations start from their stresses.  Such steps run in plain
order (book.cuh), whose results the fixture holds: failure counts and stresses
of every precision mode, recorded on a GB300 from kernels that run every solve
and transform in that order.  Fields held in FP32 agree to 2e-5 where roundings
differ; the counts are equal."""
import os

import numpy as np
import pytest

from helpers import GOLDEN, rel, rel_l2
from mth import Batch, Solver, capi, synth

pytestmark = pytest.mark.gpu

PRECISION = {"mixed": capi.MTH_MIXED, "fast": capi.MTH_MIXED_FAST, "root64": capi.MTH_MIXED_ROOT64}
FP32_FIELD = 2e-5


@pytest.fixture(scope="module")
def gold():
    return np.load(os.path.join(GOLDEN, "steep_first_steps.npz"))


def _volume(seed):
    cfg = synth.Config(cell_dim=(16, 16, 16), n_grains=20, n_steps=2, seed=seed, iter_max=20,
                       material=synth.Material(nrs=20.0, tau0f=12.0, tau0b=12.0))
    return cfg, synth.microstructure(cfg)


def _check(gold, key, step, rep, sig):
    assert rep["newton_failed"] == gold[key + "_failed"][step], key
    assert rel(rep["sig_avg"], gold[key + "_sig_avg"][step]) < FP32_FIELD, key
    if step == 0 and key + "_sig" in gold.files:
        assert rel_l2(np.asarray(sig)[::4][:, [0, 1, 2, 4, 5, 8]], gold[key + "_sig"]) < FP32_FIELD, key


@pytest.mark.parametrize("mode", sorted(PRECISION))
@pytest.mark.parametrize("seed", [4, 11, 13])
def test_volume(gold, mode, seed):
    cfg, micro = _volume(seed)
    assert gold["%s_%d_failed" % (mode, seed)][0] > 0
    with Solver(capi.params_from_config(cfg, precision=PRECISION[mode]), *micro) as s:
        for step in range(2):
            rep = s.step()
            _check(gold, "%s_%d" % (mode, seed), step, rep, s.field("sig"))


def test_batch_members(gold):
    """Members with and without failures in one batch: the loop's kernels are chosen per member,
    and again when the second step has no failures left."""
    cfgs, micro = zip(*[_volume(s) for s in (11, 5, 4)])
    with Batch([capi.params_from_config(c, precision=capi.MTH_MIXED) for c in cfgs], list(micro)) as b:
        for step in range(2):
            reps = b.step()
            for i, seed in ((0, 11), (2, 4)):
                _check(gold, "mixed_%d" % seed, step, reps[i], b.field(i, "sig"))
            assert reps[1]["newton_failed"] == 0


@pytest.mark.parametrize("tau0,seed", [(12.0, 4), (12.5, 34)])
def test_step_after_failures(tau0, seed):
    """The step after one with failures stays in plain order: the 64 voxels that come out most
    different (by up to 3e-4 of the field's rms) when it leaves that order after its first
    iteration.  The order keeps the bits; the fields' 2e-5 is allowed."""
    gold = np.load(os.path.join(GOLDEN, "steep_second_steps.npz"))
    cfg = synth.Config(cell_dim=(32, 32, 16), n_grains=20, n_steps=2, seed=seed, iter_max=20,
                       material=synth.Material(nrs=20.0, tau0f=tau0, tau0b=tau0))
    with Solver(capi.params_from_config(cfg, precision=capi.MTH_MIXED_FAST), *synth.microstructure(cfg)) as s:
        assert s.step()["newton_failed"] > 0
        s.step()
        sig = np.asarray(s.field("sig"))[gold["voxels_%d" % seed]][:, [0, 1, 2, 4, 5, 8]]
    assert np.abs(sig - gold["sig_%d" % seed]).max() < FP32_FIELD * gold["rms_%d" % seed]
