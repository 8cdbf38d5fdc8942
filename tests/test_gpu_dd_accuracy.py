"""How far the mixed dislocation-density step is from the FP64 one, over six
volumes: at most as far as an iteration with FP64 systems and Q^T rotations,
1.83e-7 (stress) and 2.13e-7 (SSD density), and two percent."""
import numpy as np
import pytest

from helpers import rel_l2
from mth import Solver, capi, synth

pytestmark = pytest.mark.gpu


def test_mixed_step_keeps_its_accuracy():
    err = []
    for seed in range(81, 87):
        cfg = synth.Config(cell_dim=(32, 32, 32), n_grains=12, n_steps=1, seed=seed, iter_max=40, dd=synth.DD())
        micro = synth.microstructure(cfg)
        out = []
        for precision in (capi.MTH_FP64, capi.MTH_MIXED):
            with Solver(capi.params_from_config(cfg, precision=precision), *micro) as s:
                s.step()
                out.append((s.field("sig"), s.field("rho_ssd")))
        err.append([rel_l2(b, a) for a, b in zip(*out)])
    sig, rho = np.mean(err, axis=0)
    assert sig <= 1.02 * 1.83e-7 and rho <= 1.02 * 2.13e-7
