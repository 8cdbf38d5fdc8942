"""The Newton steps the mixed modes' local solves take: those of a solve whose
every system is assembled at the iterate and solved in FP64 (counted with such a
kernel, volume and step by step).  A solve at the edge of the tolerance may take
one more or fewer, so the counts agree to half a percent; closing steps with an
older, unrefined Jacobian would add three."""
import pytest

from mth import Solver, capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [capi.MTH_MIXED, capi.MTH_MIXED_ROOT64])
@pytest.mark.parametrize("nrs,steps", [(10.0, (692002, 685080)), (15.0, (766004, 756412)), (20.0, (812687, 801561))])
def test_mixed_modes_take_plain_newton_steps(precision, nrs, steps):
    cfg = synth.Config(cell_dim=(32, 16, 24), n_grains=12, n_steps=3, seed=71, iter_max=20,
                       material=synth.Material(nrs=nrs))
    with Solver(capi.params_from_config(cfg, precision=precision), *synth.microstructure(cfg)) as s:
        s.step()
        for n in steps:
            assert abs(s.step()["newton_iters"] - n) < 5e-3 * n
