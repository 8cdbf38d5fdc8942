"""The Green iteration's tile passes over their line lengths: every length that
is not a power of two on every axis, short tiles (8, 18), lines longer than a
block has threads for (144, 192), z rows that are no multiple of 16 bytes (18,
54 in FP32) and a last tile of z lines that is part empty, against the oracle.
Bounds: FP64 1e-6 and mixed 1e-4, those of the other shapes (rounding of the
transforms is 1e-15 / 1e-6 of the stress; the local solve's tolerance sets the
rest)."""
import pytest

from helpers import rel, rel_l2, run_gpu, run_oracle
from mth import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(18, 24, 36), (54, 8, 72), (24, 108, 18), (36, 18, 54), (72, 36, 8), (8, 54, 24),
                                  (108, 72, 16), (16, 8, 108), (144, 8, 18), (8, 192, 144), (192, 144, 8), (12, 18, 24)])
@pytest.mark.parametrize("precision", [capi.MTH_FP64, capi.MTH_MIXED])
def test_lengths_match_oracle(dims, precision):
    cfg = synth.Config(cell_dim=dims, n_grains=9, n_steps=2, seed=57, iter_max=4)
    o, ro = run_oracle(cfg)
    s, rg = run_gpu(cfg, precision)
    tol = 1e-6 if precision == capi.MTH_FP64 else 1e-4
    for a, b in zip(rg, ro):
        assert precision == capi.MTH_MIXED or a["iterations"] == b["iterations"]
        assert rel(a["sig_avg"], b["sig_avg"]) < tol
    assert rel_l2(s.field("sig"), o.field("sig")) < tol
    assert rel_l2(s.field("strain"), o.field("strain")) < tol
    s.close()
