"""The phase-field passes on the forms their tiles and tables tell apart, bit
for bit against the oracle's sequential sweep (FP64): grids that are no
multiples of a tile, edges below a tile and its halo, tiles of more than 64 ids
(which go through the lists), neighbourhoods of more ids than the stencil
planes hold, rows of more than 48 ids (the larger hash tables), several rows
per block, and lines too long for the row bitmaps."""
import numpy as np
import pytest

import pyoracle
from mth import capi, synth
from test_gpu_drx import gpu_pf, lib  # noqa: F401

pytestmark = pytest.mark.gpu


def block_grains(dims, edge, seed):
    """Grains of edge x edge x edge voxels in a random order of ids, the last
    tenth of the ids recrystallised."""
    ax = [np.arange(n) // e for n, e in zip(dims, edge)]
    n = [a[-1] + 1 for a in ax]
    idx = (ax[0][:, None, None] * n[1] + ax[1][None, :, None]) * n[2] + ax[2][None, None, :]
    rng = np.random.default_rng(seed)
    ids = int(np.prod(n))
    grain = (rng.permutation(ids) + 1)[idx].ravel().astype(np.int32)
    rho = (100.0 + 400.0 * rng.random(ids + 1))[grain] + 20.0 * rng.random(grain.size)
    init = max(1, ids - ids // 10)
    rho[grain > init] = 1.0
    return grain, rho, init, ids


@pytest.mark.parametrize("dims,edge,steps", [
    ((13, 7, 33), (4, 4, 4), 2),       # ragged tiles
    ((4, 8, 16), (2, 4, 8), 4),        # one tile, every neighbour periodic
    ((3, 2, 5), (1, 2, 3), 2),         # smaller than a tile and its halo
    ((9, 10, 37), (2, 2, 2), 2),       # over 64 ids a tile, three rows per block
    ((6, 6, 60), (3, 3, 2), 2),        # over 48 ids a row
    ((5, 4, 130), (2, 2, 6), 3),       # a row longer than a block
    ((4, 3, 1500), (2, 2, 90), 2),     # no row bitmaps: the walk along the row
])
def test_relaxation_equals_the_sweep(lib, dims, edge, steps):  # noqa: F811
    g, rho, init, ids = block_grains(dims, edge, seed=sum(dims))
    par = capi.params_from_config(synth.Config(cell_dim=dims, drx=synth.Drx(stored_energy_scale=20.0)),
                                  precision=capi.MTH_FP64)
    table = np.zeros(ids)
    o = pyoracle.pf_relax(par, dims, g, rho, steps, init, table, kmax=capi.PF_K)
    r = gpu_pf(lib, par, dims, g, rho, steps, init, table)
    assert np.array_equal(r[0], o[0])                                     # grain map
    assert np.array_equal(r[3], o[3]) and np.array_equal(r[1], o[1])      # lists, in stored order
    assert np.array_equal(r[2].view(np.int64), o[2].view(np.int64))
    assert np.array_equal(r[4].view(np.int64), np.asarray(o[4]).view(np.int64))   # rho_avg table
