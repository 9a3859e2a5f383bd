"""The staged stencils, which grids of more than 256 columns run for multiples of 32
chains, against the direct-load kernels bit for bit: steps with and without
correlation, moment tensors, several sources and shots, two tiles of chains, ragged tiles of cells."""
import pytest

import test_fwi_onchip as OC
from hmclab_gb300 import fwi as FW
from test_fwi_strips import strips

pytestmark = pytest.mark.gpu


def _staged(C, nx=256, nz=30, **kw):
    cfg = OC._config(nx, nz, **kw)
    (dist, direct), _ = OC._pair(cfg, C)
    # off chip, with a status word and whole tiles of chains: the staged stencils
    assert strips(dist, C) == (0, 0) and C % 32 == 0 and dist.staged_tiles and not direct.staged_tiles
    OC._check(cfg, C)


@pytest.mark.parametrize("k,nt", [(1, 30), (2, 41), (3, 30), (7, 50)])
def test_snapshots(k, nt):
    _staged(32, nt=nt, snapshot_interval=k)


def test_two_tiles_of_chains_and_ragged_cells():
    _staged(64, nx=250, nz=29, nt=30, snapshot_interval=2)  # 266 columns and 45 rows of 8 x 4 tiles


@pytest.mark.parametrize("k", [1, 3])
def test_sources_and_shots(k):
    P = FW.PointSource
    shots = [[P(20, 15), P(31, 18, *FW.moment_tensor(30.0), delay=0.004), P(30, 18, *FW.moment_tensor(75.0))],
             [P(200, 9, *FW.moment_tensor(110.0))]]
    _staged(32, nt=60, shots=shots, snapshot_interval=k)
