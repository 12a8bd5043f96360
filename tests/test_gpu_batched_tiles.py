"""
The default tile shapes of a batch (one wave of short tiles; short tiles for
the smallest disks of a larger batch): the rule on the host, and the states of
a few small batches against each disk's own run, bit for bit.
"""

import numpy as np
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

from sailfish_b200.batched import BatchedSolver, Disk, default_tiles  # noqa: E402
from sailfish_b200.cbdiso_2d import Solver  # noqa: E402
from sailfish_b200.setups import CircumbinaryDisk  # noqa: E402


@pytest.mark.parametrize("sizes", [[(1, 1)], [(64, 64)] * 3, [(5, 4000), (4000, 5)], [(128, 128)] * 200,
                                   [(1024, 1024)] * 24, [(128, 128), (2048, 2048)], [(96, 97), (97, 96)] * 7])
def test_rule_covers_every_size(sizes):
    tiles = default_tiles(sizes)
    assert set(tiles) == set(sizes)
    units = 0
    for ni, nj in sizes:
        width, rows = tiles[ni, nj]
        assert width == (128 if nj > 96 else 64) and 1 <= rows <= 32
        units += -(-nj // width) * -(-ni // rows)
    # one wave, or tiles of at least 8 rows
    assert units <= 148 * 6 or all(rows >= 8 for _, rows in tiles.values())


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(48, 48), (1, 130, 97), (128, 64, 256), (200, 200, 300, 500, 130, 640)])
def test_states_equal_single_runs(sizes):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    disks = []
    for q, n in enumerate(sizes):
        setup = CircumbinaryDisk(domain_radius=6.0, mass_ratio=0.4 + 0.1 * q, eccentricity=0.1, nu=1e-3)
        disks.append(Disk(setup, setup.mesh(n)))
    b = BatchedSolver(disks)
    b.run(3)
    for i, d in enumerate(disks):
        s = Solver(setup=d.setup, mesh=d.mesh, physics=d.setup.physics, options=dict(rk_order=2, plm_theta=1.5))
        s.run(3)
        assert np.array_equal(b.solution(i), s.solution)
