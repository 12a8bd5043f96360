"""
The tile shape of a disk by its own size, which callers pass in `tiles`.
"""

import pytest

pytest.importorskip("torch")

from sailfish_b200.batched import default_tile  # noqa: E402


@pytest.mark.parametrize("size,tile", [((1, 1), (64, 16)), ((511, 96), (64, 16)), ((512, 96), (64, 32)),
                                       ((511, 97), (128, 16)), ((512, 97), (128, 32)), ((4096, 4096), (128, 32))])
def test_default_tile(size, tile):
    assert default_tile(*size) == tile
