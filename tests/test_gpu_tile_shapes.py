"""Tile shapes at the ends of what is accepted: wider than an FP64 box row may
be as one dimension of a tensor map, lower than a line segment (whose rows
then lie beyond the box), one row, four columns.  Every node must get the bits
it gets on the default tile, and every flow here stays finite."""
import numpy as np
import pytest

from test_gpu_line_sweeps import FLOWS, STEPS
from uq_b200.solver import Batch

pytestmark = pytest.mark.gpu

SIZES = [(261, 17), (140, 9), (33, 24), (5, 70)]  # beyond two 128-wide tiles, ragged both ways


def _run(cases, prec, tile):
    b = Batch(cases, prec, tile=tile)
    b.step(STEPS)
    out = [b.dist(s) for s in range(len(cases))]
    assert not b.status().any()
    b.close()
    return out


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("fm", [0, 1])
def test_extreme_tile_shapes_agree_bit_for_bit(cuda_device, prec, fm):
    cases = [FLOWS[f](nx, ny, rkmethod=rk, fmethod=fm) for rk in (0, 1, 3) for f in sorted(FLOWS) for nx, ny in SIZES]
    want = _run(cases, prec, (32, 8))
    assert all(np.isfinite(f).all() and np.isfinite(h).all() for f, h in want)
    for tile in ((128, 2), (32, 1), (32, 2), (4, 64)):
        got = _run(cases, prec, tile)
        for k, ((f, h), (fw, hw)) in enumerate(zip(got, want)):
            assert np.array_equal(f, fw) and np.array_equal(h, hw), (tile, k)
