"""Batches of more samples than a grid holds along y (65,535): creation,
bulk fields, single samples.  Every sample must do what it does in a batch of
a few, bit for bit."""
import numpy as np
import pytest

from uq_b200 import workloads as W
from uq_b200.solver import Batch

pytestmark = pytest.mark.gpu

KINDS = 5  # samples repeat with this period; it divides no launch's share


@pytest.mark.parametrize("extra", [0, 1, 65536])  # a full launch, one sample in the last, two full and one
def test_more_samples_than_a_grid_dimension(cuda_device, extra):
    few = [W.random_state(4, 3, seed, bc="periodic", du=0.02, drho=0.02, dT=0.02) for seed in range(KINDS)]
    n = 65535 + extra
    many, ref = Batch([few[k % KINDS] for k in range(n)], "f32"), Batch(few, "f32")

    def same():
        ref.step(1)
        many.step(1)
        want, got = ref.macro_all(), many.macro_all()
        for q in ("rho", "ux", "uy", "T", "p"):
            have = np.stack([m[q] for m in got])
            full = np.stack([m[q] for m in want])[np.arange(n) % KINDS]
            assert np.array_equal(have, full) and np.all(np.isfinite(have)), q
        f, h = many.dist(n - 1)
        fr, hr = ref.dist((n - 1) % KINDS)
        assert np.array_equal(f, fr) and np.array_equal(h, hr)
        assert not many.status().any()

    same()
    rng = np.random.default_rng(4)
    fields = [{"rho": rng.uniform(0.98, 1.02, (4, 3)), "T": rng.uniform(0.98, 1.02, (4, 3)),
               "ux": rng.uniform(-0.02, 0.02, (4, 3)), "uy": rng.uniform(-0.02, 0.02, (4, 3))} for _ in range(KINDS)]
    ref.set_macro_all(fields)
    many.set_macro_all([fields[k % KINDS] for k in range(n)])
    same()
    many.close()
    ref.close()
