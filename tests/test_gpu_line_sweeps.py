"""The stencil kernels' line sweeps, general tiles, joined steps and field
transfers at the sizes where they can go wrong: edges of the 32 x 8 tiles,
remainders, single tiles and boxes that reach every edge of the domain.

FP64 is compared with the oracle: rounding (1e-16 a step) grows by less than
a factor of 10 over 9 steps of these flows, 1e-11 is the suite's bound for a
dozen steps.  Other tile shapes, steps taken phase by phase and joined steps
do the same operations on every node: bit for bit, in both precisions.
"""
import numpy as np
import pytest

from golden_util import rel_l2
from oracle import oracle as O
from uq_b200 import workloads as W
from uq_b200.solver import Batch

pytestmark = pytest.mark.gpu

STEPS = 9  # one graph of eight joined steps and one of one step
SMALL = dict(du=0.02, drho=0.02, dT=0.02)
# one tile, tiles cut by one and by all but one node, several tiles each way,
# narrower than the ghost columns
SIZES = [(32, 8), (33, 9), (31, 7), (64, 24), (5, 6), (97, 17)]


def _obstacle(nx, ny, **kw):
    """A Couette flow around a solid block: general tiles among swept ones."""
    case = W.couette(nx=nx, ny=ny, **kw)
    for k in ("density", "pressure", "temp", "velocityX", "velocityY"):
        case[k] = np.append(case[k], 1.0 if k in ("density", "temp") else 0.0)
    case["cellType"] = np.append(case["cellType"], 2)
    case["numProps"] = len(case["density"])
    case["bnd"] = case["bnd"].copy()
    case["bnd"][nx // 2:nx // 2 + 2, ny // 2:ny // 2 + 2] = case["numProps"] - 1
    return case


FLOWS = {
    "couette": lambda nx, ny, **kw: W.couette(nx=nx, ny=ny, steps=STEPS, seed=3, **kw),
    "obstacle": lambda nx, ny, **kw: _obstacle(nx, ny, steps=STEPS, seed=4, **kw),
    "riemann": lambda nx, ny, **kw: W.riemann(nx=nx, ny=ny, tau=0.02, steps=STEPS, **kw),
    "plate": lambda nx, ny, **kw: W.flat_plate(nx=nx, ny=ny, tau=0.02, mach=0.2, Tc_Tref=1.5, steps=STEPS, **kw),
    "periodic": lambda nx, ny, **kw: W.random_state(nx, ny, 5, bc="periodic", steps=STEPS, **SMALL, **kw),
    "mirror": lambda nx, ny, **kw: W.random_state(nx, ny, 6, bc="mirror", solid_frac=0.05, steps=STEPS, **SMALL, **kw),
}


def _dists(cases, prec, **kw):
    b = Batch(cases, prec, **kw)
    b.step(STEPS)
    out = [b.dist(s) for s in range(len(cases))], b.status()
    b.close()
    return out


@pytest.mark.parametrize("flow", sorted(FLOWS))
@pytest.mark.parametrize("rk,fm", [(1, 1), (1, 0), (0, 1)])
def test_fp64_tile_edges_match_oracle(cuda_device, flow, rk, fm):
    cases = [FLOWS[flow](nx, ny, rkmethod=rk, fmethod=fm) for nx, ny in SIZES]
    got, status = _dists(cases, "f64")
    for case, size, (f, h), st in zip(cases, SIZES, got, status):
        o = O.Oracle(case)
        failed, _ = o.step(STEPS)
        assert (st == 0) == (not failed), size
        if failed:
            continue
        fo, ho = o.dist()
        assert rel_l2(f, fo) < 1e-11 and rel_l2(h, ho) < 1e-11, (size, rel_l2(f, fo), rel_l2(h, ho))


@pytest.mark.parametrize("prec", ["f32", "f64"])
@pytest.mark.parametrize("rks,fm", [((1,), 1), ((0,), 0), ((2,), 1), ((3,), 0), ((1, 0, 1, 2, 3), 1)])
def test_forms_of_a_step_agree_bit_for_bit(cuda_device, prec, rks, fm):
    pairs = [(f, size) for f in sorted(FLOWS) for size in SIZES[1:5]]
    cases = [FLOWS[f](nx, ny, rkmethod=rks[k % len(rks)], fmethod=fm) for k, (f, (nx, ny)) in enumerate(pairs)]
    want, _ = _dists(cases, prec)
    for kw in (dict(tile=(16, 16)), dict(tile=(64, 4)), dict(use_graph=False)):
        got, _ = _dists(cases, prec, **kw)
        for k, ((f, h), (fw, hw)) in enumerate(zip(got, want)):
            assert np.array_equal(f, fw, equal_nan=True) and np.array_equal(h, hw, equal_nan=True), (kw, k)
    # nine steps one at a time, none joined
    b = Batch(cases, prec)
    for _ in range(STEPS):
        b.step(1)
    for k, (fw, hw) in enumerate(want):
        f, h = b.dist(k)
        assert np.array_equal(f, fw, equal_nan=True) and np.array_equal(h, hw, equal_nan=True), k
    b.close()


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_fields_in_and_out_at_ragged_sizes(cuda_device, prec):
    """Fields set for all samples at once, and sample by sample, and read back
    both ways; macroscopic values come back to the rounding of the stored
    type (13 additions: 16 eps)."""
    cases = [FLOWS["periodic"](nx, ny) for nx, ny in SIZES]
    b, c = Batch(cases, prec), Batch(cases, prec)
    rng = np.random.default_rng(8)
    fields = [{k: rng.uniform(*r, (nx, ny)) for k, r in
               (("rho", (0.9, 1.1)), ("ux", (-0.1, 0.1)), ("uy", (-0.1, 0.1)), ("T", (0.9, 1.1)))} for nx, ny in SIZES]
    b.set_macro_all(fields)
    for s, v in enumerate(fields):
        c.set_macro(s, v["rho"], v["ux"], v["uy"], v["T"])
    eps = np.finfo(np.float32 if prec == "f32" else np.float64).eps
    every = b.macro_all()
    for s, v in enumerate(fields):
        one = c.macro(s)
        for k in one:
            assert np.array_equal(one[k], every[s][k]), (s, k)
        for k in v:
            assert np.max(np.abs(one[k] - v[k])) <= 16 * eps, (s, k)
        f, h = b.dist(s)
        fc, hc = c.dist(s)
        assert np.array_equal(f, fc) and np.array_equal(h, hc), s
        b.set_dist(s, f, h)
        fb, hb = b.dist(s)
        assert np.array_equal(f, fb) and np.array_equal(h, hb), s
    b.close()
    c.close()


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_residual_sums_every_tile(cuda_device, prec):
    """The residual, the RMS change of T over the nodes, from the fields before
    and after the step."""
    cases = [FLOWS["periodic"](nx, ny) for nx, ny in SIZES + [(200, 130)]]
    b = Batch(cases, prec)
    b.step(1)
    before = [b.macro(s)["T"] for s in range(b.n)]
    b.step(1, residual=True)
    got = b.residuals()
    for s, T in enumerate(before):
        want = np.sqrt(np.mean((b.macro(s)["T"] - T) ** 2))
        assert abs(got[s] - want) <= 1e-12 + (1e-6 if prec == "f32" else 1e-11) * want, (s, got[s], want)
    b.close()
