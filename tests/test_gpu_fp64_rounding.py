"""Rounding of one FP64 step, against the same step in extended precision.

The bound is the FP64 oracle's own error, the scheme evaluated as the
reference writes it: the kernels reorder sums, use reciprocals and work on
differences, and none of that may cost accuracy.  Root mean square over three
states, f and h together.
"""
import numpy as np
import pytest

from oracle import oracle as O
from uq_b200 import workloads as W
from uq_b200.solver import Batch

FLOWS = {
    "couette": lambda seed, **kw: W.couette(nx=40, ny=45, seed=seed, tau=0.03, noise=1e-4, **kw),
    "plate": lambda seed, **kw: W.flat_plate(nx=40, ny=45, tau=2e-3 / seed, mach=1.5 + 0.2 * seed, Tc_Tref=4.0, **kw),
    "riemann": lambda seed, **kw: W.riemann(nx=40, ny=45, tau=1e-3 * seed, Tc_Tref=1.5, **kw),
}


def _start(case):
    """A state a few steps on, from the oracle: every gradient is there."""
    o = O.Oracle(case)
    o.step(3)
    return o.dist()


def _error(got, want):
    e = [((g - w).astype(np.float64), w.astype(np.float64)) for g, w in zip(got, want)]
    return sum(np.sum(d ** 2) / np.sum(w ** 2) for d, w in e)


def _errors(flow, rk, fm, step):
    """(error of `step`, error of the FP64 oracle)"""
    mine = oracle = 0.0
    for seed in (1, 2, 3):
        case = FLOWS[flow](seed, rkmethod=rk, fmethod=fm, steps=1)
        f, h = _start(case)
        want = O.Extended(case).step_from(f, h)
        o = O.Oracle(case)
        o.set_dist(f, h)
        assert o.step(1)[0] == 0
        oracle += _error(o.dist(), want)
        mine += _error(step(case, f, h), want)
    return np.sqrt(mine), np.sqrt(oracle)


def _gpu(case, f, h):
    b = Batch([case], "f64")
    b.set_dist(0, f, h)
    b.step(1)
    assert b.status()[0] == 0
    out = b.dist(0)
    b.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("flow", sorted(FLOWS))
@pytest.mark.parametrize("rk,fm", [(1, 1), (1, 0), (0, 1), (0, 0)])
def test_a_step_rounds_no_worse_than_the_reference_arithmetic(cuda_device, flow, rk, fm):
    mine, oracle = _errors(flow, rk, fm, _gpu)
    assert mine <= oracle, (mine, oracle)


def test_extended_oracle_is_the_oracle():
    """The two oracles differ by FP64 rounding: a step is some hundred
    operations on values near 1."""
    zero, oracle = _errors("couette", 1, 1, lambda case, f, h: O.Extended(case).step_from(f, h))
    assert zero == 0 and 1e-17 < oracle < 100 * np.finfo(np.float64).eps
