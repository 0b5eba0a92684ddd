"""FP64 far from 1: relaxation times and densities at which the intermediate
products of a face or a relaxation are large.  Each case has a twin in an
ordinary range with the same flow."""
import numpy as np
import pytest

from uq_b200 import workloads as W
from uq_b200.solver import Batch

pytestmark = pytest.mark.gpu


def _run(cases, steps=3):
    b = Batch(cases, "f64")
    b.step(steps)
    out = [b.macro(s) for s in range(b.n)]
    b.close()
    return out


@pytest.mark.parametrize("rk", [0, 1])
def test_vanishing_relaxation_time(cuda_device, rk):
    """mu -> 0: the stages relax onto their equilibria and dt/tau times the
    distance left over has a finite limit, approached as tau/dt: at 1e-30 and
    at 1e-160 the same numbers to rounding (a dozen steps' bound)."""
    a, b = _run([W.couette(nx=40, ny=24, seed=1, tau=tau, rkmethod=rk) for tau in (1e-30, 1e-160)])
    for q in ("rho", "ux", "uy", "T"):
        assert np.all(np.isfinite(b[q])) and np.max(np.abs(a[q] - b[q])) < 1e-11, q


@pytest.mark.parametrize("rk", [0, 1])
def test_large_densities(cuda_device, rk):
    """Density and viscosity times 2^36 and 2^80: WENO5's epsilon (1e-6)
    against squared differences of 1e-4 x 6e10 and more is below 1e-18, so
    the two are the same flow to rounding.  (Its mass check is absolute and
    fails for both.)"""
    def at(scale):
        c = W.couette(nx=40, ny=24, seed=2, tau=0.05, rkmethod=rk, noise=1e-2)
        c["density"] = np.asarray(c["density"]) * scale
        c["mu"] *= scale
        return c

    a, b = _run([at(2.0 ** 36), at(2.0 ** 80)])
    for q, s in (("rho", 2.0 ** 44), ("ux", 1.0), ("uy", 1.0), ("T", 1.0)):
        assert np.all(np.isfinite(b[q])) and np.max(np.abs(b[q] / s - a[q])) < 1e-11 * max(1.0, np.max(np.abs(a[q]))), q
