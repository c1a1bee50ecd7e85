"""The FP64 cell solve's reciprocal denominators are correctly rounded, and those of infinite denominators are zero.

At DG degree 0 a cell without inflow has psi = q / (|xi|/dx + |eta|/dy + sigma_t + 1/dt), formed as q times the reciprocal:
a unit source shows the reciprocal itself.
"""
import numpy as np
import pytest

from conftest import rel_err, to_oracle
from idcsweep import abi
from idcsweep.problems import random_problem

pytestmark = pytest.mark.gpu
SHAPES = [(0, 0), (8, 1)]   # the lane kernel and the modal kernel


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("exponent", [-1000, -1, 0, 3, 1000, 1020])
def test_reciprocal_is_correctly_rounded(shape, exponent):
    """One cell, 2048 random denominators between 2^(1 - exponent) and 2^(-exponent - 3): bitwise the IEEE quotient."""
    n = 512
    rng = np.random.default_rng(exponent + 2000)
    sx, sy = np.repeat((1, 1, -1, -1), n), np.repeat((1, -1, 1, -1), n)
    xi, eta = sx * rng.uniform(0.1, 1.0, 4 * n), sy * rng.uniform(0.1, 1.0, 4 * n)
    side = 2.0 ** exponent   # (a power of two: |xi| / dx is exact)
    src = np.zeros((3, 3, 4 * n, 1, 1))
    src[1, 1] = 1.0
    with abi.SweepContext(1, 1, 0, 0.0, side, 0.0, side) as c:
        c.set_ordinates(xi, eta, np.full(4 * n, 1.0), n * np.arange(5))
        c.set_sigma(np.zeros((3, 3)), np.zeros((3, 3)))
        c.set_tile_shape(*shape)
        c.sweep(src, np.inf)
    with np.errstate(under="ignore"):
        want = 1.0 / (np.abs(xi) / side + np.abs(eta) / side)
    assert np.array_equal(src[1, 1, :, 0, 0], want)


@pytest.mark.parametrize("shape", SHAPES)
def test_infinite_denominators(restatement, shape):
    """A black cell (sigma_t infinite) at degree 0 has psi = 0 and passes on vacuum; so does every cell of a time step so
    short that 1/dt overflows."""
    P = random_problem(5, 4, 0, 8, seed=9)
    P.sigma_t.reshape(7, 6)[3, 2] = np.inf
    P.sigma_s.reshape(7, 6)[3, 2] = 0.0
    ref = restatement.sweep(to_oracle(P), P.source, P.dt).reshape(P.psi_shape())
    assert np.all(ref[3, 2] == 0.0) and np.all(np.isfinite(ref))
    with abi.SweepContext(P.nx, P.ny, P.p, P.ax, P.bx, P.ay, P.by) as c:
        c.set_ordinates(P.xi, P.eta, P.w, P.quad)
        c.set_sigma(P.sigma_t, P.sigma_s)
        c.set_tile_shape(*shape)
        psi = P.source.copy()
        c.sweep(psi, P.dt)
        assert np.all(psi[3, 2] == 0.0)
        assert rel_err(psi[1:-1, 1:-1], ref[1:-1, 1:-1]) < 1e-12
        psi = P.source.copy()
        c.sweep(psi, 1e-310)
        assert np.all(psi[1:-1, 1:-1] == 0.0)
