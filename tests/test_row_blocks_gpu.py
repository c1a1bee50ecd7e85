"""Edges of the lane kernel's tiles and of the solvers' one-launch kernels, against the CPU restatement.

* Sweeps: row counts around whole thread blocks (3, 4 or 7 warps of 32/seg rows) and one row block, columns around the
  copy and trace rings, quadrants with unequal, odd and zero ordinate counts (row segments that start and end off a
  16-byte boundary), arrays off a 16- and a 32-byte boundary.
* DSA: grids around the cluster shapes (512 cells per block, 1 to 16 blocks, 1 to 8 cells per thread) and beyond the
  largest; the preconditioned solve must converge in fewer iterations to the same flux.
* Batches: the moments-only sweeps of uneven members, one of them converged long before the others.
"""
import numpy as np
import pytest

from conftest import rel_err, to_oracle
from idcsweep import abi
from idcsweep.problems import Problem, random_problem

pytestmark = pytest.mark.gpu
TOL64 = 1e-12   # FP64 sweeps against the restatement (the bar of tests/test_sweep_gpu.py)


def _ctx(P):
    c = abi.SweepContext(P.nx, P.ny, P.p, P.ax, P.bx, P.ay, P.by)
    c.set_ordinates(P.xi, P.eta, P.w, P.quad)
    c.set_sigma(P.sigma_t, P.sigma_s)
    return c


def _uneven(nx, ny, p, counts, seed, dt):
    """Random ordinates, counts[k] in quadrant k, on random_problem's cross sections."""
    base = random_problem(nx, ny, p, 4, seed=seed, dt=dt)
    rng = np.random.default_rng(seed)
    sx, sy = (1, 1, -1, -1), (1, -1, 1, -1)
    xi = np.concatenate([sx[k] * rng.uniform(0.1, 0.9, n) for k, n in enumerate(counts)])
    eta = np.concatenate([sy[k] * rng.uniform(0.1, 0.9, n) for k, n in enumerate(counts)])
    w = rng.uniform(0.5, 1.5, xi.size) * 4 * np.pi / xi.size
    src = rng.uniform(-0.5, 1.0, (nx + 2, ny + 2, xi.size, p + 1, p + 1))
    quad = np.concatenate([[0], np.cumsum(counts)])
    return Problem(nx, ny, p, xi, eta, w, quad, base.sigma_t, base.sigma_s, src, base.ax, base.bx, base.ay, base.by, dt)


def _device(a, offset):
    """`a` on the GPU, its data `offset` doubles past an aligned allocation."""
    import torch
    buf = torch.zeros(a.size + offset, dtype=torch.float64, device="cuda")
    view = buf[offset:]
    view.copy_(torch.from_numpy(np.ascontiguousarray(a)).ravel())
    return view


@pytest.mark.parametrize("p", [0, 1, 2])
@pytest.mark.parametrize("seg", [4, 8, 16])
@pytest.mark.parametrize("nx,ny,counts,offset", [(9, 7 * 8 + 1, (3, 3, 3, 3), 0), (1, 29, (5, 1, 0, 7), 1),
                                                 (17, 3 * 2 - 1, (16, 17, 1, 2), 2), (8, 97, (7, 9, 11, 4), 3)])
def test_tile_edges(restatement, p, seg, nx, ny, counts, offset):
    import torch
    P = _uneven(nx, ny, p, counts, seed=nx + ny + p, dt=0.3)
    ref = restatement.sweep(to_oracle(P), P.source, P.dt).reshape(P.psi_shape())
    ref_phi = restatement.pmv(to_oracle(P), ref).reshape(P.phi_shape())
    with _ctx(P) as c:
        c.set_tile_shape(seg, 0)
        src, out = _device(P.source, offset), _device(np.full(P.source.shape, 7.0), offset)
        phi = torch.zeros(P.phi_shape(), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        c.sweep_out(src.data_ptr(), out.data_ptr(), P.dt, phi.data_ptr(), loc=abi.LOC_DEVICE)
        got = out.cpu().numpy().reshape(P.psi_shape())
        assert rel_err(got[1:-1, 1:-1], ref[1:-1, 1:-1]) < TOL64
        assert rel_err(phi.cpu().numpy(), ref_phi) < TOL64
        got[1:-1, 1:-1] = 7.0
        assert np.all(got == 7.0)   # no store outside the interior cells
        c.sweep(src.data_ptr(), P.dt, phi.data_ptr(), loc=abi.LOC_DEVICE)   # in place
        assert rel_err(src.cpu().numpy().reshape(P.psi_shape())[1:-1, 1:-1], ref[1:-1, 1:-1]) < TOL64


@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 513), (64, 16), (91, 90), (92, 90), (129, 127), (182, 181), (256, 256),
                                   (257, 256)])
def test_dsa_cluster_shapes(nx, ny):
    P = random_problem(nx, ny, 0, 4, seed=nx * 7 + ny, inflow=False, sigma_range=(0.5, 5.0))
    P.sigma_s[:] = 0.98 * P.sigma_t
    runs = {}
    with _ctx(P) as c:
        for kind in (abi.PRECOND_NONE, abi.PRECOND_DSA):
            c.set_preconditioner(kind, 40)
            psi = P.source.copy()
            its, _ = c.gmres_solve(psi, P.dt, abs_tol=1e-10, restart=60, max_its=2000)
            runs[kind] = (its, psi)
    if min(nx, ny) >= 16:   # (a strip a cell wide leaks too much for diffusion to describe it)
        assert runs[abi.PRECOND_DSA][0] < runs[abi.PRECOND_NONE][0]
    # two solves to one residual: the difference is the residual times the inverse's norm (c = 0.98: about 1 / (1 - c))
    assert rel_err(runs[abi.PRECOND_DSA][1], runs[abi.PRECOND_NONE][1]) < 1e-8


def test_batched_moments_only_sweeps_of_uneven_members():
    import torch
    probs = [random_problem(5, 3, 1, 4, seed=1, inflow=False, sigma_range=(0.1, 0.2)),   # converges at once
             random_problem(40, 61, 2, 6, seed=2, inflow=False, sigma_range=(0.5, 5.0)),
             random_problem(33, 24, 2, 8, seed=3, inflow=False, sigma_range=(0.5, 5.0)),
             random_problem(70, 20, 1, 10, seed=4, inflow=False, sigma_range=(0.5, 5.0))]
    ctxs, alone, work = [], [], []
    for P in probs:
        P.sigma_s[:] = 0.95 * P.sigma_t
        c = _ctx(P)
        c.set_preconditioner(abi.PRECOND_DSA, 20)
        x = P.source.copy()
        its, _ = c.gmres_solve(x, P.dt, abs_tol=1e-9, restart=5, max_its=500)
        ctxs.append(c)
        alone.append((its, x))
        work.append(torch.from_numpy(P.source).cuda())
    torch.cuda.synchronize()
    with abi.Batch() as b:
        for c in ctxs:
            b.add(c)
        its, res = b.gmres_solve([x.data_ptr() for x in work], abs_tol=1e-9, restart=5, max_its=500)
    for k, (n, x) in enumerate(alone):
        assert abs(its[k] - n) <= 1 and res[k] <= 1e-9
        assert rel_err(work[k].cpu().numpy(), x) < 1e-8
    for c in ctxs:
        c.close()
