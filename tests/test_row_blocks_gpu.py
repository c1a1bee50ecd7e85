"""Edges of the lane kernel's tiles and of the solvers' one-launch kernels, against the CPU restatement.

* Sweeps: few chains (thread blocks of 3 warps of 32/seg rows), rows around one row block, columns around the copy and
  trace rings, quadrants with unequal, odd and zero ordinate counts (row segments that start and end off a 16-byte
  boundary), arrays off a 16- and a 32-byte boundary.
* Sweeps of every instance (plain, FP32, transposed, moments-only, two sources) with as many chains as take thread blocks
  of 4 and of 7 warps, rows around whole blocks, and more items than blocks in flight, so that blocks take several.
* DSA: grids around the cluster shapes (512 cells per block, 1 to 16 blocks, 1 to 8 cells per thread) and beyond the
  largest; the preconditioned solve must converge in fewer iterations to the same flux (a single application is compared
  in test_solver_kernels_gpu.py).
* Batches: the moments-only sweeps of uneven members, one of them converged long before the others.
"""
import numpy as np
import pytest

from conftest import rel_err, to_oracle
from idc_ref import idc_steps
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


def _warps(p, seg, counts, ny):
    """The rule for the warps of a thread block (3, 4 or 7), and the launch's items."""
    widest = -(-max(counts) // -(-max(counts) // seg))
    chains = sum(-(-n // widest) for n in counts)
    items = {w: chains * -(-ny // (w * 32 // seg)) for w in (3, 4, 7)}
    w = 3 if items[3] <= 148 else 4 if items[4] <= (148 * 4 // 3 if p == 2 else 148) else 7
    return w, items[w]


# segment width, columns, rows, ordinates per quadrant: 128 = 4 blocks of 4 warps, 280 = 5 of 7; two chunks and more
SHAPES = [(4, 17, 127, (36, 35, 33, 34)), (4, 15, 128, (36, 35, 33, 34)), (4, 16, 129, (36, 35, 33, 34)),
          (4, 16, 279, (36, 35, 33, 34)), (4, 7, 280, (36, 35, 33, 34)), (4, 17, 281, (36, 35, 33, 34)),
          (16, 16, 183, (33, 31, 32, 17)), (8, 15, 533, (9, 7, 8, 10))]


def test_shapes_reach_what_they_claim():
    got = {(p, *_warps(p, seg, counts, ny)) for p in (0, 1, 2) for seg, nx, ny, counts in SHAPES}
    for p in (0, 1, 2):
        assert any(q == p and w == 4 for q, w, n in got)
        assert any(q == p and w == 7 and n > 148 for q, w, n in got)


@pytest.mark.parametrize("p", [0, 1, 2])
@pytest.mark.parametrize("seg,nx,ny,counts", SHAPES)
def test_larger_thread_blocks(restatement, p, seg, nx, ny, counts):
    import torch
    P = _uneven(nx, ny, p, counts, seed=nx + ny + p, dt=0.3)
    O = to_oracle(P)
    core = np.s_[1:-1, 1:-1]
    with _ctx(P) as c:
        c.set_tile_shape(seg, 0)
        src, out = _device(P.source, 1), _device(np.zeros(P.source.shape), 3)
        phi = torch.zeros(P.phi_shape(), dtype=torch.float64, device="cuda")

        def psi():
            return out.cpu().numpy().reshape(P.psi_shape())[core]

        ref = restatement.sweep(O, P.source, P.dt).reshape(P.psi_shape())
        ref_phi = restatement.pmv(O, ref).reshape(P.phi_shape())
        # FP32: 2^-24 times the operations along the longest path, about 10 a cell
        for prec, tol in ((abi.PREC_FP64, TOL64), (abi.PREC_FP32, 2.0 ** -24 * 10 * (nx + ny))):
            c.sweep_out(src.data_ptr(), out.data_ptr(), P.dt, phi.data_ptr(), prec, abi.LOC_DEVICE)
            assert rel_err(psi(), ref[core]) < tol, prec
            assert rel_err(phi.cpu().numpy(), ref_phi) < tol, prec

        ref = restatement.sweep_adjoint(O, P.source, P.dt).reshape(P.psi_shape())
        c.sweep_adjoint(src.data_ptr(), out.data_ptr(), P.dt, phi.data_ptr(), loc=abi.LOC_DEVICE)
        assert rel_err(psi(), ref[core]) < TOL64
        assert rel_err(phi.cpu().numpy()[core], ref[core].sum(axis=2)) < TOL64

        x = np.random.default_rng(ny).uniform(-0.5, 1.0, P.phi_shape())
        scattered = np.zeros(P.psi_shape())
        scattered[core] = restatement.smv(O, x, np.zeros(P.psi_shape())).reshape(P.psi_shape())[core]
        ref_phi = restatement.pmv(O, restatement.sweep(O, scattered, P.dt)).reshape(P.phi_shape())
        dx = torch.from_numpy(x).cuda()
        c.sweep_fused(None, None, P.dt, dx.data_ptr(), 1.0, phi.data_ptr())
        assert rel_err(phi.cpu().numpy(), ref_phi) < TOL64


@pytest.mark.parametrize("p,seg,nx,ny,counts", [(0, 4, 16, 129, (36, 35, 33, 34)), (1, 8, 15, 533, (9, 7, 8, 10)),
                                                (1, 4, 17, 127, (36, 35, 33, 34)), (2, 16, 6, 183, (33, 31, 32, 17))])
def test_larger_thread_blocks_two_sources(restatement, p, seg, nx, ny, counts):
    """One explicit IDC step, whose correction sweeps have two sources, each with its own row segments' alignment."""
    P = _uneven(nx, ny, p, counts, seed=nx + ny + p, dt=0.05)
    P.source[0], P.source[-1], P.source[:, 0], P.source[:, -1] = 0.0, 0.0, 0.0, 0.0
    psi = np.zeros(P.psi_shape())
    want = idc_steps(restatement, to_oracle(P), psi, P.source, P.dt, 1, M=3, K=1, scattering="explicit")
    with _ctx(P) as c:
        c.set_tile_shape(seg, 0)
        c.idc_integrate(psi, P.source, P.dt, 1, 3, 1, abi.SCATTER_EXPLICIT, use_graph=False)
    assert rel_err(psi[1:-1, 1:-1], want[1:-1, 1:-1]) < TOL64


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
