"""Device arrays that the caller is still filling: a call waits for what was queued before it on the default stream."""
import numpy as np
import pytest

from idcsweep import abi
from idcsweep.problems import random_problem

pytestmark = pytest.mark.gpu
DEV = abi.LOC_DEVICE


def _context(P):
    c = abi.SweepContext(P.nx, P.ny, P.p, P.ax, P.bx, P.ay, P.by)
    c.set_ordinates(P.xi, P.eta, P.w, P.quad)
    c.set_sigma(P.sigma_t, P.sigma_s)
    return c


def _batch(call):
    def run(c, P, a):
        with abi.Batch() as b:
            b.add(c)
            call(b, P, a)
    return run


# entry point -> a call on the device arrays a = {psi, src, out: psi-shaped; phi, det, gq: moment-shaped; gt, gs: cell-shaped}
CALLS = {
    "sweep": lambda c, P, a: c.sweep(a["psi"], P.dt, a["phi"], loc=DEV),
    "sweep_out": lambda c, P, a: c.sweep_out(a["src"], a["out"], P.dt, a["phi"], loc=DEV),
    "sweep_out_many": lambda c, P, a: c.sweep_out_many([a["src"], a["psi"]], [a["out"], a["psi"]], None, P.dt, loc=DEV),
    "sweep_fused": lambda c, P, a: c.sweep_fused(a["src"], a["out"], P.dt, a["det"], 1.0, a["phi"]),
    "sweep_adjoint": lambda c, P, a: c.sweep_adjoint(a["src"], a["out"], P.dt, a["phi"], loc=DEV),
    "pmv": lambda c, P, a: c.pmv(2.0, 0.5, a["src"], a["phi"], loc=DEV),
    "smv": lambda c, P, a: c.smv(2.0, 0.5, a["det"], a["psi"], loc=DEV),
    "lmv": lambda c, P, a: c.lmv(2.0, 0.5, a["src"], a["psi"], loc=DEV),
    "lmv_transpose": lambda c, P, a: c.lmv_transpose(2.0, 0.5, a["src"], a["psi"]),
    "source_iteration": lambda c, P, a: c.source_iteration(a["psi"], P.dt, 1e-6, 20, loc=DEV),
    "gmres_solve": lambda c, P, a: c.gmres_solve(a["psi"], P.dt, 1e-8, loc=DEV),
    "idc_integrate": lambda c, P, a: c.idc_integrate(a["psi"], a["src"], 0.01, 1, 3, 1, loc=DEV),
    "idc_integrate implicit": lambda c, P, a: c.idc_integrate(a["psi"], a["src"], 0.01, 1, 3, 1, abi.SCATTER_IMPLICIT,
                                                              abs_tol=1e-10, loc=DEV),
    "adjoint_grad": lambda c, P, a: c.adjoint_grad(a["src"], a["det"], a["gt"], a["gs"], a["gq"], P.dt, 1e-10, loc=DEV),
    "adjoint_transient": lambda c, P, a: c.adjoint_transient(a["psi"], a["src"], a["det"], 0.05, 1, 0, a["gt"], a["gs"],
                                                             a["gq"], a["out"], 1e-10, loc=DEV),
    "adjoint_idc": lambda c, P, a: c.adjoint_idc(a["psi"], a["src"], a["det"], 0.05, 1, 3, 1, 0, a["gt"], a["gs"], a["gq"],
                                                 a["out"], 1e-10, loc=DEV),
    "batch sweep": _batch(lambda b, P, a: b.sweep([a["src"]], [a["out"]], [a["phi"]], P.dt)),
    "batch gmres_solve": _batch(lambda b, P, a: b.gmres_solve([a["psi"]], P.dt, 1e-8)),
}


@pytest.mark.parametrize("name", CALLS)
def test_call_waits_for_the_default_stream(name):
    import torch
    P = random_problem(24, 20, 1, 4, seed=3, dt=0.3, inflow=False, sigma_range=(0.5, 3.0))
    P.sigma_s[:] = 0.5 * P.sigma_t
    rng = np.random.default_rng(1)
    psi, phi, cells = P.psi_shape(), P.phi_shape(), (P.nx + 2, P.ny + 2)
    shapes = dict(psi=psi, src=psi, out=psi, phi=phi, det=phi, gq=phi, gt=cells, gs=cells)
    given = {k: torch.from_numpy(rng.uniform(0.1, 1.0, s)).cuda() for k, s in shapes.items()}
    arrays = {k: torch.zeros_like(t) for k, t in given.items()}
    pointers = {k: t.data_ptr() for k, t in arrays.items()}
    with _context(P) as c:
        def run(busy):
            for t in arrays.values():
                t.zero_()
            torch.cuda.synchronize()
            if busy:
                torch.cuda._sleep(20_000_000)   # about 10 ms of work before the arrays are filled
            for k, t in arrays.items():
                t.copy_(given[k])
            if not busy:
                torch.cuda.synchronize()
            CALLS[name](c, P, pointers)
            return {k: t.clone() for k, t in arrays.items()}

        want = run(False)
        run(False)          # (what the first calls allocate is there: nothing else waits for the GPU)
        got = run(True)
    assert any(not torch.equal(want[k], given[k]) for k in want)
    for k in want:
        assert torch.equal(got[k], want[k]), k


@pytest.mark.parametrize("degree", [0, 1])
def test_set_sigma_waits_for_the_default_stream(degree):
    """Cross sections constant on each cell, and (degree 1) given by their Legendre moments."""
    import torch
    P = random_problem(24, 20, 1, 4, seed=3, dt=0.3)
    if degree:
        slopes = np.random.default_rng(2).uniform(-0.1, 0.1, (P.sigma_t.size, 4))
        slopes[:, 0] = 1.0
        P.sigma_t, P.sigma_s = P.sigma_t.reshape(-1, 1) * slopes, P.sigma_s.reshape(-1, 1) * slopes
    want, got = P.source.copy(), P.source.copy()
    with abi.SweepContext(P.nx, P.ny, P.p, P.ax, P.bx, P.ay, P.by, sigma_degree=degree) as c:
        c.set_ordinates(P.xi, P.eta, P.w, P.quad)
        c.set_sigma(P.sigma_t, P.sigma_s)
        c.sweep(want, P.dt)
        st, ss = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (P.sigma_t, P.sigma_s))
        a, b = torch.ones_like(st), torch.ones_like(ss)
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)
        a.copy_(st)
        b.copy_(ss)
        c.set_sigma(a.data_ptr(), b.data_ptr(), loc=DEV)
        c.sweep(got, P.dt)
    assert np.array_equal(got, want)
