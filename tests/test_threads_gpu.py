"""Contexts of several host threads: one context per thread, every call as if it were alone."""
import threading
import time

import numpy as np
import pytest

from idcsweep import abi
from idcsweep.problems import Problem, random_problem

pytestmark = pytest.mark.gpu


def _uniform(n, seed):
    """2x2 cells of DG degree 2 with n ordinates per quadrant: many short chains of row blocks."""
    base = random_problem(2, 2, 2, 4, seed=seed, dt=0.5)
    rng = np.random.default_rng(seed)
    sx, sy = np.repeat((1, 1, -1, -1), n), np.repeat((1, -1, 1, -1), n)
    xi, eta = sx * rng.uniform(0.1, 0.9, 4 * n), sy * rng.uniform(0.1, 0.9, 4 * n)
    src = rng.uniform(-0.5, 1.0, (4, 4, 4 * n, 3, 3))
    return Problem(2, 2, 2, xi, eta, np.full(4 * n, np.pi / n), n * np.arange(5), base.sigma_t, base.sigma_s, src,
                   base.ax, base.bx, base.ay, base.by, 0.5)


@pytest.mark.parametrize("shapes", [((16, 0), (16, 0)), ((8, 1), (8, 3))])
def test_threads_with_unequal_blocks(shapes):
    """Contexts whose sweeps launch one kernel with different amounts of shared memory (lane kernel: 16 and 960 ordinates
    per quadrant are 4 and 240 chains, so thread blocks of 3 and of 7 warps; modal kernel: 1 and 3 warps), in host threads
    of their own: no call fails or changes its result."""
    import torch
    errors, ctxs = [], []
    start = threading.Barrier(4)

    def run(k, n, shape):
        try:
            P = _uniform(n, seed=k)
            c = abi.SweepContext(P.nx, P.ny, P.p, P.ax, P.bx, P.ay, P.by)
            ctxs.append(c)
            c.set_ordinates(P.xi, P.eta, P.w, P.quad)
            c.set_sigma(P.sigma_t, P.sigma_s)
            c.set_tile_shape(*shape)
            src = torch.from_numpy(P.source).cuda()
            out, first = torch.zeros_like(src), torch.zeros_like(src)
            torch.cuda.synchronize()
            start.wait()
            c.sweep_out(src.data_ptr(), first.data_ptr(), P.dt, None, loc=abi.LOC_DEVICE)
            end = time.monotonic() + 3.0
            while time.monotonic() < end and not errors:
                c.sweep_out(src.data_ptr(), out.data_ptr(), P.dt, None, loc=abi.LOC_DEVICE)
            assert torch.equal(out, first)
        except Exception as e:   # noqa: BLE001 (a thread's exception is reported by the test)
            errors.append(repr(e))
            start.abort()

    threads = [threading.Thread(target=run, args=(k, *((960, shapes[1]) if k % 2 else (16, shapes[0])))) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for c in ctxs:
        c.close()
    assert not errors, errors
