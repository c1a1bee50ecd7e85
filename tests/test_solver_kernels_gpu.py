"""The solvers' one-launch kernels by themselves, against plain float64 arithmetic: a DSA application (the thread-block
cluster up to 65536 cells, the cooperative kernel beyond) and one CGS2 orthogonalisation, at the edges of their shapes and
of their job lists, and with waits that give up.
"""
import ctypes as C

import numpy as np
import pytest

from idcsweep import abi

pytestmark = pytest.mark.gpu
DEV_OK, DEV_TIMEOUT = 0, 1   # the device error word


class GridDims(C.Structure):
    _fields_ = [("nx", C.c_int), ("ny", C.c_int), ("nq", C.c_int), ("P", C.c_int), ("dx", C.c_double), ("dy", C.c_double)]


class DsaJob(C.Structure):
    _fields_ = [("g", GridDims), ("sigma_s", C.c_void_p), ("v", C.c_void_p), ("out", C.c_void_p), ("ws", C.c_void_p),
                ("error", C.c_void_p), ("spin_limit", C.c_longlong)]


class Cgs2Job(C.Structure):
    _fields_ = [("V", C.c_void_p), ("w", C.c_void_p), ("n", C.c_size_t), ("nv", C.c_int), ("part", C.c_void_p),
                ("coef", C.c_void_p), ("host", C.c_void_p), ("count", C.c_void_p), ("error", C.c_void_p),
                ("spin_limit", C.c_longlong)]


@pytest.fixture(scope="module")
def lib():
    lib = abi.load_library()
    names = dict(dsa_workspace="_ZN3idc21dsa_workspace_doublesEii",
                 dsa_setup="_ZN3idc9dsa_setupERKNS_8GridDimsEPKdS4_PdP11CUstream_st",
                 dsa_precondition="_ZN3idc16dsa_preconditionEPKNS_6DsaJobEiibiP11CUstream_st",
                 cgs2_scratch="_ZN3idc20cgs2_scratch_doublesEv",
                 launch_cgs2="_ZN3idc11launch_cgs2EPKNS_7Cgs2JobEiiP11CUstream_st")
    fn = {k: getattr(lib, v) for k, v in names.items()}
    fn["dsa_workspace"].restype = fn["cgs2_scratch"].restype = C.c_size_t
    fn["dsa_setup"].argtypes = [C.POINTER(GridDims)] + [C.c_void_p] * 4
    fn["dsa_precondition"].argtypes = [C.POINTER(DsaJob), C.c_int, C.c_int, C.c_bool, C.c_int, C.c_void_p]
    fn["launch_cgs2"].argtypes = [C.POINTER(Cgs2Job), C.c_int, C.c_int, C.c_void_p]
    return fn


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


# ---- DSA ----------------------------------------------------------------------------------------------------------

class Dsa:
    """One grid's preconditioner: inputs and workspace on the GPU, and the same application in numpy."""

    def __init__(self, lib, nx, ny, P, seed, spin_limit=1 << 22):
        import torch
        rng = np.random.default_rng(seed)
        self.nx, self.ny, self.N = nx, ny, P * P
        self.st = rng.uniform(0.5, 5.0, (nx + 2, ny + 2))
        self.ss = self.st * rng.uniform(0.8, 0.99, self.st.shape)
        self.v = rng.standard_normal((nx + 2, ny + 2, self.N))
        self.g = GridDims(nx, ny, 4, P, 0.07, 0.11)
        self.dev = [torch.from_numpy(a).cuda() for a in (self.st, self.ss, self.v)]
        self.out = torch.full_like(self.dev[2], np.nan)
        self.ws = torch.zeros(lib["dsa_workspace"](nx, ny), dtype=torch.float64, device="cuda")
        self.error = torch.zeros(1, dtype=torch.int32, device="cuda")
        self.lib = lib
        self.setup()
        self.spin_limit = spin_limit

    def setup(self):
        import torch
        torch.cuda.synchronize()
        assert self.lib["dsa_setup"](C.byref(self.g), self.dev[0].data_ptr(), self.dev[1].data_ptr(), self.ws.data_ptr(), None) == 0

    def job(self):
        return DsaJob(self.g, self.dev[1].data_ptr(), self.dev[2].data_ptr(), self.out.data_ptr(), self.ws.data_ptr(),
                      self.error.data_ptr(), self.spin_limit)

    def want(self, steps, transpose):
        dx, dy, core = self.g.dx, self.g.dy, (slice(1, -1), slice(1, -1))
        st, ss = self.st[core], self.ss[core]
        D, sa = 1 / (3 * st), st - ss
        fx = 2 * D[:-1] * D[1:] / (D[:-1] + D[1:]) / dx ** 2
        fy = 2 * D[:, :-1] * D[:, 1:] / (D[:, :-1] + D[:, 1:]) / dy ** 2
        ex, ey = D / (2 * D + dx / 4) / dx, D / (2 * D + dy / 4) / dy   # Marshak edges
        diag = sa.copy()
        diag[:-1] += fx
        diag[1:] += fx
        diag[:, :-1] += fy
        diag[:, 1:] += fy
        for edge, coef in ((np.s_[0], ex), (np.s_[-1], ex), (np.s_[:, 0], ey), (np.s_[:, -1], ey)):
            diag[edge] += coef[edge]

        def apply(u):
            y = diag * u
            y[:-1] -= fx * u[1:]
            y[1:] -= fx * u[:-1]
            y[:, :-1] -= fy * u[:, 1:]
            y[:, 1:] -= fy * u[:, :-1]
            return y

        r = self.v[core][..., 0] * (1.0 if transpose else ss)
        x, p, rz = np.zeros_like(r), np.zeros_like(r), 0.0
        for _ in range(steps):   # Jacobi-preconditioned conjugate gradients
            z = r / diag
            new = np.sum(r * z)
            p = z + (new / rz if rz else 0.0) * p
            rz = new
            q = apply(p)
            a = rz / np.sum(p * q) if rz else 0.0
            x += a * p
            r = r - a * q
        out = self.v.copy()
        out[core][..., 0] += x * (ss if transpose else 1.0)
        return out


def _apply(lib, dsas, steps, transpose):
    import torch
    torch.cuda.synchronize()
    jobs = (DsaJob * len(dsas))(*[d.job() for d in dsas])
    assert lib["dsa_precondition"](jobs, len(dsas), steps, transpose, _sms(), None) == 0
    torch.cuda.synchronize()


def _check(d, steps, transpose):
    # a few CG steps from zero: the two forms of CG differ by rounding, 2^-53 times the sums' length (under 2^17) at worst
    assert d.error.item() == DEV_OK
    got, want = d.out.cpu().numpy(), d.want(steps, transpose)
    assert np.abs(got - want).max() < 1e-11 * np.abs(want).max()
    ghost = np.ones(got.shape[:2], bool)
    ghost[1:-1, 1:-1] = False
    assert np.array_equal(got[ghost], d.v[ghost]) and np.array_equal(got[..., 1:], d.v[..., 1:])


# cells: around one block of 512 threads, two, 16 (8192), two, four and eight cells a thread, the largest cluster, beyond
@pytest.mark.parametrize("nx,ny", [(1, 1), (73, 7), (512, 1), (1, 512), (27, 19), (41, 25), (64, 128), (2731, 3), (127, 129),
                                   (128, 128), (145, 113), (128, 256), (331, 99), (257, 255), (256, 256), (65537, 1),
                                   (260, 256)])
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("steps", [1, 6])
def test_dsa_application(lib, nx, ny, transpose, steps):
    d = Dsa(lib, nx, ny, 1 + (nx + ny) % 3, seed=nx * 11 + ny)
    _apply(lib, [d], steps, transpose)
    _check(d, steps, transpose)


def test_dsa_job_lists(lib):
    """30 grids of one cluster shape (more than one launch holds), others between them, and one beyond the clusters."""
    dsas = [Dsa(lib, 20 + k, 10, 1 + k % 3, seed=k) for k in range(30)]
    dsas[7:7] = [Dsa(lib, 60, 40, 2, seed=101), Dsa(lib, 260, 256, 1, seed=102)]
    dsas.append(Dsa(lib, 150, 100, 3, seed=103))
    _apply(lib, dsas, 5, False)
    for d in dsas:
        _check(d, 5, False)


def test_dsa_grid_barrier_gives_up(lib):
    """Beyond the clusters every block waits at a counter: with a bound of no polls the waits give up and the error word
    says so; after a new set-up the same application is right."""
    d = Dsa(lib, 300, 256, 1, seed=5, spin_limit=0)
    _apply(lib, [d], 50, False)
    assert d.error.item() == DEV_TIMEOUT
    d.error.zero_()
    d.spin_limit = 1 << 22
    d.setup()
    _apply(lib, [d], 4, False)
    _check(d, 4, False)


# ---- CGS2 ---------------------------------------------------------------------------------------------------------

class Cgs2:
    def __init__(self, lib, n, nv, seed, spin_limit=1 << 22):
        import torch
        rng = np.random.default_rng(seed)
        q, _ = np.linalg.qr(rng.standard_normal((max(n, nv), nv))) if nv <= n else (np.zeros((n, nv)), None)
        self.V, self.w0, self.nv, self.n = np.ascontiguousarray(q.T), rng.standard_normal(n), nv, n
        self.dV, self.w = torch.from_numpy(self.V).cuda(), torch.from_numpy(self.w0).cuda()
        self.scratch = torch.zeros(128 + lib["cgs2_scratch"](), dtype=torch.float64, device="cuda")
        self.host = torch.full((129,), -1.0, dtype=torch.float64).pin_memory()
        self.error = torch.zeros(1, dtype=torch.int32, device="cuda")
        self.spin_limit = spin_limit

    def job(self):
        part = self.scratch.data_ptr() + 8 * 128
        return Cgs2Job(self.dV.data_ptr(), self.w.data_ptr(), self.n, self.nv, part, self.scratch.data_ptr(),
                       self.host.data_ptr(), self.scratch.data_ptr() + 8 * (self.scratch.numel() - 1),
                       self.error.data_ptr(), self.spin_limit)

    def check(self):
        V, w = self.V, self.w0.copy()
        c1 = V @ w
        w -= V.T @ c1
        c2 = V @ w
        w -= V.T @ c2
        host, nv = self.host.numpy(), self.nv
        scale = np.linalg.norm(self.w0)
        tol = 1e-13 * scale   # sums of up to 2^17 rounded products of unit vectors and w: 2^-53 times their square root
        assert np.abs(self.w.cpu().numpy() - w).max() < tol
        assert np.abs(host[:nv] + host[64:64 + nv] - (c1 + c2)).max() < tol
        assert abs(host[127] - w @ w) < tol * scale
        assert host[128:].view(np.int32)[0] == DEV_OK
        assert np.abs(V @ self.w.cpu().numpy()).max() < tol   # what the second pass is for


def _orthogonalise(lib, jobs):
    import torch
    torch.cuda.synchronize()
    arr = (Cgs2Job * len(jobs))(*[j.job() for j in jobs])
    assert lib["launch_cgs2"](arr, len(jobs), _sms(), None) == 0
    torch.cuda.synchronize()


# vectors of one element, a block's threads and around, every SM's block and around; 1 to 60 of them, around the 4 of a pass
@pytest.mark.parametrize("n", [61, 511, 512, 513, 512 * 148 - 1, 512 * 148 + 1, 100003])
@pytest.mark.parametrize("nv", [1, 3, 4, 5, 60])
def test_cgs2(lib, n, nv):
    import torch
    j = Cgs2(lib, n, nv, seed=n + nv)
    _orthogonalise(lib, [j])
    j.check()
    j.w.copy_(torch.from_numpy(j.w0))   # the counter is left as it was found: again
    _orthogonalise(lib, [j])
    j.check()


def test_cgs2_one_element(lib):
    j = Cgs2(lib, 1, 1, seed=3)
    _orthogonalise(lib, [j])
    assert abs(j.w.item()) < 1e-15 * abs(j.w0[0]) + 1e-300
    j.check()


def test_cgs2_job_lists(lib):
    """More problems than one launch holds, of uneven lengths and numbers of vectors."""
    jobs = [Cgs2(lib, 70 + 997 * (k % 9) ** 2, 1 + (7 * k) % 60, seed=k) for k in range(40)]
    _orthogonalise(lib, jobs)
    for j in jobs:
        j.check()


def test_cgs2_barrier_gives_up(lib):
    import torch
    j = Cgs2(lib, 512 * 148, 60, seed=8, spin_limit=0)
    _orthogonalise(lib, [j])
    assert j.error.item() == DEV_TIMEOUT
    j.error.zero_()
    j.scratch[-1] = 0.0   # the counter, as the solvers re-arm it
    j.w.copy_(torch.from_numpy(j.w0))
    j.spin_limit = 1 << 22
    _orthogonalise(lib, [j])
    j.check()
