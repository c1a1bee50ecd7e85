"""Performance cases of the transport-sweep library: what its users have it do, through its public entry points
(``idcsweep.abi``, the ctypes mirror of the C ABI).

Every case is one of these kinds; a case's plain values say which and how large.

* ``sweep``      one out-of-place sweep source -> psi with its moments phi (``idc_sweep_out``): the operator that every
                 solver and time integrator of the reference calls (``SweepOperator::Apply`` with ``Pmv``).
* ``host``       several sweeps of host-resident arrays (``idc_sweep_out_many`` on pinned host memory): what the
                 reference's own C++ objects hand to the library.
* ``si``         source iteration to 1e-10 (``idc_source_iteration``): the reference's SISolver.
* ``gmres``      Peierls-form GMRES(30) with DSA (``idc_gmres_solve``): steady problems with strong scattering.
* ``batch``      the same solves for several uneven problems at once (``idc_batch_gmres_solve``).
* ``idc``        IDC time steps from a given state (``idc_idc_integrate``): scattering explicit (one sweep per substep) or
                 implicit (one GMRES solve per substep).
* ``adjoint``    gradients of a detector response (``idc_adjoint_grad``): the transposed sweep inside GMRES.

Cross sections are log-normal per cell (the heterogeneous media of the benchmark) or the 7 x 7 absorber lattice with
block values that vary with the seed; sources are isotropic, positive and cell-wise random, angular where a time step
hands one over; ghost cells carry inflow where a case says so.  All sizes come from the benchmark's configurations, from
the tests, or lie between them.
"""
import math
import os
import sys

import numpy as np
import torch

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "idc-transport-solver_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)
from idcsweep import abi  # noqa: E402
from idcsweep.quadrature import level_symmetric_2d  # noqa: E402

DEVICE = "cuda:0"
LENGTH = 7.0   # every domain is LENGTH wide in x; cells are square


def listed():
    return [
        # one sweep of the reference's own case (64 x 64 lattice, Q1, S8, an implicit-Euler step): the smallest call, all
        # launch latency and wavefront fill
        dict(name="sweep 64 Q1 S8", kind="sweep", nx=64, ny=64, p=1, sn=8, dt=0.01, medium="lattice", inflow=False,
             precision="fp64"),
        # the benchmark's headline: one steady sweep of the heterogeneous medium
        dict(name="sweep 256 Q2 S16", kind="sweep", nx=256, ny=256, p=2, sn=16, dt=0.0, medium="lognormal",
             inflow=False, precision="fp64"),
        # sides that no tile divides, 15 ordinates in a quadrant, an implicit step with inflow: a time step of a ragged grid
        dict(name="sweep 131x197 Q2 S10", kind="sweep", nx=131, ny=197, p=2, sn=10, dt=0.5, medium="lognormal",
             inflow=True, precision="fp64"),
        # the lowest degree in use after the benchmark's two, many ordinates on a large grid
        dict(name="sweep 300x200 Q0 S16", kind="sweep", nx=300, ny=200, p=0, sn=16, dt=0.0, medium="lognormal",
             inflow=True, precision="fp64"),
        # FP32 cell solves with FP64 refinement, the option that the benchmark reports beside FP64
        dict(name="refined 192x160 Q2 S12", kind="sweep", nx=192, ny=160, p=2, sn=12, dt=0.0, medium="lognormal",
             inflow=False, precision="fp32_refined"),
        # host-resident right-hand sides, as the plugin inside the reference holds them
        dict(name="host 96 Q2 S12 x4", kind="host", nx=96, ny=96, p=2, sn=12, dt=0.25, medium="lognormal", inflow=True,
             count=4),
        # the reference's own solve: one implicit-Euler step of the lattice by source iteration
        dict(name="si 64 Q1 S8", kind="si", nx=64, ny=64, p=1, sn=8, dt=0.01, medium="lattice", inflow=False),
        # the benchmark's steady solve at full size, scattering ratio up to 0.999
        dict(name="gmres 256 Q2 S16", kind="gmres", nx=256, ny=256, p=2, sn=16, dt=0.0, medium="lognormal",
             inflow=False, tol=1e-10, inner=30),
        # a batch of uneven problems solved together (side:degree:S_N of each member)
        dict(name="batch 8 uneven", kind="batch", members="32:1:4,64:2:8,96:1:16,128:2:4,160:1:8,192:2:12,256:1:12,320:1:4",
             tol=1e-8, inner=20),
        # IMEX-IDC time steps of the large lattice: 4 Gauss-Lobatto nodes, 3 corrections
        dict(name="imex 512 Q1 S12", kind="idc", nx=512, ny=512, p=1, sn=12, dt=0.005, medium="lattice", inflow=False,
             steps=2, nodes=4, corrections=3, scattering="explicit"),
        # an implicit-scattering IDC step of the small lattice: a GMRES solve per substep
        dict(name="idc 64 Q1 S8", kind="idc", nx=64, ny=64, p=1, sn=8, dt=0.05, medium="lattice", inflow=False, steps=1,
             nodes=3, corrections=2, scattering="implicit"),
        # gradients of a detector response with respect to every cell's parameters
        dict(name="adjoint 128 Q1 S8", kind="adjoint", nx=128, ny=128, p=1, sn=8, dt=0.0, medium="lognormal",
             inflow=False, tol=1e-12, inner=20),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    p, sn = rng.choice([0, 1, 1, 2, 2]), rng.choice([4, 6, 8, 10, 12, 14, 16])
    kind = rng.choice(["sweep", "sweep", "sweep", "host", "si", "gmres", "batch", "idc", "adjoint"])
    case = dict(kind=kind)
    if kind == "batch":
        members = ["%d:%d:%d" % (side(24, 200), rng.choice([1, 2]), rng.choice([4, 6, 8, 10, 12]))
                   for _ in range(rng.randint(3, 8))]
        case.update(members=",".join(members), tol=1e-8, inner=20)
        return case
    top = {"sweep": 256, "host": 96, "si": 128, "gmres": 200, "idc": 128, "adjoint": 160}[kind]
    case.update(nx=side(24, top), ny=side(24, top), p=p, sn=sn, dt=rng.choice([0.0, 0.05, 0.5]),
                medium=rng.choice(["lognormal", "lattice"]), inflow=rng.choice([False, True]))
    if kind == "sweep":
        case["precision"] = rng.choice(["fp64", "fp64", "fp32_refined"])
    elif kind == "host":
        case["count"] = rng.randint(2, 4)
    elif kind == "si":
        case["dt"] = rng.choice([0.01, 0.05])   # steady problems take GMRES: source iteration is for time steps
    elif kind == "gmres":
        case.update(tol=rng.choice([1e-8, 1e-10]), inner=rng.choice([20, 30]))
    elif kind == "idc":
        implicit = rng.random() < 0.5
        case.update(dt=rng.choice([0.01, 0.05]), steps=1 if implicit else rng.randint(1, 3), nodes=rng.choice([3, 4]),
                    corrections=rng.randint(1, 3), scattering="implicit" if implicit else "explicit")
        if implicit:
            case.update(nx=min(case["nx"], 96), ny=min(case["ny"], 96))
    elif kind == "adjoint":
        case.update(dt=0.0, inflow=False, tol=1e-12, inner=20)
    return case


# ---- inputs ----------------------------------------------------------------------------------------------------

def _members(case):
    if case["kind"] != "batch":
        return [case]
    out = []
    for m in case["members"].split(","):
        n, p, sn = (int(v) for v in m.split(":"))
        out.append(dict(nx=n, ny=n, p=p, sn=sn, dt=0.0, medium="lognormal", inflow=False))
    return out


def _dt(case):
    return case["dt"] if case["dt"] > 0 else math.inf


def _problem(m, gen):
    """Cross sections, source and (for time steps) initial state of one problem, on the GPU, from the generator."""
    nx, ny, P = m["nx"], m["ny"], m["p"] + 1
    xi, eta, w, quad = level_symmetric_2d(m["sn"])
    nq = xi.size

    def rand(*shape):
        return torch.rand(shape, dtype=torch.float64, device=DEVICE, generator=gen)

    sigma_t = torch.zeros(nx + 2, ny + 2, dtype=torch.float64, device=DEVICE)
    sigma_s = torch.zeros_like(sigma_t)
    if m["medium"] == "lognormal":
        g = torch.randn(nx, ny, dtype=torch.float64, device=DEVICE, generator=gen)
        sigma_t[1:-1, 1:-1] = torch.exp(g)
        sigma_s[1:-1, 1:-1] = (0.5 + 0.499 * rand(nx, ny)) * sigma_t[1:-1, 1:-1]
        strength = 0.5 + rand(nx, ny)
    else:   # 7 x 7 blocks: absorbers of about 10, scatterers of about 1, the source in the middle block
        bi = (torch.arange(nx, device=DEVICE) * 7 // nx)[:, None].expand(nx, ny)
        bj = (torch.arange(ny, device=DEVICE) * 7 // ny)[None, :].expand(nx, ny)
        ring = (bi >= 1) & (bi <= 5) & (bj >= 1) & (bj <= 5)
        absorber = ring & ((bi + bj) % 2 == 0) & ~((bi == 3) & (bj == 3))
        block = (0.8 + 0.4 * rand(7, 7))[bi, bj]
        sigma_t[1:-1, 1:-1] = torch.where(absorber, 10.0 * block, block)
        sigma_s[1:-1, 1:-1] = torch.where(absorber, 0.0 * block, block)
        strength = ((bi == 3) & (bj == 3)).double() * (0.5 + rand(nx, ny)) + 1e-3
    source = torch.zeros(nx + 2, ny + 2, nq, P, P, dtype=torch.float64, device=DEVICE)
    moments = 0.1 * (rand(nx, ny, 1, P, P) - 0.5) * strength[:, :, None, None, None]
    moments[:, :, 0, 0, 0] = strength
    source[1:-1, 1:-1] = moments / (4.0 * math.pi)
    if math.isfinite(_dt(m)):   # a time step adds the last state, which depends on the direction
        source[1:-1, 1:-1] += 0.05 * rand(nx, ny, nq, 1, 1)
    if m["inflow"]:
        for edge in (source[0, 1:-1], source[-1, 1:-1], source[1:-1, 0], source[1:-1, -1]):
            edge[:, :, 0, 0] = 0.1 * rand(edge.shape[0], nq)
    return dict(nx=nx, ny=ny, P=P, nq=nq, xi=xi, eta=eta, w=w, quad=quad, dt=_dt(m), sigma_t=sigma_t, sigma_s=sigma_s,
                source=source, width=LENGTH, height=LENGTH * ny / nx)


def _inputs(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    problems = [_problem(m, gen) for m in _members(case)]
    pr = problems[0]
    extra = {}
    if case["kind"] == "host":
        f = 0.5 + torch.rand(case["count"], pr["nq"], 1, 1, dtype=torch.float64, device=DEVICE, generator=gen)
        extra["sources"] = [(pr["source"] * f[k]).contiguous() for k in range(case["count"])]
    if case["kind"] == "idc":
        psi0 = torch.zeros_like(pr["source"])
        psi0[1:-1, 1:-1, :, 0, 0] = 0.02 * torch.rand(pr["nx"], pr["ny"], 1, dtype=torch.float64, device=DEVICE,
                                                     generator=gen)
        if case["inflow"]:
            for s in ((0, slice(1, -1)), (-1, slice(1, -1)), (slice(1, -1), 0), (slice(1, -1), -1)):
                psi0[s] = pr["source"][s]
        extra["psi0"] = psi0
    if case["kind"] == "adjoint":   # the cell integrals over a window at the right third
        c = torch.zeros(pr["nx"] + 2, pr["ny"] + 2, pr["P"], pr["P"], dtype=torch.float64, device=DEVICE)
        m = min(16, pr["nx"], pr["ny"])
        i0, j0 = 2 * (pr["nx"] - m) // 3, (pr["ny"] - m) // 2
        c[1 + i0:1 + i0 + m, 1 + j0:1 + j0 + m, 0, 0] = (pr["width"] / pr["nx"]) * (pr["height"] / pr["ny"])
        extra["detector"] = c
    return problems, extra


def _context(pr):
    ctx = abi.SweepContext(pr["nx"], pr["ny"], pr["P"] - 1, 0.0, pr["width"], 0.0, pr["height"])
    ctx.set_ordinates(pr["xi"], pr["eta"], pr["w"], pr["quad"])
    ctx.set_sigma(pr["sigma_t"].data_ptr(), pr["sigma_s"].data_ptr(), loc=abi.LOC_DEVICE)
    return ctx


def _phi(pr):
    return torch.zeros(pr["nx"] + 2, pr["ny"] + 2, pr["P"], pr["P"], dtype=torch.float64, device=DEVICE)


def prepare(case, seed):
    problems, extra = _inputs(case, seed)
    torch.cuda.synchronize()
    ctxs = [_context(pr) for pr in problems]
    pr, ctx = problems[0], ctxs[0]
    s = dict(case=case, ctxs=ctxs, problems=problems, **extra)
    kind = case["kind"]
    if kind in ("gmres", "batch", "adjoint", "idc") and case.get("scattering") != "explicit":
        for c in ctxs:
            c.set_preconditioner(abi.PRECOND_DSA, case.get("inner", 20))
    if kind == "host":
        s["sources"] = [x.cpu().pin_memory() for x in extra["sources"]]
        s["psi"] = [torch.zeros_like(x).pin_memory() for x in s["sources"]]
        s["phi"] = [_phi(pr).cpu().pin_memory() for _ in s["sources"]]
        del pr["source"]
        return s
    s["psi"] = [torch.zeros_like(q["source"]) for q in problems]
    s["phi"] = [_phi(q) for q in problems]
    if kind == "batch":
        s["batch"] = abi.Batch()
        for c in ctxs:
            s["batch"].add(c)
    if kind == "adjoint":   # the forward solution that the gradients are taken at
        s["psi"][0].copy_(pr["source"])
        torch.cuda.synchronize()
        ctx.gmres_solve(s["psi"][0].data_ptr(), pr["dt"], abs_tol=1e-13, loc=abi.LOC_DEVICE)
        s["dsigma_t"], s["dsigma_s"] = torch.zeros_like(pr["sigma_t"]), torch.zeros_like(pr["sigma_t"])
    torch.cuda.synchronize()
    return s


def run(state):
    case, pr, ctx = state["case"], state["problems"][0], state["ctxs"][0]
    kind, psi, phi = case["kind"], state["psi"], state["phi"]
    if kind == "sweep":
        prec = abi.PREC_FP32_REFINED if case["precision"] == "fp32_refined" else abi.PREC_FP64
        ctx.sweep_out(pr["source"].data_ptr(), psi[0].data_ptr(), pr["dt"], phi[0].data_ptr(), prec, loc=abi.LOC_DEVICE)
        return {"psi": psi[0], "phi": phi[0]}
    if kind == "host":
        ctx.sweep_out_many([x.numpy() for x in state["sources"]], [x.numpy() for x in psi], [x.numpy() for x in phi],
                           pr["dt"], abi.PREC_FP64)
        return {"psi": psi, "phi": phi}
    if kind == "adjoint":
        ctx.adjoint_grad(psi[0].data_ptr(), state["detector"].data_ptr(), state["dsigma_t"].data_ptr(),
                         state["dsigma_s"].data_ptr(), phi[0].data_ptr(), pr["dt"], abs_tol=case["tol"],
                         loc=abi.LOC_DEVICE)
        return {"dsigma_t": state["dsigma_t"], "dsigma_s": state["dsigma_s"], "dsource": phi[0]}
    # the solvers work in place: the source (or the state) goes into psi first; the library runs on its own stream
    for x, q in zip(psi, state["problems"]):
        x.copy_(state["psi0"] if kind == "idc" else q["source"])
    torch.cuda.current_stream().synchronize()
    if kind == "si":
        ctx.source_iteration(psi[0].data_ptr(), pr["dt"], abs_tol=1e-10, max_its=5000, loc=abi.LOC_DEVICE)
    elif kind == "gmres":
        ctx.gmres_solve(psi[0].data_ptr(), pr["dt"], abs_tol=case["tol"], loc=abi.LOC_DEVICE)
    elif kind == "batch":
        state["batch"].gmres_solve([x.data_ptr() for x in psi], abs_tol=case["tol"])
    elif kind == "idc":
        how = abi.SCATTER_EXPLICIT if case["scattering"] == "explicit" else abi.SCATTER_IMPLICIT
        ctx.idc_integrate(psi[0].data_ptr(), pr["source"].data_ptr(), pr["dt"], case["steps"], case["nodes"],
                          case["corrections"], how, abs_tol=1e-12, loc=abi.LOC_DEVICE)
    return {"psi": psi}


# ---- what a pass cannot do without --------------------------------------------------------------------------------

def work(case):
    """Bytes: every input array read once and every output array written once (interior cells).  Operations: the
    arithmetic of the sweeps that the pass makes: 4 P^3 multiply-adds for the two transforms of a cell's source and
    solution in the eigenbasis of the one-dimensional operator, and about 4 per unknown for the solve; a solver is
    counted with the sweeps of a right-hand side, one iteration and the final psi."""
    nbytes = flops = 0
    for m in _members(case):
        cells, P = m["nx"] * m["ny"], m["p"] + 1
        N, nq = P * P, level_symmetric_2d(m["sn"])[0].size
        psi, one = 8 * cells * nq * N, 2 * cells * nq * (4 * P ** 3 + 4 * N)
        kind = case["kind"]
        if kind == "sweep":
            nbytes += 2 * psi + 8 * cells * (1 + N)
            flops += one
        elif kind == "host":
            nbytes += case["count"] * (2 * psi + 8 * cells * N) + 8 * cells
            flops += case["count"] * one
        elif kind == "idc":
            nbytes += 3 * psi + 16 * cells
            flops += one * case["steps"] * (case["nodes"] - 1) * (case["corrections"] + 1)
        elif kind == "adjoint":
            nbytes += psi + 8 * cells * (4 + 2 * N)
            flops += 2 * one
        else:
            nbytes += 2 * psi + 16 * cells
            flops += 3 * one
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind in ("sweep", "host"):
        # from the plain 64-bit solve: FP64 up to 1.7e-14, refined FP32 cell solves up to 2.3e-12
        return {"rel": 1e-11 if case.get("precision") == "fp32_refined" else 7e-14}
    if kind == "idc" and case["scattering"] == "explicit":
        return {"rel": 1e-12}   # sweeps and quadrature sums only: no iteration's stopping rule
    # solves that stop at an absolute residual: two solutions differ by about that residual times the inverse's norm
    return {"rel": 1e-9}


# ---- the same in plain 64-bit torch --------------------------------------------------------------------------------

class _Plain:
    """Sweeps, moments and operators of one problem, cell by cell in wavefront order with dense solves."""

    def __init__(self, pr):
        self.pr = pr
        nx, ny, P, nq = pr["nx"], pr["ny"], pr["P"], pr["nq"]
        self.N = P * P
        t = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=DEVICE)
        self.w = t(pr["w"])
        ax, ay = t(np.abs(pr["xi"])) * nx / pr["width"], t(np.abs(pr["eta"])) * ny / pr["height"]
        d = np.arange(P)
        M = (2 * d[:, None] + 1) * np.where((d[None, :] < d[:, None]) & ((d[:, None] - d[None, :]) % 2 == 1), -1, 1)
        u, M, eye = t((-1.0) ** d * (2 * d + 1)), t(M), torch.eye(P, dtype=torch.float64, device=DEVICE)
        # cell matrices without the sigma term, and the couplings of the x and y upwind neighbours
        self.A = ax[:, None, None] * torch.kron(M, eye) + ay[:, None, None] * torch.kron(eye, M)
        up = torch.outer(u, torch.ones_like(u))
        self.Cx, self.Cy = ax[:, None, None] * torch.kron(up, eye), ay[:, None, None] * torch.kron(eye, up)
        self.eye = torch.eye(self.N, dtype=torch.float64, device=DEVICE)
        xn, yn = t(np.asarray(pr["xi"]) < 0).bool(), t(np.asarray(pr["eta"]) < 0).bool()
        sd = t((-1.0) ** d)
        one = torch.ones_like(sd)
        self.sign = (torch.where(xn[:, None, None], sd, one)[:, 0, :, None]
                     * torch.where(yn[:, None, None], sd, one)[:, 0, None, :])          # [q][d][e]
        quad = [int(v) for v in pr["quad"]]
        self.quads = [(slice(quad[k], quad[k + 1]), [dim for dim, neg in ((0, k >= 2), (1, k & 1)) if neg])
                      for k in range(4) if quad[k + 1] > quad[k]]
        self.inverse = {}

    def flip(self, a):
        """Every quadrant mirrored to xi, eta > 0 (its own inverse): [i][j][q][d][e] arrays."""
        out = torch.empty_like(a)
        for q, dims in self.quads:
            out[:, :, q] = torch.flip(a[:, :, q], dims) if dims else a[:, :, q]
        return out * self.sign

    def sigma(self, inv_dt):
        s = (self.pr["sigma_t"] + inv_dt)[:, :, None, None, None].expand(-1, -1, self.pr["nq"], 1, 1)
        out = torch.empty(s.shape, dtype=torch.float64, device=DEVICE)
        for q, dims in self.quads:
            out[:, :, q] = torch.flip(s[:, :, q], dims) if dims else s[:, :, q]
        return out

    def sweep(self, source, dt, transposed=False):
        """psi with (Omega.grad + sigma_t + 1/dt) psi = source on interior cells, inflow from source's ghost cells; or
        the transpose's solution with zero inflow.  The result keeps source's ghost cells."""
        nx, ny, N, nq = self.pr["nx"], self.pr["ny"], self.N, self.pr["nq"]
        x = self.flip(source).reshape(nx + 2, ny + 2, nq, N, 1)
        s = self.sigma(1.0 / dt)
        A, Cx, Cy = self.A, self.Cx, self.Cy
        step = 1
        if transposed:
            A, Cx, Cy, step = A.mT, Cx.mT, Cy.mT, -1
            x = x.clone()
            x[0], x[-1], x[:, 0], x[:, -1] = 0.0, 0.0, 0.0, 0.0
        keep = self.inverse.setdefault((dt, transposed), {}) if nx * ny * nq * N * N < 1.5e8 else None
        for t in range(nx + ny - 1):
            dg = t if step == 1 else nx + ny - 2 - t
            i = torch.arange(max(0, dg - ny + 1), min(nx, dg + 1), device=DEVICE) + 1
            j = dg + 2 - i
            b = x[i, j] + Cx @ x[i - step, j] + Cy @ x[i, j - step]
            if keep is None:
                x[i, j] = torch.linalg.solve(A + s[i, j] * self.eye, b)
            else:
                if t not in keep:
                    keep[t] = torch.linalg.inv(A + s[i, j] * self.eye)
                x[i, j] = keep[t] @ b
        out = self.flip(x.reshape(source.shape))
        for e in ((0,), (-1,), (slice(None), 0), (slice(None), -1)):
            out[e] = source[e]
        return out

    def moments(self, psi, weighted=True):
        out = torch.zeros_like(psi[:, :, 0])
        a = psi[1:-1, 1:-1]
        out[1:-1, 1:-1] = torch.einsum("ijqde,q->ijde", a, self.w if weighted else torch.ones_like(self.w))
        return out

    def scatter(self, phi):
        """The isotropic scattering source sigma_s phi / (4 pi), the same for every ordinate."""
        return (self.pr["sigma_s"][:, :, None, None] * phi / (4.0 * math.pi))[:, :, None]

    def with_interior(self, base, add):
        out = base.clone()
        out[1:-1, 1:-1] += add[1:-1, 1:-1]
        return out

    def residual(self, psi):
        """(Omega.grad + sigma_t - S P) psi on interior cells, psi's ghost cells as inflow."""
        nx, ny, N, nq = self.pr["nx"], self.pr["ny"], self.N, self.pr["nq"]
        x, s = self.flip(psi).reshape(nx + 2, ny + 2, nq, N, 1), self.sigma(0.0)
        y = torch.zeros_like(x)
        c = x[1:-1, 1:-1]
        y[1:-1, 1:-1] = (self.A @ c + s[1:-1, 1:-1] * c - self.Cx @ x[:-2, 1:-1] - self.Cy @ x[1:-1, :-2])
        y = self.flip(y.reshape(psi.shape))
        return y - self.scatter(self.moments(psi))

    def krylov(self, op, b, tol):
        """GMRES without restart on op(x) = b, to a relative residual."""
        n0 = float(b.norm())
        V, H = [b.reshape(-1) / n0], np.zeros((400, 400))
        for k in range(120):
            wv = op(V[k].reshape(b.shape)).reshape(-1)
            for _ in range(2):
                B = torch.stack(V)
                h = B @ wv
                wv = wv - h @ B
                H[: k + 1, k] += h.cpu().numpy()
            H[k + 1, k] = float(wv.norm())
            e = np.zeros(k + 2)
            e[0] = n0
            y, *_ = np.linalg.lstsq(H[: k + 2, : k + 1], e, rcond=None)
            r = np.linalg.norm(H[: k + 2, : k + 1] @ y - e)
            if r < tol * n0:
                break
            V.append(wv / H[k + 1, k])
        return (torch.as_tensor(y, device=DEVICE) @ torch.stack(V[: len(y)])).reshape(b.shape)

    def solve(self, source, dt, tol=1e-14):
        """psi with (Omega.grad + sigma_t + 1/dt - S P) psi = source."""
        zero = torch.zeros_like(source)
        b = self.moments(self.sweep(source, dt))
        op = lambda f: f - self.moments(self.sweep(self.with_interior(zero, self.scatter(f)), dt))
        phi = self.krylov(op, b, tol)
        return self.sweep(self.with_interior(source, self.scatter(phi)), dt)

    def adjoint(self, detector, dt, tol=1e-14):
        """lambda with (Omega.grad + sigma_t + 1/dt - S P)^T lambda = P^T detector."""
        zero = torch.zeros_like(self.pr["source"])
        spread = lambda m: self.with_interior(zero, self.w[:, None, None] * m[:, :, None])
        back = lambda m: self.sweep(spread(m), dt, transposed=True)
        ss = self.pr["sigma_s"][:, :, None, None] / (4.0 * math.pi)
        op = lambda m: m - ss * self.moments(back(m), weighted=False)
        return back(self.krylov(op, detector, tol))


def _lobatto(M):
    """Gauss-Lobatto nodes on [0, 1] and W[i, j], the integral of the j-th Lagrange polynomial over [t_{i-1}, t_i]."""
    poly = np.polynomial
    c = np.zeros(M)
    c[-1] = 1.0
    inner = np.sort(poly.legendre.legroots(poly.legendre.legder(c))) if M > 2 else np.array([])
    t = np.concatenate([[0.0], 0.5 * (inner + 1.0), [1.0]])
    W = np.zeros((M, M))
    for j in range(M):
        y = np.zeros(M)
        y[j] = 1.0
        F = poly.polynomial.polyint(np.linalg.solve(np.vander(t, increasing=True), y))
        W[1:, j] = np.diff(poly.polynomial.polyval(t, F))
    return t, W


def _idc(pl, psi, Q, dt, case):
    """Non-hybrid IDC steps in update form; explicit scattering lags it to the previous node and corrects it."""
    M, K, explicit = case["nodes"], case["corrections"], case["scattering"] == "explicit"
    t, W = _lobatto(M)
    for _ in range(case["steps"]):
        st, ph = [psi] + [None] * (M - 1), [pl.moments(psi)] + [None] * (M - 1)

        def advance(n, add, phi_s):
            hdt = (t[n] - t[n - 1]) * dt
            src = pl.with_interior(Q, add + st[n - 1] / hdt)
            st[n] = pl.sweep(pl.with_interior(src, pl.scatter(phi_s)), hdt) if explicit else pl.solve(src, hdt)
            ph[n] = pl.moments(st[n])

        for n in range(1, M):
            advance(n, 0.0, ph[n - 1])
        for _k in range(K):
            res, old = [pl.residual(x) for x in st], list(ph)
            for n in range(1, M):
                add = sum(((1.0 if n == m else 0.0) - W[n, m] / (t[n] - t[n - 1])) * res[m] for m in range(M))
                advance(n, add, ph[n - 1] - old[n - 1] + old[n])
        psi = st[M - 1]
    return psi


def exact(case, seed):
    kind = case["kind"]
    cost = sum(m["nx"] * m["ny"] * level_symmetric_2d(m["sn"])[0].size * (m["p"] + 1) ** 2 for m in _members(case))
    sweeps = {"sweep": 1, "host": 2, "si": 8, "gmres": 30, "batch": 30, "adjoint": 60}.get(kind)
    if kind == "idc":
        sweeps = case["steps"] * (case["nodes"] - 1) * (case["corrections"] + 1)
        sweeps *= 1 if case["scattering"] == "explicit" else 20
    if cost * sweeps > 1.2e9 or sum(m["nx"] + m["ny"] for m in _members(case)) * sweeps > 30000:
        return None
    problems, extra = _inputs(case, seed)
    pr, pl = problems[0], _Plain(problems[0])
    zero_ghosts = lambda a: pl.with_interior(torch.zeros_like(a), a)
    if kind == "sweep":
        psi = pl.sweep(pr["source"], pr["dt"])
        return {"psi": zero_ghosts(psi), "phi": pl.moments(psi)}   # the call writes interior cells only
    if kind == "host":
        psi = [pl.sweep(x, pr["dt"]) for x in extra["sources"]]
        return {"psi": [zero_ghosts(x).cpu() for x in psi], "phi": [pl.moments(x).cpu() for x in psi]}
    if kind == "si":
        phi = torch.zeros_like(_phi(pr))
        for _ in range(200):
            psi = pl.sweep(pl.with_interior(pr["source"], pl.scatter(phi)), pr["dt"])
            last, phi = phi, pl.moments(psi)
            if float((phi - last).norm()) <= 1e-14 * float(phi.norm()):
                break
        return {"psi": [psi]}
    if kind in ("gmres", "batch"):
        return {"psi": [_Plain(q).solve(q["source"], q["dt"]) for q in problems]}
    if kind == "idc":
        return {"psi": [_idc(pl, extra["psi0"], pr["source"], pr["dt"], case)]}
    psi = pl.solve(pr["source"], pr["dt"])
    lam = pl.adjoint(extra["detector"], pr["dt"])
    total, phi = pl.moments(lam, weighted=False), pl.moments(psi)
    inner = lambda a: torch.nn.functional.pad(a[1:-1, 1:-1], (1, 1, 1, 1))
    return {"dsigma_t": -inner((lam * psi).sum(dim=(2, 3, 4))),
            "dsigma_s": inner((total * phi).sum(dim=(2, 3))) / (4.0 * math.pi), "dsource": total / (4.0 * math.pi)}
