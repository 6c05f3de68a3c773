"""Performance cases of the solver: calls as a user's program makes them.

A case is a plain dict.  `prepare` builds the mesh, the parameter text and the
solver(s) of a case from a seed (the seed draws the flow state, the grid
jitter, the airfoils' shapes and angles), `run` makes one pass through the
public entry points and returns its results, `work` counts the bytes and
operations the pass cannot do without, `exact` is the same result from plain
FP64 tensor code where the result is a defined number.

Kinds of cases:

* explicit  set a state, run time steps, read the state back: Sod shock tube
            (Roe, Barth-Jespersen), double Mach reflection (triangles, FP64
            or FP32 fluxes), Riemann problems (quads), cylinder wake
            (Navier-Stokes, triangles);
* residual  one call of the right-hand side (the drop-in for the reference's
            fvTimeDerivative) with the limited gradients, for programs that
            keep their own time loop;
* implicit  steady airfoil: backward Euler, Newton, GMRES with LU-SGS;
* lusgs     one application of the preconditioner;
* batch     many airfoils, or many explicit cases, advanced together;
* serve     a short request stream through the server.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

import ccfd_b200 as cc
from ccfd_b200 import meshgen, workloads

GAM = 1.4
RK3 = (0.0, 0.1918, 0.4929, 1.0)  # stage coefficients of timeOrder 2, three stages


# ------------------------------------------------------------------- cases
def listed() -> list[dict]:
    return [
        # the small plain configuration: 8,000 cells, where launches and
        # latency count; 64 steps of a transient run between two outputs
        {"name": "sod_8k", "kind": "explicit", "flow": "sod", "nx": 400, "ny": 20, "flux": 2, "limiter": 1,
         "mixed": False, "steps": 64},
        # a host program's own time loop: one right-hand side with gradients
        # on a mid-sized, odd-sized triangle mesh
        {"name": "residual_dmr_63k", "kind": "residual", "flow": "dmr", "nx": 353, "ny": 89, "flux": 5,
         "limiter": 2, "mixed": False},
        # the explicit throughput configuration
        {"name": "dmr_500k", "kind": "explicit", "flow": "dmr", "nx": 1000, "ny": 250, "flux": 5, "limiter": 2,
         "mixed": False, "steps": 16},
        # the same with FP32 reconstruction and fluxes
        {"name": "dmr_500k_mixed", "kind": "explicit", "flow": "dmr", "nx": 1000, "ny": 250, "flux": 5,
         "limiter": 2, "mixed": True, "steps": 16},
        # a large Riemann problem of the served stream (quads)
        {"name": "riemann_1m", "kind": "explicit", "flow": "riemann", "nx": 1024, "ny": 1024, "flux": 5,
         "limiter": 2, "mixed": False, "steps": 16},
        # a cylinder-wake window of the served stream (Navier-Stokes)
        {"name": "cylinder_ns_200k", "kind": "explicit", "flow": "cylinder", "nx": 447, "ny": 223, "flux": 2,
         "limiter": 2, "mixed": False, "steps": 16},
        # the implicit Navier-Stokes configuration's airfoil
        {"name": "airfoil_ns_32k", "kind": "implicit", "ni": 256, "nj": 128, "ns": True, "mixed": False,
         "steps": 2},
        # a single Euler airfoil of the batched distribution in mixed precision
        {"name": "airfoil_mixed_odd", "kind": "implicit", "ni": 301, "nj": 97, "ns": False, "mixed": True,
         "steps": 2},
        # the preconditioner alone, as a program with its own Krylov loop calls it
        {"name": "lusgs_32k", "kind": "lusgs", "ni": 256, "nj": 128, "mixed": False},
        # airfoils of the batched distribution solved together
        {"name": "batch_airfoils_8", "kind": "batch", "flow": "airfoil", "members": 8, "mixed": False, "steps": 2},
        # uneven explicit cases stepped together, 16 steps per call as the
        # serving loop advances its members
        {"name": "batch_explicit_5", "kind": "batch", "flow": "explicit", "members": 5, "mixed": False,
         "steps": 48},
        # a short served stream: requests of all three kinds from submission
        # to the results
        {"name": "serve_6", "kind": "serve", "requests": 6},
    ]


def _log_uniform(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    u = rng.random()
    if u < 0.40:
        flow = rng.choice(["sod", "dmr", "riemann", "cylinder"])
        cells = _log_uniform(rng, 4_000, 1_000_000)
        aspect = {"sod": 20.0, "dmr": 4.0, "riemann": 1.0, "cylinder": 2.0}[flow]
        quads = cells / (2 if flow in ("dmr", "cylinder") else 1)
        ny = max(8, int(math.sqrt(quads / aspect)))
        nx = max(16, int(quads / ny))
        if flow == "riemann":
            nx = ny
        return {"kind": "explicit", "flow": flow, "nx": nx, "ny": ny, "flux": rng.choice([2, 3, 5]),
                "limiter": rng.choice([1, 2]), "mixed": rng.random() < 0.3, "steps": rng.choice([8, 16, 17, 32])
                if cells > 1e5 else rng.choice([16, 33, 64])}
    if u < 0.55:
        cells = _log_uniform(rng, 4_000, 500_000)
        ny = max(8, int(math.sqrt(cells / 2 / 4.0)))
        return {"kind": "residual", "flow": rng.choice(["dmr", "cylinder"]), "nx": max(16, int(cells / 2 / ny)),
                "ny": ny, "flux": rng.choice([2, 3, 5]), "limiter": rng.choice([1, 2]), "mixed": False}
    if u < 0.75:
        return {"kind": "implicit", "ni": rng.randint(128, 400), "nj": rng.randint(64, 160),
                "ns": rng.random() < 0.4, "mixed": rng.random() < 0.4, "steps": rng.choice([1, 2])}
    if u < 0.85:
        return {"kind": "lusgs", "ni": rng.randint(128, 512), "nj": rng.randint(64, 200),
                "mixed": rng.random() < 0.4}
    if u < 0.97:
        if rng.random() < 0.5:
            return {"kind": "batch", "flow": "airfoil", "members": rng.randint(2, 7),
                    "mixed": rng.random() < 0.5, "steps": rng.choice([1, 2])}
        return {"kind": "batch", "flow": "explicit", "members": rng.randint(2, 5), "mixed": False,
                "steps": rng.choice([16, 32, 48])}
    return {"kind": "serve", "requests": rng.randint(3, 6)}


# ------------------------------------------------------- meshes and parameters
def _cart_lines(nx: int, ny: int, x1: float, y1: float, codes) -> str:
    return (f"meshType = 1\nnElemsX = {nx}\nnElemsY = {ny}\nX0 = (/0.0, 0.0/)\nXmax = (/{x1!r}, {y1!r}/)\n"
            "nBCsegments = (/1, 1, 1, 1/)\n" + "".join(f"meshBCtype = {c}\n" for c in codes))


def _riemann_ini(nx: int, ny: int, flux: int) -> str:
    text = meshgen.riemann2d_ini("riemann", [(1.0, 0.0, 0.0, 1.0)] * 4, steps=10**9, flux=flux)
    mesh = "meshType = 0\nmeshFormat = .msh\nmeshFile = riemann\n"
    assert mesh in text
    return text.replace(mesh, _cart_lines(nx, ny, 1.0, 1.0, (401, 401, 401, 401)))


def _explicit_case(case: dict, seed: int) -> cc.CaseData:
    flow, nx, ny = case["flow"], case["nx"], case["ny"]
    precision = f"precision = {1 if case['mixed'] else 0}\n"
    if flow == "sod":
        ini = meshgen.sod_ini(nx, ny, flux=case["flux"], limiter=case["limiter"]) + "venk_k = 5.0\n" + precision
        return cc.CaseData.from_text(ini)
    if flow == "riemann":
        ini = _riemann_ini(nx, ny, case["flux"]).replace("limiter = 2", f"limiter = {case['limiter']}") + precision
        return cc.CaseData.from_text(ini)
    with tempfile.TemporaryDirectory() as tmp:
        path = os.path.join(tmp, "mesh.msh")
        if flow == "dmr":
            meshgen.dmr_mesh(nx, ny, seed=seed).write_gmsh(path)
            ini = meshgen.dmr_ini("mesh", flux=case["flux"], limiter=case["limiter"],
                                  precision=1 if case["mixed"] else 0)
        else:
            meshgen.cylinder_mesh(nx, ny).write_gmsh(path)
            ini = meshgen.cylinder_ini("mesh", steps=10**9, flux=case["flux"]).replace(
                "limiter = 2", f"limiter = {case['limiter']}") + precision
        return cc.CaseData.from_text(ini, tmp)


def _flow_state(flow: str, seed: int, x: np.ndarray, y: np.ndarray) -> np.ndarray:
    """A developed-looking primitive state [N, 4] at the points (x, y): the
    flow's shocks, contacts or free stream, disturbed everywhere by a few
    seeded waves."""
    rng = np.random.Generator(np.random.PCG64(seed))
    one = np.ones_like(x)
    if flow == "sod":
        left = x < 0.4999999
        q = [np.where(left, 1.0, 0.125), 0.3 * one, 0.0 * one, np.where(left, 1.0, 0.1)]
        length = 1.0
    elif flow == "dmr":
        post = x < 1.0 / 6.0 + y / math.sqrt(3.0)
        q = [np.where(post, 8.0, 1.4), np.where(post, 8.25 * math.cos(math.pi / 6), 0.0),
             np.where(post, -8.25 * math.sin(math.pi / 6), 0.0), np.where(post, 116.5, 1.0)]
        length = 1.0
    elif flow == "riemann":
        right, top = x > 0.4999999, y > 0.4999999  # a cell centred on the line falls on one side
        states = [(rng.uniform(0.1, 2.0), rng.uniform(-1.0, 1.0), rng.uniform(-1.0, 1.0), rng.uniform(0.1, 2.0))
                  for _ in range(4)]
        q = [np.where(top, np.where(right, states[0][k], states[1][k]),
                      np.where(right, states[3][k], states[2][k])) for k in range(4)]
        length = 1.0
    else:
        q = [one, 0.2 * math.sqrt(GAM) * one, 0.0 * one, one]
        length = 20.0
    out = np.stack(q, axis=1)
    sound = np.sqrt(GAM * out[:, 3] / out[:, 0])
    amp = 0.01 if flow == "cylinder" else 0.03
    for _ in range(4):
        kx, ky = rng.uniform(-8.0, 8.0, 2) * (math.pi / length)
        wave = np.sin(kx * x + ky * y + rng.uniform(0.0, 2.0 * math.pi))
        c = rng.uniform(-amp, amp, 4)
        out[:, 0] *= 1.0 + c[0] * wave
        out[:, 3] *= 1.0 + c[3] * wave
        out[:, 1] += c[1] * sound * wave
        out[:, 2] += c[2] * sound * wave
    return out


def _case_state(case: cc.CaseData, flow: str, seed: int) -> np.ndarray:
    bary = case.mesh()["cell_bary"]
    return _flow_state(flow, seed, np.ascontiguousarray(bary[:, 0]), np.ascontiguousarray(bary[:, 1]))


def _airfoil_case(spec: dict, mixed: bool, ns: bool) -> cc.CaseData:
    with tempfile.TemporaryDirectory() as tmp:
        if not ns:
            return workloads.airfoil_case(spec, tmp, "airfoil", precision=1 if mixed else 0)
        meshgen.naca_ogrid(0.0, 0.0, 0.12, spec["ni"], spec["nj"], h0=1e-4).write_gmsh(
            os.path.join(tmp, "airfoil.msh"))
        ini = meshgen.airfoil_ini("airfoil", mach=0.5, alpha=spec["alpha"], navier_stokes=True, cfl=10.0,
                                  precision=1 if mixed else 0)
        return cc.CaseData.from_text(ini, tmp)


def _airfoil_spec(seed: int, ni: int, nj: int) -> dict:
    spec = workloads.airfoil_specs(1, seed)[0]
    return {**spec, "ni": ni, "nj": nj}


# members of the explicit batch and requests of the stream, from the seed
def _batch_members(case: dict, seed: int) -> list[dict]:
    sizes = [("riemann", 256, 256, 5), ("cylinder", 158, 158, 2), ("riemann", 401, 401, 5),
             ("dmr", 240, 60, 5), ("riemann", 300, 300, 5)][:case["members"]]
    return [{"kind": "explicit", "flow": f, "nx": nx, "ny": ny, "flux": flux, "limiter": 2, "mixed": case["mixed"],
             "steps": case["steps"]} for f, nx, ny, flux in sizes]


def _requests(case: dict, seed: int) -> list[dict]:
    rng = np.random.Generator(np.random.PCG64(seed))

    def riemann(n):
        states = [(rng.uniform(0.1, 2.0), rng.uniform(-1.0, 1.0), rng.uniform(-1.0, 1.0), rng.uniform(0.1, 2.0))
                  for _ in range(4)]
        return {"kind": "riemann", "n": n, "states": states, "steps": 64}

    def cylinder(n_theta, n_r):
        return {"kind": "cylinder", "n_theta": n_theta, "n_r": n_r, "steps": 128}

    def airfoil(k, ni, nj):
        return {"kind": "airfoil", "airfoil": _airfoil_spec(seed * 131 + k, ni, nj), "steps": 1}

    return [riemann(256), airfoil(1, 160, 80), cylinder(158, 158), riemann(333), airfoil(4, 203, 64),
            cylinder(197, 128)][:case["requests"]]


# ----------------------------------------------------------------- prepare, run
class _Job:
    """One solver with the state it starts from and a pinned result buffer."""

    def __init__(self, data: cc.CaseData, state: np.ndarray, mixed: bool):
        self.data = data
        self.solver = cc.Solver(data)
        self._in = torch.from_numpy(state).pin_memory()
        self._out = torch.empty_like(self._in).pin_memory()
        self.state, self.out = self._in.numpy(), self._out.numpy()
        # a mixed-precision run's fields are kept in FP32, the type of its fluxes
        self.dtype = np.float32 if mixed else np.float64

    def reset(self) -> None:
        self.solver.time = 0.0
        self.solver.set_state(self.state)

    def field(self) -> np.ndarray:
        return self.solver.get_state(out=self.out).astype(self.dtype, copy=False)


def _job(case: dict, seed: int) -> _Job:
    if case["kind"] in ("implicit", "lusgs"):
        spec = _airfoil_spec(seed, case["ni"], case["nj"])
        data = _airfoil_case(spec, case["mixed"], case.get("ns", False))
        return _Job(data, data.prim0(), case["mixed"])
    data = _explicit_case(case, seed)
    return _Job(data, _case_state(data, case["flow"], seed), case["mixed"])


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "batch":
        if case["flow"] == "airfoil":
            # uneven grids of the distribution's lower half, so that a pass stays short
            jobs = [_job({"kind": "implicit", "ni": 128 + 37 * k, "nj": 64 + (53 * k) % 97, "ns": False,
                          "mixed": case["mixed"]}, seed * 131 + k) for k in range(case["members"])]
        else:
            jobs = [_job(m, seed * 131 + k) for k, m in enumerate(_batch_members(case, seed))]
        return {"case": case, "jobs": jobs}
    if kind == "serve":
        with tempfile.TemporaryDirectory() as tmp:
            reqs = [(workloads.stream_case(r, tmp, f"request{k}"), r["steps"])
                    for k, r in enumerate(_requests(case, seed))]
        return {"case": case, "requests": reqs}
    job = _job(case, seed)
    state = {"case": case, "job": job}
    if kind == "residual":
        job.reset()
    if kind == "lusgs":
        job.reset()
        job.solver.build_matrix(0.0, job.solver.calc_time_step())
        rng = np.random.Generator(np.random.PCG64(seed))
        state["rhs"] = rng.standard_normal((job.solver.n, 4))
    return state


def _report(rep: dict, dtype) -> dict:
    return {"t": np.array([rep["t"]], dtype=dtype), "residual": np.array(rep["residual"][:4], dtype=dtype)}


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind in ("explicit", "implicit"):
        job = state["job"]
        job.reset()
        rep = job.solver.run(case["steps"])
        out = {"state": job.field(), **_report(rep, job.dtype)}
        if kind == "implicit":
            out["clcd"] = np.array([rep["cl"], rep["cd"]], dtype=job.dtype)
        return out
    if kind == "residual":
        ut, grad = state["job"].solver.fv_time_derivative(0.0, with_grad=True)
        return {"ut": ut, "grad": grad}
    if kind == "lusgs":
        return {"x": state["job"].solver.lusgs(state["rhs"]).astype(state["job"].dtype, copy=False)}
    if kind == "batch":
        batch = cc.Batch(0)
        for job in state["jobs"]:
            job.reset()
            batch.add(job.solver, case["steps"])
        left = case["steps"]
        while left > 0:
            batch.step(min(left, 16))
            left -= 16
        reps = [batch.report(job.solver) for job in state["jobs"]]
        batch.close()
        return [{"state": job.field(), **_report(rep, job.dtype)} for job, rep in zip(state["jobs"], reps)]
    server = cc.Server(0)
    ids = [server.submit(data, steps) for data, steps in state["requests"]]
    while True:
        queued, running, _ = server.poll(16)
        if queued + running == 0:
            break
    out = [server.result(i)[1] for i in ids]
    server.close()
    return out


# ------------------------------------------------------------------------ work
# A pass over time steps cannot do without its residual evaluations, each a
# pass over the mesh and the state: their bytes are counted per evaluation.
def _explicit_work(case: dict) -> tuple[float, float]:
    """Bytes and operations of one residual evaluation with its update."""
    tri = case["flow"] in ("dmr", "cylinder")
    n = case["nx"] * case["ny"] * (2 if tri else 1)
    sides, faces = (3, 1.5) if tri else (4, 2.0)
    ns = case["flow"] == "cylinder"
    # state in and out, stage-start state, 1/area, eps^2; neighbour, flux code,
    # weights and offset per side; normal, length and cells per face
    bytes_cell = 32 + 32 + 32 + 8 + (8 if case["limiter"] == 2 else 0) + sides * 40 + faces * (32 + (24 if ns else 0))
    # gradient 20, limiter 40 / 76 per side; reconstruction, flux, rotation per face; update
    flops_cell = sides * (20 + (76 if case["limiter"] == 2 else 40)) + faces * (230 + (110 if ns else 0)) + 30
    return n * float(bytes_cell), n * float(flops_cell)


def _implicit_work(n: int, steps: int, ns: bool, mixed: bool) -> tuple[float, float]:
    """Bytes and operations of implicit steps at the usual two Newton
    iterations per step, four Krylov iterations each, eight colours."""
    b, f = _explicit_work({"flow": "riemann", "nx": n, "ny": 1, "limiter": 2})
    word = 4 if mixed else 8
    sweep = n * (2 * 16 + 2 * 2 * 16 + 5 * 4) * word
    newton, krylov = 2 * steps, 8 * steps
    evals = newton * (1 + 4 * 8) + krylov + steps
    bytes_ = evals * b + krylov * (sweep + 10 * n * 4 * word)
    flops = evals * f + krylov * n * (6 * 32 + 100.0)
    return bytes_, flops * (1.3 if ns else 1.0)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "explicit":
        n_state = case["nx"] * case["ny"] * (2 if case["flow"] in ("dmr", "cylinder") else 1) * 64.0
        b, f = _explicit_work(case)
        return {"bytes": 3 * case["steps"] * b + n_state, "flops": 3 * case["steps"] * f}
    if kind == "residual":
        n = case["nx"] * case["ny"] * 2
        b, f = _explicit_work(case)
        return {"bytes": b + 64.0 * n, "flops": f}
    if kind == "implicit":
        b, f = _implicit_work(case["ni"] * case["nj"], case["steps"], case["ns"], case["mixed"])
        return {"bytes": b, "flops": f}
    if kind == "lusgs":
        n, word = case["ni"] * case["nj"], 4 if case["mixed"] else 8
        return {"bytes": n * float((2 * 16 + 2 * 2 * 16 + 5 * 4) * word), "flops": n * 6 * 32.0}
    if kind == "batch" and case["flow"] == "airfoil":
        parts = [_implicit_work((128 + 37 * k) * (64 + (53 * k) % 97), case["steps"], False, case["mixed"])
                 for k in range(case["members"])]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    total = {"bytes": 0.0, "flops": 0.0}
    for m in (_batch_members(case, 0) if kind == "batch" else _requests(case, 0)):
        if m["kind"] == "airfoil":
            b, f = _implicit_work(m["airfoil"]["ni"] * m["airfoil"]["nj"], m["steps"], False, False)
            w = {"bytes": b, "flops": f}
        elif m["kind"] in ("riemann", "cylinder"):
            w = work({"kind": "explicit", "flow": m["kind"], "nx": m.get("n", m.get("n_theta")),
                      "ny": m.get("n", m.get("n_r")), "limiter": 2, "steps": m["steps"]})
        else:
            w = work(m)
        total = {k: total[k] + w[k] for k in total}
    return total


# ----------------------------------------------------------------------- exact
# Plain FP64 tensor code of the scheme: second-order finite volumes on one
# kind of cell (all triangles or all quads), least-squares gradients with the
# Barth-Jespersen or Venkatakrishnan limiter, Roe / HLL / HLLC and the viscous
# flux, three-stage Runge-Kutta with the global CFL time step.
class _Mesh:
    def __init__(self, nodes: np.ndarray, cells: np.ndarray, edges: np.ndarray, dev):
        n, s = cells.shape
        a, b = cells, np.roll(cells, -1, axis=1)
        big = len(nodes) + 1
        key = np.concatenate([(np.minimum(a, b) * big + np.maximum(a, b)).ravel(),
                              np.minimum(edges[:, 0], edges[:, 1]) * big + np.maximum(edges[:, 0], edges[:, 1])])
        order = np.argsort(key, kind="stable").reshape(-1, 2)  # cell sides come before boundary edges
        other = np.full(len(key), -1)
        other[order[:, 0]], other[order[:, 1]] = order[:, 1], order[:, 0]
        side = other[:n * s]
        code = np.where(side >= n * s, edges[np.maximum(side - n * s, 0), 2], 0)
        t = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=dev)
        xy = t(nodes)
        pa, pb = xy[t(a)], xy[t(b)]
        self.bary = pa.mean(dim=1)
        mid = 0.5 * (pa + pb)
        nrm = torch.stack([pb[..., 1] - pa[..., 1], pa[..., 0] - pb[..., 0]], -1)
        self.len = nrm.norm(dim=-1)
        nrm = nrm / self.len[..., None]
        self.gp = mid - self.bary[:, None]
        self.nrm = torch.where(((nrm * self.gp).sum(-1) < 0)[..., None], -nrm, nrm)
        self.mid = mid
        self.code = t(code.reshape(n, s))
        self.ghost = self.code > 0
        self.side = t(np.where(side >= n * s, 0, side).reshape(n, s))
        self.nb = self.side // s
        mirror = self.bary[:, None] + 2.0 * (self.gp * self.nrm).sum(-1).abs()[..., None] * self.nrm
        self.there = torch.where(self.ghost[..., None], mirror, self.bary[self.nb])
        self.bb = self.there - self.bary[:, None]
        g = torch.einsum("nki,nkj->nij", self.bb, self.bb)
        self.w = torch.einsum("nij,nkj->nki", torch.linalg.inv(g), self.bb)
        p = xy[t(cells)]
        q = p.roll(-1, dims=1)
        self.area = 0.5 * (p[..., 0] * q[..., 1] - p[..., 1] * q[..., 0]).sum(1).abs()
        self.s = 0.5 * (self.nrm.abs() * self.len[..., None]).sum(1)


def _raw_mesh(case: dict, seed: int):
    nx, ny = case["nx"], case["ny"]
    if case["flow"] == "dmr":
        m = meshgen.dmr_mesh(nx, ny, seed=seed)
        return m.nodes, m.tria[:, :3], m.bc
    if case["flow"] == "cylinder":
        m = meshgen.cylinder_mesh(nx, ny)
        return m.nodes, m.tria[:, :3], m.bc
    x, y = np.meshgrid(np.linspace(0, 1, nx + 1), np.linspace(0, 1.0 if case["flow"] == "riemann" else 0.05, ny + 1))
    j, i = np.meshgrid(np.arange(ny), np.arange(nx), indexing="ij")
    a = (j * (nx + 1) + i).ravel()
    wall = 401 if case["flow"] == "riemann" else 101
    row, col = np.arange(nx), np.arange(ny)
    edges = [np.stack([row, row + 1, 0 * row + wall], 1),
             np.stack([row + ny * (nx + 1), row + ny * (nx + 1) + 1, 0 * row + wall], 1),
             np.stack([col * (nx + 1), (col + 1) * (nx + 1), 0 * col + 401], 1),
             np.stack([col * (nx + 1) + nx, (col + 1) * (nx + 1) + nx, 0 * col + 401], 1)]
    return np.stack([x.ravel(), y.ravel()], 1), np.stack([a, a + 1, a + nx + 2, a + nx + 1], 1), np.concatenate(edges)


def _cons(p):
    e = p[..., 3] / (GAM - 1) + 0.5 * p[..., 0] * (p[..., 1] ** 2 + p[..., 2] ** 2)
    return torch.stack([p[..., 0], p[..., 0] * p[..., 1], p[..., 0] * p[..., 2], e], -1)


def _prim(c):
    u, v = c[..., 1] / c[..., 0], c[..., 2] / c[..., 0]
    p = (GAM - 1) * (c[..., 3] - 0.5 * (c[..., 1] * u + c[..., 2] * v))
    small = torch.full_like(p, 1e-10)
    return torch.stack([torch.where(c[..., 0] < 1e-19, small, c[..., 0]), u, v, torch.where(p < 1e-19, small, p)], -1)


def _rotate(q, n, back=False):
    s = -1.0 if back else 1.0
    return torch.stack([q[..., 0], n[..., 0] * q[..., 1] + s * n[..., 1] * q[..., 2],
                        n[..., 0] * q[..., 2] - s * n[..., 1] * q[..., 1], q[..., 3]], -1)


def _far_field(q, n, far):
    """Characteristic far field; the wave speeds of the transformation take
    the interior velocity's x component."""
    inner, outer = _cons(_rotate(q, n)), _cons(_rotate(far.expand_as(q), n))
    c = torch.sqrt(GAM * q[..., 3] / q[..., 0])
    u = q[..., 1]
    h = c * c / (GAM - 1) + 0.5 * u * u
    one = torch.ones_like(u)
    right = torch.stack([torch.stack([one, one, one], -1), torch.stack([u - c, u, u + c], -1),
                         torch.stack([h - u * c, 0.5 * u * u, h + u * c], -1)], -2)
    left = torch.linalg.inv(right)
    pick = lambda v: torch.stack([v[..., 0], v[..., 1], v[..., 3]], -1)[..., None]
    wi, wo = (left @ pick(inner))[..., 0], (left @ pick(outer))[..., 0]
    vn = n[..., 0] * far[1] + n[..., 1] * far[2]
    cf = torch.sqrt(GAM * far[3] / far[0])
    w = torch.where(torch.stack([vn - cf > 0, vn > 0, vn + cf > 0], -1), wi, wo)
    g = (right @ w[..., None])[..., 0]
    mt = torch.where(vn > 0, inner[..., 2], outer[..., 2])
    return _rotate(_prim(torch.stack([g[..., 0], g[..., 1], mt, g[..., 2]], -1)), n, back=True)


def _dmr_solution(x, time, dx_ref):
    s = torch.tanh((x[..., 0] - (1.0 / 6.0 + (20.0 * time + x[..., 1]) / math.sqrt(3.0))) * (math.pi / (0.2 * dx_ref)))
    summ, diff = (9.4, 57.157676649772950686, -33.0, 566.0), (6.6, 57.157676649772950686, -33.0, 561.0)
    return _prim(torch.stack([0.5 * (a - b * s) for a, b in zip(summ, diff)], -1))


class _Scheme:
    def __init__(self, case: dict, seed: int):
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.m = _Mesh(*_raw_mesh(case, seed), dev)
        self.case = case
        self.ns = case["flow"] == "cylinder"
        self.far = torch.tensor([1.0, 0.2 * math.sqrt(GAM), 0.0, 1.0], dtype=torch.float64, device=dev)
        self.mu, self.pr = (0.2 * math.sqrt(GAM) / 100.0, 0.72) if self.ns else (0.0, 0.72)
        self.total = self.m.area.sum()
        self.dx_ref = torch.sqrt(self.total / len(self.m.area))
        b = self.m.bary.cpu().numpy()
        self.start = torch.as_tensor(_flow_state(case["flow"], seed, b[:, 0].copy(), b[:, 1].copy()), device=dev)
        self.cells, self.sides = torch.nonzero(self.m.ghost, as_tuple=True)
        self.bcode = self.m.code[self.cells, self.sides]

    def _ghost(self, q, n, x, time):
        local = _rotate(q, n)
        slip = _rotate(torch.stack([local[:, 0], -local[:, 1], local[:, 2], local[:, 3]], 1), n, back=True)
        stick = torch.stack([q[:, 0], -q[:, 1], -q[:, 2], q[:, 3]], 1)
        out = q.clone()
        code = self.bcode[:, None]
        out = torch.where(code == 101, slip, out)
        out = torch.where(code == 201, stick, out)
        if self.case["flow"] == "dmr":
            out = torch.where(code == 601, _dmr_solution(x, time, self.dx_ref), out)
        if self.ns:
            out = torch.where(code == 501, _far_field(q, n, self.far), out)
        return out

    def gradients(self, q, time):
        m = self.m
        qn = q[m.nb]
        k = (self.cells, self.sides)
        qn[k] = self._ghost(q[self.cells], m.nrm[k], m.there[k], time)
        grad = torch.einsum("nki,nkv->nvi", m.w, qn - q[:, None])
        low, high = torch.minimum(qn.amin(1), q) - q, torch.maximum(qn.amax(1), q) - q
        d = torch.einsum("nvi,nki->nkv", grad, m.gp)
        lim = torch.where(d > 0, high[:, None], low[:, None])
        safe = torch.where(d == 0, torch.ones_like(d), d)
        if self.case["limiter"] == 1:
            phi = torch.clamp(lim / safe, max=1.0)
        else:
            e = ((5.0 * torch.sqrt(m.area)) ** 3)[:, None, None]
            phi = ((lim * lim + e) * safe + 2.0 * d * d * lim) / (lim * lim + 2.0 * d * d + d * lim + e) / safe
        phi = torch.where(d == 0, torch.ones_like(d), phi).amin(1).clamp(max=1.0)
        return grad * phi[..., None], qn

    def residual(self, q, time):
        m = self.m
        if self.case["mixed"]:
            raise ValueError("the scheme's FP64 form")
        grad, qn = self.gradients(q, time)
        left = q[:, None] + torch.einsum("nvi,nki->nkv", grad, m.gp)
        right = left.reshape(-1, 4)[m.side]
        k = (self.cells, self.sides)
        right[k] = self._ghost(left[k], m.nrm[k], m.mid[k], time)
        f = _rotate(self._flux(_rotate(left, m.nrm), _rotate(right, m.nrm)), m.nrm, back=True)
        if self.ns:
            gn = torch.where(m.ghost[..., None, None], torch.zeros_like(grad[:1, None]), grad[m.nb])
            dist = m.bb.norm(dim=-1)
            b = m.bb / dist[..., None]
            g = 0.5 * (grad[:, None] + gn)
            corr = (g * b[..., None, :]).sum(-1) - (qn - q[:, None]) / dist[..., None]
            g = g - corr[..., None] * b[..., None, :]
            f = f - self._viscous(0.5 * (left + right), g, m.nrm)
        f = f * m.len[..., None]
        return -f.sum(1) / m.area[:, None], grad

    def _viscous(self, s, g, n):
        mu, r, u, v, p = self.mu, s[..., 0], s[..., 1], s[..., 2], s[..., 3]
        ux, uy, vx, vy = g[..., 1, 0], g[..., 1, 1], g[..., 2, 0], g[..., 2, 1]
        txx, tyy, txy = mu * (4 / 3 * ux - 2 / 3 * vy), mu * (4 / 3 * vy - 2 / 3 * ux), mu * (uy + vx)
        heat = mu * GAM / ((GAM - 1) * self.pr) * (r[..., None] * g[..., 3, :] - p[..., None] * g[..., 0, :]) \
            / (r * r)[..., None]
        ex, ey = u * txx + v * txy + heat[..., 0], u * txy + v * tyy + heat[..., 1]
        x, y = n[..., 0], n[..., 1]
        return torch.stack([0 * x, txx * x + txy * y, txy * x + tyy * y, ex * x + ey * y], -1)

    def _flux(self, a, b):
        ua, ub = _cons(a), _cons(b)

        def physical(p, u):
            return torch.stack([u[..., 1], u[..., 1] * p[..., 1] + p[..., 3], u[..., 1] * p[..., 2],
                                p[..., 1] * (u[..., 3] + p[..., 3])], -1)

        fa, fb = physical(a, ua), physical(b, ub)
        ra, rb = torch.sqrt(a[..., 0]), torch.sqrt(b[..., 0])
        mean = lambda x, y: (ra * x + rb * y) / (ra + rb)
        ha, hb = (ua[..., 3] + a[..., 3]) / a[..., 0], (ub[..., 3] + b[..., 3]) / b[..., 0]
        u, v, h = mean(a[..., 1], b[..., 1]), mean(a[..., 2], b[..., 2]), mean(ha, hb)
        c = torch.sqrt((GAM - 1) * (h - 0.5 * (u * u + v * v)))
        ca, cb = torch.sqrt(GAM * a[..., 3] / a[..., 0]), torch.sqrt(GAM * b[..., 3] / b[..., 0])
        if self.case["flux"] == 2:
            return self._roe(a, b, ua, ub, fa, fb, u, v, h, c, ca, cb)
        sr = torch.maximum(b[..., 1] + cb, u + c)
        sl = torch.minimum(a[..., 1] - ca, u - c)
        if self.case["flux"] == 3:
            star = ((sr[..., None] * fa - sl[..., None] * fb) + (sr * sl)[..., None] * (ub - ua)) / (sr - sl)[..., None]
        else:
            da, db = a[..., 0] * (sl - a[..., 1]), b[..., 0] * (sr - b[..., 1])
            sm = (b[..., 3] - a[..., 3] + a[..., 1] * da - b[..., 1] * db) / (da - db)

            def half(p, uu, f, s, d):
                fac = d / (s - sm)
                e = fac * (uu[..., 3] / p[..., 0] + (sm - p[..., 1]) * (sm + p[..., 3] / d))
                return f + s[..., None] * (torch.stack([fac, sm * fac, p[..., 2] * fac, e], -1) - uu)

            star = torch.where((sm >= 0)[..., None], half(a, ua, fa, sl, da), half(b, ub, fb, sr, db))
        return torch.where((sl > 0)[..., None], fa, torch.where((sr < 0)[..., None], fb, star))

    @staticmethod
    def _roe(a, b, ua, ub, fa, fb, u, v, h, c, ca, cb):
        lam = torch.stack([u - c, u, u, u + c], -1)
        la = torch.stack([a[..., 1] - ca, a[..., 1], a[..., 1], a[..., 1] + ca], -1)
        lb = torch.stack([b[..., 1] - cb, b[..., 1], b[..., 1], b[..., 1] + cb], -1)
        da = torch.clamp(torch.maximum(lam - la, lb - lam), min=0.0)
        safe = torch.where(da > 0, da, torch.ones_like(da))
        mag = torch.where(lam.abs() < da, 0.5 * (lam * lam / safe + da), lam.abs())
        d = ub - ua
        de = d[..., 3] - (d[..., 2] - v * d[..., 0]) * v
        w2 = -(GAM - 1) / (c * c) * (d[..., 0] * (u * u - h) + de - d[..., 1] * u)
        w1 = -0.5 / c * (d[..., 1] - d[..., 0] * (u + c)) - 0.5 * w2
        w4 = d[..., 0] - w1 - w2
        w3 = d[..., 2] - v * d[..., 0]
        one, zero = torch.ones_like(u), torch.zeros_like(u)
        vecs = (torch.stack([one, u - c, v, h - u * c], -1), torch.stack([one, u, v, 0.5 * (u * u + v * v)], -1),
                torch.stack([zero, zero, one, v], -1), torch.stack([one, u + c, v, h + u * c], -1))
        out = fa + fb
        for k, w in enumerate((w1, w2, w3, w4)):
            out = out - (w * mag[..., k])[..., None] * vecs[k]
        return 0.5 * out

    def time_step(self, q):
        m = self.m
        cfl = 0.5 if self.case["flow"] == "sod" else 0.8
        a = torch.sqrt(GAM * q[:, 3] / q[:, 0])
        dt = (cfl * m.area / ((q[:, 1].abs() + a) * m.s[:, 0] + (q[:, 2].abs() + a) * m.s[:, 1])).amin()
        if self.ns:
            ssv = max(4.0 / 3.0, GAM / self.pr) * self.mu * (m.s ** 2).sum(1)
            dt = torch.minimum(dt, (0.9 * q[:, 0] ** 2 * m.area ** 2 / (4.0 * ssv)).amin())
        return dt

    def run(self, steps: int) -> dict:
        q, t = self.start, torch.zeros((), dtype=torch.float64, device=self.start.device)
        for _ in range(steps):
            u0, dt = _cons(q), self.time_step(q)
            for s in range(1, 4):
                r, _ = self.residual(q, t + RK3[s - 1] * dt)
                q = _prim(u0 + RK3[s] * dt * r)
            t = t + dt
        res = torch.sqrt((self.m.area[:, None] * r * r).sum(0) / self.total)
        return {"state": q.cpu().numpy(), "t": t.reshape(1).cpu().numpy(), "residual": res.cpu().numpy()}


def exact(case: dict, seed: int):
    """FP64 values of the explicit results (the mixed runs' too: the same
    scheme evaluated in 64 bits).  Implicit steps and the blocks of the
    preconditioner have none: they are inexact Newton iterates and finite
    differences.  The served stream holds such steps, and its explicit
    requests are the same path as the explicit cases."""
    kind = case["kind"]
    if kind == "explicit":
        return _Scheme({**case, "mixed": False}, seed).run(case["steps"])
    if kind == "residual":
        s = _Scheme(case, seed)
        ut, grad = s.residual(s.start, 0.0)
        return {"ut": ut.cpu().numpy(), "grad": grad.transpose(1, 2).reshape(-1, 8).cpu().numpy()}
    if kind == "batch" and case["flow"] == "explicit":
        return [_Scheme({**m, "mixed": False}, seed * 131 + k).run(case["steps"])
                for k, m in enumerate(_batch_members(case, seed))]
    return None
