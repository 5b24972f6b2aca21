"""The workloads the framework's speed is judged by, through its public entry points.

Four kinds of call, as a user's program makes them:

* ``transient``: a forward solve held by ``Solver`` (mesh read, planned and assembled in
  ``prepare``): factorizations of every step size, all time steps, receivers, results on
  the host.  ``server`` sends several models to a running ``Server`` and waits for them;
  ``directory`` is the drop-in call that reads a directory and writes the output files.
* ``stationary``: the grounded wire's initial field from a directory's files to its files.
* ``system``: the in-process solver boundary ``pardiso_64``: new values in a known pattern
  are factorized, then solved with, as a time loop does on each change of step size.
* ``residual``: the device check ||b - A x|| of given columns.

Sizes: the served stream's meshes go from 30^3 to 100^3 cells, the tests' from 6^3 to 40^3,
the benchmarks are 40^3 and 80^3 with 1 or 32 wires.  Time grids are the benchmarks' first
step-size decades, cut so that a pass stays below two seconds; each decade costs one
factorization, as in the full grids.
"""
from __future__ import annotations

import dataclasses
import importlib
import math
import os
import tempfile

import numpy as np
import torch

PKG = "a-e_formulations_3d_timedomain_em_horizontalgroundedwiresource_b200"
tdem = importlib.import_module(PKG)
mg = importlib.import_module(PKG + ".modelgen")
outputs = importlib.import_module(PKG + ".outputs")

FIRST_STEP = 2e-5  # seconds: the first step of the 80^3 benchmark's grid to 0.1 s


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a residual check of one column on the smallest mesh: nothing but latency
        dict(name="residual_9cubed", kind="residual", nx=9, ny=9, nz=9, cols=1),
        # the check of a 32-source block on a mesh whose matrix is larger than L2
        dict(name="residual_32cols", kind="residual", nx=65, ny=65, nz=64, cols=32),
        # the tests' smallest transient: every launch is latency
        dict(name="cube8_A2", kind="transient", mesh="small", cells=8, form="A", scheme=2, wires=1,
             decades=3, steps=6, precision=64),
        # a few wires on a small mesh, E-form and BDF2
        dict(name="cube13_E3_5wires", kind="transient", mesh="small", cells=13, form="E", scheme=3, wires=5,
             decades=3, steps=7, precision=64),
        # the plain-method benchmark in full: 40^3 half-space, backward Euler, 120 steps
        dict(name="halfspace40_A2", kind="transient", mesh="halfspace", cells=40, form="A", scheme=2, wires=1,
             decades=6, steps=20, precision=64),
        # the headline mesh: 80^3 layers and block, E-form, BDF2, one wire
        dict(name="layers80_E3", kind="transient", mesh="layers", cells=80, form="E", scheme=3, wires=1,
             decades=1, steps=20, precision=64),
        # a survey of 32 wires over one earth solved as one block per step
        dict(name="layers48_A3_32wires", kind="transient", mesh="layers", cells=48, form="A", scheme=3, wires=32,
             decades=2, steps=10, precision=64),
        # the FP32-held factor with FP64 refinement, on an odd mesh
        dict(name="layers35_E2_mixed", kind="transient", mesh="layers", cells=35, form="E", scheme=2, wires=1,
             decades=2, steps=9, precision=32),
        # four requests of a served stream's smaller sizes at once, planning included
        dict(name="server_4requests", kind="server", mesh="layers", cells=30, form="A", scheme=3, wires=1,
             decades=3, steps=10, precision=64, requests=4),
        # the drop-in call: files in, files out
        dict(name="directory24_E2", kind="directory", mesh="layers", cells=24, form="E", scheme=2, wires=2,
             decades=3, steps=8, precision=64),
        # the initial field that feeds a transient
        dict(name="stationary28", kind="stationary", mesh="layers", cells=28, wires=2),
        # another program's solver calls
        dict(name="system_41x36x29", kind="system", nx=41, ny=36, nz=29, cols=3, solves=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["transient", "residual", "system", "server", "directory", "stationary"],
                       [10, 2, 2, 1, 1, 1])[0]
    if kind == "residual":
        return dict(kind=kind, nx=_log_int(rng, 5, 70), ny=_log_int(rng, 5, 70), nz=_log_int(rng, 5, 70),
                    cols=_log_int(rng, 1, 64))
    if kind == "system":
        return dict(kind=kind, nx=_log_int(rng, 8, 48), ny=_log_int(rng, 8, 48), nz=_log_int(rng, 8, 32),
                    cols=_log_int(rng, 1, 32), solves=rng.randint(1, 6))
    if kind == "stationary":
        return dict(kind=kind, mesh="layers", cells=rng.randint(14, 34), wires=rng.randint(1, 4))
    c = dict(kind=kind, form=rng.choice("AE"), scheme=rng.choice([2, 3]), precision=64,
             decades=rng.randint(1, 4), steps=rng.randint(8, 16))
    if kind == "server":
        return dict(c, mesh="layers", cells=rng.randint(16, 36), wires=1, requests=rng.randint(2, 6))
    if kind == "directory":
        return dict(c, mesh="layers", cells=rng.randint(14, 32), wires=rng.randint(1, 3))
    mesh = rng.choice(["small", "layers", "layers", "halfspace"])
    cells = _log_int(rng, 6, 14) if mesh == "small" else _log_int(rng, 24 if mesh == "halfspace" else 16, 60)
    wires = _log_int(rng, 1, 32) if rng.random() < 0.5 else 1
    if cells > 48:  # the largest meshes with one or two wires
        wires = min(wires, 2)
    if wires == 1 and cells <= 44 and rng.random() < 0.2:
        c["precision"] = 32
    return dict(c, mesh=mesh, cells=cells, wires=wires)


# ---------------------------------------------------------------------------
# transient models on disk
# ---------------------------------------------------------------------------
def _wires(count, shift):
    """count 100 m wires along x on a grid of four columns around the origin."""
    if count == 1:
        return [((-50.0 + shift, 0.0, 0.0), (50.0 + shift, 0.0, 0.0))]
    rows = -(-count // 4)
    return [((a[0] + shift, a[1], a[2]), (b[0] + shift, b[1], b[2]))
            for a, b in mg.wire_grid_sources(min(4, count), rows)[:count]]


def _model(case, seed):
    """The model of a case: its mesh by the sizes, its earth and wires by the seed."""
    rng = np.random.default_rng(seed)
    cells, wires = case["cells"], case["wires"]
    decades, steps = case.get("decades", 1), case.get("steps", 8)
    t_end = FIRST_STEP * steps * (2 ** decades - 1)
    times = mg.decade_time_grid(t_end, decades, steps)
    shift = float(rng.uniform(-8.0, 8.0))
    if case["mesh"] == "small":
        spec = mg.small_model(cells=cells, n_sources=wires)
        spec = dataclasses.replace(
            spec, times=times,
            sources=[((a[0] + shift, a[1], a[2]), (b[0] + shift, b[1], b[2])) for a, b in spec.sources],
            boxes=[mg.Box(-30.0, 30.0, -30.0, 30.0, -50.0, -20.0, float(rng.uniform(0.1, 0.4)))])
    elif case["mesh"] == "halfspace":
        spec = mg.halfspace_model(cells=cells, n_air=(3 * cells) // 8, sigma=float(rng.uniform(0.005, 0.02)))
        spec = dataclasses.replace(spec, times=times)
    else:  # the served stream's mesh rule, which at 80 cells gives the benchmark's mesh
        core_half = 200.0
        n_core = max(8, cells // 2)
        core_h = 2 * core_half / n_core
        x = mg.symmetric_axis(core_half, core_h, (cells - n_core) // 2, 5000.0)
        n_air = max(4, cells // 4)
        n_earth = cells - n_air
        n_core_z = max(2, min(n_earth // 2, int(300.0 / core_h)))
        z = mg.vertical_axis(n_core_z * core_h, core_h, n_earth - n_core_z, 5000.0, n_air, 5000.0)
        layers = [(0.0, 0.01), (-50.0, 0.1), (-300.0, 0.001)]
        layers = [(top, s * float(rng.uniform(0.5, 2.0))) for top, s in layers]
        rec = mg.receivers_on_y_axis(21)
        spec = mg.ModelSpec(x=x, y=x.copy(), z=z, layers=layers, boxes=mg.random_blocks(seed, count=2), sources=[],
                            receivers_b=[rec], receivers_e=[rec], times=times)
    if case["mesh"] != "small":
        sources = _wires(wires, shift)
        spec = dataclasses.replace(spec, sources=sources, receivers_b=[spec.receivers_b[0]] * wires,
                                   receivers_e=[spec.receivers_e[0]] * wires)
    return spec


def _directory(case, seed, initial_field=True):
    d = tempfile.TemporaryDirectory(prefix="tdem_case_")
    spec = _model(case, seed)
    mg.write_model(d.name, spec)
    if initial_field:
        mg.write_analytic_initial_field(d.name, spec)
    return d, spec


# ---------------------------------------------------------------------------
# systems on tensor grids: K_sigma + c M_sigma, trilinear elements, sigma by layer
# ---------------------------------------------------------------------------
def _axis_matrices(h, weight, free_end):
    """(diagonal, off-diagonal) of the 1D stiffness and mass matrices of linear elements
    of lengths h; the first node is fixed (left out), and so is the last unless free_end."""
    k, m = weight / h, weight * h
    kd, md = k.copy(), m / 3
    kd[:-1] += k[1:]
    md[:-1] += m[1:] / 3
    ko, mo = -k[1:], m[1:] / 6
    if not free_end:
        kd, md, ko, mo = kd[:-1], md[:-1], ko[:-1], mo[:-1]
    return (kd, ko), (md, mo)


def _grid_system(case, seed):
    rng = np.random.default_rng(seed)
    axes = []
    for n, free in ((case["nx"], False), (case["ny"], False), (case["nz"], True)):
        cells = n if free else n + 1
        h = 10.0 * 1.04 ** np.abs(np.arange(cells) - (0 if free else cells / 2)) * rng.uniform(0.9, 1.1, cells)
        weight = 10.0 ** rng.uniform(-3, -1, 1 + cells // 8)[np.arange(cells) // 8] if free else np.ones(cells)
        axes.append(_axis_matrices(h, weight, free))
    return axes, 1e-4  # c: the shift of the mass matrix, 1/m^2


def _dense(tri):
    return np.diag(tri[0]) + np.diag(tri[1], 1) + np.diag(tri[1], -1)


def _band(tri, n, offset):
    """Entry (i, i + offset) of a tridiagonal matrix for every i (0 outside)."""
    out = np.zeros(n)
    if offset == 0:
        out[:] = tri[0]
    elif offset == 1:
        out[:-1] = tri[1]
    else:
        out[1:] = tri[1]
    return out


def _grid_csr(case, axes, shift, upper):
    """(row pointers, columns, values), 0-based, of the system's full or upper part."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    iz, iy, ix = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    cols, vals, keep = [], [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                step = (dz * ny + dy) * nx + dx
                if upper and step < 0:
                    continue
                (kx, mx), (ky, my), (kz, mz) = [
                    (_band(a[0], m, o), _band(a[1], m, o)) for a, m, o in zip(axes, (nx, ny, nz), (dx, dy, dz))]
                v = (mz[:, None, None] * (ky[:, None] * mx + my[:, None] * (kx + shift * mx))
                     + kz[:, None, None] * (my[:, None] * mx))
                ok = ((ix + dx >= 0) & (ix + dx < nx) & (iy + dy >= 0) & (iy + dy < ny)
                      & (iz + dz >= 0) & (iz + dz < nz))
                cols.append(np.arange(n) + step)
                vals.append(v.reshape(-1))
                keep.append(ok.reshape(-1))
    keep = np.stack(keep, 1)
    ptr = np.concatenate([[0], np.cumsum(keep.sum(1))])
    return ptr.astype(np.int64), np.stack(cols, 1)[keep], np.ascontiguousarray(np.stack(vals, 1)[keep])


def _columns(case, seed):
    return np.random.default_rng(seed + 1).standard_normal((case["cols"], case["nx"] * case["ny"] * case["nz"]))


class _SystemHandle:
    """MKL's pt array; the handle is released with the object."""

    def __init__(self):
        self.pt = np.zeros(64, dtype=np.int64)

    def __del__(self):
        one = np.ones(2, dtype=np.int64)
        try:
            tdem.pardiso_64(self.pt, -1, np.zeros(1), one, one)
        except Exception:
            pass


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def _check(code):
    if code != 0:
        raise RuntimeError("pardiso_64 returned %d" % code)


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "transient":
        d, _ = _directory(case, seed)
        state["solver"] = tdem.Solver(d.name, case["form"], case["scheme"], precision=case["precision"])
        d.cleanup()
    elif kind == "server":
        state["dirs"] = [_directory(case, 1000 * seed + k)[0] for k in range(case["requests"])]
        state["server"] = tdem.Server(max_active=4, prep_threads=2)
    elif kind == "directory":
        state["dir"], _ = _directory(case, seed)
    elif kind == "stationary":
        state["dir"], state["spec"] = _directory(case, seed, initial_field=False)
    elif kind == "system":
        axes, shift = _grid_system(case, seed)
        ia, ja, a = _grid_csr(case, axes, shift, upper=True)
        ia, ja = ia + 1, ja.astype(np.int64) + 1
        b = _columns(case, seed)
        state.update(a=a, ia=ia, ja=ja, b=b, handle=_SystemHandle())
        # the first factorization brings the analysis of the pattern with it
        _check(tdem.pardiso_64(state["handle"].pt, 12, a, ia, ja, nrhs=case["cols"]))
    else:
        axes, shift = _grid_system(case, seed)
        ptr, col, val = _grid_csr(case, axes, shift, upper=False)
        gpu = [torch.from_numpy(v).cuda() for v in (ptr, col.astype(np.int32), val)]
        x = torch.from_numpy(_columns(case, seed)).cuda()
        # right-hand sides that x solves to a part in 10^5
        b = _product(*gpu, x) * (1.0 + 1e-5 * torch.from_numpy(_columns(case, seed + 7)).cuda())
        state.update(csr=gpu, x=x, b=b, norms=torch.zeros(2 * case["cols"], dtype=torch.float64, device="cuda"))
    return state


def _product(ptr, col, val, x):
    rows = torch.repeat_interleave(torch.arange(len(ptr) - 1, device=x.device), ptr[1:] - ptr[:-1])
    out = torch.zeros_like(x)
    for j in range(x.shape[0]):
        out[j].index_add_(0, rows, val * x[j][col.long()])
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "transient":
        solver = state["solver"]
        solver.run()
        return dict(zip(("e", "emf", "b"), solver.results()))
    if kind == "server":
        server = state["server"]
        ids = [server.submit(d.name, case["form"], case["scheme"]) for d in state["dirs"]]
        return [dict(zip(("e", "emf", "b"), server.results(i, server.wait(i)))) for i in ids]
    if kind == "directory":
        d = state["dir"].name
        tdem.run_directory(d, case["form"], case["scheme"])
        return {name: np.concatenate([np.stack([t for _, t in outputs.read_transients(
            os.path.join(d, "%s.%d" % (name, w + 1)))]) for w in range(case["wires"])])
            for name in ("eall_anom", "edsall_anom", "ball_anom")}
    if kind == "stationary":
        d = state["dir"].name
        tdem.stationary_directory(d)
        return {name: np.fromfile(os.path.join(d, name + ".dat")) for name in ("v3a", "a0")}
    if kind == "system":
        pt, a, ia, ja, b = state["handle"].pt, state["a"], state["ia"], state["ja"], state["b"]
        _check(tdem.pardiso_64(pt, 12, a, ia, ja, nrhs=case["cols"]))
        x = np.empty_like(b)
        for _ in range(case["solves"]):
            _check(tdem.pardiso_64(pt, 33, a, ia, ja, nrhs=case["cols"], b=b, x=x))
        return x
    ptr, col, val = state["csr"]
    x, b, norms = state["x"], state["b"], state["norms"]
    n = x.shape[1]
    tdem.residual_norms(0, n, ptr.data_ptr(), col.data_ptr(), val.data_ptr(), x.data_ptr(), b.data_ptr(), n,
                        case["cols"], norms.data_ptr(), torch.cuda.current_stream().cuda_stream)
    return norms


# ---------------------------------------------------------------------------
# work and exact values
# ---------------------------------------------------------------------------
def work(case):
    """Bytes and flops of one pass.  A transient's: the matrix and each step size's factor
    written once, the factor read twice by each step (the two triangular solves), and the
    factorizations' and solves' flops.  The factor's size under nested dissection of an n-edge
    mesh is fitted to the plans of the 40^3 and 80^3 meshes."""
    kind = case["kind"]
    if kind == "residual":
        n, nnz = _grid_counts(case, upper=False)
        return {"bytes": 12.0 * nnz + 8.0 * n + 16.0 * n * case["cols"], "flops": (2.0 * nnz + 5.0 * n) * case["cols"]}
    if kind == "system":
        n, nnz = _grid_counts(case, upper=True)
        entries, flops = 6.0 * n ** (4 / 3), 40.0 * n ** 2
        solves = case["solves"]
        return {"bytes": 16.0 * nnz + 8.0 * entries * (1 + 2 * solves) + 16.0 * n * case["cols"] * solves,
                "flops": flops + 4.0 * entries * case["cols"] * solves}
    n = 3.0 * case["cells"] ** 3
    entries, flops = 2.25e9 * (n / 1.536e6) ** (4 / 3), 1.38e13 * (n / 1.536e6) ** 2
    if kind == "stationary":  # a scalar potential and one component of the vector potential
        n = n / 3
        entries, flops = 6.0 * n ** (4 / 3), 40.0 * n ** 2
        return {"bytes": 500.0 * n + 2 * 8.0 * entries * 3 + 32.0 * n * case["wires"],
                "flops": 2 * flops + 4.0 * entries * 4 * case["wires"]}
    factorizations = case["decades"] + (case["scheme"] == 3)
    steps = case["decades"] * case["steps"]
    held = case["precision"] / 8.0
    one = {"bytes": 16.0 * 33 * n + held * entries * (factorizations + 2 * steps) + 8.0 * n * case["wires"] * 4 * steps,
           "flops": flops * factorizations + 4.0 * entries * case["wires"] * steps}
    return {k: v * case.get("requests", 1) for k, v in one.items()}


def _grid_counts(case, upper):
    sizes = (case["nx"], case["ny"], case["nz"])
    n, full = math.prod(sizes), math.prod(3 * m - 2 for m in sizes)
    return n, (full + n) // 2 if upper else full


def exact(case, seed):
    """A system's solution by diagonalising its tensor grid axis by axis, and the residual
    norms by torch, in 64 bits.  The transients and the initial field have none here: their
    oracle (element matrices, dipoles, receiver smoothing and a sparse direct solver) is a
    program of its own and takes minutes at most of these sizes."""
    if case["kind"] == "system":
        axes, shift = _grid_system(case, seed)
        lam, vec = [], []
        for k, m in axes:
            lower = np.linalg.cholesky(_dense(m))
            inv = np.linalg.inv(lower)
            w, q = np.linalg.eigh(inv @ _dense(k) @ inv.T)
            lam.append(w)
            vec.append(inv.T @ q)
        denom = lam[2][:, None, None] + lam[1][:, None] + lam[0] + shift
        vx, vy, vz = vec

        def solve(r):
            t = np.einsum("czyx,xi,yj,zk->ckji", r, vx, vy, vz, optimize=True) / denom
            return np.einsum("ckji,xi,yj,zk->czyx", t, vx, vy, vz, optimize=True)

        (kx, mx), (ky, my), (kz, mz) = [(_dense(k), _dense(m)) for k, m in axes]

        def apply(u):
            ux, uk = u @ mx, u @ (kx + shift * mx)
            p = np.einsum("jy,czyx->czjx", my, ux)
            q = np.einsum("jy,czyx->czjx", ky, ux) + np.einsum("jy,czyx->czjx", my, uk)
            return np.einsum("kz,czyx->ckyx", kz, p) + np.einsum("kz,czyx->ckyx", mz, q)

        b = _columns(case, seed).reshape(case["cols"], case["nz"], case["ny"], case["nx"])
        x = solve(b)
        for _ in range(2):
            x = x + solve(b - apply(x))
        return x.reshape(case["cols"], -1)
    if case["kind"] == "residual":
        s = prepare(case, seed)
        r = s["b"] - _product(*s["csr"], s["x"])
        return torch.stack([r.norm(dim=1), s["b"].norm(dim=1)], 1).reshape(-1)
    return None
