"""The work that users of this library have it do, as cases that can be timed.

A case is one call pattern of the public Python API (which is the C ABI) at one
size: time stepping of the drift-diffusion-Poisson system (a `Context`, driven by
`step`, by `run_to_steady_state` or by the four stage calls), a streamed warm-started
I-V sweep, the drop-in direct solver (`LU`), and the neural operator's inference and
training.  The sizes are the configurations' and the tests': single instances on
16x16 to 80x80 cells per region, groups of a few instances of one mesh, and the
64-slot batch.

Fields of FP64 and of refined (FP32 factors, FP64 residuals) runs are returned in 64
bits.  Mixed-precision runs carry the accuracy of FP32 solves in every increment;
their fields are returned as the 32-bit tensors that the operator's training and the
plots take.
"""
import math

import numpy as np
import torch

import pecs_gb300 as pg
from pecs_gb300 import learned

OPERATOR = "pecs_gb300/models/warmstart_ref6.npz"
PRECISION = {"fp64": pg.PREC_FP64, "ir": pg.PREC_FP32_IR, "mixed": pg.PREC_FP32_MIXED}


def listed():
    return [
        # One instance on a coarse mesh, driven stage by stage as a host time loop with
        # its own hooks between the stages does: the smallest calls, all latency.
        {"name": "stages-8x8", "kind": "run", "drive": "stages", "mesh": "half", "nx": 8, "nxe": 8, "ny": 8,
         "degree": 1, "pairing": 0, "grading": 1.0, "inst": 1, "precision": "fp64", "iters": 0, "steps": 4},
        # The p-n junction configuration: semiconductor only, 100 steps in one call.
        {"name": "pn-16x16", "kind": "run", "drive": "step", "mesh": "pn", "nx": 16, "nxe": 0, "ny": 16,
         "degree": 1, "pairing": 1, "grading": 1.0, "inst": 1, "precision": "fp64", "iters": 0, "steps": 100},
        # The half cell marched towards its steady state in FP64: the plain method.
        {"name": "half-64-fp64", "kind": "run", "drive": "march", "mesh": "half", "nx": 64, "nxe": 64, "ny": 64,
         "degree": 1, "pairing": 0, "grading": 1.0, "inst": 1, "precision": "fp64", "iters": 0, "steps": 20},
        # One mesh group of an uneven I-V sweep (a dozen points share a mesh), FP64, on a
        # ragged mesh graded towards the interface.
        {"name": "group-29x37-k2-fp64", "kind": "run", "drive": "march", "mesh": "half", "nx": 29, "nxe": 23,
         "ny": 37, "degree": 2, "pairing": 0, "grading": 4.0, "inst": 12, "precision": "fp64", "iters": 0,
         "steps": 6},
        # The same with FP32 factors and increment solves asked for, on a finer mesh.
        {"name": "group-64-k2-mixed", "kind": "run", "drive": "march", "mesh": "half", "nx": 64, "nxe": 64,
         "ny": 64, "degree": 2, "pairing": 0, "grading": 1.0, "inst": 8, "precision": "mixed", "iters": 0,
         "steps": 6},
        # Three biases on a large mesh, FP32 storage refined to FP64 accuracy, the
        # configurations' RT_k x DGQ_k Poisson element.
        {"name": "large-72-k2-ir", "kind": "run", "drive": "march", "mesh": "half", "nx": 72, "nxe": 72, "ny": 72,
         "degree": 2, "pairing": 1, "grading": 1.0, "inst": 3, "precision": "ir", "iters": 3, "steps": 4},
        # The throughput batch: 64 instances, FP32 factors, increment solves.
        {"name": "batch64-mixed", "kind": "run", "drive": "march", "mesh": "half", "nx": 64, "nxe": 64, "ny": 64,
         "degree": 1, "pairing": 0, "grading": 1.0, "inst": 64, "precision": "mixed", "iters": 0, "steps": 60},
        # The whole call: points predicted, probed and streamed through the slots (capped
        # after a few steps), final fields returned on the host.
        {"name": "warm-sweep", "kind": "sweep", "slots": 64, "points": 72, "steps": 20},
        # The direct solver as a host finite-element code calls it: one system, host arrays.
        {"name": "lu-host-16x16", "kind": "lu", "nx": 16, "ny": 16, "block": 4, "classes": True, "rhs": 1,
         "host": True},
        # ... and several right-hand sides that are on the GPU already.
        {"name": "lu-device-37x41", "kind": "lu", "nx": 37, "ny": 41, "block": 4, "classes": True, "rhs": 4,
         "host": False},
        # The operator's prediction for a sweep's points: network, decode, full vectors.
        {"name": "predict-256", "kind": "predict", "batch": 256},
        # One training batch of the operator: loss and gradients.
        {"name": "gradients-256", "kind": "gradients", "batch": 256, "hidden": 704, "layers": 3, "rank": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stages", "step", "march", "march", "march", "march", "sweep", "lu", "lu", "predict",
                       "gradients"])
    if kind in ("stages", "step", "march"):
        top = {"stages": 16, "step": 24, "march": 64}[kind]
        degree, pairing = rng.choice([1, 2]), rng.choice([0, 0, 1])
        nx, ny = _log_int(rng, 5, top), _log_int(rng, 5, top)
        mesh = rng.choice(["half", "half", "pn"])
        nxe = _log_int(rng, 5, top) if mesh == "half" else 0
        precision = rng.choice(["fp64", "fp64", "ir", "mixed"]) if kind == "march" else "fp64"
        # at most the largest listed case's unknowns over all instances
        room = 64 * 8192 * 4 // ((nx + nxe) * ny * (degree + 1) ** 2)
        inst = 1 if kind == "stages" else _log_int(rng, 1, max(1, min(64, room)))
        if precision == "fp64" and inst > 16:
            inst = 16 + inst % 32
        return {"kind": "run", "drive": kind, "mesh": mesh, "nx": nx, "nxe": nxe, "ny": ny, "degree": degree,
                "pairing": pairing, "grading": rng.choice([1.0, 1.0, 3.0]), "inst": inst,
                "precision": precision, "iters": 3 if precision == "ir" else 0,
                "steps": {"stages": rng.randint(1, 5), "step": rng.randint(5, 60),
                          "march": rng.randint(2, 11)}[kind]}
    if kind == "sweep":
        slots = rng.randint(33, 64)
        return {"kind": "sweep", "slots": slots, "points": slots + rng.randint(1, 16), "steps": rng.randint(6, 20)}
    if kind == "lu":
        block = rng.choice([1, 4, 4, 9])
        top = {1: 64, 4: 40, 9: 26}[block]
        return {"kind": "lu", "nx": _log_int(rng, 3, top), "ny": _log_int(rng, 3, top), "block": block,
                "classes": rng.random() < 0.7, "rhs": _log_int(rng, 1, 12), "host": rng.random() < 0.5}
    if kind == "predict":
        return {"kind": "predict", "batch": _log_int(rng, 1, 512)}
    return {"kind": "gradients", "batch": _log_int(rng, 16, 512), "hidden": _log_int(rng, 64, 704),
            "layers": rng.randint(1, 3), "rank": _log_int(rng, 16, 64)}


# -- time stepping -------------------------------------------------------------------


def _points(case, seed):
    """Parameters of the case's instances: drawn bias, generation, doping, lifetime and rate."""
    if case["mesh"] == "pn":
        rng = np.random.default_rng(seed)
        base = pg.pn_junction(nx_semi=case["nx"], ny=case["ny"], degree=case["degree"],
                              poisson_pairing=case["pairing"])
        return [base.copy(phi_app=float(rng.uniform(-0.5, 0.5)), tau_n=t, tau_p=t)
                for t in np.exp(rng.uniform(math.log(0.1), math.log(10.0), case["inst"])).tolist()]
    base = pg.half_cell(nx_semi=case["nx"], nx_elec=case["nxe"], ny=case["ny"], degree=case["degree"],
                        poisson_pairing=case["pairing"], grading=case["grading"])
    return [learned.instance_params(t, base) for t in learned.sample(case["inst"], seed)]


def _prepare_run(case, seed):
    ctx = pg.Context(_points(case, seed), precision=PRECISION[case["precision"]], ir_max_iters=case["iters"],
                     increment_solves=case["precision"] == "mixed")
    fields = {f: torch.zeros(case["inst"], ctx.ndofs[f], dtype=torch.float64, device="cuda") for f in ctx.fields()}
    return {"case": case, "ctx": ctx, "fields": fields}


def _run_run(s):
    case, ctx = s["case"], s["ctx"]
    out = {}
    ctx.initialize()
    if case["drive"] == "step":
        ctx.step(case["steps"])
    elif case["drive"] == "march":
        steps, rel = ctx.run_to_steady_state(case["steps"], 1e-8, 50)
        out["steps"], out["rel"] = steps, rel
    else:
        for _ in range(case["steps"]):
            ctx.assemble_carrier_rhs()
            ctx.solve_carriers()
            ctx.assemble_poisson_rhs()
            ctx.solve_poisson()
    for f, t in s["fields"].items():
        for i in range(case["inst"]):
            ctx.get_state_device(f, i, t[i].data_ptr())
        out["field%d" % f] = t
    out["current"] = ctx.interface_current()
    if case["precision"] == "mixed":
        out = {k: v.float() if isinstance(v, torch.Tensor) else v if v.dtype.kind == "i" else v.astype(np.float32)
               for k, v in out.items()}
    return out


def _work_run(case):
    """One pass: every step needs each stored factor entry once, the right-hand-side data
    and the states.  A nested-dissection factor of N cells with b unknowns each has about
    12 b^2 N log2 N entries (carriers; the mixed Poisson system about a third of that)."""
    b = (case["degree"] + 1) ** 2
    kp = case["degree"] + case["pairing"]
    cells = [c * case["ny"] for c in (case["nx"], case["nxe"]) if c]
    carrier = sum(12.0 * b * b * n * math.log2(max(2, n)) for n in cells)
    n = sum(cells)
    poisson = 4.3 * (3 * kp * kp) ** 2 * n * math.log2(max(2, n))
    size = 8 if case["precision"] == "fp64" else 4
    state = case["inst"] * n * (2 * 3 * b + 3 * kp * kp)
    steps = case["steps"]
    return {"bytes": steps * ((carrier + poisson) * size + 24.0 * state),
            "flops": steps * 2.0 * case["inst"] * (2 * carrier + poisson)}


# -- the streamed sweep --------------------------------------------------------------


def _prepare_sweep(case, seed):
    base = pg.half_cell(6)
    thetas = learned.sample(case["points"], seed)
    ctx = pg.Context([learned.instance_params(thetas[i % case["points"]], base) for i in range(case["slots"])],
                     precision=pg.PREC_FP32_MIXED, increment_solves=True)
    return {"case": case, "ctx": ctx, "op": learned.NeuralOperator.load(OPERATOR), "base": base, "thetas": thetas}


def _run_sweep(s):
    steps, fallback, current, fields = learned.stream_warm_sweep(
        s["ctx"], s["op"], s["thetas"], s["base"], max_steps=s["case"]["steps"], tol=1e-8, check_every=10,
        want_fields=True)
    out = {"field%d" % f: a.astype(np.float32) for f, a in fields.items()}
    out.update(steps=steps, fallback=fallback.astype(np.int64), current=current.astype(np.float32))
    return out


def _work_sweep(case):
    one = {"degree": 1, "pairing": 0, "nx": 64, "nxe": 64, "ny": 64, "precision": "mixed", "inst": case["slots"],
           "steps": case["steps"] * -(-case["points"] // case["slots"])}
    return _work_run(one)


# -- the direct solver ---------------------------------------------------------------


def _ldg_matrix(case, seed):
    """A matrix with the structure of an LDG carrier system on an nx x ny grid: per cell two
    blocks of currents (block-diagonal mass matrix) and one of densities, currents and
    densities coupled within the cell and across its faces, one block after another in the
    vector.  Returns (n, rows, columns, values) and each unknown's cell and class."""
    rng = np.random.default_rng(seed)
    nx, ny, b = case["nx"], case["ny"], case["block"]
    nc = nx * ny
    cell = np.arange(nc)
    i, j = cell % nx, cell // nx
    pairs = {0: (cell, cell)}
    for d, (ok, step) in enumerate([(i > 0, -1), (i < nx - 1, 1), (j > 0, -nx), (j < ny - 1, nx)], 1):
        pairs[d] = (cell[ok], cell[ok] + step)
    rows, cols, vals = [], [], []

    def add(br, bc, at, block):
        r = br * nc * b + at[0][:, None, None] * b + np.arange(b)[:, None]
        c = bc * nc * b + at[1][:, None, None] * b + np.arange(b)[None, :]
        rows.append(np.broadcast_to(r, block.shape).ravel())
        cols.append(np.broadcast_to(c, block.shape).ravel())
        vals.append(block.ravel())

    def some(at, scale):
        return scale / math.sqrt(b) * rng.uniform(-1, 1, (at[0].size, b, b))

    for comp in (0, 1):
        add(comp, comp, pairs[0], np.eye(b) + some(pairs[0], 0.2))
        for d in (0, 1 + 2 * comp, 2 + 2 * comp):
            add(comp, 2, pairs[d], some(pairs[d], 1.0))
            add(2, comp, pairs[d], some(pairs[d], 1.0))
    for d in range(5):
        block = some(pairs[d], 0.5)
        if d == 0:
            block += 8.0 * np.eye(b)
        add(2, 2, pairs[d], block)
    dof_cell = np.tile(np.repeat(cell, b), 3)
    dof_class = np.repeat([0, 0, 1], nc * b)
    return 3 * nc * b, np.concatenate(rows), np.concatenate(cols), np.concatenate(vals), dof_cell, dof_class


def _lu_rhs(case, n, seed):
    return np.random.default_rng(seed + 1).standard_normal((case["rhs"], n))


def _prepare_lu(case, seed):
    n, rows, cols, vals, dof_cell, dof_class = _ldg_matrix(case, seed)
    order = np.lexsort((cols, rows))
    indptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    nx, ny = case["nx"], case["ny"]
    xy = np.stack([np.tile(np.arange(nx) + 0.5, ny), np.repeat(np.arange(ny) + 0.5, nx)], axis=1)
    lu = pg.LU((vals[order], cols[order], indptr), dof_cell, xy, dof_class=dof_class if case["classes"] else None)
    b = _lu_rhs(case, n, seed)
    if case["host"]:
        return {"case": case, "lu": lu, "b": b if case["rhs"] > 1 else b[0]}
    b = torch.from_numpy(b).cuda()
    return {"case": case, "lu": lu, "b": b, "x": torch.zeros_like(b)}


def _run_lu(s):
    if s["case"]["host"]:
        return s["lu"].solve(s["b"])
    s["lu"].solve_device(s["b"].data_ptr(), s["x"].data_ptr(), nrhs=s["case"]["rhs"])
    return s["x"]


def _exact_lu(case, seed):
    n, rows, cols, vals, _, _ = _ldg_matrix(case, seed)
    if n > 20000:
        return None
    a = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    a[torch.from_numpy(rows).cuda(), torch.from_numpy(cols).cuda()] = torch.from_numpy(vals).cuda()
    x = torch.linalg.solve(a, torch.from_numpy(_lu_rhs(case, n, seed)).cuda().T).T.contiguous()
    return x[0] if case["host"] and case["rhs"] == 1 else x


def _work_lu(case):
    n = case["nx"] * case["ny"]
    entries = 12.0 * case["block"] ** 2 * n * math.log2(max(2, n))
    return {"bytes": 8.0 * entries + 16.0 * case["rhs"] * 3 * n * case["block"],
            "flops": 2.0 * case["rhs"] * entries}


# -- the neural operator -------------------------------------------------------------


def _prepare_predict(case, seed):
    op = learned.NeuralOperator.load(OPERATOR)
    n_u, n_phi = 64 * 64 * 4, 2 * 64 * 64
    lay = learned.Layout(3 * n_u, n_u, 2 * n_u, 24768, n_phi, 24768 - n_phi)
    x = torch.from_numpy(learned.normalize(learned.sample(case["batch"], seed))).cuda()
    return {"op": op, "lay": lay, "x": x}


def _run_predict(s):
    return s["op"].predict_vectors(s["x"], s["lay"])


def _exact_predict(case, seed):
    d = np.load(OPERATOR)
    cuda = lambda v: torch.from_numpy(np.asarray(v, dtype=np.float64)).cuda()  # noqa: E731
    widths, params, at = [int(w) for w in d["widths"]], cuda(d["params"]), 0
    y = cuda(learned.normalize(learned.sample(case["batch"], seed)))
    for k, (m, n) in enumerate(zip(widths[:-1], widths[1:])):
        y = y @ params[at:at + m * n].reshape(n, m).T + params[at + m * n:at + m * n + n]
        at += m * n + n
        y = torch.tanh(y) if k < len(widths) - 2 else y
    n_u = 64 * 64 * 4
    top = slice(0, 2 * n_u)
    logs = cuda(d["mean"])[top] + cuda(d["scale"])[top] * ((y * cuda(d["cscale"])) @ cuda(d["basis"])[top].T)
    out = torch.zeros(2, case["batch"], 3 * n_u, dtype=torch.float64, device="cuda")
    out[0, :, 2 * n_u:], out[1, :, 2 * n_u:] = logs[:, :n_u].exp(), logs[:, n_u:].exp()
    return out[0], out[1]


def _work_predict(case):
    n_u, weights = 64 * 64 * 4, 6 * 704 + 2 * 704 * 704 + 704 * 64
    return {"bytes": 2.0 * weights + 4.0 * 2 * n_u * 65 + 8.0 * case["batch"] * 2 * 3 * n_u,
            "flops": 2.0 * case["batch"] * (weights + 2 * n_u * 64)}


def _network(case, seed):
    """Widths, packed parameters and one batch (inputs in [-1, 1], targets of unit size)."""
    rng = np.random.default_rng(seed)
    widths = [6] + [case["hidden"]] * case["layers"] + [case["rank"]]
    params = []
    for m, n in zip(widths[:-1], widths[1:]):
        params += [rng.uniform(-1, 1, m * n) * math.sqrt(3.0 / m), 0.1 * rng.standard_normal(n)]
    x, t = rng.uniform(-1, 1, (case["batch"], 6)), rng.standard_normal((case["batch"], case["rank"]))
    return widths, np.concatenate(params).astype(np.float32), x.astype(np.float32), t.astype(np.float32)


def _prepare_gradients(case, seed):
    widths, params, x, t = _network(case, seed)
    mlp = learned.Mlp(widths)
    mlp.set_params(params)
    return {"mlp": mlp, "x": torch.from_numpy(x).cuda(), "t": torch.from_numpy(t).cuda(), "batch": case["batch"]}


def _run_gradients(s):
    grad, loss = s["mlp"].gradients(s["x"].data_ptr(), s["t"].data_ptr(), s["batch"])
    return {"grad": grad, "loss": np.float32(loss)}


def _exact_gradients(case, seed):
    widths, params, x, t = _network(case, seed)
    p = torch.from_numpy(params).double().cuda().requires_grad_()
    y, at = torch.from_numpy(x).double().cuda(), 0
    for k, (m, n) in enumerate(zip(widths[:-1], widths[1:])):
        y = y @ p[at:at + m * n].reshape(n, m).T + p[at + m * n:at + m * n + n]
        at += m * n + n
        y = torch.tanh(y) if k < len(widths) - 2 else y
    loss = ((y - torch.from_numpy(t).double().cuda()) ** 2).mean()
    loss.backward()
    return {"grad": p.grad, "loss": np.float64(loss.item())}


def _work_gradients(case):
    weights = 6 * case["hidden"] + (case["layers"] - 1) * case["hidden"] ** 2 + case["hidden"] * case["rank"]
    return {"bytes": 2.0 * weights + 4.0 * weights + 4.0 * case["batch"] * (6 + case["rank"]),
            "flops": 6.0 * case["batch"] * weights}


# -- the five functions --------------------------------------------------------------


def prepare(case, seed):
    return {"run": _prepare_run, "sweep": _prepare_sweep, "lu": _prepare_lu, "predict": _prepare_predict,
            "gradients": _prepare_gradients}[case["kind"]](case, seed) | {"kind": case["kind"]}


def run(state):
    return {"run": _run_run, "sweep": _run_sweep, "lu": _run_lu, "predict": _run_predict,
            "gradients": _run_gradients}[state["kind"]](state)


def work(case):
    return {"run": _work_run, "sweep": _work_sweep, "lu": _work_lu, "predict": _work_predict,
            "gradients": _work_gradients}[case["kind"]](case)


def exact(case, seed):
    """None for the time-stepping cases: their 64-bit values need the whole discretisation
    restated and its systems solved densely, minutes and tens of GB at most of the sizes."""
    e = {"lu": _exact_lu, "predict": _exact_predict, "gradients": _exact_gradients}.get(case["kind"])
    return e(case, seed) if e else None
