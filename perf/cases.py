"""The work this framework is run for, as measurable cases.

A case is one call a user's program repeats: a time step of a shell (hydro or
MHD, each in the sizes and with the options the runs of this repository use),
a step of an ensemble of shells, the derivative operators on PyTorch tensors
with their gradients, the refresh of a learned closure and a training step of
its network.  ``listed`` are the cases, ``draw`` gives more of the same
ranges, ``prepare`` builds what a program holds before the call, ``run`` is
one pass through the public entry points and ``work`` the bytes and
operations no implementation of the pass can do without.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "css-code_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from css_b200 import closure, ensemble, problem, torch_ops  # noqa: E402
from css_b200.context import Simulation  # noqa: E402
from css_b200.params import NPROF, PROF_NAMES, default_params  # noqa: E402

MAX_CELLS = 256 * 512 * 1024  # the largest shell of this repository's workloads
OPEN_STEPS = 4  # steps from a restart with open faces


def _step(name, dims, blocks, magnetic, precision=0, physics="closed", stepper=4):
    return {"name": name, "kind": "step", "nr": dims[0], "nth": dims[1], "nphi": dims[2], "nnr": blocks[0],
            "nnt": blocks[1], "nnp": blocks[2], "magnetic": magnetic, "precision": precision, "physics": physics,
            "stepper": stepper}


def listed():
    return [
        # the smallest shell of the workloads (smoke run, first convection
        # tests): a step of a fraction of a millisecond, launches count
        _step("hydro-64x64x128", (64, 64, 128), (2, 2, 4), False),
        # the ordinary hydro convection run
        _step("hydro-128x256x512", (128, 256, 512), (4, 8, 16), False),
        # an ordinary dynamo run
        _step("mhd-128x128x256", (128, 128, 256), (4, 4, 8), True),
        # the production dynamo run, the framework's headline configuration
        _step("mhd-256x512x1024", (256, 512, 1024), (8, 16, 32), True),
        # the mixed-precision form of the dynamo run (FP32 stage states)
        _step("mhd-mixed-128x128x256", (128, 128, 256), (4, 4, 8), True, precision=1),
        # a shell of the parameter study on its own: sizes that no 32-point
        # block divides (5 x 11 x 19 blocks of 20, 16 and 16 points)
        _step("hydro-ragged-100x176x304", (100, 176, 304), (5, 11, 19), False),
        # both radial faces open, entropy rain through the top: a few steps
        # from a restart state (opened faces are stepped on from a closed run)
        _step("hydro-open-64x128x256", (64, 128, 256), (2, 4, 8), False, physics="open"),
        # explicit viscosity and resistivity in a dynamo run (a direct
        # simulation at the resolution it is affordable at)
        _step("mhd-viscous-64x128x256", (64, 128, 256), (2, 4, 8), True, physics="viscous"),
        # a parameter study: eight uneven shells, half of them MHD, stepped
        # together in the mixed form
        {"name": "ensemble-8", "kind": "ensemble", "members": 8, "study_seed": 7, "precision": 1},
        # the three first derivatives of a scalar field and their gradients,
        # as a loss on derivatives of a field uses them
        {"name": "deriv-128x256x512", "kind": "deriv", "nr": 128, "nth": 256, "nphi": 512, "nnr": 4, "nnt": 8,
         "nnp": 16, "order": 1, "fields": 1, "dtype": "float64"},
        # the learned closure's refresh on the coarse grid of the MHD study:
        # features of every cell, the network, the speed^2 it gives
        {"name": "closure-64x128x256", "kind": "closure", "nr": 64, "nth": 128, "nphi": 256},
        # one Adam step of the closure network on the study's batch
        {"name": "train-16384", "kind": "train", "rows": 16384},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _blocks(n, least):
    """Blocks of even size in [10, 256], near 32 points, dividing n evenly."""
    best = None
    for nb in range(least, n // 10 + 1):
        m = n // nb
        if n % nb == 0 and m % 2 == 0 and 10 <= m <= 256 and nb <= 64:
            key = (0 if m in (16, 32) else 1, abs(m - 32))
            if best is None or key < best[0]:
                best = (key, nb)
    return best[1] if best else None


def _draw_dims(rng, cells_hi, least=(2, 2, 3), ragged=False):
    while True:
        if ragged:  # the parameter study's ranges
            nr, nth, nphi = 4 * rng.randint(12, 40), 16 * rng.randint(4, 16), 16 * rng.randint(8, 32)
        else:
            nr, nth, nphi = (32 * _log_int(rng, 2, 8), 32 * _log_int(rng, 2, 16), 32 * _log_int(rng, 3, 32))
        if nr * nth * nphi > cells_hi:
            continue
        nb = [_blocks(n, lo) for n, lo in zip((nr, nth, nphi), least)]
        if all(nb):
            return (nr, nth, nphi), nb


def draw(rng):
    kind = rng.choice(["hydro", "mhd", "ragged", "mixed", "physics", "ensemble", "deriv", "closure", "train"])
    if kind == "ensemble":
        return {"kind": "ensemble", "members": rng.randint(2, 12), "study_seed": rng.randint(0, 9999),
                "precision": rng.choice([0, 1, 1])}
    if kind == "deriv":
        (nr, nth, nphi), nb = _draw_dims(rng, 128 * 256 * 512, ragged=rng.random() < 0.5)
        return {"kind": "deriv", "nr": nr, "nth": nth, "nphi": nphi, "nnr": nb[0], "nnt": nb[1], "nnp": nb[2],
                "order": rng.choice([1, 1, 2]), "fields": rng.choice([1, 1, 3]),
                "dtype": rng.choice(["float64", "float64", "float32"])}
    if kind == "closure":
        return {"kind": "closure", "nr": 8 * rng.randint(3, 8), "nth": 8 * rng.randint(4, 16),
                "nphi": 16 * rng.randint(4, 16)}
    if kind == "train":
        return {"kind": "train", "rows": _log_int(rng, 500, 65536)}
    physics, precision, stepper = "closed", 0, 4
    if kind == "physics":
        physics = rng.choice(["open", "viscous", "radheat", "closed"])
        stepper = rng.choice([2, 3, 4]) if physics == "closed" else 4
    if kind == "mixed":
        precision = 1
    magnetic = kind == "mhd" or (kind != "hydro" and physics != "open" and rng.random() < 0.5)
    top = {"hydro": MAX_CELLS // 2, "mhd": MAX_CELLS // 2}.get(kind, 128 * 256 * 256)
    dims, nb = _draw_dims(rng, top, ragged=kind in ("ragged",) or (kind in ("physics", "mixed") and rng.random() < 0.3))
    c = _step("", dims, nb, magnetic, precision, physics, stepper)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
class _Resident:
    """The device state of a run as a tensor's memory (keeps the run alive)."""

    def __init__(self, sim):
        ptr, n = sim.device_state()
        self.sim = sim
        self.__cuda_array_interface__ = {"shape": sim.shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


def _resident(sim):
    return torch.as_tensor(_Resident(sim), device="cuda")


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)


def _fill(p, prof, info, gen, out):
    """The seeded state of problem.initial_state with convective motions, made
    on the device field by field into out (nv, nr, nphi, nth)."""
    dev = out.device
    bg = problem.background(_one_phi(p), prof, info)[:, :, 0, :]  # (nv, nr, nth)
    theta, phi, _, dphi = problem.angles(p)
    r = prof.reshape(NPROF, p.nr)[PROF_NAMES.index("r_ind")]
    yv = math.pi * (r - p.r1) / (p.r2 - p.r1)
    xv = math.pi * (theta - p.th1) / (p.th2 - p.th1)
    rt = np.ones_like(r) if (p.top_inout and p.bot_inout) else 1.0 - np.cos(yv) ** 16
    taper = torch.as_tensor(rt[:, None, None] * (1.0 - np.cos(xv)[None, None, :] ** 16), device=dev)
    # a few convection cells around the shell under the noise
    cells = torch.as_tensor(np.sin(yv)[:, None, None] * np.cos(8.0 * phi)[None, :, None] * np.sin(3.0 * xv)[None, None, :],
                            device=dev)
    shape = tuple(out.shape[1:])
    for iv in range(out.shape[0]):
        f = out[iv]
        if iv >= 5:  # random vector potential, rms field about 1e-3 of equipartition
            f.copy_(torch.rand(shape, generator=gen, device=dev, dtype=torch.float64))
            t2 = (1.0 - np.cos(yv)[:, None, None] ** 2) * (1.0 - np.cos(xv)[None, None, :] ** 2)
            f.mul_(2.0).sub_(1.0).mul_(torch.as_tensor(t2, device=dev) * (0.01 * (p.r2 - p.r1) / p.nr))
            continue
        f.copy_(torch.randn(shape, generator=gen, device=dev, dtype=torch.float64))
        f.mul_(taper)
        base = torch.as_tensor(bg[iv], device=dev)[:, None, :]
        if iv == 0:
            f.mul_(1e-5).add_(1.0).mul_(base)
        elif iv == 4:
            f.add_(cells).mul_(1e-4).add_(1.0).mul_(base)
        else:
            f.mul_(0.1).add_(cells).mul_(1e-3)
            if iv in (1, 3):  # no flow through the walls
                f[:, :, 0] = 0.0
                f[:, :, -1] = 0.0
            if iv == 3 and not p.top_inout:
                f[-1] = 0.0
            if iv == 3 and not p.bot_inout:
                f[0] = 0.0


def _one_phi(p):
    q = p.copy()
    q.nphi = 1
    return q


def _simulation(p, n_rho, ra, seed):
    prof, info = problem.polytrope(p, n_rho, ra=ra)
    sim = Simulation(p, prof)
    gen = _gen(seed)
    if p.precision:  # the backgrounds of the FP32 stage states come with an upload
        v = torch.empty(sim.shape, dtype=torch.float64, device="cuda")
        _fill(p, prof, info, gen, v)
        sim.upload(v.cpu().numpy())
    else:
        _fill(p, prof, info, gen, _resident(sim))
        torch.cuda.synchronize()
    dt = sim.step_size(0.3)["dtmax"]  # Courant 0.3: room for the motions to grow
    return sim, dt


def _prepare_step(c, seed):
    p = default_params(c["nr"], c["nth"], c["nphi"], (c["nnr"], c["nnt"], c["nnp"]), magnetic=c["magnetic"])
    p.precision = c["precision"]
    p.time_stepper = c["stepper"]
    if c["magnetic"]:
        p.sld_prm = 0.5
    if c["physics"] == "viscous":
        p.laplacian = 1
    elif c["physics"] == "radheat":
        p.do_radheat = 1
    elif c["physics"] == "open":
        p.top_inout = p.bot_inout = p.do_entropy_rain = 1
        p.delta_s = 1e-4
    sim, dt = _simulation(p, 5.0 if c["magnetic"] else 3.0, 1e6 if c["magnetic"] else 1e5, seed)
    if c["physics"] == "open":
        sim.inout_init()
        rng = np.random.default_rng(seed)
        sq = np.stack([rng.uniform(p.th1, p.th2, 24), rng.uniform(p.phi1, p.phi2, 24), rng.uniform(0.02, 0.08, 24),
                       np.ones(24), rng.uniform(-2e-3, -1e-3, 24), rng.uniform(-2e-4, -1e-4, 24)], axis=1)
        sim.set_clock(0, 0.0, dt)
        sim.build_squalls(sq)
    s = {"sim": sim, "dt": dt, "out": _resident(sim)}
    if c["physics"] == "open":
        s["restart"] = s["out"].clone()
        s["stream"] = torch.cuda.Stream()
        torch.cuda.synchronize()
        sim.set_stream(s["stream"].cuda_stream)
    return s


def _prepare_ensemble(c, seed):
    sims, dts = [], []
    for i, s in enumerate(ensemble.shell_specs(c["members"], seed=c["study_seed"])):
        p = default_params(s["nr"], s["nth"], s["nphi"], s["decomp"], magnetic=s["magnetic"])
        p.omega_0 = 0.5 / s["ro"]
        p.precision = c["precision"]
        if s["magnetic"]:
            p.sld_prm = 1.0 / s["pm"]
        sim, dt = _simulation(p, 3.0, s["ra"], seed * 100 + i)
        sims.append(sim)
        dts.append(dt)
    return {"sims": sims, "ens": ensemble.Ensemble(sims), "dts": np.array(dts), "out": [_resident(s) for s in sims]}


def _deriv_inputs(c, seed):
    gen = _gen(seed)
    shape = ((c["fields"],) if c["fields"] > 1 else ()) + (c["nr"], c["nphi"], c["nth"])
    dtype = getattr(torch, c["dtype"])
    v = [torch.randn(shape, generator=gen, device="cuda", dtype=dtype) for _ in range(4)]
    return v[0], v[1:]


def _prepare_deriv(c, seed):
    p = default_params(c["nr"], c["nth"], c["nphi"], (c["nnr"], c["nnt"], c["nnp"]))
    prof, _ = problem.polytrope(p, 3.0, ra=1e5)
    x, g = _deriv_inputs(c, seed)
    # PyTorch's work runs on a stream of its own, as in a training loop
    return {"sim": Simulation(p, prof), "x": x.requires_grad_(True), "g": g, "order": c["order"],
            "stream": torch.cuda.Stream()}


def _weights(rng):
    dims = (144, 128, 128, 128, 16)
    real = (135, 128, 128, 128, 12)
    out = []
    for k in range(4):
        w = np.zeros((dims[k], dims[k + 1]), dtype=np.float32)
        a = math.sqrt(6.0 / (real[k] + real[k + 1]))
        w[:real[k], :real[k + 1]] = rng.uniform(-a, a, (real[k], real[k + 1]))
        b = np.zeros(dims[k + 1], dtype=np.float32)
        b[:real[k + 1]] = rng.uniform(-0.1, 0.1, real[k + 1])
        out.append((w, b))
    return out


def _closure_inputs(c, seed):
    dims = (c["nth"], c["nphi"], c["nr"])
    gen = _gen(seed)
    f = torch.randn((7, c["nr"], c["nphi"], c["nth"]), generator=gen, device="cuda", dtype=torch.float64)
    amp = torch.tensor([1e-2, 1e-2, 1e-2, 1e-3, 5e-2, 5e-2, 5e-2], dtype=torch.float64, device="cuda")
    f *= amp[:, None, None, None]
    rng = np.random.default_rng(seed)
    qscale = np.array([1e-2, 1e-2, 1e-2, 8e-2, 7e-4], dtype=np.float32)
    tscale = rng.uniform(0.5, 2.0, 12).astype(np.float32) * np.float32(1e-4)
    return dims, f, qscale, tscale, _weights(rng)


def _prepare_closure(c, seed):
    dims, f, qscale, tscale, wb = _closure_inputs(c, seed)
    clo = closure.Closure(seed=0)
    for k, (w, b) in enumerate(wb):
        clo.net.set_params(k, w, b)
    clo.qscale, clo.tscale = qscale, tscale
    return {"clo": clo, "dims": dims, "fields": f.reshape(-1)}


def _train_inputs(c, seed):
    gen = _gen(seed)
    n = c["rows"]
    x = torch.zeros(n, closure.XPAD, dtype=torch.bfloat16, device="cuda")
    x[:, :135] = torch.randn((n, 135), generator=gen, device="cuda").to(torch.bfloat16)
    t = torch.zeros(n, closure.YPAD, dtype=torch.float32, device="cuda")
    t[:, :12] = torch.randn((n, 12), generator=gen, device="cuda")
    return x, t, _weights(np.random.default_rng(seed))


def _prepare_train(c, seed):
    x, t, wb = _train_inputs(c, seed)
    net = closure.Mlp(max_rows=65536)
    for k, (w, b) in enumerate(wb):
        net.set_params(k, w, b)
    return {"net": net, "x": x, "t": t, "rows": c["rows"]}


def prepare(case, seed):
    make = {"step": _prepare_step, "ensemble": _prepare_ensemble, "deriv": _prepare_deriv,
            "closure": _prepare_closure, "train": _prepare_train}[case["kind"]]
    return {"kind": case["kind"], **make(case, seed)}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "step" and "restart" in s:
        with torch.cuda.stream(s["stream"]):
            s["out"].copy_(s["restart"])
        s["sim"].set_clock(0, 0.0, s["dt"])
        s["sim"].step_rk4(s["dt"], OPEN_STEPS)
        return s["out"]
    if kind == "step":
        s["sim"].step_rk4(s["dt"], 1)
        return s["out"]
    if kind == "ensemble":
        s["ens"].step(s["dts"], 1)
        return s["out"]
    if kind == "deriv":
        ops = ((torch_ops.dbydr, torch_ops.dbydt, torch_ops.dbydp) if s["order"] == 1 else
               (torch_ops.d2bydr2, torch_ops.d2bydt2, torch_ops.d2bydp2))
        with torch.cuda.stream(s["stream"]):
            ys = [f(s["x"], s["sim"]) for f in ops]
            gx, = torch.autograd.grad(ys, s["x"], s["g"])
        return {"dr": ys[0].detach(), "dt": ys[1].detach(), "dp": ys[2].detach(), "gx": gx}
    if kind == "closure":
        d = closure.build_inputs(s["fields"], s["dims"], s["clo"].qscale)
        return {"features": d["x"], "speed2": s["clo"].speed2(d)}
    loss = s["net"].train_step(s["x"], s["t"], s["rows"], 1e-3)
    return {"loss": loss, "grads": [s["net"].grads(k) for k in range(4)]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
_MACS = 144 * 128 + 2 * 128 * 128 + 128 * 16
# FP64 operations of a cell in one step, counted from the equations: per
# stage about 10 for each line solve (13 and 18 lines of an RHS, 4 more for
# B = curl A) and the pointwise terms, and once the slope-limited diffusion
_STAGE_FLOPS = {5: 18 * 10 + 170, 8: 24 * 10 + 6 * 10 + 280}


def _step_work(cells, nv, stages=4):
    # the state in, the state out; what goes on between is one program's
    # choice
    return {"bytes": 16.0 * nv * cells, "flops": cells * (stages * _STAGE_FLOPS[nv] + 75.0 * nv)}


def work(c):
    if c["kind"] == "step":
        w = _step_work(c["nr"] * c["nth"] * c["nphi"], 8 if c["magnetic"] else 5, c["stepper"])
        return {k: v * OPEN_STEPS for k, v in w.items()} if c["physics"] == "open" else w
    if c["kind"] == "ensemble":
        ws = [_step_work(ensemble.cells(s), 8 if s["magnetic"] else 5)
              for s in ensemble.shell_specs(c["members"], seed=c["study_seed"])]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    if c["kind"] == "deriv":
        n = c["nr"] * c["nth"] * c["nphi"] * c["fields"]
        size = 8 if c["dtype"] == "float64" else 4
        # x and the three incoming gradients read, three outputs and the
        # gradient written; three solves and three adjoint solves
        return {"bytes": 8.0 * size * n, "flops": 60.0 * n}
    if c["kind"] == "closure":
        n = c["nr"] * c["nth"] * c["nphi"]
        return {"bytes": n * (7 * 8 + 144 * 2 + 8.0), "flops": 2.0 * _MACS * n}
    n = c["rows"]
    return {"bytes": n * (144 * 2 + 16 * 4.0) + 6 * 4.0 * _MACS, "flops": 2.0 * n * (3 * _MACS - 144 * 128)}


# ---------------------------------------------------------------------------
# the outputs in 64 bits without this framework
# ---------------------------------------------------------------------------
def _d1_block(m, lo_wall, hi_wall):
    """A y = B x of one block's compact first derivative (unit spacing), B over
    the block's points and four halo points on either side."""
    A, B = np.eye(m), np.zeros((m, m + 8))
    for j in range(m):
        if j > 0:
            A[j, j - 1] = 1.0 / 3.0
        if j < m - 1:
            A[j, j + 1] = 1.0 / 3.0
        B[j, [j + 3, j + 5]] = -7.0 / 9.0, 7.0 / 9.0
        B[j, [j + 2, j + 6]] = -1.0 / 36.0, 1.0 / 36.0
    ex = np.array([-1.0, 9.0, -45.0, 0.0, 45.0, -9.0, 1.0]) / 60.0  # explicit value at the halo point
    for wall, row, sgn, halo in ((lo_wall, 0, 1, 3), (hi_wall, m - 1, -1, m + 4)):
        if not wall:
            B[row, halo - 3:halo + 4] -= ex / 3.0
            continue
        A[row] = 0.0
        B[row] = 0.0
        at = [row + 4 + sgn * k for k in range(5)]
        A[row, [row, row + sgn, row + 2 * sgn]] = 1.0, 6.0, 3.0
        B[row, at[:4]] = sgn * np.array([-10.0 / 3.0, -3.0, 6.0, 1.0 / 3.0])
        r2 = row + sgn
        A[r2, [row, r2, r2 + sgn]] = 0.125, 1.0, 0.75
        B[r2] = 0.0
        B[r2, at] = sgn * np.array([-43.0 / 96.0, -5.0 / 6.0, 9.0 / 8.0, 1.0 / 6.0, -1.0 / 96.0])
    return np.linalg.solve(A, B)


def _d2_block(m, lo_wall, hi_wall):
    A, B = np.eye(m), np.zeros((m, m + 8))
    for j in range(m):
        if j > 0:
            A[j, j - 1] = 2.0 / 11.0
        if j < m - 1:
            A[j, j + 1] = 2.0 / 11.0
        B[j, j + 2:j + 7] += np.array([3.0 / 44.0, 12.0 / 11.0, -2.0 * (3.0 / 44.0 + 12.0 / 11.0), 12.0 / 11.0,
                                       3.0 / 44.0])
    ex = np.array([2.0, -27.0, 270.0, -490.0, 270.0, -27.0, 2.0]) / 180.0
    for wall, row, sgn, halo in ((lo_wall, 0, 1, 3), (hi_wall, m - 1, -1, m + 4)):
        if not wall:
            B[row, halo - 3:halo + 4] -= ex * 2.0 / 11.0
            continue
        A[row] = 0.0
        B[row] = 0.0
        at = [row + 4 + sgn * k for k in range(6)]
        A[row, [row, row + sgn]] = 1.0, 137.0 / 13.0
        B[row, at] = [1955.0 / 156.0, -4057.0 / 156.0, 1117.0 / 78.0, -55.0 / 78.0, -29.0 / 156.0, 7.0 / 156.0]
        r2 = row + sgn
        A[r2] = 0.0
        A[r2, [row, r2, r2 + sgn]] = 0.1, 1.0, -0.35
        B[r2] = 0.0
        B[r2, at[:5]] = [1.2375, -3.0, 2.325, -0.6, 0.0375]
    return np.linalg.solve(A, B)


def _deriv_exact(x, axis, order, coords, nb, periodic):
    """Block-closed compact derivative of x along axis."""
    n = x.shape[axis]
    m = n // nb
    v = x.movedim(axis, -1)
    out = []
    for b in range(nb):
        lo, hi = (not periodic and b == 0), (not periodic and b == nb - 1)
        M = (_d1_block if order == 1 else _d2_block)(m, lo, hi)
        d = (m - 1) / (coords[(b + 1) * m - 1] - coords[b * m])
        M = torch.as_tensor(M * d ** order, device=x.device)
        idx = torch.arange(b * m - 4, (b + 1) * m + 4, device=x.device)
        idx = idx % n if periodic else idx.clamp(0, n - 1)  # the clamped ones meet zero columns
        out.append(v.index_select(-1, idx) @ M.T)
    return torch.cat(out, -1).movedim(-1, axis)


def _mlp_exact(x, wb):
    h = x
    for k, (w, b) in enumerate(wb):
        h = h @ w + b
        if k < 3:
            h = torch.nn.functional.gelu(h, approximate="tanh")
    return h


def exact(case, seed):
    kind = case["kind"]
    if kind == "deriv":
        x, gs = _deriv_inputs(case, seed)
        x = x.double().requires_grad_(True)
        p = default_params(case["nr"], case["nth"], case["nphi"], (case["nnr"], case["nnt"], case["nnp"]))
        theta, phi, _, _ = problem.angles(p)
        rx = np.arange(case["nr"]) / float(case["nr"] - 1)
        ys = [_deriv_exact(x, -3, case["order"], rx, case["nnr"], False),
              _deriv_exact(x, -1, case["order"], theta, case["nnt"], False),
              _deriv_exact(x, -2, case["order"], phi, case["nnp"], True)]
        gx, = torch.autograd.grad(ys, x, [g.double() for g in gs])
        return {"dr": ys[0].detach(), "dt": ys[1].detach(), "dp": ys[2].detach(), "gx": gx}
    if kind == "closure":
        dims, f, qscale, tscale, wb = _closure_inputs(case, seed)
        ds = torch.empty_like(f[3])
        ds[1:-1] = (f[3][2:] - f[3][:-2]) / 2.0
        ds[0], ds[-1] = f[3][1] - f[3][0], f[3][-1] - f[3][-2]
        q = torch.stack([f[0], f[1], f[2], (f[4] ** 2 + f[5] ** 2 + f[6] ** 2).sqrt(), ds], -1)
        q /= torch.as_tensor(qscale, device=f.device).double()
        nr, nphi, nth = f.shape[1:]
        at = lambda n: torch.arange(n, device=f.device)  # noqa: E731
        cols = []
        for dr in (-1, 0, 1):
            for dt in (-1, 0, 1):
                for dp in (-1, 0, 1):
                    v = q.index_select(0, (at(nr) + dr).clamp(0, nr - 1))
                    v = v.index_select(1, (at(nphi) + dp) % nphi).index_select(2, (at(nth) + dt).clamp(0, nth - 1))
                    cols.append(v.reshape(-1, 5).float())
        x = torch.zeros((nr * nphi * nth, 144), dtype=torch.float32, device=f.device)
        x[:, :135] = torch.cat(cols, -1)
        del cols
        wb = [(torch.as_tensor(w, device=f.device).double(), torch.as_tensor(b, device=f.device).double())
              for w, b in wb]
        ts = torch.as_tensor(tscale, device=f.device).double()
        s2 = torch.empty(x.shape[0], dtype=torch.float64, device=f.device)
        for k in range(0, x.shape[0], 1 << 18):
            y = _mlp_exact(x[k:k + (1 << 18)].double(), wb)
            s2[k:k + (1 << 18)] = (y[:, [0, 3, 5]] * ts[[0, 3, 5]]).sum(-1).clamp(min=0.0)
        return {"features": x.reshape(-1), "speed2": s2}
    if kind == "train":
        x, t, wb = _train_inputs(case, seed)
        prm = [(torch.as_tensor(w, device=x.device).double().requires_grad_(True),
                torch.as_tensor(b, device=x.device).double().requires_grad_(True)) for w, b in wb]
        loss = ((_mlp_exact(x.double(), prm) - t.double())[:, :12] ** 2).mean()
        g = torch.autograd.grad(loss, [v for wb_ in prm for v in wb_])
        return {"loss": loss.item(), "grads": [(g[2 * k].clone(), g[2 * k + 1].clone()) for k in range(4)]}
    # a step has no value apart from the scheme's own arithmetic, which is
    # 64-bit throughout (32-bit stage states in the mixed form)
    return None

