"""The work that users of this solver have it do, as cases that can be timed.

A case is a dict of plain values.  `prepare` makes what a program has in hand before the call
(a handle or a batch with its initial field, device buffers, pinned host arrays), `run` makes
one pass through the public entry points and returns everything the pass computes, `work` says
what a pass cannot do without, and `exact` gives the same outputs in 64 bits where the case is a
periodic box (the boundary cases have no value here).

Kinds:
  buffers   steps of a periodic box on the caller's own device buffers
            (mrlbm_step_periodic_noalloc), the moments staying on the device;
  box       a Taylor-Green run of a handle: `steps` time steps, then the field on the host;
  exchange  a coupled program: upload a field, a few steps, download the field;
  cylinder  flow past a cylinder (the shipped case and its rescalings, or a walled channel):
            `steps` steps with the wall forces sampled, then the force history and the field;
  annulus   Taylor-Couette flow between cylinders, the same outputs;
  batch     uneven cylinder channels advanced together, every case's forces and field.

Fields of runs with 16-bit storage are handed on in 16 bits, scaled as the storage scales them
(all that such a run holds), to analysis on the GPU.  Force histories come back in 32 bits, the
precision of their per-node terms.
"""
import ctypes
import math

import numpy as np
import torch

from mrlbm_3d_cuda_gb300 import Batch, Simulation, cases, native

STORAGES = {"f32": native.STORAGE_F32, "f16": native.STORAGE_F16, "bf16": native.STORAGE_BF16,
            "hybrid": native.STORAGE_F16_U32}
NODE_BYTES = {"f32": 40, "f16": 20, "bf16": 20, "hybrid": 28}   # stored moments of one node
STEP_FLOPS = 300                                                # of one node and step


def listed():
    return [
        # a small box stepped one call at a time: the call's own latency
        {"name": "buffers_64", "kind": "buffers", "nx": 64, "ny": 64, "nz": 64, "steps": 1, "diag": False},
        # the 256^3 box of the headline benchmark, on the caller's buffers
        {"name": "buffers_256", "kind": "buffers", "nx": 256, "ny": 256, "nz": 256, "steps": 8, "diag": False},
        # a large box, one step (5.4 GB read and as much written)
        {"name": "buffers_512", "kind": "buffers", "nx": 512, "ny": 512, "nz": 512, "steps": 2, "diag": False},
        # Taylor-Green vortex with FP16 storage, mass and energy sampled on the way
        {"name": "box_f16_256", "kind": "box", "n": 256, "steps": 200, "storage": "f16", "sr": False,
         "diag_every": 20},
        # the same scheme on a box whose sides fit no tile, field exchanged with another program
        # every few steps
        {"name": "exchange_ragged", "kind": "exchange", "nx": 200, "ny": 136, "nz": 92, "steps": 20},
        # the smallest configured cylinder (128 x 64 x 32, D 16): launches and latency
        {"name": "channel_small", "kind": "cylinder", "nx": 128, "ny": 64, "nz": 32, "d": 16, "u": 0.05,
         "re": 30.0, "steps": 100, "force_every": 1, "storage": "f32", "sr": False, "periodic_y": False,
         "periodic_z": True, "convective": False},
        # the shipped cylinder case (336 x 144 x 48, D 16), drag and lift every step
        {"name": "cylinder_d16", "kind": "cylinder", "nx": 336, "ny": 144, "nz": 48, "d": 16, "u": 0.1,
         "re": 100.0, "steps": 100, "force_every": 1, "storage": "f32", "sr": False, "periodic_y": True,
         "periodic_z": True, "convective": True},
        # the same rescaled to D 32 (672 x 288 x 96) in the hybrid storage, rounded stochastically
        {"name": "cylinder_d32_hybrid", "kind": "cylinder", "nx": 672, "ny": 288, "nz": 96, "d": 32, "u": 0.1,
         "re": 100.0, "steps": 100, "force_every": 10, "storage": "hybrid", "sr": True, "periodic_y": True,
         "periodic_z": True, "convective": True},
        # the shipped annulus (136 x 136 x 256): curved walls in every tile, torque sampled
        {"name": "annulus_shipped", "kind": "annulus", "nx": 136, "ny": 136, "nz": 256, "r_in": 32.0,
         "r_out": 64.0, "u": 0.03, "re": 70.0, "steps": 100, "force_every": 10, "storage": "f32", "sr": False,
         "periodic_z": True},
        # annulus between end plates with BF16 storage
        {"name": "annulus_plates_bf16", "kind": "annulus", "nx": 160, "ny": 160, "nz": 128, "r_in": 32.0,
         "r_out": 64.0, "u": 0.05, "re": 60.0, "steps": 100, "force_every": 10, "storage": "bf16", "sr": True,
         "periodic_z": False},
        # a sweep over diameters and Reynolds numbers, advanced as one batch
        {"name": "batch_12", "kind": "batch", "count": 12, "sizes": 1234, "steps": 40, "force_every": 10,
         "storage": "f32"},
    ]


def _near(rng, lo, hi, multiple):
    """A multiple of `multiple` between lo and hi, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, multiple * round(v / multiple))


def _steps(rng, nodes, most, budget=2.5e9):
    return max(1, min(most, int(rng.uniform(0.3, 1.0) * budget / nodes)))


def draw(rng):
    kind = rng.choice(["buffers", "buffers", "box", "exchange", "cylinder", "cylinder", "annulus", "batch"])
    storage = rng.choice(["f32", "f32", "f32", "f16", "bf16", "hybrid"])
    sr = storage != "f32" and rng.random() < 0.5
    if kind == "buffers":
        nx, ny, nz = (_near(rng, 32, 480, m) for m in (8, 8, 4))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": min(8, _steps(rng, nx * ny * nz, 8)),
                "diag": rng.random() < 0.25}
    if kind == "box":
        n = _near(rng, 48, 256, 8)
        # rounding differences add up over FP32 steps: short runs
        return {"kind": kind, "n": n, "steps": _steps(rng, n ** 3, 40 if storage == "f32" else 200),
                "storage": storage, "sr": sr, "diag_every": rng.choice([0, 1, 7, 20])}
    if kind == "exchange":
        nx, ny, nz = (_near(rng, 40, 240, m) for m in (8, 8, 4))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": rng.randint(1, 20)}
    if kind == "annulus":
        r_out = rng.uniform(18.0, 76.0)
        side = 8 * math.ceil((2 * r_out + 6) / 8)
        nz = _near(rng, 16, 256, 4)
        gap = r_out * rng.uniform(0.45, 0.6)
        u = rng.uniform(0.02, 0.05)
        return {"kind": kind, "nx": side, "ny": side, "nz": nz, "r_in": round(r_out - gap, 2),
                "r_out": round(r_out, 2), "u": round(u, 4), "re": round(u * gap / rng.uniform(0.012, 0.03), 2),
                "steps": _steps(rng, side * side * nz, 100), "force_every": rng.choice([1, 10]),
                "storage": storage, "sr": sr, "periodic_z": rng.random() < 0.6}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(3, 12), "sizes": rng.randint(1, 10 ** 6),
                "steps": rng.randint(10, 40), "force_every": rng.choice([0, 1, 10]),
                "storage": rng.choice(["f32", "f32", "f16"])}
    d = rng.randint(10, 36)
    nx, ny, nz = 8 * math.ceil(12 * d / 8), 8 * math.ceil(6 * d / 8), _near(rng, 16, 96, 4)
    u = rng.uniform(0.04, 0.1)
    return {"kind": "cylinder", "nx": nx, "ny": ny, "nz": nz, "d": d, "u": round(u, 4),
            "re": round(u * d / rng.uniform(0.014, 0.03), 2), "steps": _steps(rng, nx * ny * nz, 100),
            "force_every": rng.choice([1, 10]), "storage": storage, "sr": sr, "periodic_y": rng.random() < 0.5,
            "periodic_z": rng.random() < 0.7, "convective": rng.random() < 0.5}


# ---- inputs ---------------------------------------------------------------------------------

def _modes(nx, ny, nz, seed):
    """(10, nz, ny, nx) FP32 moments of a seeded smooth periodic flow, on the GPU: three shear
    modes per velocity component, |u| up to 0.05, a density wave, m_ab = u_a u_b off equilibrium."""
    g = np.random.default_rng(seed)
    axes = [2 * math.pi * torch.arange(n, device="cuda", dtype=torch.float64) / n for n in (nx, ny, nz)]
    X, Y, Z = axes[0][None, None, :], axes[1][None, :, None], axes[2][:, None, None]
    out = torch.empty((10, nz, ny, nx), device="cuda", dtype=torch.float32)

    def wave(amplitude):
        v = 0.0
        for _ in range(3):
            k = g.integers(0, 3, size=3)
            v = v + amplitude / 3 * torch.sin(int(k[0]) * X + int(k[1]) * Y + int(k[2]) * Z + g.uniform(0, 2 * math.pi))
        return v.expand(nz, ny, nx)

    out[0] = wave(2e-3)
    for a in range(3):
        out[1 + a] = wave(0.05)
    for f, (a, b) in enumerate(((1, 1), (2, 2), (3, 3), (1, 2), (1, 3), (2, 3))):
        torch.mul(out[a], out[b], out=out[4 + f])
        out[4 + f] += wave(2e-4)
    return out


def _to_storage(m):
    """Lexicographic (10, nz, ny, nx) -> the solver's x-blocked layout (mrlbm.h), flat."""
    _, nz, ny, nx = m.shape
    nxb = -(-nx // 32)
    out = torch.zeros((nz, ny, nxb, 10, 32), device=m.device, dtype=m.dtype)
    for b in range(nxb):
        w = min(32, nx - 32 * b)
        out[:, :, b, :, :w] = m[..., 32 * b: 32 * b + w].permute(1, 2, 0, 3)
    return out.reshape(-1)


def _desc(case, seed):
    """Case descriptor and the initial field (kind, parameters)."""
    k, s = case["kind"], STORAGES[case.get("storage", "f32")]
    noise = float(seed % 1000003)
    if k == "box":
        d = cases.periodic_box(case["n"], u0=0.05, re=1600.0 * case["n"] / 256, storage=s)
        init = native.INIT_TAYLOR_GREEN, (0.035 + 1.5e-2 * (seed * 0.6180339887 % 1.0), float(d.length))
    elif k == "exchange":
        d = cases.periodic_box(case["nx"], case["ny"], case["nz"], u0=0.05, re=200.0, storage=s)
        init = None
    elif k == "annulus":
        d = cases.annulus(case["nx"], case["ny"], case["nz"], case["r_in"], case["r_out"], case["u"], case["re"],
                          periodic_z=case["periodic_z"], storage=s)
        # an axial stream through the gap (spiral Couette flow)
        init = native.INIT_NOISY_UNIFORM, (0.0, 0.0, case["u"], 0.05, noise)
    else:
        c = 4.0 * case["d"] + 0.5 * (case["d"] - 1)
        # the shipped case's 4 D upstream where it fits, else 3 D to each side wall
        yc = c if case["ny"] >= 9 * case["d"] else 0.5 * case["ny"]
        xc = c if case["nx"] >= 12 * case["d"] else 0.25 * case["nx"]
        d = cases.cylinder_channel(case["nx"], case["ny"], case["nz"], case["d"], xc, yc, case["u"], case["re"],
                                   periodic_y=case["periodic_y"], periodic_z=case["periodic_z"],
                                   convective=case["convective"], storage=s)
        init = native.INIT_NOISY_UNIFORM, (case["u"], 0.0, 0.0, 0.01, noise)
    d.stochastic_rounding = int(case.get("sr", False))
    return d, init


def _batch_descs(case):
    """The sweep: D, Re and the channel around them drawn from the case's own number."""
    g = np.random.default_rng(case["sizes"])
    out = []
    for _ in range(case["count"]):
        d, nu = int(g.integers(8, 33)), float(g.uniform(0.013, 0.03))
        nx, ny, nz = 8 * -(-12 * d // 8), 8 * -(-6 * d // 8), min(4 * -(-3 * d // 4), 64)
        out.append(cases.cylinder_channel(nx, ny, nz, d, 4.0 * d, 3.0 * d, 0.05, 0.05 * d / nu,
                                          storage=STORAGES[case["storage"]]))
    return out


def _field_buffers(sim, storage):
    """Pinned host array for the field; in 16-bit storage also its scales and the 16-bit copy that
    stays on the GPU for analysis there."""
    host = torch.empty((10,) + sim.shape, dtype=torch.float32, pin_memory=True)
    if storage == "f32":
        return host, None, None, None
    u = sim.desc.u_max
    scale = torch.tensor([1 / u ** 2] + 3 * [1 / u] + 6 * [1 / u ** 2]).reshape(10, 1, 1, 1).cuda()
    wide = torch.empty(host.shape, dtype=torch.float32, device="cuda")
    return host, scale, wide, torch.empty_like(wide, dtype=torch.bfloat16 if storage == "bf16" else torch.float16)


def _read_field(sim, buffers):
    host, scale, wide, half = buffers
    sim.moments(out=host.numpy())
    if half is None:
        return host
    return half.copy_(wide.copy_(host, non_blocking=True).mul_(scale))


def prepare(case, seed):
    k = case["kind"]
    if k == "buffers":
        a = _to_storage(_modes(case["nx"], case["ny"], case["nz"], seed))
        return {"case": case, "a": a, "b": torch.zeros_like(a), "omega": 1.0 / 0.53}
    if k == "batch":
        batch = Batch(_batch_descs(case))
        for i, c in enumerate(batch.cases):
            c.init(native.INIT_NOISY_UNIFORM, (0.05, 0.0, 0.0, 0.01, float((seed + 7919 * i) % 1000003)))
        batch.set_sampling(case["force_every"])
        return {"case": case, "batch": batch, "out": [_field_buffers(c, case["storage"]) for c in batch.cases]}
    desc, init = _desc(case, seed)
    sim = Simulation(desc, init=False)
    state = {"case": case, "sim": sim, "out": _field_buffers(sim, case.get("storage", "f32"))}
    if init is None:
        field = torch.empty((10,) + sim.shape, dtype=torch.float32, pin_memory=True)
        state["field"] = field.copy_(_modes(case["nx"], case["ny"], case["nz"], seed))
    else:
        sim.init(*init)
        sim.set_sampling(case.get("force_every", 0), case.get("diag_every", 0))
    return state


# ---- one pass -------------------------------------------------------------------------------

def _forces(sim, steps, every):
    """The forces sampled in the last `steps` steps, oldest first: (samples, 2 walls, 5)."""
    return sim.force_history(-(-steps // every))[1].astype(np.float32)


def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "buffers":
        lib = native.lib()
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        sums = (ctypes.c_double * 2)() if case["diag"] else None
        for _ in range(case["steps"]):
            a, b = state["a"], state["b"]
            native.check(lib.mrlbm_step_periodic_noalloc(a.data_ptr(), b.data_ptr(), case["nx"], case["ny"],
                                                         case["nz"], state["omega"], 1.0, sums, stream))
            state["a"], state["b"] = b, a
        out = [state["a"]]
        if sums is not None:
            out.append(np.array(sums[:], dtype=np.float32))
        return out
    if k == "batch":
        b = state["batch"]
        b.step(case["steps"])
        b.sync()
        out = [_read_field(c, o) for c, o in zip(b.cases, state["out"])]
        if case["force_every"]:
            out += [_forces(c, case["steps"], case["force_every"]) for c in b.cases]
        return out
    sim = state["sim"]
    if k == "exchange":
        sim.set_moments(state["field"].numpy())
        sim.step(case["steps"])
        return [_read_field(sim, state["out"])]
    sim.step(case["steps"])
    sim.sync()
    out = []
    if k == "box":
        every = case["diag_every"]
        if every:
            out.append(sim.diagnostics(-(-case["steps"] // every))[1].astype(np.float32))
    else:
        out.append(_forces(sim, case["steps"], case["force_every"]))
    return [_read_field(sim, state["out"])] + out


# ---- what a pass cannot do without -----------------------------------------------------------

def work(case):
    """Stored moments read and written once per step; fields that cross to or from the host
    once.  Flops: one node update."""
    k = case["kind"]
    if k == "batch":
        nodes = sum(d.nx * d.ny * d.nz for d in _batch_descs(case))
    elif k == "box":
        nodes = case["n"] ** 3
    else:
        nodes = case["nx"] * case["ny"] * case["nz"]
    node = NODE_BYTES[case.get("storage", "f32")]
    host = {"buffers": 0, "exchange": 2 * 40}.get(k, 40)
    return {"bytes": float(nodes) * (2 * node * case["steps"] + host), "flops": float(nodes) * STEP_FLOPS * case["steps"]}


# ---- the periodic boxes in 64 bits -------------------------------------------------------------

def _exact_steps(m, steps, omega):
    """`steps` steps of the moment-representation LBM on (10, nz, ny, nx) float64 moments (rho -
    rho0 first, rho0 = 1): every population rebuilt from its neighbour's moments, D3Q27 weights
    as FP32 tables hold them; returns the moments and each step's (mass, energy) before collision."""
    w = [float(np.float32(v)) for v in (8 / 27, 2 / 27, 1 / 54, 1 / 216)]
    pairs = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
    sums = []
    for _ in range(steps):
        rho = 1.0 + m[0]
        lin = [3.0 * rho * m[1 + a] for a in range(3)]
        quad = [(4.5 if a == b else 9.0) * rho * m[4 + f] for f, (a, b) in enumerate(pairs)]
        base = rho * (1.0 - 1.5 * (m[4] + m[5] + m[6]))
        new = torch.zeros_like(m)
        for cx in (-1, 0, 1):
            for cy in (-1, 0, 1):
                for cz in (-1, 0, 1):
                    c = (cx, cy, cz)
                    f = base.clone()
                    for a in range(3):
                        if c[a]:
                            f += c[a] * lin[a]
                    for q, (a, b) in zip(quad, pairs):
                        if c[a] * c[b]:
                            f += c[a] * c[b] * q
                    f *= w[abs(cx) + abs(cy) + abs(cz)]
                    f = torch.roll(f, (cz, cy, cx), (0, 1, 2))
                    new[0] += f
                    for a in range(3):
                        if c[a]:
                            new[1 + a] += c[a] * f
                    for i, (a, b) in enumerate(pairs):
                        if c[a] * c[b]:
                            new[4 + i] += c[a] * c[b] * f
        rho = new[0].clone()
        new[0] -= 1.0
        for i in range(1, 10):
            new[i] /= rho
        sums.append((float(rho.sum()), 0.5 * float((new[1] ** 2 + new[2] ** 2 + new[3] ** 2).sum())))
        for i, (a, b) in enumerate(pairs):
            new[4 + i] -= (1.0 / 3.0 if a == b else 0.0)
            new[4 + i] = (1.0 - omega) * new[4 + i] + omega * new[1 + a] * new[1 + b]
        m = new
    return m, sums


def exact(case, seed):
    k = case["kind"]
    if k == "buffers":
        m = _modes(case["nx"], case["ny"], case["nz"], seed).double()
        m, sums = _exact_steps(m, case["steps"], float(np.float32(1.0 / 0.53)))
        out = [_to_storage(m)]
        return out + [np.array(sums[-1])] if case["diag"] else out
    if k == "exchange":
        d, _ = _desc(case, seed)
        m = _modes(case["nx"], case["ny"], case["nz"], seed).double()
        return [_exact_steps(m, case["steps"], _omega(d.u_max, d.length, d.re))[0]]
    if k != "box":
        return None
    d, (_, (u0, L)) = _desc(case, seed)
    n = case["n"]
    x = torch.arange(n, device="cuda", dtype=torch.float64) / L
    X, Y, Z = x[None, None, :], x[None, :, None], x[:, None, None]
    m = torch.zeros((10, n, n, n), device="cuda", dtype=torch.float64)
    m[1] = u0 * torch.sin(X) * torch.cos(Y) * torch.cos(Z)
    m[2] = -u0 * torch.cos(X) * torch.sin(Y) * torch.cos(Z)
    m[0] = 3.0 * u0 * u0 / 16.0 * (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0)
    m[4], m[5], m[7] = m[1] ** 2, m[2] ** 2, m[1] * m[2]
    m, sums = _exact_steps(m, case["steps"], _omega(d.u_max, d.length, d.re))
    if case["storage"] != "f32":
        u = d.u_max
        m *= torch.tensor([1 / u ** 2] + 3 * [1 / u] + 6 * [1 / u ** 2], device="cuda", dtype=torch.float64).reshape(10, 1, 1, 1)
    every = case["diag_every"]
    return [m] + ([np.array(sums[::every])] if every else [])


def _omega(u, length, re):
    """The relaxation rate the descriptor stands for: tau = 1/2 + 3 u L / Re."""
    return 1.0 / (0.5 + 3.0 * u * length / re)
