"""Workloads of the S(Q,omega) engine, each one pass through the package's public entry points
with synthetic inputs made from a seed (ABO3 supercells, amorphous Al92U8 boxes, amplitude stores).

Kinds of case: the drop-in finufft calls an unmodified mp_sqom makes ("dropin"), the device-pointer
plan ("plan"), trajectories of crystals ("crystal") and of amorphous boxes ("alloy") through a job,
the time transforms of a stored trajectory ("spectrum", "maps"), mp_sql's spherical average ("sql")
and a burst of small requests to the server ("requests").
"""
import ctypes
import math
import random

import numpy as np
import torch

from mp_tools_gb300 import _lib
from mp_tools_gb300.serve import Request, Server
from mp_tools_gb300.sqom import QGrid, SqomJob, TimeAxis
from mp_tools_gb300.sql import SqlGrid, transform_histogram

f32 = np.float32
A_CELL = 4.19
BASIS = [(0.0, 0.0, 0.0), (0.5, 0.5, 0.5), (0.5, 0.5, 0.0), (0.5, 0.0, 0.5), (0.0, 0.5, 0.5)]
SIGMA = [0.05, 0.05, 0.08, 0.08, 0.08]                     # Angstrom
B_COH = [0.507, 0.716, 0.5803, 0.5803, 0.5803]             # A, B, O, O, O
XFF = [[6.4202, 3.0387, 1.9002, 0.7426, 1.5936, 31.5472, 1.9646, 85.0886, 1.1151],
       [36.0228, 0.5293, 23.4128, 3.3253, 14.9491, 16.0927, 4.1880, 100.6130, 13.3966]]
DT = 0.01                                                  # ps between frames


def listed():
    return [
        # the reference's own call: one species and frame of its BZO (hk0) example, host arrays
        {"name": "dropin_plane", "kind": "dropin", "dim": 2, "cells": 32, "m0": 160, "m1": 160,
         "m2": 1, "eps": 1e-6},
        # a host program that keeps its points on the device: two strength vectors, odd sizes
        {"name": "plan_volume_fp32", "kind": "plan", "dim": 3, "points": 200003, "m0": 127,
         "m1": 120, "m2": 101, "eps": 1e-5, "bits": 32, "ntrans": 2},
        # mp_sqom's usual run: an (hk0) plane, total S(Q) and E=const maps, 32 frames of the BZO
        # example's supercell
        {"name": "plane_fp32", "kind": "crystal", "dim": 2, "cells": 32, "frames": 32, "zones": 5,
         "bits": 32, "eps": 1e-6, "centre": 0, "window": 0, "econst": 2},
        # the same in plain FP64 off the origin of Q space with the spatial Hann window
        {"name": "plane_fp64_window", "kind": "crystal", "dim": 2, "cells": 20, "frames": 16,
         "zones": 6, "bits": 64, "eps": 1e-6, "centre": 2, "window": 1, "econst": 1},
        # static S(Q) volume in plain FP64: the first benchmark configuration
        {"name": "static_fp64", "kind": "crystal", "dim": 3, "cells": 20, "frames": 1, "zones": 8,
         "bits": 64, "eps": 1e-9, "centre": 0, "window": 0, "econst": 0},
        # the headline: frames of the batched amorphous alloy with X-ray weights
        {"name": "alloy_batch", "kind": "alloy", "atoms": 1000000, "frames": 8, "modes": 192,
         "eps": 1e-7},
        # inelastic crystal volume, five species on three grids
        {"name": "crystal_inelastic", "kind": "crystal", "dim": 3, "cells": 64, "frames": 2,
         "zones": 4, "bits": 32, "eps": 1e-6, "centre": 0, "window": 0, "econst": 0},
        # the largest configuration: one static frame on a 1152^3 fine grid
        {"name": "large_static", "kind": "crystal", "dim": 3, "cells": 136, "frames": 1, "zones": 4,
         "bits": 32, "eps": 1e-5, "centre": 0, "window": 0, "econst": 0},
        # Gaussian-window spectrum and total S(Q) of a stored 512-frame run
        {"name": "spectrum", "kind": "spectrum", "cells": 24, "zones": 4, "frames": 512},
        # E=const, E(Q) and I(Q,t) maps of a stored plane run
        {"name": "plane_maps", "kind": "maps", "cells": 40, "zones": 8, "frames": 200, "bins": 4},
        # mp_sql: |Q| histogram of the reference's 30,000-atom example box, host frame in
        {"name": "sql_average", "kind": "sql", "atoms": 30000, "frames": 1, "q_range": 6.0},
        # a burst of small jobs at the request server, results back on the host
        {"name": "requests", "kind": "requests", "jobs": 8, "edge": 16, "frames": 24, "zones": 3},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["dropin", "plan", "crystal", "crystal", "plane", "plane", "alloy", "alloy",
                       "spectrum", "maps", "sql", "requests"])
    if kind == "dropin":
        dim = rng.choice([2, 2, 3])
        top = 400 if dim == 2 else 72
        return {"kind": kind, "dim": dim, "cells": log(8, 48), "m0": log(24, top), "m1": log(24, top),
                "m2": 1 if dim == 2 else log(24, top), "eps": rng.choice([1e-4, 1e-6, 1e-9])}
    if kind == "plan":
        dim = rng.choice([2, 3])
        top = 600 if dim == 2 else 160
        return {"kind": kind, "dim": dim, "points": log(3000, 500000), "m0": log(30, top),
                "m1": log(30, top), "m2": 1 if dim == 2 else log(30, top),
                "eps": rng.choice([1e-4, 1e-5, 1e-6]), "bits": rng.choice([32, 32, 64]),
                "ntrans": rng.choice([1, 2, 3])}
    if kind == "plane":
        return {"kind": "crystal", "dim": 2, "cells": log(8, 44), "frames": log(4, 48),
                "zones": rng.randint(2, 8), "bits": rng.choice([32, 32, 64]),
                "eps": rng.choice([1e-5, 1e-6]), "centre": rng.choice([0, 0, 1, 2]),
                "window": rng.choice([0, 0, 1]), "econst": rng.choice([0, 1, 2])}
    if kind == "crystal":
        bits = rng.choice([32, 32, 32, 64])
        cells = log(8, 72 if bits == 32 else 20)
        return {"kind": kind, "dim": 3, "cells": cells, "frames": log(1, 8) if cells < 33 else 1,
                "zones": rng.randint(2, 4 if cells > 24 else 7), "bits": bits,
                "eps": rng.choice([1e-5, 1e-6]) if bits == 32 else rng.choice([1e-6, 1e-9]),
                "centre": rng.choice([0, 0, 0, 1]), "window": rng.choice([0, 0, 0, 1]), "econst": 0}
    if kind == "alloy":
        return {"kind": kind, "atoms": log(5000, 1000000), "frames": log(1, 8),
                "modes": 2 * log(16, 110), "eps": rng.choice([1e-5, 1e-6, 1e-7])}
    if kind == "spectrum":
        return {"kind": kind, "cells": log(6, 24), "zones": rng.randint(2, 4),
                "frames": rng.choice([32, 64, 128, 256, 512])}
    if kind == "maps":
        return {"kind": kind, "cells": log(12, 44), "zones": rng.randint(2, 7),
                "frames": log(30, 260), "bins": rng.randint(1, 4)}
    if kind == "sql":
        return {"kind": kind, "atoms": log(2000, 60000), "frames": rng.choice([1, 1, 2, 3]),
                "q_range": round(rng.uniform(3.0, 7.0), 2)}
    return {"kind": kind, "jobs": rng.randint(2, 10), "edge": log(8, 20), "frames": log(2, 32),
            "zones": rng.randint(2, 4)}


# ------------------------------------------------------------------------------- inputs
def device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def generator(seed):
    g = torch.Generator(device=device())
    g.manual_seed(int(seed))
    return g


def crystal_frames(cells, frames, seed):
    """(frames, 5 cells^3, 4) float32 in lattice units: ideal ABO3 sites, every atom vibrating at
    a frequency of its own (1-20 THz) with Gaussian amplitudes."""
    d, g = device(), generator(seed)
    i = torch.arange(cells, device=d, dtype=torch.float32) - cells // 2
    site = torch.stack(torch.meshgrid(i, i, i, indexing="ij"), -1).reshape(-1, 3)
    n = site.shape[0]
    out = torch.zeros((frames, 5 * n, 4), dtype=torch.float32, device=d)
    for s in range(5):
        u = torch.randn((2, n, 3), generator=g, device=d) * (SIGMA[s] / A_CELL)
        w = 2 * math.pi * (1.0 + 19.0 * torch.rand((n, 1), generator=g, device=d))
        base = site + torch.tensor(BASIS[s], device=d)
        for t in range(frames):
            out[t, s * n:(s + 1) * n, :3] = base + u[0] * torch.cos(w * (t * DT)) + u[1] * torch.sin(w * (t * DT))
    return out


def alloy_frames(atoms, frames, seed):
    """(frames, atoms, 4) float32 in Angstrom: a disordered box at 0.06 atoms per cubic Angstrom
    (random sites of a fine lattice, displaced), Al then U, walking 0.1 Angstrom per frame."""
    d, g = device(), generator(seed)
    box = (atoms / 0.06) ** (1.0 / 3.0)
    side = int(math.ceil((1.3 * atoms) ** (1.0 / 3.0)))
    pick = torch.randperm(side ** 3, generator=g, device=d)[:atoms]
    site = torch.stack([pick % side, (pick // side) % side, pick // (side * side)], -1).to(torch.float32)
    p = (site + 0.5 + 0.7 * (torch.rand((atoms, 3), generator=g, device=d) - 0.5)) * (box / side)
    out = torch.zeros((frames, atoms, 4), dtype=torch.float32, device=d)
    for t in range(frames):
        if t:
            p = p + 0.1 * torch.randn((atoms, 3), generator=g, device=d)
        p = torch.remainder(p, box)
        out[t, :, :3] = p - box / 2
    return out, [atoms - int(round(0.08 * atoms)), int(round(0.08 * atoms))], box


def store_series(n_frames, n_q, seed):
    """(n_frames, n_q) complex64 amplitudes: an elastic part, a fluctuation with memory."""
    d, g = device(), generator(seed)
    x = torch.randn((n_q, 2), generator=g, device=d)
    mean = 3.0 * torch.randn((n_q, 2), generator=g, device=d)
    out = torch.empty((n_frames, n_q, 2), dtype=torch.float32, device=d)
    for t in range(n_frames):
        x = 0.95 * x + 0.3 * torch.randn((n_q, 2), generator=g, device=d)
        out[t] = 100.0 * (mean + x)
    return torch.view_as_complex(out)


def dropin_inputs(case, seed):
    """Phases and strengths of one species as mp_sqom forms them (FP32 phases, Q centre 2 2 0)."""
    n = case["cells"]
    r = crystal_frames(n, 1, seed)[0, n ** 3:2 * n ** 3, :3].cpu().numpy()
    tpe = f32(2 * math.pi / n)
    x = [np.ascontiguousarray((r[:, k] * tpe).astype(np.float64)) for k in range(case["dim"])]
    r64 = r.astype(np.float64)
    return x, np.ascontiguousarray(np.exp(-2j * np.pi * (2.0 * r64[:, 0] + 2.0 * r64[:, 1])))


def plan_inputs(case, seed):
    d, g = device(), generator(seed)
    real = torch.float32 if case["bits"] == 32 else torch.float64
    x = (2 * torch.rand((case["dim"], case["points"]), generator=g, device=d, dtype=torch.float64) - 1) * math.pi
    x = x.to(real).clamp(-3.1415925, 3.1415925)
    c = torch.view_as_complex(torch.randn((case["ntrans"], case["points"], 2), generator=g, device=d, dtype=real))
    return x, c


def request_list(case, seed):
    r = random.Random("%(jobs)d %(edge)d %(frames)d %(zones)d" % case)
    out = []
    for k in range(case["jobs"]):
        edge = r.randint(max(4, case["edge"] // 2), case["edge"])
        frames = r.randint(max(1, case["frames"] // 4), case["frames"])
        out.append((edge, frames, r.randint(2, case["zones"]), 1000 * int(seed) + k))
    return out


def q_grid(case):
    n = case["cells"]
    dim = 2 if case["kind"] == "maps" else case.get("dim", 3)
    centre = float(case.get("centre", 0))
    return QGrid(_lib.CELL, (n,) * 3, n_bz=case["zones"], a_par=(A_CELL,) * 3, ndim=dim,
                 q_center=(centre, centre, 0.0))


def store_job(case, grid, seed):
    """A job whose amplitude store holds an earlier run's amplitudes (read back into it)."""
    job = SqomJob(grid, species_counts=[1000], n_frames=case["frames"], eps=1e-5)
    job.amplitudes_device().copy_(store_series(case["frames"], grid.n_modes, seed))
    return job


# ------------------------------------------------------------------------------- passes
def prepare(case, seed):
    kind = case["kind"]
    if kind == "dropin":
        x, c = dropin_inputs(case, seed)
        fk = np.zeros(case["m0"] * case["m1"] * case["m2"], np.complex128)
        return {"case": case, "x": x, "c": c, "fk": fk, "lib": _lib.load()}
    if kind == "plan":
        x, c = plan_inputs(case, seed)
        m = [case["m0"], case["m1"], case["m2"]][:case["dim"]]
        return {"case": case, "x": x, "c": c, "plan": Plan(m, case),
                "fk": torch.empty((case["ntrans"],) + tuple(m[::-1]), dtype=c.dtype, device="cuda")}
    if kind == "crystal":
        grid = q_grid(case)
        frames = crystal_frames(case["cells"], case["frames"], seed)
        job = SqomJob(grid, species_counts=[case["cells"] ** 3] * 5, n_frames=case["frames"],
                      precision=_lib.FP32 if case["bits"] == 32 else _lib.FP64, eps=case["eps"],
                      weight_mode=_lib.WEIGHT_NEUTRON, b_coh=B_COH, window=bool(case["window"]))
        return job_state(case, job, grid, frames)
    if kind == "alloy":
        frames, counts, box = alloy_frames(case["atoms"], case["frames"], seed)
        grid = QGrid(_lib.BULK, (1, 1, 1), n_bz=alloy_range(case, box), a_par=(box,) * 3, ndim=3)
        job = SqomJob(grid, species_counts=counts, n_frames=case["frames"], eps=case["eps"],
                      weight_mode=_lib.WEIGHT_XRAY, xff=XFF, ff_convention=_lib.FF_STANDARD)
        return job_state(case, job, grid, frames)
    if kind == "spectrum":
        grid = q_grid(case)
        n_freq = case["frames"] // 2 + 1
        return {"case": case, "job": store_job(case, grid, seed),
                "sqw": torch.empty((n_freq, grid.n_modes), dtype=torch.float32, device="cuda"),
                "sq": torch.empty(grid.n_modes, dtype=torch.float32, device="cuda")}
    if kind == "maps":
        grid = q_grid(case)
        nx, ny = grid.n_q[0], grid.n_q[1]
        return {"case": case, "job": store_job(case, grid, seed), "time": TimeAxis(case["frames"], DT),
                "path": np.arange(nx, dtype=np.int64) + (ny // 2) * nx, "q2": grid.q2_norm(),
                "sqw": torch.empty((case["bins"], grid.n_modes), dtype=torch.float32, device="cuda")}
    if kind == "sql":
        frames, counts, box = alloy_frames(case["atoms"], case["frames"], seed)
        return {"case": case, "frames": frames.cpu().numpy(), "counts": counts,
                "grid": SqlGrid(case["q_range"], (box,) * 3)}
    jobs = []
    for k, (edge, frames, zones, s) in enumerate(request_list(case, seed)):
        fr = crystal_frames(edge, frames, s).cpu().pin_memory()
        grid = QGrid(_lib.CELL, (edge,) * 3, n_bz=zones, a_par=(A_CELL,) * 3, ndim=3)
        jobs.append(Request(k, 0.0, fr, [edge ** 3] * 5, grid,
                            dict(eps=1e-5, weight_mode=_lib.WEIGHT_NEUTRON, b_coh=B_COH), t_step=DT))
    return {"case": case, "jobs": jobs, "server": Server(budget_bytes=40 << 30)}


class Plan:
    """The C plan of a device-pointer program, kept for its points to come."""

    def __init__(self, m, case):
        self.lib, self.handle = _lib.load(), ctypes.c_void_p()
        modes = (ctypes.c_int64 * 3)(*(list(m) + [1] * (3 - len(m))))
        stream = torch.cuda.current_stream().cuda_stream
        _lib.check(self.lib.mpsq_nufft_makeplan(
            case["dim"], modes, -1, case["ntrans"], case["eps"],
            _lib.FP32 if case["bits"] == 32 else _lib.FP64, ctypes.c_void_p(stream),
            ctypes.byref(self.handle)), "makeplan")

    def __del__(self):
        if self.handle:
            self.lib.mpsq_nufft_destroy(self.handle)


def job_state(case, job, grid, frames):
    job.set_frames(frames)
    s = {"case": case, "job": job, "sq": torch.empty(grid.n_modes, dtype=torch.float32, device="cuda")}
    # the amplitudes are a result too, except on the largest grids, where S(Q) alone is asked for
    # (a view of the job's store: it keeps its job alive, wherever it goes)
    s["cs"] = job.amplitudes_device() if grid.n_modes < 1 << 26 else None
    if s["cs"] is not None:
        s["cs"].job = job
    bins = case.get("econst", 0) if case["frames"] >= 4 else 0
    s["time"] = TimeAxis(case["frames"], DT)
    s["sqw"] = torch.empty((bins, grid.n_modes), dtype=torch.float32, device="cuda") if bins else None
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "dropin":
        return dropin(s)
    if kind == "plan":
        p, x, c = s["plan"], s["x"], s["c"]
        at = [ctypes.c_void_p(x[k].data_ptr()) for k in range(case["dim"])] + [None]
        _lib.check(p.lib.mpsq_nufft_setpts(p.handle, x.shape[1], at[0], at[1], at[2]), "setpts")
        _lib.check(p.lib.mpsq_nufft_execute(p.handle, ctypes.c_void_p(c.data_ptr()),
                                            ctypes.c_void_p(s["fk"].data_ptr())), "execute")
        return {"fk": s["fk"]}
    if kind in ("crystal", "alloy"):
        job = s["job"]
        job.transform()
        out = {"sq": job.sq_total(out=s["sq"])}
        if s["cs"] is not None:
            out["cs"] = s["cs"]
        if s["sqw"] is not None:
            for b in range(s["sqw"].shape[0]):
                job.sqw_econst(s["time"], b + 1, out=s["sqw"][b])
            out["sqw"] = s["sqw"]
        return out
    if kind == "spectrum":
        job = s["job"]
        return {"sqw": job.sqw_gauss(t_step=DT, out=s["sqw"]), "sq": job.sq_total(out=s["sq"])}
    if kind == "maps":
        job, ta = s["job"], s["time"]
        for b in range(case["bins"]):
            job.sqw_econst(ta, 1 + 2 * b, q2_norm=s["q2"], out=s["sqw"][b])
        return {"sqw": s["sqw"], "cut": job.sqw_dispersion(ta, s["path"]),
                "iqt": job.iqt(ta.n_int, case["frames"] // 4),
                "iqt_cut": job.iqt_dispersion(ta.n_int, s["path"])}
    if kind == "sql":
        h = transform_histogram(s["frames"], s["counts"], s["grid"], 0.01, eps=1e-6)
        return {"hist": h.astype(np.float32)}     # sums of FP32 products
    results, _ = s["server"].run(s["jobs"])
    return {"%02d" % k: [results[k].sq, results[k].sqw] for k in sorted(results)}


def dropin(s):
    case, L = s["case"], s["lib"]
    at = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    n, flag, eps, ier = ctypes.c_int64(len(s["c"])), ctypes.c_int(-1), ctypes.c_double(case["eps"]), ctypes.c_int(0)
    m = [ctypes.byref(ctypes.c_int64(case[k])) for k in ("m0", "m1", "m2")][:case["dim"]]
    call = L.finufft2d1_ if case["dim"] == 2 else L.finufft3d1_
    call(ctypes.byref(n), *[at(x) for x in s["x"]], at(s["c"]), ctypes.byref(flag), ctypes.byref(eps),
         *m, at(s["fk"]), None, ctypes.byref(ier))
    if ier.value:
        raise RuntimeError(L.mpsq_last_error())
    return {"fk": s["fk"]}


# --------------------------------------------------------------------- what a pass is made of
def even(n):
    return n + (n % 2 if n > 1 else 0)


def crystal_modes(cells, zones):
    """Modes per axis: whole zones in steps of one per cell, truncated as the grid does, even."""
    return max(1, even(int(2 * math.pi * float(f32(zones)) / float(f32(2 * math.pi / cells)))))


def alloy_range(case, box):
    """Q range (1/Angstrom) that gives the case's modes per axis."""
    return float(f32((case["modes"] + 0.25) * 2 * math.pi / box))


def transform_work(points, dim, modes, eps, grids, value, spread):
    """Spreading every point over its support and the transform of the wanted modes' fine grid."""
    w = math.ceil(math.log10(1 / eps)) + 1
    return spread * points * w ** dim + grids * 5 * modes * math.log2(max(2, modes))


def work(case):
    kind = case["kind"]
    if kind in ("dropin", "plan"):
        m = case["m0"] * case["m1"] * case["m2"]
        n, size, nt = (case["cells"] ** 3, 8, 1) if kind == "dropin" else (case["points"], case["bits"] // 8, case["ntrans"])
        return {"bytes": size * (n * (case["dim"] + 2 * nt) + 2 * m * nt),
                "flops": transform_work(n * nt, case["dim"], m, case["eps"], nt, size, 4)}
    if kind in ("crystal", "alloy"):
        n = 5 * case["cells"] ** 3 if kind == "crystal" else case["atoms"]
        dim = case.get("dim", 3)
        m = (crystal_modes(case["cells"], case["zones"]) if kind == "crystal" else case["modes"]) ** dim
        c, f = case.get("bits", 32) // 4, case["frames"]
        grids = 1 if kind == "alloy" else 5 if case["centre"] else 3
        maps = case.get("econst", 0) if f >= 4 else 0
        return {"bytes": f * (16 * n + c * m) + 4 * m * (1 + maps),
                "flops": f * transform_work(n, dim, m, case["eps"], grids, c, 2) + maps * m * 2.0 * f * f}
    if kind == "spectrum":
        m, f = crystal_modes(case["cells"], case["zones"]) ** 3, case["frames"]
        return {"bytes": 8 * f * m + 4 * m * (f // 2 + 2), "flops": m * (5 * f * math.log2(f) + 12 * f)}
    if kind == "maps":
        nx, f = crystal_modes(case["cells"], case["zones"]), case["frames"]
        n_int, n_freq, n0 = hann_sizes(f)
        return {"bytes": nx * nx * (8 * f + 4 * (case["bins"] + 1)) + 4 * nx * (n_freq + n0),
                "flops": 8.0 * n0 * n_int * (nx * nx * case["bins"] + nx * n_freq)}
    if kind == "sql":
        box = (case["atoms"] / 0.06) ** (1 / 3)
        m = (2 * int(case["q_range"] * box / (2 * math.pi) + 0.5) + 1) ** 3
        f = case["frames"]
        return {"bytes": 16 * case["atoms"] * f + 16 * int(case["q_range"] / 0.01),
                "flops": f * (transform_work(case["atoms"], 3, m, 1e-6, 1, 8, 2) + 16 * m)}
    b = fl = 0
    for edge, frames, zones, _ in request_list(case, 0):
        m = crystal_modes(edge, zones) ** 3
        b += frames * (80 * edge ** 3 + 8 * m) + 20 * m
        fl += frames * transform_work(5 * edge ** 3, 3, m, 1e-5, 3, 8, 2)
    return {"bytes": b, "flops": fl}


def hann_sizes(frames):
    """Length of the sliding window (odd), its frequency bins and its start frames."""
    n = frames // 2
    n = max(1, min(n + 1 - n % 2, frames))
    return n, (n - 1) // 2 + 1, frames - n + 1


# -------------------------------------------------------------------- results in 64 bits
def direct(x, c, m):
    """sum_j c_j exp(-i k.x_j) for k = -m/2 .. (m-1)/2, x fastest: matrix products per axis."""
    k = [torch.arange(n, device=c.device, dtype=torch.float64) - n // 2 for n in m]
    out = torch.zeros(tuple(m[::-1]), dtype=torch.complex128, device=c.device)
    for a in range(0, c.shape[0], 65536):
        b = slice(a, a + 65536)
        e = [torch.polar(torch.ones((), dtype=torch.float64, device=c.device), -k[i][:, None] * x[i][b][None, :])
             for i in range(len(m))]
        right = e[0].T.contiguous()
        if len(m) == 2:
            out += (e[1] * c[b]) @ right
            continue
        for z in range(m[2]):
            out[z] += (e[1] * (e[2][z] * c[b])) @ right
    return out.reshape(-1)


def cheap(points, modes):
    return 8.0 * points * modes < 6e12


def hann(n):
    i = torch.arange(n, dtype=torch.float64, device=device())
    return (0.5 * (1 - torch.cos(2 * math.pi * i / (n - 1)))).to(torch.float32).double() if n > 1 else i + 1


def econst(x, j, frames, norm2, scale=None):
    """Sliding Hann-window map of the centred series at the 1-based bin j."""
    n, _, n0 = hann_sizes(frames)
    i = torch.arange(n, dtype=torch.float64, device=x.device)
    ph = torch.polar(hann(n), -2 * math.pi * (j - 1) * (i - n // 2) / n)
    y = x - x.mean(0)
    if scale is not None:
        y = y * scale
    s = torch.zeros(y.shape[1], dtype=torch.float64, device=x.device)
    for t in range(n0):
        s += (ph @ y[t:t + n]).abs() ** 2
    return s / (0.5 * n0 * n) * DT / norm2


def exact_job(case, frames, counts, x_of, m, weights):
    """Amplitudes, S(Q) and E=const maps of a job."""
    f, n = frames.shape[0], sum(counts)
    if not cheap(f * n, math.prod(m)):
        return None
    dim, centre = len(m), float(case.get("centre", 0))
    cs = torch.zeros((f, math.prod(m)), dtype=torch.complex128, device=frames.device)
    for t in range(f):
        a = 0
        for s, cnt in enumerate(counts):
            r = frames[t, a:a + cnt, :3].double()
            a += cnt
            x = x_of(r)
            turns = centre * r[:, 0] + centre * r[:, 1]
            c = torch.polar(torch.ones_like(turns), -2 * math.pi * (turns - torch.floor(turns)))
            if case.get("window"):
                for k in range(dim):
                    c = c * (1 + torch.cos(x[k]))
            cs[t] += weights[s] * direct(x, c, m)
    if case.get("window"):
        cs *= 0.25 if dim == 2 else 0.125
    out = {"sq": (cs.abs() ** 2).mean(0) / float(n) ** 2}
    if math.prod(m) < 1 << 26:
        out["cs"] = cs
    bins = case.get("econst", 0) if f >= 4 else 0
    if bins:
        out["sqw"] = torch.stack([econst(cs, b + 1, f, float(n) ** 2) for b in range(bins)])
    return out


def exact_crystal(case, frames):
    cells, dim = case["cells"], case.get("dim", 3)
    tpe = float(f32(2 * math.pi / cells))
    m = [crystal_modes(cells, case["zones"])] * dim
    return exact_job(case, frames, [cells ** 3] * 5, lambda r: [r[:, k] * tpe for k in range(dim)], m, B_COH)


def form_factor(xff, s2):
    return xff[8] + sum(xff[2 * i] * torch.exp(-xff[2 * i + 1] * s2) for i in range(4))


def exact_alloy(case, seed):
    if not cheap(case["atoms"] * case["frames"], case["modes"] ** 3):
        return None
    frames, counts, box = alloy_frames(case["atoms"], case["frames"], seed)
    span = f32(f32(box) / 2) - f32(-f32(box) / 2)
    tpe = float(f32(2 * math.pi / float(span)))
    m = case["modes"]
    zone = f32(alloy_range(case, box))
    dq = f32(zone / m)
    q0 = float(f32(f32(-0.5) * zone) + f32(m // 2) * dq)
    q = q0 + float(dq) * (torch.arange(m, dtype=torch.float64, device=frames.device) - m // 2)
    q2 = (q[:, None, None] ** 2 + q[None, :, None] ** 2 + q[None, None, :] ** 2).reshape(-1)
    w = [form_factor(x, q2 / (16 * math.pi ** 2)) for x in XFF]
    return exact_job(case, frames, counts, lambda r: [r[:, k] * tpe for k in range(3)], [m] * 3, w)


def exact_spectrum(case, seed):
    f, m = case["frames"], crystal_modes(case["cells"], case["zones"]) ** 3
    x = store_series(f, m, seed)
    t = torch.arange(f, dtype=torch.float64, device=x.device)
    g = torch.exp(-4 * math.log(2.0) * ((t - 0.5 * (f - 1)) / (f / 2)) ** 2)
    sqw = torch.empty((f // 2 + 1, m), dtype=torch.float64, device=x.device)
    sq = torch.empty(m, dtype=torch.float64, device=x.device)
    for a in range(0, m, 65536):
        y = x[:, a:a + 65536].to(torch.complex128)
        sq[a:a + 65536] = (y.abs() ** 2).mean(0) / 1e6
        y = torch.fft.fft((y - y.mean(0)) * g[:, None], dim=0)[:f // 2 + 1]
        sqw[:, a:a + 65536] = y.abs() ** 2 * (DT / 1e6 / float(g.sum()))
    return {"sqw": sqw, "sq": sq}


def exact_maps(case, seed):
    f, nx = case["frames"], crystal_modes(case["cells"], case["zones"])
    n, n_freq, n0 = hann_sizes(f)
    x = store_series(f, nx * nx, seed).to(torch.complex128)
    q = [f32(-0.5) * f32(case["zones"]) + np.arange(nx, dtype=f32) * f32(f32(case["zones"]) / nx)] * 2
    q2 = (q[0][None, :] ** 2 + q[1][:, None] ** 2).astype(f32)
    inv = np.where(q2 >= 1e-8, 1 / np.sqrt(np.maximum(q2, 1e-30)), 1.0).astype(f32).reshape(-1)
    inv = torch.from_numpy(inv).to(x.device).double()
    sqw = torch.stack([econst(x, 1 + 2 * b, f, 1e6, inv) for b in range(case["bins"])])
    y = x - x.mean(0)
    row = slice((nx // 2) * nx, (nx // 2) * nx + nx)
    p = y[:, row]
    i = torch.arange(n, dtype=torch.float64, device=x.device)
    ft = torch.polar(hann(n).expand(n_freq, n), -2 * math.pi * torch.arange(n_freq, device=x.device)[:, None] * i / n)
    cut = sum((ft @ p[t:t + n]).abs() ** 2 for t in range(n0)).T / (0.5 * n0 * n) * (DT / 1e6)
    lag = f // 4
    iqt = (y[lag:lag + n] * y[:n].conj()).real.sum(0) / n / 1e6
    iqt_cut = torch.stack([(p[t:t + n] * p[:n].conj()).real.sum(0) for t in range(n0)], 1) / 1e6
    return {"sqw": sqw, "cut": cut, "iqt": iqt, "iqt_cut": iqt_cut}


def exact_sql(case, seed):
    frames, counts, box = alloy_frames(case["atoms"], case["frames"], seed)
    dq = f32(2 * math.pi) / f32(box)
    half = int(math.floor(float(f32(0.5) * f32(2 * case["q_range"]) / dq) + 0.5))
    m = [2 * half + 1] * 3
    if not cheap(case["atoms"] * case["frames"], math.prod(m)):
        return None
    # |Q| in single precision as the scaled sum of squares of Fortran's NORM2, binned by NINT
    v = (torch.arange(m[0], device=frames.device) - half).to(torch.float32) * float(dq)
    q = torch.stack(torch.meshgrid(v, v, v, indexing="ij"), -1).reshape(-1, 3).flip(1).abs()
    scale, ssq = torch.zeros_like(q[:, 0]), torch.ones_like(q[:, 0])
    for k in range(3):
        a = q[:, k]
        up = (a != 0) & (scale < a)
        r = torch.where(up, scale / a, a / scale)
        r2 = r * r
        ssq = torch.where(up, 1.0 + ssq * r2, torch.where(a != 0, ssq + r2, ssq))
        scale = torch.where(up, a, scale)
    qn = scale * torch.sqrt(ssq)
    n_hist = 1 + int(f32(case["q_range"]) / f32(0.01))
    bins = torch.floor((qn / float(f32(0.01))).double() + 0.5).long()
    keep = (qn <= float(f32(case["q_range"]))) & (bins < n_hist)
    bins = torch.where(keep, bins, torch.full_like(bins, n_hist))
    out = torch.zeros((2, 2, n_hist + 1), dtype=torch.float64, device=frames.device)
    one = torch.ones((), dtype=torch.float64, device=frames.device)
    for t in range(case["frames"]):
        amp, a = [], 0
        for cnt in counts:
            r = frames[t, a:a + cnt, :3].double()
            a += cnt
            amp.append(direct([r[:, k] * float(dq) for k in range(3)], one.expand(cnt).to(torch.complex128), m) / sum(counts))
        for i in range(2):
            for j in range(2):
                out[i, j].index_add_(0, bins, (amp[i] * amp[j].conj()).real)
    return {"hist": out[:, :, :n_hist]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "dropin":
        x, c = dropin_inputs(case, seed)
        d = device()
        m = [case["m0"], case["m1"], case["m2"]][:case["dim"]]
        return {"fk": direct([torch.from_numpy(v).to(d) for v in x], torch.from_numpy(c).to(d), m)} if cheap(len(c), math.prod(m)) else None
    if kind == "plan":
        x, c = plan_inputs(case, seed)
        m = [case["m0"], case["m1"], case["m2"]][:case["dim"]]
        if not cheap(c.numel(), math.prod(m)):
            return None
        return {"fk": torch.stack([direct(x.double(), v.to(torch.complex128), m) for v in c])}
    if kind == "crystal":
        if not cheap(5 * case["cells"] ** 3 * case["frames"], crystal_modes(case["cells"], case["zones"]) ** case["dim"]):
            return None
        return exact_crystal(case, crystal_frames(case["cells"], case["frames"], seed))
    if kind == "alloy":
        return exact_alloy(case, seed)
    if kind == "spectrum":
        return exact_spectrum(case, seed)
    if kind == "maps":
        return exact_maps(case, seed)
    if kind == "sql":
        return exact_sql(case, seed)
    out = {}
    for k, (edge, frames, zones, s) in enumerate(request_list(case, seed)):
        if not cheap(5 * edge ** 3 * frames, crystal_modes(edge, zones) ** 3 * case["jobs"]):
            return None
        bins = min(4, hann_sizes(frames)[1]) if frames >= 4 else 0
        got = exact_crystal({"cells": edge, "zones": zones, "econst": bins}, crystal_frames(edge, frames, s))
        out["%02d" % k] = [got["sq"], got.get("sqw")]
    return out
