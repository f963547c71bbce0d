"""The work users have this framework do, as cases that can be timed and compared.

Seven kinds of case, each through a public entry point:

* ``section``  - sweeps of one simulation on the caller's device memory
  (``run_device``), up to L = 24 with the state on chip, beyond that streamed;
* ``command``  - one section of the ``csg`` command: ``Engine.run`` and the
  observable records of its end;
* ``batch``    - simulations of different L advanced together by a tuned
  ``Batch``, and their observables;
* ``serving``  - a burst of requests through ``Server``, until the last result
  is fetched;
* ``resume``   - what the command does at its start and end: load a
  checkpoint, take the records of that state, save a checkpoint;
* ``analysis`` - the result table of a record series on the GPU
  (``csg_analyze_records``).

A Monte Carlo pass advances its state: the next pass goes on where it ended.
Spins, energies, overlaps and histograms are whole numbers; floating values
are the records and the result tables only.
"""
import ctypes
import importlib.util
import math
import pathlib
import random
import sys
import time

import numpy as np
import torch

_PKG = pathlib.Path(__file__).resolve().parent.parent / "spin-glass_b200"


def _package():
    if "spin_glass_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            "spin_glass_b200", _PKG / "__init__.py", submodule_search_locations=[str(_PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["spin_glass_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["spin_glass_b200"]


csg = _package()

# a device buffer of each accumulator csg_device_obs can take: name, dtype, shape
_OBS = [("e_sum", torch.int64, "ctx"), ("m_sum", torch.int64, "ctx"), ("q_sum", torch.int64, "tx"),
        ("q2_sum", torch.int64, "tx"), ("q4_sum", torch.int64, "tx2"), ("hist", torch.int32, "h"),
        ("e_last", torch.int32, "ctx"), ("m_last", torch.int32, "ctx"), ("d_last", torch.int32, "tx"),
        ("swap_acc", torch.int64, "ct"), ("boundary", torch.int64, "1")]


def _section(name, L, words, copies, temps, sweeps, swap=1, meas=1, H=0.0, t_min=0.2, t_max=2.0, m=False):
    c = {"name": name, "kind": "section", "L": L, "words": words, "copies": copies, "temps": temps,
         "sweeps": sweeps, "swap": swap, "meas": meas, "H": H, "t_min": t_min, "t_max": t_max, "m": m}
    if name is None:
        del c["name"]
    return c


def listed():
    return [
        # the smallest call: a first look at one word of samples, a few sweeps
        _section("smoke_L8", 8, 1, 2, 8, 16, t_min=0.5),
        # a study of a few samples: 32 of them, exchange and measurement every sweep
        _section("plain_L12", 12, 1, 2, 16, 512, t_min=0.5),
        # the production size, exchange and measurement every sweep
        _section("production_L16", 16, 32, 2, 24, 128),
        # the production size in a field, on the command's schedule
        _section("field_L16", 16, 32, 2, 24, 256, swap=16, meas=1024, H=0.1875, t_min=0.5, t_max=8.0, m=True),
        # a ragged shape: one copy, few words, three quads, exchanges only
        _section("ragged_L20", 20, 5, 1, 12, 100, swap=4, meas=0, t_min=0.5),
        # large lattices, streamed through L2 (64 MB) and HBM (227 MB of spins)
        _section("stream_L32", 32, 8, 2, 32, 16, t_min=0.5),
        _section("stream_L48", 48, 8, 2, 32, 8, t_min=0.5),
        # one section of the csg command in its shipped configuration
        {"name": "command_L16", "kind": "command", "L": 16, "words": 64, "temps": 24, "sweeps": 1024,
         "swap": 16, "H": 0.0},
        # three lattice sizes advanced together by one graph launch
        {"name": "batch_L12_L14_L16", "kind": "batch", "members": "12:16:16,14:12:20,16:8:24",
         "sweeps": 1024, "swap": 16, "meas": 1024},
        # a burst of six requests of different sizes
        {"name": "serving_burst", "kind": "serving",
         "requests": "8:4:16:4096,10:1:24:2048,12:16:16:2048,14:6:20:1024,16:8:24:1024,16:1:32:3072"},
        # the ends of an invocation of the command: checkpoint in, records, checkpoint out
        {"name": "resume_L16", "kind": "resume", "L": 16, "words": 32, "temps": 24, "H": 0.0},
        # the table of half an invocation's records (2048 samples, 24 temperatures)
        {"name": "analysis_L16", "kind": "analysis", "L": 16, "n_meas": 128, "samples": 2048, "temps": 24},
    ]


def _updates(L, words, copies, temps, sweeps):
    return words * copies * temps * L ** 3 * sweeps


_MOST = _updates(16, 64, 2, 24, 1024)  # word updates of the largest listed case


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5))))))


def draw(rng: random.Random):
    kind = rng.choices(["section", "stream", "command", "batch", "serving", "resume", "analysis"],
                       [8, 4, 2, 2, 1, 1, 2])[0]
    if kind == "section":
        L = rng.choice([4, 6, 8, 8, 10, 10, 12, 12, 14, 14, 16, 16, 18, 20, 22, 24])
        temps = 4 * rng.randint(1, 4 if L > 16 else 8)
        words = _log_int(rng, 1, 64)
        copies = rng.choice([1, 2, 2, 2])
        field = rng.random() < 0.3
        most = max(4, _MOST // (4 * _updates(L, words, copies, temps, 1)))
        return _section(None, L, words, copies, temps, min(_log_int(rng, 4, 1500), most),
                        swap=rng.choice([1, 1, 3, 16]), meas=rng.choice([0, 1, 5, 64]),
                        H=round(rng.uniform(0.02, 1.5), 4) if field else 0.0,
                        t_min=round(rng.uniform(0.2, 0.6), 3), t_max=round(rng.uniform(1.5, 4.0), 3),
                        m=rng.random() < 0.3)
    if kind == "stream":
        L = 2 * _log_int(rng, 13, 32)
        temps, words, copies = 4 * rng.randint(1, 8), _log_int(rng, 1, 8), rng.choice([1, 2, 2, 2])
        most = max(1, _MOST // (4 * _updates(L, words, copies, temps, 1)))
        return _section(None, L, words, copies, temps, min(_log_int(rng, 1, 40), most),
                        swap=rng.choice([1, 1, 3, 16]), meas=rng.choice([0, 1, 5]),
                        H=round(rng.uniform(0.02, 1.5), 4) if rng.random() < 0.25 else 0.0,
                        t_min=round(rng.uniform(0.4, 0.8), 3), t_max=round(rng.uniform(1.5, 3.0), 3),
                        m=rng.random() < 0.3)
    if kind == "command":
        return {"kind": "command", "L": rng.choice([8, 10, 12, 14, 16]), "words": _log_int(rng, 1, 40),
                "temps": 4 * rng.randint(3, 6), "sweeps": rng.choice([256, 500, 1024]),
                "swap": rng.choice([4, 10, 16]), "H": rng.choice([0.0, 0.0625, 0.125, 0.1875])}
    if kind == "batch":
        sides = rng.sample([8, 10, 12, 14, 16], rng.randint(2, 3))
        return {"kind": "batch", "members": ",".join("%d:%d:%d" % (L, _log_int(rng, 2, 14), 4 * rng.randint(3, 6)) for L in sides),
                "sweeps": _log_int(rng, 100, 1100), "swap": rng.choice([1, 4, 16]), "meas": rng.choice([8, 64, 1024])}
    if kind == "serving":
        return {"kind": "serving", "requests": ",".join(
            "%d:%d:%d:%d" % (rng.choice([8, 10, 12, 14, 16]), _log_int(rng, 1, 12), 4 * rng.randint(4, 8),
                             _log_int(rng, 300, 2500)) for _ in range(rng.randint(3, 6)))}
    if kind == "resume":
        return {"kind": "resume", "L": rng.choice([8, 10, 12, 14, 16]), "words": _log_int(rng, 1, 24),
                "temps": 4 * rng.randint(2, 6), "H": rng.choice([0.0, 0.0625, 0.1875])}
    return {"kind": "analysis", "L": rng.choice([8, 12, 16]), "n_meas": _log_int(rng, 3, 120),
            "samples": 32 * _log_int(rng, 1, 64), "temps": rng.randint(4, 24)}


# ---------------------------------------------------------------------------
# what a user's program has in hand
# ---------------------------------------------------------------------------

def _run_seed(seed, k=0):
    return (seed * 0x9E3779B1 + 0x5EED0001 + k) & 0xFFFFFFFFFFFF


def _prepare_section(case, seed):
    L, W, C, T = case["L"], case["words"], case["copies"], case["temps"]
    cfg, betas = csg.make_config(
        L, W, C, csg.geometric_betas(T, case["t_min"], case["t_max"]), H=case["H"], seed=_run_seed(seed),
        sweeps_per_swap=case["swap"], sweeps_per_meas=case["meas"],
        flags=csg.CSG_MEASURE_M if case["m"] else 0)
    spins = torch.empty((W, C, T // 4, L ** 3, 4), dtype=torch.int32, device="cuda")
    bonds = torch.empty((W, 3, L ** 3), dtype=torch.int32, device="cuda")
    csg.init_device(cfg, spins.data_ptr(), bonds.data_ptr(), torch.cuda.current_stream().cuda_stream)
    shapes = {"ctx": (W, C, T, 32), "tx": (W, T, 32), "tx2": (W, T, 32, 2), "h": (T, L ** 3 + 1), "ct": (C, T), "1": (1,)}
    obs = {n: torch.zeros(shapes[s], dtype=d, device="cuda") for n, d, s in _OBS}
    ptrs = csg.DeviceObs(**{n: v.data_ptr() for n, v in obs.items()})
    return {"cfg": cfg, "betas": betas, "spins": spins, "bonds": bonds, "obs": obs, "ptrs": ptrs,
            "sweeps": case["sweeps"], "sweep": 0, "run": _run_section}


def _run_section(s):
    csg.run_device(s["cfg"], s["spins"].data_ptr(), s["bonds"].data_ptr(), s["ptrs"], s["sweep"], s["sweeps"],
                   torch.cuda.current_stream().cuda_stream)
    s["sweep"] += s["sweeps"]
    return {"spins": s["spins"], **s["obs"]}


def _prepare_command(case, seed):
    e = csg.Engine(case["L"], case["words"], 2, csg.reference_betas(case["temps"]), H=case["H"], seed=_run_seed(seed),
                   sweeps_per_swap=case["swap"], sweeps_per_meas=case["sweeps"], flags=csg.CSG_MEASURE_M)
    e.init_lattice()
    return {"engine": e, "sweeps": case["sweeps"], "run": _run_command}


def _run_command(s):
    s["engine"].run(s["sweeps"])
    return {"records": s["engine"].obs_records()}


def _prepare_batch(case, seed):
    members = []
    for k, m in enumerate(case["members"].split(",")):
        L, W, T = map(int, m.split(":"))
        members.append(dict(L=L, n_words=W, n_copies=2, betas=csg.geometric_betas(T, 0.2, 2.0), seed=_run_seed(seed, k),
                            sweeps_per_swap=case["swap"], sweeps_per_meas=case["meas"]))
    b = csg.Batch(members)
    for m in b.members:
        m.init_lattice()
    b.tune(16)
    return {"batch": b, "sweeps": case["sweeps"], "obs": [m.new_observables() for m in b.members], "run": _run_batch}


def _numbers(o):
    return {n: getattr(o, n) for n in ("e_sum", "q_sum", "q2_sum", "q4_sum", "hist", "e_last", "d_last", "swap_acc")}


def _run_batch(s):
    s["batch"].run(s["sweeps"])
    return [_numbers(m.observables(o)) for m, o in zip(s["batch"].members, s["obs"])]


def _prepare_serving(case, seed):
    requests = []
    for k, r in enumerate(case["requests"].split(",")):
        L, W, T, n = map(int, r.split(":"))
        requests.append(dict(n_sweeps=n, L=L, n_words=W, n_copies=2, betas=csg.geometric_betas(T, 0.2, 2.0),
                             seed=_run_seed(seed, k), sweeps_per_swap=1, sweeps_per_meas=16, meas_start=n // 2))
    return {"server": csg.Server(16 << 30, 32, 1024), "requests": requests, "run": _run_serving}


def _run_serving(s):
    ids = [s["server"].submit(**r) for r in s["requests"]]
    got = {}
    while len(got) < len(ids):
        done, _, _ = s["server"].poll()
        for i in done:
            o = s["server"].result(i)
            got[i] = {n: getattr(o, n) for n in ("e_sum", "q2_sum", "q4_sum", "hist", "e_last", "d_last", "swap_acc")}
        if not done:
            time.sleep(50e-6)
    return [got[i] for i in ids]


def _checkpoint(case, seed):
    """A checkpoint in the reference's layout: uint32 [2 * samples, N], bits 0..T-1 the
    spins by temperature, bits 26..31 the bonds -x,+x,-y,+y,-z,+z (1: ferromagnetic)."""
    L, S, T = case["L"], 32 * case["words"], case["temps"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    spins = torch.randint(0, 1 << T, (S, 2, L, L, L), generator=g, device="cuda", dtype=torch.int64)
    bond = torch.randint(0, 2, (3, S, 1, L, L, L), generator=g, device="cuda", dtype=torch.int64)
    ref = spins
    for k in range(3):  # x, y, z: the last axis is x
        ref = ref | (bond[k] << (27 + 2 * k)) | (torch.roll(bond[k], 1, dims=4 - k) << (26 + 2 * k))
    return spins, bond, ref.reshape(2 * S, L ** 3)


def _prepare_resume(case, seed):
    ref = _checkpoint(case, seed)[2].cpu().numpy().astype(np.uint32)
    e = csg.Engine(case["L"], case["words"], 2, csg.reference_betas(case["temps"]), H=case["H"], seed=_run_seed(seed),
                   sweeps_per_swap=16, sweeps_per_meas=1024, flags=csg.CSG_MEASURE_M)
    return {"engine": e, "ref": ref, "run": _run_resume}


def _run_resume(s):
    s["engine"].load_checkpoint(s["ref"], 0)
    return {"records": s["engine"].obs_records(), "checkpoint": s["engine"].save_checkpoint()}


def _records(case, seed):
    """A record series (e[2], m[2], q_0, q_1_r[3], q_1_i[3]) whose overlaps widen towards the cold end."""
    n, d, t = case["n_meas"], case["samples"], case["temps"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    rec = torch.randn((n, d, t, 11), generator=g, device="cuda")
    width = torch.linspace(0.8, 0.05, t, device="cuda").reshape(t, 1)
    level = torch.linspace(-1.7, -0.5, t, device="cuda").reshape(t, 1)
    rec[..., 0:2] = level + 0.05 * rec[..., 0:2]
    rec[..., 2:4] *= 0.1
    rec[..., 4:5] *= width
    rec[..., 5:11] *= 0.3 * width
    return rec


def _prepare_analysis(case, seed):
    return {"rec": _records(case, seed), "dims": (case["n_meas"], case["samples"], case["temps"], case["L"]),
            "run": _run_analysis}


def _run_analysis(s):
    n, d, t, L = s["dims"]
    table = np.zeros((t, 8))
    csg._check(csg.lib().csg_analyze_records(
        ctypes.c_void_p(s["rec"].data_ptr()), n, d, t, L, table.ctypes.data_as(ctypes.c_void_p),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return {"table": table}


_PREPARE = {"section": _prepare_section, "command": _prepare_command, "batch": _prepare_batch,
            "serving": _prepare_serving, "resume": _prepare_resume, "analysis": _prepare_analysis}


def prepare(case, seed):
    torch.cuda.current_device()
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

_OPS = 47  # 32-bit integer operations of one update of a 32-sample word


def _sim_work(L, W, C, T, sweeps, passes):
    """Bytes: the state in and out and the bonds, `passes` times, and the accumulators; operations: the updates."""
    words = W * C * T * L ** 3
    obs = W * C * T * 32 * 24 + (W * T * 32 * 36 + T * (L ** 3 + 1) * 4 if C == 2 else 0)
    return passes * (8 * words + 12 * W * L ** 3) + obs, _OPS * words * sweeps


def work(case):
    kind = case["kind"]
    if kind == "section":
        # a lattice that stays on chip is read and written once a call, a streamed one once a sweep
        b, f = _sim_work(case["L"], case["words"], case["copies"], case["temps"], case["sweeps"],
                         1 if case["L"] <= 24 else case["sweeps"])
    elif kind == "command":
        b, f = _sim_work(case["L"], case["words"], 2, case["temps"], case["sweeps"], 1)
        b += 32 * case["words"] * case["temps"] * 44
    elif kind in ("batch", "serving"):
        b = f = 0
        for m in case["members" if kind == "batch" else "requests"].split(","):
            v = list(map(int, m.split(":")))
            mb, mf = _sim_work(v[0], v[1], 2, v[2], v[3] if kind == "serving" else case["sweeps"], 1)
            b, f = b + mb, f + mf
    elif kind == "resume":
        S, N, T = 32 * case["words"], case["L"] ** 3, case["temps"]
        b, f = 2 * (2 * S * N * 4) + S * T * 44, 20 * case["words"] * 2 * T * N
    else:
        n = case["n_meas"] * case["samples"] * case["temps"]
        b, f = n * 44 + case["temps"] * 64, n * 18
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the floating results in 64 bits
# ---------------------------------------------------------------------------

def _exact_records(case, seed):
    """e, m, q_0 and q_1 of a checkpoint's state, by their definitions."""
    L, S, T = case["L"], 32 * case["words"], case["temps"]
    N = L ** 3
    spins, bond, _ = _checkpoint(case, seed)
    J = (2 * bond - 1).double()
    a = torch.arange(L, device="cuda", dtype=torch.float64) * (2 * math.pi / L)
    rec = torch.empty((S, T, 11), dtype=torch.float64, device="cuda")
    for t in range(T):
        s = (2 * ((spins >> t) & 1) - 1).double()
        bonds = sum(J[k] * s * torch.roll(s, -1, dims=4 - k) for k in range(3))
        m = s.sum(dim=(2, 3, 4))
        rec[:, t, 0:2] = -(bonds.sum(dim=(2, 3, 4)) + case["H"] * m) / N
        rec[:, t, 2:4] = m / N
        q = s[:, 0] * s[:, 1]
        rec[:, t, 4] = q.sum(dim=(1, 2, 3)) / N
        for k in range(3):
            plane = q.sum(dim=[d for d in (1, 2, 3) if d != 3 - k])
            rec[:, t, 5 + k] = (plane * torch.cos(a)).sum(dim=1) / N
            rec[:, t, 8 + k] = (plane * torch.sin(a)).sum(dim=1) / N
    return rec


def _exact_table(case, seed):
    """chi_0, xi_L/L, e, m and their errors: thermal means per sample, then mean and variance over samples."""
    L, d = case["L"], case["samples"]
    rec = _records(case, seed).double()
    q2 = (rec[..., 4:11] ** 2).mean(dim=0)
    e, m = rec[..., 0:2].mean(dim=(0, 3)), rec[..., 2:4].mean(dim=(0, 3))

    def moments(x):
        return x.mean(dim=0), x.var(dim=0, unbiased=False)

    (q_a, q_v), (e_a, e_v), (m_a, m_v) = moments(q2), moments(e), moments(m)
    chi0, chi0_v = q_a[:, 0], q_v[:, 0]
    chi1, chi1_v = q_a[:, 1:].sum(dim=1) / 3, q_v[:, 1:].sum(dim=1) / 3
    chif = chi0 / chi1
    chif_v = chif ** 2 * (chi0_v / chi0 ** 2 + chi1_v / chi1 ** 2)
    xi = torch.sqrt(chif - 1) / (2 * math.sin(math.pi / L)) / L
    xi_v = (xi / (2 * (chif - 1))) ** 2 * chif_v
    return torch.stack([chi0, torch.sqrt(chi0_v / d), xi, torch.sqrt(xi_v / d), e_a, torch.sqrt(e_v / d),
                        m_a, torch.sqrt(m_v / d)], dim=1)


def exact(case, seed):
    if case["kind"] == "resume":
        return {"records": _exact_records(case, seed), "checkpoint": None}
    if case["kind"] == "analysis":
        return {"table": _exact_table(case, seed)}
    return None
