"""Timed cases of the tree-gravity library, through its public Python binding.

Each case is one pass that a program of this library makes: a force evaluation
of a system that has just moved (load, build, walk), a walk of an active subset
between rebuilds, a replayed graph step of an ensemble, a batch of served
requests, an energy check, or the Peano-Hilbert ordering of the particles.
The models are the workloads of ics.py (Plummer sphere, galaxy, clustered
system, ensembles), drawn here on the device so that inputs are quick to make.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gizmo-public_b200"))
import ggb200  # noqa: E402

KERNEL_FAC = 2.8        # kernel radius / Plummer-equivalent softening
N_CLUMPS = 1000
DRIFT_DT = 1e-3         # drift between rebuilds, in the models' time unit
FLOPS = 20              # per interaction: offset, r^2, 1/r, force factor, accumulation, potential
# interactions per target of the reference's own tree at ErrTolForceAcc 0.001 and 2^22 particles
INTERACTIONS = {"plummer": 1400.0, "galaxy": 5880.0, "clustered": 1790.0}


def listed():
    return [
        # one of the smallest systems a server is sent: launches and latency
        dict(name="plummer_1k", call="step", model="plummer", n=1000, tol=0.001, group=32),
        # the isolated Plummer sphere at GIZMO's default tolerance
        dict(name="plummer_65k", call="step", model="plummer", n=65536, tol=0.0025, group=32),
        # the galaxy (two softenings) at an ordinary size
        dict(name="galaxy_262k", call="step", model="galaxy", n=262144, tol=0.0025, group=32),
        # the galaxy at its full size
        dict(name="galaxy_4m", call="step", model="galaxy", n=4194304, tol=0.001, group=32),
        # the clustered system at its full size, with the group size the tuner picks for it
        dict(name="clustered_16m", call="step", model="clustered", n=16777216, tol=0.0008, group=64),
        # individual timesteps: a rebuild, a drift, then the walk of a random 10% of the particles
        dict(name="clustered_4m_active", call="active", model="clustered", n=4194304, tol=0.0008, group=32,
             fraction=0.1),
        # the energy check of a snapshot: the potential-only walk
        dict(name="plummer_262k_potential", call="potential", model="plummer", n=262144, tol=0.0025, group=32),
        # GIZMO's own call: host arrays in, host arrays out, odd particle count
        dict(name="clustered_1m_host", call="host", model="clustered", n=1000003, tol=0.0008, group=32),
        # an ensemble of independent clusters stepped by one captured graph
        dict(name="ensemble_1024_graph", call="graph", model="plummer", systems=1024, smallest=256, largest=32768,
             tol=0.001, group=32),
        # a batch of requests as the server runs it: separate host arrays, asynchronous walk, results fetched
        dict(name="served_48", call="served", model="plummer", systems=48, smallest=1000, largest=65536, tol=0.001,
             group=32),
        # Peano-Hilbert keys and the key sort alone (the domain decomposition's ordering)
        dict(name="order_8m", call="order", model="clustered", n=8388608),
        dict(name="order_100k", call="order", model="plummer", n=100003),
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of its range, odd sizes as likely as even ones."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["step", "step", "step", "active", "potential", "host", "graph", "served", "order"])
    if call in ("graph", "served"):
        return dict(call=call, model="plummer", systems=_log_int(rng, 8, 1024 if call == "graph" else 48),
                    smallest=_log_int(rng, 256, 1000), largest=_log_int(rng, 4096, 32768),
                    tol=rng.choice([0.001, 0.0025]), group=rng.choice([32, 32, 64]))
    model = rng.choice(["plummer", "galaxy", "clustered"])
    if call == "order":
        return dict(call=call, model=model, n=_log_int(rng, 1000, 8388608))
    largest = {"plummer": 1000000, "galaxy": 2000000, "clustered": 8388608}[model]
    case = dict(call=call, model=model, n=_log_int(rng, 1000, min(largest, 2000000) if call == "host" else largest),
                tol=rng.choice([0.001, 0.0025]), group=rng.choice([32, 32, 64]))
    if call == "active":
        case["fraction"] = rng.choice([0.01, 0.1, 0.3])
    return case


# ------------------------------------------------------------------ models (float64, on the device)

def _rand(n, gen):
    return torch.rand(n, dtype=torch.float64, device="cuda", generator=gen)


def _sphere(n, gen):
    z, phi = 2.0 * _rand(n, gen) - 1.0, 2.0 * math.pi * _rand(n, gen)
    s = torch.sqrt(1.0 - z * z)
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), z], dim=1)


def _plummer(n, gen, rmax=20.0):
    """M = a = 1 Plummer sphere truncated at rmax."""
    u = _rand(n, gen).clamp_min(1e-12) * (rmax ** 3 / (1.0 + rmax * rmax) ** 1.5)
    return _sphere(n, gen) * torch.rsqrt(u ** (-2.0 / 3.0) - 1.0)[:, None]


def _galaxy(n, gen):
    """Hernquist halo and exponential disk, 3,000,000 : 1,194,304 particles; the disk's softening is half the halo's."""
    nh = max(1, int(round(n * 3000000 / 4194304)))
    nd = n - nh
    s = torch.sqrt(_rand(nh, gen) * (100.0 / 101.0) ** 2)
    halo = _sphere(nh, gen) * (s / (1.0 - s))[:, None]
    radius = -0.05 * (torch.log(_rand(nd, gen).clamp_min(1e-300)) + torch.log(_rand(nd, gen).clamp_min(1e-300)))
    phi = 2.0 * math.pi * _rand(nd, gen)
    z = 0.005 * torch.atanh((2.0 * _rand(nd, gen) - 1.0).clamp(-1 + 1e-12, 1 - 1e-12))
    disk = torch.stack([radius * torch.cos(phi), radius * torch.sin(phi), z], dim=1)
    mass = torch.cat([torch.full((nh,), 1.0 / nh, dtype=torch.float64, device="cuda"),
                      torch.full((nd,), 0.05 / max(nd, 1), dtype=torch.float64, device="cuda")])
    h = torch.cat([torch.full((nh,), KERNEL_FAC * 0.01, dtype=torch.float64, device="cuda"),
                   torch.full((nd,), KERNEL_FAC * 0.005, dtype=torch.float64, device="cuda")])
    return torch.cat([halo, disk]), mass, h


def _clustered(n, gen):
    """Plummer clumps of log-normal mass, centres uniform in the unit sphere, and a 20% uniform background."""
    share = 10.0 ** torch.randn(N_CLUMPS, dtype=torch.float64, device="cuda", generator=gen)
    scale = 0.01 * (share / share.mean()) ** (1.0 / 3.0)
    centre = _sphere(N_CLUMPS, gen) * (_rand(N_CLUMPS, gen) ** (1.0 / 3.0))[:, None]
    nc = int(0.8 * n)
    clump = torch.searchsorted(torch.cumsum(share / share.sum(), 0), torch.sort(_rand(nc, gen))[0])
    clump = clump.clamp_max(N_CLUMPS - 1)
    return torch.cat([centre[clump] + _plummer(nc, gen) * scale[clump][:, None],
                      _sphere(n - nc, gen) * (_rand(n - nc, gen) ** (1.0 / 3.0))[:, None]])


def _system(model, n, gen):
    """Positions, masses, kernel radii."""
    if model == "galaxy":
        return _galaxy(n, gen)
    pos = _clustered(n, gen) if model == "clustered" else _plummer(n, gen)
    eps = 1e-4 if model == "clustered" else 0.01
    one = torch.ones(n, dtype=torch.float64, device="cuda")
    return pos, one / n, one * (KERNEL_FAC * eps)


def _sizes(case):
    """Sizes of a batch's systems, evenly spread over the logarithm of their range (the same for every seed)."""
    k, lo, hi = case["systems"], case["smallest"], case["largest"]
    return [int(lo * (hi / lo) ** (((i * 0.6180339887498949) % 1.0))) for i in range(k)]


def _systems(case, gen):
    return [_system(case["model"], n, gen) for n in _sizes(case)]


def _records(pos, mass, h):
    """The library's 32-byte device records {double x, y, z; float m, h}."""
    rec = torch.empty((pos.shape[0], 4), dtype=torch.float64, device="cuda")
    rec[:, :3] = pos
    single = rec.view(torch.float32)
    single[:, 6] = mass.float()
    single[:, 7] = h.float()
    return rec


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if "systems" in case:
        return _systems(case, gen), gen
    return _system(case["model"], case["n"], gen), gen


def _active(case, gen):
    k = max(1, int(round(case["fraction"] * case["n"])))
    return torch.sort(torch.randperm(case["n"], device="cuda", generator=gen)[:k])[0].to(torch.int32)


def _cube(pos):
    """A root cube around the particles, as a caller of the key kernel has it."""
    lo, hi = pos.min(0)[0], pos.max(0)[0]
    centre = (0.5 * (lo + hi)).cpu().tolist()
    length = 1.001 * float((hi - lo).max())
    return dict(center=centre, corner=[c - 0.5 * length for c in centre], len=length)


# ------------------------------------------------------------------ a pass

_graph_stream = None


def _stream(case):
    """The stream a program runs the context on: torch's own, or a capturable one for graph steps."""
    global _graph_stream
    if case["call"] != "graph":
        return torch.cuda.current_stream().cuda_stream
    if _graph_stream is None:
        _graph_stream = torch.cuda.Stream()
    return _graph_stream.cuda_stream


def prepare(case, seed):
    call = case["call"]
    data, gen = _inputs(case, seed)
    if call == "order":
        n = case["n"]
        ids = torch.arange(n, dtype=torch.int32, device="cuda")
        state = dict(case=case, pos=data[0].contiguous(), cube=_cube(data[0]), ids=ids, vals=torch.empty_like(ids),
                     keys=torch.empty(n, dtype=torch.int64, device="cuda"))
        torch.cuda.synchronize()
        return state
    state = dict(case=case, tree=ggb200.GravityTree(group_size=case["group"]))
    tree = state["tree"]
    if call == "served":
        state["systems"] = [dict(pos=p.cpu().numpy(), mass=m.cpu().numpy(), h=h.cpu().numpy()) for p, m, h in data]
        return state
    if call == "host":
        state["host"] = [a.cpu().numpy() for a in data]
        tree.load(*state["host"])
        tree.build()
        acc, pot, _, _ = tree.evaluate(err_tol_theta=0.7)      # the start-up pass gives OldAcc
        state["old"] = np.linalg.norm(acc, axis=1)
        state["out"] = (acc, pot)
        return state
    torch.cuda.synchronize()
    tree.set_stream(_stream(case))
    if call == "graph":
        state["rec"] = torch.cat([_records(*s) for s in data])
        state["counts"] = _sizes(case)
    else:
        state["rec"], state["counts"] = _records(*data), [case["n"]]
    n = state["rec"].shape[0]
    state["acc"] = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    state["pot"] = torch.empty(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    tree.load_device(state["rec"], state["counts"])
    tree.build()
    tree.evaluate_device(state["acc"], state["pot"], err_tol_theta=0.7)     # the start-up pass gives OldAcc
    tree.synchronize()
    if call == "graph":
        tree.evaluate_device(state["acc"], state["pot"], err_tol_force_acc=case["tol"])
        tree.synchronize()
        tree.capture_step(state["acc"], state["pot"], err_tol_force_acc=case["tol"])
        return state
    state["old"] = state["acc"].norm(dim=1)
    if call == "active":
        state["active"] = _active(case, gen)
        state["vel"] = 0.5 * torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=gen)
        k = state["active"].shape[0]
        state["acc"], state["pot"] = state["acc"][:k].clone(), state["pot"][:k].clone()
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "order":
        n = case["n"]
        state["vals"].copy_(state["ids"])
        ggb200.peano_hilbert_keys(state["pos"], n, state["cube"], state["keys"])
        ggb200.radix_sort_pairs(state["keys"], state["vals"], n, key_bits=63)
        return state["keys"], state["vals"]
    tree, tol = state["tree"], case["tol"]
    if call == "graph":
        tree.launch_step()
        return state["acc"], state["pot"]
    if call == "served":
        tree.load_systems(state["systems"])
        tree.build()
        tree.evaluate_async(err_tol_theta=0.7, copy_acc=False, copy_pot=False)
        tree.evaluate_async(err_tol_force_acc=tol)
        acc, pot, _ = tree.fetch()
        return acc, pot
    if call == "host":
        tree.load(*state["host"])
        tree.build()
        acc, pot, _, _ = tree.evaluate(old_acc=state["old"], err_tol_force_acc=tol, out=state["out"])
        return acc, pot
    tree.load_device(state["rec"], state["counts"])
    if call == "active":
        tree.load_velocities(state["vel"])
    tree.build()
    if call == "potential":
        tree.evaluate_potential_device(state["pot"], d_old_acc=state["old"], err_tol_force_acc=tol)
        return state["pot"]
    if call == "active":
        tree.drift(DRIFT_DT)
        tree.evaluate_device(state["acc"], state["pot"], d_active=state["active"],
                             n_active=state["active"].shape[0], d_old_acc=state["old"], err_tol_force_acc=tol)
    else:
        tree.evaluate_device(state["acc"], state["pot"], d_old_acc=state["old"], err_tol_force_acc=tol)
    return state["acc"], state["pot"]


# ------------------------------------------------------------------ work, tolerance, exact results

def work(case):
    """Records and OldAcc in, results out; the reference tree's interactions, fewer for looser tolerances and smaller systems."""
    if case["call"] == "order":
        return dict(bytes=24 * case["n"] + 12 * case["n"], flops=0)
    sizes = _sizes(case) if "systems" in case else [case["n"]]
    nbytes = flops = 0.0
    for n in sizes:
        targets = n * case.get("fraction", 1.0)
        per = INTERACTIONS[case["model"]] * math.sqrt(0.001 / case["tol"]) * math.log2(n) / 22.0
        vel = 24 * n if case["call"] == "active" else 0
        nbytes += (32 + 8) * n + vel + (8 if case["call"] == "potential" else 32) * targets
        flops += FLOPS * targets * min(per, n - 1)
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    # A tree force is an approximation: against the direct sum it measured 1e-4 to 2.3e-3 (accelerations) and 5e-5 to
    # 2.3e-3 (potentials) in the 2-norm over these cases.  Two trees that open the same nodes differ by 32-bit
    # rounding only, but a node at its opening threshold may go either way, so the bound is the tree's own error.
    # Keys and order are whole numbers.
    return "exact" if case["call"] == "order" else {"rel": 2e-3}


# direct sums of up to this many pairs take a few seconds in float64
MAX_PAIRS = 8e10


def _direct(pos, mass, h, targets=None):
    """Direct summation in float64: accelerations and potentials without G, self term left out."""
    n = pos.shape[0]
    tg = torch.arange(n, device="cuda") if targets is None else targets.long()
    acc = torch.empty((tg.shape[0], 3), dtype=torch.float64, device="cuda")
    pot = torch.empty(tg.shape[0], dtype=torch.float64, device="cuda")
    source = torch.cat([pos, torch.ones_like(pos[:, :1])], dim=1)
    rows = max(1, int(6e7) // n)
    for b in range(0, tg.shape[0], rows):
        i = tg[b:b + rows]
        r = torch.cdist(pos[i], pos, compute_mode="donot_use_mm_for_euclid_dist")
        hp = torch.maximum(h[i][:, None], h[None, :])
        rinv = torch.where(r > 0, 1.0 / r, torch.zeros_like(r))
        p = rinv * mass[None, :]
        f = p * rinv * rinv
        near = torch.nonzero((r < hp) & (r > 0), as_tuple=True)
        hn, mn = hp[near], mass[near[1]]
        u = r[near] / hn
        inner = u < 0.5
        # cubic spline softening of kernel radius h
        wf = torch.where(inner, 32.0 / 3.0 + u * u * (32.0 * u - 38.4),
                         64.0 / 3.0 - 48.0 * u + 38.4 * u * u - 32.0 / 3.0 * u ** 3 - 1.0 / (15.0 * u ** 3))
        wp = torch.where(inner, -2.8 + u * u * (16.0 / 3.0 + u * u * (6.4 * u - 9.6)),
                         -3.2 + 1.0 / (15.0 * u) + u * u * (32.0 / 3.0 + u * (-16.0 + u * (9.6 - 32.0 / 15.0 * u))))
        f[near] = mn * wf / hn ** 3
        p[near] = -mn * wp / hn
        s = f @ source
        acc[b:b + rows] = s[:, :3] - pos[i] * s[:, 3:]
        pot[b:b + rows] = -p.sum(1)
    return acc, pot


def exact(case, seed):
    if case["call"] == "order":
        return None
    sizes = _sizes(case) if "systems" in case else [case["n"]]
    if sum(n * n * case.get("fraction", 1.0) for n in sizes) > MAX_PAIRS:
        return None
    data, gen = _inputs(case, seed)
    if "systems" in case:
        # masses and kernel radii are held in 32 bits on the device
        parts = [_direct(p, m.float().double(), h.float().double()) for p, m, h in data]
        acc, pot = torch.cat([a for a, _ in parts]), torch.cat([p for _, p in parts])
        return (acc.cpu().numpy(), pot.cpu().numpy()) if case["call"] == "served" else (acc, pot)
    pos, mass, h = data[0], data[1].float().double(), data[2].float().double()
    if case["call"] == "active":
        active = _active(case, gen)
        vel = 0.5 * torch.randn((case["n"], 3), dtype=torch.float64, device="cuda", generator=gen)
        return _direct(pos + vel * DRIFT_DT, mass, h, active)
    acc, pot = _direct(pos, mass, h)
    if case["call"] == "potential":
        return pot
    return (acc.cpu().numpy(), pot.cpu().numpy()) if case["call"] == "host" else (acc, pot)
