"""The work users of the cuda methods have them do, as cases that can be timed.

Every case goes through a public entry point: `cuda.BruteForce` / `cuda.BarnesHut`
`.compute` on host arrays, or the C ABI on device buffers, as a program does that keeps
its bodies resident. Sizes are the workloads of bench.py and the tests, or odd sizes of
the same ranges; bodies are drawn on the GPU from the seed with the distributions of
`particular_gb300.ics`.

A program creates its CudaResources once: cases share one per kind. A case that replays a
CUDA graph, or walks a kept tree, holds the resources whose graph or tree that is.
"""
import ctypes
import math

import numpy as np
import torch

from particular_gb300 import Acceleration, AccelerationSoftened, CudaResources, cuda
from particular_gb300 import _native as N

DEV = "cuda"


def listed():
    return [
        # One evaluation of a small cluster from host arrays: launches, copies, latency.
        {"name": "bf_host_1024", "kind": "bf_host", "n": 1024, "soft": 1e-3},
        # All pairs of a Plummer sphere, bodies resident: the FP32 pipe.
        {"name": "bf_plummer_131072", "kind": "bf", "n": 131072, "m": 0, "soft": 0.01},
        # Massless test particles in the field of a few thousand massive bodies
        # (an Ordered storage), unsoftened and checked.
        {"name": "bf_test_particles", "kind": "bf", "n": 1000003, "m": 3001, "soft": 0.0},
        # The reference's own f32 sum, bit for bit (regression runs against the CPU).
        {"name": "bf_exact_10007", "kind": "bf_exact", "n": 10007, "soft": 0.01},
        # f64 bodies (glam DVec3), all pairs: orbits that need double.
        {"name": "bf_dvec3_6007", "kind": "bf_dvec3", "n": 6007, "soft": 0.01},
        # The reference's criterion benchmark: a small tree from host arrays, unsoftened.
        {"name": "bh_host_10000", "kind": "bh_host", "n": 10000, "theta": 0.7, "soft": 0.0},
        # The default method (the reference's rule) on a galaxy of a million bodies.
        {"name": "bh_reference_1048576", "kind": "bh", "n": 1048576, "theta": 0.5, "flags": 0, "soft": 0.01},
        # The fast accurate configuration at the largest size: quadrupoles, group walk,
        # local expansion, error-bound opening.
        {"name": "bh_error_bound_4194304", "kind": "bh", "n": 4194304, "theta": 2.0,
         "flags": N.PT_BH_QUADRUPOLE | N.PT_BH_GROUP | N.PT_BH_LOCAL | N.PT_BH_RELATIVE, "soft": 0.01},
        # f64 bodies on the tree, from host arrays.
        {"name": "bh_dvec3_50021", "kind": "bh_dvec3", "n": 50021, "theta": 0.5, "soft": 0.01},
        # Ten leapfrog steps of a galaxy, tree rebuilt each step, one CUDA graph.
        {"name": "leapfrog_bh_131072", "kind": "leapfrog", "n": 131072, "method": "bh", "theta": 0.8,
         "flags": 0, "steps": 10, "soft": 0.01},
        # A thousand small clusters of uneven size advanced together.
        {"name": "ensemble_1024", "kind": "ensemble", "systems": 1024, "lo": 64, "hi": 8192, "steps": 10,
         "soft": 0.01},
        # A tree built once, walked for probe points that are not in it.
        {"name": "tree_probe_100003", "kind": "tree", "n": 100003, "m": 1048576, "theta": 0.6,
         "flags": N.PT_BH_QUADRUPOLE | N.PT_BH_GROUP, "soft": 0.01},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bf_host", "bf", "bf_test", "bf_exact", "bf_dvec3", "bh_host", "bh", "bh_error_bound",
                       "bh_dvec3", "leapfrog", "ensemble", "tree"])
    soft = rng.choice([0.0, 0.003, 0.01, 0.05])
    if kind == "bf_host":
        return {"kind": kind, "n": _log_int(rng, 2, 8192), "soft": soft}
    if kind == "bf":
        return {"kind": kind, "n": _log_int(rng, 1024, 131072), "m": 0, "soft": soft}
    if kind == "bf_test":
        return {"kind": "bf", "n": _log_int(rng, 5000, 1000003), "m": _log_int(rng, 3, 4096), "soft": soft}
    if kind == "bf_exact":
        return {"kind": kind, "n": _log_int(rng, 64, 20000), "soft": soft}
    if kind == "bf_dvec3":
        return {"kind": kind, "n": _log_int(rng, 64, 6007), "soft": soft}
    if kind == "bh_host":
        return {"kind": kind, "n": _log_int(rng, 500, 65536), "theta": rng.uniform(0.3, 1.0), "soft": soft}
    if kind == "bh":
        flags = rng.choice([0, N.PT_BH_QUADRUPOLE, N.PT_BH_GROUP, N.PT_BH_QUADRUPOLE | N.PT_BH_GROUP,
                            N.PT_BH_QUADRUPOLE | N.PT_BH_GROUP | N.PT_BH_LOCAL])
        return {"kind": kind, "n": _log_int(rng, 65536, 1048576), "theta": rng.uniform(0.45, 0.9), "flags": flags,
                "soft": soft}
    if kind == "bh_error_bound":
        return {"kind": "bh", "n": _log_int(rng, 131072, 4194304), "theta": rng.choice([1.0, 1.5, 2.0]),
                "flags": N.PT_BH_QUADRUPOLE | N.PT_BH_GROUP | N.PT_BH_LOCAL | N.PT_BH_RELATIVE, "soft": 0.01}
    if kind == "bh_dvec3":
        return {"kind": kind, "n": _log_int(rng, 500, 50021), "theta": rng.uniform(0.45, 0.9), "soft": soft}
    if kind == "leapfrog":
        if rng.random() < 0.3:
            return {"kind": kind, "n": _log_int(rng, 512, 32768), "method": "bf", "theta": 0.0, "flags": 0,
                    "steps": rng.randint(2, 10), "soft": 0.01}
        return {"kind": kind, "n": _log_int(rng, 4096, 131072), "method": "bh", "theta": rng.uniform(0.6, 1.0),
                "flags": rng.choice([0, N.PT_BH_QUADRUPOLE | N.PT_BH_GROUP]), "steps": rng.randint(2, 10),
                "soft": 0.01}
    if kind == "ensemble":
        return {"kind": kind, "systems": _log_int(rng, 32, 1024), "lo": 64, "hi": _log_int(rng, 512, 8192),
                "steps": rng.randint(2, 10), "soft": rng.choice([0.01, 0.05])}
    return {"kind": "tree", "n": _log_int(rng, 1000, 100003), "m": _log_int(rng, 65536, 1048576),
            "theta": rng.uniform(0.5, 0.9), "flags": rng.choice([0, N.PT_BH_QUADRUPOLE | N.PT_BH_GROUP]),
            "soft": 0.01}


# ---- bodies ------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _directions(g, n):
    z = _uniform(g, -1.0, 1.0, n)
    phi = _uniform(g, 0.0, 2.0 * math.pi, n)
    s = torch.sqrt(1.0 - z * z)
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), z], 1)


def _plummer(g, n, a, mass):
    """Positions and velocities of a Plummer sphere; a and mass may be per body. The speed
    fraction q has density q^2 (1 - q^2)^(7/2): q^2 is Beta(3/2, 9/2), from squared normals."""
    u = torch.clamp(_uniform(g, 0.0, 0.999, n), min=1e-12)
    r = a / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
    z = torch.randn(12, n, generator=g, device=DEV, dtype=torch.float64).square_()
    q = torch.sqrt(z[:3].sum(0) / z.sum(0))
    v = q * math.sqrt(2.0) * (1.0 + (r / a) ** 2) ** -0.25 * (mass / a) ** 0.5
    return _directions(g, n) * r[:, None], _directions(g, n) * v[:, None]


def _bulge_disk(g, n):
    """70% Plummer bulge (a = 0.5) and 30% exponential disk (scale length 2, height 0.05) on
    circular orbits; equal masses summing to 1."""
    nb = int(round(0.7 * n))
    nd = n - nb
    xb, vb = _plummer(g, nb, 0.5, nb / n)
    R = -2.0 * torch.log(torch.clamp(_uniform(g, 0.0, 1.0, nd) * _uniform(g, 0.0, 1.0, nd), min=1e-300))
    phi = _uniform(g, 0.0, 2.0 * math.pi, nd)
    z = 0.05 * torch.atanh(torch.clamp(_uniform(g, -1.0, 1.0, nd), -1 + 1e-12, 1 - 1e-12))
    c, s = torch.cos(phi), torch.sin(phi)
    xd = torch.stack([R * c, R * s, z], 1)
    x = torch.cat([xb, xd])
    r = x.square().sum(1).sqrt()
    inside = torch.empty(n, device=DEV, dtype=torch.float64)
    inside[torch.argsort(r)] = torch.arange(1, n + 1, device=DEV, dtype=torch.float64) / n
    vc = torch.sqrt(inside[nb:] / torch.clamp(r[nb:], min=1e-6))
    vd = torch.stack([-s * vc, c * vc, torch.zeros_like(vc)], 1)
    return x, torch.cat([vb, vd]), torch.full((n,), 1.0 / n, device=DEV, dtype=torch.float64)


def _rows(x, w, dtype=torch.float32):
    return torch.cat([x, w.reshape(-1, 1).expand(x.shape[0], 1)], 1).to(dtype).contiguous()


def _sizes(case):
    """The systems' sizes: log-uniform between lo and hi, in no order, the case's own."""
    u = np.linspace(math.log(case["lo"]), math.log(case["hi"]), case["systems"])
    return np.random.RandomState(case["systems"]).permutation(np.rint(np.exp(u)).astype(np.int64))


def _bodies(case, seed):
    """The case's bodies as (targets, sources, velocities); sources None: the targets."""
    g = _generator(seed)
    kind = case["kind"]
    if kind == "bf_host":  # uniform cube, masses in [0.5, 1.5]
        x, w = _uniform(g, -1.0, 1.0, case["n"], 3), _uniform(g, 0.5, 1.5, case["n"])
        return _rows(x, w), None, None
    if kind == "bh_host":  # the criterion benchmark's cube
        x, w = _uniform(g, -5e3, 5e3, case["n"], 3), _uniform(g, 1e3, 1e9, case["n"])
        return _rows(x, w), None, None
    if kind in ("bf", "bf_exact", "bf_dvec3"):
        n, m = case["n"], case.get("m", 0)
        x, _ = _plummer(g, m or n, 1.0, 1.0)
        rows = _rows(x, torch.full((m or n,), 1.0 / (m or n), device=DEV, dtype=torch.float64),
                     torch.float64 if kind == "bf_dvec3" else torch.float32)
        if not m:
            return rows, None, None
        # an Ordered storage: the affecting bodies first, then massless ones
        t, _ = _plummer(g, n - m, 2.0, 1.0) if n > m else (x[:0], None)
        return torch.cat([rows, _rows(t, torch.zeros(1, device=DEV, dtype=torch.float64))])[:n].contiguous(), rows, None
    if kind == "ensemble":
        sizes = torch.from_numpy(_sizes(case)).to(DEV)
        k = torch.repeat_interleave(torch.arange(case["systems"], device=DEV), sizes)
        a = _uniform(g, 0.5, 2.0, case["systems"])[k]
        x, v = _plummer(g, int(sizes.sum()), a, torch.ones_like(a))
        return _rows(x, 1.0 / sizes[k].double()), None, _rows(v, torch.zeros(1, device=DEV, dtype=torch.float64))
    if kind == "tree":
        x, _, w = _bulge_disk(g, case["m"])
        t, _ = _plummer(g, case["n"], 1.0, 1.0)
        return _rows(t, torch.zeros(1, device=DEV, dtype=torch.float64)), _rows(x, w), None
    x, v, w = _bulge_disk(g, case["n"])
    return (_rows(x, w, torch.float64 if kind == "bh_dvec3" else torch.float32), None,
            _rows(v, torch.zeros(1, device=DEV, dtype=torch.float64)))


# ---- a program's state and its calls --------------------------------------------

_shared = {}


def _new_resources():
    """Resources that enqueue on the program's one stream, in order with its other work."""
    if "stream" not in _shared:
        _shared["stream"] = torch.cuda.Stream()
    res = CudaResources(0)
    res.set_stream(_shared["stream"].cuda_stream)
    return res


def _resources(kind):
    if kind not in _shared:
        _shared[kind] = _new_resources()
    return _shared[kind]


def _interaction(soft):
    return AccelerationSoftened(soft) if soft else Acceleration.checked()


DT = 1e-3


def prepare(case, seed):
    L, kind = N.lib(), case["kind"]
    aff, src, vel = _bodies(case, seed)
    soft = case["soft"]
    s = {"case": case, "aff": aff, "src": aff if src is None else src}
    own = kind in ("leapfrog", "ensemble", "tree")  # it keeps a graph or a tree
    s["res"] = _new_resources() if own else _resources(kind)
    h = s["res"].handle
    if kind in ("bf_host", "bh_host", "bh_dvec3"):
        s["aff"] = aff.cpu().numpy()
        if kind == "bf_host":
            s["method"] = cuda.BruteForce(s["res"], _interaction(soft))
        else:
            s["method"] = cuda.BarnesHut(case["theta"], s["res"], _interaction(soft), dvec3=kind == "bh_dvec3")
        return s
    s["out"] = torch.empty(aff.shape[0], 3, device=DEV, dtype=aff.dtype)
    if kind == "bh" and case["flags"] & N.PT_BH_RELATIVE:
        N.check(L.pt_bh_set_relative_alpha(h, 2.75e-3))
        N.check(L.pt_bh_set_relative_monopole(h, 0.15))
        N.check(L.pt_bh_set_local_ratio(h, 0.11))
    elif kind == "bh":
        N.check(L.pt_bh_set_local_ratio(h, 0.1))
    torch.cuda.synchronize()
    if kind == "leapfrog":
        s["vel"] = vel
        s["m"] = N.PT_METHOD_BARNES_HUT if case["method"] == "bh" else N.PT_METHOD_BRUTE_FORCE
        if case["method"] == "bh":
            N.check(L.pt_bh_accel_f32_device(h, aff.data_ptr(), aff.shape[0], aff.data_ptr(), aff.shape[0],
                                             case["theta"], soft, case["flags"], s["out"].data_ptr()))
        else:
            N.check(L.pt_bf_accel_f32_device(h, aff.data_ptr(), aff.shape[0], aff.data_ptr(), aff.shape[0], soft, 1,
                                             case["flags"], s["out"].data_ptr()))
    elif kind == "ensemble":
        s["vel"] = vel
        s["offsets"] = _offsets(case)
        s["optr"] = s["offsets"].ctypes.data_as(ctypes.c_void_p)
    elif kind == "tree":
        N.check(L.pt_bh_build_device(h, src.data_ptr(), src.shape[0], None))
    return s


def _offsets(case):
    return np.concatenate([[0], np.cumsum(_sizes(case))]).astype(np.uint32)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind in ("bf_host", "bh_host", "bh_dvec3"):
        return state["method"].compute(state["aff"])
    L, h = N.lib(), state["res"].handle
    aff, src, out, soft = state["aff"], state["src"], state["out"], case["soft"]
    n, m = aff.shape[0], src.shape[0]
    if kind == "bf":
        N.check(L.pt_bf_accel_f32_device(h, aff.data_ptr(), n, src.data_ptr(), m, soft, 1, 0, out.data_ptr()))
    elif kind == "bf_exact":
        N.check(L.pt_bf_accel_f32_device(h, aff.data_ptr(), n, src.data_ptr(), m, soft, 1, N.PT_BF_EXACT,
                                         out.data_ptr()))
    elif kind == "bf_dvec3":
        N.check(L.pt_bf_accel_dvec3_device(h, aff.data_ptr(), n, src.data_ptr(), m, soft, 1, out.data_ptr()))
    elif kind == "bh":
        N.check(L.pt_bh_accel_f32_device(h, aff.data_ptr(), n, src.data_ptr(), m, case["theta"], soft, case["flags"],
                                         out.data_ptr()))
    elif kind == "tree":
        N.check(L.pt_bh_walk_device(h, aff.data_ptr(), n, case["theta"], soft, case["flags"], out.data_ptr()))
    elif kind == "leapfrog":
        N.check(L.pt_leapfrog_device(h, aff.data_ptr(), state["vel"].data_ptr(), out.data_ptr(), n, DT, case["steps"],
                                     state["m"], case["theta"], soft, case["flags"], 1))
        return [aff, state["vel"], out]
    else:
        N.check(L.pt_ensemble_run(h, state["optr"], case["systems"], aff.data_ptr(), state["vel"].data_ptr(), DT,
                                  case["steps"], soft, 1))
        return [aff, state["vel"]]
    return out


# ---- what a pass cannot do without -----------------------------------------------

def _pairs_per_body(case, n):
    """Nodes a body's walk adds up, fitted to the reference rule's counts on these galaxies
    (476 at theta 0.8 and 1288 at theta 0.5 for 20000 bodies)."""
    theta = case["theta"]
    if case.get("flags", 0) & N.PT_BH_RELATIVE:
        theta = 0.8  # the error bound opens about as much as this angle
    return min(n, 21.0 * theta ** -2.1 * math.log2(max(n, 2)))


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        s = _sizes(case).astype(np.float64)
        return {"bytes": float(64.0 * s.sum()), "flops": float(20.0 * (s * s).sum() * (case["steps"] + 1))}
    n = case["n"]
    m = case.get("m", 0) or n
    word = 8 if kind in ("bf_dvec3", "bh_dvec3") else 4
    bytes_ = word * (3.0 * n + 3.0 * n + (4.0 * m if case.get("m", 0) else n))
    if kind in ("bf", "bf_host", "bf_exact", "bf_dvec3"):
        return {"bytes": bytes_, "flops": 20.0 * n * m}
    each = 20.0 * m if case.get("method") == "bf" else 20.0 * _pairs_per_body(case, m)
    steps = case.get("steps", 1)
    if kind == "leapfrog":
        bytes_ = 4.0 * n * (7 + 9)  # bodies and velocities in; bodies, velocities and accelerations out
    return {"bytes": bytes_, "flops": each * n * steps}


# ---- the same in 64 bits -----------------------------------------------------------

def _accel64(t, s, eps):
    """All-pairs accelerations of t (n, >= 3) from s (m, 4) in double; coincident pairs add nothing."""
    out = torch.empty(t.shape[0], 3, device=DEV, dtype=torch.float64)
    x, y, z, w = (s[:, k][None, :] for k in range(4))
    step = max(1, (1 << 26) // max(1, s.shape[0]))
    for a in range(0, t.shape[0], step):
        b = min(t.shape[0], a + step)
        dx, dy, dz = x - t[a:b, 0:1], y - t[a:b, 1:2], z - t[a:b, 2:3]
        r2 = dx * dx
        r2.addcmul_(dy, dy).addcmul_(dz, dz)
        f = torch.rsqrt(r2 + eps * eps) if eps else torch.where(r2 > 0, torch.rsqrt(r2), torch.zeros_like(r2))
        f = f * f * f * w
        out[a:b, 0], out[a:b, 1], out[a:b, 2] = (f * dx).sum(1), (f * dy).sum(1), (f * dz).sum(1)
    return out


def exact(case, seed):
    kind = case["kind"]
    eps = case["soft"] if kind in ("bf_dvec3", "bh_dvec3") else float(np.float32(case["soft"]))
    if kind == "ensemble":
        offsets = _offsets(case).astype(np.int64)
        evals, pairs = case["steps"] + 1, float((np.diff(offsets).astype(np.float64) ** 2).sum())
    else:
        evals = case["steps"] + 1 if kind == "leapfrog" else 1
        pairs = float(case["n"]) * (case.get("m", 0) or case["n"])
    if pairs * evals > 2.5e11:
        return None
    aff, src, vel = _bodies(case, seed)
    t = aff.double()
    if evals == 1:
        a = _accel64(t, t if src is None else src.double(), eps)
        return a.cpu().numpy() if kind in ("bf_host", "bh_host", "bh_dvec3") else a
    spans = [(0, case["n"])] if kind == "leapfrog" else list(zip(offsets[:-1].tolist(), offsets[1:].tolist()))
    acc, v, dt = torch.empty_like(t[:, :3]), vel.double(), float(np.float32(DT))
    for step in range(evals):
        for a, b in spans:
            acc[a:b] = _accel64(t[a:b], t[a:b], eps)
        last = step == evals - 1
        v[:, :3] += acc * (0.5 * dt if step == 0 or last else dt)
        if not last:
            t[:, :3] += v[:, :3] * dt
    return [t, v, acc] if kind == "leapfrog" else [t, v]
