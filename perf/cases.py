"""The builds that a program has this library do, as measurable cases.

A case names a mesh family, its size, a grid resolution, the build options and
the entry point the mesh goes through.  The families, sizes and options are
those of the repository's own workloads (svo_b200.meshgen, bench.py, tests/):
jittered icospheres and tori (closed surfaces, indexed), a torus soup with
sliver triangles (no index list), and a heightfield.  Every result is returned
whole: nodes, vertices, edges and keys as the device arrays the result owns
(no copy), as raw integers, since they are bit-exact by contract.

  entry "build"   Context.build, the mesh in device memory
  entry "each"    Context.build of several such meshes, one after another
  entry "batch"   Context.build_batch over several meshes of the batch
                  distribution (sizes and resolutions differ)
  entry "serve"   a Server: all requests submitted, then collected in
                  completion order; results borrowed until the next pass
  entry "host"    the drop-in user's path: mesh in host arrays, nodes and
                  keys read back to host arrays
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-svo_b200"))
import svo_b200  # noqa: E402

_ARRAYS = ("nodes", "vertices", "edges", "keys")


def _case(mesh, tris, res, entry="build", meshes=1, full=False, dedup=False, strict=False, vert_edge=True, keys=True,
          res_y=0, res_z=0):
    """res_y/res_z: 0 = the same as res."""
    return {"mesh": mesh, "tris": tris, "res": res, "res_y": res_y, "res_z": res_z, "entry": entry, "meshes": meshes,
            "full": full, "dedup": dedup, "strict": strict, "vert_edge": vert_edge, "keys": keys}


def listed():
    named = [
        # the smallest call: a low-polygon collision mesh at a coarse grid; launches and host waits count
        ("tiny_icosphere_320_res32", _case("icosphere", 320, 32)),
        # the first configuration of the benchmark: one ordinary model, the reference's default options
        ("icosphere_20k_res128", _case("icosphere", 20480, 128)),
        # models of different sizes one after another, the last pass's octrees still in use
        ("session_6_models", _case("mixed", 40000, 512, entry="each", meshes=6)),
        # few large triangles on a fine grid: each covers thousands of voxels
        ("icosphere_320_res512", _case("icosphere", 320, 512)),
        # strict arithmetic (a build compared with a CPU one) with real neighbour tables, on a grid that is neither a
        # cube nor a power of two
        ("torus_30k_res300x200x100_strict_full", _case("torus", 30000, 300, res_y=200, res_z=100, strict=True, full=True)),
        # unique vertex/edge/face keys for meshing, read back to host memory as their consumer does
        ("icosphere_80k_res200_dedup", _case("icosphere", 81920, 200, dedup=True)),
        # a terrain tile
        ("heightfield_1M_res1024_full", _case("heightfield", 1000000, 1024, full=True)),
        # scanned geometry without an index list, slivers among it (the benchmark's second configuration)
        ("torus_slivers_1M_soup_res512", _case("slivers", 1000000, 512)),
        # the largest build: the benchmark's headline configuration
        ("heightfield_5M_res2048_full_dedup", _case("heightfield", 4999122, 2048, full=True, dedup=True)),
        # many models at once (an asset import), sizes and resolutions mixed
        ("batch_15_meshes", _case("mixed", 80000, 512, entry="batch", meshes=15)),
        # requests of several clients over one server
        ("serve_8_requests", _case("mixed", 40000, 256, entry="serve", meshes=8)),
        # the reference's own users: host arrays in, host arrays out
        ("host_icosphere_20k_res96", _case("icosphere", 20480, 96, entry="host", vert_edge=False)),
    ]
    return [dict(c, name=n) for n, c in named]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choices(["build", "each", "batch", "serve", "host"], [0.65, 0.08, 0.1, 0.08, 0.09])[0]
    if entry in ("each", "batch", "serve"):
        n = rng.randint(2, 15 if entry == "batch" else 10)
        return _case("mixed", _log_int(rng, 2000, 80000), rng.choice([128, 256, 512]), entry=entry, meshes=n,
                     full=rng.random() < 0.2, strict=rng.random() < 0.2)
    if entry == "host":
        return _case(rng.choice(["icosphere", "torus"]), _log_int(rng, 300, 80000), _log_int(rng, 24, 128), entry=entry,
                     vert_edge=False, strict=rng.random() < 0.2)
    mesh = rng.choice(["icosphere", "torus", "slivers", "heightfield"])
    if mesh == "slivers":  # every triangle is far from its neighbours: nodes grow with the triangles
        tris, res = _log_int(rng, 2000, 1000000), _log_int(rng, 32, 512)
    elif mesh == "heightfield":
        tris, res = _log_int(rng, 2000, 4999122), _log_int(rng, 64, 2048)
    else:
        tris, res = _log_int(rng, 320, 320000), _log_int(rng, 32, 1024)
    thin = rng.random() < 0.15
    dedup = rng.random() < 0.25 and (res <= 256 or res > 1024)
    return _case(mesh, tris, res, full=rng.random() < 0.35, dedup=dedup, strict=rng.random() < 0.2,
                 vert_edge=rng.random() < 0.8, keys=rng.random() < 0.9,
                 res_y=max(8, _log_int(rng, res // 4, res)) if thin else 0,
                 res_z=max(8, _log_int(rng, res // 4, res)) if thin else 0)


# ---- meshes (points float32 [n, 3], triangles int32 [m, 3] or None), on the GPU ----

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _uniform(g, n, lo, hi):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _unit(x):
    return x / x.norm(dim=-1, keepdim=True)


def _icosphere(tris, g):
    """A subdivided icosahedron of about `tris` triangles, its radii jittered by 2%."""
    phi = (1.0 + 5.0 ** 0.5) / 2.0
    v = torch.tensor([[-1, phi, 0], [1, phi, 0], [-1, -phi, 0], [1, -phi, 0], [0, -1, phi], [0, 1, phi], [0, -1, -phi],
                      [0, 1, -phi], [phi, 0, -1], [phi, 0, 1], [-phi, 0, -1], [-phi, 0, 1]], dtype=torch.float64,
                     device="cuda")
    f = torch.tensor([[0, 11, 5], [0, 5, 1], [0, 1, 7], [0, 7, 10], [0, 10, 11], [1, 5, 9], [5, 11, 4], [11, 10, 2],
                      [10, 7, 6], [7, 1, 8], [3, 9, 4], [3, 4, 2], [3, 2, 6], [3, 6, 8], [3, 8, 9], [4, 9, 5], [2, 4, 11],
                      [6, 2, 10], [8, 6, 7], [9, 8, 1]], device="cuda")
    v = _unit(v)
    for _ in range(max(1, min(7, round(math.log(tris / 20.0, 4))))):
        a = torch.cat([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]]).sort(dim=1).values
        uniq, inv = torch.unique(a[:, 0] * v.shape[0] + a[:, 1], return_inverse=True)
        mid = _unit(v[uniq // v.shape[0]] + v[uniq % v.shape[0]])
        inv = inv + v.shape[0]
        n = f.shape[0]
        m01, m12, m20 = inv[:n], inv[n:2 * n], inv[2 * n:]
        v = torch.cat([v, mid])
        f = torch.cat([torch.stack([f[:, 0], m01, m20], 1), torch.stack([f[:, 1], m12, m01], 1),
                       torch.stack([f[:, 2], m20, m12], 1), torch.stack([m01, m12, m20], 1)])
    v = v * (1.0 + _uniform(g, (v.shape[0], 1), -0.02, 0.02))
    lo, hi = v.amin(0), v.amax(0)
    return (v - lo) / (hi - lo).max(), f


def _quads(nu, nv, wrap):
    """Two triangles per cell of an nu x nv vertex grid."""
    ku, kv = (nu, nv) if wrap else (nu - 1, nv - 1)
    i = torch.arange(ku, device="cuda")[:, None]
    j = torch.arange(kv, device="cuda")[None, :]
    i1, j1 = (i + 1) % nu, (j + 1) % nv
    a, b, c, d = i * nv + j, i1 * nv + j, i1 * nv + j1, i * nv + j1
    return torch.cat([torch.stack([a, b, c], -1).reshape(-1, 3), torch.stack([a, c, d], -1).reshape(-1, 3)])


def _torus(tris, g, big=0.35, small=0.12):
    nu = max(8, int(math.sqrt(tris / 2.0 * 1.8)))
    nv = max(4, int(tris / 2.0 / nu))
    u = (torch.arange(nu, device="cuda", dtype=torch.float64) * (2 * math.pi / nu))[:, None]
    w = (torch.arange(nv, device="cuda", dtype=torch.float64) * (2 * math.pi / nv))[None, :]
    ring = big + small * torch.cos(w)
    v = torch.stack([ring * torch.cos(u), ring * torch.sin(u), (small * torch.sin(w)).expand(nu, nv)], -1).reshape(-1, 3)
    return v + 0.5 + 0.01 * small * _normal(g, v.shape[0], 3), _quads(nu, nv, True)


def _slivers(tris, g):
    """Soup: nine tenths a torus, one tenth slivers 0.005-0.05 long, 50-500 times as long as wide."""
    v, f = _torus(tris * 9 // 10, g)
    n = max(1, tris - f.shape[0])
    c = _uniform(g, (n, 3), 0.05, 0.95)
    length, aspect = _uniform(g, (n, 1), 0.005, 0.05), _uniform(g, (n, 1), 50.0, 500.0)
    d = _unit(_normal(g, n, 3))
    e = _normal(g, n, 3)
    e = _unit(e - (e * d).sum(1, keepdim=True) * d)
    p2 = c + e * (length / aspect) + d * length * _uniform(g, (n, 1), -0.5, 0.5)
    s = torch.stack([c - d * length / 2, c + d * length / 2, p2], 1)
    return torch.cat([v[f], s]).reshape(-1, 3), None


def _heightfield(tris, g):
    """z = 0.5 + 16 sinusoids over a square vertex grid."""
    n = max(3, int(round(math.sqrt(tris / 2.0))) + 1)
    amp, wave = _uniform(g, 16, 0.0, 0.03), _uniform(g, 16, 1.0, 40.0)
    ang, phase = _uniform(g, 16, 0.0, 2 * math.pi), _uniform(g, 16, 0.0, 2 * math.pi)
    x = torch.linspace(0.0, 1.0, n, device="cuda", dtype=torch.float64)[:, None]
    y = torch.linspace(0.0, 1.0, n, device="cuda", dtype=torch.float64)[None, :]
    z = torch.full((n, n), 0.5, device="cuda", dtype=torch.float64)
    for k in range(16):
        z += amp[k] * torch.sin(wave[k] * (torch.cos(ang[k]) * x + torch.sin(ang[k]) * y) + phase[k])
    return torch.stack([x.expand(n, n), y.expand(n, n), z], -1).reshape(-1, 3), _quads(n, n, False)


_FAMILY = {"icosphere": _icosphere, "torus": _torus, "slivers": _slivers, "heightfield": _heightfield}


def _meshes(case, seed):
    """[(points, tris, res), ...] of a case.

    The shapes belong to the case, so that a case has one octree size: the seed sets the unit the model is in
    (coordinates times a power of two: exact, so the same voxels at other positions) and where its triangle and
    vertex lists start."""
    g = _gen(sum(ord(c) for c in case["mesh"]) + case["tris"])
    if case["mesh"] != "mixed":
        v, f = _FAMILY[case["mesh"]](case["tris"], g)
        res = (case["res"], case["res_y"] or case["res"], case["res_z"] or case["res"])
        found = [(v, f, res)]
    else:
        # the batch distribution: icospheres and tori, triangles log-uniform up to `tris`, resolutions
        # up to `res` in turn (the first mesh has the largest)
        found = []
        for k in range(case["meshes"]):
            u = torch.rand(3, generator=g, device="cuda").tolist()
            tris = int(math.exp(math.log(320.0) + u[0] * (math.log(case["tris"]) - math.log(320.0))))
            v, f = _icosphere(tris, g) if k % 2 else _torus(tris, g, 0.25 + 0.15 * u[1], 0.05 + 0.1 * u[2])
            found.append((v, f, max(32, case["res"] >> (k % 4))))
    scale = 2.0 ** (seed % 13 - 6)
    turn = 1 + seed * 7919 % 99991
    out = []
    for v, f, r in found:
        v = v.to(torch.float32) * scale
        if f is None:
            v = v.roll(3 * (turn % (v.shape[0] // 3)), 0)
        else:
            by = turn % v.shape[0]
            v = v.roll(by, 0)
            f = ((f + by) % v.shape[0]).to(torch.int32).roll(turn % f.shape[0], 0).contiguous()
        out.append((v.contiguous(), f, r))
    return out


# ---- a pass ----

_CTX = None


def _context():
    """The process's context: a program makes one and keeps it."""
    global _CTX
    if _CTX is None:
        _CTX = svo_b200.Context(0)
    return _CTX


def _flags(case):
    return ((svo_b200.FLAG_FULL_NEIGHBORS if case["full"] else 0) | (svo_b200.FLAG_DEDUP if case["dedup"] else 0) |
            (svo_b200.FLAG_STRICT_FP if case["strict"] else 0) | (0 if case["vert_edge"] else svo_b200.FLAG_NO_VERT_EDGE) |
            (0 if case["keys"] else svo_b200.FLAG_NO_KEYS))


def prepare(case, seed):
    meshes = _meshes(case, seed)
    if case["entry"] == "host":
        meshes = [(v.cpu().numpy(), f.cpu().numpy(), r) for v, f, r in meshes]
    state = {"case": dict(case), "meshes": meshes, "ctx": _context(), "flags": _flags(case), "host": {}}
    if case["entry"] == "serve":
        torch.cuda.synchronize()  # the server's workers read the meshes on streams of their own
        state["server"] = svo_b200.Server(state["ctx"], 6 << 30, workers=3, max_batch=64, flags=state["flags"])
        state["held"] = []
    return state


class _Array:
    """A result's device array, for torch.as_tensor; keeps the result and its owner (a server) alive."""

    def __init__(self, result, owner, ptr, shape, typestr):
        self.result, self.owner = result, owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


def _device_arrays(result, flags, owner=None):
    """Nodes (21 8-byte words each), vertices (2), edges (7 4-byte words) and keys of a result, where they lie."""
    out = {}
    for name in _ARRAYS:
        if (name in ("vertices", "edges") and flags & svo_b200.FLAG_NO_VERT_EDGE) or \
                (name == "keys" and flags & svo_b200.FLAG_NO_KEYS):
            continue
        n = getattr(result, "num_" + name)
        shape, kind = {"nodes": ((n, 21), "<i8"), "vertices": ((n, 2), "<i8"), "edges": ((n, 7), "<i4"),
                       "keys": ((n,), "<i8")}[name]
        out[name] = torch.as_tensor(_Array(result, owner, result.device_ptr(name), shape, kind), device="cuda")
    return out


def _dedup_lists(state, result):
    """The three key lists in pinned host memory that the program keeps (they have no device accessor)."""
    out = []
    for kind in range(3):
        n = svo_b200.lib().svo_result_num_dedup(result.handle, kind)
        buf = state["host"].get(kind)
        if buf is None or buf.numel() < n:
            buf = state["host"][kind] = torch.empty(n + n // 4, dtype=torch.int64, pin_memory=True)
        rc = svo_b200.lib().svo_result_copy_dedup(result.handle, kind, buf.data_ptr(), n)
        if rc != svo_b200.OK:
            raise RuntimeError("svo_result_copy_dedup: status %d" % rc)
        out.append(buf[:n])
    return out


def run(state):
    case, flags, ctx = state["case"], state["flags"], state["ctx"]
    if case["entry"] == "each":
        results = [ctx.build(*m, flags) for m in state["meshes"]]
        return {"bbox": np.stack([r.bbox for r in results]), "meshes": [_device_arrays(r, flags) for r in results]}
    if case["entry"] == "batch":
        results, _, rc = ctx.build_batch(state["meshes"], flags)
        if rc != svo_b200.OK:
            raise RuntimeError("build_batch: status %d" % rc)
        return {"bbox": np.stack([r.bbox for r in results]), "meshes": [_device_arrays(r, flags) for r in results]}
    if case["entry"] == "serve":
        server = state["server"]
        for ticket in state["held"]:
            server.release(ticket)
        state["held"] = [server.submit(*m) for m in state["meshes"]]
        got = {}
        for _ in state["held"]:
            ticket, result, status, _ = server.next()
            if status != svo_b200.OK:
                raise RuntimeError("request: status %d" % status)
            got[ticket] = result
        results = [got[t] for t in state["held"]]
        return {"bbox": np.stack([r.bbox for r in results]),
                "meshes": [_device_arrays(r, flags, server) for r in results]}
    points, tris, res = state["meshes"][0]
    result = ctx.build(points, tris, res, flags)
    out = {"bbox": result.bbox}
    if case["entry"] == "host":
        # as integer words: the records are structures
        out["nodes"] = result.nodes().view(np.int64)
        out["keys"] = result.keys().view(np.int64)
        return out
    out.update(_device_arrays(result, flags))
    if case["dedup"]:
        if case["res"] <= 256:
            out["dedup"] = _dedup_lists(state, result)
        else:
            # gigabytes that only a copy to host memory can reach: the build makes them, their sizes are
            # what a program asks for before it makes room; the smaller dedup cases return the lists
            out["dedup"] = [svo_b200.lib().svo_result_num_dedup(result.handle, k) for k in range(3)]
    return out


def work(case):
    """Each input read once, each output written once (the outputs' sizes follow from the mesh: one pass is run)."""
    state = prepare(case, 1)
    out = run(state)
    total = sum(v.nbytes + (0 if f is None else f.nbytes) for v, f, _ in state["meshes"])
    for arrays in out.get("meshes", [out]):
        for name in _ARRAYS:
            if name in arrays:
                total += arrays[name].nbytes
    total += sum(8 * x if isinstance(x, int) else x.nbytes for x in out.get("dedup", []))
    return {"bytes": total, "flops": 0}


def exact(case, seed):
    """The bounding cubes in 64 bits (the longest axis' cube around the mesh, widened by 1/10001 on each side); the
    octree's arrays are integers and bit patterns, which have to stay the same."""
    cubes = []
    for v, _, _ in _meshes(case, seed):
        lo, hi = v.double().amin(0), v.double().amax(0)
        pad = ((hi - lo).max() - (hi - lo)) / 2
        lo, hi = lo - pad, hi + pad
        eps = (hi - lo) / 10001.0
        lo, hi = lo - eps, hi + eps
        cubes.append(torch.cat([lo, hi, hi - lo]).cpu().numpy())
    if case["entry"] in ("each", "batch", "serve"):
        return {"bbox": np.stack(cubes), "meshes": None}
    return {"bbox": cubes[0], "nodes": None}
