"""The workloads this library's speed is measured on.

Every case goes through the public Python entry points (or the C call they wrap) the way a
program that builds octrees does: one context per program, meshes that change from call to
call.  Inputs are the repository's own synthetic families -- jittered icospheres, value-noise
heightfields and the skewed triangle soup -- made on the GPU from the seed.

Outputs are the two octree files as they are in memory: node records as 64-bit words, data
records as 32-bit words (colours and normals by bit pattern), in buffers of the program's own
that are sized once per case and zero past the octree, and the build's counts beside them.
They are whole numbers and have to stay equal bit for bit, so no case has a value in 64-bit
floating point to compare with.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import ooc_svo_builder_gb300 as ooc
from ooc_svo_builder_gb300 import tri


def listed():
    dev = {"call": "device", "limit": 2048, "payload": False, "color": "model", "levels": False}
    pay = dict(dev, payload=True)
    return [
        # the smallest useful call: an 80-triangle prop at gridsize 64, latency only
        dict(dev, name="sphere80_g64", mesh="sphere", size=1, grid=64),
        # the first benchmark workload: 20,480 triangles, svo_builder_binary -s 256
        dict(dev, name="sphere20k_g256", mesh="sphere", size=5, grid=256),
        # a small odd-sized asset with every averaged level: svo_builder -s 128 -levels -c linear
        dict(pay, name="soup3001_g128_levels", mesh="soup", size=3001, grid=128, color="linear", levels=True),
        # the headline workload: 2,093,058 triangles with colours, svo_builder -s 1024
        dict(pay, name="field1024_g1024", mesh="field", size=1024, grid=1024),
        # terrain whose vertices do not line up with the grid: 980,000 triangles, -levels -c normal
        dict(pay, name="field701_g512_levels", mesh="field", size=701, grid=512, color="normal", levels=True),
        # a payload mesh over eight partitions: svo_builder -s 2048 -l 2048
        dict(pay, name="soup300k_g2048_payload", mesh="soup", size=300_001, grid=2048),
        # the largest workload: 20M triangles, 64 partitions, svo_builder_binary -s 4096 -l 2048
        dict(dev, name="soup20M_g4096", mesh="soup", size=20_000_000, grid=4096),
        # one host mesh in, host octree out (what the command line does between its files)
        dict(pay, name="host_field512_g512", call="host", mesh="field", size=512, grid=512),
        # many uneven meshes in one call, octrees resident on the device
        {"name": "batch128", "call": "batch", "count": 128, "most": 200_000, "grid": 512},
        # a dense soup in one partition, where triangles overlap: 4M triangles, svo_builder_binary -s 1024
        dict(dev, name="soup4M_g1024", mesh="soup", size=4_000_000, grid=1024),
        # the occupancy pass alone for callers that may not allocate
        dict(dev, name="occupancy100k_g512", call="occupancy", mesh="soup", size=100_003, grid=512),
        # triangles that do not fit the device budget: read again for every group of partitions
        dict(dev, name="outofcore400k_g1024", call="stream", mesh="soup", size=400_000, grid=1024, limit=128),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(("device", "device", "device", "device", "host", "batch", "occupancy", "stream"))
    if call == "batch":
        return {"call": call, "count": _log(rng, 2, 128), "most": _log(rng, 2_000, 200_000),
                "grid": rng.choice((128, 256, 512))}
    payload = rng.random() < 0.5
    c = {"call": call, "limit": 2048, "payload": payload, "levels": rng.random() < 0.25,
         "color": rng.choice(("model", "model", "fixed", "linear", "normal"))}
    if call == "occupancy":
        c.update(mesh="soup", size=_log(rng, 500, 1_000_000), grid=rng.choice((64, 128, 256, 512, 1024)))
        return c
    if call == "stream":
        c.update(mesh="soup", size=_log(rng, 20_000, 400_000), grid=1024, limit=128)
        return c
    c["mesh"] = rng.choice(("sphere", "field", "soup"))
    if c["mesh"] == "sphere":
        c.update(size=rng.randint(1, 6), grid=rng.choice((64, 128, 256, 512, 1024)))
    elif c["mesh"] == "field":
        c.update(size=_log(rng, 33, 1025 if call == "device" else 513), grid=rng.choice((128, 256, 512, 1024)))
    else:
        c["grid"] = rng.choice((64, 128, 256, 512, 1024, 2048, 4096) if call == "device" else (64, 256, 512))
        most = 100_000 if call == "host" else (600_000 if payload else 4_000_000)
        c["size"] = _log(rng, 200, most)
        if c["grid"] >= 256 and rng.random() < 0.25:  # a low memory limit: 8 partitions
            c["limit"] = c["grid"] ** 3 // (1 << 20) // 8
    return c


# ---- inputs: [T, 9] or [T, 21] float32 records on the GPU, from the seed alone ----

def _records(v0, v1, v2, colors=None):
    parts = [v0, v1, v2]
    if colors is not None:
        n = torch.linalg.cross(v0 - v1, v1 - v2)
        parts += [n / n.norm(dim=1, keepdim=True).clamp_min(1e-20), *colors]
    return torch.cat([p.float() for p in parts], 1).contiguous()


def _sphere(subdiv, payload, seed):
    t = tri.icosphere_tris(subdiv, radius=0.4, jitter=0.002, seed=seed, payload=payload)
    return torch.from_numpy(t).cuda()


def _field(n, payload, g):
    x = torch.linspace(0.0, 1.0, n, device="cuda", dtype=torch.float64)
    X, Y = torch.meshgrid(x, x, indexing="ij")
    H = torch.zeros_like(X)
    for o, f in enumerate((4, 8, 16, 32)):
        lat = torch.rand((f + 1, f + 1), device="cuda", dtype=torch.float64, generator=g)
        i = (x * f).long().clamp_max(f - 1)
        s = x * f - i
        s = s * s * (3 - 2 * s)
        a, b = lat[i][:, i], lat[i + 1][:, i]
        c, d = lat[i][:, i + 1], lat[i + 1][:, i + 1]
        sx, sy = s[:, None], s[None, :]
        H += 0.5 ** o * ((a * (1 - sx) + b * sx) * (1 - sy) + (c * (1 - sx) + d * sx) * sy)
    P = torch.stack([X, Y, 0.3 + 0.15 * H], -1).reshape(-1, 3).float()
    idx = torch.arange(n * n, device="cuda").reshape(n, n)
    a, b = idx[:-1, :-1].reshape(-1), idx[1:, :-1].reshape(-1)
    c, d = idx[:-1, 1:].reshape(-1), idx[1:, 1:].reshape(-1)
    F = torch.cat([torch.stack([a, b, d], 1), torch.stack([a, d, c], 1)])
    col = torch.rand((n * n, 3), device="cuda", generator=g) if payload else None
    return _records(*(P[F[:, k]] for k in range(3)), None if col is None else [col[F[:, k]] for k in range(3)])


def _unit(n, g):
    u = torch.randn((n, 3), device="cuda", generator=g)
    return u / u.norm(dim=1, keepdim=True)


def _soup(T, grid, payload, g, spheres=200):
    """Half small triangles on spheres, half log-normal edges (median 4 voxels, sigma 1, at most 512)."""
    u = 1.0 / grid
    ns = T // 2
    r = lambda *s: torch.rand(s, device="cuda", generator=g)  # noqa: E731
    centre, radius = 0.2 + 0.6 * r(spheres, 3), 0.01 + 0.19 * r(spheres, 1)
    which = torch.randint(0, spheres, (ns,), device="cuda", generator=g)
    dirs = _unit(ns, g)
    pos = centre[which] + dirs * radius[which]
    axis = torch.zeros_like(dirs)
    flat = dirs[:, 0].abs() < 0.9
    axis[:, 0], axis[:, 1] = flat.float(), (~flat).float()
    t1 = torch.linalg.cross(dirs, axis)
    t1 = t1 / t1.norm(dim=1, keepdim=True)
    t2 = torch.linalg.cross(dirs, t1)
    edge, ang = (0.2 + 0.8 * r(ns, 1)) * (u / math.sqrt(3.0)), 2 * math.pi * r(ns, 1)
    small = [pos + (torch.cos(ang + k * 2 * math.pi / 3) * t1 + torch.sin(ang + k * 2 * math.pi / 3) * t2) * edge
             for k in range(3)]
    nb = T - ns
    c = r(nb, 3)
    L = torch.clamp_max(4.0 * torch.exp(torch.randn((nb, 1), device="cuda", generator=g)), 512.0) * (u / 2)
    v = [torch.cat([small[k], c + _unit(nb, g) * L]).clamp_(-0.5, 1.5) for k in range(3)]
    perm = torch.randperm(T, device="cuda", generator=g)
    v = [x[perm] for x in v]
    return _records(*v, [r(T, 3) for _ in range(3)] if payload else None)


def _mesh(kind, size, grid, payload, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "sphere":
        return _sphere(size, payload, seed)
    if kind == "field":
        return _field(size, payload, g)
    return _soup(size, grid, payload, g)


def _many(case):
    """(mesh kind, size, gridsize, payload) of every mesh of a batch: log-uniform triangle counts, half
    spheres and half soups, gridsizes and modes mixed."""
    count = case["count"]
    rng = np.random.default_rng(count)
    grids = [s for s in (64, 128, 256, 512) if s <= case["grid"]]
    T = np.exp(np.linspace(math.log(64), math.log(case["most"]), count))[rng.permutation(count)]
    N = np.resize(grids, count)[rng.permutation(count)]
    out = []
    for i in range(count):
        payload, sphere = bool(rng.integers(0, 2)), rng.random() < 0.5
        if sphere:
            s = int(np.clip(np.floor(np.log(max(T[i], 80) / 20.0) / np.log(4.0)), 1, 6))
            out.append(("sphere", s, int(N[i]), payload))
        else:
            out.append(("soup", int(T[i]), int(N[i]), payload))
    return out


# ---- state, run ----

class _DeviceBytes:
    """Library-owned device memory as a CUDA array; keeps its context alive."""

    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 3}


class _Sink:
    """An application's sink: both files gathered in host memory of its own."""

    def __init__(self, nodes, data):
        self.files = [np.zeros((nodes, 3), np.int64), np.zeros((data, 8), np.int32)]
        self.n = [0, 0]
        self.cb = ooc.SINK(self._take)

    def _take(self, user, kind, ptr, n):
        f = self.files[kind]
        if self.n[kind] + n > f.nbytes:
            return 1
        ctypes.memmove(f.ctypes.data + self.n[kind], ptr, n)
        self.n[kind] += n
        return 0


def _counts(info):
    return [info["n_nodes"], info["n_data"], info["n_filled"]]


def prepare(case, seed):
    call = case["call"]
    s = {"call": call}
    if call == "batch":
        many = _many(case)
        s["meshes"] = [_mesh(k, size, N, pay, seed * 131 + i).cpu().pin_memory()
                       for i, (k, size, N, pay) in enumerate(many)]
        s["builder"] = ooc.Builder(0)
        arr = (ooc.Mesh * len(many))()
        for m, t, (_, _, N, pay) in zip(arr, s["meshes"], many):
            m.tris, m.n_tris, m.params = t.data_ptr(), t.shape[0], ooc.make_params(N, 2048, geometry_only=not pay)
        s["array"], s["infos"] = arr, (ooc.BuildInfo * len(many))()
        room = sum(n * 24 + d * 32 + 512 for n, d in (_room(*m, False) for m in many))
        s["arena"] = torch.zeros(room // 8, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        return s
    mesh = (case["mesh"], case["size"], case["grid"], case["payload"])
    t = _mesh(*mesh, seed)
    s["params"] = ooc.make_params(case["grid"], case["limit"], geometry_only=not case["payload"],
                                  color=case["color"], levels=case["levels"])
    if call == "occupancy":
        s["tris"] = t
        s["bits"] = torch.empty(max(1, case["grid"] ** 3 // 32), dtype=torch.int32, device="cuda")
        return s
    s["builder"] = ooc.Builder(0)
    nodes, data = _room(*mesh, case["levels"])
    if call == "device":
        s["tris"] = t
        s["nodes"] = torch.zeros((nodes, 3), dtype=torch.int64, device="cuda")
        s["data"] = torch.zeros((data, 8), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()  # the build runs on the context's own stream
        return s
    s["tris"] = t.cpu().pin_memory()
    s["sink"] = _Sink(nodes, data)
    if call == "stream":
        s["builder"].set_stream_budget(s["tris"].nbytes * 7 // 10)
    return s


def run(state):
    call = state["call"]
    if call == "device":
        b, t = state["builder"], state["tris"]
        info = b.build_device(t.data_ptr(), t.shape[0], state["params"])
        nodes, data = b.result_device()  # valid until the context's next build: the program keeps a copy
        state["nodes"][:info["n_nodes"]].copy_(
            torch.as_tensor(_DeviceBytes(nodes, (info["n_nodes"], 3), "<i8", b), device="cuda"))
        state["data"][:info["n_data"]].copy_(
            torch.as_tensor(_DeviceBytes(data, (info["n_data"], 8), "<i4", b), device="cuda"))
        return [state["nodes"], state["data"], *_counts(info)]
    if call in ("host", "stream"):
        t, sink = state["tris"], state["sink"]
        sink.n = [0, 0]
        info = state["builder"].build_ptr(t.data_ptr(), t.shape[0], state["params"], sink.cb)
        return [*sink.files, *_counts(info)]
    if call == "batch":
        a = state["arena"]
        arena = ooc.DeviceArena(a.data_ptr(), a.numel() * 8, 0)
        state["builder"].build_batch_device_ptrs(state["array"], len(state["meshes"]), arena, state["infos"])
        return [a, np.array([[i.n_nodes, i.n_data, i.n_filled] for i in state["infos"]], np.int64)]
    t, bits = state["tris"], state["bits"]
    rc = ooc.voxelize_occupancy_noalloc(state["params"], t.data_ptr(), t.shape[0], bits.data_ptr(), bits.numel(),
                                        torch.cuda.current_stream().cuda_stream)
    if rc != ooc.OOC_OK:
        raise RuntimeError("ooc_voxelize_occupancy_noalloc: %d" % rc)
    return bits


# ---- sizes: estimates, from builds of these meshes ----

def _size(kind, size, grid):
    """(triangles, filled voxels, nodes) of a mesh: 1.55 voxels per unit of a sphere's area, 1.72 per
    cell of a heightfield's floor, 20.4 per soup triangle (less where they overlap), and the nodes
    above them."""
    if kind == "sphere":
        T, filled = 20 * 4 ** size, 1.55 * 4 * math.pi * 0.16 * grid * grid
    elif kind == "field":
        T, filled = 2 * (size - 1) ** 2, 1.72 * grid * grid
    else:
        T, cells = size, float(grid) ** 3
        filled = cells * -math.expm1(-20.4 * size / cells)
    return T, filled, filled * (1.35 if kind != "soup" else 1.65 - 0.5 * filled / grid ** 3)


def _room(kind, size, grid, payload, levels):
    """Node and data records a program makes room for."""
    _, filled, nodes = _size(kind, size, grid)
    nodes = int(min(1.25 * nodes + 100_000, grid ** 3 * 8 // 7 + 64))
    return nodes, 2 + (nodes if levels else int(min(1.25 * filled + 100_000, grid ** 3)) if payload else 0)


def work(case):
    """Bytes a pass cannot do without: the triangles read once, both octree files written once."""
    if case["call"] == "batch":
        meshes, levels = _many(case), False
    else:
        meshes, levels = [(case["mesh"], case["size"], case["grid"], case["payload"])], case["levels"]
    total = 0.0
    for kind, size, grid, payload in meshes:
        T, filled, nodes = _size(kind, size, grid)
        if case["call"] == "occupancy":  # vertices only, and the bitfield
            total += T * 36 + grid ** 3 / 8
            continue
        records = (filled if payload else 0) + (nodes - filled if levels else 0)
        total += T * (84 if payload else 36) + nodes * 24 + records * 32
    return {"bytes": total, "flops": 0}


def exact(case, seed):
    return None
