"""What the decoder is measured on: the calls that programs using it make.

Every case goes through the public Python API (``ParaDeltaV5GpuDecoder``,
``BatchDecoder``, ``DecodeServer``, ``cull_meshlets``), on streams that this
package's encoder writes from seeded meshes: terrain (a heightfield of six
octaves of value noise, the regular grids of ``bench.py`` and the tests),
displaced spheres with shuffled vertices (scan-like, closed) and tori.  The
encoder is the producer of the inputs, on the host, and is not timed.

A case's fields: ``path`` (which calls, see ``run``), the mesh (``mesh`` and its
sizes, or ``meshes`` and a range of triangles for many), ``bits`` per longest
axis (0: the encoder's default, a world-space error of 0.0005), the meshlet
caps ``max_verts`` / ``max_tris`` and the ``predictor``.
"""
import math
import os
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from meshpress_gb300 import ParaDeltaV5GpuDecoder, cull_meshlets, encoder, synth
from meshpress_gb300.batch import BatchDecoder
from meshpress_gb300.serve import DecodeServer

CAPS = {"max_verts": 256, "max_tris": 256, "predictor": "generalized"}  # the encoder's defaults
PATHS = ("device", "async", "normalised", "host", "oneshot", "meshlets", "pldt5", "batch", "serve")


def listed():
    return [
        # one terrain tile, as a streaming renderer decodes tile by tile and looks at each one's status: the smallest call
        {"name": "tile_33", "path": "device", "mesh": "terrain", "nx": 33, "ny": 33, "bits": 12, **CAPS},
        # an asset decoded once from its bytes into new host arrays, at the encoder's default precision: open, decode, copy, close
        {"name": "oneshot_torus", "path": "oneshot", "mesh": "torus", "nu": 151, "nv": 77, "bits": 0, **CAPS},
        # a renderer that takes a decode's rows by meshlet and culls them: the small meshlets such a renderer draws, odd sizes
        {"name": "meshlets_torus_64", "path": "meshlets", "mesh": "torus", "nu": 403, "nv": 201, "bits": 14, "max_verts": 64, "max_tris": 124,
         "predictor": "generalized"},
        # an ordinary mesh on the device, decodes queued one after the other without waiting for each one's status
        {"name": "terrain_513", "path": "async", "mesh": "terrain", "nx": 513, "ny": 513, "bits": 12, **CAPS},
        # a scan-like closed mesh at 16 bits, the reference's decode() results: normalised positions and int32 triangles
        {"name": "normalised_sphere_7", "path": "normalised", "mesh": "sphere", "level": 7, "bits": 16, **CAPS},
        # ragged terrain of survey precision: codes above 16 bits, with the canonical predictor
        {"name": "terrain_1025x771_20bit", "path": "device", "mesh": "terrain", "nx": 1025, "ny": 771, "bits": 20, "max_verts": 256, "max_tris": 256,
         "predictor": "canonical"},
        # the closed mesh of 1.3 million triangles
        {"name": "sphere_8", "path": "device", "mesh": "sphere", "level": 8, "bits": 12, **CAPS},
        # the largest single mesh: 8.4 million triangles
        {"name": "terrain_2049", "path": "device", "mesh": "terrain", "nx": 2049, "ny": 2049, "bits": 12, **CAPS},
        # a scene of mixed meshes in one launch
        {"name": "batch_128", "path": "batch", "meshes": 128, "t_min": 1000, "t_max": 200000, "bits": 12, **CAPS},
        # new bytes from the host into a kept decoder, results into kept pinned host memory: a loader's loop
        {"name": "host_terrain_641", "path": "host", "mesh": "terrain", "nx": 641, "ny": 641, "bits": 14, **CAPS},
        # a stream of the reference class's own format, PLDT v5
        {"name": "pldt5_terrain_361", "path": "pldt5", "mesh": "terrain", "nx": 361, "ny": 361, "bits": 12, **CAPS},
        # requests to the decode server, submitted together and waited for one by one
        {"name": "serve_24", "path": "serve", "meshes": 24, "t_min": 5000, "t_max": 200000, "bits": 12, **CAPS},
    ]


def draw(rng):
    path = rng.choice(PATHS)
    c = {"path": path, "bits": rng.choice((0, 10, 11, 12, 12, 13, 14, 16, 18, 20))}
    if path == "pldt5":  # its residuals are fixed by the precision; the range of its golden streams
        c["bits"] = rng.choice((10, 12, 14, 16))
    c["max_verts"], c["max_tris"] = rng.choice(((256, 256), (256, 256), (128, 256), (64, 124)))
    # the decoder takes fitted weights as long as their sums fit 32 bits: not always at 20 bits
    c["predictor"] = "canonical" if c["bits"] == 20 else rng.choice(("generalized", "generalized", "canonical"))
    if path in ("batch", "serve"):
        c["meshes"] = round(math.exp(rng.uniform(math.log(2), math.log(128 if path == "batch" else 30))))
        c["t_min"] = round(math.exp(rng.uniform(math.log(500), math.log(5000))))
        c["t_max"] = round(c["t_min"] * math.exp(rng.uniform(math.log(2), math.log(40))))
        return c
    # triangles: over the whole range where the mesh stays on the device, up to two million where it is copied or converted too
    t = math.exp(rng.uniform(math.log(2000), math.log(8.3e6 if path in ("device", "async") else 2.0e6)))
    c["mesh"] = rng.choice(("terrain", "terrain", "sphere", "torus"))
    if c["mesh"] == "sphere":
        c["level"] = min(range(3, 9), key=lambda k: abs(math.log(20 * 4 ** k / t)))
    else:
        cells, aspect = t / 2, math.exp(rng.uniform(-1, 1))
        a = max(3, round(math.sqrt(cells * aspect)))
        b = max(3, round(cells / a))
        c.update({"nx": a + 1, "ny": b + 1} if c["mesh"] == "terrain" else {"nu": a, "nv": b})
    return c


def _triangles(case):
    """Triangles of the case's mesh or meshes (of many: of the mean of their log-uniform range)."""
    if "meshes" in case:
        a, b = case["t_min"], case["t_max"]
        return case["meshes"] * (b - a) / math.log(b / a)
    if case["mesh"] == "sphere":
        return 20 * 4 ** case["level"]
    return 2 * (case["nx"] - 1) * (case["ny"] - 1) if case["mesh"] == "terrain" else 2 * case["nu"] * case["nv"]


def work(case):
    """The stream read once (about 1.8 bytes a triangle at 12 bits, 0.28 more or less a bit), 12 bytes a triangle and 12 bytes a decoded vertex
    (0.62 a triangle with 256-vertex meshlets, 0.72 with 64) written once.  Entropy decoding has no operation count worth a rate."""
    rows = {64: 0.72, 128: 0.66}.get(case["max_verts"], 0.62)
    return {"bytes": _triangles(case) * (1.8 + 0.28 * ((case["bits"] or 12) - 12) + 12 + 12 * rows), "flops": 0}


# ---- inputs ----------------------------------------------------------------
def _terrain(nx, ny, seed):
    """A heightfield on the unit square: six octaves of smooth value noise, made on the GPU, and the regular grid's triangles."""
    g = torch.Generator().manual_seed(int(seed))
    z = torch.zeros((ny, nx), dtype=torch.float64, device="cuda")
    for o in range(6):
        n = 4 * 2 ** o + 1
        lattice = (torch.rand((1, 1, n, n), generator=g, dtype=torch.float64) * 2 - 1).cuda()
        z += (0.15 / 2 ** o) * torch.nn.functional.interpolate(lattice, size=(ny, nx), mode="bicubic", align_corners=True)[0, 0]
    x, y = np.meshgrid(np.linspace(0.0, 1.0, nx), np.linspace(0.0, 1.0, ny), indexing="xy")
    return np.stack([x.ravel(), y.ravel(), z.cpu().numpy().ravel()], axis=1), synth.grid_triangles(nx, ny)


def _mesh(case, seed):
    if case["mesh"] == "terrain":
        return _terrain(case["nx"], case["ny"], seed)
    if case["mesh"] == "sphere":
        return synth.icosphere(case["level"], seed=seed)
    rng = np.random.default_rng(seed)
    return synth.torus(case["nu"], case["nv"], R=float(rng.uniform(2.0, 5.0)), r=1.0)


def _encode(case, mesh):
    precision = ({"precision_error": synth.bbox_bits_error(case["bits"]), "precision_mode": "bbox_frac"} if case["bits"] else
                 {"precision_error": 0.0005, "precision_mode": "world"})
    caps = {"max_verts": case["max_verts"], "max_tris": case["max_tris"]}
    if case["path"] == "pldt5":
        return encoder.encode_pldt5(*mesh, **caps, **precision)
    return encoder.encode(*mesh, predictor=case["predictor"], **caps, **precision)


def _streams(case, seed):
    """The case's encoded meshes."""
    if "meshes" not in case:
        return [_encode(case, _mesh(case, seed))]
    # the kinds and sizes belong to the case, the shapes to the seed
    specs = synth.mixed_batch_specs(case["meshes"], t_min=case["t_min"], t_max=case["t_max"])
    rng = np.random.default_rng(seed)
    for kind, sizes in specs:
        sizes.update({"ratio": float(rng.uniform(2.0, 5.0))} if kind == "torus" else {"seed": int(rng.integers(1 << 31))})
    with ThreadPoolExecutor(max_workers=min(16, os.cpu_count() or 1)) as ex:  # the encoder leaves Python
        return list(ex.map(lambda s: _encode(case, synth.build_spec(*s)), specs))


# ---- the calls -------------------------------------------------------------
def prepare(case, seed):
    enc = _streams(case, seed)
    path = case["path"]
    s = {"path": path, "data": enc[0].data}
    if path == "batch":
        s["batch"] = BatchDecoder([e.data for e in enc])
    elif path == "serve":
        s["blobs"] = [e.data for e in enc]
        s["server"] = DecodeServer(4 << 30, pinned_budget_bytes=64 << 20)
        s["open"] = []
    elif path != "oneshot":
        s["dec"] = ParaDeltaV5GpuDecoder(enc[0].data)
    if path == "host":
        n_v, n_t = s["dec"].n_v_total, s["dec"].n_t_total
        s["out"] = (torch.empty((n_v, 3), dtype=torch.float32, pin_memory=True).numpy(),
                    torch.empty((n_t, 3), dtype=torch.int32, pin_memory=True).numpy().view(np.uint32))
    if path == "meshlets":
        # a camera that looks into the mesh's box from one side: some meshlets lie outside its six planes
        rng = np.random.default_rng(seed)
        normal = rng.normal(size=3)
        normal /= np.linalg.norm(normal)
        s["planes"] = np.array([[*normal, 0.3], [*-normal, 4.0], [1, 0, 0, 3], [-1, 0, 0, 3], [0, 1, 0, 3], [0, -1, 0, 3]], np.float32)
    return s


def run(s):
    path = s["path"]
    if path in ("device", "async"):  # into the decoder's own tensors
        tris, verts = s["dec"].decode_to_device(check=path == "device")
        return {"verts": verts, "tris": tris.view(torch.int32)}
    if path == "normalised":
        verts, tris = s["dec"].decode(normalised=True)
        return {"verts": verts, "tris": tris}
    if path == "pldt5":
        tris, verts = s["dec"].decode_to_device()
        return {"verts": verts, "tris": tris.view(torch.int32)}
    if path == "host":
        s["dec"].reload(s["data"])
        verts, tris = s["dec"].decode_to_host(out=s["out"])
        return {"verts": verts, "tris": tris.view(np.int32)}
    if path == "oneshot":
        dec = ParaDeltaV5GpuDecoder(s["data"])
        verts, tris = dec.decode_to_host()
        dec.close()
        return {"verts": verts, "tris": tris.view(np.int32)}
    if path == "meshlets":
        tris, verts = s["dec"].decode_to_device()
        v_first, t_first = s["dec"].meshlet_ranges()
        bounds = s["dec"].meshlet_bounds(verts)
        visible, count = cull_meshlets(bounds, s["planes"])
        return {"verts": verts, "tris": tris.view(torch.int32), "v_first": v_first, "t_first": t_first, "bounds": bounds,
                "visible": visible, "count": count}
    if path == "batch":
        tris, verts = s["batch"].decode()
        return {"verts": verts, "tris": tris.view(torch.int32)}
    # serve: the last burst's results go back to the server when the next burst comes
    for rid in s["open"]:
        s["server"].release(rid)
    s["open"] = [s["server"].submit(b) for b in s["blobs"]]
    got = [s["server"].wait(rid) for rid in s["open"]]
    verts, tris = [r.verts for r in got], [r.tris.view(torch.int32) for r in got]
    for t in verts + tris:
        t.server = s["server"]  # the results are views of the server's arena: it lives as long as they do
    return {"verts": verts, "tris": tris}


# ---- the same in 64 bits ----------------------------------------------------
def _header(data):
    """center, scale, g_min, g_range, g_bits of a DPR4 stream's global header (big-endian)."""
    f = np.frombuffer(data, ">f4", 4, 6).astype(np.float64)
    g = np.frombuffer(data, ">f4", 6, 26).astype(np.float64)
    return f[:3], f[3], g[:3], g[3:], np.frombuffer(data, np.uint8, 3, 50).astype(np.int64)


def _positions(e, normalised=False):
    """float64 positions of a stream's rows, from its header and the integer codes that its writer put into it."""
    center, scale, g_min, g_range, bits = _header(e.data)
    mx = np.maximum((1 << bits) - 1, 1).astype(np.float64)
    x = g_min + e.codes.astype(np.float64) / mx * np.where(bits > 0, g_range, 0.0)
    return x if normalised else x * scale + center


def _first_rows(data):
    """First vertex row of each meshlet, from the offset table and the meshlets' 16-bit vertex counts."""
    n = int(np.frombuffer(data, ">u4", 1, 82)[0])
    at = np.frombuffer(data, ">u4", n, 86).astype(np.int64)
    b = np.frombuffer(data, np.uint8).astype(np.int64)
    i = at >> 3
    n_local = ((b[i] << 16 | b[i + 1] << 8 | b[i + 2]) >> (8 - (at & 7))) & 0xFFFF
    return np.concatenate([[0], np.cumsum(n_local)])


def exact(case, seed):
    path = case["path"]
    if path == "pldt5":  # its rows come from a float64 predictor through the whole entropy-coded stream
        return None
    enc = _streams(case, seed)
    verts = [_positions(e, path == "normalised") for e in enc]
    out = {"verts": verts if path == "serve" else np.concatenate(verts), "tris": [None] * len(enc) if path == "serve" else None}
    if path == "meshlets":
        first = _first_rows(enc[0].data)[:-1]
        out["bounds"] = np.concatenate([np.minimum.reduceat(verts[0], first), np.maximum.reduceat(verts[0], first)], axis=1)
        out.update(v_first=None, t_first=None, visible=None, count=None)
    return out
