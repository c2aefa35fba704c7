"""PLDT v5 streams written token by token, where the decoder's kernels have
edges: part groups of meshlets, either group size, meshlets that only the general kernel takes (tokens,
bytes), nine-bit ids, raw ids the FIFO still holds, every substream tag,
codewords longer than a window, values beyond 32 bits, vertices that the walk
never reaches, canonical and fitted weights.  No tolerance: positions and
indices equal the oracle's."""
import struct

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meshpress_gb300 import _build
    _build.build_decoder()
    oracle.build()
    return torch


def _b(v, n):
    return format(int(v), f"0{n}b")[-n:] if n else ""


def _code(u, tag, k):
    if tag == 1:
        return "0" * (u >> k) + "1" + _b(u, k)
    s = (u >> k) + 1
    n = s.bit_length() - 1
    return "0" * n + "1" + _b(s, n) + _b(u, k)


def _meshlet(rng, c, n_boundary):
    n_bnd, n_int, again = c["bnd"], c["int"], c.get("again", 0.0)
    n_local = n_bnd + n_int
    width = max(1, n_local.bit_length())
    out, fifo, lens, left = [], [], [], c["tris"]
    while left:
        lens.append(int(min(left, rng.integers(1, c.get("strip", 20) + 1))))
        left -= lens[-1]
    fresh = list(rng.permutation(n_local)[: c.get("reach", n_local)])
    known = []
    for n in lens:
        out.append(_b(0 if n == 1 and rng.random() < 0.5 else n, 16))
        for t in range(n + 2):
            if t >= 3:
                out.append(_b(rng.integers(2), 1))  # edge code
            held = [v for v in known if v in fifo]
            if fifo and rng.random() < 0.25:
                at = int(rng.integers(len(fifo)))
                out.append("0" + _b(len(fifo) - 1 - at, 5))  # counted from the oldest
                fifo.insert(0, fifo.pop(at))
                continue
            gone = [v for v in known if v not in fifo]
            if held and rng.random() < again:
                v = held[rng.integers(len(held))]
                fifo.remove(v)
            elif fresh and (not gone or rng.random() < 0.7):
                v = int(fresh.pop())
                known.append(v)
            elif gone:
                v = gone[rng.integers(len(gone))]
            else:
                at = int(rng.integers(len(fifo)))
                out.append("0" + _b(len(fifo) - 1 - at, 5))
                fifo.insert(0, fifo.pop(at))
                continue
            out.append("1" + _b(v, width))
            fifo = [v] + fifo[:15]
    conn = "".join(out)
    refs = ""
    if n_bnd:
        r = np.sort(rng.choice(n_boundary, n_bnd, replace=False))
        k = int(rng.integers(0, 4))
        refs = _b(r[0], 32) + (_b(k, 8) + "".join(_code(int(d) - 1, 1, k) for d in np.diff(r)) if n_bnd > 1 else "")
    subs = []
    for tag in c["tags"] if n_int else ():
        k = int(rng.integers(0, 9))
        if tag == 0:
            k = c.get("fixed", k)
            subs.append(_b(0, 8) + _b(int(rng.integers(-900, 900)) & 0xFFFF, 16) + _b(k, 8) +
                        "".join(_b(rng.integers(0, 1 << k), k) for _ in range(n_int)))
            continue
        u = [int(x) for x in rng.integers(0, 3 << k, n_int)]
        for i in range(n_int):
            if rng.random() < c.get("long", 0.0):  # (an Exp-Golomb prefix may have 32 zeros)
                u[i] = int(rng.integers(40, c.get("ones", 150))) << k if tag == 1 else int(rng.integers(1 << 30, (1 << 32) - 1)) << k
        subs.append(_b(tag, 8) + _b(k, 8) + "".join(_code(x, tag, k) for x in u))
    return _b(n_bnd, 16) + _b(n_int, 16) + _b(c["tris"], 16) + _b(len(lens), 16) + refs + conn + "".join(subs)


def _stream(c, seed):
    rng = np.random.default_rng(seed)
    nb = max(c["bnd"] * 2, 1)
    head = struct.pack(">IBB12f", 0x504C4454, 5, 16, 0.5, -1.0, 2.0, 3.0, 1e-4, -1.0, -1.0, -1.0, 2.0, 2.0, 2.0, 0.0)[:-4]
    head += bytes((12, 12, 12)) + struct.pack(">4I3f", 0, 0, nb, c["n"], *c.get("w", (1.0, 1.0, -1.0)))
    bits = "".join(_b(x, 8) for x in head)
    for _ in range(3):  # boundary table
        q = rng.integers(0, 1 << 12, nb)
        d = np.diff(q)
        bits += _b(q[0], 12) + (_b(8, 8) + "".join(_code(int(2 * x if x >= 0 else -2 * x - 1), 1, 8) for x in d) if nb > 1 else "")
    bits += "0" * (-len(bits) % 8)
    at, offs, body = len(bits) + 32 * c["n"], [], []
    for i in range(c["n"]):
        m = _meshlet(rng, c, nb)
        offs.append(_b(at, 32))
        body.append(m)
        at += len(m)
    bits += "".join(offs) + "".join(body)
    bits += "0" * (-len(bits) % 8)
    return int(bits, 2).to_bytes(len(bits) // 8, "big")


W = (0.95, 0.8, -0.75)
CASES = {
    "one": {"n": 1, "bnd": 0, "int": 3, "tris": 1, "tags": (1, 2, 0)},
    "seven": {"n": 7, "bnd": 9, "int": 20, "tris": 60, "tags": (2, 1, 0), "w": W},
    "eight_again": {"n": 8, "bnd": 5, "int": 30, "tris": 90, "tags": (1, 1, 1), "again": 0.2},
    "nine_long": {"n": 9, "bnd": 1, "int": 40, "tris": 80, "tags": (1, 2, 2), "long": 0.1, "w": W},
    "fixed_32": {"n": 10, "bnd": 3, "int": 33, "tris": 70, "tags": (0, 0, 0), "fixed": 32},
    "all_boundary": {"n": 3, "bnd": 17, "int": 0, "tris": 40, "tags": ()},
    "unreached": {"n": 17, "bnd": 6, "int": 50, "tris": 40, "reach": 30, "tags": (2, 0, 1)},
    "nine_bit_ids": {"n": 5, "bnd": 120, "int": 136, "tris": 450, "tags": (1, 2, 1), "w": W},
    "groups_of_16": {"n": 2800, "bnd": 4, "int": 5, "tris": 8, "tags": (1, 2, 0), "again": 0.02},
    "most_bytes": {"n": 9, "bnd": 2, "int": 250, "tris": 300, "tags": (1, 1, 1), "long": 0.7, "ones": 300, "w": W},
    "most_tokens": {"n": 4, "bnd": 30, "int": 100, "tris": 728, "strip": 200, "tags": (1, 2, 0), "again": 0.05},
    "more_tokens": {"n": 4, "bnd": 30, "int": 100, "tris": 800, "strip": 200, "tags": (1, 2, 0), "again": 0.05},
    "more_bytes": {"n": 3, "bnd": 2, "int": 254, "tris": 400, "tags": (1, 1, 1), "long": 2.0, "ones": 400, "w": W},
}


@pytest.mark.parametrize("name", CASES)
def test_written_streams(torch_cuda, name):
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    for seed in range(1 if CASES[name]["n"] > 1000 else 3):
        data = _stream(CASES[name], seed)
        opos, oidx = oracle.decode_v5(data)
        dec = ParaDeltaV5GpuDecoder(data)
        pos, idx = dec.decode_to_host()
        dec.close()
        assert np.array_equal(idx.astype(np.int64), oidx)
        assert np.array_equal(pos.view(np.uint32), opos.view(np.uint32))
