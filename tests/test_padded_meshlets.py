"""Batches of streams whose last meshlets are padded by hundreds of megabytes: the
sums by which the kernels form rounds of staged meshlets stay below 2^32, so such
a meshlet, and none after it, is taken for one that fits."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import oracle
from meshpress_gb300 import _build, _lib, encoder, synth

# Nine of these add up to 2^32 + 176 bytes.
REGION = 477218608

SUMS = r"""
#include <cuda_runtime.h>
#include "stride_common.cuh"
// a warp's inclusive sums, as the kernels form them; whether lane i fits `room`
extern "C" void sums(const unsigned long long* bytes, uint32_t n, uint32_t room, uint8_t* fits) {
    uint32_t c = 0;
    for (uint32_t i = 0; i < n; i++) {
        const uint32_t s = stride::staged_bytes(16ull, 16ull + bytes[i]);
        c += s + ((s & 16u) ? 0u : 16u);
        fits[i] = c <= room;
    }
}
"""


def test_sums_of_padded_meshlets_do_not_wrap(tmp_path):
    src, out = tmp_path / "sums.cpp", tmp_path / "sums.so"
    src.write_text(SUMS)
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build._nvcc()))), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fPIC", "-shared", "-I", cuda, "-I", "/usr/local/cuda/include", "-I", _build.CSRC,
                    str(src), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    rng = np.random.default_rng(1)
    for room in (5440, 227 * 1024):
        for case in range(200):
            n = 32
            b = 16 * rng.integers(1, 200, n).astype(np.uint64)
            big = rng.choice(n, int(rng.integers(0, 20)), replace=False)
            b[big] = REGION if case % 2 else 16 * rng.integers(1 << 16, 1 << 25, len(big)).astype(np.uint64)
            fits = np.zeros(n, np.uint8)
            lib.sums(b.ctypes.data_as(ctypes.c_void_p), n, room, fits.ctypes.data_as(ctypes.c_void_p))
            true = np.cumsum([int(x) | 16 if int(x) & 16 else int(x) + 16 for x in b]) <= room
            assert np.array_equal(fits.astype(bool), true)


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["meshlet", "anchor"])
def test_batch_of_padded_streams(where):
    """The team kernel sums from the meshlets' first bytes, the others from their anchors."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _build.build_decoder()
    oracle.build()
    from meshpress_gb300.batch import BatchDecoder
    V, T = synth.heightfield_grid(5, seed=4)
    mesh = encoder.encode(V, T, precision_error=synth.bbox_bits_error(12), precision_mode="bbox_frac").data
    assert np.frombuffer(mesh, ">u4", 1, 82)[0] == 1
    opos, oidx = oracle.decode(mesh)
    st = oracle.side_table(mesh)
    first = int(st["start_bit" if where == "meshlet" else "resid_bit"][0]) >> 3 & ~15
    padded = mesh + bytes(first + REGION - len(mesh))
    b = BatchDecoder([padded] * 9 + [mesh] * 39)
    n_v, n_t = len(opos), len(oidx)
    for shape in [(1, 4), (2, 4), (4, 4)] if where == "meshlet" else [(4, 2), (4, 1), (1, 3)]:
        cfg = _lib.LaunchCfg()
        cfg.warps_per_cta, cfg.persistent, cfg.stage_bytes, cfg.code_bytes = *shape, 16384, 16384
        b.set_config(cfg)
        tris, verts = b.decode()
        t, v = tris.cpu().numpy().astype(np.int64), verts.cpu().numpy()
        for i in range(48):
            assert np.array_equal(v[i * n_v:(i + 1) * n_v].view(np.uint32), opos.view(np.uint32))
            assert np.array_equal(t[i * n_t:(i + 1) * n_t], oidx)
    b.close()
