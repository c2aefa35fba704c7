"""The allocation-free entry point's fixed scratch: the tables that a small mesh
gets beside what its size needs cost no stream its place in it."""
import ctypes

import numpy as np
import pytest

import oracle
from meshpress_gb300 import _lib, encoder, synth


def _data(bits=None):
    """A small mesh at 12 bits; with `bits`, of a header that says so (never decoded)."""
    V, T = synth.heightfield_grid(33, seed=23)
    d = bytearray(encoder.encode(V, T, precision_error=synth.bbox_bits_error(12), precision_mode="bbox_frac",
                                 predictor="canonical").data)
    if bits:
        d[50:53] = bytes((bits,) * 3)
    return bytes(d)


def _most(data):
    """Longest stream (this one, padded) that fits the scratch.  The size is
    checked before the outputs, null here, and only the header is read."""
    lib = _lib.load()
    lo, hi = len(data), 1 << 28
    assert lib.stride_decode_static(data, lo, None, None, None) == _lib.STRIDE_ERR_ARG
    while hi - lo > 1:
        mid = (lo + hi) // 2
        rc = lib.stride_decode_static(data, mid, None, None, None)
        assert rc in (_lib.STRIDE_ERR_ARG, _lib.STRIDE_ERR_NOMEM)
        lo, hi = (mid, hi) if rc == _lib.STRIDE_ERR_ARG else (lo, mid)
    return lo


def test_tables_of_a_small_mesh_refuse_no_stream(built_libs):
    assert _most(_data()) == _most(_data(16))  # 16 bits: too many codes for such tables


@pytest.mark.gpu
def test_longest_stream_of_a_small_mesh():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meshpress_gb300 import _build
    _build.build_decoder()
    oracle.build()
    data = _data()
    opos, oidx = oracle.decode(data)
    long = data + bytes(_most(data) - len(data))
    info = _lib.inspect(data)
    idx = torch.zeros((int(info.n_t), 3), dtype=torch.int32, device="cuda")
    pos = torch.zeros((int(info.n_v), 3), dtype=torch.float32, device="cuda")
    s = ctypes.c_void_p(int(torch.cuda.current_stream().cuda_stream))
    _lib.check(_lib.load().stride_decode_static(long, len(long), s, ctypes.c_void_p(idx.data_ptr()),
                                                ctypes.c_void_p(pos.data_ptr())), "stride_decode_static")
    assert np.array_equal(pos.cpu().numpy().view(np.uint32), opos.view(np.uint32))
    assert np.array_equal(idx.cpu().numpy().astype(np.int64), oidx)
