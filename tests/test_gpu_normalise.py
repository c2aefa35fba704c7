"""decode(normalised=True): float32 of decode_dup's float64 expression
g_min + q / mx * g_range (encoder/paradelta_v5_dup.py:607-616), bit for bit,
for code widths from a constant axis to 24 bits, row counts that are no
multiple of the kernel's four values a thread, and codes at an offset that
allows no 16-byte access."""
import ctypes

import numpy as np
import pytest

import _golden
import oracle
from meshpress_gb300 import encoder, synth

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


def _expected(data):
    _, _, codes = oracle.decode(data, with_codes=True)
    h = oracle.parse_header(data)
    ref = np.empty(codes.shape, np.float64)
    for d in range(3):
        mx = (1 << int(h.g_bits[d])) - 1
        q = codes[:, d].astype(np.float64)
        ref[:, d] = float(h.g_min[d]) + (q / mx * float(h.g_range[d]) if mx else 0.0)
    return ref.astype(np.float32)


def _stream(name):
    if isinstance(name, str):
        return _golden.load(name)["data"]
    bits, n = name
    V, T = synth.heightfield_grid(n, ny=n + 1, seed=bits)
    return encoder.encode(V, T, precision_error=synth.bbox_bits_error(bits), precision_mode="bbox_frac",
                          predictor="canonical").data


@pytest.mark.parametrize("name", ["tri1_b12", "crafted_a", "crafted_b", "crafted_c", (1, 9), (12, 33), (16, 18), (20, 24),
                                  (24, 12)], ids=str)
def test_normalised_bit_exact(torch_cuda, name):
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    torch = torch_cuda
    data = _stream(name)
    dec = ParaDeltaV5GpuDecoder(data)
    vn, tris = dec.decode(normalised=True)
    want = _expected(data)
    assert np.array_equal(vn.cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert np.array_equal(tris.cpu().numpy().astype(np.int64), oracle.decode(data)[1])
    # unaligned arrays
    n = dec.n_v_total
    codes = torch.empty(3 * n + 1, dtype=torch.int32, device="cuda")[1:]
    out = torch.full((3 * n + 1,), np.nan, dtype=torch.float32, device="cuda")
    codes.copy_(torch.from_numpy(oracle.decode(data, with_codes=True)[2].astype(np.int32).reshape(-1)))
    rc = dec._lib.stride_normalise_codes(dec._h, None, ctypes.c_void_p(codes.data_ptr()), ctypes.c_void_p(out[1:].data_ptr()))
    torch.cuda.synchronize()
    assert rc == 0 and np.array_equal(out[1:].cpu().numpy().view(np.uint32), want.reshape(-1).view(np.uint32))
    assert np.isnan(float(out[0]))
    dec.close()
