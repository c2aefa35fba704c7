"""A meshlet larger than the team kernel's stage (a last meshlet may be padded)
is read in place: it decodes as a staged one does, and its header is checked as
in the other launch shapes: a residual k above 24 is rejected, whatever its low
bits say."""
import numpy as np
import pytest

import oracle
from meshpress_gb300 import _lib, encoder, synth

pytestmark = pytest.mark.gpu

PAD = bytes(1 << 18)  # above an SM's shared memory
SHAPES = [(1, 4), (2, 4), (4, 4), (4, 2), (4, 1), (1, 3)]  # warps per CTA, shape


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meshpress_gb300 import _build
    _build.build_decoder()
    oracle.build()
    return torch


def _mesh(bits):
    V, T = synth.heightfield_grid(9, seed=3)
    return encoder.encode(V, T, precision_error=synth.bbox_bits_error(bits), precision_mode="bbox_frac",
                          predictor="canonical").data


def _decode(data, shape):
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    dec = ParaDeltaV5GpuDecoder(data)
    cfg = _lib.LaunchCfg()
    cfg.warps_per_cta, cfg.persistent, cfg.stage_bytes, cfg.code_bytes = *shape, 16384, 16384
    dec.set_launch_config(cfg)
    try:
        tris, verts = dec.decode_to_device()
        return verts.cpu().numpy(), tris.cpu().numpy()
    finally:
        dec.close()


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bits", [12, 20])
def test_padded_meshlet(torch_cuda, bits, shape):
    data = _mesh(bits)
    opos, oidx = oracle.decode(data)
    pos, idx = _decode(data + PAD, shape)
    assert np.array_equal(pos.view(np.uint32), opos.view(np.uint32)) and np.array_equal(idx.astype(np.int64), oidx)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bits", [12, 20])
def test_residual_k_out_of_range(torch_cuda, bits, shape):
    from meshpress_gb300._lib import StrideFormatError
    data = _mesh(bits)
    n = int(np.frombuffer(data, ">u4", 1, 82)[0])
    anchor = int(oracle.side_table(data)["resid_bit"][n - 1])  # of the last meshlet
    for i in range(6):
        for flip in (0x20, 0x40, 0x80):
            bad = bytearray(data + PAD)
            at = anchor + sum(data[50:53]) + 16 * i + 8  # the pair's k, after its tag
            for b in range(8):
                if flip >> (7 - b) & 1:
                    bad[at + b >> 3] ^= 0x80 >> (at + b & 7)
            with pytest.raises(StrideFormatError):
                _decode(bytes(bad), shape)
