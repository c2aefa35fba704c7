"""A handle whose calls were captured in a CUDA graph: the status is the
replay's, and eager calls after a captured one work."""
import numpy as np
import pytest

import oracle
from meshpress_gb300 import encoder, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def data():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meshpress_gb300 import _build
    _build.build_decoder()
    oracle.build()
    V, T = synth.noise_heightfield(65, seed=3)
    return encoder.encode(V, T, precision_error=synth.bbox_bits_error(12), precision_mode="bbox_frac").data


def _same(data, tris, verts):
    opos, oidx = oracle.decode(data)
    assert np.array_equal(verts.cpu().numpy().view(np.uint32), opos.view(np.uint32))
    assert np.array_equal(tris.cpu().numpy().astype(np.int64), oidx)


def test_status_of_a_replayed_decode(data):
    import torch
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    from meshpress_gb300._lib import StrideFormatError
    dec = ParaDeltaV5GpuDecoder(data)
    tris, verts = dec.decode_to_device()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        dec.decode_into(tris, verts, check=False)
    dec.decode_to_device()  # eager, and its status seen
    bad = bytearray(data)
    bad[86 + 4 * 5:90 + 4 * 5] = (8 * len(data)).to_bytes(4, "big")  # meshlet 5 starts at the end
    dec.reload(bytes(bad))
    graph.replay()
    torch.cuda.synchronize()
    with pytest.raises(StrideFormatError):
        dec.check()
    with pytest.raises(StrideFormatError):
        dec.meshlet_bounds(verts)
    dec.reload(data)
    tris.view(torch.int32).zero_(), verts.zero_()
    graph.replay()
    torch.cuda.synchronize()
    dec.check()
    _same(data, tris, verts)
    dec.close()


def test_calls_after_captured_ones(data):
    import torch
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    dec = ParaDeltaV5GpuDecoder(data)
    tris, verts = dec.decode_to_device()
    ranges, bounds, side = dec.meshlet_ranges(), dec.meshlet_bounds(verts), dec.side_table()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        c_ranges, c_bounds, c_side = dec.meshlet_ranges(), dec.meshlet_bounds(verts), dec.side_table()
    graph.replay()
    for _ in range(2):
        again = (*dec.meshlet_ranges(), dec.meshlet_bounds(verts), *dec.side_table())
        for got in ((*c_ranges, c_bounds, *c_side), again):
            for x, y in zip(got, (*ranges, bounds, *side)):
                assert torch.equal(x, y)
        dec.reload(data)
        tris, verts = dec.decode_to_device()
        _same(data, tris, verts)
    dec.close()
