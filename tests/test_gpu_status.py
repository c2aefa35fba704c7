"""The status word, which the scan starts anew for each decode: an error in any
of its blocks is reported with its meshlet, and neither the error nor the
counters of a failed decode reach the next one, in every launch shape."""
import numpy as np
import pytest

import oracle
from meshpress_gb300 import _lib, encoder, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def good():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meshpress_gb300 import _build
    _build.build_decoder()
    oracle.build()
    V, T = synth.noise_heightfield(257, seed=3)  # 650 meshlets: three scan blocks
    data = encoder.encode(V, T, precision_error=synth.bbox_bits_error(12), precision_mode="bbox_frac").data
    return data, oracle.decode(data)


@pytest.mark.parametrize("shape", [(4, 1), (4, 2), (1, 3), (2, 4)])
def test_errors_stay_with_their_decode(good, shape):
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    from meshpress_gb300._lib import StrideFormatError
    data, (opos, oidx) = good
    n = int(np.frombuffer(data, ">u4", 1, 82)[0])
    dec = ParaDeltaV5GpuDecoder(data)
    cfg = _lib.LaunchCfg()
    cfg.warps_per_cta, cfg.persistent, cfg.stage_bytes, cfg.code_bytes = *shape, 16384, 16384
    dec.set_launch_config(cfg)
    for k in (0, 255, 256, 300, n - 1):
        bad = bytearray(data)
        at = 86 + 4 * k
        bad[at:at + 4] = (8 * len(data) if k else 8 * (86 + 4 * n) + 1).to_bytes(4, "big")
        dec.reload(bytes(bad))
        for _ in range(2):
            with pytest.raises(StrideFormatError, match=rf"meshlet {k}\)"):
                dec.decode_to_device()
            with pytest.raises(StrideFormatError, match=rf"meshlet {k}\)"):
                dec.check()  # what stride_finish has read
        dec.reload(data)
        for _ in range(2):
            tris, verts = dec.decode_to_device()
            assert np.array_equal(verts.cpu().numpy().view(np.uint32), opos.view(np.uint32))
            assert np.array_equal(tris.cpu().numpy().astype(np.int64), oidx)
    dec.close()


def test_memory_of_closed_handles(good):
    """Handles closed with work still queued on two streams hand their memory to
    the next ones, larger and smaller: every output is its own stream's."""
    import torch
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    blobs = [good[0]] + [encoder.encode(*synth.noise_heightfield(n, seed=n), precision_error=synth.bbox_bits_error(12),
                                        precision_mode="bbox_frac").data for n in (33, 129, 200)]
    want = [oracle.decode(b) for b in blobs]
    got = []
    for r in range(24):
        k = (r * 7) % len(blobs)
        dec = ParaDeltaV5GpuDecoder(blobs[(k + 1) % len(blobs)])
        dec.reload(blobs[k], stream=streams[r % 2])  # may grow
        with torch.cuda.stream(streams[r % 2]):
            tris, verts = dec.decode_to_device(check=False)
            bounds = dec.meshlet_bounds(verts, stream=streams[r % 2])
        streams[1 - r % 2].wait_stream(streams[r % 2])
        with torch.cuda.stream(streams[1 - r % 2]):
            again = dec.meshlet_bounds(verts, stream=streams[1 - r % 2])
        dec.close()
        got.append((k, tris, verts, bounds, again))
    torch.cuda.synchronize()
    for k, tris, verts, bounds, again in got:
        opos, oidx = want[k]
        assert np.array_equal(verts.cpu().numpy().view(np.uint32), opos.view(np.uint32))
        assert np.array_equal(tris.cpu().numpy().astype(np.int64), oidx)
        assert torch.equal(bounds, again)
        b = bounds.cpu().numpy()
        assert np.array_equal(b[:, :3].min(0), opos.min(0)) and np.array_equal(b[:, 3:].max(0), opos.max(0))


def test_threads_with_meshes_of_different_sizes(good):
    """Launch attributes, pinned words and closed handles' memory are shared by
    the process: eight threads open, decode and close their own meshes at once."""
    import threading
    import torch
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    blobs = [encoder.encode(*synth.noise_heightfield(n, seed=n), precision_error=synth.bbox_bits_error(b),
                            precision_mode="bbox_frac", max_verts=v, max_tris=t).data
             for n, b, v, t in ((33, 12, 64, 124), (65, 16, 256, 256), (97, 10, 128, 256), (129, 12, 256, 256))]
    want = [oracle.decode(b) for b in blobs]
    bad = []

    def work(k):
        try:
            s = torch.cuda.Stream()
            for r in range(12):
                i = (k + r) % len(blobs)
                dec = ParaDeltaV5GpuDecoder(blobs[i])
                if r % 2:
                    pos, idx = dec.decode_to_host(stream=s)
                else:
                    with torch.cuda.stream(s):
                        tris, verts = dec.decode_to_device(stream=s)
                        pos, idx = verts.cpu().numpy(), tris.cpu().numpy()
                dec.close()
                if not (np.array_equal(pos.view(np.uint32), want[i][0].view(np.uint32)) and
                        np.array_equal(idx.astype(np.int64), want[i][1])):
                    bad.append((k, r))
        except Exception as e:  # noqa: BLE001 -- reported below
            bad.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
