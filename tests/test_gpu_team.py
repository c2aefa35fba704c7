"""The team kernel (launch shape 4), the default of meshes of up to 9,728
meshlets: bit-exact against the oracle where its layout has edges -- part
groups of 4, 8 and 16 meshlets, nine-bit local ids, raw ids the FIFO still
holds, residuals wider than the code plane, codewords longer than the window,
groups that do not fit their shared memory (decoded in rounds) and meshlets
read in place.  No tolerance: positions, indices and codes are equal."""
import numpy as np
import pytest

import _golden
import oracle
from meshpress_gb300 import _lib, encoder, synth

pytestmark = pytest.mark.gpu

SHAPES = [1, 2, 4]  # 4, 8, 16 meshlets per CTA


@pytest.fixture(scope="module")
def torch_cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meshpress_gb300 import _build
    _build.build_decoder()
    oracle.build()
    return torch


def _cfg(w):
    c = _lib.LaunchCfg()
    c.warps_per_cta, c.persistent = w, 4
    return c


def _decode(torch, data, w):
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    dec = ParaDeltaV5GpuDecoder(data)
    dec.set_launch_config(_cfg(w))
    codes = torch.full((dec.n_v_total, 3), -1, dtype=torch.int32, device="cuda")
    tris, verts = dec._outputs()
    dec.decode_into(tris, verts, codes=codes)
    out = (verts.cpu().numpy(), tris.view(torch.int32).cpu().numpy().view(np.uint32), codes.cpu().numpy())
    dec.close()
    return out


def _same(data, pos, idx):
    opos, oidx = oracle.decode(data)
    assert np.array_equal(idx.astype(np.int64), oidx)
    assert np.array_equal(pos.view(np.uint32), opos.view(np.uint32))


@pytest.mark.parametrize("w", SHAPES)
@pytest.mark.parametrize("name", _golden.names())
def test_golden_streams(torch_cuda, name, w):
    """crafted_a holds raw ids that the FIFO still holds (the exact pass)."""
    g = _golden.load(name)
    pos, idx, codes = _decode(torch_cuda, g["data"], w)
    _golden.check_against(g, pos, idx, codes)


def _spikes(bits):
    """A grid whose heights jump by most of the box at some vertices:
    residuals beyond 16 bits, codewords beyond 32."""
    V, T = synth.heightfield_grid(33, seed=4)
    rng = np.random.default_rng(bits)
    V[rng.choice(len(V), 40, replace=False), 2] += 60.0 * rng.choice([-1.0, 1.0], 40)
    return V, T


MESHES = {
    "one_meshlet": (lambda: synth.heightfield_grid(5, seed=1), 12, {}),
    "ids_of_nine_bits": (lambda: synth.heightfield_grid(128, ny=2, seed=2), 12, {}),
    "part_groups": (lambda: synth.heightfield_grid(40, seed=3), 13, {"max_verts": 24, "max_tris": 40}),
    "seventeen_to_a_window": (lambda: synth.torus(60, 31, R=3.0, r=1.0), 14, {"max_verts": 64, "max_tris": 124}),
    "spikes_16": (lambda: _spikes(16), 16, {}),
    "spikes_24": (lambda: _spikes(24), 24, {"predictor": "canonical"}),
    "sphere_18": (lambda: synth.icosphere(4, seed=5), 18, {"predictor": "canonical"}),
    "coarse_1": (lambda: synth.icosphere(3, seed=6), 1, {}),
}


@pytest.mark.parametrize("w", SHAPES)
@pytest.mark.parametrize("name", sorted(MESHES))
def test_meshes_at_the_edges(torch_cuda, name, w):
    make, bits, kw = MESHES[name]
    e = encoder.encode(*make(), precision_error=synth.bbox_bits_error(bits), precision_mode="bbox_frac", **kw)
    pos, idx, codes = _decode(torch_cuda, e.data, w)
    _same(e.data, pos, idx)
    assert np.array_equal(codes, e.codes)


@pytest.mark.parametrize("w", SHAPES)
def test_batch_in_rounds_and_in_place(torch_cuda, w):
    """Shared memory is sized by the average meshlet: among 300 meshes of two
    triangles, groups with ordinary meshlets go in rounds, and meshlets of
    24-bit noise, larger than all of it, are read in place."""
    from meshpress_gb300.batch import BatchDecoder
    rng = np.random.default_rng(7)
    V, T = synth.heightfield_grid(2, seed=1)
    tiny = encoder.encode(V, T, precision_error=synth.bbox_bits_error(8), precision_mode="bbox_frac").data
    V, T = synth.heightfield_grid(24, seed=8)
    plain = encoder.encode(V, T, precision_error=synth.bbox_bits_error(12), precision_mode="bbox_frac").data
    noise = encoder.encode(rng.uniform(-1, 1, (len(V), 3)), T, precision_error=synth.bbox_bits_error(24),
                           precision_mode="bbox_frac", predictor="canonical").data
    blobs = [tiny] * 300
    for at, b in ((10, plain), (11, plain), (12, plain), (13, plain), (100, noise), (201, noise), (202, plain)):
        blobs[at] = b
    b = BatchDecoder(blobs)
    b.set_config(_cfg(w))
    tris, verts = b.decode()
    t, v = tris.view(torch_cuda.int32).cpu().numpy().view(np.uint32), verts.cpu().numpy()
    for i in (0, 9, 10, 11, 12, 13, 14, 99, 100, 101, 200, 201, 202, 203, 299):
        _same(blobs[i], v[b.v_offset[i]:b.v_offset[i + 1]], t[b.t_offset[i]:b.t_offset[i + 1]])
    b.close()


@pytest.mark.parametrize("w", SHAPES)
def test_bit_flips_rejected_or_equal(torch_cuda, w):
    rng = np.random.default_rng(11 + w)
    V, T = synth.heightfield_grid(24, seed=9)
    base = encoder.encode(V, T, precision_error=synth.bbox_bits_error(12), precision_mode="bbox_frac").data
    for _ in range(40):
        d = bytearray(base)
        bit = int(rng.integers(86 * 8, 8 * len(d)))
        d[bit >> 3] ^= 0x80 >> (bit & 7)
        try:
            opos, oidx = oracle.decode(bytes(d))
        except Exception:  # noqa: BLE001
            opos = None
        try:
            pos, idx, _ = _decode(torch_cuda, bytes(d), w)
        except ValueError:
            continue
        assert opos is not None, f"bit {bit}: accepted, the oracle rejects it"
        assert np.array_equal(idx.astype(np.int64), oidx) and np.array_equal(pos.view(np.uint32), opos.view(np.uint32))


def test_default_shape_by_size(torch_cuda):
    """4, 8 and 16 meshlets per CTA by the number of meshlets; the fused
    kernel's config stays what a handle is given."""
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    for n, caps, per in ((33, {}, 4), (129, {"max_verts": 24, "max_tris": 32}, 8), (225, {"max_verts": 24, "max_tris": 32}, 16)):
        V, T = synth.heightfield_grid(n, seed=10)
        e = encoder.encode(V, T, precision_error=synth.bbox_bits_error(11), precision_mode="bbox_frac", **caps)
        dec = ParaDeltaV5GpuDecoder(e.data)
        tris, verts = dec.decode_to_device()
        assert dec._persistent_blocks == -(-dec.n_meshlets // per)
        _same(e.data, verts.cpu().numpy(), tris.view(torch_cuda.int32).cpu().numpy().view(np.uint32))
        dec.close()
