"""A handle says which launch shape its decodes take."""
import pytest

from meshpress_gb300 import _lib, encoder, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,shape", [(12, 1), (20, 4)])
def test_shape_above_the_team_kernels_bound(bits, shape):
    """Above 9,728 meshlets codes above 16 bits keep the team kernel, others take the two kernels."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meshpress_gb300 import ParaDeltaV5GpuDecoder, _build
    _build.build_decoder()
    V, T = synth.heightfield_grid(401, seed=5)
    dec = ParaDeltaV5GpuDecoder(encoder.encode(V, T, precision_error=synth.bbox_bits_error(bits), precision_mode="bbox_frac",
                                               predictor="canonical", max_verts=24, max_tris=32).data)
    assert 9728 < dec.n_meshlets <= 17024
    assert dec.launch_config().persistent == shape
    assert int(dec.info.kernels) == (2 if shape == 4 else 3)
    cfg = _lib.LaunchCfg()
    cfg.warps_per_cta, cfg.persistent, cfg.stage_bytes, cfg.code_bytes = 4, 2, 16384, 12288
    dec.set_launch_config(cfg)
    assert dec.launch_config().as_dict() == cfg.as_dict()
    dec.close()
