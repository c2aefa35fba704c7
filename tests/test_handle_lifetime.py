"""Handles whose calls fail or are captured: their memory and their status.
The host code of csrc/stride_api.cu on a fake CUDA runtime (handle_harness.cpp)
in which a launch or an allocation fails when the test says so; no GPU."""
import ctypes
import os
import shutil
import subprocess

import pytest

from meshpress_gb300 import _lib, encoder, synth

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
_P, _SZ, _ULL = ctypes.c_void_p, ctypes.c_size_t, ctypes.c_ulonglong
CORRUPT = 6 << 32 | 3  # a status word: corrupt payload, meshlet 3
S = ctypes.c_void_p(0x1000)  # a stream


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        include = "/usr/local/cuda/include"
    out = str(tmp_path_factory.mktemp("handles") / "handles.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fPIC", "-shared", "-Wl,-Bsymbolic", "-I", include,
                    "-I", os.path.join(REPO, "include"), "-I", os.path.join(REPO, "meshpress_gb300", "csrc"),
                    os.path.join(HERE, "handle_harness.cpp"), "-o", out], check=True)
    lib = ctypes.CDLL(out)
    for name, res, args in _lib.SIGNATURES:
        if hasattr(lib, name):
            getattr(lib, name).restype, getattr(lib, name).argtypes = res, args
    lib.fake_most.argtypes = [_SZ]
    lib.fake_capture.argtypes = lib.fake_pending.argtypes = [_P]
    lib.fake_decode.argtypes = [ctypes.c_int, _ULL]
    lib.fake_replay.argtypes = [_ULL]
    return lib


@pytest.fixture()
def lib(built):
    built.fake_reset()
    return built


def _stream(n):
    V, T = synth.heightfield_grid(n, seed=n)
    return encoder.encode(V, T, precision_error=synth.bbox_bits_error(12), precision_mode="bbox_frac").data


SMALL, LARGE = _stream(9), _stream(65)
OUT = ctypes.create_string_buffer(1 << 20)
AT = ctypes.c_void_p(ctypes.addressof(OUT) + 15 & ~15)


def _open(lib, data=SMALL):
    h = _P()
    assert lib.stride_open(data, len(data), ctypes.byref(h)) == 0
    return h


CALLS = {
    "decode": lambda lib, h: lib.stride_decode(h, S, AT, AT, None),
    "timed": lambda lib, h: lib.stride_decode_timed(h, S, AT, AT, None),
    "host": lambda lib, h: lib.stride_decode_host(h, S, AT, AT),
}


@pytest.mark.parametrize("call", CALLS)
def test_memory_of_a_failed_decode_is_not_handed_on(lib, call):
    """A launch that fails leaves the scan before it on the stream: the handle's
    memory goes back to the driver, whose cudaFree waits, and not to the next handle."""
    h = _open(lib)
    assert CALLS[call](lib, h) == 0
    lib.stride_close(h)
    assert not lib.fake_returned()  # kept for the next handle
    h = _open(lib)
    lib.fake_decode(_lib.STRIDE_ERR_CUDA, 0)
    assert CALLS[call](lib, h) == _lib.STRIDE_ERR_CUDA
    lib.fake_decode(0, 0)
    lib.stride_close(h)
    assert lib.fake_returned()


@pytest.mark.parametrize("shape", [4, 1])
def test_failed_host_decode_leaves_nothing_running(lib, shape):
    """In the one-kernel and the two-kernel shape."""
    h = _open(lib)
    cfg = _lib.LaunchCfg()
    cfg.warps_per_cta, cfg.persistent, cfg.stage_bytes, cfg.code_bytes = 4, shape, 16384, 16384
    assert lib.stride_set_config(h, ctypes.byref(cfg)) == 0
    lib.fake_decode(_lib.STRIDE_ERR_CUDA, 0)
    assert lib.stride_decode(h, S, AT, AT, None) == _lib.STRIDE_ERR_CUDA
    assert lib.fake_pending(S)  # a device decode does not wait
    assert lib.stride_decode_host(h, S, AT, AT) == _lib.STRIDE_ERR_CUDA
    assert not lib.fake_pending(S)
    lib.stride_close(h)


OUTPUTS = {
    "ranges": lambda lib, h, s=S: lib.stride_meshlet_ranges(h, s, AT, AT),
    "bounds": lambda lib, h, s=S: lib.stride_meshlet_bounds(h, s, AT, AT),
    "side_table": lambda lib, h, s=S: lib.stride_side_table(h, s, AT, AT),
}


@pytest.mark.parametrize("call", OUTPUTS)
def test_outputs_after_a_reload_that_could_not_allocate(lib, call):
    h = _open(lib)
    assert lib.stride_decode(h, S, AT, AT, None) == 0
    assert lib.stride_finish(h, S, None) == 0
    assert OUTPUTS[call](lib, h) == 0
    lib.fake_most(len(SMALL))
    assert lib.stride_reload(h, LARGE, len(LARGE), S) == _lib.STRIDE_ERR_CUDA
    n = lib.fake_outputs()
    assert OUTPUTS[call](lib, h) != 0
    assert lib.fake_outputs() == n and not lib.fake_freed_used()  # nothing launched on the memory given back
    lib.fake_most(1 << 40)
    assert lib.stride_reload(h, LARGE, len(LARGE), S) == 0
    assert lib.stride_decode(h, S, AT, AT, None) == 0
    assert OUTPUTS[call](lib, h) == 0
    lib.stride_close(h)


def test_status_of_a_replayed_decode(lib):
    """A decode captured, then one run eagerly and checked, then the captured one
    replayed: the status is the replay's."""
    h = _open(lib)
    lib.fake_capture(S)
    assert lib.stride_decode(h, S, AT, AT, None) == 0
    lib.fake_capture(None)
    assert lib.stride_decode(h, S, AT, AT, None) == 0
    assert lib.stride_finish(h, S, None) == 0
    bad = ctypes.c_uint32()
    for err, rc in ((CORRUPT, _lib.STRIDE_ERR_CORRUPT), (0, 0)):
        lib.fake_replay(err)
        assert lib.stride_status(h, 1, ctypes.byref(bad)) == rc
        assert lib.stride_finish(h, S, ctypes.byref(bad)) == rc
        assert bad.value == (3 if err else 0)
        for call in OUTPUTS.values():
            assert call(lib, h) == rc
    lib.stride_close(h)


@pytest.mark.parametrize("call", OUTPUTS)
def test_calls_after_a_captured_one(lib, call):
    """A call captured after an eager one, and eager calls after it."""
    h = _open(lib)
    assert lib.stride_decode(h, S, AT, AT, None) == 0
    assert lib.stride_finish(h, S, None) == 0
    assert OUTPUTS[call](lib, h) == 0
    lib.fake_capture(S)
    assert OUTPUTS[call](lib, h) == 0
    lib.fake_capture(None)
    assert OUTPUTS[call](lib, h) == 0
    assert lib.stride_reload(h, SMALL, len(SMALL), S) == 0
    assert lib.stride_decode(h, S, AT, AT, None) == 0
    assert lib.stride_finish(h, S, None) == 0
    lib.stride_close(h)
    assert lib.fake_returned()  # the capture's replays may still use it
