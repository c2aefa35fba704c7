"""Damaged PLDT v5 streams in each of the decoder's kernels: eight and sixteen
meshlets per CTA and the general kernel, with long codewords, wide values, boundary
references, unreached vertices and raw ids that the FIFO still holds.  A stream that
the oracle rejects is rejected, any other rejected or decoded to the oracle's output,
and most damage to fixed-width values is decoded."""
import numpy as np
import pytest

import oracle
from test_gpu_pldt5_team import CASES, _stream, torch_cuda  # noqa: F401

pytestmark = pytest.mark.gpu

# case -> meshlets per CTA
KERNELS = {"seven": 8, "eight_again": 8, "nine_long": 8, "fixed_32": 8, "unreached": 8, "nine_bit_ids": 8, "most_tokens": 8,
           "most_bytes": 8, "groups_of_16": 16, "more_tokens": 0, "more_bytes": 0}


def _body(data, n):
    """First byte of the n meshlets: what the first entry of the table before it says."""
    at = oracle.parse_header_v5(data).boundary_bit // 8
    while int.from_bytes(data[at:at + 4], "big") != 8 * (at + 4 * n):
        at += 1
    return at + 4 * n


def _damaged(data, rng, name):
    n_m = CASES[name]["n"]
    body = _body(data, n_m)
    first = np.frombuffer(data, ">u4", n_m, body - 4 * n_m)
    for n in (len(data) - 1, (body + len(data)) // 2, body + 8):
        yield data[:n]
    for k in range(40):
        b = bytearray(data)
        # every other one near a meshlet's start: header, boundary references, strips
        at = int(rng.integers(8 * body, 8 * len(b)))
        if k % 2:
            at = min(int(first[rng.integers(len(first))]) + int(rng.integers(0, 200)), 8 * len(b) - 1)
        b[at >> 3] ^= 0x80 >> (at & 7)
        yield bytes(b)


@pytest.mark.parametrize("name", KERNELS)
def test_damaged_streams(torch_cuda, name):  # noqa: F811
    from meshpress_gb300 import ParaDeltaV5GpuDecoder
    from meshpress_gb300._lib import StrideFormatError
    data = _stream(CASES[name], 0)
    dec = ParaDeltaV5GpuDecoder(data)
    assert dec._lib.pldt5_meshlets_per_cta(dec._h) == KERNELS[name]
    dec.close()
    decoded = rejected = 0
    for bad in _damaged(data, np.random.default_rng(21), name):
        try:
            want = oracle.decode_v5(bad)
        except oracle.OracleError:
            want = None
        try:
            dec = ParaDeltaV5GpuDecoder(bad)
            try:
                pos, idx = dec.decode_to_host()
            finally:
                dec.close()
        except StrideFormatError:
            rejected += 1
            continue
        assert want is not None, "decoded, the oracle rejects it"
        assert np.array_equal(idx.astype(np.int64), want[1])
        assert np.array_equal(pos.view(np.uint32), want[0].view(np.uint32))
        decoded += 1
    assert rejected
    # four fifths of this stream are its values: of the twenty flips anywhere sixteen, on average
    assert name != "fixed_32" or decoded >= 8
