"""The load-time conversions take whole 16-byte words where buffers and rows allow and single values elsewhere: the same bytes
either way, at row lengths around a lane's, a warp's and an iteration's share, and the oracle's where it has them. Exact."""

import ctypes
import threading

import numpy as np
import pytest
import torch

from dromos_b200 import abi
from oracle import dromos_oracle as O
from tests import util

pytestmark = pytest.mark.gpu


def at_offset(nbytes, offset):
    """A device buffer of nbytes that starts `offset` bytes behind a 256-byte boundary."""
    return torch.zeros(nbytes + 256, dtype=torch.uint8, device="cuda")[offset:offset + nbytes]


def quantize(lx, w_dev, wtype, rows, K, offset):
    data = at_offset(rows * K // 2 if wtype == abi.W_NVFP4 else rows * K, offset)
    scale = at_offset(rows * K // 16 if wtype == abi.W_NVFP4 else 4 * rows, 0)
    lw = abi.make_weight(wtype, data, scale)
    assert lx.lx_quantize_weight(abi.ptr(w_dev), ctypes.byref(lw), rows, K, util.stream_ptr()) == 0
    out = at_offset(2 * rows * K, 2 * offset)
    assert lx.lx_dequantize_weight(ctypes.byref(lw), abi.ptr(out), rows, K, util.stream_ptr()) == 0
    return util.host(data), util.host(scale), np.float32(lw.glob), util.host(out)


@pytest.mark.parametrize("wtype,K", [(abi.W_INT8, 1), (abi.W_INT8, 8), (abi.W_INT8, 248), (abi.W_INT8, 256), (abi.W_INT8, 1000), (abi.W_INT8, 1032), (abi.W_FP8, 250), (abi.W_FP8, 264),
                                     (abi.W_FP8, 2056), (abi.W_NVFP4, 16), (abi.W_NVFP4, 272), (abi.W_NVFP4, 4112)])
def test_same_bytes_at_every_alignment(lx, wtype, K):
    rows = 35
    w = util.bf16_normal((rows, K), 0.02, K)
    w[4] = 0
    w[5, 0] = 0x8000
    if K > 16:
        w[6, K // 2] = 0x7FC1  # NaN: no part of a row's or block's maximum
    aligned = at_offset(2 * rows * K, 0)
    aligned.copy_(torch.from_numpy(w.view(np.uint8).reshape(-1)))
    ragged = at_offset(2 * rows * K, 2)
    ragged.copy_(aligned)
    want = quantize(lx, aligned, wtype, rows, K, 0)
    for src, offset in ((aligned, 1), (ragged, 0), (ragged, 1)):
        got = quantize(lx, src, wtype, rows, K, offset)
        for a, b in zip(want, got):
            assert np.atleast_1d(a).tobytes() == np.atleast_1d(b).tobytes()
    if K > 16:
        w[6, K // 2] = 0  # (the oracle has no rule for NaN)
        if wtype == abi.W_NVFP4:
            assert want[0].reshape(rows, -1)[6, K // 4] & 15 == 7  # NaN saturates like a large positive value
    oracle = O.quantize_weight(w, wtype)
    keep = np.ones((rows,), bool)
    keep[6] = False
    data = oracle.data.view(np.uint8).reshape(rows, -1)
    assert np.array_equal(want[0].reshape(rows, -1)[keep], data[keep])


@pytest.mark.parametrize("wtype", [abi.W_INT8, abi.W_FP8, abi.W_NVFP4])
@pytest.mark.parametrize("rows,K", [(1, 16), (1, 20000), (9, 16384), (4729, 1024), (4737, 1040), (1579, 3088), (4800, 256), (5001, 272)])
def test_expanded_values_for_few_wide_and_many_short_rows(lx, wtype, rows, K):
    """Rows in one piece or several, of one word a lane or four (from 4 x 148 blocks of eight pieces of 1024 values on), against
    the values one at a time (an output that is not on 16 bytes)."""
    w = torch.randn((rows, K), generator=torch.Generator(device="cuda").manual_seed(K), device="cuda").to(torch.bfloat16)
    want = quantize(lx, w, wtype, rows, K, 1)
    got = quantize(lx, w, wtype, rows, K, 0)
    for a, b in zip(want, got):
        assert np.atleast_1d(a).tobytes() == np.atleast_1d(b).tobytes()


@pytest.mark.parametrize("rows,K", [(5, 1000), (9, 1024), (3, 1160), (2, 1), (7, 120), (6, 128)])
def test_bf16x_same_bytes_at_every_alignment(lx, rows, K):
    w = util.bf16_normal((rows, K), 0.02, rows)
    w[0, ::3] = 0x0080  # more patches than slots
    w[rows - 1, K - 1] = 0x3F80
    want = O.bf16x_encode(w)
    for offset in (0, 2):
        src = at_offset(2 * rows * K, offset)
        src.copy_(torch.from_numpy(w.view(np.uint8).reshape(-1)))
        n = lx.lx_bf16x_bytes(abi.ptr(src), rows, K, util.stream_ptr())
        assert n == want.size
        enc = torch.full((n + 8,), 0xAB, dtype=torch.uint8, device="cuda")
        assert lx.lx_bf16x_encode(abi.ptr(src), rows, K, abi.ptr(enc), n, util.stream_ptr()) == 0
        assert np.array_equal(util.host(enc)[:n], want) and bool((enc[n:] == 0xAB).all())
        if n > rows * O.bf16x_row_bytes(K):
            assert lx.lx_bf16x_encode(abi.ptr(src), rows, K, abi.ptr(enc), n - 1, util.stream_ptr()) == 1
            assert lx.lx_bf16x_encode(abi.ptr(src), rows, K, abi.ptr(enc), n, util.stream_ptr()) == 0
        for out_offset in (0, 2):
            out = at_offset(2 * rows * K, out_offset)
            assert lx.lx_bf16x_decode(abi.ptr(enc), rows, K, abi.ptr(out), util.stream_ptr()) == 0
            assert np.array_equal(util.host(out), w.view(np.uint8).reshape(-1))


def test_sizes_asked_for_from_many_threads(lx):
    K = 512
    made = []
    for i in range(4):
        w = util.bf16_normal((16 + i, K), 0.02, i)
        w[: i + 1, ::3] = 0x0080
        made.append((util.dev(w), 16 + i, O.bf16x_encode(w).size))
    torch.cuda.synchronize()
    wrong = []

    def work(w_dev, rows, size):
        stream = torch.cuda.Stream()
        for _ in range(20):
            n = lx.lx_bf16x_bytes(abi.ptr(w_dev), rows, K, ctypes.c_void_p(stream.cuda_stream))
            if n != size:
                wrong.append((rows, n, size))

    threads = [threading.Thread(target=work, args=made[i % 4]) for i in range(12)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_bf16x_refused_buffer_holds_no_counts(lx):
    """A buffer one byte short of the overflow records: refused, nothing past it written, and every row in it either without patches or
    with patches in its own slots (a reader that ignores the status follows no record)."""
    rows, K = 300, 1000
    w = util.bf16_normal((rows, K), 0.02, 3)
    w[::7, ::3] = 0x0080
    row_bytes = O.bf16x_row_bytes(K)
    src = util.dev(w)
    n = lx.lx_bf16x_bytes(abi.ptr(src), rows, K, util.stream_ptr())
    assert n > rows * row_bytes
    for size in (rows * row_bytes, n - 1):
        enc = torch.full((n + 8,), 0xAB, dtype=torch.uint8, device="cuda")
        assert lx.lx_bf16x_encode(abi.ptr(src), rows, K, abi.ptr(enc), size, util.stream_ptr()) == 1
        host_bytes = util.host(enc)
        slots = host_bytes[: rows * row_bytes].reshape(rows, row_bytes)[:, :4].copy().view(np.uint32)[:, 0]
        assert np.all((slots == 0xFFFFFFFF) | (slots < 0x80000000))
        assert np.all(slots[::7] == 0xFFFFFFFF)
        assert np.all(host_bytes[rows * row_bytes:] == 0xAB)
    assert lx.lx_bf16x_encode(abi.ptr(src), rows, K, abi.ptr(enc), n, util.stream_ptr()) == 0
    assert np.array_equal(util.host(enc)[:n], O.bf16x_encode(w))
