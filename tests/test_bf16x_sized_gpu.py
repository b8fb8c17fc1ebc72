"""lx_b200_bf16x_encode_sized: the bytes and the size of lx_bf16x_bytes + lx_bf16x_encode; lx_b200_bf16x_encode_rest, which finishes
elsewhere what turned out not to fit: the same bytes, and none outside its buffer. A stored weight's buffer is its encoding and no more."""

import ctypes

import numpy as np
import pytest
import torch

from dromos_b200 import abi, host
from oracle import dromos_oracle as O
from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,K,every", [(1, 128, 0), (9, 1000, 0), (5, 1024, 2), (300, 1000, 7), (3000, 512, 1), (2, 8192, 1), (6000, 256, 1)])
def test_size_and_bytes(lx, rows, K, every):
    w = util.bf16_normal((rows, K), 0.02, rows)
    if every:
        w[::every, ::3] = 0x0080  # more patches than slots
    want, base = O.bf16x_encode(w), rows * O.bf16x_row_bytes(K)
    src, need = util.dev(w), ctypes.c_int64(-1)
    for room in (0, want.size - base, max(0, want.size - base - 1), want.size - base + 100):
        enc = torch.full((base + room + 8,), 0xAB, dtype=torch.uint8, device="cuda")
        st = lx.lx_b200_bf16x_encode_sized(abi.ptr(src), rows, K, abi.ptr(enc), base + room, ctypes.byref(need), util.stream_ptr())
        assert need.value == want.size
        assert st == (0 if want.size <= base + room else abi.ERR_SCRATCH)
        if st == 0:
            assert np.array_equal(util.host(enc)[: want.size], want)
        assert bool((enc[base + room:] == 0xAB).all())
        if st:
            for rest in (want.size, want.size + 24, base + (want.size - base) // 2 // 8 * 8, base):
                out = torch.full((rest + 64,), 0xAB, dtype=torch.uint8, device="cuda")
                assert lx.lx_b200_bf16x_encode_rest(abi.ptr(src), rows, K, abi.ptr(enc), abi.ptr(out), rest, util.stream_ptr()) == 0
                assert rest < want.size or np.array_equal(util.host(out)[: want.size], want)
                assert bool((out[rest if rest < want.size else want.size:] == 0xAB).all())
    if want.size > base:  # finished where the rows are
        enc = torch.full((want.size,), 0xAB, dtype=torch.uint8, device="cuda")
        assert lx.lx_b200_bf16x_encode_sized(abi.ptr(src), rows, K, abi.ptr(enc), base, ctypes.byref(need), util.stream_ptr()) == abi.ERR_SCRATCH
        assert bool((enc[base:] == 0xAB).all())
        assert lx.lx_b200_bf16x_encode_rest(abi.ptr(src), rows, K, abi.ptr(enc), abi.ptr(enc), want.size, util.stream_ptr()) == 0
        assert np.array_equal(util.host(enc), want)
    stored = host.store_weight(lx, torch.from_numpy(w.view(np.int16)).cuda().view(torch.bfloat16), abi.W_BF16X)
    assert stored.data.numel() == want.size and np.array_equal(util.host(stored.data), want)
    assert stored.data.untyped_storage().nbytes() == want.size and stored.data.storage_offset() == 0  # what torch.save would write


def test_store_weight_without_room_for_two_buffers(lx, monkeypatch):
    rows, K = 300, 1000
    w = util.bf16_normal((rows, K), 0.02, 1)
    w[::7, ::3] = 0x0080
    want = O.bf16x_encode(w)
    src = torch.from_numpy(w.view(np.int16)).cuda().view(torch.bfloat16)
    real, sizes = torch.empty, []

    def empty(*a, **k):
        sizes.append(a[0])
        if len(sizes) == 2:
            raise torch.OutOfMemoryError("no room")
        return real(*a, **k)

    monkeypatch.setattr(torch, "empty", empty)
    stored = host.store_weight(lx, src, abi.W_BF16X)
    monkeypatch.undo()
    assert sizes == [rows * O.bf16x_row_bytes(K), want.size, want.size]
    assert np.array_equal(util.host(stored.data), want)


def test_refused_arguments(lx):
    src, enc, need = torch.zeros(4096, dtype=torch.uint8, device="cuda"), torch.zeros(4096, dtype=torch.uint8, device="cuda"), ctypes.c_int64(-1)
    base = 2 * O.bf16x_row_bytes(128)
    call = lx.lx_b200_bf16x_encode_sized
    assert call(abi.ptr(src), 0, 128, abi.ptr(enc), 4096, ctypes.byref(need), util.stream_ptr()) == 1
    assert call(abi.ptr(src), 2, 0, abi.ptr(enc), 4096, ctypes.byref(need), util.stream_ptr()) == 1
    assert call(abi.ptr(src), 2, 128, abi.ptr(enc), base - 1, ctypes.byref(need), util.stream_ptr()) == 1
    assert call(abi.ptr(src), 2, 128, enc.data_ptr() + 4, base, ctypes.byref(need), util.stream_ptr()) == 1
    assert call(None, 2, 128, abi.ptr(enc), base, ctypes.byref(need), util.stream_ptr()) == 1
    assert call(abi.ptr(src), 2, 128, abi.ptr(enc), base, None, util.stream_ptr()) == 1
    assert need.value == -1
    rest = lx.lx_b200_bf16x_encode_rest
    assert rest(abi.ptr(src), 0, 128, abi.ptr(src), abi.ptr(enc), 4096, util.stream_ptr()) == 1
    assert rest(abi.ptr(src), 2, 0, abi.ptr(src), abi.ptr(enc), 4096, util.stream_ptr()) == 1
    assert rest(abi.ptr(src), 2, 128, abi.ptr(src), abi.ptr(enc), base - 1, util.stream_ptr()) == 1
    assert rest(abi.ptr(src), 2, 128, abi.ptr(src), enc.data_ptr() + 4, base, util.stream_ptr()) == 1
    assert rest(abi.ptr(src), 2, 128, None, abi.ptr(enc), base, util.stream_ptr()) == 1
    assert rest(None, 2, 128, abi.ptr(src), abi.ptr(enc), base, util.stream_ptr()) == 1
