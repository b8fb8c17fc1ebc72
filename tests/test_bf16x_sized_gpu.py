"""lx_b200_bf16x_encode_sized: the bytes and the size of lx_bf16x_bytes + lx_bf16x_encode, and what it answers when the buffer is too
small for the overflow records (then rows after the first that overflow are only counted: the size is exact all the same)."""

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
    stored = host.store_weight(lx, torch.from_numpy(w.view(np.int16)).cuda().view(torch.bfloat16), abi.W_BF16X)
    assert stored.data.numel() == want.size and np.array_equal(util.host(stored.data), want)


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
