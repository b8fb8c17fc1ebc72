"""The decode GEMV on weights that start on a 16-byte boundary but not on a 32-byte one: bit for bit the product of the same
weight on a 256-byte boundary."""

import ctypes

import pytest
import torch

from dromos_b200 import abi, host
from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wtype", [abi.W_BF16, abi.W_INT8, abi.W_FP8, abi.W_NVFP4])
@pytest.mark.parametrize("M", [1, 5, 8])
def test_weight_on_any_16_bytes(lx, wtype, M):
    N, K = 330, 1024
    gen = torch.Generator(device="cuda").manual_seed(M)
    sw = host.store_weight(lx, (torch.randn((N, K), generator=gen, device="cuda") * 0.02).to(torch.bfloat16), wtype)
    x = torch.randn((M, K), generator=gen, device="cuda").to(torch.bfloat16)
    raw = sw.data.view(torch.uint8).reshape(-1)
    room = torch.zeros(raw.numel() + 256, dtype=torch.uint8, device="cuda")
    out = []
    for offset in (0, 16):
        data = room[offset:offset + raw.numel()]
        data.copy_(raw)
        w = abi.make_weight(wtype, data, sw.scale, sw.glob)
        y = torch.full((M, N), float("nan"), device="cuda")
        assert lx.lx_gemv_w(abi.ptr(x), abi.BF16, K, ctypes.byref(w), None, abi.BF16, abi.ptr(y), abi.F32, N, M, N, K, 1.0, 0.0, util.stream_ptr()) == 0
        util.check_status(lx)
        out.append(y)
    assert torch.equal(out[0], out[1]) and bool(torch.isfinite(out[0]).all())
