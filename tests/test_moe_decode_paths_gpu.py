"""Few-token routed experts: rows on their word's boundary go step by step without bounds, others word by word. The same words in
the same order, so the same bits: a latent two bytes off its boundary takes the second way through the gate/up rows. Row lengths
around a step (512 values of the 8-bit formats and NVFP4, 256 of bf16) and a batch of steps."""

import pytest
import torch

from dromos_b200 import abi, host
from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wtype", [abi.W_BF16, abi.W_INT8, abi.W_FP8, abi.W_NVFP4])
@pytest.mark.parametrize("L,I", [(256, 16), (512, 528), (2064, 272), (2560, 1024)])
def test_same_bits_with_and_without_bounds(lx, wtype, L, I):
    E, T, top_k = 5, 3, 4
    gen = torch.Generator(device="cuda").manual_seed(L)
    make = lambda *shape: host.store_weight(lx, (torch.randn(shape, generator=gen, device="cuda") * 0.05).to(torch.bfloat16), wtype)
    gate_up, down = make(E, 2 * I, L), make(E, L, I)
    ids = torch.stack([torch.randperm(E, generator=gen, device="cuda")[:top_k] for _ in range(T)]).to(torch.int32)
    weights = torch.rand((T, top_k), generator=gen, device="cuda")
    room = torch.empty(T * L + 8, dtype=torch.bfloat16, device="cuda")
    values = torch.randn((T * L,), generator=gen, device="cuda").to(torch.bfloat16)
    ws = torch.empty(max(256, lx.lx_moe_decode_workspace_bytes(T, I, top_k)), dtype=torch.uint8, device="cuda")
    out = []
    for offset in (0, 1):
        latent = room[offset:offset + T * L]
        latent.copy_(values)
        y = torch.full((T, L), float("nan"), device="cuda")
        assert lx.lx_moe_experts_decode(abi.ptr(latent), abi.ptr(ids), abi.ptr(weights), gate_up.ref(), down.ref(), abi.ptr(y), abi.ptr(ws), T, L, I, top_k,
                                        util.stream_ptr()) == 0
        util.check_status(lx)
        out.append(y)
    assert torch.equal(out[0], out[1]) and bool(torch.isfinite(out[0]).all())


@pytest.mark.parametrize("wtype", [abi.W_BF16, abi.W_INT8, abi.W_FP8, abi.W_NVFP4, abi.W_BF16X])
@pytest.mark.parametrize("L,I", [(888, 16), (1032, 272), (2560, 1040)])
def test_same_bits_on_small_and_large_grids(lx, wtype, L, I):
    """Eight tokens take two output rows per warp (from 444 blocks on; 148 for BF16X) and, for the 8-bit formats, the gate/up kernel with
    more blocks per SM (from 296); a token alone neither."""
    E, T, top_k = 5, 8, 4
    step = 16 if wtype in (abi.W_INT8, abi.W_FP8, abi.W_NVFP4) else 8
    L = L // step * step
    gen = torch.Generator(device="cuda").manual_seed(L + I)
    make = lambda *shape: host.store_weight(lx, (torch.randn(shape, generator=gen, device="cuda") * 0.05).to(torch.bfloat16), wtype)
    gate_up, down = make(E, 2 * I, L), make(E, L, I)
    ids = torch.stack([torch.randperm(E, generator=gen, device="cuda")[:top_k] for _ in range(T)]).to(torch.int32)
    weights = torch.rand((T, top_k), generator=gen, device="cuda")
    latent = torch.randn((T, L), generator=gen, device="cuda").to(torch.bfloat16)
    ws = torch.empty(max(256, lx.lx_moe_decode_workspace_bytes(T, I, top_k)), dtype=torch.uint8, device="cuda")

    def experts(x, i, w):
        y = torch.full((x.shape[0], L), float("nan"), device="cuda")
        assert lx.lx_moe_experts_decode(abi.ptr(x), abi.ptr(i), abi.ptr(w), gate_up.ref(), down.ref(), abi.ptr(y), abi.ptr(ws), x.shape[0], L, I, top_k,
                                        util.stream_ptr()) == 0
        return y

    batch = experts(latent, ids, weights)
    for t in range(T):
        assert torch.equal(experts(latent[t:t + 1], ids[t:t + 1].contiguous(), weights[t:t + 1].contiguous())[0], batch[t])
    util.check_status(lx)
    assert bool(torch.isfinite(batch).all())
