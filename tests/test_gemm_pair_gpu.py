"""lx_gemm_w beyond 64 rows (pairs of SMs): bit for bit the same rows as calls of at most 64 rows, which other tests hold
against the oracle. The products multiply the same digits in the same order, so no tolerance is needed. Sizes at the edges
of the tiles: 256 weight rows, 16..256 columns, 128 bytes of K, one pass of 2048 rows."""

import pytest
import torch

from dromos_b200 import abi, host
from tests import util

pytestmark = pytest.mark.gpu

KINDS = [("bf16", abi.W_BF16, 0), ("int8", abi.W_INT8, 0), ("fp8", abi.W_FP8, 0), ("int8-int8", abi.W_INT8, 1), ("fp8-fp8", abi.W_FP8, 2)]
SHAPES = [(65, 256, 512), (70, 300, 528), (129, 513, 1040), (257, 1000, 2304), (700, 2500, 4096), (2049, 264, 272)]
# Several tiles per pair of SMs (3 to 21 by kind, on 74 pairs), so that both accumulators are used again and again; a short K, so that
# reading one out takes longer than filling the other.
DEEP = [(600, 14376, 272), (1000, 28700, 272)]


@pytest.mark.parametrize("name,wtype,math", KINDS, ids=[k[0] for k in KINDS])
@pytest.mark.parametrize("M,N,K", SHAPES, ids=lambda v: str(v))
def test_rows_equal_those_of_small_calls(lx, name, wtype, math, M, N, K):
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    sw = host.store_weight(lx, (torch.randn((N, K), generator=gen, device="cuda") * 0.02).to(torch.bfloat16), wtype)
    bias = torch.randn((N,), generator=gen, device="cuda")
    for x_f32, pad in ((False, 0), (False, 3), (True, 0)):  # rows that are read in place, unaligned rows, rounded rows
        wide = torch.randn((M, K + pad), generator=gen, device="cuda")
        wide = wide if x_f32 else wide.to(torch.bfloat16)
        x = wide[:, :K]
        out = []
        for rows in (M, 64):
            y = torch.full((M, N + 5), 0.25, device="cuda")
            for m0 in range(0, M, rows):
                m = min(rows, M - m0)
                ws = torch.full((lx.lx_gemm_workspace_bytes(m, K, math),), 0xFF, dtype=torch.uint8, device="cuda")
                assert lx.lx_gemm_w(abi.ptr(x[m0:]), abi.F32 if x_f32 else abi.BF16, x.stride(0), sw.ref(), math, abi.ptr(bias), abi.F32, abi.ptr(y[m0:]),
                                    abi.F32, N + 5, m, N, K, 0.5, 0.75, abi.ptr(ws), util.stream_ptr()) == 0
            util.check_status(lx)
            out.append(y)
        assert torch.equal(out[0], out[1]), f"{name} x_f32={x_f32} pad={pad}"
        assert torch.all(out[0][:, N:] == 0.25)


@pytest.mark.parametrize("name,wtype,math", KINDS, ids=[k[0] for k in KINDS])
@pytest.mark.parametrize("y_dtype,beta", [(torch.float32, 0.0), (torch.float32, 0.75), (torch.bfloat16, 0.0), (torch.bfloat16, 0.75)],
                         ids=["f32", "f32-beta", "bf16", "bf16-beta"])
@pytest.mark.parametrize("M,N,K", [(70, 300, 528)] + DEEP, ids=lambda v: str(v))
def test_many_tiles_and_output_types(lx, name, wtype, math, y_dtype, beta, M, N, K):
    gen = torch.Generator(device="cuda").manual_seed(N)
    sw = host.store_weight(lx, (torch.randn((N, K), generator=gen, device="cuda") * 0.02).to(torch.bfloat16), wtype)
    bias = torch.randn((N,), generator=gen, device="cuda")
    x = torch.randn((M, K), generator=gen, device="cuda").to(torch.bfloat16)
    old = torch.randn((M, N + 5), generator=gen, device="cuda").to(y_dtype)
    dt = abi.F32 if y_dtype == torch.float32 else abi.BF16
    out = []
    for rows in (M, 64):
        y = old.clone()
        if not beta:
            y[:, :N] = float("nan")  # not read
        for m0 in range(0, M, rows):
            m = min(rows, M - m0)
            ws = torch.full((lx.lx_gemm_workspace_bytes(m, K, math),), 0xFF, dtype=torch.uint8, device="cuda")
            assert lx.lx_gemm_w(abi.ptr(x[m0:]), abi.BF16, x.stride(0), sw.ref(), math, abi.ptr(bias), abi.F32, abi.ptr(y[m0:]), dt, N + 5, m, N, K, 0.5, beta,
                                abi.ptr(ws), util.stream_ptr()) == 0
        util.check_status(lx)
        out.append(y)
    assert torch.equal(out[0], out[1]) and bool(torch.isfinite(out[0]).all())
    assert torch.equal(out[0][:, N:], old[:, N:])
