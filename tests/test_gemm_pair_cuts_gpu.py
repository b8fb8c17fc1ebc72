"""lx_gemm_w beyond 64 rows where the last tiles are cut between two pairs of SMs: bit for bit the rows of calls of at most 64
rows, whose tiles are whole. The f32 sums change hands as they are, so no tolerance is needed."""

import pytest
import torch

from dromos_b200 import abi, host
from tests import util

pytestmark = pytest.mark.gpu

KINDS = [("bf16", abi.W_BF16, 0), ("int8", abi.W_INT8, 0), ("fp8", abi.W_FP8, 0), ("int8-int8", abi.W_INT8, 1), ("fp8-fp8", abi.W_FP8, 2)]
# Tiles of 256 weight rows x 64 .. 256 columns on 74 pairs of SMs: a little more than one tile per pair, nearly two, one and a half
# (shares that hold no whole tile), several whole turns first, a ragged end of rows and columns; cuts close to a tile's end.
SHAPES = [(256, 19200, 2048), (250, 36900, 1024), (512, 14336, 4096), (1000, 20001, 1552), (2049, 10000, 1024), (300, 9700, 4096)]


def product(lx, sw, math, x, y, ws_fill, m, N, K, beta):
    ws = torch.full((lx.lx_gemm_workspace_bytes(m, K, math),), ws_fill, dtype=torch.uint8, device="cuda")
    dt = abi.F32 if y.dtype == torch.float32 else abi.BF16
    x_dt = abi.F32 if x.dtype == torch.float32 else abi.BF16
    assert lx.lx_gemm_w(abi.ptr(x), x_dt, x.stride(0), sw.ref(), math, None, abi.F32, abi.ptr(y), dt, y.stride(0), m, N, K, 1.0, beta, abi.ptr(ws),
                        util.stream_ptr()) == 0
    return ws


@pytest.mark.parametrize("name,wtype,math", KINDS, ids=[k[0] for k in KINDS])
@pytest.mark.parametrize("M,N,K", SHAPES, ids=lambda v: str(v))
def test_rows_of_cut_tiles_equal_those_of_small_calls(lx, name, wtype, math, M, N, K):
    gen = torch.Generator(device="cuda").manual_seed(N)
    sw = host.store_weight(lx, (torch.randn((N, K), generator=gen, device="cuda") * 0.02).to(torch.bfloat16), wtype)
    x = torch.randn((M, K), generator=gen, device="cuda").to(torch.bfloat16)
    old = torch.randn((M, N), generator=gen, device="cuda")
    want = old.clone()
    for m0 in range(0, M, 64):
        product(lx, sw, math, x[m0:], want[m0:], 0xFF, min(64, M - m0), N, K, 0.5)
    for fill in (0xFF, 0x00):  # the flags are the call's own to clear
        y = old.clone()
        product(lx, sw, math, x, y, fill, M, N, K, 0.5)
        util.check_status(lx)
        assert torch.equal(y, want)


def test_cut_tiles_in_replayed_graphs_and_on_two_streams(lx):
    """The same workspace again and again (flags of the call before in it), and calls side by side with a workspace each."""
    M, N, K = 512, 14336, 1024
    gen = torch.Generator(device="cuda").manual_seed(1)
    sw = host.store_weight(lx, (torch.randn((N, K), generator=gen, device="cuda") * 0.02).to(torch.bfloat16), abi.W_BF16)
    xs = [torch.randn((M, K), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(2)]
    want = []
    for x in xs:
        y = torch.zeros((M, N), device="cuda")
        for m0 in range(0, M, 64):
            product(lx, sw, 0, x[m0:], y[m0:], 0, 64, N, K, 0.0)
        want.append(y)
    torch.cuda.synchronize()
    ys = [torch.zeros((M, N), device="cuda") for _ in xs]
    wss = [torch.empty(lx.lx_gemm_workspace_bytes(M, K, 0), dtype=torch.uint8, device="cuda") for _ in xs]

    def call(i):
        assert lx.lx_gemm_w(abi.ptr(xs[i]), abi.BF16, K, sw.ref(), 0, None, abi.F32, abi.ptr(ys[i]), abi.F32, N, M, N, K, 1.0, 0.0, abi.ptr(wss[i]),
                            torch.cuda.current_stream().cuda_stream) == 0

    streams = [torch.cuda.Stream() for _ in xs]
    torch.cuda.synchronize()
    for _ in range(10):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                call(i)
    torch.cuda.synchronize()
    util.check_status(lx)
    assert torch.equal(ys[0], want[0]) and torch.equal(ys[1], want[1])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=streams[0]):
        call(0)
        call(0)
    for y in ys:
        y.zero_()
    torch.cuda.synchronize()
    for _ in range(5):
        graph.replay()
    torch.cuda.synchronize()
    util.check_status(lx)
    assert torch.equal(ys[0], want[0])
