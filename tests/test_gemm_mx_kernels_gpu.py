"""lx_gemm_w on NVFP4 weights: each of its kernels (digits of a step in two instructions, or in one of up to 128 or 256 columns) with more
stages of K than a thread has scales in flight, odd counts of them, several chunks and a shorter last one, remainders, infinities,
signed scales and everything an epilogue adds; N is what picks the kernel, and lx_b200_gemm_mx_plan says that it does. Bounds as in
test_gemm_mx_gpu.py."""

import ctypes

import pytest
import torch

from dromos_b200 import abi, host
from tests import util
from tests.test_gemm_mx_gpu import product, values, weight

pytestmark = pytest.mark.gpu

ONE_128, ONE_256, TWO = (False, False), (False, True), (True, True)


def plan(lx, M, N, K):
    out = (ctypes.c_int32 * 16)()
    assert lx.lx_b200_gemm_mx_plan(M, N, K, torch.cuda.get_device_properties(0).multi_processor_count, out) == 0
    return {"kernel": (out[3] > 0, out[2] > 128), "rows": out[0], "chunks": out[1], "shorter": out[6] < out[4]}


@pytest.mark.parametrize("kernel,M,N,K,chunks,shorter", [
    (TWO, 40, 14336, 1280, 1, False), (TWO, 64, 14336, 2304, 1, False), (TWO, 130, 28672, 1280, 3, False),
    (ONE_256, 24, 14336, 2304, 1, False), (ONE_256, 64, 8192, 4096, 2, False), (ONE_256, 100, 3000, 2304, 4, True), (ONE_256, 150, 9000, 1280, 5, True),
    (ONE_128, 16, 14336, 2304, 1, False), (ONE_128, 40, 4096, 2304, 3, True), (ONE_128, 33, 1000, 4096, 3, True)])
def test_every_kernel(lx, kernel, M, N, K, chunks, shorter):
    p = plan(lx, M, N, K)
    assert (p["kernel"], p["chunks"], p["shorter"]) == (kernel, chunks, shorter), "the rule sends this to another kernel: pick another N"
    gen = torch.Generator(device="cuda").manual_seed(M + K)
    sw = weight(lx, N, K, gen)
    sw.scale.view(N, K // 16)[::3, ::5] |= 0x80
    w64 = values(sw.data, sw.scale, sw.glob, N, K)
    inf = float("inf")
    for x_f32 in (False, True):
        x = torch.randn((M, K + 3), generator=gen, device="cuda")[:, :K]  # (rows of f32 and of bf16 that begin on no 16 bytes)
        x[0, K - 3], x[M // 2, 300], x[M - 1, 5::16] = 3e5, 2e4, 4e3  # stages that go again: the last, the second, all of them
        x[3, 7], x[3, K - 1], x[M - 2, 20] = inf, -inf, inf
        x[5, K // 2] = float("nan")
        x = x if x_f32 else x.to(torch.bfloat16)
        y = product(lx, x, sw, M, N, K)
        xr = x.to(torch.bfloat16).double()
        finite = torch.isfinite(xr).all(dim=1)
        want = torch.where(finite[:, None], xr, 0.0) @ w64.T
        # (an outlier of 4000 in every block, added to thousands of small values: each of the K / 64 sums may be cut off at 2^-23 of it)
        assert float(((y[finite].double() - want[finite]).norm(dim=1) / want[finite].norm(dim=1)).max()) <= 1e-6 + K // 64 * 2.0**-23
        assert bool(torch.isnan(y[5]).all())
        for m in (3, M - 2):
            infinite = torch.where(torch.isinf(xr[m]), xr[m], 0.0)
            terms = infinite[torch.isinf(xr[m])][None, :] * w64[:, torch.isinf(xr[m])]  # (0 x infinity is NaN)
            exact = terms.sum(dim=1)
            assert torch.equal(torch.nan_to_num(y[m].double(), nan=0.5, posinf=1, neginf=-1), torch.nan_to_num(exact, nan=0.5, posinf=1, neginf=-1))
        for m in sorted({0, 1, 4, M // 2, M - 9, M - 1, p["rows"] * (p["chunks"] - 1)}):
            assert torch.equal(product(lx, x[m:m + 1], sw, 1, N, K)[0], y[m]), m
        # bias, alpha, beta, bf16 outputs: half a step of bf16 and the error of the sum
        old, bias = torch.randn((M, N), generator=gen, device="cuda").to(torch.bfloat16), torch.randn((N,), generator=gen, device="cuda")
        z = product(lx, x, sw, M, N, K, 0.75, old.clone(), bias, 0.5).double()
        full = 0.5 * (want + bias.double()) + 0.75 * old.double()
        bound = 2.0**-8 * full.abs() + (1e-6 + K // 64 * 2.0**-23) * want.norm(dim=1, keepdim=True)
        assert bool(((z - full).abs() <= bound)[finite].all())
    assert lx.lx_b200_last_error() == 0


@pytest.mark.parametrize("M", [33, 40, 64, 100])
def test_bits_do_not_depend_on_the_split(lx, M):
    """The same rows of a weight as part of matrices of different sizes, which are cut differently: the same bits."""
    K, sizes = 1280, (700, 4096, 9000, 14336, 28672)
    gen = torch.Generator(device="cuda").manual_seed(M)
    whole = weight(lx, sizes[-1], K, gen)
    x = torch.randn((M, K), generator=gen, device="cuda").to(torch.bfloat16)
    x[::7, K - 200] = 1e5
    results, cuts = [], set()
    for N in sizes:
        part = host.StoredWeight(whole.wtype, whole.data.view(-1)[: N * K // 2], whole.scale.view(-1)[: N * K // 16], whole.glob)
        results.append(product(lx, x, part, M, N, K)[:, : sizes[0]])
        cuts.add(plan(lx, M, N, K)["rows"])
    assert len(cuts) >= 2
    for y in results[1:]:
        assert torch.equal(y, results[0])
    util.check_status(lx)


def test_a_workspace_of_the_size_asked_for_is_enough(lx):
    """What lies behind the workspace's bytes is left alone, whichever way N has the rows cut."""
    for M, N, K in ((33, 1000, 4096), (40, 4096, 1280), (64, 4096, 4096), (100, 346, 1280), (1000, 1000, 256), (1025, 260, 256)):
        gen = torch.Generator(device="cuda").manual_seed(N)
        sw = weight(lx, N, K, gen)
        x = torch.randn((M, K), generator=gen, device="cuda").to(torch.bfloat16)
        n = lx.lx_gemm_workspace_bytes(M, K, 0)
        ws = torch.full((n + 4096,), 0xA5, dtype=torch.uint8, device="cuda")
        y = torch.empty((M, N), device="cuda")
        assert lx.lx_gemm_w(abi.ptr(x), abi.BF16, K, sw.ref(), 0, None, abi.F32, abi.ptr(y), abi.F32, N, M, N, K, 1.0, 0.0, abi.ptr(ws), util.stream_ptr()) == 0
        util.check_status(lx)
        assert bool((ws[n:] == 0xA5).all())
        assert torch.equal(y, product(lx, x, sw, M, N, K))
