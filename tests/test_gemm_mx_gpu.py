"""lx_gemm_w on NVFP4 weights (weights multiplied as stored, activations as base-13 digits): against 64-bit sums at the edges of its
layouts (chunks of 8 to 64 rows, launches of 1024, weight panels, 256 values of K; weights of so few rows go in chunks of 16 or 32, and
the kernel of two instructions per step is in test_gemm_mx_kernels_gpu.py), rows that do not depend on the call they come in,
small values beside large ones, and the values that have no digits.

Bound: digits and remainders hold a value exactly, or within 2^-41 of its row's largest, or leave out what is below 2^-24 * K / 512 of the
row's typical values; products of digits are exact, their sums f32, and seven sums are put together with one f32 rounding each (the
last at full size): 1e-6 is twice the 4.8e-7 that may be left out at K = 4096."""

import ctypes

import numpy as np
import pytest
import torch

from dromos_b200 import abi, host
from tests import util

pytestmark = pytest.mark.gpu

LEVELS = [0, 0.5, 1, 1.5, 2, 3, 4, 6, -0.0, -0.5, -1, -1.5, -2, -3, -4, -6]


def values(data, scale, glob, N, K):
    q = data.view(N, K // 2)
    lut = torch.tensor(LEVELS, dtype=torch.float64, device="cuda")
    v = torch.stack((lut[(q & 15).long()], lut[(q >> 4).long()]), dim=2).view(N, K)
    return v * scale.view(N, K // 16).view(torch.float8_e4m3fn).double().repeat_interleave(16, 1) * glob


def product(lx, x, sw, M, N, K, beta=0.0, y=None, bias=None, alpha=1.0):
    y = torch.full((M, N), float("nan"), device="cuda") if y is None else y
    ws = torch.full((lx.lx_gemm_workspace_bytes(M, K, 0),), 0xFF, dtype=torch.uint8, device="cuda")
    assert lx.lx_gemm_w(abi.ptr(x), abi.F32 if x.dtype == torch.float32 else abi.BF16, x.stride(0), sw.ref(), 0, abi.ptr(bias), abi.F32, abi.ptr(y),
                        abi.BF16 if y.dtype == torch.bfloat16 else abi.F32, y.stride(0), M, N, K, alpha, beta, abi.ptr(ws), util.stream_ptr()) == 0
    util.check_status(lx)
    return y


def weight(lx, N, K, gen):
    return host.store_weight(lx, (torch.randn((N, K), generator=gen, device="cuda") * 0.02).to(torch.bfloat16), abi.W_NVFP4)


@pytest.mark.parametrize("M,N,K", [(1, 1, 256), (8, 31, 512), (9, 250, 1024), (16, 5000, 256), (18, 129, 2048), (32, 300, 512), (36, 1000, 1280), (37, 97, 256),
                                   (40, 4737, 512), (48, 640, 768), (56, 200, 512), (57, 300, 512), (64, 130, 4096), (65, 300, 512), (130, 2000, 1024), (1025, 260, 256)])
def test_against_64_bits_and_rows_alone(lx, M, N, K):
    gen = torch.Generator(device="cuda").manual_seed(M + N)
    sw = weight(lx, N, K, gen)
    w64 = values(sw.data, sw.scale, sw.glob, N, K)
    for x_f32, pad in ((False, 0), (False, 3), (True, 0)):
        wide = torch.randn((M, K + pad), generator=gen, device="cuda")
        x = (wide if x_f32 else wide.to(torch.bfloat16))[:, :K]
        y = product(lx, x, sw, M, N, K)
        want = x.to(torch.bfloat16).double() @ w64.T
        assert float((y.double() - want).norm() / want.norm()) <= 1e-6
        for m in {0, M // 2, M - 1}:
            assert torch.equal(product(lx, x[m:m + 1], sw, 1, N, K)[0], y[m])


def test_bias_alpha_beta_and_bf16_outputs(lx):
    M, N, K = 45, 333, 512
    gen = torch.Generator(device="cuda").manual_seed(1)
    sw = weight(lx, N, K, gen)
    x = torch.randn((M, K), generator=gen, device="cuda").to(torch.bfloat16)
    bias, old = torch.randn((N,), generator=gen, device="cuda"), torch.randn((M, N + 3), generator=gen, device="cuda")
    want = 0.5 * (x.double() @ values(sw.data, sw.scale, sw.glob, N, K).T + bias.double()) + 0.75 * old[:, :N].double()
    y = product(lx, x, sw, M, N, K, 0.75, old.clone()[:, :N], bias, 0.5)
    assert float((y.double() - want).norm() / want.norm()) <= 1e-6
    y = product(lx, x, sw, M, N, K, 0.0, torch.empty((M, N), dtype=torch.bfloat16, device="cuda"), bias, 0.5)
    assert float((y.double() - (want - 0.75 * old[:, :N].double())).norm() / want.norm()) <= 2.0**-8


def test_values_without_digits(lx):
    M, N, K = 12, 200, 512
    gen = torch.Generator(device="cuda").manual_seed(2)
    sw = weight(lx, N, K, gen)
    w64 = values(sw.data, sw.scale, sw.glob, N, K)
    x = torch.randn((M, K), generator=gen, device="cuda").to(torch.bfloat16)
    x[1, 7], x[2, 100] = float("inf"), float("-inf")
    x[3, 5] = float("nan")
    x[4] = 0
    x[5] *= 1e-30
    x[6] *= 1e30
    x[7, 3], x[7, 300] = 1e20, 1e-20
    x[8, ::5] = 0
    y = product(lx, x, sw, M, N, K).double()
    want = x.double() @ w64.T
    for m in (1, 2):  # an infinity times its weight, NaN where that is zero
        assert torch.equal(torch.nan_to_num(y[m], nan=0.5, posinf=1, neginf=-1), torch.nan_to_num(want[m], nan=0.5, posinf=1, neginf=-1))
    assert bool(torch.isnan(y[3]).all()) and bool((y[4] == 0).all())
    for m in (0, 5, 6, 7, 8, 9, 10, 11):
        assert float((y[m] - want[m]).norm() / want[m].norm()) <= 1e-6, m


def test_scales_with_a_sign(lx):
    M, N, K = 16, 140, 512
    gen = torch.Generator(device="cuda").manual_seed(3)
    sw = weight(lx, N, K, gen)
    sw.scale[::3] |= 0x80
    x = torch.randn((M, K), generator=gen, device="cuda").to(torch.bfloat16)
    want = x.double() @ values(sw.data, sw.scale, sw.glob, N, K).T
    assert float((product(lx, x, sw, M, N, K).double() - want).norm() / want.norm()) <= 1e-6


@pytest.mark.parametrize("M,N,K", [(3, 200, 512), (16, 300, 4096), (40, 130, 1024), (64, 97, 2560), (130, 300, 2048)])
@pytest.mark.parametrize("outliers", ["every-block", "every-other-value", "one"])
@pytest.mark.parametrize("factor", [64, 256, 1024, 4096, 2**13, 2**15, 2**20])
def test_small_values_beside_outliers(lx, M, N, K, outliers, factor):
    """Outputs whose weights are zero wherever the row has an outlier: what is left of the sum is as exact as any other. (Values of 0.05
    beside 0.05 * 2^20: 2^-41 of the outlier is 2^-21 of such a value, and few are rounded at all.) The other outputs are the
    outlier's product with thousands of small ones added to it: each of the K / 64 sums may be cut off at 2^-23 of it."""
    gen = torch.Generator(device="cuda").manual_seed(factor + M)
    sw = weight(lx, N, K, gen)
    at = {"every-block": torch.arange(5, K, 16), "every-other-value": torch.arange(1, K, 2), "one": torch.tensor([K // 2 + 11])}[outliers].cuda()
    rows = torch.arange(0, M, 2, device="cuda")  # plain rows stand beside them
    x = torch.randn((M, K), generator=gen, device="cuda") * 0.05
    x[rows[:, None], at[None, :]] *= factor
    x = x.to(torch.bfloat16)
    sw.data.view(N, K // 2)[: N // 2, at // 2] &= 0x0F  # (at is odd: the high half of its byte)
    y = product(lx, x, sw, M, N, K)
    want = x.double() @ values(sw.data, sw.scale, sw.glob, N, K).T
    for part, bound in ((slice(0, N // 2), 1e-6), (slice(N // 2, N), 1e-6 + K // 64 * 2.0**-23)):
        assert float(((y[:, part].double() - want[:, part]).norm(dim=1) / want[:, part].norm(dim=1)).max()) <= bound
    for m in {0, 1, M - 1}:
        assert torch.equal(product(lx, x[m:m + 1], sw, 1, N, K)[0], y[m])


def test_one_value_of_any_size(lx):
    """Weights that pick one activation each, rows whose values are of every size: 2^-33 of the row's largest and above come out as
    they are."""
    M, K = 16, 512
    N = K
    sw = weight(lx, N, K, torch.Generator(device="cuda").manual_seed(5))
    eye = torch.zeros((N, K // 2), dtype=torch.uint8, device="cuda")
    k = torch.arange(K, device="cuda")
    eye[k, k // 2] = torch.where(k % 2 == 0, 2, 0x20).to(torch.uint8)  # code 2 is 1.0
    sw.data.copy_(eye.view(-1).view(sw.data.dtype).view(sw.data.shape))
    sw.scale.view(torch.uint8).fill_(0x38)  # 1.0
    gen = torch.Generator(device="cuda").manual_seed(6)
    x = torch.randn((M, K), generator=gen, device="cuda") * torch.exp2(-torch.randint(0, 31, (M, K), generator=gen, device="cuda").float())
    x = x.to(torch.bfloat16)
    x[:, 7] = 3.5
    x = torch.where(x.abs() < 2.0**-31, torch.zeros_like(x), x)  # 2^-33 of 2 .. 4
    y = product(lx, x, sw, M, N, K)
    assert torch.equal(y / sw.glob, (x.double() * sw.glob).float() / sw.glob)


@pytest.mark.parametrize("M,K,x_f32", [(16, 512, False), (16, 512, True), (70, 2048, False), (1100, 256, True)])
def test_rows_with_infinities(lx, M, K, x_f32):
    """Any number of infinities: an infinity where all their products agree in sign, NaN where they do not or a weight is zero."""
    N = 150
    gen = torch.Generator(device="cuda").manual_seed(7)
    sw = weight(lx, N, K, gen)
    x = torch.randn((M, K), generator=gen, device="cuda")
    inf = float("inf")
    x[1, 7], x[1, 200] = inf, inf
    x[2, 3], x[2, 40] = inf, -inf
    x[3, 5], x[3, 6], x[3, K - 1] = -inf, -inf, -inf
    x[M - 1] = inf
    x[M - 2, K - 1], x[M - 2, 0] = inf, 3.4e38 if x_f32 else inf  # (the largest f32 values are infinite in bf16)
    x[M - 3, 9], x[M - 3, 10] = inf, float("nan")
    x = x if x_f32 else x.to(torch.bfloat16)
    y = product(lx, x, sw, M, N, K).double()
    finite = torch.isfinite(x.to(torch.bfloat16)).all(dim=1)
    w64 = values(sw.data, sw.scale, sw.glob, N, K)
    want = torch.where(torch.isfinite(x.to(torch.bfloat16)), 0.0, x.to(torch.bfloat16).double())[~finite] @ w64.T
    got = y[~finite]
    assert torch.equal(torch.nan_to_num(got, nan=0.5, posinf=1, neginf=-1), torch.nan_to_num(want, nan=0.5, posinf=1, neginf=-1))
    assert bool(torch.isinf(got[0]).any()) and bool(torch.isnan(got[0]).any())
    plain = x[finite].to(torch.bfloat16).double() @ w64.T
    assert float((y[finite] - plain).norm() / plain.norm()) <= 1e-6
    # with everything an epilogue adds, in bf16
    old, bias = torch.randn((M, N), generator=gen, device="cuda").to(torch.bfloat16), torch.randn((N,), generator=gen, device="cuda")
    y = product(lx, x, sw, M, N, K, 0.75, old.clone(), bias, -0.5)[~finite].double()
    assert torch.equal(torch.nan_to_num(y, nan=0.5, posinf=1, neginf=-1), torch.nan_to_num(-want, nan=0.5, posinf=1, neginf=-1))


@pytest.mark.parametrize("M,N,K", [(24, 28700, 512), (64, 40000, 256), (200, 14353, 512), (300, 9000, 768), (1000, 5000, 256)])
def test_several_tiles_per_sm(lx, M, N, K):
    """Tiles one after the other on an SM, of one chunk and of several, beginning in the middle of a panel of weights and going on into the
    next (300 and 1000 rows on 148 SMs), with stages that go again in some chunks and not in others."""
    gen = torch.Generator(device="cuda").manual_seed(M)
    sw = weight(lx, N, K, gen)
    x = torch.randn((M, K), generator=gen, device="cuda")
    x[torch.arange(0, M, 70, device="cuda"), K - 3] = 3e5
    x = x.to(torch.bfloat16)
    y = product(lx, x, sw, M, N, K)
    w64 = values(sw.data, sw.scale, sw.glob, N, K)
    for m0 in range(0, M, 128):
        want = x[m0:m0 + 128].double() @ w64.T
        got = y[m0:m0 + 128].double()
        assert float(((got - want).norm(dim=1) / want.norm(dim=1)).max()) <= 1e-6
    for m in {0, 1, M // 2, 70 * ((M - 1) // 70), M - 1}:
        assert torch.equal(product(lx, x[m:m + 1], sw, 1, N, K)[0], y[m])
    # bf16 outputs added to old ones: half a step of bf16 (its 8 bits: at most 2^-8 of the value) and the error of the sum
    old = torch.randn((M, N), generator=gen, device="cuda").to(torch.bfloat16)
    bias = torch.randn((N,), generator=gen, device="cuda")
    z = product(lx, x, sw, M, N, K, 0.75, old.clone(), bias, 0.5).double()
    for m0 in range(0, M, 128):
        want = 0.5 * (x[m0:m0 + 128].double() @ w64.T + bias.double()) + 0.75 * old[m0:m0 + 128].double()
        bound = 2.0**-8 * want.abs() + 1e-6 * want.norm(dim=1, keepdim=True)
        assert bool(((z[m0:m0 + 128] - want).abs() <= bound).all())


@pytest.mark.parametrize("M,K", [(16, 512), (64, 4096)])
def test_a_row_does_not_depend_on_what_its_neighbours_keep(lx, M, K):
    """Rows that keep their remainders (an outlier beside small values) and rows that drop theirs (one small value, 2^-18 of the rest) in
    the same stages: each as it is alone."""
    N = 200
    gen = torch.Generator(device="cuda").manual_seed(K)
    sw = weight(lx, N, K, gen)
    x = torch.randn((M, K), generator=gen, device="cuda").abs() + 0.5
    x[:, 33] = 1.7 * 2.0**-18
    x[::3, 40] = 2.0**14
    x = x.to(torch.bfloat16)
    y = product(lx, x, sw, M, N, K)
    want = x.double() @ values(sw.data, sw.scale, sw.glob, N, K).T
    assert float(((y.double() - want).norm(dim=1) / want.norm(dim=1)).max()) <= 1e-6
    for m in range(M):
        assert torch.equal(product(lx, x[m:m + 1], sw, 1, N, K)[0], y[m]), m
