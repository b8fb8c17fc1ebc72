"""BF16X rows whose 16 slices of K are 0 to 12 steps of 64 values long and begin in either half of a block (a warp takes four steps
out of shared memory at once): bit for bit the product of the bf16 matrix. Patches in every part of a row."""

import numpy as np
import pytest
import torch

from dromos_b200 import abi
from oracle import dromos_oracle as O
from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [64, 192, 1024, 1088, 3136, 4096, 4160, 4352, 4480, 5056, 6208, 12288], ids=str)
def test_bf16x_equals_bf16(lx, K):
    N = 3 * 148 * 16 + 48 if K <= 4480 else 176
    rng = np.random.default_rng(K)
    w = util.bf16_normal((N, K), 0.02, K)
    for r in rng.integers(0, N, 40):
        w[r, rng.integers(0, K, 3)] = O.f32_to_bf16_bits(np.float32([2.0**-60]))[0]
    w[5, ::7] = O.f32_to_bf16_bits(np.float32([-(2.0**-70)]))[0]  # more patches than slots
    a, b = util.DeviceWeight(util.make_weight(w, O.W_BF16)), util.DeviceWeight(util.make_weight(w, O.W_BF16X))
    for x_dt, x in ((abi.BF16, util.dev(util.bf16_normal((8, K), 1.0, 6))), (abi.F32, util.dev(util.f32_normal((8, K), 1.0, 6)))):
        for M in (1, 8):
            out = [torch.full((M, N), float("nan"), device="cuda") for _ in range(2)]
            for weight, y in zip((a, b), out):
                assert util.gemv(lx, x, x_dt, K, weight, y, abi.F32, N, M, N, K) == 0
            util.check_status(lx)
            assert torch.equal(out[0].view(torch.int32), out[1].view(torch.int32)), f"M={M} x={x_dt}"
