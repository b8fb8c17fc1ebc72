"""How lx_gemm_w cuts up products on NVFP4 weights (lx_b200_gemm_mx_plan: the function the launches use, nothing launched), swept over
sizes on the CPU: the rings and their barriers lie inside the shared memory asked for, accumulators and scales side by side in
tensor memory, the chunks hold every row, and a workspace of lx_gemm_workspace_bytes, which is asked for without N, holds whatever N picks."""

import ctypes

import pytest

from dromos_b200 import abi

SMEM_MAX, TMEM_COLUMNS, SMS = 226 * 1024, 512, 148
NAMES = ("rows", "chunks", "cols0", "cols1", "x_bytes", "last_cols0", "last_x_bytes", "sub", "R", "SW", "SX", "turns", "sf0", "buffers", "smem", "workspace")


@pytest.fixture(scope="module")
def lib():
    return abi.Library(abi.default_library_path())


def plan(lib, M, N, K, sms=SMS):
    out = (ctypes.c_int32 * 16)()
    assert lib.lx_b200_gemm_mx_plan(M, N, K, sms, out) == 0, (M, N, K)
    return dict(zip(NAMES, out))


def test_bad_arguments(lib):
    out = (ctypes.c_int32 * 16)()
    for args in ((0, 64, 256, 148), (1025, 64, 256, 148), (1, 0, 256, 148), (1, 64, 0, 148), (1, 64, 128, 148), (1, 64, 256, 0)):
        assert lib.lx_b200_gemm_mx_plan(*args, out) == abi.ERR_INVALID, args
    assert lib.lx_b200_gemm_mx_plan(1, 64, 256, 148, None) == abi.ERR_INVALID


# What the query answered while all products went in chunks of 64 rows: buffers of that size are in use.
KNOWN = {(1, 4096): 328068, (8, 4096): 328096, (17, 4096): 852420, (33, 4096): 1311236, (40, 4096): 1311264, (64, 8192): 3932928,
         (100, 4096): 3539856, (1000, 4096): 31463584, (2000, 512): 3937536, (33, 4000): 1311236}


@pytest.mark.parametrize("M,K", KNOWN)
def test_the_workspace_is_as_large_as_ever(lib, M, K):
    assert lib.lx_gemm_workspace_bytes(M, K, 0) == KNOWN[M, K]


def columns(rows):
    return (7 * ((rows + 7) // 8 * 8) + 15) // 16 * 16


@pytest.mark.parametrize("K", [256, 1280, 4096, 8192, 53248, 2**21])
def test_plans(lib, K):
    stages, seen = K // 256, set()
    for M in [*range(1, 81), 88, 96, 97, 100, 128, 129, 130, 150, 192, 200, 255, 300, 512, 525, 777, 1000, 1023, 1024]:
        have = lib.lx_gemm_workspace_bytes(M, K, 0)
        for N in (1, 40, 250, 346, 1000, 1773, 4096, 9000, 14336, 28672):
            p = plan(lib, M, N, K)
            # rows
            assert p["rows"] % 8 == 0 and p["rows"] <= 64 and (p["chunks"] - 1) * p["rows"] < M <= p["chunks"] * p["rows"]
            last = M - (p["chunks"] - 1) * p["rows"]
            split = p["rows"] < ((M + (M + 63) // 64 - 1) // ((M + 63) // 64) + 7) // 8 * 8
            scales = 16 * (32 if p["cols0"] > 128 else 16) if split else 2048 * ((p["cols0"] + 127) // 128)
            assert split or p["chunks"] == 1 or p["cols1"]
            if p["cols1"]:
                assert p["rows"] > 32 and p["sub"] == 1 and p["cols0"] == 4 * p["rows"] <= 256 and p["cols1"] >= 3 * p["rows"]
                assert (p["last_cols0"], p["last_x_bytes"]) == (p["cols0"], p["x_bytes"])
            else:
                assert p["rows"] <= 32 and p["sub"] == 2 and p["cols0"] == columns(p["rows"]) <= 256
                assert p["last_cols0"] == columns(last) and p["last_x_bytes"] == 128 * columns(last) + scales
            cols = p["cols0"] + p["cols1"]
            assert p["x_bytes"] == 128 * cols + scales and p["x_bytes"] % 128 == p["last_x_bytes"] % 128 == 0  # bulk copies: 16 bytes
            # workspace: digits and remainders, a byte per row and eight stages, a factor per row
            used = 2 * stages * ((p["chunks"] - 1) * p["x_bytes"] + p["last_x_bytes"]) + p["chunks"] * ((stages + 7) // 8) * 64 + 4 * M
            if used < 2**31:
                assert p["workspace"] == used
            assert used <= have
            # shared memory: the rings, the scales' exchange, the barriers and the stages that go again
            assert 1 <= p["R"] <= 128 and p["SW"] >= 2 and p["SX"] >= 2
            box = (p["R"] + 7) // 8 * 1024
            rings = p["sub"] * (p["SW"] * box + p["SX"] * p["x_bytes"] + 2 * 128 * 16)
            assert rings + 8 * (2 * p["SW"] + 2 * p["SX"] + 13) + 8 + p["chunks"] * ((stages + 7) // 8) <= p["smem"] <= SMEM_MAX
            assert 128 * 128 <= p["smem"] - (p["sub"] * p["SW"] - 1) * box  # the tensor core reads 128 rows from the last box too
            # tensor memory
            assert p["turns"] in (1, 2, 4) and p["buffers"] in (1, 2) and p["buffers"] * cols <= p["sf0"]
            assert p["sf0"] + p["turns"] * p["sub"] * (16 + 16 * ((p["cols0"] + 127) // 128)) == TMEM_COLUMNS
            seen.add((p["cols1"] > 0, p["cols0"] > 128, split, split and last <= p["rows"] - 8))
    if K <= 8192:
        # each of the five kernels, and last chunks of fewer columns
        assert {s[:3] for s in seen} == {(False, False, False), (False, False, True), (False, True, False), (False, True, True), (True, True, False)}
        assert {s[:2] for s in seen if s[3]} == {(False, False), (False, True)}


def test_small_weights_are_split_and_large_ones_are_not(lib):
    assert plan(lib, 64, 28672, 8192)["rows"] == 64 and plan(lib, 64, 14336, 4096)["rows"] == 64
    assert plan(lib, 64, 4096, 4096)["rows"] == 16 and plan(lib, 64, 8192, 4096)["rows"] == 32
    assert plan(lib, 1024, 4096, 2**21)["rows"] == 64  # no split whose flags would take the rings' room
