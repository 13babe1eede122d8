"""The plan of the GEMM without a gather: tile width, parts of a cut tail, units of two tiles.  148 SMs are 74 pairs."""
import pytest

from symm_mem_recipes_b200._ext import C


@pytest.mark.parametrize("M,N,K,kw,want", [
    # with a residual two tiles at a time begin at K 3072: the plan knows what the launcher does
    (2048, 8192, 3584, dict(residual=True), (256, 74)), (2048, 8192, 3584, {}, (256, 0)),
    (4096, 8192, 3072, dict(residual=True), (256, 222)), (4096, 8192, 3064, dict(residual=True), (256, 0)),
    (16384, 3584, 8192, {}, (256, 444)), (16384, 3584, 8192, dict(elem_bytes=1), (256, 0)),
    (2048, 14336, 8192, dict(epilogue=1), (256, 222)), (2048, 14336, 8192, dict(epilogue=2), (256, 222)),
    # measured: 192 columns 66.5 us, 256 columns with two tiles at a time 69.6
    (1240, 8192, 3584, dict(residual=True), (192, 0)),
    # a width that is asked for
    (16384, 3584, 8192, dict(block_n=192), (192, 0)), (16384, 3584, 8192, dict(block_n=128), (128, 0)),
    (16384, 3584, 8192, dict(num_sms=32), (256, 448)), (8192, 1280, 8192, dict(block_n=256), (256, 0)),
])
def test_width_and_units(M, N, K, kw, want):
    plan = C.matmul_plan(M, N, K, **kw)
    assert (plan[0], plan[2]) == want


def test_units_are_whole_waves_of_256_column_tiles():
    for M in (129, 1000, 5000, 16384):
        for N in (512, 1280, 2304, 8192):
            for K in (1024, 3584, 5120, 8192):
                for kw in ({}, dict(residual=True), dict(epilogue=2), dict(num_sms=100), dict(elem_bytes=1)):
                    width, _, units = C.matmul_plan(M, N, K, **kw)
                    cols = N // 256 if kw.get("epilogue") else -(-N // 256)
                    pairs = kw.get("num_sms", 148) // 2
                    assert units == 0 or (width == 256 and units % pairs == 0 and units <= -(-M // 256) * (cols // 2))
