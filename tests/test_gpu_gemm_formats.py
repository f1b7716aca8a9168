"""The tensor-core GEMM at the edges of its tiles, in every mode, against the fp64 product.

Rows: one, both sides of the 64 below which every mode runs in the native format, both sides of a 128-row tile, a ragged
third tile, more tiles than SMs (several per block). Columns: the least, both sides of a column tile's width of 64, 128 and 256, several tiles. Contraction: less than
a step of 32, a ragged last step, both sides of the 1024 after which the native format's exact sums are read out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 4, 4), (1, 256, 32), (63, 60, 36), (64, 64, 64), (65, 68, 60), (127, 128, 128), (128, 132, 96), (129, 192, 100),
          (257, 256, 1020), (257, 260, 1024), (130, 64, 1028), (300, 512, 2052), (5000, 256, 256), (2500, 768, 512),
          (40001, 64, 160), (40001, 128, 96), (40001, 256, 288)]


@pytest.fixture(scope="module")
def calc(lib_path, models):
    from pet_kokkos_b200 import Calculator
    c = Calculator(*models("tiny"))
    yield c
    c.close()


@pytest.mark.parametrize("mode", ["native", "3xtf32", "tf32", "bf16"])
@pytest.mark.parametrize("shape", SHAPES)
def test_against_fp64(calc, shape, mode):
    m, n, k = shape
    rng = np.random.default_rng(m + n + k)
    A = rng.normal(size=(m, k)).astype(np.float32)
    W = rng.normal(size=(n, k)).astype(np.float32)
    if m > 3:  # rows whose scale lies far from the others', and one of zeros
        A[0] *= 1e30
        A[1] *= 1e-30
        A[2] = 0.0
    ref = A.astype(np.float64) @ W.T.astype(np.float64)
    size = np.abs(A).astype(np.float64) @ np.abs(W).T.astype(np.float64)  # what the rounding errors are relative to
    band = {"native": 2.0 ** -22, "3xtf32": 2.0 ** -20 + k * 2.0 ** -25, "tf32": 2.0 ** -10, "bf16": 2.0 ** -7}[mode]
    for transposed in (True, False):
        C = calc.gemm(A, W if transposed else np.ascontiguousarray(W.T), mode, transposed)
        assert np.isfinite(C).all()
        assert (np.abs(C - ref) <= band * size).all(), (shape, mode, (np.abs(C - ref) / np.maximum(size, 1e-300)).max())
        if m > 3:
            assert (C[2] == 0.0).all()


def test_native_sums_are_not_biased(calc):
    """The tensor core truncates its accumulator; the native format's split keeps that out of the result. A bias shows as a
    slope against the exact product: fp32 fused multiply-adds have none either (below 1e-8)."""
    rng = np.random.default_rng(3)
    for k in (32, 256, 2048):
        A = np.abs(rng.normal(size=(700, k))).astype(np.float32)
        W = np.abs(rng.normal(size=(256, k))).astype(np.float32)
        ref = A.astype(np.float64) @ W.T.astype(np.float64)
        C = calc.gemm(A, W, "native").astype(np.float64)
        assert abs((C * ref).sum() / (ref * ref).sum() - 1.0) < 1e-8
        assert np.sqrt(((C - ref) ** 2).mean()) < 1e-7 * np.sqrt((ref ** 2).mean())


@pytest.mark.parametrize("mode", ["native", "3xtf32"])
def test_a_pair_of_blocks_gives_the_bits_of_one(calc, mode):
    """Large GEMMs run on pairs of blocks that share a 256-row tile; a row's bits stay those of the one-block kernel. A ragged
    last tile whose second block has no rows, one that has a few, two column tiles, steps beyond a ring's length."""
    rng = np.random.default_rng(11)
    for m, n, k in [(38400 + 100, 256, 320), (38400 + 130, 256, 96), (20000, 512, 1056)]:
        A = rng.normal(size=(m, k)).astype(np.float32)
        W = rng.normal(size=(n, k)).astype(np.float32)
        for _ in range(3):  # (operands handed from block to block: look at more than one run)
            C = calc.gemm(A, W, mode)
            for r0 in (0, 12800, m - 3000):
                assert np.array_equal(C[r0:r0 + 3000], calc.gemm(A[r0:r0 + 3000], W, mode)), (m, n, k, r0)


@pytest.mark.parametrize("mode", ["native", "3xtf32", "tf32", "bf16"])
@pytest.mark.parametrize("shape", [(64, 64, 1024), (1, 128, 4096), (129, 256, 1024), (300, 192, 2048), (1000, 512, 2048),
                                   (648, 1024, 4096), (640, 256, 1056), (40, 64, 8192), (70, 128, 1152)])
def test_blocks_that_share_a_tile(calc, shape, mode):
    """Few tiles and a long contraction: the blocks of a cluster sum a run of it each and finish a slice of the columns each.
    Two, four and eight of them, tile widths of 64, 128 and 256, ragged rows, a length that cannot be shared out."""
    m, n, k = shape
    rng = np.random.default_rng(m + n + k)
    A = rng.normal(size=(m, k)).astype(np.float32)
    W = rng.normal(size=(n, k)).astype(np.float32)
    C = calc.gemm(A, W, mode)
    size = np.abs(A).astype(np.float64) @ np.abs(W).T.astype(np.float64)
    band = {"native": 2.0 ** -22, "3xtf32": 2.0 ** -20 + k * 2.0 ** -25, "tf32": 2.0 ** -10, "bf16": 2.0 ** -7}[mode]
    assert (np.abs(C - A.astype(np.float64) @ W.T.astype(np.float64)) <= band * size).all()
    if mode == "native":  # among so many rows that nothing is shared, the same rows have the same bits
        many = np.concatenate([A, rng.normal(size=(20000, k)).astype(np.float32)])
        assert np.array_equal(C, calc.gemm(many, W, mode)[:m])
