"""The weight GEMM where values lie far from the largest of their row: the error stays relative to sum |a||w|, output by output, as
that of fused multiply-adds in fp32 would (2^-22 of it at most over a few hundred terms, in the native format; where most of a
sum goes over the native format's second accumulator, the truncating sum's 2^-20 + k 2^-25 of 3xTF32)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BAND = {"native": lambda k: 2.0 ** -22, "3xtf32": lambda k: 2.0 ** -20 + k * 2.0 ** -25, "tf32": lambda k: 2.0 ** -10, "bf16": lambda k: 2.0 ** -7}


@pytest.fixture(scope="module")
def calc(lib_path, models):
    from pet_kokkos_b200 import Calculator
    c = Calculator(*models("tiny"))
    yield c
    c.close()


def worst(calc, A, W, mode):
    ref = A.astype(np.float64) @ W.T.astype(np.float64)
    size = np.abs(A).astype(np.float64) @ np.abs(W).T.astype(np.float64)
    w = 0.0
    for transposed in (True, False):
        C = calc.gemm(A, W if transposed else np.ascontiguousarray(W.T), mode, transposed)
        assert np.isfinite(C).all()
        w = max(w, (np.abs(C - ref) / size).max())
    return w


@pytest.mark.parametrize("mode", ["native", "3xtf32", "tf32", "bf16"])
@pytest.mark.parametrize("shape", [(70, 72, 100), (300, 128, 256), (129, 512, 264), (130, 64, 1028), (300, 192, 2048), (19300, 256, 96)])
def test_rows_of_a_weight_on_scales_of_their_own(calc, shape, mode):
    """Output rows of a weight that lie up to 2^-60 below the others, and one of zeros."""
    m, n, k = shape
    rng = np.random.default_rng(m + n + k)
    A = rng.normal(size=(m, k)).astype(np.float32)
    W = rng.normal(size=(n, k)).astype(np.float32)
    W *= np.float32(2.0) ** rng.integers(-30, 31, size=(n, 1)).astype(np.float32)
    W[5] *= np.float32(1e-3)
    w = worst(calc, A, W, mode)
    assert w <= BAND[mode](k), np.log2(w)
    W[3] = 0.0
    assert (calc.gemm(A, W, mode)[:, 3] == 0.0).all()


@pytest.mark.parametrize("mode", ["native", "3xtf32", "tf32", "bf16"])
@pytest.mark.parametrize("spread", [2, 4, 6, 8])
@pytest.mark.parametrize("shape", [(70, 72, 100), (300, 128, 256), (129, 512, 264), (130, 64, 1028), (300, 192, 2048), (19300, 256, 96)])
def test_columns_that_share_a_factor(calc, shape, spread, mode):
    """A column of A larger by a power of two and the weight's smaller by it (a gain before a linear layer, say): the products are
    what they were, most values lie 2^-spread and more below the largest of their rows, on both sides."""
    m, n, k = shape
    rng = np.random.default_rng(m + n + k + spread)
    f = np.float32(2.0) ** rng.integers(-spread, spread + 1, size=k).astype(np.float32)
    A = rng.normal(size=(m, k)).astype(np.float32) * f
    W = rng.normal(size=(n, k)).astype(np.float32) / f
    w = worst(calc, A, W, mode)
    assert w <= BAND["3xtf32" if mode == "native" else mode](k), np.log2(w)


@pytest.mark.parametrize("shape", [(70, 72, 100), (300, 128, 256), (19300, 256, 96)])
def test_rows_of_activations_with_outliers(calc, shape):
    """A few columns of A 2^6 to 2^12 above the others, with and without a weight that undoes them."""
    m, n, k = shape
    rng = np.random.default_rng(m + n + k)
    for up in (6, 9, 12):
        A, W = rng.normal(size=(m, k)).astype(np.float32), rng.normal(size=(n, k)).astype(np.float32)
        A[:, :3] *= np.float32(2.0) ** up
        assert worst(calc, A, W, "native") <= BAND["3xtf32"](k)
        W[:, :3] /= np.float32(2.0) ** up
        assert worst(calc, A, W, "native") <= BAND["3xtf32"](k)


def test_bits_of_a_row_with_every_product(calc):
    """A weight that asks for every product: a row's bits are still its own, alone, among many and where blocks share a tile."""
    rng = np.random.default_rng(2)
    for n, k in [(256, 256), (64, 2048)]:
        f = np.float32(2.0) ** rng.integers(-6, 7, size=k).astype(np.float32)
        A = rng.normal(size=(20000, k)).astype(np.float32) * f
        W = rng.normal(size=(n, k)).astype(np.float32) / f
        C = calc.gemm(A, W, "native")
        for r in (1, 70, 700):
            assert np.array_equal(C[:r], calc.gemm(A[:r], W, "native"))
