"""The weight GEMM in each mode against a float64 product (the reference's tests/test_gemm_modes.cpp:34-103)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def random_matrix(r, c, seed):
    """Activation-like: unit normal entries, a few eight times larger (test_gemm_modes.cpp:34-44)."""
    rng = np.random.default_rng(seed)
    m = rng.normal(size=(r, c))
    i, j = np.meshgrid(np.arange(r), np.arange(c), indexing="ij")
    m[(i + j) % 97 == 0] *= 8.0
    return m.astype(np.float32)


def rel_error(C, A, W, transposed):
    ref = A.astype(np.float64) @ (W.T if transposed else W).astype(np.float64)
    return np.abs(C - ref).max() / np.abs(ref).max()


@pytest.fixture(scope="module")
def calc(lib_path, models):
    from pet_kokkos_b200 import Calculator
    c = Calculator(*models("tiny"))
    yield c
    c.close()


@pytest.mark.parametrize("transposed", [True, False])
@pytest.mark.parametrize("shape", [(300, 256, 192), (1000, 512, 1024), (129, 64, 40)])
def test_mode_error_bands(calc, transposed, shape):
    m, k, n = shape
    A = random_matrix(m, k, 1)
    W = random_matrix(n, k, 2) if transposed else random_matrix(k, n, 2)
    native = rel_error(calc.gemm(A, W, "native", transposed), A, W, transposed)
    tf32 = rel_error(calc.gemm(A, W, "tf32", transposed), A, W, transposed)
    x3 = rel_error(calc.gemm(A, W, "3xtf32", transposed), A, W, transposed)
    print(f"{shape} {'A W^T' if transposed else 'A W'}: native {native:.2e} tf32 {tf32:.2e} 3xtf32 {x3:.2e}")
    assert native < 1e-6                      # test_gemm_modes.cpp:88
    assert 10 * native < tf32 < 1e-2          # :89-90: as accurate as its precision, and no more
    assert x3 < 2e-5 and x3 < tf32 / 20       # fp32-class: the split recovers the bits tf32 drops


def test_native_rows_do_not_depend_on_the_batch(calc):
    """A row's bits are the same whatever the number of rows (the reference's batch-invariant GEMMs)."""
    A = random_matrix(700, 256, 3)
    W = random_matrix(512, 256, 4)
    full = calc.gemm(A, W, "native")
    part = calc.gemm(A[:77], W, "native")
    assert (full[:77] == part).all()


@pytest.mark.parametrize("fmt", ["tf32x2", "f16x2", "f16x3", "f16x3_full"])
def test_pairs_of_blocks_give_the_bits_of_one_block(calc, fmt):
    """A product of several parts runs on pairs of CTAs that share a 256 x 256 tile (tcgen05.mma.cta_group::2, each CTA with half of
    the weight's tile) once there are tiles enough, on single CTAs below. Both add the same products in the same order, so a row's
    bits are the same either way; one result is also held to the fp64 product. Shapes: every row tile full, a ragged last tile
    (and a pair whose second CTA has no rows at all), two column tiles, a contraction that is not a multiple of the 32-column
    stage, a long contraction."""
    rng = np.random.default_rng(5)
    for m, n, k in [(19200, 256, 256), (19001, 256, 264), (10100, 512, 512), (38500, 256, 992)]:  # (from 1024 columns on, blocks share a tile where there are few)
        A = rng.normal(size=(m, k)).astype(np.float32)
        W = rng.normal(size=(n, k)).astype(np.float32)
        pair = calc.debug_gemm(A, W, fmt)[0]
        for r0 in (0, m - 2000):
            assert np.array_equal(pair[r0:r0 + 2000], calc.debug_gemm(A[r0:r0 + 2000], W, fmt)[0]), (m, n, k, r0)
        ref = A.astype(np.float64) @ W.T.astype(np.float64)
        err = np.abs(pair - ref).max() / np.abs(ref).max()
        assert err <= 2e-6 + 0.5 * (3 * k / 8) * 2.0 ** -24, (m, n, k, err)


@pytest.mark.parametrize("mode", ["3xtf32", "tf32", "bf16"])
def test_token_row_gemm_of_the_benchmark(calc, mode):
    """The most frequent GEMM of the 1728-atom benchmark at its full size (atoms + kept edges = 122 138 rows, d_pet 256
    in and out), in every tensor-core mode, against the fp64 product (an ncu capture of it is
    summarised under profiles/)."""
    m, n, k = 122138, 256, 256
    rng = np.random.default_rng(0)
    A = rng.normal(size=(m, k)).astype(np.float32)
    W = rng.normal(size=(n, k)).astype(np.float32)
    C = calc.gemm(A, W, mode)
    C = calc.gemm(A, W, mode)  # the second launch is the one a profile reads: the first one loads the kernel
    ref = A[:4096].astype(np.float64) @ W.T.astype(np.float64)
    err = np.abs(C[:4096] - ref).max() / np.abs(ref).max()
    tail = A[-300:].astype(np.float64) @ W.T.astype(np.float64)
    err = max(err, np.abs(C[-300:] - tail).max() / np.abs(tail).max())
    band = {"3xtf32": 2e-6 + 0.5 * (3 * k / 8) * 2.0 ** -24, "tf32": 2e-3, "bf16": 2e-2}[mode]
    assert err <= band, (mode, err)
