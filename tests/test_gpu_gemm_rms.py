"""The RMSNorm that a GEMM takes with it: rows over their root mean squares, then the product, against fp64.

Row lengths with a remainder in the last step of 32 (16 for the tf32 parts) columns, an odd number of steps, one step; rows that leave
ragged tiles; one CTA a tile, pairs of CTAs, two GEMMs in one launch. The band is the operand format's on the sums of products of unit rows
(as in test_gpu_gemm_epilogues.py) and 2^-20 for the norm (K squares added up in fp32, the root's reciprocal, a product)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMATS = ["f16x3", "f16x3_full", "f16x2", "tf32x2"]
SHAPES = [(1, 8, 4), (65, 72, 36), (129, 200, 68), (300, 128, 96), (70, 320, 1152), (9600, 512, 256), (19201, 256, 100)]
EPS = 1.1920928955078125e-07


@pytest.fixture(scope="module")
def calc(lib_path, models):
    from pet_kokkos_b200 import Calculator
    c = Calculator(*models("tiny"))
    yield c
    c.close()


def problem(m, n, k, seed):
    rng = np.random.default_rng(seed)
    A = rng.normal(size=(m, k)) * 2.0 ** rng.integers(-20, 21, size=(m, 1))  # rows on scales of their own
    A[m // 2] = 0.0
    return A.astype(np.float32), (rng.normal(size=(n, k)) / np.sqrt(k)).astype(np.float32), rng.normal(size=n).astype(np.float32)


def expected(A, W, bias):
    d = lambda x: np.asarray(x, np.float64)
    x = d(A) / np.sqrt((d(A) ** 2).mean(1, keepdims=True) + EPS)
    return x @ d(W).T + d(bias), np.abs(x) @ np.abs(d(W)).T + np.abs(d(bias))


def band(fmt, k):
    return 2.0 ** -20 + {"f16x3": 2.0 ** -22, "f16x3_full": 2.0 ** -22}.get(fmt, 2.0 ** -20 + k * 2.0 ** -25)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("epi", ["plain", "swiglu"])
@pytest.mark.parametrize("fmt", FORMATS)
def test_against_fp64(calc, fmt, epi, shape):
    A, W, bias = problem(*shape, 3)
    z, size = expected(A, W, bias)
    C, pre, _ = calc.debug_gemm(A, W, fmt, epi, bias=bias, rms=True)
    got = C if epi == "plain" else pre
    assert np.isfinite(C).all()
    assert (np.abs(got - z) <= band(fmt, shape[2]) * size).all(), (np.abs(got - z) / size).max()
    if epi == "plain" and fmt.startswith("f16x3"):  # a row's bits do not depend on the others
        r = max(1, shape[0] // 3)
        assert np.array_equal(C[:r], calc.debug_gemm(A[:r], W, fmt, epi, bias=bias, rms=True)[0])


def warp_norm(A):
    """1 / rms in fp32 as a norm by itself has it: 32 lanes' sums of squares, added in pairs, a quotient of a root."""
    k = A.shape[1]
    x = np.zeros((len(A), -(-k // 32) * 32), np.float32)
    x[:, :k] = A
    s = np.zeros((len(A), 32), np.float32)
    for part in np.moveaxis(x.reshape(len(A), -1, 32), 1, 0):
        s = (part.astype(np.float64) ** 2 + s).astype(np.float32)  # one rounding: a fused multiply and add
    for o in (16, 8, 4, 2, 1):
        s = s + s[:, np.arange(32) ^ o]
    return np.float32(1) / np.sqrt(s[:, 0] / np.float32(k) + np.float32(EPS))


@pytest.mark.parametrize("shape", [(3000, 64, 100), (3000, 64, 128), (19201, 256, 256), (3000, 64, 512), (3000, 128, 1024), (3000, 256, 2048)])
@pytest.mark.parametrize("fmt", FORMATS)
def test_the_scale_is_no_further_off_than_a_norm_by_itself(calc, fmt, shape):
    """A column of ones against a weight that reads it alone: the product is the row's 1 / rms as it stands, no other sum with it."""
    m, n, k = shape
    A = np.random.default_rng(11).normal(size=(m, k)).astype(np.float32)
    A[:, k // 2] = 1.0
    W = np.zeros((n, k), np.float32)
    W[3, k // 2] = 1.0
    got = calc.debug_gemm(A, W, fmt, "plain", rms=True)[0][:, 3].astype(np.float64)
    true = 1.0 / np.sqrt((A.astype(np.float64) ** 2).mean(1) + EPS)
    off = lambda x: np.sqrt(np.mean((x / true - 1.0) ** 2)) * 2.0 ** 24
    print(fmt, shape, "off %.3f of 2^-24, by itself %.3f" % (off(got), off(warp_norm(A))))
    assert off(got) <= off(warp_norm(A))


TWO = [((130, 512, 512), (4460, 256, 128)), ((2900, 2048, 256), (19000, 512, 256))]  # a CTA a tile; and pairs of CTAs


@pytest.mark.parametrize("shapes", TWO)
@pytest.mark.parametrize("fmt", FORMATS)
def test_two_in_one_launch(calc, fmt, shapes):
    """The atoms' rows and the edges', one of them normed or both: the bits of one after the other."""
    for normed in ((True, True), (True, False), (False, True)):
        given = []
        for shape, rms in zip(shapes, normed):
            A, W, bias = problem(*shape, 5)
            given.append(dict(A=A, W=W, fmt=fmt, epilogue="swiglu", bias=bias, rms=rms))
        before = calc.kernel_launches
        results = calc.debug_gemm_two(*given)
        launches = calc.kernel_launches - before - (2 if fmt.startswith("f16") else 0)  # (the passes that look for A's row maxima)
        assert launches == (2 if fmt == "f16x3_full" else 1)
        for x, g in zip(results, given):
            assert np.array_equal(x[0], calc.debug_gemm(**g)[0])


def test_infinite_rows_and_refusals(calc):
    """A row whose squares overflow is over an infinite root, as the norm by itself has it; formats of one part are refused by name."""
    A, W, bias = problem(70, 64, 64, 7)
    A[3] = 2.0 ** 100
    C = calc.debug_gemm(A, W, "f16x3", "plain", bias=bias, rms=True)[0]
    assert np.isfinite(C).all() and np.array_equal(C[3], bias)
    for fmt in ("f16", "bf16", "tf32"):
        with pytest.raises(Exception, match="after a norm"):
            calc.debug_gemm(A, W, fmt, "plain", rms=True)
