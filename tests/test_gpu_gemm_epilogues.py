"""Every epilogue of the tensor-core GEMM in every operand format that runs it, at ragged widths, against fp64; the sigmoid and its limits.

The widths are no multiple of a column tile (64, 128, 256) nor of a chunk of the epilogue (16 or 32 columns), the rows none of a
row tile; one shape is large enough for pairs of blocks, one long enough for blocks that share a tile. The bands are the operand
format's band on the sums (as in test_gpu_gemm_formats.py), carried through the epilogue by its derivative, and a few roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMATS = ["f16x3", "f16x3_full", "f16x2", "f16", "bf16", "tf32x2", "tf32"]
FORWARD = ["plain", "silu", "swiglu", "compress"]
BACKWARD = ["silu_bwd", "swiglu_bwd"]  # never packed in the tf32 formats
CASES = [(f, e) for f in FORMATS for e in FORWARD + (BACKWARD if not f.startswith("tf32") else [])]
SHAPES = [(1, 8, 4), (65, 72, 36), (129, 200, 68), (300, 136, 100), (257, 264, 1028), (70, 320, 1152), (9600, 520, 96), (19201, 256, 100)]


@pytest.fixture(scope="module")
def calc(lib_path, models):
    from pet_kokkos_b200 import Calculator
    c = Calculator(*models("tiny"))
    yield c
    c.close()


def band_of(fmt, k):
    return {"f16x3": 2.0 ** -22, "f16x3_full": 2.0 ** -22, "f16x2": 2.0 ** -20 + k * 2.0 ** -25, "tf32x2": 2.0 ** -20 + k * 2.0 ** -25, "f16": 2.0 ** -10,
            "tf32": 2.0 ** -10, "bf16": 2.0 ** -7}[fmt]


def sigmoid(x):
    with np.errstate(over="ignore"):
        return 1.0 / (1.0 + np.exp(-x))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fmt,epi", CASES)
def test_against_fp64(calc, fmt, epi, shape):
    m, n, k = shape
    rng = np.random.default_rng(m + n + k)
    draw = lambda *s: rng.normal(size=s).astype(np.float32)
    A, W = draw(m, k), (draw(n, k) / np.sqrt(k)).astype(np.float32)
    args, d = {}, lambda x: np.asarray(x, np.float64)
    acc = d(A) @ d(W).T
    err = band_of(fmt, k) * (np.abs(d(A)) @ np.abs(d(W)).T)
    u = 2.0 ** -21  # the sigmoid (2^-22) and the roundings after it
    if epi in FORWARD:
        args["bias"] = draw(n)
        z = acc + d(args["bias"])
        if epi == "plain":
            args["res"], args["res_row0"] = draw(m, n), m // 3
            z[m // 3:] += d(args["res"])[m // 3:]
        if epi == "compress":
            args.update(tab=draw(5, n), species=rng.integers(0, 5, size=m), wx=draw(n, 4), vec=rng.normal(size=(m, 3)))
            args["dist"] = np.linalg.norm(args["vec"], axis=1)
            z += d(args["tab"])[args["species"]] + d(args["wx"]) [None, :, 3] * args["dist"][:, None] + args["vec"] @ d(args["wx"])[:, :3].T
        err = err + 2.0 ** -20 * (np.abs(z) + 4.0)  # the terms added one after the other, each of them of order one
        if epi == "plain":
            ref, tol = z, err
        elif epi == "swiglu":
            v, g = z[:, 0::2], sigmoid(z[:, 1::2])
            ref = v * g
            tol = err[:, 0::2] * g + np.abs(v) * 0.25 * err[:, 1::2] + u * np.abs(ref)
        else:
            ref, tol = z * sigmoid(z), 1.1 * err + u * np.abs(z)
    elif epi == "silu_bwd":
        args["pre"] = draw(m, n)
        x = d(args["pre"])
        s = sigmoid(x)
        slope = s * (1.0 + x * (1.0 - s))
        ref, tol = acc * slope, err * np.abs(slope) + u * (1.0 + np.abs(x)) * np.abs(acc)
    else:
        args["pre"] = draw(m, 2 * n)
        v, s = d(args["pre"])[:, 0::2], sigmoid(d(args["pre"])[:, 1::2])
        ref, tol = np.empty((m, 2 * n)), np.empty((m, 2 * n))
        ref[:, 0::2], ref[:, 1::2] = acc * s, acc * v * s * (1.0 - s)
        tol[:, 0::2], tol[:, 1::2] = err * s + u * np.abs(acc), (err * 0.25 + u * np.abs(acc)) * np.abs(v)
    for transposed in (True, False):
        C, pre, row_max = calc.debug_gemm(A, W if transposed else W.T, fmt, epi, w_transposed=transposed, **args)
        assert np.isfinite(C).all()
        assert (np.abs(C - ref) <= tol).all(), (np.abs(C - ref) / tol).max()
        if pre is not None:
            assert (np.abs(pre - z) <= err).all(), (np.abs(pre - z) / err).max()
            other = calc.debug_gemm(A, W if transposed else W.T, fmt, epi, w_transposed=transposed, want_pre=False, **args)[0]
            assert np.array_equal(C, other)  # the same without the saved pre-activation
        assert np.array_equal(row_max, np.abs(C).max(axis=1))


def gates(calc, x):
    """sigmoid(x) as the SwiGLU epilogue computes it: values of one beside gates of x, both from the bias."""
    n = 2 * len(x)
    bias = np.ones(n, np.float32)
    bias[1::2] = x
    C, pre, _ = calc.debug_gemm(np.zeros((3, 4), np.float32), np.zeros((n, 4), np.float32), "f16x3", "swiglu", bias=bias)
    assert np.array_equal(pre[0], bias, equal_nan=True) and np.array_equal(C[0], C[2], equal_nan=True)
    return C[1]


def test_the_sigmoid(calc):
    """Within 2^-22 of itself (expf within one ulp, the sum, the last step of the reciprocal), with the quotient's limits; a result
    that is no normal number may be zero."""
    rng = np.random.default_rng(0)
    x = np.concatenate([np.linspace(-87.3, 87.3, 20000), rng.normal(size=40000), 1e-3 * rng.normal(size=4000), [0.0] * 4]).astype(np.float32)
    ref = sigmoid(x.astype(np.float64))
    assert (np.abs(gates(calc, x) - ref) <= 2.0 ** -22 * ref).all()
    low = np.linspace(-90.0, -87.3, 4000).astype(np.float32)
    assert (np.abs(gates(calc, low) - sigmoid(low.astype(np.float64))) <= 2.0 ** -126).all()
    far = np.array([-88.8, -1e3, -1e38, -np.inf, 1e3, 1e38, np.inf, 90.0], np.float32)
    assert np.array_equal(gates(calc, far), np.array([0, 0, 0, 0, 1, 1, 1, 1], np.float32))


@pytest.mark.parametrize("epi", ["silu", "swiglu", "silu_bwd", "swiglu_bwd", "compress"])
def test_what_is_not_a_number_stays_so(calc, epi):
    """A NaN in a gate or a pre-activation gives NaN in its own outputs and nowhere else."""
    m, n, k = 70, 72, 36
    rng = np.random.default_rng(1)
    A, W = rng.normal(size=(m, k)), rng.normal(size=(n, k))
    args, want = {}, np.zeros((m, {"swiglu": n // 2, "swiglu_bwd": 2 * n}.get(epi, n)), bool)
    if epi.endswith("bwd"):
        args["pre"] = rng.normal(size=(m, 2 * n if epi == "swiglu_bwd" else n))
        args["pre"][7, 11] = np.nan
        want[7, 10:12] = True  # the gate of a pair: both adjoints
        if epi == "silu_bwd":
            want[7, 10] = False
    else:
        args["bias"] = rng.normal(size=n)
        args["bias"][11] = np.nan
        want[:, 5 if epi == "swiglu" else 11] = True
        if epi == "compress":
            args.update(tab=rng.normal(size=(5, n)), species=rng.integers(0, 5, size=m), wx=rng.normal(size=(n, 4)), vec=rng.normal(size=(m, 3)),
                        dist=np.ones(m))
    assert np.array_equal(np.isnan(calc.debug_gemm(A, W, "f16x3", epi, **args)[0]), want)


def test_large_negative_values_do_not_pass_the_gate(calc):
    """silu(-1e38) is -0, not -1e38 times the smallest normal number."""
    bias = np.array([-1e38, -3e38, -1e30, 0.0], np.float32)
    C = calc.debug_gemm(np.zeros((2, 4), np.float32), np.zeros((4, 4), np.float32), "f16x3", "silu", bias=bias)[0]
    assert (C == 0.0).all()


def test_what_no_kernel_takes_is_refused(calc):
    """The backward epilogues are never packed in the tf32 formats: asked for, they fail by name."""
    for fmt in ("tf32", "tf32x2"):
        for epi, wide in (("silu_bwd", 1), ("swiglu_bwd", 2)):
            with pytest.raises(Exception, match="no kernel for this operand format"):
                calc.debug_gemm(np.ones((70, 8)), np.ones((32, 8)), fmt, epi, pre=np.zeros((70, 32 * wide)))
