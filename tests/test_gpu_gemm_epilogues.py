"""Every epilogue of the tensor-core GEMM in every operand format that runs it, at ragged widths, against fp64.

The widths are no multiple of a column tile (64, 128, 256) nor of a chunk of the epilogue (16 or 32 columns), the rows none of a
row tile; one shape is large enough for pairs of blocks, one long enough for blocks that share a tile. The bands are the operand
format's band on the sums (as in test_gpu_gemm_formats.py), carried through the epilogue by its derivative, and a few roundings."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMATS = ["f16x3", "f16x2", "f16", "bf16", "tf32x2", "tf32"]
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
    return {"f16x3": 2.0 ** -22, "f16x2": 2.0 ** -20 + k * 2.0 ** -25, "tf32x2": 2.0 ** -20 + k * 2.0 ** -25, "f16": 2.0 ** -10,
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
