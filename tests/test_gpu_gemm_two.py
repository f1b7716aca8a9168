"""Two GEMMs that are handed over together run as one launch where that is expected to be faster: the same bits as one after the other.

The shapes reach every cut: few tiles of both (a tile a CTA), more tiles than CTAs with whole and partial rounds of the first GEMM's,
pairs of CTAs, tiles of the first shared by a cluster beside whole ones of the second. Row counts leave ragged tiles, and in one case a
pair whose second CTA has no rows. Launches are counted: one for both, but for weights whose values are spread, tf32 operands, and one
residual of two, and where the first one's 128 steps make the shared launch no faster."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMATS = ["f16x3", "f16x3_full", "f16x2", "f16", "bf16", "tf32x2", "tf32"]
CASES = [(f, e) for f in FORMATS for e in ["plain", "silu", "swiglu"] + (["silu_bwd", "swiglu_bwd"] if not f.startswith("tf32") else [])]
# rows, columns and contraction of the first and of the second
SHAPES = [((21, 512, 128), (366, 128, 128)), ((21, 128, 1024), (366, 128, 256)), ((64, 512, 2048), (4460, 128, 512)),
          ((648, 256, 1024), (24646, 256, 256)), ((300, 1024, 512), (40001, 256, 128)), ((2900, 2048, 256), (19000, 512, 256)),
          ((1, 64, 36), (30001, 64, 100)), ((130, 256, 4096), (129, 512, 64))]


@pytest.fixture(scope="module")
def calc(lib_path, models):
    from pet_kokkos_b200 import Calculator
    c = Calculator(*models("tiny"))
    yield c
    c.close()


@pytest.mark.parametrize("shapes", SHAPES)
@pytest.mark.parametrize("fmt,epi", CASES)
def test_the_bits_of_one_after_the_other(calc, fmt, epi, shapes):
    rng = np.random.default_rng(7)
    draw = lambda *s: rng.normal(size=s).astype(np.float32)
    given = []
    for m, n, k in shapes:
        g = dict(A=draw(m, k), W=(draw(n, k) / np.sqrt(k)).astype(np.float32), fmt=fmt, epilogue=epi)
        if epi.endswith("bwd"):
            g["pre"] = draw(m, 2 * n if epi == "swiglu_bwd" else n)
        else:
            g["bias"] = draw(n)
        if epi == "plain":
            g.update(res=draw(m, n), res_row0=m // 3)
        given.append(g)
    for kind in ("alike", "one residual"):
        if kind == "one residual":
            if epi != "plain":
                break
            given[1].pop("res"), given[1].pop("res_row0")
        apart = [calc.debug_gemm(**g) for g in given]
        for g, (C, _, _), (m, n, k) in zip(given, apart, shapes):  # (the single GEMM has its own tests: here that it is the right one)
            if epi == "plain" and "res" not in g:
                ref = g["A"][:200].astype(np.float64) @ g["W"].T.astype(np.float64) + g["bias"]
                assert np.abs(C[:200] - ref).max() <= 0.05 * np.abs(ref).max()
        # The formats of one or two parts add a long K in another order where a cluster shares a tile, which the cut decides: their
        # sums of k products of unit variance, truncated k/16 times on the way, may be 2^-23 (k/16) of sum |a||w| apart.
        # (No other epilogue shares a tile.)
        exact = epi != "plain" or fmt.startswith("f16x3") or max(k for _, _, k in shapes) < 1024
        before = calc.kernel_launches
        results = calc.debug_gemm_two(*given)
        launches = calc.kernel_launches - before - (2 if fmt.startswith("f16") else 0)  # (the passes that look for A's row maxima)
        if fmt in ("f16x3_full", "tf32") or kind == "one residual":
            assert launches == 2
        elif shapes != SHAPES[-1]:
            assert launches == 1
        for together, alone, (m, n, k) in zip(results, apart, shapes):
            for x, y in zip(together, alone):
                if exact or x is None:
                    assert x is y is None or np.array_equal(x, y)
                else:
                    assert np.abs(x - y).max() <= 2.0 ** -23 * (k / 16 + 2) * np.sqrt(k) * max(1.0, np.abs(y).max())
