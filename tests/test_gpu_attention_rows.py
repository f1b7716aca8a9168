"""The attention's backward by itself, on rows of dO that lie apart: what a query with a small row of dO gives dQ and dK, against fp64.

A query's row of dS reaches dQ on the scale of its own largest value, so dQ keeps the format's bits as long as the staged dO does (fp16 parts
on the tile's scale: two or three parts down to 2^-17 of the largest and more, one part to 2^-24 and more). dK sums over queries, on the tile's
scale: every row counts down to 2^-40 of the tile's bound.

The bands add up errors of their own signs by their squares, six of them wide. r is what a product of two operands loses in the format: 2^-12
of it in one part; 2^-21 and 2^-22 in two and three, the tensor core's truncations among it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = {"native": 2.0 ** -22, "tf32x3": 2.0 ** -21, "tf32": 2.0 ** -12}
SIZES = [(9, 16), (17, 32), (64, 16), (65, 32), (80, 32), (81, 32), (40, 64)]  # (tokens, head size)


@pytest.fixture(scope="module")
def calc(lib_path, models):
    from pet_kokkos_b200 import Calculator
    c = Calculator(*models("tiny"))
    yield c
    c.close()


def truth(q, k, v, g, cut, sc, r):
    """dQ, dK and the cutoffs' shares in fp64, each with its band."""
    sq = lambda x: x * x
    s = sc * q @ k.T + np.log(np.concatenate([[1.0], cut]))
    p = np.exp(s - s.max(1, keepdims=True))
    p /= p.sum(1, keepdims=True)
    dp = g @ v.T
    ds = p * (dp - (p * dp).sum(1, keepdims=True))
    score = sq(r * sc) * (sq(q) @ sq(k).T) + sq(2.0 ** -23 * s)  # variances; the last of a score's rounding and of exp
    mean = (sq(p) * score).sum(1, keepdims=True)
    prod = sq(r) * (sq(g) @ sq(v).T)
    out = (sq(p) * (prod + sq(dp) * (score + mean + sq(r)))).sum(1, keepdims=True)
    each = sq(p) * (prod + out) + sq(ds) * (score + mean + sq(r))
    band = lambda x: 6 * np.sqrt(x)
    return ((sc * ds @ k, band(sq(sc) * (each + sq(r * ds)) @ sq(k))), (sc * ds.T @ q, band(sq(sc) * (each + sq(r * ds)).T @ sq(q))),
            (ds.sum(0), band(each.sum(0))))


def one_atom(calc, mode, q, k, v, g, cut):
    """Two heads with the same rows, the atom between two others with rows of their own."""
    n, hd = q.shape
    D, T = 2 * hd, n + 4
    rng = np.random.default_rng(1)
    qkv, dm = rng.normal(size=(T, 3 * D)), rng.normal(size=(T, D))
    off = np.array([0, 1, n, n + 1])
    rows = np.concatenate([[1], 3 + 1 + np.arange(n - 1)])
    both = lambda x: np.concatenate([x, x], 1)
    qkv[rows] = np.concatenate([both(q), both(k), both(v)], 1)
    dm[rows] = both(g)
    cuts = np.concatenate([[0.5], cut, [0.25]])
    sc = hd ** -0.5
    merged, adj, cfh = calc.debug_attention(qkv, dm, off, cuts, 2, mode, sc)
    assert np.isfinite(adj).all() and np.isfinite(merged).all()
    adj = adj[rows].astype(np.float64)
    assert np.array_equal(adj[:, :hd], adj[:, hd:D])
    return adj[:, :hd], adj[:, D:D + hd], cfh[rows, 0]


def tokens(n, hd, seed):
    rng = np.random.default_rng(seed)
    f32 = lambda x: x.astype(np.float32).astype(np.float64)
    q, k, v, g = (f32(rng.normal(size=(n, hd))) for _ in range(4))
    return q, k, v, g, f32(rng.uniform(0.05, 1.0, size=n - 1))


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("mode", list(MODES))
def test_a_small_row_keeps_its_bits_in_dq(calc, mode, size):
    n, hd = size
    q, k, v, g, cut = tokens(n, hd, 3)
    down = {n // 3: 16, n - 1: 17} if mode != "tf32" else {n // 3: 23, n - 1: 24}
    for r, d in down.items():
        g[r] *= 2.0 ** -d
    dq, dk, cfh = one_atom(calc, mode, q, k, v, g, cut)
    for what, got, (t, band) in zip(("dq", "dk", "cut"), (dq, dk, cfh), truth(q, k, v, g, cut, hd ** -0.5, MODES[mode])):
        print(mode, size, what, (np.abs(got - t) / band).max(), (np.abs(got - t) / band).reshape(n, -1).max(1)[list(down)])
        assert (np.abs(got - t) <= band).all(), (what, (np.abs(got - t) / band).max())


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("mode", list(MODES))
def test_a_small_row_counts_in_dk(calc, mode, size):
    """Queries with large rows of dO see key 0 alone (scores 200 binades apart: the other weights are zero), so the other keys' dK is
    what the small rows give them."""
    n, hd = size
    q, k, v, g, cut = tokens(n, hd, 5)
    far = np.float64(np.float32(np.sqrt(100.0 * hd ** 0.5)))
    q[:, 0], k[:, 0] = 0.0, -far
    k[0, 0] = far
    small = np.arange(n) % 2 == 1
    q[~small, 0] = far
    g[small] *= 2.0 ** -26
    dq, dk, cfh = one_atom(calc, mode, q, k, v, g, cut)
    _, (tk, band), _ = truth(q, k, v, g, cut, hd ** -0.5, max(MODES[mode], 2.0 ** -14))  # dO's own rows, 2^-26 down, have 13 bits left
    # a row of dS on the tile's scale: to 2^-25 where the bound, 2.1 |dO| |V| taken up to a power of two, is at 2^15
    bound = 4.2 * np.sqrt((g ** 2).sum(1).max() * (v ** 2).sum(1).max())
    grid = 2.0 ** -40 * bound * hd ** -0.5 * np.abs(q).sum(0)
    off = np.abs(dk[1:] - tk[1:])
    print(mode, size, "dk off", (off / (band[1:] + grid)).max(), "if dropped", (np.abs(tk[1:]) / (band[1:] + grid)).max())
    assert (off <= band[1:] + grid).all()
