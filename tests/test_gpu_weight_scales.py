"""A network whose weights are rescaled by powers of two that cancel exactly (a head's values against the output projection, a
head's queries against its keys, a gate's values against the layer after it, a norm's gains against the layer after it) is the
same function. The evaluation has to stay within the bands of the plain network: no tensor may be held to the scale of another."""
import numpy as np
import pytest
import torch

from oracle import pet_oracle as po
from pet_kokkos_b200 import checkpoint as ck, structures as st

pytestmark = pytest.mark.gpu


def heads_apart(t, h, rng):
    """Heads on scales of their own, values against the output projection and queries against keys."""
    D, hd = h["d_pet"], h["head_dim"]
    for p in [n[:-len(".input_linear.weight")] for n in t if n.endswith(".input_linear.weight")]:
        for head in range(h["num_heads"]):
            s, q = np.float32(2.0) ** rng.integers(-8, 9, size=2).astype(np.float32)
            at = slice(head * hd, (head + 1) * hd)
            for name in (".input_linear.weight", ".input_linear.bias"):
                t[p + name][head * hd:(head + 1) * hd] *= q
                t[p + name][D + head * hd:D + (head + 1) * hd] /= q
                t[p + name][2 * D + head * hd:2 * D + (head + 1) * hd] *= s
            t[p + ".output_linear.weight"][:, at] /= s


def features_apart(t, h, rng):
    """Columns of queries and keys, values of gates and gains of norms on scales of their own."""
    D = h["d_pet"]
    e = lambda n: np.float32(2.0) ** rng.integers(-6, 7, size=n).astype(np.float32)
    for p in [n[:-len(".w_in.weight")] for n in t if n.endswith(".w_in.weight")]:
        f = t[p + ".w_out.weight"].shape[1]
        s = e(f)
        t[p + ".w_in.weight"][:f] *= s[:, None]
        t[p + ".w_in.bias"][:f] *= s
        t[p + ".w_out.weight"] /= s
    for p in [n[:-len(".attention.input_linear.weight")] for n in t if n.endswith(".attention.input_linear.weight")]:
        s = e(D)
        for name in (".attention.input_linear.weight", ".attention.input_linear.bias"):
            t[p + name][:D] = (t[p + name][:D].T * s).T
            t[p + name][D:2 * D] = (t[p + name][D:2 * D].T / s).T
        g = e(D)
        t[p + ".norm_attention.weight"] *= g
        t[p + ".attention.input_linear.weight"] /= g
        g = e(D)
        t[p + ".norm_mlp.weight"] *= g
        t[p + ".mlp.w_in.weight"] /= g


@pytest.mark.parametrize("gemm", ["native", "3xtf32"])
@pytest.mark.parametrize("heads", [1, 2, 4])  # head sizes 64, 32, 16
@pytest.mark.parametrize("how", [heads_apart, features_apart])
def test_same_function(lib_path, tmp_path, how, heads, gemm):
    from pet_kokkos_b200 import Calculator
    shape = dict(d_pet=64, num_heads=heads, d_feedforward=64, cutoff=4.5)
    jp, sp = ck.write_random_checkpoint(tmp_path / "plain", shape, seed=5, init="scaled")
    meta, tens = ck.load_checkpoint(jp, sp)
    systems = [st.diamond(2, jitter=0.05, seed=0), st.random_mixture(40, 8.0, seed=3)]
    ref = po.evaluate(meta, tens, systems, dtype=torch.float64)
    there = {k: np.array(v, np.float32) for k, v in tens.items()}
    how(there, meta["hypers"], np.random.default_rng(7))
    ck.write_safetensors(tmp_path / "apart.safetensors", there)
    f_scale, e_scale = max(1.0, np.abs(ref["forces"]).max()), max(1.0, np.abs(ref["per_atom_energy"]).sum())
    f_band, e_band = {"native": (1e-5, 1e-6), "3xtf32": (3e-4, 3e-5)}[gemm]
    off = []
    for weights in (sp, str(tmp_path / "apart.safetensors")):
        c = Calculator(jp, weights, gemm=gemm)
        r = c.compute(systems)
        c.close()
        off.append((np.abs(r.forces - ref["forces"]).max() / f_scale, np.abs(r.energy - ref["energy"]).max() / e_scale))
        print(how.__name__, heads, gemm, "dF %.2e dE %.2e" % off[-1])
        assert off[-1][0] <= f_band and off[-1][1] <= e_band, off
    assert off[1][0] <= 4 * off[0][0] + 2e-6, off  # and about as good as the plain network's


def outliers(t, h, rng, binades):
    """An eighth of the features of every block's tokens and node rows stand out by 2^binades; the norms' gains damp them by as much."""
    up = np.float32(2.0) ** binades
    pick = lambda n: rng.choice(n, n // 8, replace=False)
    at, node = pick(h["d_pet"]), pick(h["d_node"])
    for n in t:
        if n.endswith((".compress.2.weight", ".compress.2.bias", ".center_contraction.weight", ".center_contraction.bias")):
            t[n][at] *= up
        if n.endswith((".center_expansion.weight", ".center_expansion.bias")):
            t[n][node] *= up
        if n.endswith(".center_contraction.weight"):
            t[n][:, node] /= up
        if n.endswith((".norm_attention.weight", ".norm_mlp.weight", ".norm_center_features.weight")):
            some = node if "center" in n else at
            t[n] *= up * np.float32(8.0 ** -0.5)  # the root mean square is the outliers' now
            t[n][some] /= up


@pytest.mark.parametrize("gemm", ["native", "3xtf32"])
@pytest.mark.parametrize("init,binades", [("scaled", 2), ("scaled", 4), ("n002", 3), ("n002", 6), ("n002", 12), ("n002", 20)])
def test_outliers_that_a_gain_damps(lib_path, tmp_path, init, binades, gemm):
    from pet_kokkos_b200 import Calculator
    shape = dict(d_pet=64, num_heads=2, d_feedforward=64, cutoff=4.5)
    jp, sp = ck.write_random_checkpoint(tmp_path / "plain", shape, seed=5, init=init)
    meta, tens = ck.load_checkpoint(jp, sp)
    systems = [st.diamond(2, jitter=0.05, seed=0), st.random_mixture(40, 8.0, seed=3)]
    there = {k: np.array(v, np.float32) for k, v in tens.items()}
    outliers(there, meta["hypers"], np.random.default_rng(7), binades)
    ck.write_safetensors(tmp_path / "out.safetensors", there)
    ref, fp32 = (po.evaluate(meta, there, systems, dtype=d) for d in (torch.float64, torch.float32))
    f_scale, e_scale = np.abs(ref["forces"]).max(), np.abs(ref["per_atom_energy"]).sum()
    c = Calculator(jp, str(tmp_path / "out.safetensors"), gemm=gemm)
    r = c.compute(systems)
    c.close()
    off = lambda forces, energy: (np.abs(forces - ref["forces"]).max() / f_scale, np.abs(energy - ref["energy"]).max() / e_scale)
    print("outliers", init, binades, gemm, "dF %.2e dE %.2e" % off(r.forces, r.energy), "fp32 dF %.2e dE %.2e" % off(fp32["forces"], fp32["energy"]))
    f_band, e_band = {"native": (1e-5, 1e-6), "3xtf32": (3e-4, 3e-5)}[gemm]
    dF, dE = off(r.forces, r.energy)
    assert dF <= f_band and dE <= e_band


def one_feature_damped(tmp_path, gain):
    jp, sp = ck.write_random_checkpoint(tmp_path / "plain", dict(d_pet=64, num_heads=2, d_feedforward=64, cutoff=4.5), seed=5, init="n002")
    meta, tens = ck.load_checkpoint(jp, sp)
    there = {k: np.array(v, np.float32) for k, v in tens.items()}
    for n in there:
        if n.endswith((".norm_attention.weight", ".norm_mlp.weight", ".norm_center_features.weight")):
            there[n][5] = gain
    ck.write_safetensors(tmp_path / "damped.safetensors", there)
    return meta, jp, sp, str(tmp_path / "damped.safetensors")


@pytest.mark.parametrize("gemm,damped,apart", [("native", 2.0 ** -6, True), ("native", 0.9, False), ("3xtf32", 2.0 ** -6, False),
                                               ("3xtf32", 2.0 ** -13, True), ("3xtf32", 0.0, False), ("bf16", 2.0 ** -13, False)])
def test_a_gain_that_spreads_a_weight_stays_out_of_it(lib_path, tmp_path, gemm, damped, apart):
    """Three norms a block run by themselves then, and nothing else changes: the GEMMs keep the format in which two of them share a launch
    (64 atoms: all do that can)."""
    from pet_kokkos_b200 import Calculator
    meta, jp, sp, damped_sp = one_feature_damped(tmp_path, damped)
    launches = []
    for weights in (sp, damped_sp):
        c = Calculator(jp, weights, gemm=gemm)
        c.compute([st.diamond(2, jitter=0.05, seed=0)])
        before = c.kernel_launches
        c.compute([st.diamond(2, jitter=0.05, seed=1)])
        launches.append(c.kernel_launches - before)
        c.close()
    h = meta["hypers"]
    assert launches[1] - launches[0] == (3 * h["num_gnn_layers"] * h["num_attention_layers"] if apart else 0), launches


def test_norms_apart_under_every_tier(lib_path, tmp_path, monkeypatch):
    """The rows and row maxima of norms by themselves in passes that make them again, edges in chunks: the same bits."""
    from pet_kokkos_b200 import Calculator
    monkeypatch.setenv("PET_EDGE_CHUNK", "900")
    _, jp, _, sp = one_feature_damped(tmp_path, 2.0 ** -6)
    results = []
    for tier in ("never", "wide", "layers"):
        c = Calculator(jp, sp, recompute=tier)
        r = c.compute([st.diamond(2, jitter=0.05, seed=0)])
        results.append((r.energy, r.forces, r.virial))
        c.close()
    for other in results[1:]:
        for x, y in zip(results[0], other):
            assert np.array_equal(x, y)
