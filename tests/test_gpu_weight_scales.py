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
