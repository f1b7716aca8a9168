"""The tensor-core attention on fp16 parts at the edges of its blocks: atoms with 1 to 17 tokens and on both sides of 32, 48, 80, 128
and 160 (blocks of 16, the widths the kernels are cut for, the warps' second turn), in every mode, against the fp64 oracle.

A cluster of n atoms within the cutoff of one another gives every atom n tokens."""
import numpy as np
import pytest
import torch

from oracle import pet_oracle as po
from pet_kokkos_b200 import checkpoint as ck, structures as st

pytestmark = pytest.mark.gpu


def cluster(n, seed):
    rng = np.random.default_rng(seed)
    pos = rng.normal(size=(4 * n + 8, 3))
    pos *= (rng.uniform(0, 1, len(pos)) ** (1 / 3) / np.linalg.norm(pos, axis=1))[:, None] * 2.2
    return st.make_system(rng.choice([1, 6, 7, 8], size=n), pos[:n], np.zeros((3, 3)), (False, False, False))


@pytest.mark.parametrize("heads", [1, 2, 4])  # head sizes 64, 32, 16
@pytest.mark.parametrize("gemm", ["native", "3xtf32", "tf32"])
def test_block_edges(lib_path, tmp_path, heads, gemm):
    from pet_kokkos_b200 import Calculator
    shape = dict(d_pet=64, num_heads=heads, d_feedforward=64, cutoff=4.5)
    jp, sp = ck.write_random_checkpoint(tmp_path / "m", shape, seed=5, init="scaled")
    meta, tens = ck.load_checkpoint(jp, sp)
    c = Calculator(jp, sp, gemm=gemm)
    sizes = [1, 2, 15, 16, 17, 31, 32, 33, 48, 49, 79, 80, 81, 128, 129, 160, 161, 177]
    for n in sizes:
        system = cluster(n, n)
        r = c.compute([system])
        ref = po.evaluate(meta, tens, [system], dtype=torch.float64)
        force = max(1.0, np.abs(ref["forces"]).max())
        energy = max(1.0, np.abs(ref["per_atom_energy"]).sum())
        f_band, e_band = {"native": (1e-5, 1e-6), "3xtf32": (3e-4, 3e-5), "tf32": (3e-2, 3e-2)}[gemm]
        assert np.abs(r.forces - ref["forces"]).max() <= f_band * force, (n, np.abs(r.forces - ref["forces"]).max() / force)
        assert np.abs(r.energy - ref["energy"]).max() <= e_band * energy, (n, np.abs(r.energy - ref["energy"]).max() / energy)
    if gemm == "native":  # together: the CTAs are cut for the longest atom, the results stay each structure's own, to the bit
        systems = [cluster(n, n) for n in (5, 40, 90)]
        r = c.compute(systems)
        assert (r.energy == np.concatenate([c.compute([s]).energy for s in systems])).all()
    c.close()
