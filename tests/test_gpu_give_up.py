"""What an evaluation does when a tensor-core kernel has given up on a bounded wait: nothing here makes one wait. The word that
such a kernel raises is raised by the test hook instead."""
import numpy as np
import pytest
import torch

from pet_kokkos_b200 import structures as st

pytestmark = pytest.mark.gpu


@pytest.fixture()
def calc(lib_path, models):
    from pet_kokkos_b200 import Calculator
    c = Calculator(*models("tiny"))
    yield c
    c.close()


def test_the_calculator_it_happened_to_reports_it(lib_path, models, calc):
    """The word belongs to a calculator: another one on the same device neither reports it nor clears it."""
    from pet_kokkos_b200 import Calculator
    other = Calculator(*models("tiny"))
    system = st.diamond(2, jitter=0.05, seed=0)
    good = calc.compute(system)
    calc.debug_give_up()
    assert np.array_equal(other.compute(system).forces, good.forces)
    with pytest.raises(RuntimeError, match="gave up"):
        calc.compute(system)
    assert np.array_equal(calc.compute(system).forces, good.forces)  # reported once
    other.close()


def on_the_device(calc):
    """The results where they lie, read once the calculator's stream has got there."""
    r, stream = calc.device_results()
    torch.cuda.ExternalStream(stream).synchronize()
    n = r.n_atoms
    out = {}
    for name, shape in (("energy", (1,)), ("per_atom_energy", (n,)), ("forces", (n, 3)), ("virial", (6,))):
        p = getattr(r, name)
        if p:
            class Lies:
                __cuda_array_interface__ = {"shape": shape, "typestr": "<f8", "data": (p, False), "version": 3}
            out[name] = torch.as_tensor(Lies(), device="cuda").cpu().numpy()
    return out


@pytest.mark.parametrize("forces", [True, False])
@pytest.mark.parametrize("how", ["staged", "step"])
def test_results_left_on_the_device(calc, how, forces):
    """They are read there without a host that asks: an evaluation that gave up leaves NaN in all of them, the next one fails, the
    one after it is good again."""
    from pet_kokkos_b200 import EdgeListView
    system = st.diamond(2, jitter=0.05, seed=0)
    raw = calc.neighbor_list(system)
    offsets = np.concatenate([[0], np.cumsum(np.bincount(raw["i"], minlength=system["n_atoms"]))]).astype(np.int32)
    calc.set_neighbors(EdgeListView(positions=system["positions"], atomic_numbers=system["atomic_numbers"], offsets=offsets,
                                    neighbors=raw["j"], shifts=raw["shift"], cell=system["cell"]))
    calc.stage([system])

    def evaluate():
        if how == "step":
            calc.compute_step_on_device(system["positions"], cell=system["cell"], compute_forces=forces)
        else:
            calc.compute_staged(forces)

    evaluate()
    good = on_the_device(calc)
    assert len(good) == (4 if forces else 2) and all(np.isfinite(v).all() for v in good.values())
    evaluate()
    calc.debug_give_up()
    assert all(np.isnan(v).all() for v in on_the_device(calc).values())
    with pytest.raises(RuntimeError, match="gave up"):
        evaluate()
    evaluate()
    again = on_the_device(calc)
    assert all(np.array_equal(again[k], good[k]) for k in good)
    evaluate()
    calc.debug_give_up()
    calc.device_results()
    if how == "staged":  # ... or the host asks for the same evaluation's results
        with pytest.raises(RuntimeError, match="gave up"):
            calc.fetch()
        evaluate()
        assert np.array_equal(on_the_device(calc)["energy"], good["energy"])
