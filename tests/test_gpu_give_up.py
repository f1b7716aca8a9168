"""What an evaluation does when a tensor-core kernel has given up on a bounded wait: nothing here makes one wait. The word that
such a kernel raises is raised by the test hook instead."""
import numpy as np
import pytest

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
