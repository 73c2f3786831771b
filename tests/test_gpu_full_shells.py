"""Molecules whose basis is fully occupied, down to one function, against the CPU oracle."""

import numpy as np
import pytest

from oracle import oracle
from vibeqc_b200 import Calculator

pytestmark = pytest.mark.gpu

AUX = "def2-tzvp"
# charge, multiplicity; N functions and electrons of each spin in STO-3G
CASES = {
    "He": ([("He", (0.1, 0.2, 0.3))], 0, 1),  # 1, 1 + 1
    "H-": ([("H", (0.0, 0.0, 0.0))], -1, 1),  # 1, 1 + 1
    "Ne": ([("Ne", (0.0, 0.1, 0.0))], 0, 1),  # 5, 5 + 5
    "He2": ([("He", (0.0, 0.0, 0.0)), ("He", (0.0, 0.3, 4.0))], 0, 1),  # 2, 2 + 2
    "H": ([("H", (0.1, -0.2, 0.3))], 0, 2),  # 1, 1 + 0
}


@pytest.mark.parametrize("precision", ["fp64", "mixed", "auto"])
@pytest.mark.parametrize("name", list(CASES))
def test_full_shells_match_oracle(name, precision):
    atoms, charge, mult = CASES[name]
    unrestricted = mult != 1
    calc = Calculator(method="uhf" if unrestricted else "rhf", basis="sto-3g", auxiliary_basis=AUX,
                      device="cuda", density_fitting="cuda", precision=precision)
    got = calc.singlepoint(atoms, charge=charge, multiplicity=mult)
    run = oracle.df_uhf if unrestricted else oracle.df_rhf
    want = run(atoms, "sto-3g", AUX, charge=charge, **({"multiplicity": mult} if unrestricted else {}))
    de, df = (1e-8, 1e-7) if precision == "fp64" else (1e-6, 1e-5)
    assert got.converged
    assert abs(got.energy - want.energy) < de
    assert np.abs(got.forces - want.forces).max() < df
