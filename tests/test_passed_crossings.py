"""The step's system where two crossings have passed each other along a yarn
(du < 0 on an edge): the product's element code on the host against the CPU
oracle, every row of A and b. Both evaluate the same formulas in FP64 in
different orders; 1e-12 of a row's largest entry is what the other comparisons
of the two allow."""
import numpy as np
import pytest

import passed_cases
from emu_py import EmuCloth


@pytest.mark.parametrize("weave,k,kf", passed_cases.CASES)
def test_system_matches_oracle(weave, k, kf):
    from oracle.oracle import ClothSpec, OracleCloth
    kw = passed_cases.kwargs(weave, kf)
    oc, em = OracleCloth(ClothSpec(**kw)), EmuCloth(**kw)
    st = passed_cases.state(oc.get_state(), kw, k)
    oc.set_state(st)
    em.set_state(st)
    oc.fill()
    A_ref, b_ref = oc.system(1e-3)
    em.assemble(1e-3)
    A, b = em.system()
    err = np.abs(A - A_ref).max(1) / np.abs(A_ref).max(1)
    assert err.max() <= 1e-12, (int(err.argmax()), err.max())
    assert np.abs(b - b_ref).max() <= 1e-12 * np.abs(b_ref).max()
