"""CSR arguments of the stand-alone solves that are refused before any device call."""
import numpy as np
import pytest

from mixsolver_b200 import solver as S


@pytest.mark.parametrize("ptr", [[0, 1, 2], [1, 2, 0], [1, 9, 3], [1, -5, 3]],
                         ids=["0-based", "negative length", "row beyond the last entry", "negative row"])
@pytest.mark.parametrize("solve", [S.cg_jacobi, S.cg_ic0, S.bicgstab_ilu0, S.pcg_poly])
def test_row_pointers_out_of_range_are_refused(ptr, solve):
    with pytest.raises(RuntimeError, match=r"status -1\b.*row pointer"):
        solve(np.array(ptr), np.array([1, 2], np.int32), np.ones(2), np.ones(2), np.zeros(2), 1e-8, 5)
