"""Observables with entries that are not finite are not Hermitian (CPU)."""
import numpy as np
import pytest

import mossquantum_b200 as mq


@pytest.mark.parametrize("matrix,coeff", [([[np.inf, 0], [0, 1]], 1.0), ([[0, np.inf], [np.inf, 0]], 1.0), ([[1, 0], [0, 1]], np.inf),
                                          ([[1, 0], [0, -1]], np.nan), ([[np.nan, 0], [0, 1]], 1.0)])
def test_not_finite(matrix, coeff):
    with np.errstate(invalid="ignore"):
        assert not mq.QubitsOperator([mq.QubitsTerm([1], [np.array(matrix)], coeff)]).is_hermitian()
