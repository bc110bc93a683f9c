"""A coarsest matrix with a column of NaN is a breakdown in every factorisation kernel: no row
is chosen as its pivot.  Needs a GB300."""
import numpy as np
import pytest

import femgpu
from test_gpu_coarsest import dense_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,column", [(1, 0), (40, 0), (40, 39), (392, 100), (393, 0), (400, 170), (700, 699)])
def test_nan_column_is_a_breakdown(n, column, precision):
    M = 2.0 * np.eye(n) + np.diag(np.full(n - 1, 0.25), 1)
    M[:, column] = np.nan
    with femgpu.Solver(solverType=0, maxLevels=1, topSize=1, precision=precision) as s:
        s.set_matrix_csr(*dense_csr(M))
        with pytest.raises(femgpu.FemgpuError) as e:
            s.setup()
        assert e.value.status == 4  # FEMGPU_ERR_BREAKDOWN
        s.set_matrix_csr(*dense_csr(np.eye(n) * 2.0))
        s.setup()
        assert np.array_equal(s.vcycle(np.ones(n)), np.full(n, 0.5))
