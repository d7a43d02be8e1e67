"""The dense solve at the edges of its blocks (32 states, 8 warps of rows) and
at its largest size, bit for bit against the oracle's substitution (GPU)."""
import numpy as np
import pytest

from conftest import oracle_mod, pkg
from test_gpu_integrate import _from_dev_vec, _to_dev_mat, _to_dev_vec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["C", "F"])
@pytest.mark.parametrize("nn,n", [(1, 1), (2, 33), (7, 31), (8, 32), (9, 65), (16, 200), (54, 97), (55, 1000),
                                  (169, 40), (176, 33), (177, 3), (5, 128 * 152 - 1),
                                  (5, 128 * 152 + 3), (32, 256 * 152 + 1)])
def test_lu_solve_edges_bitwise(cuda_device, order, nn, n):
    orc = oracle_mod()
    integ = pkg("integrate")
    rng = np.random.default_rng(nn)
    lu, piv, _ = orc.lu_factor(rng.standard_normal((n, nn, nn)), 1.0, 1.0)
    b = rng.standard_normal((n, nn))
    x = integ.lu_solve(_to_dev_mat(lu, order, cuda_device), _to_dev_vec(piv, order, cuda_device),
                       _to_dev_vec(b, order, cuda_device), order=order)
    assert np.array_equal(_from_dev_vec(x, order), orc.lu_solve(lu, piv, b))
