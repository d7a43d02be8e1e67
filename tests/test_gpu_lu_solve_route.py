"""The dense solve on both sides of the sizes at which it goes from 32 states per
block to a thread per state: both substitute in the oracle's order, so both are
its results bit for bit (GPU)."""
import numpy as np
import pytest

from conftest import oracle_mod, pkg
from test_gpu_integrate import _from_dev_vec, _to_dev_mat, _to_dev_vec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,nn,per_sm", [("C", 40, 128), ("C", 44, 56), ("C", 54, 128), ("C", 72, 80), ("C", 100, 56),
                                             ("F", 33, 576)])
@pytest.mark.parametrize("more", [-1, 0])
def test_solve_across_the_route(cuda_device, order, nn, per_sm, more):
    import torch
    orc, integ = oracle_mod(), pkg("integrate")
    n = per_sm * torch.cuda.get_device_properties(cuda_device).multi_processor_count + more
    rng = np.random.default_rng(nn)
    m = 96  # matrices, repeated
    lu, piv, _ = orc.lu_factor(rng.standard_normal((m, nn, nn)), 1.0, 1.0)
    b = rng.standard_normal((m, nn))
    want = orc.lu_solve(lu, piv, b)
    idx = np.arange(n) % m
    x = integ.lu_solve(_to_dev_mat(lu[idx], order, cuda_device), _to_dev_vec(piv[idx], order, cuda_device),
                       _to_dev_vec(b[idx], order, cuda_device), order=order)
    assert np.array_equal(_from_dev_vec(x, order), want[idx])
