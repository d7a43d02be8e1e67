"""Dense solves of different sizes from several threads at once (GPU): each
launch finds the shared memory it needs, whatever the others ask for."""
import threading

import numpy as np
import pytest

from conftest import oracle_mod, pkg
from test_gpu_integrate import _from_dev_vec, _to_dev_mat, _to_dev_vec

pytestmark = pytest.mark.gpu


def test_concurrent_solves_of_different_sizes(cuda_device):
    import torch
    orc, integ = oracle_mod(), pkg("integrate")
    rng = np.random.default_rng(4)
    jobs = []
    for nn in (169, 33, 120, 64):
        lu, piv, _ = orc.lu_factor(rng.standard_normal((8, nn, nn)), 1.0, 1.0)
        b = rng.standard_normal((8, nn))
        jobs.append((_to_dev_mat(lu, "F", cuda_device), _to_dev_vec(piv, "F", cuda_device),
                     _to_dev_vec(b, "F", cuda_device), orc.lu_solve(lu, piv, b)))
    torch.cuda.synchronize()
    errors = []

    def work(lu, piv, b, want):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(2000):
                    x = integ.lu_solve(lu, piv, b.clone(), order="F")
                torch.cuda.current_stream().synchronize()
            if not np.array_equal(_from_dev_vec(x, "F"), want):
                errors.append("wrong result")
        except Exception as e:  # the thread's, shown by the assertion below
            errors.append(str(e))

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
