"""Workers with more additions in a batch than are staged at a time (GPU).

The 500-species mechanism's sparse Jacobian gives a worker of a tile 50
additions per batch and more, against 24 to 48 staged ones, so that its lanes
refill their stage together; sizes for tiles of 1, 2, 4 and 8 states, against
the oracle at both ends of the batch.
"""
import numpy as np
import pytest

from conftest import load_mech, oracle_mod, pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 609, 1217, 2433])
def test_restaged_additions_match_oracle(cuda_device, n):
    import torch
    mech = load_mech("synthetic500")
    ev = pkg("api").Evaluator(mech)
    P, phi = pkg("states").draw_states(mech.n_species, n, seed=91, x_floor=1e-12)
    phi[:, 0] = 2000.0 + 0.3 * (phi[:, 0] - 800.0)  # entries beyond 1e150 at lower temperatures
    J = ev.jacobian(torch.from_numpy(P).to(cuda_device), torch.from_numpy(phi).to(cuda_device), jac_format="sparse")
    pick = np.unique([0, 1, 31, n // 2, n - 2, n - 1])
    pick = pick[(pick >= 0) & (pick < n)]
    got = J[torch.from_numpy(pick).to(cuda_device)].cpu().numpy()
    Jref = oracle_mod().Oracle(mech).jacobian(P[pick], phi[pick])
    ptr, ind = ev.jacobian_indices("C")
    rows = np.repeat(np.arange(mech.nn), np.diff(ptr))
    scale = np.abs(Jref).max(axis=2)[:, rows]
    scale[scale == 0] = 1.0
    assert np.isfinite(got).all()
    assert float((np.abs(got - Jref[:, rows, ind]) / scale).max()) < 1e-8
