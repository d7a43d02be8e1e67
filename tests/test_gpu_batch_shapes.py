"""Batches of every size give the same results, whichever kernel shape they take.

Small and medium batches are evaluated in tiles of 1 to 32 states, a block per
tile; batches of about a wave and more by a thread per state.  Every sum over
reactions and species has one fixed order in all of them, so the species rates
are equal bit for bit, and the Jacobian but for the contraction of a few
products (one rounding of a term: 1e-14 of the row's largest entry).  Sizes at
the edges: one state, a partly filled tile, one state past a tile, past a round
of tiles, past a wave.
"""
import numpy as np
import pytest

from conftest import load_mech, oracle_mod, pkg, row_rel_err

pytestmark = pytest.mark.gpu

# tiles of 1, 2, 4, 8, 16, 32 states on 152 SMs, and a thread per state
SIZES = [1, 2, 303, 305, 609, 1217, 2433, 4863, 4865, 9729, 20001]
_ev = {}


def evaluator(name):
    if name not in _ev:
        _ev[name] = pkg("api").Evaluator(load_mech(name))
    return _ev[name]


@pytest.mark.parametrize("name,n", [("h2o2", 70001), ("gri30", 61003), ("testmech", 65537), ("synthetic_small", 60001)])
@pytest.mark.parametrize("conp", [True, False])
@pytest.mark.parametrize("order,fmt", [("C", "sparse"), ("F", "full")])
def test_batch_sizes_agree(cuda_device, name, n, conp, order, fmt):
    import torch
    mech, ev = load_mech(name), evaluator(name)
    if name == "gri30":
        fmt = "sparse"
    P, phi = pkg("states").draw_states(mech.n_species, n, seed=61, x_floor=1e-12, conp=conp)
    tP = torch.from_numpy(P).to(cuda_device)
    tx = torch.from_numpy(phi).to(cuda_device)

    def run(k):
        x = tx[:k].contiguous() if order == "C" else tx[:k].t().contiguous()
        r = ev.species_rates(tP[:k].contiguous(), x, order=order, conp=conp)
        J = ev.jacobian(tP[:k].contiguous(), x, order=order, conp=conp, jac_format=fmt)
        g = ev.vjp(tP[:k].contiguous(), x, x, order=order, conp=conp)
        return [a if order == "C" else a.movedim(-1, 0) for a in (r, J, g)]

    r0, J0, g0 = run(n)
    ptr, ind = ev.jacobian_indices(order)
    line = np.repeat(np.arange(mech.nn), np.diff(ptr))
    row = torch.from_numpy(line if order == "C" else ind.astype(np.int64)).to(cuda_device)
    big = torch.zeros(J0.shape[0], mech.nn, dtype=torch.float64, device=cuda_device)
    if fmt == "sparse":
        big.scatter_reduce_(1, row.expand(J0.shape[0], -1), J0.abs(), "amax")
        scale = big[:, row]
    else:  # [state, col, row] for order F
        scale = J0.abs().amax(1, keepdim=True).expand_as(J0)
    for k in SIZES:
        r, J, g = run(k)
        assert torch.equal(r, r0[:k]), k
        ok = (J - J0[:k]).abs() <= 1e-14 * scale[:k]
        assert bool(ok.all()), (k, int((~ok).sum()))
        assert float((g - g0[:k]).abs().max() / g0.abs().max()) <= 1e-13, k


@pytest.mark.parametrize("name", ["gri30", "synthetic_small"])
@pytest.mark.parametrize("n", [1, 33, 700])
def test_small_batches_match_oracle(cuda_device, name, n):
    import torch
    mech, ev = load_mech(name), evaluator(name)
    P, phi = pkg("states").draw_states(mech.n_species, n, seed=62, x_floor=1e-12)
    J = ev.jacobian(torch.from_numpy(P).to(cuda_device), torch.from_numpy(phi).to(cuda_device)).cpu().numpy()
    assert row_rel_err(J, oracle_mod().Oracle(mech).jacobian(P, phi)) < 1e-8
