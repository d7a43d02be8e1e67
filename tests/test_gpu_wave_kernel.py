"""The thread-per-state kernels (GPU).  The Jacobian in both register forms: a
launch of at most two blocks of 128 states per SM, and a larger one.  They are
the same code, so they may differ by the contraction of a few products: 1e-14 of
a row's largest entry."""
import pytest

from conftest import load_mech, pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conp", [True, False])
@pytest.mark.parametrize("order,fmt", [("C", "sparse"), ("F", "full")])
def test_register_forms_agree(cuda_device, conp, order, fmt):
    import torch
    mech = load_mech("h2o2")
    ev = pkg("api").Evaluator(mech)
    few = 2 * 128 * torch.cuda.get_device_properties(cuda_device).multi_processor_count
    n = few + 1
    P, phi = pkg("states").draw_states(mech.n_species, n, seed=95, x_floor=1e-12, conp=conp)
    tP, tx = torch.from_numpy(P).to(cuda_device), torch.from_numpy(phi).to(cuda_device)

    def run(k):
        x = tx[:k].contiguous() if order == "C" else tx[:k].t().contiguous()
        J = ev.jacobian(tP[:k].contiguous(), x, order=order, conp=conp, jac_format=fmt)
        return J if order == "C" else J.movedim(-1, 0).contiguous()

    a, b = run(few), run(n)[:few]
    if fmt == "full":  # [state, col, row]
        scale = b.abs().amax(1, keepdim=True)
    else:  # H2/O2's pattern is full
        assert ev.nnz == mech.nn ** 2
        a, b = a.view(few, mech.nn, mech.nn), b.view(few, mech.nn, mech.nn)
        scale = b.abs().amax(2, keepdim=True)
    assert bool(torch.isfinite(a).all())
    assert float(((a - b).abs() / scale).max()) <= 1e-14


# whole waves with a rest that a thread per state takes in a launch of its own,
# one that it takes in the same launch, and one for the tiles
@pytest.mark.parametrize("rest", [32000, 70000, 9001])
@pytest.mark.parametrize("order", ["C", "F"])
def test_rest_after_whole_waves(cuda_device, rest, order):
    import torch
    mech = load_mech("h2o2")
    ev = pkg("api").Evaluator(mech)
    n = 4 * 128 * torch.cuda.get_device_properties(cuda_device).multi_processor_count + rest
    P, phi = pkg("states").draw_states(mech.n_species, n, seed=96, x_floor=1e-12)
    tP, tx = torch.from_numpy(P).to(cuda_device), torch.from_numpy(phi).to(cuda_device)

    def run(i, j):
        x = tx[i:j].contiguous() if order == "C" else tx[i:j].t().contiguous()
        q = tP[i:j].contiguous()
        out = (ev.species_rates(q, x, order=order), ev.jacobian(q, x, order=order), ev.vjp(q, x, x, order=order))
        return [a if order == "C" else a.movedim(-1, 0) for a in out]

    r, J, g = run(0, n)
    for i, j in ((0, 40000), (n - 40000, n), (n - 200, n)):
        r1, J1, g1 = run(i, j)
        assert torch.equal(r[i:j], r1)
        scale = J1.abs().amax(2 if order == "C" else 1, keepdim=True)
        assert float(((J[i:j] - J1).abs() / scale).max()) <= 1e-14
        gs = torch.einsum("nrc,nr->nc" if order == "C" else "ncr,nr->nc", J1.abs(), tx[i:j].abs())
        assert float(((g[i:j] - g1).abs() / gs).max()) <= 1e-13
