"""CUDA graphs: once a call has been made with a number of states, calls with
any smaller number allocate nothing and can be captured (GPU)."""
import pytest

from conftest import load_mech, pkg

pytestmark = pytest.mark.gpu

# a thread per state, and tiles of 32 to 1 states
SIZES = [60000, 20000, 9000, 4000, 2000, 1000, 500, 200, 3]


@pytest.mark.parametrize("name", ["h2o2", "gri30"])
@pytest.mark.parametrize("order,fmt", [("C", "full"), ("F", "sparse")])
@pytest.mark.parametrize("warm", [100000, 20000])
def test_smaller_batches_can_be_captured(cuda_device, name, order, fmt, warm):
    import torch
    mech = load_mech(name)
    ev = pkg("api").Evaluator(mech)
    P, phi = pkg("states").draw_states(mech.n_species, warm, seed=71, x_floor=1e-12)
    tP, tx = torch.from_numpy(P).to(cuda_device), torch.from_numpy(phi).to(cuda_device)

    def inputs(n):
        return tP[:n].contiguous(), tx[:n].contiguous() if order == "C" else tx[:n].t().contiguous()

    def call(q, x):
        return (ev.species_rates(q, x, order=order), ev.jacobian(q, x, order=order, jac_format=fmt),
                ev.vjp(q, x, x, order=order))

    call(*inputs(warm))
    torch.cuda.synchronize()
    graphs = []
    for n in SIZES:
        if n > warm:
            continue
        q, x = inputs(n)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out = call(q, x)
        graphs.append((n, g, q, x, out))
    for n, g, q, x, out in graphs:
        g.replay()
        torch.cuda.synchronize()
        for a, b in zip(out, call(q, x)):
            assert torch.equal(a, b), n
