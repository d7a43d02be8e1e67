"""Reactions whose pre-exponential factor is zero (GPU): ln A is -inf, and the
reaction adds nothing.  One of each kind of record: an elementary reaction, a
mass-action pattern, a third-body pattern and a fall-off's low-pressure limit,
on both evaluation kernels."""
import os

import numpy as np
import pytest

from conftest import DATA, oracle_mod, pkg, row_rel_err

pytestmark = pytest.mark.gpu

ZEROED = ["H+O2<=>O+OH                              2.650E+16",
          "2OH<=>O+H2O                              3.570E+04",
          "H+O2+M<=>HO2+M                           2.800E+18",
          "     LOW  /  2.300E+18"]
N_CHECKED = 300


@pytest.fixture(scope="module")
def mechanism(tmp_path_factory):
    with open(os.path.join(DATA, "h2o2.inp")) as f:
        text = f.read()
    for line in ZEROED:
        assert text.count(line) == 1
        head = line[:-9]
        text = text.replace(line, head + "0.000E+00")
    path = tmp_path_factory.mktemp("mech") / "zero_rates.inp"
    path.write_text(text)
    with np.errstate(divide="ignore"):
        return pkg().load_mechanism(str(path))


# 300 states are evaluated in tiles, 40,000 by a thread per state
@pytest.mark.parametrize("n", [N_CHECKED, 40000])
@pytest.mark.parametrize("conp", [True, False])
def test_zero_rates_add_nothing(cuda_device, mechanism, n, conp):
    import torch
    ev = pkg("api").Evaluator(mechanism)
    P, phi = pkg("states").draw_states(mechanism.n_species, n, seed=81, x_floor=1e-12, conp=conp)
    tP, tx = torch.from_numpy(P).to(cuda_device), torch.from_numpy(phi).to(cuda_device)
    m = N_CHECKED
    orc = oracle_mod().Oracle(mechanism)
    ref, scale = (f(P[:m], phi[:m], conp=conp) for f in (orc.species_rates, orc.rates_scale))
    J = orc.jacobian(P[:m], phi[:m], conp=conp)
    assert np.isfinite(ref).all() and np.isfinite(J).all()
    r = ev.species_rates(tP, tx, conp=conp)[:m].cpu().numpy()
    assert float((np.abs(r - ref) / (np.abs(ref) + scale)).max()) < 1e-10
    assert row_rel_err(ev.jacobian(tP, tx, conp=conp)[:m].cpu().numpy(), J) < 1e-8
    v = np.random.default_rng(82).standard_normal(phi.shape)
    g = ev.vjp(tP, tx, torch.from_numpy(v).to(cuda_device), conp=conp)[:m].cpu().numpy()
    d = np.abs(g - np.einsum("nrc,nr->nc", J, v[:m]))
    assert float((d / np.einsum("nrc,nr->nc", np.abs(J), np.abs(v[:m]))).max()) < 1e-9
