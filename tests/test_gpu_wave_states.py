"""The numerically hard states through the thread-per-state kernel (GPU).

Batches of a few hundred states are evaluated in tiles, so the states of the
edge tests (temperatures at and beyond the clamps, equilibrium constants on both
sides of the split, zero moles, bath-rich mixtures) are repeated here to a whole
wave of the Jacobian kernel and compared with the oracle: species rates,
Jacobian and J^T v.  Also, with both kernels: the 'approximate' Jacobian type, a
mechanism that does not conserve mass (row E's weights are not sums of
coefficients) and a Jacobian pattern that leaves out terms (rows T and E are then
sums over the stored entries).  Tolerances are the small batches'.
"""
import copy
import os

import numpy as np
import pytest

from conftest import DATA, bath_rich_states, load_mech, oracle_mod, pkg, row_rel_err
from test_gpu_edges import _gibbs_b, _rates_err

pytestmark = pytest.mark.gpu

RU = 8314.4621


def wave(device):
    import torch
    return 4 * 128 * torch.cuda.get_device_properties(device).multi_processor_count


def put(a, order, n, device):
    """The states of a (m, NN) or (m,) repeated to n, in the data order."""
    import torch
    a = torch.from_numpy(np.ascontiguousarray(a)).to(device)
    a = a.repeat((-(-n // a.shape[0]),) + (1,) * (a.dim() - 1))[:n]
    return a.contiguous() if order == "C" or a.dim() == 1 else a.t().contiguous()


def run(ev, P, phi, v, order, conp, fmt, n, device):
    """Rates, dense Jacobian [row, col] and J^T v of the m states at the start of n."""
    m, nn = phi.shape
    tP, tx, tv = put(P, order, n, device), put(phi, order, n, device), put(v, order, n, device)

    def host(a):
        a = a if order == "C" else a.movedim(-1, 0)
        return a[:m].cpu().numpy().reshape(m, -1)

    r = host(ev.species_rates(tP, tx, order=order, conp=conp))
    J = host(ev.jacobian(tP, tx, order=order, conp=conp, jac_format=fmt))
    g = host(ev.vjp(tP, tx, tv, order=order, conp=conp))
    if fmt == "sparse":
        ptr, ind = ev.jacobian_indices(order)
        line = np.repeat(np.arange(nn), np.diff(ptr))
        full = np.zeros((m, nn, nn))
        full[:, line if order == "C" else ind, ind if order == "C" else line] = J
        J = full
    else:
        J = J.reshape(m, nn, nn)
        J = J if order == "C" else J.transpose(0, 2, 1)
    return r, J, g


def check(mech, P, phi, order, conp, fmt, device, n, vjp=True):
    v = np.random.default_rng(97).standard_normal(phi.shape)
    r, J, g = run(pkg("api").Evaluator(mech), P, phi, v, order, conp, fmt, n, device)
    o = oracle_mod().Oracle(mech)
    ref, Jref = o.species_rates(P, phi, conp=conp), o.jacobian(P, phi, conp=conp)
    assert np.isfinite(r).all() and np.isfinite(J).all() and np.isfinite(g).all()
    assert _rates_err(r, ref, o.rates_scale(P, phi, conp=conp)) < 1e-10
    assert row_rel_err(J, Jref) < 1e-8
    if vjp:
        scale = np.einsum("nrc,nr->nc", np.abs(Jref), np.abs(v))
        err = np.abs(g - np.einsum("nrc,nr->nc", Jref, v)) / np.where(scale > 0, scale, 1.0)
        assert err.max() < 1e-9


def hard_states(mech, kind):
    draw = pkg("states").draw_states
    if kind == "bath_rich":
        return bath_rich_states(mech, 150, 21, True)
    if kind == "zero_moles":
        P, phi = draw(mech.n_species, 257, seed=8, x_floor=1e-12)
        phi = phi.copy()
        phi[:, 2:][np.random.default_rng(8).random(phi[:, 2:].shape) < 0.5] = 0.0
        phi[0, 2:] = 0.0
        return P, phi
    if kind == "limits":
        T = np.array([80.0, 100.0, 100.5, 300.0, 999.999999, 1000.0, 1000.000001, 2500.0, 3500.0, 6000.0,
                      9999.0, 10000.0, 12000.0])
    else:  # "split"
        n, rng = 256, np.random.default_rng(41)
        T = np.where(np.arange(n) % 3 == 0, rng.uniform(250.0, 700.0, n), rng.uniform(700.0, 3000.0, n))
        assert 0.1 < (np.abs(_gibbs_b(mech, T)).max(axis=1) > 138.0).mean() < 0.5
    P, phi = draw(mech.n_species, T.size, seed=21, x_floor=1e-12)
    phi = phi.copy()
    phi[:, 2:] *= (phi[:, 0] / T)[:, None]
    phi[:, 0] = T
    return P, phi


@pytest.mark.parametrize("name,kind", [("h2o2", "limits"), ("gri30", "limits"), ("gri30", "split"),
                                       ("gri30", "zero_moles"), ("gri30", "bath_rich"), ("testmech", "bath_rich"),
                                       ("synthetic_small", "bath_rich")])
@pytest.mark.parametrize("order", ["C", "F"])
def test_hard_states(cuda_device, name, kind, order):
    mech = load_mech(name)
    P, phi = hard_states(mech, kind)
    # the edge tests compare J^T v where the Jacobian's own tolerance carries over
    check(mech, P, phi, order, True, "full", cuda_device, wave(cuda_device), vjp=kind in ("split", "bath_rich"))


@pytest.mark.parametrize("name", ["h2o2", "gri30", "testmech", "synthetic_small"])
@pytest.mark.parametrize("conp", [True, False])
def test_vjp_on_its_own_scale(cuda_device, name, conp):
    mech = load_mech(name)
    P, phi = bath_rich_states(mech, 150, 21, conp)
    check(mech, P, phi, "C", conp, "sparse", cuda_device, wave(cuda_device))


@pytest.mark.parametrize("name", ["h2o2", "gri30", "testmech", "synthetic_small"])
@pytest.mark.parametrize("order,fmt", [("C", "sparse"), ("F", "full")])
def test_approximate_jacobian(cuda_device, name, order, fmt):
    mech = load_mech(name, jac_type="approximate")
    P, phi = pkg("states").draw_states(mech.n_species, 200, seed=21, x_floor=1e-12)
    if name in ("testmech", "synthetic_small"):
        P, phi = bath_rich_states(mech, 200, 21, True)
    check(mech, P, phi, order, True, fmt, cuda_device, wave(cuda_device), vjp=False)


@pytest.mark.parametrize("blocks", [2, 3, 4])
def test_large_mechanism(cuda_device, blocks):
    """The 500-species mechanism, whose Jacobian kernel holds three blocks per SM
    (two in the form for fewer blocks, four where a rest of one joins the last wave)."""
    import torch
    torch.cuda.empty_cache()
    mech = load_mech("synthetic500")
    P, phi = pkg("states").draw_states(mech.n_species, 6, seed=18)
    check(mech, P, phi, "F", True, "sparse", cuda_device, blocks * wave(cuda_device) // 4, vjp=False)
    torch.cuda.empty_cache()


@pytest.mark.parametrize("waves", [0, 1])
@pytest.mark.parametrize("conp", [True, False])
def test_mechanism_that_does_not_conserve_mass(cuda_device, tmp_path, waves, conp):
    with open(os.path.join(DATA, "h2o2.inp")) as f:
        text = f.read()
    for a, b in (("O+H2<=>H+OH   ", "O+H2<=>H+HO2  "), ("2H+M<=>H2+M  ", "2H+M<=>H2O+M ")):
        assert text.count(a) == 1
        text = text.replace(a, b)
    path = tmp_path / "unbalanced.inp"
    path.write_text(text)
    mech = pkg().load_mechanism(str(path))
    P, phi = bath_rich_states(mech, 200, 23, conp)
    check(mech, P, phi, "C", conp, "full", cuda_device, waves * wave(cuda_device) or 200)


@pytest.mark.parametrize("waves", [0, 1])
@pytest.mark.parametrize("name", ["h2o2", "testmech"])
@pytest.mark.parametrize("order", ["C", "F"])
def test_pattern_that_leaves_out_terms(cuda_device, waves, name, order):
    base = load_mech(name)
    nn, last = base.nn, base.n_species - 1
    rng = np.random.default_rng(7)
    ptr, ind = base.pattern("C")
    rows = np.repeat(np.arange(nn), np.diff(ptr))
    keep = (rows < 2) | (ind < 2) | (rng.random(ind.size) > 0.3)
    mask = np.zeros((nn, nn), dtype=bool)
    mask[rows[keep], ind[keep]] = True
    mech = copy.copy(base)
    off = lambda a: np.concatenate([[0], np.cumsum(a)])
    mech.val = dict(base.val, jac_inds=dict(
        base.val["jac_inds"],
        crs={"row_ptr": off(mask.sum(1)), "col_ind": np.nonzero(mask)[1]},
        ccs={"col_ptr": off(mask.sum(0)), "row_ind": np.nonzero(mask.T)[1]}))
    P, phi = bath_rich_states(base, 120, 25, True)
    n = waves * wave(cuda_device) or 120
    _, J, _ = run(pkg("api").Evaluator(mech), P, phi, phi, order, True, "sparse", n, cuda_device)
    # the whole Jacobian's rows T and E less the entries left out
    o = oracle_mod().Oracle(base)
    ref = o.jacobian(P, phi)
    cp, h, _ = o.chem_utils(phi)
    T, V = phi[:, 0], phi[:, 1]
    c = phi[:, 2:] / V[:, None]
    cp_tot = (cp[:, :last] * c).sum(1) + cp[:, last] * (P / (RU * T) - c.sum(1))
    sp = pkg("pack").PackedTables(base).species
    hw = h[:, :last] - h[:, last:] * sp[:last, 1]
    out = np.where(mask, 0.0, 1.0)[2:, 2:] * ref[:, 2:, 2:]
    dT = np.einsum("nk,nkj->nj", hw, out) / (V * cp_tot)[:, None]
    dE = -(T * RU / P)[:, None] * np.einsum("k,nkj->nj", sp[:last, 2], out) + (V / T)[:, None] * dT
    scale = np.abs(ref).max(axis=-1, keepdims=True)
    scale[scale == 0] = 1.0  # a species that no reaction changes
    ref[:, 0, 2:] += dT
    ref[:, 1, 2:] += dE
    assert np.abs(dT).max() > 0 and np.abs(dE).max() > 0
    assert float((np.abs(J - ref * mask) / scale).max()) < 1e-8
