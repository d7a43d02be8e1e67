"""pjg_vjp_noalloc with a small mechanism, whose larger batches take larger tiles
(GPU): the same products as pjg_vjp on both sides of the change, and no device
memory taken by either size's first call."""
import pytest

from conftest import load_mech, pkg
from test_zz_no_alloc import _call, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["C", "F"])
@pytest.mark.parametrize("n", [1, 2432, 2433, 30001])
def test_noalloc_small_mechanism(cuda_device, order, n):
    import torch
    L = pkg("_lib")
    lib = L.load()
    mech = load_mech("h2o2")
    tP, tphi = _inputs(mech, n, order, cuda_device, 7)
    v = torch.randn(tphi.shape, dtype=torch.float64, device=cuda_device)
    got, ref = torch.full_like(tphi, float("nan")), torch.empty_like(tphi)
    warm, fresh = pkg("api").DeviceMechanism(mech), pkg("api").DeviceMechanism(mech)
    assert _call(lib, "pjg_vjp_noalloc", warm, n, order, tP, tphi, v, ref) == 0, L.last_error()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert _call(lib, "pjg_vjp_noalloc", fresh, n, order, tP, tphi, v, got) == 0, L.last_error()
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    assert _call(lib, "pjg_vjp", fresh, n, order, tP, tphi, v, ref) == 0, L.last_error()
    torch.cuda.synchronize()
    assert bool(torch.isfinite(got).all())
    assert float((got - ref).abs().max() / ref.abs().max()) <= 1e-12
