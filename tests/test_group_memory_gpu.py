"""A context for whose jump groups there is no device memory left is created all
the same, on the row tiles' tables, and computes what it computes with them.

Tolerance: FP64 1e-12 of the largest output (some hundred terms in another
order)."""
import numpy as np
import pytest

from bigstickpublick_b200 import model

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


def test_context_without_room_for_its_groups():
    import torch
    from bigstickpublick_b200.engine import Hamiltonian
    t = model.build_tables(model.pf_model(6, 2, seed=5))
    a = t.a
    jumps = sum(int(a["pxend"][b] - a["pxstart"][b] + 1) for b in range(len(a["optype"])) if a["optype"][b] == 4)
    groups = 16 * jumps   # the jumps alone: the least that the groups take
    assert groups > 32 << 20
    x = torch.from_numpy(np.random.default_rng(7).standard_normal(t.dim)).cuda()
    y = torch.zeros_like(x)
    h = Hamiltonian(t)
    full = h.stats()["derived_bytes"]
    h.applyh(x, y)
    with_groups = y.cpu().numpy()
    before = _free()
    h.close()
    used = _free() - before
    assert used > groups
    hog = torch.empty(_free() - used + groups // 2, dtype=torch.uint8, device="cuda")
    try:
        h = Hamiltonian(t)
        assert h.stats()["derived_bytes"] <= full - groups
        y.fill_(float("nan"))
        h.applyh(x, y)
        torch.cuda.synchronize()
        got = y.cpu().numpy()
        h.close()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert np.abs(got - with_groups).max() < 1e-12 * np.abs(with_groups).max()
    assert not np.array_equal(got, with_groups)   # another kernel's order: the groups were not there
