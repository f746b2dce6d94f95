"""The batch autotuner chooses for the persistent launch only: a batch whose members
all have jump groups keeps its setting (there is nothing to time), a batch with a
member that has none (pf 2p4n) gets one of the candidates, and its results keep
their bits."""
import pytest

from bigstickpublick_b200 import model

pytestmark = pytest.mark.gpu


def _apply(b):
    import torch
    g = torch.Generator(device="cuda").manual_seed(2)
    vin = [torch.randn(d, dtype=torch.float32, device="cuda", generator=g) for d in b.dims]
    vout = [torch.empty_like(v) for v in vin]
    b.applyh(vin, vout)
    torch.cuda.synchronize()
    return vout


def test_members_with_groups_keep_their_setting():
    from bigstickpublick_b200.engine import Batch
    b = Batch([model.build_tables(model.sd_model(p, 3, seed=p, jz2=(p + 3) % 2)) for p in (2, 3, 4)])
    for items, ctas in ((1, 3), (8, 5), (2, 16)):
        assert b.lib.bsg_batch_set_tuning(b.h, items, ctas) == 0
        got = b.autotune()
        assert (got["items"], got["ctas_per_sm"]) == (items, ctas) and 0 < got["ms"] < 1e3
    b.close()


def test_mixed_members():
    import torch
    from bigstickpublick_b200.engine import Batch
    b = Batch([model.build_tables(model.sd_model(3, 3, seed=1)), model.build_tables(model.pf_model(2, 4, seed=2))])
    before = _apply(b)
    got = b.autotune()
    assert got["items"] in (1, 2, 4, 8) and got["ctas_per_sm"] in (4, 8) and 0 < got["ms"] < 1e3
    assert all(torch.equal(x, y) for x, y in zip(before, _apply(b)))
    b.close()
