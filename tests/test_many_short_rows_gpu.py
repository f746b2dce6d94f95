"""Single vectors on many rows of a few positions run with more CTAs to an SM: the
same bits as the batch's kernel, which does not (sd 6p2n, 862 rows; pf 4p1n, 3,681),
and the oracle's sums, stored and accumulated."""
import numpy as np
import pytest

from bigstickpublick_b200 import model
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shell,p,n", [("sd", 6, 2), ("pf", 4, 1), ("sd", 5, 1)])
@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_bits_and_sums(shell, p, n, dt):
    import torch
    from bigstickpublick_b200.engine import Batch, Hamiltonian
    mk = model.sd_model if shell == "sd" else model.pf_model
    t = model.build_tables(mk(p, n, seed=3, jz2=(p + n) % 2))
    rows = np.diff(np.append(t.a["pstart"], t.dim))
    assert len(rows) > 592 and np.median(rows) <= 16
    x = torch.from_numpy(np.random.default_rng(p).standard_normal(t.dim).astype(dt)).cuda()
    y, z = torch.full_like(x, float("nan")), torch.full_like(x, float("nan"))
    h, b = Hamiltonian(t), Batch([t])
    h.applyh(x, y)
    b.applyh([x], [z])
    torch.cuda.synchronize()
    assert torch.equal(y, z)
    ref = oracle.applyh(t, x.cpu().numpy())
    assert np.abs(y.cpu().numpy() - ref).max() < (1e-12 if dt == np.float64 else 2e-5) * np.abs(ref).max()
    base = z.clone().normal_()
    w = base.clone()
    h.applyh(x, w, accumulate=True)
    torch.cuda.synchronize()
    assert torch.equal(w, base + y)
    h.close()
    b.close()
