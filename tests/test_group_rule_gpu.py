"""The rule that sends applyH to the jump groups or to the row tiles, on both
sides of its lines, against the oracle: rows of a few positions, fewer and more
of them than CTAs fit at once (sd 4p2n, 6p2n, pf 3p1n); rows of about a hundred, below and above twice as many (pf 3p3n,
4p3n); blocks of one, two and four 16-byte loads.

Tolerances as in test_rowgroup_gpu.py: FP64 1e-12 of the largest output, FP32
2e-5 (sums of some hundred terms in another order)."""
import numpy as np
import pytest

from bigstickpublick_b200 import model
import oracle

pytestmark = pytest.mark.gpu

SPACES = {
    "sd 4p2n": (lambda: model.sd_model(4, 2, seed=2), 471),
    "sd 6p2n": (lambda: model.sd_model(6, 2, seed=2), 862),
    "pf 3p1n": (lambda: model.pf_model(3, 1, seed=5), 932),
    "pf 3p3n": (lambda: model.pf_model(3, 3, seed=5), 1140),
    "pf 4p3n": (lambda: model.pf_model(4, 3, seed=5, jz2=1), 4829),
}
TOL = {np.float64: 1e-12, np.float32: 2e-5}


@pytest.mark.parametrize("name", list(SPACES))
def test_both_sides_of_the_rule(name):
    import torch
    from bigstickpublick_b200.engine import Hamiltonian
    mk, rows = SPACES[name]
    t = model.build_tables(mk())
    pstart = t.a["pstart"]
    assert len(pstart) == rows
    # a run of rows in the middle and the last ones: the oracle walks them alone
    cuts = [(int(pstart[k]), int(pstart[k + 12])) for k in (0, rows // 2)] + [(int(pstart[-12]), t.dim)]
    h = Hamiltonian(t)
    rng = np.random.default_rng(rows)
    for dt in (np.float64, np.float32):
        for nb in (1, 2, 4, 8, 16):
            x = rng.standard_normal((t.dim, nb)).astype(dt)
            got = h.applyh(torch.from_numpy(x).cuda().reshape(t.dim, nb) if nb > 1 else torch.from_numpy(x[:, 0].copy()).cuda())
            torch.cuda.synchronize()
            got = got.cpu().numpy().reshape(t.dim, nb)
            for lo, hi in cuts:
                ref = oracle.applyh_rows(t, x.reshape(-1), lo, hi, nb=nb).reshape(t.dim, nb)[lo:hi]
                assert np.abs(ref).max() > 0
                assert np.abs(got[lo:hi] - ref).max() < TOL[dt] * np.abs(ref).max(), (dt, nb, lo)
    h.close()
