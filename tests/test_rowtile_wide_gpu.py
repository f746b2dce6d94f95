"""The row-tile kernels on the spaces and blocks that the jump groups leave to them,
with rows of several hundred and several thousand positions: few long rows (pf 2p5n,
190 of up to 1,651; pf 2p6n, up to 3,952), where single FP32 vectors take 256-position
tiles (k_rows_f1<8, ...>), FP64 ones 128 (k_rows_d1<4, ...>) and blocks of eight 64
(k_rows<..., 8, 2, ...>); and sd 6p6n blocks of two 16-byte loads (FP32 nb = 8, FP64
nb = 4).  Since the jump groups, pf 4p4n and pf 6p6n of test_applyh_sizes_gpu.py, and
sd 6p6n there but for FP32 nb = 8, run k_rowgroup.

Tolerances: FP64 1e-12 and FP32 2e-5 of the largest output, as there."""
import numpy as np
import pytest

from bigstickpublick_b200 import model
import oracle

pytestmark = pytest.mark.gpu

TOL = {np.float64: 1e-12, np.float32: 2e-5}
BLOCKS = {
    "pf 2p5n": [(np.float32, 1), (np.float64, 1), (np.float32, 8), (np.float64, 8), (np.float32, 16), (np.float64, 3)],
    "pf 2p6n": [(np.float32, 1), (np.float64, 1), (np.float32, 8), (np.float64, 2)],
    "sd 6p6n": [(np.float32, 8), (np.float64, 4)],
}


@pytest.mark.parametrize("name", list(BLOCKS))
def test_rows_against_the_oracle(name):
    import torch
    from bigstickpublick_b200.engine import Hamiltonian
    p, n = int(name[3]), int(name[5])
    t = model.build_tables((model.sd_model if name[:2] == "sd" else model.pf_model)(p, n, seed=5, jz2=(p + n) % 2))
    pstart = t.a["pstart"]
    nr = len(pstart)
    h = Hamiltonian(t)
    for dt, nb in BLOCKS[name]:
        x = np.random.default_rng(nb).standard_normal((t.dim, nb)).astype(dt)
        xd = torch.from_numpy(x).cuda().reshape((t.dim, nb) if nb > 1 else (t.dim,))
        y = torch.full_like(xd, float("nan"))
        h.applyh(xd, y)
        z = torch.ones_like(xd)
        h.applyh(xd, z, accumulate=True)
        torch.cuda.synchronize()
        assert torch.equal(z, 1 + y)
        y = y.cpu().numpy().reshape(t.dim, nb)
        for r in (0, nr // 2, nr - 2):
            lo, hi = int(pstart[r]), int(pstart[r + 2]) if r + 2 < nr else t.dim
            ref = oracle.applyh_rows(t, x.reshape(-1), lo, hi, nb=nb).reshape(t.dim, nb)[lo:hi]
            assert np.abs(y[lo:hi] - ref).max() < TOL[dt] * np.abs(ref).max(), (dt, nb, r)
    h.close()
