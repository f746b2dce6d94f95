"""Host-pointer applyH with room on the device for one of its two staging vectors
only: refused with BSG_ERR_NOMEM, also the second time, and served once there is room
(the staging vector that was found stays)."""
import numpy as np
import pytest

from bigstickpublick_b200 import model

pytestmark = pytest.mark.gpu


def test_room_for_one_vector():
    import torch
    from bigstickpublick_b200.engine import BsgError, Hamiltonian
    t = model.build_tables(model.pf_model(4, 4, seed=5))   # 251 MB for 16 FP64 vectors
    h = Hamiltonian(t)
    x = np.random.default_rng(1).standard_normal((t.dim, 16))
    one = h.applyh(x[:, :1].copy()[:, 0])   # kernels and small staging in place
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - x.nbytes - x.nbytes // 2, dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            with pytest.raises(BsgError, match="memory"):
                h.applyh(x)
    finally:
        del hog
        torch.cuda.empty_cache()
    got = h.applyh(x)
    assert np.abs(got[:, 0] - one).max() < 1e-12 * np.abs(one).max()
    h.close()
