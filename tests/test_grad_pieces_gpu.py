"""Row-major states of a gradient go to the device in pieces of 64 MB: the same
bits as column-major ones over several pieces and a last short one, and no room
needed for a second copy of them."""
import numpy as np
import pytest

from bigstickpublick_b200 import model

pytestmark = pytest.mark.gpu

NS = 40   # 209,715 of the 1,963,461 basis states a piece


def test_pieces_and_room():
    import torch
    from bigstickpublick_b200.engine import Hamiltonian
    t = model.build_tables(model.pf_model(4, 4, seed=5))
    h = Hamiltonian(t)
    v = np.random.default_rng(3).standard_normal((t.dim, NS)) * (1.0 / np.sqrt(t.dim))
    cols = h.grad(np.asfortranarray(v))
    h.close()   # with its scratch
    h = Hamiltonian(t)
    h.grad(np.ascontiguousarray(v[:, :2]))   # tile list, kernels
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - v.nbytes - (320 << 20), dtype=torch.uint8, device="cuda")
    try:
        rows = h.grad(v)
    finally:
        del hog
        torch.cuda.empty_cache()
    h.close()
    assert sorted(rows) == sorted(cols)
    for key in cols:
        assert np.array_equal(rows[key], cols[key]), key
