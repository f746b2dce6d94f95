"""Host-pointer applyH from 4 MB on, where the row kernel's launches run in
row-range chunks and the copies of vout run beside them: the same bits as one
launch on device pointers, in both modes and with interleaved blocks.  One
FP64 vector (3.8 MB) lies below the line and runs whole."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ham():
    from bigstickpublick_b200 import model
    from bigstickpublick_b200.engine import Hamiltonian
    t = model.build_tables(model.pf_model(4, 3, seed=3, jz2=1))
    h = Hamiltonian(t, device=0)
    yield t, h
    h.close()


@pytest.mark.parametrize("nb,dt", [(1, np.float64), (2, np.float64), (3, np.float32), (4, np.float32)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_equals_the_device_call(ham, nb, dt, accumulate):
    import torch
    t, h = ham
    bytes_ = t.dim * nb * np.dtype(dt).itemsize
    assert (bytes_ >= 4 << 20) == (nb > 1) and bytes_ < 32 << 20
    rng = np.random.default_rng(nb + 10 * accumulate)
    shape = (t.dim, nb) if nb > 1 else (t.dim,)
    x = rng.standard_normal(shape).astype(dt)
    base = rng.standard_normal(shape).astype(dt) if accumulate else None
    host = h.applyh(x, None if base is None else base.copy(), accumulate=accumulate)
    dev = h.applyh(torch.from_numpy(x).cuda(), torch.from_numpy(base).cuda() if accumulate else None,
                   accumulate=accumulate)
    torch.cuda.synchronize()
    assert np.array_equal(host, dev.cpu().numpy())
