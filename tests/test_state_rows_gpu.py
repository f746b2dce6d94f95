"""Row-major state blocks (bsg_grad_rows, bsg_density1b_rows) give the bits of
the column-major entry points: odd and even state counts (odd ones are padded on
the device), one state, and blocks that are neither (copied)."""
import numpy as np
import pytest

from bigstickpublick_b200 import model

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ham():
    from bigstickpublick_b200.engine import Hamiltonian
    t = model.build_tables(model.sd_model(3, 2, seed=3, jz2=1))
    h = Hamiltonian(t)
    yield t, h
    h.close()


@pytest.mark.parametrize("ns", [1, 2, 3, 5, 8])
def test_rows_equal_columns(ham, ns):
    t, h = ham
    v = np.random.default_rng(ns).standard_normal((t.dim, ns))
    wide = np.zeros((t.dim, 2 * ns))
    wide[:, ::2] = v
    blocks = {"rows": np.ascontiguousarray(v), "cols": np.asfortranarray(v), "strided": wide[:, ::2]}
    grads = {k: h.grad(b) for k, b in blocks.items()}
    dens = {k: h.density1b(b) for k, b in blocks.items()}
    for k in ("rows", "strided"):
        for key in grads["cols"]:
            assert grads[k][key].shape[0] == ns
            assert np.array_equal(grads[k][key], grads["cols"][key]), (k, key)
        for key in ("p", "n"):
            assert np.array_equal(dens[k][key], dens["cols"][key]), (k, key)
