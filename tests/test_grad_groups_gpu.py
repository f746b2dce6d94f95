"""The adjoint takes up to five states in one pass over the records of a space
that fills the chip: each state's gradient has the bits that it has alone, for
every size of a group (2 and 3 states; 4 and 5; 6 as 3 + 3; 7 as 3 + 4)."""
import numpy as np
import pytest

from bigstickpublick_b200 import model

pytestmark = pytest.mark.gpu


def test_grouped_states_equal_single_states():
    from bigstickpublick_b200.engine import Hamiltonian
    t = model.build_tables(model.sd_model(6, 6, seed=3))
    h = Hamiltonian(t)
    v = np.random.default_rng(2).standard_normal((t.dim, 7))
    v /= np.linalg.norm(v, axis=0)
    alone = [h.grad(v[:, k:k + 1]) for k in range(7)]
    for ns in range(2, 8):
        got = h.grad(np.ascontiguousarray(v[:, :ns]))
        for key in got:
            for k in range(ns):
                assert np.array_equal(got[key][k], alone[k][key][0]), (ns, key, k)
    h.close()
