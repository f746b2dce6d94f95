"""bsg_applyh_noalloc after a host applyH whose launches ran in row ranges (4 MB of
output and more on the jump groups): the tile lists that such a call caches lift the
limit of the static array's 65,536 tiles like those of a whole launch.  pf 8p1n has
83,550 rows; three FP64 vectors of it are 5.3 MB."""
import ctypes as C

import numpy as np
import pytest

from bigstickpublick_b200 import model

pytestmark = pytest.mark.gpu


def test_noalloc_after_a_chunked_host_call():
    from bigstickpublick_b200.engine import Hamiltonian
    t = model.build_tables(model.pf_model(8, 1, seed=5, jz2=1))
    assert len(t.a["pstart"]) > 65536 and 4 << 20 <= t.dim * 24 < 8 << 20
    h = Hamiltonian(t)
    lib = h.lib
    lib.bsg_applyh_noalloc.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_int]
    lib.bsg_applyh_noalloc.restype = C.c_int
    x = np.random.default_rng(1).standard_normal((t.dim, 3))
    y = np.zeros_like(x)
    call = lambda out: lib.bsg_applyh_noalloc(h.h, x.ctypes.data, out.ctypes.data, 3, 8, 0)
    assert call(y) == 7 and not y.any()   # BSG_ERR_ARG: no list yet
    ref = h.applyh(x)
    for _ in range(2):
        y.fill(np.nan)
        assert call(y) == 0
        assert np.array_equal(y, ref)
    h.close()
