"""The jump-group row kernel and the rule that sends calls to it, against the
oracle's loops: rows of less than a slice, of a few slices (eight one-warp
parts) and longer (one part of several warps); operators used by 1, 2, 3, 4 and
more jumps of a row; blocks whose 16-byte loads take 1, 2 or 4 vectors, and the
same blocks on a base that allows only single loads; three-body operators split
into sub-operators.

Tolerances: FP64 1e-12 of the largest output (sums of some hundred terms, each
rounding 1.1e-16, in another order); FP32 2e-5 (the same with 6e-8)."""
import numpy as np
import pytest

from bigstickpublick_b200 import model
import oracle

pytestmark = pytest.mark.gpu

SYSTEMS = {
    "sd 1p1n": lambda: model.build_tables(model.sd_model(1, 1, seed=11)),
    "pf 4p1n": lambda: model.build_tables(model.pf_model(4, 1, seed=6, jz2=1)),        # rows of one or two positions
    "sd 3p4n": lambda: model.build_tables(model.sd_model(3, 4, seed=2, jz2=1)),        # eight parts
    "pf 2p4n": lambda: model.build_tables(model.pf_model(2, 4, seed=5)),               # few long rows: the row-tile kernel
    "pf 3p4n": lambda: model.build_tables(model.pf_model(3, 4, seed=5, jz2=1)),        # one part, rows of some hundred
    "sd 3p3n three-body": lambda: model.build_tables3(model.sd_model(3, 3, seed=4), w2=1.0, w3=0.1, seed=9),
}
TOL = {np.float64: 1e-12, np.float32: 2e-5}


@pytest.fixture(scope="module")
def built():
    from bigstickpublick_b200.engine import Hamiltonian
    out = {}
    for name, mk in SYSTEMS.items():
        t = mk()
        out[name] = (t, Hamiltonian(t, pn_table_max=32 if "three" in name else 0))
    yield out
    for _, h in out.values():
        h.close()


def _run(h, x, nb, offset, base=None):
    """applyH on device vectors whose storage starts `offset` elements in."""
    import torch
    dt = torch.float64 if x.dtype == np.float64 else torch.float32
    shape = x.shape

    def place(v):
        store = torch.empty(v.size + offset, dtype=dt, device="cuda")
        store[offset:] = torch.from_numpy(np.ascontiguousarray(v).reshape(-1)).cuda()
        return store[offset:].view(shape)

    vin = place(x)
    vout = place(np.full_like(x, np.nan) if base is None else base)
    h.applyh(vin, vout, accumulate=base is not None)
    torch.cuda.synchronize()
    return vout.cpu().numpy()


@pytest.mark.parametrize("name", list(SYSTEMS))
@pytest.mark.parametrize("dt", [np.float64, np.float32])
@pytest.mark.parametrize("nb,offset", [(1, 0), (1, 1), (2, 0), (3, 0), (4, 0), (4, 1), (5, 0), (6, 0), (8, 0), (16, 0), (16, 2)])
def test_against_oracle(built, name, dt, nb, offset):
    if name == "pf 3p4n" and nb not in (1, 3, 4):
        pytest.skip("the oracle takes long on this space")
    t, h = built[name]
    rng = np.random.default_rng(100 * nb + offset)
    x = rng.standard_normal((t.dim, nb)).astype(dt) if nb > 1 else rng.standard_normal(t.dim).astype(dt)
    ref = oracle.applyh(t, x.reshape(-1), nb=nb).reshape(x.shape)
    got = _run(h, x, nb, offset)
    assert np.abs(got - ref).max() < TOL[dt] * np.abs(ref).max()
    assert np.array_equal(_run(h, x, nb, offset), got)
    base = rng.standard_normal(x.shape).astype(dt)
    assert np.array_equal(_run(h, x, nb, offset, base), base + got)


@pytest.mark.parametrize("name", ["pf 4p1n", "sd 3p4n", "pf 3p4n"])
@pytest.mark.parametrize("nb", [1, 2])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_non_finite_inputs_reach_the_same_outputs(built, name, nb, bad):
    """The staged rows, their zero places and the grouped sums add no product
    that the loops do not have."""
    t, h = built[name]
    x = np.random.default_rng(5).standard_normal((t.dim, nb) if nb > 1 else t.dim)
    x.reshape(t.dim, -1)[t.dim // 3, 0] = bad
    ref = oracle.applyh(t, x.reshape(-1), nb=nb).reshape(x.shape)
    got = _run(h, x, nb, 0)
    assert 0 < np.isfinite(ref).sum() < ref.size
    assert np.array_equal(np.isfinite(got), np.isfinite(ref))
    assert np.array_equal(np.isnan(got), np.isnan(ref))
