"""A matrix element that is not finite reaches the outputs that it couples and no
others: contexts with one stay on the row tiles, which do not read the unused record
places that the jump groups multiply with a zero input.  Twelve labels are tried one
by one, each the one that a PN bundle's first proton and first neutron jump use (the
first element of the jump's row of elements); the outputs' finite, infinite and
not-a-number places must be the oracle's."""
import numpy as np
import pytest

from bigstickpublick_b200 import model
import oracle

pytestmark = pytest.mark.gpu


def _first_labels(t):
    """hmatpn labels (0-based) of every PN bundle's first pair of jumps."""
    a, s = t.a, t.s
    nl_p, nl_n = int(s["nhsps_pl"]), int(s["nhsps_nl"])
    ld = nl_n + int(s["nhsps_nr"]) + 1
    out = []
    for b in range(int(s["nbundles"])):
        if a["optype"][b] != 4 or a["pxend"][b] < a["pxstart"][b] or a["nxend"][b] < a["nxstart"][b]:
            continue
        p, n = int(a["pxstart"][b]) - 1, int(a["nxstart"][b]) - 1
        at = lambda pc, nc: (int(pc) + nl_p) * ld + int(nc) + nl_n
        out.append(int(a["cpnpair"][at(a["p1b_cop"][p], a["n1b_cop"][n])] + a["dpnpair"][at(a["p1b_dop"][p], a["n1b_dop"][n])]) - 1)
    return sorted(set(out))


@pytest.mark.parametrize("name", ["pf 4p1n", "sd 3p4n"])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_non_finite_elements(name, bad):
    from bigstickpublick_b200.engine import Hamiltonian
    shell, p, n = ("pf", 4, 1) if name.startswith("pf") else ("sd", 3, 4)
    t = model.build_tables((model.pf_model if shell == "pf" else model.sd_model)(p, n, seed=6, jz2=1))
    good = t.a["hmatpn"].copy()
    x = np.random.default_rng(5).standard_normal(t.dim)
    labels = _first_labels(t)
    partial = 0
    for k in labels[::max(1, len(labels) // 12)][:12]:
        t.a["hmatpn"][:] = good
        t.a["hmatpn"][k] = bad
        ref = oracle.applyh(t, x)
        h = Hamiltonian(t)
        for v in (x, x.astype(np.float32)):
            got = h.applyh(v)
            assert np.array_equal(np.isfinite(got), np.isfinite(ref)), (k, v.dtype)
            assert np.array_equal(np.isnan(got), np.isnan(ref)), (k, v.dtype)
        h.close()
        partial += 0 < np.isfinite(ref).sum() < ref.size
    assert partial > 3
