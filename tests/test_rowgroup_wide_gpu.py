"""The jump-group kernel on long rows, where a row takes one part of 256, 512 or
1,024 threads: pf 3p5n (rows up to 1,651: 256 threads for single vectors, 512 where a
load takes two FP64 or four FP32 vectors) and pf 3p6n (up to 3,952: 512 and 1,024),
stored and accumulated, on a few output rows against the oracle's share of them; and
the FP64 columns that Lanczos has it write, by the Ritz values of short runs against
a projection formed with the same context's applyH.

Tolerances: FP64 1e-12 and FP32 2e-5 of the largest output (sums of up to a few
thousand terms in another order); Ritz values 1e-10 of the largest (two
orthogonalizations of six vectors in FP64)."""
import numpy as np
import pytest

from bigstickpublick_b200 import model
import oracle

pytestmark = pytest.mark.gpu

TOL = {np.float64: 1e-12, np.float32: 2e-5}


@pytest.fixture(scope="module", params=[(3, 5), (3, 6)], ids=["pf 3p5n", "pf 3p6n"])
def space(request):
    from bigstickpublick_b200.engine import Hamiltonian
    p, n = request.param
    t = model.build_tables(model.pf_model(p, n, seed=5, jz2=(p + n) % 2))
    h = Hamiltonian(t)
    yield t, h
    h.close()


@pytest.mark.parametrize("dt,nb", [(np.float64, 1), (np.float64, 2), (np.float64, 4), (np.float32, 1), (np.float32, 2),
                                   (np.float32, 4), (np.float32, 8)])
def test_rows_against_the_oracle(space, dt, nb):
    import torch
    t, h = space
    pstart = t.a["pstart"]
    n = len(pstart)
    rng = np.random.default_rng(nb)
    x = rng.standard_normal((t.dim, nb)).astype(dt)
    base = rng.standard_normal((t.dim, nb)).astype(dt)
    shape = (t.dim, nb) if nb > 1 else (t.dim,)
    xd = torch.from_numpy(x).cuda().reshape(shape)
    y = torch.full_like(xd, float("nan"))
    h.applyh(xd, y)
    z = torch.from_numpy(base).cuda().reshape(shape)
    h.applyh(xd, z, accumulate=True)
    torch.cuda.synchronize()
    assert torch.equal(z, torch.from_numpy(base).cuda().reshape(shape) + y)
    y = y.cpu().numpy().reshape(t.dim, nb)
    for r in (0, n // 2, n - 2):
        lo, hi = int(pstart[r]), int(pstart[r + 2]) if r + 2 < n else t.dim
        ref = oracle.applyh_rows(t, x.reshape(-1), lo, hi, nb=nb).reshape(t.dim, nb)[lo:hi]
        assert np.abs(y[lo:hi] - ref).max() < TOL[dt] * np.abs(ref).max()


@pytest.mark.parametrize("nb", [1, 2])
def test_lanczos_columns(space, nb):
    import torch
    t, h = space
    m = 6
    v = torch.zeros(t.dim, m, dtype=torch.float64, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(nb)
    v[:, :nb] = torch.linalg.qr(torch.randn(t.dim, nb, dtype=torch.float64, device="cuda", generator=g))[0]
    pivot = v[:, :nb].cpu().numpy()
    hv = torch.zeros_like(v)
    for k in range(0, m, nb):
        x = v[:, k:k + nb].contiguous()
        w = h.applyh(x if nb > 1 else x[:, 0]).reshape(t.dim, nb)
        hv[:, k:k + nb] = w
        if k + nb < m:
            for _ in range(2):
                w = w - v[:, :k + nb] @ (v[:, :k + nb].T @ w)
                w = torch.linalg.qr(w)[0]
            v[:, k + nb:k + 2 * nb] = w
    small = v.T @ hv
    ref = torch.linalg.eigvalsh(0.5 * (small + small.T)).cpu().numpy()
    got, _, _ = h.lanczos(nkeep=2, niter=m // nb, nb=nb, matvec_prec=8, lanc_prec=8, fixed_iter=True,
                          pivot=np.ascontiguousarray(pivot) if nb > 1 else pivot[:, 0].copy())
    assert np.abs(got[:2] - ref[:2]).max() < 1e-10 * np.abs(ref).max()


def test_contexts_of_different_sizes_in_turn():
    """The shared-memory limit belongs to a kernel, not to a context: contexts whose
    launches need different amounts, used in turn, each keep their results."""
    import torch
    from bigstickpublick_b200.engine import Hamiltonian
    specs = [model.pf_model(3, 6, seed=5, jz2=1), model.sd_model(3, 4, seed=2, jz2=1), model.pf_model(2, 6, seed=5),
             model.pf_model(3, 4, seed=5, jz2=1)]
    hams, xs, first = [], [], []
    for s in specs:
        t = model.build_tables(s)
        hams.append(Hamiltonian(t))
        xs.append([torch.randn(t.dim, 2, dtype=dt, device="cuda") for dt in (torch.float32, torch.float64)])
        first.append([(hams[-1].applyh(x[:, 0].contiguous()).clone(), hams[-1].applyh(x).clone()) for x in xs[-1]])
    for k in (2, 0, 1, 3, 0):
        for x, (one, two) in zip(xs[k], first[k]):
            assert torch.equal(hams[k].applyh(x), two)
            assert torch.equal(hams[k].applyh(x[:, 0].contiguous()), one)
    for h in hams:
        h.close()
