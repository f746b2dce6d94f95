"""The work that users of this framework have it do, as timed cases.

Each case is one call (or one solve) through the public Python interface on
seeded synthetic interactions: Hamiltonian applications from the smallest
basis to the pf 6p6n one, in FP32 and FP64, on single vectors and blocks, on
device and on host vectors; a three-body Hamiltonian; a batch of systems; a
Lanczos solve; eigenvalue gradients; one-body transition densities.

``exact`` evaluates the same sums in FP64 with plain torch, straight from the
reference-layout tables (jumps, phases, matrix elements, opbundles).
"""
import math

import numpy as np
import torch

from bigstickpublick_b200 import engine, model

SPE, PP, NN, PN, PPP, NNN, PPN, PNN = 1, 2, 3, 4, 7, 8, 9, 10


def _case(kind, shell, np_, nn, prec=64, nb=1, acc=False, **more):
    return dict(kind=kind, shell=shell, protons=np_, neutrons=nn, prec=prec, nb=nb, acc=acc, **more)


def listed():
    return [
        # smallest basis (dim 640): what a user tries first, and members of a
        # scan over nuclei; launch latency
        dict(_case("applyh", "sd", 2, 2), name="sd2p2n_f64"),
        # mid-shell sd (dim 93,710), single precision as lanc_prec = 4 ships
        dict(_case("applyh", "sd", 6, 6, prec=32), name="sd6p6n_f32"),
        # pf shell (dim 1,963,461) in double precision, the plain solver's matvec
        dict(_case("applyh", "pf", 4, 4), name="pf4p4n_f64"),
        # the same space as block Lanczos applies it: eight vectors at once
        dict(_case("applyh", "pf", 4, 4, prec=32, nb=8), name="pf4p4n_f32_nb8"),
        # odd nucleus (2Jz = 1, dim 6,004,205), rows of uneven length,
        # vec2 = vec2 + H vec1 as the Fortran loop calls it
        dict(_case("applyh", "pf", 5, 4, prec=32, acc=True), name="pf5p4n_f32_acc"),
        # the largest single-GPU space (dim 109,954,620)
        dict(_case("applyh", "pf", 6, 6, prec=32), name="pf6p6n_f32"),
        # the drop-in call: host vectors in and out through the C interface
        dict(_case("applyh_host", "pf", 4, 4, prec=32, acc=True), name="pf4p4n_f32_host"),
        # three-body forces (PPP, PPN, PNN, NNN bundles)
        dict(_case("applyh3", "pf", 3, 4, prec=32), name="pf3p4n_threebody_f32"),
        # 256 independent sd Hamiltonians of uneven size in one launch
        dict(_case("batch", "sd", 0, 0, prec=32, systems=256), name="batch256_f32"),
        # a whole solve: 300 Lanczos iterations, full reorthogonalization
        dict(_case("lanczos", "sd", 6, 6, niter=300, nkeep=5), name="sd6p6n_lanczos_f64"),
        # Hellmann-Feynman gradients of five states
        dict(_case("grad", "sd", 6, 6, states=5), name="sd6p6n_grad"),
        # one-body transition densities of all pairs of ten states
        dict(_case("density", "pf", 4, 4, states=10), name="pf4p4n_density"),
    ]


def draw(rng):
    kind = rng.choice(["applyh"] * 6 + ["applyh_host", "applyh3", "batch", "lanczos", "grad", "density"])
    prec = rng.choice([32, 64])
    if kind == "applyh":
        if rng.random() < 0.5:
            shell, p, n, nb = "sd", rng.randint(2, 8), rng.randint(2, 8), rng.choice([1, 1, 1, 2, 3, 4, 8, 16])
        else:
            shell, p, n = "pf", rng.randint(2, 5), rng.randint(2, 5)
            nb = rng.choice([1, 1, 1, 2, 4, 8]) if p + n <= 8 else 1
        return _case(kind, shell, p, n, prec=prec, nb=nb, acc=rng.random() < 0.3)
    if kind == "applyh_host":
        shell = rng.choice(["sd", "pf"])
        return _case(kind, shell, rng.randint(3, 5), rng.randint(2, 4), prec=prec, acc=rng.random() < 0.5)
    if kind == "applyh3":
        shell = rng.choice(["sd", "pf"])
        return _case(kind, shell, rng.randint(2, 3), rng.randint(2, 4), prec=prec, nb=rng.choice([1, 1, 2]))
    if kind == "batch":
        return _case(kind, "sd", 0, 0, prec=prec, systems=int(round(math.exp(rng.uniform(math.log(8), math.log(256))))))
    if kind == "lanczos":
        return _case(kind, "sd", rng.randint(4, 7), rng.randint(4, 7), niter=rng.randint(200, 300), nkeep=rng.randint(1, 5),
                     nb=rng.choice([1, 1, 2]))
    if kind == "grad":
        shell = rng.choice(["sd", "pf"])
        return _case(kind, shell, rng.randint(2, 6) if shell == "sd" else rng.randint(2, 3), rng.randint(2, 6) if shell == "sd" else 3,
                     states=rng.randint(1, 5))
    return _case("density", rng.choice(["sd", "pf"]), rng.randint(2, 4), rng.randint(3, 4), states=rng.randint(1, 16))


# ------------------------------------------------------------------ inputs
def _spec(case, seed):
    make = model.sd_model if case["shell"] == "sd" else model.pf_model
    p, n = case["protons"], case["neutrons"]
    return make(p, n, seed=1 + seed, jz2=(p + n) % 2)


def _tables(case, seed):
    if case["kind"] == "applyh3":
        return model.build_tables3(_spec(case, seed), w2=1.0, w3=0.1, seed=1 + seed)
    return model.build_tables(_spec(case, seed))


def _batch_tables(case, seed):
    """Valence counts of the seeded sd batch (2 to 8 of each kind, the same
    nuclei for every seed), each nucleus with an interaction of its own."""
    specs = []
    for i in range(case["systems"]):
        m = model.batch_member(i)
        specs.append(model.sd_model(m.np_, m.nn, seed=1000 * (seed % 100000) + i, jz2=m.jz2))
    return model.build_tables_many(specs)


def _dtype(case):
    return torch.float32 if case["prec"] == 32 else torch.float64


def _vectors(dim, k, seed, dtype, start=0.0):
    """(vin, vout) of dim x k (dim for k = 1): a normalized random vector per
    column, as a Lanczos step meets it, and the vector to write or add to."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (dim,) if k == 1 else (dim, k)
    v = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).to(dtype) * (1.0 / math.sqrt(dim))
    w = torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).to(dtype) * (1.0 / math.sqrt(dim)) if start else torch.zeros_like(v)
    return v, w


def _states(dim, k, seed):
    """k orthonormal random vectors on the host (dim x k, FP64): the states of
    a chaotic spectrum have Gaussian amplitudes."""
    v, _ = _vectors(dim, k, seed, torch.float64)
    q, _ = torch.linalg.qr(v.reshape(dim, k))
    return np.ascontiguousarray(q.cpu().numpy())


def prepare(case, seed):
    kind, dt = case["kind"], _dtype(case)
    if kind == "batch":
        tabs = _batch_tables(case, seed)
        b = engine.Batch(tabs)
        x, y = _vectors(sum(b.dims), 1, seed, dt)
        return dict(kind=kind, batch=b, out=y, vin=list(x.split(b.dims)), vout=list(y.split(b.dims)))
    t = _tables(case, seed)
    h = engine.Hamiltonian(t)
    if kind in ("applyh", "applyh3"):
        x, y = _vectors(t.dim, case["nb"], seed, dt, case["acc"])
        return dict(kind=kind, h=h, x=x, y=y, acc=case["acc"])
    if kind == "applyh_host":
        x, y = _vectors(t.dim, case["nb"], seed, dt, case["acc"])
        return dict(kind=kind, h=h, x=x.cpu().numpy(), y=y.cpu().numpy(), acc=case["acc"])
    if kind == "lanczos":
        x, _ = _vectors(t.dim, case["nb"], seed, torch.float64)
        return dict(kind=kind, h=h, pivot=_pivot(x).cpu().numpy(), niter=case["niter"], nkeep=case["nkeep"], nb=case["nb"])
    return dict(kind=kind, h=h, states=_states(t.dim, case["states"], seed))


def _pivot(x):
    if x.ndim == 1:
        return x / x.norm()
    return torch.linalg.qr(x)[0].contiguous()


def run(state):
    kind = state["kind"]
    if kind in ("applyh", "applyh3", "applyh_host"):
        return state["h"].applyh(state["x"], state["y"], accumulate=state["acc"])
    if kind == "batch":
        state["batch"].applyh(state["vin"], state["vout"])
        return state["out"]
    if kind == "lanczos":
        e, _, _ = state["h"].lanczos(nkeep=state["nkeep"], niter=state["niter"], nb=state["nb"], matvec_prec=8, lanc_prec=8,
                                     fixed_iter=True, pivot=state["pivot"])
        return e
    if kind == "grad":
        return state["h"].grad(state["states"])
    return state["h"].density1b(state["states"])


# ------------------------------------------------------------------- work
def _pairs(t):
    """(optype, proton side, neutron side) sizes of every opbundle's loop."""
    a = t.a
    for b in range(int(t.s["nbundles"])):
        op = int(a["optype"][b])
        npx = max(0, int(a["pxend"][b] - a["pxstart"][b] + 1))
        nnx = max(0, int(a["nxend"][b] - a["nxstart"][b] + 1))
        if t.threebody and op in (PP, NN, PN):
            continue
        yield op, npx, nnx


def _updates(t):
    return sum(p * n for _, p, n in _pairs(t))


def _table_bytes(t):
    arrays = list(t.a.values()) + (list(t.a3.values()) if t.threebody else [])
    return sum(x.nbytes for x in arrays)


def work(case):
    kind, size = case["kind"], case["prec"] // 8
    if kind == "batch":
        tabs = _batch_tables(case, 0)
        return {"bytes": sum(_table_bytes(t) + 2 * size * t.dim for t in tabs), "flops": 2 * sum(_updates(t) for t in tabs)}
    t = _tables(case, 0)
    if kind == "lanczos":
        # per step: one application, and the overlaps with and the removal of every earlier vector
        m, nb = case["niter"], case["nb"]
        steps = m // nb
        return {"bytes": 8 * t.dim * (3 * m + 2 * nb * steps * (steps + 1) // 2) + _table_bytes(t),
                "flops": 2 * _updates(t) * m + 4 * t.dim * nb * nb * (steps * (steps + 1) // 2)}
    if kind == "grad":
        k = case["states"]
        return {"bytes": 8 * k * (t.dim + t.s["nmatpp"] + t.s["nmatnn"] + t.s["nmatpn"]) + _table_bytes(t), "flops": 2 * k * _updates(t)}
    if kind == "density":
        k, d = case["states"], t.extra["density"]
        rows = sum(max(0, int(d["pxend"][b] - d["pxstart"][b] + 1)) * max(0, int(d["nxend"][b] - d["nxstart"][b] + 1))
                   for b in range(int(d["nbundles"])))
        nq = int(t.s["nhsps_pl"] + t.s["nhsps_pr"])
        return {"bytes": 8 * k * t.dim + 16 * k * k * nq * nq + sum(x.nbytes for x in d.values() if hasattr(x, "nbytes")),
                "flops": 2 * k * k * rows}
    nb = case["nb"]
    return {"bytes": (3 if case["acc"] else 2) * size * nb * t.dim + _table_bytes(t), "flops": 2 * nb * _updates(t)}


# ------------------------------------------------------------------- exact
_CHUNK = 1 << 25


def _loops(t):
    """Every opbundle's updates out[o] += me * in[i], in chunks, as
    (o, i, me, label name, label, sign): indices 0-based, me the float matrix
    element times its phases in FP64, label 0-based in the named table."""
    a, s, dev = t.a, t.s, "cuda"
    up = {}

    def col(name, table=None):
        key = (name, table is not None)
        if key not in up:
            up[key] = torch.from_numpy(np.ascontiguousarray((table or a)[name])).to(dev)
        return up[key]

    def side(kind, b, ends, table=None):
        """(in, out, phase, range) of one side's jumps of a bundle."""
        lo, hi = ends
        r = slice(lo - 1, hi)
        i, f = col(kind + "_isd", table)[r], col(kind + "_fsd", table)[r]
        if b:
            i, f = f, i
        return i, f, col(kind + "_phase", table)[r].double(), r

    nl_p, nl_n = int(s["nhsps_pl"]), int(s["nhsps_nl"])
    ld = int(s["nhsps_nl"] + s["nhsps_nr"] + 1)
    for b in range(int(s["nbundles"])):
        op, back, cs = int(a["optype"][b]), chr(int(a["hchar"][b])) == "b", max(1, int(a["cstride"][b]))
        px, nx = (int(a["pxstart"][b]), int(a["pxend"][b])), (int(a["nxstart"][b]), int(a["nxend"][b]))
        if px[1] < px[0] or nx[1] < nx[0] or (t.threebody and op in (PP, NN, PN)):
            continue
        a3 = t.a3
        ps, ns = col("pstart")[px[0] - 1:px[1]:cs] if op in (SPE, NN, NNN) else None, \
            col("nstart")[nx[0] - 1:nx[1]:cs] if op in (SPE, PP, PPP) else None
        if op == SPE:
            me = (col("pspe_h")[px[0] - 1:px[1]][:, None] + col("nspe_h")[nx[0] - 1:nx[1]][None, :]).double().reshape(-1)
            o = (ps[:, None] + ns[None, :] - 1).reshape(-1)
            yield o, o, me, None, None, None
            continue
        if op in (PP, PPP, NN, NNN):
            pside = op in (PP, PPP)
            three = op in (PPP, NNN)
            kind = {PP: "p2b", PPP: "p3b", NN: "n2b", NNN: "n3b"}[op]
            hm = {PP: "hmatpp", PPP: "hmatppp", NN: "hmatnn", NNN: "hmatnnn"}[op]
            i, f, ph, r = side(kind, back, px if pside else nx, a3 if three else None)
            lab = col(kind + "_op", a3 if three else None)[r].long() - 1
            me = col(hm, a3 if three else None)[lab].double() * ph
            other = ns if pside else ps
            step = max(1, _CHUNK // len(other))
            for c in range(0, len(i), step):
                w = slice(c, c + step)
                yield ((f[w][:, None] + other[None, :] - 1).reshape(-1), (i[w][:, None] + other[None, :] - 1).reshape(-1),
                       me[w][:, None].expand(-1, len(other)).reshape(-1), hm, lab[w][:, None].expand(-1, len(other)).reshape(-1),
                       ph[w][:, None].expand(-1, len(other)).reshape(-1))
            continue
        pi, pf, pph, pr = side("p2b" if op == PPN else "p1b", back, px)
        ni, nf, nph, nr = side("n2b" if op == PNN else "n1b", back, nx)
        if op == PN:
            ca, cb, hm, table = col("cpnpair"), col("dpnpair"), "hmatpn", None
            xa, xc = (col("p1b_cop")[pr].long() + nl_p) * ld, (col("p1b_dop")[pr].long() + nl_p) * ld
            yb, yd = col("n1b_cop")[nr].long() + nl_n, col("n1b_dop")[nr].long() + nl_n
        elif op == PPN:
            npp = int(t.s3["npairs_p"])
            ca, cb, hm, table = col("cppntriplet", a3).long(), col("dppntriplet", a3).long(), "hmatppn", a3
            xa, xc = col("p2b_cop", a3)[pr].long() - 1, col("p2b_dop", a3)[pr].long() - 1
            yb, yd = (col("n1b_cop")[nr].long() + nl_n) * npp, (col("n1b_dop")[nr].long() + nl_n) * npp
        else:
            npn = int(t.s3["npairs_n"])
            ca, cb, hm, table = col("cpnntriplet", a3).long(), col("dpnntriplet", a3).long(), "hmatpnn", a3
            xa, xc = (col("p1b_cop")[pr].long() + nl_p) * npn, (col("p1b_dop")[pr].long() + nl_p) * npn
            yb, yd = col("n2b_cop", a3)[nr].long() - 1, col("n2b_dop", a3)[nr].long() - 1
        h = col(hm, table)
        step = max(1, _CHUNK // len(ni))
        for c in range(0, len(pi), step):
            w = slice(c, c + step)
            lab = (ca[xa[w][:, None] + yb[None, :]] + cb[xc[w][:, None] + yd[None, :]] - 1).reshape(-1)
            ph = (pph[w][:, None] * nph[None, :]).reshape(-1)
            yield ((pf[w][:, None] + nf[None, :] - 1).reshape(-1), (pi[w][:, None] + ni[None, :] - 1).reshape(-1),
                   h[lab].double() * ph, hm, lab, ph)


def _apply(t, x, y):
    """y + H x in FP64 for x of dim or dim x k."""
    for o, i, me, _, _, _ in _loops(t):
        y.index_add_(0, o, me * x[i] if x.ndim == 1 else me[:, None] * x[i])
    return y


def _matrix(t):
    """H as a sparse FP64 matrix."""
    parts = [(o, i, me) for o, i, me, _, _, _ in _loops(t)]
    o, i, me = (torch.cat(p) for p in zip(*parts))
    return torch.sparse_coo_tensor(torch.stack([o, i]), me, (t.dim, t.dim)).coalesce().to_sparse_csr()


def _solve(t, pivot, m, nkeep):
    """Lowest Ritz values of a Lanczos run of m vectors, orthogonalized twice
    against all earlier ones (the projected matrix formed in full)."""
    h, nb = _matrix(t), pivot.shape[1]
    v = torch.zeros(t.dim, m, dtype=torch.float64, device="cuda")
    v[:, :nb] = pivot
    hv = torch.zeros_like(v)
    for k in range(0, m - m % nb, nb):
        hv[:, k:k + nb] = w = h @ v[:, k:k + nb]
        if k + 2 * nb > m:
            break
        for _ in range(2):
            w = w - v[:, :k + nb] @ (v[:, :k + nb].T @ w)
        q, _ = torch.linalg.qr(w)
        for _ in range(2):
            q = q - v[:, :k + nb] @ (v[:, :k + nb].T @ q)
            q, _ = torch.linalg.qr(q)
        v[:, k + nb:k + 2 * nb] = q
    used = m - m % nb
    small = v[:, :used].T @ hv[:, :used]
    return torch.linalg.eigvalsh(0.5 * (small + small.T))[:nkeep].cpu().numpy()


def _gradients(t, states):
    x = torch.from_numpy(states).cuda()
    size = {"hmatpp": t.s["nmatpp"], "hmatnn": t.s["nmatnn"], "hmatpn": t.s["nmatpn"]}
    g = {n: torch.zeros(int(k), x.shape[1], dtype=torch.float64, device="cuda") for n, k in size.items()}
    for o, i, _, name, lab, ph in _loops(t):
        if name is None:
            return None
        for k in range(x.shape[1]):
            g[name][:, k].index_add_(0, lab, ph * x[o, k] * x[i, k])
    return {n[4:]: v.T.contiguous().cpu().numpy() for n, v in g.items()}


def _densities(t, states):
    a, s, d = t.a, t.s, t.extra["density"]
    x = torch.from_numpy(states).cuda()
    k = x.shape[1]
    out = []
    for op, sp, nl, nq in ((5, "p", int(s["nhsps_pl"]), int(s["nhsps_pl"] + s["nhsps_pr"])),
                           (6, "n", int(s["nhsps_nl"]), int(s["nhsps_nl"] + s["nhsps_nr"]))):
        dens = torch.zeros(nq * nq, k, k, dtype=torch.float64, device="cuda")
        for b in range(int(d["nbundles"])):
            if int(d["optype"][b]) != op:
                continue
            cs, back = int(d["cstride"][b]), chr(int(d["hchar"][b])) == "b"
            j = ("px", "nx") if op == 5 else ("nx", "px")
            j0, j1, c0, c1 = (int(d[n][b]) for n in (j[0] + "start", j[0] + "end", j[1] + "start", j[1] + "end"))
            n = (c1 - c0 + cs) // cs
            if j1 < j0 or n < 1:
                continue
            # the other species' SDs are an arithmetic progression of basis states
            if op == 5:
                rows = int(a["nstart"][c0 - cs]) - 2 + cs + cs * np.arange(n)
            else:
                stride = int(a["pstart"][c0 - 1 + cs] - a["pstart"][c0 - 1]) if n > 1 else 0
                rows = int(a["pstart"][c0 - 1]) - 1 + stride * np.arange(n)
            rows = torch.from_numpy(rows).cuda()
            get = lambda name: torch.from_numpy(d[sp + "1b_" + name][j0 - 1:j1].astype(np.int64)).cuda()
            isd, fsd, c, dd, ph = get("isd"), get("fsd"), get("cop"), get("dop"), get("phase").double()
            c, dd = (torch.where(q < 0, -q - 1, nl + q - 1) for q in (c, dd))
            if back:
                isd, fsd, c, dd = fsd, isd, dd, c
            step = max(1, _CHUNK // (n * k))
            for w in range(0, len(isd), step):
                z = slice(w, w + step)
                m = torch.bmm(x[fsd[z][:, None] + rows].transpose(1, 2), x[isd[z][:, None] + rows]) * ph[z][:, None, None]
                dens.index_add_(0, (c * nq + dd)[z], m)
        out.append(dens.permute(1, 2, 0).reshape(k, k, nq, nq).cpu().numpy())
    return {"p": out[0], "n": out[1]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        tabs = _batch_tables(case, seed)
        dims = [t.dim for t in tabs]
        x, _ = _vectors(sum(dims), 1, seed, _dtype(case))
        return torch.cat([_apply(t, v, torch.zeros_like(v)) for t, v in zip(tabs, x.double().split(dims))])
    t = _tables(case, seed)
    n = _updates(t)
    if n * case["nb"] > 2.5e10:
        return None
    if kind in ("applyh", "applyh3", "applyh_host"):
        x, y = _vectors(t.dim, case["nb"], seed, _dtype(case), case["acc"])
        r = _apply(t, x.double(), y.double())
        return r.cpu().numpy() if kind == "applyh_host" else r
    if kind == "lanczos":
        if n > 3e8:
            return None
        x, _ = _vectors(t.dim, case["nb"], seed, torch.float64)
        return _solve(t, _pivot(x).reshape(t.dim, -1), case["niter"], case["nkeep"])
    states = _states(t.dim, case["states"], seed)
    return _gradients(t, states) if kind == "grad" else _densities(t, states)
