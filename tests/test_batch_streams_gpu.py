"""Batched applyH calls that are in flight together: each call's vectors are its
own, on two streams and from two host threads, for members with jump groups (one
launch, a CTA per row) and without (the persistent launch and its work counter:
pf 2p4n, few long rows).  A call on a capturing stream is refused and spoils
neither the capture nor the batch.

The results of a call alone are compared with the oracle (tolerances as in
test_batch_gpu.py); calls in flight together must then give the same bits."""
import threading

import numpy as np
import pytest

from bigstickpublick_b200 import model
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def batch():
    from bigstickpublick_b200.engine import Batch
    tabs = [model.build_tables(model.sd_model(5, 5, seed=20 + i)) for i in range(10)]
    tabs += [model.build_tables(model.sd_model(2, 3, seed=40, jz2=1)), model.build_tables(model.pf_model(2, 4, seed=41))]
    b = Batch(tabs)
    yield tabs, b
    b.close()


def _vectors(tabs, seed, dt):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    vin = [torch.randn(t.dim, dtype=dt, device="cuda", generator=g) for t in tabs]
    return vin, [torch.full_like(v, float("nan")) for v in vin]


def _alone(b, vin, vout):
    import torch
    torch.cuda.synchronize()
    b.applyh(vin, vout)
    torch.cuda.synchronize()
    r = [y.clone() for y in vout]
    for y in vout:
        y.fill_(float("nan"))
    torch.cuda.synchronize()
    return r


@pytest.mark.parametrize("prec", [8, 4])
def test_mixed_members_against_oracle(batch, prec):
    import torch
    tabs, b = batch
    vin, vout = _vectors(tabs, 1, torch.float64 if prec == 8 else torch.float32)
    got = _alone(b, vin, vout)
    for k in (0, 9, 10, 11):
        ref = oracle.applyh(tabs[k], vin[k].cpu().numpy())
        assert np.abs(got[k].cpu().numpy() - ref).max() < (1e-12 if prec == 8 else 2e-5) * np.abs(ref).max()


@pytest.mark.parametrize("first", ["side", "default"])
@pytest.mark.parametrize("prec", [8, 4])
def test_two_streams_with_other_vectors(batch, prec, first):
    import torch
    tabs, b = batch
    dt = torch.float64 if prec == 8 else torch.float32
    sets = [_vectors(tabs, s, dt) for s in (2, 3)]
    ref = [_alone(b, *s) for s in sets]
    streams = [torch.cuda.Stream() if first == "side" else torch.cuda.default_stream(), torch.cuda.Stream()]
    for _ in range(5):
        for (vin, vout), s in zip(sets, streams):
            b.applyh(vin, vout, stream=s.cuda_stream)
    torch.cuda.synchronize()
    for (_, vout), r in zip(sets, ref):
        assert all(torch.equal(x, y) for x, y in zip(vout, r))


def test_two_host_threads(batch):
    import torch
    tabs, b = batch
    sets = [_vectors(tabs, s, torch.float32) for s in (4, 5)]
    ref = [_alone(b, *s) for s in sets]
    failed = []

    def work(k):
        s = torch.cuda.Stream()
        try:
            for _ in range(20):
                b.applyh(*sets[k], stream=s.cuda_stream)
            s.synchronize()
        except Exception as e:   # reported below: a thread's exception is otherwise lost
            failed.append(e)

    th = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not failed
    torch.cuda.synchronize()
    for (_, vout), r in zip(sets, ref):
        assert all(torch.equal(x, y) for x, y in zip(vout, r))


def test_capturing_stream_is_refused(batch):
    import torch
    from bigstickpublick_b200.engine import BsgError
    tabs, b = batch
    vin, vout = _vectors(tabs, 6, torch.float32)
    ref = _alone(b, vin, vout)
    x = torch.zeros(8, device="cuda")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x += 1
        with pytest.raises(BsgError):
            b.applyh(vin, vout)
    g.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 1.0
    assert all(torch.equal(x, y) for x, y in zip(_alone(b, vin, vout), ref))
