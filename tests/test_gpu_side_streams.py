"""Calls that fork onto side streams, as seen from the caller's stream: what
that stream wrote just before is what they read, what they write is ready for
it, and it may overwrite or free both right after.  A wait in front of each
call makes a fork that does not wait read the old input."""

import ctypes

import pytest

from felizjueves_b200 import _lib, configs
from felizjueves_b200.fock import FockEngine

pytestmark = pytest.mark.gpu

SLEEP = 3_000_000  # clock cycles, about 1.5 ms


def _check(run, D0, ref, bar):
    """run(D) -> outputs, on a stream of its own: zero D, wait, write D, run,
    copy the outputs, overwrite everything."""
    import torch
    D = torch.zeros_like(D0)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        for _ in range(3):
            torch.cuda._sleep(SLEEP)
            D.copy_(D0)
            outs = run(D)
            got = [o.clone() for o in outs]
            D.zero_()
            for o in outs:
                o.fill_(float("nan"))
    st.synchronize()
    for a, b in zip(got, ref):
        assert float((a - b).abs().max()) <= bar


@pytest.mark.parametrize("threshold", [0.0, 1e-9])
def test_coulomb(cuda, lib_built, threshold):
    import torch
    w = configs.cluster(4, 9)
    eng = FockEngine(w.basis)
    D0 = torch.tensor(w.D, device=cuda)
    J = eng.coulomb(D0, tau=1e-12, threshold=threshold).clone()
    out = torch.zeros_like(J)
    _check(lambda D: [eng.coulomb(D, tau=1e-12, threshold=threshold, J=out)], D0, [J], 0.0)


def test_one_electron(cuda, lib_built):
    """The nuclei are host values; D only orders the call."""
    import torch
    w = configs.cluster(6, 9)
    nuclei = [(float(1 + i % 9), tuple(map(float, c))) for i, c in enumerate(w.coords)]
    eng = FockEngine(w.basis)
    ref = [m.clone() for m in eng.one_electron(nuclei)]
    _check(lambda D: list(eng.one_electron(nuclei)), torch.zeros(4, device=cuda), ref, 0.0)


def test_df_eri3(cuda, lib_built):
    import torch
    from felizjueves_b200.df import DFEngine
    w = configs.cluster(2, 5)
    df = DFEngine(w.basis, configs.aux_basis(w))
    n = len(df.aux.shells)
    ref = df.eri3_block(0, n, tau=0.0).clone()
    out = torch.zeros_like(ref)

    def run(D):
        return [df.eri3_block(0, n, tau=0.0, out=out)]

    _check(run, torch.zeros(4, device=cuda), [ref], 0.0)


@pytest.mark.parametrize("precision,threshold", [(_lib.FJB_FP64, 0.0), (_lib.FJB_ROUTED, 1e-9)])
def test_batch(cuda, lib_built, precision, threshold):
    import torch
    from felizjueves_b200.batch import BatchBuilder
    bb = BatchBuilder([configs.cluster(n, 4200 + n) for n in (3, 2, 4)])
    L, b = _lib.load(), bb._merged()

    def build():
        rc = L.fjb_batch_build(b, int(precision), ctypes.c_double(threshold),
                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0

    build()
    ref = [m.clone() for o in bb.out for m in o]
    src = [D.clone() for D in bb.D]
    for D in bb.D:
        D.zero_()

    def run(_):
        for D, s in zip(bb.D, src):
            D.copy_(s)
        build()
        for D in bb.D:
            D.zero_()
        return [m for o in bb.out for m in o]

    _check(run, torch.zeros(4, device=cuda), ref, 1e-11 if precision == _lib.FJB_FP64 else 1e-8)


def test_two_handles_on_two_streams(cuda, lib_built):
    """Builds of two handles enqueued in turn on two streams, one of them in a
    capture in between: each gets its own result."""
    import torch
    ws = [configs.cluster(3, 9), configs.cluster(4, 5)]
    engs, Ds, refs = [], [], []
    for w in ws:
        eng = FockEngine(w.basis)
        eng.plan(w.D, w.tau, w.n_mag, export=False)
        D = torch.tensor(w.D, device=cuda)
        engs.append(eng)
        Ds.append(D)
        refs.append([m.clone() for m in eng.build(D)])
    sts = [torch.cuda.Stream() for _ in ws]
    outs = [[torch.zeros_like(D) for _ in range(3)] for D in Ds]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    for rep in range(3):
        for eng, D, st, o in zip(engs, Ds, sts, outs):
            with torch.cuda.stream(st):
                torch.cuda._sleep(SLEEP)
                eng.build(D, J=o[0], K=o[1], G=o[2])
        if rep == 0:
            torch.cuda.synchronize()
            with torch.cuda.graph(g):
                engs[0].build(Ds[0], J=outs[0][0], K=outs[0][1], G=outs[0][2])
    torch.cuda.synchronize()
    for o, ref in zip(outs, refs):
        for a, b in zip(o, ref):
            assert float((a - b).abs().max()) <= 1e-11
            a.zero_()
    g.replay()
    torch.cuda.synchronize()
    for a, b in zip(outs[0], refs[0]):
        assert float((a - b).abs().max()) <= 1e-11
