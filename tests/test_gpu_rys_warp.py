"""The warp-autonomous Rys kernel (rys_warp.cuh) at the sizes where its split
can go wrong: fewer kets than a group (one atom), units cut into slices (small
systems) and not (a system whose units outnumber the grid), every class it is
built for (set_rys(2)), and contraction degrees that leave ragged table rounds
-- against the register kernel and the HGP interpreter (set_rys(0)), whose
boundary and transfers are other code, at the plain FP64 bar."""

import numpy as np
import pytest

from felizjueves_b200 import configs
from felizjueves_b200.fock import FockEngine
from felizjueves_b200.shell import Basis, Shell, primitive_norm

pytestmark = pytest.mark.gpu


def _ragged(seed):
    """Three centres with s, p, d, f shells of degrees 1, 2, 5 and 7."""
    rng = np.random.default_rng(seed)
    shells = []
    for c in rng.uniform(0.0, 4.0, (3, 3)):
        for l, deg in ((0, 7), (0, 1), (1, 5), (1, 1), (2, 2), (2, 1), (3, 1), (3, 2)):
            ex = [0.25 * 2.7 ** k * (1 + 0.1 * l) for k in range(deg)]
            shells.append(Shell(l, tuple(map(float, c)), ex, [primitive_norm(l, e) / deg for e in ex]))
    B = Basis(tuple(shells))
    return B, configs.random_density(rng, B.n_ao, 6)


def _system(name):
    if name == "ragged":
        return _ragged(3)
    w = configs.cluster(int(name), 5 + int(name))
    return w.basis, w.D


@pytest.mark.parametrize("name", ["1", "2", "7", "ragged"])
def test_warp_kernel_matches_other_engines(cuda, lib_built, name):
    basis, D = _system(name)
    eng = FockEngine(basis)
    eng.plan(D, 1e-12, 4, export=False)
    out = {}
    for mode in (0, 1, 2):
        eng.set_rys(mode)
        out[mode] = (eng.build_host(D), sum(s["computed"] for s in eng.launch_stats()))
    scale = max(1.0, np.abs(out[0][0][0]).max() / 100.0)  # 1e-13 of the largest element above 100
    for mode in (1, 2):
        assert out[mode][1] == out[0][1]  # every quartet once, slices or not
        for a, b in zip(out[mode][0], out[0][0]):
            assert np.abs(a - b).max() <= 1e-11 * scale


@pytest.mark.parametrize("name", ["1", "7", "ragged"])
def test_warp_kernel_fp32_tier(cuda, lib_built, name):
    """Every unit in FP32, unchecked, mode 2: FP32 accuracy relative to G."""
    from felizjueves_b200 import _lib
    basis, D = _system(name)
    eng = FockEngine(basis)
    eng.plan(D, 1e-12, 4, export=False)
    G = eng.build_host(D)[2]
    eng.set_rys(2)
    eng.set_route_check(0.0)
    G32 = eng.build_host(D, precision=_lib.FJB_ROUTED, threshold=1e30)[2]
    assert 0.0 < np.abs(G32 - G).max() <= 1e-5 * np.abs(G).max()


def test_long_queues_are_taken_several_items_at_a_time(cuda, lib_built):
    """75 p and 50 f shells: (pp|pf) and (pf|pf) have more than 64 work units
    a team of the kernel twice over, so its teams take them two or more at a
    time.  Every quartet once, and the result of the other engines."""
    rng = np.random.default_rng(1)
    shells = []
    for l, n in ((1, 75), (3, 50)):
        for e, c in zip(rng.uniform(0.4, 1.2, n), rng.uniform(0.0, 2.0, (n, 3))):
            shells.append(Shell(l, tuple(map(float, c)), [float(e)], [primitive_norm(l, float(e))]))
    B = Basis(tuple(shells))
    D = configs.random_density(rng, B.n_ao, 8)
    eng = FockEngine(B)
    eng.plan(D, 1e-12, 4, export=False)
    out = {}
    for mode in (0, 1):
        eng.set_rys(mode)
        out[mode] = (eng.build_host(D), sum(s["computed"] for s in eng.launch_stats()))
    units = {(r["la"], r["lb"], r["lc"], r["ld"]): r["units"] for r in eng.class_stats()}
    assert units[1, 1, 1, 3] >= 2 * 64 * 148 * 16  # a warp a team, at most 16 an SM
    assert units[1, 3, 1, 3] >= 2 * 64 * 148 * 4   # 128 threads a team, at most 4 an SM
    assert out[0][1] == out[1][1]
    for a, b in zip(out[1][0], out[0][0]):
        # sums of 5e7 terms in another order, each to 1e-16 of the largest
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


@pytest.mark.parametrize("ls", [(1,), (0, 1)])
def test_small_classes_keep_their_fp32_bodies(cuda, lib_built, ls):
    """A system whose classes have a few units each, every unit in FP32: the
    classes of s and p shells run the FP32 register bodies that they run in
    large systems, so the default mode's result is mode 0's to FP64 rounding
    (a Rys build's, mode 2, differs by FP32 rounding)."""
    from felizjueves_b200 import _lib
    rng = np.random.default_rng(7)
    shells = []
    for c in rng.uniform(0.0, 5.0, (4, 3)):
        for l in ls:
            ex = [0.4 * 2.9 ** k for k in range(3)]
            shells.append(Shell(l, tuple(map(float, c)), ex, [primitive_norm(l, e) / 3 for e in ex]))
    B = Basis(tuple(shells))
    D = configs.random_density(rng, B.n_ao, 6)
    eng = FockEngine(B)
    eng.plan(D, 1e-12, 4, export=False)
    eng.set_route_check(0.0)
    G = {}
    for mode in (0, 1, 2):
        eng.set_rys(mode)
        G[mode] = eng.build_host(D, precision=_lib.FJB_ROUTED, threshold=1e30)[2]
    scale = np.abs(G[0]).max()
    assert np.abs(G[2] - G[0]).max() > 1e-9 * scale
    assert np.abs(G[1] - G[0]).max() <= 1e-12 * scale


@pytest.mark.parametrize("precision,threshold", [(0, 0.0), (1, 1e-9)])
def test_overlapped_build_order(cuda, lib_built, precision, threshold):
    """A small build forks its class launches onto side streams: D written
    just before it on the caller's stream is the D it reads, its outputs are
    ready for that stream, and the captured graph gives the same."""
    import torch
    w = configs.cluster(4, 9)
    eng = FockEngine(w.basis)
    eng.plan(w.D, w.tau, w.n_mag, export=False)
    ref = [torch.tensor(m, device=cuda) for m in eng.build_host(w.D)]
    D0 = torch.tensor(w.D, device=cuda)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    for graph in (False, True, False):
        D, outs = torch.zeros_like(D0), [torch.zeros_like(D0) for _ in range(3)]
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            for _ in range(3):
                D.zero_()
                D.add_(D0)
                eng.build(D, J=outs[0], K=outs[1], G=outs[2], precision=precision, threshold=threshold, graph=graph)
                got = [o.clone() for o in outs]
                for o in outs:
                    o.fill_(float("nan"))
        st.synchronize()
        for a, b in zip(got, ref):
            assert float((a - b).abs().max()) <= (1e-11 if precision == 0 else 1e-8)


def test_build_on_a_priority_stream(cuda, lib_built):
    """A build on a high-priority stream, between two on a default one."""
    import torch
    w = configs.cluster(3, 9)
    eng = FockEngine(w.basis)
    eng.plan(w.D, w.tau, w.n_mag, export=False)
    want = eng.build_host(w.D)
    D = torch.tensor(w.D, device=cuda)
    for prio in (0, -5, 0, -5):
        st = torch.cuda.Stream(priority=prio)
        st.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(st):
            got = [m.clone() for m in eng.build(D)]
        st.synchronize()
        for a, b in zip(got, want):
            assert np.abs(a.cpu().numpy() - b).max() <= 1e-11


def test_first_build_captured_overlaps(cuda, lib_built):
    """A handle's first build inside the caller's own capture: the recorded
    graph runs its classes side by side, so their times add up to well more
    than the build's, as an eager build's do."""
    import torch
    w = configs.cluster(3, 9)
    ref = FockEngine(w.basis)
    ref.plan(w.D, w.tau, w.n_mag, export=False)
    want = ref.build_host(w.D)
    del ref
    eng = FockEngine(w.basis)
    eng.plan(w.D, w.tau, w.n_mag, export=False)
    D = torch.tensor(w.D, device=cuda)
    outs = [torch.zeros_like(D) for _ in range(3)]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        eng.build(D, J=outs[0], K=outs[1], G=outs[2])
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    for a, b in zip(outs, want):
        assert np.abs(a.cpu().numpy() - b).max() <= 1e-11
    total = eng.last_build_stats()[0]
    assert sum(r["ms"] for r in eng.class_stats()) > 2.0 * total


@pytest.mark.parametrize("atoms", [1, 2, 5])
def test_j_engine_orders_and_reproduces(cuda, lib_built, oracle_lib, atoms):
    """The J-engine's Rys classes with fewer kets than a warp's step (one
    atom: one ff record) and ragged last steps, against the oracle; and the
    same bits on every build (one writer an element, fixed order)."""
    import torch
    w = configs.cluster(atoms, 3)
    eng = FockEngine(w.basis)
    D = torch.tensor(w.D, device=cuda)
    J = eng.coulomb(D, tau=0.0).clone()
    again = eng.coulomb(D, tau=0.0).clone()
    torch.cuda.synchronize()
    assert torch.equal(J, again)
    if atoms < 5:
        Jo, _ = oracle_lib.jk(oracle_lib.OracleBasis.of(w.basis), w.D)
        assert np.abs(J.cpu().numpy() - Jo).max() <= 1e-11
    else:
        eng.plan(w.D, 0.0, 4, export=False)
        assert float((J - eng.build(D)[0]).abs().max()) <= 1e-11
