"""The Rys kernel (rys_warp.cuh): the large classes' boundary by Rys
quadrature, then the build's HRR and digest.  Held to the oracle at the
plain FP64 bar (1e-11 max-abs) on clusters with every class to (ff|ff), to
the HGP interpreter it replaces, and in FP32 (the routed path's tier) to the
FP64 build at FP32 accuracy."""

import numpy as np
import pytest

from felizjueves_b200 import configs
from felizjueves_b200.fock import FockEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms,seed", [(3, 5), (4, 7), (2, 3)])
def test_rys_build_matches_oracle(cuda, lib_built, oracle_lib, atoms, seed):
    w = configs.cluster(atoms, seed)
    eng = FockEngine(w.basis)
    eng.plan(w.D, 0.0, 4)
    J, K, G = eng.build_host(w.D)
    Jo, Ko = oracle_lib.jk(oracle_lib.OracleBasis.of(w.basis), w.D)
    assert np.abs(J - Jo).max() <= 1e-11
    assert np.abs(K - Ko).max() <= 1e-11
    assert np.abs(G - (Jo - 0.5 * Ko)).max() <= 1e-11


def test_rys_matches_interpreter(cuda, lib_built):
    """Same plan, same density: the Rys engine against the HGP interpreter
    on a screened 6-atom cluster (contraction degrees to 9 x 9)."""
    w = configs.cluster(6, 11)
    eng = FockEngine(w.basis)
    eng.plan(w.D, w.tau, w.n_mag)
    Jr, Kr, Gr = eng.build_host(w.D)
    eng.set_rys(False)
    Ji, Ki, Gi = eng.build_host(w.D)
    eng.set_rys(True)
    for a, b in ((Jr, Ji), (Kr, Ki), (Gr, Gi)):
        assert np.abs(a - b).max() <= 1e-11


def test_rys_fp32_tier(cuda, lib_built, oracle_lib):
    """Every unit routed to FP32: the Rys kernel's FP32 tier and, for the
    classes of at most 100 boundary values, the FP32 register bodies, against
    the oracle at FP32 accuracy relative to G."""
    from felizjueves_b200 import _lib, router
    w = configs.cluster(3, 5)
    eng = FockEngine(w.basis)
    eng.plan(w.D, w.tau, w.n_mag)
    _, _, G32 = eng.build_host(w.D, precision=_lib.FJB_ROUTED, threshold=1e30)
    n32, n64 = router.route_stats(eng)
    Jo, Ko = oracle_lib.jk(oracle_lib.OracleBasis.of(w.basis), w.D)
    Go = Jo - 0.5 * Ko
    assert n64 == 0 and n32 > 0
    assert np.abs(G32 - Go).max() / np.abs(Go).max() <= 1e-5


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_each_engine_matches_oracle(cuda, lib_built, oracle_lib, mode):
    """The same cluster on each engine, FP64 at the plain bar and every unit
    in FP32 at FP32 accuracy: mode 0 the register kernels and the interpreter,
    2 the Rys kernel for every class it has, 1 the default choice."""
    from felizjueves_b200 import _lib
    w = configs.cluster(3, 5)
    eng = FockEngine(w.basis)
    eng.plan(w.D, 0.0, 4, export=False)
    eng.set_rys(mode)
    J, K, G = eng.build_host(w.D)
    engines = {(r["la"], r["lb"], r["lc"], r["ld"]): r["engine"] for r in eng.class_stats()}
    assert len(engines) == 55
    if mode == 0:  # 24 register classes, 31 interpreted
        assert list(engines.values()).count(1) == 24 and 2 not in engines.values()
    else:  # every class but those of an ss bra and (sp|sp), (sp|sd)
        rys = {c for c, e in engines.items() if e == 2}
        assert rys == {c for c in engines if c[:2] != (0, 0) and c not in ((0, 1, 0, 1), (0, 1, 0, 2))}
    Jo, Ko = oracle_lib.jk(oracle_lib.OracleBasis.of(w.basis), w.D)
    Go = Jo - 0.5 * Ko
    for a, b in ((J, Jo), (K, Ko), (G, Go)):
        assert np.abs(a - b).max() <= 1e-11
    eng.set_route_check(0.0)
    G32 = eng.build_host(w.D, precision=_lib.FJB_ROUTED, threshold=1e30)[2]
    assert 0.0 < np.abs(G32 - Go).max() <= 1e-5 * np.abs(Go).max()


@pytest.mark.parametrize("atoms,seed", [(3, 5), (6, 11)])
def test_fp32_tier_within_the_tap_s_error(cuda, lib_built, atoms, seed):
    """fjb_eri_blocks_fp32 evaluates the HGP recurrences in FP32, what mode 0
    runs; the default tier, whose large classes run the Rys kernel, is no
    further from FP64 on the 64-atom workload's shells (measured: K 0.3 to
    0.45 of it)."""
    from felizjueves_b200 import _lib
    w = configs.cluster(atoms, seed)
    eng = FockEngine(w.basis)
    eng.plan(w.D, w.tau, w.n_mag, export=False)
    eng.set_route_check(0.0)
    K = eng.build_host(w.D)[1]
    err = {}
    for mode in (0, 1):
        eng.set_rys(mode)
        err[mode] = np.linalg.norm(eng.build_host(w.D, precision=_lib.FJB_ROUTED, threshold=1e30)[1] - K)
    assert 0.0 < err[1] <= err[0]
