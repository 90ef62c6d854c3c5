"""The autotuner (autotune.py) times what it sets: on an engine whose Rys
kernel ignores the class configuration, whose overlapped class times hold one
another's, and whose configured kernels have known times, it finds each
class's fastest candidate and leaves the engine's modes as they were."""

import contextlib

import pytest

from felizjueves_b200 import autotune
from felizjueves_b200.fock import FockEngine

CLASSES = [(0, 0, 0, 0), (0, 1, 1, 1), (3, 3, 3, 3)]


class Engine:
    """Class (c, i) runs candidate k in 1 + ((k + i) % n) ms, serial and off the Rys kernel."""

    serial_hgp = FockEngine.serial_hgp

    def __init__(self, candidates, rys, overlap):
        self.candidates, self._rys_mode, self._overlap = candidates, rys, overlap
        self.cfg, self.cfg32, self.routed = {}, {}, False
        self.built, self.fail = [], False

    def set_rys(self, mode):
        self._rys_mode = mode

    def set_overlap(self, on):
        self._overlap = on

    def set_class_config(self, c, threads, slots):
        if c == CLASSES[2] and threads == 1:
            raise ValueError("no register kernel")
        self.cfg[c] = (threads, slots)

    def set_class_config32(self, c, threads, slots):
        self.cfg32[c] = (threads, slots)

    def build(self, D, precision=0, threshold=0.0):
        if self.fail:
            raise RuntimeError("build")
        self.routed = precision == 1
        self.built.append((self._rys_mode, self._overlap))

    def class_stats(self):
        cfg = self.cfg32 if self.routed else self.cfg
        out = []
        for i, c in enumerate(CLASSES):
            n = len(self.candidates)
            k = self.candidates.index(cfg[c]) if c in cfg else 0
            ms = 1.0 if self._rys_mode else 1.0 + (k + i) % n
            out.append(dict(zip(("la", "lb", "lc", "ld"), c), ms=ms))
        if self._overlap:
            out = [dict(r, ms=sum(x["ms"] for x in out)) for r in out]
        return out


@pytest.fixture
def no_gpu(monkeypatch):
    import torch
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: None)


@pytest.mark.parametrize("rys,overlap", [(1, True), (2, False), (0, True)])
@pytest.mark.parametrize("tune,cands,key", [(autotune.autotune, autotune.CANDIDATES, "choice"),
                                            (autotune.autotune32, autotune.CANDIDATES32, "choice32")])
def test_finds_the_fastest(no_gpu, tune, cands, key, rys, overlap):
    eng = Engine(list(cands), rys, overlap)
    choice = tune(eng, None)[key]
    for i, c in enumerate(CLASSES):
        best = [k for k in range(len(cands)) if (k + i) % len(cands) == 0][0]
        assert tuple(choice[",".join(map(str, c))]) == cands[best]
        assert (eng.cfg32 if key == "choice32" else eng.cfg)[c] == cands[best]
    assert set(eng.built) == {(0, False)}
    assert (eng._rys_mode, eng._overlap) == (rys, overlap)


def test_modes_restored_after_a_failure(no_gpu):
    eng = Engine(list(autotune.CANDIDATES), 2, True)
    eng.fail = True
    with contextlib.suppress(RuntimeError):
        autotune.autotune(eng, None)
    assert (eng._rys_mode, eng._overlap) == (2, True)


@pytest.mark.gpu
def test_times_the_configured_kernels(cuda, lib_built):
    """On the engine: the interpreter at (128, 0) and the register kernel are
    told apart where the default mode runs the Rys kernel for both, the build
    is the same with what was found, and serial class times add up to the
    build's."""
    import numpy as np
    import torch
    from felizjueves_b200 import configs
    w = configs.cluster(3, 5)
    eng = FockEngine(w.basis)
    eng.plan(w.D, w.tau, w.n_mag, export=False)
    D = torch.tensor(w.D, device=cuda)
    G = eng.build(D)[2].clone()
    assert {r["engine"] for r in eng.class_stats() if r["la"] + r["ld"] > 0 and r["lb"] > 1} == {2}
    t = autotune.autotune(eng, D, ((1, 0), (128, 0)), reps=3)
    ms = t["ms"]["0,1,1,1"]
    assert abs(ms["1x0"] / ms["128x0"] - 1.0) > 0.05  # two kernels, not one twice
    assert np.abs((eng.build(D)[2] - G).cpu().numpy()).max() <= 1e-11
    eng.set_overlap(False)
    eng.build(D)
    torch.cuda.synchronize()
    assert sum(r["ms"] for r in eng.class_stats()) <= 1.02 * eng.last_build_stats()[0]
