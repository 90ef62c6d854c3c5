"""The J-engine's FP32 tier (fjb_coulomb_mixed) is decided for chunks of 32
sorted kets by the chunk's largest bound, at every order.  Few shells of
similar exponents and a density that puts the first ket of every order far
above the rest: a build whose threshold no chunk's first ket is under is the
FP64 build to the bit, although most record pairs are under it."""

import numpy as np
import pytest

from felizjueves_b200 import configs
from felizjueves_b200.fock import FockEngine
from felizjueves_b200.shell import Basis, Shell, primitive_norm

pytestmark = pytest.mark.gpu

# record pairs of an order: 15 ff, 15 df, 16 dd and pf, 6 pd, 3 pp -- several
# steps of 4 to 8 kets of every Rys order (7 to 12), one chunk of 32
_SHELLS = [3] * 5 + [2] * 3 + [1] * 2


def _system():
    rng = np.random.default_rng(4)
    shells = []
    for i, l in enumerate(_SHELLS):
        e = 0.5 + 0.01 * i
        shells.append(Shell(l, tuple(map(float, rng.uniform(-0.4, 0.4, 3))), [e], [primitive_norm(l, e)]))
    B = Basis(tuple(shells))
    D = 1e-5 * configs.random_density(rng, B.n_ao, 6)
    ends = list(B.offsets[1:]) + [B.n_ao]
    for a, b in ((0, 1), (0, 5), (0, 8), (5, 6), (5, 8), (8, 9)):  # one shell pair of each order to the front
        D[B.offsets[a]:ends[a], B.offsets[b]:ends[b]] += 1.0
        D[B.offsets[b]:ends[b], B.offsets[a]:ends[a]] += 1.0
    return B, D


def test_tier_decided_by_chunks_of_32(cuda, lib_built):
    import torch
    B, D = _system()
    eng = FockEngine(B)
    p = eng.j_plan_lists(D)
    G, key, L = (np.asarray(p[k]) for k in ("G", "key", "L"))
    counts = [int((L == l).sum()) for l in set(L.tolist())]
    assert max(counts) <= 32  # one chunk an order
    thr = 0.5 * G.min() * min(key[L == l].max() for l in set(L.tolist()))
    under = sum(int((g * key < thr).sum()) for g in G)
    assert under > 0.5 * len(G) ** 2  # most pairs are under it, no chunk's first is
    Dt = torch.tensor(D, device=cuda)
    J64 = eng.coulomb(Dt, tau=0.0).clone()
    J = eng.coulomb(Dt, tau=0.0, threshold=float(thr)).clone()
    J32 = eng.coulomb(Dt, tau=0.0, threshold=1e30).clone()
    torch.cuda.synchronize()
    assert not torch.equal(J32, J64)
    assert torch.equal(J, J64)
