"""The split operands of the tensor-core DF contractions (df_split_kernel) and
the J pass (df_jmat_kernel) at the edges of their tiles: fewer rows than a
tile, columns that end inside a 64-wide K tile, aux blocks whose boundary
falls inside a lane's pair (odd n), a tile and one row more -- J and K of
random symmetric factors against the FP64 contractions of the same factors."""

import pytest

from felizjueves_b200 import configs
from felizjueves_b200.df import DFEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,n", [(1, 1), (3, 7), (5, 64), (2, 129), (9, 130), (40, 33)])
def test_df_contractions_at_tile_edges(cuda, lib_built, nq, n):
    import torch
    w = configs.cluster(1, 3)
    df = DFEngine(w.basis, configs.aux_basis(w))
    g = torch.Generator(device="cpu").manual_seed(nq * 1000 + n)
    B = torch.randn((nq, n, n), dtype=torch.float64, generator=g)
    B = (B + B.transpose(1, 2)).contiguous().to(cuda)
    D = torch.randn((n, n), dtype=torch.float64, generator=g)
    D = (D + D.T).contiguous().to(cuda)
    J, K = df.jk(D, "bf16x3", B=B)
    J0, K0 = df.jk(D, "fp64", B=B)
    assert float((J - J0).norm() / J0.norm()) <= 1e-13
    # The bound: the tensor cores truncate each FP32 accumulation, at most 2^-23
    # of the running sum, one a K = 16 step and product -- 24 a 64-wide K tile --
    # in either GEMM (contractions of n and of nq n terms); the operands' own
    # 2^-24 is inside it.  (A first bound of two roundings in random directions
    # missed that the truncations add up: 3.1e-6 at (5, 64).)
    steps = 24 * (-(-nq * n // 64) + -(-n // 64))
    assert float((K - K0).norm() / K0.norm()) <= steps * 2.0 ** -23
