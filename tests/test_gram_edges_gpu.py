"""The tall-skinny Gram kernel (qg_gram_small_d) at the edges of its tiles: parts of 32 columns,
steps of 8 rows, blocks with fewer rows than warps, rows of odd length (scalar loads).
Tolerance: each of N products and additions rounds once, |error| <= N eps sum |a b| in any order;
the rows here are below 2^12, so 2^12 * 1.1e-16 of sum |a b| is a bound."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 7, 8, 255, 258, 4001])
@pytest.mark.parametrize("ma,mb", [(1, 1), (8, 31), (32, 32), (33, 9), (64, 64), (63, 65)])
def test_gram_tile_edges(cuda_ctx, N, ma, mb):
    import torch
    from qumasun_b200.engine import check, lib
    rng = np.random.default_rng(N * 100 + ma)
    A, B = rng.normal(size=(ma, N)), rng.normal(size=(mb, N))
    Ad, Bd = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    out = torch.full((mb, ma), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    check(lib().qg_gram_small_d(cuda_ctx.h, N, ma, mb, C.c_void_p(Ad.data_ptr()), C.c_void_p(Bd.data_ptr()), 0.5,
                                C.c_void_p(out.data_ptr())), "qg_gram_small_d")
    err = np.abs(out.cpu().numpy().T - 0.5 * (A @ B.T))
    assert (err <= 2.0 ** 12 * 1.2e-16 * (np.abs(A) @ np.abs(B).T) + 1e-300).all()
