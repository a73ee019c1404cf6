"""The plain form's base case picks its tile (64, 32 or 16 on a side) per
launch and skips blocks outside the leaf.  Every tile accumulates an entry
over k in the same order, so the pick never changes a bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 3, 8, 9, 14, 16, 17, 31, 33, 64, 65, 98, 129, 250, 500, 777, 1030])
def test_picked_tile_bit_identical_to_fixed_tile(caps, cuda, m):
    import torch
    rng = np.random.default_rng(m)
    A = torch.from_numpy(rng.uniform(-1, 1, m * m)).to(cuda)
    B = torch.from_numpy(rng.uniform(-1, 1, m * m)).to(cuda)
    out = {}
    for tile in ("64x64", "128x64", "32x32"):
        out[tile] = torch.full((m * m,), float("nan"), dtype=torch.float64, device=cuda)
        caps.leaf_gemm(A, B, out[tile], m, tile=tile)
    torch.cuda.synchronize()
    assert torch.equal(out["64x64"], out["128x64"]) and torch.equal(out["64x64"], out["32x32"])
    Ai = rng.integers(-50, 51, (m, m)).astype(np.float64)
    Bi = rng.integers(-50, 51, (m, m)).astype(np.float64)
    caps.leaf_gemm(torch.from_numpy(Ai.T.copy().reshape(-1)).to(cuda),
                   torch.from_numpy(Bi.T.copy().reshape(-1)).to(cuda), out["64x64"], m)
    torch.cuda.synchronize()
    exact = (Ai.astype(np.int64) @ Bi.astype(np.int64)).astype(np.float64)
    assert np.array_equal(out["64x64"].cpu().numpy().reshape(m, m).T, exact)


@pytest.mark.parametrize("m,n,k", [(70, 33, 21), (9, 200, 5), (300, 17, 130), (1, 1, 1), (640, 520, 35)])
def test_rectangular_edges_exact_on_integers(caps, cuda, m, n, k):
    import torch
    rng = np.random.default_rng(m + n + k)
    A = rng.integers(-50, 51, (m, k)).astype(np.float64)
    B = rng.integers(-50, 51, (k, n)).astype(np.float64)
    C = torch.full((m * n,), float("nan"), dtype=torch.float64, device=cuda)
    caps.rect_mm(torch.from_numpy(A.T.copy().reshape(-1)).to(cuda), torch.from_numpy(B.T.copy().reshape(-1)).to(cuda),
                 C, m, n, k)
    torch.cuda.synchronize()
    assert np.array_equal(C.cpu().numpy().reshape(n, m).T, (A.astype(np.int64) @ B.astype(np.int64)).astype(np.float64))
