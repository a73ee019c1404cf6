"""Tall, narrow rectangular products: a launch holds 65535 row tiles, so the
tile the plain form picks must keep within that (integers: exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# the last height whose tiles of 16 fit, the first beyond it, heights beyond
# tiles of 32, and the last that tiles of 64 hold
@pytest.mark.parametrize("m,n,k", [(1048560, 8, 4), (1048561, 8, 4), (1100000, 65, 2), (2000000, 16, 3),
                                   (2097121, 9, 5), (4194240, 2, 1)])
def test_tall_rectangular_product_exact_on_integers(caps, cuda, m, n, k):
    import torch
    rng = np.random.default_rng(m)
    A = rng.integers(-50, 51, (k, m)).astype(np.float64)  # transposed: rows are A's columns
    B = rng.integers(-50, 51, (n, k)).astype(np.float64)
    C = torch.full((m * n,), float("nan"), dtype=torch.float64, device=cuda)
    caps.rect_mm(torch.from_numpy(A.reshape(-1)).to(cuda), torch.from_numpy(B.reshape(-1)).to(cuda), C, m, n, k)
    torch.cuda.synchronize()
    assert np.array_equal(C.cpu().numpy().reshape(n, m), B @ A)
