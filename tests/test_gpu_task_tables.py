"""A plan's task tables reach the device as a launch's arguments up to 1 KiB and
16 KiB, and by a staged copy above: a rectangular product of N column blocks
has a table of 64 N bytes, so N around 16 and 256 takes every way.  Integer
data: exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [1, 15, 16, 17, 255, 256, 257, 1000])
def test_tables_of_every_size(caps, cuda, blocks):
    import torch
    m, k, n = 8, 24, 8 * blocks
    rng = np.random.default_rng(blocks)
    A = rng.integers(-50, 51, (m, k)).astype(np.float64)
    out = []
    for _ in range(2):  # a second call's tables replace the first's
        B = rng.integers(-50, 51, (k, n)).astype(np.float64)
        C = torch.full((m * n,), float("nan"), dtype=torch.float64, device=cuda)
        caps.rect_mm(torch.from_numpy(A.T.copy().reshape(-1)).to(cuda), torch.from_numpy(B.T.copy().reshape(-1)).to(cuda),
                     C, m, n, k, 1, "d", [1, blocks, 1])
        out.append((B, C))
    torch.cuda.synchronize()
    for B, C in out:
        assert np.array_equal(C.cpu().numpy().reshape(n, m).T, (A.astype(np.int64) @ B.astype(np.int64)).astype(np.float64))
