"""'d' steps in sequence keep the operand sums and the products in the C
quadrants and three buffers: the same bits as a 'b' step's, in every buffer
alignment and for odd quarters (their sums take the unaligned path)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("form,n,r,bs,pat", [("plain", 4, 2, 1, "dd"), ("plain", 28, 2, 7, "dd"),
                                             ("plain", 620, 2, 1, "db"), ("split", 4, 1, 1, "d"),
                                             ("split", 310, 1, 1, "d"), ("split", 620, 2, 1, "dd"),
                                             ("split", 620, 2, 1, "bd"), ("split", 1036, 2, 7, "dd")])
def test_lean_steps_bit_identical_to_b_steps(caps, cuda, form, n, r, bs, pat, offset):
    import torch
    rng = np.random.default_rng(n + r + offset)

    def buffer(x):
        t = torch.full((n * n + 2,), float("nan"), dtype=torch.float64, device=cuda)
        t[offset:offset + n * n] = torch.from_numpy(x).to(cuda) if x is not None else float("nan")
        return t

    a, b = buffer(rng.uniform(-1, 1, n * n)), buffer(rng.uniform(-1, 1, n * n))
    d = caps.MatDescriptor.make(n, r, bs)
    got = {}
    for p in (pat, "b" * r):
        c = buffer(None)
        limit = caps.workspace_size(d, p, form=form) if p == pat else 0
        view = slice(offset, offset + n * n)
        caps.multiply(a[view], b[view], c[view], d, p, form=form, workspace_limit=limit)
        torch.cuda.synchronize()
        got[p] = c.cpu().numpy()
    assert np.array_equal(got[pat], got["b" * r], equal_nan=True)
    assert np.isnan(got[pat]).sum() == 2  # nothing outside the matrix is written
