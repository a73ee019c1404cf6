"""The layout reorder copies long block columns by warps and short ones by
elements or pairs of elements; every block size around its limits, odd and
even sizes, aligned and unaligned matrices, against the oracle's permutation
(values are moved, not computed: exact)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,r,bs", [(12, 1, 2), (90, 1, 3), (124, 1, 31), (128, 1, 32), (198, 1, 33), (400, 2, 50),
                                    (318, 1, 159), (318, 1, 1), (640, 2, 160), (640, 2, 1), (644, 2, 161), (1036, 2, 7),
                                    (1028, 2, 1), (777, 0, 1), (777, 0, 111), (512, 4, 4), (1500, 1, 250)])
@pytest.mark.parametrize("shift", [0, 1])
def test_reorder_paths_match_oracle(caps, oracle_mod, cuda, n, r, bs, shift):
    import torch
    x = np.random.default_rng(n + bs).uniform(-1, 1, n * n)
    d = caps.MatDescriptor.make(n, r, bs)
    buf = [torch.full((n * n + 1,), float("nan"), dtype=torch.float64, device=cuda)[shift:shift + n * n] for _ in range(3)]
    buf[0].copy_(torch.from_numpy(x))
    caps.to_caps_layout(buf[0], buf[1], d)
    caps.from_caps_layout(buf[1], buf[2], d)
    torch.cuda.synchronize()
    assert np.array_equal(buf[1].cpu().numpy(), oracle_mod.to_caps(x, n, r, bs))
    assert torch.equal(buf[0], buf[2])
