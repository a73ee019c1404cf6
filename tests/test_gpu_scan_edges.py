"""The split form's exponent scan cuts a leaf into units by its size and the
number of leaves; the unit that ends a leaf side sets the counts.  Integer
data whose bits come from a single entry anywhere in the leaf make any entry
the scan misses or counts twice show: the moduli, and the exact product."""
import numpy as np
import pytest

from test_gpu_residue_counts import expected_moduli, leaf, model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 15, 31, 33, 64, 127, 257, 510, 513, 1025])
def test_scan_finds_the_widest_entry_wherever_it_is(caps, oracle_mod, cuda, m):
    rng = np.random.default_rng(m)
    for i, k in {(0, 0), (m - 1, m - 1), (0, m - 1), (m // 2, m // 3)}:
        A = rng.integers(-1, 2, (m, m)).astype(np.float64)
        B = rng.integers(-1, 2, (m, m)).astype(np.float64)
        A[i, k] = 2.0 ** 20 + 1
        B[k, i] = -(2.0 ** 18) - 1
        C, L = leaf(caps, cuda, A, B)
        ref, (ta, tb) = model(oracle_mod, A, B)
        assert ta >= 21 and tb >= 19 and L == expected_moduli(ta, tb, m)
        assert np.array_equal(C, ref)
        assert np.array_equal(C, (A.astype(np.int64) @ B.astype(np.int64)).astype(np.float64))


def test_several_leaves_of_one_group_each_scanned(caps, cuda):
    """A batched group: the widest entry sits in another leaf each time, and
    every product stays exact (the operand bits are the group's)."""
    import torch
    n, count = 96, 5
    rng = np.random.default_rng(4)
    for wide in range(count):
        A = rng.integers(-3, 4, (count, n, n)).astype(np.float64)
        B = rng.integers(-3, 4, (count, n, n)).astype(np.float64)
        A[wide, 95, 17] = 2.0 ** 22 + 1
        As = [torch.from_numpy(x.T.copy().reshape(-1)).to(cuda) for x in A]
        Bs = [torch.from_numpy(x.T.copy().reshape(-1)).to(cuda) for x in B]
        Cs = [torch.full((n * n,), float("nan"), dtype=torch.float64, device=cuda) for _ in A]
        caps.multiply_batched(As, Bs, Cs, [n] * count, form="split")
        for a, b, c in zip(A, B, Cs):
            got = c.cpu().numpy().reshape(n, n).T
            assert np.array_equal(got, (a.astype(np.int64) @ b.astype(np.int64)).astype(np.float64))
