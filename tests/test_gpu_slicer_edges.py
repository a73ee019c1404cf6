"""The slicers round and cut operands without branches (residues: two limbs for
few operand bits and four otherwise): magnitudes on every side of the shifts,
ties and rounding carries, against the oracle's models, bit for bit."""
import numpy as np
import pytest

from test_gpu_residue_counts import leaf, model

pytestmark = pytest.mark.gpu


def magnitudes(m, rng):
    """Rows whose entries lie 0..90 binades below the row's largest, with ties
    (half units at the cut) and all-ones significands that carry."""
    e = np.arange(m) % 91
    x = np.ldexp(1.0, -e)[None, :] * np.where(rng.random((m, m)) < 0.5, 1.0, -1.0)
    kind = rng.integers(0, 4, (m, m))
    x = np.where(kind == 1, x * (2.0 - 2.0 ** -52), x)
    x = np.where(kind == 2, x * 1.5, x)
    x = np.where(kind == 3, x * (1.0 + 2.0 ** -52 * rng.integers(0, 2 ** 30, (m, m))), x)
    x[:, 0] = 1.0
    return x


@pytest.mark.parametrize("bits", [2, 13, 26, 27, 28, 40, 48, 52, 55])
@pytest.mark.parametrize("m", [96, 131])
def test_rounding_at_every_shift_bitexact_vs_model(caps, oracle_mod, cuda, m, bits):
    rng = np.random.default_rng(m + bits)
    A, B = magnitudes(m, rng), magnitudes(m, rng).T.copy()
    C, _ = leaf(caps, cuda, A, B, operand_bits=bits)
    assert np.array_equal(C, model(oracle_mod, A, B, bits)[0])


@pytest.mark.parametrize("scale_a,scale_b", [(2.0 ** -1060, 2.0 ** 900), (2.0 ** 900, 2.0 ** -1000),
                                             (2.0 ** -1070, 1.0)])
def test_subnormal_and_huge_operands(caps, oracle_mod, cuda, scale_a, scale_b):
    m = 64
    rng = np.random.default_rng(3)
    A, B = rng.uniform(-1, 1, (m, m)) * scale_a, rng.uniform(-1, 1, (m, m)) * scale_b
    C, _ = leaf(caps, cuda, A, B)
    assert np.array_equal(C, model(oracle_mod, A, B)[0])


@pytest.mark.parametrize("m", [96, 131])
@pytest.mark.parametrize("slices", [0, 3])
def test_digit_rounding_at_every_shift_bitexact_vs_model(caps, oracle_mod, cuda, m, slices):
    import torch
    rng = np.random.default_rng(m)
    A, B = magnitudes(m, rng), magnitudes(m, rng).T.copy()
    B[:, 1] *= 2.0 ** -1000  # with the tail of the column subnormal
    a, b = A.T.copy().reshape(-1), B.T.copy().reshape(-1)
    C = torch.full((m * m,), float("nan"), dtype=torch.float64, device=cuda)
    caps.leaf_gemm(torch.from_numpy(a).to(cuda), torch.from_numpy(b).to(cuda), C, m, form="split", scheme="digits",
                   slices=slices)
    torch.cuda.synchronize()
    cnt = caps.counters()
    assert np.array_equal(C.cpu().numpy(), oracle_mod.split_gemm(a, b, m, cnt["split_slices"], cnt["split_diagonals"]))
