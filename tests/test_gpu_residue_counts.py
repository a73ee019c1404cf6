"""The residue scheme's reconstruction at every modulus count: its word counts
and constants are compiled per count, so each is run against the oracle's
128-bit model, bit for bit (the oracle rounds the exact product once, as the
kernel must: no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODULI = [181, 180, 179, 173, 169, 167, 163, 161, 157, 151, 149, 139, 137, 131, 127, 121, 113]


def expected_moduli(ta, tb, m):
    kp = (m + 15) // 16 * 16
    need = ta + tb + (kp - 1).bit_length() + 1
    prod = 1
    for L, p in enumerate(MODULI, 1):
        prod *= p
        if prod.bit_length() - 1 >= need:
            return L
    return None


def leaf(caps, cuda, A, B, **kw):
    import torch
    m = A.shape[0]
    dA = torch.from_numpy(np.ascontiguousarray(A.T).reshape(-1)).to(cuda)
    dB = torch.from_numpy(np.ascontiguousarray(B.T).reshape(-1)).to(cuda)
    dC = torch.full_like(dA, float("nan"))
    caps.leaf_gemm(dA, dB, dC, m, form="split", scheme="residues", **kw)
    torch.cuda.synchronize()
    return dC.cpu().numpy().reshape(m, m).T, caps.counters()["split_moduli"]


def model(oracle_mod, A, B, bits=55):
    m = A.shape[0]
    ref, t = oracle_mod.split_gemm_residues(A.T.copy().reshape(-1), B.T.copy().reshape(-1), m, bits)
    return ref.reshape(m, m).T, t


# the largest operand bits each count holds (the least room for |C'|): 1 .. 17 moduli
CASES = [(14, 1)] + [(130, b) for b in (2, 6, 10, 14, 17, 21, 25, 28, 32, 36, 39, 43, 46, 50, 53, 55)]
assert [expected_moduli(b, b, m) for m, b in CASES] == list(range(1, 18))


@pytest.mark.parametrize("m,bits", CASES)
def test_every_modulus_count_bitexact_vs_model(caps, oracle_mod, cuda, m, bits):
    rng = np.random.default_rng(bits)
    A = rng.uniform(-1, 1, (m, m)) * 2.0 ** rng.integers(-3, 4, (m, m))
    B = rng.uniform(-1, 1, (m, m))
    A[5] = 0.0
    # rows and columns at the largest scaled value, all of one sign: the
    # largest |C'| the modulus count has to hold
    A[7], A[8] = 1.0 - 2.0 ** -53, -1.0
    B[:, 3], B[:, 4] = 1.0 - 2.0 ** -53, 1.0
    C, L = leaf(caps, cuda, A, B, operand_bits=bits)
    ref, (ta, tb) = model(oracle_mod, A, B, bits)
    assert max(ta, tb) == bits and L == expected_moduli(ta, tb, m) == expected_moduli(bits, bits, m)
    assert np.array_equal(C, ref)
