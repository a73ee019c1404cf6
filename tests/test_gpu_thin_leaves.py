"""Leaves of up to 128 rows fill half a unit of the residue GEMM; launches of
many of them run in parts, as (leaf, modulus) items: the bits of single
leaves, in no more time a leaf than a small launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 343 leaves at once against one by one; 32 stays whole units
@pytest.mark.parametrize("m", [32, 33, 64, 100, 128])
@pytest.mark.parametrize("kind", ["uniform", "wide", "int"])
def test_many_thin_leaves_match_single_ones(caps, cuda, m, kind):
    import torch
    n, r = 8 * m, 3
    rng = np.random.default_rng(m)
    a, b = rng.uniform(-1, 1, (2, n * n))
    if kind == "wide":
        a, b = a * 2.0 ** rng.integers(-20, 21, n * n), b * 2.0 ** rng.integers(-20, 21, n * n)
    if kind == "int":
        a, b = np.round(a * 1024), np.round(b * 1024)
    A, B = torch.from_numpy(a).to(cuda), torch.from_numpy(b).to(cuda)
    d = caps.MatDescriptor.make(n, r)
    lean = caps.workspace_size(d, "ddd", form="split", scheme="residues")
    out, launches = {}, {}
    for pat, limit in (("bbb", 0), ("ddd", lean)):
        out[pat] = torch.full_like(A, float("nan"))
        caps.multiply(A, B, out[pat], d, pat, form="split", scheme="residues", workspace_limit=limit)
        torch.cuda.synchronize()
        launches[pat] = caps.counters()["kernel_launches"]
    assert launches["ddd"] > 343 * 4  # one leaf a launch group
    assert torch.equal(out["bbb"], out["ddd"])


def test_many_thin_leaves_take_no_longer_each(caps, cuda):
    """GEMM time a leaf: 2401 leaves of 128 at once take 0.9 of what 49 take (the
    small launch fills its last round of SMs less), as whole units 1.2."""
    import torch
    each = {}
    caps.set_phase_timing(True)
    try:
        for r in (2, 4):
            n = 128 << r
            A = torch.rand(n * n, dtype=torch.float64, device=cuda) * 2 - 1
            C = torch.empty_like(A)
            times = []
            for _ in range(8):
                caps.multiply(A, A, C, caps.MatDescriptor.make(n, r), "b" * r, form="split", scheme="residues")
                torch.cuda.synchronize()
                times.append(caps.counters()["time_leaf_gemm"])
            each[r] = min(times[2:]) / 7 ** r
    finally:
        caps.set_phase_timing(False)
    assert each[4] < 1.05 * each[2], each
