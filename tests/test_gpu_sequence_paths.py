"""Steps in sequence against steps in one batch.  Without a workspace limit
small 'd' steps run as 'b' steps; the size of the sequence as the limit keeps
them apart, so the same multiply goes through single-leaf launches ((leaf,
modulus) items) and through one large launch (whole units): bit for bit."""
import numpy as np
import pytest

from test_gpu_residue_counts import CASES, expected_moduli

pytestmark = pytest.mark.gpu


def both_ways(caps, cuda, n, r, pat, data, **kw):
    """(C, counters) of `pat` in sequence and of 'b' steps throughout."""
    import torch
    A, B = (torch.from_numpy(x).to(cuda) for x in data)
    d = caps.MatDescriptor.make(n, r)
    out = []
    for p, limit in ((pat, caps.workspace_size(d, pat, form="split", scheme="residues")), ("b" * r, 0)):
        C = torch.full_like(A, float("nan"))
        caps.multiply(A, B, C, d, p, form="split", scheme="residues", workspace_limit=limit, **kw)
        torch.cuda.synchronize()
        out.append((C, caps.counters()))
    return out


@pytest.mark.parametrize("m,bits", CASES)
def test_whole_units_match_items_at_every_modulus_count(caps, cuda, m, bits):
    n, r = 8 * m, 3
    data = np.random.default_rng(bits).uniform(-1, 1, (2, n * n))
    (c, one), (b, all_) = both_ways(caps, cuda, n, r, "ddd", data, operand_bits=bits)
    # (the last leaf alone may need fewer bits than the cap, and a modulus less)
    assert one["split_moduli"] <= all_["split_moduli"] == expected_moduli(bits, bits, m)
    assert one["kernel_launches"] > 343 * 4 > all_["kernel_launches"]  # 343 launch groups, and one
    assert (c == b).all()


@pytest.mark.parametrize("m", [130, 300])
@pytest.mark.parametrize("kind", ["uniform", "wide", "int"])
@pytest.mark.parametrize("pat", ["ddd", "ddb"])
def test_whole_units_match_items(caps, cuda, m, kind, pat):
    n, r = 8 * m, 3
    rng = np.random.default_rng(m)
    data = rng.uniform(-1, 1, (2, n * n))
    if kind == "wide":
        data *= 2.0 ** rng.integers(-20, 21, (2, n * n))
    if kind == "int":
        data = np.round(data * 1024)
    (c, one), (b, all_) = both_ways(caps, cuda, n, r, pat, data)
    assert one["kernel_launches"] > (343 if pat == "ddd" else 49) * 4 > all_["kernel_launches"]
    assert (c == b).all()


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("n,r,pat", [(512, 1, "d"), (896, 2, "dd"), (1024, 2, "bd"), (1024, 2, "db"), (2048, 2, "dd")])
def test_steps_in_sequence_match_b_steps(caps, cuda, n, r, pat, wide):
    rng = np.random.default_rng(7 * n + r)
    data = rng.uniform(-1, 1, (2, n * n))
    if wide:
        data *= 2.0 ** rng.integers(-20, 21, (2, n * n))
    (c, seq), (b, batch) = both_ways(caps, cuda, n, r, pat, data)
    assert seq["split_moduli"] > 0 and seq["kernel_launches"] > batch["kernel_launches"]
    assert (c == b).all()
