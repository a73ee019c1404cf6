"""The residue GEMM hands out whole units in large launches and (unit, modulus)
items in launches of up to 160 units.  A 'b' step batches its leaves into one
launch and a 'd' step runs them one by one, so the same multiply goes both
ways; the products are exact and the sums the same, so the results agree bit
for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# leaves of 96 (one row tile), 130 (two row tiles, ragged), 300 (an odd third
# row tile and a second column tile): 343 leaves at once, 7 at a time, one by one
@pytest.mark.parametrize("m", [96, 130, 300])
@pytest.mark.parametrize("kind", ["uniform", "wide", "int"])
def test_whole_units_and_items_agree(caps, cuda, m, kind):
    import torch
    n, r = 8 * m, 3
    rng = np.random.default_rng(m)
    A = rng.uniform(-1, 1, n * n)
    B = rng.uniform(-1, 1, n * n)
    if kind == "wide":
        A *= 2.0 ** rng.integers(-20, 21, n * n)
        B *= 2.0 ** rng.integers(-20, 21, n * n)
    if kind == "int":
        A, B = np.round(A * 1024), np.round(B * 1024)
    dA, dB = torch.from_numpy(A).to(cuda), torch.from_numpy(B).to(cuda)
    out = {}
    for pat in ("bbb", "ddb", "ddd"):
        out[pat] = torch.full_like(dA, float("nan"))
        caps.multiply(dA, dB, out[pat], caps.MatDescriptor.make(n, r), pat, form="split", scheme="residues")
    torch.cuda.synchronize()
    assert torch.equal(out["bbb"], out["ddb"]) and torch.equal(out["bbb"], out["ddd"])


@pytest.mark.parametrize("m", [16, 128, 144, 256, 272, 400, 640])
def test_items_at_tile_edges_bitexact_vs_model(caps, oracle_mod, cuda, m):
    from test_gpu_residue_counts import leaf, model
    rng = np.random.default_rng(m)
    A, B = rng.uniform(-1, 1, (m, m)), rng.uniform(-1, 1, (m, m))
    C, _ = leaf(caps, cuda, A, B)
    assert np.array_equal(C, model(oracle_mod, A, B)[0])
