"""Small 'd' steps run as 'b' steps where the workspace budget allows it.  A
budget of exactly what the pattern needs in sequence forbids it, so the same
call runs both ways: the bits must agree, and the budget must hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["plain", "split"])
@pytest.mark.parametrize("n,r,bs,pat,hybrid", [(56, 2, 1, "dd", 1), (56, 2, 7, "dd", 1), (392, 2, 7, "bd", 1),
                                               (112, 3, 1, "hdd", 1), (112, 3, 1, "hdd", 3), (310, 1, 1, "d", 1),
                                               (1032, 3, 1, "ddd", 1), (2600, 1, 1, "d", 1), (2080, 2, 1, "bd", 1)])
def test_merged_steps_bit_identical_to_steps_in_sequence(caps, cuda, form, n, r, bs, pat, hybrid):
    import torch
    rng = np.random.default_rng(n + r)
    A = torch.from_numpy(rng.uniform(-1, 1, n * n)).to(cuda)
    B = torch.from_numpy(rng.uniform(-1, 1, n * n)).to(cuda)
    d = caps.MatDescriptor.make(n, r, bs, hybrid)
    lean = caps.workspace_size(d, pat, form=form)
    out, used = {}, {}
    for limit in (0, lean):
        out[limit] = torch.full_like(A, float("nan"))
        caps.multiply(A, B, out[limit], d, pat, form=form, workspace_limit=limit)
        torch.cuda.synchronize()
        used[limit] = caps.counters()
    assert torch.equal(out[0], out[lean])
    assert used[lean]["workspace_peak_bytes"] <= lean
    if hybrid == 1 and (form == "split" or n // 2 ** r <= 154):
        assert used[0]["kernel_launches"] < used[lean]["kernel_launches"]
    assert used[0]["additions"] == used[lean]["additions"]
    with pytest.raises(caps.CapsError) as e:
        caps.multiply(A, B, out[0], d, pat, form=form, workspace_limit=lean - 256)
    assert e.value.status == 3  # CAPS_ERR_BUDGET


@pytest.mark.parametrize("form", ["plain", "split"])
def test_host_entry_with_merged_inner_steps(caps, cuda, form):
    import torch
    n, r = 240, 3
    rng = np.random.default_rng(5)
    a, b = rng.uniform(-1, 1, n * n), rng.uniform(-1, 1, n * n)
    c = np.full(n * n, np.nan)
    d = caps.MatDescriptor.make(n, r)
    caps.multiply(a, b, c, d, "ddd", form=form)
    dC = torch.empty(n * n, dtype=torch.float64, device=cuda)
    caps.multiply(torch.from_numpy(a).to(cuda), torch.from_numpy(b).to(cuda), dC, d, "bbb", form=form)
    torch.cuda.synchronize()
    assert np.array_equal(c, dC.cpu().numpy())


def test_full_device_falls_back_to_steps_in_sequence(caps, cuda):
    """An allocation that fails for the merged steps (host-side injection) is
    tried again for the steps in sequence, where those take less."""
    import torch
    n, r = 1024, 2
    rng = np.random.default_rng(9)
    A = torch.from_numpy(rng.uniform(-1, 1, n * n)).to(cuda)
    B = torch.from_numpy(rng.uniform(-1, 1, n * n)).to(cuda)
    d = caps.MatDescriptor.make(n, r)
    want, got = torch.empty_like(A), torch.empty_like(A)
    caps.multiply(A, B, want, d, "dd", form="split")
    torch.cuda.synchronize()
    caps.release_cache()
    caps.debug_fail_allocations(1)
    try:
        caps.multiply(A, B, got, d, "dd", form="split")
        torch.cuda.synchronize()
        assert caps.counters()["workspace_peak_bytes"] <= caps.workspace_size(d, "dd", form="split")
        caps.release_cache()
        caps.debug_fail_allocations(2)
        with pytest.raises(caps.CapsError) as e:
            caps.multiply(A, B, got, d, "dd", form="split")
        assert e.value.status == 5  # CAPS_ERR_ALLOC
    finally:
        caps.debug_fail_allocations(0)
    assert torch.equal(want, got)
