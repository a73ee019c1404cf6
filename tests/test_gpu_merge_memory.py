"""Without a workspace limit, small 'd' steps run as 'b' steps only as far as that
takes a small part of the free device memory, and never by allocating under a
stream capture; a caller who shares the GPU keeps the memory that the pattern
leaves (caps_workspace_size is what the steps in sequence take)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def operands(n, cuda):
    import torch
    rng = np.random.default_rng(n)
    return [torch.from_numpy(rng.uniform(-1, 1, n * n)).to(cuda) for _ in range(2)]


def test_merged_steps_leave_a_shared_device_its_memory(caps, cuda):
    import torch
    n, pat = 4096, "dd"
    A, B = operands(n, cuda)
    d = caps.MatDescriptor.make(n, 2)
    lean = caps.workspace_size(d, pat, form="split")
    out, peak = [], []
    caps.release_cache()
    torch.cuda.empty_cache()
    rest = 24 << 30
    if torch.cuda.mem_get_info()[0] < rest + (100 << 30):
        pytest.skip("needs an otherwise empty device")
    for share in (True, False):
        held = torch.empty(torch.cuda.mem_get_info()[0] - rest, dtype=torch.uint8, device=cuda) if share else None
        C = torch.full_like(A, float("nan"))
        caps.multiply(A, B, C, d, pat, form="split")
        torch.cuda.synchronize()
        out.append(C)
        peak.append(caps.counters()["workspace_peak_bytes"])
        del held
        torch.cuda.empty_cache()
        caps.release_cache()
    assert peak[0] == lean  # merged it would take 4.7 GB, more than 24 GB / 16
    assert peak[1] > lean   # with the device to itself
    assert torch.equal(out[0], out[1])


def test_capture_takes_the_workspace_there_is(caps, cuda):
    """A workspace that holds the steps in sequence is enough under a capture,
    which cannot allocate more for merged ones."""
    import torch
    n, pat = 56, "dd"
    A, B = operands(n, cuda)
    d = caps.MatDescriptor.make(n, 2)
    want, got = torch.empty_like(A), torch.full_like(A, float("nan"))
    caps.release_cache()
    caps.multiply(A, B, want, d, pat, workspace_limit=caps.workspace_size(d, pat))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        caps.multiply(A, B, got, d, pat)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(want, got)
