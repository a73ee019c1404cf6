"""Matrices of 2^31 elements and more: positions take 64-bit divisions, which
blocks of 32 and more pay once per block column, not once per element."""
import pytest

pytestmark = pytest.mark.gpu

N = 46592  # 512 * 91: N^2 >= 2^31, 17.4 GB


@pytest.fixture(scope="module")
def buffers(caps, cuda):
    import torch
    if torch.cuda.mem_get_info()[0] < 120e9:
        pytest.skip("needs 120 GB of device memory")
    out = [torch.arange(N * N, dtype=torch.float64, device=cuda)]
    out += [torch.empty_like(out[0]) for _ in range(2)]
    yield out
    out.clear()
    torch.cuda.empty_cache()


def milliseconds(f):
    import torch
    f()
    times = []
    for _ in range(5):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        e[0].record()
        f()
        e[1].record()
        torch.cuda.synchronize()
        times.append(e[0].elapsed_time(e[1]))
    return min(times)


@pytest.mark.parametrize("r,bs", [(1, 128), (2, 64), (3, 32), (3, 16)])
def test_large_reorder_is_the_layout(caps, cuda, buffers, r, bs):
    import torch
    x, y, z = buffers
    d = caps.MatDescriptor.make(N, r, bs)
    caps.to_caps_layout(x, y, d)
    caps.from_caps_layout(y, z, d)
    torch.cuda.synchronize()
    assert torch.equal(x, z)
    # column-major (columns first) split into quadrant bits, blocks and entries
    nb = (N >> r) // bs
    k = r + 2
    dims = [2] * r + [nb, bs]
    order = [j for i in range(k) for j in (i, k + i)]
    z.copy_(x.reshape(dims + dims).permute(order).reshape(-1))
    assert torch.equal(y, z)


@pytest.mark.parametrize("bs", [64, 128])
def test_large_reorder_in_blocks_is_no_chain_of_divisions(caps, cuda, buffers, bs):
    """Against the same reorder in whole leaf columns, which runs at the copy
    rate: blocks of 64 take 1.4 times as long by runs and 4.0 times with
    divisions for every element; the bound lies between."""
    x, y, _ = buffers
    for move in (caps.to_caps_layout, caps.from_caps_layout):
        leaf = milliseconds(lambda: move(x, y, caps.MatDescriptor.make(N, 1)))
        assert milliseconds(lambda: move(x, y, caps.MatDescriptor.make(N, 1, bs))) < 2.5 * leaf
