"""The plain form's tile option: a fixed tile is one, not the default's pick."""
import ctypes

import pytest


def accepted(caps, opt):
    out = ctypes.c_longlong()
    return caps.lib().caps_workspace_size(caps.MatDescriptor.make(512, 1), b"b", ctypes.byref(opt), ctypes.byref(out)) == 0


def test_each_tile_is_a_value_of_its_own(caps):
    values = [caps.options(tile=t).plain_tile for t in ("default", "64x64", "32x32", "128x64")]
    assert values[0] == caps.options().plain_tile and len(set(values)) == 4
    assert all(accepted(caps, caps.options(tile=v)) for v in values)
    assert not any(accepted(caps, caps.options(tile=v)) for v in (-1, 3, 5))


@pytest.mark.gpu
@pytest.mark.parametrize("m,r", [(1, 0), (63, 0), (64, 0), (65, 0), (129, 0), (500, 0), (1030, 0),
                                 (500, 1), (77, 2), (130, 2)])
def test_fixed_tiles_and_the_default_agree(caps, cuda, m, r):
    """Single leaves (which the default runs in tiles of 16) and batches of 7 and
    49 of them (64 for 7 of 500): an entry's products add up in one order."""
    import torch
    n = m << r
    A, B = (torch.rand(n * n, dtype=torch.float64, device=cuda, generator=torch.Generator(cuda).manual_seed(i)) - 0.5
            for i in (m, m + 1))
    out = []
    for tile in ("default", "64x64", "32x32", "128x64"):
        out.append(torch.full_like(A, float("nan")))
        caps.multiply(A, B, out[-1], caps.MatDescriptor.make(n, r), "b" * r, tile=tile)
    torch.cuda.synchronize()
    assert all(torch.equal(out[0], o) for o in out[1:])


@pytest.mark.gpu
def test_64_runs_where_the_default_picks_16(caps, cuda):
    """A leaf of 1024 is 256 tiles of 64, two on the busiest of 152 SMs, or 4096
    of 16, 27 of a sixteenth the work: 1.19 times the time for tiles of 64."""
    import torch
    m = 1024
    A = torch.rand(m * m, dtype=torch.float64, device=cuda)
    C = torch.empty_like(A)
    times = {}
    for tile in ("default", "64x64"):
        for _ in range(8):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            caps.leaf_gemm(A, A, C, m, tile=tile)
            e[1].record()
            torch.cuda.synchronize()
            times[tile] = min(times.get(tile, 1e9), e[0].elapsed_time(e[1]))
    assert times["64x64"] > 1.08 * times["default"], times
