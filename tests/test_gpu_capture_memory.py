"""A sector batch captured in a graph when the device has no room for the scaled copy of its vectors: the
graph records the kernels that need none, instead of failing at its launch."""

import numpy as np
import pytest

from ls_helpers import LAT, ls

pytestmark = pytest.mark.gpu


def test_capture_without_room_for_the_scaled_vectors():
    import torch
    n, k = 22, 16
    ops = []
    for m in range(n):
        b = ls.SpinBasis(n, n // 2, 1, ls.Symmetries(LAT.chain_symmetries(n, m)))
        b.build(exact_norms=True)
        ops.append(ls.Operator(b, LAT.xxz(LAT.chain_bonds(n), 1.0, 1.5)))
    batch = ls.SectorBatch(ops, k=k)
    assert batch.batched
    gen = torch.Generator(device="cuda").manual_seed(3)
    for s in range(batch.number_sectors):
        batch.x(s).copy_(torch.view_as_complex(torch.randn((batch.sizes[s], k, 2), generator=gen, dtype=torch.float64,
                                                           device="cuda")))
    expected = batch.run(check=True).clone()
    copy = sum(batch.sizes) * k * 16
    assert copy > 64 << 20
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room = torch.cuda.mem_get_info()[0] - copy // 2
    hold = torch.empty(room, dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < copy
        batch.Y.zero_()
        batch.capture()
        batch.replay()
        torch.cuda.synchronize()
        y = batch.Y
        batch.check_errors()
        worst = max(float((y[s] - expected[s]).abs().square().sum() / expected[s].abs().square().sum())
                    for s in range(batch.number_sectors))
    finally:
        del hold
        torch.cuda.empty_cache()
    # a row sums at most 23 products
    assert worst <= (1e-14) ** 2
