"""Kernels outside the QSA path at the sizes where their work split changes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one span, the largest list of the small table, the first of the large one, the largest of that, the first of a second launch
@pytest.mark.parametrize("n", [1, 96, 97, 1200, 1201])
def test_state_copy_table_sizes(n):
    from crucible_strix_halo_b200 import layers
    gen = torch.Generator(device="cuda").manual_seed(n)
    sizes = [4 * (1 + (7 * i) % 13) for i in range(n)]
    sizes[n // 2] = 4 * 4099                                     # several pieces and a ragged last one
    spans = [torch.randint(0, 1 << 30, (s,), device="cuda", dtype=torch.int32, generator=gen) for s in sizes]
    want = torch.cat(spans)
    point = layers.SlotCheckpoint(spans)
    point.save()
    assert torch.equal(point.buffer.view(torch.int32), want)
    for s in spans:
        s.zero_()
    point.restore()
    assert torch.equal(torch.cat(spans), want)
