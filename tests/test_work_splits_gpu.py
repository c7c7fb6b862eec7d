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


# each cut of a projection: the narrow tiles of few rows, K over clusters of 2 to 8, one and two waves of CTA pairs; rows and
# columns at and around the edges of a tile
@pytest.mark.parametrize("R,K,N", [(1, 512, 1280), (7, 4096, 2048), (8, 6144, 2560), (9, 2560, 4064), (64, 4096, 2080), (127, 2048, 12352),
                                   (129, 2048, 1312), (20, 1024, 1312), (130, 2048, 5600), (200, 2048, 12352), (257, 4096, 2048), (333, 6144, 2560), (513, 2560, 16480), (1025, 2048, 9856), (2047, 2048, 12320)])
def test_projection_cuts(R, K, N):
    from crucible_strix_halo_b200 import capi, layers
    gen = torch.Generator(device="cuda").manual_seed(R + N)
    x = torch.randn(R, K, device="cuda", generator=gen).bfloat16()
    w = (torch.randn(N, K, device="cuda", generator=gen) / K ** 0.5).bfloat16()
    outs = [torch.full((R, c), float("nan"), device="cuda") for c in (N - 96, 96)]
    layers.proj_gemm(x, w, outs)
    assert capi.lib.cr_device_check() == 0
    ref = x.float() @ w.float().t()
    assert (torch.cat(outs, 1) - ref).abs().max().item() < 2e-4          # order of the fp32 additions only
