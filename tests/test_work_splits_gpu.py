"""Kernels outside the QSA path at the sizes where their work split changes."""
import ctypes as C

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


# chunked scan against the serial one: a single ragged chunk, rows fewer than the ring holds, both sides of the size where a
# CTA takes one value head (296 / value heads chunks), one to three value heads per key head
@pytest.mark.parametrize("geometry", [(16, 32), (16, 48), (4, 4)])
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("R", [1, 17, 63, 64, 385, 576, 577])
def test_gdn_chunk_prefill_splits(geometry, bf16, R):
    from crucible_strix_halo_b200 import capi, layers
    g = capi.Geometry(256, 16, 2, geometry[1], geometry[0])
    gen = torch.Generator(device="cuda").manual_seed(R)
    rn = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=gen) * std
    C, Hv, pos0 = g.gdn_channels, g.gdn_vheads, 100
    dt = torch.bfloat16 if bf16 else torch.float32
    w = layers.GdnWeights(g, rn(C, 4, std=0.5), rn(Hv) - 1, rn(Hv, std=0.5), 1 + rn(128, std=0.1))
    qkv, z, ab = rn(R, C).to(dt), rn(R, Hv * 128).to(dt), rn(R, 2 * Hv).to(dt)
    hist = rn(16, C).bfloat16().float()
    state = rn(Hv * 16384 + 64, std=0.1)
    got = []
    for algo in (capi.GDN_SERIAL_F32, capi.GDN_CHUNK_TC):
        s = layers.GdnSession(g)
        s.hist.copy_(hist)
        s.state.copy_(state)
        plan = layers.GdnPrefillPlan(w, R, in_dtype=capi.IN_BF16 if bf16 else capi.IN_F32)
        got.append((plan.run(s, qkv, z, ab, pos0, algo).clone(), s.state_view().clone(), s.hist.clone()))
    assert capi.lib.cr_device_check() == 0
    (o0, s0, h0), (o1, s1, h1) = got
    ring = hist.clone()
    for r in range(max(0, R - 16), R):
        ring[(pos0 + r) % 16] = qkv[r].float()
    assert torch.equal(h0, ring) and torch.equal(h1, ring)
    assert (o1 - o0).abs().max() < 4e-3 * o0.abs().max() and (s1 - s0).abs().max() < 4e-3 * s0.abs().max()


# Calls of a few rows run through the step's recurrence, 14 to 26 rows in two launches: the serial fp32 scan over the same rows differs
# by the order of fp32 additions only (128 terms, 26 rows: a few 1e-6), which the output format then rounds.  Positions without a
# full halo, every row format, the packed layout, states off the 16-byte boundary (which take the chunked scan, tf32).
@pytest.mark.parametrize("heads", [(16, 32), (16, 48), (4, 4)])
@pytest.mark.parametrize("R,pos0", [(1, 0), (1, 3), (2, 1), (4, 100), (12, 5), (13, 2), (14, 0), (17, 100), (25, 1), (26, 77), (27, 9)])
@pytest.mark.parametrize("bf16,fmt,offset", [(False, "f32", 0), (True, "bf16", 0), (True, "exl3", 0), (False, "packed", 0), (False, "f32", 1)])
def test_gdn_prefill_of_few_rows(heads, R, pos0, bf16, fmt, offset):
    from crucible_strix_halo_b200 import capi, layers
    g = capi.Geometry(256, 16, 2, heads[1], heads[0])
    gen = torch.Generator(device="cuda").manual_seed(100 * R + pos0)
    rn = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=gen) * std
    width, Hv = g.gdn_channels, g.gdn_vheads
    dt = torch.bfloat16 if bf16 else torch.float32
    w = layers.GdnWeights(g, rn(width, 4, std=0.5), rn(Hv) - 1, rn(Hv, std=0.5), 1 + rn(128, std=0.1), suh=1 + rn(Hv * 128, std=0.1))
    qkv, z, ab = rn(R, width).to(dt), rn(R, Hv * 128).to(dt), rn(R, 2 * Hv).to(dt)
    hist, state = rn(16, width).bfloat16().float(), rn(Hv * 16384, std=0.1)
    code = {"f32": capi.OUT_RAW_F32, "bf16": capi.OUT_RAW_BF16}.get(fmt, capi.OUT_EXL3_WHT)
    got = []
    for algo in (capi.GDN_SERIAL_F32, capi.GDN_CHUNK_TC):
        s = layers.GdnSession(g)
        s.state = torch.zeros(s.state.numel() + 4, device="cuda")[offset:offset + s.state.numel()]
        s.state[:Hv * 16384] = state
        s.hist.copy_(hist)
        plan = layers.GdnPrefillPlan(w, max(R, 27), in_dtype=capi.IN_BF16 if bf16 else capi.IN_F32, fmt=code)
        out = torch.zeros((R + 5) * Hv * 128, device="cuda", dtype=plan.out.dtype) if fmt == "packed" else plan.out
        d = capi.dptr
        args = capi.GdnPrefillArgs(capi.GdnArgs(d(qkv), d(z), None, None, d(w.conv), d(w.A_log), d(w.dt_bias), d(w.gamma), d(s.hist), d(s.state), d(w.suh), d(out),
                                                None, pos0, R, 0, R, R + 5 if fmt == "packed" else 0, 3 if fmt == "packed" else 0),
                                   d(ab), plan.in_dtype, d(plan.workspace), plan.workspace.numel(), None)
        capi.check(capi.lib.cr_gdn_prefill(C.byref(g), C.byref(args), algo, code, None))
        got.append(((out if fmt == "packed" else plan.out[:R]).float().clone(), s.state[:Hv * 16384].clone(), s.hist.clone()))
    assert capi.lib.cr_device_check() == 0
    (o0, s0, h0), (o1, s1, h1) = got
    ring = hist.clone()
    for r in range(max(0, R - 16), R):
        ring[(pos0 + r) % 16] = qkv[r].float()
    assert torch.equal(h0, ring) and torch.equal(h1, ring)
    chunked = R > 26 or offset
    tol = 4e-3 if chunked else 2e-5
    assert (s1 - s0).abs().max() < tol * s0.abs().max()
    step = {"f32": 0.0, "bf16": 2.0 ** -8}.get(fmt, 3e-3)                  # one step of the format (fp16 is rounded twice before its transform)
    assert (o1 - o0).abs().max() < (tol + step) * o0.abs().max()


# The un-gated readout is an output like the others: asking for it changes neither the route of a call nor a bit of its results.
@pytest.mark.parametrize("R", [1, 13, 14, 26, 27])
@pytest.mark.parametrize("bf16", [False, True])
def test_raw_readout_changes_nothing_else(R, bf16):
    from crucible_strix_halo_b200 import capi, layers
    g = capi.Geometry(256, 16, 2, 32, 16)
    gen = torch.Generator(device="cuda").manual_seed(R)
    rn = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=gen) * std
    width, Hv = g.gdn_channels, g.gdn_vheads
    dt = torch.bfloat16 if bf16 else torch.float32
    w = layers.GdnWeights(g, rn(width, 4, std=0.5), rn(Hv) - 1, rn(Hv, std=0.5), 1 + rn(128, std=0.1))
    qkv, z, ab = rn(R, width).to(dt), rn(R, Hv * 128).to(dt), rn(R, 2 * Hv).to(dt)
    hist, state = rn(16, width), rn(Hv * 16384, std=0.1)
    got = []
    for algo, raw in ((capi.GDN_CHUNK_TC, False), (capi.GDN_CHUNK_TC, True), (capi.GDN_SERIAL_F32, True)):
        s = layers.GdnSession(g)
        s.state[:Hv * 16384] = state
        s.hist.copy_(hist)
        plan = layers.GdnPrefillPlan(w, R, in_dtype=capi.IN_BF16 if bf16 else capi.IN_F32, raw_y=raw)
        if raw:
            plan.raw_y.fill_(float("nan"))
        out = plan.run(s, qkv, z, ab, 1000, algo).clone()
        got.append((out, s.state.clone(), s.hist.clone(), plan.raw_y))
    for x, y in zip(got[0][:3], got[1][:3]):
        assert torch.equal(x, y)
    y, want = got[1][3], got[2][3]
    assert (y - want).abs().max() < (4e-3 if R > 26 else 2e-5) * want.abs().max()


# Calls in a row on one plan, with nothing between them: every call writes its operands where the one before had its own, and its
# scan must not take those for new.  The workspace of the first call holds marks that say everything is written.  Rows: a CTA
# with a unit for one half, units for both, several per half; more chunks than the scan's loader looks at in one go (32).
@pytest.mark.parametrize("geometry", [(16, 32), (16, 48)])
@pytest.mark.parametrize("R", [64, 577, 1999, 2113])
def test_gdn_prefill_calls_share_a_workspace(geometry, R):
    from crucible_strix_halo_b200 import capi, layers
    g = capi.Geometry(256, 16, 2, geometry[1], geometry[0])
    gen = torch.Generator(device="cuda").manual_seed(R)
    rn = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=gen) * std
    C, Hv = g.gdn_channels, g.gdn_vheads
    w = layers.GdnWeights(g, rn(C, 4, std=0.5), rn(Hv) - 1, rn(Hv, std=0.5), 1 + rn(128, std=0.1))
    inputs = [(rn(R, C), rn(R, Hv * 128), rn(R, 2 * Hv)) for _ in range(2)]
    state = [rn(Hv * 16384 + 64, std=0.1) for _ in range(2)]

    def session(i):
        s = layers.GdnSession(g)
        s.state.copy_(state[i])
        return s

    serial = layers.GdnPrefillPlan(w, R)
    want = []
    for i in range(2):
        s = session(i)
        want.append((serial.run(s, *inputs[i], 0, capi.GDN_SERIAL_F32).clone(), s.state_view()))
    plan = layers.GdnPrefillPlan(w, R)
    plan.workspace.fill_(0xFF)                                   # marks set, operands NaN
    got = [session(k & 1) for k in range(12)]
    torch.cuda.synchronize()
    for k, s in enumerate(got):
        out = plan.run(s, *inputs[k & 1], 0, capi.GDN_CHUNK_TC)
    assert capi.lib.cr_device_check() == 0
    out1, _ = want[1]
    assert (out - out1).abs().max() < 4e-3 * out1.abs().max()    # the last call had the second inputs
    for k, s in enumerate(got):
        ref = want[k & 1][1]
        assert (s.state_view() - ref).abs().max() < 4e-3 * ref.abs().max(), k


# The raw-row ring at an address that is a multiple of 4 bytes only: what a call reads of it (the three rows before the call) and
# what it writes are the same as with an aligned ring, bit for bit.
@pytest.mark.parametrize("algo", ["serial", "chunk"])
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("offset", [1, 2, 3])
def test_gdn_prefill_ring_at_any_float_address(algo, bf16, offset):
    from crucible_strix_halo_b200 import capi, layers
    g = capi.Geometry(256, 16, 2, 4, 2)
    gen = torch.Generator(device="cuda").manual_seed(offset)
    rn = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=gen) * std
    C, Hv, R, pos0 = g.gdn_channels, 4, 21, 5
    dt = torch.bfloat16 if bf16 else torch.float32
    w = layers.GdnWeights(g, rn(C, 4, std=0.5), rn(Hv) - 1, rn(Hv, std=0.5), 1 + rn(128, std=0.1))
    qkv, z, ab, hist = rn(R, C).to(dt), rn(R, Hv * 128).to(dt), rn(R, 2 * Hv).to(dt), rn(16, C).bfloat16().float()
    plan = layers.GdnPrefillPlan(w, R, in_dtype=capi.IN_BF16 if bf16 else capi.IN_F32)
    got = []
    for shift in (0, offset):
        s = layers.GdnSession(g)
        room = torch.zeros(16 * C + 4, device="cuda")
        s.hist = room[shift:shift + 16 * C].view(16, C)
        s.hist.copy_(hist)
        out = plan.run(s, qkv, z, ab, pos0, capi.GDN_SERIAL_F32 if algo == "serial" else capi.GDN_CHUNK_TC)
        got.append((out.clone(), s.state.clone(), s.hist.clone(), room[:shift].sum() + room[shift + 16 * C:].sum()))
    assert all(torch.equal(a, b) for a, b in zip(*got)) and got[1][3] == 0


# A GDN step alone and beside 1 to 5 other sessions: its heads run as clusters of four, of two (2 sessions x 32 heads; 48 heads),
# as single CTAs with an SM each and two to an SM, and give the same bits.  Rows and replayed rows from the fewest to the most,
# more replayed rows than are staged at once, rows that are recorded where replayed ones lay.
@pytest.mark.parametrize("heads", [32, 48])
@pytest.mark.parametrize("R,replay,commit", [(1, 0, 1), (4, 2, 1), (9, 8, 1), (13, 17, 5), (13, 0, 13)])
@pytest.mark.parametrize("fmt", [0, 1, 2])
def test_gdn_step_clusters(heads, R, replay, commit, fmt):
    from crucible_strix_halo_b200 import capi, layers
    g = capi.Geometry(512, 16, 2, heads, 16)
    gen = torch.Generator(device="cuda").manual_seed(R)
    rn = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=gen) * std
    C, W = g.gdn_channels, heads * 128
    w = layers.GdnWeights(g, rn(C, 4, std=0.5), rn(heads) - 1, rn(heads, std=0.5), 1 + rn(128, std=0.1), ab=rn(2 * heads, 512, std=0.05), suh=1 + rn(W, std=0.1))
    rows = [(rn(R, C), rn(R, W), rn(R, 512)) for _ in range(6)]
    begin = [(rn(heads * 16384 + 64, std=0.1), rn(16, C), torch.cat([rn(heads, 20, 256, std=0.2), torch.rand(heads, 20, 2, device="cuda", generator=gen)], 2)) for _ in range(6)]

    def span(i):
        s = layers.GdnSession(g, pend_rows=20)
        for to, x in zip((s.state, s.hist, s.pend), begin[i]):
            to.copy_(x)
        qkv, z, x = rows[i]
        return dict(session=s, qkv=qkv, z=z, x=x, pos0=7, replay=replay, commit=commit)

    def results(spans, outs):
        s = spans[0]["session"]
        return outs[0], s.state, s.hist, s.pend

    alone = [span(0)]
    want = results(alone, layers.gdn_step(w, alone, fmt))
    assert torch.isfinite(want[0].float()).all() and torch.isfinite(want[1]).all()
    for n in (2, 3, 4, 6):
        spans = [span(i) for i in range(n)]
        assert all(torch.equal(a, b) for a, b in zip(want, results(spans, layers.gdn_step(w, spans, fmt)))), n


# Stage timing keeps a call on one stream but times the form of the chunk-local kernel that the call runs without it: units on CTAs
# of their own in a call of several parts, two units to a CTA in a call of one.
@pytest.mark.parametrize("R,form", [(2500, "gdn_chunk_local_kernel"), (1500, "gdn_chunk_local_kernel<2>")])
def test_gdn_stage_timing_times_the_live_form(R, form):
    from crucible_strix_halo_b200 import capi, layers
    g = capi.Geometry(256, 16, 2, 32, 16)
    gen = torch.Generator(device="cuda").manual_seed(R)
    rn = lambda *s, std=1.0: torch.randn(*s, device="cuda", generator=gen) * std
    w = layers.GdnWeights(g, rn(g.gdn_channels, 4, std=0.5), rn(32) - 1, rn(32, std=0.5), 1 + rn(128, std=0.1))
    inputs = rn(R, g.gdn_channels), rn(R, 4096), rn(R, 64)
    old = capi.set_options(gdn_part_chunks=32)
    try:
        outs = []
        for timing in (0, 1):
            capi.check(capi.lib.cr_profile_enable(timing))
            plan = layers.GdnPrefillPlan(w, R)
            outs.append(plan.run(layers.GdnSession(g), *inputs, 0, capi.GDN_CHUNK_TC))
        names = capi.profile_collect()
    finally:
        capi.check(capi.lib.cr_profile_enable(0))
        capi.set_options(gdn_part_chunks=old.gdn_part_chunks)
    assert [n for n in names if "local" in n] == [form] and torch.equal(*outs)
