"""QSA kernels at the sizes where their work split changes: stream counts, clusters and head groups of the attention,
bitmap windows of the union lists.  References: plain torch in float64 / a dictionary merge."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _weights(Hq):
    from crucible_strix_halo_b200 import capi, layers
    g = capi.Geometry(256, Hq, 2, 4, 2)
    one = [torch.ones(n) for n in (256, 256, 128, 128)]
    return capi, layers, g, layers.QsaWeights(g, *one)


def _selection(gen, pos):
    """(sel, nsel) of the row at position pos: 512 of its complete blocks, or dense."""
    nb = (pos + 1) // 4
    if nb <= 512:
        return torch.zeros(512, dtype=torch.int32, device="cuda"), -1
    return torch.randperm(nb, generator=gen, device="cuda")[:512].sort().values.int(), 512


def _attend(q, k, v, sel, nsel, pos):
    """Gated attention of one row, float64: q [Hq, 512], k / v fp16 [ctx, 2, 256]."""
    nb = (pos + 1) // 4
    if nsel < 0:
        at = torch.arange(pos + 1, device="cuda")
    else:
        at = torch.cat([(sel.long()[:, None] * 4 + torch.arange(4, device="cuda")).reshape(-1), torch.arange(4 * nb, pos + 1, device="cuda")])
    gqa = q.shape[0] // 2
    out = []
    for g in range(2):
        Q = q[g * gqa:(g + 1) * gqa].double()
        p = torch.softmax(Q[:, :256] @ k[at, g].double().T / 16, dim=1)
        out.append((p @ v[at, g].double()) * torch.sigmoid(Q[:, 256:]))
    return torch.cat(out)


# units = sessions x rows x 2 KV heads; 8 streams a CTA (16 heads) or 6 (18 and 24 heads): one position, fewer tiles than
# streams, clusters of 8 / 4 / 2, one CTA per unit, several units per CTA, ragged last CTA
@pytest.mark.parametrize("Hq,sessions,rows,ctx", [(16, 1, 1, 1), (16, 1, 1, 37), (16, 1, 1, 1501), (16, 1, 2, 2052), (16, 4, 1, 9003), (16, 7, 2, 2600),
                                                   (16, 8, 9, 3001), (16, 17, 13, 2301), (24, 1, 4, 2051), (24, 3, 1, 700), (18, 5, 5, 2301), (24, 9, 13, 2301), (16, 8, 1, 9003), (24, 2, 4, 9003), (16, 15, 1, 9003), (24, 9, 2, 9003), (16, 18, 1, 9003)])
def test_attention_work_splits(Hq, sessions, rows, ctx):
    capi, layers, g, w = _weights(Hq)
    gen = torch.Generator(device="cuda").manual_seed(ctx + Hq)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    spans, outs, arr = [], [], (capi.QsaArgs * sessions)()
    zero = torch.zeros(rows, 640, device="cuda")
    for i in range(sessions):
        pos0 = ctx - rows - (i % 3 if ctx > rows + 3 else 0)      # tails of different lengths
        s = layers.QsaSession(g, ctx, max_rows=rows)
        s.k.copy_(rn(ctx, 2, 256)); s.v.copy_(rn(ctx, 2, 256))
        for r in range(rows):
            s.sel[r], n = _selection(gen, pos0 + r)
            s.nsel[r] = n
        q = rn(rows, Hq, 512)
        q[:, :, :256] *= 2.0
        outs.append(torch.full((rows, Hq * 256), 7.0, device="cuda"))
        spans.append((s, q, pos0))
        arr[i] = layers.qsa_args(w, s, q, zero, zero, zero, outs[i], pos0)
    scratch = torch.empty(capi.lib.cr_qsa_scratch_bytes(C.byref(g), sessions * rows), device="cuda", dtype=torch.uint8)
    capi.check(capi.lib.cr_qsa_attn(C.byref(g), arr, sessions, capi.dptr(scratch), scratch.numel(), capi.OUT_RAW_F32, None))
    torch.cuda.synchronize()
    for i, (s, q, pos0) in enumerate(spans):
        for r in range(rows):
            ref = _attend(q[r], s.k, s.v, s.sel[r], int(s.nsel[r]), pos0 + r)
            err = (outs[i][r].view(Hq, 256).double() - ref).abs().max().item()
            assert err < 2e-5, "session %d row %d: %g" % (i, r, err)


@pytest.mark.parametrize("pos0,R", [(4 * 262144 - 9, 20), (4 * 524288 + 3, 33)])
def test_union_lists_past_one_bitmap_window(pos0, R):
    capi, layers, g, w = _weights(16)
    rng = np.random.default_rng(pos0)
    ses = layers.QsaSession(g, 64, max_rows=R)
    common = rng.choice((pos0 + 1) // 4, 300, replace=False)
    sel = np.empty((R, 512), np.int32)
    for r in range(R):
        own = rng.choice((pos0 + 1) // 4, 700, replace=False)
        sel[r] = np.sort(np.concatenate([common, np.setdiff1d(own, common)[:212]]))
    ses.sel.copy_(torch.from_numpy(sel)); ses.nsel.fill_(512)
    z = torch.zeros(R, 16, 512, device="cuda")
    args = layers.qsa_args(w, ses, z, z, z, z, z, pos0)
    args.sstride = (pos0 + R) // 4                               # nothing reads the scores or the cache here
    ints, RT = capi.lib.cr_qsa_union_list_ints(C.byref(g), R), 16
    tiles = (R + RT - 1) // RT
    lst, cnt = torch.zeros(ints, dtype=torch.int32, device="cuda"), torch.zeros(tiles, dtype=torch.int32, device="cuda")
    u = capi.QsaUnion(lst.data_ptr(), cnt.data_ptr())
    capi.check(capi.lib.cr_qsa_union_build(C.byref(g), (capi.QsaArgs * 1)(args), C.byref(u), None))
    got = lst.cpu().numpy().reshape(tiles, -1, 2)
    for t in range(tiles):
        want = {}
        for r in range(t * RT, min(R, (t + 1) * RT)):
            blocks = list(sel[r]) + ([(pos0 + r + 1) // 4] if (pos0 + r + 1) % 4 else [])
            for b in blocks:
                want[int(b)] = want.get(int(b), 0) | 1 << (r - t * RT)
        np.testing.assert_array_equal(got[t, :int(cnt[t])], np.array(sorted(want.items()), np.int32))


# histogram levels of the selection: everything in one bin, crowded bins that are divided, many equal keys around the
# threshold, an outlier that leaves the window below the largest key empty; rows read four elements at a time and singly
@pytest.mark.parametrize("nb", [600, 4096, 4097, 9001, 20000])
@pytest.mark.parametrize("pattern", ["close", "steps", "outlier", "zeros", "ramp"])
def test_selection_threshold_patterns(nb, pattern):
    capi, layers, g, w = _weights(16)
    gen = torch.Generator(device="cuda").manual_seed(nb)
    u = torch.rand(3, nb, device="cuda", generator=gen)
    sc = {"close": 1.0 + u * 1e-5, "steps": (u * 7).floor() / 7, "outlier": u * 1e-6, "zeros": torch.where(u < 0.95, torch.zeros_like(u), u),
          "ramp": torch.arange(nb, device="cuda").expand(3, nb) * 1e-3}[pattern]
    if pattern == "outlier":
        sc[:, 5] = 3e4
    for pad in (0, 1, 4):                                            # sstride a multiple of four or not
        s = layers.QsaSession(g, 4 * nb + 8, max_rows=3)
        s.sstride = nb + pad
        s.scores = torch.zeros(3, s.sstride, device="cuda")
        s.scores[:, :nb] = sc
        z = torch.zeros(3, 16, 512, device="cuda")
        args = layers.qsa_args(w, s, z, z, z, z, z, 4 * nb - 1)
        cs, ci = torch.empty(3, 512, device="cuda"), torch.empty(3, 512, device="cuda", dtype=torch.int32)
        capi.check(capi.lib.cr_qsa_shard_candidates(C.byref(g), C.byref(args), 0, nb, capi.dptr(cs), capi.dptr(ci), None))
        for r in range(3):
            v = sc[r].double().cpu().numpy()
            want = np.sort(np.lexsort((np.arange(nb), -v))[:512])
            np.testing.assert_array_equal(ci[r].cpu().numpy(), want)
            np.testing.assert_array_equal(cs[r].cpu().numpy(), sc[r].cpu().numpy()[want])


# more rows than the chip holds at 1,024 threads each: 256 threads a row up to 14,336 blocks, 512 above; a full list, lists that
# overflow (few distinct scores, mostly zeros), rows read four elements at a time and singly
@pytest.mark.parametrize("last_nb", [700, 3072, 3073, 14336, 14337, 17000])
@pytest.mark.parametrize("pattern,pad", [("random", 0), ("random", 1), ("seven", 0), ("zeros", 3)])
def test_selection_of_many_rows(last_nb, pattern, pad):
    capi, layers, g, w = _weights(16)
    R = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 9
    gen = torch.Generator(device="cuda").manual_seed(last_nb)
    pos0 = 4 * last_nb - R
    s = layers.QsaSession(g, pos0 + R, max_rows=R)
    s.sstride = last_nb + pad
    s.scores = torch.zeros(R, s.sstride, device="cuda")
    tiles = torch.randn(s.ik_pool.numel() // 4096, 128, 32, device="cuda", generator=gen)
    if pattern == "seven":
        tiles = tiles[:1, :, :7].repeat(tiles.shape[0], 1, 5)[:, :, :32].contiguous()
    if pattern == "zeros":
        tiles *= (torch.rand(tiles.shape[0], 1, 32, device="cuda", generator=gen) < 300 / last_nb)
    s.ik_pool.copy_(tiles.flatten())
    idx = torch.randn(R, 640, device="cuda", generator=gen)
    z = torch.zeros(R, 16, 512, device="cuda")
    args = layers.qsa_args(w, s, z, z, z, idx, z, pos0)
    capi.check(capi.lib.cr_qsa_select(C.byref(g), C.byref(args), 1, None, 0, None))
    sc, sel, nsel = s.scores.cpu().numpy(), s.sel.cpu().numpy(), s.nsel.cpu().numpy()
    for r in range(0, R, 3):
        nb = (pos0 + r + 1) // 4
        if nb <= capi.SEL_BLOCKS:
            assert nsel[r] == -1
            continue
        assert nsel[r] == 512
        want = np.sort(np.lexsort((np.arange(nb), -sc[r, :nb].astype(np.float64)))[:512])
        np.testing.assert_array_equal(sel[r], want)


# many rows of equal scores past 196,608 blocks: the bitmap of the ties runs past the short list over the histogram's place and ends where the
# selection's own begins
@pytest.mark.parametrize("last_nb", [196608, 200003, 262144])
def test_selection_of_many_long_rows_of_ties(last_nb):
    capi, layers, g, w = _weights(16)
    R = 2 * torch.cuda.get_device_properties(0).multi_processor_count + 9
    gen = torch.Generator(device="cuda").manual_seed(last_nb)
    s = layers.QsaSession(g, 64, max_rows=R)                            # no cache row is written
    s.ik_pool = torch.zeros((last_nb + 31) // 32, 128, 32, device="cuda")
    some = torch.randperm(last_nb, device="cuda", generator=gen)[:300]
    s.ik_pool[some // 32, :, some % 32] = torch.randn(300, 128, device="cuda", generator=gen)
    s.ik_pool = s.ik_pool.flatten()
    s.sstride = last_nb
    s.scores = torch.zeros(R, s.sstride, device="cuda")
    idx, z = torch.randn(R, 640, device="cuda", generator=gen), torch.zeros(R, 16, 512, device="cuda")
    pos0 = 4 * last_nb - R
    args = layers.qsa_args(w, s, z, z, z, idx, z, pos0)
    capi.check(capi.lib.cr_qsa_select(C.byref(g), C.byref(args), 1, None, 0, None))
    for r in range(0, R, 38):
        nb = (pos0 + r + 1) // 4
        v = s.scores[r, :nb].cpu().numpy()
        assert (v > 0).sum() < 512 and int(s.nsel[r]) == 512
        best = np.nonzero(v > 0)[0]
        want = np.sort(np.concatenate([best, np.nonzero(v == 0)[0][:512 - len(best)]]))
        np.testing.assert_array_equal(s.sel[r].cpu().numpy(), want)


# a rank's partials from query rows off the 16-byte boundary (fragments from global memory) and on it (through shared memory)
@pytest.mark.parametrize("Hq", [16, 24])
@pytest.mark.parametrize("p0,p1", [(0, 4000), (1024, 2600)])
def test_shard_attention_of_shifted_rows(Hq, p0, p1):
    capi, layers, g, w = _weights(Hq)
    gen = torch.Generator(device="cuda").manual_seed(Hq + p0)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    R, start = 3, 2997
    s = layers.QsaSession(g, start + R, max_rows=R)
    s.k.copy_(rn(*s.k.shape).half()); s.v.copy_(rn(*s.v.shape).half())
    for r in range(R):
        s.sel[r] = torch.randperm((start + r + 1) // 4, device="cuda", generator=gen)[:512].sort().values.int()
    s.nsel.fill_(512)
    q, z, got = rn(R, Hq, 512), torch.zeros(R, 640, device="cuda"), []
    for shift in (0, 2):
        buf = torch.zeros(q.numel() + 4, device="cuda")
        rows = buf[shift:shift + q.numel()].view_as(q)
        rows.copy_(q)
        args = layers.qsa_args(w, s, rows, z, z, z, z, start)
        part = torch.zeros(R, Hq, 258, device="cuda")
        capi.check(capi.lib.cr_qsa_shard_attn(C.byref(g), C.byref(args), p0, p1, capi.dptr(part), None, 0, None))
        got.append(part)
    assert torch.equal(got[0], got[1]) and got[0][..., 1].min().item() > 0


# rows of a step at the lines between a CTA per row (read twice, held in registers) and a cluster per row
@pytest.mark.parametrize("nb,sessions", [(14336, 3), (14337, 3), (20479, 2), (20480, 2), (20481, 20), (32768, 20), (32769, 20), (32768, 3), (65537, 2), (65537, 20)])
@pytest.mark.parametrize("pattern,pad", [("random", 0), ("random", 1), ("zeros", 0)])
def test_selection_of_step_rows(nb, sessions, pattern, pad):
    capi, layers, g, w = _weights(16)
    gen = torch.Generator(device="cuda").manual_seed(nb + sessions)
    pool = torch.randn((nb + 31) // 32, 128, 32, device="cuda", generator=gen)
    if pattern == "zeros":
        pool *= torch.rand(pool.shape[0], 1, 32, device="cuda", generator=gen) < 300 / nb
    spans, args, z = [], (capi.QsaArgs * sessions)(), torch.zeros(1, 16, 512, device="cuda")
    for i in range(sessions):
        s = layers.QsaSession(g, 64)                                    # the spans share one pool and write no cache
        s.ik_pool = pool.flatten()
        s.sstride = nb + pad
        s.scores = torch.zeros(1, s.sstride, device="cuda")
        idx = torch.randn(1, 640, device="cuda", generator=gen)
        args[i] = layers.qsa_args(w, s, z, z, z, idx, z, 4 * nb - 1)
        spans.append((s, idx))
    capi.check(capi.lib.cr_qsa_select(C.byref(g), args, sessions, None, 0, None))
    for s, _ in spans:
        v = s.scores[0, :nb].double().cpu().numpy()
        want = np.sort(np.lexsort((np.arange(nb), -v))[:512])
        np.testing.assert_array_equal(s.sel[0].cpu().numpy(), want)
        assert int(s.nsel[0]) == 512


# rows of every length beside a long one, by clusters: shares of a few dozen elements, all of which pass, up to the first that has 64 to
# offer in each; rows that attend everything in between
@pytest.mark.parametrize("long_nb", [21000, 57501, 70001])
def test_selection_of_mixed_rows_by_clusters(long_nb):
    capi, layers, g, w = _weights(16)
    gen = torch.Generator(device="cuda").manual_seed(long_nb)
    lengths = [513, 519, 300, 2051, 4095, 4096, 4097, 4103, 7651, 9001, long_nb]
    pool = torch.randn((long_nb + 31) // 32, 128, 32, device="cuda", generator=gen).flatten()
    spans, args, z = [], (capi.QsaArgs * len(lengths))(), torch.zeros(1, 16, 512, device="cuda")
    for i, nb in enumerate(lengths):
        s = layers.QsaSession(g, 64)                                    # the spans share one pool and write no cache
        s.ik_pool, s.sstride = pool, nb
        s.scores = torch.zeros(1, nb, device="cuda")
        idx = torch.randn(1, 640, device="cuda", generator=gen)
        args[i] = layers.qsa_args(w, s, z, z, z, idx, z, 4 * nb - 1)
        spans.append((s, idx))
    capi.check(capi.lib.cr_qsa_select(C.byref(g), args, len(lengths), None, 0, None))
    for (s, _), nb in zip(spans, lengths):
        if nb <= capi.SEL_BLOCKS:
            assert int(s.nsel[0]) == -1
            continue
        v = s.scores[0].double().cpu().numpy()
        np.testing.assert_array_equal(s.sel[0].cpu().numpy(), np.sort(np.lexsort((np.arange(nb), -v))[:512]))
        assert int(s.nsel[0]) == 512


# scores of spans of 3 to 16 rows: every number of row quartets, ragged last tiles, several tiles to a warp (the longest), spans of
# different length in a launch, a pool off the 16-byte boundary (scalar loads), score rows off it
@pytest.mark.parametrize("starts,R,pad,shift", [([2050, 9003], 3, 0, 0), ([4096], 4, 1, 0), ([2300, 2041], 5, 0, 0), ([9003], 9, 2, 0), ([33001], 13, 0, 0),
                                                ([6000], 16, 3, 0), ([262100, 200001], 4, 0, 0), ([9003], 6, 0, 1), ([9003], 12, 1, 3)])
def test_span_scores(starts, R, pad, shift):
    capi, layers, g, w = _weights(16)
    gen = torch.Generator(device="cuda").manual_seed(R)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    spans, args, keep = [], (capi.QsaArgs * len(starts))(), []
    for i, start in enumerate(starts):
        s = layers.QsaSession(g, start + R, max_rows=R)
        s.ik_pool = rn(s.ik_pool.numel() + 4)[shift:]
        s.sstride = (start + R) // 4 + pad
        s.scores = torch.full((R, s.sstride), -7.0, device="cuda")
        idx, z = rn(R, 640), torch.zeros(R, 16, 512, device="cuda")
        args[i] = layers.qsa_args(w, s, z, z, z, idx, z, start)
        spans.append((s, idx, start))
        keep.append(z)
    capi.check(capi.lib.cr_qsa_select(C.byref(g), args, len(starts), None, 0, None))
    for s, idx, start in spans:
        nb_all = (start + R) // 4
        tiles = s.ik_pool[:s.ik_pool.numel() // 4096 * 4096].view(-1, 128, 32).double()
        pool = tiles.transpose(1, 2).reshape(-1, 128)[:nb_all]
        want = torch.relu(torch.einsum("rhd,bd->rhb", idx[:, :512].view(R, 4, 128).double(), pool)).sum(1) / 128 ** 0.5
        for r in range(R):
            nb = (start + r + 1) // 4
            if nb > capi.SEL_BLOCKS:
                assert (s.scores[r, :nb].double() - want[r, :nb]).abs().max().item() < 2e-4, r
                assert (s.scores[r, nb:] == -7.0).all(), r                          # nothing past a row's blocks


# scores of one and two rows, of every block and of a range, from pools on and off the 16-byte boundary (which the wide loads want):
# the order of the 128 products of a dot differs, fp32 throughout; pairs of rows in more CTAs than the form with half a tile in flight has places
@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("starts,R,b0,b1", [([2051], 1, 0, 0), ([9003, 2300], 2, 0, 0), ([79997] * 4, 2, 0, 0), ([9003], 1, 700, 2200), ([9004], 2, 5, 2251)])
def test_short_span_scores_of_shifted_pools(starts, R, b0, b1, shift):
    capi, layers, g, w = _weights(16)
    gen = torch.Generator(device="cuda").manual_seed(R + b0)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    spans, args, keep = [], (capi.QsaArgs * len(starts))(), []
    for i, start in enumerate(starts):
        s = layers.QsaSession(g, start + R, max_rows=R)
        s.ik_pool = rn(s.ik_pool.numel() + 4)[shift:]
        s.scores = torch.full((R, s.sstride), -7.0, device="cuda")
        idx, z = rn(R, 640), torch.zeros(R, 16, 512, device="cuda")
        args[i] = layers.qsa_args(w, s, z, z, z, idx, z, start)
        spans.append((s, idx, start))
        keep.append(z)
    cs, ci = torch.zeros(R, 512, device="cuda"), torch.zeros(R, 512, device="cuda", dtype=torch.int32)
    if b1:
        capi.check(capi.lib.cr_qsa_shard_select(C.byref(g), args, b0, b1, capi.dptr(cs), capi.dptr(ci), None))
    else:
        capi.check(capi.lib.cr_qsa_select(C.byref(g), args, len(starts), None, 0, None))
    for s, idx, start in spans:
        tiles = s.ik_pool[:s.ik_pool.numel() // 4096 * 4096].view(-1, 128, 32).double()
        pool = tiles.transpose(1, 2).reshape(-1, 128)[:(start + R) // 4]
        want = torch.relu(torch.einsum("rhd,bd->rhb", idx[:, :512].view(R, 4, 128).double(), pool)).sum(1) / 128 ** 0.5
        for r in range(R):
            nb = (start + r + 1) // 4
            lo, hi = (b0, min(b1, nb)) if b1 else (0, nb)
            if nb > capi.SEL_BLOCKS:
                assert (s.scores[r, lo:hi].double() - want[r, lo:hi]).abs().max().item() < 2e-4, r
            else:
                lo = hi = 0
            assert (s.scores[r, :lo] == -7.0).all() and (s.scores[r, hi:] == -7.0).all(), r


# Spans of 3 to 16 rows are scored on tensor cores whatever the address of a pool; one pool off the 16-byte boundary beside another on it
@pytest.mark.parametrize("R", [3, 7, 9, 16])
def test_shifted_pools_stay_on_tensor_cores(R):
    capi, layers, g, w = _weights(16)
    gen = torch.Generator(device="cuda").manual_seed(R)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    args, keep = (capi.QsaArgs * 2)(), []
    for i, shift in enumerate((0, 3)):
        s = layers.QsaSession(g, 6001 + R, max_rows=R)
        s.ik_pool = rn(s.ik_pool.numel() + 4)[shift:]
        idx, z = rn(R, 640), torch.zeros(R, 16, 512, device="cuda")
        args[i] = layers.qsa_args(w, s, z, z, z, idx, z, 6001)
        keep.append((s, idx, z))
    capi.check(capi.lib.cr_profile_enable(1))
    try:
        capi.check(capi.lib.cr_qsa_select(C.byref(g), args, 2, None, 0, None))
        names = capi.profile_collect()
    finally:
        capi.check(capi.lib.cr_profile_enable(0))
    assert "qsa_score_mma_kernel" in names and "qsa_score_kernel" not in names, names
    for s, idx, _ in keep:
        pool = s.ik_pool[:s.ik_pool.numel() // 4096 * 4096].view(-1, 128, 32).transpose(1, 2).reshape(-1, 128)[:(6001 + R) // 4].double()
        want = torch.relu(torch.einsum("rhd,bd->rhb", idx[:, :512].view(R, 4, 128).double(), pool)).sum(1) / 128 ** 0.5
        for r in range(R):
            nb = (6001 + r + 1) // 4
            assert (s.scores[r, :nb].double() - want[r, :nb]).abs().max().item() < 2e-4, r


# Rotations of far positions against 64 bits: text positions, and multimodal ones with an axis each, around the angle past which the
# reduction changes (105,615), up to 4 M and at the end of the integers that a float holds; the plain table and a YaRN one, whose
# multiplier scales both.  A head of ones in the first 32 channels comes out as cosines and sines times one factor.  Bound: cosf and
# sinf 2 ulp (2^-23 below one), the remainder's first-order term 2^-24, the norm's factor and the products 5 roundings of 2^-24.
@pytest.mark.parametrize("factor", [1, 4])
@pytest.mark.parametrize("first", [0, 105000, 105600, 262144, 1048576, 4000000, 16775000])
@pytest.mark.parametrize("axes", [1, 3])
def test_rotation_of_far_positions(first, axes, factor):
    from crucible_strix_halo_b200 import capi, layers
    g = capi.Geometry(256, 16, 2, 4, 2)
    one = [torch.ones(n) for n in (256, 256, 128, 128)]
    w = layers.QsaWeights(g, *one, rope_factor=factor)
    rng = np.random.default_rng(first + axes)
    R = 2048
    pos = np.arange(first, first + R, dtype=np.int32)[:, None].repeat(3, 1)
    if axes == 3:
        pos = np.stack([pos[:, 0], rng.integers(0, first + R, R), rng.integers(0, 4194304, R)], 1).astype(np.int32)
    q = torch.zeros(R, 16, 512, device="cuda")
    q[:, :, :32] = 1.0
    q[:, 1::2, :32], q[:, 1::2, 32:64] = 0.0, 1.0
    s, z = layers.QsaSession(g, 64, max_rows=1), torch.zeros(R, 640, device="cuda")
    table = torch.zeros(R, 4, device="cuda", dtype=torch.int32)
    table[:, :3] = torch.from_numpy(pos)
    args = layers.qsa_args(w, s, q, z, z, z, z, first if axes == 1 else 0, mrope=table if axes == 3 else None)
    args.sstride = (first + R) // 4                              # the query half touches neither scores nor cache
    capi.check(capi.lib.cr_qsa_prep_queries(C.byref(g), C.byref(args), 1, None))
    rope = w.rope.cpu().numpy()
    j = np.arange(32)
    axis = np.where(j % 3 == 1, 1, np.where((j % 3 == 2) & (j < 30), 2, 0))
    ang = (pos[:, axis].astype(np.float32) * rope[:32]).astype(np.float64)              # the fp32 angle is the rotation's definition
    scale = float(rope[32]) / np.sqrt(32 / 256 + 1e-6)
    got = q[:, :, :64].cpu().numpy().astype(np.float64) / scale
    want = np.cos(ang), np.sin(ang)
    for h in range(16):
        c, sn = (want[0], want[1]) if h % 2 == 0 else (-want[1], want[0])
        err = max(np.abs(got[:, h, :32] - c).max(), np.abs(got[:, h, 32:] - sn).max())
        assert err < 8 * 2.0 ** -24, (h, err * 2.0 ** 24)


# A compact raw ring beside a full raw cache: calls that start inside a block, whose pooled mean reads ring slots that the call's own
# rows take, fewer and more rows than slots.  The pooled keys and the newest raw keys are the same, bit for bit.
@pytest.mark.parametrize("slots", [16, 37])
@pytest.mark.parametrize("start,R", [(0, 1), (1, 3), (5, 15), (6, 14), (7, 1), (7, 16), (30, 17), (35, 33), (1501, 117), (2047, 38)])
def test_compact_ring_matches_full_cache(slots, start, R):
    capi, layers, g, w = _weights(16)
    gen = torch.Generator(device="cuda").manual_seed(start)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    full, ring = layers.QsaSession(g, start + R, max_rows=R), layers.QsaSession(g, start + R, max_rows=R, raw_slots=slots)
    raw = rn(start + R, 128)
    old = full.ik_raw.view(-1, 128)
    old[:start] = raw[:start]
    for p in range(max(0, start - slots), start):
        ring.ik_raw.view(-1, 128)[p % slots] = raw[p]
    q, k, v, idx = rn(R, g.q_heads, 512), rn(R, 512), rn(R, 512), rn(R, 640)
    idx[:, 512:] = raw[start:]
    outs = [layers.QsaPrefillPlan(w, R).run(s, q.clone(), k.clone(), v.clone(), idx.clone(), start) for s in (full, ring)]
    done = torch.arange(start // 4, (start + R) // 4, device="cuda")                # blocks this call completes
    for s in (full, ring):
        assert torch.equal(s.ik_pool.view(-1, 128, 32)[done // 32, :, done % 32], full.ik_pool.view(-1, 128, 32)[done // 32, :, done % 32])
    for p in range(max(start, start + R - slots), start + R):
        assert torch.equal(ring.ik_raw.view(-1, 128)[p % slots], raw[p]) and torch.equal(old[p], raw[p])
    if start == 0:
        assert torch.equal(outs[0], outs[1])


# scores of prefill parts: dense rows in front of scored ones, ragged row tiles, fewer visits than CTA pairs, runs of a pair
# that cross into the next row tile
@pytest.mark.parametrize("start,R", [(2040, 70), (2100, 17), (9003, 117), (33000, 65), (6001, 257), (20000, 700)])
def test_prefill_part_scores(start, R):
    from crucible_strix_halo_b200 import capi, layers
    g = capi.GEOM_BENCH
    gen = torch.Generator(device="cuda").manual_seed(start)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    w = layers.QsaWeights(g, 1 + 0.1 * rn(256), 1 + 0.1 * rn(256), 1 + 0.1 * rn(128), 1 + 0.1 * rn(128))
    s = layers.QsaSession(g, start + R, max_rows=R)
    s.ik_pool.copy_(rn(s.ik_pool.numel()))
    q, k, v, idx = rn(R, g.q_heads, 512), rn(R, 512), rn(R, 512), rn(R, 640)
    layers.QsaPrefillPlan(w, R).run(s, q, k, v, idx, start)
    assert capi.lib.cr_device_check() == 0
    pool = s.pool_rows((start + R) // 4).double()
    want = torch.relu(torch.einsum("rhd,bd->rhb", idx[:, :512].view(R, 4, 128).double(), pool)).sum(1) / 128 ** 0.5
    for r in range(R):
        nb = (start + r + 1) // 4
        if nb > capi.SEL_BLOCKS:
            assert (s.scores[r, :nb].double() - want[r, :nb]).abs().max().item() < 2e-4, r


# rows on both sides of the first selection: spans without any selecting row (no selection launch), with one, and both in a step
@pytest.mark.parametrize("starts,R", [([1500], 1), ([2046], 1), ([2050], 1), ([2045, 700], 5), ([10, 2051], 3)])
def test_step_marks_dense_rows(starts, R):
    from crucible_strix_halo_b200 import capi, layers
    g = capi.GEOM_BENCH
    gen = torch.Generator(device="cuda").manual_seed(R)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    w = layers.QsaWeights(g, 1 + 0.1 * rn(256), 1 + 0.1 * rn(256), 1 + 0.1 * rn(128), 1 + 0.1 * rn(128))
    spans = []
    for p in starts:
        s = layers.QsaSession(g, p + R, R)
        s.nsel.fill_(77)
        spans.append(dict(session=s, q=rn(R, g.q_heads, 512), k=rn(R, 512), v=rn(R, 512), idx=rn(R, 640), pos0=p))
    layers.QsaStepPlan(w, len(starts) * R).run(spans)
    for x in spans:
        want = [-1 if (x["pos0"] + r + 1) // 4 <= capi.SEL_BLOCKS else capi.SEL_BLOCKS for r in range(R)]
        assert x["session"].nsel.tolist() == want


# Which kernel serves a part: one wave row-wise; then all tiles one way by their lists together (75 rows, a ragged part, as many tiles as
# have an SM each); then tile by tile, a ragged last tile with the one before it, unless it has too many entries per row (129 and 1,185
# rows: a tile of one).  Tiles that share their blocks, tiles that do not, and both in turn, against the row-wise kernel (tolerance of
# the fp16 queries and probabilities of the tiled one).
@pytest.mark.parametrize("Hq", [16, 24])
@pytest.mark.parametrize("R", [16, 17, 74, 75, 129, 148, 1184, 1185, 1204])
@pytest.mark.parametrize("pattern", ["shared", "scattered", "mixed", "mixed last shared"])
def test_prefill_kernel_choice(Hq, R, pattern):
    capi, layers, g, w = _weights(Hq)
    start = 20480
    gen = torch.Generator(device="cuda").manual_seed(R)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    s = layers.QsaSession(g, start + R, max_rows=R)
    s.k.copy_(rn(start + R, 2, 256)); s.v.copy_(rn(start + R, 2, 256))
    RT = 128 // (Hq // 2)
    tile = torch.arange(R, device="cuda") // RT
    last = int(tile[-1])
    share = {"shared": tile >= 0, "scattered": tile < 0, "mixed": (tile - last) % 2 == 1, "mixed last shared": (tile - last) % 2 == 0}[pattern]
    score = rn(R, start // 4) * torch.where(share, 0.05, 1.0)[:, None] + rn(last + 1, start // 4)[tile] * share[:, None]
    s.sel.copy_(score.topk(512, dim=1).indices.sort(dim=1).values.int())
    s.nsel.fill_(512)
    q = rn(R, Hq, 512)
    zero = torch.zeros(R, 640, device="cuda")
    got = {}
    for mode in (0, -1):
        old = capi.set_options(qsa_union_rows=mode)
        try:
            plan = layers.QsaPrefillPlan(w, R)
            plan.q_hi.copy_(q[:, :, :256])
            plan.out.fill_(float("nan"))
            a = capi.QsaPrefillArgs(layers.qsa_args(w, s, q, zero, zero, zero, plan.out, start), capi.dptr(plan.q_hi), capi.dptr(plan.scratch), plan.scratch.numel())
            capi.check(capi.lib.cr_qsa_prefill_attend(C.byref(g), C.byref(a), 0, capi.OUT_RAW_F32, None))
            torch.cuda.synchronize()
            got[mode] = plan.out
        finally:
            capi.check(capi.lib.cr_set_options(C.byref(old)))
    assert capi.lib.cr_device_check() == 0
    assert (got[0] - got[-1]).abs().max().item() < 4e-3
