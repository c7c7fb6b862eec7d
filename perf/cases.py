"""Performance cases of the attention path: what a program that serves a hybrid QSA / Gated DeltaNet model calls, through
crucible_strix_halo_b200.layers.

Kinds of case
  step         one decode or speculative-verify step of a batch of sessions through a GDN layer and a QSA layer
               (layers.gdn_step, layers.QsaStepPlan.run); rows = 1 is plain decoding, rows > 1 a verify span of one
               certain row and rows - 1 drafts behind a pass that left `replay` accepted rows to fold in
  qsa_prefill  one part of a prompt through a QSA layer against the cache before it (layers.QsaPrefillPlan.run)
  gdn_prefill  a prompt, or a part of one, through a GDN layer's core (layers.GdnPrefillPlan.run)
  gdn_layer    the same between its projections: input GEMM, core, output GEMM (layers.proj_gemm around the plan)
  proj         one projection GEMM (layers.proj_gemm)
  checkpoint   a stream's device state saved to a checkpoint and restored from it (layers.SlotCheckpoint)

Geometry "bench": hidden 2048, 16 query / 2 KV heads, 32 / 16 GDN heads.  Geometry "reference": 2560, 24 / 2, 48 / 16.
"""
import math

import torch

from crucible_strix_halo_b200 import capi, layers

GEOMETRY = {"bench": capi.GEOM_BENCH, "reference": capi.GEOM_REF}
FORMAT = {"f32": capi.OUT_RAW_F32, "bf16": capi.OUT_RAW_BF16, "exl3": capi.OUT_EXL3_WHT}
SELECTED = 512                      # blocks of 4 positions a row attends once it has more complete blocks than that


def listed():
    return [
        # One user, short context: every position is attended, launches and host work decide.  The smallest call.
        dict(name="decode_1x1501", kind="step", geometry="bench", sessions=1, context=1501, rows=1, replay=0, out="f32", ring=0),
        # Four sessions at the longest context: the pool scan streams 134 MB.
        dict(name="decode_4x262144", kind="step", geometry="bench", sessions=4, context=262144, rows=1, replay=0, out="bf16", ring=16),
        # One user with draft tokens, the engine's own geometry and output-projection format: the everyday step.
        dict(name="verify_1x32003", kind="step", geometry="reference", sessions=1, context=32003, rows=4, replay=2, out="exl3", ring=16),
        # A serving batch that verifies eight drafts per session at a long context.
        dict(name="verify_8x131072", kind="step", geometry="bench", sessions=8, context=131072, rows=9, replay=4, out="bf16", ring=0),
        # A short chat turn behind a conversation of nine thousand tokens.
        dict(name="qsa_turn_117_at_9003", kind="qsa_prefill", geometry="bench", start=9003, rows=117, follow=0.98, out="bf16", ring=16),
        # A full part in the middle of a prompt, the selections of neighbouring rows overlapping as they do in text.
        dict(name="qsa_part_2048_at_30720", kind="qsa_prefill", geometry="reference", start=30720, rows=2048, follow=0.98, out="exl3", ring=0),
        # The last part of the longest prompt, with unrelated indexer queries: the most scattered selections.
        dict(name="qsa_part_2048_at_260096", kind="qsa_prefill", geometry="bench", start=260096, rows=2048, follow=0.0, out="bf16", ring=0),
        # A part as the engine cuts prompts (2,048 rows at most), fp32 projection rows, engine geometry and output format.
        dict(name="gdn_part_1999", kind="gdn_prefill", geometry="reference", start=6144, rows=1999, input="f32", out="exl3"),
        # A whole 32K prompt in one call, bf16 projection rows.
        dict(name="gdn_prompt_32768", kind="gdn_prefill", geometry="bench", start=0, rows=32768, input="bf16", out="bf16"),
        # A short chat turn through a whole GDN layer: projections and core, few rows.
        dict(name="gdn_layer_333", kind="gdn_layer", geometry="bench", start=9003, rows=333),
        # The input projection of a GDN layer over a 32K prompt.
        dict(name="gdn_in_proj_32768", kind="proj", rows=32768, inner=2048, columns=12352, out="bf16"),
        # The in-slot checkpoint of a 48-layer stream: 36 GDN layers, 12 QSA layers.
        dict(name="checkpoint_48_layers", kind="checkpoint", geometry="bench", gdn_layers=36, qsa_layers=12, position=4003),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "qsa_prefill", "qsa_prefill", "gdn_prefill", "gdn_prefill", "gdn_layer", "proj", "checkpoint"])
    geometry = rng.choice(["bench", "reference"])
    if kind == "step":
        sessions, rows = rng.choice([1, 1, 2, 3, 4, 6, 8, 12, 16]), rng.choice([1, 1, 1, 2, 3, 4, 5, 6, 7, 8, 9])
        return dict(kind=kind, geometry=geometry, sessions=sessions, context=_log(rng, 300, min(262144, 1048576 // sessions)), rows=rows,
                    replay=rng.randint(0, min(8, rows - 1)), out=rng.choice(["f32", "bf16", "exl3"]), ring=rng.choice([0, 16]))
    if kind == "qsa_prefill":
        rows = rng.choice([2048, _log(rng, 1, 2048)])
        return dict(kind=kind, geometry=geometry if rows < 2048 else "bench", start=_log(rng, 1, 260096) - 1, rows=rows, follow=rng.choice([0.0, 0.9, 0.98]),
                    out=rng.choice(["f32", "bf16", "exl3"]), ring=rng.choice([0, 16]))
    if kind == "gdn_prefill":
        return dict(kind=kind, geometry=geometry, start=_log(rng, 1, 200000) - 1, rows=_log(rng, 1, 32768 if geometry == "bench" else 16384),
                    input=rng.choice(["f32", "bf16"]), out=rng.choice(["f32", "bf16", "exl3"]))
    if kind == "gdn_layer":
        return dict(kind=kind, geometry=geometry, start=_log(rng, 1, 200000) - 1, rows=_log(rng, 1, 8192))
    if kind == "proj":
        inner = rng.choice([2048, 2560, 4096])
        return dict(kind=kind, rows=_log(rng, 1, 32768 * 2048 // inner), inner=inner, columns=32 * rng.randint(40, 386), out=rng.choice(["f32", "bf16"]))
    qsa_layers = rng.randint(1, 12)
    return dict(kind=kind, geometry=geometry, gdn_layers=3 * qsa_layers, qsa_layers=qsa_layers, position=rng.randint(1, 4095))


# ---- inputs ----------------------------------------------------------------------------------------------------

class _Values:
    """Seeded values on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        return torch.empty(*shape, device="cuda", dtype=dtype).normal_(mean, std, generator=self.gen)

    def fill(self, *tensors, std=1.0):
        for t in tensors:
            t.normal_(0.0, std, generator=self.gen)

    def uniform(self, *shape):
        return torch.rand(*shape, device="cuda", generator=self.gen)

    def follow(self, rows, width, rho):
        """Unit-variance rows of which each is rho times the one before it plus news."""
        x = self.normal(rows, width)
        if not rho:
            return x
        i = torch.arange(rows, device="cuda", dtype=torch.float32)
        lag = i[:, None] - i[None, :]
        mix = torch.where(lag >= 0, rho ** lag.clamp(min=0), torch.zeros_like(lag))
        mix[:, 1:] *= math.sqrt(1 - rho * rho)
        return mix @ x


def _gdn_weights(v, g, step=False, suh=False):
    Hv = g.gdn_vheads
    return layers.GdnWeights(g, v.normal(g.gdn_channels, 4, std=0.5), v.normal(Hv, std=1.5, mean=-1.0).clamp(-5, 1.5), v.normal(Hv, std=0.5),
                             v.normal(128, std=0.1, mean=1.0), ab=v.normal(2 * Hv, g.hidden, std=0.05) if step else None,
                             suh=v.normal(Hv * 128, std=0.1, mean=1.0) if suh else None)


def _qsa_weights(v, g, suh=False):
    norms = [v.normal(n, std=0.1, mean=1.0) for n in (256, 256, 128, 128)]
    return layers.QsaWeights(g, *norms, suh=v.normal(g.q_heads * 256, std=0.1, mean=1.0) if suh else None)


def _qsa_rows(v, g, sessions, rows, follow=0.0):
    """Projection rows of a QSA layer, one dict per session.  q and idx lie in one buffer that the layer overwrites when it
    normalises them; `fresh` holds what the projection of the next pass puts there."""
    nq = g.q_heads * 512
    fresh = v.normal(sessions, rows * (nq + 640))
    if follow:
        for f in fresh:
            f[rows * nq:].view(rows, 640)[:, :512] = v.follow(rows, 512, follow)
    work = torch.empty_like(fresh)
    got = [dict(q=w[:rows * nq].view(rows, g.q_heads, 512), idx=w[rows * nq:].view(rows, 640), k=v.normal(rows, g.kv_heads * 256),
                v=v.normal(rows, g.kv_heads * 256)) for w in work]
    return got, fresh, work


def _qsa_session(v, g, context, rows, ring):
    s = layers.QsaSession(g, context, max_rows=rows, raw_slots=ring)
    v.fill(s.k, s.v, s.ik_raw, s.ik_pool)
    return s


def _gdn_session(v, g, pend_rows=8):
    s = layers.GdnSession(g, pend_rows=pend_rows)
    v.fill(s.state_view(), std=0.05)
    v.fill(s.hist)
    return s


def _pool(sessions, name):
    slots = torch.zeros(len(sessions), *getattr(sessions[0], name).shape, device="cuda", dtype=getattr(sessions[0], name).dtype)
    for s, slot in zip(sessions, slots):
        setattr(s, name, slot)
    return slots


def _written(k, v, ik_pool, start, rows):
    """What a step or a part writes into QSA caches: its K and V rows and the pool tiles it completes blocks in."""
    got = [k[..., start:start + rows, :, :], v[..., start:start + rows, :, :]]
    b0, b1 = start // 4, (start + rows) // 4
    return got + ([ik_pool[..., b0 // 32 * 4096:((b1 - 1) // 32 + 1) * 4096]] if b1 > b0 else [])


def prepare(case, seed):
    v, kind = _Values(seed), case["kind"]
    if kind == "proj":
        R, K, N = case["rows"], case["inner"], case["columns"]
        out = torch.empty(R, N, device="cuda", dtype=torch.bfloat16 if case["out"] == "bf16" else torch.float32)
        return dict(kind=kind, x=v.normal(R, K, dtype=torch.bfloat16), w=v.normal(N, K, std=K ** -0.5, dtype=torch.bfloat16), outs=[out])
    g = GEOMETRY[case["geometry"]]
    VW = g.gdn_vheads * 128
    if kind == "step":
        R, S, start, suh = case["rows"], case["sessions"], case["context"] - case["rows"], case["out"] == "exl3"
        commit = 1 if R > 1 else R
        gw, qw = _gdn_weights(v, g, step=True, suh=suh), _qsa_weights(v, g, suh)
        gs, qs = [layers.GdnSession(g, pend_rows=16 if R > 8 else 8) for _ in range(S)], [layers.QsaSession(g, case["context"], R, raw_slots=case["ring"]) for _ in range(S)]
        # the sessions' buffers are slots of one pool each, as a serving engine holds them
        pools = {n: _pool(gs, n) for n in ("state", "hist", "pend")} | {n: _pool(qs, n) for n in ("k", "v", "ik_raw", "ik_pool")}
        v.fill(*(pools[n] for n in ("hist", "k", "v", "ik_raw", "ik_pool")))
        v.fill(pools["state"][:, :g.gdn_vheads * 16384], std=0.05)
        v.fill(pools["pend"], std=0.1)
        pools["pend"][..., 256:] = 0.5 + 0.5 * v.uniform(S, g.gdn_vheads, gs[0].pend_rows, 2)           # decay and beta of the pending rows
        gdn = [dict(session=s, qkv=v.normal(R, g.gdn_channels), z=v.normal(R, VW), x=v.normal(R, g.hidden), pos0=start,
                    replay=case["replay"], commit=commit) for s in gs]
        rows, fresh, work = _qsa_rows(v, g, S, R)
        qsa = [dict(session=s, pos0=start, **r) for s, r in zip(qs, rows)]
        after = [pools["state"], pools["hist"], pools["pend"]] + _written(pools["k"], pools["v"], pools["ik_pool"], start, R)
        return dict(kind=kind, gw=gw, gdn=gdn, qsa=qsa, fresh=fresh, work=work, plan=layers.QsaStepPlan(qw, S * R, fmt=FORMAT[case["out"]]), fmt=FORMAT[case["out"]], after=after)
    if kind == "qsa_prefill":
        R, start = case["rows"], case["start"]
        w, s = _qsa_weights(v, g, case["out"] == "exl3"), _qsa_session(v, g, start + R, R, case["ring"])
        rows, fresh, work = _qsa_rows(v, g, 1, R, case["follow"])
        return dict(kind=kind, plan=layers.QsaPrefillPlan(w, R, fmt=FORMAT[case["out"]]), session=s, rows=rows[0], fresh=fresh, work=work, start=start,
                    after=_written(s.k, s.v, s.ik_pool, start, R))
    if kind == "gdn_prefill":
        R, bf = case["rows"], case["input"] == "bf16"
        dt = torch.bfloat16 if bf else torch.float32
        w = _gdn_weights(v, g, suh=case["out"] == "exl3")
        plan = layers.GdnPrefillPlan(w, R, in_dtype=capi.IN_BF16 if bf else capi.IN_F32, fmt=FORMAT[case["out"]])
        return dict(kind=kind, plan=plan, session=_gdn_session(v, g), start=case["start"], qkv=v.normal(R, g.gdn_channels, dtype=dt),
                    z=v.normal(R, VW, dtype=dt), ab=v.normal(R, 2 * g.gdn_vheads, dtype=dt))
    if kind == "gdn_layer":
        R, bf = case["rows"], dict(device="cuda", dtype=torch.bfloat16)
        widths = (g.gdn_channels, VW, 2 * g.gdn_vheads)
        return dict(kind=kind, plan=layers.GdnPrefillPlan(_gdn_weights(v, g), R, in_dtype=capi.IN_BF16, fmt=capi.OUT_RAW_BF16), session=_gdn_session(v, g),
                    start=case["start"], x=v.normal(R, g.hidden, dtype=torch.bfloat16), w_in=v.normal(sum(widths), g.hidden, std=g.hidden ** -0.5, dtype=torch.bfloat16),
                    w_out=v.normal(g.hidden, VW, std=VW ** -0.5, dtype=torch.bfloat16), rows=[torch.empty(R, n, **bf) for n in widths],
                    hidden=[torch.empty(R, g.hidden, **bf)])
    # checkpoint: compact raw rings and one open pool tile per QSA layer, as a slot of a serving engine holds them
    gs = [_gdn_session(v, g) for _ in range(case["gdn_layers"])]
    for s in gs:
        v.fill(s.pend)
    qs = [_qsa_session(v, g, 4096, 1, 16) for _ in range(case["qsa_layers"])]
    point = layers.SlotCheckpoint(layers.checkpoint_spans(gs, qs, case["position"]))
    return dict(kind=kind, point=point, after=[point.buffer, gs[0].state, gs[-1].pend, qs[-1].ik_pool])


def run(state):
    kind = state["kind"]
    if kind == "step":
        gdn_out = layers.gdn_step(state["gw"], state["gdn"], state["fmt"])
        state["work"].copy_(state["fresh"])
        return dict(gdn=gdn_out, qsa=state["plan"].run(state["qsa"]), after=state["after"])
    if kind == "qsa_prefill":
        state["work"].copy_(state["fresh"])
        r = state["rows"]
        return dict(out=state["plan"].run(state["session"], r["q"], r["k"], r["v"], r["idx"], state["start"]), after=state["after"])
    if kind == "gdn_prefill":
        s = state["session"]
        out = state["plan"].run(s, state["qkv"], state["z"], state["ab"], state["start"], capi.GDN_CHUNK_TC)
        return dict(out=out, state=s.state, hist=s.hist)
    if kind == "gdn_layer":
        s = state["session"]
        qkv, z, ab = layers.proj_gemm(state["x"], state["w_in"], state["rows"])
        core = state["plan"].run(s, qkv, z, ab, state["start"], capi.GDN_CHUNK_TC)
        return dict(out=layers.proj_gemm(core, state["w_out"], state["hidden"]), state=s.state, hist=s.hist)
    if kind == "proj":
        return layers.proj_gemm(state["x"], state["w"], state["outs"])
    state["point"].save()
    state["point"].restore()
    return state["after"]


# ---- what a pass cannot do without -------------------------------------------------------------------------------

OUT_BYTES = {"f32": 4, "bf16": 2, "exl3": 2}


def _attended(p):
    nb = (p + 1) // 4
    return p + 1 if nb <= SELECTED else 4 * SELECTED + (p + 1) % 4


def _qsa_work(g, start, rows, out_bytes, distinct):
    """Of one span: pooled keys once, K / V of `distinct` positions once, projection rows in, cache rows and outputs out."""
    nb = (start + rows) // 4
    scored = sum((start + r + 1) // 4 for r in range(rows) if (start + r + 1) // 4 > SELECTED)
    kv = 2 * g.kv_heads * 256
    moved = (nb * 512 if nb > SELECTED else 0) + distinct * kv * 2 + rows * 4 * (g.q_heads * 512 + kv + 640) + rows * (kv * 2 + 128 + g.q_heads * 256 * out_bytes)
    return moved, scored * 4 * 128 * 2 + sum(_attended(start + r) for r in range(rows)) * g.q_heads * 256 * 4


def _gdn_flops(g, rows):
    return rows * g.gdn_vheads * 128 * 128 * 2 * 3          # S^T k, the rank-one update, S^T q


def work(case):
    kind = case["kind"]
    if kind == "proj":
        R, K, N = case["rows"], case["inner"], case["columns"]
        return {"bytes": 2 * (R * K + N * K) + R * N * OUT_BYTES[case["out"]], "flops": 2 * R * K * N}
    g = GEOMETRY[case["geometry"]]
    C, VW, Hv, R = g.gdn_channels, g.gdn_vheads * 128, g.gdn_vheads, case.get("rows", 1)
    state = Hv * 128 * 128 * 4
    if kind == "step":
        S, start, o = case["sessions"], case["context"] - R, OUT_BYTES[case["out"]]
        # rows of a span differ in what they select: each row's positions count, up to the whole context
        distinct = min(start + R, sum(_attended(start + r) for r in range(R)))
        moved, flops = _qsa_work(g, start, R, o, distinct)
        pend = (case["replay"] + (R - 1 if R > 1 else 0)) * Hv * 258 * 4
        gdn = 2 * state + R * (4 * (C + VW + g.hidden) + VW * o + 4 * C) + 3 * C * 4 + pend
        return {"bytes": S * (moved + gdn) + 2 * Hv * g.hidden * 2 + C * 16, "flops": S * (flops + _gdn_flops(g, R + case["replay"]) + R * 4 * Hv * g.hidden)}
    if kind == "qsa_prefill":
        start = case["start"]
        distinct = min(start + R, sum(_attended(start + r) for r in range(R)))
        moved, flops = _qsa_work(g, start, R, OUT_BYTES[case["out"]], distinct)
        return {"bytes": moved, "flops": flops}
    if kind == "gdn_prefill":
        i = 2 if case["input"] == "bf16" else 4
        return {"bytes": R * (i * (C + VW + 2 * Hv) + VW * OUT_BYTES[case["out"]]) + 2 * state + 19 * C * 4 + C * 16, "flops": _gdn_flops(g, R)}
    if kind == "gdn_layer":
        N, H = C + VW + 2 * Hv, g.hidden
        return {"bytes": 2 * (2 * R * H + N * H + H * VW) + 2 * state + 19 * C * 4 + C * 16, "flops": 2 * R * H * (N + VW) + _gdn_flops(g, R)}
    n = case["gdn_layers"] * (4 * (Hv * 16384 + 64) + 64 * C + 4 * Hv * 8 * 258) + case["qsa_layers"] * (16 * 512 + (16384 if case["position"] % 128 else 0))
    return {"bytes": 4 * n, "flops": 0}                      # the spans read and written once by the save, once by the restore


def tolerance(case):
    if case["kind"] == "checkpoint":
        return "exact"
    if case["kind"] == "proj":
        return {"rel": 1e-5 if case["out"] == "f32" else 5e-3}
    if case["kind"] == "step":
        # fp32 products over fp16 K / V; a block whose score ties with the 512th within fp32 rounding may be exchanged,
        # which moves one row of the output by a few per cent
        return {"rel": {"f32": 2e-3, "bf16": 1e-2, "exl3": 5e-3}[case["out"]]}
    if case["kind"] == "qsa_prefill":
        return {"rel": 1e-2}                                 # fp16 queries and probabilities, score ties as above
    return {"rel": 1e-2 if case.get("out", "bf16") == "bf16" else 3e-3}   # tf32 operands of the chunked recurrence
