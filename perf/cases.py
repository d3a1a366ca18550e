"""The work that this library is used for, as cases that can be timed: MoE sublayers over INT4 group-32 expert pages in a
VRAM pool, from one token to a batch, through the calls a serving program makes.

A case names a layer shape, an activation type and one of seven ways to use the library (``kind``):

  step_host   one token from and to host memory per layer, the layer bound once (MoeDecoder.bind_host_step)
  layer       one token already on the device, router and experts in one call (MoeDecoder.forward_layer)
  stack       residual add + RMS norm + MoE sublayer per layer, recorded once as a CUDA graph and replayed: what an
              engine runs between its attention blocks; one token (MoeDecoder) or a batch (GroupedDecoder)
  tokens      a batch of tokens through one layer, every distinct expert read once (GroupedDecoder.forward)
  ep_share    the same for an expert-parallel rank that owns a range of the experts (GroupedDecoder.experts with a range)
  ep_pairs    an expert-parallel rank's launches of a step with one token per rank: the pairs it owns plus the shared
              expert of its own token (select_local_pairs, moe_layer_int4_paged_grouped)
  paged       the per-page calls in the order an engine drives them, with the routing read back by the host
              (run_moe_sublayer_paged_calls)

Weights, tokens and routing are seeded synthetic data of the distributions that synth.py gives.  Every layer of a pass
has its own token, as in a decode step, so that one layer's rounding does not reroute the next.  A pass reads more
weight bytes than the L2 cache holds, except for the small shapes, which a serving program finds in L2 too.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vic_b200 import kernels
from vic_b200.buffer_manager import QueryPlanner
from vic_b200.core_types import KIMI, MIXTRAL, SCORING_SIGMOID, SCORING_SOFTMAX, MoeShape
from vic_b200.ep import PAIRS_PER_LAUNCH
from vic_b200.grouped import GroupedDecoder, zipf_logit_offset
from vic_b200.moe import MoeDecoder, run_moe_sublayer_paged_calls
from vic_b200.synth import build_synthetic_moe, synth_activation

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
EP_WORLD = 8          # expert-parallel cases: rank 1 of eight


def _case(name, kind, shape, layers, tokens, dtype, **options):
    c = {"kind": kind, "hidden": shape.hidden, "intermediate": shape.intermediate, "experts": shape.num_experts,
         "top_k": shape.top_k, "shared": shape.shared_experts, "sigmoid": shape.scoring == SCORING_SIGMOID,
         "scaling": shape.scaling_factor, "layers": layers, "tokens": tokens, "dtype": dtype, "skew": False, "bias": False}
    c.update(options)
    if name:
        c["name"] = name
    return c


SMALL = MoeShape("small", 1024, 2048, 6, 3, 1, SCORING_SIGMOID, 2.5, True)
RAGGED = MoeShape("ragged", 1024, 4000, 6, 3, 1, SCORING_SIGMOID, 2.5, True)


def listed():
    return [
        # the smallest call: a small layer's token from and to host memory, where launches and the wait are the cost
        _case("small_step_host", "step_host", SMALL, 1, 1, "bf16"),
        # sizes that no tile divides (4000 rows, ragged last pages), fp32 activations, a selection bias
        _case("ragged_layer_fp32", "layer", RAGGED, 1, 1, "fp32", bias=True),
        # decode of one request through host buffers: the headline workload end to end, two layers per pass
        _case("kimi_step_host", "step_host", KIMI, 2, 1, "bf16"),
        # decode of one request inside an engine's graph: norm and sublayer
        _case("kimi_stack_1", "stack", KIMI, 2, 1, "bf16"),
        # decode of one request through wide experts (intermediate 14336), softmax over the selected, fp16
        _case("mixtral_layer_fp16", "layer", MIXTRAL, 2, 1, "fp16"),
        # the library behind an engine that launches page by page
        _case("kimi_paged", "paged", KIMI, 1, 1, "fp32"),
        # small decode batch, skewed load (a few experts are popular)
        _case("kimi_tokens_8", "tokens", KIMI, 1, 8, "bf16", skew=True),
        # usual decode batch inside an engine's graph, evenly loaded experts: about 190 distinct ones
        _case("kimi_stack_32", "stack", KIMI, 1, 32, "bf16"),
        # largest batch of one step, skewed load: from idle experts to one that most tokens choose
        _case("kimi_tokens_128", "tokens", KIMI, 1, 128, "bf16", skew=True),
        # a prefill chunk of odd length through few wide experts: about 12 tokens for each
        _case("mixtral_tokens_50", "tokens", MIXTRAL, 1, 50, "fp16"),
        # an expert-parallel rank's share of a decode batch of odd size
        _case("kimi_ep_share_29", "ep_share", KIMI, 1, 29, "bf16"),
        # an expert-parallel rank's share of one token from each of eight ranks
        _case("kimi_ep_pairs_8", "ep_pairs", KIMI, 2, 8, "bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any kind, layer shapes from the small test sizes to the two full ones, 1 to 128 tokens."""
    while True:
        kind = rng.choice(["step_host", "layer", "layer", "stack", "stack", "tokens", "tokens", "tokens", "ep_share", "ep_pairs", "paged"])
        pick = rng.random()
        if pick < 0.35:
            # the large layer with fewer experts and other routing widths
            sh = MoeShape("drawn", KIMI.hidden, KIMI.intermediate, 16 * rng.randint(4, 24), rng.randint(4, 8), rng.randint(0, 1),
                          SCORING_SIGMOID, 2.5, True)
        elif pick < 0.5 and kind not in ("ep_share", "ep_pairs"):
            sh = MoeShape("drawn", MIXTRAL.hidden, MIXTRAL.intermediate, rng.choice([8, 12, 16]), rng.randint(1, 4), 0, SCORING_SOFTMAX, 1.0, True)
        else:
            # tensor-core and expert-parallel launches take multiples of 256, the one-token calls any multiple of 32
            step = 32 if kind in ("step_host", "layer", "paged") else 256
            hidden = max(step, _log_int(rng, 512, 7168) // step * step)
            inter = max(step, _log_int(rng, 512, 6144) // step * step)
            if kind == "ep_pairs":
                inter = rng.choice([1024, 2048])
            experts = _log_int(rng, 4, 256)
            if kind in ("ep_share", "ep_pairs"):
                experts = max(2 * EP_WORLD, experts // EP_WORLD * EP_WORLD)
            top_k = rng.randint(1, min(8, experts))
            sigmoid = rng.random() < 0.6
            sh = MoeShape("drawn", hidden, inter, experts, top_k, rng.randint(0, 1), SCORING_SIGMOID if sigmoid else SCORING_SOFTMAX,
                          rng.choice([1.0, 2.5]) if sigmoid else 1.0, True)
        if kind in ("tokens", "ep_share") or (kind == "stack" and rng.random() < 0.5):
            tokens = _log_int(rng, 2, 128)
        elif kind == "ep_pairs":
            tokens = rng.choice([2, 4, EP_WORLD])
        else:
            tokens = 1
        layers = rng.randint(1, 2) if kind in ("step_host", "layer", "stack", "ep_pairs") and tokens <= 8 else 1
        dtype = "fp32" if kind == "paged" else "bf16" if kind == "ep_pairs" else rng.choice(["bf16", "bf16", "fp16", "fp32"])
        c = _case(None, kind, sh, layers, tokens, dtype, skew=kind in ("tokens", "ep_share") and rng.random() < 0.5,
                  bias=kind == "layer" and rng.random() < 0.3)
        # (the direct kernels keep every selected expert's intermediate in shared memory)
        if (sh.top_k + sh.shared_experts) * sh.intermediate > 9 * 8192:
            continue
        if work(c)["bytes"] <= 3.9e9 and sh.num_experts * sh.expert_bytes * layers <= 20e9:
            return c


def _shape(case):
    return MoeShape("case", case["hidden"], case["intermediate"], case["experts"], case["top_k"], case["shared"],
                    SCORING_SIGMOID if case["sigmoid"] else SCORING_SOFTMAX, case["scaling"], True)


def _ep_range(sh):
    n = sh.num_experts // EP_WORLD
    return n, 2 * n       # rank 1


def prepare(case, seed):
    sh, dev, kind = _shape(case), torch.device("cuda"), case["kind"]
    L, T, dt = case["layers"], case["tokens"], DTYPES[case["dtype"]]
    lo, hi = _ep_range(sh) if kind in ("ep_share", "ep_pairs") else (0, sh.num_experts)
    model = build_synthetic_moe(sh, L, dev, seed=seed, slot_seed=seed + 1, experts=None if hi - lo == sh.num_experts else range(lo, hi))
    g = torch.Generator(device=dev).manual_seed(seed + 2)
    xs = synth_activation(sh, g, dev, dt, L * T).view(L, T, sh.hidden)
    s = {"kind": kind, "sh": sh, "L": L, "T": T, "xs": xs, "model": model, "range": (lo, hi), "offset": None, "bias": None}
    if case["skew"]:
        s["offset"] = torch.from_numpy(zipf_logit_offset(sh.num_experts, seed + 3)).to(dev)
    if case["bias"]:
        s["bias"] = 0.1 * torch.randn(sh.num_experts, generator=g, device=dev)
    if kind in ("step_host", "layer", "ep_pairs") or (kind == "stack" and T == 1):
        s["dec"] = MoeDecoder(model)
    if kind in ("tokens", "ep_share") or (kind == "stack" and T > 1):
        s["gd"] = GroupedDecoder(model, max_tokens=T)
    if kind == "step_host":
        s["stream"] = torch.cuda.Stream(device=dev)
        s["host"] = [xs[l, 0].cpu().pin_memory() for l in range(L)]
        s["steps"] = [s["dec"].bind_host_step(l, dt, s["stream"]) for l in range(L)]
    elif kind == "layer":
        s["out"] = torch.zeros(L, sh.hidden, device=dev)
        s["ids"] = torch.zeros(L, 16, dtype=torch.int16, device=dev)
    elif kind == "stack":
        s["h0"] = synth_activation(sh, g, dev, torch.float32, L * T).view(L, T, sh.hidden)
        s["attn"] = (0.3 * torch.randn(L, T, sh.hidden, generator=g, device=dev)).to(torch.bfloat16)
        s["norm"] = (1.0 + 0.1 * torch.randn(L, sh.hidden, generator=g, device=dev)).to(torch.float16)
        s["h"], s["x"] = torch.zeros_like(s["h0"]), torch.zeros(T, sh.hidden, dtype=dt, device=dev)
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _stack(s)
            side.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"], stream=side):
                _stack(s)
        torch.cuda.current_stream().wait_stream(side)
    elif kind == "ep_pairs":
        # the messages of the eight ranks as they lie in the receive buffer: tokens, expert ids, routing weights
        dec = s["dec"]
        s["ids"] = torch.zeros(L, T, 16, dtype=torch.int16, device=dev)
        s["w"] = torch.zeros(L, T, 16, device=dev)
        for l in range(L):
            for t in range(T):
                dec.route(l, xs[l, t])
                s["ids"][l, t].copy_(dec.ids)
                s["w"][l, t].copy_(dec.weights)
        cap = T * sh.top_k
        s["pe"], s["pt"] = (torch.zeros(cap, dtype=torch.int16, device=dev) for _ in range(2))
        s["pw"], s["n"] = torch.zeros(cap, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
        s["act"] = torch.zeros((PAIRS_PER_LAUNCH + 1) * sh.intermediate, dtype=torch.float16, device=dev)
        s["out"] = torch.zeros(L, T, sh.hidden, device=dev)
    elif kind == "paged":
        s["planner"], s["bufs"] = QueryPlanner(model.pool, sh.pages_per_segment), {}
        s["w16"] = [model.router_w[l].to(torch.float16) for l in range(L)]
    return s


def _stack(s):
    """The layers' sublayers, each on its own hidden state: h += attention output, x = norm(h), h += moe(x)."""
    s["h"].copy_(s["h0"])
    for l in range(s["L"]):
        kernels.residual_rms_norm(s["h"][l], s["attn"][l], s["norm"][l], 1e-6, s["x"], early_dependents=True)
        if s["T"] == 1:
            s["dec"].forward_layer(l, s["x"][0], out=s["h"][l, 0], accumulate=True, hold=True)
        else:
            s["gd"].forward(l, s["x"], out=s["h"][l], accumulate=True, hold=True)


def run(s):
    kind, sh, L = s["kind"], s["sh"], s["L"]
    if kind == "step_host":
        for l in range(L):
            s["steps"][l].run(s["host"][l].data_ptr())
        return [step.out for step in s["steps"]]
    if kind == "layer":
        for l in range(L):
            s["dec"].forward_layer(l, s["xs"][l, 0], out=s["out"][l], bias=s["bias"])
            s["ids"][l].copy_(s["dec"].ids)
        return s["out"], s["ids"]
    if kind == "stack":
        s["graph"].replay()
        return s["h"]
    if kind == "tokens":
        out = s["gd"].forward(0, s["xs"][0], logit_offset=s["offset"])
        return out, s["gd"].ids[:s["T"]], s["gd"].weights[:s["T"]]
    if kind == "ep_share":
        gd = s["gd"]
        gd.route(0, s["xs"][0], s["offset"])
        out = gd.experts(0, s["xs"][0], expert_range=s["range"], shared=False)
        return out, gd.ids[:s["T"]]
    if kind == "ep_pairs":
        dec, (lo, hi) = s["dec"], s["range"]
        for l in range(L):
            kernels.select_local_pairs(s["ids"][l], 32, s["w"][l], 64, s["T"], sh.top_k, lo, hi, s["pe"], s["pw"], s["pt"], s["pe"].numel(), s["n"])
            for b in range(0, s["pe"].numel(), PAIRS_PER_LAUNCH):
                kernels.moe_layer_int4_paged_grouped(
                    s["xs"][l], kernels.x_dtype_code(s["xs"]), s["xs"].stride(1) * s["xs"].element_size(), s["T"], dec.tables[l], sh.num_experts,
                    dec.shared_tables[l] if b == 0 else 0, 1, s["pe"], s["pw"], s["pt"], PAIRS_PER_LAUNCH, b, s["n"], 1.0, s["act"],
                    s["out"][l], sh.hidden, b > 0, sh.hidden, sh.intermediate, sh.pages_per_segment, sh.gate_up.rows_per_page,
                    sh.down.rows_per_page, dec.status)
        return s["out"]
    out, activation, _ = run_moe_sublayer_paged_calls(s["model"], 0, s["xs"][0, 0], s["planner"], s["w16"][0], s["bufs"])
    return out, np.array([e for e, _ in activation], dtype=np.int64), np.array([w for _, w in activation], dtype=np.float32)


def _selected(case):
    """(pairs, distinct experts) of one layer that the pass computes, from the routing that tokens of this kind get: router
    weights N(0, 0.02) against N(0, 1) columns make logits N(0, 0.02 sqrt(hidden)), the skewed cases add the offset."""
    sh, T = _shape(case), case["tokens"]
    rng = np.random.default_rng(5)
    logits = rng.standard_normal((T, sh.num_experts)) * 0.02 * math.sqrt(sh.hidden)
    if case["skew"]:
        logits = logits + zipf_logit_offset(sh.num_experts, 5)
    ids = np.argsort(-logits, axis=1)[:, :sh.top_k].reshape(-1)
    if case["kind"] in ("ep_share", "ep_pairs"):
        lo, hi = _ep_range(sh)
        ids = ids[(ids >= lo) & (ids < hi)]
    return len(ids), len(set(ids.tolist()))


def work(case):
    sh, L, T, kind = _shape(case), case["layers"], case["tokens"], case["kind"]
    pairs, distinct = _selected(case)
    if kind == "ep_pairs":
        distinct = pairs      # (a pair reads its expert: two tokens of a step rarely share one of 384)
    shared = sh.shared_experts and kind != "ep_share"
    weights = (distinct + (1 if shared else 0)) * sh.expert_bytes
    router = 0 if kind == "ep_pairs" else sh.num_experts * sh.hidden * (2 if kind == "paged" else 4)
    xbytes = {"bf16": 2, "fp16": 2, "fp32": 4}[case["dtype"]]
    rows = T * sh.hidden * (xbytes + 4 if kind != "stack" else 4 + 2 + 4)
    own = (1 if kind == "ep_pairs" else T) if shared else 0
    flops = 2.0 * (pairs + own) * 3 * sh.hidden * sh.intermediate + (0 if kind == "ep_pairs" else 2.0 * T * sh.num_experts * sh.hidden)
    return {"bytes": L * (weights + router + rows), "flops": L * flops}


def tolerance(case):
    # A sublayer rounds gate, up, their SiLU product and every expert's down projection to fp16.  Against the same layer in
    # 64 bits (dequantised pages, the same routing) the outputs of all kinds and shapes differ by 4.1e-4 to 5.1e-4 relative
    # and by at most 3.1e-3 of their root mean square (tensor-core and one-token paths alike); four times that is stated.
    # Where the hidden state is part of the output it hides some of the difference.  Expert ids are whole: none may differ.
    return {"rel": 1.7e-3, "max": 1.2e-2}


# ── the same in 64 bits ──────────────────────────────────────────────────────────────────────

PAGE_BYTES = 2 << 20


def _matrix64(model, layer, expert, segment):
    """One INT4 matrix of the pool as float64: per page [rows x K/2] code bytes (low nibble = even column, weight =
    (nibble - 8) * scale), then [rows x K/32] fp16 scales."""
    store, parts = model.pool.storage, []
    for pg in sorted((p for p in model.by_expert[layer, expert] if p.pid.segment == segment), key=lambda p: p.row_start):
        raw, n = store[pg.slot * PAGE_BYTES:(pg.slot + 1) * PAGE_BYTES], pg.row_count * pg.cols // 2
        codes = raw[:n].view(pg.row_count, pg.cols // 2)
        scales = raw[n:n + pg.row_count * pg.cols // 16].clone().view(torch.float16).view(pg.row_count, pg.cols // 32)
        w = torch.stack((codes & 15, codes >> 4), dim=2).view(pg.row_count, pg.cols).double() - 8.0
        parts.append((w.view(pg.row_count, -1, 32) * scales.double()[:, :, None]).view(pg.row_count, pg.cols))
    return torch.cat(parts)


def _experts64(model, layer, x, pairs, shared_tokens):
    """Sum over a token's experts of weight * down(silu(gate x) * up x); pairs: [(token, expert, weight)]."""
    out = torch.zeros_like(x)
    by_expert = {}
    for t, e, w in pairs:
        by_expert.setdefault((e, 0), []).append((t, w))
    if shared_tokens:
        by_expert[0xFFFF, 14] = [(t, 1.0) for t in shared_tokens]     # (the shared expert's segments are 14, 15, 16)
    for (e, seg), use in by_expert.items():
        rows = torch.tensor([t for t, _ in use], device=x.device)
        xe = x[rows]
        act = torch.nn.functional.silu(xe @ _matrix64(model, layer, e, seg + 1).T) * (xe @ _matrix64(model, layer, e, seg).T)
        y = act @ _matrix64(model, layer, e, seg + 2).T
        out.index_add_(0, rows, y * torch.tensor([w for _, w in use], device=x.device, dtype=torch.float64)[:, None])
    return out


def _route64(sh, x, w, offset, bias):
    logits = x @ w.double().T
    if offset is not None:
        logits = logits + offset.double()
    if sh.scoring == SCORING_SOFTMAX:
        top, ids = torch.topk(logits, sh.top_k, dim=1)
        return ids, torch.softmax(top, dim=1)
    score = torch.sigmoid(logits)
    ids = torch.topk(score if bias is None else score + bias.double(), sh.top_k, dim=1).indices
    wt = score.gather(1, ids)
    return ids, wt / wt.sum(1, keepdim=True) * sh.scaling_factor


def exact(case, seed):
    """What run returns, in 64 bits from the dequantised pages; expert ids, which are whole numbers, are left out."""
    s = prepare(case, seed)
    kind, sh, L, T, model = s["kind"], s["sh"], s["L"], s["T"], s["model"]
    (lo, hi), outs, weights = s["range"], [], None
    model.by_expert = {}
    for p in model.pages:
        model.by_expert.setdefault((p.pid.layer, p.pid.expert), []).append(p)
    for l in range(L):
        x, h = s["xs"][l].double(), None
        if kind == "stack":
            h = s["h0"][l].double() + s["attn"][l].double()
            # (the sublayer's input is rounded to its activation type on the way)
            x = (h / torch.sqrt((h * h).mean(1, keepdim=True) + 1e-6) * s["norm"][l].double()).to(s["x"].dtype).double()
        if kind == "ep_pairs":
            ids, wt = s["ids"][l][:, :sh.top_k].long(), s["w"][l][:, :sh.top_k].double()
        else:
            ids, wt = _route64(sh, x, s["w16"][0] if kind == "paged" else model.router_w[l], s["offset"], s["bias"])
        weights = wt
        pairs = [(t, e, w) for t, (es, ws) in enumerate(zip(ids.tolist(), wt.tolist())) for e, w in zip(es, ws) if lo <= e < hi]
        shared = [] if not sh.shared_experts or kind == "ep_share" else [1] if kind == "ep_pairs" else range(T)
        out = _experts64(model, l, x, pairs, shared)
        outs.append(out if h is None else h + out)
    if kind == "step_host":
        return [o[0].cpu() for o in outs]
    if kind == "layer":
        return torch.cat(outs), None
    if kind in ("stack", "ep_pairs"):
        return torch.stack(outs)
    if kind == "tokens":
        full = torch.zeros(T, s["gd"].weights.shape[1], dtype=torch.float64, device=x.device)
        full[:, :sh.top_k] = weights
        return outs[0], None, full
    if kind == "ep_share":
        return outs[0], None
    return outs[0][0], None, weights[0].cpu().numpy()
