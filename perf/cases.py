"""The work that is measured: what a program of this framework has the GPU do, through its public entry points.

Kinds of case, and what each stands for in real use:

* ``step``     one whole decode or verify step (embedding, every layer, head, commit) as a captured graph: what ``generate``
               replays for every token.  Returns the logits, the new K/V rows and the recurrent states.
* ``prefill``  a whole ``DecodeEngine.prefill`` call on a prompt: wide chunks, then 8-row steps for the rest.  Returns the
               state that it leaves (K/V rows, recurrent states) and the logits of its last step.
* ``gdn``, ``attn``, ``moe``   layers of one kind (``Gdn.forward``, ``FullAttn.forward``, ``Moe.forward``) on 1..8 token rows:
               one row is plain decode, 2..4 the MTP verify, 8 the DFlash verify and the chunked prefill.
* ``head``     final norm, logits, sampling and commit (``Head.forward``).
* ``linear``   quantise a block of token rows and multiply it with a projection of the checkpoint
               (``ops.tc_gemm.act_quant`` + ``fp8_gemm``): every projection of a prefill chunk.

``tp`` is the width of the tensor-parallel group whose rank-0 shard is run (one process, no exchange): 8 is the deployment
of the served model, 1 the single-GPU configuration of ``bench.py``.  A layer case runs a few layers with weights, rows and
caches of their own one after the other, as a program that owns a stack does, so that the weights come from memory and not
from the L2 cache that the pass before left; a captured graph of the pass is what such a program keeps.  Weights are
N(0, 0.02) in e4m3 with 128 x 128 block scales, the initialisation of this repository's benchmark.
"""

import math

import torch

from nexrt_b200.attn import FullAttn
from nexrt_b200.config import ShardSpec, full_config
from nexrt_b200.decode_engine import DecodeEngine
from nexrt_b200.gdn import Gdn
from nexrt_b200.head import Head
from nexrt_b200.moe import Moe
from nexrt_b200.ops.tc_gemm import act_quant, fp8_gemm
from nexrt_b200.runtime.capture import graph_capture
from nexrt_b200.runtime.context import StepContext
from nexrt_b200.runtime.control import Ctl
from nexrt_b200.weights import random_rank_model

DEV = torch.device("cuda", 0)
FP8 = torch.float8_e4m3fn
CFG = full_config()
H = CFG.hidden
MAX_KEYS = 256 * 1024   # the served model's context length


def listed():
    return [
        # the single-GPU benchmark of this repository: 4 layers of the full width, one token at a 1K context
        {"name": "step_1row_tp1", "kind": "step", "tp": 1, "rows": 1, "keys": 1024, "layers": 4},
        # a short chat prompt: five 64-row chunks, one 8-row step and a ragged one
        {"name": "prefill_333_tp8", "kind": "prefill", "tp": 8, "tokens": 333, "wide": 64, "layers": 4},
        # plain decode in the deployment: the smallest calls, where latency counts
        {"name": "gdn_1row_tp8", "kind": "gdn", "tp": 8, "rows": 1, "layers": 4},
        {"name": "attn_1row_1k_tp8", "kind": "attn", "tp": 8, "rows": 1, "keys": 1024, "layers": 4},
        {"name": "moe_1row_tp8", "kind": "moe", "tp": 8, "rows": 1, "layers": 4},
        {"name": "head_1row_tp8", "kind": "head", "tp": 8, "rows": 1, "temperature": 0.0},
        # plain decode behind a book-length document
        {"name": "attn_1row_200k_tp8", "kind": "attn", "tp": 8, "rows": 1, "keys": 200000, "layers": 1},
        # the 4-row MTP verify and the 8-row DFlash verify
        {"name": "moe_4rows_tp8", "kind": "moe", "tp": 8, "rows": 4, "layers": 4},
        {"name": "gdn_8rows_tp8", "kind": "gdn", "tp": 8, "rows": 8, "layers": 4},
        {"name": "attn_8rows_32k_tp8", "kind": "attn", "tp": 8, "rows": 8, "keys": 32768, "layers": 2},
        {"name": "moe_8rows_tp8", "kind": "moe", "tp": 8, "rows": 8, "layers": 4},
        # the attention front of a 64-row prefill chunk on a two-GPU shard, exact three-term activations
        {"name": "linear_64rows", "kind": "linear", "rows": 64, "out": 10240, "terms": 3},
    ]


def draw(rng):
    # no attention layer on exactly two rows: its front refuses them (a launch error), as the step and the ragged end of a prompt do
    kind = rng.choice(["gdn", "gdn", "attn", "attn", "attn", "moe", "moe", "moe", "head", "linear", "step", "prefill"])
    tp = rng.choice([1, 2, 4, 8, 8])
    rows = rng.choice([1, 1, 3, 4, 4, 5, 6, 7, 8, 8])
    layers = max(1, tp // 2)
    std = round(math.exp(rng.uniform(math.log(0.02), math.log(2.0))), 4)      # the residual rows grow along the stack
    if kind == "gdn":
        return {"kind": kind, "tp": tp, "rows": rng.choice([rows, rows, 2]), "layers": layers, "position": 16 * rng.randint(0, 8000) + rng.randint(0, 8), "std": std}
    if kind == "moe":
        return {"kind": kind, "tp": tp, "rows": rng.choice([rows, rows, 2]), "layers": layers, "std": std}
    if kind == "attn":
        keys = int(round(math.exp(rng.uniform(math.log(16), math.log(MAX_KEYS - 16)))))
        return {"kind": kind, "tp": tp, "rows": rows, "keys": keys, "layers": 1 if keys > 65536 else max(1, layers // 2), "std": std}
    if kind == "head":
        return {"kind": kind, "tp": tp, "rows": rows, "temperature": rng.choice([0.0, 0.6, 0.9]), "std": std}
    if kind == "linear":
        return {"kind": kind, "rows": rng.choice([16, 24, 32, 64, 96, 128]), "out": 128 * rng.randint(8, 160), "terms": rng.choice([1, 2, 3])}
    if kind == "step":
        return {"kind": kind, "tp": 8, "rows": rows, "keys": rng.randint(32, 8192), "layers": rng.choice([1, 2, 4])}
    return {"kind": kind, "tp": 8, "tokens": rng.choice([n for n in range(70, 333) if n % 8 != 2]), "wide": rng.choice([0, 64, 64, 128]), "layers": 4}


# ---- inputs: plain torch, from the seed alone -------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 11)


def _randn(g, *shape, std=0.02):
    return torch.randn(*shape, generator=g, device=DEV) * std


def _fp8(g, *shape):
    """N(0, 0.02) matrices ``[..., R, C]`` as e4m3 with one fp32 scale per 128 x 128 block."""
    *lead, R, C = shape
    n = math.prod(lead)
    q = torch.empty(n, R, C, dtype=FP8, device=DEV)
    s = torch.empty(n, R // 128, C // 128, device=DEV)
    step = max(1, (1 << 27) // (R * C))
    for i in range(0, n, step):
        m = min(step, n - i)
        w = _randn(g, m, R // 128, 128, C // 128, 128)
        sc = w.abs().amax(dim=(2, 4)) / 448.0
        s[i : i + m] = sc
        q[i : i + m] = (w / sc[:, :, None, :, None]).to(FP8).view(m, R, C)
    return q.view(*shape), s.view(*lead, R // 128, C // 128)


POSITION = 16 * 61 + 3   # committed length of a layer case without a context of its own: odd, its rows do not wrap in the rings
STD = 0.1                # residual rows early in the stack, where what a layer adds weighs more than what it is added to


def _gdn_weights(g, spec):
    nv, C = spec.gdn_v, spec.gdn_qkv_rows
    fw, fs = _fp8(g, spec.gdn_front_rows, H)
    ow, os_ = _fp8(g, H, spec.gdn_local)
    return {
        "kind": "linear", "in_ln": 1.0 + _randn(g, H), "front_w": fw, "front_s": fs, "ba_w": _randn(g, 2 * nv, H).bfloat16(),
        "conv_w": _randn(g, C, 4, std=0.2).bfloat16().float(), "a_log": _randn(g, nv), "dt_bias": _randn(g, nv),
        "gnorm_w": (1.0 + _randn(g, 128)).bfloat16().float(), "out_w": ow, "out_s": os_,
    }


def _gdn_state(g, spec):
    """What the layer holds after some tokens: the last three pre-convolution rows and the recurrent state."""
    return _randn(g, spec.gdn_qkv_rows, 3, std=1.0), _randn(g, spec.gdn_v, 128, 128, std=0.05)


def _attn_weights(g, spec):
    hd = CFG.head_dim
    fw, fs = _fp8(g, spec.attn_front_rows, H)
    ow, os_ = _fp8(g, H, spec.attn_local)
    return {"kind": "full", "in_ln": 1.0 + _randn(g, H), "front_w": fw, "front_s": fs, "qn": 1.0 + _randn(g, hd), "kn": 1.0 + _randn(g, hd),
            "out_w": ow, "out_s": os_}


def _attn_cache(g, spec, keys):
    """K rows are normalised per head (unit rms), V rows have the spread of the projection."""
    shape = (spec.kv_heads, keys, CFG.head_dim)
    return torch.randn(shape, generator=g, device=DEV).bfloat16(), (torch.randn(shape, generator=g, device=DEV) * 1.3).bfloat16()


def _moe_weights(g, spec):
    E, I = CFG.n_experts, spec.inter
    w13, w13s = _fp8(g, E + 1, 2 * I, H)
    w2, w2s = _fp8(g, E + 1, H, I)
    return {"post_ln": 1.0 + _randn(g, H), "router_w": _randn(g, E + 1, H).bfloat16(), "w13": w13, "w13_s": w13s, "w2": w2, "w2_s": w2s}


def _rows(g, case):
    return _randn(g, case["rows"], H, std=case.get("std", STD)).bfloat16()


def _head_weights(g, spec):
    return {"final_ln": 1.0 + _randn(g, H), "lm_head": _randn(g, spec.vocab, H).bfloat16()}


# ---- what a program keeps ---------------------------------------------------------------------------------------------
def _context(spec):
    return StepContext(CFG, spec, DEV, comm_world=1, comm_rank=0)


def _captured(fn):
    """A graph of one pass, after an eager one (the launchers' lazy initialisation must not run under capture)."""
    side = torch.cuda.Stream(DEV)
    side.wait_stream(torch.cuda.current_stream(DEV))
    with torch.cuda.stream(side):
        fn()
    torch.cuda.synchronize(DEV)
    graph = torch.cuda.CUDAGraph()
    with graph_capture(graph, side):
        fn()
    torch.cuda.synchronize(DEV)
    return graph


def _prepare_layers(case, seed):
    kind, M = case["kind"], case["rows"]
    spec = ShardSpec(CFG, case["tp"], 0)
    g = _gen(seed)
    ctxs, blocks, outs = [], [], []
    x = torch.zeros(case["layers"], 8, H, dtype=torch.bfloat16, device=DEV)     # the residual rows of every layer
    rows = torch.zeros(case["layers"], M, H, dtype=torch.bfloat16, device=DEV)
    for i in range(case["layers"]):
        c = _context(spec)
        c.x = x[i]
        if kind == "gdn":
            P = case.get("position", POSITION)
            b = Gdn(c, _gdn_weights(g, spec), state_ring=9)
            b.load_state(P, *_gdn_state(g, spec))
            outs.append([c.x[:M], b.state_ring[(P + M) % 9], b.conv_ring[P % 16 : P % 16 + M]])
        elif kind == "attn":
            P = case["keys"]
            b = FullAttn(c, _attn_weights(g, spec), cache_len=P + 16)
            b.load_kv(*_attn_cache(g, spec, P))
            outs.append([c.x[:M], b.k_cache[:, P : P + M], b.v_cache[:, P : P + M]])
        else:
            P = POSITION
            b = Moe(c, _moe_weights(g, spec))
            outs.append([c.x[:M]])
        c.ctl[Ctl.COMMITTED_LEN] = P
        rows[i] = _rows(g, case)
        ctxs.append(c)
        blocks.append(b)

    def one_pass():
        x[:, :M].copy_(rows)                # the layers' input rows (a layer adds its output to them)
        for b in blocks:
            b.forward(M)

    return {"graph": _captured(one_pass), "outs": outs, "keep": (ctxs, blocks, x, rows)}


def _prepare_head(case, seed):
    M = case["rows"]
    spec = ShardSpec(CFG, case["tp"], 0)
    g = _gen(seed)
    c = _context(spec)
    w = _head_weights(g, spec)
    rows = _rows(g, case)
    head = Head(c, w)
    if case["temperature"] > 0:
        head.set_sampling_config(int(seed) + 1, case["temperature"], 0.95, 20)
    logits = head.enable_logits()
    c.x[:M] = rows
    ctl = c.ctl.clone()
    ctl[Ctl.COMMITTED_LEN] = POSITION

    def one_pass():
        c.ctl.copy_(ctl)                    # the head commits: the control block of this step
        head.forward(M)

    return {"graph": _captured(one_pass), "outs": [logits[:M], c.ctl[Ctl.EMITTED : Ctl.EMITTED + 1]], "keep": (c, head, ctl)}


def _prepare_linear(case, seed):
    g = _gen(seed)
    wq, sw = _fp8(g, case["out"], H)
    x = torch.randn(case["rows"], H, generator=g, device=DEV).bfloat16()
    gamma = 1.0 + _randn(g, H)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    return {"linear": (x, gamma, wq, sw, status), "terms": case["terms"]}


def _engine(case, seed, keys):
    cfg = CFG.truncated(case["layers"])
    model = random_rank_model(cfg, case["tp"], 0, DEV, seed=int(seed))
    eng = DecodeEngine(0, 1, DEV, ext=model, cfg=cfg, shape_tp=case["tp"], max_rows=8, cache_len=keys + 64)
    eng.head.enable_logits()
    return cfg, eng


def _prepare_step(case, seed):
    M, P = case["rows"], case["keys"]
    cfg, eng = _engine(case, seed, P)
    g = _gen(seed)
    layers = {}
    for i, m in enumerate(eng.mixers):
        if isinstance(m, FullAttn):
            k, v = _attn_cache(g, eng.spec, P)
            layers[i] = {"k_cache": k, "v_cache": v}
        else:
            conv, state = _gdn_state(g, eng.spec)
            layers[i] = {"conv_state": conv, "recurrent_state": state}
    ids = torch.randint(0, cfg.vocab, (M,), generator=g, device=DEV).tolist()
    eng.load_prefill({"L": P, "first_token": ids[0], "layers": layers})
    eng.set_rows(ids)
    graph = eng.capture(M)
    outs = [eng.head.logits[:M]]
    for m in eng.mixers:
        outs.append([m.k_cache[:, P : P + M], m.v_cache[:, P : P + M]] if isinstance(m, FullAttn) else [m.state_ring[(P + M) % m.state_ring_len]])
    return {"step": (eng, graph, eng.ctx.ctl.clone()), "outs": outs}


def _prepare_prefill(case, seed):
    cfg, eng = _engine(case, seed, case["tokens"])
    g = _gen(seed)
    ids = torch.randint(0, cfg.vocab, (case["tokens"],), generator=g, device=DEV).tolist()
    eng.reset(first_token=ids[0])
    eng.capture(8)
    n = case["tokens"]
    outs = [eng.head.logits[(n - 1) % 8 if case["wide"] == 0 else (n - 1 - (n - 1) // case["wide"] * case["wide"]) % 8]]
    for m in eng.mixers:
        outs.append([m.k_cache[:, :n], m.v_cache[:, :n]] if isinstance(m, FullAttn) else [m.state_ring[n % m.state_ring_len]])
    return {"prefill": (eng, ids, case["wide"]), "outs": outs}


def prepare(case, seed):
    if case["kind"] in ("gdn", "attn", "moe"):
        return _prepare_layers(case, seed)
    return {"head": _prepare_head, "linear": _prepare_linear, "step": _prepare_step, "prefill": _prepare_prefill}[case["kind"]](case, seed)


def run(state):
    if "graph" in state:
        state["graph"].replay()
    elif "linear" in state:
        x, gamma, wq, sw, status = state["linear"]
        xq, sx = act_quant(x, gamma, CFG.rms_eps, state["terms"])
        y = fp8_gemm(wq, sw, xq, sx, status=status)
        return y if state["terms"] == 1 else y.view(state["terms"], x.shape[0], -1).sum(0)   # one row block per term
    elif "step" in state:
        eng, graph, ctl = state["step"]
        eng.ctx.ctl.copy_(ctl)              # the same step again: rings and caches are indexed by position
        graph.replay()
    else:
        eng, ids, wide = state["prefill"]
        eng.prefill(ids, wide=wide)
    return state["outs"]


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def _layer_work(kind, spec, M, keys=0):
    """(bytes, flops) of one layer: weights and caches read once, rows read and written once."""
    rows = 4.0 * M * H
    if kind == "gdn":
        w = spec.gdn_front_rows * H + H * spec.gdn_local
        st = 4.0 * spec.gdn_v * 128 * 128 * (M + 1)     # the state before the step and the one after every row
        return w * (1 + 4 / 16384) + 4.0 * spec.gdn_v * H + st + rows, 2.0 * M * w + 8.0 * M * spec.gdn_v * 128 * 128
    if kind == "attn":
        w = spec.attn_front_rows * H + H * spec.attn_local
        kv = 4.0 * spec.kv_heads * (keys + M) * CFG.head_dim
        return w * (1 + 4 / 16384) + kv + rows, 2.0 * M * w + 4.0 * M * spec.q_heads * (keys + M) * CFG.head_dim
    E, I, K = CFG.n_experts, spec.inter, CFG.top_k
    used = E * (1 - (1 - K / E) ** M) + 1               # distinct experts of M rows with independent routes
    return used * 3.0 * I * H * (1 + 4 / 16384) + 2.0 * (E + 1) * H + rows, 2.0 * M * (3.0 * I * H * (K + 1) + (E + 1) * H)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        T, R, P = case["rows"], case["out"], case["terms"]
        return {"bytes": R * H * (1 + 4 / 16384) + 2.0 * T * H + 4.0 * T * R, "flops": 2.0 * P * T * R * H}
    spec = ShardSpec(CFG, case["tp"], 0)
    if kind == "head":
        return {"bytes": 2.0 * spec.vocab * H + case["rows"] * (2.0 * H + 4.0 * spec.vocab), "flops": 2.0 * case["rows"] * spec.vocab * H}
    if kind in ("gdn", "attn", "moe"):
        b, f = _layer_work(kind, spec, case["rows"], case.get("keys", 0))
        return {"bytes": b * case["layers"], "flops": f * case["layers"]}
    if kind == "step":
        plan = [(case["rows"], case["keys"], 1)]
    else:
        chunk = case["wide"] or 8
        n = case["tokens"]
        whole = (n - 1) // chunk if case["wide"] else n // 8
        rest = n - whole * chunk
        plan = [(chunk, n // 2, whole)] + ([(8, n, rest // 8)] if rest >= 8 else []) + ([(rest % 8, n, 1)] if rest % 8 else [])
    total = {"bytes": 0.0, "flops": 0.0}
    for M, keys, times in plan:
        for kind_ in CFG.layer_types[: case["layers"]]:
            for part in ("attn" if kind_ == "full" else "gdn", "moe"):
                # a chunk keeps the recurrent state along its rows and writes the last one only
                b, f = _layer_work(part, spec, M, keys)
                if part == "gdn" and M > 8:
                    b -= 4.0 * spec.gdn_v * 128 * 128 * (M - 1)
                total["bytes"] += b * times
                total["flops"] += f * times
        if M <= 8:
            total["bytes"] += 2.0 * spec.vocab * H * times
            total["flops"] += 2.0 * M * spec.vocab * H * times
    return total


# ---- how far two correct implementations may be apart -----------------------------------------------------------------
def tolerance(case):
    kind = case["kind"]
    if kind == "linear":
        # fp32 sums in another order, and a scale one unit in the last place off turns a few roundings of the last term
        return {"rel": 2e-2 / 16 ** case["terms"], "max": 0.2 / 16 ** case["terms"]}
    if kind == "head":
        return {"rel": 2e-4, "max": 2e-3, "differ": 0.0}  # activations as bf16 hi + lo
    if kind in ("gdn", "attn", "moe"):
        return {"rel": 4e-3, "max": 4e-2}                 # results in bf16 (one unit in the last place is up to 2^-7 of a value)
    if kind == "step":
        return {"rel": 1e-2, "max": 0.1}                  # a change of rounding in one layer goes through all that follow
    return {"rel": 2e-2, "max": 0.9}                      # hundreds of tokens: a routing near tie may turn for one of them


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------
def _deq(q, s):
    return (q.double().unflatten(-2, (-1, 128)).unflatten(-1, (-1, 128)) * s.double()[..., :, None, :, None]).flatten(-2).flatten(-3, -2)


def _rms(x, w=None, eps=CFG.rms_eps):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return y if w is None else y * w.double()


def _silu(x):
    return x * torch.sigmoid(x)


def _exact_gdn(spec, M, x, w, conv, state):
    D, nqk, nv, C = 128, spec.gdn_qk, spec.gdn_v, spec.gdn_qkv_rows
    xn = _rms(x, w["in_ln"])
    pre = xn @ _deq(w["front_w"], w["front_s"]).T
    ba = xn @ w["ba_w"].double().T
    hist = torch.cat([conv.double().T, pre[:, :C]])
    y, S = [], state.double()
    for m in range(M):
        qkv = _silu((hist[m : m + 4].T * w["conv_w"].double()).sum(1))
        q, k, v = qkv[: nqk * D].view(nqk, D), qkv[nqk * D : 2 * nqk * D].view(nqk, D), qkv[2 * nqk * D :].view(nv, D)
        l2 = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)
        q, k = l2(q).repeat_interleave(nv // nqk, 0) * D**-0.5, l2(k).repeat_interleave(nv // nqk, 0)
        beta = torch.sigmoid(ba[m, :nv])
        decay = torch.exp(-torch.exp(w["a_log"].double()) * torch.nn.functional.softplus(ba[m, nv:] + w["dt_bias"].double()))
        S = S * decay[:, None, None]
        S = S + k[:, :, None] * ((v - (S * k[:, :, None]).sum(1)) * beta[:, None])[:, None, :]
        o = _rms((S * q[:, :, None]).sum(1)) * w["gnorm_w"].double() * _silu(pre[m, C:].view(nv, D))
        y.append(o.reshape(-1))
    return [x + torch.stack(y) @ _deq(w["out_w"], w["out_s"]).T, S.transpose(1, 2), pre[:, :C]]


def _exact_attn(spec, M, x, w, K, V):
    hd, nq, nk, P = CFG.head_dim, spec.q_heads, spec.kv_heads, K.shape[1]
    pre = _rms(x, w["in_ln"]) @ _deq(w["front_w"], w["front_s"]).T
    qg = pre[:, : 2 * nq * hd].view(M, nq, 2, hd)
    q, gate = _rms(qg[:, :, 0], w["qn"]), qg[:, :, 1]
    k, v = pre[:, 2 * nq * hd :].view(M, 2, nk, hd).unbind(1)
    k = _rms(k, w["kn"])
    half = CFG.rotary_dim // 2
    # position times inverse frequency in 32 bits, as the model defines its rotation
    inv = (1.0 / (CFG.rope_theta ** (torch.arange(0, CFG.rotary_dim, 2, dtype=torch.float32) / CFG.rotary_dim))).to(DEV)
    ang = (torch.arange(P, P + M, device=DEV, dtype=torch.float32)[:, None] * inv)[:, None].double()

    def rope(t):
        a, b = t[..., :half], t[..., half : 2 * half]
        return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin(), t[..., 2 * half :]], -1)

    q, k = rope(q), rope(k)
    ctx = torch.empty(M, nq, hd, dtype=torch.float64, device=DEV)
    for h in range(nk):
        Kh, Vh = torch.cat([K[h].double(), k[:, h]]), torch.cat([V[h].double(), v[:, h]])
        qs = q[:, h * (nq // nk) : (h + 1) * (nq // nk)]
        s = qs @ Kh.T * hd**-0.5
        s = s.masked_fill(torch.arange(P + M, device=DEV) > torch.arange(P, P + M, device=DEV)[:, None, None], -math.inf)
        ctx[:, h * (nq // nk) : (h + 1) * (nq // nk)] = torch.softmax(s, -1) @ Vh
    y = (ctx * torch.sigmoid(gate)).flatten(1) @ _deq(w["out_w"], w["out_s"]).T
    return [x + y, k.transpose(0, 1), v.transpose(0, 1)]


def _exact_moe(spec, M, x, w):
    E, I = CFG.n_experts, spec.inter
    xn = _rms(x, w["post_ln"])
    logits = xn @ w["router_w"].double().T
    tw, te = torch.softmax(logits[:, :E], -1).topk(CFG.top_k)
    tw = tw / tw.sum(-1, keepdim=True)
    y = x.clone()
    for m in range(M):
        for wt, e in [*zip(tw[m].tolist(), te[m].tolist()), (torch.sigmoid(logits[m, E]).item(), E)]:
            gu = _deq(w["w13"][e], w["w13_s"][e]) @ xn[m]
            y[m] += wt * (_deq(w["w2"][e], w["w2_s"][e]) @ (_silu(gu[:I]) * gu[I:]))
    return [y]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "prefill"):
        return None
    g = _gen(seed)
    if kind == "linear":
        wq, sw = _fp8(g, case["out"], H)
        x = torch.randn(case["rows"], H, generator=g, device=DEV).bfloat16()
        return _rms(x.double(), 1.0 + _randn(g, H)) @ _deq(wq, sw).T
    spec, M = ShardSpec(CFG, case["tp"], 0), case["rows"]
    if kind == "head":
        w = _head_weights(g, spec)
        xn = _rms(_rows(g, case).double(), w["final_ln"])
        return [torch.cat([xn @ part.double().T for part in w["lm_head"].split(16384)], 1), None]
    out = []
    for _ in range(case["layers"]):
        if kind == "gdn":
            w, st = _gdn_weights(g, spec), _gdn_state(g, spec)
            out.append(_exact_gdn(spec, M, _rows(g, case).double(), w, *st))
        elif kind == "attn":
            w, kv = _attn_weights(g, spec), _attn_cache(g, spec, case["keys"])
            out.append(_exact_attn(spec, M, _rows(g, case).double(), w, *kv))
        else:
            w = _moe_weights(g, spec)
            out.append(_exact_moe(spec, M, _rows(g, case).double(), w))
    return out
