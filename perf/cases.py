"""What a user of this library has it do, as cases that can be timed: passes of a speculative decoder, prompts, batched steps, and the
operators that are called on their own.  Every case goes through the package's public calls.

Models and shapes are the benchmark's: `c3` (48 layers, 512 experts top-10, EXL3 3-bit experts, Q8_0 projections, EXL3 4-bit head
screened by its 2-bit proxy, Q8_KV cache) and `tiny` (4 layers, everything Q8_0).  The weights of a model are laid out once a process
and serve every session of it, as in a server; what a seed decides is the conversation: history, tokens, activations."""
import numpy as np
import torch

import __graft_entry__ as graft

pkg = graft.load_package()
md, lib, synth = pkg.model, pkg.lib, pkg.synth

C3 = dict(n_layer=48, hidden=2048, streams=4, hc_rank=256, vocab=151936, n_head=16, n_kv_head=2, head_dim=256, rope_dims=64,
          n_expert=512, n_expert_used=10, expert_ff=512, shared_ff=512, ssm_k_heads=16, ssm_v_heads=32, ssm_head_dim=128, conv_k=4,
          attn_interval=4, eps=1e-6, rope_theta=1e7)
MODELS = {"c3": C3, "tiny": md.TINY}
MOE = {"c2": dict(hidden=2048, n_expert=512, top_k=10, expert_ff=512, shared_ff=512),      # benchmark config 2
       "c1": dict(hidden=512, n_expert=32, top_k=4, expert_ff=256, shared_ff=512)}         # benchmark config 1
TYPES = {"exl3": lib.TYPE_EXL3(3), "iq3_s": lib.TYPE_IQ3_S, "q8_0": lib.TYPE_Q8_0}
TREE = [-1, 0, 0, 0, 1, 1, 4, 6]       # benchmark config 4's draft tree, as many rows as a pass holds
REQUEST = 256                          # positions a request decodes before the next one takes its session
#: The Q8_0 projections of a c3 layer: qkv + gate of a DeltaNet layer together, qkv, gate, the output projection, an attention layer's k.
PROJECTIONS = [(12288, 2048), (8192, 2048), (4096, 2048), (2048, 4096), (512, 2048)]


def listed():
    return [
        # the smallest thing a session does: a verify pass of the tiny model early in a conversation (launches, host path)
        {"name": "tiny-pass-4", "kind": "pass", "model": "tiny", "rows": 4, "ctx": 256},
        # decoding one conversation at the headline context: nothing to draft (1 row), and K = 3 drafts (4 rows)
        {"name": "pass-1", "kind": "pass", "model": "c3", "rows": 1, "ctx": 24576},
        {"name": "pass-4", "kind": "pass", "model": "c3", "rows": 4, "ctx": 24576},
        # a draft tree, the widest pass there is
        {"name": "tree-8", "kind": "tree", "model": "c3", "rows": 8, "ctx": 24576},
        # a conversation's prompt, of a length that is no multiple of anything
        {"name": "prompt-507", "kind": "prompt", "model": "c3", "tokens": 507, "ctx": 0},
        # serving: many conversations stepped together at benchmark config 5's contexts, and their prompts fed together
        {"name": "step-32", "kind": "step", "model": "c3", "sequences": 32, "ctx": 15000},
        {"name": "feed-16", "kind": "feed", "model": "c3", "sequences": 16, "tokens": 75},
        # the MoE sublayer on its own, for a host with its own session: a verify pass's 4 rows in two expert formats, a batch's 256 rows
        {"name": "moe-exl3-4", "kind": "moe", "shape": "c2", "format": "exl3", "rows": 4},
        {"name": "moe-iq3s-4", "kind": "moe", "shape": "c2", "format": "iq3_s", "rows": 4},
        {"name": "moe-rows-256", "kind": "rows", "shape": "c2", "rows": 256},
        # a projection over the rows of a batch and over a long prompt
        {"name": "cols-256", "kind": "cols", "rows": 12288, "cols": 2048, "tokens": 256},
        {"name": "cols-4093", "kind": "cols", "rows": 12288, "cols": 2048, "tokens": 4093},
    ]


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["pass", "pass", "tree", "prompt", "step", "feed", "moe", "moe", "rows", "cols", "cols"])
    if kind in ("pass", "tree"):
        model = rng.choice(["c3", "c3", "tiny"])
        return {"kind": kind, "model": model, "rows": rng.randint(1 if kind == "pass" else 3, 8), "ctx": _spread(rng, 200, 24576 if model == "c3" else 4000)}
    if kind == "prompt":
        return {"kind": kind, "model": rng.choice(["c3", "c3", "tiny"]), "tokens": _spread(rng, 20, 507), "ctx": rng.choice([0, _spread(rng, 256, 9600)])}
    if kind == "step":
        return {"kind": kind, "model": "c3", "sequences": _spread(rng, 2, 32), "ctx": _spread(rng, 500, 15000)}
    if kind == "feed":
        return {"kind": kind, "model": "c3", "sequences": rng.randint(2, 16), "tokens": _spread(rng, 20, 75)}
    if kind == "moe":
        return {"kind": kind, "shape": rng.choice(["c2", "c2", "c1"]), "format": rng.choice(sorted(TYPES)), "rows": rng.randint(1, 8)}
    if kind == "rows":
        return {"kind": kind, "shape": "c2", "rows": 8 * rng.randint(1, 32)}
    rows, cols = rng.choice(PROJECTIONS)
    return {"kind": kind, "rows": rows, "cols": cols, "tokens": _spread(rng, 1, 4093)}


# ---- what a program lays out once ----------------------------------------------------------------------------------------------------
_once = {}


def _model(name):
    """The model in HBM and its token cycles' successor table.  The four kinds of weights that a layer of `c3` can have (three DeltaNet
    layers and one of attention) are made once and every later layer is a copy of its own of them: 33 GB that a pass streams."""
    if name not in _once:
        cfg = MODELS[name]
        if name == "c3":
            M = md.make_model(dict(cfg, n_layer=4), dense_type=lib.TYPE_Q8_0, expert_type=TYPES["exl3"], seed=1, device="cuda",
                              cycle_alpha=0.95, cycle_beta=0.7, head_type=lib.TYPE_EXL3(4))
            for l in range(4, cfg["n_layer"]):
                for key in [k for k in M["tensors"] if k.startswith("blk.%d." % (l % 4))]:
                    M["tensors"]["blk.%d.%s" % (l, key.split(".", 2)[2])] = M["tensors"][key]
                M["moe"].append(M["moe"][l % 4])
            M["cfg"]["n_layer"] = cfg["n_layer"]
        else:
            M = md.make_model(cfg, seed=1, device="cuda", cycle_alpha=0.95, cycle_beta=0.7)
        _once[name] = (md.DeviceModel(M, "cuda:0"), md.token_cycles(cfg["vocab"], 1)[0].numpy())
        del M
        torch.cuda.empty_cache()
    return _once[name]


def _layers(shape, fmt):
    """A few MoE layers that calls take in turn, so that a call's experts come from HBM as they do inside a model."""
    key = (shape, fmt)
    if key not in _once:
        s = MOE[shape]
        _once[key] = [pkg.moe.MoeLayer(synth.make_moe_layer(s["hidden"], s["n_expert"], s["top_k"], s["expert_ff"], s["shared_ff"], TYPES[fmt], TYPES[fmt],
                                                            seed=1 + i, device="cuda"), "cuda:0") for i in range(3 if fmt == "exl3" else 2)]
    return _once[key]


def _matrices(rows, cols):
    key = (rows, cols)
    if key not in _once:
        n = max(2, min(12, (200 << 20) // (rows * cols)))      # larger together than L2 where a dozen can be
        _once[key] = [synth.quantize_q8_0(synth.normal((rows, cols), 0.02, 1 + i, "projection", "cuda")).reshape(-1) for i in range(n)]
    return _once[key]


# ---- one case ------------------------------------------------------------------------------------------------------------------------
def _contexts(case, seed):
    """The history of every sequence of a step: a short, a middle and a long one in turn (benchmark config 5: 3k, 9.6k, 15k)."""
    r = np.random.default_rng(seed)
    return [max(16, int(case["ctx"] * (0.2, 0.64, 1.0)[int(k)])) for k in r.integers(0, 3, case["sequences"])]


def _prompt(n, vocab, seed):
    return md.make_prompt(n, vocab, seed=seed, cycles=_once["cycles", vocab])


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("pass", "tree", "prompt", "step", "feed"):
        dm, succ = _model(case["model"])
        vocab, proxy = MODELS[case["model"]]["vocab"], case["model"] == "c3"
        if ("cycles", vocab) not in _once:
            _once["cycles", vocab] = md.token_cycles(vocab, 1)[1]
        s = {"kind": kind, "rng": np.random.default_rng(seed), "succ": succ, "vocab": vocab, "seed": seed}
        if kind in ("pass", "tree"):
            s.update(sess=md.Session(dm, case["ctx"] + REQUEST + 64, head_proxy=proxy), rows=case["rows"], ctx=[case["ctx"]], next=[int(s["rng"].integers(0, vocab))])
            s["sess"].fill_synthetic(case["ctx"], seed=seed)
        elif kind == "prompt":
            s.update(sess=md.Session(dm, case["ctx"] + case["tokens"] + 64, head_proxy=proxy), ctx=[case["ctx"]], prompt=_prompt(case["tokens"], vocab, seed))
        else:
            n = case["sequences"]
            s["ctx"] = _contexts(case, seed) if kind == "step" else [0] * n
            s["batch"] = md.Batch(dm, n, max(s["ctx"]) + (REQUEST if kind == "step" else case["tokens"]) + 64, head_proxy=proxy,
                                  rows_max=min(256, 8 * n))
            if kind == "step":
                s["next"] = [int(t) for t in s["rng"].integers(0, vocab, n)]
                for sess, ctx in zip(s["batch"].sessions, s["ctx"]):
                    sess.fill_synthetic(ctx, seed=seed)
            else:   # prompts of different lengths, up to the case's
                s["prompts"] = [_prompt(max(4, case["tokens"] - int(s["rng"].integers(0, case["tokens"] // 2))), vocab, seed + 17 * b) for b in range(n)]
        return s
    if kind in ("moe", "rows"):
        layers = _layers(case["shape"], case.get("format", "exl3"))
        x = synth.normal((15 if kind == "moe" else 4, case["rows"], MOE[case["shape"]]["hidden"]), 1.0, seed, "x", "cuda").to(torch.bfloat16).float()
        return {"kind": kind, "layers": layers, "x": [v.contiguous() for v in x], "turn": 0}
    x = synth.normal((case["tokens"], case["cols"]), 1.0, seed, "x", "cuda")
    return {"kind": kind, "ops": [pkg.mma_cols.MmaCols(w, case["rows"], case["cols"], case["tokens"]) for w in _matrices(case["rows"], case["cols"])], "x": x, "turn": 0}


def _drafts(s, nxt, rows):
    """The pass's own token and the drafts after it: the model's habit (the next tokens of the cycle), which it follows most of the time."""
    ids = [nxt]
    for _ in range(rows - 1):
        ids.append(int(s["succ"][ids[-1]]))
    return ids


def _read(sess):
    """The pass's result and its commit, as the decoder's loop does it: (rows kept, next token), the rows' top-64 values and ids."""
    (keep, nxt), top, _ = sess.result()
    sess.commit(keep)
    return keep, nxt, [np.array([keep, nxt]), top[:, :64].view(np.float32), top[:, 64:].astype(np.int64)]


def run(state):
    s = state
    kind = s["kind"]
    if kind in ("pass", "tree"):
        sess = s["sess"]
        if len(sess) + 8 > s["ctx"][0] + REQUEST:      # the request is done: the next one's history
            sess.fill_synthetic(s["ctx"][0], seed=s["seed"])
        if kind == "pass":
            sess.verify(_drafts(s, s["next"][0], s["rows"]), accept=1)
        else:                                          # draft tokens uniform over the vocabulary
            sess.verify_tree([s["next"][0]] + [int(t) for t in s["rng"].integers(0, s["vocab"], s["rows"] - 1)], TREE[:s["rows"]], accept=1)
        _, s["next"][0], out = _read(sess)
        return out
    if kind == "prompt":
        sess = s["sess"]
        if s["ctx"][0]:
            sess.fill_synthetic(s["ctx"][0], seed=s["seed"])
        else:
            sess.reset()
        sess.prefill(s["prompt"])
        _, top, _ = sess.result()
        sess.commit(top.shape[0])
        sess.verify([int(top[-1, 64])], accept=1)      # and the first step of the answer, which stands on all the prompt left behind
        return _read(sess)[2] + [top[-1:, :64].view(np.float32), top[-1:, 64:].astype(np.int64)]
    if kind == "step":
        ss = s["batch"].sessions
        for sess, ctx in zip(ss, s["ctx"]):
            if len(sess) + 8 > ctx + REQUEST:
                sess.fill_synthetic(ctx, seed=s["seed"])
        s["batch"].verify([_drafts(s, t, 1 + b % 4) for b, t in enumerate(s["next"])], accept=1)      # some drafted, some had nothing to draft
        out = []
        for b, sess in enumerate(ss):
            _, s["next"][b], o = _read(sess)
            out.append(o)
        return [np.concatenate(v) for v in zip(*out)]
    if kind == "feed":
        ss = s["batch"].sessions
        for sess in ss:
            sess.reset()
        s["batch"].prefill(s["prompts"])
        out = []
        for sess in ss:
            _, top, _ = sess.result()
            sess.commit(top.shape[0])
            out.append([top[-1:, :64].view(np.float32), top[-1:, 64:].astype(np.int64)])   # the last row's are the prompt's
        return [np.concatenate(v) for v in zip(*out)]
    turn, s["turn"] = s["turn"], s["turn"] + 1
    if kind == "cols":
        return s["ops"][turn % len(s["ops"])](s["x"])
    layer, x = s["layers"][turn % len(s["layers"])], s["x"][turn % len(s["x"])]
    return layer.moe_batch(x) if kind == "moe" else layer.moe_rows(x)


# ---- what a case cannot do without ---------------------------------------------------------------------------------------------------
def _expert_bytes(shape, fmt):
    """Bytes of one expert's three matrices."""
    h, f = shape["hidden"], shape["expert_ff"]
    n = 3 * h * f
    return n * 3 // 8 + 3 * (2 * (h + f) + 4) if fmt == "exl3" else n // 256 * 110 if fmt == "iq3_s" else n // 32 * 34


def _moe_work(shape, fmt, rows):
    """Every expert that some row chose once (as many as independent rows choose of them), the shared expert, the router."""
    h, f, ne, k = shape["hidden"], shape["expert_ff"], shape["n_expert"], shape["top_k"]
    distinct = ne * (1 - (1 - k / ne) ** rows)
    one, shared = _expert_bytes(shape, fmt), _expert_bytes(dict(shape, expert_ff=shape["shared_ff"]), fmt)
    return {"bytes": distinct * one + shared + 4 * (ne + 1) * h + 8 * rows * h, "flops": 2 * rows * (3 * h * (k * f + shape["shared_ff"]) + ne * h)}


def _session_work(model, seqs):
    """One pass over every (rows, history, rows with a head) of `seqs`: all weights once, each sequence's cache and recurrent state once."""
    c = MODELS[model]
    fmt = "exl3" if model == "c3" else "q8_0"
    h, vocab, hd = c["hidden"], c["vocab"], c["head_dim"]
    ch = c["streams"] * h
    rows, heads = sum(q[0] for q in seqs), sum(q[2] for q in seqs)
    n_attn = c["n_layer"] // c["attn_interval"]
    n_delta = c["n_layer"] - n_attn
    kd, vd = c["ssm_k_heads"] * c["ssm_head_dim"], c["ssm_v_heads"] * c["ssm_head_dim"]
    qd, kvd = c["n_head"] * hd, c["n_kv_head"] * hd
    hyper = 2 * (2 * c["hc_rank"] + c["streams"]) * ch                       # two reads a layer, bf16
    dense = n_delta * h * (2 * kd + 3 * vd + 2 * c["ssm_v_heads"]) + n_attn * h * (3 * qd + 2 * kvd)
    moe = _moe_work(dict(hidden=h, n_expert=c["n_expert"], top_k=c["n_expert_used"], expert_ff=c["expert_ff"], shared_ff=c["shared_ff"]), fmt, rows)
    head = vocab * h // 4 + vocab * (h // 128) * 2 + min(1187, 128 * heads) * 128 * h // 2 if model == "c3" else vocab * h // 32 * 34
    state = 2 * 4 * (c["ssm_v_heads"] * c["ssm_head_dim"] ** 2 + (c["conv_k"] - 1) * (2 * kd + vd))
    cache = 2 * c["n_kv_head"] * (hd + (hd // 32 * 2 + 15) // 16 * 16)        # K and V of a position in a layer
    past = sum(n * past + n * (n + 1) // 2 for n, past, _ in seqs)             # (row, position) pairs attention looks at
    return {"bytes": c["n_layer"] * (moe["bytes"] + 2 * hyper) + dense * 34 // 32 + head + rows * h * 34 // 32 + 512 * heads +
            len(seqs) * n_delta * state + n_attn * cache * sum(n + p for n, p, _ in seqs),
            "flops": c["n_layer"] * (moe["flops"] + 2 * rows * hyper) + 2 * rows * dense + 2 * heads * vocab * h +
            n_attn * 4 * past * qd + n_delta * rows * 8 * c["ssm_v_heads"] * c["ssm_head_dim"] ** 2}


def work(case):
    kind = case["kind"]
    if kind in ("pass", "tree"):
        return _session_work(case["model"], [(case["rows"], case["ctx"], case["rows"])])
    if kind == "prompt":
        return _session_work(case["model"], [(case["tokens"], case["ctx"], (case["tokens"] - 1) % 8 + 1)])
    if kind == "step":
        return _session_work(case["model"], [(1 + b % 4, int(case["ctx"] * 0.61), 1 + b % 4) for b in range(case["sequences"])])
    if kind == "feed":
        return _session_work(case["model"], [(case["tokens"] * 3 // 4, 0, 4)] * case["sequences"])
    if kind in ("moe", "rows"):
        return _moe_work(MOE[case["shape"]], case.get("format", "exl3"), case["rows"])
    r, c, n = case["rows"], case["cols"], case["tokens"]
    return {"bytes": r * c // 32 * 34 + 4 * n * (r + c), "flops": 2 * n * r * c}


def tolerance(case):
    """Exact weights, 32-bit sums: 1e-5 for one operator (the projections take f16 inputs by definition, with 32-bit sums).  A whole
    pass sends such differences through up to 48 layers, where two experts or two tokens of nearly the same weight may change places."""
    if case["kind"] in ("moe", "rows", "cols"):
        return {"rel": 1e-5}
    return {"rel": 1e-3, "differ": 0.01}
