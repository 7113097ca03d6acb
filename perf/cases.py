"""Performance cases of the token loop: the calls a serving program makes on a `Graph`, from one token of one
conversation to prompts of thousands of tokens and batches of many conversations.

Two checkpoints of the repository's own configurations, both with the draft layer: `a3b` (a 12-layer prefix of the
benchmark's 512-expert shape: nine DeltaNet and three attention layers, the mix of the whole) and `tiny`. Twelve layers
and not forty-eight, because routing is discrete: an expert at a near-tie falls either way in two correct
implementations, and every further layer spreads what that changed until their outputs say nothing about each other.
A server loads its checkpoint once and keeps it, so one synthetic model per configuration lives here for the whole
process; what changes with the seed is what changes from request to request: token ids, contexts, and the caches and
recurrent state behind them.

A case is a dict:
    model    "a3b" or "tiny"
    kind     "step"    one token of one conversation (Graph.extend), every logit back on the host
             "slots"   one token for each of `rows` conversations in one batched pass (Graph.decode_rows)
             "round"   one speculative round: `rows` - 1 draft steps and a verify pass of `rows` rows, half the drafts kept
             "prompt"  a new conversation of `rows` tokens (Graph.forward), cut into passes of `chunk` rows
             "turn"    `rows` further tokens of a conversation that already holds `context` cells (Graph.extend)
    rows     as above (1 for a step)
    context  cells the conversation holds before the pass; "slots": the longest, the others are drawn from a quarter of it up
    chunk    rows per pass the graph is created for (GraphOpts.max_tokens)
"""
import ctypes
import importlib

import numpy as np

pkg = importlib.import_module("strix-halo-vulkan_b200")

DRAFT_VOCAB = {"a3b": 65536, "tiny": 16384}   # ids the draft head projects onto (spec.DRAFT_VOCAB_DEFAULT; half of tiny's)
ROUTER_STD = 0.1                              # a trained router is decisive: its tenth expert weighs little beside its first
HEADROOM = 256                                # positions a decode case advances before it goes back to its start
_models = {}


def _case(name, model, kind, rows, context, chunk):
    c = dict(model=model, kind=kind, rows=rows, context=context, chunk=chunk)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call there is: one token through four small layers (latency and launches only)
        _case("tiny-step", "tiny", "step", 1, 100, 64),
        # one conversation being answered: the benchmark's headline step, after a prompt of 2048
        _case("step-2k", "a3b", "step", 1, 2048, 2048),
        # the same late in a long conversation
        _case("step-30k", "a3b", "step", 1, 30000, 2048),
        # a few conversations decode together (the largest group that shares the single-row schedule is eight)
        _case("slots-5", "a3b", "slots", 5, 3000, 64),
        # a small server's batch, between the single-row schedule and the tensor-core passes
        _case("slots-12", "a3b", "slots", 12, 12000, 64),
        # a busy server: the benchmark's 64 slots with contexts of 8 to 32 thousand cells
        _case("slots-64", "a3b", "slots", 64, 32000, 64),
        # speculative decoding of one conversation at the default depth of 2
        _case("round-3", "a3b", "round", 3, 1000, 1024),
        # a one-line question
        _case("prompt-37", "a3b", "prompt", 37, 0, 2048),
        # a question with a page of text, an odd length
        _case("prompt-701", "a3b", "prompt", 701, 0, 2048),
        # the benchmark's prompt, one pass
        _case("prompt-2048", "a3b", "prompt", 2048, 0, 2048),
        # a document: four full passes of 4096 rows and a ragged fifth
        _case("prompt-20001", "a3b", "prompt", 20001, 0, 4096),
        # the next user message (or a tool's answer) in a conversation of some thousand tokens
        _case("turn-200", "a3b", "turn", 200, 6000, 2048),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    model = "tiny" if rng.random() < 0.15 else "a3b"
    kind = rng.choice(["step", "slots", "slots", "round", "prompt", "prompt", "prompt", "turn", "turn"])
    if kind == "step":
        return _case(None, model, kind, 1, _log(rng, 16, 32000), 2048)
    if kind == "slots":
        return _case(None, model, kind, _log(rng, 2, 80), _log(rng, 256, 32000), 80)
    if kind == "round":
        return _case(None, model, kind, rng.randint(2, 5), _log(rng, 64, 2048), 1024)
    if kind == "prompt":
        return _case(None, model, kind, _log(rng, 2, 16000), 0, rng.choice([2048, 4096]))
    return _case(None, model, kind, _log(rng, 2, 2048), _log(rng, 128, 30000), 2048)


def _config(name):
    cfg = pkg.config.CONFIGS[name]
    return pkg.config.variant(cfg, has_draft=1, n_layer=min(12, cfg["n_layer"]))


def _model(name):
    """The checkpoint, generated on the device as Model.synthetic does it, with wider router weights."""
    if name not in _models:
        cfg, lib = _config(name), pkg.lib.load()
        fields = pkg.config.graph_fields(cfg)
        handle = ctypes.c_void_p()
        pkg.lib.check(lib.b200_model_new(ctypes.byref(pkg.lib.Config(**fields)), 0, ctypes.byref(handle)))
        for i, (tensor, typ, dims, (rule, p0, p1)) in enumerate(pkg.config.manifest(cfg)):
            p1 = ROUTER_STD if tensor.endswith("ffn_gate_inp.weight") else p1
            d = (ctypes.c_int64 * len(dims))(*dims)
            pkg.lib.check(lib.b200_model_add_synthetic(handle, tensor.encode(), typ, len(dims), d, i, int(rule != "normal"), p0, p1))
        pkg.lib.check(lib.b200_model_finalize(handle))
        _models[name] = pkg.Model(handle, fields)
    return _models[name]


class State:
    """A graph at the point a request finds it in, and the request."""


def prepare(case, seed):
    cfg, model = _config(case["model"]), _model(case["model"])
    kind, rows, context = case["kind"], case["rows"], case["context"]
    rng = np.random.default_rng(seed)
    s = State()
    s.kind, s.start, s.left = kind, context, HEADROOM
    slots = rows if kind == "slots" else 1
    room = rows if kind in ("prompt", "turn") else HEADROOM + 8
    s.g = g = pkg.Graph(model, n_kv=context + room + 8, max_tokens=max(case["chunk"], slots), slots=slots,
                        speculative=kind == "round", spec_rows=rows if kind == "round" else 0)
    s.ids = rng.integers(0, cfg["vocab"], rows).astype(np.int32)
    if kind == "slots":
        s.slots = np.arange(rows, dtype=np.int32)
        s.start = rng.integers(max(1, context // 4), context + 1, rows).tolist()
        for i, cells in enumerate(s.start):
            g.use_slot(i)
            g.synth_context(cells, seed=(seed * 1009 + i) & 0x7FFFFFFF)
    elif kind == "round":
        # a real prompt: the draft's cache is filled from the trunk's residual rows
        sp = pkg.spec.Speculator(g, depth=rows - 1, draft_vocab=DRAFT_VOCAB[case["model"]])
        sp.prime(rng.integers(0, cfg["vocab"], context).astype(np.int32), pick=lambda logits: int(s.ids[0]))
        s.h, s.vocab_k, s.keep = sp.h[None, :], DRAFT_VOCAB[case["model"]], 1 + (rows - 1) // 2
    elif context:
        g.synth_context(context, seed=seed & 0x7FFFFFFF)
    return s


def run(s):
    g = s.g
    if s.kind == "prompt":
        return g.forward(s.ids)
    if s.kind == "turn":
        g.set_past(s.start)
        return g.extend(s.ids)
    if s.kind == "round":
        at = g.past()
        out = []
        h = s.h
        for k in range(len(s.ids) - 1):
            res, logits = g.draft_rows(h, s.ids[k:k + 1], s.vocab_k)
            out.append(logits)
            h = res[-1:]
        g.speculate(True)
        logits, residual = g.extend_rows(s.ids)
        g.keep(s.keep)
        g.speculate(False)
        g.set_past(at)
        g.draft_rewind(at - 1)
        return out + [logits, residual]
    if s.left == 0:  # back to the first position
        s.left = HEADROOM
        for i, cells in enumerate(s.start if s.kind == "slots" else [s.start]):
            g.use_slot(i)
            g.set_past(cells)
    s.left -= 1
    if s.kind == "slots":
        return g.decode_rows(s.slots, s.ids)
    return g.extend(s.ids)


def _pass_work(cfg, rows, logit_rows, cells, layers, draft_vocab=0):
    """(bytes, flops) of `rows` rows that together attend to `cells` cells: weights once (the routed experts that many
    random rows touch), key / value cells and recurrent state, logits out. `layers`: (attention, DeltaNet) layers."""
    gguf, config = pkg.gguf, pkg.config
    n_at, n_dn, draft = layers
    nE, used = cfg["n_expert"], cfg["n_expert_used"]
    touched = nE * (1.0 - (1.0 - used / nE) ** rows)
    nbytes = flops = 0.0
    for name, typ, dims, _ in config.manifest(cfg):
        mine = name.startswith(f"blk.{cfg['n_layer']}.")
        b, k = gguf.tensor_bytes(typ, dims), float(np.prod(dims))
        if name == "token_embd.weight":
            nbytes += gguf.row_bytes(typ, dims[0]) * rows
        elif name == "output.weight":
            part = draft_vocab / cfg["vocab"] if draft else 1.0
            nbytes += b * part
            flops += 2.0 * k * part * logit_rows
        elif mine == draft:
            if "_exps." in name:
                nbytes += b / nE * touched
                flops += 2.0 * k / nE * used * rows
            else:
                nbytes += b
                flops += 2.0 * k * rows
    state = cfg["dn_heads_v"] * cfg["dn_head_dim"] ** 2
    nbytes += n_at * 2 * cfg["n_head_kv"] * cfg["head_dim"] * 2 * rows
    flops += n_dn * 6.0 * state * rows + n_at * 4.0 * cfg["head_dim"] * cfg["n_head"] * cells
    nbytes += 4.0 * logit_rows * (draft_vocab if draft else cfg["vocab"])
    return nbytes, flops, state * 4.0


def work(case):
    cfg = _config(case["model"])
    kind, rows, context = case["kind"], case["rows"], case["context"]
    n_at = sum(pkg.config.is_attention_layer(cfg, l) for l in range(cfg["n_layer"]))
    n_dn = cfg["n_layer"] - n_at
    cell = 2 * cfg["n_head_kv"] * cfg["head_dim"] * 2.0   # bytes of a cell's keys and values in one layer
    seqs = rows if kind == "slots" else 1
    ctx = context * 0.625 if kind == "slots" else context   # mean of the drawn contexts
    pairs = rows * ctx + rows if kind == "slots" else rows * context + rows * (rows + 1) / 2.0
    every = rows if kind in ("slots", "round") else 1
    b, f, state = _pass_work(cfg, rows, every, pairs, (n_at, n_dn, False))
    b += n_dn * state * seqs * (1.0 if kind == "prompt" else 2.0)    # a new conversation's state is only written
    if kind == "round":
        b += n_dn * state * (rows - 1)                               # the state after every row, so that any prefix can be kept
    b += n_at * cell * ctx * seqs
    if kind == "round":
        for _ in range(rows - 1):
            db, df, _ = _pass_work(cfg, 1, 1, context, (1, 0, True), DRAFT_VOCAB[case["model"]])
            b, f = b + db + cell * context, f + df
    return {"bytes": b, "flops": f}


def tolerance(case):
    # Every matmul input is stored as fp16 and top-k routing is discrete: two correct implementations that add in
    # different orders differ by fp16 steps in each of twelve layers, and now and then by an expert at a near-tie. The
    # same tokens through passes of other sizes (fp16-rounded or exact weights) measured 1e-3 to 1.5e-2.
    return {"rel": 0.025, "max": 0.3}
