"""Performance cases of the DFlash step: what a serving process asks of this library, call by call.

Models are the seeded synthetic ones of `qwen-llm_b200/synthetic.py` at the benchmark geometries (the dense 9B-class
hybrid with its 5-layer drafter, the 35B-A3B-shaped routed-expert hybrid).  A process loads a model once and keeps it,
so the weights here depend on the geometry only and are kept for the life of the process; prompts, blocks, drafts and
logits come from the seed.  Sessions belong to a request.
"""
import functools
import importlib
import math

import numpy as np

pkg = importlib.import_module("qwen-llm_b200")
syn = importlib.import_module("qwen-llm_b200.synthetic")

BYTES_PER_WEIGHT = {pkg.Q4_K: 144 / 256, pkg.Q5_K: 176 / 256, pkg.Q6_K: 210 / 256, pkg.BF16: 2.0, pkg.F32: 4.0}
DECODE_PATTERN = [3, 3, 4, 3, 4]    # drafts accepted per step in the decode loop: 4.4 tokens per step
SHORT_CAPACITY, LONG_CAPACITY = 4096, 32768


def listed():
    return [
        # the verify / accept step on two bare matrices (one layer and a head), host activations in, accepted prefix out
        {"name": "matrix_step_16", "kind": "matrices", "rows": 16},
        # plain decoding: one token, its logits to the host sampler
        {"name": "token", "kind": "token", "model": "dense", "ctx": 300},
        # one greedy verify block of a chat-length sequence
        {"name": "verify_block", "kind": "verify", "model": "dense", "ctx": 600, "rows": 16, "logits": False},
        # a verify block of a long sequence (tiled cache), its logits to the host sampler
        {"name": "verify_long_sampled", "kind": "verify", "model": "dense", "ctx": 17001, "rows": 16, "logits": True},
        # a verify block on the routed-expert model
        {"name": "verify_experts", "kind": "verify", "model": "experts", "ctx": 200, "rows": 16, "logits": True},
        # one draft of 16 tokens
        {"name": "draft_block", "kind": "draft", "model": "dense", "ctx": 700},
        # a short chat turn: new request, 77-token prompt, every captured row back on the host
        {"name": "prompt_77_rows", "kind": "prompt", "model": "dense", "tokens": 77, "rows_out": True},
        # an ordinary prompt and a long one: new request, drafter fed on the device, last logits back
        {"name": "prompt_512", "kind": "prompt", "model": "dense", "tokens": 512, "rows_out": False},
        {"name": "prompt_2048", "kind": "prompt", "model": "dense", "tokens": 2048, "rows_out": False},
        # a prompt on the routed-expert model
        {"name": "prompt_experts_300", "kind": "prompt", "model": "experts", "tokens": 300, "rows_out": False},
        # a request resumed from the prefix cache, then the greedy outer loop: draft, verify, accept, roll back
        {"name": "decode_48", "kind": "decode", "model": "dense", "ctx": 512, "tokens": 48},
        # sampled acceptance of one block on the host (T 0.7, top-p 0.95), four drafts accepted, the fifth corrected
        {"name": "accept_sampled", "kind": "accept", "rows": 16, "vocab": 151936, "accepted": 4, "temperature": 0.7, "top_p": 0.95},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matrices", "token", "verify", "verify", "verify", "draft", "prompt", "prompt", "prompt", "decode", "accept"])
    if kind == "matrices":
        return {"kind": kind, "rows": rng.randint(1, 16)}
    if kind == "token":
        return {"kind": kind, "model": rng.choice(["dense", "dense", "experts"]), "ctx": _log_int(rng, 16, 3000)}
    if kind == "verify":
        model = rng.choice(["dense", "dense", "experts"])
        rows = 16 if rng.random() < 0.6 else rng.randint(2, 15)
        return {"kind": kind, "model": model, "ctx": _log_int(rng, 16, 20000 if model == "dense" else 2000), "rows": rows, "logits": model == "experts" or rng.random() < 0.3}
    if kind == "draft":
        return {"kind": kind, "model": "dense", "ctx": _log_int(rng, 16, 20000)}
    if kind == "prompt":
        model = rng.choice(["dense", "dense", "experts"])
        tokens = _log_int(rng, 17, 2048 if model == "dense" else 900)
        return {"kind": kind, "model": model, "tokens": tokens, "rows_out": tokens <= 512 and rng.random() < 0.3}
    if kind == "decode":
        return {"kind": kind, "model": "dense", "ctx": _log_int(rng, 32, 2000), "tokens": rng.randint(8, 64)}
    return {"kind": kind, "rows": 16, "vocab": rng.choice([32000, 151936]), "accepted": rng.randint(0, 15), "temperature": rng.choice([0.6, 0.7, 1.0]),
            "top_p": rng.choice([0.8, 0.9, 0.95, 1.0])}


# ---------------------------------------------------------------------------------------------------------------
# what a serving process keeps
# ---------------------------------------------------------------------------------------------------------------
class Model:
    def __init__(self, which):
        self.arch = syn.arch_9b() if which == "dense" else syn.arch_35b_a3b()
        entries = syn.target_entries(self.arch, seed=100)
        self.model = syn.build_model(self.arch, entries)
        syn.free_entries(entries)
        self.drafter, self.taps = None, [7, 15, 23, 31, 39]
        if which == "dense":
            cfg = syn.dflash_config_9b(self.arch)
            entries = syn.drafter_entries(self.arch, cfg, seed=101)
            self.drafter = syn.build_drafter(self.model, cfg, entries)
            syn.free_entries(entries)
            self.taps = self.drafter.layer_ids()


@functools.lru_cache(maxsize=None)
def _model(which):
    return Model(which)


@functools.lru_cache(maxsize=None)
def _matrices():
    """A 4096 x 4096 Q4_K matrix and a 4096 -> 32000 Q6_K head."""
    out = []
    for dtype, n_in, n_out in ((pkg.Q4_K, 4096, 4096), (pkg.Q6_K, 4096, 32000)):
        _, _, _, ptr, n_bytes = pkg.synth_tensor("w", dtype, n_in, n_out, 7 + n_out, 0.02)
        out.append(pkg.QMatrix(dtype, n_in, n_out, pkg.device_to_host(ptr, n_bytes)))
        pkg.device_free(ptr)
    return out


class State:
    """What one request holds; its device memory goes when it does."""

    def __init__(self, case):
        self.case, self.m, self.sess, self.scr, self.ds = case, None, None, None, None

    def close(self):
        for x in (self.sess, self.scr, self.ds):
            if x is not None:
                x.close()
        self.sess = self.scr = self.ds = None

    def __del__(self):
        self.close()


def _capacity(ctx):
    return SHORT_CAPACITY if ctx + 128 <= SHORT_CAPACITY else LONG_CAPACITY


@functools.lru_cache(maxsize=2)
def _long_prefix(which, n, drafter):
    """Snapshot of a long fixed prefix, as a prefix cache holds it."""
    s = State({})
    s.m = m = _model(which)
    s.sess, s.scr = pkg.Session(m.model, LONG_CAPACITY, True), pkg.Scratch(m.model, 16, len(m.taps))
    s.ds = pkg.DSession(m.drafter, LONG_CAPACITY) if drafter else None
    ids = np.random.default_rng(n).integers(0, m.arch.vocab_size, size=n)
    pkg.prefill(m.model, s.sess, s.scr, m.taps, ids, 0, feed_drafter=s.ds, want_logits=False)
    return pkg.session_snapshot(m.model, s.sess, s.ds)


def _at_context(case, rng, drafter):
    """A request after `ctx` tokens: (state, last logits)."""
    s = State(case)
    s.m = m = _model(case["model"])
    ctx, cap = case["ctx"], _capacity(case["ctx"])
    s.sess, s.scr = pkg.Session(m.model, cap, True), pkg.Scratch(m.model, 16, len(m.taps))
    s.ds = pkg.DSession(m.drafter, cap) if drafter else None
    start = 0
    if cap == LONG_CAPACITY:
        start = ctx - 200
        pkg.session_restore_snapshot(m.model, s.sess, s.ds, _long_prefix(case["model"], start, drafter))
    ids = rng.integers(0, m.arch.vocab_size, size=ctx - start)
    logits, _ = pkg.prefill(m.model, s.sess, s.scr, m.taps, ids, start, feed_drafter=s.ds)
    return s, logits


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, np.random.default_rng(seed))


def run(state):
    return globals()["_run_" + state.case["kind"]](state)


# ---- matrices ---------------------------------------------------------------------------------------------------
def _prepare_matrices(case, rng):
    s = State(case)
    w1, head = _matrices()
    s.pipe = pkg.C1Pipeline(w1, head)
    s.x = rng.standard_normal((case["rows"], 4096)).astype(np.float32)
    s.draft = rng.integers(0, 32000, size=case["rows"]).astype(np.int32)
    return s


def _run_matrices(s):
    argmax, gap, accepted, _ = s.pipe.step(s.x, s.draft)
    return {"argmax": argmax, "gap": gap, "accepted": accepted}


# ---- one token --------------------------------------------------------------------------------------------------
def _prepare_token(case, rng):
    s, logits = _at_context(case, rng, False)
    s.token = int(np.argmax(logits))
    return s


def _run_token(s):
    m, at = s.m, s.case["ctx"]
    logits, _ = pkg.single_token(m.model, s.sess, s.scr, [], s.token, at, want_hidden=False)
    pkg.restore_pre_block(m.model, s.sess, s.scr, at)     # so that the next pass finds the same context
    return logits


# ---- verify block -----------------------------------------------------------------------------------------------
def _prepare_verify(case, rng):
    s, _ = _at_context(case, rng, False)
    s.block = rng.integers(0, s.m.arch.vocab_size, size=case["rows"]).astype(np.int32)
    return s


def _run_verify(s):
    m, at = s.m, s.case["ctx"]
    argmax, gap, logits = pkg.packed_verify(m.model, s.sess, s.scr, m.taps, s.block, at, want_logits=s.case["logits"])
    pkg.restore_pre_block(m.model, s.sess, s.scr, at)     # as for a block of which nothing is kept
    return logits if s.case["logits"] else {"argmax": argmax, "gap": gap}


# ---- draft block ------------------------------------------------------------------------------------------------
def _prepare_draft(case, rng):
    s, _ = _at_context(case, rng, True)
    s.carry = int(rng.integers(0, s.m.arch.vocab_size))
    return s


def _run_draft(s):
    return s.ds.draft_block(s.carry, s.case["ctx"])[0]


# ---- prompt: a new request up to its first logits ---------------------------------------------------------------
def _prepare_prompt(case, rng):
    s = State(case)
    s.m = _model(case["model"])
    s.scr = pkg.Scratch(s.m.model, 16, len(s.m.taps))
    s.ids = rng.integers(0, s.m.arch.vocab_size, size=case["tokens"]).astype(np.int32)
    return s


def _run_prompt(s):
    m, cap = s.m, _capacity(s.case["tokens"])
    sess = pkg.Session(m.model, cap, True)
    ds = pkg.DSession(m.drafter, cap) if m.drafter is not None else None
    try:
        logits, rows = pkg.prefill(m.model, sess, s.scr, m.taps, s.ids, 0, feed_drafter=ds, want_hidden=s.case["rows_out"])
    finally:
        sess.close()
        if ds is not None:
            ds.close()
    return {"logits": logits, "rows": rows}


# ---- decode: the greedy outer loop ------------------------------------------------------------------------------
def _prepare_decode(case, rng):
    n = case["tokens"]
    s, s.first = _at_context(case, rng, True)
    m = s.m
    s.snapshot = pkg.session_snapshot(m.model, s.sess, s.ds)
    truth, _ = pkg.generate(m.model, s.sess, s.scr, s.ds, pkg.Sampler(), s.first, n)
    # drafts replay the true continuation with one wrong token after every few, so that steps accept 3, 3, 4, 3, 4
    s.drafts, at, step = np.concatenate([truth, np.zeros(16, np.int32)]).astype(np.int32), 1, 0
    while at < n:
        at += DECODE_PATTERN[step % len(DECODE_PATTERN)]
        if at < n:
            s.drafts[at] = (s.drafts[at] + 1) % m.arch.vocab_size
        at, step = at + 1, step + 1
    return s


def _run_decode(s):
    m = s.m
    pkg.session_restore_snapshot(m.model, s.sess, s.ds, s.snapshot)
    return pkg.generate(m.model, s.sess, s.scr, s.ds, pkg.Sampler(), s.first, s.case["tokens"], replay_history=s.drafts, replay_runs_drafter=True,
                        replay_unchecked=True)[0]


# ---- sampled acceptance on the host -----------------------------------------------------------------------------
def _prepare_accept(case, rng):
    """Logits like a language model's: a broad body, a few dozen plausible tokens, one clear favourite in the rows whose
    draft is accepted and none in the row that ends the prefix."""
    s = State(case)
    n, V, a = case["rows"], case["vocab"], case["accepted"]
    s.logits = (rng.standard_normal((n, V), dtype=np.float32) * 2.0).astype(np.float32)
    favourite = rng.integers(0, V, size=n)
    for r in range(n):
        s.logits[r, rng.integers(0, V, size=40)] += rng.uniform(4.0, 9.0, size=40).astype(np.float32)
        s.logits[r, favourite[r]] = 40.0 if r < a else 9.0
    s.block = np.concatenate([rng.integers(0, V, size=1), favourite[:n - 1]]).astype(np.int32)
    if a < n - 1:
        s.block[a + 1] = int(np.argmin(s.logits[a]))      # a draft that the target would not sample
    s.sampler = pkg.Sampler(temperature=case["temperature"], top_p=case["top_p"], seed=int(rng.integers(1 << 60)))
    return s


def _run_accept(s):
    d = pkg.accept_prefix(s.block, s.logits, s.case["vocab"], None, s.sampler, 4096, ())
    return {"accepted": np.array(d["accepted_drafts"], dtype=np.int32), "carry": int(d["next_carry"][1]), "kept": d["retain_input_count"]}


# ---------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------
def _target_work(which, rows, ctx, head_rows):
    """Bytes and operations of `rows` tokens after `ctx`: weights, cache and state once, two operations per weight and row."""
    a = syn.arch_9b() if which == "dense" else syn.arch_35b_a3b()
    H, hd = a.hidden_size, a.attn_head_dim
    q, kv, v = a.n_q_heads * hd, a.n_kv_heads * hd, a.gdn_n_v_heads * 128
    conv = (2 * a.gdn_n_k_heads + a.gdn_n_v_heads) * 128
    n_attn = a.n_layer // a.full_attention_interval
    n_gdn = a.n_layer - n_attn
    B4, B5, B6 = BYTES_PER_WEIGHT[pkg.Q4_K], BYTES_PER_WEIGHT[pkg.Q5_K], BYTES_PER_WEIGHT[pkg.Q6_K]
    attn_w, gdn_w = H * (2 * q + 2 * kv) + q * H, H * (conv + v) + v * H
    weight_bytes = n_attn * attn_w * B4 + n_gdn * (H * conv * B6 + H * v * B4 + v * H * B5 + 8 * H * a.gdn_n_v_heads) + (a.vocab_size * H * B6 if head_rows else 0)
    flops = 2.0 * rows * (n_attn * attn_w + n_gdn * (gdn_w + 2 * H * a.gdn_n_v_heads)) + 2.0 * head_rows * a.vocab_size * H
    if a.expert_count:
        fe, used, E = a.expert_feed_forward_length, a.expert_used_count, a.expert_count
        touched = E * (1.0 - (1.0 - used / E) ** rows)      # expected under the near-uniform routing of random weights
        per_expert = H * fe * (2 * B4 + B6)
        weight_bytes += a.n_layer * ((touched + 1) * per_expert + 4.0 * H * (E + 1))
        flops += 2.0 * rows * a.n_layer * (3 * H * fe * (used + 1) + H * (E + 1))
    else:
        F = a.intermediate_size
        weight_bytes += a.n_layer * H * F * (2 * B4 + B6)
        flops += 2.0 * rows * a.n_layer * 3 * H * F
    keys = rows * ctx + rows * (rows + 1) / 2
    state = n_attn * (ctx + rows) * 2 * kv * 2 + n_gdn * 2 * (v * 128 + 3 * conv) * 4
    flops += n_attn * 4.0 * q * keys + n_gdn * rows * 8.0 * v * 128
    return weight_bytes + state, flops


def _drafter_work(rows, ctx, new_columns, whole):
    a = syn.arch_9b()
    c = syn.dflash_config_9b(a)
    H, F, q, kv = c.hidden_size, c.intermediate_size, c.n_q_heads * c.head_dim, c.n_kv_heads * c.head_dim
    fc, per_kv = c.n_target_layers * H * H, 2 * H * kv
    per_layer = H * (q + 2 * kv) + q * H + 3 * H * F
    seen = sum(min(ctx, c.swa_window) if c.layer_is_swa[i] else ctx for i in range(c.n_layer))
    n_bytes = flops = 0.0
    if whole:
        n_bytes += 2.0 * c.n_layer * per_layer + a.vocab_size * H * BYTES_PER_WEIGHT[pkg.Q6_K] + seen * 2 * kv * 4
        flops += 2.0 * rows * (c.n_layer * per_layer + a.vocab_size * H) + 4.0 * q * rows * seen
    if new_columns:
        n_bytes += 2.0 * fc + (0 if whole else 2.0 * c.n_layer * per_kv) + new_columns * c.n_layer * 2 * kv * 4
        flops += 2.0 * new_columns * (fc + c.n_layer * per_kv)
    return n_bytes, flops


def work(case):
    kind = case["kind"]
    if kind == "matrices":
        n, H, V = case["rows"], 4096, 32000
        return {"bytes": H * H * BYTES_PER_WEIGHT[pkg.Q4_K] + V * H * BYTES_PER_WEIGHT[pkg.Q6_K] + n * (4 * H + 16), "flops": 2.0 * n * H * (H + V)}
    if kind == "accept":
        read = min(case["accepted"] + 1, case["rows"])
        return {"bytes": 4.0 * read * case["vocab"], "flops": 8.0 * read * case["vocab"]}
    if kind == "token":
        b, f = _target_work(case["model"], 1, case["ctx"], 1)
        return {"bytes": b + 4.0 * 151936, "flops": f}
    if kind == "verify":
        b, f = _target_work(case["model"], case["rows"], case["ctx"], case["rows"])
        return {"bytes": b + (4.0 * 151936 * case["rows"] if case["logits"] else 0), "flops": f}
    if kind == "draft":
        b, f = _drafter_work(16, case["ctx"], 0, True)
        return {"bytes": b, "flops": f}
    if kind == "prompt":
        b, f = _target_work(case["model"], case["tokens"], 0, 1)
        b += 4.0 * 151936 + (case["tokens"] * 5 * 4096 * 4.0 if case["rows_out"] else 0)
        if case["model"] == "dense":   # of the drafter's context, what is appended within the call has to be projected by the next draft at the latest
            db, df = _drafter_work(0, 0, case["tokens"], False)
            b, f = b + db, f + df
        return {"bytes": b, "flops": f}
    # decode: 4.4 tokens a step, each step one draft with the columns of the step before and one verify
    steps = math.ceil(max(case["tokens"] - 1, 1) / 4.4)
    vb, vf = _target_work("dense", 16, case["ctx"], 16)
    db, df = _drafter_work(16, case["ctx"], 5, True)
    return {"bytes": steps * (vb + db), "flops": steps * (vf + df)}


def tolerance(case):
    if case["kind"] in ("accept", "decode", "draft"):
        return "exact"
    if case["kind"] == "matrices":
        return {"rel": 1e-4}      # a difference of two logits: f32-class logits (1e-6) over gaps a tenth of their size
    # K and V are kept in fp16.  The experts' random router has logits of 20 and more, so that a last-bit difference before
    # it moves the route weights by some 1e-4.
    return {"rel": 3e-3 if case["model"] == "experts" else 1e-3}
