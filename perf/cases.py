"""The work that a user of this framework has it do, as cases for timing and for comparing two builds.

Two ways in are covered.  The engine (Engine.verify / commit / draft, their lanes forms, lookup, prompt, save_state /
load_state) is what a serving process drives: one model with its weights on the GPU and many conversations, each a
sequence of the engine.  The operators (router_route, moe_experts, attn, dense) are what a host program calls that brings
its own scheduler and replaces its kernels one at a time.

Model: the synthetic Qwen3-Next-style model of the benchmark (hidden 2048, 512 experts top-10 + shared expert, gated
attention in every 4th layer, gated DeltaNet in the others, vocabulary 151,936, one draft layer with a draft vocabulary) at
its own widths and a quarter of its depth: 12 layers repeat the benchmark's 3 : 1 pattern three times, and their expert
weights (8 GB) are far larger than L2 as the full model's are.  The weights are one fixed random model per process, as a
server loads one file; a case's conversation (cache rows, recurrent states, tokens) comes from its seed.
"""
import math

import numpy as np
import torch

import fnx_b200 as F

LAYERS, HIDDEN, EXPERTS, TOP_K, FFN, VOCAB, DRAFT_VOCAB = 12, 2048, 512, 10, 512, 151936, 40528
N_ATTN, N_GDN, KV_WIDTH, MAX_ROWS = 3, 9, 512, 32
IN_ATTN, IN_GDN, MIX = 9216, 12352, 4096            # rows of the input projections; width of the mixers' outputs
SLOTS = MAX_ROWS + 1                                # state slots of a sequence's ring
IQ3S = 110 / 256                                    # bytes of a weight
ATTN = [l for l in range(LAYERS) if (l + 1) % 4 == 0]
P_KEEP = 0.72                                       # chance that a draft-layer draft stands (the benchmark's rate)

# greedy engine: a chat server's conversations; sampled engine: few long ones
ENGINES = {"greedy": dict(n_seq=26, max_ctx=40960 + 1024), "sampled": dict(n_seq=14, max_ctx=131072 + 4096)}


def listed():
    return [
        # plain decoding, one token per pass, in a short chat: the smallest call, where launches and latency count
        {"name": "decode 1 row", "kind": "decode", "rows": 1, "draft": 0, "ctx": 600},
        # the framework's headline: a committed token and four draft-layer drafts, then commit and the next draft chain
        {"name": "decode 5 rows", "kind": "decode", "rows": 5, "draft": 4, "ctx": 4096},
        # an editing session: prompt-lookup branch beside the draft chain, verified as a tree, a branch kept
        {"name": "tree 20 rows", "kind": "tree", "rows": 20, "draft": 4, "ctx": 32768},
        # concurrent chats of different draft counts sharing greedy windows
        {"name": "lanes 7 ragged", "kind": "lanes", "engine": "greedy", "lanes": 7, "rows": 0, "draft": 2, "ctx": 3000},
        # long documents served together at temperature 0.7
        {"name": "lanes 4x5 sampled 131k", "kind": "lanes", "engine": "sampled", "lanes": 4, "rows": 5, "draft": 4, "ctx": 131072},
        # a new chat's first message
        {"name": "prompt 333", "kind": "prompt", "tokens": 333, "ctx": 0},
        # the next long message (a pasted file) of a live conversation
        {"name": "prompt 3001 at 16384", "kind": "prompt", "tokens": 3001, "ctx": 16384},
        # a long document read cold
        {"name": "prompt 38912", "kind": "prompt", "tokens": 38912, "ctx": 0},
        # a conversation parked in host memory for another one, and brought back
        {"name": "park and resume 4096", "kind": "park", "ctx": 4096},
        # operators: the MoE block of a five-row window, routing included
        {"name": "op moe 5 rows", "kind": "moe", "rows": 5},
        # operators: window attention over a long cache
        {"name": "op attn 5 rows 32768", "kind": "attn", "rows": 5, "ctx": 32768, "tree": False},
        # operators: the input projections of the layers one after another, norm fused
        {"name": "op dense 12352x2048 5 rows", "kind": "dense", "out": 12352, "cols": 2048, "rows": 5, "norm": True, "accumulate": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "tree", "lanes", "lanes", "prompt", "prompt", "park", "moe", "attn", "dense"])
    if kind == "decode":
        rows = rng.randint(1, 8)
        return {"kind": kind, "rows": rows, "draft": rng.choice([0, 2, 3, 4]), "ctx": _log(rng, 20, 32768)}
    if kind == "tree":
        return {"kind": kind, "rows": rng.randint(7, 32), "draft": rng.choice([2, 4]), "ctx": _log(rng, 500, 36000)}
    if kind == "lanes":
        if rng.random() < 0.5:
            return {"kind": kind, "engine": "greedy", "lanes": rng.randint(2, 8), "rows": rng.choice([0, 1, 2, 3, 4]), "draft": rng.choice([0, 1, 2, 4]), "ctx": _log(rng, 50, 24000)}
        return {"kind": kind, "engine": "sampled", "lanes": rng.randint(1, 4), "rows": rng.randint(1, 5), "draft": rng.choice([0, 3, 4]), "ctx": _log(rng, 2000, 131072)}
    if kind == "prompt":
        ctx = rng.choice([0, 0, _log(rng, 100, 16384)])
        return {"kind": kind, "tokens": _log(rng, 12, 38912 - 2 * ctx if ctx < 16384 else 6144), "ctx": ctx}
    if kind == "park":
        return {"kind": kind, "ctx": _log(rng, 150, 16384)}
    if kind == "moe":
        return {"kind": kind, "rows": rng.randint(1, 24)}
    if kind == "attn":
        return {"kind": kind, "rows": rng.randint(1, 20), "ctx": _log(rng, 50, 131072), "tree": rng.random() < 0.3}
    cols = rng.choice([512, 1024, 2048, 2048, 4096])
    return {"kind": "dense", "out": 16 * _log(rng, 16, 1024), "cols": cols, "rows": rng.randint(1, 8 if cols == 4096 else 12), "norm": rng.random() < 0.6,
            "accumulate": rng.random() < 0.4}


# ------------------------------------------------------------------------------------------------ one model per process
class _Server:
    """An engine with its weights and the sequences that no conversation holds."""

    def __init__(self, name):
        self.cfg = F.flash_next_config(n_layer=LAYERS, max_rows=MAX_ROWS, draft_vocab=DRAFT_VOCAB, **ENGINES[name])
        self.eng = F.Engine(self.cfg)
        self.eng.init_synthetic(seed=0, sigma=0.02)
        if name == "sampled":
            self.eng.set_sampling(F.Sampling(0.7, 1.0, 0.0, 0), seed=4)
        self.free = list(range(self.cfg.n_seq))
        c = self.cfg
        rows = c.max_ctx + c.max_rows
        t = self.eng.tensor
        self.kv = {p: [t(p + n, torch.float16, (c.n_seq, rows, KV_WIDTH)) for n in ("k_cache", "v_cache")] for p in ["l%d." % l for l in ATTN] + ["mtp."]}
        self.state = {l: t("l%d.state" % l, torch.float32, (c.n_seq, SLOTS, 32, 128, 128)) for l in range(LAYERS) if l not in ATTN}
        self.hist = {l: t("l%d.conv_hist" % l, torch.float32, (c.n_seq, SLOTS, 3, 8192)) for l in self.state}
        self.ctx = t("seq.ctx", torch.int32, (c.n_seq, rows))
        self.logits = t("buf.logits", torch.float32, (MAX_ROWS, VOCAB))


_servers, _moe_weights = {}, []


def _server(name):
    if name not in _servers:
        _servers[name] = _Server(name)
    return _servers[name]


class _State:
    """What a case holds between passes; its sequences go back to the engine with it."""

    def __init__(self, case):
        self.case, self.srv, self.seqs, self.i = case, None, [], 0

    def take(self, name, n):
        self.srv = _server(name)
        if len(self.srv.free) < n:
            raise MemoryError("no free sequences")
        self.seqs = [self.srv.free.pop() for _ in range(n)]

    def __del__(self):
        if self.srv is not None:
            self.srv.free.extend(self.seqs)


def _conversation(srv, seq, ctx, g, tokens):
    """Sequence `seq` at position ctx: cache rows, recurrent states and tokens of the values that a read context leaves."""
    srv.eng.reset(seq)
    if ctx == 0:
        return
    srv.eng.set_position(seq, ctx)
    for pair in srv.kv.values():
        for t in pair:
            t[seq, :ctx].normal_(0.0, 1.0, generator=g)
    for l in srv.state:
        srv.state[l][seq, 0].normal_(0.0, 0.02, generator=g)
        srv.hist[l][seq, 0].normal_(0.0, 0.5, generator=g)
    srv.ctx[seq, :ctx] = torch.from_numpy(tokens[:ctx]).cuda()


def _edited_text(rng, n):
    """Token ids in which spans of the earlier text recur, as in an editing session."""
    out = np.empty(n, np.int32)
    i = 0
    while i < n:
        m = int(rng.integers(14, 134))
        out[i:i + m] = rng.integers(0, VOCAB, size=len(out[i:i + m]))
        i += m
        if i < n and i > 300:
            m = int(rng.integers(20, 200))
            at = int(rng.integers(0, i - 250)) if i > 260 else 0
            m = min(m, n - i)
            out[i:i + m] = out[at:at + m]
            i += m
    return out


def _tree(rng, rows, chain):
    """Parents of a window: the root, a chain of drafts, and branches of the lookup rows that leave the chain at some row."""
    par = [-1]
    for t in range(1, rows):
        if t <= chain:
            par.append(t - 1)
        elif t == chain + 1 or rng.random() < 0.1:
            par.append(int(rng.integers(0, chain)))
        else:
            par.append(t - 1)
    return par


def _path_to(par, node):
    path = []
    while node >= 0:
        path.append(node)
        node = par[node]
    return path[::-1]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    s = _State(case)
    kind = case["kind"]
    n_plan = 16   # the windows' tokens and what of each is kept, drawn ahead: the drafts of a random model would never stand
    if kind in ("decode", "tree", "prompt", "park"):
        s.take("greedy", 1)
        ctx = case["ctx"]
        s.ctx = ctx
        s.tokens = _edited_text(rng, max(ctx, 1))
        _conversation(s.srv, s.seqs[0], ctx, g, s.tokens)
    if kind == "decode":
        T = case["rows"]
        s.windows = [rng.integers(0, VOCAB, size=T).tolist() for _ in range(n_plan)]
        s.keep = [1 + _run_of(rng, T - 1) for _ in range(n_plan)]
        s.end = ctx + min(2048, s.srv.cfg.max_ctx - MAX_ROWS - ctx)
    elif kind == "tree":
        T = case["rows"]
        s.windows, s.parents, s.paths = [], [], []
        for _ in range(n_plan):
            par = _tree(rng, T, min(4, T - 2))
            s.windows.append(rng.integers(0, VOCAB, size=T).tolist())
            s.parents.append(par)
            s.paths.append(_path_to(par, int(rng.integers(0, T))))
        at = rng.integers(2, max(3, ctx), size=n_plan)      # the tokens that the edit has reached
        s.roots = [int(s.tokens[i]) for i in np.minimum(at, ctx - 1)]
        s.end = ctx + min(2048, s.srv.cfg.max_ctx - MAX_ROWS - ctx)
    elif kind == "lanes":
        n = case["lanes"]
        s.take(case["engine"], n)
        s.ctx = case["ctx"]
        s.pos0 = []
        for j, q in enumerate(s.seqs):                       # conversations of different lengths
            at = max(1, s.ctx - int(rng.integers(0, max(2, s.ctx // 8))))
            s.pos0.append(at)
            _conversation(s.srv, q, at, g, rng.integers(0, VOCAB, size=at, dtype=np.int32))
        rows = _lane_rows(case)
        rng.shuffle(rows)
        s.windows = [[rng.integers(0, VOCAB, size=r).tolist() for r in rows] for _ in range(n_plan)]
        s.keep = [[1 + _run_of(rng, r - 1) for r in rows] for _ in range(n_plan)]
        s.end = s.ctx + 1024
    elif kind == "prompt":
        s.new = rng.integers(0, VOCAB, size=case["tokens"]).tolist()
    elif kind == "moe":
        s.w = _moe_block_weights()
        s.x = torch.empty((case["rows"], HIDDEN), device="cuda").normal_(0.0, 1.0, generator=g)
        s.norm = torch.ones(HIDDEN, device="cuda")
    elif kind == "attn":
        T, ctx = case["rows"], case["ctx"]
        s.qg = torch.empty((T, 16, 512), device="cuda").normal_(0.0, 1.0, generator=g)
        s.kc, s.vc = (torch.empty((ctx + T, 2, 256), dtype=torch.float16, device="cuda").normal_(0.0, 1.0, generator=g) for _ in range(2))
        s.pos0 = torch.tensor([ctx], dtype=torch.int32, device="cuda")
        s.parent = torch.tensor(_tree(rng, T, max(1, min(4, T - 2))), dtype=torch.int32, device="cuda") if case["tree"] and T > 2 else None
        s.scratch = torch.empty(F.lib().fnx_attn_scratch_bytes(T, 16, 256), dtype=torch.uint8, device="cuda")
    elif kind == "dense":
        rows, cols = case["out"], case["cols"]
        s.w = []
        for _ in range(LAYERS):
            w = torch.empty(rows * cols, device="cuda").normal_(0.0, 0.02, generator=g)
            s.w.append(F.iq3s_retile(F.iq3s_quantize(w), rows, cols))
        s.x = torch.empty((LAYERS, case["rows"], cols), device="cuda").normal_(0.0, 1.0, generator=g)
        s.norm = torch.ones(cols, device="cuda") if case["norm"] else None
        s.base = torch.empty((LAYERS, case["rows"], rows), device="cuda").normal_(0.0, 1.0, generator=g)
        s.out = s.base.clone()
        s.err = F.new_err()
    torch.cuda.synchronize()
    return s


def _lane_rows(case):
    """Rows of the lanes: all alike, or (rows = 0) 1, 4, 3, 2 and round again, as lanes of different draft counts have."""
    return [case["rows"] or 1 + 3 * j % 4 for j in range(case["lanes"])]


def _run_of(rng, most):
    """How many drafts of a chain stand."""
    n = 0
    while n < most and rng.random() < P_KEEP:
        n += 1
    return n


def _moe_block_weights():
    if not _moe_weights:
        def matrix(rows, cols, stream):
            w = F.fill_normal(torch.empty(rows * cols, device="cuda"), 0.02, 0, stream)
            return F.iq3s_retile(F.iq3s_quantize(w), rows, cols)
        gu = torch.cat([matrix(2 * FFN, HIDDEN, 100 + e) for e in range(EXPERTS)])
        dn = torch.cat([matrix(HIDDEN, FFN, 1000 + e) for e in range(EXPERTS)])
        wr = F.fill_normal(torch.empty((EXPERTS + 1, HIDDEN), device="cuda"), 0.02, 0, 7)
        _moe_weights.append((wr, gu, dn, matrix(2 * FFN, HIDDEN, 50), matrix(HIDDEN, FFN, 51)))
    return _moe_weights[0]


# ------------------------------------------------------------------------------------------------ one pass
def run(s):
    kind = s.case["kind"]
    if kind in ("decode", "tree", "lanes"):
        return _round(s, kind)
    if kind == "prompt":
        return _prompt(s)
    if kind == "park":
        return _park(s)
    if kind == "moe":
        wr, gu, dn, sgu, sdn = s.w
        r = F.router_route(wr, s.x, TOP_K, norm_w=s.norm)
        out, h, part = F.moe_experts(gu, dn, sgu, sdn, r, s.x, FFN, TOP_K, norm_w=s.norm)
        return {"out": out, "topi": r["topi"], "topw": r["topw"], "logits": r["logits"]}
    if kind == "attn":
        return F.attn(s.qg, s.kc, s.vc, s.pos0, s.parent, scratch=s.scratch)
    if s.case["accumulate"]:       # the sums start from the same rows in every pass, as a residual that a layer adds to
        s.out.copy_(s.base)
    for l in range(LAYERS):
        F.dense(s.w[l], s.case["out"], s.case["cols"], s.x[l], norm_w=s.norm, out=s.out[l], accumulate=s.case["accumulate"], err=s.err)
    return s.out


def _round(s, kind):
    """A decoding round: the window, what of it stands, the drafts of the next one.  A conversation that has grown by the
    room it was given goes back to its first length."""
    e, case, i = s.srv.eng, s.case, s.i % len(s.windows)
    s.i += 1
    k = case["draft"]
    if kind == "lanes":
        if any(e.pos(q) + 5 > s.end for q in s.seqs):
            for q, at in zip(s.seqs, s.pos0):
                e.set_position(q, at)
        got = e.verify_lanes_rows(s.seqs, s.windows[i])
        e.commit_lanes(s.seqs, s.keep[i])
        drafts = e.draft_lanes(s.seqs, k) if k else []
        T, used = sum(len(w) for w in s.windows[i]), -(-len(s.seqs) * DRAFT_VOCAB // VOCAB) if k else 0
        emitted = [t for lane in got for t in lane[2]]
    else:
        q = s.seqs[0]
        if e.pos(q) + MAX_ROWS > s.end:
            e.set_position(q, s.ctx)
        window = s.windows[i]
        if kind == "tree":
            chain = min(4, len(window) - 2)
            found = e.lookup(len(window) - 1 - chain, root=s.roots[i], seq=q)     # the lookup branch takes the rows after the chain
            window = window[:chain + 1] + found + window[chain + 1 + len(found):]
            window[0] = s.roots[i]
            got = e.verify(window, s.parents[i], seq=q)
            e.commit(s.paths[i], seq=q)
        else:
            got = e.verify(window, seq=q)
            e.commit(list(range(s.keep[i])), seq=q)
        drafts = [e.draft(k, seq=q)] if k else []
        T, used = len(window), 1 if k else 0
        emitted = got[2]
    # (the draft layer's own logits use the first rows of the buffer)
    r = {"emitted": np.asarray(emitted, np.int32), "drafts": np.asarray(drafts, np.int32), "logits": s.srv.logits[used:T]}
    return {n: v for n, v in r.items() if len(v)}


def _prompt(s):
    """The prompt into a cleared conversation, or behind the rows of a live one (which goes back to its first length when it is full)."""
    e, q, n = s.srv.eng, s.seqs[0], len(s.new)
    if s.ctx == 0:
        e.reset(q)
        s.i = 0
    elif e.pos(q) + n > min(s.ctx + 4 * n, s.srv.cfg.max_ctx - MAX_ROWS):
        e.set_position(q, s.ctx)
    at = e.pos(q)
    e.prompt(s.new, seq=q)
    s.i += n
    l, cur = max(s.srv.state), s.i % SLOTS
    return {"logits": s.srv.logits[:1], "state": s.srv.state[l][q, cur], "hist": s.srv.hist[l][q, cur],
            "k": s.srv.kv["l%d." % ATTN[-1]][0][q, at:at + n], "v": s.srv.kv["l%d." % ATTN[-1]][1][q, at:at + n]}


def _park(s):
    e, q = s.srv.eng, s.seqs[0]
    buf = e.save_state(seq=q)
    e.load_state(buf, seq=q)
    l = max(s.srv.state)
    return {"image": np.frombuffer(buf, np.uint8), "k": s.srv.kv["l%d." % ATTN[-1]][0][q, :s.ctx], "state": s.srv.state[l][q, 0]}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def _distinct(T):
    """Expected experts that T rows' picks fall on."""
    return EXPERTS * (1 - (1 - TOP_K / EXPERTS) ** T)


def _row_weights():
    """Weights that one row meets in the layers: mixers' projections and the picked and shared experts."""
    return N_ATTN * (IN_ATTN + HIDDEN * MIX / HIDDEN) * HIDDEN + N_GDN * (IN_GDN + HIDDEN * MIX / HIDDEN) * HIDDEN + LAYERS * (TOP_K + 1) * 3 * FFN * HIDDEN


def _window(lanes, T, ctx):
    """(bytes, flops) of a verify window of T rows in all over `lanes` contexts."""
    w = N_ATTN * (IN_ATTN + MIX) * HIDDEN + N_GDN * (IN_GDN + MIX) * HIDDEN + LAYERS * (_distinct(T) + 1) * 3 * FFN * HIDDEN + VOCAB * HIDDEN
    b = w * IQ3S + LAYERS * (EXPERTS + 1) * HIDDEN * 4                             # weights, router
    b += N_ATTN * (lanes * ctx + T) * 2 * KV_WIDTH * 2                             # cache rows
    b += N_GDN * (lanes + T) * (32 * 128 * 128 + 3 * 8192) * 4 + T * VOCAB * 4     # states read and written, logits
    f = 2 * T * (_row_weights() + VOCAB * HIDDEN) + 4 * N_ATTN * T * (ctx + T) * MIX + 6 * N_GDN * T * 32 * 128 * 128
    return b, f


def _draft(lanes, rows, ctx):
    """(bytes, flops) of one draft-layer call of `rows` rows in all."""
    w = (2 * HIDDEN + IN_ATTN + MIX) * HIDDEN + (_distinct(rows) + 1) * 3 * FFN * HIDDEN + DRAFT_VOCAB * HIDDEN
    b = w * IQ3S + (EXPERTS + 1) * HIDDEN * 4 + (lanes * ctx + rows) * 2 * KV_WIDTH * 2
    f = 2 * rows * ((2 * HIDDEN + IN_ATTN + MIX) * HIDDEN + (TOP_K + 1) * 3 * FFN * HIDDEN) + 2 * lanes * DRAFT_VOCAB * HIDDEN + 4 * rows * ctx * MIX
    return b, f


def work(case):
    kind = case["kind"]
    if kind in ("decode", "tree", "lanes"):
        lanes = case.get("lanes", 1)
        T = sum(_lane_rows(case)) if kind == "lanes" else case["rows"]
        parts = [_window(lanes, T, case["ctx"])]
        if case["draft"]:
            kept = lanes + (T - lanes) / 2
            parts += [_draft(lanes, kept, case["ctx"])] + [_draft(lanes, lanes, case["ctx"])] * (case["draft"] - 1)
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if kind == "prompt":
        n, ctx = case["tokens"], case["ctx"]
        b, f = _window(1, 1, ctx + n)
        w = N_ATTN * (IN_ATTN + MIX) * HIDDEN + N_GDN * (IN_GDN + MIX) * HIDDEN + LAYERS * (_distinct(n) + 1) * 3 * FFN * HIDDEN
        return {"bytes": b + w * IQ3S + N_ATTN * (ctx + n) * 2 * KV_WIDTH * 2 + n * HIDDEN * 2,
                "flops": f + n * (2 * _row_weights() + 4 * N_ATTN * (ctx + n / 2) * MIX + 6 * N_GDN * 32 * 128 * 128)}
    if kind == "park":
        return {"bytes": 4 * ((N_ATTN + 1) * case["ctx"] * 2 * KV_WIDTH * 2 + N_GDN * (32 * 128 * 128 + 3 * 8192) * 4), "flops": 0}
    T = case["rows"]
    if kind == "moe":
        return {"bytes": (_distinct(T) + 1) * 3 * FFN * HIDDEN * IQ3S + (EXPERTS + 1) * HIDDEN * 4 + 2 * T * HIDDEN * 4,
                "flops": 2 * T * ((TOP_K + 1) * 3 * FFN + EXPERTS + 1) * HIDDEN}
    if kind == "attn":
        return {"bytes": (case["ctx"] + T) * 2 * KV_WIDTH * 2 + T * 3 * MIX * 4, "flops": 4 * T * (case["ctx"] + T) * MIX}
    rows, cols = case["out"], case["cols"]
    return {"bytes": LAYERS * (rows * cols * IQ3S + T * (cols + rows * (2 if case["accumulate"] else 1)) * 4), "flops": 2 * LAYERS * T * rows * cols}


def tolerance(case):
    """The matrix products round activations to two int8 levels (windows: 1 / 65,024 of a block's largest value) or to f16
    (prompts); with random weights a row's tenth and eleventh expert are often closer than what that leaves, and a row that
    takes the other one is off by some 1e-2.  Attention's weights are f16.  A parked image is a copy."""
    kind = case["kind"]
    if kind == "park":
        return "exact"
    if kind in ("decode", "tree", "lanes", "prompt"):
        return {"rel": 1e-2, "max": 0.5, "differ": 0.01}
    if kind == "moe":
        return {"rel": 1e-3, "max": 0.1, "differ": 0.01}
    return {"rel": 1e-3 if kind == "attn" else 1e-4}
