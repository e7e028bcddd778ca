"""The engine's own weight layout against the interchange layout: the same weights, windows and prompts, two engines.

fnx_engine_tensor hands a weight matrix out in the interchange layout, and windows read it there from then on; an engine whose
matrices were never asked for reads its own four-bit layout.  Both hold the same numbers and quantise the rows the same way, so
their results differ by the order of f32 sums and by rows whose codes move by one step of 1 / 65,024 of a block's largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
import fnx_b200 as F  # noqa: E402

MATRICES = ("w_in", "w_out", "experts_gu", "experts_dn", "shared_gu", "shared_dn")


def small(**over):
    d = dict(n_layer=4, hidden=1024, n_expert=32, top_k=4, ffn=256, n_q_head=8, n_kv_head=1, gdn_k_head=2, gdn_v_head=4, vocab=2048, max_ctx=2048, max_rows=32, n_seq=4)
    d.update(over)
    return F.flash_next_config(**d)


def wide():   # the benchmark's widths: 4,096-column output projections (split over clusters), 16-row padding of the draft head
    return F.flash_next_config(n_layer=4, n_expert=32, vocab=4096, max_ctx=512, max_rows=32, n_seq=4, draft_vocab=1040)


def pair(cfg):
    engines = []
    for tiles in (False, True):
        e = F.Engine(cfg)
        e.init_synthetic(seed=5, sigma=0.02)
        if tiles:
            names = [f"l{l}.{m}" for l in range(cfg.n_layer) for m in MATRICES] + ["mtp." + m for m in MATRICES] + ["mtp.fc_hid", "mtp.fc_emb", "head"]
            for n in names + (["mtp.head"] if cfg.draft_vocab else []):
                e.tensor(n, torch.uint8)
        engines.append(e)
    return engines


def rows(e, cfg, T):
    r = e.tensor("buf.R", torch.float32).cpu().numpy().reshape(cfg.max_rows, cfg.hidden)[:T]
    lg = e.tensor("buf.logits", torch.float32).cpu().numpy().reshape(cfg.max_rows, cfg.vocab)[:T]
    return r.copy(), lg.copy()


def close(a, b, what):
    err = float(np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b))
    assert err < 3e-4, (what, err)


@pytest.mark.parametrize("make", [small, wide])
def test_windows_and_drafts_agree_between_the_layouts(make):
    cfg = make()
    a, b = pair(cfg)
    try:
        rng = np.random.default_rng(3)
        for T in (1, 4, 5, 9, 16, 20, 21, 32):   # row groups 1 .. 5, one launch and two
            toks = rng.integers(0, cfg.vocab, size=T).tolist()
            got = [e.verify(toks) for e in (a, b)]
            for x, y, w in zip(rows(a, cfg, T), rows(b, cfg, T), ("rows", "logits")):
                close(x, y, (T, w))
            assert got[0] == got[1]
            keep = list(range(min(T, 3)))
            for e in (a, b):
                e.commit(keep)
            assert a.draft(3) == b.draft(3)
        par = [-1, 0, 1, 0, 3, 1, 2]
        toks = rng.integers(0, cfg.vocab, size=7).tolist()
        assert a.verify(toks, par) == b.verify(toks, par)
        for x, y in zip(rows(a, cfg, 7), rows(b, cfg, 7)):
            close(x, y, "tree")
        lanes = [rng.integers(0, cfg.vocab, size=n).tolist() for n in (1, 4, 5)]
        assert a.verify_lanes_rows([1, 2, 3], lanes) == b.verify_lanes_rows([1, 2, 3], lanes)
        for x, y in zip(rows(a, cfg, 10), rows(b, cfg, 10)):
            close(x, y, "lanes")
        for e in (a, b):
            e.commit_lanes([1, 2, 3], [1, 2, 5])
        assert a.draft_lanes([1, 2, 3], 2) == b.draft_lanes([1, 2, 3], 2)
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("n", [70, 1200])   # the products that decode as they go, and the ones from weights decoded once
def test_prompts_agree_between_the_layouts(n):
    cfg = small()
    a, b = pair(cfg)
    try:
        toks = np.random.default_rng(4).integers(0, cfg.vocab, size=n).tolist()
        for e in (a, b):
            e.prompt(toks)
        close(rows(a, cfg, 1)[1], rows(b, cfg, 1)[1], n)
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("E,n", [(32, 1), (32, 8), (32, 9), (32, 48),          # jobs of eight rows up to 2n = 4E
                                 (32, 49), (32, 64), (32, 65), (32, 144), (32, 145),
                                 (2, 63), (2, 64), (2, 65), (2, 129)])    # weights through tensor memory: jobs of 64 rows
def test_prompt_products_at_the_edges_of_their_jobs(E, n):
    """Every row of a prompt, in both layouts, at the lengths where a job or a row group is full, one short or one over.

    (A prompt's last token is a window's, so n rows are n + 1 tokens.)  With a router of zeros every row picks experts 0 and 1, in both engines alike, so these two have exactly n rows and no near tie
    can part the layouts.  The keys of an attention layer behind one DeltaNet layer and its experts are compared row by row: what
    the products read and leave is rounded to f16 three times on the way there (norms, SwiGLU, the key), 2^-11 of a value each."""
    cfg = small(n_layer=2, attn_every=2, n_expert=E, top_k=2, max_ctx=256)
    a, b = pair(cfg)
    try:
        toks = np.random.default_rng(6).integers(0, cfg.vocab, size=n + 1).tolist()
        keys = []
        for e in (a, b):
            for l in range(2):
                e.tensor(f"l{l}.router", torch.float32)[:E * cfg.hidden] = 0.0
            e.prompt(toks)
            keys.append(e.tensor("l1.k_cache", torch.float16).float().reshape(-1, cfg.n_kv_head * cfg.head_dim)[:n].cpu().numpy())
        err = np.linalg.norm(keys[0] - keys[1], axis=1) / np.linalg.norm(keys[1], axis=1)
        assert err.max() < 3 * 2.0 ** -11, (int(err.argmax()), float(err.max()))
    finally:
        a.close()
        b.close()


@pytest.mark.parametrize("n", [11, 15, 16, 17, 32, 33, 47, 63, 79, 113])
def test_prompt_products_at_every_sixteen_rows(n):
    """As above, where the products' N changes (a job's rows in sixteens) and where the dense jobs take fewer rows, for all of them to run at once."""
    test_prompt_products_at_the_edges_of_their_jobs(2, n)


@pytest.mark.parametrize("n", [320, 385, 513, 1100])   # in- and output projection: decoded as they go, or once; tiles of 256 rows full, one over
def test_prompt_projections_of_both_forms(n):
    """As above, at the benchmark's widths: the keys are a projection of rows that an output projection and experts left (f16 three times)."""
    cfg = F.flash_next_config(n_layer=2, attn_every=2, n_expert=2, top_k=2, vocab=2048, max_ctx=1280, max_rows=32, n_seq=1)
    a, b = pair(cfg)
    try:
        toks = np.random.default_rng(7).integers(0, cfg.vocab, size=n + 1).tolist()
        keys = []
        for e in (a, b):
            e.prompt(toks)
            keys.append(e.tensor("l1.k_cache", torch.float16).float().reshape(-1, cfg.n_kv_head * cfg.head_dim)[:n].cpu().numpy())
        err = np.linalg.norm(keys[0] - keys[1], axis=1) / np.linalg.norm(keys[1], axis=1)
        assert err.max() < 3 * 2.0 ** -11, (int(err.argmax()), float(err.max()))
    finally:
        a.close()
        b.close()


def test_a_matrix_asked_for_comes_back_in_the_interchange_layout():
    """Bit for bit the tiles that the same seeded weights give through the operators, padded rows included."""
    cfg = small(draft_vocab=1040)
    e = F.Engine(cfg)
    try:
        e.init_synthetic(seed=5, sigma=0.02)
        w = torch.empty(1040 * cfg.hidden, device="cuda")
        F.fill_normal(w, 0.02, 5, (61 * 16 + 2) << 12)
        want = F.iq3s_retile(F.iq3s_quantize(w), 1040, cfg.hidden)
        assert torch.equal(e.tensor("mtp.head", torch.uint8), want)
        gu = 2 * cfg.ffn
        w = torch.empty(gu * cfg.hidden, device="cuda")
        F.fill_normal(w, 0.02, 5, ((1 * 16 + 4) << 12) | 7)
        per = F.iq3s_bytes(gu, cfg.hidden)
        assert torch.equal(e.tensor("l1.experts_gu", torch.uint8)[7 * per:8 * per], F.iq3s_retile(F.iq3s_quantize(w), gu, cfg.hidden))
    finally:
        e.close()


@pytest.mark.parametrize("n", [30, 200])
def test_scales_past_the_largest_f16(tmp_path, n):
    """A block scale d (1 + 2 s) that overflows f16, in a file's matrix: a prompt's weights of that block are infinite with the sign of theirs, in
    both layouts (every value of the normed rows is 1 here, so a row of the values' projection with weights of one sign sums to that infinity)."""
    from gguf_files import model_meta, tiny_model_tensors, write_gguf
    cfg = small(n_layer=1, attn_every=1, n_expert=4, top_k=2, vocab=512, max_ctx=512)
    a = F.Engine(cfg)
    a.init_synthetic(seed=5, sigma=0.02)
    tensors = tiny_model_tensors(F, a, cfg)
    a.close()
    tensors["token_embd.weight"][7] = 1.0
    blk = tensors["blk.0.attn_v.weight"][0].reshape(-1, cfg.hidden // 256, 110)
    for row, signs in ((0, 0x00), (1, 0xFF)):
        blk[row, :, :2] = np.frombuffer(np.float16(60000).tobytes(), np.uint8)
        blk[row, :, 74:106] = signs
        blk[row, :, 106:] = 0xFF
    path = tmp_path / "huge.gguf"
    write_gguf(path, model_meta(cfg), tensors)
    for asked in (False, True):
        g = F.Gguf(path)
        e = F.Engine(g.model_config(max_ctx=cfg.max_ctx, max_rows=cfg.max_rows))
        try:
            e.load_gguf(g)
            if asked:
                e.tensor("l0.w_in", torch.uint8)
            with pytest.raises(F.FnxError):              # (the logits are not finite)
                e.prompt([7] * (n + 1))
            v = e.tensor("l0.v_cache", torch.float16).reshape(-1, cfg.n_kv_head * cfg.head_dim)[:n]
            assert torch.isposinf(v[:, 0]).all() and torch.isneginf(v[:, 1]).all() and torch.isfinite(v[:, 2:]).all(), asked
        finally:
            e.close()


@pytest.mark.parametrize("n", [48, 200])   # jobs of eight rows and of 64
def test_scales_that_are_large_but_fit(tmp_path, n):
    """Experts with a few rows of block scales d of 1,000 (and normed rows small enough for it): the decode's form for large scales, against the
    interchange layout, key by key as in test_prompt_products_at_the_edges_of_their_jobs."""
    from gguf_files import model_meta, tiny_model_tensors, write_gguf
    cfg = small(n_layer=2, attn_every=2, n_expert=32, top_k=2, vocab=512, max_ctx=512)
    a = F.Engine(cfg)
    a.init_synthetic(seed=5, sigma=0.02)
    tensors = tiny_model_tensors(F, a, cfg)
    a.close()
    # a large row's block sums at most 1,000 x 15 x (256 x 1,024)^1/2 x 3e-5 = 230 of a normed row of 1,024: silu(gate) x up stays inside f16
    tensors["blk.0.post_attention_norm.weight"] *= 3e-5
    for l in range(2):
        tensors[f"blk.{l}.ffn_gate_inp.weight"][:] = 0.0
    for name, cols in (("ffn_gate_exps", cfg.hidden), ("ffn_up_exps", cfg.hidden), ("ffn_down_exps", cfg.ffn)):
        blk = tensors[f"blk.0.{name}.weight"][0].reshape(cfg.n_expert, -1, cols // 256, 110)
        blk[:, 3::40, 0, :2] = np.frombuffer(np.float16(1000).tobytes(), np.uint8)
        blk[:, 3::40, 0, 106:] = 0
    path = tmp_path / "large.gguf"
    write_gguf(path, model_meta(cfg), tensors)
    keys = []
    for asked in (False, True):
        g = F.Gguf(path)
        e = F.Engine(g.model_config(max_ctx=cfg.max_ctx, max_rows=cfg.max_rows))
        try:
            e.load_gguf(g)
            if asked:
                for m in MATRICES[2:]:
                    e.tensor("l0." + m, torch.uint8)
            e.prompt(np.random.default_rng(6).integers(0, cfg.vocab, size=n + 1).tolist())
            assert e.error_bits() == 0
            keys.append(e.tensor("l1.k_cache", torch.float16).float().reshape(-1, cfg.n_kv_head * cfg.head_dim)[:n].cpu().numpy())
        finally:
            e.close()
    err = np.linalg.norm(keys[0] - keys[1], axis=1) / np.linalg.norm(keys[1], axis=1)
    assert err.max() < 3 * 2.0 ** -11, (int(err.argmax()), float(err.max()))
