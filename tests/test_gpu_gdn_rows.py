"""DeltaNet windows at the edges of their batches of four rows, of the clusters that leave a row quantised, and of a ring's end."""
import numpy as np
import pytest

from helpers import rel_err
from test_gpu_ops import _gdn_inputs, dev

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("T", [3, 4, 5, 8, 9, 13, 17, 32])
def test_rows_of_a_window_are_the_oracles_and_each_alone(F, O, T):
    """Against the oracle (the bars of test_gdn_core_matches_oracle), a chain and a tree; and the chain's rows one window each: the same bits."""
    nk, nv, hs, NS = 2, 4, 128, 33
    rng = np.random.default_rng(T)
    cur = NS - 2                                       # the slots pass the ring's end
    ch, qkvz, ab, convw, dt, a, nw = _gdn_inputs(rng, T, nk, nv, hs)
    S = (0.1 * rng.standard_normal((NS, nv, hs, hs))).astype(np.float32)
    hist = rng.standard_normal((NS, 3, ch)).astype(np.float32)
    const = [dev(v) for v in (convw, dt, a, nw)]

    def run(rows, d_S, d_hist, at, parent=None):
        return F.gdn_core(dev(qkvz[rows]), dev(ab[rows]), d_hist, *const, d_S, dev(np.array([at], np.int32)), parent, nk, nv, hs)

    for parent in (None, [-1] + [int(rng.integers(max(0, t - 4), t)) for t in range(1, T)]):
        d_S, d_hist, S1, h1 = dev(S), dev(hist), S.copy(), hist.copy()
        y = run(slice(0, T), d_S, d_hist, cur, None if parent is None else dev(np.array(parent, np.int32)))
        ref = O.gdn_core(qkvz, ab, h1, convw, dt, a, nw, S1, cur, parent, nk, nv, hs)
        assert rel_err(y.cpu().numpy(), ref) < 2e-3 and rel_err(d_S.cpu().numpy(), S1) < 1e-4
        assert np.array_equal(d_hist.cpu().numpy(), h1)
        if parent is None:
            together = y, d_S, d_hist
    d_S, d_hist = dev(S), dev(hist)
    for t in range(T):
        assert torch.equal(run(slice(t, t + 1), d_S, d_hist, (cur + t) % NS)[0], together[0][t]), f"row {t}"
    assert torch.equal(d_S, together[1]) and torch.equal(d_hist, together[2])


def _small_config(F, nv=4):
    return F.flash_next_config(n_layer=4, hidden=1024, n_expert=32, top_k=4, ffn=256, n_q_head=8, n_kv_head=1, gdn_k_head=nv // 2, gdn_v_head=nv, vocab=2048, max_ctx=256, max_rows=16,
                               n_seq=6)


@pytest.mark.parametrize("nv,lens", [(4, [1, 1]), (4, [1, 2]), (4, [2, 1]), (4, [1, 1, 1]), (4, [2, 2]), (4, [4, 4]), (4, [5, 4]), (64, [1, 2, 1, 1]), (64, [1, 2, 1, 1, 1])])
def test_rows_in_several_lanes_give_the_bits_of_each_alone(F, nv, lens):
    """On either side of the eight rows in all, and of the 128 clusters (value heads / 2 x lanes), beyond which the rows are quantised by a kernel of their own; and the next window from the
    states that these leave."""
    cfg = _small_config(F, nv)
    eng = F.Engine(cfg)
    try:
        eng.init_synthetic(seed=0, sigma=0.02)
        toks = np.random.default_rng(1).integers(0, cfg.vocab, size=10).tolist()
        logits = eng.tensor("buf.logits", torch.float32).view(cfg.max_rows, cfg.vocab)
        for s in range(6):
            eng.reset(s)
        eng.verify(toks, seq=0)
        together, seqs, at = logits[:10].clone(), [3, 1, 2, 5, 4][:len(lens)], [0] * len(lens)
        for _ in range(2):
            eng.verify_lanes_rows(seqs, [toks[a:a + n] for a, n in zip(at, lens)])
            want = torch.cat([together[a:a + n] for a, n in zip(at, lens)])
            assert torch.equal(logits[:len(want)], want), at
            eng.commit_lanes(seqs, lens)
            at = lens
    finally:
        eng.close()


@pytest.mark.parametrize("T", [8, 9, 12])
def test_a_row_of_an_engine_gives_the_same_bits_in_wide_windows(F, T):
    """On either side of the eight rows beyond which the output projection's rows are quantised by a kernel of their own, alone and in two lanes."""
    cfg = _small_config(F)
    eng = F.Engine(cfg)
    try:
        eng.init_synthetic(seed=0, sigma=0.02)
        toks = np.random.default_rng(T).integers(0, cfg.vocab, size=T).tolist()
        logits = eng.tensor("buf.logits", torch.float32).view(cfg.max_rows, cfg.vocab)
        for s in range(3):
            eng.reset(s)
        eng.verify(toks, seq=0)
        together = logits[:T].clone()
        n = min(T - 4, 5)
        eng.verify_lanes_rows([1, 2], [toks[:n], toks[:4]])
        assert torch.equal(logits[:n], together[:n]) and torch.equal(logits[n:n + 4], together[:4])
        for i, t in enumerate(toks):
            eng.verify([t], seq=0)
            assert torch.equal(logits[0], together[i]), f"row {i}"
            eng.commit([0], seq=0)
    finally:
        eng.close()


def _lanes(F, d_x, d_ab, d_hist, const, d_S, cur, seqs, lens, max_rows, y, nk, nv):
    L, P, hs = F.lib(), F.ptr, 128
    row0 = dev(np.concatenate([[0], np.cumsum(lens)]).astype(np.int32))
    F.check(L.fnx_gdn_core_lanes(P(d_x), d_x.stride(0), P(d_ab), d_ab.stride(0), P(d_hist), d_hist.stride(0), *map(P, const), P(d_S), d_S.stride(0), P(cur), d_S.shape[1],
                                 P(dev(np.array(seqs, np.int32))), P(row0), len(lens), max_rows, P(y), nk, nv, hs, 1e-6, F._stream()))


@pytest.mark.parametrize("lens,seqs", [([1], [2]), ([1, 1], [1, 0]), ([4, 5, 1], [2, 0, 1]), ([2, 3, 8, 0, 9], [4, -1, 0, 3, 1]), ([32], [0])])
def test_lanes_of_the_operator_are_each_alone(F, lens, seqs):
    """The lanes form against fnx_gdn_core of each lane: the same bits, from a longest lane of one row to one of FNX_MAX_ROWS; an empty lane and one of a negative sequence change nothing."""
    nk, nv, hs, n_seq = 2, 4, 128, 5
    NS, T = max(lens) + 1, sum(lens)
    rng = np.random.default_rng(T)
    ch, qkvz, ab, convw, dt, a, nw = _gdn_inputs(rng, T, nk, nv, hs)
    const = [dev(v) for v in (convw, dt, a, nw)]
    d_S, d_hist = dev((0.1 * rng.standard_normal((n_seq, NS, nv, hs, hs))).astype(np.float32)), dev(rng.standard_normal((n_seq, NS, 3, ch)).astype(np.float32))
    want_S, want_hist, at = d_S.clone(), d_hist.clone(), rng.integers(0, NS, size=n_seq).astype(np.int32)
    d_x, d_ab = dev(qkvz), dev(ab)
    y = torch.full((T, nv * hs), 7.0, device="cuda")
    want = y.clone()
    _lanes(F, d_x, d_ab, d_hist, const, d_S, dev(at), seqs, lens, max(lens), y, nk, nv)
    r = 0
    for n, s in zip(lens, seqs):
        if n and s >= 0:
            want[r:r + n] = F.gdn_core(d_x[r:r + n], d_ab[r:r + n], want_hist[s], *const, want_S[s], dev(at[s:s + 1]), None, nk, nv, hs)
        r += n
    assert torch.equal(y, want) and torch.equal(d_S, want_S) and torch.equal(d_hist, want_hist)


def test_lanes_of_more_rows_than_a_window_are_refused(F):
    """FNX_MAX_ROWS + 1 rows a lane: refused whatever the lanes hold (here: nothing, so that a call that is taken has no row to work on)."""
    nk, nv, hs, NS = 2, 4, 128, 40
    ch, qkvz, ab, convw, dt, a, nw = _gdn_inputs(np.random.default_rng(0), 1, nk, nv, hs)
    args = [F, dev(qkvz), dev(ab), torch.zeros((1, NS, 3, ch), device="cuda"), [dev(v) for v in (convw, dt, a, nw)], torch.zeros((1, NS, nv, hs, hs), device="cuda"),
            dev(np.zeros(1, np.int32)), [0], [0]]
    _lanes(*args, F.MAX_ROWS, torch.zeros((1, nv * hs), device="cuda"), nk, nv)
    with pytest.raises(F.FnxError, match="lanes of up to 33 rows"):
        _lanes(*args, F.MAX_ROWS + 1, torch.zeros((1, nv * hs), device="cuda"), nk, nv)
    torch.cuda.synchronize()
