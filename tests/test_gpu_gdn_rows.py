"""DeltaNet windows at the edges of their batches of four rows, of the rows that a kernel leaves quantised, and of a ring's end."""
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


@pytest.mark.parametrize("T", [8, 9, 12])
def test_a_row_of_an_engine_gives_the_same_bits_in_wide_windows(F, T):
    """On either side of the row count from which the output projection's rows are quantised by a kernel of their own, alone and in lanes."""
    cfg = F.flash_next_config(n_layer=4, hidden=1024, n_expert=32, top_k=4, ffn=256, n_q_head=8, n_kv_head=1, gdn_k_head=2, gdn_v_head=4, vocab=2048, max_ctx=256, max_rows=16,
                              n_seq=3)
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
