"""The sampler's 64 candidates at the edges of their selection: eight slices of a row, a warp's second largest, more equal values than a slice keeps."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("V", [64, 65, 511, 513, 8191, 8200, 9000, 40003, 151936, 300007])
def test_top_tokens_are_the_largest_keys(F, V):
    rng = np.random.default_rng(V)
    rows = [rng.standard_normal(V), np.zeros(V), np.round(rng.standard_normal(V) * 2), np.arange(V), -np.arange(V), rng.standard_normal(V)]
    logits = np.stack(rows).astype(np.float32)
    logits[5, V // 2:] = -np.inf                         # (a mask; infinities are values like others)
    logits[5, : V // 3] = 3.0                            # more equal ones than a slice keeps, where the row is long
    logits[0, V - 1] = np.inf
    logits[2, :3] = [0.0, -0.0, 0.0]                     # (of two zeros the positive one is the larger)
    bits = logits.view(np.uint32).astype(np.uint64)
    key = np.where(bits >> 31, ~bits & 0xFFFFFFFF, bits | 0x80000000) << np.uint64(32) | (0xFFFFFFFF - np.arange(V, dtype=np.uint64))
    want = np.argsort(key, axis=1)[:, ::-1][:, :64]      # value first, the lower index among equals
    v, i = F.top_tokens(torch.from_numpy(logits).cuda())
    assert np.array_equal(i.cpu().numpy(), want)
    assert np.array_equal(v.cpu().numpy().view(np.uint32), np.take_along_axis(logits, want, 1).view(np.uint32))
    # a row that does not start on a 16-byte boundary
    flat = torch.from_numpy(np.concatenate([np.zeros(1, np.float32), logits[0]])).cuda()
    _, one = F.top_tokens(flat[1:].view(1, V))
    assert np.array_equal(one.cpu().numpy()[0], want[0])


def test_top_tokens_and_argmax_of_more_rows_than_a_grids_second_dimension(F):
    T, V = 65_537, 70
    logits = torch.randn((T, V), device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    v, i = F.top_tokens(logits)
    want = logits.sort(dim=1, descending=True)   # (equal values may come in another order: the values are compared, and that the ids lead to them)
    assert torch.equal(v, want.values[:, :64]) and torch.equal(logits.gather(1, i.long()), v)
    assert torch.equal(F.argmax(logits)[1], want.values[:, 0])


def test_accept_sample_with_draft_distributions(F, O):
    """Drafts of their own distributions (up to 64 candidates, in any order) beside fixed ones: counts and tokens as the oracle's."""
    rng = np.random.default_rng(12)
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    for it in range(80):
        T, V = int(rng.integers(1, 9)), 2000
        cv, ci = O.top_tokens((rng.standard_normal((T, V)) * 3).astype(np.float32))
        tok = rng.integers(0, V, size=T).astype(np.int32)
        qi, qp, qn = np.zeros((T, 64), np.int32), np.zeros((T, 64)), np.zeros(T, np.int32)
        for t in range(T):
            if rng.random() < 0.7:
                m = int(rng.integers(1, 65))
                p = rng.random(m)
                qn[t], qi[t, :m], qp[t, :m] = m, ci[t, rng.permutation(64)[:m]], p / p.sum()
            if t + 1 < T and rng.random() < 0.8:
                tok[t + 1] = ci[t, int(rng.integers(0, 4))]
        s = [O.Sampling(0.7, 1.0, 0.0, 0), O.Sampling(1.0, 0.9, 0.05, 40), O.Sampling(0.3, 1.0, 0.2, 0), O.Sampling(2.0, 0.5, 0.0, 7)][it % 4]
        n, em = O.accept_sample(cv, ci, tok, s, seed=9, seq=it, step=3, q_ids=qi, q_p=qp, q_n=qn)
        gn, _, gem = F.accept_sample(cuda(cv), cuda(ci), cuda(tok), F.Sampling(s.temperature, s.top_p, s.min_p, s.top_k), 9, it, cuda(np.array([3], np.int32)), cuda(qi),
                                     cuda(qp), cuda(qn))
        assert gn == n and gem == list(em), it


@pytest.mark.parametrize("T,V", [(1, 1), (3, 5), (2, 31), (5, 1023), (1, 40528), (3, 40525), (32, 32771), (20, 151936), (1100, 64)])
def test_argmax_over_a_cluster(F, T, V):
    """Eight slices of a row, aligned to 16 bytes or not: the first of the largest values, and a row with a value that is not finite is reported."""
    rng = np.random.default_rng(V)
    logits = np.round(rng.standard_normal((T, V)) * 3).astype(np.float32) + 0.0    # (many ties; no negative zeros, which are below the positive one)
    i, v, err = F.argmax(torch.from_numpy(logits).cuda())
    assert np.array_equal(i.cpu().numpy(), logits.argmax(1)) and np.array_equal(v.cpu().numpy(), logits.max(1)) and int(err.item()) == 0
    logits[T - 1, V - 1] = -np.inf
    assert int(F.argmax(torch.from_numpy(logits).cuda())[2].item()) == 16


@pytest.mark.parametrize("T", [15, 16, 25, 33, 34, 74, 75])
@pytest.mark.parametrize("V", [65, 700, 1023, 1024, 8191, 8192, 16383, 16384, 50001, 100000])
def test_rows_by_eight_blocks_to_one(F, T, V):
    """Either side of where a row's blocks become fewer: the candidates and the largest of rows without ties, with many, and all alike."""
    g = torch.Generator(device="cuda").manual_seed(T * V)
    logits = torch.randn((T, V), device="cuda", generator=g) + 0.0
    logits[T // 2:] = torch.round(logits[T // 2:] * 2) + 0.0             # (no negative zeros)
    logits[T - 1] = -1.5
    logits[T - 2] = torch.round(logits[T - 2] * 1e6) * 1e-6 + 1000.0     # (values that share most of their bits)
    want_v, want_i = logits.sort(dim=1, descending=True, stable=True)    # the lower index among equals
    v, i = F.top_tokens(logits)
    assert torch.equal(v, want_v[:, :64]) and torch.equal(i.long(), want_i[:, :64])
    i, v, err = F.argmax(logits)
    assert torch.equal(v, want_v[:, 0]) and torch.equal(i.long(), want_i[:, 0]) and int(err.item()) == 0
