"""The job list of a window, word for word: either side of eight rows, experts that four, five and all rows picked, ranges of experts, the most
experts and picks there can be."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def jobs_of(topi, E, lo, hi, shared, tok):
    T, K = topi.shape
    out = []
    for e in range(lo, hi):
        at = [(t, t * K + k) for t in range(T) for k in range(K) if topi[t, k] == e]
        out += [(e, at[i:i + tok]) for i in range(0, len(at), tok)]
    routed = len(out)
    if shared:
        at = [(t, T * K + t) for t in range(T)]
        out += [(E, at[i:i + tok]) for i in range(0, T, tok)]
    words = np.zeros((len(out), 2 + 2 * tok), np.int32)
    for w, (e, at) in zip(words, out):
        w[:2] = e, len(at)
        w[2:2 + len(at)] = [t for t, _ in at]
        w[2 + tok:2 + tok + len(at)] = [o for _, o in at]
    return words, routed


@pytest.mark.parametrize("T", [1, 2, 4, 5, 7, 8, 9, 20, 32])
@pytest.mark.parametrize("E,K,same", [(8, 8, 0), (16, 4, 1), (33, 10, 0), (512, 10, 0), (512, 10, 1), (1024, 32, 0)])
def test_job_list_word_for_word(F, T, E, K, same):
    H = 256
    g = torch.Generator(device="cuda").manual_seed(E + T)
    x = torch.randn((1 if same else T, H), device="cuda", generator=g).expand(T, H).contiguous()   # (rows alike pick alike)
    wr = 0.1 * torch.randn((E + 1, H), device="cuda", generator=g)
    for lo, hi, shared in ((0, E, True), (E // 4, E - 1, False), (E // 2, E // 2, True)):
        r = F.router_route(wr, x, K, e_lo=lo, e_hi=hi, add_shared=shared)
        want, _ = jobs_of(r["topi"].cpu().numpy(), E, lo, hi, shared, F.JOB_TOK)
        n = int(r["njobs"][0].item())
        got = r["jobs"].cpu().numpy().tobytes()
        got = np.frombuffer(got, np.int32).reshape(-1, 2 + 2 * F.JOB_TOK)[:n]
        assert n == len(want) and np.array_equal(got, want), (lo, hi)
