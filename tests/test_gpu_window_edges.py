"""Window kernels at the edges of their tiles: attention's 64-position chunks, splits and 128-row tiles, for several head ratios and for
lanes; the router's top K among ties."""
import numpy as np
import pytest

from helpers import rel_err

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# weights are rounded to f16 (2^-11 of each), scores carry f16 keys on both sides: far below the bar of the other attention tests
TOL_ATTN = 2e-3


def _caches(rng, rows, nkv):
    return [rng.standard_normal((rows, nkv, 256)).astype(np.float16) for _ in range(2)]


@pytest.mark.parametrize("pos0,T,nq,nkv", [(0, 1, 16, 2), (63, 1, 16, 2), (64, 16, 16, 2), (59, 5, 16, 2), (60, 17, 16, 2), (4735, 1, 16, 2), (4736, 32, 16, 2),
                                           (200, 32, 4, 4), (130, 7, 6, 2), (9500, 2, 8, 1)])
def test_window_attention_at_tile_edges(F, O, pos0, T, nq, nkv):
    rng = np.random.default_rng(pos0 * 31 + T)
    kc, vc = _caches(rng, pos0 + T, nkv)
    qg = rng.standard_normal((T, nq, 512)).astype(np.float32)
    qg[:, :, :256] *= 3.0                      # the running maxima move
    parent = None if T < 3 else np.array([-1] + [int(rng.integers(0, t)) for t in range(1, T)], np.int32)
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    d_pos = cuda(np.array([pos0], np.int32))
    for par in (None, parent) if parent is not None else (None,):
        got = F.attn(cuda(qg), cuda(kc), cuda(vc), d_pos, None if par is None else cuda(par)).cpu().numpy()
        assert rel_err(got, O.attn(qg, kc.view(np.uint16), vc.view(np.uint16), pos0, par)) < TOL_ATTN


def test_lane_attention_is_each_lane_alone(F):
    """Seven lanes of 1 to 5 rows at uneven positions: every row the bits that its lane alone gives."""
    nq, nkv, rows_each = 16, 2, [1, 4, 3, 2, 5, 1, 3]
    pos = np.array([0, 63, 64, 700, 4800, 5, 130], np.int32)
    rng = np.random.default_rng(3)
    stride, T, n = 4900, sum(rows_each), len(rows_each)
    row0 = np.concatenate([[0], np.cumsum(rows_each)]).astype(np.int32)
    kc, vc = (torch.from_numpy(c).cuda() for c in _caches(rng, n * stride, nkv))
    qg = torch.from_numpy(rng.standard_normal((T, nq, 512)).astype(np.float32)).cuda()
    out = torch.empty((T, nq, 256), device="cuda")
    L = F.lib()
    scratch = torch.empty(L.fnx_attn_scratch_bytes(T, nq, 256), dtype=torch.uint8, device="cuda")
    d_pos, d_row0 = torch.from_numpy(pos).cuda(), torch.from_numpy(row0).cuda()
    lanes = torch.arange(n, dtype=torch.int32, device="cuda")
    F.check(L.fnx_attn_lanes(F.ptr(qg), nq * 512, F.ptr(kc), F.ptr(vc), stride, F.ptr(out), T, n, nq, nkv, 256, F.ptr(d_pos), F.ptr(lanes), F.ptr(d_row0), F.ptr(scratch), None))
    torch.cuda.synchronize()
    for j in range(n):
        a, b = row0[j], row0[j + 1]
        alone = F.attn(qg[a:b].contiguous(), kc[j * stride:(j + 1) * stride], vc[j * stride:(j + 1) * stride], d_pos[j:j + 1])
        assert torch.equal(alone, out[a:b]), j


@pytest.mark.parametrize("E,K,ties", [(512, 10, "few"), (512, 10, "all"), (32, 4, "none"), (16, 10, "few"), (700, 32, "few"), (1024, 10, "few"), (10, 10, "none")])
def test_router_picks_in_order_among_ties(F, E, K, ties):
    """Integer logits through one-hot rows: the picks are the K largest, the lower expert first among equals."""
    T, H = 32, 256
    rng = np.random.default_rng(E + K)
    lg = np.zeros((T, E), np.float32) if ties == "all" else rng.standard_normal((T, E)).astype(np.float32)
    if ties == "few":
        lg = np.round(2 * lg)
    x = np.zeros((T, H), np.float32)
    x[np.arange(T), np.arange(T)] = 1
    W = np.zeros((E + 1, H), np.float32)
    W[:E, :T] = lg.T
    r = F.router_route(torch.from_numpy(W).cuda(), torch.from_numpy(x).cuda(), K)
    assert np.array_equal(r["topi"].cpu().numpy(), np.argsort(-lg, axis=1, kind="stable")[:, :K])
