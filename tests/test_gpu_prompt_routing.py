"""A prompt's routing at the edges of its kernels: the router's tiles of sixteen rows by sixteen experts, and the job lists either side of
the number of picks that one block takes."""
import numpy as np
import pytest

from test_gpu_ops import _moe_fixture

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("E,H,T", [(15, 256, 33), (16, 1024, 47), (31, 2048, 48), (32, 512, 49), (512, 2048, 64), (512, 2048, 65)])
@pytest.mark.parametrize("normed", [False, True])
def test_router_tiles(F, E, H, T, normed):
    """Against float64: each product is good to 3 x 2^-22 of itself (two splits, the dropped low x low), the partial sums of sixteen
    columns and the f32 sums behind them to some 2^-21 of the sum of magnitudes together."""
    rng = np.random.default_rng(E + T)
    wr = (0.02 * rng.standard_normal((E + 1, H))).astype(np.float32)
    x = (3.0 * rng.standard_normal((T, H))).astype(np.float32)
    nw = (1.0 + 0.05 * rng.standard_normal(H)).astype(np.float32)
    cuda = lambda a: torch.from_numpy(a).cuda()
    _, _, lg = F.router_rows(cuda(wr), cuda(x), 4, norm_w=cuda(nw) if normed else None)
    xn = x.astype(np.float64)
    if normed:
        xn = xn / np.sqrt((xn * xn).mean(axis=1, keepdims=True) + 1e-6) * nw
    bound = (3 * 2.0 ** -22 + 2.0 ** -21) * (np.abs(xn) @ np.abs(wr.astype(np.float64)).T)
    assert (np.abs(lg.cpu().numpy() - xn @ wr.astype(np.float64).T) < bound).all()


@pytest.mark.parametrize("T", [1, 819])   # ten picks a row: 8,190 fill one block's list, 8,200 take the lists of several
def test_job_lists_do_not_show_in_the_rows(F, T):
    """A row's experts give the same bits whichever rows it comes with and wherever its entry lies."""
    E, H, Fn, K = 16, 512, 256, 10
    fx = _moe_fixture(F, E, H, Fn, seed=29)
    x = torch.randn((820, H), device="cuda", generator=torch.Generator(device="cuda").manual_seed(8))
    topi, topw, logits = F.router_rows(fx["wr"], x, K)
    run = lambda n: F.moe_prefill(fx["gu_t"], fx["dn_t"], fx["sh_gu_t"], fx["sh_dn_t"], topi[:n].contiguous(), topw[:n].contiguous(), logits[:n].contiguous(), x[:n].contiguous(), Fn)
    (some, err), (every, err2) = run(T), run(820)
    assert int(err.item()) == 0 and int(err2.item()) == 0
    assert torch.equal(some, every[:T])


@pytest.mark.parametrize("K,add_shared", [(1, True), (10, True), (11, False), (11, True), (12, True), (24, True), (32, True)])
def test_combine_of_many_picks(F, K, add_shared):
    """The weighted sum of a row's addends (eleven at a time) at the edges of its passes, with every expert on this rank and with a range of
    them.  Every value is one f32 multiply-add per addend, in pick order."""
    E, H, Fn, T = 32, 512, 256, 19
    fx = _moe_fixture(F, E, H, Fn, seed=31)
    g = torch.Generator(device="cuda").manual_seed(K)
    x = torch.randn((T, H), device="cuda", generator=g)
    topi = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(t))[:K] for t in range(T)]).int().cuda()
    topw = torch.rand((T, K), device="cuda", generator=g)
    topw[3, 0] = 0.0
    logits = torch.randn((T, E + 1), device="cuda", generator=g)
    old = torch.randn((T, H), device="cuda", generator=g)
    run = lambda w, **kw: F.moe_prefill(fx["gu_t"], fx["dn_t"], fx["sh_gu_t"], fx["sh_dn_t"], topi, w, logits, x, Fn, **kw)[0]
    unit = []                                            # each addend by itself, weight 1
    for k in range(K):
        w = torch.zeros_like(topw)
        w[:, k] = 1.0
        unit.append(run(w, add_shared=False).double())
    want = sum(topw[:, k:k + 1].double() * unit[k] for k in range(K))
    size = sum(topw[:, k:k + 1].double() * unit[k].abs() for k in range(K))
    if add_shared:
        sh = run(torch.zeros_like(topw), add_shared=True).double()
        want, size = want + sh, size + sh.abs()
    bound = (K + 3) * 2.0 ** -24 * (size + old.abs().double()) + 1e-30
    assert ((run(topw, add_shared=add_shared).double() - want).abs() <= bound).all()
    assert ((run(topw, add_shared=add_shared, out=old.clone(), accumulate=True).double() - (want + old.double())).abs() <= bound).all()
    part = run(topw, add_shared=add_shared, e_lo=0, e_hi=E // 2)
    rest = run(topw, add_shared=False, e_lo=E // 2, e_hi=E, out=part.clone(), accumulate=True)
    assert ((rest.double() - want).abs() <= 2 * bound).all()


@pytest.mark.parametrize("K,T", [(1, 3), (10, 40), (11, 19), (24, 21),   # one block's job list, one pass of addends and more
                                 (10, 830), (4, 1030)])                    # several blocks' list; rows by tensor copies
@pytest.mark.parametrize("half", [False, True])
def test_a_pick_that_names_no_expert_adds_nothing(F, K, T, half):
    """Ids of -1 and E (a masked row, a masked pick) with weights that are not 0: no job has them, so nobody writes their addends, and the
    sum is that of the other picks, bit for bit, whatever the scratch held."""
    E, H, Fn = 32, 512, 256
    fx = _moe_fixture(F, E, H, Fn, seed=31)
    g = torch.Generator(device="cuda").manual_seed(K)
    x, logits, topw = torch.randn((T, H), device="cuda", generator=g), torch.randn((T, E + 1), device="cuda", generator=g), torch.rand((T, K), device="cuda", generator=g) + 0.1
    topi = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(t))[:K] for t in range(T)]).int().cuda()
    out_of_range = torch.rand((T, K), device="cuda", generator=g) < 0.3
    out_of_range[0] = True
    ids = torch.where(out_of_range, torch.where(topi % 2 == 0, -1, E).int(), topi)
    nbytes = F.lib().fnx_moe_prefill_scratch_bytes(T, K, E, H, Fn)
    run = lambda i, w, **kw: F.moe_prefill(fx["gu_t"], fx["dn_t"], fx["sh_gu_t"], fx["sh_dn_t"], i, w, logits, x, Fn, e_hi=E // 2 if half else E,
                                           scratch=torch.full((nbytes,), 255, dtype=torch.uint8, device="cuda"), **kw)[0]   # (floats of 0xFFFFFFFF: NaN)
    for shared in (True, False):
        got, want = run(ids, topw, add_shared=shared), run(topi, torch.where(out_of_range, 0.0, topw), add_shared=shared)
        assert torch.isfinite(want).all() and torch.equal(got, want), shared


@pytest.mark.parametrize("lo,hi", [(0, 32), (0, 16)])
@pytest.mark.parametrize("K", [4, 12])
def test_addends_that_are_not_finite(F, K, lo, hi):
    """Picks of weight 0 leave nothing of theirs in a row, finite or not; the shared expert is no pick: where its gate has gone to 0, what is
    not finite in it still shows."""
    E, H, Fn, T = 32, 512, 256, 9
    fx = _moe_fixture(F, E, H, Fn, seed=31)
    g = torch.Generator(device="cuda").manual_seed(K)
    x, old = torch.randn((T, H), device="cuda", generator=g), torch.randn((T, H), device="cuda", generator=g)
    x[4:6] = float("inf")                                # (every expert's results for these two rows are NaN)
    topi = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(t))[:K] for t in range(T)]).int().cuda()
    topw, logits = torch.rand((T, K), device="cuda", generator=g) + 0.1, torch.randn((T, E + 1), device="cuda", generator=g)
    topw[4:6] = 0.0
    logits[4:6, E] = -200.0
    run = lambda shared: F.moe_prefill(fx["gu_t"], fx["dn_t"], fx["sh_gu_t"], fx["sh_dn_t"], topi, topw, logits, x, Fn, e_lo=lo, e_hi=hi, add_shared=shared, out=old.clone(),
                                       accumulate=True)[0]
    routed, every = run(False), run(True)
    assert torch.equal(routed[4:6], old[4:6]) and torch.isnan(every[4:6]).all()
    assert torch.isfinite(routed).all() and torch.isfinite(torch.cat([every[:4], every[6:]])).all()
