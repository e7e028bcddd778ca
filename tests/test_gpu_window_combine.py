"""The window's weighted sum: picks that name no expert of the range, picks of weight 0, over addends that nobody wrote."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

E, H = 48, 512


def fixture(T, K):
    """A routing in which picks are masked (id -1 or E, a weight that is not 0) or weigh 0, their addends NaN; and the same with all of
    these at weight 0 over finite addends."""
    g = torch.Generator(device="cuda").manual_seed(100 * T + K)
    rn = lambda *s: torch.randn(s, device="cuda", generator=g)
    topi = torch.stack([torch.randperm(E, generator=torch.Generator().manual_seed(t))[:K] for t in range(T)]).int().cuda()
    topw = torch.rand((T, K), device="cuda", generator=g) + 0.1
    masked, zero = (torch.rand((T, K), device="cuda", generator=g) < 0.25 for _ in range(2))
    masked[0] = True                                     # (a whole row)
    part = rn(T * K + T, H)
    dirty = part.clone()
    dirty[:T * K][(masked | zero).reshape(-1)] = float("nan")
    ids = torch.where(masked, torch.where(topi % 2 == 0, -1, E).int(), topi)
    w = torch.where(zero, 0.0, topw)
    return dict(ids=ids, w=w, dirty=dirty, topi=topi, w0=torch.where(masked, 0.0, w), part=part, logits=rn(T, E + 1), old=rn(T, H))


def combine(F, part, topi, topw, logits, lo, hi, shared, old):
    T, K = topi.shape
    out = old.clone()
    F.check(F.lib().fnx_moe_combine(F.ptr(part), F.ptr(topi), F.ptr(topw), F.ptr(logits), T, E, H, K, lo, hi, int(shared), F.ptr(out), 1, None))
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("T,K", [(1, 1), (5, 10), (20, 11), (32, 32)])
@pytest.mark.parametrize("lo,hi,shared", [(0, E, True), (0, E, False), (0, E // 2, True), (E // 2, E, False)])
def test_picks_that_do_not_count_add_nothing(F, T, K, lo, hi, shared):
    f = fixture(T, K)
    want = combine(F, f["part"], f["topi"], f["w0"], f["logits"], lo, hi, shared, f["old"])
    got = combine(F, f["dirty"], f["ids"], f["w"], f["logits"], lo, hi, shared, f["old"])
    assert torch.isfinite(want).all() and torch.equal(got, want)


@pytest.mark.parametrize("T,K", [(1, 1), (5, 10), (13, 17), (32, 32)])
def test_the_form_that_leaves_the_image_leaves_them_out_too(F, T, K):
    f = fixture(T, K)
    want = combine(F, f["dirty"], f["ids"], f["w"], f["logits"], 0, E, True, f["old"])
    got = f["old"].clone()
    F.moe_combine_image(f["dirty"], dict(topi=f["ids"], topw=f["w"], logits=f["logits"]), T, E, H, K, got, torch.ones(H, device="cuda"))
    assert torch.isfinite(want).all() and torch.equal(got, want)
