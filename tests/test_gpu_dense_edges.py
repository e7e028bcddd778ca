"""The operators' dense product where its work is cut: one 16-row unit, a unit a block, one more; fewer items than warps; one to three blocks of rows
a warp to quantise, and more."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows", [16, 48, 148 * 16, 149 * 16])
@pytest.mark.parametrize("cols,T", [(256, 1), (256, 12), (512, 5), (1024, 9), (2048, 3), (2048, 5), (2048, 6), (2048, 12), (4096, 1), (4096, 8)])
@pytest.mark.parametrize("normed", [False, True])
def test_dense_against_64_bits(F, rows, cols, T, normed):
    g = torch.Generator(device="cuda").manual_seed(rows + cols + T)
    tiles = F.iq3s_retile(F.iq3s_quantize(torch.randn(rows * cols, device="cuda", generator=g) * 0.02), rows, cols)
    w = F.iq3s_dequant_tiles(tiles, rows, cols).double()
    x = torch.randn((T, cols), device="cuda", generator=g)
    nw = 1.0 + 0.1 * torch.randn(cols, device="cuda", generator=g) if normed else None
    old = torch.randn((T, rows), device="cuda", generator=g)
    out, err = old.clone(), F.new_err()
    F.dense(tiles, rows, cols, x, norm_w=nw, out=out, accumulate=True, err=err)
    plain = F.dense(tiles, rows, cols, x, norm_w=nw, err=err)
    plain = plain[0] if isinstance(plain, tuple) else plain
    assert int(err.item()) == 0
    xw = x.double() * nw.double() if normed else x.double()
    r = (x.double().pow(2).mean(1, keepdim=True) + 1e-6).rsqrt() if normed else torch.ones((T, 1), dtype=torch.float64, device="cuda")
    want = r * (xw @ w.T)
    # the codes leave amax / 65,024 of a value (a quarter more: the levels' own f32 arithmetic); the f32 sums 2^-23 of what they add, a dozen steps
    amax = xw.abs().view(T, cols // 256, 256).amax(2, keepdim=True).expand(-1, -1, 256).reshape(T, cols)
    bound = r * (1.25 * (amax / 65024) @ w.abs().T + 12 * 2.0 ** -23 * (xw.abs() @ w.abs().T))
    assert ((plain.double() - want).abs() <= bound).all()
    assert ((out.double() - (want + old.double())).abs() <= bound + 2.0 ** -23 * (want.abs() + old.abs().double())).all()
    if T > 1:   # a row's bits are its own
        alone = F.dense(tiles, rows, cols, x[T - 1:].contiguous(), norm_w=nw, err=err)
        assert torch.equal((alone[0] if isinstance(alone, tuple) else alone)[-1], plain[-1])
