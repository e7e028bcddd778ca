"""Products with both operands by tensor copies: the rows a block takes depend on how many there are, a row's bits do not."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("rows,cols", [(2048, 512), (528, 256), (12352, 256)])
def test_a_row_does_not_depend_on_its_tile(F, rows, cols, accumulate):
    g = torch.Generator(device="cuda").manual_seed(rows)
    w = F.iq3s_retile(F.iq3s_quantize(torch.randn(rows * cols, device="cuda", generator=g) * 0.02), rows, cols)
    x, old = torch.randn((5000, cols), device="cuda", generator=g), torch.randn((5000, rows), device="cuda", generator=g)

    def run(n):
        out, err = F.dense_prompt(w, rows, cols, x[:n].contiguous(), out=old[:n].clone(), accumulate=accumulate)
        assert int(err.item()) == 0
        return out
    every = run(5000)
    ref = x.half().double() @ F.iq3s_dequant_tiles(w, rows, cols).half().double().T + (old.double() if accumulate else 0)
    # f16 operands, exact products; the tensor core's f32 sums cut off, some 2^-23 of what they add a step of sixteen columns; weights round twice (scale, value)
    size = x.half().abs().double() @ F.iq3s_dequant_tiles(w, rows, cols).abs().double().T + old.abs().double()
    assert ((every.double() - ref).abs() <= (2.0 ** -10 + cols / 16 * 2.0 ** -23) * size).all()
    for n in (1024, 1025, 1279, 1700, 2047, 3001, 4097):
        assert torch.equal(run(n), every[:n]), n


def test_router_rows_do_not_depend_on_their_tile(F):
    g = torch.Generator(device="cuda").manual_seed(3)
    wr, x = 0.02 * torch.randn((513, 512), device="cuda", generator=g), torch.randn((4000, 512), device="cuda", generator=g)
    every = F.router_rows(wr, x, 10)
    for n in (1024, 1500, 3001, 3999):
        for a, b in zip(F.router_rows(wr, x[:n].contiguous(), 10), every):
            assert torch.equal(a, b[:n]), n
