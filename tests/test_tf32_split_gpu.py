"""Precision of the three-term TF32 products after the split without conversion instructions: every operand is
represented to 2^-22 or better, over the whole exponent range that products of two operands leave finite, and a NaN or an
infinity in a row stays in that row.  Row counts around the 128-row tiles, single- and multi-chunk weights."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 129, 18945])
@pytest.mark.parametrize("cin,cout", [(64, 64), (64, 704), (192, 64), (704, 64)])
def test_row_products_against_float64(rows, cin, cout):
    from ictc_o3.operators import _tc_matmul
    gen = torch.Generator(device="cuda").manual_seed(rows + cin)
    scale = torch.exp2(torch.randint(-40, 41, (rows, 1), generator=gen, device="cuda").float())
    x = torch.randn(rows, cin, generator=gen, device="cuda") * scale
    w = torch.randn(cout, cin, generator=gen, device="cuda")
    got = _tc_matmul(x, w).double()
    bound = (x.double().abs() @ w.double().abs().t())
    # split: 2 x 2^-22 per product, dropped small x small term: 2^-22, fp32 accumulation of 3 cin / 8 partial sums
    worst = float(((got - x.double() @ w.double().t()).abs() / bound).max())
    assert worst < 3 * 2.0 ** -22 + (3 * cin // 8) * 2.0 ** -24, worst


def test_not_a_number_and_infinity_stay_in_their_rows():
    from ictc_o3.operators import _tc_matmul
    x = torch.ones(300, 64, device="cuda")
    x[7, 3], x[140, 63] = float("nan"), float("inf")
    x[200] = torch.tensor(0x7FFFFFFF, dtype=torch.int32, device="cuda").view(torch.float32)
    y = _tc_matmul(x, torch.full((64, 64), 0.5, device="cuda"))
    bad = torch.zeros(300, dtype=torch.bool, device="cuda")
    bad[[7, 140, 200]] = True
    assert bool((~torch.isfinite(y[bad])).all()) and bool((y[~bad] == 32.0).all())
