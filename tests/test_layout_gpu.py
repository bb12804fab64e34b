"""mul_ir <-> ir_mul row conversion: exact against reshapes, at tile edges, with ragged channel counts and shifted buffers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _turn(rows, channels, blocks, to_ir_mul):
    out, start = [], 0
    for count, m in blocks:
        piece = rows[:, start:start + count * m * channels]
        shape = (channels, m) if to_ir_mul else (m, channels)
        out.append(piece.reshape(len(rows), count, *shape).transpose(2, 3).reshape(len(rows), -1))
        start += count * m * channels
    return torch.cat(out, dim=1)


@pytest.mark.parametrize("rows", [1, 2, 11, 1185, 9473])
@pytest.mark.parametrize("channels,blocks", [(64, ((3, 1), (4, 3), (4, 5))), (64, ((1, 1), (1, 3), (1, 5))), (4, ((1, 7), (0, 3), (2, 1))),
                                             (12, ((2, 5), (3, 1), (0, 3))), (6, ((1, 3), (2, 5))), (8, ((1, 9), (2, 2)))])
def test_rows_equal_reshapes(rows, channels, blocks):
    from ictc_o3.operators import convert_layout
    width = channels * sum(c * m for c, m in blocks)
    store = torch.randn(rows * width + 1, device="cuda", generator=torch.Generator("cuda").manual_seed(rows))
    for flat in (store[:-1].reshape(rows, width), store[1:].reshape(rows, width)):       # aligned, and 4 bytes off
        for direction in (True, False):
            got = convert_layout(flat, channels, blocks, direction)
            assert torch.equal(got, _turn(flat, channels, blocks, direction))
