"""What a split-precision member allocates (mcv_footprint_bytes; host only): the
state twice, the increments twice, RK4's sums, phi_s in both widths, the raw
boundary in both widths, and one 96-byte record of linear references for each
8x8-cell tile of the persistent tile forms, which alone keep them; up to the
256-byte alignment of the arrays."""
import pytest

from mcv_sw_b200 import api


@pytest.mark.parametrize("order", [3, 4])
@pytest.mark.parametrize("nc", [2, 9, 48, 256, 1024])
@pytest.mark.parametrize("scheme,sums", [(3, 0), (4, 3)])
def test_split_precision_member(order, nc, scheme, sums):
    H = order - 1
    n = nc * H + 1
    npx = n + 2 * H
    points = 6 * npx * ((npx + 15) // 16 * 16)
    tiles = ((nc + 7) // 8) ** 2
    member = points * (7 * 8 + (7 + sums) * 4) + 24 * n * (16 + 32) + 96 * 6 * tiles + 16
    footprint = [api.lib().mcv_footprint_bytes(order, nc, scheme, 1, m) for m in (1, 5)]
    assert abs(footprint[1] - footprint[0] - 4 * member) <= 32 * 256
