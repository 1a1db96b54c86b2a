"""The weight gradient's persistent kernel where its tile split can go wrong,
against the FP64 oracle on the same bfloat16 inputs: images smaller than one
tile of 96 positions, a batch whose tiles do not divide among the CTAs (a CTA's
range starts and ends inside images), a last tile that is mostly padding, and
rows longer than a tile.

The kernel sums in binary32, the oracle in float64: 1e-5 of the sum of absolute
terms plus 1e-5, as for the other weight-gradient tests.

The tensor core's binary32 accumulator rounds towards zero, so a sum of one sign
falls short by up to 2^-23 of its running value with every addition: half a
chain's length times 2^-23 of the total. A chain is 66 additions (11 tiles) at
most, 3.9e-6; adding up the chains (7 per CTA and 25 in the reduction, to
nearest, 2^-24 each of a running sum) gives up to 1.0e-6. The last test asks
for 5e-6 however many images a CTA walks."""
import ctypes as C

import numpy as np
import pytest

import conv_oracle as co
from pfb200 import check, lib

pytestmark = pytest.mark.gpu

SHAPES = [(1, 2, 2), (1, 2, 46), (3, 2, 47), (150, 5, 18), (1, 3, 300), (31, 16, 17)]


def _bf16(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).to(torch.bfloat16).cuda().contiguous()


@pytest.mark.parametrize("cx,cy", [(16, 32), (32, 32), (32, 16), (16, 16)])
@pytest.mark.parametrize("B,H,W", SHAPES)
def test_tile_edges(cx, cy, B, H, W):
    import torch
    rng = np.random.default_rng(7 * B + H + W + cx)
    xd = _bf16(co.to_padded(rng.standard_normal((B, H, W, cx))))
    yd = _bf16(co.to_padded(rng.standard_normal((B, H, W, cy))))
    x = co.from_padded(xd.float().cpu().numpy().astype(np.float64), H, W)
    y = co.from_padded(yd.float().cpu().numpy().astype(np.float64), H, W)
    nbytes = lib().pfb_conv3x3_wgrad_workspace(B, H, W, cx, cy)
    # one word past a 16-byte boundary: the partial sums then go out by words
    for skip in (0, 1):
        ws = torch.full((nbytes // 4 + 1,), float("nan"), device="cuda")
        dw = torch.full((cy, cx, 3, 3), 3.0, device="cuda")
        db = torch.full((cy,), 3.0, device="cuda")
        check(lib().pfb_conv3x3_wgrad(xd.data_ptr(), yd.data_ptr(), ws.data_ptr() + 4 * skip, nbytes,
                                      dw.data_ptr(), db.data_ptr(), B, H, W, cx, cy, None), "wgrad")
        torch.cuda.synchronize()
        v = C.c_uint()
        check(lib().pfb_conv_status(C.byref(v), 1), "status")
        assert v.value == 0
        rdw, rdb = co.conv3x3_wgrad(x, y)
        sdw, sdb = co.conv3x3_wgrad(np.abs(x), np.abs(y))
        assert np.all(np.abs(dw.cpu().numpy() - rdw) <= 1e-5 * sdw + 1e-5)
        assert np.all(np.abs(db.cpu().numpy() - rdb) <= 1e-5 * sdb + 1e-5)


@pytest.mark.parametrize("cx,cy", [(32, 32), (16, 16)])
@pytest.mark.parametrize("B,H,W", [(256, 64, 64), (1024, 32, 32), (1024, 9, 13)])
def test_error_does_not_grow_with_the_batch(cx, cy, B, H, W):
    """x and dY of one sign in batches of many tiles per CTA (the ring of six
    stages wraps up to twelve times)."""
    import torch
    rng = np.random.default_rng(B + cx)
    xd = _bf16(co.to_padded(np.abs(rng.standard_normal((B, H, W, cx), np.float32))))
    yd = _bf16(co.to_padded(np.abs(rng.standard_normal((B, H, W, cy), np.float32))))
    nbytes = lib().pfb_conv3x3_wgrad_workspace(B, H, W, cx, cy)
    ws = torch.full((nbytes // 4,), float("nan"), device="cuda")
    dw = torch.full((cy, cx, 3, 3), 3.0, device="cuda")
    db = torch.full((cy,), 3.0, device="cuda")
    check(lib().pfb_conv3x3_wgrad(xd.data_ptr(), yd.data_ptr(), ws.data_ptr(), nbytes, dw.data_ptr(),
                                  db.data_ptr(), B, H, W, cx, cy, None), "wgrad")
    torch.cuda.synchronize()
    rdw, rdb = co.conv3x3_wgrad(co.from_padded(xd.float().cpu().numpy(), H, W),
                                co.from_padded(yd.float().cpu().numpy(), H, W))
    assert np.max(np.abs(dw.cpu().numpy() / rdw - 1.0)) <= 5e-6
    assert np.max(np.abs(db.cpu().numpy() / rdb - 1.0)) <= 5e-6
