"""The 3D update of cells with a pending recentring shift, which takes the
per-voxel form of an item, against the unshifted update, which takes the form
that tests rows of four: the same values at the moved places, bit for bit, and a
DESTINATION_CLIP for each supported value that leaves the brick."""
import numpy as np
import pytest

import pfb200
from helpers3d import DeviceState3D, small_centres, small_params

pytestmark = pytest.mark.gpu

CLIP = pfb200.FLAG3D_NAMES.index("destination_clip")
GEOMS = ["periodic", "slab", "channel"]
EPS = np.float32(1.0e-5)


def update(s, shift):
    """phi_out and S_out of one update of every cell with this shift pending."""
    cells = s.get_cells()
    cells["flags"] = 0
    cells["pending_shift_x"], cells["pending_shift_y"], cells["pending_shift_z"] = shift
    s.cells.copy_(s.torch.from_numpy(cells.view(np.uint8).copy()).to(s.cells.device))
    s.flags.zero_()
    s.S[1 - s.cur].zero_()
    s.phi[1 - s.cur].fill_(7.0)
    s.update(s.update_args())
    s.torch.cuda.synchronize()
    return s.get_phi(1 - s.cur), s.get_S(1 - s.cur)


def moved(phi, shift):
    """(phi at the destination of each source voxel, the values left outside)."""
    out, lost = np.zeros_like(phi), phi.copy()
    B = phi.shape[1]
    dst, src = [slice(None)], [slice(None)]
    for s in shift[::-1]:
        dst.append(slice(max(0, -s), B - max(0, s)))
        src.append(slice(max(0, s), B - max(0, -s)))
    out[tuple(dst)] = phi[tuple(src)]
    lost[tuple(src)] = 0.0
    return out, lost


@pytest.mark.parametrize("geometry", GEOMS)
@pytest.mark.parametrize("shift", [(1, 0, 0), (0, -1, 0), (0, 0, 2), (4, 0, 0), (-3, 2, -1), (-4, 4, 4)])
def test_shifted_update_moves_the_unshifted_one(geometry, shift):
    p = small_params(geometry, N=5)
    s = DeviceState3D(p, small_centres(p), "pfb")
    phi0, S0 = update(s, (0, 0, 0))
    assert not s.get_flags().any()
    phi1, S1 = update(s, shift)
    assert not s.get_flags().any()
    want, lost = moved(phi0, shift)
    assert np.max(np.abs(lost)) <= EPS
    assert phi1.tobytes() == want.tobytes()
    np.testing.assert_array_equal(S1, S0)  # what leaves the brick is below half a quantum


@pytest.mark.parametrize("geometry", GEOMS)
@pytest.mark.parametrize("shift", [(2, 0, 0), (-1, 3, 0), (0, -4, 1)])
def test_clip_decides_on_the_value_the_update_gives(geometry, shift):
    """Values spread over a few units in the last place around the support
    threshold: DESTINATION_CLIP counts those of the unshifted update above it."""
    p = small_params(geometry, N=5)
    s = DeviceState3D(p, small_centres(p), "pfb")
    rng = np.random.default_rng(11)
    shape = s.get_phi().shape
    level = np.full(shape[:2], EPS, np.float32)  # of each plane
    S = s.S[s.cur]
    S.zero_()

    def updated(rel):
        f = (level[:, :, None, None] * (1 + rel)).astype(np.float32)
        s.phi[s.cur].copy_(s.torch.from_numpy(f).to(S.device))
        return update(s, (0, 0, 0))[0]

    noise = rng.uniform(-1.0, 1.0, shape)
    for _ in range(5):  # the update's mean effect on each plane taken out
        mid = np.median(updated(0.0 * noise)[:, :, 8:32, 8:32], axis=(2, 3))
        level = np.where(mid > 0, level * EPS / np.maximum(mid, 1e-9), level).astype(np.float32)
    phi0 = updated(4e-7 * noise)
    _, lost = moved(phi0, shift)
    near = np.abs(np.abs(lost) / EPS - 1.0) < 4e-7
    assert near.sum() > 1000
    want = int((np.abs(lost) > EPS).sum())
    update(s, shift)
    assert int(s.get_flags()[CLIP]) == want


def test_shifted_cells_take_one_form():
    """300 cells (B = 40) all shifted by one row run about 2.0 times as long as
    unshifted; with both forms in the warps along an edge it was 3.6 times."""
    p = small_params("channel", N=300, Nx=200, Ny=200)
    s = DeviceState3D(p, small_centres(p), "pfb")
    torch = s.torch

    def micros(shift):
        update(s, shift)
        u, ts = s.update_args(), []
        for _ in range(9):
            s.S[1 - s.cur].zero_()
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            s.update(u)
            e[1].record()
            e[1].synchronize()
            ts.append(e[0].elapsed_time(e[1]) * 1e3)
        return sorted(ts)[4]

    assert micros((0, 1, 0)) <= 2.7 * micros((0, 0, 0))
