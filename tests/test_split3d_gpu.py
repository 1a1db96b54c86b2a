"""The 3D step cut into more parts for systems of few cells: every split gives
the same bits. A measurement (clusters of 4 or 8) and an update (4 parts, or
as many as fill the SMs) of a selection of a system's cells equal those of the
whole system for the same cells, also for bricks of which an SM holds one, for
shifted cells and for 16-bit pools (whose in-place modes update a few cells at a
time)."""
import numpy as np
import pytest

import pfb200
from helpers3d import DeviceState3D, small_centres, small_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geometry", ["periodic", "slab", "channel"])
@pytest.mark.parametrize("count", [1, 37, 38, 50, 73])
def test_split_does_not_change_the_bits(geometry, count):
    N = 80
    p = small_params(geometry, N=N, Nx=160, Ny=160, **({"Nz": 160} if geometry == "periodic" else {}))
    a = DeviceState3D(p, small_centres(p), "pfb")
    b = DeviceState3D(p, small_centres(p), "pfb")
    a.step_once()
    b.clone_from(a)
    ids = np.random.default_rng(count).permutation(N)[:count].astype(np.int32)
    sel = b.torch.from_numpy(ids).to(b.cells.device)
    for s, chosen in ((a, None), (b, sel)):
        m, u = s.measure_args(tumble=True, surface=True), s.update_args()
        if chosen is not None:
            for args in (m, u):
                args.selection.ids, args.selection.count = chosen.data_ptr(), count
        s.S[1 - s.cur].zero_()
        s._call("measure_cells_only", m)
        s._call("apply_cell_motion", m)
        s.update(u)
        s.torch.cuda.synchronize()
    ca, cb = a.get_cells()[ids], b.get_cells()[ids]
    for f in ca.dtype.names:
        np.testing.assert_array_equal(ca[f], cb[f], err_msg=f)
    assert a.get_phi(1 - a.cur)[ids].tobytes() == b.get_phi(1 - b.cur)[ids].tobytes()
    assert int(a.get_flags().sum()) == int(b.get_flags().sum()) == 0


@pytest.mark.parametrize("geometry", ["periodic", "slab", "channel"])
def test_split_of_wide_bricks_and_shifted_cells(geometry):
    N, count = 74, 9
    p = small_params(geometry, N=N, B=80, Nx=160, Ny=160,
                     **({"Nz": 160} if geometry == "periodic" else {"Nz": 112} if geometry == "slab" else {}))
    a = DeviceState3D(p, small_centres(p), "pfb")
    b = DeviceState3D(p, small_centres(p), "pfb")
    a.step_once()
    b.clone_from(a)
    rng = np.random.default_rng(1)
    ids = rng.permutation(N)[:count].astype(np.int32)
    shift = rng.integers(-4, 5, (N, 3))
    sel = b.torch.from_numpy(ids).to(b.cells.device)
    for s, chosen in ((a, None), (b, sel)):
        m, u = s.measure_args(tumble=True, surface=True), s.update_args()
        if chosen is not None:
            for args in (m, u):
                args.selection.ids, args.selection.count = chosen.data_ptr(), count
        s.S[1 - s.cur].zero_()
        s._call("measure_cells_only", m)
        cells = s.get_cells()
        for k, f in enumerate(("pending_shift_x", "pending_shift_y", "pending_shift_z")):
            cells[f] = shift[:, k]
        s.cells.copy_(s.torch.from_numpy(cells.view(np.uint8).copy()).to(s.cells.device))
        s.update(u)
        s.torch.cuda.synchronize()
    ca, cb = a.get_cells()[ids], b.get_cells()[ids]
    for f in ca.dtype.names:
        np.testing.assert_array_equal(ca[f], cb[f], err_msg=f)
    assert a.get_phi(1 - a.cur)[ids].tobytes() == b.get_phi(1 - b.cur)[ids].tobytes()
    assert int(a.get_flags().sum()) == int(b.get_flags().sum()) == 0


@pytest.mark.parametrize("storage", [1, 2])
def test_split_of_16_bit_pools(storage):
    p = small_params("periodic", N=80, Nx=160, Ny=160, Nz=160, phi_storage=storage)
    c = small_centres(p)
    out = []
    for mode, slots in (("throughput", 0), ("balanced", 2)):
        s = pfb200.Sim3D(p, c, memory_mode=mode, scratch_slots=slots)
        s.advance(12)
        out.append((s.cells().tobytes(), s.phi().tobytes(), s.S().tobytes()))
        assert not s.flags().any()
        s.close()
    assert out[0] == out[1]
