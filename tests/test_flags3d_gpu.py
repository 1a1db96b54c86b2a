"""Every sticky flag that the 3D measurement and update raise from the field,
against the CPU oracle on the same planted state: a NaN, an infinity, |phi| > 2,
an aggregate word below the cell's own quanta, one that wraps, contact with the
top of a slab, and a supported value pushed out of the brick, in unshifted and
shifted cells. The kernels test a row of four first and look at single voxels
only where that calls for it; counts must equal the oracle's, which tests every
voxel. Fields agree to 1e-6 (the oracle rounds in another order)."""
import ctypes as C

import numpy as np
import pytest

import oracle3d
import pfb200
from helpers3d import DeviceState3D, small_params

pytestmark = pytest.mark.gpu

N_CELLS, AT = 3, (19, 22)  # voxel (z, y) of the planted value; x varies over a row of four
FLAG = {n: i for i, n in enumerate(pfb200.FLAG3D_NAMES)}
KINDS = ["none", "nan", "inf", "clamp", "negative", "overflow", "clip", "top"]


def planted(geometry, kind, x):
    """A state of three cells, the second of which holds the planted value."""
    p = small_params(geometry, N=N_CELLS, dt=1e-3)
    mid = {"periodic": 40.0, "slab": 20.0, "channel": 12.0}[geometry]
    s = DeviceState3D(p, np.array([[20.0, 20.0, mid], [50.0, 50.0, mid], [50.0, 20.0, mid]]), "pfb")
    cells = s.get_cells()
    if kind == "top":
        # the brick's planes from the cell's middle up lie above the domain
        cells["origin_z"][1] = p.Nz - 1 - 22
    s.cells.copy_(s.torch.from_numpy(cells.view(np.uint8).copy()).to(s.cells.device))
    z, y = AT
    value = {"nan": np.nan, "inf": np.inf, "clamp": 2.3}.get(kind)
    if value is not None:
        s.phi[s.cur][1, z, y, x] = value
    if kind == "clip":
        s.phi[s.cur][1, z, y, 0] = 0.5
    s.S[s.cur].zero_()
    a = pfb200._abi3d.ScatterArgs3D()
    a.phi, a.cells, a.S = s.phi[s.cur].data_ptr(), s.cells.data_ptr(), s.S[s.cur].data_ptr()
    a.global_flags, a.layout, a.N, a.B = s.flags.data_ptr(), s.layout, s.N, s.B
    s._call("scatter_current", a)
    cells["flags"] = 0
    s.cells.copy_(s.torch.from_numpy(cells.view(np.uint8).copy()).to(s.cells.device))
    s.flags.zero_()
    word = (int(cells["origin_z"][1]) + z) % p.Nz, (int(cells["origin_y"][1]) + y) % p.Ny, \
        (int(cells["origin_x"][1]) + x) % p.Nx
    out = s.torch.zeros_like(s.S[0])
    if kind == "negative":
        s.S[s.cur][word] = 1
    if kind == "overflow":
        out[word] = -16  # 2^32 - 16: the cell's quanta wrap it
    s.torch.cuda.synchronize()
    return p, s, out


def host(s):
    wall = None if s.wall is None else s.wall.cpu().numpy()
    return s.get_cells(), s.get_phi(), s.get_S(), np.zeros(10, np.uint32), wall


def ptr(a):
    return None if a is None else a.ctypes.data


@pytest.mark.parametrize("geometry", ["periodic", "slab", "channel"])
@pytest.mark.parametrize("kind", [k for k in KINDS if k not in ("overflow", "clip")])
@pytest.mark.parametrize("x", [20, 23])
def test_measurement(geometry, kind, x):
    if kind == "top" and geometry != "slab":
        pytest.skip("only a slab has a top")
    p, s, _ = planted(geometry, kind, x)
    cells, phi, S, flags, wall = host(s)
    s._call("measure_cells_only", s.measure_args(tumble=False, surface=True))
    got = s.get_cells()
    oracle3d.olib().oracle3d_measure(0, ptr(phi), ptr(S), ptr(cells), ptr(flags), 0, C.byref(s.layout),
                                     s.N, s.B, ptr(wall), p.dt, p.lambda_, p.kappa, p.xi, p.tau, 1, 0,
                                     0, 1, 0)
    np.testing.assert_array_equal(s.get_flags(), flags)
    for f in ("flags", "phi_max", "bb_lo_x", "bb_hi_x", "bb_lo_y", "bb_hi_y", "bb_lo_z", "bb_hi_z"):
        np.testing.assert_array_equal(got[f], cells[f], err_msg=f)
    np.testing.assert_allclose(got["V"], cells["V"], rtol=1e-12)
    want = {"nan": "nonfinite", "inf": "nonfinite", "negative": "S_negative",
            "top": "slab_top_contact"}.get(kind)
    assert want is None or flags[FLAG[want]] > 0


@pytest.mark.parametrize("geometry", ["periodic", "slab", "channel"])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("x,shift", [(20, (0, 0, 0)), (23, (0, 0, 0)), (21, (0, 0, -1)), (22, (1, -2, 1)),
                                     (23, (4, 0, 0))])
def test_update(geometry, kind, x, shift):
    if kind == "top" and geometry != "slab":
        pytest.skip("only a slab has a top")
    if kind == "clip" and shift[0] <= 0:
        pytest.skip("nothing leaves through the planted face")
    p, s, S_out = planted(geometry, kind, x)
    cells = s.get_cells()
    cells["pending_shift_x"], cells["pending_shift_y"], cells["pending_shift_z"] = shift
    s.cells.copy_(s.torch.from_numpy(cells.view(np.uint8).copy()).to(s.cells.device))
    cells, phi, S, flags, wall = host(s)
    S1 = S_out.cpu().numpy().view(np.uint32).copy()
    s.S[1 - s.cur].copy_(S_out)
    u = s.update_args()
    s.update(u)
    phi1 = np.zeros_like(phi)
    oracle3d.olib().oracle3d_update(ptr(phi), ptr(phi1), ptr(S), ptr(S1), ptr(cells), ptr(flags),
                                    C.byref(s.layout), s.N, s.B, ptr(wall), u.dt, u.V0, u.volume_scale,
                                    u.bulk_scale, u.interaction_coeff, 0)
    np.testing.assert_array_equal(s.get_flags(), flags)
    np.testing.assert_array_equal(s.get_cells()["flags"], cells["flags"])
    assert np.max(np.abs(s.get_phi(1 - s.cur) - phi1)) <= 1e-6
    d = (s.get_S(1 - s.cur) - S1).view(np.int32)  # q = phi^2 2^27: 2 |phi| 1e-6 2^27 and rounding
    assert np.max(np.abs(d)) <= 2 * 2.3 * 1e-6 * 2 ** 27 + N_CELLS
    want = {"nan": "nonfinite", "inf": "nonfinite", "clamp": "q_clamp", "negative": "S_negative",
            "overflow": "S_overflow", "clip": "destination_clip", "top": "slab_top_contact"}.get(kind)
    assert (flags[FLAG[want]] > 0) if want else not flags.any()
