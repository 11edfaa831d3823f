"""The line-scan sweeps' own waits (tbl_line.cu) give up within a second or so
when nothing comes: at a shared-memory barrier, for a row of the plane below and
for the carry of the segment before.  The handle reports the time-out from then on;
other handles are not affected."""
import ctypes as C

import pytest

from turbulentbl_gb300 import abi
from turbulentbl_gb300.synth import small_workload, make_state

pytestmark = pytest.mark.gpu


def give_up(g, which):
    """A warp's wait of the handle's sweeps runs out: the error word and the seconds."""
    f = g.lib.tbl_selftest_sweep_wait
    f.argtypes = [C.c_void_p, C.c_int32, C.POINTER(C.c_int32), C.POINTER(C.c_double)]
    f.restype = C.c_int
    obs, secs = C.c_int32(0), C.c_double(0.0)
    st = f(g._h, which, C.byref(obs), C.byref(secs))
    return st, obs.value, secs.value


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("which", [0, 1, 2])
def test_a_wait_of_the_sweeps_gives_up(which, mixed):
    from turbulentbl_gb300.lib import TblGpu
    wl = small_workload(nx=40, nz_span=8, ny_wall=14, kmax=20)
    mesh, rp, st = make_state(wl, nproc=2)
    if mixed:
        rp.precision = abi.TBL_PREC_MIXED
    g = TblGpu(mesh, rp)
    g.upload(st)
    assert g.step(1, check=False)[0] == abi.TBL_OK
    assert give_up(g, 3)[0] == abi.TBL_ERR_BAD_ARG
    status, observed, seconds = give_up(g, which)
    assert status == abi.TBL_OK and observed == abi.TBL_ERR_TIMEOUT
    assert 0.02 < seconds < 5.0
    assert g.step(1, check=False)[0] == abi.TBL_ERR_TIMEOUT
    g.close()
    g = TblGpu(mesh, rp)
    g.upload(st)
    assert g.step(1, check=False)[0] == abi.TBL_OK
    g.close()


def test_a_timeout_is_reported_by_the_backward_window():
    """The adjoint's sweeps run after the window's last step: the error word is
    read with their own residuals."""
    from turbulentbl_gb300.lib import TblGpu
    from turbulentbl_gb300.runner import TblError
    wl = small_workload(nx=24, nz_span=8, ny_wall=14, kmax=20)
    mesh, rp, st = make_state(wl, nproc=2)
    rp.cum = 50
    g = TblGpu(mesh, rp)
    g.upload(st)
    x = mesh.dx * mesh.nx
    g.forward_window(2, 0.25 * x, 0.75 * x, 2)
    g.backward_window()
    assert give_up(g, 1)[:2] == (abi.TBL_OK, abi.TBL_ERR_TIMEOUT)
    with pytest.raises(TblError) as e:
        g.backward_window()
    assert e.value.status == abi.TBL_ERR_TIMEOUT
    g.close()


@pytest.mark.parametrize("mixed", [False, True])
def test_a_timeout_is_not_taken_for_a_nan(mixed):
    from turbulentbl_gb300.lib import TblGpu
    wl = small_workload(nx=24, nz_span=8, ny_wall=14, kmax=20)
    mesh, rp, st = make_state(wl, nproc=2)
    rp.mmax = 20
    if mixed:
        rp.precision = abi.TBL_PREC_MIXED
    st["u"] = st["u"].copy(order="F")
    st["u"][5, 5, 5] = float("nan")
    g = TblGpu(mesh, rp)
    g.upload(st)
    assert g.step(1, check=False)[0] == abi.TBL_ERR_NAN
    assert give_up(g, 1)[:2] == (abi.TBL_OK, abi.TBL_ERR_TIMEOUT)
    g.upload(st)
    assert g.step(1, check=False)[0] == abi.TBL_ERR_TIMEOUT
    g.close()
