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
