"""The wavefront sweeps (tbl_sweep.cu) against the oracle, on lines longer than
the line-scan sweeps take (from 1538 points in FP64, 3074 in mixed precision):
a row lag of a whole chunk (4 span rows) and of one position, two 32-row blocks,
plane groups of a slab as one cluster (40 planes in 3 slabs, the last slab's top
CTA idle) and with progress flags in global memory (40 planes in one slab, ten
plane groups)."""
import numpy as np
import pytest

from turbulentbl_gb300 import abi
from turbulentbl_gb300.synth import small_workload, make_state
from oracle.bind import OracleRunner

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed,nx,nzs,nyw,P", [
    (False, 1538, 4, 14, 2), (False, 1539, 5, 40, 3), (False, 1541, 6, 40, 1), (False, 1600, 36, 12, 1),
    (True, 3074, 4, 14, 2), (True, 3075, 5, 40, 3), (True, 3081, 6, 40, 1), (True, 3074, 36, 12, 1)])
def test_steps_match_the_oracle(mixed, nx, nzs, nyw, P):
    """Tolerances of the FP64 parity tests (1e-12) and of the mixed ones (1e-5,
    1e-4 for p)."""
    from turbulentbl_gb300.lib import TblGpu
    wl = small_workload(nx=nx, nz_span=nzs, ny_wall=nyw, kmax=20, errtol=1e-10 if mixed else 1e-8)
    mesh, rp, st = make_state(wl, nproc=P)
    o = OracleRunner(mesh, rp)
    o.upload(st)
    if mixed:
        rp.precision = abi.TBL_PREC_MIXED
    g = TblGpu(mesh, rp)
    g.upload(st)
    for _ in range(2):
        o.step(1)
        g.step(1)
    if not mixed:
        assert g.last_counts() == o.last_counts()
    a, b = o.download(), g.download()
    g.close()
    for f in ("u", "v", "w", "p"):
        tol = (1e-4 if f == "p" else 1e-5) if mixed else 1e-12
        err = np.linalg.norm(b[f] - a[f]) / np.linalg.norm(a[f])
        assert err <= tol, (f, err)
