"""The line-scan sweeps (tbl_line.cu) against the oracle where their split of
a grid changes: one and several warps per line (a partial chunk, a last warp
of one lane), 1, 2, 4 and 8 points per lane, rows that fill the rings' halves
exactly or leave a remainder, slabs of many and of few planes (one and several
planes per CTA, an incomplete last CTA, as many planes as registers allow)."""
import numpy as np
import pytest

from turbulentbl_gb300 import abi
from turbulentbl_gb300.synth import small_workload, make_state
from oracle.bind import OracleRunner

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("precision", [abi.TBL_PREC_FP64, abi.TBL_PREC_MIXED])
@pytest.mark.parametrize("nx,nzs,nyw,P", [(34, 8, 14, 2), (35, 9, 30, 1), (130, 4, 18, 3), (131, 5, 17, 2),
                                          (133, 16, 12, 1), (258, 13, 27, 4), (300, 7, 60, 8),
                                          (390, 8, 110, 1), (40, 12, 110, 2), (520, 9, 13, 2), (1030, 6, 11, 1)])
def test_steps_match_the_oracle(nx, nzs, nyw, P, precision):
    """Tolerances of the FP64 parity tests (1e-12) and of the mixed ones
    (1e-5, 1e-4 for p): the scan changes rounding only."""
    from turbulentbl_gb300.lib import TblGpu
    mixed = precision == abi.TBL_PREC_MIXED
    wl = small_workload(nx=nx, nz_span=nzs, ny_wall=nyw, kmax=20, errtol=1e-10 if mixed else 1e-8)
    mesh, rp, st = make_state(wl, nproc=P)
    o = OracleRunner(mesh, rp)
    o.upload(st)
    rp.precision = precision
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
        assert rel(b[f], a[f]) <= tol, (f, rel(b[f], a[f]))
