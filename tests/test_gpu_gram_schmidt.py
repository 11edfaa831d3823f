"""Restart lengths at the edges of the Gram-Schmidt passes (tbl_krylov.cu)
against the oracle: blocks of eight basis vectors in FP64 (a last block of one,
seven, eight vectors, one block and several); in mixed precision groups of up to
eight in the dot pass, back substitution of more than 32 columns, the largest
restart length."""
import numpy as np
import pytest

from turbulentbl_gb300 import abi
from turbulentbl_gb300.synth import small_workload, make_state
from oracle.bind import OracleRunner

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,kmax", [(abi.TBL_PREC_FP64, k) for k in (7, 8, 9, 16, 17, 33)] +
                                           [(abi.TBL_PREC_MIXED, k) for k in (7, 8, 9, 33, 63)])
@pytest.mark.parametrize("nx,nzs,nyw,P", [(34, 8, 14, 2), (133, 16, 12, 1)])
def test_restart_lengths_match_the_oracle(nx, nzs, nyw, P, precision, kmax):
    """FP64: 1e-12, as in the parity tests; a perturbation of the initial state
    by one rounding unit moves the oracle's p by 4e-14 and leaves its iteration
    counts.  Mixed: 1e-5, 1e-4 for p, as in the mixed tests."""
    from turbulentbl_gb300.lib import TblGpu
    mixed = precision == abi.TBL_PREC_MIXED
    wl = small_workload(nx=nx, nz_span=nzs, ny_wall=nyw, kmax=20 if mixed else kmax, errtol=1e-10 if mixed else 1e-8)
    mesh, rp, st = make_state(wl, nproc=P)
    o = OracleRunner(mesh, rp)
    o.upload(st)
    o.step(2)
    rp.precision = precision
    if mixed:
        rp.mixed_kmax = kmax
        rp.mixed_max_outer = 60  # the shortest restarts need more refinements than the default 20
    g = TblGpu(mesh, rp)
    g.upload(st)
    g.step(2)
    if not mixed:
        assert g.last_counts() == o.last_counts()
    a, b = o.download(), g.download()
    g.close()
    for f in ("u", "v", "w", "p"):
        tol = (1e-4 if f == "p" else 1e-5) if mixed else 1e-12
        err = np.linalg.norm(b[f] - a[f]) / np.linalg.norm(a[f])
        assert err <= tol, (f, err)
