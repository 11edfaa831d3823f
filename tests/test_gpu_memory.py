"""Device memory of a handle: the fields and Krylov vectors of the solver, and
little besides.  A box that fills the GPU is sized by them."""
import pytest

from turbulentbl_gb300 import abi
from turbulentbl_gb300.synth import small_workload, make_state

pytestmark = pytest.mark.gpu
RB, RBP = abi.TBL_FLAG_RB_ORDER, abi.TBL_FLAG_RB_PRECOND


@pytest.mark.parametrize("mixed,flags", [(False, 0), (True, 0), (False, RB), (True, RB | RBP)])
def test_footprint(mixed, flags):
    """256 x 98 x 97 in 8 slabs, 30 vectors.  FP64: p', its right-hand side, u, v,
    w, p, their 3 right-hand sides, 3 explicit terms, the SSOR work field, 3
    fluctuations and 31 vectors; mixed: p', right-hand side and 3 fluctuations in
    FP64, 3 x 3 + 5 fields and 32 vectors in FP32.  Besides, up to 1.6 FP64 fields
    (what the sweeps hand from block to block or from slab to slab, and the allocator's
    2 MB granules) and 8 MB of statistics and partial sums."""
    import torch
    from turbulentbl_gb300.lib import TblGpu
    wl = small_workload(nx=256, nz_span=96, ny_wall=96, kmax=30)
    mesh, rp, _ = make_state(wl, nproc=8)
    rp.flags = flags
    if mixed:
        rp.precision, rp.mixed_kmax = abi.TBL_PREC_MIXED, 30
    torch.zeros(1, device="cuda")
    TblGpu(mesh, rp).close()  # loads the kernels
    before = torch.cuda.mem_get_info()[0]
    g = TblGpu(mesh, rp)
    used = before - torch.cuda.mem_get_info()[0]
    g.close()
    points = (mesh.nx + 14) // 8 * 8 * mesh.ny * mesh.nz
    fields = 5 * 8 + (14 + 32) * 4 if mixed else (16 + 31) * 8
    assert used <= points * (fields + 1.6 * 8) + 8e6, used / points


def test_a_box_that_leaves_no_room_for_the_exchange_still_runs():
    """256 x 98 x 97 in one slab, 3 vectors: the line-scan sweeps' exchange is 31 MB
    there.  With half of that left they are not taken, the handle is created all
    the same, and the step is the other sweeps' (1e-12, as in the parity tests)."""
    import gc

    import numpy as np
    import torch
    from turbulentbl_gb300.lib import TblGpu
    gc.collect()  # no handle of another test is to be freed meanwhile
    wl = small_workload(nx=256, nz_span=96, ny_wall=96, kmax=3)
    mesh, rp, st = make_state(wl, nproc=1)
    rp.flags, counts = abi.TBL_FLAG_REPLAY, [4, 4, 4, 2, 3, 3]

    def run():
        g = TblGpu(mesh, rp)
        g.set_replay(counts)
        g.upload(st)
        n0 = g.launches()
        assert g.step(1, check=False)[0] == abi.TBL_OK
        out, n = g.download(), g.launches() - n0
        g.close()
        return out, n
    torch.zeros(1, device="cuda")
    wide = small_workload(nx=1540, nz_span=4, ny_wall=96, kmax=3)  # loads the other sweeps' kernels
    m2, rp2, st2 = make_state(wide, nproc=1)
    g = TblGpu(m2, rp2)
    g.upload(st2)
    g.step(1, check=False)
    g.close()
    a, na = run()
    free = torch.cuda.mem_get_info()[0]
    g = TblGpu(mesh, rp)
    used = free - torch.cuda.mem_get_info()[0]
    g.close()
    ballast = torch.empty(free - used + 16 * 2 ** 20, dtype=torch.uint8, device="cuda")
    try:
        b, nb = run()
    finally:
        del ballast
        torch.cuda.empty_cache()
    assert nb != na  # other kernels
    for f in ("u", "v", "w", "p"):
        err = np.linalg.norm(b[f] - a[f]) / np.linalg.norm(a[f])
        assert err <= 1e-12, (f, err)
