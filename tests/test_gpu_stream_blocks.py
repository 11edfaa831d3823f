"""Streamwise and span SSOR blocks on lines of several warps (tbl_line.cu) and on
lines that the wavefront sweeps take (tbl_sweep.cu) against a NumPy model of the
block preconditioner: in the line-scan sweeps the carry from warp to warp and the
scan over the lanes are cut inside a warp's segment, at every number of points
per lane.

The model is the NumPy oracle with its sweeps along a line as first-order
filters, the preconditioner's lines cut into up to four blocks of whole chunks (4
points in FP64, 8 in mixed precision) and its rows into blocks of 32 in sweep
order.  A cycle of three vectors is stopped short of convergence, where p' still
is what the preconditioner made it: blocks a chunk off, or not cut at all, move
it by 1% and more."""
import numpy as np
import pytest
from scipy.signal import lfilter

from turbulentbl_gb300 import abi
from turbulentbl_gb300.synth import small_workload, make_state
from oracle.np_oracle import NpOracle

pytestmark = pytest.mark.gpu
KIT = 3


class BlockModel(NpOracle):
    block = None  # points per streamwise block, counted from i = 0
    rows = None   # rows per span block, counted in sweep order

    def gs(self, target=None):
        t, nx, ny = -self.rp.dt / self.rp.re, self.nx, self.ny
        i = slice(1, nx - 1)
        e, w = slice(2, nx), slice(0, nx - 2)
        sweeps = []
        for c in range(3):
            F, Q = self.U[c], self.Q[c]
            for n in range(target[c]):
                old = F.copy()
                for r, (bn, en) in enumerate(self.slabs):
                    for k in range(bn, en + 1):
                        d = 1.0 + t * self.Ap[k]
                        lo = old if k == bn and r > 0 else F
                        hi = old if k == en and r < len(self.slabs) - 1 else F
                        for j in range(1, ny - 1):
                            q = (Q[i, j, k] - t * self.Aw * F[e, j, k] - t * self.As * (F[i, self.jp1[j], k]
                                 + F[i, self.jm1[j], k]) - t * self.At[k] * hi[i, j, k + 1]
                                 - t * self.Ab[k] * lo[i, j, k - 1]) / d
                            ci = -t * self.Aw / d
                            F[i, j, k] = lfilter([1.0], [1.0, -ci], q, zi=[ci * F[0, j, k]])[0]
            sweeps.append(target[c])
        return sweeps

    def _line(self, f, ci, d):
        out = np.empty_like(f)  # f: points 1 .. nx-2; d: 1 forward, -1 backward
        cuts = [0] + [q - 1 for q in range(self.block, self.nx - 1, self.block)] + [len(f)]
        for a, b in zip(cuts[:-1], cuts[1:]):
            out[a:b] = lfilter([1.0], [1.0, -ci], f[a:b][::d])[::d]
        return out

    def ssor(self, R):
        om, nx, ny = self.rp.omega, self.nx, self.ny
        i = slice(1, nx - 1)
        out = np.zeros_like(R)
        for bn, en in self.slabs:
            x = np.zeros((nx, ny, en - bn + 3))
            for k in range(bn, en + 1):
                s, kl = -om / self.Ap[k], k - bn + 1
                for j in range(1, ny - 1):
                    before = x[i, j - 1, kl] * ((j - 1) % self.rows != 0)
                    f = s * (R[i, j, k] + self.As * before + self.Ab[k] * x[i, j, kl - 1])
                    x[i, j, kl] = self._line(f, s * self.Aw, 1)
            for k in range(bn, en + 1):
                x[i, 1:ny - 1, k - bn + 1] *= ((2 - om) / om) * self.Ap[k]
            for k in range(en, bn - 1, -1):
                s, kl = -om / self.Ap[k], k - bn + 1
                for j in range(ny - 2, 0, -1):
                    before = x[i, j + 1, kl] * ((ny - 2 - j) % self.rows != 0)
                    f = s * (x[i, j, kl] + self.As * before + self.At[k] * x[i, j, kl + 1])
                    x[i, j, kl] = self._line(f, s * self.Aw, -1)
            out[i, 1:ny - 1, bn:en + 1] = x[i, 1:ny - 1, 1:en - bn + 2]
        return out


def _case(nx, span, mixed, stream):
    wl = small_workload(nx=nx, nz_span=span, ny_wall=14, kmax=KIT, errtol=1e-10)
    mesh, rp, st = make_state(wl, nproc=2)
    chunk = 8 if mixed else 4
    n = (nx - 2) // chunk + 1
    nib = min(4, n) if stream else 1
    return mesh, rp, st, chunk * ((n + nib - 1) // nib)


SPAN, STREAM = abi.TBL_FLAG_SSOR_SPAN_BLOCKS, abi.TBL_FLAG_SSOR_STREAM_BLOCKS


@pytest.mark.parametrize("mixed,nx,span,flags", [
    (False, 134, 6, STREAM), (False, 203, 6, STREAM), (False, 203, 40, SPAN), (False, 802, 6, STREAM),
    (True, 264, 6, STREAM), (True, 602, 6, STREAM), (True, 602, 40, SPAN | STREAM),
    (False, 1540, 6, STREAM), (False, 1538, 40, SPAN | STREAM), (True, 3076, 6, STREAM), (True, 3074, 40, SPAN)])
def test_cut_lines_match_the_model(mixed, nx, span, flags):
    """p' after three vectors, interior, relative to its norm.  One rounding unit
    of the state (1e-16) moves the model's by 5e-14, an FP32 one (6e-8) by 2e-5:
    1e-10 in FP64, 2e-3 in mixed precision."""
    from turbulentbl_gb300.lib import TblGpu
    mesh, rp, st, block = _case(nx, span, mixed, bool(flags & STREAM))
    rp.flags = flags
    if mixed:
        rp.precision = abi.TBL_PREC_MIXED
        rp.mixed_kmax, rp.mixed_max_outer, rp.mixed_inner_tol = KIT, 1, 1e-30
        g = TblGpu(mesh, rp)
        g.upload(st)
        status, rec = g.step(1, check=False)
        assert status == abi.TBL_ERR_NOT_CONVERGED
        assert rec[0]["gmres_iters"] == KIT
        counts = list(rec[0]["gs_sweeps"]) + [1, KIT]
    else:
        counts = [20, 20, 20, 1, KIT]
        rp.flags |= abi.TBL_FLAG_REPLAY
        g = TblGpu(mesh, rp)
        g.set_replay(counts)
        g.upload(st)
        g.step(1, check=False)
    b = g.download(fields=("pcorr",))["pcorr"]
    g.close()
    m = BlockModel(mesh, rp)
    m.block = block
    m.rows = 32 if flags & SPAN else mesh.ny
    m.upload(st)
    m.step(counts)
    inner = (slice(1, -1),) * 3
    err = np.linalg.norm(b[inner] - m.PC[inner]) / np.linalg.norm(m.PC[inner])
    assert err <= (2e-3 if mixed else 1e-10), err
