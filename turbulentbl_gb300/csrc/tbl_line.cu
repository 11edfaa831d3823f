// tbl_line.cu -- line-scan sweeps: lexicographic Gauss-Seidel and the
// forward/backward block-SSOR preconditioner, one whole line (j, k) at a time.
//
// A sweep is the triangular solve
//   x(i,j,k) = f(i,j,k) + ci x(i-1,j,k) + cj x(i,j-1,k) + ck x(i,j,k-1)
// with coefficients constant on a plane.  Along a line it is a first-order
// linear recurrence, so the line is solved by a scan over the lanes of a few
// warps instead of point after point: the dependency chain of a slab of K
// planes and J rows is J + K line steps, where the point-by-point wavefront
// (tbl_sweep.cu) needs nx/4 + K + 9 J/32 steps of at least twice the length.
// The scan is exact in exact arithmetic; it only changes the rounding.
//
//   * a warp owns 32 E consecutive points of every line of one plane, E per
//     lane; S warps span a line; the row above stays in registers;
//   * within a lane: a chain of E - 1 FMAs; across the lanes: Kogge-Stone on
//     y(l) = b(l) + ci^E y(l-1); levels whose factor |ci|^(E 2^l) is below
//     2^-60 (2^-32 in FP32), 1/100 of a rounding unit, add nothing and are
//     left out (typically 2 of the 5 remain in FP32 and 3 in FP64);
//   * the carry into a warp's segment comes from the warp before it through a
//     mailbox in shared memory, one slot per row, whose value is its own flag
//     (slots start as a NaN pattern that no result has), and is added after
//     the scan, so that the chain between the warps of a line is one FMA;
//   * the plane below is handed over row by row with st.async into a ring in
//     the consumer's shared memory (its own CTA or the next CTA of the
//     cluster), ordered by the ring slots' mbarriers;
//   * slabs of more planes than a cluster holds continue in the next cluster
//     through a global exchange buffer whose words are their own flags.
//
// All waits are bounded; a wait that gives up sets the error word, and every
// warp stays until the cluster's closing barrier, so no CTA leaves while
// another may still reach its shared memory.
#include <algorithm>

#include "tbl_internal.cuh"
#include "tbl_kernels.cuh"
#include "tbl_sync.cuh"

namespace tbl {

constexpr int LINE_XR = 4;            // ring slots (rows) per warp
constexpr int LINE_MAX_WARPS = 16;    // warps of a CTA at most
constexpr int LINE_MAX_SLOTS = 8192;  // carry mailbox slots of a CTA at most (64 KB in FP64)
constexpr int LINE_MAX_SMEM = 160 * 1024;  // above the largest CTA: 64 KB of rings, 64 KB of mailboxes, barriers

template <typename V>
struct LineArgs {
    Geom g;
    const SlabDesc* slabs;
    int* err;
    const int* skip;
    int S, KP;         // warps per line, planes per CTA
    int nc, ngrp;      // CTAs per cluster, clusters per slab column
    int nblk, rows;    // span blocks per slab, rows of a block (the last may have fewer)
    int cb;            // SSOR streamwise blocks: chunks per block (0 = one block)
    const double *Ab, *At, *rAp;
    double aw, as, omega;
    const V* gsc;      // GS: [p0|p1|p2|p3] x nz of the handle's coefficient table
    const V* gsb;      // GS: nz coefficients of U(k-1)
    V* out[3];         // GS: fields; SSOR: out[0]
    const V* in[3];    // GS: precomputed old-value terms; SSOR: in[0]
    int comp[3];
    V* halo_out;       // GS: [comp][side][slab] planes of the next sweep's halo
    int P;
    V* xch;            // [set][slab][block][cluster boundary][row][32 E S]
};

template <typename V> struct LineBits;
template <> struct LineBits<double> {
    using U = unsigned long long;
    static __device__ __forceinline__ U of(double v) { return (U)__double_as_longlong(v); }
    static __device__ __forceinline__ double from(U b) { return __longlong_as_double((long long)b); }
    static constexpr double tiny = 8.7e-19;  // 2^-60
};
template <> struct LineBits<float> {
    using U = unsigned;
    static __device__ __forceinline__ U of(float v) { return __float_as_uint(v); }
    static __device__ __forceinline__ float from(U b) { return __uint_as_float(b); }
    static constexpr float tiny = 2.3e-10f;  // 2^-32
};
// "not written yet": all bits set, a NaN that a result is never stored as
template <typename V>
__device__ __forceinline__ V line_flagged(V v) {
    using B = LineBits<V>;
    return B::of(v) == ~(typename B::U)0 ? B::from((~(typename B::U)0) >> 1) : v;
}

template <typename V, int E>
__device__ __forceinline__ void line_load(V (&v)[E], const V* p, bool rev) {
    constexpr int W = 16 / sizeof(V);
    V t[E];
#pragma unroll
    for (int b = 0; b < E / W; ++b) {
        const int4 q = __ldcg(reinterpret_cast<const int4*>(p) + b);
        *reinterpret_cast<int4*>(&t[b * W]) = q;
    }
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = rev ? t[E - 1 - e] : t[e];
}
template <typename V, int E>
__device__ __forceinline__ void line_store(V* p, const V (&v)[E], bool rev) {
    constexpr int W = 16 / sizeof(V);
    V t[E];
#pragma unroll
    for (int e = 0; e < E; ++e) t[e] = rev ? v[E - 1 - e] : v[e];
#pragma unroll
    for (int b = 0; b < E / W; ++b)
        *(reinterpret_cast<int4*>(p) + b) = *reinterpret_cast<const int4*>(&t[b * W]);
}

template <int MODE, typename V, int E, int D>
__global__ void __launch_bounds__(32 * LINE_MAX_WARPS) k_line(const LineArgs<V> a) {
    if (a.skip && *a.skip) return;  // every CTA reads the same word, written by an earlier launch
    using B = LineBits<V>;
    constexpr bool GS = MODE == 0, BWD = MODE == 2;
    constexpr unsigned XBYTES = 32 * E * sizeof(V);
    const Geom& g = a.g;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int S = a.S, KP = a.KP, NW = S * KP;
    const int seg = wid % S, kp = wid / S;
    const int set = blockIdx.y;
    // grid.x: [slab][span block][cluster of the column][CTA of the cluster]
    const int rank = blockIdx.x % a.nc, grp = (blockIdx.x / a.nc) % a.ngrp;
    const int blk = (blockIdx.x / (a.nc * a.ngrp)) % a.nblk, slab = blockIdx.x / (a.nc * a.ngrp * a.nblk);
    const SlabDesc sl = a.slabs[slab];
    const int J = g.ny - 2, K = sl.K;
    const int comp = GS ? a.comp[set] : 0;
    const int j0 = blk * a.rows, nrow = min(a.rows, J - j0);  // logical rows [j0, j0 + nrow)
    const int kl = (grp * a.nc + rank) * KP + kp;             // logical plane
    const bool live = kl < K;
    const int kidx = BWD ? K - 1 - kl : kl;
    const int k = sl.bn + (live ? kidx : 0);

    // shared memory: rings of the warps | ring barriers (full, empty) | carry mailboxes
    extern __shared__ __align__(16) unsigned char s_dyn[];
    V* const ring = reinterpret_cast<V*>(s_dyn) + (size_t)wid * LINE_XR * 32 * E;
    unsigned long long* const bars = reinterpret_cast<unsigned long long*>(s_dyn + (size_t)NW * LINE_XR * XBYTES);
    unsigned long long* const full = bars + wid * 2 * LINE_XR;
    unsigned long long* const empty = full + LINE_XR;
    V* const mail = reinterpret_cast<V*>(bars + NW * 2 * LINE_XR);  // [warp][row]
    for (int q = threadIdx.x; q < NW * a.rows; q += blockDim.x)
        reinterpret_cast<typename B::U*>(mail)[q] = ~(typename B::U)0;
    if (lane == 0) {
        for (int q = 0; q < LINE_XR; ++q) {
            mbar_init(&full[q], 1);
            mbar_init(&empty[q], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int q = 0; q < LINE_XR; ++q) mbar_arrive_expect_tx(&full[q], XBYTES);
    }
    __syncthreads();
    cluster_sync_all();  // barriers initialised and armed in every CTA of the cluster

    if (live) {
        const bool first = kl == 0;
        const bool last_of_grp = rank == a.nc - 1 && kp == KP - 1;
        const bool from_ring = !first && !(rank == 0 && kp == 0);
        const bool from_xch = !first && !from_ring;
        const bool has_up = kl + 1 < K;
        const bool to_ring = has_up && !last_of_grp, to_xch = has_up && last_of_grp;
        const unsigned up_rank = kp < KP - 1 ? rank : rank + 1, dn_rank = kp > 0 ? rank : rank - 1;
        const int up_wid = kp < KP - 1 ? wid + S : seg, dn_wid = kp > 0 ? wid - S : (KP - 1) * S + seg;
        // shared-memory addresses in the neighbours' CTAs (the layout is the same in all)
        V* const up_ring = reinterpret_cast<V*>(s_dyn) + (size_t)up_wid * LINE_XR * 32 * E;
        const unsigned up_data = mapa_rank(smem_u32(up_ring + lane * E), to_ring ? up_rank : rank);
        const unsigned up_full = mapa_rank(smem_u32(bars + up_wid * 2 * LINE_XR), to_ring ? up_rank : rank);
        const unsigned dn_empty =
            mapa_rank(smem_u32(bars + dn_wid * 2 * LINE_XR + LINE_XR), from_ring ? dn_rank : rank);
        const size_t xrow = (size_t)32 * E * S;
        const size_t xbase = (((size_t)set * a.P + slab) * a.nblk + blk) * (a.ngrp > 1 ? a.ngrp - 1 : 0);
        V* const xin = from_xch ? a.xch + (xbase + grp - 1) * a.rows * xrow + (size_t)(seg * 32 + lane) * E : nullptr;
        V* const xout = to_xch ? a.xch + (xbase + grp) * a.rows * xrow + (size_t)(seg * 32 + lane) * E : nullptr;

        // this lane's points: chunk ch of the line in sweep order, i = i0 .. i0 + E - 1
        const int C = (g.nx - 2) / E + 1;
        const int ch = seg * 32 + lane;
        const bool on = ch < C;
        const int pc = BWD ? C - 1 - ch : ch;
        const int i0 = on ? E * pc : 0;
        bool ok[E];
        bool all_ok = true;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int i = i0 + (BWD ? E - 1 - e : e);
            ok[e] = on && i >= 1 && i <= g.nx - 2;
            all_ok = all_ok && ok[e];
        }
        const bool edge = __any_sync(0xffffffffu, !all_ok);  // the warp holds a line end
        // chunks before this one in its streamwise block
        int dist = ch;
        if (!GS && a.cb > 0) dist = BWD ? min(C, (pc / a.cb + 1) * a.cb) - 1 - pc : pc % a.cb;

        V ci, cj, ck;
        if (GS) {
            ci = a.gsc[g.nz + k];
            cj = a.gsc[2 * g.nz + k];
            ck = a.gsb[k];
        } else {
            const double wr = -a.omega * a.rAp[k];
            ci = (V)(wr * a.aw);
            cj = (V)(wr * a.as);
            ck = (V)(wr * (BWD ? a.At[k] : a.Ab[k]));
        }
        V cpw[E];  // ci^(e+1)
        cpw[0] = ci;
#pragma unroll
        for (int e = 1; e < E; ++e) cpw[e] = cpw[e - 1] * ci;
        V pw = cpw[E - 1];        // ci^(E 2^l)
        V lev[5], acar = V(1);    // scan factors of this lane; factor of the segment's carry-in, ci^(E (lane+1))
        int nlev = 0;
#pragma unroll
        for (int l = 0; l < 5; ++l) {
            const int d = 1 << l;
            lev[l] = (lane >= d && dist >= d) ? pw : V(0);
            if (abs(pw) >= B::tiny) nlev = l + 1;
            if ((lane + 1) & d) acar *= pw;
            pw = pw * pw;
        }
        if (lane == 31) acar = pw;
        if (dist <= lane) acar = V(0);  // the block starts inside the segment (always so in segment 0)
        const bool starts = dist == 0;

        // line pointers; logical row r of the block
        const int jfirst = BWD ? J - 1 - j0 : j0;
        const long long rstep = BWD ? -(long long)g.sx : (long long)g.sx;
        const long long base = (long long)g.sx * ((long long)(1 + jfirst) + (long long)g.ny * k) + i0;
        const V* inp = a.in[comp] + base;
        V* outp = a.out[comp] + base;
        V* hout = nullptr;
        if (GS) {
            const size_t hb = (size_t)comp * 2 * a.P;
            const long long hl = (long long)g.sx * (1 + jfirst) + i0;
            if (kidx == 0 && slab > 0) hout = a.halo_out + (hb + a.P + (slab - 1)) * (size_t)g.ps + hl;
            if (kidx == K - 1 && slab < a.P - 1) hout = a.halo_out + (hb + (slab + 1)) * (size_t)g.ps + hl;
        }
        V* const my_mail = mail + (size_t)wid * a.rows;
        const V* const prev_mail = mail + (size_t)(wid - 1) * a.rows;

        V pf[D][E], xj[E], x0[GS ? E : 1];
#pragma unroll
        for (int u = 0; u < D; ++u) {
#pragma unroll
            for (int e = 0; e < E; ++e) pf[u][e] = V(0);
            if (on && u < nrow) line_load<V, E>(pf[u], inp + u * rstep, BWD);
        }
#pragma unroll
        for (int e = 0; e < E; ++e) xj[e] = V(0);
        bool dead = false;

        auto row = [&](const int r, V(&in)[E]) {
            V f[E];
#pragma unroll
            for (int e = 0; e < E; ++e) f[e] = fma(cj, xj[e], in[e]);
            if (on && r + D < nrow) line_load<V, E>(in, inp + (r + D) * rstep, BWD);
            if (GS && r == nrow - 1) {  // periodic: the last row reads the first row's new values
#pragma unroll
                for (int e = 0; e < E; ++e) f[e] = fma(cj, x0[GS ? e : 0], f[e]);
            }
            // ---- the plane below
            if (from_ring) {
                const int s = r % LINE_XR;
                if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (unsigned)(r / LINE_XR) & 1u))) { dead = true; return; }
                V xk[E];
                const V* src = ring + (s * 32 + lane) * E;
#pragma unroll
                for (int e = 0; e < E; ++e) xk[e] = src[e];
                __syncwarp();
                if (lane == 0 && r + LINE_XR < nrow) {  // hand the slot back when it is written again
                    mbar_arrive_expect_tx(&full[s], XBYTES);
                    mbar_arrive_remote(dn_empty + 8u * s);
                }
#pragma unroll
                for (int e = 0; e < E; ++e) f[e] = fma(ck, xk[e], f[e]);
            } else if (from_xch) {
                V xk[E];
                long long spins = 0;
                bool have;
                do {
                    const volatile typename B::U* src = reinterpret_cast<const volatile typename B::U*>(xin + r * xrow);
                    have = true;
#pragma unroll
                    for (int e = 0; e < E; ++e) {
                        const typename B::U v = src[e];
                        have = have && v != ~(typename B::U)0;
                        xk[e] = B::from(v);
                    }
                    if (++spins > SPIN_LIMIT) break;
                } while (!__all_sync(0xffffffffu, have));
                if (!__all_sync(0xffffffffu, have)) { dead = true; return; }
                typename B::U* dst = reinterpret_cast<typename B::U*>(xin + r * xrow);
#pragma unroll
                for (int e = 0; e < E; ++e) dst[e] = ~(typename B::U)0;  // empty again for the next launch
#pragma unroll
                for (int e = 0; e < E; ++e) f[e] = fma(ck, xk[e], f[e]);
            }
            // ---- the line: local chain, scan over the lanes, carry of the segment before
            V x[E];
            x[0] = f[0];
#pragma unroll
            for (int e = 1; e < E; ++e) x[e] = fma(ci, x[e - 1], f[e]);
            V b = x[E - 1];
#pragma unroll
            for (int l = 0; l < 5; ++l)
                if (l < nlev) b = fma(lev[l], __shfl_up_sync(0xffffffffu, b, 1 << l), b);
            V c = V(0);
            if (seg > 0) {
                const volatile typename B::U* m = reinterpret_cast<const volatile typename B::U*>(prev_mail + r);
                typename B::U v;
                long long spins = 0;
                while ((v = *m) == ~(typename B::U)0)
                    if (++spins > SPIN_LIMIT) break;
                if (__any_sync(0xffffffffu, v == ~(typename B::U)0)) { dead = true; return; }
                c = B::from(v);
                b = fma(acar, c, b);
            }
            if (seg < S - 1 && lane == 31) *const_cast<volatile V*>(my_mail + r) = line_flagged(b);
            V y = __shfl_up_sync(0xffffffffu, b, 1);
            if (lane == 0) y = c;
            if (starts) y = V(0);
#pragma unroll
            for (int e = 0; e < E - 1; ++e) x[e] = fma(cpw[e], y, x[e]);
            x[E - 1] = b;
            if (edge) {
#pragma unroll
                for (int e = 0; e < E; ++e) x[e] = ok[e] ? x[e] : V(0);
            }
            // ---- hand the row to the plane above, then to global memory
            if (to_ring) {
                const int s = r % LINE_XR;
                if (r >= LINE_XR &&
                    !__all_sync(0xffffffffu, mbar_wait(&empty[s], (unsigned)(r / LINE_XR - 1) & 1u))) {
                    dead = true;
                    return;
                }
                xpush<E>(up_data + (unsigned)(s * XBYTES), up_full + 8u * s, x);
            } else if (to_xch) {
                volatile V* dst = xout + r * xrow;
#pragma unroll
                for (int e = 0; e < E; ++e) dst[e] = line_flagged(x[e]);
            }
            if (on) {
                if (!GS || !edge) {
                    line_store<V, E>(outp + r * rstep, x, BWD);
                    if (GS && hout) line_store<V, E>(hout + r * rstep, x, BWD);
                } else {  // the faces i = 0 and nx-1 keep their boundary values
#pragma unroll
                    for (int e = 0; e < E; ++e)
                        if (ok[e]) {
                            outp[r * rstep + e] = x[e];
                            if (hout) hout[r * rstep + e] = x[e];
                        }
                }
            }
#pragma unroll
            for (int e = 0; e < E; ++e) xj[e] = x[e];
            if (GS && r == 0) {
#pragma unroll
                for (int e = 0; e < E; ++e) x0[GS ? e : 0] = x[e];
            }
        };
        for (int r0 = 0; r0 < nrow && !dead; r0 += D) {
#pragma unroll
            for (int u = 0; u < D; ++u)
                if (r0 + u < nrow && !dead) row(r0 + u, pf[u]);
        }
        if (dead && lane == 0) atomicExch(a.err, TBL_ERR_TIMEOUT);
        __syncwarp();
    }
    cluster_sync_all();  // pushes into a CTA's shared memory have landed or will not come
}

// ------------------------------------------------------------------ host
template <typename V> constexpr int line_e() { return 4; }
template <typename V> constexpr int line_d() { return sizeof(V) == 8 ? 4 : 8; }

template <int MODE, typename V>
static const void* line_fn() { return (const void*)k_line<MODE, V, line_e<V>(), line_d<V>()>; }

static size_t line_smem(int S, int KP, int rows, size_t vsize, int E) {
    const size_t nw = (size_t)S * KP;
    return nw * LINE_XR * 32 * E * vsize + nw * 2 * LINE_XR * 8 + nw * rows * vsize;
}

static void line_cfg(const tbl_handle* h, const LineShape& q, int nsets, cudaLaunchConfig_t& cfg,
                     cudaLaunchAttribute* at) {
    cfg = {};
    cfg.gridDim = dim3((unsigned)(h->P * q.nblk * q.ngrp * q.nc), (unsigned)nsets);
    cfg.blockDim = dim3((unsigned)(32 * q.S * q.KP));
    cfg.dynamicSmemBytes = q.smem;
    cfg.stream = h->stream;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)q.nc;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}

// Splits a slab column of Kmax planes over CTAs and clusters for one kernel.
// False when the line sweeps do not take this grid.
static bool line_plan(const tbl_handle* h, const void* fn, size_t vsize, int E, int rows, int nblk, int want_kp,
                      LineShape& q) {
    const int C = (h->g.nx - 2) / E + 1;
    int kmax = 1;
    for (int r = 0; r < h->P; ++r) kmax = std::max(kmax, h->en[r] - h->bn[r] + 1);
    q = LineShape();
    q.S = (C + 31) / 32;
    q.rows = rows;
    q.nblk = nblk;
    if (q.S > LINE_MAX_WARPS || (long long)q.S * rows > LINE_MAX_SLOTS) return false;
    const int kp_max = std::max(1, LINE_MAX_WARPS / q.S);
    for (q.KP = std::min(want_kp, kp_max); q.KP <= kp_max; ++q.KP)
        for (int most = 16; most >= 8; most -= 8) {  // 16 CTAs where the device takes such clusters
            if ((long long)q.S * q.KP * rows > LINE_MAX_SLOTS) return false;
            const int ctas = (kmax + q.KP - 1) / q.KP;
            q.ngrp = (ctas + most - 1) / most;
            q.nc = (ctas + q.ngrp - 1) / q.ngrp;
            q.smem = line_smem(q.S, q.KP, rows, vsize, E);
            cudaLaunchConfig_t cfg;
            cudaLaunchAttribute at[1];
            line_cfg(h, q, 1, cfg, at);
            int ncl = 0;
            if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, LINE_MAX_SMEM) != cudaSuccess ||
                cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
                cudaOccupancyMaxActiveClusters(&ncl, fn, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                continue;
            }
            // the clusters of a column wait on one another: all of a launch's clusters must be resident
            q.sets = ncl < 1 ? 0 : q.ngrp == 1 ? 3 : std::min(3, ncl / (h->P * nblk * q.ngrp));
            if (q.sets >= 1) return true;
        }
    return false;
}

template <typename V>
static int line_init(tbl_handle* h) {
    const int J = h->g.ny - 2;
    const int kp = sizeof(V) == 8 ? 1 : 1;
    const bool span = (h->cfg.flags & TBL_FLAG_SSOR_SPAN_BLOCKS) != 0;
    const int brows = span ? std::min(32, J) : J, nblk = span ? (J + 31) / 32 : 1;
    h->line[0].S = h->line[1].S = h->line[2].S = 0;
    LineShape q[3];
    if (line_plan(h, line_fn<0, V>(), sizeof(V), line_e<V>(), J, 1, kp, q[0])) h->line[0] = q[0];
    if (line_plan(h, line_fn<1, V>(), sizeof(V), line_e<V>(), brows, nblk, kp, q[1]) &&
        line_plan(h, line_fn<2, V>(), sizeof(V), line_e<V>(), brows, nblk, kp, q[2])) {
        h->line[1] = q[1];
        h->line[2] = q[2];
    }
    size_t words = 0;
    for (int m = 0; m < 3; ++m) {
        const LineShape& s = h->line[m];
        if (s.S > 0)
            words = std::max(words, (size_t)(m == 0 ? std::min(3, s.sets) : 1) * h->P * s.nblk * (s.ngrp - 1) * s.rows *
                                        32 * line_e<V>() * s.S);
    }
    if (words > 0) {
        TBL_CUDA_TRY(cudaMalloc(&h->line_xch, words * sizeof(V)));
        TBL_CUDA_TRY(cudaMemset(h->line_xch, 0xff, words * sizeof(V)));
    }
    return TBL_OK;
}

int line_create(tbl_handle* h) {
    return h->cfg.precision == TBL_PREC_MIXED ? line_init<float>(h) : line_init<double>(h);
}

template <typename V>
static LineArgs<V> line_args(tbl_handle* h, const LineShape& q) {
    LineArgs<V> a = {};
    a.g = h->g;
    a.slabs = h->slabs;
    a.err = h->err;
    a.S = q.S; a.KP = q.KP; a.nc = q.nc; a.ngrp = q.ngrp; a.nblk = q.nblk; a.rows = q.rows;
    a.P = h->P;
    a.Ab = h->Ab; a.At = h->At; a.rAp = h->rAp;
    a.aw = 1.0 / (h->cfg.dx * h->cfg.dx);
    a.as = 1.0 / (h->cfg.dy * h->cfg.dy);
    a.omega = h->cfg.omega;
    a.xch = (V*)h->line_xch;
    return a;
}

template <int MODE, typename V>
static int line_launch(tbl_handle* h, const LineShape& q, LineArgs<V>& a, int nsets) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    line_cfg(h, q, nsets, cfg, at);
    TBL_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_line<MODE, V, line_e<V>(), line_d<V>()>, a));
    h->launches++;
    return TBL_OK;
}

template <typename V>
int launch_line_gs(tbl_handle* h, V* const F[3], V* const PRE[3], V* halo_out, const int* comps, int ncomp) {
    const LineShape& q = h->line[0];
    const size_t nz = (size_t)h->g.nz;
    LineArgs<V> a = line_args<V>(h, q);
    a.gsc = sizeof(V) == 8 ? (const V*)h->gs_coef : (const V*)h->gs_coef_f;
    a.gsb = a.gsc + (sizeof(V) == 8 ? 7 : 4) * nz;
    a.halo_out = halo_out;
    for (int c = 0; c < 3; ++c) { a.out[c] = F[c]; a.in[c] = PRE[c]; }
    for (int c0 = 0; c0 < ncomp; c0 += q.sets) {
        const int n = std::min(ncomp - c0, q.sets);
        for (int c = 0; c < n; ++c) a.comp[c] = comps[c0 + c];
        const int s = line_launch<0, V>(h, q, a, n);
        if (s != TBL_OK) return s;
    }
    return TBL_OK;
}

template <typename V>
int launch_line_ssor(tbl_handle* h, bool bwd, const V* in, V* out, const int* skip) {
    const LineShape& q = h->line[bwd ? 2 : 1];
    LineArgs<V> a = line_args<V>(h, q);
    a.in[0] = in;
    a.out[0] = out;
    a.skip = skip;
    // streamwise blocks of the same points as the wavefront sweep's
    if (h->ssor_nib > 1) {
        const int ch = sweep_chunk(sizeof(V)), C = (h->g.nx - 2) / ch + 1;
        a.cb = (C + h->ssor_nib - 1) / h->ssor_nib * (ch / line_e<V>());
    }
    return bwd ? line_launch<2, V>(h, q, a, 1) : line_launch<1, V>(h, q, a, 1);
}

template int launch_line_gs<double>(tbl_handle*, double* const[3], double* const[3], double*, const int*, int);
template int launch_line_gs<float>(tbl_handle*, float* const[3], float* const[3], float*, const int*, int);
template int launch_line_ssor<double>(tbl_handle*, bool, const double*, double*, const int*);
template int launch_line_ssor<float>(tbl_handle*, bool, const float*, float*, const int*);

}  // namespace tbl
