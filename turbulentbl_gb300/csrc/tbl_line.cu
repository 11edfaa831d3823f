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
//   * the plane below comes row by row: from another warp of the CTA straight
//     into a ring in shared memory, from another CTA through a global exchange
//     buffer whose words are their own flags too, which a courier warp polls
//     and copies into the ring (the loads of a poll in flight would otherwise
//     stall the sweeping warps); the rows' operands are fetched by bulk copies,
//     four rows at a time.
//
// CTAs take their planes by ticket, the lowest planes of all slabs first, so
// that a CTA only ever waits for CTAs that have started: the launch needs no
// co-residency.  All waits are bounded (about a second); a wait that gives up
// sets the error word and the warps that depend on it give up in turn.  Rows it
// did not take stay in the exchange buffer, so the error word is never cleared:
// a handle that has timed out reports it from then on.
//
// What bounds it: the serial chain of J + K rows.  An FP64 row with 1 point per
// lane takes about 900 cycles at 128 x 66 x 64, of which 320 are the scan (an
// FP64 FMA of 64 and two shuffles a level) and 180 the other FMAs; the rest, and
// most of an FP32 row's 620, is the issue of about 170 instructions from one
// warp per scheduler, where a branch costs 20 to 30 cycles taken or not.  At
// 512 x 130 x 128 two FP64 warps share a pipe: 1400.  A hand-over to the next
// CTA takes about 1 us.  What left the row for that reason: operand copies (100
// cycles each to issue; a feeder warp does it), selects and tests at its ends.
// SSOR sweep, wavefront -> line scan: 130 -> 53 us (128 x 66 x 64, FP64, 8
// slabs), 389 -> 176 us (512 x 130 x 128, FP64), 95 -> 34 us and 251 -> 74 us
// (FP32); GS sweep of three components 54 us at 128 and 305 at 512 (FP64), with its
// precomputed terms 280 -> 64 and 620 -> 493 us.
// A first form with thread-block clusters (st.async into the next CTA's ring)
// was slower at 512 (243 us): clusters of 15 CTAs doubled up on SMs.  Register
// prefetch of the operands was slower too (their loads share scoreboards with
// the shuffles: every row waited for them).
#include <algorithm>
#include <climits>

#include "tbl_internal.cuh"
#include "tbl_kernels.cuh"
#include "tbl_sync.cuh"

namespace tbl {

constexpr int LINE_XR = 8;           // ring slots (rows) per warp, in two halves that are handed back whole
// sweeping warps of a CTA at most, so that the registers of E points per lane fit
constexpr int line_max_warps(int E) { return E >= 4 ? 12 : 16; }
constexpr int LINE_MAX_COURIERS = 4;
constexpr int LINE_MAX_SMEM = 222 * 1024;
// mbarriers per warp: the plane below's row is in a slot; a half of the slots
// has been read; a half's operands have landed
constexpr int LINE_BARS = LINE_XR + 4;

template <typename V>
struct LineArgs {
    Geom g;
    const LineCta* ctas;     // CTAs of one component, lowest planes first
    unsigned* ticket;        // [taken, finished]
    int* err;
    const int* skip;
    int S, KP, NC, nsets;  // warps per line, planes per CTA, couriers, components
    int rows;              // rows of a span block (the last may have fewer)
    int cb;                // SSOR streamwise blocks: chunks per block (0 = one block)
    const double *Ab, *At, *rAp;
    double aw, as, omega;
    const V* gsc;      // GS: [p0|p1|p2|p3] x nz of the handle's coefficient table
    const V* gsb;      // GS: nz coefficients of U(k-1)
    V* out[3];         // GS: fields; SSOR: out[0]
    const V* in[3];    // GS: precomputed old-value terms; SSOR: in[0]
    int comp[3];
    V* xch;            // [set][plane handed over][span row][32 E S], empty words all ones
    int nxp;           // planes handed over (one component)
};

template <typename V> struct LineBits;
template <> struct LineBits<double> {
    static __device__ __forceinline__ unsigned hi(double v) { return (unsigned)__double2hiint(v); }
    static __device__ __forceinline__ double nan() { return __hiloint2double(0x7fffffff, -1); }
    static __device__ __forceinline__ double empty() { return __hiloint2double(-1, -1); }
    static constexpr double tiny = 8.7e-19;  // 2^-60
};
template <> struct LineBits<float> {
    static __device__ __forceinline__ unsigned hi(float v) { return __float_as_uint(v); }
    static __device__ __forceinline__ float nan() { return __uint_as_float(0x7fffffffu); }
    static __device__ __forceinline__ float empty() { return __uint_as_float(0xffffffffu); }
    static constexpr float tiny = 2.3e-10f;  // 2^-32
};
// "Not written yet" is a NaN with its high word all ones; results with that
// high word are stored as another NaN.
template <typename V>
__device__ __forceinline__ bool line_empty(V v) { return LineBits<V>::hi(v) == 0xffffffffu; }
__device__ __forceinline__ double line_value(double v) { return line_empty(v) ? LineBits<double>::nan() : v; }
__device__ __forceinline__ float line_value(float v) { return v; }  // FP32 arithmetic gives one NaN, 0x7fffffff

// E values of the exchange buffer; each value is read and written whole.
__device__ __forceinline__ void xch_ld(double (&v)[1], const double* p) {
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v[0]) : "l"(p) : "memory");
}
__device__ __forceinline__ void xch_ld(double (&v)[2], const double* p) {
    asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "l"(p) : "memory");
}
__device__ __forceinline__ void xch_ld(double (&v)[4], const double* p) {
    xch_ld(reinterpret_cast<double(&)[2]>(v[0]), p);
    xch_ld(reinterpret_cast<double(&)[2]>(v[2]), p + 2);
}
__device__ __forceinline__ void xch_ld(float (&v)[2], const float* p) {
    asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(v[0]), "=f"(v[1]) : "l"(p) : "memory");
}
__device__ __forceinline__ void xch_ld(float (&v)[4], const float* p) {
    asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void xch_ld(float (&v)[8], const float* p) {
    xch_ld(reinterpret_cast<float(&)[4]>(v[0]), p);
    xch_ld(reinterpret_cast<float(&)[4]>(v[4]), p + 4);
}
__device__ __forceinline__ void xch_put(double* p, const double (&v)[1]) {
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v[0]) : "memory");
}
__device__ __forceinline__ void xch_put(double* p, const double (&v)[2]) {
    asm volatile("st.relaxed.gpu.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v[0]), "d"(v[1]) : "memory");
}
__device__ __forceinline__ void xch_put(double* p, const double (&v)[4]) {
    xch_put(p, reinterpret_cast<const double(&)[2]>(v[0]));
    xch_put(p + 2, reinterpret_cast<const double(&)[2]>(v[2]));
}
__device__ __forceinline__ void xch_put(float* p, const float (&v)[2]) {
    asm volatile("st.relaxed.gpu.global.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v[0]), "f"(v[1]) : "memory");
}
__device__ __forceinline__ void xch_put(float* p, const float (&v)[4]) {
    asm volatile("st.relaxed.gpu.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3])
                 : "memory");
}
__device__ __forceinline__ void xch_put(float* p, const float (&v)[8]) {
    xch_put(p, reinterpret_cast<const float(&)[4]>(v[0]));
    xch_put(p + 4, reinterpret_cast<const float(&)[4]>(v[4]));
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}

// E values in memory order <-> in sweep order, by the widest accesses.
template <int BYTES> struct LineWord { using T = int4; };
template <> struct LineWord<8> { using T = int2; };
template <typename V, int E>
__device__ __forceinline__ void line_read(V (&v)[E], const V* p, bool rev) {
    using T = typename LineWord<E * sizeof(V)>::T;
    constexpr int W = sizeof(T) / sizeof(V);
    V t[E];
#pragma unroll
    for (int b = 0; b < E / W; ++b) *reinterpret_cast<T*>(&t[b * W]) = *(reinterpret_cast<const T*>(p) + b);
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = rev ? t[E - 1 - e] : t[e];
}
template <typename V, int E>
__device__ __forceinline__ void line_store(V* p, const V (&v)[E], bool rev) {
    using T = typename LineWord<E * sizeof(V)>::T;
    constexpr int W = sizeof(T) / sizeof(V);
    V t[E];
#pragma unroll
    for (int e = 0; e < E; ++e) t[e] = rev ? v[E - 1 - e] : v[e];
#pragma unroll
    for (int b = 0; b < E / W; ++b) *(reinterpret_cast<T*>(p) + b) = *reinterpret_cast<const T*>(&t[b * W]);
}
// `bytes` of global memory into this CTA's shared memory, counted by a barrier.
__device__ __forceinline__ void line_fetch(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// Chunks of E points of a line, points 0 .. nx-2 at least, a whole number of
// 16-byte words (a backward segment starts that many chunks from the end).
template <typename V, int E>
__host__ __device__ constexpr int line_chunks(int nx) {
    constexpr int M = E * sizeof(V) >= 16 ? 1 : 16 / (E * (int)sizeof(V));
    return ((nx - 2) / E + 1 + M - 1) / M * M;
}

template <typename V, int E>
__device__ __forceinline__ bool line_arrived(const V (&w)[E]) {
    bool have = true;
#pragma unroll
    for (int e = 0; e < E; ++e) have = have && !line_empty(w[e]);
    return have;
}
// A courier's wait for one segment of a row of the plane below.
template <typename V, int E>
__device__ __forceinline__ void xch_wait(V (&w)[E], const V* p, bool& good) {
    for (long long spins = 0; good;) {
        xch_ld(w, p);
        if (__all_sync(0xffffffffu, line_arrived(w))) break;
        good = ++spins < SPIN_LIMIT / 16;
    }
}
// A warp's wait for the carry into its segment.
template <typename V>
__device__ __forceinline__ bool carry_wait(V& c, const volatile V* p) {
    for (long long spins = 0; spins < SPIN_LIMIT; ++spins) {
        c = *p;
        if (!__any_sync(0xffffffffu, line_empty(c))) return true;
    }
    return false;
}

template <int MODE, typename V, int E>
__global__ void __launch_bounds__(32 * (line_max_warps(E) + LINE_MAX_COURIERS + 1), 1) k_line(const LineArgs<V> a) {
    dependent_wait();
    if (a.skip && *a.skip) return;  // every CTA reads the same word, written by an earlier launch
    using B = LineBits<V>;
    constexpr bool GS = MODE == 0, BWD = MODE == 2;
    constexpr unsigned ALL = 0xffffffffu;
    constexpr int XR = LINE_XR, H = XR / 2;
    constexpr unsigned LBYTES = 32 * E * sizeof(V);  // a warp's segment of a row
    const Geom& g = a.g;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int S = a.S, KP = a.KP, NW = S * KP;

    // shared memory: rings of the warps, a slot holding a row's operands and the
    // row of the plane below | their barriers | carry mailboxes [warp][row]
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ unsigned s_ticket;
    V* const rings = reinterpret_cast<V*>(s_dyn);
    unsigned long long* const bars = reinterpret_cast<unsigned long long*>(s_dyn + (size_t)NW * XR * 2 * LBYTES);
    V* const mail = reinterpret_cast<V*>(bars + NW * LINE_BARS);
    if (threadIdx.x == 0) s_ticket = atomicAdd(a.ticket, 1u);
    for (int q = threadIdx.x; q < NW * a.rows; q += blockDim.x) mail[q] = B::empty();
    __syncthreads();
    const int set = (int)(s_ticket % (unsigned)a.nsets);
    const LineCta cta = a.ctas[s_ticket / (unsigned)a.nsets];
    const int J = g.ny - 2, K = cta.K;
    const int comp = GS ? a.comp[set] : 0;
    const int j0 = cta.blk * a.rows, nrow = min(a.rows, J - j0);  // logical rows [j0, j0 + nrow)
    const int jfirst = BWD ? J - 1 - j0 : j0;                     // logical row 0
    const int seg = wid % S, kp = wid / S;
    const int kl = cta.kg * KP + kp;  // logical plane
    const bool sweeps = wid < NW && kl < K;
    const int kidx = BWD ? K - 1 - kl : kl;
    const int k = cta.bn + (sweeps ? kidx : 0);
    const bool below = kl > 0;  // a plane of the slab comes before this one
    unsigned long long* const full = bars + (sweeps ? wid : 0) * LINE_BARS;
    unsigned long long *const empty = full + XR, *const opfull = full + XR + 2;
    if (sweeps && lane < LINE_BARS) mbar_init(&full[lane], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncthreads();

    const size_t xrow = (size_t)32 * E * S;
    // exchange rows of a plane handed over, this lane's values of segment 0
    auto xch_plane = [&](int p) {
        return a.xch + ((((size_t)set * a.nxp + p) * J + j0) * S * 32 + lane) * E;
    };
    // The row segments of a warp's operands in global memory: chunks [c0, ..) of
    // the line, at chunk c0 - clo of the slot.
    const int C = line_chunks<V, E>(g.nx);
    if (wid == NW + a.NC) {
        // Feeder: the rows' operands, half a ring at a time, lane w for warp w (a
        // bulk copy takes its thread about 100 cycles to issue).
        const int fl = cta.kg * KP + lane / S, fs = lane % S;
        const bool feeds = lane < NW && fl < K;
        unsigned long long* const fb = bars + (feeds ? lane : 0) * LINE_BARS;
        const int clo = BWD ? C - 32 * (fs + 1) : 32 * fs, c0 = max(clo, 0);
        const unsigned bytes =
            min((unsigned)(g.sx - E * c0), 32u * E - (unsigned)(E * (c0 - clo))) * (unsigned)sizeof(V);
        const long long rstep = BWD ? -(long long)g.sx : (long long)g.sx;
        const int fk = cta.bn + (feeds ? (BWD ? K - 1 - fl : fl) : 0);
        const V* src = a.in[comp] + (long long)g.sx * ((long long)(1 + jfirst) + (long long)g.ny * fk) + E * c0;
        const unsigned dst = smem_u32(rings) + ((unsigned)(feeds ? lane : 0) * XR * 2 * 32 + (unsigned)(c0 - clo)) * E *
                                                   (unsigned)sizeof(V);
        const int nh = feeds ? (nrow + H - 1) / H : 0;
        int m = 0;
        long long spins = 0;
        bool fail = false;
        while (__any_sync(ALL, m < nh && !fail)) {
            const bool go = m < nh && !fail && (m < 2 || mbar_test(&fb[XR + (m & 1)], (unsigned)(m / 2 - 1) & 1u));
            if (go) {
                const int n = min(H, nrow - m * H);
                mbar_arrive_expect_tx(&fb[XR + 2 + (m & 1)], bytes * n);
                for (int w = 0; w < n; ++w, src += rstep)
                    line_fetch(dst + (unsigned)((m & 1) * H + w) * 2 * LBYTES, src, bytes, smem_u32(&fb[XR + 2 + (m & 1)]));
                ++m;
                spins = 0;
            } else if (m < nh && ++spins > SPIN_LIMIT) {
                fail = true;
            }
            if (!__any_sync(ALL, go)) __nanosleep(64);
        }
        // every copy has landed before the CTA ends
        for (int q = max(0, m - 2); q < m; ++q)
            if (!mbar_wait(&fb[XR + 2 + (q & 1)], (unsigned)(q / 2) & 1u)) fail = true;
        if (fail) atomicExch(a.err, TBL_ERR_TIMEOUT);
    } else if (wid >= NW) {
        // Courier: the top plane of the CTA below, row by row, into the rings of
        // this CTA's first plane; its words are emptied for the next launch.
        const int sg0 = wid - NW;
        const bool has = cta.kg > 0 && cta.kg * KP < K;
        V* const src = xch_plane(has ? cta.xp - 1 : 0);
        V none[E];
#pragma unroll
        for (int e = 0; e < E; ++e) none[e] = B::empty();
        auto hand = [&](int r, int sg, const V(&w)[E]) {
            const int u = r & (XR - 1);
            line_store<V, E>(rings + (((size_t)sg * XR + u) * 64 + 32 + lane) * E, w, false);
            __syncwarp();
            if (lane == 0) mbar_arrive(bars + sg * LINE_BARS + u);
            xch_put(src + r * xrow + (size_t)sg * 32 * E, none);
        };
        bool good = true;
        if (has && S <= a.NC) {  // one segment
            unsigned long long* const fb = bars + sg0 * LINE_BARS + XR;
            for (int r = 0; r < nrow && good; ++r) {
                if ((r & (H - 1)) == 0 && r >= XR)
                    good = __all_sync(ALL, mbar_wait(&fb[(r & (XR - 1)) / H], (unsigned)(r / XR - 1) & 1u));
                V w[E];
                xch_wait<V, E>(w, src + r * xrow + (size_t)sg0 * 32 * E, good);
                if (good) hand(r, sg0, w);
            }
        } else if (has) {
            // Several segments: a look at a word takes an L2 round trip, 700 cycles
            // of a row's 1400, so one at each is in flight and none is waited for
            // alone (taken in turn, 180 against 174 us a sweep at 512 x 130 x 128
            // in FP64; a courier for each, whose registers the sweeping warps lack,
            // 187; this loop for one segment costs a hand-over 0.3 us).
            constexpr int CS = (line_max_warps(E) + LINE_MAX_COURIERS - 1) / LINE_MAX_COURIERS;
            int row[CS];  // the next row of segments sg0, sg0 + NC, ..
#pragma unroll
            for (int c = 0; c < CS; ++c) row[c] = sg0 + c * a.NC < S ? 0 : nrow;
            long long spins = 0;
            for (bool more = true; more && good; good = ++spins < SPIN_LIMIT / 16) {
                V w[CS][E];
#pragma unroll
                for (int c = 0; c < CS; ++c)
                    if (row[c] < nrow) xch_ld(w[c], src + row[c] * xrow + (size_t)(sg0 + c * a.NC) * 32 * E);
                more = false;
#pragma unroll
                for (int c = 0; c < CS; ++c) {
                    if (row[c] >= nrow) continue;
                    const int r = row[c], u = r & (XR - 1), sg = sg0 + c * a.NC;
                    bool have = line_arrived(w[c]);
                    if ((u & (H - 1)) == 0 && r >= XR)
                        have = mbar_test(bars + sg * LINE_BARS + XR + u / H, (unsigned)(r / XR - 1) & 1u) && have;
                    if (__all_sync(ALL, have)) {
                        hand(r, sg, w[c]);
                        ++row[c];
                        spins = 0;
                    }
                    more = more || row[c] < nrow;
                }
            }
        }
        if (!good && lane == 0) atomicExch(a.err, TBL_ERR_TIMEOUT);
    } else if (sweeps) {
        V* const ring = rings + (size_t)wid * XR * 64 * E;
        const bool has_up = kl + 1 < K;
        const bool to_ring = has_up && kp < KP - 1, to_xch = has_up && kp == KP - 1;
        V* const up_ring = ring + (size_t)S * XR * 64 * E + (32 + lane) * E;
        unsigned long long* const up_full = full + S * LINE_BARS;
        V* xout = to_xch ? xch_plane(cta.xp) + (size_t)seg * 32 * E : nullptr;

        const long long rstep = BWD ? -(long long)g.sx : (long long)g.sx;

        // this lane's points: chunk ch of the line in sweep order, i = i0 .. i0 + E - 1
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
        const bool whole = all_ok, edge = __any_sync(ALL, !all_ok);  // the warp holds a line end
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
        V* outp = a.out[comp] + (long long)g.sx * ((long long)(1 + jfirst) + (long long)g.ny * k) + i0;
        volatile V* const my_mail = mail + (size_t)wid * a.rows;
        const volatile V* const prev_mail = mail + (size_t)(seg > 0 ? wid - 1 : wid) * a.rows;

        V gr[E], xj[E], x0[GS ? E : 1];
#pragma unroll
        for (int e = 0; e < E; ++e) xj[e] = V(0);

        // Row q's right-hand side with the plane below's share: ask() looks
        // without waiting, get() waits.  An ask that came too early has read a
        // stale slot, and get() follows.  Lanes beyond the line read what is
        // there: no point of the line depends on them.
        // The first plane of a slab has zeros in the slots of the plane below, and
        // looks at its operands' barrier in place of theirs.
        const V* const slot0 = ring + (BWD ? 31 - lane : lane) * E;
        V* const below0 = ring + (32 + lane) * E;
        if (!below) {
            V none[E];
#pragma unroll
            for (int e = 0; e < E; ++e) none[e] = V(0);
            for (int s = 0; s < XR; ++s) line_store<V, E>(below0 + s * 64 * E, none, false);
        }
        auto take = [&](int s, V(&o)[E]) {
            V xk[E];
            line_read<V, E>(o, slot0 + s * 64 * E, BWD);
            line_read<V, E>(xk, below0 + s * 64 * E, false);
#pragma unroll
            for (int e = 0; e < E; ++e) o[e] = fma(ck, xk[e], o[e]);
        };
        auto there = [&](int s) { return below ? &full[s] : &opfull[s / H]; };
        auto ask = [&](int s, unsigned ph, V(&o)[E]) -> bool {
            bool rdy = mbar_test(there(s), ph);
            if ((s & (H - 1)) == 0) rdy = mbar_test(&opfull[s / H], ph) && rdy;
            rdy = __all_sync(ALL, rdy);
            take(rdy ? s : (s ^ 1), o);  // the address waits for the test
            return rdy;
        };
        bool dead = false;  // a wait gave up: nothing waits any more, and the results mean nothing
        auto get = [&](int s, unsigned ph, V(&o)[E]) {
            bool got = dead || mbar_wait(there(s), ph);
            if ((s & (H - 1)) == 0) got = (dead || mbar_wait(&opfull[s / H], ph)) && got;
            if (!__all_sync(ALL, got)) dead = true;
            take(s, o);
        };
        // The H rows up to q have been read: their slots are handed back to the
        // plane below and to the feeder.
        auto done = [&](int q, int s) {
            if ((s & (H - 1)) != H - 1) return;
            __syncwarp();
            if (lane == 0 && q + H + 1 < nrow) mbar_arrive(&empty[s / H]);
        };

        // One row: gr holds its right-hand side and the plane below's share.
        // What the next row needs from the plane below is looked at while this
        // row's scan runs, and waited for only after this row has been handed on.
        // (Every branch and every instruction of a row counts: the chain of rows
        // is one warp's issue.)
        auto row = [&](const int r, const int u, const unsigned ph) {
            V x[E];
#pragma unroll
            for (int e = 0; e < E; ++e) x[e] = fma(cj, xj[e], gr[e]);
            if (GS && r == nrow - 1) {  // periodic: the last row reads the first row's new values
                __syncwarp();           // (a branch: predicated FMAs would cost FP64 issue in every row)
#pragma unroll
                for (int e = 0; e < E; ++e) x[e] = fma(cj, x0[GS ? e : 0], x[e]);
            }
            V c = seg > 0 ? prev_mail[r] : V(0);
            // the line: local chain, scan over the lanes
#pragma unroll
            for (int e = 1; e < E; ++e) x[e] = fma(ci, x[e - 1], x[e]);
            V b = x[E - 1];
            b = fma(lev[0], __shfl_up_sync(ALL, b, 1), b);
            b = fma(lev[1], __shfl_up_sync(ALL, b, 2), b);
            if (nlev > 2) {
                b = fma(lev[2], __shfl_up_sync(ALL, b, 4), b);
                if (nlev > 3) {
                    b = fma(lev[3], __shfl_up_sync(ALL, b, 8), b);
                    if (nlev > 4) b = fma(lev[4], __shfl_up_sync(ALL, b, 16), b);
                }
            }
            const bool more = r + 1 < nrow;
            const int s1 = (u + 1) % XR;
            const unsigned ph1 = u + 1 == XR ? ph ^ 1u : ph;
            const bool rdy = ask(s1, ph1, gr);  // (after the last row: what a slot holds, and not used)
            // the carry of the segment before
            if (seg > 0) {
                if (__any_sync(ALL, line_empty(c)) && !dead && !carry_wait(c, &prev_mail[r])) dead = true;
                b = fma(acar, c, b);
            }
            if (seg < S - 1 && lane == 31) my_mail[r] = line_value(b);
            V y = __shfl_up_sync(ALL, b, 1);
            if (lane == 0) y = c;
            if (starts) y = V(0);
#pragma unroll
            for (int e = 0; e < E - 1; ++e) x[e] = fma(cpw[e], y, x[e]);
            x[E - 1] = b;
            // GS: the boundary value at i = 0 enters the line only.  The other points
            // outside 1..nx-2 are zero (BWD) or come after the line's last.
            if (GS && ch == 0) x[0] = V(0);
            // hand the row to the plane above, then to global memory
            if (to_ring) {
                if ((u & (H - 1)) == 0 && r >= XR && !dead &&
                    !__all_sync(ALL, mbar_wait(&up_full[XR + u / H], ph ^ 1u)))
                    dead = true;
                line_store<V, E>(up_ring + u * 64 * E, x, false);
                __syncwarp();
                if (lane == 0) mbar_arrive(&up_full[u]);
            } else if (to_xch) {
                V w[E];
#pragma unroll
                for (int e = 0; e < E; ++e) w[e] = line_value(x[e]);
                xch_put(xout, w);
                xout += xrow;
            }
            if (whole) line_store<V, E>(outp, x, BWD);
            if (E > 1 && edge) {  // a line end in the chunk: the points outside keep their values
#pragma unroll
                for (int e = 0; e < E; ++e)
                    if (!whole && ok[e]) outp[BWD ? E - 1 - e : e] = x[e];
            }
            outp += rstep;
#pragma unroll
            for (int e = 0; e < E; ++e) xj[e] = x[e];
            if (GS && u == 0 && r == 0) {
#pragma unroll
                for (int e = 0; e < E; ++e) x0[GS ? e : 0] = x[e];
            }
            if (!rdy && more) get(s1, ph1, gr);
            if (more) done(r + 1, s1);
        };
        get(0, 0u, gr);
        unsigned ph = 0;
        for (int r0 = 0; r0 < nrow; r0 += XR, ph ^= 1u) {
#pragma unroll
            for (int u = 0; u < XR; ++u)
                if (r0 + u < nrow) row(r0 + u, u, ph);
        }
        if (dead && lane == 0) atomicExch(a.err, TBL_ERR_TIMEOUT);
        __syncwarp();
    }
    __syncthreads();  // the last CTA to finish leaves the tickets as it found them
    if (threadIdx.x == 0 && atomicAdd(a.ticket + 1, 1u) + 1 == gridDim.x) {
        a.ticket[0] = 0u;
        a.ticket[1] = 0u;
    }
}

// One warp waits as the sweeps do, at a barrier (which = 0), for a row of the plane
// below (1) or for a carry (2), for what nobody brings.
template <typename V>
__global__ void __launch_bounds__(32) k_line_wait(int which, V* word, int* err) {
    constexpr int E = sizeof(V) == 8 ? 1 : 4;
    __shared__ unsigned long long s_bar;
    __shared__ V s_mail;
    if (threadIdx.x == 0) {
        mbar_init(&s_bar, 1);
        s_mail = LineBits<V>::empty();
    }
    __syncwarp();
    bool got;
    if (which == 0) {
        got = mbar_wait(&s_bar, 0);
    } else if (which == 1) {
        V w[E];
        got = true;
        xch_wait<V, E>(w, word + threadIdx.x * E, got);
    } else {
        V c;
        got = carry_wait(c, &s_mail);
    }
    if (!got && threadIdx.x == 0) atomicExch(err, TBL_ERR_TIMEOUT);
}

// ------------------------------------------------------------------ host
// Kernels by points per lane: 1, 2, 4 in FP64, 4, 8 in FP32.
template <int MODE, typename V>
static void (*line_fn(int E))(const LineArgs<V>) {
    if constexpr (sizeof(V) == 8) return E == 1 ? k_line<MODE, V, 1> : E == 2 ? k_line<MODE, V, 2> : k_line<MODE, V, 4>;
    else return E == 4 ? k_line<MODE, V, 4> : k_line<MODE, V, 8>;
}
template <typename V>
static int line_chunks_of(int E, int nx) {
    if constexpr (sizeof(V) == 8)
        return E == 1 ? line_chunks<V, 1>(nx) : E == 2 ? line_chunks<V, 2>(nx) : line_chunks<V, 4>(nx);
    else return E == 4 ? line_chunks<V, 4>(nx) : line_chunks<V, 8>(nx);
}

// Splits the slab columns over CTAs of KP planes for one kernel.  False when
// the line sweeps do not take the grid: lines of more warps than a CTA may
// have, or rows that the mailboxes have no room for.
template <typename V>
static bool line_plan(const tbl_handle* h, int rows, int nblk, int E, int kp, LineShape& q) {
    q = LineShape();
    q.E = E;
    q.S = (line_chunks_of<V>(E, h->g.nx) + 31) / 32;
    if (q.S > line_max_warps(E)) return false;
    q.KP = std::min(kp, line_max_warps(E) / q.S);
    q.NC = std::min(q.S, LINE_MAX_COURIERS);
    q.rows = rows;
    q.nblk = nblk;
    const size_t plane = q.S * (LINE_XR * 64 * E * sizeof(V) + LINE_BARS * 8 + rows * sizeof(V));
    q.KP = std::min(q.KP, (int)(LINE_MAX_SMEM / plane));
    if (q.KP < 1) return false;
    q.smem = q.KP * plane;
    for (int r = 0; r < h->P; ++r) {
        const int nkg = (h->en[r] - h->bn[r] + 1 + q.KP - 1) / q.KP;
        q.ncta += nkg * nblk;
        q.nxp += nkg - 1;
    }
    return true;
}

// Lets the kernel of a plan have its shared memory (and loads it: only the
// chosen plan's, which tbl_create waits for).
template <int MODE, typename V>
static bool line_ready(const LineShape& q) {
    if (cudaFuncSetAttribute((const void*)line_fn<MODE, V>(q.E), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             LINE_MAX_SMEM) == cudaSuccess)
        return true;
    (void)cudaGetLastError();
    return false;
}

// A Gauss-Seidel launch sweeps three components at once, so its CTAs are
// counted in waves of one per SM: a second CTA on an SM shares its FP64 pipes
// or waits for its registers, and starts its chain late.  The plan takes the
// fewest waves, and of those the fewest points per lane and then planes per
// CTA.  FP64, E, KP = 2, 2 / 2, 3 / 4, 2 / 4, 3, us: 124 / 118 / 139 / 135 at
// 256 x 98 x 96 (one wave each); 194 / 157 / 203 / 182 at 256 x 130 x 128 and
// 341 / - / 343 / 300 at 512 x 130 x 128 (two, one, two, one; the last took 284
// before the couriers kept a look at each segment in flight, 5% that the SSOR
// sweeps gain: 180 -> 174, twice per Arnoldi step).  FP32, 4, 2 /
// 4, 3 / 8, 4: 111 / 98 / 103 at 512 x 130 x 128 (two, one, one), 119 / 131 /
// 99 at 512 x 102 x 190 (two, two, one); from two planes to three or four the
// hand-overs saved weigh as much.  FP32 lines of four warps or more take 8
// points (4 / 8: 60 / 64 at 384 x 98 x 96, 95 / 89 at 400 x 130 x 128, 97 / 91 at
// 512 x 130 x 128).
template <typename V>
static bool line_plan_gs(const tbl_handle* h, int rows, int E0, LineShape& q) {
    int best = INT_MAX;
    for (int E = E0; E <= (sizeof(V) == 8 ? 4 : 8); E *= 2)
        for (int kp = sizeof(V) == 8 ? 2 : 3; kp <= 4; ++kp) {
            LineShape t;
            if (!line_plan<V>(h, rows, 1, E, kp, t)) continue;
            const int waves = (3 * t.ncta + h->n_sm - 1) / h->n_sm;
            if (waves < best) {
                best = waves;
                q = t;
            }
        }
    return best < INT_MAX;
}

// The CTAs of a launch, the lowest of every column first.
static int line_table(const tbl_handle* h, LineShape& q) {
    std::vector<LineCta> t;
    std::vector<int> xp(h->P, 0);  // exchange planes before the column's
    for (int r = 1; r < h->P; ++r) xp[r] = xp[r - 1] + (h->en[r - 1] - h->bn[r - 1] + 1 + q.KP - 1) / q.KP - 1;
    for (int kg = 0; (int)t.size() < q.ncta; ++kg)
        for (int r = 0; r < h->P; ++r)
            if (kg * q.KP < h->en[r] - h->bn[r] + 1)
                for (int blk = 0; blk < q.nblk; ++blk)
                    t.push_back({h->bn[r], h->en[r] - h->bn[r] + 1, blk, kg, xp[r] + kg});
    TBL_CUDA_TRY(cudaMalloc(&q.ctas, t.size() * sizeof(LineCta)));
    TBL_CUDA_TRY(cudaMemcpy(q.ctas, t.data(), t.size() * sizeof(LineCta), cudaMemcpyHostToDevice));
    return TBL_OK;
}

template <typename V>
static int line_init(tbl_handle* h) {
    const int J = h->g.ny - 2, nx = h->g.nx;
    const bool span = (h->cfg.flags & TBL_FLAG_SSOR_SPAN_BLOCKS) != 0;
    const int brows = span ? std::min(32, J) : J, nblk = span ? (J + 31) / 32 : 1;
    // SSOR: points per lane and planes per CTA.  An FP64 row costs about 65
    // cycles per FMA that a warp issues, so few points per lane spread a line
    // over more of the SM's four FP64 pipes, but every warp pays for the scan.
    // Forward and backward sweep, E = 1 / 2: 100 / 117 us at 128 x 66 x 64,
    // 116 / 118 at 160 x 66 x 81, 138 / 140 at 201 x 77 x 59, level but for
    // seven warps a line instead of four, 188 / 173 at 256 x 98 x 96; E = 2 / 4: 317 / 356 at 512 x 130 x 128, 341 / 356 at
    // 700 x 130 x 100, 304 / 276 at 850 x 92 x 90.  FP32 rows are bound by
    // latency: 4 points, and two planes per CTA save a hand-over (152 / 147 /
    // 178 with 1 / 2 / 3 at 512 x 130 x 128); from five warps a line on, the
    // registers leave one CTA per SM and 8 points are better (4 / 8 points:
    // 316 / 260 at 768 x 194 x 144, 198 / 172 at 600 x 130 x 128, 147 / 153 at
    // 512).
    int E, kp;
    if (sizeof(V) == 8) {
        E = nx <= 161 ? 1 : nx <= 769 ? 2 : 4;
        kp = 1;
    } else {
        E = nx <= 513 ? 4 : 8;
        kp = 2;
    }
    LineShape q[3];
    const bool ssor = !(h->cfg.flags & TBL_FLAG_RB_PRECOND) && line_plan<V>(h, brows, nblk, E, kp, q[1]) &&
                      line_plan<V>(h, brows, nblk, E, kp, q[2]) && line_ready<1, V>(q[1]) && line_ready<2, V>(q[2]);
    const bool gs = !(h->cfg.flags & TBL_FLAG_RB_ORDER) &&
                    line_plan_gs<V>(h, J, sizeof(V) == 4 && nx > 385 ? 8 : E, q[0]) && line_ready<0, V>(q[0]);
    if (!gs && !ssor) return TBL_OK;
    size_t words = 32 * 8;  // the self-test's at least
    for (int m = 0; m < 3; ++m)
        if (m == 0 ? gs : ssor)
            words = std::max(words, (size_t)(m == 0 ? 3 : 1) * q[m].nxp * J * 32 * q[m].E * q[m].S);
    // Up to a few percent of the handle's memory: where only that is missing the
    // wavefront sweeps do with less.
    const cudaError_t e = cudaMalloc(&h->line_xch, words * sizeof(V));
    if (e == cudaErrorMemoryAllocation) {
        (void)cudaGetLastError();
        h->line_xch = nullptr;
        return TBL_OK;
    }
    TBL_CUDA_TRY(e);
    TBL_CUDA_TRY(cudaMemset(h->line_xch, 0xff, words * sizeof(V)));
    TBL_CUDA_TRY(cudaMalloc(&h->line_ticket, 2 * sizeof(unsigned)));
    TBL_CUDA_TRY(cudaMemset(h->line_ticket, 0, 2 * sizeof(unsigned)));
    for (int m = 0; m < 3; ++m) {
        if (m == 0 ? !gs : !ssor) continue;
        h->line[m] = q[m];
        const int st = line_table(h, h->line[m]);
        if (st != TBL_OK) return st;
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
    a.ctas = q.ctas;
    a.ticket = h->line_ticket;
    a.err = h->err;
    a.S = q.S; a.KP = q.KP; a.NC = q.NC; a.rows = q.rows;
    a.Ab = h->Ab; a.At = h->At; a.rAp = h->rAp;
    a.aw = 1.0 / (h->cfg.dx * h->cfg.dx);
    a.as = 1.0 / (h->cfg.dy * h->cfg.dy);
    a.omega = h->cfg.omega;
    a.xch = (V*)h->line_xch;
    a.nxp = q.nxp;
    return a;
}

template <int MODE, typename V>
static int line_launch(tbl_handle* h, const LineShape& q, LineArgs<V>& a, int nsets) {
    a.nsets = nsets;
    TBL_CUDA_TRY(launch_dependent(line_fn<MODE, V>(q.E), dim3(q.ncta * nsets), dim3(32 * (q.S * q.KP + q.NC + 1)), q.smem,
                                  h->stream, a));
    h->launches++;
    return TBL_OK;
}

template <typename V>
int launch_line_gs(tbl_handle* h, V* const F[3], V* const PRE[3], const int* comps, int ncomp) {
    const LineShape& q = h->line[0];
    const size_t nz = (size_t)h->g.nz;
    LineArgs<V> a = line_args<V>(h, q);
    a.gsc = sizeof(V) == 8 ? (const V*)h->gs_coef : (const V*)h->gs_coef_f;
    a.gsb = a.gsc + (sizeof(V) == 8 ? 7 : 4) * nz;
    for (int c = 0; c < 3; ++c) { a.out[c] = F[c]; a.in[c] = PRE[c]; }
    for (int c = 0; c < ncomp; ++c) a.comp[c] = comps[c];
    return line_launch<0, V>(h, q, a, ncomp);
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
        a.cb = (C + h->ssor_nib - 1) / h->ssor_nib * (ch / q.E);
    }
    return bwd ? line_launch<2, V>(h, q, a, 1) : line_launch<1, V>(h, q, a, 1);
}

// The exchange buffer holds no row between launches.
int line_selftest(tbl_handle* h, int which) {
    if (which < 0 || which > 2 || !h->line_xch) return TBL_ERR_BAD_ARG;
    if (h->cfg.precision == TBL_PREC_MIXED) k_line_wait<float><<<1, 32, 0, h->stream>>>(which, (float*)h->line_xch, h->err);
    else k_line_wait<double><<<1, 32, 0, h->stream>>>(which, (double*)h->line_xch, h->err);
    TBL_CUDA_TRY(cudaGetLastError());
    h->launches++;
    return TBL_OK;
}

template int launch_line_gs<double>(tbl_handle*, double* const[3], double* const[3], const int*, int);
template int launch_line_gs<float>(tbl_handle*, float* const[3], float* const[3], const int*, int);
template int launch_line_ssor<double>(tbl_handle*, bool, const double*, double*, const int*);
template int launch_line_ssor<float>(tbl_handle*, bool, const float*, float*, const int*);

}  // namespace tbl
