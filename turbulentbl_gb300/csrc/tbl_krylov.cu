// tbl_krylov.cu -- GMRES(kmax) building blocks in FP64
// (dnstbl2/dnstbl.f90:952-1208): modified Gram-Schmidt passes over blocks of
// basis vectors with fused grid reductions, Givens rotations and back
// substitution in one warp, and the solution update p' += V y.
//
// Vector kernels stream the whole padded volume: Krylov vectors are zero
// outside the interior, so boundary and padding entries add nothing to the dot
// products and stay zero under the updates.
#include "tbl_internal.cuh"
#include "tbl_reduce.cuh"
#include "tbl_kernels.cuh"
#include "tbl_sync.cuh"

namespace tbl {

// Grid of the streaming reductions: one resident wave (8 blocks of 256 threads
// per SM), so no partial second wave idles part of the GPU at the tail.
int red_blocks(tbl_handle* h) {
    long long n2 = h->g.vol / 2;
    long long b = (n2 + RED_THREADS * 4 - 1) / (RED_THREADS * 4);
    const long long wave = 8LL * (h->n_sm > 0 ? h->n_sm : 148);
    if (b > wave) b = wave;
    if (b > h->red.max_blocks) b = h->red.max_blocks;
    if (b < 1) b = 1;
    return (int)b;
}

// sum(a*b) over the volume -> *out (op 1: sqrt)
__global__ void __launch_bounds__(RED_THREADS, 8) k_dot(long long n2, const double2* __restrict__ a,
                                                     const double2* __restrict__ b, RedWork rw, int slot,
                                                     double* out, int op) {
    __shared__ double s_red[RED_THREADS / 32];
    double acc = 0.0;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n2; q += (long long)gridDim.x * blockDim.x) {
        double2 x = a[q], y = b[q];
        acc += x.x * y.x;
        acc += x.y * y.y;
    }
    double bt = block_sum(acc, s_red);
    grid_finish(bt, rw, slot, gridDim.x, blockIdx.x, out, op);
}

// L2 eviction-priority policy for data that should stay in L2 across
// kernels (evict-last), and 16-byte loads and stores under it.
__device__ __forceinline__ unsigned long long l2_keep_policy() {
    unsigned long long p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ double2 ld_keep(const double2* a, unsigned long long pol) {
    double2 v;
    asm volatile("ld.global.L2::cache_hint.v2.f64 {%0, %1}, [%2], %3;" : "=d"(v.x), "=d"(v.y) : "l"(a), "l"(pol));
    return v;
}
__device__ __forceinline__ void st_keep(double2* a, double2 v, unsigned long long pol) {
    asm volatile("st.global.L2::cache_hint.v2.f64 [%0], {%1, %2}, %3;" ::"l"(a), "d"(v.x), "d"(v.y), "l"(pol)
                 : "memory");
}

// Warp sums of N FP64 values per lane (N = 16, 8 or 1), as a reduce-scatter:
// at each of the offsets 16, 8, .. a lane keeps half of its values, sends the
// other half to lane ^ offset and adds what it receives; when one is left the
// remaining offsets complete it.  Lane l then holds the warp total of value
// l / (32 / N): 16 FP64 additions per lane for 16 values instead of the 80 of 16
// shuffle trees (FP64 runs at 1/64 of the FP32 rate on this GPU).  Fixed order:
// deterministic.
template <int N>
__device__ __forceinline__ double warp_reduce_scatter(double (&a)[N]) {
    const int lane = threadIdx.x & 31;
    int off = 16;
#pragma unroll
    for (int half = N / 2; half >= 1; half >>= 1, off >>= 1) {
        const bool up = (lane & off) != 0;  // keeps the upper half of the current values
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const double keep = up ? a[i + half] : a[i];
            const double send = up ? a[i] : a[i + half];
            a[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
    }
#pragma unroll
    for (int o = 32 / (2 * N); o >= 1; o >>= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
    return a[0];
}

// The last block to publish its partials, known to all its threads; what the
// blocks wrote before is visible to it.
__device__ __forceinline__ bool last_arrival(unsigned* count, unsigned total, bool* s_last) {
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned t;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(t) : "l"(count) : "memory");
        *s_last = t == total - 1;
    }
    __syncthreads();
    return *s_last;
}

// Block partials of N consecutive values, in a fixed order, by one warp: lanes
// strided over the blocks.  Lane l has the total of value l / (32 / N).
template <int N>
__device__ __forceinline__ double sum_partials(const double* p, int max_blocks, int nb) {
    double t[N];
#pragma unroll
    for (int e = 0; e < N; ++e) t[e] = 0.0;
#pragma unroll 4
    for (int q = threadIdx.x & 31; q < nb; q += 32)
#pragma unroll
        for (int e = 0; e < N; ++e) t[e] += __ldcg(p + (size_t)e * max_blocks + q);
    return warp_reduce_scatter<N>(t);
}

// Givens rotations for column kit (1-based) (:1165-1189) by one warp.  The
// rotations so far are a chain, cur = s_i cur + c_i h_{i+1}, of one FMA each
// when the lanes have formed c_i h_{i+1} before (an FP64 instruction of one
// thread takes as long as one of a warp: four of them a rotation, 5 us at 40
// rotations); the quotients are one division on three lanes.  The global loads
// of the first 32 rotations are made before the sums that last waits for.
struct Givens {
    int kit;
    double *H, *gg, *gc, *gs;  // H: the column, its first kit values set
    DevScalars* sc;
    bool ahead;  // Arnoldi steps enqueued ahead: the cycle stops when the estimate sumav
    double stop_at;  // reaches stop_at (the host's loop test, evaluated on the same double)
    double h0, nx, c, s, gk, gkp, sumnor;
    __device__ __forceinline__ void load(int base) {
        const int i = base + (threadIdx.x & 31);
        const bool on = i < kit - 1;
        nx = on ? H[i + 1] : 0.0;
        c = on ? gc[i] : 0.0;
        s = on ? gs[i] : 0.0;
    }
    __device__ __forceinline__ void prefetch() {
        load(0);
        h0 = H[0];
        gk = gg[kit - 1];
        gkp = gg[kit];
        sumnor = sc->sumnor;
    }
    // last: the subdiagonal value; returns 1 / rec
    __device__ __forceinline__ double column(double last, double rec) {
        const int lane = threadIdx.x & 31;
        double cur = h0;
        for (int base = 0; base < kit - 1; base += 32) {
            if (base > 0) load(base);
            const int n = min(32, kit - 1 - base);
            const double p = c * nx, q = s * nx;
            double mine = 0.0;
#pragma unroll 4
            for (int t = 0; t < n; ++t) {
                if (lane == t) mine = cur;
                cur = fma(__shfl_sync(0xffffffffu, s, t), cur, __shfl_sync(0xffffffffu, p, t));
            }
            if (lane < n) H[base + lane] = fma(c, mine, -q);
        }
        const double nu = sqrt(cur * cur + last * last);
        const double quot = (lane == 0 ? cur : lane == 1 ? -last : 1.0) / (lane < 2 ? nu : rec);
        const double cn = __shfl_sync(0xffffffffu, quot, 0), sn = __shfl_sync(0xffffffffu, quot, 1);
        double diag = cur, sub = last, a = gk, b = gkp;
        if (nu > 0.0) {
            diag = cn * cur - sn * last;
            sub = 0.0;
            a = cn * gk - sn * gkp;
            b = sn * gk + cn * gkp;
        }
        const double rho = fabs(b), sumav = rho / sumnor;
        if (lane == 0) {
            if (nu > 0.0) {
                gc[kit - 1] = cn;
                gs[kit - 1] = sn;
                gg[kit - 1] = a;
                gg[kit] = b;
            }
            H[kit - 1] = diag;
            H[kit] = sub;
            sc->rho = rho;
            sc->sumav = sumav;
            if (ahead && !(sumav > stop_at)) sc->stop = 1;
        }
        return __shfl_sync(0xffffffffu, quot, 2);
    }
};

// What the FP64 Gram-Schmidt keeps of a basis vector's norm: d = 1/|v|, and with
// p the power of two of 1 <= p |v| < 2 (exact scalings), ds = d / p, ns = p |v|, p.
struct GsNorms {
    double *d, *ds, *ns, *p;
    __device__ __forceinline__ void set(int i, double norm, double rec) const {  // rec = 1 / norm
        if (!(norm > 0.0)) norm = rec = 1.0;
        const int e = min(max((__double2hiint(norm) >> 20) & 0x7ff, 1), 2045);  // norm = m 2^(e - 1023)
        const double up = __hiloint2double((2046 - e) << 20, 0), down = __hiloint2double(e << 20, 0);
        d[i] = rec;
        ds[i] = rec * down;
        ns[i] = norm * up;
        p[i] = up;
    }
};

// ---------------------------------------------------- Gram-Schmidt (FP64)
// Modified Gram-Schmidt (:1140-1161) over blocks of 8 basis vectors.  One pass
// takes a block's projections off w and forms the next block's dot products:
//   w -= sum_i (h_i d_i p_k / d_k) v_i   (i in the previous block)
//   S_i = <v_i, w>                   (i in the next block), or <w, w> at the end
// Inside a block the dots are all taken against the same w; the modified
// Gram-Schmidt coefficients follow from h_i = c_i - sum_{j<i} <v_i, v_j> h_j,
// the products of a block's vectors being formed once, with the pass in which
// their last one is the newest (the product of the block's projections, also
// when the basis has lost orthogonality).
// The basis vectors are kept as they come out of this, not divided by their
// norms: v_i d_i with d_i = 1 / |v_i| is the reference's unit vector, and w =
// p_k M^-1 A v_k with p_k the power of two that brings |v_k| between 1 and 2, so
// c_i = d_i (d_k / p_k) S_i.  The division pass is gone.  The powers of two change
// no bit of the result; without them |v_k| is the product of the subdiagonal
// values, about 0.3 each, and its square is zero after some 300 vectors.
//
// Bound: two FP64 FMAs per element and basis vector (28.8 us a vector at
// 512 x 130 x 128 and 600 G FMA/s) and two reads of every basis vector (20 us
// at 6.8 TB/s): 33.4 us a vector at 40 vectors, 43.6 with one pass per vector.
// On small grids the number of launches, a ninth as many, and what a pass does
// besides, about 10 us: 145 us at 40 vectors and 128 x 66 x 64, of which 74 are
// FP64 issue.
constexpr int GSB = 8;
struct GsPass {
    long long n2;
    double2* w;
    const double2* V;      // basis, n2 apart
    int p0, q0;            // first vector of the previous and of the next block
    int k;                 // vectors in the basis
    GsNorms n;
    double* G;             // <v_i, v_j> / (|v_i| |v_j|), j in i's block, [i][GSB]
    double *hcol, *hs;     // Hessenberg column; h_i d_i p_k / d_k
    double* partial;       // [16][max_blocks]
    unsigned* count;
    int max_blocks;
    int K1;
    double *h, *gg, *gc, *gs;
    DevScalars* sc;
    const int* skip;
    double stop_at;
};

// NP, NQ: vectors of the two blocks (0: none).  GRAM: the next block holds the
// newest vector (its last).
template <int NP, int NQ, bool GRAM>
__global__ void __launch_bounds__(RED_THREADS, 2) k_gs_pass(const GsPass a) {
    dependent_wait();
    if (a.skip && *a.skip) return;  // an Arnoldi step enqueued ahead of a converged one
    constexpr int NW = RED_THREADS / 32;
    constexpr int NV = NQ == 0 ? 1 : GRAM && NQ > 1 ? 16 : 8;  // sums of the pass
    __shared__ double s_red[16 * NW];
    __shared__ double s_val[16];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned long long keep = l2_keep_policy();
    double hp[NP > 0 ? NP : 1];
#pragma unroll
    for (int e = 0; e < NP; ++e) hp[e] = a.hs[a.p0 + e];
    double acc[NV];
#pragma unroll
    for (int e = 0; e < NV; ++e) acc[e] = 0.0;
    const long long st = (long long)gridDim.x * blockDim.x;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < a.n2; q += st) {
        double2 x = ld_keep(a.w + q, keep);
        double2 v[NP > 0 ? NP : 1], y[NQ > 0 ? NQ : 1];
#pragma unroll
        for (int e = 0; e < NP; ++e) v[e] = __ldcs(a.V + (long long)(a.p0 + e) * a.n2 + q);
#pragma unroll
        for (int e = 0; e < NQ; ++e) y[e] = __ldcs(a.V + (long long)(a.q0 + e) * a.n2 + q);
#pragma unroll
        for (int e = 0; e < NP; ++e) {
            x.x = fma(-hp[e], v[e].x, x.x);
            x.y = fma(-hp[e], v[e].y, x.y);
        }
        if (NP > 0) st_keep(a.w + q, x, keep);
#pragma unroll
        for (int e = 0; e < NQ; ++e) acc[e] = fma(y[e].y, x.y, fma(y[e].x, x.x, acc[e]));
        if (NV == 16)
#pragma unroll
            for (int e = 0; e < NQ - 1; ++e)
                acc[8 + e] = fma(y[e].y, y[NQ - 1].y, fma(y[e].x, y[NQ - 1].x, acc[8 + e]));
        if (NQ == 0) acc[0] = fma(x.y, x.y, fma(x.x, x.x, acc[0]));
    }
    const double tot = warp_reduce_scatter<NV>(acc);  // value lane / (32 / NV)
    if (lane % (32 / NV) == 0) s_red[lane / (32 / NV) * NW + wid] = tot;
    __syncthreads();
    if (threadIdx.x < (NV * NW > 32 ? NV * NW : 32)) {
        double t = s_red[threadIdx.x];
#pragma unroll
        for (int o = NW / 2; o >= 1; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (threadIdx.x % NW == 0 && threadIdx.x / NW < NV)
            a.partial[(size_t)(threadIdx.x / NW) * a.max_blocks + blockIdx.x] = t;
    }
    if (!last_arrival(a.count, gridDim.x, &s_last)) return;
    // the last block: what the solve or the rotations need, fetched while the
    // other warps sum the partials, two values a warp
    const int i = a.q0 + lane;
    double di = 0.0, dk = 0.0, nk = 0.0, grow[GSB];
    Givens gv = {a.k, a.h + (size_t)a.K1 * (a.k - 1), a.gg, a.gc, a.gs, a.sc, a.skip != nullptr, a.stop_at};
    if (wid == 0) {
        dk = a.n.ds[a.k - 1];
        nk = a.n.ns[a.k - 1];
        if (NQ == 0) {
            gv.prefetch();
        } else {
            di = lane < NQ ? a.n.d[i] : 0.0;
#pragma unroll
            for (int j = 0; j < GSB - 1; ++j)  // this lane's row of the block's products
                grow[j] = lane < NQ - GRAM && j < lane ? a.G[(size_t)i * GSB + j] : 0.0;
        }
    }
    if (NV == 1) {
        if (wid == 0) {
            const double t = sum_partials<1>(a.partial, a.max_blocks, gridDim.x);
            if (lane == 0) s_val[0] = t;
        }
        __syncwarp();
    } else {
        if (2 * wid < NV) {
            const double t = sum_partials<2>(a.partial + (size_t)(2 * wid) * a.max_blocks, a.max_blocks, gridDim.x);
            if (lane % 16 == 0) s_val[2 * wid + lane / 16] = t;
        }
        __syncthreads();
    }
    if (wid != 0) return;
    if (NQ != 0) {
        double c = lane < NQ ? di * dk * s_val[lane] : 0.0;
        if (GRAM && NQ > 1) {
#pragma unroll
            for (int j = 0; j < NQ - 1; ++j) {
                const double dj = __shfl_sync(0xffffffffu, di, j);
                if (lane == NQ - 1) {
                    grow[j] = dj * di * s_val[8 + j];
                    a.G[(size_t)i * GSB + j] = grow[j];
                }
            }
        }
#pragma unroll
        for (int j = 0; j < GSB - 1; ++j) c = fma(-grow[j], __shfl_sync(0xffffffffu, c, j), c);
        if (lane < NQ) {
            a.hcol[i] = c;
            a.hs[i] = c * di * nk;
        }
    } else {
        const double nh = sqrt(s_val[0]);
        const double r = gv.column(dk * nh, nh);
        if (lane == 0) a.n.set(a.k, nh, r);
    }
    if (lane == 0) *a.count = 0u;
}

// Start of a restart (:958-963, :1048-1056): zero h, c, s, g, y; g(1) = rho;
// sumnor at the first restart; sumav = rho/sumnor.
// n: what is kept of the norms of basis vectors kept as they come (FP64), or nulls.
__global__ void k_restart_init(int K1, double* h, double* gg, double* gc, double* gs, double* gy, DevScalars* sc,
                               int first, GsNorms n) {
    for (int q = threadIdx.x; q < K1 * K1; q += blockDim.x) h[q] = 0.0;
    for (int q = threadIdx.x; q < K1; q += blockDim.x) { gg[q] = 0.0; gc[q] = 0.0; gs[q] = 0.0; gy[q] = 0.0; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double rho = sc->rho;
        sc->stop = 0;
        if (first) sc->sumnor = rho;
        sc->sumav = rho / sc->sumnor;
        gg[0] = rho;
        if (n.d) n.set(0, rho, 1.0 / rho);
    }
}

// y from the triangular h (:1193-1200), 32 columns at a time: one warp solves
// the triangle in registers, then all threads take the 32 columns off the rows
// above.  A column at a time through global memory took 54 us at 36 columns.  The
// chain multiplies by the reciprocal of the diagonal and corrects the quotient by its
// residual, which rounds as a division does: without the correction y is a seventh
// further off (1.7e-16 against 1.5e-16 of itself, mean over systems of 3 to 60
// columns), and a division is 1000 cycles a column.  With d the
// coefficients of the basis vectors as they are kept, y_i / |v_i|.
__global__ void __launch_bounds__(128) k_backsub(int K1, int kit, const double* h, double* gg, double* gy,
                                                 const double* d) {
    __shared__ double s_y[32];
    for (int base = (kit - 1) / 32 * 32; base >= 0; base -= 32) {
        const int n = min(32, kit - base);
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x, row = base + lane;
            double H[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) H[i] = i < n && lane <= i ? h[(size_t)K1 * (base + i) + row] : 0.0;
            double g = lane < n ? gg[row] : 0.0, diag = 1.0;
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (lane == i && i < n) diag = H[i];
            const double inv = 1.0 / diag;
#pragma unroll
            for (int i = 31; i >= 0; --i) {
                const double q = g * inv;
                const double y = __shfl_sync(0xffffffffu, fma(fma(-diag, q, g), inv, q), i);
                if (lane < i) g = fma(-H[i], y, g);
            }
            const double y = lane < n ? g / diag : 0.0;
            s_y[lane] = y;
            if (lane < n) gy[row] = d ? y * d[row] : y;
        }
        __syncthreads();
        for (int j = threadIdx.x; j < base; j += blockDim.x) {
            double g = gg[j];
            for (int i = 0; i < n; ++i) g = fma(-h[(size_t)K1 * (base + i) + j], s_y[i], g);
            gg[j] = g;
        }
        __syncthreads();
    }
}

// p' += sum_i v_i y_i, accumulated in the reference's order (:1202-1205)
__global__ void k_update(long long n2, double2* __restrict__ pc, const double2* __restrict__ V, long long vstride2,
                         const double* __restrict__ gy, int kit) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n2; q += (long long)gridDim.x * blockDim.x) {
        double2 x = pc[q];
#pragma unroll 4
        for (int i = 0; i < kit; ++i) {
            double2 v = V[(long long)i * vstride2 + q];
            double y = gy[i];
            x.x = x.x + v.x * y;
            x.y = x.y + v.y * y;
        }
        pc[q] = x;
    }
}

// ||L7 p' - Q8||^2 and ||Q8||^2 over the interior -> red[9], red[10]
__global__ void __launch_bounds__(RED_THREADS) k_ppe_resid(Geom g, double aw, double as, const double* __restrict__ Ab,
                                                           const double* __restrict__ At, const double* __restrict__ Ap,
                                                           const double* __restrict__ PC, const double* __restrict__ Q8,
                                                           RedWork rw, DevScalars* sc) {
    __shared__ double s_red[RED_THREADS / 32];
    const int ni = g.nx - 2, J = g.ny - 2, nk = g.nz - 2;
    const long long n = (long long)ni * J * nk;
    double num = 0.0, den = 0.0;
    for (long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; t0 < n; t0 += (long long)gridDim.x * blockDim.x) {
        int i = 1 + (int)(t0 % ni);
        long long r = t0 / ni;
        int j = 1 + (int)(r % J);
        int k = 1 + (int)(r / J);
        long long p = (long long)i + (long long)g.sx * ((long long)j + (long long)g.ny * k);
        int jm = j == 1 ? g.ny - 2 : j - 1, jp = j == g.ny - 2 ? 1 : j + 1;
        long long pjm = (long long)i + (long long)g.sx * ((long long)jm + (long long)g.ny * k);
        long long pjp = (long long)i + (long long)g.sx * ((long long)jp + (long long)g.ny * k);
        double lap = aw * PC[p - 1] + aw * PC[p + 1] + as * PC[pjm] + as * PC[pjp] + Ab[k] * PC[p - g.ps] +
                     At[k] * PC[p + g.ps] + Ap[k] * PC[p];
        double rr = lap - Q8[p];
        num += rr * rr;
        den += Q8[p] * Q8[p];
    }
    double b1 = block_sum(num, s_red);
    __syncthreads();
    double b2 = block_sum(den, s_red);
    grid_finish(b1, rw, 9, gridDim.x, blockIdx.x, &sc->red[9], 0);
    __syncthreads();
    grid_finish(b2, rw, 10, gridDim.x, blockIdx.x, &sc->red[10], 0);
}

// ------------------------------------------------ mixed precision (FP32)
// Inner GMRES vectors are FP32; dot products accumulate in FP64 (the FP32
// products of 4 consecutive elements are summed in FP32, then added in FP64),
// and h, g, c, s, y stay FP64 (k_restart_init / Givens / k_backsub above).

__device__ __forceinline__ double dot4(float4 a, float4 b) {
    return (double)fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)));
}

__global__ void __launch_bounds__(RED_THREADS, 8) k_dot_f(long long n4, const float4* __restrict__ a,
                                                       const float4* __restrict__ b, RedWork rw, int slot,
                                                       double* out, int op) {
    __shared__ double s_red[RED_THREADS / 32];
    double acc = 0.0;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += (long long)gridDim.x * blockDim.x)
        acc += dot4(a[q], b[q]);
    double bt = block_sum(acc, s_red);
    grid_finish(bt, rw, slot, gridDim.x, blockIdx.x, out, op);
}


__global__ void k_scale_inv_f(long long n4, float4* __restrict__ w, const double* __restrict__ denom,
                              const int* __restrict__ skip) {
    if (skip && *skip) return;
    const double d = *denom;
    if (!(d > 0.0 || d < 0.0)) return;
    const float r = (float)(1.0 / d);
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += (long long)gridDim.x * blockDim.x) {
        float4 x = w[q];
        x.x *= r; x.y *= r; x.z *= r; x.w *= r;
        w[q] = x;
    }
}

// p' (FP64) += sum_i y_i v_i: the FP32 correction of one inner cycle, added in FP64
__global__ void k_update_f(long long n4, double* __restrict__ pc, const float4* __restrict__ V, long long vstride4,
                           const double* __restrict__ gy, int kit) {
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < n4; q += (long long)gridDim.x * blockDim.x) {
        float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int i = 0; i < kit; ++i) {
            const float4 v = V[(long long)i * vstride4 + q];
            const float y = (float)gy[i];
            c.x = fmaf(y, v.x, c.x); c.y = fmaf(y, v.y, c.y); c.z = fmaf(y, v.z, c.z); c.w = fmaf(y, v.w, c.w);
        }
        double2* p2 = reinterpret_cast<double2*>(pc) + 2 * q;
        double2 x0 = p2[0], x1 = p2[1];
        x0.x += (double)c.x; x0.y += (double)c.y; x1.x += (double)c.z; x1.y += (double)c.w;
        p2[0] = x0;
        p2[1] = x1;
    }
}

// ------------------------------------------------------------- host glue
int launch_dot(tbl_handle* h, const double* a, const double* b, double* out, int op) {
    int nb = red_blocks(h);
    k_dot<<<nb, RED_THREADS, 0, h->stream>>>(h->g.vol / 2, (const double2*)a, (const double2*)b, h->red, 7, out, op);
    h->launches++;
    return TBL_OK;
}

// The pass that forms the dots of the last block, n vectors, and the pass that
// takes its projections off and forms the norm.
template <int NP>
static void (*gs_newest(int n))(const GsPass) {
    switch (n) {
        case 1: return k_gs_pass<NP, 1, true>;
        case 2: return k_gs_pass<NP, 2, true>;
        case 3: return k_gs_pass<NP, 3, true>;
        case 4: return k_gs_pass<NP, 4, true>;
        case 5: return k_gs_pass<NP, 5, true>;
        case 6: return k_gs_pass<NP, 6, true>;
        case 7: return k_gs_pass<NP, 7, true>;
        default: return k_gs_pass<NP, 8, true>;
    }
}
static void (*gs_last(int n))(const GsPass) {
    switch (n) {
        case 1: return k_gs_pass<1, 0, false>;
        case 2: return k_gs_pass<2, 0, false>;
        case 3: return k_gs_pass<3, 0, false>;
        case 4: return k_gs_pass<4, 0, false>;
        case 5: return k_gs_pass<5, 0, false>;
        case 6: return k_gs_pass<6, 0, false>;
        case 7: return k_gs_pass<7, 0, false>;
        default: return k_gs_pass<8, 0, false>;
    }
}

static GsNorms gs_norms(const tbl_handle* h) {
    const size_t n = (size_t)h->cfg.kmax + 1;
    return {h->gs_d, h->gs_d + n, h->gs_d + 2 * n, h->gs_d + 3 * n};
}

// The factor of step k's matvec (k >= 1).
const double* gs_factor(const tbl_handle* h, int k) { return gs_norms(h).p + (k - 1); }

// Orthogonalises w against the k vectors of the basis, then the Givens rotation
// of the column.
int launch_gs(tbl_handle* h, double* w, int k, const int* skip, double stop_at) {
    GsPass a = {};
    a.n2 = h->g.vol / 2;
    a.w = (double2*)w;
    a.V = (const double2*)h->V;
    a.k = k;
    a.K1 = h->cfg.kmax + 1;
    a.n = gs_norms(h);
    a.G = h->gs_G;
    a.hs = h->gs_hs;
    a.h = h->h;
    a.hcol = h->h + (size_t)a.K1 * (k - 1);
    a.gg = h->gg; a.gc = h->gc; a.gs = h->gs; a.sc = h->sc;
    a.partial = h->red.partial;
    a.count = h->red.count + 15;
    a.max_blocks = h->red.max_blocks;
    a.skip = skip;
    a.stop_at = stop_at;
    long long nb = (a.n2 + RED_THREADS - 1) / RED_THREADS;
    const long long wave = 2LL * (h->n_sm > 0 ? h->n_sm : 148);
    if (nb > wave) nb = wave;
    const int nblk = (k + GSB - 1) / GSB, rest = k - (nblk - 1) * GSB;  // vectors of the last block
    for (int b = 0; b <= nblk; ++b) {
        a.p0 = (b - 1) * GSB;
        a.q0 = b * GSB;
        void (*fn)(const GsPass) = b == nblk        ? gs_last(rest)
                                   : b == nblk - 1 ? (b == 0 ? gs_newest<0>(rest) : gs_newest<GSB>(rest))
                                   : b == 0        ? k_gs_pass<0, GSB, false>
                                                   : k_gs_pass<GSB, GSB, false>;
        TBL_CUDA_TRY(launch_dependent(fn, dim3((unsigned)nb), dim3(RED_THREADS), 0, h->stream, a));
        h->launches++;
    }
    return TBL_OK;
}

int launch_restart_init(tbl_handle* h, int first) {
    const int K1 = h->cfg.kmax + 1;
    k_restart_init<<<1, 256, 0, h->stream>>>(K1, h->h, h->gg, h->gc, h->gs, h->gy, h->sc, first, gs_norms(h));
    h->launches++;
    return TBL_OK;
}

int launch_backsub_update(tbl_handle* h, int kit) {
    const int K1 = h->cfg.kmax + 1;
    k_backsub<<<1, 128, 0, h->stream>>>(K1, kit, h->h, h->gg, h->gy, h->gs_d);
    int nb = red_blocks(h);
    k_update<<<nb, RED_THREADS, 0, h->stream>>>(h->g.vol / 2, (double2*)h->PC, (const double2*)h->V, h->g.vol / 2,
                                                h->gy, kit);
    h->launches += 2;
    return TBL_OK;
}

// ------------------------- low-synchronisation Gram-Schmidt (FP32 inner GMRES)
// Modified Gram-Schmidt in its inverse compact-WY form: for a basis
// Q = [v_0 .. v_{n-1}] with L the strictly lower triangle of Q^T Q, the product
// of the n MGS projections is I - Q (I + L)^-1 Q^T (exactly, also when Q has
// lost orthogonality).  One pass forms Q^T w and the new row of L
// (Q^T v_{n-1}); a forward substitution gives the Hessenberg column t; a
// second pass applies w -= Q t and forms ||w||.  2n+3 vector passes per
// Arnoldi step instead of MGS's 4n+1; the FP64 outer refinement of the mixed
// solve makes the different rounding irrelevant to the final accuracy.
constexpr int LSG_G = 8;  // basis vectors per group (grid.y) of the dot pass

__device__ __forceinline__ float dot4f(float4 a, float4 b) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)));
}
// The pass's share of G basis vectors: S_e = <v_e, w>, T_e = <v_e, l> with l the
// newest basis vector, interleaved in acc.  The products are FP32 (the vectors
// are); each thread sums its share (about 16 float4 loads, 64 products) in FP32,
// and from these per-thread partials on every sum is FP64.  An FP64 sum per
// float4 instead cost the mixed step 14 ms at 512 x 130 x 128 (22% of its
// Gram-Schmidt time).
template <int G>
__device__ __forceinline__ void lsg_dots(long long n4, const float4* __restrict__ w, const float4* __restrict__ l,
                                         const float4* __restrict__ V, long long vstride4, double (&acc)[16]) {
#pragma unroll
    for (int e = 0; e < 16; ++e) acc[e] = 0.0;
    const long long stride = (long long)gridDim.y * blockDim.x;
    for (long long q = (long long)blockIdx.y * blockDim.x + threadIdx.x; q < n4;) {
        float fd[G], fg[G];
#pragma unroll
        for (int e = 0; e < G; ++e) { fd[e] = 0.f; fg[e] = 0.f; }
        for (int n = 0; n < 16 && q < n4; ++n, q += stride) {
            const float4 x = w[q], y = l[q];
            float4 v[G];
#pragma unroll
            for (int e = 0; e < G; ++e) v[e] = __ldcs(V + (long long)e * vstride4 + q);  // read once: evict first
#pragma unroll
            for (int e = 0; e < G; ++e) {
                fd[e] += dot4f(v[e], x);
                fg[e] += dot4f(v[e], y);
            }
        }
#pragma unroll
        for (int e = 0; e < G; ++e) {
            acc[2 * e] += (double)fd[e];
            acc[2 * e + 1] += (double)fg[e];
        }
    }
}

struct LsgArgs {
    long long n4;
    float4* w;
    const float4* V;  // basis, n4 apart
    int nv;           // its vectors
    double* partial;  // [16 per group][max_blocks]
    unsigned* count;  // [0] groups done, [1 + group] blocks done
    int max_blocks;
    int K1;
    double *L, *hcol;  // strictly lower triangle of the basis' products; Hessenberg column
    double *h, *gg, *gc, *gs;
    DevScalars* sc;
    const int* skip;
    double stop_at;
};

// d = Q^T w and the newest row of L, the basis in groups of at most LSG_G
// vectors, one per blockIdx.x (the groups of a stretch of w run together and
// share it in L2: 275 -> 263 us at 40 vectors, 512 x 130 x 128).  The last block
// of a group sums its block partials, the last group solves (I + L) t = d for
// the Hessenberg column: a forward substitution in one warp's registers, L
// fetched into shared memory while the sums are formed.
__global__ void __launch_bounds__(RED_THREADS, 2) k_lsg_dots_f(const LsgArgs a) {
    dependent_wait();
    if (a.skip && *a.skip) return;
    constexpr int NW = RED_THREADS / 32;
    __shared__ double s_red[16 * NW];
    extern __shared__ double sL[];  // nv columns of nv (odd) values
    __shared__ bool s_last;
    const int nv = a.nv, ngr = gridDim.x, grp = blockIdx.x;
    const int i0 = grp * nv / ngr, G = (grp + 1) * nv / ngr - i0;
    const float4 *l = a.V + (long long)(nv - 1) * a.n4, *V = a.V + (long long)i0 * a.n4;
    double acc[16];
    switch (G) {
        case 1: lsg_dots<1>(a.n4, a.w, l, V, a.n4, acc); break;
        case 2: lsg_dots<2>(a.n4, a.w, l, V, a.n4, acc); break;
        case 3: lsg_dots<3>(a.n4, a.w, l, V, a.n4, acc); break;
        case 4: lsg_dots<4>(a.n4, a.w, l, V, a.n4, acc); break;
        case 5: lsg_dots<5>(a.n4, a.w, l, V, a.n4, acc); break;
        case 6: lsg_dots<6>(a.n4, a.w, l, V, a.n4, acc); break;
        case 7: lsg_dots<7>(a.n4, a.w, l, V, a.n4, acc); break;
        default: lsg_dots<8>(a.n4, a.w, l, V, a.n4, acc); break;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const double tot = warp_reduce_scatter<16>(acc);  // value lane >> 1
    if ((lane & 1) == 0) s_red[(lane >> 1) * NW + wid] = tot;
    __syncthreads();
    double* const part = a.partial + (size_t)grp * 16 * a.max_blocks;
    if (threadIdx.x < 16 * NW) {
        double t = s_red[threadIdx.x];
#pragma unroll
        for (int o = NW / 2; o >= 1; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (threadIdx.x % NW == 0) part[(size_t)(threadIdx.x / NW) * a.max_blocks + blockIdx.y] = t;
    }
    if (!last_arrival(a.count + 1 + grp, gridDim.y, &s_last)) return;
    const int r = nv - 1, ld = nv | 1;
    for (int q = threadIdx.x; q < nv * nv; q += blockDim.x) {  // L's older rows, zeros elsewhere
        const int row = q / nv, col = q % nv;
        const unsigned dst = (unsigned)__cvta_generic_to_shared(sL + col * ld + row);
        if (col < row && row < r)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(a.L + (size_t)row * a.K1 + col) : "memory");
        else
            sL[col * ld + row] = 0.0;
    }
    if (wid < G) {  // <v, w> on lane 0, <v, l> on lane 16
        const double t = sum_partials<2>(part + (size_t)(2 * wid) * a.max_blocks, a.max_blocks, gridDim.y);
        const int i = i0 + wid;
        if (lane == 0) a.hcol[i] = t;
        if (lane == 16 && i < r) a.L[(size_t)r * a.K1 + i] = t;
    }
    if (threadIdx.x == 0) a.count[1 + grp] = 0u;
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (!last_arrival(a.count, ngr, &s_last) || wid != 0) return;
    // rows lane and lane + 32 (nv <= 63); the newest row's products straight from memory
    double t0 = lane < nv ? __ldcg(a.hcol + lane) : 0.0, t1 = 32 + lane < nv ? __ldcg(a.hcol + 32 + lane) : 0.0;
    for (int j = lane; j < r; j += 32) sL[j * ld + r] = __ldcg(a.L + (size_t)r * a.K1 + j);
    __syncwarp();
    if (nv <= 32) {
#pragma unroll 4
        for (int j = 0; j < r; ++j) t0 = fma(-(lane < nv ? sL[j * ld + lane] : 0.0), __shfl_sync(0xffffffffu, t0, j), t0);
    } else {
#pragma unroll 4
        for (int j = 0; j < r; ++j) {
            const double tj = __shfl_sync(0xffffffffu, j < 32 ? t0 : t1, j & 31);
            t0 = fma(-sL[j * ld + lane], tj, t0);
            t1 = fma(-(32 + lane < nv ? sL[j * ld + 32 + lane] : 0.0), tj, t1);
        }
    }
    if (lane < nv) a.hcol[lane] = t0;
    if (32 + lane < nv) a.hcol[32 + lane] = t1;
    if (lane == 0) *a.count = 0u;
}

// w -= sum_i t_i v_i (FP32), eight vectors' loads in flight per thread (four,
// with six blocks per SM: 249 -> 217 us at 40 vectors, 512 x 130 x 128, 35 -> 27
// at 128 x 66 x 64), then in the last block ||w|| (sqrt of the deterministic
// sum) and the column's Givens rotation.
__global__ void __launch_bounds__(RED_THREADS, 4) k_lsg_update_f(const LsgArgs a, RedWork rw, int slot) {
    dependent_wait();
    if (a.skip && *a.skip) return;
    __shared__ double s_red[RED_THREADS / 32];
    __shared__ float s_t[64];
    __shared__ bool s_last;
    const int nv = a.nv;
    if (threadIdx.x < 64) s_t[threadIdx.x] = threadIdx.x < nv ? (float)a.hcol[threadIdx.x] : 0.f;
    __syncthreads();
    double acc = 0.0;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < a.n4;
         q += (long long)gridDim.x * blockDim.x) {
        float4 x = a.w[q];
        for (int i = 0; i < nv; i += 8) {
            float4 v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e)  // read once: evict first
                v[e] = i + e < nv ? __ldcs(a.V + (long long)(i + e) * a.n4 + q) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float ti = s_t[i + e];
                x.x = fmaf(-ti, v[e].x, x.x);
                x.y = fmaf(-ti, v[e].y, x.y);
                x.z = fmaf(-ti, v[e].z, x.z);
                x.w = fmaf(-ti, v[e].w, x.w);
            }
        }
        a.w[q] = x;
        acc += (double)dot4f(x, x);
    }
    const double bt = block_sum(acc, s_red);
    if (threadIdx.x == 0) rw.partial[(size_t)slot * rw.max_blocks + blockIdx.x] = bt;
    if (!last_arrival(rw.count + slot, gridDim.x, &s_last)) return;
    Givens gv = {nv, a.hcol, a.gg, a.gc, a.gs, a.sc, a.skip != nullptr, a.stop_at};
    if (threadIdx.x < 32) gv.prefetch();
    double t = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) t += __ldcg(rw.partial + (size_t)slot * rw.max_blocks + b);
    t = block_sum(t, s_red);
    if (threadIdx.x >= 32) return;
    const double nrm = sqrt(__shfl_sync(0xffffffffu, t, 0));
    gv.column(nrm, 1.0);
    if (threadIdx.x == 0) {
        a.sc->red[8] = nrm;  // the next step's matvec divides by it
        rw.count[slot] = 0u;
    }
}

// Orthogonalises W against the kit <= 63 vectors of the FP32 basis, then the
// Givens rotation of the column.
int launch_lsg_f(tbl_handle* h, float* W, int kit, const int* skip, double stop_at) {
    LsgArgs a = {};
    a.K1 = h->cfg.mixed_kmax + 1;
    if (kit > 63 || kit > a.K1) return TBL_ERR_BAD_ARG;
    a.n4 = h->g.vol / 4;
    a.w = (float4*)W;
    a.V = (const float4*)h->Vf;
    a.nv = kit;
    a.partial = h->lsg_partial;
    a.count = h->red.count + 15;  // and one for each of at most 8 groups
    a.max_blocks = h->red.max_blocks;
    a.L = h->lsg_L;
    a.hcol = h->h + (size_t)a.K1 * (kit - 1);
    a.gg = h->gg; a.gc = h->gc; a.gs = h->gs; a.sc = h->sc;
    a.skip = skip;
    a.stop_at = stop_at;
    // one resident wave over all groups: two blocks per SM, one where a block
    // has at most 8 rounds, which then count less than the partials to be summed
    // (14.4 -> 11.3 us at 4 vectors, 128 x 66 x 64; 48 -> 59 at 20, 333 x 99 x 85)
    const int ngr = (kit + LSG_G - 1) / LSG_G, sms = h->n_sm > 0 ? h->n_sm : 148;
    const long long one = (a.n4 + RED_THREADS - 1) / RED_THREADS;  // one float4 per thread
    long long nbd = (one * ngr <= 8LL * sms ? 1LL : 2LL) * sms / ngr;
    if (nbd > one) nbd = one;
    if (nbd > h->red.max_blocks) nbd = h->red.max_blocks;
    if (nbd < 1) nbd = 1;
    TBL_CUDA_TRY(launch_dependent(k_lsg_dots_f, dim3(ngr, (unsigned)nbd), dim3(RED_THREADS),
                                  (size_t)kit * (kit | 1) * sizeof(double), h->stream, a));
    long long nbu = 4LL * sms;  // one resident wave at 4 blocks per SM
    if (nbu > one) nbu = one;
    TBL_CUDA_TRY(launch_dependent(k_lsg_update_f, dim3((unsigned)nbu), dim3(RED_THREADS), 0, h->stream, a, h->red, 7));
    h->launches += 2;
    return TBL_OK;
}

int launch_dot_f(tbl_handle* h, const float* a, const float* b, double* out, int op) {
    int nb = red_blocks(h);
    k_dot_f<<<nb, RED_THREADS, 0, h->stream>>>(h->g.vol / 4, (const float4*)a, (const float4*)b, h->red, 7, out, op);
    h->launches++;
    return TBL_OK;
}

int launch_scale_by_inv_f(tbl_handle* h, float* w, const double* denom, const int* skip) {
    int nb = red_blocks(h);
    k_scale_inv_f<<<nb, RED_THREADS, 0, h->stream>>>(h->g.vol / 4, (float4*)w, denom, skip);
    h->launches++;
    return TBL_OK;
}

int launch_backsub_update_f(tbl_handle* h, int kit) {
    const int K1 = h->cfg.mixed_kmax + 1;
    k_backsub<<<1, 128, 0, h->stream>>>(K1, kit, h->h, h->gg, h->gy, h->gs_d);
    int nb = red_blocks(h);
    k_update_f<<<nb, RED_THREADS, 0, h->stream>>>(h->g.vol / 4, h->PC, (const float4*)h->Vf, h->g.vol / 4, h->gy,
                                                  kit);
    h->launches += 2;
    return TBL_OK;
}

int launch_restart_init_k(tbl_handle* h, int first, int K1) {
    k_restart_init<<<1, 256, 0, h->stream>>>(K1, h->h, h->gg, h->gc, h->gs, h->gy, h->sc, first, GsNorms());
    h->launches++;
    return TBL_OK;
}

int launch_ppe_resid(tbl_handle* h) {
    int nb = red_blocks(h);
    k_ppe_resid<<<nb, RED_THREADS, 0, h->stream>>>(h->g, 1.0 / (h->cfg.dx * h->cfg.dx), 1.0 / (h->cfg.dy * h->cfg.dy),
                                                   h->Ab, h->At, h->Ap, h->PC, h->Q8, h->red, h->sc);
    h->launches++;
    return TBL_OK;
}

}  // namespace tbl
