// tbl_lap.cu -- the matvec in front of the SSOR sweeps, R = s(k) L7 X of an
// Arnoldi step or R = s(k) (Q8 - L7 X) of a restart (dnstbl2/dnstbl.f90:
// 995-1006, 1086-1101), with the sweeps' scale folded into the coefficients.
//
// A warp owns 32 x 16 bytes of points of a row and marches up a range of
// planes: the planes below, at and above a point stay in registers, the points
// beside it come by shuffle, the rows beside it from L1 (the block's other
// warps), so that every plane is read from L2 once per block of 8 rows.
//
// FP32 (the mixed solver's Arnoldi step): bound by memory and latency.  It also
// finishes the previous step: its input is that step's vector before the
// division by its norm, which it applies to every value it loads, and it writes
// the divided vector into the basis.  512 x 130 x 128: 50 -> 25 us (105 MB read
// and written) with TMA plane tiles in shared memory, whose barriers and
// scaling pass over each tile were the time, replaced by registers; the norm's
// reciprocal by one warp of a block, 21.5 -> 19.5 us (128 x 66 x 64: 4.7 -> 3.2).
// FP64: bound by FP64 issue, 7 operations a point (64 cycles a warp each); one
// thread per point with the scale as an eighth took 137 us, now 105 us.
#include <algorithm>

#include "tbl_internal.cuh"
#include "tbl_kernels.cuh"
#include "tbl_sync.cuh"

namespace tbl {

constexpr int LAP_ROWS = 8;   // span rows (warps) per block
constexpr int LAP_KC = 32;    // planes per block at most

// 16 bytes of values, converted to the arithmetic type
template <typename TC>
__device__ __forceinline__ void lap_load(TC (&v)[2], const double* p) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    v[0] = (TC)t.x;
    v[1] = (TC)t.y;
}
__device__ __forceinline__ void lap_load(float (&v)[4], const float* p) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void lap_store(double* p, const double (&v)[2]) {
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
}
__device__ __forceinline__ void lap_store(float* p, const float (&v)[2]) {
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}
__device__ __forceinline__ void lap_store(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

// RESID: Q8 - L7 X.  NORM: X is divided by *denom and written to vout.  factor
// multiplies the coefficients of L7 X.
template <typename TI, typename TO, typename TC, bool RESID, bool NORM>
__global__ void __launch_bounds__(32 * LAP_ROWS) k_lap(Geom g, double aw, double as, const double* __restrict__ Ab,
                                                       const double* __restrict__ At, const double* __restrict__ Ap,
                                                       const double* __restrict__ scale, int kc,
                                                       const TI* X, const double* Q8, TO* __restrict__ R,
                                                       const int* skip, const double* denom,
                                                       const double* factor, TI* __restrict__ vout) {
    constexpr int VEC = 16 / sizeof(TI);
    constexpr unsigned ALL = 0xffffffffu;
    __shared__ TC s_c[LAP_KC][6];  // s Ab, s At, s Ap, s aw, s as, s
    const int lane = threadIdx.x, k_lo = 1 + kc * blockIdx.z, k_hi = min(g.nz - 2, k_lo + kc - 1);
    for (int q = threadIdx.y * 32 + lane; q < 6 * kc; q += 32 * LAP_ROWS) {
        const int k = min(k_lo + q / 6, g.nz - 2), c = q % 6;
        const double s = scale[k];
        s_c[q / 6][c] = (TC)(s * (c == 0 ? Ab[k] : c == 1 ? At[k] : c == 2 ? Ap[k] : c == 3 ? aw : c == 4 ? as : 1.0));
    }
    dependent_wait(X);
    constexpr bool SCALED = sizeof(TI) == 8 && !RESID && !NORM;
    const int up = SCALED && factor ? __double2hiint(*factor) - 0x3ff00000 : 0;  // known when the skip word is
    if (skip && *skip) return;  // an Arnoldi step enqueued ahead of a converged one
    if (SCALED && factor)  // each thread its own entries; in the exponent, an FP64 product a warp costs 64 cycles
        for (int q = threadIdx.y * 32 + lane; q < 6 * kc; q += 32 * LAP_ROWS) {
            const double c = s_c[q / 6][q % 6];
            if (c != 0.0) s_c[q / 6][q % 6] = (TC)__hiloint2double(__double2hiint(c) + up, __double2loint(c));
        }
    __shared__ TC s_rs;
    if (NORM && threadIdx.y == LAP_ROWS - 1) {  // one warp: an FP64 division keeps its pipe for 1000 cycles
        const double d = *denom;
        const TC q = d > 0.0 || d < 0.0 ? (TC)(1.0 / d) : TC(1);
        if (lane == 0) s_rs = q;
    }
    __syncthreads();
    const int j = 1 + LAP_ROWS * blockIdx.y + threadIdx.y;
    if (j > g.ny - 2) return;
    const int jm = j == 1 ? g.ny - 2 : j - 1, jp = j == g.ny - 2 ? 1 : j + 1;
    const int first = VEC * (32 * blockIdx.x + lane);
    const int i0 = min(first, g.sx - VEC);  // lanes beyond the row load its end and store nothing
    unsigned okm = 0;
#pragma unroll
    for (int e = 0; e < VEC; ++e)
        if (first + e >= 1 && first + e <= g.nx - 2) okm |= 1u << e;
    const bool whole = okm == (1u << VEC) - 1;
    const TC rs = NORM ? s_rs : TC(1);
    auto load = [&](TC(&v)[VEC], const TI* p) {
        lap_load(v, p);
        if (NORM)
#pragma unroll
            for (int e = 0; e < VEC; ++e) v[e] *= rs;
    };
    const long long c0 = (long long)i0 + (long long)g.sx * ((long long)j + (long long)g.ny * k_lo);
    const TI* pc = X + c0;
    const long long djm = (long long)g.sx * (jm - j), djp = (long long)g.sx * (jp - j);
    TC zm[VEC], x[VEC];
    load(zm, pc - g.ps);
    load(x, pc);
    long long o = c0;
    for (int k = k_lo; k <= k_hi; ++k, pc += g.ps, o += g.ps) {
        TC zp[VEC], ym[VEC], yp[VEC];
        load(zp, pc + g.ps);
        load(ym, pc + djm);
        load(yp, pc + djp);
        TC xl = __shfl_up_sync(ALL, x[VEC - 1], 1), xr = __shfl_down_sync(ALL, x[0], 1);
        if (lane == 0) xl = i0 > 0 ? (TC)pc[-1] * rs : TC(0);
        if (lane == 31) xr = i0 + VEC < g.sx ? (TC)pc[VEC] * rs : TC(0);
        const TC* c = s_c[k - k_lo];
        TO r[VEC];
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
            TC t = c[2] * x[e];
            t = fma(c[3], e > 0 ? x[e > 0 ? e - 1 : 0] : xl, t);
            t = fma(c[3], e < VEC - 1 ? x[e < VEC - 1 ? e + 1 : e] : xr, t);
            t = fma(c[4], ym[e], t);
            t = fma(c[4], yp[e], t);
            t = fma(c[0], zm[e], t);
            t = fma(c[1], zp[e], t);
            if (RESID) t = fma(c[5], (TC)Q8[o + e], -t);
            r[e] = (TO)t;
        }
        if (whole) {
            lap_store(R + o, r);
            if (NORM) lap_store(vout + o, x);
        } else {
#pragma unroll
            for (int e = 0; e < VEC; ++e)
                if (okm >> e & 1u) {
                    R[o + e] = r[e];
                    if (NORM) vout[o + e] = (TI)x[e];
                }
        }
#pragma unroll
        for (int e = 0; e < VEC; ++e) {
            zm[e] = x[e];
            x[e] = zp[e];
        }
    }
}

template <typename TI, typename TO, typename TC>
static int lap(tbl_handle* h, const TI* X, const double* Q8, TO* R, const double* scale, const int* skip,
               const double* denom, const double* factor, TI* vout) {
    const Geom& g = h->g;
    const int vec = 16 / (int)sizeof(TI), planes = g.nz - 2;
    const unsigned gx = (unsigned)((g.nx - 2) / (32 * vec) + 1), gy = (unsigned)((g.ny - 2 + LAP_ROWS - 1) / LAP_ROWS);
    // Planes per block (each range reads two planes more than it writes).  FP32,
    // bound by latency: one wave of the 5 blocks an SM holds.  FP64, bound by the
    // FP64 pipes: 8 blocks per SM, which the SMs share evenly.  Small grids go
    // down to one plane: every SM busy counts for more than the reread planes
    // (32 x 18 x 24: 5 us a launch against 8 with 4 planes).
    const long long sms = h->n_sm > 0 ? h->n_sm : 148, tiles = (long long)gx * gy;
    const long long want = sizeof(TI) == 4 ? std::max(1LL, 5 * sms / tiles) : (8 * sms + tiles - 1) / tiles;
    const int kc = (int)std::min((long long)LAP_KC, (planes + want - 1) / want);
    const double aw = 1.0 / (h->cfg.dx * h->cfg.dx), as = 1.0 / (h->cfg.dy * h->cfg.dy);
    void (*fn)(Geom, double, double, const double*, const double*, const double*, const double*, int, const TI*,
               const double*, TO*, const int*, const double*, const double*, TI*);
    if constexpr (sizeof(TI) == 4) fn = denom ? k_lap<TI, TO, TC, false, true> : k_lap<TI, TO, TC, false, false>;
    else if constexpr (sizeof(TO) == 4) fn = k_lap<TI, TO, TC, true, false>;
    else fn = Q8 ? k_lap<TI, TO, TC, true, false> : k_lap<TI, TO, TC, false, false>;
    TBL_CUDA_TRY(launch_dependent(fn, dim3(gx, gy, (unsigned)((planes + kc - 1) / kc)), dim3(32, LAP_ROWS), 0, h->stream,
                                  g, aw, as, h->Ab, h->At, h->Ap, scale, kc, X, Q8, R, skip, denom, factor, vout));
    h->launches++;
    return TBL_OK;
}

int launch_lap(tbl_handle* h, const double* X, const double* Q8, double* R, const int* skip, const double* factor) {
    if (Q8 && factor) return TBL_ERR_BAD_ARG;
    return lap<double, double, double>(h, X, Q8, R, h->ssor_scale, skip, nullptr, factor, nullptr);
}
int launch_lap_f(tbl_handle* h, const float* X, float* R, const int* skip, const double* denom, float* vout) {
    if ((denom == nullptr) != (vout == nullptr) || (vout && vout == X)) return TBL_ERR_BAD_ARG;
    return lap<float, float, float>(h, X, nullptr, R, h->ssor_scale, skip, denom, nullptr, vout);
}
int launch_lap_resid_f(tbl_handle* h, const double* X, const double* Q8, float* R, const int* skip) {
    return lap<double, float, double>(h, X, Q8, R, h->ssor_scale, skip, nullptr, nullptr, nullptr);
}

}  // namespace tbl
