// tbl_gs.cu -- the parallel passes of the implicit diffusion's Gauss-Seidel
// iteration (1 + t L7) U = Q, t = -dt/Re (dnstbl2/dnstbl.f90:771-896): the L1
// norm of the residual, and the part of the next sweep that reads only values
// the sweep has not yet replaced when it gets there,
//   s   = Q - cE U(i+1) - cN U(j+1) - cT U(k+1)
//   PRE = (s - cN U(j-1) [first row] - cB U(k-1) [first plane of a slab]) / d
//   res = s - d U - cE U(i-1) - cN U(j-1) - cB U(k-1)
// where the last span row leaves U(j+1), the first row's new value, to the sweep,
// and PRE(i=0) is the inflow boundary value.  A check that lets the iteration go
// on has formed the next sweep's PRE on the way: one pass and 9 FP64 operations
// a point instead of two passes and 12.
//
// The access is the matvec's (tbl_lap.cu): a warp owns 32 x 16 bytes of points of
// a row and marches up the planes with the planes around it in registers.  FP64
// is bound by FP64 issue (64 cycles a warp and operation), FP32 by memory.
// 512 x 130 x 128, three components: check + PRE 525 -> 431 us in FP64 (9.5
// operations a point: 411 us at 600 G FMA/s), 220 -> 78 us in FP32; PRE alone
// 195 -> 188 and 103 -> 63 us.
#include <algorithm>

#include "tbl_internal.cuh"
#include "tbl_reduce.cuh"
#include "tbl_kernels.cuh"
#include "tbl_sync.cuh"

namespace tbl {

constexpr int GS_ROWS = 8;  // span rows (warps) per block
constexpr int GS_KC = 32;   // planes per tile at most

__device__ __forceinline__ void gs_load(double (&v)[2], const double* p) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    v[0] = t.x; v[1] = t.y;
}
__device__ __forceinline__ void gs_load(float (&v)[4], const float* p) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void gs_store(double* p, const double (&v)[2]) {
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
}
__device__ __forceinline__ void gs_store(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

template <typename T>
struct GsFields {
    const T* U[3];
    const T* Q[3];
    T* PRE[3];
    int comp[3];
};

// pc: the handle's table k_gs_coef fills, [p0|p1|p2|p3|d|cT|cB|pb] x nz, p0 = 1/d.
template <typename T, bool PRE, bool RESID>
__global__ void __launch_bounds__(32 * GS_ROWS) k_gs_parts(Geom g, T cE, T cN, const double* pc,
                                                           const int* __restrict__ slab_of_k,
                                                           const SlabDesc* __restrict__ slabs, GsFields<T> f, int gx,
                                                           int gy, int gz, int kc, RedWork rw, DevScalars* sc) {
    constexpr int VEC = 16 / sizeof(T);
    constexpr unsigned ALL = 0xffffffffu;
    __shared__ T s_c[GS_KC][4];  // 1/d, d, cT, cB
    __shared__ double s_red[GS_ROWS];
    const int lane = threadIdx.x, tid = threadIdx.y * 32 + lane;
    // (selected, not indexed: an indexed parameter is copied to local memory)
    auto pick = [](const auto& a, int i) { return i == 0 ? a[0] : i == 1 ? a[1] : a[2]; };
    const int comp = pick(f.comp, blockIdx.y), nz = g.nz;
    const T *U = pick(f.U, comp), *Q = pick(f.Q, comp);
    T* P = pick(f.PRE, comp);
    dependent_wait(pc);
    double acc = 0.0;
    for (int t = blockIdx.x; t < gx * gy * gz; t += gridDim.x) {
        const int bx = t % gx, by = t / gx % gy, bz = t / (gx * gy);
        const int k_lo = 1 + kc * bz, k_hi = min(nz - 2, k_lo + kc - 1);
        __syncthreads();
        for (int q = tid; q < 4 * kc; q += 32 * GS_ROWS) {
            const int k = min(k_lo + q / 4, nz - 2), c = q % 4;
            s_c[q / 4][c] = (T)pc[(c == 0 ? 0 : c + 3) * nz + k];
        }
        __syncthreads();
        const int j = 1 + GS_ROWS * by + threadIdx.y;
        if (j > g.ny - 2) continue;
        const int jm = j == 1 ? g.ny - 2 : j - 1, jp = j == g.ny - 2 ? 1 : j + 1;
        const bool need_m = RESID || j == 1;
        const int first = VEC * (32 * bx + lane);
        const int i0 = min(first, g.sx - VEC);  // lanes beyond the row load its end and store nothing
        unsigned okm = 0;
#pragma unroll
        for (int e = 0; e < VEC; ++e)
            if (first + e >= 1 && first + e <= g.nx - 2) okm |= 1u << e;
        long long o = (long long)i0 + (long long)g.sx * ((long long)j + (long long)g.ny * k_lo);
        const long long djm = (long long)g.sx * (jm - j), djp = (long long)g.sx * (jp - j);
        T zm[VEC], x[VEC];
        if (RESID) gs_load(zm, U + o - g.ps);
        gs_load(x, U + o);
        for (int k = k_lo; k <= k_hi; ++k, o += g.ps) {
            T zp[VEC], ym[VEC], yp[VEC], s[VEC];
            gs_load(s, Q + o);
            gs_load(zp, U + o + g.ps);
            gs_load(yp, U + o + djp);
            if (need_m) gs_load(ym, U + o + djm);
            T xl = T(0), xr = __shfl_down_sync(ALL, x[0], 1);
            if (lane == 31) xr = i0 + VEC < g.sx ? U[o + VEC] : T(0);
            if (RESID) {
                xl = __shfl_up_sync(ALL, x[VEC - 1], 1);
                if (lane == 0) xl = i0 > 0 ? U[o - 1] : T(0);
            }
            const T rd = s_c[k - k_lo][0], d = s_c[k - k_lo][1], cT = s_c[k - k_lo][2], cB = s_c[k - k_lo][3];
            const bool wrap = PRE && jp == 1, low = PRE && k == slabs[slab_of_k[k]].bn;
            T zl[VEC];  // the plane below, where PRE takes it
            if (PRE && !RESID && low) gs_load(zl, U + o - g.ps);
            T out[VEC], sum = T(0);
            // The special rows and planes are real branches (the warp sync inside
            // keeps them from becoming predicated FMAs, which cost FP64 issue all
            // the same: 12 against 9.5 operations a point).
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                s[e] = fma(-cE, e < VEC - 1 ? x[e < VEC - 1 ? e + 1 : e] : xr, s[e]);
                s[e] = fma(-cT, zp[e], s[e]);
                if (PRE) out[e] = s[e];
                s[e] = fma(-cN, yp[e], s[e]);
                if (PRE && !wrap) out[e] = s[e];
            }
            if (PRE && j == 1) {
                __syncwarp();
#pragma unroll
                for (int e = 0; e < VEC; ++e) out[e] = fma(-cN, ym[e], out[e]);
            }
            if (low) {
                __syncwarp();
#pragma unroll
                for (int e = 0; e < VEC; ++e) out[e] = fma(-cB, RESID ? zm[e] : zl[e], out[e]);
            }
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                if (PRE) out[e] *= rd;
                if (RESID) {
                    s[e] = fma(-d, x[e], s[e]);
                    s[e] = fma(-cE, e > 0 ? x[e > 0 ? e - 1 : 0] : xl, s[e]);
                    s[e] = fma(-cN, ym[e], s[e]);
                    s[e] = fma(-cB, zm[e], s[e]);
                    if (okm >> e & 1u) sum += abs(s[e]);
                }
            }
            if (RESID) acc += (double)sum;
            if (PRE) {
                if (first == 0) out[0] = x[0];  // the inflow boundary value
                if (okm == (1u << VEC) - 1 || (first == 0 && okm == (1u << VEC) - 2)) {
                    gs_store(P + o, out);
                } else {
#pragma unroll
                    for (int e = 0; e < VEC; ++e)
                        if ((okm >> e & 1u) || first + e == 0) P[o + e] = out[e];
                }
            }
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                if (RESID) zm[e] = x[e];
                x[e] = zp[e];
            }
        }
    }
    if (!RESID) return;
    // block_sum and grid_finish index by threadIdx.x: the block's sum in FP64, by rows
    acc = warp_sum(acc);
    __syncthreads();
    if (lane == 0) s_red[threadIdx.y] = acc;
    __syncthreads();
    __shared__ bool s_last;
    if (tid == 0) {
        double b = 0.0;
        for (int q = 0; q < GS_ROWS; ++q) b += s_red[q];
        rw.partial[(size_t)comp * rw.max_blocks + blockIdx.x] = b;
        __threadfence();
        s_last = atomicAdd(&rw.count[comp], 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    double tot = 0.0;
    for (int q = tid; q < (int)gridDim.x; q += 32 * GS_ROWS) tot += __ldcg(&rw.partial[(size_t)comp * rw.max_blocks + q]);
    tot = warp_sum(tot);
    __syncthreads();
    if (lane == 0) s_red[threadIdx.y] = tot;
    __syncthreads();
    if (tid == 0) {
        double b = 0.0;
        for (int q = 0; q < GS_ROWS; ++q) b += s_red[q];
        sc->red[comp] = b;
        rw.count[comp] = 0u;
    }
}

template <typename T>
static int gs_parts(tbl_handle* h, T* const U[3], T* const Q[3], T* const PRE[3], const int* comps, int ncomp, bool pre,
                    bool resid) {
    const Geom& g = h->g;
    const int vec = 16 / (int)sizeof(T), planes = g.nz - 2;
    const int gx = (g.nx - 2) / (32 * vec) + 1, gy = (g.ny - 2 + GS_ROWS - 1) / GS_ROWS;
    // planes per tile: about 8 blocks per SM over the components (16 in FP64: 16.8
    // against 17.5 ms of checks a step at 512 x 130 x 128), one plane at least
    const long long sms = h->n_sm > 0 ? h->n_sm : 148, tiles = (long long)gx * gy * ncomp;
    const long long want = ((sizeof(T) == 8 ? 16 : 8) * sms + tiles - 1) / tiles;
    const int kc = (int)std::min((long long)GS_KC, (planes + want - 1) / want), gz = (planes + kc - 1) / kc;
    const long long nb = std::min((long long)gx * gy * gz, (long long)h->red.max_blocks);
    const double t = -h->cfg.dt / (h->cfg.re);
    const T cE = (T)(t * (1.0 / (h->cfg.dx * h->cfg.dx))), cN = (T)(t * (1.0 / (h->cfg.dy * h->cfg.dy)));
    GsFields<T> f;
    for (int c = 0; c < 3; ++c) {
        f.U[c] = U[c]; f.Q[c] = Q[c]; f.PRE[c] = PRE[c];
        f.comp[c] = c < ncomp ? comps[c] : 0;
    }
    TBL_CUDA_TRY(launch_dependent(pre ? resid ? k_gs_parts<T, true, true> : k_gs_parts<T, true, false>
                                      : k_gs_parts<T, false, true>,
                                  dim3((unsigned)nb, ncomp), dim3(32, GS_ROWS), 0, h->stream, g, cE, cN, h->gs_coef,
                                  h->slab_of_k, h->slabs, f, gx, gy, gz, kc, h->red, h->sc));
    h->launches++;
    return TBL_OK;
}

// The residual of the listed components into sc->red[comp] (resid), the
// line-scan sweeps' PRE (pre), or both.
int launch_gs_parts(tbl_handle* h, const int* comps, int ncomp, bool pre, bool resid) {
    if (h->cfg.precision == TBL_PREC_MIXED) {  // delta form: the increment D and its right-hand side
        float* P[3] = {h->PREf, h->PREf + h->g.vol, h->PREf + 2 * h->g.vol};
        return gs_parts<float>(h, h->Df, h->Qf, P, comps, ncomp, pre, resid);
    }
    double* P[3] = {h->PRE, h->PRE + h->g.vol, h->PRE + 2 * h->g.vol};
    return gs_parts<double>(h, h->U, h->Q, P, comps, ncomp, pre, resid);
}

}  // namespace tbl
