// tbl_kernels.cuh -- host-side launchers shared between translation units.
#pragma once
#include "tbl_internal.cuh"

namespace tbl {

// tbl_stencil.cu
int launch_save_uold(tbl_handle* h);
int launch_inflow(tbl_handle* h);
int launch_conv_q(tbl_handle* h);
int launch_div(tbl_handle* h);
int launch_pc_zero_faces(tbl_handle* h);
int launch_project_bcs(tbl_handle* h);
int launch_div_diag(tbl_handle* h, int nblocks, int slot);
int launch_flux_shear(tbl_handle* h);
int launch_fluc_ke(tbl_handle* h, int nblocks, int slot);
int launch_stats(tbl_handle* h);
int launch_rescale(tbl_handle* h);
int launch_gs_delta_init(tbl_handle* h, int comp);
int launch_gs_delta_apply(tbl_handle* h, int comp);
int launch_gs_delta_restart(tbl_handle* h, int comp);

// tbl_gs.cu
int launch_gs_parts(tbl_handle* h, const int* comps, int ncomp, bool pre, bool resid);

// tbl_sweep.cu
int build_sweep_ctas(tbl_handle* h);
int check_cooperative(tbl_handle* h);
int launch_gs_sweep(tbl_handle* h, const int* comps, int ncomp, int parity, bool have_pre);
int launch_gs_coef(tbl_handle* h);
int launch_halo_init(tbl_handle* h, int parity);
int launch_ssor_fwd(tbl_handle* h, const double* X, const double* Q8, const int* skip = nullptr,
                    const double* factor = nullptr);
int launch_ssor_bwd(tbl_handle* h, double* out, const int* skip = nullptr);
int launch_ssor_fwd_f(tbl_handle* h, const float* Xf, const double* PCd, const double* Q8, const int* skip = nullptr,
                      const double* denom = nullptr, float* vout = nullptr);
int launch_ssor_bwd_f(tbl_handle* h, float* out, const int* skip = nullptr);
int selftest_bounded_wait(int* observed, double* seconds);

// tbl_line.cu: line-scan sweeps, where h->line[mode].S > 0
int line_create(tbl_handle* h);
int line_selftest(tbl_handle* h, int which);
template <typename V>
int launch_line_gs(tbl_handle* h, V* const F[3], V* const PRE[3], const int* comps, int ncomp);
template <typename V>
int launch_line_ssor(tbl_handle* h, bool bwd, const V* in, V* out, const int* skip);

// tbl_lap.cu: R = factor scale(k) L7 X (no factor: 1), or scale(k) (Q8 - L7 X) with Q8
int launch_lap(tbl_handle* h, const double* X, const double* Q8, double* R, const int* skip, const double* factor);
int launch_lap_f(tbl_handle* h, const float* X, float* R, const int* skip, const double* denom, float* vout);
int launch_lap_resid_f(tbl_handle* h, const double* X, const double* Q8, float* R, const int* skip);

// tbl_krylov.cu
int launch_dot(tbl_handle* h, const double* a, const double* b, double* out, int op);
int launch_gs(tbl_handle* h, double* w, int k, const int* skip, double stop_at);
const double* gs_factor(const tbl_handle* h, int k);
int launch_backsub_update(tbl_handle* h, int kit);
int launch_restart_init(tbl_handle* h, int first);
int launch_ppe_resid(tbl_handle* h);
int red_blocks(tbl_handle* h);
int launch_dot_f(tbl_handle* h, const float* a, const float* b, double* out, int op);
int launch_scale_by_inv_f(tbl_handle* h, float* w, const double* denom, const int* skip = nullptr);
int launch_backsub_update_f(tbl_handle* h, int kit);
int launch_restart_init_k(tbl_handle* h, int first, int K1);
int launch_lsg_f(tbl_handle* h, float* W, int kit, const int* skip, double stop_at);

// tbl_api.cu
int readback(tbl_handle* h, const void* dev, size_t bytes);
int put3(tbl_handle* h, double* dst, const double* src);
int get3(tbl_handle* h, double* dst, const double* src);
int gs_solve(tbl_handle* h, const int* target, tbl_step_stats& st, bool zero_ok);
int gmres(tbl_handle* h, const int32_t* rec, std::vector<int32_t>& kits, tbl_step_stats& st);
int one_step(tbl_handle* h, tbl_step_stats* out);

// tbl_adjoint.cu
void adj_free(tbl_handle* h);

}  // namespace tbl
