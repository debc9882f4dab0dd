// fi_plain.h -- kernels of the plain FP64 form (fi_plain.cu).
#pragma once
#include <cuda_runtime.h>

#include "fi_fft.cuh"

namespace fi {
// The vector a right-hand side is evaluated at: kind 0 the given u, 1 up + a k1, 2 the fourth
// BS3 stage up + a (2/9 k1 + 1/3 k2 + 4/9 k3).
struct PlainStage {
    int kind = 0;
    double a = 0.0;
    const double *up = nullptr, *k1 = nullptr, *k2 = nullptr, *k3 = nullptr;
};
__global__ void kp_head(PlainStage st, const double* u, int nx, int ny, double border, const double* ue,
                        const double* z_b_ref, const double* u_ref, double* now_u, double* z_b, double* s_m,
                        double rho_um, const double* Ha, const double* Hb, double dti, double tt, int exact, double* H,
                        const double* z_ss, const double* H_af_ref, double* H_af, double* s_i, double rho_sw_ice,
                        double rho_ice);
__global__ void kp_load_moments(const double* s_i, const double* s_sw, const double* s_l, const double* s_m,
                                const double* mask, double* s_load, double* s_full, const double* now_u, double* u,
                                int nx, int ny, double Dx, double Dy, const double* D, double nu, double* Mxx,
                                double* Myy, double* Mxy);
__global__ void kp_div_rows(const double* s_full, double g, const double* Mxx, const double* Myy, const double* Mxy,
                            int nx, int ny, double Dx, double Dy, const double* eta, double2* f, const FftPlan* plans,
                            int plan);
__global__ void kp_spec_cols(double2* f, int nx, int ny, const double* spinv, const FftPlan* plans, int plan,
                             double scale);
__global__ void kp_rows_real(const double2* f, int nx, double spy, double* raw, const FftPlan* plans, int plan);
__global__ void kp_corner_out(const double* raw, int nx, int ny, double border, double* dudt, double* now_dudt);
__global__ void kp_corner_off(const double* X, int nx, int ny, double border, double* off);
__global__ void kp_sub_off(double* X, size_t n, const double* off);
__global__ void kp_copy(double* dst, const double* src, size_t n);
__global__ void kp_haf_ice(const double* H, const double* z_b, const double* z_ss, const double* H_af_ref,
                           double* H_af, double* s_i, double rho_sw_ice, double rho_ice, size_t n);
__global__ void kp_litho(const double* ue, const double* ue_ref, double* s_l, double rho_l, size_t n);
__global__ void kp_geo_in(const double* s_load, const double* s_full, const double* s_m, const double* mask,
                          int compressible, double A, double* out, size_t n);
__global__ void kp_zss(const double* z_ss_ref, const double* dz, double z_bsl, double* z_ss, size_t n);
__global__ void kp_load_full(const double* s_i, const double* s_sw, const double* s_l, const double* s_m,
                             const double* mask, double* s_load, double* s_full, size_t n);
__global__ void kp_volumes(const double* H_af, const double* H, const double* z_ss, const double* z_b, double A,
                           double* partial, size_t n);
__global__ void kp_sealevel(const double* H, const double* H_af, const double* z_ss, const double* z_b,
                            const double* z_ss_ref, const double* mask, int interactive, double rho_sw,
                            double rho_i_sw, double* mgr, double* moc, double* hwater, double* s_sw, size_t n);
__global__ void kp_cmul(double2* P, const double2* G, size_t n);
__global__ void kp_crop(const double2* P, int Mx, int cx, int cy, double* out);
__global__ void kp_window(const double* cropped, int cx, int i1, int j1, int nx, int ny, double* out);
__global__ void kp_zero(double* X, size_t n);
__global__ void kp_stage(double* out, const double* uprev, double a, const double* k, size_t n);
__global__ void kp_err(const double* uprev, const double* u, const double* k1, const double* k2, const double* k3,
                       const double* k4, double dt, double abstol, double reltol, double* partial, size_t n);
__global__ void kp_norms2(const double* a, const double* b, const double* sk_base, double abstol, double reltol,
                          double* partial, size_t n);
__global__ void kp_initdt_terms(const double* f0, const double* f1, const double* sk_base, double abstol,
                                double reltol, double* partial, size_t n);
__global__ void kp_elra_in(const double* s_load, const double* s_l, double g, double* out, size_t n);
__global__ void kp_elra_dudt(const double* u_eq, const double* u, const double* tau, double* dudt, size_t n);
__global__ void kp_lc_in(const double* s_load, const double* s_l, double g, const double* u, double2* F, double2* U,
                         size_t n);
__global__ void kp_lc_step(double2* U, const double2* F, const double* eta, const double* pd, const double* R,
                           const double* D, double rho_m_g, double dt, size_t n);
__global__ void kp_real(const double2* U, double* u, size_t n);
__global__ void k_field_out64(const double* in, int nx, int ny, int rowmajor, double* out);
__global__ void k_field_out32(const float* in, const double* c4, double border, double off, int nx, int ny,
                              int rowmajor, double* out);
__global__ void k_field_in(const double* in, int nx, int ny, int rowmajor, double* out64, float* out32);
__global__ void k_out_stage(const double* u, const float* ue, double cue, const float* dudt, double cdu,
                            const float* dz, double cdz, double* out, size_t n);
}  // namespace fi
