// fi_plain.cu -- the plain FP64 form: the broadcast / stencil structure of the reference
// right-hand side (src/simulation.jl:335-393, src/deformation.jl:91-131 and
// src/derivatives.jl:48-191) with complex 2D FFTs as in the reference's c2c plans and a
// host-side step controller.  The Maxwell path's every-call work runs in six launches;
// the sparse update and the other rheologies keep one kernel per operation.  It is the
// comparison baseline of the fused FP32 form and a second, independent implementation.
#include "fi_device.cuh"
#include "fi_plain.h"

namespace fi {

#define GRID_STRIDE(i, n) for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)(n); \
                               i += (size_t)gridDim.x * blockDim.x)

__global__ void kp_corner_off(const double* X, int nx, int ny, double border, double* off) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        // sum(W .* X) with W = 1/4 at the corners (boundary_conditions.jl:144-148, 199-207)
        const double s = 0.25 * X[0] + 0.25 * X[nx - 1] + 0.25 * X[(size_t)(ny - 1) * nx] +
                         0.25 * X[(size_t)(ny - 1) * nx + nx - 1];
        *off = s - border;
    }
}

__global__ void kp_sub_off(double* X, size_t n, const double* off) {
    const double o = *off;
    GRID_STRIDE(i, n) X[i] -= o;
}

__global__ void kp_copy(double* dst, const double* src, size_t n) { GRID_STRIDE(i, n) dst[i] = src[i]; }

__global__ void kp_haf_ice(const double* H, const double* z_b, const double* z_ss, const double* H_af_ref,
                           double* H_af, double* s_i, double rho_sw_ice, double rho_ice, size_t n) {
    GRID_STRIDE(i, n) {
        double m = z_b[i] - z_ss[i];
        if (m > 0) m = 0;
        double v = H[i] + m * rho_sw_ice;
        v = v > 0 ? v : 0.0;
        H_af[i] = v;
        s_i[i] = rho_ice * (v - H_af_ref[i]);
    }
}

__global__ void kp_litho(const double* ue, const double* ue_ref, double* s_l, double rho_l, size_t n) {
    GRID_STRIDE(i, n) s_l[i] = rho_l * (ue[i] - ue_ref[i]);
}

__global__ void kp_geo_in(const double* s_load, const double* s_full, const double* s_m, const double* mask,
                          int compressible, double A, double* out, size_t n) {
    GRID_STRIDE(i, n) out[i] = compressible ? A * (s_load[i] + mask[i] * s_m[i]) : A * s_full[i];
}

__global__ void kp_zss(const double* z_ss_ref, const double* dz, double z_bsl, double* z_ss, size_t n) {
    GRID_STRIDE(i, n) z_ss[i] = z_ss_ref[i] + dz[i] + z_bsl;
}

__global__ void kp_load_full(const double* s_i, const double* s_sw, const double* s_l, const double* s_m,
                             const double* mask, double* s_load, double* s_full, size_t n) {
    GRID_STRIDE(i, n) {
        const double ld = mask[i] * (s_i[i] + s_sw[i] + 0.0);  // the sediment anomaly is zero
        s_load[i] = ld;
        s_full[i] = ld + mask[i] * (s_l[i] + s_m[i]);
    }
}

// ---------------------------------------------------------------------------
// One right-hand side of the Maxwell path in six launches.  At the usual sizes a launch costs
// more than the pass it makes over an L2-resident field, and one kernel per broadcast of the
// reference took about thirty.  Every product and quotient is rounded where the separate kernels
// rounded it (__dmul_rn where a following sum would otherwise absorb it), so the results are
// bitwise theirs.  A coupled 10-yr step at N = 128 (some 25 BS3 attempts): 8567 -> 3027 us.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double corner_off(double c0, double c1, double c2, double c3, double border) {
    const double s = 0.25 * c0 + 0.25 * c1 + 0.25 * c2 + 0.25 * c3;
    return s - border;
}

// the stage vector's value at i: u itself, uprev + a k1, or stage 4 (uprev + dt (a41 k1 + a42 k2 + a43 k3))
__device__ __forceinline__ double stage_value(const PlainStage& st, const double* u, size_t i) {
    if (st.kind == 0) return u[i];
    if (st.kind == 1) return st.up[i] + st.a * st.k1[i];
    return st.up[i] + st.a * (A41 * st.k1[i] + A42 * st.k2[i] + A43 * st.k3[i]);
}

// stage vector, its corner BC, bedrock, ice, height above floatation and their anomalies.  u is
// only read (its corners by every block); now_u gets the corrected vector.
__global__ void kp_head(PlainStage st, const double* u, int nx, int ny, double border, const double* ue,
                        const double* z_b_ref, const double* u_ref, double* now_u, double* z_b, double* s_m,
                        double rho_um, const double* Ha, const double* Hb, double dti, double tt, int exact, double* H,
                        const double* z_ss, const double* H_af_ref, double* H_af, double* s_i, double rho_sw_ice,
                        double rho_ice) {
    const size_t n = (size_t)nx * ny;
    const double off = corner_off(stage_value(st, u, 0), stage_value(st, u, nx - 1), stage_value(st, u, n - nx),
                                  stage_value(st, u, n - 1), border);
    GRID_STRIDE(i, n) {
        const double uv = stage_value(st, u, i) - off;
        now_u[i] = uv;
        const double zb = z_b_ref[i] + ue[i] + uv;
        z_b[i] = zb;
        s_m[i] = rho_um * (uv - u_ref[i]);
        double h;
        if (Ha) {
            h = exact ? Ha[i] : Ha[i] + (Hb[i] - Ha[i]) / dti * tt;
            H[i] = h;
        } else {
            h = H[i];
        }
        double m = zb - z_ss[i];
        if (m > 0) m = 0;
        double v = h + m * rho_sw_ice;
        v = v > 0 ? v : 0.0;
        H_af[i] = v;
        s_i[i] = rho_ice * (v - H_af_ref[i]);
    }
}

// d/dx along row r (one-sided at the ends)
__device__ __forceinline__ double dx_at(const double* r, int i, int nx, double Dx) {
    if (i == 0) return (r[1] - r[0]) / Dx;
    if (i == nx - 1) return (r[nx - 1] - r[nx - 2]) / Dx;
    return (r[i + 1] - r[i - 1]) / (2 * Dx);
}
__device__ __forceinline__ double dxx_at(const double* r, int i, int nx, double Dx) {
    const int c = i < 1 ? 1 : (i > nx - 2 ? nx - 2 : i);
    return (r[c + 1] - 2 * r[c] + r[c - 1]) / (Dx * Dx);
}
__device__ __forceinline__ double dyy_at(const double* u, int i, int j, int nx, int ny, double Dy) {
    const size_t e = (size_t)j * nx + i;
    if (j > 0 && j < ny - 1) return (u[e + nx] - 2 * u[e] + u[e - nx]) / (Dy * Dy);
    if (j == 0) return (u[e + 2 * (size_t)nx] - 2 * u[e + nx] + u[e]) / (Dy * Dy);
    return (u[e] - 2 * u[e - nx] + u[e - 2 * (size_t)nx]) / (Dy * Dy);
}
// d/dy of d/dx
__device__ __forceinline__ double dxy_at(const double* u, int i, int j, int nx, int ny, double Dx, double Dy) {
    const double* r = u + (size_t)j * nx;
    if (j == 0) return (dx_at(r + nx, i, nx, Dx) - dx_at(r, i, nx, Dx)) / Dy;
    if (j == ny - 1) return (dx_at(r, i, nx, Dx) - dx_at(r - nx, i, nx, Dx)) / Dy;
    return (dx_at(r + nx, i, nx, Dx) - dx_at(r - nx, i, nx, Dx)) / (2 * Dy);
}

// column anomalies, bending moments of now_u; u <- now_u (the BC's in-place change)
__global__ void kp_load_moments(const double* s_i, const double* s_sw, const double* s_l, const double* s_m,
                                const double* mask, double* s_load, double* s_full, const double* now_u, double* u,
                                int nx, int ny, double Dx, double Dy, const double* D, double nu, double* Mxx,
                                double* Myy, double* Mxy) {
    GRID_STRIDE(e, (size_t)nx * ny) {
        const int i = (int)(e % nx), j = (int)(e / nx);
        const double ld = __dmul_rn(mask[e], s_i[e] + s_sw[e] + 0.0);
        s_load[e] = ld;
        s_full[e] = ld + mask[e] * (s_l[e] + s_m[e]);
        const double bxx = dxx_at(now_u + (e - i), i, nx, Dx), byy = dyy_at(now_u, i, j, nx, ny, Dy);
        const double bxy = dxy_at(now_u, i, j, nx, ny, Dx, Dy);
        Mxx[e] = -D[e] * (nu * byy + bxx);
        Myy[e] = -D[e] * (nu * bxx + byy);
        Mxy[e] = -D[e] * (1 - nu) * bxy;
        u[e] = now_u[e];
    }
}

// a row of rhs = -g s_full + Mxx_xx + 2 Mxy_xy + Myy_yy, times K/(2 eta), and its row transform
__global__ void __launch_bounds__(256)
kp_div_rows(const double* s_full, double g, const double* Mxx, const double* Myy, const double* Mxy, int nx, int ny,
            double Dx, double Dy, const double* eta, double2* f, const FftPlan* plans, int plan) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ FftPlan s_plan;
    const int j = blockIdx.x;
    if (threadIdx.x == 0) s_plan = plans[plan];
    double2* b0 = (double2*)smem;
    double2* b1 = b0 + nx;
    for (int i = threadIdx.x; i < nx; i += blockDim.x) {
        const size_t e = (size_t)j * nx + i;
        const double bxx = dxx_at(Mxx + (size_t)j * nx, i, nx, Dx), byy = dyy_at(Myy, i, j, nx, ny, Dy);
        const double bxy = dxy_at(Mxy, i, j, nx, ny, Dx, Dy);
        const double rhs = __dmul_rn(-g, s_full[e]) + (bxx + (2 * bxy + byy));
        b0[i] = make_double2(rhs * 1.0 / (2 * eta[e]), 0.0);
    }
    __syncthreads();
    double2* r = fft_batch<false, double>(b0, b1, s_plan, 1, nx);
    for (int i = threadIdx.x; i < nx; i += blockDim.x) f[(size_t)j * nx + i] = r[i];
}

// a column: transform, times 1/(R |k|), inverse transform with its scale
__global__ void __launch_bounds__(256)
kp_spec_cols(double2* f, int nx, int ny, const double* spinv, const FftPlan* plans, int plan, double scale) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ FftPlan s_plan;
    const int kx = blockIdx.x;
    if (threadIdx.x == 0) s_plan = plans[plan];
    double2* b0 = (double2*)smem;
    double2* b1 = b0 + ny;
    for (int y = threadIdx.x; y < ny; y += blockDim.x) b0[y] = f[(size_t)y * nx + kx];
    __syncthreads();
    double2* r = fft_batch<false, double>(b0, b1, s_plan, 1, ny);
    double2* o = r == b0 ? b1 : b0;
    for (int y = threadIdx.x; y < ny; y += blockDim.x) {
        const double s = spinv[(size_t)y * nx + kx];
        r[y] = make_double2(r[y].x * s, r[y].y * s);
    }
    __syncthreads();
    double2* q = fft_batch<true, double>(r, o, s_plan, 1, ny);
    for (int y = threadIdx.x; y < ny; y += blockDim.x)
        f[(size_t)y * nx + kx] = make_double2(q[y].x * scale, q[y].y * scale);
}

// inverse row transform, real part times the seconds of a year
__global__ void __launch_bounds__(256)
kp_rows_real(const double2* f, int nx, double spy, double* raw, const FftPlan* plans, int plan) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ FftPlan s_plan;
    if (threadIdx.x == 0) s_plan = plans[plan];
    double2* b0 = (double2*)smem;
    double2* b1 = b0 + nx;
    const size_t r0 = (size_t)blockIdx.x * nx;
    for (int i = threadIdx.x; i < nx; i += blockDim.x) b0[i] = f[r0 + i];
    __syncthreads();
    double2* r = fft_batch<true, double>(b0, b1, s_plan, 1, nx);
    for (int i = threadIdx.x; i < nx; i += blockDim.x) raw[r0 + i] = r[i].x * spy;
}

// corner BC of raw into dudt and its copy
__global__ void kp_corner_out(const double* raw, int nx, int ny, double border, double* dudt, double* now_dudt) {
    const size_t n = (size_t)nx * ny;
    const double off = corner_off(raw[0], raw[nx - 1], raw[n - nx], raw[n - 1], border);
    GRID_STRIDE(i, n) {
        const double v = raw[i] - off;
        dudt[i] = v;
        now_dudt[i] = v;
    }
}

// block partial sums of H_af A, H_ice A and max(z_ss - z_b, 0) A (update_V_af!,
// update_V_den!, update_V_pov!, src/sealevel.jl:275-332), three per block
__global__ void kp_volumes(const double* H_af, const double* H, const double* z_ss, const double* z_b, double A,
                           double* partial, size_t n) {
    __shared__ double red[96];
    double a = 0.0, d = 0.0, p = 0.0;
    GRID_STRIDE(i, n) {
        a += H_af[i] * A;
        d += H[i] * A;
        const double w = z_ss[i] - z_b[i];
        p += (w > 0 ? w : 0.0) * A;
    }
    double v[3] = {a, d, p};
    block_sum<3>(v, red);
    if (threadIdx.x == 0)
        for (int q = 0; q < 3; q++) partial[3 * blockIdx.x + q] = v[q];
}

// update_maskgrounded!, update_maskocean!, watercolumn! and columnanom_water!
// (src/topography.jl:1-28, src/loads.jl:56-85)
__global__ void kp_sealevel(const double* H, const double* H_af, const double* z_ss, const double* z_b,
                            const double* z_ss_ref, const double* mask, int interactive, double rho_sw,
                            double rho_i_sw, double* mgr, double* moc, double* hwater, double* s_sw, size_t n) {
    GRID_STRIDE(i, n) {
        const bool gr = H_af[i] > 0;
        const double w = z_ss[i] - z_b[i];
        const bool oc = w > 0 && !gr;
        const double wc = w > 0 ? w : 0.0;
        mgr[i] = gr;
        moc[i] = oc;
        hwater[i] = (H[i] <= 1 ? wc : 0.0) + ((!gr && H[i] > 1) ? wc - H[i] * rho_i_sw : 0.0);
        s_sw[i] = interactive ? rho_sw * (z_ss[i] - z_ss_ref[i]) * (oc ? 1.0 : 0.0) * mask[i] : 0.0;
    }
}

__global__ void kp_cmul(double2* P, const double2* G, size_t n) {
    GRID_STRIDE(i, n) {
        const double2 a = P[i], b = G[i];
        P[i] = make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
    }
}

__global__ void kp_crop(const double2* P, int Mx, int cx, int cy, double* out) {
    GRID_STRIDE(e, (size_t)cx * cy) {
        const int i = (int)(e % cx), j = (int)(e / cx);
        out[e] = P[(size_t)j * Mx + i].x;
    }
}

__global__ void kp_window(const double* cropped, int cx, int i1, int j1, int nx, int ny, double* out) {
    GRID_STRIDE(e, (size_t)nx * ny) {
        const int i = (int)(e % nx), j = (int)(e / nx);
        out[e] = cropped[(size_t)(j1 + j) * cx + i1 + i];
    }
}

__global__ void kp_zero(double* X, size_t n) { GRID_STRIDE(i, n) X[i] = 0.0; }

// integrator helpers (perform_step!(integrator, ::BS3Cache))
__global__ void kp_stage(double* out, const double* uprev, double a, const double* k, size_t n) {
    GRID_STRIDE(i, n) out[i] = uprev[i] + a * k[i];
}

__global__ void kp_err(const double* uprev, const double* u, const double* k1, const double* k2, const double* k3,
                       const double* k4, double dt, double abstol, double reltol, double* partial, size_t n) {
    __shared__ double red[32];
    double acc = 0.0;
    GRID_STRIDE(i, n) {
        const double ut = dt * (BT1 * k1[i] + BT2 * k2[i] + BT3 * k3[i] + BT4 * k4[i]);
        const double a = fabs(uprev[i]), b = fabs(u[i]);
        const double r = ut / (abstol + (a > b ? a : b) * reltol);
        acc += r * r;
    }
    double v[1] = {acc};
    block_sum<1>(v, red);
    if (threadIdx.x == 0) partial[blockIdx.x] = v[0];
}

// sums of squares for the initial-dt heuristic: s0 = sum (a/sk)^2, s1 = sum (b/sk)^2
__global__ void kp_norms2(const double* a, const double* b, const double* sk_base, double abstol, double reltol,
                          double* partial, size_t n) {
    __shared__ double red[64];
    double s0 = 0.0, s1 = 0.0;
    GRID_STRIDE(i, n) {
        const double sk = abstol + fabs(sk_base[i]) * reltol;
        const double x = a[i] / sk, y = b[i] / sk;
        s0 += x * x;
        s1 += y * y;
    }
    double v[2] = {s0, s1};
    block_sum<2>(v, red);
    if (threadIdx.x == 0) { partial[2 * blockIdx.x] = v[0]; partial[2 * blockIdx.x + 1] = v[1]; }
}

__global__ void kp_initdt_terms(const double* f0, const double* f1, const double* sk_base, double abstol,
                                double reltol, double* partial, size_t n) {
    __shared__ double red[64];
    double s0 = 0.0, eq = 1.0;
    GRID_STRIDE(i, n) {
        const double sk = abstol + fabs(sk_base[i]) * reltol;
        const double x = (f1[i] - f0[i]) / sk;
        s0 += x * x;
        if (f1[i] != f0[i]) eq = 0.0;
    }
    double v[2] = {s0, eq};
    block_sum<2>(v, red);
    if (threadIdx.x == 0) { partial[2 * blockIdx.x] = v[0]; partial[2 * blockIdx.x + 1] = v[1]; }
}

// ELRA (src/deformation.jl:29-45): the convolution input -(load + litho) g K^2 and
// dudt = (u_eq - u) / tau
__global__ void kp_elra_in(const double* s_load, const double* s_l, double g, double* out, size_t n) {
    GRID_STRIDE(i, n) out[i] = -(s_load[i] + s_l[i]) * g;
}
__global__ void kp_elra_dudt(const double* u_eq, const double* u, const double* tau, double* dudt, size_t n) {
    GRID_STRIDE(i, n) dudt[i] = 1.0 / tau[i] * (u_eq[i] - u[i]);
}

// Laterally-constant Maxwell step (src/deformation.jl:52-89): F = -(load + litho) g,
// U = u as complex inputs; then U <- ((nabla - dt/2 beta) U + dt F) / (nabla + dt/2 beta)
// with nabla = 2 eta |k| R and beta = rho_m g + D |k|^4, elementwise as the reference
// broadcasts them; then u = Re(ifft(U)).
__global__ void kp_lc_in(const double* s_load, const double* s_l, double g, const double* u, double2* F, double2* U,
                         size_t n) {
    GRID_STRIDE(i, n) {
        F[i] = make_double2(-(s_load[i] + s_l[i]) * g, 0.0);
        U[i] = make_double2(u[i], 0.0);
    }
}
__global__ void kp_lc_step(double2* U, const double2* F, const double* eta, const double* pd, const double* R,
                           const double* D, double rho_m_g, double dt, size_t n) {
    GRID_STRIDE(i, n) {
        const double k = pd[i];
        const double nab = 2.0 * eta[i] * k * R[i];
        const double beta = rho_m_g + D[i] * k * k * k * k;
        const double a = nab - dt / 2 * beta, b = nab + dt / 2 * beta;
        U[i] = make_double2((a * U[i].x + dt * F[i].x) / b, (a * U[i].y + dt * F[i].y) / b);
    }
}
__global__ void kp_real(const double2* U, double* u, size_t n) { GRID_STRIDE(i, n) u[i] = U[i].x; }

// Output staging of the FP32 form: out = [u | ue - cue | dudt - cdu | dz - cdz] in FP64
// (fields whose source is null are skipped).
__global__ void k_out_stage(const double* u, const float* ue, double cue, const float* dudt, double cdu,
                            const float* dz, double cdz, double* out, size_t n) {
    GRID_STRIDE(i, n) {
        if (u) out[i] = u[i];
        if (ue) out[n + i] = (double)ue[i] - cue;
        if (dudt) out[2 * n + i] = (double)dudt[i] - cdu;
        if (dz) out[3 * n + i] = (double)dz[i] - cdz;
    }
}

// ---------------------------------------------------------------------------
// fields between the device's layout ((i, j) at i + j nx) and the caller's
// ---------------------------------------------------------------------------
// out(i, j) = in(i, j) - (corner mean of c4 - border) (c4 null: - off), FP64; rowmajor: (i, j) of
// out at i ny + j, through a 32 x 32 tile so that both sides are read and written along rows.
template <typename T>
__device__ __forceinline__ void field_out(const T* in, const double* c4, double border, double off, int nx, int ny,
                                          int rowmajor, double* out) {
    __shared__ double tile[32][33];
    if (c4) off = (0.25 * (c4[0] + c4[1] + c4[2] + c4[3])) - border;
    const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int i = i0 + threadIdx.x, j = j0 + r;
        if (i < nx && j < ny) {
            const double v = (double)in[(size_t)j * nx + i] - off;
            if (rowmajor) tile[r][threadIdx.x] = v;
            else out[(size_t)j * nx + i] = v;
        }
    }
    if (!rowmajor) return;
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int i = i0 + r, j = j0 + threadIdx.x;
        if (i < nx && j < ny) out[(size_t)i * ny + j] = tile[threadIdx.x][r];
    }
}
__global__ void k_field_out64(const double* in, int nx, int ny, int rowmajor, double* out) {
    field_out(in, nullptr, 0.0, 0.0, nx, ny, rowmajor, out);
}
__global__ void k_field_out32(const float* in, const double* c4, double border, double off, int nx, int ny,
                              int rowmajor, double* out) {
    field_out(in, c4, border, off, nx, ny, rowmajor, out);
}

// in(i, j) at i ny + j (rowmajor) or i + j nx -> the device's layout, FP64 and / or FP32
__global__ void k_field_in(const double* in, int nx, int ny, int rowmajor, double* out64, float* out32) {
    __shared__ double tile[32][33];
    const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
    for (int r = threadIdx.y; r < 32; r += 8) {
        if (rowmajor) {
            const int i = i0 + r, j = j0 + threadIdx.x;
            if (i < nx && j < ny) tile[threadIdx.x][r] = in[(size_t)i * ny + j];
        } else {
            const int i = i0 + threadIdx.x, j = j0 + r;
            if (i < nx && j < ny) tile[r][threadIdx.x] = in[(size_t)j * nx + i];
        }
    }
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8) {
        const int i = i0 + threadIdx.x, j = j0 + r;
        if (i < nx && j < ny) {
            const double v = tile[r][threadIdx.x];
            if (out64) out64[(size_t)j * nx + i] = v;
            if (out32) out32[(size_t)j * nx + i] = (float)v;
        }
    }
}

}  // namespace fi
