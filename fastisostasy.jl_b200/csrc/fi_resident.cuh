// fi_resident.cuh -- persistent BS3 step executor whose blocks keep their row tile in
// shared memory (the "resident" kernel).
//
// Same integration as fi_persist.cu (one cooperative launch per output segment, the same
// arithmetic on the same elements in the same order, so the results are bitwise those of
// k_persist and of the per-phase kernels), for layouts with at most one row tile per SM:
// block b owns row tile b for the whole launch.
//
// What bounds a single simulation is latency, not bytes or flops: an attempt is seven
// grid-wide phases, and in each a short dependent chain runs behind a grid barrier.
// k_persist spent most of a forward-row phase on round trips to L2 (inputs read in place),
// on single-thread set-up after the barrier, and on cold instruction fetch.  Here
//  * the tile's state (u, k1..k4 with their halos) and its inputs stay in shared memory
//    across phases and attempts, as far as they fit (ResLayout; an offset of -1 reads in
//    place); only the spectrum, the corner partials and two halo rows a side move
//    through L2;
//  * a grid barrier is split into arrive and wait, and the scalar work of a phase (gate,
//    stage scalars, corner sums, halo refreshes) runs in between, or on the last four warps
//    beside the transforms of the other twelve;
//  * the first inverse pass reads the spectrum and the last column pass writes it straight
//    from registers, the viscous multiplier is applied in the store of the last forward
//    column pass, and the inverse transform of stage 4's derivative is the loop's fourth
//    trip through the same code, so a BS3 attempt runs one copy of each transform;
//  * the launch has one block per task (32 at N = 64, 117 at N = 350), so that a barrier has
//    no arrivals of blocks without work.
// Measured, us per BS3 attempt, k_persist -> this kernel: N = 64 48.4 -> 30.9, 165 x 130 83 ->
// 66, N = 350 (tiles of 3 rows) 65.5 -> 46.2, N = 1024 (8 rows) 292 -> 178.
// Measured and dropped: 768 threads a block (N = 350 48.6: more warps only add instruction
// fetches and barrier time); stencils marching down columns with a row's values kept for the
// next (N = 350 51.7, N = 1024 205: half the instructions, but one dependent chain a thread).
// Conversions between FP32 and FP64 run at 16 a cycle and SM, a quarter of the FP64
// arithmetic; they and the FP64 chains are what is left of the stencil sub-steps.
#pragma once
#include "fi_grid.cuh"

namespace fi {

// ---------------------------------------------------------------------------
// split grid barrier: the counter of grid_barrier (fi_grid.cuh)
// ---------------------------------------------------------------------------
// Every block arrives once per barrier, so the count to wait for is known and the arrival needs
// no answer (a reduction, not a returning atomic).  epoch: barriers so far, kept by every thread.
__device__ __forceinline__ void grid_arrive(unsigned int* bar) {
    __syncthreads();  // the block's writes happen before thread 0's release
    if (threadIdx.x == 0)
        asm volatile("red.add.release.gpu.u64 [%0], 1;" ::"l"(reinterpret_cast<unsigned long long*>(bar)) : "memory");
}

// Returns false (in every thread of the block) when the barrier was abandoned.
__device__ __forceinline__ bool grid_wait(unsigned int* bar, unsigned int nblocks, unsigned int& epoch, int* s_ok,
                                          long long polls) {
    epoch += 1;
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned long long target = (unsigned long long)epoch * nblocks;
        const unsigned long long* cnt = reinterpret_cast<const unsigned long long*>(bar);
        const volatile unsigned int* vabort = bar + 2;
        long long npoll = 0;
        for (;;) {
            unsigned long long cur;
            asm volatile("ld.acquire.gpu.u64 %0, [%1];" : "=l"(cur) : "l"(cnt) : "memory");
            if (cur >= target) break;
            if (++npoll > polls) {
                atomicExch(bar + 2, 1u);
                ok = 0;
                break;
            }
            if ((npoll & 63) == 0 && *vabort) {
                ok = 0;
                break;
            }
            if (npoll > 4096) __nanosleep(100);
        }
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// ---------------------------------------------------------------------------
// transform passes with the caller's loads and stores (the arithmetic of ct_pass)
// ---------------------------------------------------------------------------
// Run by the first FT threads of the block; group_sync<FT> is their barrier.
// ld(b, i) and st(b, i, v): element i of transform b.  BATCH_FAST: consecutive threads take
// consecutive transforms of one butterfly (for column-major global access).
template <int FT>
__device__ __forceinline__ void group_sync() {
    if constexpr (FT != 384) __syncthreads();
    else asm volatile("bar.sync 1, %0;" ::"n"(FT) : "memory");
}

template <int FT, int R, bool INV, int L, int NS, bool BATCH_FAST, class Ld, class St>
__device__ __forceinline__ void fn_pass(const float2* __restrict__ tw, int nbatch, unsigned int mag, Ld ld, St st) {
    constexpr int nb = L / R, stride = L / (NS * R);
    const int total = nbatch * nb;
#pragma unroll 1
    for (int idx = threadIdx.x; idx < total; idx += FT) {
        int b, j;
        if (BATCH_FAST) {
            j = (int)fastdiv((unsigned)idx, (unsigned)nbatch, mag);
            b = idx - j * nbatch;
        } else {
            b = idx / nb;
            j = idx - b * nb;
        }
        const int jq = j / NS;
        const int k = j - jq * NS;
        float2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = ld(b, j + r * nb);
        if (NS > 1) {
#pragma unroll
            for (int r = 1; r < R; r++) {
                float2 w = tw[k * r * stride];
                if (INV) w.y = -w.y;
                v[r] = cmul(v[r], w);
            }
        }
        SmallDft<R, INV, float>::run(v);
        const int idxD = jq * NS * R + k;
#pragma unroll
        for (int q = 0; q < R; q++) st(b, idxD + q * NS, v[q]);
    }
}

// Passes P0 .. P1-1 of SEQ between shared buffers (row pitch `pitch`); the result is in src
// when P1 - P0 is even, else in dst.
template <int FT, bool INV, int SEQ, int P0, int P1, int NS>
__device__ __forceinline__ void sm_passes(float2* src, float2* dst, const float2* tw, int nbatch, int pitch) {
    if constexpr (P0 < P1) {
        constexpr int R = seq_radix(SEQ, P0);
        fn_pass<FT, R, INV, seq_len(SEQ), NS, false>(
            tw, nbatch, 0u, [&](int b, int i) { return src[b * pitch + i]; },
            [&](int b, int i, float2 v) { dst[b * pitch + i] = v; });
        group_sync<FT>();
        sm_passes<FT, INV, SEQ, P0 + 1, P1, NS * R>(dst, src, tw, nbatch, pitch);
    }
}

// ---------------------------------------------------------------------------
// constants of the launch (the divisions of the stencils, done once)
// ---------------------------------------------------------------------------
struct ResConst {
    double idx2, idy2, i2dx, idx, i2dy, idy;
    float fidx2, fidy2, fi2dx, fidx, fi2dy, fidy;
    unsigned int mnx, mnh;
};

// ---------------------------------------------------------------------------
// the stage's scalars, each by one full warp (fwd_static and fwd_offsets spread over lanes)
// ---------------------------------------------------------------------------
// ice_lookup with the snapshot found by ballots: the first index with tt[i] >= t is the number
// of times before t
__device__ __forceinline__ int ice_lookup_warp(const double* __restrict__ tt, int K, int flat, double t, int* i_out,
                                               double* w_out) {
    *w_out = 0.0;
    if (t < tt[0]) {
        *i_out = 0;
        return flat ? FI_OK : FI_ERR_FORCING_RANGE;
    }
    if (t > tt[K - 1]) {
        *i_out = K - 1;
        return flat ? FI_OK : FI_ERR_FORCING_RANGE;
    }
    int lo = 0;
    for (int b = 0; b < K; b += 32) {
        const int i = b + (threadIdx.x & 31);
        const unsigned before = __ballot_sync(0xffffffffu, i < K && tt[i] < t);
        lo += __popc(before);
        if (before != 0xffffffffu) break;
    }
    if (tt[lo] == t) {
        *i_out = lo;
        return FI_OK;
    }
    *i_out = lo - 1;
    *w_out = (t - tt[lo - 1]) / (tt[lo] - tt[lo - 1]);
    return FI_OK;
}

static __device__ __noinline__ void stage_static_warp(const Member& m, Ctl& c, int stage, const double* tice,
                                                      FwdScalars& s) {
    const double t = c.t, dt = c.dt;
    double a1 = 0, a2 = 0, a3 = 0, tr;
    if (stage == 2) { tr = t + C2 * dt; a1 = dt * A21; }
    else if (stage == 3) { tr = t + C3 * dt; a2 = dt * A32; }
    else { tr = t + dt; a1 = dt * A41; a2 = dt * A42; a3 = dt * A43; }
    int ii = 0, status = FI_OK;
    double w = 0.0;
    if (!m.ice_external) status = ice_lookup_warp(tice, m.K, m.ice_flat, tr, &ii, &w);
    const int lane = threadIdx.x & 31;
    // lanes 0..2: the corner means of the two elastic buffers and of the sea surface
    const double* cp = lane == 0 ? c.ue_corner[c.iue] : lane == 1 ? c.ue_corner[c.iue_zb] : c.dz_corner;
    const double cm = cmean(cp, lane < 2 ? m.border_e : m.border_g);
    if (lane == 0) {
        s.a1 = a1; s.a2 = a2; s.a3 = a3;
        s.iue = c.iue;
        s.iuz = c.iue_zb;
        s.dzbsl = c.z_bsl - m.bsl_ref_z;
        s.zbsl = c.z_bsl;
        s.gated = c.gate;
        s.stage = stage;
        s.ik = c.ik;
        s.unew = stage == 4 ? m.u[c.ibuf ^ 1] : nullptr;
        s.status = status;
        s.ice_i = ii;
        s.w = w;
        if (status != FI_OK) c.status = status;
        s.cue = cm;
    } else if (lane == 1) {
        s.cuz = cm;
    } else if (lane == 2) {
        s.cdz = cm;
    }
    __syncwarp();
}

// uc: the four corner values of the state the attempt starts from
static __device__ __noinline__ void stage_offsets_warp(const Member& m, const Ctl& c, const double* uc, FwdScalars& s) {
    const int lane = threadIdx.x & 31, q = lane & 3;
    const double *kc1 = c.kcorner[c.ik], *kc2 = c.kcorner[2], *kc3 = c.kcorner[3];
    const double bv = m.border_v;
    const double c1 = cmean(kc1, bv), c2 = cmean(kc2, bv), c3 = cmean(kc3, bv);
    double v = uc[q];
    if (s.a1 != 0.0) v += s.a1 * (kc1[q] - c1);
    if (s.a2 != 0.0) v += s.a2 * (kc2[q] - c2);
    if (s.a3 != 0.0) v += s.a3 * (kc3[q] - c3);
    double us = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) us += 0.25 * __shfl_sync(0xffffffffu, v, k);
    if (lane == 0) {
        s.c1 = c1; s.c2 = c2; s.c3 = c3;
        s.off = us - bv;
    }
    __syncwarp();
}

// Corner partials of a column task from the edge rows (0 and ny-1) of its nb columns, one set per
// Bsub columns: column_corner_term with a lane per term, summed in its order.  One full warp.
__device__ __forceinline__ void edge_corners_warp(const float2 (*edge)[16], int nx, int kx0, int nb, int Bsub,
                                                  const float2* twx, double* cpart) {
    const int lane = threadIdx.x & 31, q = lane & 3;
    double term[2];
#pragma unroll
    for (int g = 0; g < 2; g++) {
        const int b = 8 * g + (lane >> 2), kx = kx0 + b;
        term[g] = 0.0;
        if (b < nb) {
            const float2 a = edge[q >> 1][b];
            const bool right = q & 1;
            if (kx == 0) {
                term[g] = (double)a.x;
            } else if ((nx % 2 == 0) && kx == nx / 2) {
                term[g] = right ? -(double)a.x : (double)a.x;
            } else if (!right) {
                term[g] = 2.0 * (double)a.x;
            } else {
                const double wr = (double)twx[kx].x, wi = (double)twx[kx].y;
                term[g] = 2.0 * ((double)a.x * wr - (double)a.y * wi);
            }
        }
    }
    double v = 0.0;
    int sub = 0, in_sub = 0;
#pragma unroll 1
    for (int b = 0; b < nb; b++) {
        v += __shfl_sync(0xffffffffu, b < 8 ? term[0] : term[1], 4 * (b & 7) + q);
        if (++in_sub == Bsub || b == nb - 1) {
            if (lane < 4) cpart[4 * sub + lane] = v;
            v = 0.0;
            sub++;
            in_sub = 0;
        }
    }
}

// The sparse update (its phases and barriers) out of line: its transforms would only spread the
// step's code over more instruction-cache lines.
static __device__ __noinline__ bool sparse_update(const Member& m, Ctl& sc, const FftPlan* pl, unsigned char* ws,
                                                  const PersistArgs& a, unsigned int& epoch, int* s_ok,
                                                  unsigned long long* tlast) {
    const int bid = blockIdx.x, G = gridDim.x, tid = threadIdx.x;
    const unsigned int GB = G + a.bar_extra;
    for (int t = bid; t < a.n_crow; t += G) ph_conv_rows(m, pl[2], ws, t, a.h_conv);
    grid_arrive(a.bar);
    if (!grid_wait(a.bar, GB, epoch, s_ok, a.polls)) return false;
    trace_mark(a.trace, tlast, PH_CONV_ROWS);
    for (int t = bid; t < a.n_ccol; t += G) ph_conv_cols(m, pl[3], ws, t, a.B_conv);
    grid_arrive(a.bar);
    if (!grid_wait(a.bar, GB, epoch, s_ok, a.polls)) return false;
    trace_mark(a.trace, tlast, PH_CONV_COLS);
    const int iue = sc.iue;
    for (int t = bid; t < a.n_crowi; t += G)
        ph_conv_rows_inv(m, pl[2], ws, t, a.h_conv, iue, m.ctl->ue_corner[iue], m.ctl->dz_corner);
    grid_arrive(a.bar);
    if (!grid_wait(a.bar, GB, epoch, s_ok, a.polls)) return false;
    trace_mark(a.trace, tlast, PH_CONV_ROWS_INV);
    if (tid < 4) {
        const volatile double* ue_c = m.ctl->ue_corner[iue];
        const volatile double* dz_c = m.ctl->dz_corner;
        sc.ue_corner[iue][tid] = ue_c[tid];
        sc.dz_corner[tid] = dz_c[tid];
    }
    __syncthreads();
    return true;
}

// update_maskgrounded!, update_maskocean!, watercolumn!, columnanom_water! (src/topography.jl:1-28,
// src/loads.jl:56-85) of one cell after the sparse update; returns the seawater anomaly
static __device__ __noinline__ double gated_masks(const Member& m, const FwdScalars& fs, int g, double H, double haf,
                                                  double zdiff, double dzv, double mk) {
    const bool gr = haf > 0.0;
    const double w = -zdiff;  // z_ss - z_b
    const bool oc = w > 0.0 && !gr;
    const double wc = w > 0.0 ? w : 0.0;
    const double hw = (H <= 1.0 ? wc : 0.0) + ((!gr && H > 1.0) ? wc - H / m.rho_sw_ice : 0.0);
    double ssw = 0.0;
    if (m.sl_interactive && oc) ssw = m.rho_sw * (dzv + fs.zbsl) * mk;
    m.sw[g] = (float)ssw;
    m.mgr[g] = gr ? 1.0f : 0.0f;
    m.moc[g] = oc ? 1.0f : 0.0f;
    m.hwater[g] = (float)hw;
    return ssw;
}

// SX, SY: the compiled radix sequences (0: the plans' runtime passes).  RES 1: every optional
// buffer of the layout is in shared memory (the pointers are known to be shared); 0: each may be.
template <int SX, int SY, int RES>
__global__ void __launch_bounds__(res_threads(RES), 1) k_resident(const __grid_constant__ ResArgs ra) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Member sm;
    __shared__ Ctl sc;
    __shared__ FftPlan pl[4];
    __shared__ FwdScalars fs;
    __shared__ ResConst rc;
    __shared__ double s_red[RES_MAX_SUB * (RT / 32)];
    __shared__ double s_uc[2][4];
    __shared__ double s_c4[4];
    __shared__ float2 s_edge[2][16];
    __shared__ int s_ok;
    constexpr int NT = res_threads(RES), NW = NT / 32;
    // Threads that run the transforms.  A single small grid has butterflies for fewer than 384, so
    // the last warps do the scalar work of a phase beside them.
    constexpr int FT = (RES && SX != 0 && SY != 0) ? 384 : NT;
    const PersistArgs& a = ra.p;
    const ResLayout& L = ra.L;
    const int tid = threadIdx.x, bid = blockIdx.x, wid = tid >> 5, lane = tid & 31;
    const unsigned int G = gridDim.x;
    const unsigned int GB = G + a.bar_extra;  // arrivals a grid barrier waits for
    unsigned int epoch = 0;

    // ---- stage the member, the control block, the plans and the ice times ----
    copy_words(&sm, a.mem, sizeof(Member));
    __syncthreads();
    copy_words(&sc, sm.ctl, sizeof(Ctl));  // word by word over the block's threads: used after a barrier
    const Member& m = sm;
    const int nx = m.nx, ny = m.ny, NH = m.NH, h = a.h_rows, sp = m.sp;
    float2* const twx = (float2*)(smem + L.twx);
    float2* const twy = (float2*)(smem + L.twy);
    for (int i = tid; i < nx; i += NT) twx[i] = m.px.tw32[i];
    if (L.twy != L.twx)
        for (int i = tid; i < ny; i += NT) twy[i] = m.py.tw32[i];
    const double* tice = m.t_ice;
    if (L.tice >= 0 && !m.ice_external) {
        double* st = (double*)(smem + L.tice);
        for (int i = tid; i < m.K; i += NT) st[i] = m.t_ice[i];
        tice = st;
    }
    if (tid == 0) {
        pl[0] = m.px; pl[1] = m.py; pl[2] = m.pMx; pl[3] = m.pMy;
        pl[0].tw32 = twx;
        pl[1].tw32 = twy;
        rc.idx2 = 1.0 / (m.dx * m.dx); rc.idy2 = 1.0 / (m.dy * m.dy);
        rc.i2dx = 1.0 / (2 * m.dx); rc.idx = 1.0 / m.dx;
        rc.i2dy = 1.0 / (2 * m.dy); rc.idy = 1.0 / m.dy;
        rc.fidx2 = (float)rc.idx2; rc.fidy2 = (float)rc.idy2;
        rc.fi2dx = (float)rc.i2dx; rc.fidx = (float)rc.idx;
        rc.fi2dy = (float)rc.i2dy; rc.fidy = (float)rc.idy;
        rc.mnx = fastdiv_magic((unsigned)nx);
        rc.mnh = fastdiv_magic((unsigned)NH);
    }
    __syncthreads();
    // ---- segment start: loop header of the first attempt ----
    if (tid == 0) {
        Ctl* c = &sc;
        int active = (c->status == FI_OK) && (c->t < c->t_stop);
        c->pending_output = 0;
        c->nsteps_seg = 0;
        if (active) {
            loopheader_prep(c);
            if (c->status != FI_OK) active = 0;
        }
        c->active = active;
        c->gate = 0;
        if (active) gate_eval(m, c, c->t + C2 * c->dt);
    }
    __syncthreads();
    if (tid < 4) s_uc[0][tid] = __ldcg(&m.u[sc.ibuf][corner_index(tid, nx, ny)]);

    // ---- this block's row tile ----
    const bool rows_on = bid < a.n_rows;
    const int ty0 = !rows_on ? 0 : ra.tail && bid == a.n_rows - 1 ? ny - 1 : bid * h;
    const RowRanges rr = row_ranges_of(ty0, ty0 == ny - 1 ? ny : min(ty0 + h, ny - ra.tail), ny);
    const int y0 = rr.y0, y1 = rr.y1, loU = rr.loU, loT = rr.loM;
    const int nU = rr.hiU - loU, n_own = (y1 - y0) * nx, own0 = (y0 - loU) * nx;
    const unsigned int mnx = rc.mnx;
    const bool resU = RES || L.P0 >= 0, resK = RES || L.KA0 >= 0, resB = RES || L.KB >= 0, resC = RES || L.KC >= 0;
    float2* const MS = (float2*)(smem + L.MS);
    float2* const F = (float2*)(smem + L.F);
    float* const KB = (float*)(smem + (resB ? L.KB : 0));
    float* const KC = (float*)(smem + (resC ? L.KC : 0));
    // byte offsets of uprev / k1 of the attempt and of the stage vector / k4 (exchanged on acceptance)
    int oU = resU ? L.P0 : L.P1, oV = L.P1, oK1 = resK ? L.KA0 : 0, oK4 = resK ? L.KA1 : 0;
    int ice_key = -1, ue_ver = -1;  // what the resident ice and elastic rows hold
    if (rows_on) {
        if (resU) copy_words(smem + oU, m.u[sc.ibuf] + (size_t)loU * nx, nU * nx * 8);
        if (resK)
            for (int i = tid; i < nU * nx; i += NT) ((float*)(smem + oK1))[i] = m.k14[sc.ik][(size_t)loU * nx + i];
        if (RES || L.D >= 0)
            for (int i = tid; i < (rr.hiM - loT) * nx; i += NT)
                ((float*)(smem + L.D))[i] = m.D[(size_t)loT * nx + i];
        if (RES || L.visc >= 0)
            for (int i = tid; i < n_own; i += NT) ((float*)(smem + L.visc))[i] = m.visc_fac[(size_t)y0 * nx + i];
    }
    if (RES || L.mult >= 0) {  // resident only when every block has one column task
        const int kx0 = bid * a.B_cols, nb = min(a.B_cols, NH - kx0);
        for (int i = tid; i < nb * ny; i += NT) ((float*)(smem + L.mult))[i] = m.mult[(size_t)kx0 * ny + i];
    }
    bool ok = true;
    unsigned long long* trace = a.trace;
    unsigned long long tlast = (trace && bid == 0 && tid == 0) ? globaltimer_ns() : 0ull;
    __syncthreads();
    if (wid == 0 && sc.active && !sc.gate) {
        stage_static_warp(m, sc, 2, tice, fs);
        stage_offsets_warp(m, sc, s_uc[0], fs);
    }
    __syncthreads();

    while (sc.active && ok) {
#pragma unroll 1
        for (int stage = 2; stage <= 5; stage++) {
            // stage 5: k4 and the error norm.  The grid barrier behind the previous phase
            // has been waited for.
            if (stage < 5 && sc.gate) {
                // the convolutions read the column anomalies of the last call
                ok = sparse_update(m, sc, pl, (unsigned char*)MS, a, epoch, &s_ok, &tlast);
                if (!ok) break;
                ue_ver = -1;
                if (wid == 0) {
                    stage_static_warp(m, sc, stage, tice, fs);
                    if (stage == 2) stage_offsets_warp(m, sc, s_uc[0], fs);
                }
                __syncthreads();
            }
            const int inv = stage > 2;
            const int lo = stage == 5 ? y0 : loU, hi = stage == 5 ? y1 : loU + nU;
            const int npi = (hi - lo + 1) / 2;  // row pairs inverted (or combined) here
            if (inv) {
                // corner values of the previous stage's field: the last four warps sum the column
                // tasks' partials in the order of corners_from_partials; then one of them takes them
                // over and sets the stage vector's offsets
                auto corner_sums = [&]() {
                    const double* cp = m.cpart + (wid - (NW - 4));
                    double acc = 0.0;
                    for (int t = lane; t < m.ncols; t += 32) acc += __ldcg(cp + 4 * t);
                    acc = warp_sum(acc);
                    if (lane == 0) s_c4[wid - (NW - 4)] = acc;
                };
                auto take_corners = [&]() {
                    if (lane < 4) sc.kcorner[stage == 3 ? 2 : stage == 4 ? 3 : sc.ik ^ 1][lane] = s_c4[lane];
                    __syncwarp();
                    if (stage < 5) stage_offsets_warp(m, sc, s_uc[0], fs);
                };
                // inverse real row transform of the previous stage, two rows per complex FFT;
                // ping-pong between MS and a dead buffer, the result in MS
                const float2* Sp = m.S[stage == 4 ? 1 : 0] + (size_t)lo * sp;
                float2* const other = stage == 5 ? F : (float2*)(smem + oV);
                const int nrow = hi - lo;
                auto pair = [&](int p, int k) {
                    const int kk = (k < NH) ? k : nx - k;
                    const float2* Sa = Sp + (size_t)(2 * p) * sp + kk;
                    const float2 A = __ldcg(Sa);
                    const float2 B = (2 * p + 1 < nrow) ? __ldcg(Sa + sp) : make_float2(0.0f, 0.0f);
                    return (k < NH) ? make_float2(A.x - B.y, A.y + B.x) : make_float2(A.x + B.y, -A.y + B.x);
                };
                if constexpr (SX != 0) {
                    constexpr int NP = seq_npass(SX), R0 = seq_radix(SX, 0);
                    float2* first = (NP % 2) ? MS : other;
                    float2* second = (NP % 2) ? other : MS;
                    auto pass0 = [&]() {
                        fn_pass<FT, R0, true, seq_len(SX), 1, false>(
                            twx, npi, 0u, pair, [&](int b, int i, float2 v) { first[b * nx + i] = v; });
                    };
                    if constexpr (FT < NT) {
                        if (tid < FT) {
                            if (rows_on) {
                                pass0();
                                group_sync<FT>();
                                sm_passes<FT, true, SX, 1, NP, R0>(first, second, twx, npi, nx);
                            }
                        } else if (wid >= NW - 4) {
                            corner_sums();
                            asm volatile("bar.sync 2, 128;" ::: "memory");
                            if (wid == NW - 1) take_corners();
                        }
                        __syncthreads();
                    } else {
                        if (wid >= NW - 4) corner_sums();
                        if (rows_on) pass0();
                        __syncthreads();
                        if (wid == NW - 1) take_corners();
                        if (rows_on) sm_passes<FT, true, SX, 1, NP, R0>(first, second, twx, npi, nx);
                        __syncthreads();
                    }
                } else {
                    float2* first = (pl[0].npass % 2) ? other : MS;
                    float2* second = (pl[0].npass % 2) ? MS : other;
                    if (wid >= NW - 4) corner_sums();
                    if (rows_on)
                        for (int i = tid; i < npi * nx; i += NT) {
                            const int p = (int)fastdiv((unsigned)i, (unsigned)nx, mnx);
                            first[i] = pair(p, i - p * nx);
                        }
                    __syncthreads();
                    if (wid == NW - 1) take_corners();
                    if (rows_on) fft_batch<true, float>(first, second, pl[0], npi, nx);
                    __syncthreads();
                }
            }
            if (stage == 5) break;

            if (rows_on) {
                // ---- 1: stage vector rows [loU, hiU) in FP64, corner BC ----
                double* const sU = (double*)(smem + oV);
                {
                    float* const kdst = (stage == 3 ? m.k2 : m.k3) + (size_t)loU * nx;
                    const double a1 = fs.a1, a2 = fs.a2, a3 = fs.a3, c1 = fs.c1, c2 = fs.c2, c3 = fs.c3, off = fs.off;
                    const double* up = resU ? (const double*)(smem + oU) : m.u[sc.ibuf] + (size_t)loU * nx;
                    const float* k1 = resK ? (const float*)(smem + oK1) : m.k14[sc.ik] + (size_t)loU * nx;
                    const float* k2 = resB ? KB : m.k2 + (size_t)loU * nx;
                    // one element: kv is the derivative inverted here (k2 or k3)
                    auto combine = [&](int e, float kv) {
                        double u = up[e];
                        if (a1 != 0.0) u += a1 * ((double)k1[e] - c1);
                        if (a2 != 0.0) u += a2 * ((double)(stage == 3 ? kv : k2[e]) - c2);
                        if (a3 != 0.0) u += a3 * ((double)kv - c3);
                        sU[e] = u - off;
                    };
                    if (!inv) {
#pragma unroll 2
                        for (int e = tid; e < nU * nx; e += NT) combine(e, 0.0f);
                    } else {
#pragma unroll 1
                        for (int i = tid; i < npi * nx; i += NT) {
                            const int p = (int)fastdiv((unsigned)i, (unsigned)nx, mnx);
                            const float2 z = MS[i];
#pragma unroll
                            for (int q = 0; q < 2; q++) {
                                const int e = i + (p + q) * nx;  // row 2p + q, column i - p nx
                                if (e < nU * nx) {
                                    const float kv = q ? z.y : z.x;
                                    const bool own = e >= own0 && e < own0 + n_own;
                                    if (own) kdst[e] = kv;
                                    if (stage == 3) {
                                        if (resB) KB[e] = kv;
                                    } else if (resC && own) {
                                        KC[e - own0] = kv;
                                    }
                                    combine(e, kv);
                                }
                            }
                        }
                    }
                }
                // the ice snapshots and the elastic and sea-surface rows of this call
                const float* Hg =
                    (m.ice_external ? m.H_ext : m.H_tab + (size_t)fs.ice_i * nx * ny) + (size_t)y0 * nx;
                const float* ueg = m.ue[fs.iue] + (size_t)y0 * nx;
                const float* dzg = m.dz + (size_t)y0 * nx;
                if (RES || L.Ha >= 0) {
                    const int key = 2 * fs.ice_i + (fs.w != 0.0);
                    if (key != ice_key) {
                        for (int i = tid; i < n_own; i += NT) {
                            ((float*)(smem + L.Ha))[i] = Hg[i];
                            if (fs.w != 0.0) ((float*)(smem + L.Hb))[i] = Hg[(size_t)nx * ny + i];
                        }
                        ice_key = key;
                    }
                }
                if (RES || L.ue >= 0) {
                    if (ue_ver != fs.iue) {
                        for (int i = tid; i < n_own; i += NT) {
                            ((float*)(smem + L.ue))[i] = ueg[i];
                            ((float*)(smem + L.dz))[i] = dzg[i];
                        }
                        ue_ver = fs.iue;
                    }
                }
                const float* vHa = (RES || L.Ha >= 0) ? (const float*)(smem + L.Ha) : Hg;
                const float* vHb = (RES || L.Ha >= 0) ? (const float*)(smem + L.Hb) : Hg + (size_t)nx * ny;
                const float* vue = (RES || L.ue >= 0) ? (const float*)(smem + L.ue) : ueg;
                const float* vdz = (RES || L.ue >= 0) ? (const float*)(smem + L.dz) : dzg;
                const float* vD = (RES || L.D >= 0) ? (const float*)(smem + L.D) : m.D + (size_t)loT * nx;
                const float* vvisc = (RES || L.visc >= 0) ? (const float*)(smem + L.visc) : m.visc_fac + (size_t)y0 * nx;
                const bool uz_old = fs.iuz != fs.iue;  // a gated call: z_b reads the previous buffer
                const float* uzg = m.ue[fs.iuz] + (size_t)y0 * nx;
                __syncthreads();
                // ---- chunks of own rows: moments and column anomalies, then the moment divergence ----
                const int chunk = RES ? h : L.chunk;
                float* const sMxx = (float*)MS;
                float* const sMyy = sMxx + capM_of(chunk) * nx;
                float* const sMxy = sMyy + capM_of(chunk) * nx;
#pragma unroll 1
                for (int cy0 = y0; cy0 < y1; cy0 += chunk) {
                    const int cy1 = min(cy0 + chunk, y1);
                    int loM = cy0 == 0 ? 0 : cy0 - 1, hiM = cy1 == ny ? ny : cy1 + 1;
                    if (cy0 == 0) hiM = max(hiM, min(ny, 3));
                    if (cy1 == ny) loM = min(loM, ny - 3);
                    const int nM = (hiM - loM) * nx;
                    // 2a: bending moments on rows [loM, hiM) (u-derivatives in FP64)
                    {
                        const double nu = m.nu, idx2 = rc.idx2, idy2 = rc.idy2;
                        const double* const Ub0 = sU + (loM - loU) * nx;
                        const float* const Db0 = vD + (loM - loT) * nx;
#pragma unroll 1
                        for (int i = tid; i < nM; i += NT) {
                            const int rl = (int)fastdiv((unsigned)i, (unsigned)nx, mnx);
                            const int x = i - rl * nx, r = loM + rl;
                            const double* Ur = Ub0 + i;  // (r, x)
                            const bool top = r == 0, bot = r == ny - 1;
                            const double* U0 = top ? Ur + nx : bot ? Ur - nx : Ur;
                            const double* Ua = bot ? Ur : Ur + nx;
                            const double* Ub = top ? Ur : Ur - nx;
                            const bool xl = x == 0, xr = x == nx - 1, xe = xl || xr;
                            const int oc = xl ? 1 : xr ? -1 : 0;
                            const double uxx = (Ur[oc + 1] - 2.0 * Ur[oc] + Ur[oc - 1]) * idx2;
                            const double uyy = (U0[nx] - 2.0 * U0[0] + U0[-nx]) * idy2;
                            const int xp = xr ? 0 : 1, xm = xl ? 0 : -1;
                            const double sx = xe ? rc.idx : rc.i2dx, sy = (top || bot) ? rc.idy : rc.i2dy;
                            // products rounded before the difference, as with a branch per edge
                            const double da = __dmul_rn(Ua[xp] - Ua[xm], sx), db = __dmul_rn(Ub[xp] - Ub[xm], sx);
                            const double uxy = (da - db) * sy;
                            const double D = (double)Db0[i];
                            sMxx[i] = (float)(-D * (nu * uyy + uxx));
                            sMyy[i] = (float)(-D * (nu * uxx + uyy));
                            sMxy[i] = (float)(-D * (1.0 - nu) * uxy);
                        }
                    }
                    // 2b: column anomalies of the chunk's rows; -g sigma_full to F (the place of the
                    // element's right-hand side)
                    {
                        const double cue = fs.cue, cuz = fs.cuz, cdz = fs.cdz, dzbsl = fs.dzbsl;
                        const float fw = (float)fs.w;
                        double* const unew = fs.unew;
                        const int flags = m.flags, gated = fs.gated;
                        const double rho_sw_ice = m.rho_sw_ice, rho_ice = m.rho_ice, rho_litho = m.rho_litho,
                                     rho_um = m.rho_um, mg = -m.g, mA = m.A;
                        const float zbs = m.zbss_scalar;
                        const int i0 = (cy0 - y0) * nx, i1 = (cy1 - y0) * nx;
                        float* const Ff = (float*)F;
                        // start with the threads that the moment rows left idle
#pragma unroll 1
                        for (int i = i0 + (tid + NT - nM % NT) % NT; i < i1; i += NT) {
                            const int g = y0 * nx + i;
                            const int rl = (int)fastdiv((unsigned)i, (unsigned)nx, mnx);
                            const double u = sU[own0 + i];
                            const float ha = vHa[i];
                            const double H = (double)(fw != 0.0f ? ha + (vHb[i] - ha) * fw : ha);
                            const double uev = (double)vue[i] - cue;
                            const double dzv = (double)vdz[i] - cdz;
                            const double uzv = (double)(uz_old ? uzg[i] : vue[i]);
                            const double zdiff = (double)((flags & FLAG_ZBSS) ? m.zbss_ref[g] : zbs) +
                                                 (uzv - cuz) + u - dzv - dzbsl;
                            double haf = H + (zdiff < 0.0 ? zdiff : 0.0) * rho_sw_ice;
                            haf = haf > 0.0 ? haf : 0.0;
                            const double mk = (flags & FLAG_MASK) ? (double)m.mask[g] : 1.0;
                            const double hafref = (flags & FLAG_HAFREF) ? (double)m.H_af_ref[g] : 0.0;
                            double ssw = 0.0;
                            if (gated) {
                                ssw = gated_masks(m, fs, g, H, haf, zdiff, dzv, mk);
                            } else if (m.sl_interactive) {
                                ssw = (double)m.sw[g];
                            }
                            const double sload = mk * (rho_ice * (haf - hafref) + ssw);
                            double sfull = mk * (rho_ice * haf + rho_litho * uev + rho_um * u + ssw);
                            if (flags & FLAG_SIGREF) sfull -= (double)m.sigma_ref[g];
                            m.sig_load[g] = (float)sload;
                            double geo = sfull;
                            if (m.column_compressible) {
                                // A (sigma_load + m sigma_mantle) = A (sigma_full - m sigma_litho), sealevel.jl:193-197
                                const double uer = (flags & FLAG_UEREF) ? (double)m.ue_ref[g] : 0.0;
                                geo = sfull - mk * rho_litho * (uev - uer);
                            }
                            m.sig_geo[g] = (float)(mA * geo);
                            // row rl, column i - rl nx -> pair rl / 2, component rl % 2
                            Ff[2 * (i - (rl - (rl >> 1)) * nx) + (rl & 1)] = (float)(mg * sfull);
                            if (unew) unew[g] = u;
                        }
                    }
                    __syncthreads();
                    // 3: moment divergence in FP32 -> f = rhs * K/(2 eta), rows packed in pairs
                    {
                        const float idx2 = rc.fidx2, idy2 = rc.fidy2;
                        const int p0 = (cy0 - y0) >> 1, np = (cy1 - cy0 + 1) >> 1;
#pragma unroll 1
                        for (int i = tid; i < np * nx; i += NT) {
                            const int p = (int)fastdiv((unsigned)i, (unsigned)nx, mnx);
                            const int x = i - p * nx;
                            const bool xl = x == 0, xr = x == nx - 1;
                            const int oc = xl ? 1 : xr ? -1 : 0, xp = xr ? 0 : 1, xm = xl ? 0 : -1;
                            const float sx = (xl || xr) ? rc.fidx : rc.fi2dx;
                            float2 f = F[p0 * nx + i];
#pragma unroll
                            for (int q = 0; q < 2; q++) {
                                const int rv = cy0 + 2 * p + q;
                                float fv = 0.0f;
                                if (rv < cy1) {
                                    const int ro = (rv - loM) * nx + x;
                                    const bool top = rv == 0, bot = rv == ny - 1;
                                    const float* Mx = sMxx + ro;
                                    const float* My0 = sMyy + (top ? ro + nx : bot ? ro - nx : ro);
                                    const float* Ma = sMxy + (bot ? ro : ro + nx);
                                    const float* Mb = sMxy + (top ? ro : ro - nx);
                                    const float sy = (top || bot) ? rc.fidy : rc.fi2dy;
                                    const float mxx = (Mx[oc + 1] - 2.0f * Mx[oc] + Mx[oc - 1]) * idx2;
                                    const float myy = (My0[nx] - 2.0f * My0[0] + My0[-nx]) * idy2;
                                    const float da = __fmul_rn(Ma[xp] - Ma[xm], sx);
                                    const float db = __fmul_rn(Mb[xp] - Mb[xm], sx);
                                    const float mxy = (da - db) * sy;
                                    const float rhs = (q ? f.y : f.x) + (mxx + (2.0f * mxy + myy));
                                    fv = rhs * vvisc[(rv - y0) * nx + x];
                                }
                                if (q) f.y = fv; else f.x = fv;
                            }
                            F[p0 * nx + i] = f;
                        }
                    }
                    __syncthreads();
                }
                // ---- forward row transforms, split into the rows' half spectra ----
                const int np = (y1 - y0 + 1) / 2;
                const float2* res;
                if constexpr (SX != 0) {
                    if (FT == NT || tid < FT) sm_passes<FT, false, SX, 0, seq_npass(SX), 1>(F, MS, twx, np, nx);
                    if constexpr (FT < NT) __syncthreads();
                    res = (seq_npass(SX) % 2) ? MS : F;
                } else {
                    res = fft_batch<false, float>(F, MS, pl[0], np, nx);
                }
                float2* Sout = m.S[stage == 3 ? 1 : 0] + (size_t)y0 * sp;
                const unsigned int mnh = rc.mnh;
#pragma unroll 1
                for (int i = tid; i < np * NH; i += NT) {
                    const int p = (int)fastdiv((unsigned)i, (unsigned)NH, mnh);
                    const int kx = i - p * NH;
                    float2* Sa = Sout + (size_t)(2 * p) * sp + kx;
                    const float2 Z = res[p * nx + kx];
                    const float2 Zc = res[p * nx + (kx == 0 ? 0 : nx - kx)];
                    Sa[0] = make_float2(0.5f * (Z.x + Zc.x), 0.5f * (Z.y - Zc.y));
                    if (y0 + 2 * p + 1 < y1) Sa[sp] = make_float2(0.5f * (Z.y + Zc.y), -0.5f * (Z.x - Zc.x));
                }
            }
            grid_arrive(a.bar);
            // while the others arrive: count the call, evaluate the gate of the next one and, unless
            // it is open, set the next stage's scalars
            if (wid == NW - 1) {
                if (lane == 0) {
                    sc.nf += 1;
                    if (stage < 4) gate_eval(m, &sc, sc.t + (stage == 2 ? C3 : 1.0) * sc.dt);
                }
                __syncwarp();
                if (stage < 4 && !sc.gate) stage_static_warp(m, sc, stage + 1, tice, fs);
            }
            if (!(ok = grid_wait(a.bar, GB, epoch, &s_ok, a.polls))) break;
            trace_mark(trace, &tlast, PH_ROWS_FWD2 + 2 * (stage - 2));
            // ---- columns ----
            if (stage == 3 && resB && rows_on && (FT == NT || tid >= FT)) {
                // the halo rows of k2 as their owners computed them (another pairing of rows
                // rounds differently)
                constexpr int NA = FT < NT ? NT - FT : NT;
                const int nhalo = nU * nx - n_own;
                const float* kg = m.k2 + (size_t)loU * nx;
#pragma unroll 4
                for (int j = tid - (NT - NA); j < nhalo; j += NA) {
                    const int i = j < own0 ? j : j + n_own;
                    KB[i] = __ldcg(kg + i);
                }
            }
            float2* const Sc = m.S[stage == 3 ? 1 : 0];
            for (int tc = bid; tc < a.n_cols; tc += G) {
                const int kx0 = tc * a.B_cols, nb = min(a.B_cols, NH - kx0);
                if constexpr (SY != 0) {
                    constexpr int NP = seq_npass(SY), R0 = seq_radix(SY, 0), RL = seq_radix(SY, NP - 1);
                    constexpr int LL = seq_len(SY), PITCH = LL + 1;  // +1: columns start in different banks
                    if (FT == NT || tid < FT) {
                        const unsigned int mnb = fastdiv_magic((unsigned)nb);
                        float2* const b0 = MS;
                        float2* const b1 = MS + a.B_cols * PITCH;
                        float2* const Sk = Sc + kx0;
                        const float* const mk =
                            (RES || L.mult >= 0) ? (const float*)(smem + L.mult) : m.mult + (size_t)kx0 * ny;
                        fn_pass<FT, R0, false, LL, 1, true>(
                            twy, nb, mnb, [&](int b, int i) { return __ldcg(Sk + (size_t)i * sp + b); },
                            [&](int b, int i, float2 v) { b0[b * PITCH + i] = v; });
                        group_sync<FT>();
                        sm_passes<FT, false, SY, 1, NP - 1, R0>(b0, b1, twy, nb, PITCH);
                        float2* const c0 = ((NP - 2) % 2) ? b1 : b0;
                        float2* const c1 = ((NP - 2) % 2) ? b0 : b1;
                        fn_pass<FT, RL, false, LL, LL / RL, false>(
                            twy, nb, 0u, [&](int b, int i) { return c0[b * PITCH + i]; },
                            [&](int b, int i, float2 v) {
                                const float s = mk[b * LL + i];
                                c1[b * PITCH + i] = make_float2(v.x * s, v.y * s);
                            });
                        group_sync<FT>();
                        sm_passes<FT, true, SY, 0, NP - 1, 1>(c1, c0, twy, nb, PITCH);
                        float2* const d0 = ((NP - 1) % 2) ? c0 : c1;
                        fn_pass<FT, RL, true, LL, LL / RL, true>(
                            twy, nb, mnb, [&](int b, int i) { return d0[b * PITCH + i]; },
                            [&](int b, int i, float2 v) {
                                Sk[(size_t)i * sp + b] = v;
                                if (i == 0) s_edge[0][b] = v;
                                if (i == LL - 1) s_edge[1][b] = v;
                            });
                        group_sync<FT>();
                        if (wid == 0)
                            edge_corners_warp(s_edge, nx, kx0, nb, ra.B_sub, twx,
                                              m.cpart + 4 * tc * (a.B_cols / ra.B_sub));
                        if (tc + (int)G < a.n_cols) group_sync<FT>();
                    }
                } else {
                    ph_cols<0>(m, pl[1], twx, (unsigned char*)MS, tc, a.B_cols, ra.B_sub, Sc, m.cpart);
                }
            }
            grid_arrive(a.bar);
            if (!(ok = grid_wait(a.bar, GB, epoch, &s_ok, a.polls))) break;
            trace_mark(trace, &tlast, PH_COLS2 + 2 * (stage - 2));
        }
        if (!ok) break;
        // ---- k4 rows (in MS) and the embedded error norm ----
        const int ik = sc.ik, ibuf = sc.ibuf;
        if (rows_on) {
            const double dt = sc.dt, abstol = sc.abstol, reltol = sc.reltol;
            const double cc1 = cmean(sc.kcorner[ik], m.border_v), cc2 = cmean(sc.kcorner[2], m.border_v);
            const double cc3 = cmean(sc.kcorner[3], m.border_v), cs = cmean(s_c4, m.border_v);
            const size_t g0 = (size_t)y0 * nx;
            const float* k1 = resK ? (const float*)(smem + oK1) + own0 : m.k14[ik] + g0;
            const float* k2 = resB ? KB + own0 : m.k2 + g0;
            const float* k3 = resC ? KC : m.k3 + g0;
            const double* up = resU ? (const double*)(smem + oU) + own0 : m.u[ibuf] + g0;
            const double* un = resU ? (const double*)(smem + oV) + own0 : m.u[ibuf ^ 1] + g0;
            float* const k4 = (float*)(smem + oK4) + own0;
            float* const dst = m.k14[ik ^ 1] + g0;
            // one partial per ra.h_sub rows, each summed in the order of block_sum
            const int n_sub = ra.h_sub * nx;
            int nsub = 0;
#pragma unroll 1
            for (int s0 = 0; s0 < n_own; s0 += n_sub, nsub++) {
                double acc = 0.0;
                const int s1 = min(s0 + n_sub, n_own);
                // the first RT threads, so that each sums the elements it does in the other executors
#pragma unroll 1
                for (int i = s0 + (tid < RT ? tid : s1); i < s1; i += RT) {
                    const int rl = (int)fastdiv((unsigned)i, (unsigned)nx, mnx);
                    const float2 z = MS[i - (rl - (rl >> 1)) * nx];
                    const float v = (rl & 1) ? z.y : z.x;
                    dst[i] = v;
                    if (resK) k4[i] = v;
                    const double ut = dt * (BT1 * ((double)k1[i] - cc1) + BT2 * ((double)k2[i] - cc2) +
                                            BT3 * ((double)k3[i] - cc3) + BT4 * ((double)v - cs));
                    const double ua = fabs(up[i]), ub = fabs(un[i]);
                    const double e = ut / (abstol + (ua > ub ? ua : ub) * reltol);
                    acc += e * e;
                }
                acc = warp_sum(acc);
                if (lane == 0 && wid < RT / 32) s_red[nsub * (RT / 32) + wid] = acc;
            }
            __syncthreads();
            if (tid < nsub) {
                double s = 0.0;
#pragma unroll
                for (int w = 0; w < RT / 32; w++) s += s_red[tid * (RT / 32) + w];
                m.partial[y0 / ra.h_sub + tid] = s;
            }
        }
        grid_arrive(a.bar);
        if (!(ok = grid_wait(a.bar, GB, epoch, &s_ok, a.polls))) break;
        trace_mark(trace, &tlast, PH_ROWS_INV4);
        // ---- step controller, replicated (warp 0), beside the halo rows of the new state, in case
        // the step is accepted ----
        if (wid == 0) {
            if (lane < 4) s_uc[1][lane] = __ldcg(&m.u[ibuf ^ 1][corner_index(lane, nx, ny)]);
            const double acc = partials_sum(m.partial, ra.n_part);
            finish_attempt_warp(m, &sc, sqrt(acc / ((double)nx * ny)));
            __syncwarp();
            if (sc.accept_step && lane < 4) s_uc[0][lane] = s_uc[1][lane];
            __syncwarp();
            if (sc.active && !sc.gate) {
                stage_static_warp(m, sc, 2, tice, fs);
                stage_offsets_warp(m, sc, s_uc[0], fs);
            }
        } else if (rows_on && (resU || resK)) {
            // halo element j: rows above the own rows, then rows below (ibuf, ik: this attempt's)
            const int nhalo = nU * nx - n_own;
            const size_t g0 = (size_t)loU * nx;
            const double* un = m.u[ibuf ^ 1] + g0;
            const float* kn = m.k14[ik ^ 1] + g0;
#pragma unroll 2
            for (int j = tid - 32; j < nhalo; j += NT - 32) {
                const int i = j < own0 ? j : j + n_own;
                if (resU) ((double*)(smem + oV))[i] = __ldcg(un + i);
                if (resK) ((float*)(smem + oK4))[i] = __ldcg(kn + i);
            }
        }
        __syncthreads();
        if (sc.accept_step) {
            if (resU) { const int o = oU; oU = oV; oV = o; }
            if (resK) { const int o = oK1; oK1 = oK4; oK4 = o; }
        }
        trace_mark(trace, &tlast, PH_CONTROLLER);
    }
    if (!ok && tid == 0) sc.status = FI_ERR_TIMEOUT;
    __syncthreads();
    if (bid == 0) copy_words(m.ctl, &sc, sizeof(Ctl));
}

}  // namespace fi
