// fno.cu -- Fourier neural operator (FNO) surrogate of the LV-ELVA solver: forward pass,
// its adjoint (backward pass), Adam, all on the device.
//
// Network (fixed shape, S x S grid, S a multiple of 32 in [32, 256]):
//   input 6 channels -> lift (pointwise 6 -> 32) -> 4 Fourier layers of width 32
//   -> projection (pointwise 32 -> 128, GELU, 128 -> 1).
//   Fourier layer: z = SpectralConv(v) + Wloc v + b;  v' = GELU(z) (identity after the last).
//   SpectralConv keeps kx in [0, 16) (half axis, x) and ky in {0..15, S-16..S-1} (full axis,
//   y): 512 complex modes, one complex 32 x 32 channel matrix per mode; the inverse is the
//   real inverse DFT of that truncated half spectrum (weight 1 at kx = 0, 2 otherwise, 1/S^2).
//
// Every contraction but the per-mode weight gradient runs on the tensor cores (tcgen05, BF16
// operands, FP32 accumulators in tensor memory), on the GEMM of fno_gemm.cuh unless a kernel is named:
//   DFT along x:   v[(b,c,y)][x]            x F1[(part,kx)][x]            -> T
//   DFT along y:   T[(kx,b,c)][(part,y)]    x F2[(kyi,part')][(part,y)]   -> Z (per mode)
//                  (k_dft2: both at once, up to S = 128)
//   channel mix:   Z[mode][b][(part,ci)]    x Wmat[mode][(part',co)][(part,ci)]  (512 batches)
//   inverse y:     Y[(b,co,kx)][(kyi,part)] x G2[(y,part')][(kyi,part)]   -> G[(b,y)][co][(kx,part)]
//   inverse x + pointwise path, one product per row (b, y) of pixels x channels with K = 32 + 32 (k_pix):
//                  [G1[x][(kx,part)] | v[b][ci][y][x]]  x  [G[(b,y)][co][(kx,part)] | Wloc[co][ci]]
//                  (the activation v read in place from NCHW as an MN-major operand)
// The backward pass runs the same products against the transposed matrices.  The weight gradients of
// the pointwise layers are split-K products over pixels whose B operand carries a row of ones (bias
// gradient; k_wgrad) and, for the projection, the loss gradient (dQ2; k_proj_bwd).
//
// Activations live in NCHW ([b][c][y*S+x]) only: the pointwise layers and the projection
// read them as MN-major operands (pixels x channels).  All parameters are FP32 masters
// (Adam), packed to BF16 operand copies after each update.
#include <cmath>
#include <cstdio>
#include <string>
#include <vector>

#include "../../include/fastiso_b200.h"
#include "fno_gemm.cuh"

namespace fi {
namespace fno {

typedef __nv_bfloat16 bf16;

constexpr int C = 32;         // width
constexpr int KX = 16;        // kept kx
constexpr int KY = 32;        // kept ky (kyi < 16: ky = kyi; else ky = S - 32 + kyi)
constexpr int NM = KX * KY;   // complex modes per layer
constexpr int NIN = 6;        // input channels
constexpr int XC = 8;         // padded input channels (6 inputs, ones, zero)
constexpr int VC = 34;        // channels of an NCHW activation buffer: 32, ones, loss gradient
constexpr int PW = 128;       // projection width
constexpr int NLAYER = 4;
constexpr long long SPEC = (long long)NM * 2 * C * C;  // [mode][re, im][ci][co]
constexpr long long LAYER = SPEC + C * C + C;          // spectral, Wloc[co][ci], bloc[co]

// offsets into the flat FP32 parameter (and gradient) vector
struct Offsets {
    long long P, bP, layer[NLAYER], Q1, b1, Q2, b2, total;
};

inline Offsets offsets() {
    Offsets o;
    o.P = 0;                // [32][6]
    o.bP = C * NIN;         // [32]
    long long p = o.bP + C;
    for (int l = 0; l < NLAYER; l++) {
        o.layer[l] = p;
        p += LAYER;
    }
    o.Q1 = p;               // [128][32]
    o.b1 = o.Q1 + PW * C;   // [128]
    o.Q2 = o.b1 + PW;       // [128]
    o.b2 = o.Q2 + PW;       // [1]
    o.total = o.b2 + 1;
    return o;
}

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------
// GELU(a) = a Phi(a), Phi the standard normal distribution function
__device__ __forceinline__ float gelu(float a) { return 0.5f * a * (1.f + erff(a * 0.70710678118654752f)); }
// GELU and GELU'(a) = Phi(a) + a phi(a), Phi evaluated once
__device__ __forceinline__ void gelu_both(float a, float& g, float& gp) {
    const float Phi = 0.5f * (1.f + erff(a * 0.70710678118654752f));
    g = a * Phi;
    gp = Phi + a * 0.39894228040143268f * expf(-0.5f * a * a);
}
__device__ __forceinline__ float gelu_grad(float a) {
    float g, gp;
    gelu_both(a, g, gp);
    return gp;
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
// 16 values as BF16 to a 32-byte aligned address
__device__ __forceinline__ void store16(bf16* dst, const float* v) {
    uint4* d = reinterpret_cast<uint4*>(dst);
    d[0] = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
    d[1] = make_uint4(pack2(v[8], v[9]), pack2(v[10], v[11]), pack2(v[12], v[13]), pack2(v[14], v[15]));
}

// ---------------------------------------------------------------------------
// GEMM epilogues (called per row and 16-column chunk; every N below is a multiple of 16)
// ---------------------------------------------------------------------------

// 16 consecutive parameters at a multiple of 16 floats (every group's offset is a multiple of 32).  The
// non-coherent loads hold: parameters change in k_adam and in the host's copies alone, and a call ends
// with a wait for both before another pass starts.  As
// single loads beside each value's arithmetic they were two of a hidden unit's loads and waits:
// 32 samples of 128 x 128, inference 482 -> 468 us, training step 1196 -> 1174 us.
__device__ __forceinline__ void load16(float* d, const float* __restrict__ p) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p) + q);
        d[4 * q] = t.x; d[4 * q + 1] = t.y; d[4 * q + 2] = t.z; d[4 * q + 3] = t.w;
    }
}

// lift: batch z = b, row p, col c -> v0 in NCHW
struct EpiLift {
    static constexpr bool PAIR = false;
    bf16* vext;
    const float* bias;
    int S2;
    __device__ __forceinline__ void operator()(int z, int p, int c0, const float* v, int) const {
        bf16* o = vext + ((size_t)z * VC + c0) * S2 + p;
        float bc[16];
        load16(bc, bias + c0);
#pragma unroll
        for (int i = 0; i < 16; i++) o[(size_t)i * S2] = __float2bfloat16_rn(v[i] + bc[i]);
    }
    __device__ __forceinline__ void row_done(int, int) const {}
};

// DFT along x and the adjoint of the inverse along x: batch z = b, row (c, y), col n = part*16 + kx,
// out T[kx][b][c][part][y]
struct EpiDftX {
    static constexpr bool PAIR = false;
    bf16* T;
    int B, S;
    __device__ __forceinline__ void operator()(int b, int row, int n0, const float* v, int) const {
        const int c = row / S, y = row - c * S, part = n0 >> 4;
#pragma unroll
        for (int i = 0; i < 16; i++)
            T[(((size_t)i * B + b) * C + c) * 2 * S + part * S + y] = __float2bfloat16_rn(v[i]);
    }
    __device__ __forceinline__ void row_done(int, int) const {}
};

// DFT along y (and the adjoint of the inverse along y): row (kx, b, c), col n = kyi*2 + part,
// out Z[kx*KY + kyi][b][part*32 + c]
struct EpiModes {
    static constexpr bool PAIR = false;
    bf16* Z;
    int B;
    __device__ __forceinline__ void operator()(int, int row, int n0, const float* v, int) const {
        const int c = row % C, t = row / C, b = t % B, kx = t / B;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int n = n0 + i, kyi = n >> 1, part = n & 1;
            Z[((size_t)(kx * KY + kyi) * B + b) * 64 + part * 32 + c] = __float2bfloat16_rn(v[i]);
        }
    }
    __device__ __forceinline__ void row_done(int, int) const {}
};

// channel mixing (forward and adjoint): batch z = mode, row b, cols c (real) and 32 + c (imaginary),
// out Y[b][c][kx][kyi*2 + part]
struct EpiMix {
    static constexpr bool PAIR = true;
    bf16* Y;
    __device__ __forceinline__ void pair(int z, int row, int c0, const float* re, const float* im) const {
        const int kx = z / KY, kyi = z - kx * KY;
        bf16* y = Y + (((size_t)row * C + c0) * KX + kx) * 64 + kyi * 2;
#pragma unroll
        for (int i = 0; i < 16; i++) *(uint32_t*)(y + (size_t)i * KX * 64) = pack2(re[i], im[i]);
    }
    __device__ __forceinline__ void row_done(int, int) const {}
};

// inverse DFT along y (and the adjoint of the DFT along y): row (b, c, kx), col n = y*2 + part,
// out G[(b, y)][c][kx*2 + part]
struct EpiIdftY {
    static constexpr bool PAIR = false;
    bf16* G;
    int S;
    __device__ __forceinline__ void operator()(int, int row, int n0, const float* v, int) const {
        const int bc = row / KX, kx = row - bc * KX, b = bc / C, c = bc - b * C;
        bf16* g = G + (((size_t)b * S + (n0 >> 1)) * C + c) * 32 + kx * 2;
#pragma unroll
        for (int i = 0; i < 8; i++) *(uint32_t*)(g + (size_t)i * C * 32) = pack2(v[2 * i], v[2 * i + 1]);
    }
    __device__ __forceinline__ void row_done(int, int) const {}
};

// inverse DFT along x + pointwise path + bias: batch z = (b, y), row x, col c.  Saves z
// (FP32) and writes the activation, both NCHW.
struct EpiPixAct {
    static constexpr bool PAIR = false;
    const float* bias;
    float* zs;
    bf16* vext;
    int S, S2, act;
    __device__ __forceinline__ void operator()(int z, int x, int c0, const float* v, int) const {
        const int b = z / S, y = z - b * S;
        const size_t p = (size_t)y * S + x;
        float* zo = zs + ((size_t)b * C + c0) * S2 + p;
        bf16* vo = vext + ((size_t)b * VC + c0) * S2 + p;
        float bc[16];
        load16(bc, bias + c0);
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const float zz = v[i] + bc[i];
            zo[(size_t)i * S2] = zz;
            vo[(size_t)i * S2] = __float2bfloat16_rn(act ? gelu(zz) : zz);
        }
    }
    __device__ __forceinline__ void row_done(int, int) const {}
};

// gradient of a layer's input, batch z = (b, y), row x, col c, times GELU'(zs) of the layer below
// (identity when zs is null) -> dz[b][c][y*S + x] in BF16.  dz may be the operand that the product
// read: a tile's pixels are read by that tile alone, before its epilogue.
struct EpiPixBwd {
    static constexpr bool PAIR = false;
    const float* zs;
    bf16* dz;
    int S, S2;
    __device__ __forceinline__ void operator()(int z, int x, int c0, const float* v, int) const {
        const int b = z / S, y = z - b * S;
        const size_t o = ((size_t)b * C + c0) * S2 + (size_t)y * S + x;
        float zv[16];
#pragma unroll
        for (int i = 0; i < 16; i++) zv[i] = zs ? zs[o + (size_t)i * S2] : 0.f;
#pragma unroll
        for (int i = 0; i < 16; i++) dz[o + (size_t)i * S2] = __float2bfloat16_rn(zs ? v[i] * gelu_grad(zv[i]) : v[i]);
    }
    __device__ __forceinline__ void row_done(int, int) const {}
};

// projection: batch z = b, row p, col j (all 128 in one tile): q = sum_j GELU(a_j + b1_j) Q2_j + b2
struct EpiProj {
    static constexpr bool PAIR = false;
    const float* b1;
    const float* Q2;
    const float* b2;
    float* q;
    int S2;
    float acc;
    __device__ __forceinline__ void operator()(int, int, int j0, const float* v, int) {
        float bj[16], qj[16];
        load16(bj, b1 + j0);
        load16(qj, Q2 + j0);
#pragma unroll
        for (int i = 0; i < 16; i++) acc += gelu(v[i] + bj[i]) * qj[i];
    }
    __device__ __forceinline__ void row_done(int z, int p) { q[(size_t)z * S2 + p] = acc + b2[0]; }
};

// ---------------------------------------------------------------------------
// DFT along x and then y of CH channels of a sample (and the adjoint of the inverse), fused:
//   T[(c, y)][(part, kx)] = v[c][y][x] x F1[(part, kx)][x]          in tiles of 128 rows (c, y)
//   Z[mode][b][part*32 + c] = T[(c, kx)][(part, y)] x F2[(kyi, part')][(part, y)]
// T exists only as the BF16 operand of the second product in shared memory: a row's 16 values of a
// part are two 16-byte pieces of eight (c, kx) at column (part, y), the MN-major core matrices.  For
// S <= 128 (both operands and three tiles of v fit an SM: 201 KB at 128); wider grids run the two
// products of the general kernel.  CH is 8 (all 128 rows of the second product) where that gives
// enough blocks, else fewer.  One thread keeps three tiles' TMA loads in flight and issues the MMAs;
// the other work of a tile is its accumulator's way to shared memory.  With 16-byte cp.async copies
// by all threads, their issue alone took 2200 cycles of a tile's 4000.
// 32 samples of 128 x 128: 40 us in two kernels, 26 us fused with cp.async, 14 us
// (the pass: inference 600 -> 550 us, training step 1483 -> 1386 us).
// ---------------------------------------------------------------------------
constexpr int DFT2_S = 128;
constexpr int DFT2_NB = 3;  // tile buffers
constexpr int dft2_kb(int S) { return S % 64 ? 32 : 64; }  // columns of a TMA box
struct Dft2Args {
    CUtensorMap v, F1, F2;  // v: (x, (c, y), sample), boxes of 128 rows; F1, F2: all rows
    bf16* Z;
    int B, CH;
    int* err;
    long long polls;
};
constexpr int dft2_smem(int S) { return DFT2_NB * 256 * S + 64 * S + 256 * S + 512 * S + 1024; }

template <int S>
__global__ void __launch_bounds__(256) k_dft2(const __grid_constant__ Dft2Args g) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t bars[2], full[DFT2_NB], fbar[2];
    __shared__ uint32_t tmem_base;
    constexpr int KB = dft2_kb(S), BOX = 128 * KB * 2;  // bytes of a box of v
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, CH = g.CH;
    const int groups = C / CH, b = blockIdx.x / groups, c0 = (blockIdx.x - b * groups) * CH;
    const int rows = CH * S, nt = (rows + 127) >> 7;
    const uint32_t sV = (tc_smem_u32(smem_raw) + 1023) & ~1023u;  // the swizzle's alignment
    const uint32_t sF1 = sV + DFT2_NB * 256 * S, sF2 = sF1 + 64 * S, sA = sF2 + 256 * S;
    unsigned char* const smem = smem_raw + (sV - tc_smem_u32(smem_raw));
    if (tid == 0) {
        for (int i = 0; i < 2; i++) {
            mbar_init(&bars[i], 1);
            mbar_init(&fbar[i], 1);
        }
        for (int i = 0; i < DFT2_NB; i++) mbar_init(&full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
        // the matrices are constants of the network
        mbar_expect(&fbar[0], 64 * S);
        for (int x = 0; x < S; x += KB) tma_load(sF1 + x * 64, &g.F1, x, 0, 0, &fbar[0]);
        mbar_expect(&fbar[1], 256 * S);
        for (int x = 0; x < 2 * S; x += KB) tma_load(sF2 + x * 128, &g.F2, x, 0, 0, &fbar[1]);
    }
    if (warp == 1) {
        tc_alloc(&tmem_base, 128);
        tc_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;  // three accumulators of 32 columns, then the second product's 64
    dep_wait();
    if (dep_early()) dep_launch();
    // thread 0: tile t to buffer t % DFT2_NB (the rows of a last, shorter tile are followed by rows of
    // the next channels, or zeros, which only unread accumulator rows see)
    auto load_tile = [&](int t) {
        uint64_t* const bar = &full[t % DFT2_NB];
        mbar_expect(bar, 256 * S);
#pragma unroll
        for (int i = 0; i < S / KB; i++)
            tma_load(sV + (t % DFT2_NB) * 256 * S + i * BOX, &g.v, i * KB, c0 * S + t * 128, b, bar);
    };
    int nload = 0, nfull = 0, ncommit = 0;  // thread 0: tiles loaded, tiles that arrived, commits
    if (tid == 0)
        for (; nload < min(nt, DFT2_NB); nload++) load_tile(nload);
    const int quad = warp & 3, half = warp >> 2, pr = quad * 32 + lane;
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    // Commit n (tile n; the last one is the second product) goes to bars[n & 1].  A tile's product is
    // issued before the previous tile's accumulator is read, so it runs beside that epilogue; with three
    // accumulators the block barrier behind the previous commit's wait is the only one of a tile.
    bool dead = false;  // thread 0: a wait gave up
    auto wait_commit = [&](int c) {
        if (tid == 0 && !dead) dead = !mbar_wait(&bars[c & 1], (uint32_t)((c >> 1) & 1), g.polls);
        const int any = __syncthreads_or(dead);
        tc_fence_after();
        return !any;
    };
    bool ok = true;
    for (int t = 0; t <= nt; t++) {
        if (t < nt && tid == 0 && !dead) {
            if (mbar_wait(&full[t % DFT2_NB], (uint32_t)((t / DFT2_NB) & 1), g.polls) &&
                (t > 0 || mbar_wait(&fbar[0], 0, g.polls))) {
                nfull = t + 1;
                tc_fence_after();
                const uint32_t a0 = sV + (t % DFT2_NB) * 256 * S;
#pragma unroll
                for (int x = 0; x < S; x += 16)
                    tc_mma(tmem + (t % 3) * 32, tma_desc<KB>(a0 + x / KB * BOX + x % KB * 2),
                           tma_desc<KB>(sF1 + x / KB * (64 * KB) + x % KB * 2), tc_instr_desc(TC_BM, 32), x > 0);
                tc_commit(&bars[t & 1]);
                ncommit = t + 1;
            } else {
                dead = true;
            }
        }
        if (t == 0) continue;
        // tile t - 1: this thread's row (c, y), part `half`
        ok = wait_commit(t - 1);
        if (!ok) break;
        if (tid == 0 && nload < nt) load_tile(nload++);  // to the buffer of tile t - 1
        float v[16];
        tc_ld16(tmem + lanes + (uint32_t)(((t - 1) % 3) * 32 + half * 16), v);
        const int row = (t - 1) * 128 + pr;
        if (row < rows) {
            const int c = row / S, k = half * S + row - c * S;
            unsigned char* d = smem + (sA - sV) + (k >> 3) * 2048 + (2 * c) * 128 + (k & 7) * 16;
            *(uint4*)d = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
            *(uint4*)(d + 128) = make_uint4(pack2(v[8], v[9]), pack2(v[10], v[11]), pack2(v[12], v[13]), pack2(v[14], v[15]));
        }
        tc_fence_before();
    }
    const uint32_t tD2 = tmem + 64;  // the third accumulator is done too
    if (ok) {
        fence_async_smem();
        __syncthreads();
        if (tid == 0) {
            if (mbar_wait(&fbar[1], 0, g.polls)) {
                tc_fence_after();
#pragma unroll
                for (int x = 0; x < 2 * S; x += 16)
                    tc_mma(tD2, tc_smem_desc(sA + x / 8 * 2048, 2048, 128),
                           tma_desc<KB>(sF2 + x / KB * (128 * KB) + x % KB * 2), tc_instr_desc(TC_BM, 64) | (1u << 15),
                           x > 0);
                tc_commit(&bars[nt & 1]);
                ncommit = nt + 1;
            } else {
                dead = true;
            }
        }
        ok = wait_commit(nt);
    }
    if (ok) {
        if (!dep_early()) dep_launch();
        // row m = (c, kx): to shared memory as [kx][kyi][part][c] (the tiles of v are done), then out in
        // runs of CH channels
        bf16* const zt = (bf16*)smem;
        const int kxp = 64 * CH + 8;  // pitch of a kx: its rows start in different banks
        const int c = pr >> 4, kx = pr & 15;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            float v[16];
            tc_ld16(tD2 + lanes + (uint32_t)(half * 32 + q * 16), v);
            if (c < CH) {
#pragma unroll
                for (int i = 0; i < 16; i++) zt[kx * kxp + (half * 32 + q * 16 + i) * CH + c] = __float2bfloat16_rn(v[i]);
            }
        }
        tc_fence_before();
        __syncthreads();
        for (int v = tid; v < KX * 64; v += 256) {
            const int k = v >> 6, r = v & 63;  // r = kyi*2 + part
            const bf16* z = zt + k * kxp + r * CH;
            bf16* o = g.Z + ((size_t)(k * KY + (r >> 1)) * g.B + b) * 64 + (r & 1) * 32 + c0;
            if (CH == 8) *(uint4*)o = *(const uint4*)z;
            else if (CH == 4) *(uint2*)o = *(const uint2*)z;
            else if (CH == 2) *(uint32_t*)o = *(const uint32_t*)z;
            else *o = *z;
        }
    }
    if (dead) {
        if (g.err) atomicExch(g.err, FI_ERR_TIMEOUT);
        // let the copies and MMAs in flight finish first
        for (int t = nfull; t < nload; t++) mbar_wait(&full[t % DFT2_NB], (uint32_t)((t / DFT2_NB) & 1));
        for (int i = 0; i < 2; i++) mbar_wait(&fbar[i], 0);
        if (ncommit > 0) mbar_wait(&bars[(ncommit - 1) & 1], (uint32_t)(((ncommit - 1) >> 1) & 1));
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tc_dealloc(tmem, 128);
}

// ---------------------------------------------------------------------------
// inverse DFT along x + pointwise path of a row of pixels (and the adjoints of both), per row (b, y) and
// 128 pixels x:
//   out[x][c] = G1[x][(kx, part)] x G[(b, y)][c][(kx, part)] + v[b][ci][y][x] x W[c][ci]
// A ring of PIX_NB tiles: thread 256 keeps their TMA loads in flight and issues the MMAs (an accumulator
// of 32 columns a slot), two groups of four warps take the accumulators in turn.  A slot's barriers: full
// (its copies arrived), done (its MMAs finished: the accumulator is ready and the copies' place free),
// taken (the accumulator was read).  What bounds it is the epilogue's traffic (4-byte values of z along
// the pixels, BF16 activations); as tiles of the general kernel, ten blocks an SM of four warps with
// cp.async copies, block barriers and copies, products and stores all in phase, 60 us (forward) and
// 62 us (backward) at 32 samples of 128 x 128, this one 38 and 42 us (bytes: 21 us).
// ---------------------------------------------------------------------------
constexpr int PIX_NB = 4, PIX_THREADS = 288, PIX_BLOCKS = 4;  // blocks: an SM (3: training step 1291 us, 4: 1270)
constexpr int pix_kb(int S) { return S % 64 ? 32 : 64; }      // pixels of a TMA box
struct PixArgs {
    CUtensorMap G1, G, v, W;  // (K, x), (K, c, (b, y)), (pixel, ci, b), (ci, c, layer)
    int S, ntiles, layer;
    int* err;
    long long polls;
};
inline int pix_smem(int S) { return PIX_NB * (8192 + 2048) + 2048 + (S > 128 ? 2 : 1) * 8192 + 1024; }

template <int KB, class Epi>
__global__ void __launch_bounds__(PIX_THREADS, PIX_BLOCKS) k_pix(const __grid_constant__ PixArgs g, const Epi epi) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[PIX_NB], done[PIX_NB], taken[PIX_NB], fbar;
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, S = g.S;
    const int mt = (S + 127) >> 7, G1R = min(S, 128);
    const uint32_t sV = (tc_smem_u32(smem) + 1023) & ~1023u, sG = sV + PIX_NB * 8192, sW = sG + PIX_NB * 2048,
                   sG1 = sW + 2048;
    if (tid == 256) {
        for (int i = 0; i < PIX_NB; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&done[i], 1);
            mbar_init(&taken[i], 4);
        }
        mbar_init(&fbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
        // G1 is a constant of the network
        mbar_expect(&fbar, mt * G1R * 64 + 2048);
        for (int m = 0; m < mt; m++) tma_load(sG1 + m * 8192, &g.G1, 0, m * 128, 0, &fbar);
    }
    if (warp == 0) {
        tc_alloc(&tmem_base, 32 * PIX_NB);
        tc_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;
    dep_wait();
    if (dep_early()) dep_launch();
    const int n = (g.ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;  // this block's tiles
    bool dead = false;
    if (tid == 256) {
        tma_load(sW, &g.W, 0, 0, g.layer, &fbar);
        auto load = [&](int i) {
            const int tile = blockIdx.x + i * gridDim.x, z = tile / mt, m0 = (tile - z * mt) * 128, b = z / S, y = z - b * S;
            const int q = i % PIX_NB, nbox = min(128, S - m0) / KB;
            mbar_expect(&full[q], 2048 + nbox * KB * 64);
            tma_load(sG + q * 2048, &g.G, 0, 0, z, &full[q]);
            for (int k = 0; k < nbox; k++)
                tma_load(sV + q * 8192 + k * KB * 64, &g.v, y * S + m0 + k * KB, 0, b, &full[q]);
        };
        int nload = 0, nfull = 0, ncommit = 0;
        for (; nload < min(n, PIX_NB); nload++) load(nload);
        dead = !mbar_wait(&fbar, 0, g.polls);
        for (int i = 0; i < n && !dead; i++) {
            const int q = i % PIX_NB;
            const uint32_t ph = (uint32_t)(i / PIX_NB) & 1;
            dead = !mbar_wait(&full[q], ph, g.polls);
            if (dead) break;
            nfull = i + 1;
            dead = i >= PIX_NB && !mbar_wait(&taken[q], ph ^ 1, g.polls);
            if (dead) break;
            tc_fence_after();
            const int m = (int)((blockIdx.x + i * gridDim.x) % mt);
            const uint32_t d = tmem + 32 * q, id = tc_instr_desc(TC_BM, 32);
#pragma unroll
            for (int k = 0; k < 2; k++)
                tc_mma(d, tma_desc<32>(sG1 + m * 8192 + 32 * k), tma_desc<32>(sG + q * 2048 + 32 * k), id, k > 0);
#pragma unroll
            for (int k = 0; k < 2; k++)
                tc_mma(d, tma_desc_mn<KB>(sV + q * 8192 + k * KB * 32, KB * 64), tma_desc<32>(sW + 32 * k), id | (1u << 15),
                       1u);
            tc_commit(&done[q]);
            ncommit = i + 1;
            // the previous tile's slot, when its MMAs are done
            if (i > 0 && nload < n) {
                dead = !mbar_wait(&done[(i - 1) % PIX_NB], (uint32_t)((i - 1) / PIX_NB) & 1, g.polls);
                if (!dead) load(nload++);
            }
        }
        // copies and MMAs in flight finish first (also when it is an epilogue that gave up)
        mbar_wait(&fbar, 0);
        for (int i = nfull; i < nload; i++) mbar_wait(&full[i % PIX_NB], (uint32_t)(i / PIX_NB) & 1);
        if (ncommit > 0) mbar_wait(&done[(ncommit - 1) % PIX_NB], (uint32_t)((ncommit - 1) / PIX_NB) & 1);
    } else if (warp < 8) {
        const int quad = warp & 3;
        for (int i = warp >> 2; i < n; i += 2) {
            const int tile = blockIdx.x + i * gridDim.x, z = tile / mt, x = (tile - z * mt) * 128 + quad * 32 + lane;
            const int q = i % PIX_NB;
            dead = !__all_sync(0xffffffffu, mbar_wait(&done[q], (uint32_t)(i / PIX_NB) & 1, g.polls));
            if (dead) break;
            tc_fence_after();
#pragma unroll 1
            for (int c0 = 0; c0 < 32; c0 += 16) {
                float v[16];
                tc_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(32 * q + c0), v);
                if (c0) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&taken[q]);
                }
                if (x < S) epi(z, x, c0, v, 16);
            }
        }
    }
    if (dead && g.err) atomicExch(g.err, FI_ERR_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (!dep_early()) dep_launch();
    if (warp == 0) tc_dealloc(tmem, 32 * PIX_NB);
}

// ---------------------------------------------------------------------------
// weight gradients of the pointwise layers: slices of SLICE pixels
// ---------------------------------------------------------------------------
constexpr int SLICE = 512;  // pixels per split-K slice (S2 is a multiple of 1024)

// part[slice][32][NR] = sum over the slice's pixels of dz[32][p] x act[NR][p], one 128 x N tensor-core
// tile whose rows beyond 32 (and columns beyond NR) hold whatever the operand buffers overlap: only
// their own, unread, results depend on it.  Boxes of 64 pixels come by TMA; a box's MMAs start when it
// arrives and the next slice's box follows when they are done, so three blocks an SM keep 200 KB of
// copies in flight; two accumulators leave the first warp a slice's time to store.  Bytes bound it.
// 32 samples of 128 x 128 (67 MB read): 38 us as a general product in eight chunks of K, 28 us with one
// cp.async copy of a slice by 256 threads, about 20 us (training step 1237 -> 1196 us).
struct WgradArgs {
    CUtensorMap dz, act;  // (pixel, channel, b), boxes of 64 pixels x 32 and NR channels
    int ns, nslices;
    float* part;
    int* err;
    long long polls;
};
constexpr int WG_BOX = 64, WG_NBOX = SLICE / WG_BOX, WG_THREADS = 64, WG_LAG = 2;
template <int NR>
constexpr int wgrad_smem() {  // the last box's 128 rows end 12 KB behind the boxes of dz
    constexpr int B = WG_NBOX * ((NR + 7) / 8) * 1024;
    return WG_NBOX * 4096 + (B > 12288 ? B : 12288) + 2048;
}

template <int NR>
__global__ void __launch_bounds__(WG_THREADS) k_wgrad(const __grid_constant__ WgradArgs g) {
    constexpr int NG = (NR + 7) / 8, N = (NR + 15) / 16 * 16;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[WG_NBOX], done[WG_NBOX], ready[2], taken[2];
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sa = (tc_smem_u32(smem) + 1023) & ~1023u, sb = sa + WG_NBOX * 4096;
    if (tid == 32) {
        for (int i = 0; i < WG_NBOX; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&done[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&ready[i], 1);
            mbar_init(&taken[i], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 0) {
        tc_alloc(&tmem_base, 128);
        tc_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    dep_wait();
    if (dep_early()) dep_launch();
    const uint32_t tmem = tmem_base;
    const int n = (g.nslices - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;  // this block's slices
    bool dead = false;
    if (tid == 32) {
        auto load = [&](int i, int k) {
            const int z = blockIdx.x + i * gridDim.x, b = z / g.ns, px = (z - b * g.ns) * SLICE + k * WG_BOX;
            mbar_expect(&full[k], (32 + NR) * 128);
            tma_load(sa + k * 4096, &g.dz, px, 0, b, &full[k]);
            tma_load(sb + k * NG * 1024, &g.act, px, 0, b, &full[k]);
        };
        // boxes in the order of all slices: loaded, arrived, committed
        int nload = 0, nfull = 0, ncommit = 0;
        for (; nload < WG_NBOX; nload++) load(0, nload);
        for (int i = 0; i < n && !dead; i++) {
            const uint32_t d = tmem + 64 * (i & 1);
            if (i >= 2) dead = !mbar_wait(&taken[i & 1], (uint32_t)((i >> 1) - 1) & 1, g.polls);
            for (int k = 0; k < WG_NBOX && !dead; k++) {
                dead = !mbar_wait(&full[k], (uint32_t)i & 1, g.polls);
                if (dead) break;
                nfull++;
                tc_fence_after();
#pragma unroll
                for (int x = 0; x < WG_BOX; x += 16)
                    tc_mma(d, tma_desc<64>(sa + k * 4096 + 2 * x), tma_desc<64>(sb + k * NG * 1024 + 2 * x),
                           tc_instr_desc(TC_BM, N), k > 0 || x > 0);
                tc_commit(&done[k]);
                ncommit++;
                // the next slice's box to the place of the box WG_LAG before
                if (ncommit > WG_LAG && nload < n * WG_NBOX) {
                    const int c = ncommit - 1 - WG_LAG;
                    dead = !mbar_wait(&done[c % WG_NBOX], (uint32_t)(c / WG_NBOX) & 1, g.polls);
                    if (!dead) {
                        load(nload / WG_NBOX, nload % WG_NBOX);
                        nload++;
                    }
                }
            }
            if (!dead) tc_commit(&ready[i & 1]);
        }
        // copies and MMAs in flight finish first
        for (int c = nfull; c < nload; c++) mbar_wait(&full[c % WG_NBOX], (uint32_t)(c / WG_NBOX) & 1);
        if (ncommit > 0) mbar_wait(&done[(ncommit - 1) % WG_NBOX], (uint32_t)((ncommit - 1) / WG_NBOX) & 1);
    } else if (warp == 0) {
        for (int i = 0; i < n; i++) {
            dead = !__all_sync(0xffffffffu, mbar_wait(&ready[i & 1], (uint32_t)(i >> 1) & 1, g.polls));
            if (dead) break;
            tc_fence_after();
            float v[N];
#pragma unroll
            for (int c0 = 0; c0 < N; c0 += 16) tc_ld16(tmem + 64 * (i & 1) + c0, v + c0);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&taken[i & 1]);
            float* o = g.part + ((size_t)(blockIdx.x + i * gridDim.x) * C + lane) * NR;
#pragma unroll
            for (int c = 0; c < NR; c++) o[c] = v[c];
        }
    }
    if (dead && g.err) atomicExch(g.err, FI_ERR_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (!dep_early()) dep_launch();
    if (warp == 0) tc_dealloc(tmem, 128);
}

// ---------------------------------------------------------------------------
// adjoint of the projection, fused: per slice of SLICE pixels, in tiles of 128 pixels,
//   a = v Q1^T + b1 (recomputed), da = dq Q2 GELU'(a), h = GELU(a)
//   dz = da Q1 (gradient of the last layer's output, BF16 NCHW)
//   part[slice][j][c] = sum da_j v_c (c < 32), sum da_j (c = 32), sum h_j dq (c = 33)
// da and h exist only as BF16 tiles in shared memory: 16-byte pieces of 8 hidden units of a pixel,
// which serve as the pixels x units operand of dz and, transposed by the descriptors, as the
// units x pixels operand of the weight gradients; likewise the tile of v (channels 0..33) for a
// and for the weight gradients.  Three products of separate kernels moved 1.2 GB of da and h at
// 32 samples of 128 x 128; what is left is bound by the instructions of erff and expf.
// 434 us in four kernels -> 159 us (103 M instructions).
// ---------------------------------------------------------------------------
struct ProjBwdArgs {
    const bf16* v;       // last activation buffer [b][VC][S2]
    const bf16 *Q1, *Q1T;  // [128][32], [32][128]
    const float *b1, *Q2, *dq;
    bf16* dz;
    float* part;
    int S2, nslices;
    int* err;
    long long polls;
};
constexpr int PB_V = 6 * 2048, PB_V_OFF = 0, PB_Q1 = 2 * PB_V, PB_Q1T = PB_Q1 + 8192, PB_DA = PB_Q1T + 8192,
              PB_H = PB_DA + 32768, PB_W = PB_H + 32768, PB_SMEM = PB_W + 1024;

__global__ void __launch_bounds__(256, 2) k_proj_bwd(const __grid_constant__ ProjBwdArgs g) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t tmem_base;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, S2 = g.S2, ns = S2 / SLICE;
    const uint32_t s0 = tc_smem_u32(smem);
    float* const sb1 = (float*)(smem + PB_W);
    float* const sQ2 = sb1 + PW;
    // tile t of this block's sequence (4 per slice): pixels of sample b from px
    auto where = [&](int t, int& b, size_t& px) {
        const int z = blockIdx.x + (t >> 2) * gridDim.x;
        b = z / ns;
        px = (size_t)(z - b * ns) * SLICE + (t & 3) * 128;
    };
    auto stage = [&](int t) {
        int b;
        size_t px;
        where(t, b, px);
        const bf16* p = g.v + (size_t)b * VC * S2 + px;
        const uint32_t d = s0 + PB_V_OFF + (t & 1) * PB_V;
        // 16-byte piece: 8 pixels of channel c; eight neighbouring threads take eight channels of one
        // core matrix
        for (int v = tid; v < (VC + 7) / 8 * 128; v += 256) {
            const int c = (v >> 7) * 8 + (v & 7), q = (v >> 3) & 15;
            if (c < VC) cp_async16(d + (c >> 3) * 2048 + q * 128 + (c & 7) * 16, p + (size_t)c * S2 + 8 * q, true);
        }
        cp_async_commit();
    };
    const int my = g.nslices > (int)blockIdx.x ? (g.nslices - 1 - blockIdx.x) / gridDim.x + 1 : 0;
    const int ntiles = 4 * my;
    if (warp == 0) {
        tc_alloc(&tmem_base, 256);
        tc_relinquish();
    }
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_fail = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    dep_wait();
    if (dep_early()) dep_launch();
    for (int v = tid; v < PW * 4; v += 256) {
        const int r = v >> 2, q = v & 3;
        cp_async16(s0 + PB_Q1 + q * (PW * 16) + (r >> 3) * 128 + (r & 7) * 16, g.Q1 + r * C + 8 * q, true);
    }
    for (int v = tid; v < C * 16; v += 256) {
        const int r = v >> 4, q = v & 15;
        cp_async16(s0 + PB_Q1T + q * (C * 16) + (r >> 3) * 128 + (r & 7) * 16, g.Q1T + r * PW + 8 * q, true);
    }
    if (tid < PW) {
        sb1[tid] = g.b1[tid];
        sQ2[tid] = g.Q2[tid];
    }
    if (ntiles > 0) stage(0);
    const uint32_t tmem = tmem_base, tW1 = tmem + PW, tW2 = tmem + PW + 48;
    const int quad = warp & 3, half = warp >> 2, pr = quad * 32 + lane;  // pixel row of the tile, column half
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    int stage_bar = -1;  // thread 0: the barrier of its last commit (0, 1), and the phase
    uint32_t last_phase = 0;
    for (int t = 0; t < ntiles; t++) {
        const uint32_t ph = (uint32_t)(t & 1);
        const uint32_t sv = s0 + PB_V_OFF + (t & 1) * PB_V;
        cp_async_wait<0>();
        fence_async_smem();
        __syncthreads();
        // hidden layer: pixels (MN-major v, 32 channels) x units
        if (tid == 0) {
            tc_fence_after();
            for (int ks = 0; ks < 2; ks++)
                tc_mma(tmem, tc_smem_desc(sv + 2 * ks * 2048, 2048, 128),
                       tc_smem_desc(s0 + PB_Q1 + 2 * ks * (PW * 16), PW * 16, 128),
                       tc_instr_desc(TC_BM, PW) | (1u << 15), ks > 0);
            tc_commit(&bars[0]);
            stage_bar = 0;
            last_phase = ph;
        }
        // the other tile buffer was last read by the previous tile's products, which are done
        if (t + 1 < ntiles) stage(t + 1);
        int b;
        size_t px;
        where(t, b, px);
        const float gq = g.dq[(size_t)b * S2 + px + pr];
        if (tid == 0 && !mbar_wait(&bars[0], ph, g.polls)) s_fail = 1;
        __syncthreads();
        if (s_fail) break;
        tc_fence_after();
        // da and h of this thread's pixel, 64 units
        unsigned char* const dda = smem + PB_DA + (pr >> 3) * 2048 + (pr & 7) * 16;
#pragma unroll 1
        for (int j0 = half * 64; j0 < half * 64 + 64; j0 += 16) {
            float v[16], h[16];
            tc_ld16(tmem + lanes + (uint32_t)j0, v);
#pragma unroll
            for (int i = 0; i < 16; i++) {
                float ga, gpa;
                gelu_both(v[i] + sb1[j0 + i], ga, gpa);
                v[i] = gq * sQ2[j0 + i] * gpa;
                h[i] = ga;
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const float *a = v + 8 * q, *c = h + 8 * q;
                *(uint4*)(dda + ((j0 >> 3) + q) * 128) =
                    make_uint4(pack2(a[0], a[1]), pack2(a[2], a[3]), pack2(a[4], a[5]), pack2(a[6], a[7]));
                *(uint4*)(dda + (PB_H - PB_DA) + ((j0 >> 3) + q) * 128) =
                    make_uint4(pack2(c[0], c[1]), pack2(c[2], c[3]), pack2(c[4], c[5]), pack2(c[6], c[7]));
            }
        }
        tc_fence_before();
        fence_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const uint32_t da = s0 + PB_DA, hh = s0 + PB_H;
            // dz: pixels x units (K) times Q1T; the hidden accumulator's first columns are free again
            for (int ks = 0; ks < PW / 16; ks++)
                tc_mma(tmem, tc_smem_desc(da + 2 * ks * 128, 128, 2048),
                       tc_smem_desc(s0 + PB_Q1T + 2 * ks * (C * 16), C * 16, 128), tc_instr_desc(TC_BM, C), ks > 0);
            // weight gradients: units (MN-major) x pixels (K) times channels
            for (int ks = 0; ks < 8; ks++) {
                const uint32_t acc = (t & 3) > 0 || ks > 0;
                tc_mma(tW1, tc_smem_desc(da + 2 * ks * 2048, 2048, 128), tc_smem_desc(sv + 2 * ks * 128, 128, 2048),
                       tc_instr_desc(TC_BM, 48) | (1u << 15), acc);
                tc_mma(tW2, tc_smem_desc(hh + 2 * ks * 2048, 2048, 128),
                       tc_smem_desc(sv + 4 * 2048 + 2 * ks * 128, 128, 2048), tc_instr_desc(TC_BM, 16) | (1u << 15), acc);
            }
            tc_commit(&bars[1]);
            stage_bar = 1;
            last_phase = ph;
            if (!mbar_wait(&bars[1], ph, g.polls)) s_fail = 1;
        }
        __syncthreads();
        if (s_fail) break;
        tc_fence_after();
        {
            float v[16];
            tc_ld16(tmem + lanes + (uint32_t)(half * 16), v);
            bf16* o = g.dz + ((size_t)b * C + half * 16) * S2 + px + pr;
#pragma unroll
            for (int i = 0; i < 16; i++) o[(size_t)i * S2] = __float2bfloat16_rn(v[i]);
        }
        if ((t & 3) == 3) {
            const int z = blockIdx.x + (t >> 2) * gridDim.x;
            float* o = g.part + ((size_t)z * PW + pr) * VC;
            float v[16];
            if (half == 0) {
#pragma unroll
                for (int c0 = 0; c0 < 32; c0 += 16) {
                    tc_ld16(tW1 + lanes + (uint32_t)c0, v);
#pragma unroll
                    for (int i = 0; i < 16; i++) o[c0 + i] = v[i];
                }
            } else {
                tc_ld16(tW1 + lanes + 32u, v);
                o[C] = v[0];
                tc_ld16(tW2 + lanes, v);
                o[C + 1] = v[1];
            }
        }
        tc_fence_before();
        // the next tile's MMAs are issued after the next __syncthreads()
    }
    if (!dep_early()) dep_launch();
    cp_async_wait<0>();
    if (s_fail && tid == 0) {
        if (g.err) atomicExch(g.err, FI_ERR_TIMEOUT);
        if (stage_bar >= 0) mbar_wait(&bars[stage_bar], last_phase);  // let the issued MMAs finish
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tc_dealloc(tmem, 256);
}

// ---------------------------------------------------------------------------
// element-wise and reduction kernels.  Those launched programmatically take plain pointers: what they
// read may still be written while they wait, which the non-coherent loads of `const __restrict__`
// parameters do not allow.
// ---------------------------------------------------------------------------

// x [B][6][S2] FP32 -> NCHW [b][8][S2] BF16 (channel 6 = 1 for the lift's bias gradient)
__global__ void k_prep_input(const float* __restrict__ x, bf16* xe, int B, int S2) {
    dep_wait();
    dep_launch();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)B * S2) return;
    const int b = (int)(i / S2), p = (int)(i - (size_t)b * S2);
#pragma unroll
    for (int c = 0; c < NIN; c++)
        xe[((size_t)b * XC + c) * S2 + p] = __float2bfloat16_rn(x[((size_t)b * NIN + c) * S2 + p]);
    xe[((size_t)b * XC + 6) * S2 + p] = __float2bfloat16_rn(1.f);
    xe[((size_t)b * XC + 7) * S2 + p] = __float2bfloat16_rn(0.f);
}

// channel `ch` of every sample of an NCHW activation buffer := value
__global__ void k_fill_channel(bf16* v, int B, int S2, int ch, float value) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)B * S2) return;
    const int b = (int)(i / S2), p = (int)(i - (size_t)b * S2);
    v[((size_t)b * VC + ch) * S2 + p] = __float2bfloat16_rn(value);
}

// loss gradient: weighted MSE against target, loss = (1/n) sum_i w_b(i) (q_i - t_i)^2 with
// per-sample weights w (1 when null), dq = 2 w (q - t) / n; or a given dy.
// Writes dq (FP32), its BF16 copy into channel 33 of the last activation buffer, and
// accumulates sum(dq) (gradient of b2).
__global__ void __launch_bounds__(256) k_loss(const float* q, const float* target,
                                              const float* w, const float* dy, int n,
                                              int S2, float inv_n, float* dq, bf16* vext4, float* part) {
    dep_wait();
    dep_launch();
    const int i = blockIdx.x * 256 + threadIdx.x;
    float l = 0.f, d = 0.f;
    if (i < n) {
        const int b = i / S2, p = i - b * S2;
        if (target) {
            const float e = q[i] - target[i], wb = w ? w[b] : 1.f;
            l = wb * e * e * inv_n;
            d = 2.f * wb * e * inv_n;
        } else {
            d = dy[i];
        }
        dq[i] = d;
        vext4[((size_t)b * VC + 33) * S2 + p] = __float2bfloat16_rn(d);
    }
    for (int o = 16; o > 0; o >>= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, o);
        d += __shfl_xor_sync(0xffffffffu, d, o);
    }
    __shared__ float sl[8], sd[8];
    if ((threadIdx.x & 31) == 0) {
        sl[threadIdx.x >> 5] = l;
        sd[threadIdx.x >> 5] = d;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float a = 0.f, c = 0.f;
        for (int w = 0; w < 8; w++) {
            a += sl[w];
            c += sd[w];
        }
        part[blockIdx.x] = a;
        part[gridDim.x + blockIdx.x] = c;
    }
}

// the per-block partials of k_loss summed in a fixed order (one block): the loss and the
// output-bias gradient come out the same on every run
__global__ void __launch_bounds__(256) k_loss_sum(const float* part, int nblk, float* loss, float* gb2) {
    dep_wait();
    dep_launch();
    __shared__ float sl[256], sd[256];
    float a = 0.f, c = 0.f;
    for (int i = threadIdx.x; i < nblk; i += 256) {
        a += part[i];
        c += part[nblk + i];
    }
    sl[threadIdx.x] = a;
    sd[threadIdx.x] = c;
    for (int o = 128; o > 0; o >>= 1) {
        __syncthreads();
        if (threadIdx.x < o) {
            sl[threadIdx.x] += sl[threadIdx.x + o];
            sd[threadIdx.x] += sd[threadIdx.x + o];
        }
    }
    if (threadIdx.x == 0) {
        *loss = sl[0];
        *gb2 = sd[0];
    }
}

// spectral weight gradient of one mode (block = mode):
//   dWr[ci][co] = sum_b dYr[co] Zr[ci] + dYi[co] Zi[ci]
//   dWi[ci][co] = sum_b dYi[co] Zr[ci] - dYr[co] Zi[ci]
__global__ void __launch_bounds__(256) k_spec_wgrad(const bf16* Z, const bf16* dY,
                                                    float* gW, int B) {
    dep_wait();
    dep_launch();
    __shared__ float zs[64][64], ds[64][64];
    const int mode = blockIdx.x, tid = threadIdx.x;
    float sr[4] = {0.f, 0.f, 0.f, 0.f}, si[4] = {0.f, 0.f, 0.f, 0.f};
    for (int b0 = 0; b0 < B; b0 += 64) {
        const int nb = min(64, B - b0);
        __syncthreads();
        for (int i = tid; i < nb * 64; i += 256) {
            const size_t g = ((size_t)mode * B + b0) * 64 + i;
            zs[i >> 6][i & 63] = __bfloat162float(Z[g]);
            ds[i >> 6][i & 63] = __bfloat162float(dY[g]);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int idx = tid + 256 * k, ci = idx >> 5, co = idx & 31;
            for (int bb = 0; bb < nb; bb++) {
                const float zr = zs[bb][ci], zi = zs[bb][32 + ci], dr = ds[bb][co], di = ds[bb][32 + co];
                sr[k] += dr * zr + di * zi;
                si[k] += di * zr - dr * zi;
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int idx = tid + 256 * k;
        gW[(size_t)mode * 2 * C * C + idx] = sr[k];
        gW[((size_t)mode * 2 + 1) * C * C + idx] = si[k];
    }
}

// split-K partials [z][MN] summed over z into grad[base + map[i]] (map is one-to-one; a backward pass
// writes every gradient once), in a fixed order, so that gradients are the same on every run:
// each of at most 64 ranges of `per` consecutive z in order (range y and y + 32 by row y of the
// block), then the ranges in order.
__global__ void __launch_bounds__(1024) k_reduce_map(const float* part, int nz, int MN, int per,
                                                     const int* map, float* grad, long long base) {
    dep_wait();
    dep_launch();
    __shared__ float sm[64][33];
    const int i = blockIdx.x * 32 + threadIdx.x;
    for (int y = threadIdx.y; y < 64; y += 32) {
        float s = 0.f;
        if (i < MN) {
            const int z1 = min(nz, (y + 1) * per);
#pragma unroll 8
            for (int z = y * per; z < z1; z++) s += part[(size_t)z * MN + i];
        }
        sm[y][threadIdx.x] = s;
    }
    __syncthreads();
    if (threadIdx.y == 0 && i < MN) {
        float a = 0.f;
        for (int y = 0; y * per < nz; y++) a += sm[y][threadIdx.x];
        grad[base + map[i]] = a;
    }
}

// ranges: at most this many (<= 64)
static cudaError_t reduce_map(const float* part, cudaStream_t st, int nz, int MN, int ranges, const int* map,
                              float* grad, long long base) {
    return launch_dep(k_reduce_map, (MN + 31) / 32, dim3(32, 32), 0, st, part, nz, MN, (nz + ranges - 1) / ranges, map, grad,
                      base);
}

// err: no step from gradients of a pass in which a wait gave up
__global__ void k_adam(float* p, const float* g, float* m, float* v, long long n, float lr, float b1,
                       float b2, float eps, float c1, float c2, const int* err) {
    dep_wait();
    dep_launch();
    if (*err) return;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
    }
}

// spectral weights -> real 64 x 64 block matrices [[Wr, -Wi], [Wi, Wr]] (rows part'*32 + co,
// cols part*32 + ci) and their transposes; grid (mode, layer).  The weights are read and
// both matrices written along their rows, through a shared-memory copy of the mode.
__global__ void __launch_bounds__(256) k_pack_spec(const float* params, long long off0, bf16* Wm,
                                                   bf16* WmT) {
    dep_wait();
    dep_launch();
    __shared__ float w[2][C][C + 1];  // [re, im][ci][co]
    const int mode = blockIdx.x, l = blockIdx.y;
    const float* W = params + off0 + (long long)l * LAYER + (size_t)mode * 2 * C * C;
    for (int i = threadIdx.x; i < 2 * C * C; i += 256) w[i >> 10][(i >> 5) & 31][i & 31] = W[i];
    __syncthreads();
    const size_t o = ((size_t)l * NM + mode) * 4096;
    for (int i = threadIdx.x; i < 4096; i += 256) {
        // Wm row n = (pO, co), col k = (pI, ci)
        const int n = i >> 6, k = i & 63, pO = n >> 5, co = n & 31, pI = k >> 5, ci = k & 31;
        const float wr = w[0][ci][co], wi = w[1][ci][co];
        Wm[o + i] = __float2bfloat16_rn(pO == pI ? wr : (pO == 0 ? -wi : wi));
        // WmT row k' = (pI, ci), col n' = (pO, co): WmT[k'][n'] = Wm[n'][k']
        const int kk = i >> 6, nn = i & 63, pI2 = kk >> 5, ci2 = kk & 31, pO2 = nn >> 5, co2 = nn & 31;
        const float wr2 = w[0][ci2][co2], wi2 = w[1][ci2][co2];
        WmT[o + i] = __float2bfloat16_rn(pO2 == pI2 ? wr2 : (pO2 == 0 ? -wi2 : wi2));
    }
}

// pointwise weights -> BF16 operands: P [32][8], Wloc [l][co][ci] and [l][ci][co], Q1 [128][32], [32][128]
__global__ void k_pack_small(const float* params, Offsets o, bf16* Pb, bf16* Wl, bf16* WlT, bf16* Q1b,
                             bf16* Q1Tb) {
    dep_wait();
    dep_launch();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < C * XC) {
        const int c = i / XC, k = i - c * XC;
        Pb[i] = __float2bfloat16_rn(k < NIN ? params[o.P + c * NIN + k] : 0.f);
    }
    if (i < NLAYER * C * C) {
        const int l = i / (C * C), r = i - l * C * C, co = r / C, ci = r - co * C;
        const float w = params[o.layer[0] + (long long)l * LAYER + SPEC + r];
        Wl[i] = __float2bfloat16_rn(w);
        WlT[(size_t)l * C * C + ci * C + co] = __float2bfloat16_rn(w);
    }
    if (i < PW * C) {
        const int j = i / C, c = i - j * C;
        const float w = params[o.Q1 + i];
        Q1b[i] = __float2bfloat16_rn(w);
        Q1Tb[c * PW + j] = __float2bfloat16_rn(w);
    }
}

}  // namespace fno
}  // namespace fi

using namespace fi;
using namespace fi::fno;

struct fi_fno {
    int S = 0, S2 = 0, maxB = 0, device = 0, ns = 0;
    Offsets o{};
    cudaStream_t st = nullptr;
    float *params = nullptr, *grads = nullptr, *m = nullptr, *v = nullptr;
    long long adam_t = 0;
    float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    // BF16 operand copies of the parameters and the DFT matrices
    bf16 *Pb = nullptr, *Wm = nullptr, *WmT = nullptr, *Wl = nullptr, *WlT = nullptr, *Q1b = nullptr,
         *Q1Tb = nullptr;
    bf16 *F1 = nullptr, *F2 = nullptr, *G2 = nullptr, *G1 = nullptr, *F1T = nullptr, *F2T = nullptr,
         *G2T = nullptr, *G1T = nullptr;
    // activations (saved for the backward pass) and scratch
    bf16 *xe = nullptr, *vext[NLAYER + 1] = {}, *Tb = nullptr, *Zm[NLAYER] = {}, *Yb = nullptr, *Gt = nullptr,
         *dz = nullptr, *dYm = nullptr;
    float *zs[NLAYER] = {}, *q = nullptr, *dq = nullptr, *part = nullptr, *scal = nullptr;
    int *map_loc = nullptr, *map_proj = nullptr, *map_lift = nullptr, *err = nullptr;
    CUtensorMap tm_v[NLAYER], tm_dz, tm_m[4];  // activations and F1, F2, G1T, G2T for k_dft2
    CUtensorMap tm_G1, tm_F1T, tm_G, tm_W, tm_WT, tm_pv[NLAYER], tm_pdz;  // for k_pix
    CUtensorMap tm_wdz, tm_wv[NLAYER], tm_wx;  // for k_wgrad
    int nsm = 0;
    int fwdB = 0;  // batch of the last forward pass (0: none)
    std::vector<void*> allocs;
    std::string msg;
};

namespace {

int fail(fi_fno* h, int code, const std::string& m) {
    if (h) h->msg = m;
    return code;
}

#define FNO_CK(expr)                                                                         \
    do {                                                                                     \
        cudaError_t e_ = (expr);                                                             \
        if (e_ != cudaSuccess)                                                               \
            return fail(h, FI_ERR_CUDA, std::string(#expr) + ": " + cudaGetErrorString(e_)); \
    } while (0)

template <class T>
cudaError_t dalloc(fi_fno* h, T** p, size_t count) {
    void* q = nullptr;
    cudaError_t e = cudaMalloc(&q, count * sizeof(T) + 16);
    if (e != cudaSuccess) return e;
    h->allocs.push_back(q);
    *p = (T*)q;
    return cudaMemset(q, 0, count * sizeof(T) + 16);
}

// operands: K-major (rows K-contiguous) and MN-major (NCHW read as pixels x channels)
TcOperand opK(const bf16* p, int ld, long long s = 0) {
    TcOperand o;
    o.p = p;
    o.ld = ld;
    o.s = s;
    o.mn = 0;
    return o;
}
TcOperand opMN(const bf16* p, int ld, long long s = 0) {
    TcOperand o = opK(p, ld, s);
    o.mn = 1;
    return o;
}

// C[z] = A[z] B[z]^T over K columns; NTHR 128: 128 x 128 tiles of 128 threads, 0: the tile and
// threads that suit N
template <int NTHR = 0, class Epi>
cudaError_t gemm(fi_fno* h, int M, int N, int K, TcOperand A, TcOperand B, int batch, const Epi& epi) {
    TcGemmArgs g;
    g.M = M;
    g.N = N;
    g.K = K;
    g.A = A;
    g.B = B;
    g.err = h->err;
    if constexpr (NTHR == 128) return launch_gemm_tc<128, 128>(g, batch, epi, h->st);
    else return launch_gemm(g, batch, epi, h->st);
}

uint64_t splitmix64(uint64_t& s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
double unif(uint64_t& s) { return (double)(splitmix64(s) >> 11) * (1.0 / 9007199254740992.0); }

// default initialisation: pointwise layers U(-1/sqrt(fan_in), 1/sqrt(fan_in)); spectral
// weights U(0, 1/(C*C)) for the real and imaginary parts
std::vector<float> init_params(const Offsets& o, uint64_t seed) {
    std::vector<float> p(o.total);
    uint64_t s = seed;
    auto fill = [&](long long off, long long n, double lo, double hi) {
        for (long long i = 0; i < n; i++) p[off + i] = (float)(lo + (hi - lo) * unif(s));
    };
    const double a_in = 1.0 / std::sqrt((double)NIN), a_c = 1.0 / std::sqrt((double)C),
                 a_pw = 1.0 / std::sqrt((double)PW);
    fill(o.P, C * NIN, -a_in, a_in);
    fill(o.bP, C, -a_in, a_in);
    for (int l = 0; l < NLAYER; l++) {
        fill(o.layer[l], SPEC, 0.0, 1.0 / (C * C));
        fill(o.layer[l] + SPEC, C * C, -a_c, a_c);
        fill(o.layer[l] + SPEC + C * C, C, -a_c, a_c);
    }
    fill(o.Q1, PW * C, -a_c, a_c);
    fill(o.b1, PW, -a_c, a_c);
    fill(o.Q2, PW, -a_pw, a_pw);
    fill(o.b2, 1, -a_pw, a_pw);
    return p;
}

// truncated DFT matrices (FP64, rounded once to BF16); angles reduced exactly mod S
void build_dft(int S, std::vector<bf16> (&mats)[8]) {
    const double tw = 2.0 * M_PI / S, inv = 1.0 / ((double)S * S);
    auto ky_of = [S](int kyi) { return kyi < 16 ? kyi : S - KY + kyi; };
    std::vector<double> F1(32 * S), F2(64 * 2 * S), G2(2 * S * 64), G1(S * 32);
    for (int part = 0; part < 2; part++)
        for (int kx = 0; kx < KX; kx++)
            for (int x = 0; x < S; x++) {
                const double a = tw * ((kx * x) % S);
                F1[(part * 16 + kx) * S + x] = part ? -std::sin(a) : std::cos(a);
                const double w = (kx == 0 ? 1.0 : 2.0) * inv;
                G1[x * 32 + kx * 2 + part] = part ? -w * std::sin(a) : w * std::cos(a);
            }
    for (int kyi = 0; kyi < KY; kyi++)
        for (int y = 0; y < S; y++) {
            const double a = tw * (((long long)ky_of(kyi) * y) % S), c = std::cos(a), s = std::sin(a);
            // Z = sum_y (Tr + i Ti)(c - i s):  Zr = Tr c + Ti s,  Zi = -Tr s + Ti c
            F2[(kyi * 2 + 0) * 2 * S + 0 * S + y] = c;
            F2[(kyi * 2 + 0) * 2 * S + 1 * S + y] = s;
            F2[(kyi * 2 + 1) * 2 * S + 0 * S + y] = -s;
            F2[(kyi * 2 + 1) * 2 * S + 1 * S + y] = c;
            // G = sum_ky (Yr + i Yi)(c + i s):  Gr = Yr c - Yi s,  Gi = Yr s + Yi c
            G2[(0 * S + y) * 64 + kyi * 2 + 0] = c;
            G2[(0 * S + y) * 64 + kyi * 2 + 1] = -s;
            G2[(1 * S + y) * 64 + kyi * 2 + 0] = s;
            G2[(1 * S + y) * 64 + kyi * 2 + 1] = c;
        }
    auto bf = [](double d) { return __float2bfloat16_rn((float)d); };
    for (auto& m : mats) m.clear();
    mats[0].resize(32 * S);      // F1  [part*16+kx][x]
    mats[1].resize(64 * 2 * S);  // F2  [kyi*2+part'][part*S+y]
    mats[2].resize(2 * S * 64);  // G2  [y*2+part'][kyi*2+part]
    mats[3].resize(S * 32);      // G1  [x][kx*2+part]
    mats[4].resize(S * 32);      // F1T [x][kx*2+part]
    mats[5].resize(2 * S * 64);  // F2T [y*2+part][kyi*2+part']
    mats[6].resize(64 * 2 * S);  // G2T [kyi*2+part][part'*S+y]
    mats[7].resize(32 * S);      // G1T [part*16+kx][x]
    for (size_t i = 0; i < F1.size(); i++) mats[0][i] = bf(F1[i]);
    for (size_t i = 0; i < F2.size(); i++) mats[1][i] = bf(F2[i]);
    for (size_t i = 0; i < G1.size(); i++) mats[3][i] = bf(G1[i]);
    for (int x = 0; x < S; x++)
        for (int kx = 0; kx < KX; kx++)
            for (int part = 0; part < 2; part++) {
                mats[4][x * 32 + kx * 2 + part] = bf(F1[(part * 16 + kx) * S + x]);
                mats[7][(part * 16 + kx) * S + x] = bf(G1[x * 32 + kx * 2 + part]);
            }
    for (int r = 0; r < 2 * S; r++)
        for (int n = 0; n < 64; n++) {
            const int q = (r % S) * 2 + r / S;  // row (part, y) -> (y, part)
            mats[2][q * 64 + n] = bf(G2[r * 64 + n]);
            mats[5][q * 64 + n] = bf(F2[n * 2 * S + r]);
            mats[6][n * 2 * S + r] = bf(G2[r * 64 + n]);
        }
}

int pack(fi_fno* h) {
    FNO_CK(launch_dep(k_pack_spec, dim3(NM, NLAYER), 256, 0, h->st, h->params, h->o.layer[0], h->Wm, h->WmT));
    FNO_CK(launch_dep(k_pack_small, (PW * C + 255) / 256, 256, 0, h->st, h->params, h->o, h->Pb, h->Wl, h->WlT, h->Q1b,
                      h->Q1Tb));
    return FI_OK;
}

// wait for the stream; read the kernels' timeout flag and, if asked, the loss.  The flag is taken down
// for the next call; what the failed one wrote is not used: its activations serve no backward pass, and
// an Adam step (steps: those of the call) was not made.
int finish(fi_fno* h, float* loss = nullptr, int steps = 0) {
    int e = 0;
    FNO_CK(cudaMemcpyAsync(&e, h->err, sizeof(int), cudaMemcpyDeviceToHost, h->st));
    if (loss) FNO_CK(cudaMemcpyAsync(loss, h->scal, sizeof(float), cudaMemcpyDeviceToHost, h->st));
    FNO_CK(cudaStreamSynchronize(h->st));
    if (e) {
        h->fwdB = 0;
        h->adam_t -= steps;
        FNO_CK(cudaMemsetAsync(h->err, 0, sizeof(int), h->st));
        return fail(h, e, "a tensor-core GEMM wait gave up");
    }
    return FI_OK;
}

void (*dft2_kernel(int S))(Dft2Args) {
    return S == 32 ? k_dft2<32> : S == 64 ? k_dft2<64> : S == 96 ? k_dft2<96> : k_dft2<128>;
}

// truncated DFT along x and y (F1, F2), or the adjoint of the inverse (G1T, G2T), of 32 channels; m: the
// maps of v (dft2_maps)
int dft2(fi_fno* h, int B, const CUtensorMap& m, bool adjoint, const bf16* v, long long vs, bf16* Z) {
    const int S = h->S;
    if (S <= DFT2_S) {
        int CH = 8;
        while (CH > 1 && B * (C / CH) < 96) CH /= 2;
        const Dft2Args a{m, h->tm_m[adjoint ? 2 : 0], h->tm_m[adjoint ? 3 : 1], Z, B, CH, h->err, tc_wait_polls()};
        FNO_CK(launch_dep(dft2_kernel(S), B * (C / CH), 256, dft2_smem(S), h->st, a));
        return FI_OK;
    }
    const bf16 *M1 = adjoint ? h->G1T : h->F1, *M2 = adjoint ? h->G2T : h->F2;
    FNO_CK(gemm(h, C * S, 2 * KX, S, opK(v, S, vs), opK(M1, S), B, EpiDftX{h->Tb, B, S}));
    FNO_CK(gemm(h, KX * B * C, 2 * KY, 2 * S, opK(h->Tb, 2 * S), opK(M2, 2 * S), 1, EpiModes{Z, B}));
    return FI_OK;
}

// inverse DFT along x + pointwise path (m1 = G1, W) or their adjoints (F1T, WlT); v, the activation or
// gradient, by its map
template <class Epi>
int pix(fi_fno* h, int B, const CUtensorMap& m1, const CUtensorMap& v, const CUtensorMap& W, int layer, const Epi& epi) {
    const int S = h->S, ntiles = B * S * ((S + 127) / 128);
    const PixArgs a{m1, h->tm_G, v, W, S, ntiles, layer, h->err, tc_wait_polls()};
    const int grid = std::min(ntiles, PIX_BLOCKS * h->nsm);
    FNO_CK(launch_dep(pix_kb(S) == 64 ? k_pix<64, Epi> : k_pix<32, Epi>, grid, PIX_THREADS, pix_smem(S), h->st, a, epi));
    return FI_OK;
}
template <class Epi>
bool pix_attr(int S) {
    return cudaFuncSetAttribute(pix_kb(S) == 64 ? k_pix<64, Epi> : k_pix<32, Epi>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, pix_smem(256)) == cudaSuccess;
}

// the tensor maps of k_pix
bool pix_maps(fi_fno* h) {
    const int S = h->S, S2 = h->S2, KB = pix_kb(S), G1R = std::min(S, 128);
    bool ok = tma_map(&h->tm_G1, h->G1, 32, S, 32, 1, 32LL * S, 32, G1R) &&
              tma_map(&h->tm_F1T, h->F1T, 32, S, 32, 1, 32LL * S, 32, G1R) &&
              tma_map(&h->tm_G, h->Gt, 32, C, 32, h->maxB * S, 32 * C, 32, C) &&
              tma_map(&h->tm_W, h->Wl, C, C, C, NLAYER, C * C, 32, C) &&
              tma_map(&h->tm_WT, h->WlT, C, C, C, NLAYER, C * C, 32, C) &&
              tma_map(&h->tm_pdz, h->dz, S2, C, S2, h->maxB, (long long)C * S2, KB, C);
    for (int l = 0; l < NLAYER; l++)
        ok = ok && tma_map(&h->tm_pv[l], h->vext[l], S2, C, S2, h->maxB, (long long)VC * S2, KB, C);
    return ok;
}

// the tensor maps of k_dft2
bool dft2_maps(fi_fno* h) {
    const int S = h->S, S2 = h->S2, KB = dft2_kb(S);
    bool ok = true;
    for (int l = 0; l < NLAYER; l++)
        ok = ok && tma_map(&h->tm_v[l], h->vext[l], S, C * S, S, h->maxB, (long long)VC * S2, KB, 128);
    ok = ok && tma_map(&h->tm_dz, h->dz, S, C * S, S, h->maxB, (long long)C * S2, KB, 128);
    const bf16* m[4] = {h->F1, h->F2, h->G1T, h->G2T};
    for (int i = 0; i < 4; i++) {
        const int K = i % 2 ? 2 * S : S, R = i % 2 ? 2 * KY : 2 * KX;
        ok = ok && tma_map(&h->tm_m[i], m[i], K, R, K, 1, (long long)R * K, KB, R);
    }
    return ok;
}

int forward(fi_fno* h, int B, const float* x, float* y) {
    const int S = h->S, S2 = h->S2;
    const Offsets& o = h->o;
    const long long nb = (long long)B * S2, vs = (long long)VC * S2;
    k_prep_input<<<(unsigned)((nb + 255) / 256), 256, 0, h->st>>>(x, h->xe, B, S2);
    FNO_CK(cudaGetLastError());
    // lift: per sample, pixels x inputs (MN-major) times P
    FNO_CK(gemm(h, S2, C, XC, opMN(h->xe, S2, (long long)XC * S2), opK(h->Pb, XC), B,
                EpiLift{h->vext[0], h->params + o.bP, S2}));
    for (int l = 0; l < NLAYER; l++) {
        const float* lp = h->params + o.layer[l];
        const int rc = dft2(h, B, h->tm_v[l], false, h->vext[l], vs, h->Zm[l]);
        if (rc) return rc;
        // channel mixing, one batch per mode
        FNO_CK(gemm(h, B, 64, 64, opK(h->Zm[l], 64, (long long)B * 64), opK(h->Wm + (size_t)l * NM * 4096, 64, 4096),
                    NM, EpiMix{h->Yb}));
        // inverse along y: rows (b, c, kx) -> G[(b, y)][c][(kx, part)]
        FNO_CK(gemm(h, B * C * KX, 2 * S, 64, opK(h->Yb, 64), opK(h->G2, 64), 1, EpiIdftY{h->Gt, S}));
        // inverse along x + pointwise path
        const int rp = pix(h, B, h->tm_G1, h->tm_pv[l], h->tm_W, l,
                           EpiPixAct{lp + SPEC + C * C, h->zs[l], h->vext[l + 1], S, S2, l < NLAYER - 1 ? 1 : 0});
        if (rp) return rp;
    }
    // one thread sums a row's 128 columns in order: 128 threads
    FNO_CK(gemm<128>(h, S2, PW, C, opMN(h->vext[NLAYER], S2, vs), opK(h->Q1b, C), B,
                     EpiProj{h->params + o.b1, h->params + o.Q2, h->params + o.b2, y, S2, 0.f}));
    h->fwdB = B;
    return FI_OK;
}

// weight and bias gradients of a pointwise layer: dz x act (NR channels, the last one ones)
template <int NR>
int wgrad(fi_fno* h, int B, const CUtensorMap& act, int ranges, const int* map, long long base) {
    const int nz = B * h->ns;
    const WgradArgs a{h->tm_wdz, act, h->ns, nz, h->part, h->err, tc_wait_polls()};
    FNO_CK(launch_dep(k_wgrad<NR>, std::min(nz, 3 * h->nsm), WG_THREADS, wgrad_smem<NR>(), h->st, a));
    FNO_CK(reduce_map(h->part, h->st, nz, C * NR, ranges, map, h->grads, base));
    return FI_OK;
}

// the tensor maps of k_wgrad
bool wgrad_maps(fi_fno* h) {
    const int S2 = h->S2;
    bool ok = tma_map(&h->tm_wdz, h->dz, S2, C, S2, h->maxB, (long long)C * S2, WG_BOX, C) &&
              tma_map(&h->tm_wx, h->xe, S2, XC, S2, h->maxB, (long long)XC * S2, WG_BOX, NIN + 1);
    for (int l = 0; l < NLAYER; l++)
        ok = ok && tma_map(&h->tm_wv[l], h->vext[l], S2, VC, S2, h->maxB, (long long)VC * S2, WG_BOX, C + 1);
    return ok;
}

// gradients of all parameters from dq (and its BF16 copy) set by k_loss
int backward(fi_fno* h, int B) {
    const int S = h->S, S2 = h->S2;
    const Offsets& o = h->o;
    const long long cs = (long long)C * S2;
    float* gr = h->grads;
    const ProjBwdArgs pb{h->vext[NLAYER], h->Q1b, h->Q1Tb, h->params + o.b1, h->params + o.Q2, h->dq, h->dz, h->part, S2,
                         B * h->ns, h->err, tc_wait_polls()};
    FNO_CK(launch_dep(k_proj_bwd, std::min(pb.nslices, 2 * h->nsm), 256, PB_SMEM, h->st, pb));
    FNO_CK(reduce_map(h->part, h->st, B * h->ns, PW * VC, 16, h->map_proj, gr, 0));
    for (int l = NLAYER - 1; l >= 0; l--) {
        // pointwise path weights and bias: [co][ci | ones]
        int rc = wgrad<C + 1>(h, B, h->tm_wv[l], 32, h->map_loc, o.layer[l]);
        if (rc) return rc;
        // spectral path: adjoint of the inverse DFT along x, then along y
        rc = dft2(h, B, h->tm_dz, true, h->dz, cs, h->dYm);
        if (rc) return rc;
        FNO_CK(launch_dep(k_spec_wgrad, NM, 256, 0, h->st, h->Zm[l], h->dYm, gr + o.layer[l], B));
        // adjoint of the channel mixing and of the DFT along y
        FNO_CK(gemm(h, B, 64, 64, opK(h->dYm, 64, (long long)B * 64), opK(h->WmT + (size_t)l * NM * 4096, 64, 4096),
                    NM, EpiMix{h->Yb}));
        FNO_CK(gemm(h, B * C * KX, 2 * S, 64, opK(h->Yb, 64), opK(h->F2T, 64), 1, EpiIdftY{h->Gt, S}));
        // adjoint of the DFT along x + the pointwise path; then the activation of the layer below (the
        // lift has none)
        rc = pix(h, B, h->tm_F1T, h->tm_pdz, h->tm_WT, l, EpiPixBwd{l > 0 ? h->zs[l - 1] : nullptr, h->dz, S, S2});
        if (rc) return rc;
    }
    // lift weights and bias: [c][inputs | ones]
    return wgrad<NIN + 1>(h, B, h->tm_wx, 64, h->map_lift, 0);
}

int set_loss(fi_fno* h, int B, const float* target, const float* w, const float* dy) {
    const int n = B * h->S2;
    // per-block partials in the split-K scratch (free until the backward pass)
    const int nblk = (n + 255) / 256;
    FNO_CK(launch_dep(k_loss, nblk, 256, 0, h->st, h->q, target, w, dy, n, h->S2, 1.f / n, h->dq, h->vext[NLAYER],
                      h->part));
    FNO_CK(launch_dep(k_loss_sum, 1, 256, 0, h->st, h->part, nblk, h->scal, h->grads + h->o.b2));
    return FI_OK;
}

int adam(fi_fno* h, float lr) {
    h->adam_t++;
    const float c1 = (float)(1.0 / (1.0 - std::pow((double)h->beta1, (double)h->adam_t)));
    const float c2 = (float)(1.0 / (1.0 - std::pow((double)h->beta2, (double)h->adam_t)));
    FNO_CK(launch_dep(k_adam, 148 * 8, 256, 0, h->st, h->params, h->grads, h->m, h->v, h->o.total, lr, h->beta1, h->beta2,
                      h->eps, c1, c2, h->err));
    return pack(h);
}

int check_batch(fi_fno* h, int B) {
    if (B < 1 || B > h->maxB) return fail(h, FI_ERR_ARG, "batch outside [1, max_batch]");
    return FI_OK;
}

}  // namespace

extern "C" {

int fi_fno_create(int32_t S, int32_t max_batch, int32_t device, uint64_t seed, fi_fno** out) {
    if (!out) return FI_ERR_ARG;
    *out = nullptr;
    if (S < 32 || S > 256 || S % 32 || max_batch < 1 || max_batch > 256) return FI_ERR_ARG;
    fi_fno* h = new fi_fno();
    h->S = S;
    h->S2 = S * S;
    h->maxB = max_batch;
    h->device = device;
    h->o = offsets();
    h->ns = h->S2 / SLICE;
    auto bad = [&](int rc) {
        fi_fno_destroy(h);
        return rc;
    };
    if (cudaSetDevice(device) != cudaSuccess) return bad(FI_ERR_CUDA);
    if (cudaStreamCreateWithFlags(&h->st, cudaStreamDefault) != cudaSuccess) return bad(FI_ERR_CUDA);
    if (cudaDeviceGetAttribute(&h->nsm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaFuncSetAttribute(k_proj_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, PB_SMEM) != cudaSuccess ||
        (S <= DFT2_S && cudaFuncSetAttribute(dft2_kernel(S), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             dft2_smem(S)) != cudaSuccess) ||
        !pix_attr<EpiPixAct>(S) || !pix_attr<EpiPixBwd>(S) ||
        cudaFuncSetAttribute(k_wgrad<C + 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, wgrad_smem<C + 1>()) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_wgrad<NIN + 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, wgrad_smem<NIN + 1>()) !=
            cudaSuccess)
        return bad(FI_ERR_CUDA);
    const long long B = max_batch, S2 = h->S2, P = h->o.total;
    bool ok = dalloc(h, &h->params, P) == cudaSuccess && dalloc(h, &h->grads, P) == cudaSuccess &&
              dalloc(h, &h->m, P) == cudaSuccess && dalloc(h, &h->v, P) == cudaSuccess &&
              dalloc(h, &h->Pb, C * XC) == cudaSuccess && dalloc(h, &h->Wm, (size_t)NLAYER * NM * 4096) == cudaSuccess &&
              dalloc(h, &h->WmT, (size_t)NLAYER * NM * 4096) == cudaSuccess &&
              dalloc(h, &h->Wl, NLAYER * C * C) == cudaSuccess && dalloc(h, &h->WlT, NLAYER * C * C) == cudaSuccess &&
              dalloc(h, &h->Q1b, PW * C) == cudaSuccess && dalloc(h, &h->Q1Tb, PW * C) == cudaSuccess &&
              dalloc(h, &h->F1, 32 * S) == cudaSuccess && dalloc(h, &h->F2, 128 * S) == cudaSuccess &&
              dalloc(h, &h->G2, 128 * S) == cudaSuccess && dalloc(h, &h->G1, 32 * S) == cudaSuccess &&
              dalloc(h, &h->F1T, 32 * S) == cudaSuccess && dalloc(h, &h->F2T, 128 * S) == cudaSuccess &&
              dalloc(h, &h->G2T, 128 * S) == cudaSuccess && dalloc(h, &h->G1T, 32 * S) == cudaSuccess &&
              dalloc(h, &h->xe, B * XC * S2) == cudaSuccess &&
              dalloc(h, &h->Tb, S > DFT2_S ? (size_t)KX * B * C * 2 * S : 1) == cudaSuccess &&
              dalloc(h, &h->Yb, (size_t)B * C * KX * 64) == cudaSuccess &&
              dalloc(h, &h->Gt, (size_t)B * C * S * 32) == cudaSuccess &&
              dalloc(h, &h->dz, (size_t)B * C * S2) == cudaSuccess &&
              dalloc(h, &h->dYm, (size_t)NM * B * 64) == cudaSuccess &&
              dalloc(h, &h->q, (size_t)B * S2) == cudaSuccess &&
              dalloc(h, &h->dq, (size_t)B * S2) == cudaSuccess &&
              dalloc(h, &h->part, (size_t)B * h->ns * PW * VC) == cudaSuccess &&
              dalloc(h, &h->scal, 4) == cudaSuccess && dalloc(h, &h->map_loc, C * (C + 1)) == cudaSuccess &&
              dalloc(h, &h->map_proj, PW * VC) == cudaSuccess && dalloc(h, &h->map_lift, C * (NIN + 1)) == cudaSuccess &&
              dalloc(h, &h->err, 1) == cudaSuccess;
    for (int l = 0; l <= NLAYER && ok; l++) ok = dalloc(h, &h->vext[l], (size_t)B * VC * S2) == cudaSuccess;
    for (int l = 0; l < NLAYER && ok; l++)
        ok = dalloc(h, &h->zs[l], (size_t)B * C * S2) == cudaSuccess &&
             dalloc(h, &h->Zm[l], (size_t)NM * B * 64) == cudaSuccess;
    if (!ok || !pix_maps(h) || !wgrad_maps(h) || (S <= DFT2_S && !dft2_maps(h))) return bad(FI_ERR_CUDA);
    // DFT matrices
    std::vector<bf16> mats[8];
    build_dft(S, mats);
    bf16* dst[8] = {h->F1, h->F2, h->G2, h->G1, h->F1T, h->F2T, h->G2T, h->G1T};
    for (int i = 0; i < 8; i++)
        if (cudaMemcpy(dst[i], mats[i].data(), mats[i].size() * sizeof(bf16), cudaMemcpyHostToDevice) != cudaSuccess)
            return bad(FI_ERR_CUDA);
    // split-K gradient maps (targets relative to the base passed to k_reduce_map)
    const Offsets& o = h->o;
    std::vector<int> ml(C * (C + 1)), mp(PW * VC), mf(C * (NIN + 1));
    for (int co = 0; co < C; co++)
        for (int k = 0; k <= C; k++) ml[co * (C + 1) + k] = (int)(k < C ? SPEC + co * C + k : SPEC + C * C + co);
    for (int j = 0; j < PW; j++) {
        for (int c = 0; c < C; c++) mp[j * VC + c] = (int)(o.Q1 + j * C + c);
        mp[j * VC + C] = (int)(o.b1 + j);
        mp[j * VC + C + 1] = (int)(o.Q2 + j);
    }
    for (int c = 0; c < C; c++) {
        for (int k = 0; k < NIN; k++) mf[c * (NIN + 1) + k] = (int)(o.P + c * NIN + k);
        mf[c * (NIN + 1) + NIN] = (int)(o.bP + c);
    }
    if (cudaMemcpy(h->map_loc, ml.data(), ml.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->map_proj, mp.data(), mp.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(h->map_lift, mf.data(), mf.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess)
        return bad(FI_ERR_CUDA);
    // ones channel of every NCHW activation buffer (bias gradients)
    for (int l = 0; l <= NLAYER; l++) k_fill_channel<<<(unsigned)((B * S2 + 255) / 256), 256, 0, h->st>>>(
        h->vext[l], (int)B, (int)S2, C, 1.f);
    std::vector<float> p0 = init_params(o, seed);
    if (cudaMemcpy(h->params, p0.data(), P * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess)
        return bad(FI_ERR_CUDA);
    if (pack(h) != FI_OK || finish(h) != FI_OK) return bad(FI_ERR_CUDA);
    *out = h;
    return FI_OK;
}

int64_t fi_fno_num_params(const fi_fno* h) { return h ? h->o.total : -1; }

int fi_fno_get_params(fi_fno* h, float* out, int64_t n) {
    if (!h || !out || n != h->o.total) return fail(h, FI_ERR_ARG, "parameter count");
    FNO_CK(cudaSetDevice(h->device));
    FNO_CK(cudaStreamSynchronize(h->st));
    FNO_CK(cudaMemcpy(out, h->params, n * sizeof(float), cudaMemcpyDeviceToHost));
    return FI_OK;
}

int fi_fno_set_params(fi_fno* h, const float* in, int64_t n) {
    if (!h || !in || n != h->o.total) return fail(h, FI_ERR_ARG, "parameter count");
    FNO_CK(cudaSetDevice(h->device));
    FNO_CK(cudaStreamSynchronize(h->st));
    FNO_CK(cudaMemcpy(h->params, in, n * sizeof(float), cudaMemcpyHostToDevice));
    FNO_CK(cudaMemset(h->m, 0, n * sizeof(float)));
    FNO_CK(cudaMemset(h->v, 0, n * sizeof(float)));
    h->adam_t = 0;
    h->fwdB = 0;
    int rc = pack(h);
    return rc ? rc : finish(h);
}

int fi_fno_get_grads(fi_fno* h, float* out, int64_t n) {
    if (!h || !out || n != h->o.total) return fail(h, FI_ERR_ARG, "parameter count");
    FNO_CK(cudaSetDevice(h->device));
    FNO_CK(cudaStreamSynchronize(h->st));
    FNO_CK(cudaMemcpy(out, h->grads, n * sizeof(float), cudaMemcpyDeviceToHost));
    return FI_OK;
}

int fi_fno_forward(fi_fno* h, int32_t B, const float* x, float* y) {
    if (!h || !x || !y) return fail(h, FI_ERR_ARG, "null pointer");
    int rc = check_batch(h, B);
    if (rc) return rc;
    FNO_CK(cudaSetDevice(h->device));
    rc = forward(h, B, x, y);
    return rc ? rc : finish(h);
}

int fi_fno_backward(fi_fno* h, int32_t B, const float* dy) {
    if (!h || !dy) return fail(h, FI_ERR_ARG, "null pointer");
    if (B != h->fwdB) return fail(h, FI_ERR_STATE, "backward needs a forward pass of the same batch");
    FNO_CK(cudaSetDevice(h->device));
    int rc = set_loss(h, B, nullptr, nullptr, dy);
    if (!rc) rc = backward(h, B);
    return rc ? rc : finish(h);
}

int fi_fno_train_step(fi_fno* h, int32_t B, const float* x, const float* target, float lr, float* loss) {
    return fi_fno_train_step_weighted(h, B, x, target, nullptr, lr, loss);
}

int fi_fno_train_step_weighted(fi_fno* h, int32_t B, const float* x, const float* target, const float* w, float lr,
                               float* loss) {
    if (!h || !x || !target) return fail(h, FI_ERR_ARG, "null pointer");
    int rc = check_batch(h, B);
    if (rc) return rc;
    FNO_CK(cudaSetDevice(h->device));
    rc = forward(h, B, x, h->q);
    if (!rc) rc = set_loss(h, B, target, w, nullptr);
    if (!rc) rc = backward(h, B);
    if (!rc) rc = adam(h, lr);
    if (!rc) rc = finish(h, loss, 1);
    return rc;
}

int fi_fno_loss_backward(fi_fno* h, int32_t B, const float* x, const float* target, const float* w, float* loss) {
    if (!h || !x || !target) return fail(h, FI_ERR_ARG, "null pointer");
    int rc = check_batch(h, B);
    if (rc) return rc;
    FNO_CK(cudaSetDevice(h->device));
    rc = forward(h, B, x, h->q);
    if (!rc) rc = set_loss(h, B, target, w, nullptr);
    if (!rc) rc = backward(h, B);
    if (!rc) rc = finish(h, loss);
    return rc;
}

void* fi_fno_grads_device(fi_fno* h) { return h ? (void*)h->grads : nullptr; }

int fi_fno_adam(fi_fno* h, float lr) {
    if (!h) return FI_ERR_ARG;
    FNO_CK(cudaSetDevice(h->device));
    int rc = adam(h, lr);
    return rc ? rc : finish(h, nullptr, 1);
}

int fi_fno_set_adam(fi_fno* h, float beta1, float beta2, float eps) {
    if (!h || !(beta1 >= 0.f && beta1 < 1.f) || !(beta2 >= 0.f && beta2 < 1.f) || !(eps > 0.f))
        return fail(h, FI_ERR_ARG, "Adam hyper-parameters");
    h->beta1 = beta1;
    h->beta2 = beta2;
    h->eps = eps;
    return FI_OK;
}

const char* fi_fno_last_error(const fi_fno* h) { return h ? h->msg.c_str() : "null handle"; }

void fi_fno_destroy(fi_fno* h) {
    if (!h) return;
    cudaSetDevice(h->device);
    if (h->st) cudaStreamSynchronize(h->st);
    for (void* p : h->allocs) cudaFree(p);
    if (h->st) cudaStreamDestroy(h->st);
    delete h;
}

}  // extern "C"
