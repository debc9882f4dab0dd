// fno_gemm.cuh -- BF16 x BF16 -> FP32 GEMM on the 5th-generation tensor cores (tcgen05)
// for the Fourier-neural-operator surrogate.
//
//   C[z][m][n] = sum_k A[z][m][k] * B[z][n][k]
//
// Output tiles of 128 x BN.  Per K chunk of at most 64 a block copies its A and B rows into
// shared memory with cp.async (16-byte copies) in the no-swizzle canonical layout of the UMMA
// operand descriptors (8-row x 16-byte core matrices; the core matrices of one 8-row group follow
// each other along K at LBO bytes, the 8-row groups at SBO bytes); one elected thread issues a
// tcgen05.mma per 16 columns (kind::f16, BF16 inputs, FP32 accumulation in tensor memory) and
// commits them to an mbarrier.  The finished accumulator is read with tcgen05.ld (a warp owns the
// 32 TMEM lanes of its quarter) and each row's values go to an epilogue functor.  Every mbarrier
// wait is bounded: on expiry the block raises an error word, waits for its copies, frees its
// tensor memory and returns.
//
// The products of the surrogate are small (K of 8 to 512, mostly one chunk), so a tile's time is
// the latency of copy, MMA and epilogue in a row; what counts is how many tiles an SM works on at
// once and how little a tile costs beside its epilogue.  So only the K columns, rows and stages
// that a product has take copies and shared memory, and blocks walk tiles (launch_gemm_nb).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "../../include/fastiso_b200.h"

namespace fi {

constexpr int TC_BM = 128;       // tile rows (UMMA M)
constexpr int TC_BK = 64;        // K per chunk (4 UMMA of K = 16)
constexpr int TC_THREADS = 128;  // one warpgroup
constexpr long long TC_SPIN_LIMIT = 1LL << 26;

// K-major no-swizzle operand layout of `rows` rows x 64 K elements (BF16): byte offset of
// element (r, k).  Core matrix (8 rows x 8 elements = 128 B) of row group g, K group c
// at c * (rows * 16) + g * 128; inside it row r % 8 at 16 B steps.
__host__ __device__ inline uint32_t tc_operand_offset(int rows, int r, int k) {
    return (uint32_t)((k >> 3) * (rows * 16) + (r >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// UMMA shared-memory descriptor (sm_100): start >> 4 in bits [0,14), LBO >> 4 in [16,30),
// SBO >> 4 in [32,46), version 1 in [46,48), layout type 0 (no swizzle) in [61,64).
__host__ __device__ inline uint64_t tc_smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// UMMA instruction descriptor, kind::f16: FP32 accumulator, BF16 A and B, both K-major,
// N >> 3 in bits [17,23), M >> 4 in bits [24,29).
__host__ __device__ inline uint32_t tc_instr_desc(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}


// ---------------------------------------------------------------------------
// PTX wrappers (sm_100a)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t tc_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem_u32(bar)), "r"(count) : "memory");
}

// true when the phase with the given parity has completed
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(tc_smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait of at most `polls` tests; false when the limit ran out
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long polls = TC_SPIN_LIMIT) {
    for (long long i = 0; i < polls; i++)
        if (mbar_test(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_alloc(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(dst_smem)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tc_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem_u32(bar))
                 : "memory");
}

// ---------------------------------------------------------------------------
// TMA operands: boxes of `rows` rows x KB elements (KB = 64 or 32: 128- or 64-byte rows) of a K-major
// BF16 tensor (x, row, depth), one after another in shared memory (1024-byte aligned) with the
// swizzle of their row size, which is also the operand layout of the descriptor below.
// ---------------------------------------------------------------------------
// inner: row length and box columns start at multiples of KB; pitch, dpitch: elements between rows and
// between depths (multiples of 8).  Rows of a box beyond `rows` are filled with zeros.
inline bool tma_map(CUtensorMap* m, const void* p, int inner, int rows, long long pitch, int depth, long long dpitch,
                    int KB, int box_rows) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode f = [] {
        void* e = nullptr;
        cudaDriverEntryPointQueryResult q;
        const cudaError_t r = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &e, cudaEnableDefault, &q);
        return r == cudaSuccess && q == cudaDriverEntryPointSuccess ? (Encode)e : nullptr;
    }();
    if (!f) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)rows, (cuuint64_t)depth};
    const cuuint64_t strides[2] = {(cuuint64_t)pitch * 2, (cuuint64_t)dpitch * 2};
    const cuuint32_t box[3] = {(cuuint32_t)KB, (cuuint32_t)box_rows, 1}, one[3] = {1, 1, 1};
    return f(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(p), dims, strides, box, one,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, KB == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// descriptor of 16 K columns of such a box: 8-row groups 16 KB bytes apart, rows inside them swizzled.
// The next 16 columns of the box start 32 bytes on.
template <int KB>
__device__ __forceinline__ uint64_t tma_desc(uint32_t saddr) {
    return tc_smem_desc(saddr, 16, 16 * KB) | ((uint64_t)(KB == 64 ? 2 : 4) << 61);
}

// the same for an MN-major operand: boxes of KB elements along M x 32 K columns, `lbo` bytes apart along
// M; 16 columns are two groups of 8, 16 KB bytes apart
template <int KB>
__device__ __forceinline__ uint64_t tma_desc_mn(uint32_t saddr, uint32_t lbo) {
    return tc_smem_desc(saddr, lbo, 16 * KB) | ((uint64_t)(KB == 64 ? 2 : 4) << 61);
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, int x, int row, int depth, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(x), "r"(row), "r"(depth), "r"(tc_smem_u32(bar))
        : "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float* v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// ---------------------------------------------------------------------------
// programmatic dependent launch: a kernel's blocks may start while the kernel before it in the
// stream still runs.  Each one calls dep_wait() before its first access to global memory that
// another kernel touches (it returns when the kernels before have completed and their writes are
// visible).  It calls dep_launch() after that -- and after it has its tensor memory, which a waiting
// block of the next kernel must not hold in its place: at once if the grid has at most one block
// an SM (dep_early) or its blocks have one short piece of work each (the element-wise kernels), else
// when the block's tiles are done.  One thread's call counts for its block.  (Blocks of the next
// kernel that start early gather on the SMs that are free first and then walk their equal shares
// there: 32 samples of 128 x 128, every product a tile-walking GEMM, inference 659 us with the late
// call, 793 with the early one, 695 without.  In k_pix and k_wgrad alone it makes no difference:
// 462 and 466 us, training step 1176 and 1185.)  What overlaps is the launch latency and the
// prologue.  One 64 x 64 sample: 228 -> 170 us; training step of 7 samples of 96 x 96: 768 -> 612 us.
// ---------------------------------------------------------------------------
constexpr unsigned DEP_EARLY_BLOCKS = 148;
__device__ __forceinline__ bool dep_early() { return gridDim.x <= DEP_EARLY_BLOCKS; }
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t launch_dep(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

// ---------------------------------------------------------------------------
// the GEMM
// ---------------------------------------------------------------------------
// One GEMM operand.  K-major (mn = 0): element (r, k) of batch z at p[z * s + r * ld + k], rows
// K-contiguous.  MN-major (mn = 1): at p[z * s + k * ld + r], each K column contiguous along the rows (an NCHW
// activation read as pixels x channels).  The tensor cores take either form: the shared
// memory image keeps the same core-matrix grid and only the inside of each 128-byte
// core matrix is transposed, which bit 15 (A) / 16 (B) of the instruction descriptor
// announces.
struct TcOperand {
    const __nv_bfloat16* p = nullptr;
    int ld = 0;
    long long s = 0;
    int mn = 0;
};

struct TcGemmArgs {
    int M = 0, N = 0, K = 0;
    TcOperand A, B;
    int batch = 1;
    int* err = nullptr;  // set to FI_ERR_TIMEOUT when a wait gives up
    long long polls = TC_SPIN_LIMIT;  // bound of each commit wait (tc_wait_polls())
};

// Poll bound of the commit waits for the next launches: TC_SPIN_LIMIT unless a test
// lowered it with fi_debug_set_wait_limit (fno_gemm.cu).
long long tc_wait_polls();

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// kc (<= 64, a multiple of 16) product columns from k0 of one side (A or B) of the product into
// the canonical layout at shared address dst, zero outside [0, K).  Rows at or beyond nrows are
// not copied: what the buffer holds there only reaches accumulator rows or columns that no epilogue
// reads.  The rows of an MN-major operand are copied in groups of 8, so their number is a multiple of
// 8, as every K is (fi_fno_gemm refuses others).  `safe` is any valid global address (the source
// operand of a zero-filled copy, never read).
template <int ROWS, int NTHR>
__device__ __forceinline__ void tc_stage(uint32_t dst, const TcOperand& o, int z, int row0, int nrows, int k0, int kc,
                                         int K, const void* safe) {
    const int left = nrows - row0;
    if (!o.mn) {
        // one 16-byte copy = 8 consecutive K elements of one row; a thread keeps its K group.  Eight
        // neighbouring threads take the eight rows of one core matrix (contiguous in shared memory: no
        // bank conflicts), the next eight the next K group (contiguous in global memory).
        const int sh = kc <= 16 ? 1 : kc <= 32 ? 2 : 3;
        const int kv = (threadIdx.x >> 3) & ((1 << sh) - 1), gk = k0 + kv * 8;
        if (kv * 8 < kc) {
            const bool kok = gk < K;
            const int r_ = (threadIdx.x >> (3 + sh)) * 8 + (threadIdx.x & 7), step = NTHR >> sh;
            const int rows = left < ROWS ? left : ROWS;
            const __nv_bfloat16* src = o.p + (size_t)z * o.s + gk + (size_t)(row0 + r_) * o.ld;
            const size_t sstep = (size_t)step * o.ld;
            for (int r = r_; r < rows; r += step, src += sstep)
                cp_async16(dst + tc_operand_offset(ROWS, r, kv * 8), kok ? (const void*)src : safe, kok);
        }
    } else {
        // one 16-byte copy = 8 consecutive rows of one K column, stored as row (k % 8) of core matrix
        // (k / 8, r / 8); eight neighbouring threads take the eight columns of one core matrix
        constexpr int RV = ROWS / 8;
        for (int v = threadIdx.x; v < RV * kc; v += NTHR) {
            const int rv = (v >> 3) % RV, kc_ = v / (8 * RV) * 8 + (v & 7);
            const int gk = k0 + kc_;
            if (rv * 8 >= left) continue;
            const bool ok = gk < K;
            const void* src = ok ? (const void*)(o.p + (size_t)z * o.s + (size_t)gk * o.ld + row0 + rv * 8) : safe;
            cp_async16(dst + (kc_ >> 3) * (ROWS * 16) + rv * 128 + (kc_ & 7) * 16, src, ok);
        }
    }
}

// Blocks of NTHR threads walk the output tiles with the grid's stride (tile index: row tile
// fastest, then column tile, then batch).  128 threads: warp w reads accumulator rows 32 (w % 4)
// and all BN columns; 256: warps w and w + 4 share the rows and take half the columns each, which
// doubles the warps where tensor memory (512 columns an SM) holds only four 128-column tiles.
// NB stage buffers: with one (K of a single chunk) the next tile's copies start when the tile's
// MMAs are done and run beside its epilogue; with two, one chunk ahead of the MMAs.
template <int BN, int NTHR, int NB, class Epi>
__global__ void __launch_bounds__(NTHR) k_gemm_tc(const __grid_constant__ TcGemmArgs g, Epi epi) {
    static_assert(NTHR == 128 || NTHR == 256, "one or two warpgroups");
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t tmem_base;
    __shared__ int s_fail;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nch = NB == 1 ? 1 : (g.K + TC_BK - 1) / TC_BK;
    const int kc0 = g.K < TC_BK ? (g.K + 15) & ~15 : TC_BK;  // columns of a full chunk
    const uint32_t a_bytes = TC_BM * 2 * kc0, stage_bytes = a_bytes + BN * 2 * kc0;
    const uint32_t sbase = tc_smem_u32(smem);
    // 32-bit arithmetic: the launch checks that the tiles fit
    const unsigned mt = (unsigned)(g.M + TC_BM - 1) / TC_BM, nt = (unsigned)(g.N + BN - 1) / BN;
    const unsigned ntiles = mt * nt * (unsigned)g.batch;
    // an operand that is the same for every tile is copied once, where its chunks keep their buffer
    const bool keep = nch <= NB;
    const bool fixA = keep && mt == 1 && g.A.s == 0, fixB = keep && nt == 1 && g.B.s == 0;
    int m0 = 0, n0 = 0, z = 0;  // the tile whose chunks are being copied
    auto stage = [&](unsigned tile, int c, int buf, bool first) {
        if (c == 0) {
            const unsigned mnt = mt * nt, zt = tile / mnt, mn = tile - zt * mnt, nq = mn / mt;
            z = (int)zt;
            m0 = (int)(mn - nq * mt) * TC_BM;
            n0 = (int)nq * BN;
        }
        const uint32_t sa = sbase + (uint32_t)buf * stage_bytes;
        const int left = g.K - c * TC_BK, kc = left < kc0 ? (left + 15) & ~15 : kc0;
        if (first || !fixA) tc_stage<TC_BM, NTHR>(sa, g.A, z, m0, g.M, c * TC_BK, kc, g.K, g.A.p);
        if (first || !fixB) tc_stage<BN, NTHR>(sa + a_bytes, g.B, z, n0, g.N, c * TC_BK, kc, g.K, g.A.p);
        cp_async_commit();
    };
    unsigned tile = blockIdx.x;
    if (warp == 0) {
        tc_alloc(&tmem_base, BN < 32 ? 32 : BN);
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
    if (tile < ntiles) stage(tile, 0, 0, true);
    const uint32_t tmem = tmem_base;
    const uint32_t idesc = tc_instr_desc(TC_BM, BN);
    int j = 0;  // chunks so far over all tiles; chunk j uses buffer j % NB
    int last_commit = -1;  // thread 0: the last chunk whose MMAs were committed
    for (; tile < ntiles; tile += gridDim.x) {
        const int tm0 = m0, tn0 = n0, tz = z;
        const bool more = tile + gridDim.x < ntiles;
        bool fail = false;  // s_fail as read directly behind its barrier: thread 0 may set it again before the next one
        for (int c = 0; c < nch; c++, j++) {
            if (NB == 2 && (c + 1 < nch || more)) {
                // the other stage buffer was last read by the MMAs of chunk j - 1
                if (j >= 1) {
                    if (tid == 0 && !mbar_wait(&bars[(j - 1) & 1], (uint32_t)(((j - 1) >> 1) & 1), g.polls)) s_fail = 1;
                    __syncthreads();
                    if (s_fail) {
                        fail = true;
                        break;
                    }
                }
                const bool next = c + 1 == nch;
                stage(next ? tile + gridDim.x : tile, next ? 0 : c + 1, (j + 1) & 1, j + 1 < nch);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            fence_async_smem();
            __syncthreads();
            if (tid == 0) {
                tc_fence_after();
                const int buf = NB == 2 ? j & 1 : 0;
                const uint32_t a0 = sbase + (uint32_t)buf * stage_bytes, b0 = a0 + a_bytes;
                const int left = g.K - c * TC_BK, nks = ((left < kc0 ? left : kc0) + 15) >> 4;
                for (int ks = 0; ks < nks; ks++) {
                    // K step ks covers core-matrix columns 2ks and 2ks + 1
                    const uint64_t da = tc_smem_desc(a0 + 2 * ks * (TC_BM * 16), TC_BM * 16, 128);
                    const uint64_t db = tc_smem_desc(b0 + 2 * ks * (BN * 16), BN * 16, 128);
                    tc_mma(tmem, da, db, idesc | ((uint32_t)g.A.mn << 15) | ((uint32_t)g.B.mn << 16),
                           (c > 0 || ks > 0) ? 1u : 0u);
                }
                tc_commit(&bars[j & 1]);
                last_commit = j;
            }
        }
        if (fail) break;
        // tile complete: wait for its MMAs, read the accumulator, hand rows to the epilogue
        if (tid == 0 && !mbar_wait(&bars[(j - 1) & 1], (uint32_t)(((j - 1) >> 1) & 1), g.polls)) s_fail = 1;
        __syncthreads();
        if (s_fail) break;
        tc_fence_after();
        if (NB == 1 && more) stage(tile + gridDim.x, 0, 0, false);
        Epi e = epi;  // per tile: the epilogue may carry per-row state across its column chunks
        constexpr int CW = NTHR == 256 ? BN / 2 : BN;  // columns a warp reads
        const int quad = warp & 3, cb = (warp >> 2) * CW, row = tm0 + quad * 32 + lane;
        if constexpr (Epi::PAIR) {
            // columns c and c + BN / 2 together (N == BN)
            static_assert(NTHR == 128, "one warp reads both halves");
            for (int c0 = 0; c0 < BN / 2; c0 += 16) {
                float v[16], w[16];
                tc_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
                tc_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(c0 + BN / 2), w);
                if (row < g.M) e.pair(tz, row, c0, v, w);
            }
        } else {
            for (int c0 = cb; c0 < cb + CW; c0 += 16) {
                float v[16];
                tc_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
                if (row < g.M && tn0 + c0 < g.N) e(tz, row, tn0 + c0, v, g.N - (tn0 + c0));
            }
        }
        if (warp < 4 && row < g.M) e.row_done(tz, row);
        tc_fence_before();
        __syncthreads();  // the next tile's MMAs overwrite the accumulator
    }
    if (!dep_early()) dep_launch();
    cp_async_wait<0>();
    if (s_fail && tid == 0) {
        if (g.err) atomicExch(g.err, FI_ERR_TIMEOUT);
        // before the tensor memory is released, let the MMAs already issued finish
        // (their commit completes every earlier tcgen05 operation of this thread);
        // bounded again, with the full limit
        if (last_commit >= 0) mbar_wait(&bars[last_commit & 1], (uint32_t)((last_commit >> 1) & 1));
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tc_dealloc(tmem, BN < 32 ? 32 : BN);
}

// plain FP32 store: C[z][row][col], pitch ldc
struct EpiBase {
    static constexpr bool PAIR = false;  // true: pair(z, row, col, v, w) with the columns col and col + BN / 2
};
struct EpiStoreF32 : EpiBase {
    EpiStoreF32(float* C_, int ldc_, long long sC_) : C(C_), ldc(ldc_), sC(sC_) {}
    float* C;
    int ldc;
    long long sC;
    __device__ __forceinline__ void operator()(int z, int row, int col0, const float* v, int nvalid) const {
        float* c = C + (size_t)z * sC + (size_t)row * ldc + col0;
        if (nvalid >= 16 && ((uintptr_t)c & 15) == 0) {
            float4* c4 = reinterpret_cast<float4*>(c);
#pragma unroll
            for (int q = 0; q < 4; q++) c4[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            return;
        }
#pragma unroll
        for (int i = 0; i < 16; i++)
            if (i < nvalid) c[i] = v[i];
    }
    __device__ __forceinline__ void row_done(int, int) const {}
};

// Launch: at most one block per tile, and at most TC_BLOCKS_SM an SM or as many as fit (shared
// memory, registers, tensor memory; cudaOccupancyMaxActiveBlocksPerMultiprocessor answers 1 for
// kernels that allocate tensor memory, although more run).  A block that walks several tiles pays
// its launch, its tensor-memory allocation and the copies of fixed operands once, and several
// blocks an SM overlap one's epilogue with another's copies and MMAs.  One block per tile kept an
// SM at 2.7 blocks of 10 that fit (launches could not keep up): inverse x + pointwise product of
// 32 samples of 128 x 128, 4096 tiles: 83 -> 58 us, its adjoint 60 -> 38 us, lift 48 -> 27 us.
// Blocks an SM, us per inference / training step of that batch (final kernels): 4 614 / 1500, 6 619 /
// 1503, 8 603 / 1485, 10 596 / 1475.
constexpr int TC_BLOCKS_SM = 10;
template <int BN, int NTHR, int NB, class Epi>
inline cudaError_t launch_gemm_nb(const TcGemmArgs& g, int batch, const Epi& epi, cudaStream_t st) {
    const int kc0 = g.K < TC_BK ? (g.K + 15) & ~15 : TC_BK;
    const int smem = (TC_BM + BN) * kc0 * 2 * NB;
    // per device: blocks that fit the GPU with this many 16-column K steps (0: not yet asked)
    static std::atomic<int> fit[32][5];
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 32) return cudaErrorInvalidDevice;
    int blocks = fit[dev][kc0 / 16].load();
    if (blocks == 0) {
        int nsm = 0, smax = 0;
        cudaFuncAttributes fa{};
        e = cudaFuncGetAttributes(&fa, k_gemm_tc<BN, NTHR, NB, Epi>);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_gemm_tc<BN, NTHR, NB, Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     NB * (TC_BM + BN) * TC_BK * 2);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        if (e != cudaSuccess) return e;
        const int regs = (fa.numRegs + 7) / 8 * 8;
        int occ = std::min(TC_BLOCKS_SM, 512 / (BN < 32 ? 32 : BN));
        occ = std::min(occ, smax / (smem + (int)fa.sharedSizeBytes + 1024));
        occ = std::min(occ, 65536 / (regs * NTHR));
        blocks = nsm * std::max(1, occ);
        fit[dev][kc0 / 16].store(blocks);
    }
    TcGemmArgs a = g;
    a.batch = batch;
    a.polls = tc_wait_polls();
    const long long ntiles =
        (long long)((g.M + TC_BM - 1) / TC_BM) * ((g.N + BN - 1) / BN) * (long long)batch;
    if (ntiles <= 0) return cudaSuccess;
    if (ntiles * ((g.K + TC_BK - 1) / TC_BK) > 0x3fffffffLL) return cudaErrorInvalidValue;
    return launch_dep(k_gemm_tc<BN, NTHR, NB, Epi>, dim3((unsigned)std::min<long long>(ntiles, blocks)), dim3(NTHR), smem,
                      st, a, epi);
}
template <int BN, int NTHR, class Epi>
inline cudaError_t launch_gemm_tc(const TcGemmArgs& g, int batch, const Epi& epi, cudaStream_t st) {
    return g.K <= TC_BK ? launch_gemm_nb<BN, NTHR, 1>(g, batch, epi, st) : launch_gemm_nb<BN, NTHR, 2>(g, batch, epi, st);
}

// Tile width by N; 256 threads where the tile is 128 columns wide.
template <class Epi>
inline cudaError_t launch_gemm(const TcGemmArgs& g, int batch, const Epi& epi, cudaStream_t st) {
    if constexpr (Epi::PAIR) return launch_gemm_tc<64, 128>(g, batch, epi, st);  // N == 64
    else if (g.N <= 32) return launch_gemm_tc<32, 128>(g, batch, epi, st);
    else if (g.N <= 64) return launch_gemm_tc<64, 128>(g, batch, epi, st);
    else return launch_gemm_tc<128, 256>(g, batch, epi, st);
}

}  // namespace fi
