// sl_mlp.cu -- the collision-outcome surrogate: an MLP (n_in -> H x L hidden
// layers with GELU -> n_out) with BF16 weights and activations and FP32
// accumulation, trained and evaluated on the GPU by this file's kernels
// (include/spacelab_mlp.h).
//
// Every training product is one kernel, gemm_nt_tc: C[M][N] = A[M][K] .
// B[N][K]^T with A and B bf16 row-major (K contiguous) on the
// fifth-generation tensor cores: TMA copies of 128-byte-swizzled K chunks into
// shared memory, tcgen05.mma (bf16 x bf16 -> f32) into a tensor memory
// accumulator, tcgen05.ld back to registers for the epilogue.
//   forward   Z_l = X_l W_l^T + b_l,  X_{l+1} = bf16(GELU(Z_l)) and X_{l+1}^T
//   backward  dW_l = dZ_l^T X_l, db_l = the column sums of dZ_l, and
//             dX_l = dZ_l W_l, dZ_{l-1} = bf16(dX_l * GELU'(Z_{l-1})) and its
//             transpose: one launch per layer
// The operands with the batch as their K dimension are the transposed copies
// that the epilogues write; W^T is kept beside the bf16 weights by Adam.
// Training runs a step as one CUDA graph over an epoch's rows packed on the
// device.  Prediction takes all layers in one launch (mlp_forward_kernel).
// Widths are padded to multiples of 32 with zero weights that stay zero
// (their gradients are zero).  FP32 master weights are updated with Adam;
// bf16 copies feed the GEMMs.  An mma.sync m16n8k16 kernel (gemm_nt_kernel)
// is kept only as the second opinion of sl_diag_gemm_bf16.
#include "../../include/spacelab_mlp.h"
#include "../../include/spacelab_diag.h"
#include "../../include/spacelab_gpu.h"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include "sl_pdl.cuh"
#include "sl_tma.cuh"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <random>
#include <string>
#include <vector>

int sl_record_error(int code, const char* msg);

namespace {

using bf16 = __nv_bfloat16;

constexpr int kTM = 64, kTN = 64, kTK = 32, kPadK = 8;  // CTA tile; smem row pad (bank spread)

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void ldsm_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(smem_u32(p)));
}

__device__ __forceinline__ void ldsm_x2(uint32_t& r0, uint32_t& r1, const void* p)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(smem_u32(p)));
}

__device__ __forceinline__ void mma_bf16(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }

__device__ __forceinline__ float gelu_grad(float z)
{
    const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
    return cdf + z * pdf;
}

// C = A . B^T for bf16 A[M][K] (lda), B[N][K] (ldb); K % 32 == 0; any M, N.
// act: 0 identity, 1 GELU (applied to the bf16 output only).
__global__ void __launch_bounds__(128) gemm_nt_kernel(const bf16* __restrict__ A, int lda, const bf16* __restrict__ B,
                                                      int ldb, const float* __restrict__ bias, float* Cf, bf16* Cb,
                                                      int ldc, int M, int N, int K, int act)
{
    __shared__ __align__(16) bf16 As[kTM][kTK + kPadK];
    __shared__ __align__(16) bf16 Bs[kTN][kTK + kPadK];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * kTM, n0 = blockIdx.x * kTN;
    const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
    float acc[2][4][4] = {};
    for (int k0 = 0; k0 < K; k0 += kTK) {
        // 64 rows x 32 bf16 = 4 16-byte chunks per row; 128 threads x 2 chunks per matrix
        for (int q = tid; q < kTM * 4; q += 128) {
            const int r = q >> 2, c = (q & 3) * 8;
            uint4 va = make_uint4(0, 0, 0, 0), vb = make_uint4(0, 0, 0, 0);
            if (m0 + r < M) va = *reinterpret_cast<const uint4*>(A + (size_t)(m0 + r) * lda + k0 + c);
            if (n0 + r < N) vb = *reinterpret_cast<const uint4*>(B + (size_t)(n0 + r) * ldb + k0 + c);
            *reinterpret_cast<uint4*>(&As[r][c]) = va;
            *reinterpret_cast<uint4*>(&Bs[r][c]) = vb;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kTK; kk += 16) {
            uint32_t a[2][4], b[4][2];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
                ldsm_x4(a[mt][0], a[mt][1], a[mt][2], a[mt][3], &As[wm + mt * 16 + (lane & 15)][kk + (lane >> 4) * 8]);
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
                ldsm_x2(b[nt][0], b[nt][1], &Bs[wn + nt * 8 + (lane & 7)][kk + ((lane >> 3) & 1) * 8]);
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nt = 0; nt < 4; ++nt)
                    mma_bf16(acc[mt][nt], a[mt][0], a[mt][1], a[mt][2], a[mt][3], b[nt][0], b[nt][1]);
        }
        __syncthreads();
    }
    const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int row = m0 + wm + mt * 16 + g + h * 8;
                const int col = n0 + wn + nt * 8 + t4 * 2;
                if (row >= M) continue;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (col + e >= N) continue;
                    float v = acc[mt][nt][2 * h + e] + (bias ? bias[col + e] : 0.0f);
                    if (Cf) Cf[(size_t)row * ldc + col + e] = v;
                    if (Cb) Cb[(size_t)row * ldc + col + e] = __float2bfloat16(act ? gelu(v) : v);
                }
            }
}

// ------------------------------------------------------------- tcgen05 --
// C[M][N] = A[M][K] . B[N][K]^T on the fifth-generation tensor cores
// (gemm_nt_tc_kernel).  One CTA (8 warps) per 128 x 32 tile of C; its
// accumulator is 32 f32 columns x 128 lanes of tensor memory (TMEM).  K is
// taken in chunks of 64 elements (128 bytes): TMA copies the A and B chunks
// into shared memory with the 128-byte swizzle -- the K-major layout the MMA's
// shared-memory descriptors describe (8-row groups 1024 bytes apart) -- into
// one of four stages, and one thread issues up to four tcgen05.mma (M=128,
// N=32, K=16) per chunk, then tcgen05.commit to the stage's barrier so that
// the next copy into that stage waits for the MMAs reading it.  Boxes past M,
// N or K are zero-filled by the copy engine.  Every wait is bounded
// (sl_tma.cuh); a wait that runs out sets *err, the CTA waits (bounded) for
// its MMAs, frees its TMEM and returns.
//
// The training products are small -- a batch of 256 rows through 256-wide
// layers is 33 MFLOP -- so what counts is how many CTAs share one (16 of 128 x
// 32 for a layer) and that nothing needs a pass of its own: a launch holds up
// to two products and a bias gradient (the backward's dW, db and dX of one
// layer), and the epilogue writes the next product's operands in the layout
// it reads, the transposed copy too (TMEM gives a warp 32 rows of one column:
// its 2-byte stores are contiguous in the transposed copy).  The bias gradient
// adds in row order from the transposed copy, 16 bytes a load.
//
// Measured (GB300, 8-256x4-4): one epoch of 45,000 rows in batches of 256, 87.1
// -> 12.4 ms (497 -> 70 us a step: 40 launches, three copies and a wait a step
// before, 12 launches in a graph now); loss and gradient of 1024 rows, 696 ->
// 224 us.  Same bits.
constexpr int kTcM = 128, kTcN = 32, kTcK = 64, kTcStages = 4;
constexpr int kTcThreads = 256;
constexpr int kTcABytes = kTcM * kTcK * 2, kTcBBytes = kTcN * kTcK * 2;
constexpr int kTcSmem = kTcStages * (kTcABytes + kTcBBytes) + 1024 /* barriers etc. */ + 1024 /* alignment */;

// Shared-memory matrix descriptor of a K-major tile with the 128-byte
// swizzle: start address >> 4 (bits 0-13), leading byte offset (unused for
// this layout; 16 bytes, bits 16-29), stride byte offset 1024 = 8 rows x 128
// bytes (bits 32-45), descriptor version 1 (bits 46-47), base offset 0 (the
// tile is 1024-byte aligned), layout SWIZZLE_128B = 2 (bits 61-63).  The
// K = 16 sub-steps within a 128-byte row advance the start address by 32
// bytes.
__device__ __forceinline__ uint64_t tc_desc_sw128(uint32_t saddr)
{
    return (uint64_t)((saddr >> 4) & 0x3fffu) | ((uint64_t)(16 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// Instruction descriptor of kind::f16: D f32 (bits 4-5 = 1), A and B bf16
// (bits 7-9 and 10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 (bits
// 17-22), M >> 4 (bits 24-28).
__host__ __device__ constexpr uint32_t tc_idesc_bf16(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, int accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrives on `bar` once every tcgen05.mma this thread issued has completed.
__device__ __forceinline__ void tc_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(sl::tma::smem_addr(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive f32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float* v)
{
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// 16 consecutive f32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float* v)
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t bf16x2(float a, float b)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);  // a in the low half
    return *reinterpret_cast<const uint32_t*>(&v);
}

// One product and what becomes of it.  z = C + bias (if any) goes to cf; zin
// given, z = C * GELU'(zin); bf16(act ? GELU(z) : z) goes to cb and, transposed
// (leading dimension ldt), to cbt.  During training the step's rows of the
// epoch's packed inputs start at (*step + step_bias) x a_row_step rows of A and
// x b_col_step columns of B.
struct GemmJob {
    CUtensorMap a, b;
    const float *bias, *zin;
    float* cf;
    bf16 *cb, *cbt;
    int ldc, ldt, M, N, K, act;
    int a_row_step, b_col_step;
};

struct GemmLaunch {
    GemmJob job[2];
    int njobs;
    // bias gradient: db_out[c] = sum over r < db_rows of db_src[c][r], r ascending
    const bf16* db_src;
    float* db_out;
    int db_n, db_rows;
    const int* step;  // NULL: step 0
    int step_bias;
    int* bump;        // incremented once (by a launch that does not read it)
    int* err;
};

__host__ __device__ inline int gemm_tiles(const GemmJob& j) { return ((j.M + kTcM - 1) / kTcM) * ((j.N + kTcN - 1) / kTcN); }

// Bias gradients: the sums over the batch of kBiasOut outputs' gradients from
// c0 on, by one CTA.  All threads copy rows of dZ^T (16 bytes each, all in
// flight) to shared memory, and lane c of warp 0 adds row c0 + c's values there,
// in row order: a chain of FP32 adds, 4 cycles each, that from global memory
// was a chain of loads (the backward launch of 1024 rows: 20.5 us, 11.4 here).
constexpr int kBiasOut = 32, kBiasRows = 1024;
constexpr int kBiasStride = kBiasRows * 2 + 16;  // bytes; 16-byte loads of 8 lanes fall in distinct banks
static_assert(kBiasOut * kBiasStride + 1024 <= kTcSmem, "the rows fit in the GEMM's shared memory");

__device__ void bias_grad(const GemmLaunch& L, unsigned char* smem, int c0)
{
    const int tid = threadIdx.x;
    float s = 0.0f;
    for (int r0 = 0; r0 < L.db_rows; r0 += kBiasRows) {
        const int vecs = min(kBiasRows, L.db_rows - r0) / 8;  // rows a multiple of 32
        const int outs = min(kBiasOut, L.db_n - c0);
        if (r0) __syncthreads();
#pragma unroll 8
        for (int k = tid; k < outs * vecs; k += kTcThreads) {
            const int c = k / vecs, v = k - c * vecs;
            *reinterpret_cast<uint4*>(smem + c * kBiasStride + v * 16) =
                reinterpret_cast<const uint4*>(L.db_src + (size_t)(c0 + c) * L.db_rows + r0)[v];
        }
        __syncthreads();
        if (tid < outs) {
            const uint4* row = reinterpret_cast<const uint4*>(smem + tid * kBiasStride);
#pragma unroll 4
            for (int v = 0; v < vecs; ++v) {
                const uint4 q = row[v];
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    s += __uint_as_float(w[k] << 16);
                    s += __uint_as_float(w[k] & 0xffff0000u);
                }
            }
        }
    }
    if (tid < kBiasOut && c0 + tid < L.db_n) L.db_out[c0 + tid] = s;
}

__global__ void __launch_bounds__(kTcThreads) gemm_nt_tc_kernel(const __grid_constant__ GemmLaunch L)
{
    extern __shared__ unsigned char tc_raw[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_raw) + 1023) &
                                                           ~static_cast<uintptr_t>(1023));
    int tile = blockIdx.x;
    sl::pdl_next();
    const int tiles0 = gemm_tiles(L.job[0]);
    const bool second = tile >= tiles0;
    if (second) tile -= tiles0;
    if (second && (L.njobs < 2 || tile >= gemm_tiles(L.job[1]))) {
        sl::pdl_wait();
        bias_grad(L, base, (tile - (L.njobs < 2 ? 0 : gemm_tiles(L.job[1]))) * kBiasOut);
        return;
    }
    const GemmJob& J = L.job[second];

    unsigned char* sa = base;                            // [stage][128 rows][128 B]
    unsigned char* sb = base + kTcStages * kTcABytes;    // [stage][32 rows][128 B]
    uint64_t* full = reinterpret_cast<uint64_t*>(sb + kTcStages * kTcBBytes);
    uint64_t* empty = full + kTcStages;
    uint64_t* done = empty + kTcStages;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    int* failed = reinterpret_cast<int*>(tmem_slot + 1);
    const int tiles_n = (J.N + kTcN - 1) / kTcN;
    const int m0 = tile / tiles_n * kTcM, n0 = tile % tiles_n * kTcN;
    const int nk = (J.K + kTcK - 1) / kTcK;

    if (tid == 0) {
        for (int st = 0; st < kTcStages; ++st) {
            sl::tma::mbar_init(&full[st], 1);
            sl::tma::mbar_init(&empty[st], 1);
        }
        sl::tma::mbar_init(done, 1);
        *failed = 0;
        sl::tma::fence_barrier_init();
    }
    if (warp == 0) {  // 32 f32 columns of TMEM
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(sl::tma::smem_addr(tmem_slot)), "r"(kTcN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    sl::pdl_wait();
    if (blockIdx.x == 0 && tid == 0 && L.bump) *L.bump += 1;

    if (tid == 0) {
        constexpr uint32_t idesc = tc_idesc_bf16(kTcM, kTcN);
        const int step = L.step ? *L.step + L.step_bias : 0;
        const int ya = m0 + step * J.a_row_step, xb = step * J.b_col_step;
        auto issue = [&](int kc) {
            const int st = kc % kTcStages;
            sl::tma::mbar_arrive_expect_tx(&full[st], kTcABytes + kTcBBytes);
            sl::tma::load_2d(sa + st * kTcABytes, &J.a, kc * kTcK, ya, &full[st]);
            sl::tma::load_2d(sb + st * kTcBBytes, &J.b, xb + kc * kTcK, n0, &full[st]);
        };
        int issued = 0;
        for (; issued < nk && issued < kTcStages; ++issued) issue(issued);
        bool ok = true;
        int kc = 0;
        for (; kc < nk && ok; ++kc) {
            const int st = kc % kTcStages;
            const uint32_t par = (uint32_t)(kc / kTcStages) & 1u;
            if (!sl::tma::mbar_wait(&full[st], par)) { ok = false; break; }
            tc_fence_after();
            const uint32_t a0 = sl::tma::smem_addr(sa + st * kTcABytes);
            const uint32_t b0 = sl::tma::smem_addr(sb + st * kTcBBytes);
            // past K the boxes hold zeros, or another step's columns
            const int steps = min(kTcK, J.K - kc * kTcK + 15) / 16;
            for (int k = 0; k < steps; ++k)
                tc_mma(tmem, tc_desc_sw128(a0 + 32 * k), tc_desc_sw128(b0 + 32 * k), idesc, (kc | k) != 0);
            tc_commit(&empty[st]);
            // the stage before this one's gets its next copy when the MMAs that
            // read it have completed, with this one's MMAs under way
            if (kc > 0 && kc - 1 + kTcStages < nk) {
                const int q = kc - 1;
                if (!sl::tma::mbar_wait(&empty[q % kTcStages], (uint32_t)(q / kTcStages) & 1u)) { ok = false; ++kc; break; }
                issue(q + kTcStages);
                ++issued;
            }
        }
        tc_commit(done);  // arrives when every MMA issued above has completed
        if (!ok) {
            *failed = 1;
            // let the copies in flight land before the CTA's memory is reused
            for (int q = kc; q < issued; ++q)
                sl::tma::mbar_wait(&full[q % kTcStages], (uint32_t)(q / kTcStages) & 1u);
        }
    }
    __syncwarp();
    if (!sl::tma::mbar_wait(done, 0)) *failed = 1;
    tc_fence_after();
    __syncthreads();
    // the same decision in every thread (tcgen05.ld is warp-collective)
    if (*failed) {
        if (tid == 0) *L.err = 1;
    } else {
        // warp w: TMEM lanes 32 (w mod 4) .., columns 16 (w / 4) ..
        const int row = m0 + (warp & 3) * 32 + lane, c0 = (warp >> 2) * 16;
        float v[16];
        tc_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, v);
        const int col = n0 + c0;
        if (row < J.M) {
            const size_t at = (size_t)row * J.ldc + col;
            if (J.ldc % 8 == 0 && col + 16 <= J.N) {  // whole 16-byte groups
                if (J.bias)
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] += J.bias[col + i];
                if (J.zin) {
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const float4 z = *reinterpret_cast<const float4*>(J.zin + at + i);
                        v[i] *= gelu_grad(z.x);
                        v[i + 1] *= gelu_grad(z.y);
                        v[i + 2] *= gelu_grad(z.z);
                        v[i + 3] *= gelu_grad(z.w);
                    }
                }
                if (J.cf)
#pragma unroll
                    for (int i = 0; i < 16; i += 4)
                        *reinterpret_cast<float4*>(J.cf + at + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                if (J.cb) {
                    uint32_t h[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        h[i] = J.act ? bf16x2(gelu(v[2 * i]), gelu(v[2 * i + 1])) : bf16x2(v[2 * i], v[2 * i + 1]);
                    uint4* dst = reinterpret_cast<uint4*>(J.cb + at);
                    dst[0] = make_uint4(h[0], h[1], h[2], h[3]);
                    dst[1] = make_uint4(h[4], h[5], h[6], h[7]);
                    if (J.cbt) {
                        uint16_t* t = reinterpret_cast<uint16_t*>(J.cbt) + (size_t)col * J.ldt + row;
#pragma unroll
                        for (int i = 0; i < 16; ++i) t[(size_t)i * J.ldt] = (uint16_t)(h[i >> 1] >> (16 * (i & 1)));
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    if (col + i >= J.N) break;
                    const float z = v[i] + (J.bias ? J.bias[col + i] : 0.0f);
                    if (J.cf) J.cf[at + i] = z;
                    if (J.cb) J.cb[at + i] = __float2bfloat16(J.act ? gelu(z) : z);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcN) : "memory");
}

// ----------------------------------------------- the whole forward pass --
// The network's outputs for n rows in one launch.  A CTA takes 128 rows at a
// time through every layer: the bf16 activations stay in shared memory (64
// KB: up to 256 columns in 64-column chunks, the 128-byte-swizzled K-major
// layout the MMA reads), the accumulator in 256 columns of tensor memory, and
// the weights stream from L2 in 128 x 64 tiles (16 KB) through a ring of
// three.  Six warps: four for the epilogues (a thread is a row: TMEM lane ->
// bias, GELU, bf16 -> the next layer's operand), one issues the MMAs, one the
// copies.  114,944 bytes of shared memory and 256 of the 512 TMEM columns let
// two CTAs share an SM, so that one's MMAs and copies run under the other's
// epilogue, which is what bounds the pass: 1024 erff per row, ~40
// instructions each.  Rows are read and results written where the caller has
// them.  The products are accumulated K chunk by K chunk as the
// layer-by-layer kernel does, so the outputs are the same bits.
//
// Measured (GB300, 8-256x4-4, host arrays in and out): 1,000,000 rows 272 ->
// 1.72 ms, 1000 rows 289 -> 67 us, 1 row 132 -> 68 us, against a batch of
// 1024 rows at a time through six launches and three blocking copies, with
// the epilogue's stores one row per lane (55 of a layer's 58 us).
constexpr int kFwRows = 128, kFwMaxWidth = 256, kFwMaxLayers = 8, kFwStages = 3, kFwTileN = 128;
constexpr int kFwXBytes = kFwRows * kFwMaxWidth * 2, kFwWBytes = kFwTileN * kTcK * 2;
constexpr int kFwThreads = 192, kFwEpilogue = 128;
constexpr int kFwSmem = kFwXBytes + kFwStages * kFwWBytes + 256;  // + barriers, TMEM address, failure flag

// Row tiles of n rows, for any n; a tile's last row fits an int too
__host__ __device__ constexpr int fw_tiles(int n) { return n / kFwRows + (n % kFwRows != 0); }
static_assert(fw_tiles(1) == 1 && fw_tiles(kFwRows) == 1 && fw_tiles(kFwRows + 1) == 2, "row tiles");
static_assert(fw_tiles(INT_MAX) == 1 << 24, "row tiles of the largest prediction");

struct FwNet {
    CUtensorMap w[kFwMaxLayers];            // weights [dout][din], boxes of 64 x 128
    const float* bias[kFwMaxLayers];
    int din[kFwMaxLayers], dout[kFwMaxLayers];
    int layers, n_in, n_out;
};

// Waits like mbar_wait, and gives up at once when another thread of the CTA has.
__device__ __forceinline__ bool fw_wait(uint64_t* bar, uint32_t parity, volatile int* failed)
{
    if (sl::tma::mbar_test(bar, parity)) return true;
    const long long t0 = clock64();
    while (!sl::tma::mbar_test(bar, parity))
        if (*failed || clock64() - t0 > sl::tma::kWaitCycles) {
            *failed = 1;
            return false;
        }
    return true;
}

// byte of row r's 16-byte group g (8 columns) of the activations
__device__ __forceinline__ int fw_x_offset(int r, int g) { return (g >> 3) * (kFwRows * 128) + r * 128 + (((g & 7) ^ (r & 7)) << 4); }

__global__ void __launch_bounds__(kFwThreads, 2) mlp_forward_kernel(const __grid_constant__ FwNet net,
                                                                    const float* __restrict__ x, float* y, int n,
                                                                    int* err)
{
    extern __shared__ __align__(1024) unsigned char fw_raw[];
    unsigned char* sx = fw_raw;
    unsigned char* sw = fw_raw + kFwXBytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(sw + kFwStages * kFwWBytes);
    uint64_t* empty = full + kFwStages;
    uint64_t* acc_done = empty + kFwStages;   // a layer's MMAs have completed
    uint64_t* x_ready = acc_done + 1;         // a layer's operand is in shared memory
    uint64_t* drain = x_ready + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
    volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntiles = fw_tiles(n);
    // whole 16-byte groups of the caller's rows
    const bool vec_in = net.n_in % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    const bool vec_out = net.n_out % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 15u) == 0;

    if (tid == 0) {
        for (int k = 0; k < kFwStages; ++k) {
            sl::tma::mbar_init(&full[k], 1);
            sl::tma::mbar_init(&empty[k], 1);
        }
        sl::tma::mbar_init(acc_done, 1);
        sl::tma::mbar_init(x_ready, kFwEpilogue);
        sl::tma::mbar_init(drain, 1);
        *failed = 0;
        sl::tma::fence_barrier_init();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(sl::tma::smem_addr(tmem_slot)), "r"(kFwMaxWidth)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp < 4) {  // ------------------------------------------- epilogues
        const int r = warp * 32 + lane;
        uint32_t phase = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
            const int row = t * kFwRows + r;
            {  // the row's features, zero up to whole K chunks
                const float* xr = x + (size_t)row * net.n_in;
                const int groups = (net.din[0] + kTcK - 1) / kTcK * 8;
                for (int g = 0; g < groups; ++g) {
                    float f[8];
                    if (vec_in && row < n && g * 8 + 8 <= net.n_in) {
                        const float4 lo = *reinterpret_cast<const float4*>(xr + g * 8);
                        const float4 hi = *reinterpret_cast<const float4*>(xr + g * 8 + 4);
                        f[0] = lo.x; f[1] = lo.y; f[2] = lo.z; f[3] = lo.w;
                        f[4] = hi.x; f[5] = hi.y; f[6] = hi.z; f[7] = hi.w;
                    } else {
#pragma unroll
                        for (int k = 0; k < 8; ++k) f[k] = row < n && g * 8 + k < net.n_in ? xr[g * 8 + k] : 0.0f;
                    }
                    *reinterpret_cast<uint4*>(sx + fw_x_offset(r, g)) =
                        make_uint4(bf16x2(f[0], f[1]), bf16x2(f[2], f[3]), bf16x2(f[4], f[5]), bf16x2(f[6], f[7]));
                }
            }
            sl::tma::fence_proxy_async();
            sl::tma::mbar_arrive(x_ready);
            for (int l = 0; l < net.layers; ++l) {
                ok = fw_wait(acc_done, phase, failed);
                phase ^= 1u;
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                tc_fence_after();
                const float* bias = net.bias[l];
                const int N = net.dout[l];
                const bool last = l == net.layers - 1;
#pragma unroll 1
                for (int cg = 0; cg < N / 32; ++cg) {
                    float v[32];
                    tc_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(cg * 32), v);
                    if (last) {
                        float* yr = y + (size_t)row * net.n_out + cg * 32;
                        const int cols = row < n ? net.n_out - cg * 32 : 0;
#pragma unroll
                        for (int i = 0; i < 32; i += 4) {
                            const float4 b = __ldg(reinterpret_cast<const float4*>(bias + cg * 32 + i));
                            const float4 o = make_float4(v[i] + b.x, v[i + 1] + b.y, v[i + 2] + b.z, v[i + 3] + b.w);
                            if (vec_out && i < cols) {
                                *reinterpret_cast<float4*>(yr + i) = o;
                            } else {
                                if (i < cols) yr[i] = o.x;
                                if (i + 1 < cols) yr[i + 1] = o.y;
                                if (i + 2 < cols) yr[i + 2] = o.z;
                                if (i + 3 < cols) yr[i + 3] = o.w;
                            }
                        }
                        continue;
                    }
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const float4 b0 = __ldg(reinterpret_cast<const float4*>(bias + cg * 32 + g * 8));
                        const float4 b1 = __ldg(reinterpret_cast<const float4*>(bias + cg * 32 + g * 8 + 4));
                        const float* z = v + g * 8;
                        *reinterpret_cast<uint4*>(sx + fw_x_offset(r, cg * 4 + g)) =
                            make_uint4(bf16x2(gelu(z[0] + b0.x), gelu(z[1] + b0.y)),
                                       bf16x2(gelu(z[2] + b0.z), gelu(z[3] + b0.w)),
                                       bf16x2(gelu(z[4] + b1.x), gelu(z[5] + b1.y)),
                                       bf16x2(gelu(z[6] + b1.z), gelu(z[7] + b1.w)));
                    }
                }
                if (!last) {
                    for (int g = N / 8; g < (N + kTcK - 1) / kTcK * 8; ++g)
                        *reinterpret_cast<uint4*>(sx + fw_x_offset(r, g)) = make_uint4(0, 0, 0, 0);
                    tc_fence_before();
                    sl::tma::fence_proxy_async();
                    sl::tma::mbar_arrive(x_ready);
                } else {
                    tc_fence_before();  // the next tile's x_ready arrival follows these loads
                }
            }
        }
    } else if (warp == 4 && lane == 0) {  // ----------------------------- MMAs
        int q = 0;
        uint32_t xphase = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
            for (int l = 0; l < net.layers && ok; ++l) {
                ok = fw_wait(x_ready, xphase, failed);
                xphase ^= 1u;
                if (!ok) break;
                tc_fence_after();
                const int K = net.din[l], N = net.dout[l];
                for (int kc = 0; kc * kTcK < K && ok; ++kc) {
                    const uint32_t a0 = sl::tma::smem_addr(sx + kc * (kFwRows * 128));
                    const int steps = min(kTcK, K - kc * kTcK) / 16;
                    for (int n0 = 0; n0 < N; n0 += kFwTileN, ++q) {
                        const int st = q % kFwStages;
                        ok = fw_wait(&full[st], (uint32_t)(q / kFwStages) & 1u, failed);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t b0 = sl::tma::smem_addr(sw + st * kFwWBytes);
                        const uint32_t idesc = tc_idesc_bf16(kFwRows, min(kFwTileN, N - n0));
                        for (int k = 0; k < steps; ++k)
                            tc_mma(tmem + (uint32_t)n0, tc_desc_sw128(a0 + 32 * k), tc_desc_sw128(b0 + 32 * k), idesc,
                                   (kc | k) != 0);
                        tc_commit(&empty[st]);
                    }
                }
                if (ok) tc_commit(acc_done);
            }
        // every MMA issued has completed before the tensor memory is freed
        tc_commit(drain);
        if (!sl::tma::mbar_wait(drain, 0)) *failed = 1;
    } else if (warp == 5 && lane == 0) {  // ---------------------------- copies
        int q = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
            for (int l = 0; l < net.layers && ok; ++l)
                for (int k0 = 0; k0 < net.din[l] && ok; k0 += kTcK)
                    for (int n0 = 0; n0 < net.dout[l]; n0 += kFwTileN, ++q) {
                        const int st = q % kFwStages;
                        if (q >= kFwStages) ok = fw_wait(&empty[st], (uint32_t)(q / kFwStages - 1) & 1u, failed);
                        if (!ok) break;
                        sl::tma::mbar_arrive_expect_tx(&full[st], kFwWBytes);
                        sl::tma::load_2d(sw + st * kFwWBytes, &net.w[l], k0, n0, &full[st]);
                    }
        // and every copy has landed before the shared memory is given back
        for (int p = max(0, q - kFwStages); p < q; ++p)
            if (!sl::tma::mbar_wait(&full[p % kFwStages], (uint32_t)(p / kFwStages) & 1u)) *failed = 1;
    }
    __syncwarp();
    __syncthreads();
    if (tid == 0 && *failed) *err = 1;
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kFwMaxWidth)
                     : "memory");
}

// The inputs of rows idx[0 .. rows) (NULL: rows 0 ..) as bf16 rows of ld
// columns, zero past n_in and past row n, and transposed (leading dimension
// rows); targets gathered alongside.  Thread = row.
__global__ void pack_kernel(const float* __restrict__ x, const float* __restrict__ y, const int* __restrict__ idx,
                            int rows, int n, int n_in, int n_out, int ld, bf16* xb, bf16* xt, float* yb)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    const int src = idx ? idx[r] : r;
    for (int c = 0; c < ld; ++c) {
        const bf16 v = __float2bfloat16(c < n_in && src < n ? x[(size_t)src * n_in + c] : 0.0f);
        xb[(size_t)r * ld + c] = v;
        if (xt) xt[(size_t)c * rows + r] = v;
    }
    if (yb)
        for (int c = 0; c < n_out; ++c) yb[(size_t)r * n_out + c] = y[(size_t)src * n_out + c];
}

// MSE over the first n_out columns: dZ = 2 (z - y) / (M n_out), row-major and
// transposed, and the loss in one partial sum per 256 entries of dZ
__global__ void mse_grad_kernel(const float* z, int ldz, const float* y, int M, int n_out, bf16* dz, bf16* dzt, int ld,
                                float* loss_partial, const int* step, int step_bias)
{
    __shared__ float red[256];
    sl::pdl_next();
    sl::pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int st = step ? *step + step_bias : 0;
    y += (size_t)st * M * n_out;
    loss_partial += (size_t)st * gridDim.x;
    float l = 0.0f;
    if (i < M * ld) {
        const int r = i / ld, c = i - r * ld;
        float g = 0.0f;
        if (c < n_out) {
            const float e = z[(size_t)r * ldz + c] - y[(size_t)r * n_out + c];
            l = e * e;
            g = 2.0f * e / (float)(M * n_out);
        }
        dz[i] = __float2bfloat16(g);
        dzt[(size_t)c * M + r] = __float2bfloat16(g);
    }
    red[threadIdx.x] = l;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) loss_partial[blockIdx.x] = red[0];
}

// A layer's place in the parameter vector: W [dout][din] at w, then b
struct LayerAt {
    long long w;
    int din, dout;
};

// bf16 copy of parameter i, and for a weight the copy's transposed place
__device__ __forceinline__ void put_bf16(bf16* pb, bf16* wt, const LayerAt* at, int layers, int i, float v)
{
    pb[i] = __float2bfloat16(v);
    int l = 0;
    while (l + 1 < layers && i >= at[l + 1].w) ++l;
    const long long k = i - at[l].w;
    if (k < (long long)at[l].din * at[l].dout) {
        const int r = (int)(k / at[l].din), c = (int)(k - (long long)r * at[l].din);
        wt[at[l].w + (long long)c * at[l].dout + r] = __float2bfloat16(v);
    }
}

// Adam on fp32 master parameters; refreshes the bf16 copies.  mask: the
// parameter is live (padding stays 0).  coef: the step's bias corrections
// 1 - b1^t, 1 - b2^t.
__global__ void adam_kernel(float* p, const float* g, float* m, float* v, bf16* pb, bf16* wt, const LayerAt* at,
                            int layers, const uint8_t* mask, int n, float lr, float b1, float b2, float eps,
                            const float2* coef, const int* step, int step_bias)
{
    sl::pdl_next();
    sl::pdl_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (!mask[i]) return;
    const float2 c = coef[*step + step_bias];
    const float c1 = c.x, c2 = c.y;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    put_bf16(pb, wt, at, layers, i, pi);
}

__global__ void to_bf16_kernel(const float* __restrict__ in, bf16* pb, bf16* wt, const LayerAt* at, int layers, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) put_bf16(pb, wt, at, layers, i, in[i]);
}

int pad32(int x) { return (x + 31) / 32 * 32; }

// Device memory that training keeps for a data set and its packed epoch (45,000
// rows of 8 features take 9 MB).
constexpr size_t kEpochBytes = size_t(256) << 20;

}  // namespace

struct sl_mlp {
    int n_in = 0, hidden = 0, layers = 0, n_out = 0, max_batch = 0;
    int nl = 0;                          // linear layers = hidden layers + 1
    std::vector<int> din, dout;          // padded widths of each linear layer
    std::vector<size_t> w_off, b_off;    // offsets into the parameter vector
    size_t nparam = 0;
    float *P = nullptr, *G = nullptr, *Mom = nullptr, *Var = nullptr;  // fp32 params, grads, Adam moments
    bf16* Pb = nullptr;                  // bf16 copy of params (weights used by the GEMMs)
    uint8_t* mask = nullptr;             // live parameters
    bf16* Wt = nullptr;                  // its weights transposed, [din][dout] at the same offsets
    LayerAt* at = nullptr;               // the layers' places, for the kernels
    std::vector<bf16*> X, Xt;            // bf16 activations per layer input, [M][din] and [din][M]
    std::vector<float*> Z;               // fp32 pre-activations per layer [M][dout]
    bf16 *dZ[2] = {}, *dZt[2] = {};      // gradients of Z, [M][dout] and [dout][M]; a layer reads one and writes the other
    float *xin = nullptr, *yin = nullptr;
    cudaStream_t stream = nullptr;       // training's launches
    void* epoch = nullptr;               // training's copies of the data set (grown when a larger one comes, to kEpochBytes)
    size_t epoch_bytes = 0;
    int step = 0;
    int* err = nullptr;           // set by a tcgen05 GEMM whose bounded wait ran out; pinned host memory, with
    float* loss_part = nullptr;   // a batch's loss in partial sums behind it: read after a wait, without a copy
    bool tc_setup_failed = false; // a GEMM's tensor maps or launch attributes could not be set up
    bool fused = false;           // `net` is set up: the whole forward pass in one launch
    FwNet net{};
    int num_sms = 0;
    bool host_direct = false;     // the GPU reads and writes pageable host memory (cudaDevAttrPageableMemoryAccess)
    int fail_next = 0;            // diagnostics: what sl_diag_mlp_fail asked for
    void* arena = nullptr;
};

namespace {

void gemm_mma_sync(cudaStream_t st, const bf16* A, int lda, const bf16* B, int ldb, const float* bias, float* Cf,
                   bf16* Cb, int ldc, int M, int N, int K, int act)
{
    dim3 grid((N + kTN - 1) / kTN, (M + kTM - 1) / kTM);
    gemm_nt_kernel<<<grid, 128, 0, st>>>(A, lda, B, ldb, bias, Cf, Cb, ldc, M, N, K, act);
}

PFN_cuTensorMapEncodeTiled_v12000 mlp_map_encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    });
    return encode;
}

// A row-major bf16 matrix [rows][k] with leading dimension ld (elements) as a
// 2D tensor map: boxes of 64 elements (128 bytes) of k x box_rows rows, the
// 128-byte swizzle, zero fill outside the matrix.
bool make_tc_map(CUtensorMap* map, const bf16* base, int rows, int k, int ld, int box_rows)
{
    PFN_cuTensorMapEncodeTiled_v12000 encode = mlp_map_encoder();
    if (!encode || !base || (reinterpret_cast<uintptr_t>(base) & 15u) || (ld * 2) % 16) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kTcK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A job without its epilogue; false if a tensor map cannot be made.
bool make_job(GemmJob* j, const bf16* A, int rows_a, int lda, const bf16* B, int ldb, int kb, int M, int N, int K)
{
    *j = GemmJob{};
    j->M = M; j->N = N; j->K = K;
    return make_tc_map(&j->a, A, rows_a, K, lda, kTcM) && make_tc_map(&j->b, B, N, kb, ldb, kTcN);
}

bool launch_gemm(const GemmLaunch& L, cudaStream_t st)
{
    // set on every call: the attribute belongs to the current device's
    // context, and the call is a host-side table update
    if (cudaFuncSetAttribute(gemm_nt_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem) != cudaSuccess)
        return false;
    int grid = gemm_tiles(L.job[0]) + (L.njobs > 1 ? gemm_tiles(L.job[1]) : 0);
    if (L.db_out) grid += (L.db_n + kBiasOut - 1) / kBiasOut;
    return sl::launch_pdl(true, gemm_nt_tc_kernel, grid, kTcThreads, kTcSmem, st, L) == cudaSuccess;
}

// After a synchronisation: the GEMMs' setup and bounded waits.
int mlp_status(sl_mlp* h, const char* what)
{
    if (h->tc_setup_failed)
        return sl_record_error(SL_ERR_CUDA, (std::string(what) + ": tcgen05 GEMM setup (tensor maps) failed").c_str());
    if (*static_cast<volatile int*>(h->err))
        return sl_record_error(SL_ERR_TIMEOUT,
                               (std::string(what) + ": a bounded wait in the tcgen05 GEMM ran out").c_str());
    return SL_OK;
}

// At the start of a call, which finds the handle idle: what an earlier call left
// is not this one's.
void clear_status(sl_mlp* h)
{
    *h->err = 0;
    h->tc_setup_failed = false;
}

// Where a batch's inputs are: its own buffers, or the rows of a training
// epoch's (rows epoch_rows, the step's read from *step).
struct BatchInput {
    const bf16 *X0, *X0t;
    const float* y;
    int rows;           // of X0 and columns of X0t
    int* step;          // NULL: the batch starts at row 0
    float* loss_part;
};

// forward over M rows: the output pre-activation of the last layer is
// Z[nl-1] ([M][dout_last], fp32).  train: the transposed activations too.
void forward(sl_mlp* h, const BatchInput& in, int M, bool train, cudaStream_t st)
{
    for (int l = 0; l < h->nl && !h->tc_setup_failed; ++l) {
        const bool last = l == h->nl - 1;
        const int K = h->din[l], N = h->dout[l];
        GemmLaunch L{};
        GemmJob& j = L.job[0];
        L.njobs = 1;
        L.err = h->err;
        bool ok = make_job(&j, l ? h->X[l] : in.X0, l ? M : in.rows, K, h->Pb + h->w_off[l], K, K, M, N, K);
        j.bias = h->P + h->b_off[l];
        j.cf = h->Z[l];
        j.cb = last ? nullptr : h->X[l + 1];
        j.cbt = last || !train ? nullptr : h->Xt[l + 1];
        j.ldc = N;
        j.ldt = M;
        j.act = 1;
        if (l == 0) {
            L.step = in.step;
            j.a_row_step = M;
        } else if (l == 1) {
            L.bump = in.step;  // from here on *step is the step after this one
        }
        ok = ok && h->fail_next != SL_DIAG_MLP_SETUP && launch_gemm(L, st);
        if (!ok) {
            h->tc_setup_failed = true;
            h->fail_next = 0;
        }
    }
}

// backward for the M rows of the last forward; fills G
void backward(sl_mlp* h, const BatchInput& in, int M, cudaStream_t st)
{
    const int nl = h->nl, ldo = h->dout[nl - 1];
    const int nb = (M * ldo + 255) / 256;
    int cur = 0;
    sl::launch_pdl(true, mse_grad_kernel, nb, 256, 0, st, h->Z[nl - 1], ldo, in.y, M, h->n_out, h->dZ[cur], h->dZt[cur],
                   ldo, in.loss_part, in.step, -1);
    for (int l = nl - 1; l >= 0 && !h->tc_setup_failed; --l, cur ^= 1) {
        const int K = h->din[l], N = h->dout[l];
        GemmLaunch L{};
        L.njobs = 1;
        L.err = h->err;
        // dW = dZ^T X: the products run over the batch
        bool ok = make_job(&L.job[0], h->dZt[cur], N, M, l ? h->Xt[l] : in.X0t, l ? M : in.rows, l ? M : in.rows, N, K,
                           M);
        L.job[0].cf = h->G + h->w_off[l];
        L.job[0].ldc = K;
        if (l == 0) {
            L.step = in.step;
            L.step_bias = -1;
            L.job[0].b_col_step = M;
        }
        L.db_src = h->dZt[cur];
        L.db_out = h->G + h->b_off[l];
        L.db_n = N;
        L.db_rows = M;
        if (l > 0) {  // dZ of the layer below = dZ W * GELU'(Z)
            L.njobs = 2;
            GemmJob& j = L.job[1];
            ok = ok && make_job(&j, h->dZ[cur], M, N, h->Wt + h->w_off[l], N, N, M, K, N);
            j.zin = h->Z[l - 1];
            j.cb = h->dZ[cur ^ 1];
            j.cbt = h->dZt[cur ^ 1];
            j.ldc = K;
            j.ldt = M;
        }
        ok = ok && launch_gemm(L, st);
        if (!ok) h->tc_setup_failed = true;
    }
}

// The batch's own input buffers, packed from M rows of n features at x (and
// their targets at y), device-reachable; rows n .. M - 1 are zero.
BatchInput pack_batch(sl_mlp* h, const float* x, const float* y, int n, int M, cudaStream_t st)
{
    pack_kernel<<<(M + 127) / 128, 128, 0, st>>>(x, nullptr, nullptr, M, n, h->n_in, h->n_out, h->din[0], h->X[0],
                                                 h->Xt[0], nullptr);
    return BatchInput{h->X[0], h->Xt[0], y, M, nullptr, h->loss_part};
}

// The one-launch forward pass: networks of up to kFwMaxLayers linear layers of
// up to kFwMaxWidth padded columns (what fits in shared memory and TMEM).
bool setup_forward(sl_mlp* h)
{
    if (h->nl > kFwMaxLayers) return false;
    FwNet& f = h->net;
    f.layers = h->nl; f.n_in = h->n_in; f.n_out = h->n_out;
    for (int l = 0; l < h->nl; ++l) {
        if (h->din[l] > kFwMaxWidth || h->dout[l] > kFwMaxWidth) return false;
        f.din[l] = h->din[l];
        f.dout[l] = h->dout[l];
        f.bias[l] = h->P + h->b_off[l];
        if (!make_tc_map(&f.w[l], h->Pb + h->w_off[l], h->dout[l], h->din[l], h->din[l], kFwTileN)) return false;
    }
    return true;
}

// y = network(x) for n rows; x and y where the GPU can reach them
cudaError_t forward_fused(sl_mlp* h, const float* x, float* y, int n, cudaStream_t st)
{
    // set on every call: the attribute belongs to the current device's context
    cudaError_t e = cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwSmem);
    if (e != cudaSuccess) return e;
    size_t smem = kFwSmem;
    if (h->fail_next == SL_DIAG_MLP_LAUNCH) {  // more than an SM has
        smem = size_t(1) << 20;
        h->fail_next = 0;
    }
    const int tiles = fw_tiles(n);
    e = sl::launch_pdl(false, mlp_forward_kernel, (unsigned)std::min(tiles, 2 * h->num_sms), kFwThreads, smem, st, h->net,
                       x, y, n, h->err);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

// All rows in one launch, read and written where the caller has them.  *slow: a
// wait ran out.  The epilogues' reads and writes of host memory are inside the
// waits' bound, and a page may take longer (a cold mapped file).
cudaError_t predict_in_place(sl_mlp* h, const float* x, float* y, int n, bool* slow)
{
    cudaError_t e = forward_fused(h, x, y, n, nullptr);
    const cudaError_t done = cudaStreamSynchronize(nullptr);
    if (e == cudaSuccess) e = done;
    if (h->fail_next == SL_DIAG_MLP_SLOW_PAGE) {
        *h->err = 1;
        h->fail_next = 0;
    }
    *slow = *static_cast<volatile int*>(h->err) != 0;
    return e;
}

// A batch at a time through device staging.
cudaError_t predict_staged(sl_mlp* h, const float* x, float* y, int n)
{
    cudaError_t e = cudaSuccess;
    for (int s0 = 0; s0 < n && e == cudaSuccess; s0 += std::min(h->max_batch, n - s0)) {
        const int M = std::min(h->max_batch, n - s0);
        e = cudaMemcpyAsync(h->xin, x + (size_t)s0 * h->n_in, (size_t)M * h->n_in * 4, cudaMemcpyHostToDevice, nullptr);
        if (e == cudaSuccess) e = forward_fused(h, h->xin, h->yin, M, nullptr);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(y + (size_t)s0 * h->n_out, h->yin, (size_t)M * h->n_out * 4, cudaMemcpyDeviceToHost,
                                nullptr);
    }
    const cudaError_t done = cudaStreamSynchronize(nullptr);
    return e != cudaSuccess ? e : done;
}

// A caller's host array as the GPU can use it in place, or NULL
void* device_view(const sl_mlp* h, const void* p)
{
    if (h->host_direct) return const_cast<void*>(p);
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeManaged ? a.devicePointer : nullptr;
}

}  // namespace

extern "C" {

int sl_mlp_create(int n_in, int hidden, int hidden_layers, int n_out, int max_batch, uint64_t seed, sl_mlp** out)
{
    if (!out) return sl_record_error(SL_ERR_ARG, "out is NULL");
    *out = nullptr;
    if (n_in < 1 || hidden < 1 || hidden_layers < 1 || n_out < 1 || max_batch < 32 || max_batch % 32)
        return sl_record_error(SL_ERR_ARG, "need n_in, hidden, layers, n_out >= 1 and max_batch a multiple of 32");
    sl_mlp* h = new (std::nothrow) sl_mlp();
    if (!h) return sl_record_error(SL_ERR_ALLOC, "host allocation failed");
    h->n_in = n_in; h->hidden = hidden; h->layers = hidden_layers; h->n_out = n_out; h->max_batch = max_batch;
    h->nl = hidden_layers + 1;
    for (int l = 0; l < h->nl; ++l) {
        h->din.push_back(pad32(l == 0 ? n_in : hidden));
        h->dout.push_back(pad32(l == h->nl - 1 ? n_out : hidden));
    }
    size_t off = 0;
    for (int l = 0; l < h->nl; ++l) {
        h->w_off.push_back(off); off += (size_t)h->din[l] * h->dout[l];
        h->b_off.push_back(off); off += (size_t)h->dout[l];
    }
    h->nparam = off;
    int maxw = 0;
    for (int l = 0; l < h->nl; ++l) maxw = std::max(maxw, std::max(h->din[l], h->dout[l]));
    // one arena
    size_t bytes = 0;
    auto take = [&](size_t b) { size_t o = bytes; bytes = (bytes + b + 255) / 256 * 256; return o; };
    const size_t oP = take(off * 4), oG = take(off * 4), oM = take(off * 4), oV = take(off * 4), oPb = take(off * 2),
                 oMask = take(off), oWt = take(off * 2), oAt = take(h->nl * sizeof(LayerAt));
    std::vector<size_t> oX, oXt, oZ;
    for (int l = 0; l < h->nl; ++l) {
        oX.push_back(take((size_t)max_batch * h->din[l] * 2));
        oXt.push_back(take((size_t)max_batch * h->din[l] * 2));
        oZ.push_back(take((size_t)max_batch * h->dout[l] * 4));
    }
    const size_t odZ = take((size_t)max_batch * maxw * 2 * 4),
                 oxin = take((size_t)max_batch * n_in * 4), oyin = take((size_t)max_batch * n_out * 4),
                 host_bytes = 256 + ((size_t)max_batch * maxw / 256 + 1) * 4;
    if (cudaMalloc(&h->arena, bytes) != cudaSuccess || cudaMallocHost(&h->err, host_bytes) != cudaSuccess) {
        cudaFree(h->arena);
        delete h;
        return sl_record_error(SL_ERR_ALLOC, "allocation of the MLP's memory failed");
    }
    std::memset(h->err, 0, host_bytes);
    h->loss_part = reinterpret_cast<float*>(reinterpret_cast<char*>(h->err) + 256);
    char* b = static_cast<char*>(h->arena);
    h->P = (float*)(b + oP); h->G = (float*)(b + oG); h->Mom = (float*)(b + oM); h->Var = (float*)(b + oV);
    h->Pb = (bf16*)(b + oPb); h->mask = (uint8_t*)(b + oMask); h->Wt = (bf16*)(b + oWt); h->at = (LayerAt*)(b + oAt);
    for (int l = 0; l < h->nl; ++l) {
        h->X.push_back((bf16*)(b + oX[l]));
        h->Xt.push_back((bf16*)(b + oXt[l]));
        h->Z.push_back((float*)(b + oZ[l]));
    }
    for (int k = 0; k < 2; ++k) {
        h->dZ[k] = (bf16*)(b + odZ) + (size_t)(2 * k) * max_batch * maxw;
        h->dZt[k] = h->dZ[k] + (size_t)max_batch * maxw;
    }
    h->xin = (float*)(b + oxin); h->yin = (float*)(b + oyin);
    cudaMemset(h->arena, 0, bytes);
    // He-style init of live weights, zero biases and padding
    std::vector<float> p(off, 0.0f);
    std::vector<uint8_t> mk(off, 0);
    std::mt19937_64 rng(seed);
    std::normal_distribution<float> nd(0.0f, 1.0f);
    for (int l = 0; l < h->nl; ++l) {
        const int kin = l == 0 ? n_in : hidden, nout = l == h->nl - 1 ? n_out : hidden;
        const float sd = std::sqrt(2.0f / (float)kin);
        for (int r = 0; r < nout; ++r)
            for (int c = 0; c < kin; ++c) {
                const size_t i = h->w_off[l] + (size_t)r * h->din[l] + c;
                p[i] = sd * nd(rng);
                mk[i] = 1;
            }
        for (int r = 0; r < nout; ++r) mk[h->b_off[l] + r] = 1;
    }
    cudaMemcpy(h->P, p.data(), off * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(h->mask, mk.data(), off, cudaMemcpyHostToDevice);
    std::vector<LayerAt> at(h->nl);
    for (int l = 0; l < h->nl; ++l) at[l] = {(long long)h->w_off[l], h->din[l], h->dout[l]};
    cudaMemcpy(h->at, at.data(), at.size() * sizeof(LayerAt), cudaMemcpyHostToDevice);
    to_bf16_kernel<<<(int)((off + 255) / 256), 256>>>(h->P, h->Pb, h->Wt, h->at, h->nl, (int)off);
    if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaDeviceSynchronize() != cudaSuccess) {
        sl_mlp_destroy(h);
        return sl_record_error(SL_ERR_CUDA, "MLP initialisation failed");
    }
    int dev = 0, pageable = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&h->num_sms, cudaDevAttrMultiProcessorCount, dev);
    h->host_direct = cudaDeviceGetAttribute(&pageable, cudaDevAttrPageableMemoryAccess, dev) == cudaSuccess && pageable;
    h->fused = setup_forward(h);
    *out = h;
    return SL_OK;
}

int sl_mlp_destroy(sl_mlp* h)
{
    if (!h) return SL_OK;
    if (h->arena) cudaFree(h->arena);
    if (h->err) cudaFreeHost(h->err);
    if (h->epoch) cudaFree(h->epoch);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return SL_OK;
}

int sl_mlp_num_params(const sl_mlp* h, int64_t* n)
{
    if (!h || !n) return sl_record_error(SL_ERR_ARG, "null argument");
    *n = (int64_t)h->nparam;
    return SL_OK;
}

int sl_mlp_get_params(sl_mlp* h, float* params)
{
    if (!h || !params) return sl_record_error(SL_ERR_ARG, "null argument");
    if (cudaMemcpy(params, h->P, h->nparam * 4, cudaMemcpyDeviceToHost) != cudaSuccess)
        return sl_record_error(SL_ERR_CUDA, "copy failed");
    return SL_OK;
}

int sl_mlp_set_params(sl_mlp* h, const float* params)
{
    if (!h || !params) return sl_record_error(SL_ERR_ARG, "null argument");
    if (cudaMemcpy(h->P, params, h->nparam * 4, cudaMemcpyHostToDevice) != cudaSuccess)
        return sl_record_error(SL_ERR_CUDA, "copy failed");
    to_bf16_kernel<<<(int)((h->nparam + 255) / 256), 256>>>(h->P, h->Pb, h->Wt, h->at, h->nl, (int)h->nparam);
    if (cudaDeviceSynchronize() != cudaSuccess) return sl_record_error(SL_ERR_CUDA, "bf16 refresh failed");
    return SL_OK;
}

int sl_mlp_gradients(sl_mlp* h, const float* x, const float* y, int M, float* grads, float* loss)
{
    if (!h || !x || !y || M < 32 || M % 32 || M > h->max_batch)
        return sl_record_error(SL_ERR_ARG, "M must be a multiple of 32 up to max_batch");
    clear_status(h);
    // the kernels read x and y where they are, or from the staging
    const float* vx = static_cast<const float*>(device_view(h, x));
    const float* vy = static_cast<const float*>(device_view(h, y));
    if (!vx) cudaMemcpy(h->xin, x, (size_t)M * h->n_in * 4, cudaMemcpyHostToDevice);
    if (!vy) cudaMemcpy(h->yin, y, (size_t)M * h->n_out * 4, cudaMemcpyHostToDevice);
    const BatchInput in = pack_batch(h, vx ? vx : h->xin, vy ? vy : h->yin, M, M, nullptr);
    forward(h, in, M, true, nullptr);
    backward(h, in, M, nullptr);
    if (cudaDeviceSynchronize() != cudaSuccess) return sl_record_error(SL_ERR_CUDA, "MLP step failed");
    if (int r = mlp_status(h, "sl_mlp_gradients")) return r;
    if (grads) cudaMemcpy(grads, h->G, h->nparam * 4, cudaMemcpyDeviceToHost);
    if (loss) {
        const int ldo = h->dout[h->nl - 1];
        const int nb = (M * ldo + 255) / 256;
        double s = 0;
        for (int k = 0; k < nb; ++k) s += h->loss_part[k];
        *loss = (float)(s / ((double)M * h->n_out));
    }
    return SL_OK;
}

int sl_mlp_train(sl_mlp* h, const float* x, const float* y, int n, int epochs, int batch, float lr, uint64_t seed,
                 float* loss_per_epoch)
{
    if (!h || !x || !y || n < batch || batch < 32 || batch % 32 || batch > h->max_batch || epochs < 1)
        return sl_record_error(SL_ERR_ARG, "bad training arguments");
    clear_status(h);
    std::vector<int> idx(n);
    for (int i = 0; i < n; ++i) idx[i] = i;
    std::mt19937_64 rng(seed);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const int ld0 = h->din[0], ldo = h->dout[h->nl - 1];
    const int nb = (batch * ldo + 255) / 256;
    const int steps = n / batch;

    // The epoch's rows packed on the device, `seg` steps at a time.  Whole: the data
    // set is there too, and an epoch is packed at once in its order.  Otherwise,
    // beyond kEpochBytes or where the device has no room, the host gathers each
    // segment's rows.
    int seg = steps;
    bool whole = true;
    size_t bytes = 0, ox = 0, oy = 0, oidx = 0, oxp = 0, oxt = 0, oyp = 0, ocoef = 0, oloss = 0, ostep = 0;
    auto layout = [&] {
        bytes = 0;
        auto take = [&](size_t b) { size_t o = bytes; bytes = (bytes + b + 255) / 256 * 256; return o; };
        const size_t r = (size_t)seg * batch;
        ox = take((whole ? (size_t)n : r) * h->n_in * 4);
        oy = take(whole ? (size_t)n * h->n_out * 4 : 0);
        oidx = take(whole ? r * 4 : 0);
        oxp = take(r * ld0 * 2);
        oxt = take(r * ld0 * 2);
        oyp = take(r * h->n_out * 4);
        ocoef = take((size_t)seg * sizeof(float2));
        oloss = take((size_t)seg * nb * 4);
        ostep = take(sizeof(int));
    };
    layout();
    if (bytes > kEpochBytes) {
        whole = false;
        for (layout(); bytes > kEpochBytes && seg > 1; layout()) seg = (seg + 1) / 2;
    }
    if (bytes > h->epoch_bytes) {
        if (h->epoch) cudaFree(h->epoch);
        h->epoch = nullptr;
        h->epoch_bytes = 0;
        while (cudaMalloc(&h->epoch, bytes) != cudaSuccess) {
            cudaGetLastError();
            h->epoch = nullptr;
            if (!whole && seg == 1) return sl_record_error(SL_ERR_ALLOC, "sl_mlp_train: cudaMalloc of a batch failed");
            if (!whole) seg = (seg + 1) / 2;
            whole = false;
            layout();
        }
        h->epoch_bytes = bytes;
    }
    const int rows = seg * batch;
    char* e = static_cast<char*>(h->epoch);
    float *dx = (float*)(e + ox), *dy = (float*)(e + oy), *yp = (float*)(e + oyp), *dloss = (float*)(e + oloss);
    int *didx = (int*)(e + oidx), *dstep = (int*)(e + ostep);
    bf16 *xp = (bf16*)(e + oxp), *xt = (bf16*)(e + oxt);
    float2* dcoef = (float2*)(e + ocoef);
    cudaStream_t st = h->stream;
    std::vector<float> gx(whole ? 0 : (size_t)rows * h->n_in), gy(whole ? 0 : (size_t)rows * h->n_out);
    if (whole) {
        cudaMemcpyAsync(dx, x, (size_t)n * h->n_in * 4, cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(dy, y, (size_t)n * h->n_out * 4, cudaMemcpyHostToDevice, st);
    }

    // one step as a graph: it finds its rows by the step counter
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    const BatchInput in{xp, xt, yp, rows, dstep, dloss};
    bool ok = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
    if (ok) {
        forward(h, in, batch, true, st);
        backward(h, in, batch, st);
        sl::launch_pdl(true, adam_kernel, (int)((h->nparam + 255) / 256), 256, 0, st, h->P, h->G, h->Mom, h->Var, h->Pb,
                       h->Wt, h->at, h->nl, h->mask, (int)h->nparam, lr, b1, b2, eps, dcoef, dstep, -1);
        // a step without one of its products must not run: Adam would take the gradients that are there
        ok = cudaStreamEndCapture(st, &graph) == cudaSuccess && !h->tc_setup_failed &&
             cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess;
    }
    if (graph) cudaGraphDestroy(graph);
    int rc = ok                   ? SL_OK
             : h->tc_setup_failed ? mlp_status(h, "sl_mlp_train")
                                  : sl_record_error(SL_ERR_CUDA, "sl_mlp_train: the step's graph could not be made");

    std::vector<float> part((size_t)seg * nb);
    std::vector<float2> coef(seg);
    std::vector<int> next(idx);
    std::shuffle(next.begin(), next.end(), rng);
    for (int ep = 0; ep < epochs && rc == SL_OK; ++ep) {
        idx.swap(next);
        double ls = 0;
        for (int s0 = 0; s0 < steps && rc == SL_OK; s0 += seg) {
            const int ns = std::min(seg, steps - s0), nr = ns * batch;
            const int* order = idx.data() + (size_t)s0 * batch;
            for (int k = 0; k < ns; ++k) {
                ++h->step;
                coef[k] = make_float2(1.0f - std::pow(b1, (float)h->step), 1.0f - std::pow(b2, (float)h->step));
            }
            cudaMemcpyAsync(dcoef, coef.data(), (size_t)ns * sizeof(float2), cudaMemcpyHostToDevice, st);
            cudaMemsetAsync(dstep, 0, sizeof(int), st);
            if (whole) {
                cudaMemcpyAsync(didx, order, (size_t)nr * 4, cudaMemcpyHostToDevice, st);
                pack_kernel<<<(rows + 127) / 128, 128, 0, st>>>(dx, dy, didx, rows, n, h->n_in, h->n_out, ld0, xp, xt,
                                                                yp);
            } else {
                for (int r = 0; r < nr; ++r) {
                    std::memcpy(&gx[(size_t)r * h->n_in], &x[(size_t)order[r] * h->n_in], h->n_in * 4);
                    std::memcpy(&gy[(size_t)r * h->n_out], &y[(size_t)order[r] * h->n_out], h->n_out * 4);
                }
                cudaMemcpyAsync(dx, gx.data(), (size_t)nr * h->n_in * 4, cudaMemcpyHostToDevice, st);
                cudaMemcpyAsync(yp, gy.data(), (size_t)nr * h->n_out * 4, cudaMemcpyHostToDevice, st);
                pack_kernel<<<(rows + 127) / 128, 128, 0, st>>>(dx, nullptr, nullptr, rows, nr, h->n_in, h->n_out, ld0,
                                                                xp, xt, nullptr);
            }
            for (int k = 0; k < ns; ++k) cudaGraphLaunch(exec, st);
            if (s0 + ns == steps && ep + 1 < epochs) {  // the next epoch's order, under this one's last steps
                next = idx;
                std::shuffle(next.begin(), next.end(), rng);
            }
            cudaMemcpyAsync(part.data(), dloss, (size_t)ns * nb * 4, cudaMemcpyDeviceToHost, st);
            if (cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
                rc = sl_record_error(SL_ERR_CUDA, "training kernel failed");
            for (int k = 0; k < ns; ++k) {
                double s = 0;
                for (int i = 0; i < nb; ++i) s += part[(size_t)k * nb + i];
                ls += s / ((double)batch * h->n_out);
            }
        }
        if (loss_per_epoch && rc == SL_OK) loss_per_epoch[ep] = (float)(ls / std::max(1, steps));
    }
    if (exec) cudaGraphExecDestroy(exec);
    if (rc == SL_OK) rc = mlp_status(h, "sl_mlp_train");
    return rc;
}

int sl_mlp_predict(sl_mlp* h, const float* x, int n, float* y)
{
    if (!h || !x || !y || n < 1) return sl_record_error(SL_ERR_ARG, "bad arguments");
    clear_status(h);
    const int B = h->max_batch, L = h->nl, ldo = h->dout[L - 1];
    if (h->fused) {
        float* vx = static_cast<float*>(device_view(h, x));
        float* vy = static_cast<float*>(device_view(h, y));
        // staged: what the GPU cannot reach, and results over the inputs, of which
        // one CTA would write what another has yet to read
        const uintptr_t xa = reinterpret_cast<uintptr_t>(x), ya = reinterpret_cast<uintptr_t>(y);
        const bool overlap = xa < ya + (size_t)n * h->n_out * 4 && ya < xa + (size_t)n * h->n_in * 4;
        bool staged = !vx || !vy || overlap;
        cudaError_t e = cudaSuccess;
        if (!staged) {
            e = predict_in_place(h, vx, vy, n, &staged);
            if (e == cudaSuccess && staged) clear_status(h);
        }
        if (e == cudaSuccess && staged) e = predict_staged(h, x, y, n);
        if (e != cudaSuccess)
            return sl_record_error(SL_ERR_CUDA, (std::string("sl_mlp_predict: ") + cudaGetErrorString(e)).c_str());
        return mlp_status(h, "sl_mlp_predict");
    }
    std::vector<float> zb((size_t)B * ldo);
    for (int s0 = 0; s0 < n; s0 += B) {
        const int M = std::min(B, n - s0);
        const int Mp = (M + 31) / 32 * 32;
        cudaMemcpy(h->xin, x + (size_t)s0 * h->n_in, (size_t)M * h->n_in * 4, cudaMemcpyHostToDevice);
        forward(h, pack_batch(h, h->xin, nullptr, M, Mp, nullptr), Mp, false, nullptr);
        if (cudaMemcpy(zb.data(), h->Z[L - 1], (size_t)M * ldo * 4, cudaMemcpyDeviceToHost) != cudaSuccess)
            return sl_record_error(SL_ERR_CUDA, "prediction failed");
        if (int r = mlp_status(h, "sl_mlp_predict")) return r;
        for (int r = 0; r < M; ++r)
            for (int c = 0; c < h->n_out; ++c) y[(size_t)(s0 + r) * h->n_out + c] = zb[(size_t)r * ldo + c];
    }
    return SL_OK;
}

}  // extern "C"

extern "C" int sl_diag_mlp_fail(sl_mlp* h, int what)
{
    if (!h || what < 0 || what > SL_DIAG_MLP_SETUP) return sl_record_error(SL_ERR_ARG, "sl_diag_mlp_fail: bad argument");
    if (what == SL_DIAG_MLP_TIMED_OUT)
        *h->err = 1;
    else
        h->fail_next = what;
    return SL_OK;
}

extern "C" int sl_diag_gemm_bf16(int M, int N, int K, const uint16_t* A, const uint16_t* B, const float* bias,
                                 int act, int kernel, float* C, uint16_t* Cb)
{
    if (M < 1 || N < 1 || K < 1 || K % 8 || !A || !B || !C || (kernel != 0 && kernel != 1))
        return sl_record_error(SL_ERR_ARG, "sl_diag_gemm_bf16: need M, N >= 1, K a multiple of 8, kernel 0 or 1");
    if (kernel == 0 && K % kTK)
        return sl_record_error(SL_ERR_ARG, "sl_diag_gemm_bf16: the mma.sync kernel needs K a multiple of 32");
    const size_t na = (size_t)M * K, nbb = (size_t)N * K, nc = (size_t)M * N;
    size_t off = 0;
    auto take = [&](size_t b) { size_t o = off; off = (off + b + 255) / 256 * 256; return o; };
    const size_t oA = take(na * 2), oB = take(nbb * 2), oBias = take((size_t)N * 4), oC = take(nc * 4),
                 oCb = take(nc * 2), oErr = take(sizeof(int));
    void* arena = nullptr;
    if (cudaMalloc(&arena, off) != cudaSuccess) return sl_record_error(SL_ERR_ALLOC, "sl_diag_gemm_bf16: cudaMalloc");
    char* b = static_cast<char*>(arena);
    bf16* dA = (bf16*)(b + oA);
    bf16* dB = (bf16*)(b + oB);
    float* dBias = bias ? (float*)(b + oBias) : nullptr;
    float* dC = (float*)(b + oC);
    bf16* dCb = Cb ? (bf16*)(b + oCb) : nullptr;
    int* dErr = (int*)(b + oErr);
    int rc = SL_OK;
    cudaMemcpy(dA, A, na * 2, cudaMemcpyHostToDevice);
    cudaMemcpy(dB, B, nbb * 2, cudaMemcpyHostToDevice);
    if (bias) cudaMemcpy(dBias, bias, (size_t)N * 4, cudaMemcpyHostToDevice);
    cudaMemset(dErr, 0, sizeof(int));
    if (kernel == 0) {
        gemm_mma_sync(nullptr, dA, K, dB, K, dBias, dC, dCb, N, M, N, K, act);
    } else {
        GemmLaunch L{};
        L.njobs = 1;
        L.err = dErr;
        bool ok = make_job(&L.job[0], dA, M, K, dB, K, K, M, N, K);
        L.job[0].bias = dBias;
        L.job[0].cf = dC;
        L.job[0].cb = dCb;
        L.job[0].ldc = N;
        L.job[0].act = act;
        ok = ok && launch_gemm(L, nullptr);
        if (!ok) rc = sl_record_error(SL_ERR_CUDA, "sl_diag_gemm_bf16: tensor map or launch setup failed");
    }
    if (rc == SL_OK) {
        cudaError_t e = cudaDeviceSynchronize();
        if (e != cudaSuccess) rc = sl_record_error(SL_ERR_CUDA, cudaGetErrorString(e));
    }
    int herr = 0;
    if (rc == SL_OK) {
        cudaMemcpy(&herr, dErr, sizeof(int), cudaMemcpyDeviceToHost);
        if (herr) rc = sl_record_error(SL_ERR_TIMEOUT, "sl_diag_gemm_bf16: a bounded wait in the tcgen05 GEMM ran out");
    }
    if (rc == SL_OK) {
        cudaMemcpy(C, dC, nc * 4, cudaMemcpyDeviceToHost);
        if (Cb) cudaMemcpy(Cb, dCb, nc * 2, cudaMemcpyDeviceToHost);
    }
    cudaFree(arena);
    return rc;
}
