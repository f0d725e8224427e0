// BF16 tensor-core GEMM for sm_100a (tcgen05 + TMEM) and, with fused kernels of its own, the
// warm-start MLP.
//
// rf_gemm_bf16 computes C[M x N] = A[M x K] * B[N x K]^T with both operands K-major
// (row-major with K contiguous), BF16 inputs and FP32 accumulation in tensor memory:
//   - one CTA of 128 threads per 128-row tile of C (grid.x), the whole N (<= 256) per
//     CTA, K split over grid.y (split-K results are added atomically);
//   - K is walked in chunks of 64: the four warps stage the A chunk (128 x 64) and the
//     B chunk (N x 64) in shared memory in the canonical no-swizzle K-major layout
//     (8-row x 16-byte core matrices; 128 bytes between K-adjacent core matrices,
//     1024 bytes between 8-row groups), one elected thread issues four
//     tcgen05.mma.kind::f16 (M=128, K=16 each) into the TMEM accumulator and commits
//     them to an mbarrier that all threads wait on (bounded);
//   - the epilogue reads the accumulator with tcgen05.ld (warp w owns TMEM lanes
//     32w..32w+31, one row per thread) and applies bias/ReLU, a ReLU mask, or the split-K
//     atomic add, writing BF16 rows, their transpose or FP32.
// Waits give up after a bounded number of polls, raise an error flag and still free the
// tensor memory before returning.
#include <cuda_bf16.h>
#include <cstring>
#include <cmath>
#include <algorithm>
#include <vector>
#include "rf_common.cuh"

namespace rf {
namespace mlp {

enum Epi : int {
    EPI_RELU_BF16 = 0,      // h = relu(acc + bias) -> bf16 rows (+ transpose)
    EPI_LINEAR_F32 = 1,     // y = acc + bias -> fp32, first ncols_f columns
    EPI_MASK_BF16 = 2,      // dz = acc * (mask > 0) -> bf16 rows (+ transpose)
    EPI_ATOMIC_F32 = 3,     // out += scale * acc (split-K weight gradients)
};

struct GemmArgs {
    const __nv_bfloat16* A;
    const __nv_bfloat16* B;
    int M, N, K, lda, ldb;
    int chunks_per_split;
    int mode;
    const float* bias;
    const __nv_bfloat16* mask;
    int ldm;
    __nv_bfloat16* out_h;
    int ld_h;
    __nv_bfloat16* out_ht;
    int ld_ht;
    float* out_f;
    int ld_f, ncols_f;
    float scale;
    uint32_t* err;
};

#define GEMM_KC 64                      // K per staged chunk (four MMAs of K = 16)
#define GEMM_A_BYTES (128 * GEMM_KC * 2)
#define GEMM_B_MAX_BYTES (256 * GEMM_KC * 2)
#define GEMM_WAIT_LIMIT (1u << 24)

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor: canonical K-major layout without swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);            // start address
    d |= (uint64_t)((128u >> 4) & 0x3FFFu) << 16;        // leading byte offset: K-adjacent core matrices
    d |= (uint64_t)((1024u >> 4) & 0x3FFFu) << 32;       // stride byte offset: 8-row groups
    d |= (uint64_t)1 << 46;                              // descriptor version (sm_100)
    return d;                                            // base offset 0, layout type 0 (no swizzle)
}

// Instruction descriptor of kind::f16: D = F32, A = B = BF16, both K-major, M = 128.
__host__ __device__ __forceinline__ uint32_t umma_idesc(int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase) {
    for (uint32_t it = 0; it < GEMM_WAIT_LIMIT; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(bar), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Copy the 16-byte pieces of a rows x 64 chunk (rows from r0, columns from k0) into the
// canonical layout; rows >= nrows and columns >= K read as zero.
__device__ __forceinline__ void stage_chunk(uint8_t* s, const __nv_bfloat16* g, int ld, int r0, int nrows, int rows,
                                            int k0, int K) {
    const int pieces = rows * (GEMM_KC / 8);
    for (int p = threadIdx.x; p < pieces; p += blockDim.x) {
        const int r = p >> 3, kg = p & 7;
        const int gr = r0 + r, gk = k0 + kg * 8;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (gr < nrows && gk < K) v = *reinterpret_cast<const uint4*>(g + (size_t)gr * ld + gk);
        *reinterpret_cast<uint4*>(s + (r >> 3) * 1024 + kg * 128 + (r & 7) * 16) = v;
    }
}

template <int NC>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[NC]);
template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
}

__global__ void __launch_bounds__(128) k_umma_gemm(GemmArgs g) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sA = smem;
    uint8_t* sB = smem + GEMM_A_BYTES;
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t s_taddr;
    __shared__ uint32_t s_fail;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * 128;
    const int ncols = g.N <= 32 ? 32 : (g.N <= 64 ? 64 : (g.N <= 128 ? 128 : 256));
    const uint32_t bar_a = smem_u32(&bar);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_taddr)),
                     "r"(ncols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (threadIdx.x == 0) {
        s_fail = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar_a) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t taddr = s_taddr;
    const int nchunks = (g.K + GEMM_KC - 1) / GEMM_KC;
    const int c0 = blockIdx.y * g.chunks_per_split;
    const int c1 = min(nchunks, c0 + g.chunks_per_split);
    const uint32_t idesc = umma_idesc(g.N);
    uint32_t phase = 0;
    bool ok = true;
    for (int c = c0; c < c1 && ok; ++c) {
        stage_chunk(sA, g.A, g.lda, m0, g.M, 128, c * GEMM_KC, g.K);
        stage_chunk(sB, g.B, g.ldb, 0, g.N, g.N, c * GEMM_KC, g.K);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // generic writes -> tensor core reads
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int s = 0; s < GEMM_KC / 16; ++s) {
                const uint64_t da = umma_desc(smem_u32(sA + s * 256));
                const uint64_t db = umma_desc(smem_u32(sB + s * 256));
                const uint32_t acc = (c > c0 || s > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
                    :
                    : "r"(taddr), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar_a)
                         : "memory");
        }
        if (!mbar_wait(bar_a, phase)) {
            atomicOr(&s_fail, 1u);
        }
        phase ^= 1u;
        __syncthreads();                                 // the staging buffers are free again
        ok = (s_fail == 0);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    }
    if (!ok) {
        if (threadIdx.x == 0 && g.err) atomicOr(g.err, 1u);
    } else if (c1 > c0) {
        // epilogue: thread (warp w, lane l) owns row m0 + 32w + l
        const int row = m0 + warp * 32 + lane;
        for (int cb = 0; cb < g.N; cb += 16) {
            float v[16];
            tmem_ld<16>(taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)cb, v);
            if (row >= g.M) continue;
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const int col = cb + q;
                if (col >= g.N) break;
                float a = v[q];
                switch (g.mode) {
                    case EPI_RELU_BF16: {
                        a = fmaxf(a + (g.bias ? g.bias[col] : 0.f), 0.f);
                        const __nv_bfloat16 h = __float2bfloat16_rn(a);
                        g.out_h[(size_t)row * g.ld_h + col] = h;
                        if (g.out_ht) g.out_ht[(size_t)col * g.ld_ht + row] = h;
                        break;
                    }
                    case EPI_LINEAR_F32:
                        if (col < g.ncols_f) g.out_f[(size_t)row * g.ld_f + col] = (a + (g.bias ? g.bias[col] : 0.f)) * g.scale;
                        break;
                    case EPI_MASK_BF16: {
                        const float m = __bfloat162float(g.mask[(size_t)row * g.ldm + col]);
                        const __nv_bfloat16 h = __float2bfloat16_rn(m > 0.f ? a : 0.f);
                        g.out_h[(size_t)row * g.ld_h + col] = h;
                        if (g.out_ht) g.out_ht[(size_t)col * g.ld_ht + row] = h;
                        break;
                    }
                    default:
                        if (col < g.ncols_f) atomicAdd(&g.out_f[(size_t)row * g.ld_f + col], g.scale * a);
                        break;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
    }
}

}  // namespace mlp
}  // namespace rf

using namespace rf;
using namespace rf::mlp;

namespace {
uint32_t* gemm_err_word() {
    static thread_local uint32_t* w = nullptr;
    if (!w) {
        if (cudaMalloc(&w, sizeof(uint32_t)) != cudaSuccess) return nullptr;
        cudaMemset(w, 0, sizeof(uint32_t));
    }
    return w;
}
}  // namespace

extern "C" rf_status rf_gemm_bf16(const void* A, int lda, const void* B, int ldb, int M, int N, int K, int mode,
                                  const float* bias, const void* mask, int ldm, void* out_h, int ld_h, void* out_ht,
                                  int ld_ht, float* out_f, int ld_f, int ncols_f, float scale, int splits,
                                  rf_stream stream) {
    if (!A || !B || M <= 0 || N <= 0 || K <= 0 || N > 256 || (N % 16) != 0 || (K % 8) != 0 || (lda % 8) != 0 ||
        (ldb % 8) != 0 || lda < K || ldb < K || mode < 0 || mode > 3 || splits <= 0 ||
        ((uintptr_t)A % 16) != 0 || ((uintptr_t)B % 16) != 0) {
        set_error("rf_gemm_bf16: bad arguments (N multiple of 16 up to 256, K and leading dims multiples of 8, "
                  "16-byte aligned operands)");
        return RF_ERR_INVALID;
    }
    if ((mode == EPI_RELU_BF16 || mode == EPI_MASK_BF16) && (!out_h || ld_h < N || (mode == EPI_MASK_BF16 && !mask))) {
        set_error("rf_gemm_bf16: bf16 epilogue needs out_h (and mask)");
        return RF_ERR_INVALID;
    }
    if ((mode == EPI_LINEAR_F32 || mode == EPI_ATOMIC_F32) && (!out_f || ncols_f <= 0 || ncols_f > N)) {
        set_error("rf_gemm_bf16: fp32 epilogue needs out_f and 0 < ncols_f <= N");
        return RF_ERR_INVALID;
    }
    if (mode != EPI_ATOMIC_F32 && splits != 1) {
        set_error("rf_gemm_bf16: split-K only with the atomic epilogue");
        return RF_ERR_INVALID;
    }
    uint32_t* err = gemm_err_word();
    if (!err) { set_error("rf_gemm_bf16: no status word"); return RF_ERR_CUDA; }
    GemmArgs g;
    std::memset(&g, 0, sizeof(g));
    g.A = (const __nv_bfloat16*)A; g.B = (const __nv_bfloat16*)B;
    g.M = M; g.N = N; g.K = K; g.lda = lda; g.ldb = ldb;
    const int nchunks = (K + GEMM_KC - 1) / GEMM_KC;
    const int sp = splits > nchunks ? nchunks : splits;
    g.chunks_per_split = (nchunks + sp - 1) / sp;
    g.mode = mode; g.bias = bias; g.mask = (const __nv_bfloat16*)mask; g.ldm = ldm;
    g.out_h = (__nv_bfloat16*)out_h; g.ld_h = ld_h; g.out_ht = (__nv_bfloat16*)out_ht; g.ld_ht = ld_ht;
    g.out_f = out_f; g.ld_f = ld_f; g.ncols_f = ncols_f; g.scale = scale; g.err = err;
    const size_t smem = GEMM_A_BYTES + (size_t)N * GEMM_KC * 2;
    static bool attr_set = false;
    if (!attr_set) {
        RF_CUDA(cudaFuncSetAttribute(k_umma_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     GEMM_A_BYTES + GEMM_B_MAX_BYTES));
        attr_set = true;
    }
    const int gy = (nchunks + g.chunks_per_split - 1) / g.chunks_per_split;
    dim3 grid((M + 127) / 128, gy);
    k_umma_gemm<<<grid, 128, smem, (cudaStream_t)stream>>>(g);
    RF_CHECK_LAUNCH("k_umma_gemm");
    return RF_OK;
}

// Read and clear the GEMM status word (1 = an MMA completion wait gave up).
extern "C" rf_status rf_gemm_status(rf_stream stream) {
    uint32_t* err = gemm_err_word();
    if (!err) return RF_ERR_CUDA;
    uint32_t h = 0;
    RF_CUDA(cudaMemcpyAsync(&h, err, sizeof(h), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    RF_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
    if (h) {
        RF_CUDA(cudaMemsetAsync(err, 0, sizeof(uint32_t), (cudaStream_t)stream));
        set_error("rf_gemm_bf16: tensor-core completion wait timed out");
        return RF_ERR_CUDA;
    }
    return RF_OK;
}

// ===========================================================================
// Warm-start MLP: 64 -> 128 -> 128 -> 128 -> 6 (padded to 16), ReLU, BF16 weights and
// activations, FP32 accumulation in tensor memory, FP32 master weights trained with Adam
// on the mean squared error. Weights are kept in the layout of a linear layer, W[out][in].
//
// Both directions are one kernel each: a tile of 128 rows goes through every layer inside
// one CTA, its activations never leave shared memory, and a training step's weight
// gradients stay in tensor memory until the CTA has seen all its tiles. What a step must
// move is then the features and targets (152 B a row) and, for the bias sums, dZ (800 B a
// row, written and read); the arithmetic is about 235 kFLOP a row (0.31 ms at the measured
// tensor rate for 2M rows). Measured on a B200: a training step on 2M rows 2.4 ms, inference
// of 300k rows 66 us with the host's wait; layer-by-layer GEMMs with the activations and
// their transposes in memory took 58 ms and 1.58 ms. What bounds both is the chain of a tile
// (GEMM, accumulator read, conversion, shared-memory write, barrier, seven times over in
// training): the tensor cores idle in it.
//
// Every matrix in shared memory is in 8-row x 16-byte core matrices (128 contiguous
// bytes): core (rg, cg) of a buffer of R rows at cg * R * 16 + rg * 128, so that element
// (r, c) of the buffer sits at (c / 8) * R * 16 + r * 16 + (c % 8) * 2. The same bytes are
// a K-major operand with the columns as K (leading offset R * 16 between K-adjacent cores,
// stride offset 128 between 8-row groups) and an MN-major operand with the rows as K
// (leading offset 128 between 8-row groups, stride offset R * 16 between column groups):
// a layer's activations serve the next layer's GEMM and the weight gradient, its weights
// the forward and the backward pass, without a transpose anywhere.
// ===========================================================================
namespace rf {
namespace mlp {

static const int NL = 4;
static const int DIN[NL] = {64, 128, 128, 128};
static const int DOUT[NL] = {128, 128, 128, 16};     // the last layer's 6 outputs padded to 16
static const int NOUT = 6;

#define MLP_TILE 128                        // rows of a tile: the M of every MMA over rows
#define MLP_CS (MLP_TILE * 16)              // bytes of a column group of a tile (8 columns)
#define MLP_W1 0                            // weights in shared memory: W1 W2 W3 W4, then the biases
#define MLP_W2 (MLP_W1 + 128 * 64 * 2)
#define MLP_W3 (MLP_W2 + 128 * 128 * 2)
#define MLP_W4 (MLP_W3 + 128 * 128 * 2)
#define MLP_BIAS (MLP_W4 + 16 * 128 * 2)
#define MLP_DATA (MLP_BIAS + (3 * 128 + 16) * 4)
#define MLP_T_WARPS 16                      // of a training CTA, and the one that issues the MMAs
#define MLP_T_THREADS (32 * MLP_T_WARPS + 32)
#define MLP_SPLITS 64                       // splits of a training step's rows (CTAs)

// Shared memory of a training CTA: features, activations H1..H3 (the gradients dZ1..dZ3
// replace them in place), dZ4.
#define MLP_T_X MLP_DATA
#define MLP_T_H1 (MLP_T_X + 8 * MLP_CS)
#define MLP_T_H2 (MLP_T_H1 + 16 * MLP_CS)
#define MLP_T_H3 (MLP_T_H2 + 16 * MLP_CS)
#define MLP_T_D4 (MLP_T_H3 + 16 * MLP_CS)
#define MLP_T_SMEM (MLP_T_D4 + 2 * MLP_CS)
// Shared memory of an inference CTA: one 32 KB activation buffer per warpgroup.
#define MLP_F_GROUPS 4
#define MLP_F_SMEM (MLP_DATA + MLP_F_GROUPS * 16 * MLP_CS)

// Tensor memory columns of a training CTA: the working accumulator, then the gradients
// dW1^T.. with lane = output, column = input (W4: lane = input, column = output).
#define MLP_C_ACC 0
#define MLP_C_D1 128
#define MLP_C_D2 (MLP_C_D1 + 64)
#define MLP_C_D3 (MLP_C_D2 + 128)
#define MLP_C_D4 (MLP_C_D3 + 128)
#define MLP_GCOLS 336                       // gradient columns
static_assert(MLP_C_D1 + MLP_GCOLS == MLP_C_D4 + 16 && MLP_C_D4 + 16 <= 512, "tensor memory columns");
static_assert(MLP_T_SMEM <= 227 * 1024 && MLP_F_SMEM <= 227 * 1024, "shared memory of an SM");

struct MlpWeights {
    const __nv_bfloat16* W[NL];
    const float* b[NL];
};

// What a training step leaves for its bias gradients: the rows' output gradients (outputs
// 0..3 and 4..5) and dZ1..dZ3 in bf16, in the order in which k_mlp_bias adds them: by 8-column
// group and 32-row share of every 256 rows, so that each of its warps reads one contiguous stream.
struct BiasRows {
    float4* dy;              // [8 shares][nk][32 rows]
    float2* dy2;
    uint4* dz[3];            // [16 column groups][8 shares][nk][32 rows]
    long nk;                 // 256-row blocks
};

__device__ __forceinline__ uint64_t mlp_desc(uint32_t saddr, uint32_t lead, uint32_t stride) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lead >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((stride >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}
#define IDESC_A_MN (1u << 15)               // A is MN-major
#define IDESC_B_MN (1u << 16)               // B is MN-major

__device__ __forceinline__ void mlp_mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, bool acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
        :
        : "r"(d), "l"(da), "l"(db), "r"(idesc), "r"(acc ? 1u : 0u), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void mlp_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}

// acc[128][n] = A[128 rows][16 ks] * W^T: a layer's forward GEMM. W: [n][k] buffer at w.
__device__ __forceinline__ void mma_forward(uint32_t d, uint32_t a, uint32_t w, int n, int ks) {
    const uint32_t wcs = (uint32_t)n * 16u;
    for (int s = 0; s < ks; ++s)
        mlp_mma(d, mlp_desc(a + s * 2 * MLP_CS, MLP_CS, 128), mlp_desc(w + s * 2 * wcs, wcs, 128), umma_idesc(n), s > 0);
}
// acc[128][128] = dZ[128 rows][o outputs] * W: the gradient at a layer's input. W: [o][128].
__device__ __forceinline__ void mma_input_grad(uint32_t d, uint32_t dz, uint32_t w, int o) {
    const uint32_t wcs = (uint32_t)o * 16u;
    for (int s = 0; s < o / 16; ++s)
        mlp_mma(d, mlp_desc(dz + s * 2 * MLP_CS, MLP_CS, 128), mlp_desc(w + s * 256, 128, wcs),
                umma_idesc(128) | IDESC_B_MN, s > 0);
}
// g[m][n] += P^T Q over the tile's 128 rows (P: 128 columns, Q: n columns).
__device__ __forceinline__ void mma_weight_grad(uint32_t d, uint32_t p, uint32_t q, int n, bool add) {
    for (int s = 0; s < MLP_TILE / 16; ++s)
        mlp_mma(d, mlp_desc(p + s * 256, 128, MLP_CS), mlp_desc(q + s * 256, 128, MLP_CS),
                umma_idesc(n) | IDESC_A_MN | IDESC_B_MN, add || s > 0);
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// b's halves where h's are positive, else zero. h are activations after ReLU (+0 to +inf): adding
// 0x7FFF sets a half's top bit, with no carry out of it, exactly if the half is not zero, and
// the byte permutation spreads the two top bits over their halves.
__device__ __forceinline__ uint32_t mask_bf16(uint32_t b, uint32_t h) {
    uint32_t m;
    asm("prmt.b32 %0, %1, 0, 0xBB99;" : "=r"(m) : "r"(h + 0x7FFF7FFFu));
    return b & m;
}
// bf16 of max(a + bias, 0), a pair at once: rounded first, so the larger of the rounded sum and +0
// (a NaN sum gives 0, as fmaxf does in FP32).
__device__ __forceinline__ uint32_t relu_pair(uint32_t a0, uint32_t a1, float b0, float b1) {
    const __nv_bfloat162 h = __hmax2(__floats2bfloat162_rn(__uint_as_float(a0) + b0, __uint_as_float(a1) + b1),
                                     __floats2bfloat162_rn(0.f, 0.f));
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Weights (bf16 [out][in]) and biases into shared memory.
__device__ __forceinline__ void load_weights(uint8_t* smem, const MlpWeights& w) {
    const int off[NL] = {MLP_W1, MLP_W2, MLP_W3, MLP_W4}, in[NL] = {64, 128, 128, 128}, out[NL] = {128, 128, 128, 16};
    float* sb = reinterpret_cast<float*>(smem + MLP_BIAS);
#pragma unroll
    for (int l = 0; l < NL; ++l) {
        const int pieces = out[l] * in[l] / 8;
        for (int p = threadIdx.x; p < pieces; p += blockDim.x) {
            const int o = p % out[l], cg = p / out[l];
            *reinterpret_cast<uint4*>(smem + off[l] + cg * out[l] * 16 + o * 16) =
                __ldg(reinterpret_cast<const uint4*>(w.W[l] + (size_t)o * in[l] + cg * 8));
        }
        for (int o = threadIdx.x; o < out[l]; o += blockDim.x) sb[l * 128 + o] = w.b[l][o];
    }
}

// 32 accumulator columns of a row -> bias, ReLU -> four 16-byte pieces of the activations.
__device__ __forceinline__ void hidden_piece(const uint32_t (&r)[32], const float* bias, uint8_t* dst) {
    const float4* b4 = reinterpret_cast<const float4*>(bias);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 u = b4[2 * q], v = b4[2 * q + 1];
        *reinterpret_cast<uint4*>(dst + q * MLP_CS) =
            make_uint4(relu_pair(r[8 * q], r[8 * q + 1], u.x, u.y), relu_pair(r[8 * q + 2], r[8 * q + 3], u.z, u.w),
                       relu_pair(r[8 * q + 4], r[8 * q + 5], v.x, v.y), relu_pair(r[8 * q + 6], r[8 * q + 7], v.z, v.w));
    }
}

// Inference. Four warpgroups a CTA, each with its own tile, buffer, accumulator (128
// columns) and barrier: while one converts its accumulators the others' MMAs run. A
// layer's activations overwrite its input in place (its MMAs have finished reading).
__global__ void __launch_bounds__(128 * MLP_F_GROUPS, 1)
k_mlp_forward(MlpWeights w, const __nv_bfloat16* __restrict__ X, int rows, float* Y, int ldy, int ncols, int residual,
              uint32_t* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[MLP_F_GROUPS];
    __shared__ uint32_t s_taddr;
    const int warp = threadIdx.x >> 5, grp = threadIdx.x >> 7, row = threadIdx.x & 127, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_taddr)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int q = 0; q < MLP_F_GROUPS; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&bars[q])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    load_weights(smem, w);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t acc = s_taddr + (uint32_t)grp * 128u, bar = smem_u32(&bars[grp]);
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    uint8_t* H = smem + MLP_DATA + grp * 16 * MLP_CS;
    const uint32_t sH = smem_u32(H), sW = smem_u32(smem);
    const float* sb = reinterpret_cast<const float*>(smem + MLP_BIAS);
    const long ntiles = ((long)rows + MLP_TILE - 1) / MLP_TILE;
    uint32_t phase = 0;
    bool ok = true;
    auto group_sync = [&]() { asm volatile("bar.sync %0, 128;\n" ::"r"(grp + 1) : "memory"); };
    // a warp's rows are 32; its loads take 8 rows x 64 bytes at a time
    const int lr = (warp & 3) * 32 + (lane & 7), lk = lane >> 3;
    for (long tile = blockIdx.x + (long)grp * gridDim.x; tile < ntiles; tile += (long)gridDim.x * MLP_F_GROUPS) {
        const long r0 = tile * MLP_TILE;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int r = lr + (q >> 1) * 8, kg = (q & 1) * 4 + lk;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (r0 + r < rows) v = __ldg(reinterpret_cast<const uint4*>(X + (size_t)(r0 + r) * 64) + kg);
            *reinterpret_cast<uint4*>(H + kg * MLP_CS + r * 16) = v;
        }
        float xin[NOUT];
        if (residual) {
            __syncwarp();
#pragma unroll
            for (int c = 0; c < NOUT; ++c) xin[c] = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(H + row * 16)[c]);
        }
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            group_sync();
            if (row == 0) {
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const int wo = l == 0 ? MLP_W1 : l == 1 ? MLP_W2 : l == 2 ? MLP_W3 : MLP_W4;
                mma_forward(acc, sH, sW + wo, l < 3 ? 128 : 16, l == 0 ? 4 : 8);
                mlp_commit(bar);
            }
            ok = mbar_wait(bar, phase) && ok;
            phase ^= 1u;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            if (l < 3) {
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    uint32_t r[32];
                    tmem_ld32(acc + lanes + h * 32, r);
                    tmem_ld_wait();
                    hidden_piece(r, sb + l * 128 + h * 32, H + h * 4 * MLP_CS + row * 16);
                }
            }
        }
        float v[16];
        tmem_ld<16>(acc + lanes, v);
#pragma unroll
        for (int c = 0; c < 16; ++c) v[c] += sb[3 * 128 + c];
        if (residual) {
#pragma unroll
            for (int c = 0; c < NOUT; ++c) v[c] += xin[c];
        }
        if (r0 + row < rows) {
            float* y = Y + (size_t)(r0 + row) * ldy;
            if (ncols == 16 && (ldy & 3) == 0 && ((uintptr_t)Y & 15) == 0) {
#pragma unroll
                for (int c = 0; c < 16; c += 4)
                    *reinterpret_cast<float4*>(y + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
            } else {
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    if (c < ncols) y[c] = v[c];
            }
        }
    }
    if (!ok && err) atomicOr(err, 1u);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(s_taddr), "r"(512) : "memory");
    }
}

// One training step's forward and backward pass over a CTA's split of the rows (`split` rows, a
// multiple of 64; up to 64 splits). Warp w < 16 owns rows 32 (w % 4) .. + 31 of the tile and
// columns 32 (w / 4) .. + 31 of each layer; warp 16 issues the MMAs (an issuing thread is held
// about as long as its MMAs run). The chain of a tile is seven GEMMs, each followed by its
// epilogue; the weight gradients are issued behind the GEMM the chain waits for and run under
// its epilogue, as do the stores to memory. part: the CTA's gradient columns [336][128].
// A split's weight gradients are one tensor-memory accumulation over its rows in order, the
// splits those of a split-K GEMM over 64-row chunks: the FP32 accumulator's rounding over tens
// of thousands of rows is the largest error of a step, and with other splits (one per SM, every
// 148th tile: 0.97 ms a step at 2M rows against 2.4 ms) the gradients moved by 5e-5.
__global__ void __launch_bounds__(MLP_T_THREADS, 1)
k_mlp_train(MlpWeights w, const __nv_bfloat16* __restrict__ X, const float* __restrict__ T, int rows, long split,
            int residual, float* __restrict__ part, double* __restrict__ loss_part, BiasRows out_rows, uint32_t* err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t s_taddr, s_fail;
    __shared__ double s_loss[4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = (warp & 3) * 32 + lane, quart = warp >> 2;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s_taddr)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (threadIdx.x == 0) {
        s_fail = 0;
        for (int q = 0; q < 2; ++q)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&bars[q])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    load_weights(smem, w);
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tm = s_taddr, bar_a = smem_u32(&bars[0]), bar_g = smem_u32(&bars[1]);
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t sm = smem_u32(smem);
    const float* sb = reinterpret_cast<const float*>(smem + MLP_BIAS);
    const long row0 = (long)blockIdx.x * split, row1 = min((long)rows, row0 + split);
    const float inv = 2.0f / ((float)rows * (float)NOUT);
    uint32_t pa = 0, pg = 0;
    bool ok = true;
    double loss = 0.0;
    // features of a tile: warp w loads rows 8 w .. + 7, 64 bytes of each at a time
    const int lr = warp * 8 + (lane & 7), lk = lane >> 3;
    uint4 xv[2];
    auto fetch = [&](long first_row) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const long r = first_row + lr;
            xv[q] = make_uint4(0u, 0u, 0u, 0u);
            if (r < row1) xv[q] = __ldg(reinterpret_cast<const uint4*>(X + (size_t)r * 64) + q * 4 + lk);
        }
    };
    // shared-memory writes and tensor-memory reads of the stage done: the next MMAs may follow
    auto stage_sync = [&]() {
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    };
    auto wait_a = [&]() {
        if (!mbar_wait(bar_a, pa)) s_fail = 1;
        pa ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    };
    auto wait_g = [&]() {
        if (!mbar_wait(bar_g, pg)) s_fail = 1;
        pg ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    };
    bool first = true;
    if (warp == MLP_T_WARPS) {
        // the MMAs of a tile, each batch after the barrier that its operands' writers reach
        for (long r0 = row0; r0 < row1; r0 += MLP_TILE) {
            stage_sync();
            ok = s_fail == 0;
            if (!ok) break;
            const bool issue = lane == 0;
            if (issue) { mma_forward(tm + MLP_C_ACC, sm + MLP_T_X, sm + MLP_W1, 128, 4); mlp_commit(bar_a); }
            stage_sync();
            if (issue) { mma_forward(tm + MLP_C_ACC, sm + MLP_T_H1, sm + MLP_W2, 128, 8); mlp_commit(bar_a); }
            stage_sync();
            if (issue) { mma_forward(tm + MLP_C_ACC, sm + MLP_T_H2, sm + MLP_W3, 128, 8); mlp_commit(bar_a); }
            stage_sync();
            if (issue) { mma_forward(tm + MLP_C_ACC, sm + MLP_T_H3, sm + MLP_W4, 16, 8); mlp_commit(bar_a); }
            stage_sync();
            if (issue) {
                mma_input_grad(tm + MLP_C_ACC, sm + MLP_T_D4, sm + MLP_W4, 16);
                mlp_commit(bar_a);
                mma_weight_grad(tm + MLP_C_D4, sm + MLP_T_H3, sm + MLP_T_D4, 16, !first);
                mlp_commit(bar_g);
            }
            stage_sync();
            if (issue) {
                mma_input_grad(tm + MLP_C_ACC, sm + MLP_T_H3, sm + MLP_W3, 128);
                mlp_commit(bar_a);
                mma_weight_grad(tm + MLP_C_D3, sm + MLP_T_H3, sm + MLP_T_H2, 128, !first);
                mlp_commit(bar_g);
            }
            stage_sync();
            if (issue) {
                mma_input_grad(tm + MLP_C_ACC, sm + MLP_T_H2, sm + MLP_W2, 128);
                mlp_commit(bar_a);
                mma_weight_grad(tm + MLP_C_D2, sm + MLP_T_H2, sm + MLP_T_H1, 128, !first);
                mlp_commit(bar_g);
            }
            stage_sync();
            if (issue) {
                mma_weight_grad(tm + MLP_C_D1, sm + MLP_T_H1, sm + MLP_T_X, 64, !first);
                mlp_commit(bar_g);
            }
            __syncwarp();
            first = false;
        }
    } else {
        fetch(row0);
        for (long r0 = row0; r0 < row1; r0 += MLP_TILE) {
            if (!first) wait_g();                          // the last tile's dW1 has read X
#pragma unroll
            for (int q = 0; q < 2; ++q)
                *reinterpret_cast<uint4*>(smem + MLP_T_X + (q * 4 + lk) * MLP_CS + lr * 16) = xv[q];
            stage_sync();
            ok = s_fail == 0;
            if (!ok) break;
            if (r0 + MLP_TILE < row1) fetch(r0 + MLP_TILE);
            const long gr = r0 + row;
            float t[NOUT];
#pragma unroll
            for (int c = 0; c < NOUT; ++c) t[c] = (quart == 0 && gr < row1) ? __ldg(&T[(size_t)gr * NOUT + c]) : 0.f;
            // forward: H1, H2, H3
#pragma unroll
            for (int l = 0; l < 3; ++l) {
                uint8_t* H = smem + (l == 0 ? MLP_T_H1 : l == 1 ? MLP_T_H2 : MLP_T_H3) + quart * 4 * MLP_CS + row * 16;
                wait_a();
                uint32_t r[32];
                tmem_ld32(tm + lanes + MLP_C_ACC + quart * 32, r);
                tmem_ld_wait();
                hidden_piece(r, sb + l * 128 + quart * 32, H);
                stage_sync();
            }
            // output, loss and its gradient
            wait_a();
            float e[NOUT], g[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) g[c] = 0.f;
            if (quart == 0) {
                float v[16];
                tmem_ld<16>(tm + lanes + MLP_C_ACC, v);
#pragma unroll
                for (int c = 0; c < NOUT; ++c) {
                    float y = v[c] + sb[3 * 128 + c];
                    if (residual) y += __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(smem + MLP_T_X + row * 16)[c]);
                    e[c] = y - t[c];
                    if (gr < row1) g[c] = inv * e[c];
                }
                *reinterpret_cast<uint4*>(smem + MLP_T_D4 + row * 16) =
                    make_uint4(pack_bf16(g[0], g[1]), pack_bf16(g[2], g[3]), pack_bf16(g[4], g[5]), 0u);
                *reinterpret_cast<uint4*>(smem + MLP_T_D4 + MLP_CS + row * 16) = make_uint4(0u, 0u, 0u, 0u);
            }
            stage_sync();
            const size_t at = (((gr >> 5) & 7) * out_rows.nk + (gr >> 8)) * 32 + (gr & 31);     // in a stream
            if (quart == 0 && gr < row1) {
#pragma unroll
                for (int c = 0; c < NOUT; ++c) loss += (double)e[c] * e[c];
                out_rows.dy[at] = make_float4(g[0], g[1], g[2], g[3]);
                out_rows.dy2[at] = make_float2(g[4], g[5]);
            }
            // backward: dZ3, dZ2, dZ1 over H3, H2, H1
#pragma unroll
            for (int l = 2; l >= 0; --l) {
                uint8_t* H = smem + (l == 0 ? MLP_T_H1 : l == 1 ? MLP_T_H2 : MLP_T_H3) + quart * 4 * MLP_CS + row * 16;
                wait_a();
                uint32_t r[32];
                tmem_ld32(tm + lanes + MLP_C_ACC + quart * 32, r);
                tmem_ld_wait();
                uint4 z[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint4 h = *reinterpret_cast<const uint4*>(H + q * MLP_CS);
                    z[q].x = mask_bf16(pack_bf16(__uint_as_float(r[8 * q]), __uint_as_float(r[8 * q + 1])), h.x);
                    z[q].y = mask_bf16(pack_bf16(__uint_as_float(r[8 * q + 2]), __uint_as_float(r[8 * q + 3])), h.y);
                    z[q].z = mask_bf16(pack_bf16(__uint_as_float(r[8 * q + 4]), __uint_as_float(r[8 * q + 5])), h.z);
                    z[q].w = mask_bf16(pack_bf16(__uint_as_float(r[8 * q + 6]), __uint_as_float(r[8 * q + 7])), h.w);
                }
                wait_g();                                  // the weight gradient has read this buffer
#pragma unroll
                for (int q = 0; q < 4; ++q) *reinterpret_cast<uint4*>(H + q * MLP_CS) = z[q];
                stage_sync();
                if (gr < row1) {
                    uint4* dz = out_rows.dz[l] + (size_t)quart * 4 * 8 * out_rows.nk * 32 + at;
#pragma unroll
                    for (int q = 0; q < 4; ++q) dz[(size_t)q * 8 * out_rows.nk * 32] = z[q];
                }
            }
            first = false;
        }
    }
    if (ok && warp < MLP_T_WARPS) wait_g();
    __syncthreads();
    if (s_fail == 0 && warp < MLP_T_WARPS) {
        float* out = part + (size_t)blockIdx.x * MLP_GCOLS * 128;
        for (int cb = quart * 16; cb < MLP_GCOLS; cb += 64) {
            float v[16];
            tmem_ld<16>(tm + lanes + MLP_C_D1 + cb, v);
#pragma unroll
            for (int c = 0; c < 16; ++c) out[(size_t)(cb + c) * 128 + row] = v[c];
        }
    } else if (s_fail && threadIdx.x == 0) {
        atomicOr(err, 1u);
    }
    for (int o = 16; o; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (quart == 0 && lane == 0) s_loss[warp] = loss;
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) loss_part[blockIdx.x] = (s_loss[0] + s_loss[1]) + (s_loss[2] + s_loss[3]);
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tm), "r"(512) : "memory");
    }
}

__global__ void k_init_weights(float* W, float* b, int out, int in, int out_real, uint64_t seed) {
    const int n = out * in;
    const float bound = sqrtf(6.0f / (float)in) * (out_real < out ? 0.1f : 1.0f);   // He-uniform; small last layer
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        const int o = q / in;
        uint64_t z = seed + 0x9E3779B97F4A7C15ull * (uint64_t)(q + 1);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        const float u = (float)(z >> 40) * (1.0f / 16777216.0f);
        W[q] = o < out_real ? (2.0f * u - 1.0f) * bound : 0.f;
    }
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < out; q += gridDim.x * blockDim.x) b[q] = 0.f;
}

// BF16 copy of W[out][in].
__global__ void k_weights_bf16(const float* W, int n, __nv_bfloat16* Wb) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) Wb[q] = __float2bfloat16_rn(W[q]);
}

struct MlpParams {
    float *W[NL], *b[NL], *mW[NL], *vW[NL], *mb[NL], *vb[NL], *gT[NL], *gb[NL];
    __nv_bfloat16* Wb[NL];
};

__device__ __forceinline__ void adam(float* p, float* m, float* v, float g, float lr, float b1, float b2, float eps,
                                     float c1, float c2) {
    const float mm = b1 * *m + (1.f - b1) * g, vv = b2 * *v + (1.f - b2) * g * g;
    *m = mm; *v = vv;
    *p -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
}

// Column sums of a lane's n rows (a stream of 32-row lines) in row order, DEPTH loads in flight.
template <int DEPTH, typename V, typename F>
__device__ __forceinline__ void sum_stream(const V* z, int n, F add) {
    V v[DEPTH];
#pragma unroll
    for (int q = 0; q < DEPTH; ++q)
        if (q < n) v[q] = __ldcs(z + (size_t)q * 32);
    int k = 0;
    for (; k + DEPTH <= n; k += DEPTH) {
#pragma unroll
        for (int q = 0; q < DEPTH; ++q) {
            add(v[q]);
            if (k + DEPTH + q < n) v[q] = __ldcs(z + (size_t)(k + DEPTH + q) * 32);
        }
    }
#pragma unroll
    for (int q = 0; q < DEPTH; ++q)
        if (k + q < n) add(v[q]);
}

// Bias gradients: column sums of dY (FP32) and dZ1..dZ3 (bf16) over the rows in FP32, share t of
// 256 adding rows t, t + 256, ..., then trees over 32 shares (a warp each), then the eight warps'
// sums in order (k_mlp_update): the order fixes the parallelism at 256 chains a column. One warp
// a block, eight columns (one 16-byte piece a row) of a hidden layer or up to four of the output
// layer; 400 warps have to keep the memory busy, so each has 32 rows a lane in flight (2M rows:
// 0.27 ms, 5.9 TB/s; with 16 rows loaded, then added, and dY in one stream 0.75 ms).
__global__ void __launch_bounds__(32) k_mlp_bias(BiasRows r, int rows, float* __restrict__ bias_part) {
    const int b = blockIdx.x >> 3, w = blockIdx.x & 7, l = threadIdx.x, t = w * 32 + l;
    const int n = (rows - t + 255) / 256;                // rows of this share
    const size_t at = (size_t)w * r.nk * 32 + l;
    float s[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) s[c] = 0.f;
    if (b < 48) {
        sum_stream<32>(r.dz[b >> 4] + (size_t)(b & 15) * 8 * r.nk * 32 + at, n, [&](const uint4& v) {
            s[0] += __uint_as_float(v.x << 16); s[1] += __uint_as_float(v.x & 0xFFFF0000u);
            s[2] += __uint_as_float(v.y << 16); s[3] += __uint_as_float(v.y & 0xFFFF0000u);
            s[4] += __uint_as_float(v.z << 16); s[5] += __uint_as_float(v.z & 0xFFFF0000u);
            s[6] += __uint_as_float(v.w << 16); s[7] += __uint_as_float(v.w & 0xFFFF0000u);
        });
    } else if (b == 48) {
        sum_stream<32>(r.dy + at, n, [&](const float4& v) { s[0] += v.x; s[1] += v.y; s[2] += v.z; s[3] += v.w; });
    } else {
        sum_stream<32>(r.dy2 + at, n, [&](const float2& v) { s[4] += v.x; s[5] += v.y; });
    }
#pragma unroll
    for (int c = 0; c < 8; ++c)
        for (int o = 16; o; o >>= 1) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
    if (l < 8 && (b < 48 || (l < 4) == (b == 48))) {     // the last two blocks of eight share a group
        float v = s[0];
#pragma unroll
        for (int c = 1; c < 8; ++c) v = l == c ? s[c] : v;
        bias_part[((size_t)min(b, 48) * 8 + l) * 8 + w] = v;
    }
}

// Weight gradients of the step from the CTAs' partials (added in CTA order), then with lr > 0
// an Adam step of every weight and bias and the BF16 copies. One thread per gradient column
// entry: consecutive threads read consecutive lanes of each partial.
__global__ void k_mlp_update(MlpParams p, const float* __restrict__ part, const float* __restrict__ bias_part, int ncta,
                             float lr, float b1, float b2, float eps, float c1, float c2) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = q >> 7, lane = q & 127;
    if (col >= MLP_GCOLS) {                      // the last block: biases
        for (int l = 0; l < NL; ++l) {
            if (l == 3 && lane >= 16) break;
            float g = 0.f;
            if (l < 3 || lane < NOUT)
                for (int w = 0; w < 8; ++w) g += bias_part[((size_t)(l * 16 + (lane >> 3)) * 8 + (lane & 7)) * 8 + w];
            p.gb[l][lane] = g;
            if (lr > 0.f && (l < 3 || lane < NOUT))
                adam(&p.b[l][lane], &p.mb[l][lane], &p.vb[l][lane], g, lr, b1, b2, eps, c1, c2);
        }
        return;
    }
    int l, in, out;
    if (col < 64) { l = 0; in = col; out = lane; }
    else if (col < 192) { l = 1; in = col - 64; out = lane; }
    else if (col < 320) { l = 2; in = col - 192; out = lane; }
    else { l = 3; in = lane; out = col - 320; }
    float g = 0.f;
#pragma unroll 8
    for (int b = 0; b < ncta; ++b) g += __ldg(&part[((size_t)b * MLP_GCOLS + col) * 128 + lane]);
    const int nin = l == 0 ? 64 : 128, nout = l == 3 ? 16 : 128, nreal = l == 3 ? NOUT : 128;
    p.gT[l][(size_t)in * nout + out] = g;
    if (lr > 0.f && out < nreal) {
        const size_t s = (size_t)out * nin + in;
        adam(&p.W[l][s], &p.mW[l][s], &p.vW[l][s], g, lr, b1, b2, eps, c1, c2);
        p.Wb[l][s] = __float2bfloat16_rn(p.W[l][s]);
    }
}

}  // namespace mlp
}  // namespace rf

struct rf_mlp {
    rf::mlp::MlpParams p = {};
    float* part = nullptr;                       // gradient partials of the training CTAs (first training step)
    double* loss_part = nullptr;
    float* bias_part = nullptr;
    rf::mlp::BiasRows rows = {};                 // as many rows as the largest step so far
    void* rows_mem = nullptr;
    size_t rows_cap = 0;
    __nv_bfloat16* xcopy = nullptr;              // features given at an address that is not 16-byte aligned
    size_t xcopy_rows = 0;
    int sms = 0;
    int steps = 0;
    int residual = 0;           // predict the correction to the input's first 6 features
    cudaStream_t stream = nullptr;
    std::vector<void*> allocs;
};

namespace {
using namespace rf::mlp;

template <class T> rf_status mlp_alloc(rf_mlp* m, T** p, size_t n) {
    void* q = nullptr;
    RF_CUDA(cudaMalloc(&q, (n ? n : 1) * sizeof(T)));
    m->allocs.push_back(q);
    *p = (T*)q;
    return RF_OK;
}

MlpWeights mlp_weights(const rf_mlp* m) {
    MlpWeights w;
    for (int l = 0; l < NL; ++l) { w.W[l] = m->p.Wb[l]; w.b[l] = m->p.b[l]; }
    return w;
}

// CTAs of a pass over `rows`: one per tile up to one per SM (their shared memory fills it).
int mlp_grid(const rf_mlp* m, int rows) {
    const long tiles = ((long)rows + MLP_TILE - 1) / MLP_TILE;
    return (int)(tiles < m->sms ? tiles : m->sms);
}
}  // namespace

extern "C" {

rf_status rf_mlp_create(uint64_t seed, rf_mlp** out) {
    if (!out) { set_error("rf_mlp_create: null output"); return RF_ERR_INVALID; }
    rf_mlp* m = new rf_mlp();
    auto fail = [&](rf_status s) { rf_mlp_destroy(m); return s; };
    int dev = 0;
    if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize, MLP_F_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, MLP_T_SMEM) != cudaSuccess)
        return fail(cuda_status(cudaGetLastError(), "rf_mlp_create"));
    MlpParams& p = m->p;
    for (int l = 0; l < NL; ++l) {
        const size_t n = (size_t)DOUT[l] * DIN[l];
        rf_status st;
        if ((st = mlp_alloc(m, &p.W[l], n)) || (st = mlp_alloc(m, &p.b[l], DOUT[l])) ||
            (st = mlp_alloc(m, &p.mW[l], n)) || (st = mlp_alloc(m, &p.vW[l], n)) ||
            (st = mlp_alloc(m, &p.mb[l], DOUT[l])) || (st = mlp_alloc(m, &p.vb[l], DOUT[l])) ||
            (st = mlp_alloc(m, &p.gT[l], n)) || (st = mlp_alloc(m, &p.gb[l], DOUT[l])) ||
            (st = mlp_alloc(m, &p.Wb[l], n)))
            return fail(st);
        cudaMemsetAsync(p.mW[l], 0, n * 4, m->stream);
        cudaMemsetAsync(p.vW[l], 0, n * 4, m->stream);
        cudaMemsetAsync(p.mb[l], 0, DOUT[l] * 4, m->stream);
        cudaMemsetAsync(p.vb[l], 0, DOUT[l] * 4, m->stream);
        k_init_weights<<<64, 256, 0, m->stream>>>(p.W[l], p.b[l], DOUT[l], DIN[l], l == NL - 1 ? NOUT : DOUT[l],
                                                   seed + 1000003ull * l);
        k_weights_bf16<<<64, 256, 0, m->stream>>>(p.W[l], (int)n, p.Wb[l]);
    }
    if (cudaStreamSynchronize(m->stream) != cudaSuccess) return fail(cuda_status(cudaGetLastError(), "rf_mlp_create"));
    *out = m;
    return RF_OK;
}

rf_status rf_mlp_destroy(rf_mlp* m) {
    if (!m) return RF_OK;
    if (m->stream) cudaStreamSynchronize(m->stream);
    for (void* p : m->allocs) cudaFree(p);
    if (m->xcopy) cudaFree(m->xcopy);
    if (m->rows_mem) cudaFree(m->rows_mem);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return RF_OK;
}

rf_stream rf_mlp_stream(rf_mlp* m) { return m ? (rf_stream)m->stream : nullptr; }

// Inference: Y[rows][ldy] (fp32, first ncols <= 16 outputs) from X (bf16 [rows][64]).
rf_status rf_mlp_forward(rf_mlp* m, const void* X, int rows, float* Y, int ldy, int ncols) {
    if (!m || !X || !Y || rows <= 0 || ncols <= 0 || ncols > 16 || ldy < ncols || ((uintptr_t)X % 16) != 0) {
        set_error("rf_mlp_forward: bad arguments (X 16-byte aligned)");
        return RF_ERR_INVALID;
    }
    uint32_t* err = gemm_err_word();
    if (!err) { set_error("rf_mlp_forward: no status word"); return RF_ERR_CUDA; }
    k_mlp_forward<<<mlp_grid(m, rows), 128 * MLP_F_GROUPS, MLP_F_SMEM, m->stream>>>(
        mlp_weights(m), (const __nv_bfloat16*)X, rows, Y, ldy, ncols, m->residual, err);
    RF_CHECK_LAUNCH("k_mlp_forward");
    return RF_OK;
}

// Residual mode on/off: the network's output is added to the input's first 6 features
// (the last increment's motion in the warm-start features), and trained on the difference.
rf_status rf_mlp_set_residual(rf_mlp* m, int on) {
    if (!m) { set_error("rf_mlp_set_residual: null"); return RF_ERR_INVALID; }
    m->residual = on ? 1 : 0;
    return RF_OK;
}

// Gradients of the loss mean((y - t)^2) for X (bf16 [rows][64]) and targets T (fp32
// [rows][6]); *loss receives the loss before the update. With lr > 0 an Adam step
// (beta 0.9, 0.999, eps 1e-8) follows.
rf_status rf_mlp_train_step(rf_mlp* m, const void* X, const float* T, int rows, float lr, double* loss) {
    if (!m || !X || !T || rows <= 0) { set_error("rf_mlp_train_step: bad arguments"); return RF_ERR_INVALID; }
    cudaStream_t cs = m->stream;
    uint32_t* err = gemm_err_word();
    if (!err) { set_error("rf_mlp_train_step: no status word"); return RF_ERR_CUDA; }
    if (!m->part) {
        rf_status st;
        if ((st = mlp_alloc(m, &m->loss_part, MLP_SPLITS)) || (st = mlp_alloc(m, &m->bias_part, 49 * 64)) ||
            (st = mlp_alloc(m, &m->part, (size_t)MLP_SPLITS * MLP_GCOLS * 128)))
            return st;
    }
    const size_t rp = ((size_t)rows + 255) / 256 * 256;
    if (m->rows_cap < rp) {
        if (m->rows_mem) cudaFree(m->rows_mem);  // (waits for what still uses it)
        m->rows_mem = nullptr; m->rows_cap = 0;
        RF_CUDA(cudaMalloc(&m->rows_mem, rp * (24 + 3 * 256)));
        m->rows_cap = rp;
    }
    {
        char* q = (char*)m->rows_mem;
        m->rows.dy = (float4*)q;
        m->rows.dy2 = (float2*)(q + rp * 16);
        m->rows.nk = (long)(rp / 256);
        for (int l = 0; l < 3; ++l) m->rows.dz[l] = (uint4*)(q + rp * (24 + l * 256));
    }
    const void* x = X;
    if ((uintptr_t)X % 16 != 0) {                // the kernel's loads take 16 bytes: a copy where they cannot
        if (m->xcopy_rows < (size_t)rows) {
            if (m->xcopy) cudaFree(m->xcopy);
            m->xcopy = nullptr; m->xcopy_rows = 0;
            RF_CUDA(cudaMalloc(&m->xcopy, (size_t)rows * 64 * 2));
            m->xcopy_rows = rows;
        }
        RF_CUDA(cudaMemcpyAsync(m->xcopy, X, (size_t)rows * 64 * 2, cudaMemcpyDeviceToDevice, cs));
        x = m->xcopy;
    }
    // the rows in splits of whole 64-row chunks, one per 2048 rows up to MLP_SPLITS
    const long chunks = ((long)rows + 127) / 128 * 2;
    const long splits = std::max(1l, std::min((long)MLP_SPLITS, chunks / 32)), per = (chunks + splits - 1) / splits;
    const int ncta = (int)((((long)rows + 63) / 64 + per - 1) / per);    // (the last chunk can be padding alone)
    k_mlp_train<<<ncta, MLP_T_THREADS, MLP_T_SMEM, cs>>>(mlp_weights(m), (const __nv_bfloat16*)x, T, rows, per * 64, m->residual,
                                               m->part, m->loss_part, m->rows, err);
    RF_CHECK_LAUNCH("k_mlp_train");
    float c1 = 1.f, c2 = 1.f;
    const float b1 = 0.9f, b2 = 0.999f;
    if (lr > 0.f) {
        m->steps += 1;
        c1 = 1.f - std::pow(b1, (float)m->steps);
        c2 = 1.f - std::pow(b2, (float)m->steps);
    }
    k_mlp_bias<<<50 * 8, 32, 0, cs>>>(m->rows, rows, m->bias_part);
    RF_CHECK_LAUNCH("k_mlp_bias");
    k_mlp_update<<<MLP_GCOLS + 1, 128, 0, cs>>>(m->p, m->part, m->bias_part, ncta, lr, b1, b2, 1e-8f, c1, c2);
    RF_CHECK_LAUNCH("k_mlp_update");
    std::vector<double> h(ncta);
    RF_CUDA(cudaMemcpyAsync(h.data(), m->loss_part, ncta * sizeof(double), cudaMemcpyDeviceToHost, cs));
    if (rf_status st = rf_gemm_status((rf_stream)cs)) return st;      // (synchronises the stream)
    if (loss) {
        double t = 0.0;
        for (double q : h) t += q;
        *loss = t / ((double)rows * NOUT);
    }
    return RF_OK;
}

// Copy the fp32 weights out / in (host buffers; W[l] is [out][in] with the last layer's
// out = 16 rows, of which the first 6 are used). Layer sizes: 128x64, 128x128, 128x128, 16x128.
rf_status rf_mlp_get(rf_mlp* m, int layer, float* W, float* b) {
    if (!m || layer < 0 || layer >= NL) { set_error("rf_mlp_get: bad arguments"); return RF_ERR_INVALID; }
    RF_CUDA(cudaStreamSynchronize(m->stream));
    if (W) RF_CUDA(cudaMemcpy(W, m->p.W[layer], (size_t)DOUT[layer] * DIN[layer] * 4, cudaMemcpyDeviceToHost));
    if (b) RF_CUDA(cudaMemcpy(b, m->p.b[layer], (size_t)DOUT[layer] * 4, cudaMemcpyDeviceToHost));
    return RF_OK;
}
rf_status rf_mlp_set(rf_mlp* m, int layer, const float* W, const float* b) {
    if (!m || layer < 0 || layer >= NL || !W || !b) { set_error("rf_mlp_set: bad arguments"); return RF_ERR_INVALID; }
    RF_CUDA(cudaStreamSynchronize(m->stream));
    const int n = DOUT[layer] * DIN[layer];
    RF_CUDA(cudaMemcpy(m->p.W[layer], W, (size_t)n * 4, cudaMemcpyHostToDevice));
    RF_CUDA(cudaMemcpy(m->p.b[layer], b, (size_t)DOUT[layer] * 4, cudaMemcpyHostToDevice));
    k_weights_bf16<<<64, 256, 0, m->stream>>>(m->p.W[layer], n, m->p.Wb[layer]);
    RF_CHECK_LAUNCH("k_weights_bf16");
    RF_CUDA(cudaStreamSynchronize(m->stream));
    return RF_OK;
}
// The gradients of the last rf_mlp_train_step: gT is [in][out] (the transpose of W's layout).
rf_status rf_mlp_grad(rf_mlp* m, int layer, float* gT, float* gb) {
    if (!m || layer < 0 || layer >= NL) { set_error("rf_mlp_grad: bad arguments"); return RF_ERR_INVALID; }
    RF_CUDA(cudaStreamSynchronize(m->stream));
    if (gT) RF_CUDA(cudaMemcpy(gT, m->p.gT[layer], (size_t)DOUT[layer] * DIN[layer] * 4, cudaMemcpyDeviceToHost));
    if (gb) RF_CUDA(cudaMemcpy(gb, m->p.gb[layer], (size_t)DOUT[layer] * 4, cudaMemcpyDeviceToHost));
    return RF_OK;
}

}  // extern "C"
