// Flux surrogate network kernels: a BF16 multilayer perceptron trained and evaluated on the
// device with the 5th-generation tensor cores (tcgen05), FP32 accumulation in tensor memory.
//
// The surrogate maps one heliostat's inputs (sun vector, field position, aim offset, slope
// error) to the flux image it puts on the receiver; the plain trace (st_sim_run with a
// per-source flux map) makes its training data and measures its error.  It has no counterpart in the
// reference, which traces every ray.
//
// One product does every layer's work, forward and backward:
//     C[M x N] = epilogue(A[M x K] B[N x K]^T)
// with A(m, k) = A[m lam + k lak] and B(n, k) = B[n lbn + k lbk] (bf16), so the backward
// products (dX = dZ W, dW = dZ^T X) read their operands in place through strides.  Split-K: several
// CTAs share a tile's K range and add their partial sums (EPI_F32_ADD).  Two kernels:
//   k_mlp_gemm_tma, a warp-specialised TMA pipeline, for operands TMA can address (every layer
//     of a network whose widths are multiples of 8);
//   k_mlp_gemm for any strides: a CTA of 128 threads owns a 128 x BN tile of C; per 64-wide slice
//     of K it stages the A and B tiles in shared memory in the K-major, unswizzled core-matrix
//     layout the tensor cores read (8 rows x 16 bytes per core matrix), one elected thread issues
//     four tcgen05.mma (K = 16 each) into the tile's FP32 accumulator in tensor memory and commits
//     them to an mbarrier, and after the last slice the four warps read the accumulator back
//     (tcgen05.ld, one row per thread) and apply the epilogue.
//
// Every wait is bounded: an mbarrier wait that runs out sets an error flag (read with
// st_b200_mlp_error) and the kernel drains and returns, freeing its tensor memory.
#include <cstdint>
#include <cstdio>
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/st_b200.h"

namespace stb {
namespace mlp {

constexpr int kBM = 128;       // rows of a C tile (the tensor-core M)
constexpr int kBK = 64;        // K per shared-memory stage
constexpr int kThreads = 128;  // four warps: loaders, then one accumulator row each in the epilogue
constexpr unsigned kSpinLimit = 1u << 26;

// epilogues
enum Epi : int {
    EPI_BIAS_RELU_BF16 = 0,  // out_bf16 = bf16(max(acc + bias, 0))            (hidden layer)
    EPI_BIAS_F32 = 1,        // out_f32 = acc + bias                             (output layer)
    EPI_RELU_MASK_BF16 = 2,  // out_bf16 = bf16(acc) where aux_bf16 > 0, else 0  (dZ through ReLU)
    EPI_F32 = 3,             // out_f32 = acc                                    (dX of the input)
    EPI_F32_ADD = 4,         // out_f32 += acc (atomic; split-K partial sums)    (dW)
};

struct GemmArgs {
    const __nv_bfloat16 *A, *B;
    long long lam, lak, lbn, lbk;
    int M, N, K;
    int epi;
    void *C;
    long long ldc;
    const float *bias;
    const __nv_bfloat16 *aux;  // EPI_RELU_MASK_BF16: the layer's activations, leading dimension ldc
    int k_per_split;           // K range of one split (multiple of kBK)
    unsigned *err;             // set to 1 when a wait ran out
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// shared-memory matrix descriptor (tcgen05): K-major, no swizzle; start address, leading byte
// offset (between the two K-adjacent core matrices of one K = 16 step) and stride byte offset
// (between M/N-adjacent core matrices) in 16-byte units; version 1 (bits 46-47)
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= uint64_t((addr >> 4) & 0x3FFFu);
    d |= uint64_t((lbo >> 4) & 0x3FFFu) << 16;
    d |= uint64_t((sbo >> 4) & 0x3FFFu) << 32;
    d |= uint64_t(1) << 46;
    return d;  // base offset 0, leading-offset mode 0, layout 0 (no swizzle)
}

// instruction descriptor of kind::f16: D f32 (bits 4-5 = 1), A and B bf16 (bits 7-9, 10-12 =
// 1), both K-major, N / 8 at bits 17-22, M / 16 at bits 24-28
__host__ __device__ constexpr uint32_t instr_desc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(kBM >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

// wait for phase `parity` of the barrier to complete; false when the spin limit ran out
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity) {
    const uint32_t a = smem_u32(bar);
    for (unsigned it = 0; it < kSpinLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// one thread of the (converged) warp
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 16 consecutive 32-bit columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 64 accumulator columns of the warp's 32 lanes in one load and one wait
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, float v[64]) {
    uint32_t r[64];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, "
        "%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, "
        "%48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
          "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
          "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
          "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
          "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 64; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 accumulator columns of the warp's 32 lanes
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float v[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Stage rows [r0, r0 + R) x K [k0, k0 + kBK) of an operand (element (r, k) at src[r lr + k lk],
// rows < rows_end and k < k_end valid, zero elsewhere) in shared memory as K-major core
// matrices: core matrix (row group g, K chunk c) at byte ((c R/8) + g) 128, its 8 rows 16 bytes
// apart.  One 16-byte chunk (8 K values of one row) per thread and step; with K contiguous the
// chunks of a row go to neighbouring threads, otherwise neighbouring rows do (coalesced either way).
template <int R>
__device__ __forceinline__ void load_tile(unsigned char *dst, const __nv_bfloat16 *src, long long lr, long long lk,
                                          int r0, int rows_end, int k0, int k_end) {
    constexpr int kChunks = R * (kBK / 8);
    const bool k_contig = (lk == 1);
    for (int c = threadIdx.x; c < kChunks; c += kThreads) {
        const int r = k_contig ? c / (kBK / 8) : c % R;
        const int kc = k_contig ? c % (kBK / 8) : c / R;
        const int gr = r0 + r, gk = k0 + kc * 8;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (gr < rows_end) {
            const __nv_bfloat16 *p = src + gr * lr + gk * lk;
            if (k_contig && gk + 8 <= k_end && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
                v = *reinterpret_cast<const uint4 *>(p);
            } else {
                unsigned short h[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    h[e] = (gk + e < k_end) ? __bfloat16_as_ushort(p[e * lk]) : (unsigned short)0;
                v = make_uint4(h[0] | (uint32_t(h[1]) << 16), h[2] | (uint32_t(h[3]) << 16),
                               h[4] | (uint32_t(h[5]) << 16), h[6] | (uint32_t(h[7]) << 16));
            }
        }
        *reinterpret_cast<uint4 *>(dst + (size_t(kc) * (R / 8) + r / 8) * 128 + (r % 8) * 16) = v;
    }
}

// two floats rounded to bf16, lo in the low half: one packed conversion (single conversions run on the
// quarter-rate unit: 512 cycles an SM per 128 x 64 slice of the fused kernel)
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// one accumulator value of C (element `at`, column `col`) through the epilogue
__device__ __forceinline__ void epilogue1(const GemmArgs &g, long long at, int col, float v) {
    switch (g.epi) {
        case EPI_BIAS_RELU_BF16:
            static_cast<__nv_bfloat16 *>(g.C)[at] = __float2bfloat16_rn(fmaxf(v + g.bias[col], 0.f));
            break;
        case EPI_BIAS_F32:
            static_cast<float *>(g.C)[at] = v + g.bias[col];
            break;
        case EPI_RELU_MASK_BF16:
            static_cast<__nv_bfloat16 *>(g.C)[at] =
                __bfloat162float(g.aux[at]) > 0.f ? __float2bfloat16_rn(v) : __float2bfloat16_rn(0.f);
            break;
        case EPI_F32:
            static_cast<float *>(g.C)[at] = v;
            break;
        default:
            atomicAdd(static_cast<float *>(g.C) + at, v);
    }
}

// The product for operands TMA cannot address (neither stride 1, rows not 16 bytes apart or
// unaligned bases): loads of any stride, one stage.
template <int BN>
__global__ void __launch_bounds__(kThreads, 1) k_mlp_gemm(GemmArgs g) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *sa = smem;                      // kBM x kBK bf16
    unsigned char *sb = smem + kBM * kBK * 2;      // BN x kBK bf16
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t tmem_sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;
    const int kb = blockIdx.z * g.k_per_split;
    const int ke = min(g.K, kb + g.k_per_split);
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {  // the tile's FP32 accumulator: 128 lanes x BN columns of tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                     "r"(uint32_t(BN)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_sh;
    constexpr uint32_t idesc = instr_desc(BN);
    unsigned phase = 0;
    bool ok = true;
    int steps = 0;
    for (int k0 = kb; k0 < ke; k0 += kBK) {
        load_tile<kBM>(sa, g.A, g.lam, g.lak, m0, g.M, k0, ke);
        load_tile<BN>(sb, g.B, g.lbn, g.lbk, n0, g.N, k0, ke);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor cores read what was stored
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int j = 0; j < kBK / 16; ++j) {
                const uint64_t ad = smem_desc(smem_u32(sa) + uint32_t(j * 2 * (kBM / 8) * 128), (kBM / 8) * 128, 128);
                const uint64_t bd = smem_desc(smem_u32(sb) + uint32_t(j * 2 * (BN / 8) * 128), (BN / 8) * 128, 128);
                mma_bf16(tmem, ad, bd, idesc, (steps > 0 || j > 0) ? 1u : 0u);
            }
            mma_commit(&bar);
        }
        ok = mbar_wait(&bar, phase);
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // block-wide: the next stage overwrites the tiles the finished products read, and a wait
        // that ran out in any thread ends the loop for all of them
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        ++steps;
    }
    if (!ok) {
        if (lane == 0) atomicExch(g.err, 1u);
    } else if (steps > 0) {
        // epilogue: warp w reads accumulator lanes [32 w, 32 w + 32), thread = one row of C
        const int row = m0 + warp * 32 + lane;
        const bool row_ok = row < g.M;
        for (int c0 = 0; c0 < BN; c0 += 16) {
            float v[16];
            tmem_ld16(tmem + (uint32_t(warp * 32) << 16) + uint32_t(c0), v);
            if (!row_ok) continue;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int col = n0 + c0 + i;
                if (col >= g.N) continue;
                const long long at = row * g.ldc + col;
                epilogue1(g, at, col, v[i]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (!ok) mbar_wait(&bar, phase ^ 1u);  // a product still in flight finishes before its memory is freed
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(uint32_t(BN)));
}

// ---------------------------------------------------------------------------------------
// The same product with both operands brought in by TMA
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// bounded wait that also gives up as soon as another role raised the abort flag
__device__ __forceinline__ bool mbar_wait_or_abort(uint64_t *bar, unsigned parity, volatile int *abort) {
    const uint32_t a = smem_u32(bar);
    for (unsigned it = 0; it < kSpinLimit; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if (*abort) return false;
    }
    return false;
}

// one box of a tensor map -> this CTA's shared memory, its bytes counted on `bar`; x (the
// contiguous dimension) is a multiple of 64 elements everywhere below
__device__ __forceinline__ void tma_load(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// 32 bytes to global memory in one store (a whole sector per thread)
__device__ __forceinline__ void store32(void *p, const uint32_t v[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

// Matrix descriptor of a 128-byte-swizzled tile as TMA leaves it (8 rows x 128 bytes per atom,
// 1024 bytes).  K-major (a row holds 64 K values): row groups 1024 bytes apart.  MN-major (a row
// holds 64 M or N values of one K): K groups 1024 bytes apart (stride offset), the next 64 M or N
// values one 64-row box further (leading offset).
constexpr uint32_t kBoxBytes = 64 * kBK * 2;  // an MN-major box: 64 values x 64 K
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr, bool mn_major) {
    uint64_t d = uint64_t((addr >> 4) & 0x3FFFu) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) |
                 (uint64_t(2) << 61);
    return d | (uint64_t(mn_major ? (kBoxBytes >> 4) : 1u) << 16);
}

// Sixteen accumulator values of one row of C (columns col .. col + 15) through the epilogue
__device__ __forceinline__ void epilogue16(const GemmArgs &g, long long row, int col, const float v[16], bool wide) {
    const long long at = row * g.ldc + col;
    if (wide && col + 16 <= g.N) {
        if (g.epi == EPI_BIAS_RELU_BF16 || g.epi == EPI_RELU_MASK_BF16) {
            float y[16];
            if (g.epi == EPI_BIAS_RELU_BF16) {
#pragma unroll
                for (int i = 0; i < 16; ++i) y[i] = fmaxf(v[i] + __ldg(g.bias + col + i), 0.f);
            } else {
                const uint4 *a = reinterpret_cast<const uint4 *>(g.aux + at);
                const uint4 a0 = a[0], a1 = a[1];
                const uint32_t h[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    y[2 * i] = __uint_as_float(h[i] << 16) > 0.f ? v[2 * i] : 0.f;
                    y[2 * i + 1] = __uint_as_float(h[i] & 0xffff0000u) > 0.f ? v[2 * i + 1] : 0.f;
                }
            }
            uint32_t p[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                p[i] = pack_bf16(y[2 * i], y[2 * i + 1]);
            store32(static_cast<__nv_bfloat16 *>(g.C) + at, p);
        } else if (g.epi == EPI_F32_ADD) {
#pragma unroll
            for (int i = 0; i < 16; i += 4)
                atomicAdd(reinterpret_cast<float4 *>(static_cast<float *>(g.C) + at + i),
                          make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]));
        } else {
            uint32_t p[16];
#pragma unroll
            for (int i = 0; i < 16; ++i)
                p[i] = __float_as_uint(g.epi == EPI_BIAS_F32 ? v[i] + __ldg(g.bias + col + i) : v[i]);
            store32(static_cast<float *>(g.C) + at, p);
            store32(static_cast<float *>(g.C) + at + 8, p + 8);
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i)
        if (col + i < g.N) epilogue1(g, at + i, col + i, v[i]);
}

// Operands whose rows TMA can address (one stride 1, the other a multiple of 8 values, 16-byte
// aligned bases): persistent CTAs walk the (tile, K split) items; one thread keeps a ring of
// A and B tiles filled with TMA loads, one issues the tensor-core products, eight warps run the
// epilogue of the last item from one accumulator while the next item's products fill the
// other.  Either operand may be stored with its M (N) index contiguous: its boxes hold 64 such
// values by 64 K and the products read them transposed in place.  Rows and K beyond the
// matrices arrive as zeros.
// Against k_mlp_gemm (one stage, every wait exposed, element loads of transposed operands): the
// sixteen 256-wide products of a gradient pass over 16,384 rows took 140 us each there; here
// the hidden layers' take 13 to 15 (dX) and 21 (dW): a single wave of 128 tiles whose tensor pipe is
// active a tenth of the time, the rest being launch, pipeline fill and the outputs' stores.  The
// pass fell from 2.31 to 0.42 ms.
constexpr int kPipeThreads = 320;             // warps 0-7 epilogue, 8 loader, 9 products
constexpr int kPipeBytes = 192 * 1024;        // ring of operand tiles
template <int BN>
__global__ void __launch_bounds__(kPipeThreads, 1)
    k_mlp_gemm_tma(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
                   const __grid_constant__ GemmArgs g, int tiles_m, int tiles_n, long long items, int a_mn, int b_mn) {
    constexpr uint32_t kABytes = kBM * kBK * 2, kTile = kABytes + BN * kBK * 2;
    constexpr int kStages = kPipeBytes / kTile;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *smem = smem_raw + (1024u - (smem_u32(smem_raw) & 1023u)) % 1024u;
    __shared__ __align__(8) uint64_t full[kStages], empty[kStages], acc_full[2], acc_free[2], drain;
    __shared__ uint32_t tmem_sh;
    __shared__ volatile int abort_flag;
    __shared__ unsigned issued_sh, consumed_sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_free[i], 256);
        }
        mbar_init(&drain, 1);
        abort_flag = 0;
        issued_sh = consumed_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {  // two 128 x BN FP32 accumulators
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                     "r"(uint32_t(2 * BN)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_sh;
    // item -> tile and K range [k0, k0 + kBK nk); an empty split has nk = 0
    auto item = [&](long long it, int &m0, int &n0, int &k0, int &nk) {
        m0 = int(it % tiles_m) * kBM;
        n0 = int(it / tiles_m % tiles_n) * BN;
        const long long kb = it / tiles_m / tiles_n * g.k_per_split;
        const long long ke = min((long long)g.K, kb + g.k_per_split);
        k0 = int(kb);
        nk = ke > kb ? int((ke - kb + kBK - 1) / kBK) : 0;
    };
    int m0, n0, k0, nk;
    if (warp == 8) {
        // ---- loader ----
        if (lane == 0) {
            unsigned q = 0;
            for (long long it = blockIdx.x; it < items && !abort_flag; it += gridDim.x) {
                item(it, m0, n0, k0, nk);
                for (int k = 0; k < nk; ++k, ++q) {
                    const int slot = q % kStages, x = k0 + k * kBK;
                    if (q >= kStages && !mbar_wait_or_abort(&empty[slot], ((q / kStages) - 1) & 1u, &abort_flag)) {
                        abort_flag = 1;
                        break;
                    }
                    unsigned char *sa = smem + slot * kTile, *sb = sa + kABytes;
                    mbar_expect_tx(&full[slot], kTile);
                    if (a_mn)
                        for (int c = 0; c < kBM / 64; ++c) tma_load(sa + c * kBoxBytes, &ta, m0 + 64 * c, x, &full[slot]);
                    else
                        tma_load(sa, &ta, x, m0, &full[slot]);
                    if (b_mn)
                        for (int c = 0; c < BN / 64; ++c) tma_load(sb + c * kBoxBytes, &tb, n0 + 64 * c, x, &full[slot]);
                    else
                        tma_load(sb, &tb, x, n0, &full[slot]);
                }
            }
            issued_sh = q;
        }
    } else if (warp == 9) {
        // ---- products ----
        if (lane == 0) {
            const uint32_t idesc = instr_desc(BN) | (uint32_t(a_mn) << 15) | (uint32_t(b_mn) << 16);
            // a K = 16 step: 32 bytes along a K-major row, two 8-K groups of an MN-major box
            const uint32_t astep = a_mn ? 2048u : 32u, bstep = b_mn ? 2048u : 32u;
            unsigned q = 0, u = 0;
            bool ok = true;
            for (long long it = blockIdx.x; it < items && ok; it += gridDim.x) {
                item(it, m0, n0, k0, nk);
                if (nk == 0) continue;
                const int b = u & 1;
                if (u >= 2 && !mbar_wait_or_abort(&acc_free[b], ((u >> 1) - 1) & 1u, &abort_flag)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int k = 0; k < nk; ++k, ++q) {
                    const int slot = q % kStages;
                    if (!mbar_wait_or_abort(&full[slot], (q / kStages) & 1u, &abort_flag)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t sa = smem_u32(smem + slot * kTile), sb = sa + kABytes;
#pragma unroll
                    for (int j = 0; j < kBK / 16; ++j)
                        mma_bf16(tmem + uint32_t(b * BN), sw128_desc(sa + j * astep, a_mn), sw128_desc(sb + j * bstep, b_mn),
                                 idesc, (k > 0 || j > 0) ? 1u : 0u);
                    mma_commit(&empty[slot]);
                }
                if (ok) mma_commit(&acc_full[b]);
                ++u;
            }
            if (!ok) abort_flag = 1;
            consumed_sh = q;
            // every product this thread issued has finished before the CTA frees its memory
            mma_commit(&drain);
            mbar_wait(&drain, 0);
        }
    } else {
        // ---- epilogue: warp w reads accumulator lanes 32 (w % 4) .. + 31 of half the columns ----
        const int out_size = (g.epi == EPI_BIAS_RELU_BF16 || g.epi == EPI_RELU_MASK_BF16) ? 2 : 4;
        // whole 32-byte stores (aux is shaped as C and read alongside)
        const bool wide = ((reinterpret_cast<uintptr_t>(g.C) | uintptr_t(g.ldc * out_size)) & 31) == 0 &&
                          (g.epi != EPI_RELU_MASK_BF16 || (reinterpret_cast<uintptr_t>(g.aux) & 15) == 0);
        unsigned u = 0;
        bool ok = true;
        for (long long it = blockIdx.x; it < items && ok; it += gridDim.x) {
            item(it, m0, n0, k0, nk);
            if (nk == 0) continue;
            const int b = u & 1;
            // warp-uniform: the tensor-memory loads below are warp-collective
            if (!__all_sync(0xffffffffu, mbar_wait_or_abort(&acc_full[b], (u >> 1) & 1u, &abort_flag))) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const long long row = m0 + (warp & 3) * 32 + lane;
            constexpr int kHalf = BN / 2, kCols = kHalf < 64 ? kHalf : 64;
            for (int c = (warp >> 2) * kHalf; c < (warp >> 2) * kHalf + kHalf; c += kCols) {
                if (n0 + c >= g.N) break;
                const uint32_t at = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(b * BN + c);
                float v[kCols];
                if (kCols == 64) {
                    tmem_ld64(at, v);
                } else {
                    tmem_ld16(at, v);
                    tmem_ld16(at + 16, v + 16);
                }
                if (row < g.M) {
#pragma unroll
                    for (int i = 0; i < kCols; i += 16) epilogue16(g, row, n0 + c + i, v + i, wide);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&acc_free[b]);
            ++u;
        }
        if (!ok) abort_flag = 1;
    }
    __syncthreads();
    if (abort_flag) {
        if (threadIdx.x == 0) {
            atomicExch(g.err, 1u);
            // operand copies issued but never consumed land before their shared memory goes away
            for (unsigned q = consumed_sh; q < issued_sh; ++q) mbar_wait(&full[q % kStages], (q / kStages) & 1u);
        }
        __syncthreads();
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(uint32_t(2 * BN)));
}

// mean-squared-error loss over rows x cols outputs against float targets: dY = bf16(2 (y - t) /
// (rows cols)); the sum of squared differences is added to *loss (double).  Bound by reading y and
// t and writing dY once (10 bytes a value).  WIDE (targets contiguous, 16-byte aligned, a multiple
// of four values): 16-byte loads without the row division; one atomic per block in either form.
constexpr int kMseThreads = 256;
template <int WIDE>
__global__ void __launch_bounds__(kMseThreads) k_mse(int rows, int cols, const float *y, const float *t, long long ldt,
                                                     __nv_bfloat16 *dy, double *loss) {
    const long long n = (long long)rows * cols;
    const float scale = 2.0f / float(n);
    const long long stride = (long long)gridDim.x * kMseThreads;
    double acc = 0.0;
    if (WIDE) {
        const long long q = n / 4;
#pragma unroll 4
        for (long long i = blockIdx.x * (long long)kMseThreads + threadIdx.x; i < q; i += stride) {
            const float4 a = reinterpret_cast<const float4 *>(y)[i], b = reinterpret_cast<const float4 *>(t)[i];
            const float d[4] = {a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w};
            uint2 p;
            p.x = pack_bf16(scale * d[0], scale * d[1]);
            p.y = pack_bf16(scale * d[2], scale * d[3]);
            reinterpret_cast<uint2 *>(dy)[i] = p;
#pragma unroll
            for (int k = 0; k < 4; ++k) acc += double(d[k]) * double(d[k]);
        }
    } else {
        for (long long i = blockIdx.x * (long long)kMseThreads + threadIdx.x; i < n; i += stride) {
            const long long r = i / cols, c = i % cols;
            const float d = y[i] - t[r * ldt + c];
            dy[i] = __float2bfloat16_rn(scale * d);
            acc += double(d) * double(d);
        }
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    __shared__ double part[kMseThreads / 32];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kMseThreads / 32; ++w) acc += part[w];
        atomicAdd(loss, acc);
    }
}

// db[c] = sum over rows of dz[r][c].  Bound by reading dz once (L2-resident behind the product
// that wrote it).  A cluster of kSumCluster CTAs owns kSumCols columns, its CTAs splitting the
// rows: a thread adds every 512th row of its eight columns (16-byte loads), the CTA folds its
// 64 row lanes in shared memory and the cluster's first CTA adds the others' sums read through
// distributed shared memory, always in the same order (no atomics, no cleared output).  32
// columns a cluster keep 64 bytes of a row together and give 64 CTAs at 256 columns.
// One thread per column (2 blocks at 256 columns, a serial chain over the rows) took 926 us at
// 16,384 rows, two thirds of a gradient pass, which fell from 4.81 to 2.31 ms with this kernel.
constexpr int kSumCols = 32, kSumCluster = 8, kSumThreads = 256;
__global__ void __cluster_dims__(kSumCluster, 1, 1) __launch_bounds__(kSumThreads)
    k_colsum(int rows, int cols, const __nv_bfloat16 *dz, float *db) {
    namespace cg = cooperative_groups;
    constexpr int kLanes = kSumThreads / (kSumCols / 8);  // row lanes of a CTA
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ float part[kLanes][kSumCols + 1];
    __shared__ float sum[kSumCols];
    const int q = threadIdx.x % (kSumCols / 8), lane = threadIdx.x / (kSumCols / 8);
    const int c0 = int(blockIdx.x / kSumCluster) * kSumCols + 8 * q;
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    // whole 16-byte chunks of an aligned matrix; single values otherwise
    const bool wide = cols % 8 == 0 && (reinterpret_cast<uintptr_t>(dz) & 15) == 0;
    if (c0 < cols) {
#pragma unroll 4
        for (long long r = int(cluster.block_rank()) * kLanes + lane; r < rows; r += kSumCluster * kLanes) {
            const __nv_bfloat16 *p = dz + r * cols + c0;
            if (wide) {
                const uint4 v = *reinterpret_cast<const uint4 *>(p);
                const uint32_t h[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    s[2 * i] += __uint_as_float(h[i] << 16);
                    s[2 * i + 1] += __uint_as_float(h[i] & 0xffff0000u);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (c0 + i < cols) s[i] += __bfloat162float(p[i]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) part[lane][8 * q + i] = s[i];
    __syncthreads();
    for (int o = kLanes / 2; o >= kSumThreads / kSumCols; o >>= 1) {
        for (int k = threadIdx.x; k < o * kSumCols; k += kSumThreads)
            part[k / kSumCols][k % kSumCols] += part[k / kSumCols + o][k % kSumCols];
        __syncthreads();
    }
    if (threadIdx.x < kSumCols) {
        float t = 0.f;
        for (int k = 0; k < kSumThreads / kSumCols; ++k) t += part[k][threadIdx.x];
        sum[threadIdx.x] = t;
    }
    cluster.sync();
    const int c = int(blockIdx.x / kSumCluster) * kSumCols + int(threadIdx.x);
    if (cluster.block_rank() == 0 && threadIdx.x < kSumCols && c < cols) {
        float t = 0.f;
        for (int b = 0; b < kSumCluster; ++b) t += *cluster.map_shared_rank(&sum[threadIdx.x], b);
        db[c] = t;
    }
    cluster.sync();  // the other CTAs' sums stay until they are read
}

// Adam (Kingma & Ba 2015) on float master weights, with the bf16 copy the GEMMs read
__global__ void k_adam(long long n, float *w, const float *g, float *m, float *v, __nv_bfloat16 *wb, float lr,
                       float b1, float b2, float eps, float c1, float c2) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        w[i] = wi;
        if (wb) wb[i] = __float2bfloat16_rn(wi);
    }
}

__global__ void k_to_bf16(long long n, const float *x, __nv_bfloat16 *y) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        y[i] = __float2bfloat16_rn(x[i]);
}

// ---------------------------------------------------------------------------------------
// Fused inference: every layer in one persistent kernel
// ---------------------------------------------------------------------------------------
// A CTA (one per SM) walks 128-row tiles.  The tile's activations X (128 x 256 bf16, the
// K-major core-matrix layout the tensor cores read) stay in shared memory from layer to
// layer; the weights stream through a ring of shared-memory stages, each one bulk copy
// (cp.async.bulk, completion counted on the stage's mbarrier) of a block that the packing
// kernel already laid out in that layout.  Roles:
//   warps 0-7 (epilogue): load the tile's inputs into X; per layer read the accumulator back
//     64 columns at a time (warp w owns tensor-memory lanes 32 (w % 4) .. + 31, thread = row,
//     and half of the 64 columns), add the bias, ReLU, round to bf16 and write that slice of X for
//     the next layer; on the output layer apply scale/clamp and write the rows, or, for group
//     sums, whose products run transposed (W X^T: lane = output, column = row), add up its
//     output's rows in registers, 32 at a time, and add once per group to the sums;
//   warp 8, one thread (loader): issues the weight stages, kRing ahead of their use, across
//     layers and tiles (the next layer's weights arrive while the epilogue runs);
//   warp 9 (MMA issuer): per stage waits for its weights and for the 64-wide slice of X they
//     multiply; one elected thread issues the tcgen05.mma (128 x 256 x 16 each) and commits the
//     stage back to the loader; the accumulator's commit wakes the epilogue.  The whole warp runs
//     the loop and only offsets are added to ready descriptors: with a loop that only lane 0
//     entered and descriptors built per product, 128,000 rows took 206 us a pass and take 182
//     here, 128 rows 31.5 and 27.6.
// Two accumulators (2 x 256 tensor-memory columns) alternate between units (a layer, or a
// 256-wide chunk of the output layer), so a layer's products start on the first slice of X while
// the epilogue still writes the others, and an output chunk's epilogue overlaps the next
// chunk's products.  With four epilogue warps and one barrier for the whole of X the tensor
// cores waited for the epilogue of every hidden layer: 64 x 2,000 rows of the 6-layer network
// took 338 us there.  With the group sums' products transposed they take 137 us: summing each
// column over rows by shuffles between lanes held the output layer up (187 us; on the device
// 128,000 rows in groups of 2,000 182 -> 129 us, 2,000 rows 28.7 -> 23.2, 128,000 rows in groups of
// 31, whose rows were added one atomic each, 1,179 -> 236).  Every wait is bounded; one that runs
// out sets the error flag and a shared abort flag that ends every role's loop, and the CTA drains
// its own copies and products before freeing tensor memory.
constexpr int kWidth = 256;                       // hidden width: the MMA N and the next layer's K
constexpr int kRing = 4;                          // weight stages in flight
constexpr int kStageBytes = kWidth * kBK * 2;     // 32 KB: a 256 x 64 weight block
constexpr int kFirstBytes = kWidth * 16 * 2;      // 8 KB: the first layer's 256 x 16 block
constexpr int kXBytes = kBM * kWidth * 2;         // 64 KB: a 128-row activation tile
constexpr int kFusedThreads = 320;                // warps 0-7 epilogue, 8 loader, 9 products
constexpr int kSlices = kWidth / kBK;             // 64-wide slices of X
constexpr int kMaxLayers = 8;
constexpr int kMaxOut = 4096;

struct FusedArgs {
    const __nv_bfloat16 *x;
    long long ldx;
    int M, d_in, n_layers, n_out;
    const unsigned char *packed;
    const float *bias[kMaxLayers];
    float *out;
    int mode, group_rows, clamp;
    float scale;
    unsigned *err;
};

// one bulk copy global -> this CTA's shared memory, its bytes counted on `bar`
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// weight stages of one tile: the first layer's block, 4 per hidden layer, 4 per output chunk
__host__ __device__ inline int stages_per_tile(int n_layers, int n_out) {
    return 1 + 4 * (n_layers - 2) + 4 * (n_out / kWidth);
}
__device__ __forceinline__ uint32_t stage_bytes(int j) { return j == 0 ? kFirstBytes : kStageBytes; }
__device__ __forceinline__ size_t stage_offset(int j) {
    return j == 0 ? 0 : size_t(kFirstBytes) + size_t(j - 1) * kStageBytes;
}

__global__ void __launch_bounds__(kFusedThreads, 1) k_mlp_fused(FusedArgs g) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *X = smem;
    unsigned char *ring = smem + kXBytes;
    float *bias_sh = reinterpret_cast<float *>(ring + kRing * kStageBytes);  // every layer's, end to end
    __shared__ __align__(8) uint64_t full[kRing], empty[kRing], acc_full[2], acc_free[2], x_ready[kSlices], drain;
    __shared__ uint32_t tmem_sh;
    __shared__ volatile int abort_flag;
    __shared__ unsigned issued_sh, consumed_sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = (g.M + kBM - 1) / kBM;
    const int L = g.n_layers, NC = g.n_out / kWidth;
    for (int k = threadIdx.x; k < (L - 1) * kWidth + g.n_out; k += kFusedThreads) {
        const int l = min(k / kWidth, L - 1);
        bias_sh[k] = g.bias[l][k - l * kWidth];
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < kRing; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_free[i], 256);
        }
        for (int i = 0; i < kSlices; ++i) mbar_init(&x_ready[i], 256);
        mbar_init(&drain, 1);
        abort_flag = 0;
        issued_sh = consumed_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {  // two 128 x 256 FP32 accumulators
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                     "r"(uint32_t(2 * kWidth)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_sh;
    const int S = stages_per_tile(L, g.n_out);

    if (warp == 8) {
        // ---- loader ----
        if (lane == 0) {
            unsigned q = 0;
            for (int t = blockIdx.x; t < n_tiles && !abort_flag; t += gridDim.x) {
                for (int j = 0; j < S; ++j, ++q) {
                    const int slot = q % kRing;
                    if (q >= kRing && !mbar_wait_or_abort(&empty[slot], ((q / kRing) - 1) & 1u, &abort_flag)) {
                        abort_flag = 1;
                        break;
                    }
                    mbar_expect_tx(&full[slot], stage_bytes(j));
                    bulk_load(ring + slot * kStageBytes, g.packed + stage_offset(j), stage_bytes(j), &full[slot]);
                }
            }
            issued_sh = q;
        }
    } else if (warp == 9) {
        // ---- MMA issuer: the warp runs the loop (votes keep it uniform), one thread issues ----
        constexpr uint32_t idesc = instr_desc(kWidth);
        const bool leader = elect_one();
        const uint64_t x_desc = smem_desc(smem_u32(X), 2048, 128), w_desc = smem_desc(smem_u32(ring), 4096, 128);
        unsigned q = 0, slot = 0, wrap = 0, u = 0, x0 = 0, x1 = 0;  // x0, x1: phases of slice 0 (a layer each) and of the others
        bool ok = true;
        for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
            for (int l = 0; l < L && ok; ++l) {
                const int chunks = (l == L - 1) ? NC : 1;
                const int nst = (l == 0) ? 1 : kWidth / kBK;
                for (int c = 0; c < chunks && ok; ++c, ++u) {
                    const int b = u & 1;
                    if (u >= 2 && !__all_sync(0xffffffffu, mbar_wait_or_abort(&acc_free[b], ((u >> 1) - 1) & 1u, &abort_flag))) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t acc = tmem + uint32_t(b * kWidth);
                    for (int s = 0; s < nst; ++s) {
                        if (!__all_sync(0xffffffffu, mbar_wait_or_abort(&full[slot], wrap, &abort_flag)) ||
                            (c == 0 && !__all_sync(0xffffffffu, mbar_wait_or_abort(&x_ready[s], (s ? x1 : x0) & 1u, &abort_flag)))) {
                            ok = false;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        // X: a K chunk of eight every 2048 bytes (16 row groups of 128 B); weight
                        // block: every 4096 (32 row groups); a K = 16 step spans two chunks
                        const uint64_t ad = x_desc + uint64_t(s * (kBK / 8 * 2048 >> 4)), bd = w_desc + uint64_t(slot * (kStageBytes >> 4));
                        if (leader) {
                            if (l == L - 1 && g.mode == 1) {  // W X^T, 128 outputs (2048 bytes of a chunk) a half
                                constexpr uint32_t tdesc = instr_desc(kBM);
#pragma unroll
                                for (int j = 0; j < kBK / 16; ++j)
#pragma unroll
                                    for (int h = 0; h < 2; ++h)
                                        mma_bf16(acc + uint32_t(h * kBM), bd + uint64_t((j * 2 * 4096 + h * 2048) >> 4),
                                                 ad + uint64_t(j * (2 * 2048 >> 4)), tdesc, (s > 0 || j > 0) ? 1u : 0u);
                            } else {
                                mma_bf16(acc, ad, bd, idesc, s > 0 ? 1u : 0u);
                                if (l > 0) {
#pragma unroll
                                    for (int j = 1; j < kBK / 16; ++j)
                                        mma_bf16(acc, ad + uint64_t(j * (2 * 2048 >> 4)), bd + uint64_t(j * (2 * 4096 >> 4)), idesc,
                                                 1u);
                                }
                            }
                            mma_commit(&empty[slot]);
                        }
                        ++q;
                        if (++slot == kRing) {
                            slot = 0;
                            wrap ^= 1u;
                        }
                    }
                    if (ok && leader) mma_commit(&acc_full[b]);
                }
                ++x0;
                if (l > 0) ++x1;
            }
        }
        __syncwarp();
        if (leader) {
            if (!ok) abort_flag = 1;
            consumed_sh = q;
            // every product this thread issued has finished before the CTA frees its memory
            mma_commit(&drain);
            mbar_wait(&drain, 0);
        }
    } else {
        // ---- epilogue: warps 0-7, thread = row of the tile and half of every 64 columns ----
        const int r = threadIdx.x & 127, half = warp >> 2;
        unsigned u = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
            const int row = t * kBM + r;
            // inputs, zero-padded to K = 16 (two core-matrix columns, one per half)
            {
                unsigned short h[8];
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    h[e] = (row < g.M && 8 * half + e < g.d_in) ? __bfloat16_as_ushort(g.x[row * g.ldx + 8 * half + e])
                                                                : (unsigned short)0;
                *reinterpret_cast<uint4 *>(X + (half * 16 + r / 8) * 128 + (r % 8) * 16) =
                    make_uint4(h[0] | (uint32_t(h[1]) << 16), h[2] | (uint32_t(h[3]) << 16),
                               h[4] | (uint32_t(h[5]) << 16), h[6] | (uint32_t(h[7]) << 16));
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(&x_ready[0]);
            for (int l = 0; l < L && ok; ++l) {
                const int chunks = (l == L - 1) ? NC : 1;
                for (int c = 0; c < chunks; ++c, ++u) {
                    const int b = u & 1;
                    // warp-uniform: the tensor-memory loads below are warp-collective
                    if (!__all_sync(0xffffffffu, mbar_wait_or_abort(&acc_full[b], (u >> 1) & 1u, &abort_flag))) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t ta = tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(b * kWidth);
                    const float4 *bias = reinterpret_cast<const float4 *>(bias_sh + l * kWidth + c * kWidth);
                    if (l < L - 1) {
                        for (int s = 0; s < kSlices; ++s) {
                            const int c0 = s * kBK + half * 32;
                            float v[32];
                            tmem_ld32(ta + uint32_t(c0), v);
#pragma unroll
                            for (int q = 0; q < 4; ++q) {  // a K chunk of eight columns each
                                const float4 b0 = bias[c0 / 4 + 2 * q], b1 = bias[c0 / 4 + 2 * q + 1];
                                const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
                                uint32_t p[4];
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const float a0 = fmaxf(v[8 * q + 2 * i] + bb[2 * i], 0.f);
                                    const float a1 = fmaxf(v[8 * q + 2 * i + 1] + bb[2 * i + 1], 0.f);
                                    p[i] = pack_bf16(a0, a1);
                                }
                                *reinterpret_cast<uint4 *>(X + ((c0 / 8 + q) * 16 + r / 8) * 128 + (r % 8) * 16) =
                                    make_uint4(p[0], p[1], p[2], p[3]);
                            }
                            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                            if (s + 1 == kSlices) {
                                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                                mbar_arrive(&acc_free[b]);
                            }
                            mbar_arrive(&x_ready[s]);
                        }
                    } else if (g.mode == 1) {
                        // thread = output column, accumulator column = row: the sum over the tile's rows
                        // stays in the thread, one atomic per group that the tile meets
                        const int n = c * kWidth + half * kBM + r;
                        const float bn = bias_sh[l * kWidth + n];
                        const int rows = min(kBM, g.M - t * kBM);
                        int grp = t * kBM / g.group_rows;
                        int left = int(min((long long)kBM, (grp + 1LL) * g.group_rows - t * kBM));  // its rows ahead
                        float sum = 0.f;
                        auto next_group = [&]() {
                            atomicAdd(g.out + (long long)grp * g.n_out + n, sum);
                            sum = 0.f;
                            ++grp;
                            left = min(kBM, g.group_rows);
                        };
                        for (int r0 = 0; r0 < rows; r0 += 32) {
                            if (left == 0) next_group();
                            float v[32];
                            tmem_ld32(ta + uint32_t(half * kBM + r0), v);
#pragma unroll
                            for (int i = 0; i < 32; ++i) {
                                v[i] = (v[i] + bn) * g.scale;
                                if (g.clamp) v[i] = fmaxf(v[i], 0.f);
                            }
                            if (left >= 32 && rows - r0 >= 32) {
#pragma unroll
                                for (int w = 16; w >= 1; w >>= 1)
#pragma unroll
                                    for (int i = 0; i < w; ++i) v[i] += v[i + w];
                                sum += v[0];
                                left -= 32;
                                continue;
                            }
                            // rows to the end of the group, then the next groups'
#pragma unroll
                            for (int i = 0; i < 32; ++i) {
                                if (r0 + i >= rows) break;
                                if (left == 0) next_group();
                                sum += v[i];
                                --left;
                            }
                        }
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        mbar_arrive(&acc_free[b]);
                        atomicAdd(g.out + (long long)grp * g.n_out + n, sum);
                    } else {
                        const bool valid = row < g.M;
                        for (int s = 0; s < kSlices; ++s) {
                            const int c0 = s * kBK + half * 32;
                            float v[32];
                            tmem_ld32(ta + uint32_t(c0), v);
                            if (valid) {
                                float4 *o = reinterpret_cast<float4 *>(g.out + (long long)row * g.n_out + c * kWidth + c0);
#pragma unroll
                                for (int i = 0; i < 8; ++i) {
                                    const float4 bb = bias[c0 / 4 + i];
                                    float4 y = make_float4((v[4 * i] + bb.x) * g.scale, (v[4 * i + 1] + bb.y) * g.scale,
                                                           (v[4 * i + 2] + bb.z) * g.scale, (v[4 * i + 3] + bb.w) * g.scale);
                                    if (g.clamp)
                                        y = make_float4(fmaxf(y.x, 0.f), fmaxf(y.y, 0.f), fmaxf(y.z, 0.f), fmaxf(y.w, 0.f));
                                    o[i] = y;
                                }
                            }
                        }
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        mbar_arrive(&acc_free[b]);
                    }
                }
            }
        }
        if (!ok) abort_flag = 1;
    }
    __syncthreads();
    if (abort_flag) {
        if (threadIdx.x == 0) {
            atomicExch(g.err, 1u);
            // weight copies issued but never consumed land before their shared memory goes away
            for (unsigned q = consumed_sh; q < issued_sh; ++q) mbar_wait(&full[q % kRing], (q / kRing) & 1u);
        }
        __syncthreads();
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(uint32_t(2 * kWidth)));
}

// packed weights, in bf16 elements: the first layer's 256 x 16 block, then per hidden layer
// and per output chunk four 256 x 64 blocks (K slices 0-63, ..., 192-255), each block K-major
// core matrices: element (n, k) at byte ((k / 8) 32 + n / 8) 128 + (n % 8) 16 + (k % 8) 2
struct PackArgs {
    const __nv_bfloat16 *w[kMaxLayers];
    int dims[kMaxLayers + 1];
    int n_layers;
    long long n_elems;
    __nv_bfloat16 *out;
};

__global__ void k_mlp_pack(PackArgs a) {
    constexpr long long kFirst = kFirstBytes / 2, kBlock = kStageBytes / 2;
    const int L = a.n_layers;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < a.n_elems;
         e += (long long)gridDim.x * blockDim.x) {
        int l, n, k;
        long long off;
        if (e < kFirst) {
            l = 0;
            off = e * 2;
            n = int((off % 4096) / 128) * 8 + int((off % 128) / 16);
            k = int(off / 4096) * 8 + int((off % 16) / 2);
        } else {
            const long long blk = (e - kFirst) / kBlock;
            off = ((e - kFirst) % kBlock) * 2;
            int chunk = 0, slice;
            if (blk < 4LL * (L - 2)) {
                l = 1 + int(blk / 4);
                slice = int(blk % 4);
            } else {
                l = L - 1;
                chunk = int((blk - 4LL * (L - 2)) / 4);
                slice = int((blk - 4LL * (L - 2)) % 4);
            }
            n = chunk * kWidth + int((off % 4096) / 128) * 8 + int((off % 128) / 16);
            k = slice * kBK + int(off / 4096) * 8 + int((off % 16) / 2);
        }
        const int din = a.dims[l], dout = a.dims[l + 1];
        a.out[e] = (n < dout && k < din) ? a.w[l][(long long)n * din + k] : __float2bfloat16_rn(0.f);
    }
}

__device__ unsigned g_mlp_err = 0;

unsigned *err_flag() {
    static unsigned *addr[64] = {nullptr};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return nullptr;
    if (!addr[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_mlp_err) != cudaSuccess) return nullptr;
        addr[dev] = static_cast<unsigned *>(p);
    }
    return addr[dev];
}

template <int BN>
int launch_gemm(const GemmArgs &a, int splits, cudaStream_t st) {
    const size_t smem = size_t(kBM + BN) * kBK * 2;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(k_mlp_gemm<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess)
            return -1;
        attr = true;
    }
    const dim3 grid((a.M + kBM - 1) / kBM, (a.N + BN - 1) / BN, splits);
    k_mlp_gemm<BN><<<grid, kThreads, smem, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? 1 : -1;
}

// The tensor map of one operand: `rows` x `k` values, element (r, j) at p[r lr + j lk].  K-major
// (lk 1) boxes hold 64 K of `box_rows` rows, MN-major ones (lr 1) 64 rows of kBK K.  False when
// TMA cannot address it.
typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
    static const EncodeTiled fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<EncodeTiled>(p);
    }();
    return fn;
}
bool operand_map(CUtensorMap &map, const __nv_bfloat16 *p, int rows, int k, long long lr, long long lk, int box_rows,
                 int &mn_major) {
    mn_major = lk != 1;
    const long long ld = mn_major ? lk : lr;
    if ((mn_major && lr != 1) || ld <= 0 || ld % 8 || ld >= (1ll << 38) || (reinterpret_cast<uintptr_t>(p) & 15))
        return false;
    const EncodeTiled encode = encode_tiled();
    if (!encode) return false;
    const cuuint64_t dims[2] = {cuuint64_t(mn_major ? rows : k), cuuint64_t(mn_major ? k : rows)};
    const cuuint64_t stride[1] = {cuuint64_t(ld) * 2};
    const cuuint32_t box[2] = {64u, cuuint32_t(mn_major ? kBK : box_rows)}, step[2] = {1u, 1u};
    return encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16 *>(p), dims, stride, box, step,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// SMs of the current device, 0 on failure
int device_sms() {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    return n;
}

// 1 launched, -1 launch failure, 0: TMA cannot address the operands (the caller launches k_mlp_gemm)
template <int BN>
int launch_gemm_tma(const GemmArgs &a, int splits, cudaStream_t st) {
    CUtensorMap ta, tb;
    int a_mn = 0, b_mn = 0;
    if (!operand_map(ta, a.A, a.M, a.K, a.lam, a.lak, kBM, a_mn) ||
        !operand_map(tb, a.B, a.N, a.K, a.lbn, a.lbk, BN, b_mn))
        return 0;
    constexpr int smem = kPipeBytes + 1024;
    // set on every call: the attribute belongs to the current device's context
    if (cudaFuncSetAttribute(k_mlp_gemm_tma<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
        return -1;
    const int sms = device_sms();
    if (sms <= 0) return -1;
    const long long tiles_m = (a.M + (long long)kBM - 1) / kBM, tiles_n = (a.N + (long long)BN - 1) / BN;
    const long long items = tiles_m * tiles_n * splits;
    k_mlp_gemm_tma<BN><<<unsigned(items < sms ? items : sms), kPipeThreads, smem, st>>>(
        ta, tb, a, int(tiles_m), int(tiles_n), items, a_mn, b_mn);
    return cudaGetLastError() == cudaSuccess ? 1 : -1;
}

// the TMA kernel where it can read the operands, else the one that reads any strides
template <int BN>
int launch_gemm_any(const GemmArgs &a, int splits, cudaStream_t st) {
    const int rc = launch_gemm_tma<BN>(a, splits, st);
    return rc != 0 ? rc : launch_gemm<BN>(a, splits, st);
}

// the fused kernel's shape rules; -1 or the packed size in bf16 elements
long long packed_elems(int n_layers, const int *dims) {
    if (!dims || n_layers < 2 || n_layers > kMaxLayers) return -1;
    if (dims[0] < 1 || dims[0] > 16) return -1;
    for (int l = 1; l < n_layers; ++l)
        if (dims[l] != kWidth) return -1;
    const int n_out = dims[n_layers];
    if (n_out < kWidth || n_out > kMaxOut || n_out % kWidth) return -1;
    return kFirstBytes / 2 + (long long)(stages_per_tile(n_layers, n_out) - 1) * (kStageBytes / 2);
}

int launch_fused(const FusedArgs &a, cudaStream_t st) {
    // X, the weight ring and the biases (at most 7 x 256 + 4096)
    constexpr int smem = kXBytes + kRing * kStageBytes + ((kMaxLayers - 1) * kWidth + kMaxOut) * 4;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
    static int sms[64] = {0};
    if (!sms[dev]) {
        if (cudaFuncSetAttribute(k_mlp_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return -1;
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return -1;
        sms[dev] = n;
    }
    const int tiles = (a.M + kBM - 1) / kBM;
    k_mlp_fused<<<tiles < sms[dev] ? tiles : sms[dev], kFusedThreads, smem, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? 1 : -1;
}

}  // namespace mlp
}  // namespace stb

using namespace stb::mlp;

extern "C" {

int st_b200_mlp_gemm(int m, int n, int k, const void *A, long long lam, long long lak, const void *B, long long lbn,
                     long long lbk, void *C, long long ldc, int epilogue, const float *bias, const void *aux, int splits,
                     void *stream) {
    if (m <= 0 || n <= 0 || k <= 0 || !A || !B || !C || epilogue < EPI_BIAS_RELU_BF16 || epilogue > EPI_F32_ADD)
        return -1;
    if ((epilogue == EPI_BIAS_RELU_BF16 || epilogue == EPI_BIAS_F32) && !bias) return -1;
    if (epilogue == EPI_RELU_MASK_BF16 && !aux) return -1;
    if (splits < 1 || (splits > 1 && epilogue != EPI_F32_ADD)) return -1;
    GemmArgs a;
    a.A = static_cast<const __nv_bfloat16 *>(A);
    a.B = static_cast<const __nv_bfloat16 *>(B);
    a.lam = lam;
    a.lak = lak;
    a.lbn = lbn;
    a.lbk = lbk;
    a.M = m;
    a.N = n;
    a.K = k;
    a.epi = epilogue;
    a.C = C;
    a.ldc = ldc;
    a.bias = bias;
    a.aux = static_cast<const __nv_bfloat16 *>(aux);
    const int kb = (k + kBK - 1) / kBK;
    a.k_per_split = ((kb + splits - 1) / splits) * kBK;
    a.err = err_flag();
    if (!a.err) return -1;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n >= 256) return launch_gemm_any<256>(a, splits, st);
    if (n <= 64) return launch_gemm_any<64>(a, splits, st);
    return launch_gemm_any<128>(a, splits, st);
}

int st_b200_mlp_mse(int rows, int cols, const float *y, const float *target, long long ldt, void *dy, double *loss,
                    void *stream) {
    if (rows <= 0 || cols <= 0 || !y || !target || !dy || !loss) return -1;
    const bool wide = ldt == cols && (long long)rows * cols % 4 == 0 &&
                      ((reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(target)) & 15) == 0 &&
                      (reinterpret_cast<uintptr_t>(dy) & 7) == 0;
    (wide ? k_mse<1> : k_mse<0>)<<<1184, kMseThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        rows, cols, y, target, ldt, static_cast<__nv_bfloat16 *>(dy), loss);
    return cudaGetLastError() == cudaSuccess ? 1 : -1;
}

int st_b200_mlp_colsum(int rows, int cols, const void *dz, float *db, void *stream) {
    if (rows <= 0 || cols <= 0 || !dz || !db) return -1;
    const unsigned chunks = unsigned((cols + (long long)kSumCols - 1) / kSumCols);
    k_colsum<<<chunks * kSumCluster, kSumThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        rows, cols, static_cast<const __nv_bfloat16 *>(dz), db);
    return cudaGetLastError() == cudaSuccess ? 1 : -1;
}

int st_b200_mlp_adam(long long n, float *w, const float *g, float *m, float *v, void *w_bf16, float lr, float beta1,
                     float beta2, float eps, int step, void *stream) {
    if (n <= 0 || !w || !g || !m || !v || step < 1) return -1;
    const float c1 = 1.f - powf(beta1, float(step)), c2 = 1.f - powf(beta2, float(step));
    k_adam<<<592, 256, 0, static_cast<cudaStream_t>(stream)>>>(n, w, g, m, v, static_cast<__nv_bfloat16 *>(w_bf16), lr,
                                                               beta1, beta2, eps, c1, c2);
    return cudaGetLastError() == cudaSuccess ? 1 : -1;
}

int st_b200_mlp_to_bf16(long long n, const float *x, void *y, void *stream) {
    if (n <= 0 || !x || !y) return -1;
    k_to_bf16<<<592, 256, 0, static_cast<cudaStream_t>(stream)>>>(n, x, static_cast<__nv_bfloat16 *>(y));
    return cudaGetLastError() == cudaSuccess ? 1 : -1;
}

long long st_b200_mlp_packed_bytes(int n_layers, const int *dims) {
    const long long e = packed_elems(n_layers, dims);
    return e < 0 ? -1 : 2 * e;
}

int st_b200_mlp_pack(int n_layers, const int *dims, const void *const *w, void *packed, void *stream) {
    const long long e = packed_elems(n_layers, dims);
    if (e < 0 || !w || !packed) return -1;
    PackArgs a;
    for (int l = 0; l < n_layers; ++l) {
        if (!w[l]) return -1;
        a.w[l] = static_cast<const __nv_bfloat16 *>(w[l]);
    }
    for (int l = 0; l <= n_layers; ++l) a.dims[l] = dims[l];
    a.n_layers = n_layers;
    a.n_elems = e;
    a.out = static_cast<__nv_bfloat16 *>(packed);
    k_mlp_pack<<<592, 256, 0, static_cast<cudaStream_t>(stream)>>>(a);
    return cudaGetLastError() == cudaSuccess ? 1 : -1;
}

int st_b200_mlp_forward_fused(int n_layers, const int *dims, const void *packed, const float *const *bias, int m,
                              const void *x, long long ldx, float *out, int mode, int group_rows, float scale,
                              int clamp, void *stream) {
    if (packed_elems(n_layers, dims) < 0 || !packed || !bias || m <= 0 || !x || ldx < dims[0] || !out) return -1;
    if (mode < 0 || mode > 1 || (mode == 1 && group_rows < 1)) return -1;
    if ((reinterpret_cast<uintptr_t>(packed) & 15) || (reinterpret_cast<uintptr_t>(out) & 15)) return -1;
    FusedArgs a;
    for (int l = 0; l < n_layers; ++l) {
        if (!bias[l]) return -1;
        a.bias[l] = bias[l];
    }
    a.x = static_cast<const __nv_bfloat16 *>(x);
    a.ldx = ldx;
    a.M = m;
    a.d_in = dims[0];
    a.n_layers = n_layers;
    a.n_out = dims[n_layers];
    a.packed = static_cast<const unsigned char *>(packed);
    a.out = out;
    a.mode = mode;
    a.group_rows = mode == 1 ? group_rows : 1;
    a.clamp = clamp ? 1 : 0;
    a.scale = scale;
    a.err = err_flag();
    if (!a.err) return -1;
    return launch_fused(a, static_cast<cudaStream_t>(stream));
}

// the GEMM error flag of the current device (1: a wait ran out), cleared by the read
int st_b200_mlp_error(void) {
    unsigned *f = err_flag();
    if (!f) return -1;
    unsigned v = 0;
    if (cudaMemcpy(&v, f, sizeof v, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    if (v) {
        const unsigned z = 0;
        cudaMemcpy(f, &z, sizeof z, cudaMemcpyHostToDevice);
    }
    return int(v);
}

}  // extern "C"
