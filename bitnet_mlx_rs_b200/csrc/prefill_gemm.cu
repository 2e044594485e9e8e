// Prefill-time BitLinear (many tokens): int8 x ternary GEMM on the 5th-generation tensor cores.
//
//   1. quantize_rows_perm_kernel: per-token absmax int8 quantisation of x[M,K] into scratch,
//      with the 16 values of every 16-wide k group stored transposed (byte 4j+i holds k = 4i+j),
//      plus the row sums sum_k q[m,k].
//   2. prefill_gemm_kernel: persistent CTAs; the accumulator tile is 128 output features (tensor-memory
//      lanes) x up to 192 tokens (columns), i.e. the weights are the MMA's A operand.
//        warp 0      activation loads: per pair of 128-wide k slices one TMA box of int8 activations
//                    (tokens x 128 bytes x 2, 128-byte swizzle)
//        last warp   packed-weight loads: one box of 128 rows x 64 bytes per pair (64-byte swizzle), through a ring of
//                    its own that runs far ahead of the activations
//        warps 2-    expand packed weights to u8 codes {0,1,2} in registers and write them straight
//                    into TENSOR MEMORY (tcgen05.st), where the MMA reads its A operand: a thread
//                    owns one feature row; (w >> 2j) & 0x03030303 yields the four bytes
//                    k = j, j+4, j+8, j+12 of a group, i.e. word j of the transposed group order the
//                    activations were stored in.  Expanded weights never touch shared memory.
//                    (two or three groups of four warps take the pairs in turn)
//        warp 1      one thread issues tcgen05.mma kind::i8 (M=128, N=tokens, K=32; u8 x s8 -> s32),
//                    A from tensor memory, B (activations) from shared memory; two accumulators
//                    alternate between tiles
//        4 warps     epilogue: tcgen05.ld the accumulator, subtract the row sum
//                    (sum_k (code-1) q = sum_k code q - sum_k q), scale, stage 32 x 32 blocks in
//                    shared memory and write y with TMA stores
//      What bounds it: above 128 tokens the MMAs (653 clk a pair of slices at the int8 rate with 160 tokens; 745 measured where
//      k is long); at 128 and fewer the instructions of the single threads and warps that feed them, 565 to 665 clk a
//      pair.  In the MMA thread (clock reads around each part, five shapes): the wait for the pair 200 to 250, the eight MMAs
//      130 to 160 (16 to 20 each to issue), commit and ring step 110 to 270.  With its quantiser, weights from memory:
//      2048x2560x6912 40.0 us = 1813 TOPS (55.9 before the roles were taken apart and their loops run by elected threads),
//      256x8192x28672 49.7 (86.2), 64x2560x128256 32.5 us (63.1).
//      Work is dealt in whole tiles, or -- when whole tiles would leave most of a wave idle -- in
//      equal runs of k slices with an exact integer fix-up of the tiles shared by two CTAs.
//      Every barrier wait is bounded; a wait that runs out raises an error flag and the CTA
//      drains and frees its tensor memory.
//
// Semantics: TernaryProcessor::quantize_activations + ternary_matmul_generic
// (bitnet-inference/src/engine/ternary_operations.rs:117-172, :283-338) with int32 accumulation
// on the packed layout of BitPacked2BitPacker (bitnet-quant/src/quantization/packing.rs:352-394).
// The reference has no tensor-core kernel; this is what its BitLinearLayer::forward
// (transformer_layers.rs:119-202) computes for a [B*S, K] input.
#include <cuda.h>
#include <cstdlib>
#include <mutex>

#include "common.cuh"

namespace bitnet {

// Set (bit 1) when a bounded wait of the GEMM kernel ran out -- read with bitnet_device_error_flags().
__device__ unsigned g_prefill_error_flags;

constexpr int PF_BF = 128;                         // output features per tile (the MMA's M: tensor-memory lanes)
constexpr int PF_BT = 192;                         // tokens per tile (the MMA's N)
constexpr int PF_BK = 128;                         // k per slice (bytes of int8)
constexpr int PF_PAIR = 2;                         // k slices per hand-over between the roles (one barrier round per pair)
constexpr int PF_MAX_RING = 8, PF_MAX_WRING = 20;  // pairs in flight; a plan's depths depend on its tile (pf_rings)
constexpr int PF_WP_BYTES = PF_BF * PF_BK / 4;     // 4 KB packed
// Groups of four warps that expand packed weights, working on alternate pairs.  One takes about 1300 clk a pair (its waits
// 470, masks and shifts 300, the tensor-memory store 350): two keep ahead of the MMAs of a tile above 128 tokens (784 clk a
// pair at 192), narrower ones take three (64x2560x128256: 36.2 -> 33.7 us; at 192 tokens the smaller register share of the
// wider CTA makes three the slower choice, 26.3 against 27.8 us for 192x8192x18944).  Three groups are 608 threads of 96
// registers: 64 bytes of stores and 176 of loads are spilled (gate/up pair 40 and 84; none with two groups).
constexpr int pf_groups(int bt) { return bt > 128 ? 2 : 3; }
constexpr int pf_threads(int groups) { return (2 + 4 * groups + 4 + 1) * 32; }   // activation loads, MMA, expanders, epilogue, weight loads
constexpr unsigned PF_WAIT_LIMIT = 1u << 17;      // tries of at most 16 us each
constexpr unsigned PF_POLL_LIMIT = 1u << 20;      // polls of a counter in global memory
constexpr int PF_A_COLS = PF_BK / 4;               // tensor-memory columns that hold 128 bytes of k per lane
constexpr int PF_WARP_OUT_BYTES = 32 * 32 * 4;     // epilogue staging per warp: 32 tokens x 32 features fp32, two of them
constexpr int PF_OUT_BYTES = 4 * PF_WARP_OUT_BYTES;
constexpr size_t PF_SMEM = 217 * 1024;             // ring of activations, ring of packed weights, staging, alignment slack
constexpr size_t PF_RING_BYTES = PF_SMEM - 2 * PF_OUT_BYTES - 1024;
constexpr size_t PF_SLOT_BYTES = (size_t)PF_BF * PF_BT * 4;   // one partial accumulator tile

// ---- quantiser for the GEMM path ----------------------------------------------------------------

// Same exact rounding as common.cuh's quantize_one for |x*scale| <= 2^22 (trunc(|t| + c) with c the
// largest float below 0.5 equals roundf(|t|) for every float; adding 2^23 toward zero leaves the
// integer in the low mantissa bits); NaN quantises to 0.
__device__ __forceinline__ int pf_quantize_fast(float x, float scale)
{
    const float t = __fmul_rn(x, scale);
    const float a = fminf(__fadd_rn(fabsf(t), 0.49999997f), 127.0f);
    const int mag = __float_as_int(__fadd_rz(a, 8388608.0f)) & 0xff;
    const int neg = __float_as_int(t) >> 31;
    return (t == t) ? (mag ^ neg) - neg : 0;
}

// One CTA per token row, one read of the row when it fits the registers (two 16-wide groups per
// thread).  Short rows take 128-thread CTAs: more rows in flight per SM, which is what bounds this
// kernel (a row is one dependent chain load -> absmax -> quantise -> store).
// q_perm[m, 16G + 4j + i] = q[m, 16G + 4i + j]; rowsum[m] = sum_k q[m,k]; rows of q_perm are `pitch` bytes apart.
// Semantics: TernaryProcessor::quantize_activations (ternary_operations.rs:130-163).
template <int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == 128 ? 8 : 4) quantize_rows_perm_kernel(const float *__restrict__ x, size_t K, size_t pitch,
                                                                 int8_t *__restrict__ q_perm, float *__restrict__ a_scale,
                                                                 int *__restrict__ rowsum, int8_t *__restrict__ q_out,
                                                                 float *__restrict__ a_scale_out, unsigned *__restrict__ counters,
                                                                 int n_counters)
{
    // the GEMM that follows may start (allocate tensor memory, fetch packed weights) while this runs;
    // it waits for this grid before it touches anything written here
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // launched with programmatic dependent launch itself (BITNET_FLAG_PDL): x and the scratch this grid
    // overwrites belong to the kernels before it until they have finished
    asm volatile("griddepcontrol.wait;" ::: "memory");
    // the GEMM counts the parts of split tiles in these; they start at zero
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < n_counters; i += THREADS) counters[i] = 0u;
    __shared__ unsigned s_key[THREADS / 32];
    __shared__ int s_sum[THREADS / 32];
    const size_t m = blockIdx.x;
    const float *row = x + m * K;
    const int tid = threadIdx.x;
    const size_t n_groups = K / 16;
    const bool resident = n_groups <= 2 * THREADS;   // two 16-wide groups per thread stay in registers

    float4 f[2][4];
    unsigned key = 0;
    if (resident) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const size_t G = tid + u * THREADS;
            if (G < n_groups) {
                const float4 *src = reinterpret_cast<const float4 *>(row + G * 16);
#pragma unroll
                for (int v = 0; v < 4; ++v) f[u][v] = __ldg(src + v);
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
            if ((size_t)(tid + u * THREADS) < n_groups) {
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    key = max(max(key, abs_key(f[u][v].x)), max(abs_key(f[u][v].y), max(abs_key(f[u][v].z), abs_key(f[u][v].w))));
            }
    } else {
        for (size_t G = tid; G < n_groups; G += THREADS) {
            const float4 *src = reinterpret_cast<const float4 *>(row + G * 16);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const float4 g4 = __ldg(src + v);
                key = max(max(key, abs_key(g4.x)), max(abs_key(g4.y), max(abs_key(g4.z), abs_key(g4.w))));
            }
        }
    }
    key = __reduce_max_sync(0xffffffffu, key);
    if ((tid & 31) == 0) s_key[tid >> 5] = key;
    __syncthreads();
    key = 0;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) key = max(key, s_key[w]);
    const float absmax = __uint_as_float(key);
    const float scale = quant_scale(absmax);
    // a huge or tiny absmax makes the scale leave the normal range; the fast rounding assumes it has not
    const bool fast = scale >= 1e-30f && scale <= 1e30f;

    int sum = 0;
    const size_t rounds = resident ? 2 : (n_groups + THREADS - 1) / THREADS;
    for (size_t u = 0; u < rounds; ++u) {
        const size_t G = tid + u * THREADS;
        if (G >= n_groups) break;
        float4 g4[4];
        if (resident) {
#pragma unroll
            for (int v = 0; v < 4; ++v) g4[v] = u == 0 ? f[0][v] : f[1][v];
        } else {
            const float4 *src = reinterpret_cast<const float4 *>(row + G * 16);
#pragma unroll
            for (int v = 0; v < 4; ++v) g4[v] = __ldg(src + v);
        }
        int q[16];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            if (fast) {
                q[4 * v + 0] = pf_quantize_fast(g4[v].x, scale);
                q[4 * v + 1] = pf_quantize_fast(g4[v].y, scale);
                q[4 * v + 2] = pf_quantize_fast(g4[v].z, scale);
                q[4 * v + 3] = pf_quantize_fast(g4[v].w, scale);
            } else {
                q[4 * v + 0] = quantize_one(g4[v].x, scale);
                q[4 * v + 1] = quantize_one(g4[v].y, scale);
                q[4 * v + 2] = quantize_one(g4[v].z, scale);
                q[4 * v + 3] = quantize_one(g4[v].w, scale);
            }
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) sum += q[e];
        uint4 perm;
        perm.x = (q[0] & 0xff) | ((q[4] & 0xff) << 8) | ((q[8] & 0xff) << 16) | ((unsigned)(q[12] & 0xff) << 24);
        perm.y = (q[1] & 0xff) | ((q[5] & 0xff) << 8) | ((q[9] & 0xff) << 16) | ((unsigned)(q[13] & 0xff) << 24);
        perm.z = (q[2] & 0xff) | ((q[6] & 0xff) << 8) | ((q[10] & 0xff) << 16) | ((unsigned)(q[14] & 0xff) << 24);
        perm.w = (q[3] & 0xff) | ((q[7] & 0xff) << 8) | ((q[11] & 0xff) << 16) | ((unsigned)(q[15] & 0xff) << 24);
        *reinterpret_cast<uint4 *>(q_perm + m * pitch + G * 16) = perm;
        if (q_out) {
            uint4 canon;
            canon.x = (q[0] & 0xff) | ((q[1] & 0xff) << 8) | ((q[2] & 0xff) << 16) | ((unsigned)(q[3] & 0xff) << 24);
            canon.y = (q[4] & 0xff) | ((q[5] & 0xff) << 8) | ((q[6] & 0xff) << 16) | ((unsigned)(q[7] & 0xff) << 24);
            canon.z = (q[8] & 0xff) | ((q[9] & 0xff) << 8) | ((q[10] & 0xff) << 16) | ((unsigned)(q[11] & 0xff) << 24);
            canon.w = (q[12] & 0xff) | ((q[13] & 0xff) << 8) | ((q[14] & 0xff) << 16) | ((unsigned)(q[15] & 0xff) << 24);
            *reinterpret_cast<uint4 *>(q_out + m * K + G * 16) = canon;
        }
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if ((tid & 31) == 0) s_sum[tid >> 5] = sum;
    __syncthreads();
    if (tid == 0) {
        int total = 0;
#pragma unroll
        for (int w = 0; w < THREADS / 32; ++w) total += s_sum[w];
        rowsum[m] = total;
        a_scale[m] = dequant_scale(absmax);
        if (a_scale_out) a_scale_out[m] = dequant_scale(absmax);
    }
}

// The same for any K and any alignment of x: a thread makes the four bytes of one word of the transposed order, so that its
// loads of the row (cached: the first pass has just read it) and its stores are coalesced.  Bytes past K are zero.
__global__ void __launch_bounds__(256) quantize_rows_pad_kernel(const float *__restrict__ x, size_t K, size_t pitch, int8_t *__restrict__ q_perm,
                                                                float *__restrict__ a_scale, int *__restrict__ rowsum, int8_t *__restrict__ q_out,
                                                                float *__restrict__ a_scale_out, unsigned *__restrict__ counters, int n_counters)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < n_counters; i += 256) counters[i] = 0u;
    __shared__ unsigned s_key[8];
    __shared__ int s_sum[8];
    const size_t m = blockIdx.x;
    const float *row = x + m * K;
    const int tid = threadIdx.x;
    unsigned key = 0;
    for (size_t k = tid; k < K; k += 256) key = max(key, abs_key(__ldg(row + k)));
    key = __reduce_max_sync(0xffffffffu, key);
    if ((tid & 31) == 0) s_key[tid >> 5] = key;
    __syncthreads();
    key = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) key = max(key, s_key[w]);
    const float absmax = __uint_as_float(key);
    const float scale = quant_scale(absmax);
    int sum = 0;
    for (size_t w = tid; w < pitch / 4; w += 256) {
        const size_t k0 = (w >> 2) * 16 + (w & 3);
        unsigned word = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const size_t k = k0 + 4 * i;
            if (k < K) {
                const int q = quantize_one(__ldg(row + k), scale);
                sum += q;
                word |= ((unsigned)q & 0xffu) << (8 * i);
                if (q_out) q_out[m * K + k] = (int8_t)q;
            }
        }
        *reinterpret_cast<unsigned *>(q_perm + m * pitch + 4 * w) = word;
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if ((tid & 31) == 0) s_sum[tid >> 5] = sum;
    __syncthreads();
    if (tid == 0) {
        int total = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) total += s_sum[w];
        rowsum[m] = total;
        a_scale[m] = dequant_scale(absmax);
        if (a_scale_out) a_scale_out[m] = dequant_scale(absmax);
    }
}

// Rows of the flat packed stream that start in the middle of a byte, or not on the 16 bytes that TMA asks of a row, copied to
// rows of `pitch` bytes (codes past K are 0: they meet no activation).  A thread makes 16 codes from two words of the stream;
// words that reach past its end, and all words of a stream that is not 4-byte aligned, are put together from bytes.
// Code 3 becomes 1 (weight 0) on the way, as the generic kernel reads it.
__global__ void __launch_bounds__(256) repack_rows_kernel(const uint8_t *__restrict__ wp, size_t stream_bytes, size_t N, size_t K, size_t pitch,
                                                          uint8_t *__restrict__ out)
{
    const size_t words = pitch / 4, total = N * words;
    const bool aligned = (reinterpret_cast<uintptr_t>(wp) & 3) == 0;
    auto word_at = [&](size_t i) -> unsigned {   // bytes 4i .. 4i+3 of the stream, zeros past its end
        if (aligned && 4 * i + 4 <= stream_bytes) return __ldg(reinterpret_cast<const unsigned *>(wp) + i);
        unsigned v = 0;
        for (int b = 0; b < 4; ++b)
            if (4 * i + b < stream_bytes) v |= (unsigned)__ldg(wp + 4 * i + b) << (8 * b);
        return v;
    };
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        const size_t n = t / words, w = t - n * words, k0 = 16 * w;
        unsigned v = 0;
        if (k0 < K) {
            const size_t e = n * K + k0;          // flat index of the first code
            v = __funnelshift_r(word_at(e >> 4), word_at((e >> 4) + 1), 2 * (unsigned)(e & 15));
            const unsigned both = (v >> 1) & v & 0x55555555u;
            v ^= both << 1;
            if (K - k0 < 16) v &= (1u << (2 * (unsigned)(K - k0))) - 1u;
        }
        reinterpret_cast<unsigned *>(out)[t] = v;
    }
}

// ---- PTX wrappers -------------------------------------------------------------------------------

__device__ __forceinline__ unsigned pf_smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void pf_mbar_init(unsigned long long *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(pf_smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void pf_mbar_arrive(unsigned long long *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(pf_smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void pf_mbar_expect_tx(unsigned long long *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(pf_smem_u32(bar)), "r"(bytes) : "memory");
}
// Bounded wait; false (and the error flag) when the phase did not complete in time.  try_wait suspends the thread in
// hardware and wakes it when the phase completes: a nanosleep between the tries woke it up to 200 clk late, and tries
// without the long time limit (16 us) kept the barrier unit so busy that a wait for a completed phase took 130 clk, not 90.
__device__ __forceinline__ bool pf_mbar_wait(unsigned long long *bar, unsigned parity)
{
    const unsigned addr = pf_smem_u32(bar);
    for (unsigned n = 0; n < PF_WAIT_LIMIT; ++n) {
        unsigned done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity), "r"(16384)
            : "memory");
        if (done) return true;
    }
    atomicOr(&g_prefill_error_flags, 2u);
    return false;
}
// The whole warp waits (one broadcast access per try) and leaves together.
__device__ __forceinline__ bool pf_warp_wait(unsigned long long *bar, unsigned parity)
{
    return __all_sync(0xffffffffu, pf_mbar_wait(bar, parity));
}
__device__ __forceinline__ void pf_tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, unsigned long long *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
            pf_smem_u32(dst)),
        "l"(map), "r"(pf_smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}
__device__ __forceinline__ void pf_tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, unsigned long long *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            pf_smem_u32(dst)),
        "l"(map), "r"(pf_smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}
// K-major operand, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart.
__device__ __forceinline__ unsigned long long pf_smem_desc(unsigned smem_addr)
{
    return (unsigned long long)((smem_addr >> 4) & 0x3fffu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void pf_commit(unsigned long long *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(pf_smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void pf_tmem_ld32(unsigned taddr, unsigned (&r)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void pf_mma_i8_ts(unsigned tmem_d, unsigned tmem_a, unsigned long long b_desc, unsigned idesc,
                                             unsigned accumulate)
{
    // A (expanded weights) comes from tensor memory, B (activations) from shared memory
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void pf_tmem_st32(unsigned taddr, const unsigned (&r)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
// Barrier among the four epilogue warps that also ANDs a predicate (all leave a loop together).
__device__ __forceinline__ bool pf_epi_all(bool ok)
{
    unsigned out;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "barrier.cta.red.and.pred p, 1, 128, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(out)
        : "r"(ok ? 1u : 0u)
        : "memory");
    return out != 0;
}

__device__ __forceinline__ void pf_tma_store_2d(const CUtensorMap *map, int x, int y, const void *src)
{
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map),
                 "r"(pf_smem_u32(src)), "r"(x), "r"(y)
                 : "memory");
}
struct PrefillParams {
    float *y;
    int32_t *acc_out;
    const float *a_scale;
    const int *rowsum;
    int *slots;          // partial accumulator tiles, two per CTA, [token][feature] int32
    unsigned *counters;  // per tile: k slices contributed so far (zero at launch)
    float w_scale, w_scale2;       // pair: gate scale, up scale
    int seg_end0, seg_end1;        // stacked matrices: features below seg_end0 use w_scale, below seg_end1 seg_scale1, the rest seg_scale2
    float seg_scale1, seg_scale2;
    int M, K, N;
    size_t ldy;
    int m_tiles, n_tiles, k_tiles;
    int tma_store;       // y can be written with TMA (16-byte aligned rows), else plain stores
    int bt;              // tokens per tile (the MMA's N): a multiple of 32, at most PF_BT
    int ring, wring;     // activation and packed-weight pairs in flight
    int aslots;          // expanded-weight pairs in tensor memory, behind the two accumulators of bt columns
    int whole_tiles;     // ranges end on tile boundaries (no tile is split between CTAs)
    float *y_peers[8];   // output-feature split over several GPUs: every output goes to each of these (own and peer
    int n_peers;         // memory, plain stores over NVLink; TMA is used for this GPU's memory only); 0 = write y only
};

// instruction descriptor: D = s32, A = u8 (codes, tensor memory), B = s8 (activations, K-major), N = tokens, M = 128
__host__ __device__ constexpr unsigned pf_idesc(int bt) { return (2u << 4) | (0u << 7) | (1u << 10) | ((unsigned)(bt >> 3) << 17) | ((unsigned)(PF_BF >> 4) << 24); }

// The work of the whole GEMM is the sequence of (tile, k slice) units, tile-major; CTA c takes
// the contiguous range [U*c/G, U*(c+1)/G), so every CTA has the same number of k slices whatever
// the tile count.  A segment is the part of one tile inside a range.  A CTA works through its
// segments in the order: first (often a partial tile), last (often a partial tile), then the whole
// tiles in between -- the fix-up of a tile shared with a neighbour then happens early on both
// sides and hides behind the MMAs of the whole tiles, and the kernel's tail is a plain tile.
struct PfSegment {
    int tile, kb, ke;
};
struct PfSchedule {
    int t_first, kb_first;   // tile and k position of the range's first unit
    int t_last, ke_last;     // tile of the range's last unit, end of its k range
    int n_seg;
};
__device__ __forceinline__ long long pf_range_start(long long units, int c, int ctas, int k_tiles = 0)
{
    if (k_tiles > 0) {   // whole tiles only: split the tile count, not the slice count
        const unsigned tiles = (unsigned)(units / k_tiles);
        return (long long)(unsigned)((unsigned long long)tiles * (unsigned)c / (unsigned)ctas) * k_tiles;
    }
    // 32-bit arithmetic when it fits (the usual case): 64-bit division is slow on the device
    if (units < (1ll << 31) / (ctas > 0 ? ctas : 1)) return (long long)((unsigned)units * (unsigned)c / (unsigned)ctas);
    return units * c / ctas;
}
__device__ __forceinline__ PfSchedule pf_schedule(long long u_begin, long long u_end, int k_tiles)
{
    PfSchedule sch;
    sch.n_seg = 0;
    sch.t_first = sch.kb_first = sch.t_last = sch.ke_last = 0;
    if (u_end <= u_begin) return sch;
    if (u_end < (1ll << 31)) {
        sch.t_first = (int)((unsigned)u_begin / (unsigned)k_tiles);
        sch.t_last = (int)((unsigned)(u_end - 1) / (unsigned)k_tiles);
    } else {
        sch.t_first = (int)(u_begin / k_tiles);
        sch.t_last = (int)((u_end - 1) / k_tiles);
    }
    sch.kb_first = (int)(u_begin - (long long)sch.t_first * k_tiles);
    sch.ke_last = (int)(u_end - (long long)sch.t_last * k_tiles);
    sch.n_seg = sch.t_last - sch.t_first + 1;
    return sch;
}
__device__ __forceinline__ PfSegment pf_segment(const PfSchedule &sch, int idx, int k_tiles)
{
    PfSegment sg;
    if (sch.n_seg == 1) {
        sg.tile = sch.t_first; sg.kb = sch.kb_first; sg.ke = sch.ke_last;
    } else if (idx == 0) {
        sg.tile = sch.t_first; sg.kb = sch.kb_first; sg.ke = k_tiles;
    } else if (idx == 1) {
        sg.tile = sch.t_last; sg.kb = 0; sg.ke = sch.ke_last;
    } else {
        sg.tile = sch.t_first + idx - 1; sg.kb = 0; sg.ke = k_tiles;
    }
    return sg;
}

// PAIR: gate and up projection in one launch, y receives up * relu(gate)^2.  A tile is 64 features of both: rows 0-63 of the
// MMA's A operand are gate rows, rows 64-127 the up rows of the same features, so the two values of an output meet in
// one CTA, in lanes 64 apart, and the epilogue's gate warps hand theirs to the up warps through shared memory.
template <int GROUPS, bool PAIR>
__global__ void __launch_bounds__(pf_threads(GROUPS), 1)
prefill_gemm_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                    const __grid_constant__ CUtensorMap map_w2, const __grid_constant__ CUtensorMap map_y, const PrefillParams p)
{
    constexpr int EXP_WARPS = 4 * GROUPS;
    constexpr int TILE_F = PAIR ? PF_BF / 2 : PF_BF;   // output features per tile
    extern __shared__ unsigned char pf_smem_raw[];
    __shared__ __align__(8) unsigned long long s_full_w[PF_MAX_WRING];       // a pair's packed weights have landed
    __shared__ __align__(8) unsigned long long s_free_w[PF_MAX_WRING];   // a pair's packed weights are in the expanders' registers
    __shared__ __align__(8) unsigned long long s_full[PF_MAX_RING];          // a pair's activations have landed and its weights are expanded in tensor memory
    __shared__ __align__(8) unsigned long long s_done[PF_MAX_RING];          // the MMAs of a pair have read their operands
    __shared__ __align__(8) unsigned long long s_acc_full[2], s_acc_empty[2];
    __shared__ unsigned s_tmem_base;
    __shared__ unsigned s_prev_count;
    __shared__ __align__(16) int2 s_tab[4 * PF_BT];   // per epilogue warp, per token of the tile: row sum, scale bits
    __shared__ __align__(8) unsigned long long s_in[4];   // per epilogue warp: a fetched part of a split tile has landed

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // a kernel launched behind this one with programmatic dependent launch may be scheduled as CTAs here retire
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(pf_smem_raw) + 1023) & ~uintptr_t(1023));
    // activation stages start 1024-byte aligned (the 128-byte swizzle needs it); the packed weights follow
    const unsigned x_bytes = (unsigned)p.bt * PF_BK;
    auto stage_x = [&](int s) { return smem + (size_t)s * x_bytes; };
    auto stage_wp = [&](int pair) { return smem + (size_t)(p.ring * PF_PAIR) * x_bytes + (size_t)pair * (PF_PAIR * PF_WP_BYTES); };

    if (tid == 0) {
        for (int r = 0; r < p.ring; ++r) pf_mbar_init(&s_full[r], 1 + 4);
        for (int r = 0; r < p.wring; ++r) {
            pf_mbar_init(&s_full_w[r], 1);
            pf_mbar_init(&s_free_w[r], 4);
        }
        for (int r = 0; r < p.ring; ++r) pf_mbar_init(&s_done[r], 1);
        for (int w = 0; w < 4; ++w) pf_mbar_init(&s_in[w], 1);
        for (int b = 0; b < 2; ++b) {
            pf_mbar_init(&s_acc_full[b], 1);
            pf_mbar_init(&s_acc_empty[b], 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {   // all 512 tensor-memory columns: two 128 x bt s32 accumulators + the weight slots
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(pf_smem_u32(&s_tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem_base = s_tmem_base;

    const long long units = (long long)p.m_tiles * p.n_tiles * p.k_tiles;
    const int whole_k = p.whole_tiles ? p.k_tiles : 0;
    const long long u_begin = pf_range_start(units, (int)blockIdx.x, (int)gridDim.x, whole_k);
    const long long u_end = pf_range_start(units, (int)blockIdx.x + 1, (int)gridDim.x, whole_k);
    const PfSchedule sch = pf_schedule(u_begin, u_end, p.k_tiles);
    // Slices are handed between the roles in pairs: one barrier round per pair keeps the single MMA-issuing thread's
    // waits and commits off the critical path.  A pair never crosses a segment (the last one of an odd segment has one
    // slice), so that every role counts pairs and nothing else.

    // a cursor walks this CTA's pairs in segment order
    struct Cursor {
        int idx, n_tile, m_tile, kt, ke;
    };
    auto cursor_seg = [&](Cursor &c, int idx) {
        c.idx = idx;
        if (idx >= sch.n_seg) return;
        const PfSegment sg = pf_segment(sch, idx, p.k_tiles);
        c.n_tile = sg.tile / p.m_tiles;
        c.m_tile = sg.tile - c.n_tile * p.m_tiles;
        c.kt = sg.kb;
        c.ke = sg.ke;
    };
    auto advance = [&](Cursor &c) {
        if ((c.kt += PF_PAIR) >= c.ke) cursor_seg(c, c.idx + 1);
    };

    if (warp == 0) {
        // ===================== activation loads =====================
        if (elect_one()) {
            Cursor c;
            cursor_seg(c, 0);
            int xr = 0;
            unsigned phase = 1;                   // of the wait for the ring position's previous use
            asm volatile("griddepcontrol.wait;" ::: "memory");   // the int8 activations come from the quantiser grid
            while (c.idx < sch.n_seg) {
                if (!pf_mbar_wait(&s_done[xr], phase)) break;   // the MMAs of the pair that used these stages are done
                pf_mbar_expect_tx(&s_full[xr], PF_PAIR * x_bytes);
                // both slices in one box (one past the last k slice reads as zeros and meets no MMA)
                pf_tma_load_3d(stage_x(xr * PF_PAIR), &map_x, 0, c.m_tile * p.bt, c.kt, &s_full[xr]);
                if (++xr == p.ring) { xr = 0; phase ^= 1u; }
                advance(c);
            }
        }
    } else if (warp == pf_threads(GROUPS) / 32 - 1) {
        // ===================== packed-weight loads =====================
        // A thread of their own: with both kinds of loads the one producer was busy 600 clk a pair, more than the
        // MMAs of a tile of up to 128 tokens take.
        if (elect_one()) {
            Cursor c;
            cursor_seg(c, 0);
            int wr = 0;
            unsigned phase = 1;
            while (c.idx < sch.n_seg) {
                if (!pf_mbar_wait(&s_free_w[wr], phase)) break;   // the expanders hold the previous pair in registers
                pf_mbar_expect_tx(&s_full_w[wr], PF_PAIR * PF_WP_BYTES);
                pf_tma_load_2d(stage_wp(wr), &map_w, c.kt * (PF_BK / 4), c.n_tile * TILE_F, &s_full_w[wr]);
                if constexpr (PAIR)
                    pf_tma_load_2d(stage_wp(wr) + PF_PAIR * PF_WP_BYTES / 2, &map_w2, c.kt * (PF_BK / 4), c.n_tile * TILE_F, &s_full_w[wr]);
                if (++wr == p.wring) { wr = 0; phase ^= 1u; }
                advance(c);
            }
        }
    } else if (warp == 1) {
        // ===================== MMA issuer =====================
        if (elect_one()) {
            // this thread's instructions bound the kernel at narrow tiles: one wait, one commit and no index arithmetic beyond
            // two ring steps per pair
            int xr = 0;
            unsigned x_phase = 0;
            const unsigned tmem_a0 = tmem_base + 2u * (unsigned)p.bt, tmem_a_end = tmem_a0 + (unsigned)(p.aslots * PF_PAIR * PF_A_COLS);
            const unsigned long long b_step = x_bytes >> 4;   // a slice, in descriptor units
            unsigned tmem_a = tmem_a0;
            bool ok = true;
            const unsigned idesc = pf_idesc(p.bt);
            const unsigned long long b_desc0 = pf_smem_desc(pf_smem_u32(stage_x(0)));
            unsigned long long b_desc = b_desc0;
            for (int si = 0; si < sch.n_seg && ok; ++si) {
                const PfSegment sg = pf_segment(sch, si, p.k_tiles);
                const int buf = si & 1;
                if (!pf_mbar_wait(&s_acc_empty[buf], ((unsigned)(si >> 1) & 1u) ^ 1u)) break;   // epilogue drained this accumulator
                const unsigned tmem_d = tmem_base + (unsigned)(buf * p.bt);
                unsigned acc = 0;
                for (int left = sg.ke - sg.kb; left > 0; left -= PF_PAIR) {
                    if (!pf_mbar_wait(&s_full[xr], x_phase)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int ks = 0; ks < PF_BK / 32; ++ks) {  // 32 bytes of k per instruction: 8 columns / +2 16-byte units
                        pf_mma_i8_ts(tmem_d, tmem_a + 8u * ks, b_desc + 2ull * ks, idesc, acc);
                        acc = 1;
                    }
                    if (left > 1) {
#pragma unroll
                        for (int ks = 0; ks < PF_BK / 32; ++ks)
                            pf_mma_i8_ts(tmem_d, tmem_a + PF_A_COLS + 8u * ks, b_desc + b_step + 2ull * ks, idesc, 1u);
                    }
                    pf_commit(&s_done[xr]);   // TMA stages and the tensor-memory slot of the pair are free
                    if ((tmem_a += PF_PAIR * PF_A_COLS) == tmem_a_end) tmem_a = tmem_a0;
                    b_desc += PF_PAIR * b_step;
                    if (++xr == p.ring) { xr = 0; x_phase ^= 1u; b_desc = b_desc0; }
                }
                if (ok) pf_commit(&s_acc_full[buf]);
            }
        }
    } else if (warp < 2 + EXP_WARPS) {
        // ===================== weight expanders: GROUPS groups take the pairs in turn =====================
        // A thread owns one feature row of the tile: 32 packed bytes per slice become the 128 code
        // bytes of its tensor-memory lane.  (w >> 2j) & 0x03030303 is word j of a 16-wide group in
        // the transposed k order the activations were stored in.
        const int group = (warp - 2) / 4;
        const int quarter = warp & 3;            // the tensor-memory lanes this warp may touch
        const int row = quarter * 32 + lane;
        int n_pairs = 0;
        for (int si = 0; si < sch.n_seg; ++si) {
            const PfSegment sg = pf_segment(sch, si, p.k_tiles);
            n_pairs += (sg.ke - sg.kb + PF_PAIR - 1) / PF_PAIR;
        }
        const unsigned ta0 = tmem_base + ((unsigned)(quarter * 32) << 16) + 2u * (unsigned)p.bt;
        int slot = group % p.aslots;
        int first_wait = group;                  // the first pair of this group that has to wait for its slot
        while (first_wait < p.aslots) first_wait += GROUPS;
        // ring positions: packed weights, hand-over to the MMAs, the pair that used the slot before
        int wr = group, xr = group, dr = first_wait - p.aslots;
        unsigned w_phase = 0, d_phase = 0;
        for (int pp = group; pp < n_pairs; pp += GROUPS) {
            // expand both slices of the pair into registers first: this part does not need the
            // tensor-memory slot and overlaps the MMAs that still read it
            unsigned r[PF_PAIR][32];
            if (!pf_warp_wait(&s_full_w[wr], w_phase)) break;
            const unsigned char *src = stage_wp(wr) + row * (PF_PAIR * PF_BK / 4);
#pragma unroll
            for (int h = 0; h < PF_PAIR; ++h) {
                // 64-byte rows in the 64-byte swizzle: 16-byte piece i sits at i ^ ((row / 2) % 4)
                const uint4 w0 = *reinterpret_cast<const uint4 *>(src + (((2 * h) ^ ((row >> 1) & 3)) << 4));
                const uint4 w1 = *reinterpret_cast<const uint4 *>(src + (((2 * h + 1) ^ ((row >> 1) & 3)) << 4));
                const unsigned w[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    r[h][4 * g + 0] = w[g] & 0x03030303u;
                    r[h][4 * g + 1] = (w[g] >> 2) & 0x03030303u;
                    r[h][4 * g + 2] = (w[g] >> 4) & 0x03030303u;
                    r[h][4 * g + 3] = (w[g] >> 6) & 0x03030303u;
                }
            }
            __syncwarp();
            if (lane == 0) pf_mbar_arrive(&s_free_w[wr]);
            if ((wr += GROUPS) >= p.wring) { wr -= p.wring; w_phase ^= 1u; }
            if (pp >= p.aslots) {   // the MMAs that read this slot (pair pp - aslots) are done
                if (!pf_warp_wait(&s_done[dr], d_phase)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if ((dr += GROUPS) >= p.ring) { dr -= p.ring; d_phase ^= 1u; }
            }
            const unsigned ta = ta0 + (unsigned)(slot * PF_PAIR * PF_A_COLS);
            pf_tmem_st32(ta, r[0]);
            pf_tmem_st32(ta + PF_A_COLS, r[1]);   // (no MMA reads the second half when the pair is a single slice)
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) pf_mbar_arrive(&s_full[xr]);
            if ((xr += GROUPS) >= p.ring) xr -= p.ring;
            for (slot += GROUPS; slot >= p.aslots;) slot -= p.aslots;
        }
    } else {   // the four warps behind the expanders
        // ===================== epilogue (4 warps; a thread owns one feature row of the accumulator) =====================
        // Accumulator lanes are features, columns are tokens, so a warp's 32 lanes hold 32 consecutive
        // features of one token.  Each warp works on its own: a chunk of 32 tokens x 32 features goes
        // through the warp's private staging buffer ([token][feature], conflict-free) and leaves as one
        // TMA store; no barrier between the warps inside a tile.
        const int quarter = warp & 3;   // the tensor-memory lanes a warp may touch: 32 * (warp % 4)
        const int frow = quarter * 32 + lane;
        const bool epi_leader = tid == (2 + EXP_WARPS) * 32;
        unsigned char *my_stage = smem + PF_RING_BYTES + (size_t)quarter * (2 * PF_WARP_OUT_BYTES);   // two 4 KB buffers
        int sc = 0, n_staged = 0, n_in = 0;
        [[maybe_unused]] int n_xch = 0;
        // int -> fp32: 1.5 * 2^23 added to an integer below 2^22 in magnitude is that float with the integer in its low
        // bits, so one integer and one float addition convert exactly (|sum| <= 127 K); the conversion instruction runs
        // at a quarter of their rate and was a third of the epilogue
        const bool magic = p.K <= 32768;
        const int to_magic = magic ? 0x4b400000 : 0;
        bool ok = true;
        asm volatile("griddepcontrol.wait;" ::: "memory");   // row sums, scales and the zeroed counters come from the quantiser grid

        // the copy that read buffer (n_staged & 1) two sends ago has finished reading: its thread waited for it
        // right after the previous send, and the __syncwarp orders that before everybody's stores
        auto send_chunk = [&](const unsigned (&v)[32], int x, int yrow) {   // token-major, to y
            unsigned *st = reinterpret_cast<unsigned *>(my_stage + (size_t)(n_staged & 1) * PF_WARP_OUT_BYTES);
            ++n_staged;
            __syncwarp();
#pragma unroll
            for (int j = 0; j < 32; ++j) st[j * 32 + lane] = v[j];
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (elect_one()) {
                pf_tma_store_2d(&map_y, x, yrow, st);
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");   // the other buffer is free again
            }
        };
        // a part of a split tile goes to its slot feature-major: the thread's 32 values are 128
        // contiguous bytes (16-byte pieces XOR-swizzled so that the shared-memory accesses do not
        // collide); a warp's 32 rows are 4 KB contiguous in the slot
        auto send_partial = [&](const unsigned (&v)[32], int *slot_piece) {
            unsigned char *st = my_stage + (size_t)(n_staged & 1) * PF_WARP_OUT_BYTES;
            ++n_staged;
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<uint4 *>(st + lane * 128 + ((i ^ (lane & 7)) << 4)) = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (elect_one()) {
                asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(slot_piece + quarter * 32 * 32),
                             "r"(pf_smem_u32(st)), "r"(PF_WARP_OUT_BYTES)
                             : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
            }
        };
        // fetch this warp's 4 KB of another CTA's part into the staging buffer that is free, add it to v
        auto add_partial = [&](unsigned (&v)[32], const int *slot_piece) -> bool {
            unsigned char *st = my_stage + (size_t)(n_staged & 1) * PF_WARP_OUT_BYTES;
            __syncwarp();   // lane 0 has seen the last copy out of this buffer finish reading
            if (elect_one()) {
                pf_mbar_expect_tx(&s_in[quarter], PF_WARP_OUT_BYTES);
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                 pf_smem_u32(st)),
                             "l"(slot_piece + quarter * 32 * 32), "r"(PF_WARP_OUT_BYTES), "r"(pf_smem_u32(&s_in[quarter]))
                             : "memory");
            }
            const bool got = pf_warp_wait(&s_in[quarter], (unsigned)n_in & 1u);
            ++n_in;
            if (!got) return false;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint4 t = *reinterpret_cast<const uint4 *>(st + lane * 128 + ((i ^ (lane & 7)) << 4));
                v[4 * i + 0] += t.x;
                v[4 * i + 1] += t.y;
                v[4 * i + 2] += t.z;
                v[4 * i + 3] += t.w;
            }
            return true;
        };

        for (int si = 0; si < sch.n_seg && ok; ++si) {
            const PfSegment sg = pf_segment(sch, si, p.k_tiles);
            const int n_tile = sg.tile / p.m_tiles, m_tile = sg.tile % p.m_tiles;
            const int buf = sc & 1;
            const unsigned acc_ph = (unsigned)(sc >> 1) & 1u;
            ++sc;
            const bool whole = sg.kb == 0 && sg.ke == p.k_tiles;
            const int m0 = m_tile * p.bt;
            const int n = n_tile * TILE_F + (frow & (TILE_F - 1));
            const bool n_ok = n < p.N;
            const float ws = PAIR ? (quarter >= 2 ? p.w_scale2 : p.w_scale) : (n < p.seg_end0 ? p.w_scale : (n < p.seg_end1 ? p.seg_scale1 : p.seg_scale2));
            // per token of the tile: row sum and scale (each warp keeps its own copy), read back below as
            // broadcast 16-byte loads
            int2 *tab = s_tab + quarter * PF_BT;
            __syncwarp();
            for (int j = lane; j < p.bt; j += 32) {
                const int m = m0 + j;
                int2 e = make_int2(0, 0);
                if (m < p.M) {
                    e.x = to_magic - __ldg(p.rowsum + m);
                    e.y = __float_as_int(__ldg(p.a_scale + m));
                }
                tab[j] = e;
            }
            ok = pf_epi_all(pf_warp_wait(&s_acc_full[buf], acc_ph));   // the four warps go on, or give up, together
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned taddr = tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)(buf * p.bt);

            // a tile that is split between CTAs: publish this part, and whoever completes the
            // tile's k range adds the published parts to its own (integer sums: order is irrelevant)
            int c_lo = 0, c_hi = -1;   // the CTAs that hold parts of this tile (when it is split)
            bool finish = true;
            if (!whole) {
                // claim first: the CTA whose claim completes the tile's k range finishes the tile and need not
                // publish its own part; everyone else publishes and moves on
                const unsigned len = (unsigned)(sg.ke - sg.kb);
                if (epi_leader) s_prev_count = atomicAdd(p.counters + 2 * sg.tile, len);
                pf_epi_all(true);
                finish = s_prev_count + len == (unsigned)p.k_tiles;
                pf_epi_all(true);   // s_prev_count may be rewritten only after everyone has read it
                if (!finish) {
                    int *slot = p.slots + ((size_t)2 * blockIdx.x + (sg.tile != sch.t_first ? 1 : 0)) * (PF_BF * PF_BT);
#pragma unroll 1
                    for (int c = 0; c < p.bt / 32; ++c) {
                        unsigned r[32];
                        pf_tmem_ld32(taddr + (unsigned)c * 32, r);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        send_partial(r, slot + c * 32 * PF_BF);
                    }
                    if (elect_one()) {   // (the same thread of the warp every time: it owns the copies)
                        asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // this warp's pieces are written
                        asm volatile("fence.proxy.async;" ::: "memory");
                        __threadfence();
                    }
                    pf_epi_all(true);
                    if (epi_leader) {
                        __threadfence();
                        atomicAdd(p.counters + 2 * sg.tile + 1, len);
                    }
                } else {
                    // the other parts were claimed before this one, so their CTAs are running and publish
                    // without waiting for anybody: a short, bounded wait
                    if (epi_leader) {
                        const volatile unsigned *published = p.counters + 2 * sg.tile + 1;
                        unsigned seen = 0;
                        for (unsigned n = 0; n < PF_POLL_LIMIT; ++n) {
                            seen = *published;
                            if (seen + len == (unsigned)p.k_tiles) break;
                            __nanosleep(64);
                        }
                        if (seen + len != (unsigned)p.k_tiles) atomicOr(&g_prefill_error_flags, 2u);
                        __threadfence();
                    }
                    pf_epi_all(true);
                    const long long t_begin = (long long)sg.tile * p.k_tiles, t_end = t_begin + p.k_tiles;
                    c_lo = (int)(((t_begin + 1) * gridDim.x - 1) / units);   // owners of the tile's first and last unit
                    c_hi = (int)((t_end * gridDim.x - 1) / units);
                }
            }
            if (finish) {
#pragma unroll 1
                for (int c = 0; c < p.bt / 32; ++c) {
                    if (m0 + c * 32 >= p.M) break;   // warp-uniform
                    unsigned r[32];
                    pf_tmem_ld32(taddr + (unsigned)c * 32, r);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    for (int cc = c_lo; cc <= c_hi; ++cc) {
                        if (cc == (int)blockIdx.x) continue;
                        const long long t_begin = (long long)sg.tile * p.k_tiles, t_end = t_begin + p.k_tiles;
                        const long long cb = pf_range_start(units, cc, (int)gridDim.x), ce = pf_range_start(units, cc + 1, (int)gridDim.x);
                        if ((cb > t_begin ? cb : t_begin) >= (ce < t_end ? ce : t_end)) continue;   // an empty range
                        const int *piece = p.slots + ((size_t)2 * cc + (sg.tile != (int)(cb / p.k_tiles) ? 1 : 0)) * (PF_BF * PF_BT) + (c * 32) * PF_BF;
                        if (!add_partial(r, piece)) break;
                    }
                    const int m_left = p.M - (m0 + c * 32);   // tokens of this chunk that exist
                    if (p.acc_out) {   // parity-test output of the integer sums; kept out of the loop below so that it stays branch-free
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (n_ok && j < m_left) p.acc_out[(size_t)(m0 + c * 32 + j) * p.ldy + n] = (int)r[j] + tab[c * 32 + j].x - to_magic;
                    }
                    // loads first, arithmetic after: the warp issues in order, so a load placed next to
                    // its use would expose its latency 32 times
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        int4 e[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) e[i] = reinterpret_cast<const int4 *>(tab)[c * 16 + h * 8 + i];
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int j = h * 16 + 2 * i;
                            const int v0 = (int)r[j] + e[i].x, v1 = (int)r[j + 1] + e[i].z;
                            const float f0 = magic ? __fadd_rn(__int_as_float(v0), -12582912.0f) : (float)v0;
                            const float f1 = magic ? __fadd_rn(__int_as_float(v1), -12582912.0f) : (float)v1;
                            r[j] = __float_as_uint(__fmul_rn(f0, __fmul_rn(ws, __int_as_float(e[i].y))));
                            r[j + 1] = __float_as_uint(__fmul_rn(f1, __fmul_rn(ws, __int_as_float(e[i].w))));
                        }
                    }
                    if constexpr (PAIR) {
                        // Two exchange buffers and one barrier of the two warps per chunk: the gate warp writes a buffer
                        // again two chunks later, behind the barrier of the chunk between, which the up warp reaches
                        // after it has read the buffer.
                        float *xch = reinterpret_cast<float *>(smem + PF_RING_BYTES + (size_t)(quarter & 1) * (2 * PF_WARP_OUT_BYTES) +
                                                               (size_t)(n_xch & 1) * PF_WARP_OUT_BYTES);
                        ++n_xch;
                        if (quarter < 2) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) {
                                const float rl = fmaxf(__uint_as_float(r[j]), 0.0f);
                                xch[j * 32 + lane] = __fmul_rn(rl, rl);
                            }
                            asm volatile("bar.sync %0, 64;" ::"r"(2 + (quarter & 1)) : "memory");
                            continue;
                        }
                        asm volatile("bar.sync %0, 64;" ::"r"(2 + (quarter & 1)) : "memory");
#pragma unroll
                        for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__fmul_rn(__uint_as_float(r[j]), xch[j * 32 + lane]));
                    }
                    if (p.tma_store) {
                        send_chunk(r, n_tile * TILE_F + (PAIR ? (quarter & 1) : quarter) * 32, m0 + c * 32);
                    } else if (p.n_peers) {
                        // this GPU's column slice, stored into every GPU's full-width output: a warp writes 128
                        // contiguous bytes per token row and destination
                        for (int pr = 0; pr < p.n_peers; ++pr) {
                            float *ycol = p.y_peers[pr] + (size_t)(m0 + c * 32) * p.ldy + n;
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (n_ok && j < m_left) ycol[(size_t)j * p.ldy] = __uint_as_float(r[j]);
                        }
                    } else {
                        float *ycol = p.y + (size_t)(m0 + c * 32) * p.ldy + n;
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (n_ok && j < m_left) ycol[(size_t)j * p.ldy] = __uint_as_float(r[j]);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) pf_mbar_arrive(&s_acc_empty[buf]);
        }
        __syncwarp();
        if (elect_one()) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // shared memory outlives the stores
    }

    // everyone meets here, also after a wait that gave up, so that tensor memory is always freed
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    }
}

bitnet_status_t prefill_take_error_flags(unsigned *flags)
{
    unsigned v = 0, zero = 0;
    BITNET_CUDA(cudaMemcpyFromSymbol(&v, g_prefill_error_flags, sizeof(v)));
    if (v) BITNET_CUDA(cudaMemcpyToSymbol(g_prefill_error_flags, &zero, sizeof(zero)));
    *flags = v;
    return BITNET_OK;
}

// ---- host side --------------------------------------------------------------------------------------

bool prefill_supports(size_t M, size_t K, size_t N)
{
    return M >= 1 && N >= 1 && K >= 128 && K % 128 == 0 && M <= (1u << 24) && N <= (1u << 24) && K <= (1u << 20);
}

// K a multiple of 64 still has rows of packed weights that start on 16 bytes; the second half of the last slice lies past the
// end of a row and is filled with zeros by TMA (code 0: whatever the activation bytes there are, they add nothing).
bool prefill_supports_tail(size_t M, size_t K, size_t N)
{
    return M >= 1 && N >= 1 && K >= 64 && K % 64 == 0 && M <= (1u << 24) && N <= (1u << 24) && K <= (1u << 20);
}

static size_t pf_pitch(size_t K) { return align_up(K, PF_BK); }   // bytes between quantised rows
static size_t pf_q_bytes(size_t M, size_t K) { return align_up(M * pf_pitch(K), 256); }
static size_t pf_vec_bytes(size_t M) { return align_up(M * 4, 256); }

// How a problem is cut: tokens per tile, whether tiles may be split between CTAs, and the grid.
struct PfPlan {
    int bt;
    bool whole_tiles;
    size_t tiles, grid;
};
// Depths of the rings for a tile of bt tokens.  Tensor memory: whatever two accumulators of bt columns leave holds
// expanded pairs (2 at 192 tokens, 5 at 64).  Shared memory: enough activation pairs to cover a fetch from L2, the rest
// for packed weights, whose bytes in flight are what a narrow tile lives on (5 pairs of 8 KB at 192 tokens, 13 at 64).
struct PfRings {
    int ring, wring, aslots;
};
static PfRings pf_rings(int bt)
{
    PfRings r;
    r.ring = bt > 128 ? 3 : (bt > 64 ? 4 : (bt > 32 ? 5 : 8));
    r.wring = (int)((PF_RING_BYTES - (size_t)r.ring * PF_PAIR * bt * PF_BK) / (PF_PAIR * PF_WP_BYTES));
    if (r.wring > PF_MAX_WRING) r.wring = PF_MAX_WRING;
    // never more slots than ring positions: an expander that has seen the MMAs of pair pp - aslots reports pair pp on the
    // barrier that pair pp - ring used, whose phase has to be over by then
    r.aslots = (512 - 2 * bt) / (PF_PAIR * PF_A_COLS);
    if (r.aslots > r.ring) r.aslots = r.ring;
    return r;
}
static size_t pf_tiles(size_t M, size_t N, int bt, bool pair = false)
{
    const size_t f = pair ? PF_BF / 2 : PF_BF;
    return ((M + bt - 1) / bt) * ((N + f - 1) / f);
}
// Estimated device cycles of a plan, from timings of 23 shapes (16 to 2048 tokens, K 128 to 8192) at every tile and both ways
// of dealing: a k slice costs what its MMAs take (2.22 clk a token) and never less than 290; finishing a tile costs what is
// hidden behind the next tile's MMAs unless K is short (per 32 tokens 1400 and 1700 around it where three expander groups leave
// the epilogue fewer registers, 1000 and 2500 above 128 tokens; the gate/up pair writes half as much), and is seen once at the
// end; splitting tiles between CTAs costs another 4500 + 80 a token, so it pays only when whole tiles leave most of a wave idle
// (256x8192x28672, 3.03 waves of 128 tokens: 49.7 against 52.7 us; 2048x2560x6912, 4.74 of 160: 49.9 against 40.0).  Against one
// line for all tiles, which took 128 tokens where K is short: 2048x128x20000 69.7 -> 59.0 us, 2048x1024x32768 118.8 -> 100.4,
// 300x1024x32768 28.5 -> 23.6, 2048x640x5000 27.3 -> 22.9, 512x512x16384 22.3 -> 19.1, 2048x2560x6912 41.7 -> 40.0.
static double pf_plan_cost(size_t M, size_t K, size_t N, int bt, bool whole, size_t sms, bool pair)
{
    const double k = (double)((K + PF_BK - 1) / PF_BK), tiles = (double)pf_tiles(M, N, bt, pair);
    const double per_slice = 2.22 * bt > 290.0 ? 2.22 * bt : 290.0;
    const double epilogue = 1000.0 * (bt / 32);
    const double between = pair ? 700.0 + epilogue : (pf_groups(bt) == 2 ? 2500.0 + 1000.0 * (bt / 32) : 1700.0 + 1400.0 * (bt / 32));
    const double tile = k * per_slice > between ? k * per_slice : between;
    if (tiles <= (double)sms) return k * per_slice + epilogue;
    if (whole) return (double)((size_t)((tiles + sms - 1) / sms)) * tile + epilogue;
    return tiles / (double)sms * tile + epilogue + 4500.0 + 80.0 * bt;
}
// At most 128 tokens are dealt in whole tiles (splitting gains 4 % at best there, 16x8192x28672, and needs 28 MB of scratch).
static bool pf_may_split(size_t M) { return M > 128; }
static PfPlan pf_plan(size_t M, size_t K, size_t N, bool pair)
{
    const size_t sms = (size_t)device_sm_count();
    static const int env_bt = getenv("BITNET_PREFILL_BT") ? atoi(getenv("BITNET_PREFILL_BT")) : 0;
    static const int env_mode = getenv("BITNET_PREFILL_WHOLE") ? atoi(getenv("BITNET_PREFILL_WHOLE")) : -1;
    PfPlan best = {};
    double best_cost = 0.0;
    for (int bt = PF_BT; bt >= (pf_may_split(M) ? 64 : 32); bt -= 32) {
        if (env_bt >= 32 && env_bt <= PF_BT && env_bt % 32 == 0 && bt != env_bt) continue;
        for (int whole = 1; whole >= 0; --whole) {
            const bool can_split = pf_may_split(M) && !pair;
            if (can_split ? env_mode >= 0 && whole != (env_mode != 0) : whole == 0) continue;
            const double cost = pf_plan_cost(M, K, N, bt, whole != 0, sms, pair);
            if (best.bt == 0 || cost < best_cost) {
                best.bt = bt;
                best.whole_tiles = whole != 0;
                best_cost = cost;
            }
        }
    }
    if (best.bt == 0) { best.bt = PF_BT; best.whole_tiles = true; }
    best.tiles = pf_tiles(M, N, best.bt, pair);
    const size_t units = best.tiles * ((K + PF_BK - 1) / PF_BK);
    if (best.tiles <= sms) { best.grid = best.tiles; best.whole_tiles = true; }
    else best.grid = best.whole_tiles ? sms : (units < sms ? units : sms);
    return best;
}
static size_t pf_counter_bytes(size_t M, size_t N) { return align_up(pf_tiles(M, N, 64) * 8, 256); }   // claimed, published (largest tile count)

// Two to sixteen tokens: the weight-streaming kernel or this one.  Estimates in ns from both kernels at five token counts and
// twelve shapes (K 512 to 16384, N 2560 to 128256).  The weight-streaming kernel runs its steps on mma.sync and a CTA meets
// many short blocks where N is large and K small: 16x8192x28672 40.4 us against 26.0 here, 16x2560x128256 58.0 / 30.4,
// 8x2560x128256 40.9 / 33.0, 4x1024x32768 14.7 / 10.6; it stays ahead at 8x8192x28672 (18.2 / 27.0) and in the small layers
// (16x2560x2560 8.9 / 9.6).  The margins keep calls there whose times are close: its launches cost the host less.
bool prefill_beats_decode(size_t M, size_t K, size_t N)
{
    if (M < 2 || M > 16 || !prefill_supports(M, K, N)) return false;
    const size_t sms = (size_t)device_sm_count();
    const double blocks = (double)(((N + 15) / 16 + sms - 1) / sms);
    // tiles of 32 tokens in whole waves (pf_plan_cost has the cost between wider tiles; these two estimates are fitted to each other)
    const double k = (double)(K / PF_BK), tiles = (double)pf_tiles(M, N, 32);
    const double chain = tiles <= (double)sms ? k * 290.0 : (double)((size_t)((tiles + sms - 1) / sms)) * (k * 290.0 > 1700.0 ? k * 290.0 : 1700.0);
    const double here = 6500.0 + (chain + 1000.0) / 1.9;
    const double decode = M > 8 ? 6500.0 + blocks * (150.0 + 300.0 * (double)K / 1024.0) : 7000.0 + blocks * (450.0 + 55.0 * (double)K / 1024.0);
    return here * (M > 8 ? 1.05 : 1.25) < decode;
}

size_t prefill_workspace_bytes(size_t M, size_t K, size_t N)
{
    // int8 activations, fp32 scales, int32 row sums; where tiles may be split their counters and two partial tiles per CTA
    return pf_q_bytes(M, K) + 2 * pf_vec_bytes(M) + (pf_may_split(M) ? pf_counter_bytes(M, N) + 2 * (size_t)device_sm_count() * PF_SLOT_BYTES : 0);
}

// ---- widths that are no multiple of 64 ----

static bool pf_supports_any(size_t M, size_t K, size_t N) { return M >= 1 && N >= 1 && K >= 1 && M <= (1u << 24) && N <= (1u << 24) && K <= (1u << 20); }
static size_t repack_bytes(size_t N, size_t K) { return align_up(N * (pf_pitch(K) / 4), 256); }
size_t repack_workspace_bytes(size_t M, size_t K, size_t N) { return repack_bytes(N, K) + prefill_workspace_bytes(M, K, N); }
// The three launches (copy of the packed rows, quantiser, GEMM) take 9 to 12 us up to a few million weights.  The generic
// kernel walks a row code by code: 3 us and 13 ns per k for one token, 5 ns per k and token from there on, whatever N up to
// the 9472 warps it runs (1x1001x2100 16.4 us, 8 tokens 48, 40 tokens 220, here 9.7 / 10.2 / 9.8; 1x501x1001 10.3 on both),
// more beyond (1x333x10000 16.9 against 9.7; 1x3114x23861 here 35.9).
bool repack_pays(size_t M, size_t K, size_t N)
{
    return pf_supports_any(M, K, N) && ((double)K * (double)(M + 2) > 2500.0 || (double)N * (double)K > 2.0e6);
}

static bitnet_status_t encode_map_nd(CUtensorMap *map, CUtensorMapDataType dtype, cuuint32_t rank, const void *base, const cuuint64_t *dims,
                                     const cuuint64_t *strides, const cuuint32_t *box, CUtensorMapSwizzle swizzle)
{
    const cuuint32_t elem[3] = {1, 1, 1};
    // the driver entry point is looked up through the runtime, so the library does not link
    // against libcuda and still loads on a machine without a driver
    typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                 const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        BITNET_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
        if (!fn || qres != cudaDriverEntryPointSuccess)
            return fail(BITNET_ERR_CUDA_DRIVER, "cuTensorMapEncodeTiled is not available from this driver");
        encode = reinterpret_cast<EncodeFn>(fn);
    }
    const CUresult r = encode(map, dtype, rank, const_cast<void *>(base), dims, strides, box, elem,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(BITNET_ERR_CUDA_DRIVER, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return BITNET_OK;
}

static bitnet_status_t encode_map(CUtensorMap *map, const void *base, uint64_t inner, uint64_t rows, uint64_t row_stride_bytes,
                                  uint32_t box_inner, uint32_t box_rows, CUtensorMapSwizzle swizzle,
                                  CUtensorMapDataType dtype = CU_TENSOR_MAP_DATA_TYPE_UINT8)
{
    const cuuint64_t dims[2] = {inner, rows};
    const cuuint64_t strides[1] = {row_stride_bytes};
    const cuuint32_t box[2] = {box_inner, box_rows};
    return encode_map_nd(map, dtype, 2, base, dims, strides, box, swizzle);
}

// The quantised rows as slices of 128 k: a box holds `rows` tokens of PF_PAIR consecutive slices, 128-byte swizzle.
static bitnet_status_t encode_map_slices(CUtensorMap *map, const void *base, uint64_t row_bytes, uint64_t rows, uint32_t box_rows)
{
    const cuuint64_t dims[3] = {PF_BK, rows, row_bytes / PF_BK};
    const cuuint64_t strides[2] = {row_bytes, PF_BK};
    const cuuint32_t box[3] = {PF_BK, box_rows, PF_PAIR};
    return encode_map_nd(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

// The same encoder for the other tensor-core kernel of the library (uint8 elements).
bitnet_status_t tensor_map_2d(void *map_out, const void *base, uint64_t inner, uint64_t rows, uint64_t row_stride_bytes,
                              uint32_t box_inner, uint32_t box_rows, int swizzle_128b)
{
    return encode_map(static_cast<CUtensorMap *>(map_out), base, inner, rows, row_stride_bytes, box_inner, box_rows,
                      swizzle_128b ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE);
}

bitnet_status_t launch_prefill(const ForwardArgs &a, void *workspace, size_t workspace_bytes, cudaStream_t stream, bool repack)
{
    if (!(repack ? pf_supports_any(a.M, a.K, a.N) && !a.wp2 : prefill_supports_tail(a.M, a.K, a.N)))
        return fail(BITNET_ERR_UNSUPPORTED_OPERATION, "tensor-core path needs K %% 64 == 0 (M=%zu K=%zu N=%zu)", a.M, a.K, a.N);
    if (workspace_bytes < (repack ? repack_workspace_bytes(a.M, a.K, a.N) : prefill_workspace_bytes(a.M, a.K, a.N)))
        return fail(BITNET_ERR_WORKSPACE, "workspace too small for the tensor-core path");
    if (!repack && ((reinterpret_cast<uintptr_t>(a.wp) & 15) || (reinterpret_cast<uintptr_t>(a.x) & 15)))
        return fail(BITNET_ERR_INVALID_CONFIG, "packed weights and activations must be 16-byte aligned");
    if (a.wp2 && ((reinterpret_cast<uintptr_t>(a.wp2) & 15) || a.n_seg || a.n_peers || a.acc_out))
        return fail(BITNET_ERR_INVALID_CONFIG, "the gate/up pair takes 16-byte aligned weights and no stacked matrices, peer outputs or accumulator output");
    if (!repack && a.q_out && (reinterpret_cast<uintptr_t>(a.q_out) & 15)) return fail(BITNET_ERR_INVALID_CONFIG, "q_out must be 16-byte aligned");

    char *ws = static_cast<char *>(workspace);
    const size_t pitch = pf_pitch(a.K);
    const uint8_t *wp = a.wp;
    size_t w_row_bytes = a.K / 4;          // bytes of codes per packed row; what a box reads past them is zero
    if (repack) {
        uint8_t *rows = reinterpret_cast<uint8_t *>(ws);
        ws += repack_bytes(a.N, a.K);
        const size_t blocks = (a.N * (pitch / 16) + 255) / 256, cap = (size_t)device_sm_count() * 16;
        repack_rows_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, stream>>>(a.wp, (a.N * a.K + 3) / 4, a.N, a.K, pitch / 4, rows);
        BITNET_TRY(check_launch("repack_rows_kernel"));
        wp = rows;
        w_row_bytes = pitch / 4;
    }
    int8_t *q_perm = reinterpret_cast<int8_t *>(ws);
    ws += pf_q_bytes(a.M, a.K);
    float *a_scale = reinterpret_cast<float *>(ws);
    ws += pf_vec_bytes(a.M);
    int *rowsum = reinterpret_cast<int *>(ws);
    ws += pf_vec_bytes(a.M);
    unsigned *counters = reinterpret_cast<unsigned *>(ws);
    ws += pf_counter_bytes(a.M, a.N);
    int *slots = reinterpret_cast<int *>(ws);

    const bool pair = a.wp2 != nullptr;
    const PfPlan plan = pf_plan(a.M, a.K, a.N, pair);
    const int n_counters = plan.whole_tiles ? 0 : 2 * (int)plan.tiles;   // only split tiles are counted
    // The GEMM fetches its weights before it waits for the quantiser.  Rows that the launch in front of the quantiser copied
    // are there by then only if the quantiser itself started after that launch: no programmatic start behind a copy.
    const uint32_t q_flags = repack ? a.flags & ~BITNET_FLAG_PDL : a.flags;
    if (a.pre) {   // residual add and normalisation ride in the quantiser
        RowsOut rows = {};
        rows.q_perm = q_perm; rows.pitch = pitch; rows.rowsum = rowsum; rows.a_scale = a_scale;
        rows.counters = counters; rows.n_counters = n_counters;
        BITNET_TRY(launch_quantize_rows_glued(a.x, a.M, a.K, a.pre, rows, a.q_out, a.a_scale_out, q_flags, stream));
    } else {
        cudaLaunchConfig_t qcfg = {};
        cudaLaunchAttribute qattr[1];
        const bool short_rows = a.K / 16 <= 256;
        qcfg.gridDim = dim3((unsigned)a.M);
        qcfg.blockDim = dim3(short_rows ? 128 : 256);
        qcfg.stream = stream;
        qcfg.attrs = qattr;
        if (q_flags & BITNET_FLAG_PDL) {   // the caller chains launches: start while the previous kernel drains
            qattr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            qattr[0].val.programmaticStreamSerializationAllowed = 1;
            qcfg.numAttrs = 1;
        }
        if (repack) {
            qcfg.blockDim = dim3(256);
            BITNET_CUDA(cudaLaunchKernelEx(&qcfg, quantize_rows_pad_kernel, a.x, a.K, pitch, q_perm, a_scale, rowsum, a.q_out, a.a_scale_out,
                                           counters, n_counters));
        } else if (short_rows)
            BITNET_CUDA(cudaLaunchKernelEx(&qcfg, quantize_rows_perm_kernel<128>, a.x, a.K, pitch, q_perm, a_scale, rowsum, a.q_out,
                                           a.a_scale_out, counters, n_counters));
        else
            BITNET_CUDA(cudaLaunchKernelEx(&qcfg, quantize_rows_perm_kernel<256>, a.x, a.K, pitch, q_perm, a_scale, rowsum, a.q_out,
                                           a.a_scale_out, counters, n_counters));
    }
    BITNET_TRY(check_launch("quantize_rows_perm_kernel"));

    CUtensorMap map_x, map_w, map_w2, map_y;
    BITNET_TRY(encode_map_slices(&map_x, q_perm, pitch, a.M, (uint32_t)plan.bt));
    // a pair of slices per box: 64-byte rows (half the requests of 32-byte ones; columns past K read as zero and meet no MMA)
    BITNET_TRY(encode_map(&map_w, wp, w_row_bytes, a.N, w_row_bytes, PF_PAIR * PF_BK / 4, pair ? PF_BF / 2 : PF_BF, CU_TENSOR_MAP_SWIZZLE_64B));

    if (pair) BITNET_TRY(encode_map(&map_w2, a.wp2, w_row_bytes, a.N, w_row_bytes, PF_PAIR * PF_BK / 4, PF_BF / 2, CU_TENSOR_MAP_SWIZZLE_64B));
    else map_w2 = map_w;

    PrefillParams p = {};
    p.w_scale2 = a.w_scale2;
    p.seg_end0 = p.seg_end1 = 0x7fffffff;
    if (a.n_seg > 0) {
        p.seg_end0 = (int)a.seg_end[0]; p.seg_scale1 = a.seg_scale[0];
        if (a.n_seg > 1) { p.seg_end1 = (int)a.seg_end[1]; p.seg_scale2 = a.seg_scale[1]; }
    }
    p.y = a.y; p.acc_out = a.acc_out; p.a_scale = a_scale; p.rowsum = rowsum; p.w_scale = a.w_scale;
    p.slots = slots; p.counters = counters;
    p.M = (int)a.M; p.K = (int)a.K; p.N = (int)a.N; p.ldy = a.ldy ? a.ldy : a.N;
    p.bt = plan.bt;
    const PfRings rings = pf_rings(plan.bt);
    p.ring = rings.ring; p.wring = rings.wring; p.aslots = rings.aslots;
    p.whole_tiles = plan.whole_tiles ? 1 : 0;
    p.m_tiles = (int)((a.M + plan.bt - 1) / plan.bt);
    const int tile_f = pair ? PF_BF / 2 : PF_BF;
    p.n_tiles = (int)((a.N + tile_f - 1) / tile_f);
    p.k_tiles = (int)(pitch / PF_BK);
    // y leaves through TMA when its rows are 16-byte aligned; any other output takes plain stores
    p.tma_store = ((reinterpret_cast<uintptr_t>(a.y) & 15) == 0 && (p.ldy % 4) == 0) ? 1 : 0;
    p.n_peers = a.n_peers;
    for (int r = 0; r < a.n_peers && r < 8; ++r) p.y_peers[r] = a.y_peers[r];
    if (a.n_peers) {
        if (a.acc_out) return fail(BITNET_ERR_INVALID_CONFIG, "peer outputs and acc_out exclude each other");
        p.tma_store = 0;   // peer memory takes plain stores
    }
    if (p.tma_store)
        BITNET_TRY(encode_map(&map_y, a.y, a.N, a.M, p.ldy * 4, 32, 32, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_DATA_TYPE_FLOAT32));
    else
        map_y = map_w;   // unused by the kernel

    {   // once per device, under a lock: host threads launch concurrently (one per stream)
        static std::mutex mu;
        static bool attr_set[64] = {false};
        int dev = 0;
        BITNET_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lock(mu);
        if (dev < 0 || dev >= 64 || !attr_set[dev]) {
            for (auto kernel : {prefill_gemm_kernel<2, false>, prefill_gemm_kernel<3, false>, prefill_gemm_kernel<2, true>, prefill_gemm_kernel<3, true>})
                BITNET_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PF_SMEM));
            if (dev >= 0 && dev < 64) attr_set[dev] = true;
        }
    }
    const int grid = (int)plan.grid;
    // programmatic dependent launch: the GEMM's prologue and weight fetch overlap the quantiser's tail
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)pf_threads(pf_groups(plan.bt)));
    cfg.dynamicSmemBytes = PF_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto kernel = pf_groups(plan.bt) == 2 ? (pair ? prefill_gemm_kernel<2, true> : prefill_gemm_kernel<2, false>)
                                          : (pair ? prefill_gemm_kernel<3, true> : prefill_gemm_kernel<3, false>);
    BITNET_CUDA(cudaLaunchKernelEx(&cfg, kernel, map_x, map_w, map_w2, map_y, p));
    return check_launch("prefill_gemm_kernel");
}

}  // namespace bitnet
