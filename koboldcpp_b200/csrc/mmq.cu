// mmq.cu -- (a7) prefill GEMM over GGUF block formats on the 5th-generation tensor cores (tcgen05 + TMEM).
//
//   dst[n][m] = sum_k W[m][k] * X[n][k],  W quantised (Q4_0, Q8_0, Q4_K, Q5_K, Q6_K), X f32, any N.
//
// Replaces ggml_cuda_op_mul_mat_q / mul_mat_q<type,...> (mma.sync m16n8k32 int8 tiles with ALU-side unpack and two CTA
// barriers per 128-K half step, ggml/src/ggml-cuda/mmq.cuh:2495-2905) and the cuBLAS dequantise-then-GEMM
// fallback that koboldcpp uses by default (ggml-cuda.cu:1186-1284: whole-tensor dequant to f16 in HBM, then cublasGemmEx).
//
// B200 design (the one dense contraction of the path: tensor-pipe bound once N is a few hundred):
//   * weights are dequantised ON THE FLY into bf16 operand tiles in shared memory (never to HBM), in the 128-byte-swizzled K-major layout
//     the tensor core reads; activations are converted f32 -> bf16 once per call by a pre-pass;
//   * tcgen05.mma (kind::f16, bf16 x bf16 -> f32), the f32 accumulators in TMEM; a shared-memory ring with mbarrier full/empty pairs,
//     tcgen05.commit releases a stage when the MMAs that read it retire -- no CTA-wide barrier in the K loop.
// mmq_pair.cuh holds the kernel of almost every call (K a multiple of 256, dense rows); here are mmq_tc_kernel for rows of 32-value blocks with other
// K, a dense kernel for stacks at odd strides, MUL_MAT_ID's grouping, and the entry points.
// Why bf16 and not kind::i8: per-32 (per-16 for Q6_K) group scales would force a TMEM read-out after every K=32 MMA,
// which is epilogue-bound; bf16 operands keep the whole K loop inside the tensor pipe.  Activations carry 8 mantissa bits
// (q8_1 carries 7 + sign per 32-block), weights are rounded once from their exact f32 dequantised value.
#include "tcgen05.cuh"

#include <cuda_bf16.h>

#include <atomic>
#include <cstdlib>
#include <mutex>

namespace b200 {

constexpr int MQ_BM = 128, MQ_BK = 64, MQ_STAGES = 4;
constexpr int MQ_PRODUCERS = 128;              // threads; warps 0..3
constexpr int MQ_THREADS = MQ_PRODUCERS + 32;  // + the MMA warp

// ---------------------------------------------------------------- raw block loads from 2-byte aligned global addresses
template <int NW>
__device__ __forceinline__ void ld_words(const unsigned char *p, unsigned (&w)[NW]) {
    const uintptr_t a = (uintptr_t)p;
    const unsigned *q = reinterpret_cast<const unsigned *>(a & ~(uintptr_t)3);
    const unsigned sh = (unsigned)(a & 3) * 8;
    if (sh == 0) {
#pragma unroll
        for (int i = 0; i < NW; i++) w[i] = __ldg(q + i);
    } else {
        unsigned prev = __ldg(q);
#pragma unroll
        for (int i = 0; i < NW; i++) {
            const unsigned nxt = __ldg(q + i + 1);
            w[i] = __funnelshift_r(prev, nxt, sh);
            prev = nxt;
        }
    }
}
__device__ __forceinline__ float f16lo(unsigned w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xffff))); }
__device__ __forceinline__ float f16hi(unsigned w) { return __half2float(__ushort_as_half((unsigned short)(w >> 16))); }
__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const unsigned *>(&h);
}

// ---------------------------------------------------------------- 64 consecutive weights of one row -> 32 packed bf16x2 words
// Formats with blocks of 32 values.  Arithmetic follows dequantize_row_* (ggml-quants.c:1523, 1617) in f32; the result is rounded once to bf16.
#define BYTE_OF(w, i) (((w)[(i) >> 2] >> (8 * ((i) & 3))) & 0xffu)

// bytes of the 256-value group a K-step of 64 belongs to (one K-quant super-block, or 8 q4_0 / q8_0 blocks)
__host__ __device__ constexpr int group256_bytes(int t) { return type_block_bytes(t) * 256 / type_block_values(t); }

template <int TYPE>
struct Dequant64;  // run(g, c, o): g -> first byte of the 256-value group, c = 64-value chunk 0..3 inside it

template <>
struct Dequant64<B200_TYPE_Q4_0> {
    static __device__ __forceinline__ void run(const unsigned char *g, int c, unsigned (&o)[32]) {
        unsigned w[9];
        ld_words<9>(g + c * 2 * Q4_0_BYTES, w);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const float d = __half2float(__ushort_as_half((unsigned short)(BYTE_OF(w, 18 * b) | (BYTE_OF(w, 18 * b + 1) << 8))));
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
                const unsigned q0 = BYTE_OF(w, 18 * b + 2 + j), q1 = BYTE_OF(w, 18 * b + 3 + j);
                o[16 * b + j / 2]     = pack_bf16(d * (float)((int)(q0 & 15) - 8), d * (float)((int)(q1 & 15) - 8));
                o[16 * b + 8 + j / 2] = pack_bf16(d * (float)((int)(q0 >> 4) - 8), d * (float)((int)(q1 >> 4) - 8));
            }
        }
    }
};

// Q4_1 / Q5_0 / Q5_1 (dequantize_row_q4_1 / q5_0 / q5_1, ggml-quants.c:1543-1615): x d + m, or (x5 - 16) d; the fifth bit of value j
// is bit j of qh.  Byte offsets inside a block: d 0, [m 2], [qh 4 bytes], qs 16 bytes.
template <int TYPE>
struct LegacyLayout {
    static constexpr bool HAS_M = TYPE != B200_TYPE_Q5_0, HAS_H = TYPE != B200_TYPE_Q4_1;
    static constexpr int BB = type_block_bytes(TYPE), QH = 2 + (HAS_M ? 2 : 0), QS = QH + (HAS_H ? 4 : 0);
};
template <int TYPE>
struct Dequant64Legacy {
    static __device__ __forceinline__ void run(const unsigned char *g, int c, unsigned (&o)[32]) {
        using L = LegacyLayout<TYPE>;
        constexpr int NWL = (2 * L::BB + 3) / 4;
        unsigned w[NWL];
        ld_words<NWL>(g + c * 2 * L::BB, w);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const int base = L::BB * b;
            const float d = __half2float(__ushort_as_half((unsigned short)(BYTE_OF(w, base) | (BYTE_OF(w, base + 1) << 8))));
            float m = 0.f;
            if constexpr (L::HAS_M) m = __half2float(__ushort_as_half((unsigned short)(BYTE_OF(w, base + 2) | (BYTE_OF(w, base + 3) << 8))));
            unsigned qh = 0;
            if constexpr (L::HAS_H) qh = BYTE_OF(w, base + L::QH) | (BYTE_OF(w, base + L::QH + 1) << 8) | (BYTE_OF(w, base + L::QH + 2) << 16) | (BYTE_OF(w, base + L::QH + 3) << 24);
            if constexpr (TYPE == B200_TYPE_Q5_0) m = d * -16.0f;
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
                const unsigned q0 = BYTE_OF(w, base + L::QS + j), q1 = BYTE_OF(w, base + L::QS + 1 + j);
                const unsigned l0 = (q0 & 15) | (((qh >> j) & 1u) << 4), l1 = (q1 & 15) | (((qh >> (j + 1)) & 1u) << 4);
                const unsigned h0 = (q0 >> 4) | (((qh >> (16 + j)) & 1u) << 4), h1 = (q1 >> 4) | (((qh >> (17 + j)) & 1u) << 4);
                o[16 * b + j / 2]     = pack_bf16(d * (float)l0 + m, d * (float)l1 + m);
                o[16 * b + 8 + j / 2] = pack_bf16(d * (float)h0 + m, d * (float)h1 + m);
            }
        }
    }
};
template <> struct Dequant64<B200_TYPE_Q4_1> : Dequant64Legacy<B200_TYPE_Q4_1> {};
template <> struct Dequant64<B200_TYPE_Q5_0> : Dequant64Legacy<B200_TYPE_Q5_0> {};
template <> struct Dequant64<B200_TYPE_Q5_1> : Dequant64Legacy<B200_TYPE_Q5_1> {};

// IQ4_NL (dequantize_row_iq4_nl, ggml-quants.c:3743): dl * level[nibble], the levels looked up eight at a
// time with the byte permute unit (iq4_levels, b200_common.cuh).  q(k) must yield byte k of the sub-block's 16 nibble bytes;
// o16[0..7] receive values 0..15 (low nibbles), o16[8..15] values 16..31 (high nibbles).
template <int K> __device__ __forceinline__ float s8_f(unsigned x) { return (float)(int)(signed char)((x >> (8 * K)) & 0xffu); }
template <typename QFn>
__device__ __forceinline__ void iq4_unpack32(QFn q, float dl, unsigned *o16) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const unsigned w = q(4 * i) | (q(4 * i + 1) << 8) | (q(4 * i + 2) << 16) | (q(4 * i + 3) << 24);
        unsigned lo, hi;
        iq4_levels(w, lo, hi);
        o16[2 * i]         = pack_bf16(dl * s8_f<0>(lo), dl * s8_f<1>(lo));
        o16[2 * i + 1]     = pack_bf16(dl * s8_f<2>(lo), dl * s8_f<3>(lo));
        o16[8 + 2 * i]     = pack_bf16(dl * s8_f<0>(hi), dl * s8_f<1>(hi));
        o16[8 + 2 * i + 1] = pack_bf16(dl * s8_f<2>(hi), dl * s8_f<3>(hi));
    }
}
// 6-bit scale of IQ4_XS sub-block ib, minus 32: nibble ib of scales_l (as one word) | bits 2ib, 2ib+1 of scales_h << 4
__device__ __forceinline__ float iq4xs_scale(unsigned sl, unsigned sh, int ib) {
    return (float)((int)(((sl >> (4 * ib)) & 0xFu) | (((sh >> (2 * ib)) & 3u) << 4)) - 32);
}
template <>
struct Dequant64<B200_TYPE_IQ4_NL> {
    static __device__ __forceinline__ void run(const unsigned char *g, int c, unsigned (&o)[32]) {
        unsigned w[9];
        ld_words<9>(g + c * 2 * IQ4_NL_BYTES, w);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const int base = IQ4_NL_BYTES * b;
            const float d = __half2float(__ushort_as_half((unsigned short)(BYTE_OF(w, base) | (BYTE_OF(w, base + 1) << 8))));
            iq4_unpack32([&](int k) { return BYTE_OF(w, base + 2 + k); }, d, o + 16 * b);
        }
    }
};
template <>
struct Dequant64<B200_TYPE_Q8_0> {
    static __device__ __forceinline__ void run(const unsigned char *g, int c, unsigned (&o)[32]) {
        unsigned w[17];
        ld_words<17>(g + c * 2 * Q8_0_BYTES, w);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const float d = __half2float(__ushort_as_half((unsigned short)(BYTE_OF(w, 34 * b) | (BYTE_OF(w, 34 * b + 1) << 8))));
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                const int q0 = (int)(signed char)BYTE_OF(w, 34 * b + 2 + j), q1 = (int)(signed char)BYTE_OF(w, 34 * b + 3 + j);
                o[16 * b + j / 2] = pack_bf16(d * (float)q0, d * (float)q1);
            }
        }
    }
};

// ---------------------------------------------------------------- activation pre-pass: f32 [N][K] -> bf16 [N_pad][K] (pad rows zero)
// A CTA's share of a row, XB_PIECES times 256 pieces of four values: bf16 of them (no row: zeros).  A thread has all its loads in flight at once; with one of 16 bytes a
// thread, 512 rows of 4096 values took 3.5 us beside the product that reads them, 2.3 now, 512 of 11008 6.6, now 4.5.
constexpr int XB_PIECES = 4;
static unsigned xb_blocks(int64_t K) { return (unsigned)((K / 4 + 256 * XB_PIECES - 1) / (256 * XB_PIECES)); }
__device__ __forceinline__ void row_to_bf16(const float *row, int64_t K, __nv_bfloat16 *out) {
    const int64_t i0 = (int64_t)blockIdx.x * (256 * XB_PIECES) + threadIdx.x;
    float4 v[XB_PIECES];
#pragma unroll
    for (int u = 0; u < XB_PIECES; u++) {
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row && (i0 + 256 * u) * 4 < K) v[u] = ld_behind(reinterpret_cast<const float4 *>(row) + i0 + 256 * u);
    }
#pragma unroll
    for (int u = 0; u < XB_PIECES; u++)
        if ((i0 + 256 * u) * 4 < K) *reinterpret_cast<uint2 *>(out + (i0 + 256 * u) * 4) = make_uint2(pack_bf16(v[u].x, v[u].y), pack_bf16(v[u].z, v[u].w));
}
__global__ void __launch_bounds__(256) mmq_x_to_bf16_kernel(const float *__restrict__ x, int64_t x_stride, int64_t K, int64_t N, int64_t n_pad, __nv_bfloat16 *__restrict__ out,
                                     int64_t x_batch) {
    pdl_enter(x);
    const int64_t n = blockIdx.y;
    x += (int64_t)blockIdx.z * x_batch;            // a batch of independent products: blockIdx.z
    out += (int64_t)blockIdx.z * n_pad * K;
    row_to_bf16(n < N ? x + n * x_stride : nullptr, K, out + n * K);
}

struct MmqParams {
    const unsigned char *W;
    size_t w_row_bytes;
    const __nv_bfloat16 *Xb;  // [n_pad][K]
    float *dst;
    int64_t dst_stride, K, M, N;
    // grouped mode (MUL_MAT_ID batches, b200_mul_mat_id_q): a device-built tile table {n_tiles, (expert, first
    // sorted row, end row) ...}; W advances by expert_bytes per expert; sorted row i is stored at dst[row_dst[i] + m]
    const int *tile_tab;
    const int *row_dst;
    size_t expert_bytes;
    int ksplit;  // parts of K that the pairs of a cluster take (mmq_pair_kernel, not grouped)
    // batch of independent products of one shape (not grouped): W advances by w_batch_bytes, dst by dst_batch floats, the
    // bf16 activations by n_pad rows
    int n_batch;
    size_t w_batch_bytes;
    int64_t dst_batch, n_pad;
    int n_expert;  // grouped: experts in the stack
    long long wait_limit = PAIR_WAIT_LIMIT;  // mmq_pair_kernel: clock cycles
};

template <int TYPE, int BN>
__global__ void __launch_bounds__(MQ_THREADS, 1) mmq_tc_kernel(const __grid_constant__ MmqParams p) {
    constexpr int A_BYTES = MQ_BM * MQ_BK * 2, B_BYTES = BN * MQ_BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);  // SW128 atoms: 1024-byte aligned
    __shared__ __align__(8) unsigned long long full_bar[MQ_STAGES], empty_bar[MQ_STAGES], tmem_full_bar;
    __shared__ unsigned tmem_base_s;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const int64_t m0 = (int64_t)blockIdx.x * MQ_BM, n0 = (int64_t)blockIdx.y * BN;
    const int nkb = (int)(p.K / MQ_BK);

    if (tid == 0) {
        for (int s = 0; s < MQ_STAGES; s++) { mbar_init(&full_bar[s], MQ_PRODUCERS); mbar_init(&empty_bar[s], 1); }
        mbar_init(&tmem_full_bar, 1);
        mbar_fence_init();
    }
    if (warp == 4) tmem_alloc(&tmem_base_s, BN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = tmem_base_s;

    if (warp < 4) {
        // ===== producers: thread t owns weight row m0 + t and activation rows t, t + 128 of the tile
        const int64_t m = m0 + tid;
        const bool row_ok = m < p.M;
        const unsigned char *wrow = p.W + (size_t)(row_ok ? m : 0) * p.w_row_bytes;
        const unsigned a_off = (unsigned)((tid >> 3) * 1024 + (tid & 7) * 128);
        for (int kb = 0; kb < nkb; kb++) {
            const int s = kb % MQ_STAGES;
            const unsigned ph = (unsigned)(kb / MQ_STAGES) & 1u;
            mbar_wait(&empty_bar[s], ph ^ 1u);
            unsigned char *a_s = smem + (size_t)s * STAGE_BYTES, *b_s = a_s + A_BYTES;
#pragma unroll
            for (int r0 = 0; r0 < BN; r0 += MQ_PRODUCERS) {
                const int r = r0 + tid;
                if (r < BN) {
                    const unsigned char *src = reinterpret_cast<const unsigned char *>(p.Xb + (n0 + r) * p.K + (int64_t)kb * MQ_BK);
                    unsigned char *drow = b_s + (r >> 3) * 1024 + (r & 7) * 128;
#pragma unroll
                    for (int c = 0; c < 8; c++) cp_async16(drow + ((c ^ (r & 7)) << 4), src + 16 * c);
                }
            }
            cp_async_commit();
            unsigned o[32];
            if (row_ok) Dequant64<TYPE>::run(wrow + (size_t)(kb >> 2) * group256_bytes(TYPE), kb & 3, o);
            else {
#pragma unroll
                for (int i = 0; i < 32; i++) o[i] = 0u;
            }
#pragma unroll
            for (int c = 0; c < 8; c++)
                *reinterpret_cast<uint4 *>(a_s + a_off + ((c ^ (tid & 7)) << 4)) = make_uint4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
            cp_async_wait<0>();
            fence_proxy_async_smem();  // generic-proxy writes (st.shared, cp.async) -> visible to the tensor core's async proxy
            mbar_arrive(&full_bar[s]);
        }
        // ===== epilogue: TMEM lane quarter `warp` -> dst[n][m]
        mbar_wait(&tmem_full_bar, 0u);
        tc_fence_after();
        float *drow = p.dst + m;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 32) {
            float v[32];
            tmem_ld32(tmem_base + ((unsigned)(warp * 32) << 16) + (unsigned)c0, v);
            if (row_ok) {
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const int64_t n = n0 + c0 + j;
                    if (n < p.N) drow[n * p.dst_stride] = v[j];
                }
            }
        }
        tc_fence_before();
    } else {
        // ===== MMA issuer
        constexpr unsigned idesc = umma_idesc_bf16(MQ_BM, BN);
        for (int kb = 0; kb < nkb; kb++) {
            const int s = kb % MQ_STAGES;
            const unsigned ph = (unsigned)(kb / MQ_STAGES) & 1u;
            mbar_wait(&full_bar[s], ph);
            tc_fence_after();
            if (lane == 0) {
                const unsigned a_addr = smem_u32(smem + (size_t)s * STAGE_BYTES), b_addr = a_addr + A_BYTES;
#pragma unroll
                for (int k = 0; k < MQ_BK / 16; k++) {
                    // 16 bf16 = 32 bytes further along K inside the swizzle atom: +2 in the (address >> 4) field
                    tc_mma_bf16(tmem_base, umma_desc_sw128(a_addr) + 2u * k, umma_desc_sw128(b_addr) + 2u * k, idesc, (kb | k) != 0 ? 1u : 0u);
                }
                tc_commit(&empty_bar[s]);
                if (kb == nkb - 1) tc_commit(&tmem_full_bar);
            }
            __syncwarp();
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 4) {
        tc_fence_after();
        tmem_dealloc(tmem_base, BN);
    }
}

// small integers become floats without I2F: PRMT drops the byte into the mantissa of 2^23 (0x4B0000bb = 8388608 + b), one exact FADD removes the bias
template <int K> __device__ __forceinline__ float byte_f(unsigned x) {  // float(byte K of x), exact
    return __uint_as_float(__byte_perm(x, 0x4B000000u, 0x7650 + K)) - 8388608.0f;
}

// ================================================================ dense bf16 rows whose products lie at odd strides
// What one tensor map cannot cover (an expert or batch stride that is no multiple of the row stride): the weight rows pass through the
// producers' registers, the activations arrive by TMA (cp.async.bulk.tensor.2d, 128-byte swizzle applied by the copy engine), issued by a
// dedicated warp as soon as a stage is free.  Everything else runs on the pair kernel (mmq_pair.cuh).
constexpr int MQ2_STAGES = 4;
constexpr int MQ2_THREADS = MQ_PRODUCERS + 64;  // + MMA warp + TMA warp

template <int BN, bool GROUPED>  // GROUPED: experts; else a batch of products
__global__ void __launch_bounds__(MQ2_THREADS, 1) mmq_tc2_kernel(const __grid_constant__ TmapBytes tmB, const __grid_constant__ MmqParams p) {
    constexpr int A_BYTES = MQ_BM * MQ_BK * 2, B_BYTES = BN * MQ_BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    int64_t n0 = (int64_t)blockIdx.y * BN, n_end = p.N;
    const unsigned char *Wbase = p.W;
    if constexpr (GROUPED) {  // uniform over the CTA: tiles past the table's end have nothing to do
        if ((int)blockIdx.y >= __ldg(p.tile_tab)) return;
        const int *te = p.tile_tab + 1 + 3 * blockIdx.y;
        Wbase += (size_t)__ldg(te) * p.expert_bytes;
        n0 = __ldg(te + 1);
        n_end = __ldg(te + 2);
    }
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) unsigned long long full_bar[MQ2_STAGES], empty_bar[MQ2_STAGES], tmem_full_bar;
    __shared__ unsigned tmem_base_s;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const int64_t m0 = (int64_t)blockIdx.x * MQ_BM;
    const int nkb = (int)(p.K / MQ_BK), zb = GROUPED ? 0 : (int)blockIdx.z;
    if (!GROUPED) Wbase += (size_t)zb * p.w_batch_bytes;

    if (tid == 0) {
        for (int s = 0; s < MQ2_STAGES; s++) { mbar_init(&full_bar[s], MQ_PRODUCERS + 1); mbar_init(&empty_bar[s], 1); }
        mbar_init(&tmem_full_bar, 1);
        mbar_fence_init();
    }
    if (warp == 4) tmem_alloc(&tmem_base_s, BN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = tmem_base_s;

    if (warp < 4) {
        const int64_t m = m0 + tid;
        const bool row_ok = m < p.M;
        const unsigned char *wrow = Wbase + (size_t)(row_ok ? m : 0) * p.w_row_bytes;
        const unsigned a_off = (unsigned)((tid >> 3) * 1024 + (tid & 7) * 128);
        auto publish = [&](int kb, const unsigned (&o)[32]) {
            const int s = kb % MQ2_STAGES;
            mbar_wait(&empty_bar[s], ((unsigned)(kb / MQ2_STAGES) & 1u) ^ 1u);
            unsigned char *a_s = smem + (size_t)s * STAGE_BYTES;
#pragma unroll
            for (int q = 0; q < 8; q++)
                *reinterpret_cast<uint4 *>(a_s + a_off + ((q ^ (tid & 7)) << 4)) = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
            fence_proxy_async_smem();
            mbar_arrive(&full_bar[s]);
        };
        {
            // dense bf16 rows: a K step is 128 bytes of the thread's row, stored as it is; the next step's bytes are in flight meanwhile
            const uint4 *q4 = reinterpret_cast<const uint4 *>(wrow);
            uint4 cur[8], nxt[8];
#pragma unroll
            for (int i = 0; i < 8; i++) cur[i] = row_ok ? __ldg(q4 + i) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
            for (int kb = 0; kb < nkb; kb++) {
                if (kb + 1 < nkb) {
#pragma unroll
                    for (int i = 0; i < 8; i++) nxt[i] = row_ok ? __ldg(q4 + (size_t)(kb + 1) * 8 + i) : make_uint4(0u, 0u, 0u, 0u);
                }
                unsigned o[32];
#pragma unroll
                for (int i = 0; i < 8; i++) { o[4 * i] = cur[i].x; o[4 * i + 1] = cur[i].y; o[4 * i + 2] = cur[i].z; o[4 * i + 3] = cur[i].w; }
                publish(kb, o);
#pragma unroll
                for (int i = 0; i < 8; i++) cur[i] = nxt[i];
            }
        }
        mbar_wait(&tmem_full_bar, 0u);
        tc_fence_after();
        float *drow = p.dst + m + (int64_t)zb * p.dst_batch;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 32) {
            float v[32];
            tmem_ld32(tmem_base + ((unsigned)(warp * 32) << 16) + (unsigned)c0, v);
            if (row_ok) {
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    const int64_t n = n0 + c0 + j;
                    if (n >= n_end) continue;
                    if constexpr (GROUPED) drow[(int64_t)__ldg(p.row_dst + n)] = v[j];  // scatter: sorted row -> (token, slot)
                    else drow[n * p.dst_stride] = v[j];
                }
            }
        }
        tc_fence_before();
    } else if (warp == 4) {
        constexpr unsigned idesc = umma_idesc_bf16(MQ_BM, BN);
        for (int kb = 0; kb < nkb; kb++) {
            const int s = kb % MQ2_STAGES;
            mbar_wait(&full_bar[s], (unsigned)(kb / MQ2_STAGES) & 1u);
            tc_fence_after();
            if (lane == 0) {
                const unsigned a_addr = smem_u32(smem + (size_t)s * STAGE_BYTES), b_addr = a_addr + A_BYTES;
#pragma unroll
                for (int k = 0; k < MQ_BK / 16; k++)
                    tc_mma_bf16(tmem_base, umma_desc_sw128(a_addr) + 2u * k, umma_desc_sw128(b_addr) + 2u * k, idesc, (kb | k) != 0 ? 1u : 0u);
                tc_commit(&empty_bar[s]);
                if (kb == nkb - 1) tc_commit(&tmem_full_bar);
            }
            __syncwarp();
        }
        tc_fence_before();
    } else {
        // ===== TMA warp: activation tiles [BN rows x 64 bf16] into the swizzled B slot of each free stage
        if (lane == 0) {
            for (int kb = 0; kb < nkb; kb++) {
                const int s = kb % MQ2_STAGES;
                mbar_wait(&empty_bar[s], ((unsigned)(kb / MQ2_STAGES) & 1u) ^ 1u);
                mbar_expect_tx(&full_bar[s], (unsigned)B_BYTES);
                tma_load_2d(smem + (size_t)s * STAGE_BYTES + A_BYTES, &tmB, kb * MQ_BK, (int)n0 + zb * (int)p.n_pad, &full_bar[s]);
            }
        }
    }
    __syncthreads();
    if (warp == 4) {
        tc_fence_after();
        tmem_dealloc(tmem_base, BN);
    }
}

// ---------------------------------------------------------------- host side
// set by a GEMM whose pipeline gave up; pinned host memory, so that reading it after a synchronisation costs nothing.  Allocated before the first
// launch that may set it, whoever makes it and on whichever thread; legal while a stream is being captured.
static std::atomic<int *> g_gemm_timeout{nullptr};
static int gemm_status_prepare() {
    static std::mutex lock;
    if (g_gemm_timeout.load(std::memory_order_acquire)) return B200_OK;
    std::lock_guard<std::mutex> guard(lock);
    if (g_gemm_timeout.load(std::memory_order_relaxed)) return B200_OK;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    B200_CUDA_TRY(cudaThreadExchangeStreamCaptureMode(&mode));
    int *p = nullptr;
    const cudaError_t rc = cudaHostAlloc((void **)&p, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped);
    cudaThreadExchangeStreamCaptureMode(&mode);
    B200_CUDA_TRY(rc);
    *p = 0;
    g_gemm_timeout.store(p, std::memory_order_release);
    return B200_OK;
}
// the word itself, for kernels of other files whose waits have a limit
int gemm_status_word(int **p) {
    const int rc = gemm_status_prepare();
    *p = rc == B200_OK ? g_gemm_timeout.load(std::memory_order_acquire) : nullptr;
    return rc;
}

static int64_t mmq_bn(int64_t N) { return N <= 32 ? 32 : N <= 64 ? 64 : N <= 128 ? 128 : 256; }
static int64_t mmq_n_pad(int64_t N) { const int64_t bn = mmq_bn(N); return (N + bn - 1) / bn * bn; }

template <int TYPE, int BN>
static int mmq_launch(const MmqParams &p, cudaStream_t st) {
    constexpr size_t smem = (size_t)MQ_STAGES * (MQ_BM * MQ_BK * 2 + BN * MQ_BK * 2) + 1024;
    static bool attr_set_dev[16] = {};  // cudaFuncSetAttribute is per device
    int cur_dev = 0;
    B200_CUDA_TRY(cudaGetDevice(&cur_dev));
    bool &attr_set = attr_set_dev[cur_dev & 15];
    if (!attr_set) {
        B200_CUDA_TRY(cudaFuncSetAttribute(mmq_tc_kernel<TYPE, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set = true;
    }
    dim3 grid((unsigned)((p.M + MQ_BM - 1) / MQ_BM), (unsigned)((p.N + BN - 1) / BN));
    mmq_tc_kernel<TYPE, BN><<<grid, MQ_THREADS, smem, st>>>(p);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

// a 2-D bf16 tensor map of `rows` rows of K values, boxes of `box_rows` x 64, 128-byte swizzle
static int encode_rows(TmapBytes &tm, const void *base, int64_t K, int64_t rows, size_t row_bytes, int box_rows) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) { set_error("b200_mul_mat_q: cuTensorMapEncodeTiled not available"); return B200_ERR_CUDA; }
    const unsigned long long gdim[2] = {(unsigned long long)K, (unsigned long long)rows}, gstr[1] = {(unsigned long long)row_bytes};
    const unsigned box[2] = {(unsigned)MQ_BK, (unsigned)box_rows}, estr[2] = {1, 1};
    // CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 = 9, INTERLEAVE_NONE = 0, SWIZZLE_128B = 3, L2_PROMOTION_L2_256B = 3, FLOAT_OOB_FILL_NONE = 0
    const int rc = enc(&tm, 9, 2, (void *)base, gdim, gstr, box, estr, 0, 3, 3, 0);
    if (rc != 0) { set_error("b200_mul_mat_q: cuTensorMapEncodeTiled failed (%d)", rc); return B200_ERR_CUDA; }
    return B200_OK;
}

}  // namespace b200
#include "mmq_pair.cuh"
namespace b200 {

template <int BN, bool GROUPED>
static int mmq2_launch(const MmqParams &p, int64_t n_pad, cudaStream_t st, unsigned grid_y = 0) {
    constexpr size_t smem = (size_t)MQ2_STAGES * (MQ_BM * MQ_BK * 2 + BN * MQ_BK * 2) + 1024;
    static bool attr_set_dev[16] = {};  // cudaFuncSetAttribute is per device
    int cur_dev = 0;
    B200_CUDA_TRY(cudaGetDevice(&cur_dev));
    bool &attr_set = attr_set_dev[cur_dev & 15];
    if (!attr_set) {
        B200_CUDA_TRY(cudaFuncSetAttribute(mmq_tc2_kernel<BN, GROUPED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set = true;
    }
    TmapBytes tm;
    const int rc = encode_rows(tm, p.Xb, p.K, n_pad * p.n_batch, (size_t)p.K * 2, BN);
    if (rc != B200_OK) return rc;
    const dim3 grid((unsigned)((p.M + MQ_BM - 1) / MQ_BM), GROUPED ? grid_y : (unsigned)((p.N + BN - 1) / BN), (unsigned)p.n_batch);
    mmq_tc2_kernel<BN, GROUPED><<<grid, MQ2_THREADS, smem, st>>>(tm, p);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

template <int TYPE>
static int mmq_dispatch_bn(const MmqParams &p, cudaStream_t st) {
    if constexpr (TYPE == B200_TYPE_BF16) {  // dense rows: any K that is a multiple of the K step
        const int64_t n_pad = mmq_n_pad(p.N);
        // products whose weight rows lie at one stride over all of them: one tensor map covers the stack
        if (p.n_batch == 1 || p.w_batch_bytes % p.w_row_bytes == 0) return mmq_pair_launch<TYPE, false>(p, n_pad, p.n_batch > 1 ? (int64_t)(p.w_batch_bytes / p.w_row_bytes) : 0, 0, 0, st);
        switch (mmq_bn(p.N)) {
            case 32: return mmq2_launch<32, false>(p, n_pad, st);
            case 64: return mmq2_launch<64, false>(p, n_pad, st);
            case 128: return mmq2_launch<128, false>(p, n_pad, st);
            default: return mmq2_launch<256, false>(p, n_pad, st);
        }
    } else {
        if (p.K % 256 == 0) return mmq_pair_launch<TYPE, false>(p, mmq_n_pad(p.N), 0, 0, 0, st);
    }
    if constexpr (type_block_values(TYPE) == 32) {  // (a K-quant's rows are whole groups of 256 values)
        switch (mmq_bn(p.N)) {
            case 32: return mmq_launch<TYPE, 32>(p, st);
            case 64: return mmq_launch<TYPE, 64>(p, st);
            case 128: return mmq_launch<TYPE, 128>(p, st);
            default: return mmq_launch<TYPE, 256>(p, st);
        }
    }
    return B200_ERR_UNSUPPORTED;
}


// ================================================================ (a9) MUL_MAT_ID for batches: group by expert on the device
// Replaces the batch branch of ggml_cuda_mul_mat_id (ggml/src/ggml-cuda.cu:2066-2139: ids copied to the host +
// stream sync, then per expert k_copy_src1_to_contiguous -> mul_mat -> k_copy_dst_from_contiguous, :1954-2001).  Here nothing
// leaves the device: one small kernel counts the (token, slot) pairs per expert, prefix-sums them, writes the sorted row lists and
// the tile table; a gather pass converts the selected activation rows to bf16 in sorted order; ONE grouped tensor-core launch
// walks the tile table (every tile belongs to one expert) and scatters its f32 results straight to dst[(token, slot)].
constexpr int MID_MAX_EXPERTS = 256;
struct MidTables {      // int offsets into the table area of the workspace
    int *tile_tab;      // 1 + 3 * max_tiles
    int *row_src;       // n_rows: float offset of the activation row of sorted row i
    int *row_dst;       // n_rows: float offset of dst row of sorted row i
};
__global__ void __launch_bounds__(1024, 1) mid_group_kernel(const int32_t *__restrict__ ids, int64_t ids_stride, int n_used, int T, int n_expert, int n_b_rows,
                                                            int64_t b_stride_row, int64_t b_stride_tok, int64_t d_stride_row, int64_t d_stride_tok, int BN,
                                                            MidTables t) {
    __shared__ int count[MID_MAX_EXPERTS], off[MID_MAX_EXPERTS + 1], cursor[MID_MAX_EXPERTS];
    pdl_enter(ids);
    for (int e = threadIdx.x; e < n_expert; e += blockDim.x) { count[e] = 0; cursor[e] = 0; }
    __syncthreads();
    const int n = n_used * T;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int e = ids[(int64_t)(i / n_used) * ids_stride + i % n_used];
        if (e >= 0 && e < n_expert) atomicAdd(&count[e], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0, nt = 0;
        for (int e = 0; e < n_expert; e++) {
            off[e] = acc;
            for (int r0 = acc; r0 < acc + count[e]; r0 += BN) {
                t.tile_tab[1 + 3 * nt] = e;
                t.tile_tab[2 + 3 * nt] = r0;
                t.tile_tab[3 + 3 * nt] = acc + count[e];
                nt++;
            }
            acc += count[e];
        }
        off[n_expert] = acc;
        t.tile_tab[0] = nt;
    }
    __syncthreads();
    // rows of invalid expert ids are left out (their dst rows stay untouched; the reference asserts on them); the slots behind
    // the last valid row are given a harmless source so the gather pass needs no count
    for (int i = off[n_expert] + threadIdx.x; i < n; i += blockDim.x) { t.row_src[i] = 0; t.row_dst[i] = 0; }
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int tok = i / n_used, s = i % n_used;
        const int e = ids[(int64_t)tok * ids_stride + s];
        if (e < 0 || e >= n_expert) continue;
        const int pos = off[e] + atomicAdd(&cursor[e], 1);
        t.row_src[pos] = (int)(tok * b_stride_tok + (s % n_b_rows) * b_stride_row);
        t.row_dst[pos] = (int)(tok * d_stride_tok + s * d_stride_row);
    }
}
// gather + convert: sorted row i <- bf16(b[row_src[i]]), K values
__global__ void __launch_bounds__(256) mid_gather_bf16_kernel(const float *__restrict__ b, const int *__restrict__ row_src, int64_t K, __nv_bfloat16 *__restrict__ out) {
    pdl_enter(b, row_src);
    const int64_t n = blockIdx.y;
    row_to_bf16(b + (int64_t)ld_behind(row_src + n), K, out + n * K);
}

static int64_t mid_bn(int64_t n_rows, int n_expert) { return mmq_bn((n_rows + n_expert - 1) / n_expert); }
static int64_t mid_max_tiles(int64_t bn, int64_t n_rows, int n_expert) { return (n_rows + bn - 1) / bn + n_expert; }
// experts whose rows lie at one stride over the stack (quantised ones need no stack): the pair kernel
static bool mid_pair(int type, size_t w_row_bytes, size_t expert_bytes) { return type != B200_TYPE_BF16 || expert_bytes % w_row_bytes == 0; }
// there the width of a tile follows its rows, so the table's tiles are as wide as the accumulators allow unless experts are small
static int64_t mid_tile(bool pair, int64_t n_rows, int n_expert) {
    const int64_t bn = mid_bn(n_rows, n_expert);
    return !pair ? bn : bn < 128 ? 2 * bn : 256;
}
static size_t mid_xb_bytes(int64_t n_rows, int64_t K) { return ((size_t)n_rows * (size_t)K * 2 + 255) / 256 * 256; }

template <int TYPE>
static int mid_dispatch_bn(const MmqParams &p, int64_t bn, int64_t n_rows, unsigned grid_y, cudaStream_t st) {
    if (mid_pair(TYPE, p.w_row_bytes, p.expert_bytes)) return mmq_pair_launch<TYPE, true>(p, n_rows, (int64_t)(p.expert_bytes / p.w_row_bytes), grid_y, bn, st);
    if constexpr (TYPE == B200_TYPE_BF16)
    switch (bn) {
        case 32: return mmq2_launch<32, true>(p, n_rows, st, grid_y);
        case 64: return mmq2_launch<64, true>(p, n_rows, st, grid_y);
        case 128: return mmq2_launch<128, true>(p, n_rows, st, grid_y);
        default: return mmq2_launch<256, true>(p, n_rows, st, grid_y);
    }
    return B200_ERR_UNSUPPORTED;
}

}  // namespace b200

using namespace b200;

extern "C" int b200_gemm_status(void) {
    const volatile int *p = g_gemm_timeout.load(std::memory_order_acquire);
    return p ? *p : 0;
}

extern "C" size_t b200_mul_mat_q_workspace_bytes(int type, int64_t K, int64_t M, int64_t N) {
    (void)type; (void)M;
    if (K <= 0 || N <= 0) return 0;
    return (size_t)mmq_n_pad(N) * (size_t)K * 2 + 256;
}

extern "C" int b200_mul_mat_q(int type, const void *W, size_t w_row_bytes, const float *X, int64_t x_stride, float *dst, int64_t dst_stride,
                              int64_t K, int64_t M, int64_t N, void *workspace, size_t workspace_bytes, b200_stream_t stream) {
    return b200_mul_mat_q_wait(type, W, w_row_bytes, X, x_stride, dst, dst_stride, K, M, N, workspace, workspace_bytes, PAIR_WAIT_LIMIT, stream);
}

extern "C" int b200_mul_mat_q_wait(int type, const void *W, size_t w_row_bytes, const float *X, int64_t x_stride, float *dst, int64_t dst_stride, int64_t K, int64_t M,
                                   int64_t N, void *workspace, size_t workspace_bytes, int64_t wait_cycles, b200_stream_t stream) {
    if (wait_cycles < 0) { set_error("b200_mul_mat_q_wait: limit below zero"); return B200_ERR_INVALID; }
    if (!W || !dst) { set_error("b200_mul_mat_q: NULL argument"); return B200_ERR_INVALID; }
    const int bv = type_block_values(type);
    if (!(type == B200_TYPE_Q4_0 || type == B200_TYPE_Q8_0 || type == B200_TYPE_Q4_K || type == B200_TYPE_Q5_K || type == B200_TYPE_Q6_K ||
          type == B200_TYPE_Q4_1 || type == B200_TYPE_Q5_0 || type == B200_TYPE_Q5_1 || type == B200_TYPE_Q2_K || type == B200_TYPE_Q3_K ||
          type == B200_TYPE_IQ4_NL || type == B200_TYPE_IQ4_XS || type == B200_TYPE_BF16)) {
        set_error("b200_mul_mat_q: unsupported weight type %d", type);
        return B200_ERR_UNSUPPORTED;
    }
    if (K <= 0 || K % bv || M < 0 || N < 0) { set_error("b200_mul_mat_q: bad shape K=%lld M=%lld N=%lld", (long long)K, (long long)M, (long long)N); return B200_ERR_INVALID; }
    if (K % MQ_BK) { set_error("b200_mul_mat_q: K=%lld must be a multiple of %d", (long long)K, MQ_BK); return B200_ERR_UNSUPPORTED; }
    if (M == 0 || N == 0) return B200_OK;
    const size_t row_bytes = (size_t)(K / bv) * type_block_bytes(type);
    if (w_row_bytes < row_bytes || (w_row_bytes & 1) || ((uintptr_t)W & 1)) { set_error("b200_mul_mat_q: weight stride/alignment"); return B200_ERR_INVALID; }
    if ((type == B200_TYPE_Q4_K || type == B200_TYPE_Q5_K || type == B200_TYPE_BF16) && ((w_row_bytes & 15) || ((uintptr_t)W & 15))) {
        set_error("b200_mul_mat_q: q4_K / q5_K / bf16 rows must be 16-byte aligned");
        return B200_ERR_UNSUPPORTED;
    }
    if (X && (((uintptr_t)X & 15) || (x_stride & 3))) { set_error("b200_mul_mat_q: X must be 16-byte aligned with a row stride multiple of 4"); return B200_ERR_UNSUPPORTED; }
    const size_t need = b200_mul_mat_q_workspace_bytes(type, K, M, N);
    if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 15)) {
        set_error("b200_mul_mat_q: workspace of %zu bytes (16-byte aligned) required, %zu given", need, workspace_bytes);
        return B200_ERR_INVALID;
    }
    const cudaStream_t st = (cudaStream_t)stream;
    const int64_t n_pad = mmq_n_pad(N);
    if (n_pad > 65535) { set_error("b200_mul_mat_q: N too large"); return B200_ERR_UNSUPPORTED; }
    __nv_bfloat16 *xb = (__nv_bfloat16 *)workspace;
    if (X) {  // (X == NULL: the workspace holds the bf16 activations of the previous call with this K and N)
        dim3 g1(xb_blocks(K), (unsigned)n_pad);
        B200_CUDA_TRY(launch_chained(mmq_x_to_bf16_kernel, g1, 256, 0, st, X, x_stride, K, N, n_pad, xb, (int64_t)0));
    }
    MmqParams p;
    p.W = (const unsigned char *)W; p.w_row_bytes = w_row_bytes; p.Xb = xb; p.dst = dst; p.dst_stride = dst_stride; p.K = K; p.M = M; p.N = N;
    p.tile_tab = nullptr; p.row_dst = nullptr; p.expert_bytes = 0;
    p.n_batch = 1; p.w_batch_bytes = 0; p.dst_batch = 0; p.n_pad = n_pad; p.n_expert = 1;
    p.wait_limit = wait_cycles;
    switch (type) {
        case B200_TYPE_Q4_0: return mmq_dispatch_bn<B200_TYPE_Q4_0>(p, st);
        case B200_TYPE_Q8_0: return mmq_dispatch_bn<B200_TYPE_Q8_0>(p, st);
        case B200_TYPE_Q4_K: return mmq_dispatch_bn<B200_TYPE_Q4_K>(p, st);
        case B200_TYPE_Q5_K: return mmq_dispatch_bn<B200_TYPE_Q5_K>(p, st);
        case B200_TYPE_Q6_K: return mmq_dispatch_bn<B200_TYPE_Q6_K>(p, st);
        case B200_TYPE_Q4_1: return mmq_dispatch_bn<B200_TYPE_Q4_1>(p, st);
        case B200_TYPE_Q5_0: return mmq_dispatch_bn<B200_TYPE_Q5_0>(p, st);
        case B200_TYPE_Q5_1: return mmq_dispatch_bn<B200_TYPE_Q5_1>(p, st);
        case B200_TYPE_Q2_K: return mmq_dispatch_bn<B200_TYPE_Q2_K>(p, st);
        case B200_TYPE_Q3_K: return mmq_dispatch_bn<B200_TYPE_Q3_K>(p, st);
        case B200_TYPE_IQ4_NL: return mmq_dispatch_bn<B200_TYPE_IQ4_NL>(p, st);
        case B200_TYPE_IQ4_XS: return mmq_dispatch_bn<B200_TYPE_IQ4_XS>(p, st);
        case B200_TYPE_BF16: return mmq_dispatch_bn<B200_TYPE_BF16>(p, st);
    }
    return B200_ERR_UNSUPPORTED;
}

// A batch of independent products of one shape over dense bf16 weights (the per-head matrices of an attention layer) in ONE
// launch: product b reads W + b * w_batch_bytes and X + b * x_batch and writes dst + b * dst_batch.
extern "C" int b200_mul_mat_bf16_batched(const void *W, size_t w_row_bytes, size_t w_batch_bytes, const float *X, int64_t x_stride, int64_t x_batch, float *dst,
                                         int64_t dst_stride, int64_t dst_batch, int64_t K, int64_t M, int64_t N, int32_t n_batch, void *workspace,
                                         size_t workspace_bytes, b200_stream_t stream) {
    if (!W || !X || !dst || n_batch < 1 || n_batch > 65535) { set_error("b200_mul_mat_bf16_batched: bad argument"); return B200_ERR_INVALID; }
    if (K <= 0 || K % MQ_BK || M <= 0 || N <= 0) { set_error("b200_mul_mat_bf16_batched: K=%lld must be a positive multiple of %d", (long long)K, MQ_BK); return B200_ERR_UNSUPPORTED; }
    if (((uintptr_t)W | w_row_bytes | w_batch_bytes | (uintptr_t)X) & 15 || (x_stride & 3) || (x_batch & 3)) { set_error("b200_mul_mat_bf16_batched: operands must be 16-byte aligned"); return B200_ERR_UNSUPPORTED; }
    const int64_t n_pad = mmq_n_pad(N);
    const size_t need = (size_t)n_pad * (size_t)K * 2 * (size_t)n_batch + 256;
    if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 15) || n_pad * n_batch > 0x7fffffff) {
        set_error("b200_mul_mat_bf16_batched: workspace of %zu bytes (16-byte aligned) required, %zu given", need, workspace_bytes);
        return B200_ERR_INVALID;
    }
    const cudaStream_t st = (cudaStream_t)stream;
    __nv_bfloat16 *xb = (__nv_bfloat16 *)workspace;
    dim3 g1(xb_blocks(K), (unsigned)n_pad, (unsigned)n_batch);
    B200_CUDA_TRY(launch_chained(mmq_x_to_bf16_kernel, g1, 256, 0, st, X, x_stride, K, N, n_pad, xb, x_batch));
    MmqParams p;
    p.W = (const unsigned char *)W; p.w_row_bytes = w_row_bytes; p.Xb = xb; p.dst = dst; p.dst_stride = dst_stride; p.K = K; p.M = M; p.N = N;
    p.tile_tab = nullptr; p.row_dst = nullptr; p.expert_bytes = 0;
    p.n_batch = n_batch; p.w_batch_bytes = w_batch_bytes; p.dst_batch = dst_batch; p.n_pad = n_pad; p.n_expert = 1;
    return mmq_dispatch_bn<B200_TYPE_BF16>(p, st);
}

extern "C" size_t b200_mul_mat_id_q_workspace_bytes(int type, int64_t K, int64_t M, int64_t n_used, int64_t T, int32_t n_expert) {
    (void)type; (void)M;
    const int64_t n_rows = n_used * T;
    if (K <= 0 || n_rows <= 0 || n_expert <= 0) return 0;
    return mid_xb_bytes(n_rows, K) + sizeof(int) * (size_t)(1 + 3 * mid_max_tiles(mid_bn(n_rows, n_expert), n_rows, n_expert) + 2 * n_rows) + 256;
}

extern "C" int b200_mul_mat_id_q(int type, const void *as, size_t w_row_bytes, size_t expert_bytes, int32_t n_expert, const int32_t *ids,
                                 int64_t ids_stride, const float *b, int64_t b_stride_row, int64_t b_stride_tok, float *dst, int64_t dst_stride_row,
                                 int64_t dst_stride_tok, int64_t K, int64_t M, int64_t n_used, int64_t n_b_rows, int64_t T, void *workspace,
                                 size_t workspace_bytes, b200_stream_t stream) {
    if (!as || !ids || !b || !dst) { set_error("b200_mul_mat_id_q: NULL argument"); return B200_ERR_INVALID; }
    if (!(type == B200_TYPE_Q4_0 || type == B200_TYPE_Q8_0 || type == B200_TYPE_Q4_K || type == B200_TYPE_Q5_K || type == B200_TYPE_Q6_K ||
          type == B200_TYPE_Q4_1 || type == B200_TYPE_Q5_0 || type == B200_TYPE_Q5_1 || type == B200_TYPE_Q2_K || type == B200_TYPE_Q3_K ||
          type == B200_TYPE_IQ4_NL || type == B200_TYPE_IQ4_XS || type == B200_TYPE_BF16)) {
        set_error("b200_mul_mat_id_q: unsupported weight type %d", type);
        return B200_ERR_UNSUPPORTED;
    }
    const int64_t k_unit = type == B200_TYPE_BF16 ? MQ_BK : 256;  // dense rows step by one K tile, quantised rows by a 256-value group
    if (K <= 0 || K % k_unit || M < 0 || T < 0 || n_used < 1 || n_b_rows < 1 || n_expert < 1 || n_expert > MID_MAX_EXPERTS) {
        set_error("b200_mul_mat_id_q: bad shape (K must be a multiple of %d, at most %d experts)", (int)k_unit, MID_MAX_EXPERTS);
        return K % k_unit ? B200_ERR_UNSUPPORTED : B200_ERR_INVALID;
    }
    if (M == 0 || T == 0) return B200_OK;
    if (type == B200_TYPE_BF16 && ((w_row_bytes | expert_bytes | (uintptr_t)as) & 15)) { set_error("b200_mul_mat_id_q: bf16 rows must be 16-byte aligned"); return B200_ERR_UNSUPPORTED; }
    const int bv = type_block_values(type);
    const size_t row_bytes = (size_t)(K / bv) * type_block_bytes(type);
    if (w_row_bytes < row_bytes || ((w_row_bytes | expert_bytes | (uintptr_t)as) & 1)) { set_error("b200_mul_mat_id_q: weight stride/alignment"); return B200_ERR_INVALID; }
    if ((type == B200_TYPE_Q4_K || type == B200_TYPE_Q5_K) && ((w_row_bytes | expert_bytes | (uintptr_t)as) & 15)) {
        set_error("b200_mul_mat_id_q: q4_K/q5_K rows must be 16-byte aligned");
        return B200_ERR_UNSUPPORTED;
    }
    if (((uintptr_t)b & 15) || ((b_stride_row | b_stride_tok) & 3)) { set_error("b200_mul_mat_id_q: b rows must be 16-byte aligned"); return B200_ERR_UNSUPPORTED; }
    const int64_t n_rows = n_used * T;
    const int64_t span_b = (T - 1) * b_stride_tok + (n_b_rows - 1) * b_stride_row, span_d = (T - 1) * dst_stride_tok + (n_used - 1) * dst_stride_row;
    if (n_rows > 65535 || span_b > 0x7fffffff || span_d > 0x7fffffff) { set_error("b200_mul_mat_id_q: batch too large"); return B200_ERR_UNSUPPORTED; }
    const size_t need = b200_mul_mat_id_q_workspace_bytes(type, K, M, n_used, T, n_expert);
    if (!workspace || workspace_bytes < need || ((uintptr_t)workspace & 255)) {
        set_error("b200_mul_mat_id_q: workspace of %zu bytes (256-byte aligned) required, %zu given", need, workspace_bytes);
        return B200_ERR_INVALID;
    }
    const cudaStream_t st = (cudaStream_t)stream;
    const int64_t bn = mid_tile(mid_pair(type, w_row_bytes, expert_bytes), n_rows, n_expert), max_tiles = mid_max_tiles(bn, n_rows, n_expert);
    __nv_bfloat16 *xb = (__nv_bfloat16 *)workspace;
    MidTables t;
    t.tile_tab = (int *)((unsigned char *)workspace + mid_xb_bytes(n_rows, K));
    t.row_src = t.tile_tab + 1 + 3 * max_tiles;
    t.row_dst = t.row_src + n_rows;
    B200_CUDA_TRY(launch_chained(mid_group_kernel, 1, 1024, 0, st, ids, ids_stride, (int)n_used, (int)T, (int)n_expert, (int)n_b_rows, b_stride_row, b_stride_tok, dst_stride_row,
                                 dst_stride_tok, (int)bn, t));
    dim3 g1(xb_blocks(K), (unsigned)n_rows);
    B200_CUDA_TRY(launch_chained(mid_gather_bf16_kernel, g1, 256, 0, st, b, t.row_src, K, xb));
    MmqParams p;
    p.W = (const unsigned char *)as; p.w_row_bytes = w_row_bytes; p.Xb = xb; p.dst = dst; p.dst_stride = 0; p.K = K; p.M = M; p.N = n_rows;
    p.tile_tab = t.tile_tab; p.row_dst = t.row_dst; p.expert_bytes = expert_bytes;
    p.n_batch = 1; p.w_batch_bytes = 0; p.dst_batch = 0; p.n_pad = 0; p.n_expert = n_expert;
    switch (type) {
        case B200_TYPE_Q4_0: return mid_dispatch_bn<B200_TYPE_Q4_0>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_Q8_0: return mid_dispatch_bn<B200_TYPE_Q8_0>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_Q4_K: return mid_dispatch_bn<B200_TYPE_Q4_K>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_Q5_K: return mid_dispatch_bn<B200_TYPE_Q5_K>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_Q6_K: return mid_dispatch_bn<B200_TYPE_Q6_K>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_Q4_1: return mid_dispatch_bn<B200_TYPE_Q4_1>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_Q5_0: return mid_dispatch_bn<B200_TYPE_Q5_0>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_Q5_1: return mid_dispatch_bn<B200_TYPE_Q5_1>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_Q2_K: return mid_dispatch_bn<B200_TYPE_Q2_K>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_Q3_K: return mid_dispatch_bn<B200_TYPE_Q3_K>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_IQ4_NL: return mid_dispatch_bn<B200_TYPE_IQ4_NL>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_IQ4_XS: return mid_dispatch_bn<B200_TYPE_IQ4_XS>(p, bn, n_rows, (unsigned)max_tiles, st);
        case B200_TYPE_BF16: return mid_dispatch_bn<B200_TYPE_BF16>(p, bn, n_rows, (unsigned)max_tiles, st);
    }
    return B200_ERR_UNSUPPORTED;
}
