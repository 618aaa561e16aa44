// mmvq_mma.cuh -- decode GEMV for 4 (q6_K: 6) to 8 columns over q4_K / q5_K / q6_K weights on the int8 tensor cores.  Included by mmvq.cu.
//
// Same arithmetic as SliceDot (exact integer sums of quants and q8_1 activations per sub-block, scaled in f32), but the integer sums of 16 weight
// rows against all columns come from mma.sync s8 tiles: the dp4a form spends 8 instructions a column and 32 weights and was issue-bound, 56.8 us for
// 27648 x 5120 q5_K and 4 columns (97 MB, 1.7 TB/s); 34.6 us here, 8 columns 101.5 -> 37.8.  What bounds it now is still issue: unpacking and
// scaling, the same for any column count, and the columns' quantisation, which every CTA does for itself (8 values a thread and no division of
// indexes: with 4 values and a division it cost 2 us for 2048 values x 4 columns, 1 us now).
//   * a warp takes 16 rows x one 256-value block at a time; their raw bytes (16-byte cp.async pieces, rows may start at any even byte) wait in a
//     ring of its own, one or two blocks ahead; the ring is filled before the wait for the producer kernel;
//   * the activations of all columns are quantised once per CTA into shared memory, in the order in which a lane reads its operand;
//   * KS warps share a row tile, each a part of K; their sums meet in shared memory in a fixed order.  KS is chosen so that rows and K parts
//     fill the device evenly.
#pragma once

namespace b200 {

constexpr int MV_NW = MMVQ_NW, MV_ROWS = 16;
template <int TYPE> constexpr int mv_pieces() { return (type_block_bytes(TYPE) + (TYPE == B200_TYPE_Q6_K ? 14 : 0) + 15) / 16; }
template <int TYPE> constexpr int mv_row() { return (mv_pieces<TYPE>() | 1) * 16; }  // 8 rows start in 8 different groups of 4 banks
// activations of one (32-value block, column): 32 int8, then d and s (q6_K: and -32 times the sums of both halves)
template <int TYPE> constexpr int mv_scale_bytes() { return TYPE == B200_TYPE_Q6_K ? 16 : 8; }
constexpr int mv_cols(int n) { return (n + 1) & ~1; }  // columns' scales are read two at a time

struct MvParams {
    MmvqParams m;
    int n, ks, slots, n_tiles;     // columns, warps a row tile, ring slots
    unsigned div_n8;               // 2^32 / (K / 8), rounded up: item / (K / 8) is exact while item x K / 8 < 2^32
    int tile0[B200_GEMV_MAX_JOBS]; // first row tile of each job
};

__device__ __forceinline__ void mv_mma32(int (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mv_mma16(int (&c)[4], unsigned a0, unsigned a1, unsigned b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(b0));
}
// exact floats of integers below 2^22 in magnitude without a conversion: the integer was added to the bits of 1.5 * 2^23
constexpr int MV_MAGIC = 0x4B400000;
__device__ __forceinline__ float mv_float(int biased) { return __int_as_float(biased) - 12582912.0f; }
__device__ __forceinline__ float mv_byte(unsigned w, int k) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650 + k)) - 8388608.0f; }
// word at a 2-byte aligned shared address
__device__ __forceinline__ unsigned mv_word(const unsigned char *p) {
    const unsigned a = smem_u32(p);
    const unsigned *w = reinterpret_cast<const unsigned *>(p - (a & 2u));
    return __funnelshift_r(w[0], w[1], (a & 2u) * 8u);
}

// one 256-value block of rows g and g + 8: acc[0..1] += row g, columns 2 t4 and 2 t4 + 1; acc[2..3] += row g + 8.  r0, r1: the rows' first bytes; bq: this lane's
// operand (column g) of the block's first 32 values, next ones bq_step bytes on; sc: the scales of column 2 t4, next 32 values sc_step bytes on
template <int TYPE>
__device__ __forceinline__ void mv_block(const unsigned char *r0, const unsigned char *r1, int t4, bool col, const unsigned char *bq, int bq_step, const unsigned char *sc, int sc_step,
                                         float (&acc)[4]) {
    if constexpr (TYPE == B200_TYPE_Q6_K) {
        const float d0 = h2f(*reinterpret_cast<const unsigned short *>(r0 + 208)), d1 = h2f(*reinterpret_cast<const unsigned short *>(r1 + 208));
        float sd[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int half = 0; half < 2; half++) {
            unsigned qh0[2], qh1[2], s0[2], s1[2];  // both 16-byte halves' high bits; the half's 8 scales
#pragma unroll
            for (int e = 0; e < 2; e++) {
                qh0[e] = mv_word(r0 + 128 + 32 * half + 16 * e + 4 * t4);
                qh1[e] = mv_word(r1 + 128 + 32 * half + 16 * e + 4 * t4);
                s0[e] = mv_word(r0 + 192 + 8 * half + 4 * e);
                s1[e] = mv_word(r1 + 192 + 8 * half + 4 * e);
            }
#pragma unroll
            for (int rl = 0; rl < 2; rl++) {
                unsigned q0[2], q1[2];
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    q0[e] = mv_word(r0 + 64 * half + 32 * rl + 16 * e + 4 * t4);
                    q1[e] = mv_word(r1 + 64 * half + 32 * rl + 16 * e + 4 * t4);
                }
#pragma unroll
                for (int hi = 0; hi < 2; hi++) {
                    const int blk = 4 * half + 2 * hi + rl;
                    const uint2 b = col ? *reinterpret_cast<const uint2 *>(bq + blk * bq_step) : make_uint2(0u, 0u);
                    const int4 ca = *reinterpret_cast<const int4 *>(sc + blk * sc_step), cb = *reinterpret_cast<const int4 *>(sc + blk * sc_step + 16);  // d, s, -32 sums
                    const int sh = 2 * (2 * hi + rl);
                    int c0[4] = {ca.z, cb.z, ca.z, cb.z}, c1[4] = {ca.w, cb.w, ca.w, cb.w};
                    mv_mma16(c0, ((q0[0] >> (4 * hi)) & 0x0F0F0F0Fu) | (((qh0[0] >> sh) & 0x03030303u) << 4), ((q1[0] >> (4 * hi)) & 0x0F0F0F0Fu) | (((qh1[0] >> sh) & 0x03030303u) << 4), b.x);
                    mv_mma16(c1, ((q0[1] >> (4 * hi)) & 0x0F0F0F0Fu) | (((qh0[1] >> sh) & 0x03030303u) << 4), ((q1[1] >> (4 * hi)) & 0x0F0F0F0Fu) | (((qh1[1] >> sh) & 0x03030303u) << 4), b.y);
                    // scales 2 (2 hi + rl) and + 1 of the half: word hi, bytes 2 rl and 2 rl + 1
                    const int a0 = (int)(signed char)(s0[hi] >> (16 * rl)), a1 = (int)(signed char)(s0[hi] >> (16 * rl + 8)), e0 = (int)(signed char)(s1[hi] >> (16 * rl)),
                              e1 = (int)(signed char)(s1[hi] >> (16 * rl + 8));
                    const float da = __int_as_float(ca.x), db = __int_as_float(cb.x);
                    // (16 x 32 x 127 x 128 is above 2^22: this sum is converted)
                    sd[0] += da * (float)(c0[0] * a0 + c1[0] * a1);
                    sd[1] += db * (float)(c0[1] * a0 + c1[1] * a1);
                    sd[2] += da * (float)(c0[2] * e0 + c1[2] * e1);
                    sd[3] += db * (float)(c0[3] * e0 + c1[3] * e1);
                }
            }
        }
        acc[0] += d0 * sd[0]; acc[1] += d0 * sd[1]; acc[2] += d1 * sd[2]; acc[3] += d1 * sd[3];
    } else {
        constexpr int QS = TYPE == B200_TYPE_Q4_K ? 16 : 48;
        const uint4 h0 = *reinterpret_cast<const uint4 *>(r0), h1 = *reinterpret_cast<const uint4 *>(r1);
        // scales and minima of sub-blocks 0..3 and 4..7, one per byte (get_scale_min_k4)
        const unsigned sc0[2] = {h0.y & 0x3f3f3f3fu, (h0.w & 0x0f0f0f0fu) | ((h0.y >> 2) & 0x30303030u)}, mn0[2] = {h0.z & 0x3f3f3f3fu, ((h0.w >> 4) & 0x0f0f0f0fu) | ((h0.z >> 2) & 0x30303030u)};
        const unsigned sc1[2] = {h1.y & 0x3f3f3f3fu, (h1.w & 0x0f0f0f0fu) | ((h1.y >> 2) & 0x30303030u)}, mn1[2] = {h1.z & 0x3f3f3f3fu, ((h1.w >> 4) & 0x0f0f0f0fu) | ((h1.z >> 2) & 0x30303030u)};
        unsigned f[4] = {0u, 0u, 0u, 0u};  // q5_K: the fifth bits
        if constexpr (TYPE == B200_TYPE_Q5_K) {
            f[0] = *reinterpret_cast<const unsigned *>(r0 + 16 + 4 * t4); f[2] = *reinterpret_cast<const unsigned *>(r0 + 32 + 4 * t4);
            f[1] = *reinterpret_cast<const unsigned *>(r1 + 16 + 4 * t4); f[3] = *reinterpret_cast<const unsigned *>(r1 + 32 + 4 * t4);
        }
        float sd[4] = {0.f, 0.f, 0.f, 0.f}, sm[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 4; c++) {
            unsigned q[4];  // rows g, g + 8 of the chunk's first 16 bytes, then of its last
            q[0] = *reinterpret_cast<const unsigned *>(r0 + QS + 32 * c + 4 * t4); q[2] = *reinterpret_cast<const unsigned *>(r0 + QS + 32 * c + 16 + 4 * t4);
            q[1] = *reinterpret_cast<const unsigned *>(r1 + QS + 32 * c + 4 * t4); q[3] = *reinterpret_cast<const unsigned *>(r1 + QS + 32 * c + 16 + 4 * t4);
#pragma unroll
            for (int hi = 0; hi < 2; hi++) {
                const int sb = 2 * c + hi;
                unsigned x[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    x[i] = (q[i] >> (4 * hi)) & 0x0F0F0F0Fu;
                    if constexpr (TYPE == B200_TYPE_Q5_K) x[i] += ((f[i] >> sb) & 0x01010101u) * 16u;
                }
                const uint2 b = col ? *reinterpret_cast<const uint2 *>(bq + sb * bq_step) : make_uint2(0u, 0u);
                const float4 ds = *reinterpret_cast<const float4 *>(sc + sb * sc_step);  // d, s of column 2 t4; d, s of column 2 t4 + 1
                int k[4] = {0, 0, 0, 0};
                mv_mma32(k, x[0], x[1], x[2], x[3], b.x, b.y);
                const int a = (int)((sc0[sb >> 2] >> (8 * (sb & 3))) & 0xffu), e = (int)((sc1[sb >> 2] >> (8 * (sb & 3))) & 0xffu);
                const float ma = mv_byte(mn0[sb >> 2], sb & 3), me = mv_byte(mn1[sb >> 2], sb & 3);
                if constexpr (TYPE == B200_TYPE_Q4_K) {  // 32 x 15 x 127 x 63 < 2^22
                    sd[0] += ds.x * mv_float(k[0] * a + MV_MAGIC); sd[1] += ds.z * mv_float(k[1] * a + MV_MAGIC);
                    sd[2] += ds.x * mv_float(k[2] * e + MV_MAGIC); sd[3] += ds.z * mv_float(k[3] * e + MV_MAGIC);
                } else {                                 // 32 x 31 x 127 x 63 is not
                    sd[0] += ds.x * (float)(k[0] * a); sd[1] += ds.z * (float)(k[1] * a);
                    sd[2] += ds.x * (float)(k[2] * e); sd[3] += ds.z * (float)(k[3] * e);
                }
                sm[0] += ds.y * ma; sm[1] += ds.w * ma; sm[2] += ds.y * me; sm[3] += ds.w * me;
            }
        }
        const float d0 = h2f((unsigned short)(h0.x & 0xffff)), n0 = h2f((unsigned short)(h0.x >> 16)), d1 = h2f((unsigned short)(h1.x & 0xffff)), n1 = h2f((unsigned short)(h1.x >> 16));
        acc[0] += d0 * sd[0] - n0 * sm[0]; acc[1] += d0 * sd[1] - n0 * sm[1];
        acc[2] += d1 * sd[2] - n1 * sm[2]; acc[3] += d1 * sd[3] - n1 * sm[3];
    }
}

template <int TYPE>
__global__ void __launch_bounds__(MV_NW * 32, 1) mmvq_mma_kernel(const __grid_constant__ MvParams p) {
    constexpr int BB = type_block_bytes(TYPE), PIECES = mv_pieces<TYPE>(), ROW = mv_row<TYPE>(), PER = (MV_ROWS * PIECES + 31) / 32, SB = mv_scale_bytes<TYPE>();
    constexpr bool ALIGNED = TYPE != B200_TYPE_Q6_K;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ float red[MV_NW];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int N = p.n, NC = mv_cols(N), KS = p.ks, SLOTS = p.slots, nsb = (int)(p.m.K / 256), nblk = nsb * 8;
    unsigned char *aq = smem, *as = aq + (size_t)nblk * N * 32;                 // int8 operands; scales
    float *part = reinterpret_cast<float *>(as + (size_t)nblk * NC * SB);       // [2][MV_NW][16 rows x 8 columns]
    unsigned char *ring = reinterpret_cast<unsigned char *>(part + 2 * MV_NW * 128) + (size_t)warp * SLOTS * MV_ROWS * ROW;

    const int groups = MV_NW / KS, grp = warp / KS, kp = warp - grp * KS;       // this warp's group of KS, its part of K
    const int sb0 = kp * nsb / KS, nb = (kp + 1) * nsb / KS - sb0;
    const int step = (int)gridDim.x * groups, first = (int)blockIdx.x + grp * (int)gridDim.x;
    struct Tile { const unsigned char *W; int job; int64_t row; };
    auto tile = [&](int t) {
        int j = 0;
        while (j + 1 < p.m.n_jobs && t >= p.tile0[j + 1]) j++;
        return Tile{(const unsigned char *)p.m.jobs[j].W, j, (int64_t)(t - p.tile0[j]) * MV_ROWS};
    };
    // ---- raw blocks: SLOTS - 1 ahead, over tile ends too; rows past a matrix read its last one
    int ct = first, left = 0, slot_in = 0;
    const unsigned char *src[PER];
    unsigned to[PER];
#pragma unroll
    for (int j = 0; j < PER; j++) { const int i = lane + 32 * j; to[j] = smem_u32(ring) + (unsigned)(i / PIECES * ROW + i % PIECES * 16); }
    auto copy_block = [&]() {
        if (left == 0 && ct < p.n_tiles && nb > 0) {
            const Tile ti = tile(ct);
            ct += step;
            left = nb;
#pragma unroll
            for (int j = 0; j < PER; j++) {
                const int i = lane + 32 * j, r = (i / PIECES) & (MV_ROWS - 1);
                const int64_t row = ti.row + r < p.m.jobs[ti.job].M ? ti.row + r : p.m.jobs[ti.job].M - 1;
                src[j] = ti.W + (size_t)row * p.m.w_row_bytes + (size_t)sb0 * BB + (ALIGNED ? i % PIECES * 16 : 0);
            }
        }
        if (left > 0) {
            left--;
            const unsigned so = (unsigned)(slot_in * MV_ROWS * ROW);
#pragma unroll
            for (int j = 0; j < PER; j++) {
                const int i = lane + 32 * j;
                const bool mine = 32 * (j + 1) <= MV_ROWS * PIECES || i < MV_ROWS * PIECES;
                if constexpr (ALIGNED) {
                    if (mine) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to[j] + so), "l"(src[j]) : "memory");
                } else {
                    const unsigned off = (unsigned)(uintptr_t)src[j] & 15u, at = (unsigned)(i % PIECES * 16);
                    if (mine && at < off + BB) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to[j] + so), "l"(src[j] + (int)(at - off)) : "memory");
                }
                src[j] += BB;
            }
        }
        cp_async_commit();
        slot_in = slot_in + 1 == SLOTS ? 0 : slot_in + 1;
    };
    if (p.m.in_order) pdl_wait();
    for (int i = 0; i < SLOTS - 1; i++) copy_block();
    pdl_wait();
    pdl_trigger();

    // ---- the columns as q8_1, once per CTA: word w (4 values) of a block lies at 2 (w & 3) + (w >> 2), so that a lane's two words are neighbours
    {
        const float *X = behind(p.m.jobs[0].X), *norm_w = behind(p.m.norm_w);
        const int n8 = (int)(p.m.K / 8), items = N * n8;  // 8 values each; 4 neighbouring lanes hold a block (n8 is a multiple of 32)
        __shared__ float nscale[8];
        if (p.m.norm_w != nullptr) {
            for (int n = 0; n < N; n++) {
                const float s = rms_scale(X + (int64_t)n * p.m.x_stride, p.m.K, p.m.norm_eps, red);
                if (threadIdx.x == 0) nscale[n] = s;
            }
            __syncthreads();
        }
        const bool keep = blockIdx.x == 0;
        auto column = [&](int i) { return (int)__umulhi((unsigned)i, p.div_n8); };
        for (int base = 0; base < items; base += 2 * MV_NW * 32) {
            float4 v[2][2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int i = base + u * MV_NW * 32 + threadIdx.x, n = column(i);
                const float4 *x = reinterpret_cast<const float4 *>(X + (int64_t)n * p.m.x_stride) + 2 * (i - n * n8);
                const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
                v[u][0] = i < items ? __ldcg(x) : zero;
                v[u][1] = i < items ? __ldcg(x + 1) : zero;
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int i = base + u * MV_NW * 32 + threadIdx.x, n = column(i), i8 = i - n * n8;
                if (p.m.norm_w != nullptr && i < items) {
                    const float s = nscale[n];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float4 w = ld_behind(reinterpret_cast<const float4 *>(norm_w) + 2 * i8 + h);
                        float4 &x = v[u][h];
                        x.x = x.x * s; x.y = x.y * s; x.z = x.z * s; x.w = x.w * s;
                        if (keep && p.m.norm_out) reinterpret_cast<float4 *>(p.m.norm_out + (int64_t)n * p.m.K)[2 * i8 + h] = x;
                        x.x = x.x * w.x; x.y = x.y * w.y; x.z = x.z * w.z; x.w = x.w * w.w;
                        if (keep && p.m.norm_mul_out) reinterpret_cast<float4 *>(p.m.norm_mul_out + (int64_t)n * p.m.K)[2 * i8 + h] = x;
                    }
                }
                float d, s;
                int lo, hi, sum16;
                quantize_q8_1_group4(v[u][0], v[u][1], lo, hi, d, s, sum16);
                const int hi16 = __shfl_xor_sync(0xffffffffu, sum16, 2);
                if (i < items) {
                    const int blk = i8 >> 2, part = i8 & 3;
                    int *q = reinterpret_cast<int *>(aq + ((size_t)blk * N + n) * 32) + 4 * (part & 1) + (part >> 1);  // words 2 part and 2 part + 1
                    q[0] = lo;
                    q[2] = hi;
                    if (part == 0) {
                        unsigned char *sc = as + ((size_t)blk * NC + n) * SB;
                        *reinterpret_cast<float2 *>(sc) = make_float2(d, s);
                        if constexpr (TYPE == B200_TYPE_Q6_K) *reinterpret_cast<int2 *>(sc + 8) = make_int2(-32 * sum16, -32 * hi16);
                    }
                }
            }
        }
    }
    __syncthreads();

    const bool col = g < N;
    const int cp2 = 2 * t4 < NC ? 2 * t4 : NC - 2;  // (lanes of columns that do not exist read others' scales; their sums are not stored)
    const unsigned char *bq0 = aq + (col ? g : 0) * 32 + 8 * t4, *sc0 = as + cp2 * SB;
    const int bq_step = N * 32, sc_step = NC * SB;
    int slot = 0, buf = 0;
    for (int t = first; t < p.n_tiles; t += step) {
        const Tile ti = tile(t);
        const int64_t M = p.m.jobs[ti.job].M, last = M - 1;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        unsigned at0 = 0, at1 = 0;  // where in its slot row the block starts
        if constexpr (!ALIGNED) {
            const uintptr_t base = (uintptr_t)ti.W + (size_t)sb0 * BB;
            at0 = (unsigned)(base + (size_t)(ti.row + g < M ? ti.row + g : last) * p.m.w_row_bytes) & 15u;
            at1 = (unsigned)(base + (size_t)(ti.row + g + 8 < M ? ti.row + g + 8 : last) * p.m.w_row_bytes) & 15u;
        }
        for (int b = 0; b < nb; b++) {
            if (SLOTS == 3) cp_async_wait<1>(); else cp_async_wait<0>();
            __syncwarp();  // the block has landed for all lanes, and all have left the one before
            copy_block();
            const unsigned char *rows = ring + slot * MV_ROWS * ROW;
            mv_block<TYPE>(rows + g * ROW + at0, rows + (g + 8) * ROW + at1, t4, col, bq0 + (size_t)(sb0 + b) * 8 * bq_step, bq_step, sc0 + (size_t)(sb0 + b) * 8 * sc_step, sc_step, acc);
            if constexpr (!ALIGNED) { at0 = (at0 + BB) & 15u; at1 = (at1 + BB) & 15u; }
            slot = slot + 1 == SLOTS ? 0 : slot + 1;
        }
        // ---- the group's sums meet in a fixed order: part[buf][warp][row][column]
        float *mine = part + ((size_t)buf * MV_NW + warp) * 128;
        *reinterpret_cast<float2 *>(mine + g * 8 + 2 * t4) = make_float2(acc[0], acc[1]);
        *reinterpret_cast<float2 *>(mine + (g + 8) * 8 + 2 * t4) = make_float2(acc[2], acc[3]);
        if (KS > 1) asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(KS * 32) : "memory");
        else __syncwarp();
        const float *all = part + ((size_t)buf * MV_NW + grp * KS) * 128;
        for (int i = kp * 32 + lane; i < 128; i += KS * 32) {
            const int r = i & 15, n = i >> 4;
            if (n >= N || ti.row + r >= M) continue;
            float v = 0.f;
            for (int k = 0; k < KS; k++) v += all[k * 128 + r * 8 + n];
            const int64_t o = (int64_t)n * p.m.dst_stride + ti.row + r;
            if (p.m.raw_dst[ti.job]) p.m.raw_dst[ti.job][o] = v;
            p.m.jobs[ti.job].dst[o] = p.m.residual[ti.job] ? v + p.m.residual[ti.job][o] : v;
        }
        buf ^= 1;
    }
    cp_async_wait<0>();
}

// -1000: not for this kernel (shared memory)
template <int TYPE>
static int launch_mmvq_mma(const MmvqParams &m, int N, cudaStream_t st, bool pdl) {
    MvParams p;
    p.m = m;
    p.m.in_order = !pdl;
    p.n = N;
    p.div_n8 = (unsigned)(((1ull << 32) + m.K / 8 - 1) / (m.K / 8));
    int64_t tiles = 0;
    for (int j = 0; j < m.n_jobs; j++) { p.tile0[j] = (int)tiles; tiles += (m.jobs[j].M + MV_ROWS - 1) / MV_ROWS; }
    p.n_tiles = (int)tiles;
    const int rc = device_props();
    if (rc) return rc;
    const int nsb = (int)(m.K / 256);
    const size_t acts = (size_t)nsb * 8 * (N * 32 + mv_cols(N) * mv_scale_bytes<TYPE>()) + 2 * MV_NW * 128 * sizeof(float), slot = (size_t)MV_NW * MV_ROWS * mv_row<TYPE>(), cap = g_smem_optin - 2048;
    p.slots = acts + 3 * slot <= cap ? 3 : 2;
    if (acts + p.slots * slot > cap) return -1000;
    // the longest warp's blocks: rounds of row tiles times its part of K, and half a block's time a round for the meeting
    double best = -1;
    for (int ks = 1; ks <= MV_NW; ks *= 2) {
        const int64_t at_once = (int64_t)g_sm_count * (MV_NW / ks);
        const double cost = (double)((tiles + at_once - 1) / at_once) * ((nsb + ks - 1) / ks + 0.5);
        if (best < 0 || cost < best) { best = cost; p.ks = ks; }
    }
    const size_t smem = acts + p.slots * slot;
    const auto kern = mmvq_mma_kernel<TYPE>;
    static bool attr_set_dev[16] = {};  // cudaFuncSetAttribute is per device
    int cur_dev = 0;
    B200_CUDA_TRY(cudaGetDevice(&cur_dev));
    bool &attr_set = attr_set_dev[cur_dev & 15];
    if (!attr_set) {
        B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
        attr_set = true;
    }
    const int64_t per_cta = MV_NW / p.ks, ctas = (tiles + per_cta - 1) / per_cta;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ctas < g_sm_count ? ctas : g_sm_count));
    cfg.blockDim = dim3(MV_NW * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p));
    return B200_OK;
}

}  // namespace b200
