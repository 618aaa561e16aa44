// mmvq_mma.cuh -- decode GEMV for 2 to 8 columns over q4_0 / q8_0 / q4_K / q5_K / q6_K weights on the int8 tensor cores.  Included by mmvq.cu.
//
// Same arithmetic as SliceDot (exact integer sums of quants and q8_1 activations per sub-block, scaled in f32), but the integer sums of 16 weight
// rows against all columns come from mma.sync s8 tiles.  What bounds it is issue: unpacking the weights, the same for any column count, and scaling the sums.
//   * a tile has eight columns.  Fewer are packed: of four (two) the tile's columns hold two (four) sub-blocks, each with the activations of its own and zeros
//     for the others', so that one set of sums, and one scaling, serves two (four) sub-blocks.
//   * the sums start from the bits of 1.5 * 2^23, which makes floats of them without a conversion; a sub-block's scale is multiplied in by the same FMA that
//     takes that start away (exact: below 2^24).
//   * minima of q4_K and q5_K (mins . sums of the activations) are one f16 tile a 256-value block, packed as the columns are: both factors are f16 values.
//   * a warp takes 16 rows x one 256-value block at a time; their raw bytes (16-byte cp.async pieces, rows may start at any even byte) wait in a
//     ring of its own, one to three blocks ahead; the ring is filled before the wait for the producer kernel;
//   * the activations of all columns are quantised once per CTA into shared memory, in the order in which a lane reads its operand.  All loads of
//     MV_U x 4096 values are in flight at once, and the norm's squares are taken from the same registers;
//   * KS warps share a row tile, each a part of K; their sums meet in shared memory in a fixed order; two CTAs share row tiles, half of K each, where the columns
//     are long or, with four columns or more, row tiles few.
#pragma once

namespace b200 {

constexpr int MV_NW = MMVQ_NW, MV_ROWS = 16, MV_U = 4;
constexpr bool mv_aligned(int t) { return t == B200_TYPE_Q4_K || t == B200_TYPE_Q5_K; }
template <int TYPE> constexpr int mv_bytes() { return type_block_bytes(TYPE) * 256 / type_block_values(TYPE); }  // of 256 values
template <int TYPE> constexpr int mv_pieces() { return (mv_bytes<TYPE>() + (mv_aligned(TYPE) ? 0 : 14) + 15) / 16; }
template <int TYPE> constexpr int mv_row() { return (mv_pieces<TYPE>() | 1) * 16; }  // 8 rows start in 8 different groups of 4 banks
// beside 32 int8 of a (32-value block, column): d; q4_0: and -8 s; q6_K: and -32 times the sums of both halves
template <int TYPE> constexpr int mv_scale_bytes() { return TYPE == B200_TYPE_Q6_K ? 12 : TYPE == B200_TYPE_Q4_0 ? 8 : 4; }
constexpr int mv_cols(int n) { return (n + 1) & ~1; }  // columns' scales are read two at a time
// bytes of all columns' activations: operands [block][column][32] | scales | q4_K, q5_K: s in f16, [256-value block][column][8]
template <int TYPE> constexpr size_t mv_act_bytes(int64_t K, int n) {
    return (size_t)(K / 32) * (n * 32 + mv_cols(n) * mv_scale_bytes<TYPE>()) + (mv_aligned(TYPE) ? (size_t)(K / 256) * n * 16 : 0);
}

struct MvParams {
    MmvqParams m;
    int n, ks, slots, n_tiles;     // columns, warps a row tile, ring slots
    int c, batch;                  // CTAs that share row tiles, each a part of K; row tiles whose sums wait for one another's parts
    unsigned div_nsb[2];           // 2^32 / (256-value blocks of the CTA's part), rounded up
    int tile0[B200_GEMV_MAX_JOBS]; // first row tile of each job
};

__device__ __forceinline__ void mv_mma32(int (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1, const int (&c)[4]) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c[0]), "r"(c[1]), "r"(c[2]), "r"(c[3]));
}
__device__ __forceinline__ void mv_mma16(int (&c)[4], unsigned a0, unsigned a1, unsigned b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a0), "r"(a1), "r"(b0));
}
__device__ __forceinline__ void mv_mma_f16(float (&d)[4], unsigned a0, unsigned a1, unsigned b0) {  // 16 x 8 x 8
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "f"(0.f));
}
// exact floats of integers below 2^22 in magnitude without a conversion: the integer was added to the bits of 1.5 * 2^23
constexpr int MV_MAGIC = 0x4B400000;
__device__ __forceinline__ float mv_float(int biased) { return __int_as_float(biased) - 12582912.0f; }
__device__ __forceinline__ float mv_byte(unsigned w, int k) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650 + k)) - 8388608.0f; }
// Shared memory by 32-bit addresses and constant offsets.  (Through pointers a word at a 2-byte aligned address took about ten instructions, and a q6_K block 1000.)
extern __shared__ __align__(128) unsigned char mv_smem[];
template <typename T> __device__ __forceinline__ T mv_ld(unsigned at) { return *reinterpret_cast<const T *>(mv_smem + at); }
// words of a run that starts at a 2-byte aligned address: two loads and a shift by what the run's start asks for
struct MvRun {
    unsigned at, sh;
    __device__ __forceinline__ explicit MvRun(unsigned a) : at(a & ~3u), sh((a & 2u) * 8u) {}
    __device__ __forceinline__ unsigned word(int off) const { return __funnelshift_r(mv_ld<unsigned>(at + off), mv_ld<unsigned>(at + off + 4), sh); }
};

// (int)roundf(x) for |x| < 128: the fraction is cut off behind the addition of the float below one half.  (One half itself would lift 0.49999997 to 1; checked for
// every float of the range.)
__device__ __forceinline__ int round_away(float x) { return __float2int_rz(__fadd_rn(x, copysignf(0.49999997f, x))); }
// quantize_q8_1_group4, the same values from fewer instructions.  (A launch of one column, which waits for the latency of a single block and not for issue, is 2 %
// slower with it: 1024 x 1024 q4_K 3.01 -> 3.11 us.)
__device__ __forceinline__ void mv_quantize(const float4 a, const float4 b, int &lo, int &hi, float &d16, float &s16, int &sum16) {
    float amax = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
                       fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    // amax / 127 rounded to nearest: a quotient by the rounded reciprocal is corrected by its remainder (Markstein's theorem; checked for every mantissa), where
    // the remainder is no denormal and amax finite
    constexpr float r127 = 1.0f / 127.0f;
    const float dq = __fmul_rn(amax, r127);
    float d = __fmaf_rn(__fmaf_rn(-127.0f, dq, amax), r127, dq);
    if (!(amax > 1e-25f && amax < 1e38f)) d = __fdiv_rn(amax, 127.0f);
    const float id = d != 0.0f ? __frcp_rn(d) : 0.0f;
    const int q0 = round_away(__fmul_rn(a.x, id)), q1 = round_away(__fmul_rn(a.y, id)), q2 = round_away(__fmul_rn(a.z, id)), q3 = round_away(__fmul_rn(a.w, id));
    const int q4 = round_away(__fmul_rn(b.x, id)), q5 = round_away(__fmul_rn(b.y, id)), q6 = round_away(__fmul_rn(b.z, id)), q7 = round_away(__fmul_rn(b.w, id));
    lo = (int)prmt(prmt((unsigned)q0, (unsigned)q1, 0x0040u), prmt((unsigned)q2, (unsigned)q3, 0x0040u), 0x5410u);
    hi = (int)prmt(prmt((unsigned)q4, (unsigned)q5, 0x0040u), prmt((unsigned)q6, (unsigned)q7, 0x0040u), 0x5410u);
    int s = dp4a(hi, 0x01010101, dp4a(lo, 0x01010101, 0));
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    sum16 = s;
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    d16 = __half2float(__float2half_rn(d));
    s16 = __half2float(__float2half_rn(__fmul_rn((float)s, d)));
}
__device__ __forceinline__ float4 mv_ldcg(const float4 *p) {  // (stays where it stands among the copies)
    float4 v;
    asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned mv_cluster_rank() { unsigned r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void mv_cluster_meet() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// what CTA `rank` of the cluster has written to its shared variable before the meeting
__device__ __forceinline__ float mv_cluster_ld(const float *p, unsigned rank) {
    float v;
    asm volatile("{\n.reg .b32 a;\nmapa.shared::cluster.u32 a, %1, %2;\nld.shared::cluster.f32 %0, [a];\n}\n" : "=f"(v) : "r"(smem_u32(p)), "r"(rank) : "memory");
    return v;
}

// What a lane needs to know of the packing.  NP: columns of a packed group (2, 4 or 8, >= n).  As the operand's column, lane g holds column g % NP of sub-block
// g / NP of a set; its sums are those of columns col and col + 1 of sub-block `sub` of the set.
template <int NP>
struct MvLane {
    static constexpr int G = 8 / NP;
    int t4, gb, sub;
    unsigned mask[G];                  // all ones in the tile that takes this lane's operand
    unsigned bq, sc, su, su_mask;      // operand of the lane's column in the first block; scales from column col on; (K-quants) its f16 sums, and which of the two
    unsigned bq_step, sc_step, ai;     // from a block to the next; ai: q6_K, from the scales to the integer sums
};
__device__ __forceinline__ int mv_sbyte(unsigned w, int k) { return (int)(signed char)(w >> (8 * k)); }

// one 256-value block of rows g and g + 8: acc[0..1] += row g, columns col and col + 1 of sub-block `sub`; acc[2..3] += row g + 8.  r0, r1: the
// rows' first bytes
template <int TYPE, int NP>
__device__ __forceinline__ void mv_block(unsigned r0, unsigned r1, const MvLane<NP> &L, int sb, float (&acc)[4]) {
    constexpr int G = MvLane<NP>::G;
    const int t4 = L.t4;
    const int magic[4] = {MV_MAGIC, MV_MAGIC, MV_MAGIC, MV_MAGIC};
    const unsigned bq = L.bq + sb * 8 * L.bq_step, sc = L.sc + sb * 8 * L.sc_step;
    if constexpr (TYPE == B200_TYPE_Q6_K) {
        // sub-blocks of 16.  NP 8: both halves of a 32-value block in tiles of their own; NP 4: one tile, each half in four of its columns; NP 2: and two
        // blocks, values 64 apart, in one set
        const float d0 = h2f(mv_ld<unsigned short>(r0 + 208)), d1 = h2f(mv_ld<unsigned short>(r1 + 208));
        const MvRun u0(r0), u1(r1), v0(r0 + 4 * t4), v1(r1 + 4 * t4);
        float sd[4] = {0.f, 0.f, 0.f, 0.f};
        const unsigned ci = sc + L.ai + sb * 8 * L.sc_step;  // the block's integer sums
        const int e = L.sub & 1, eb = L.gb & 1, hs = NP == 2 ? L.sub >> 1 : 0, hb = NP == 2 ? L.gb >> 1 : 0;
#pragma unroll
        for (int half = 0; half < 2; half++) {
            unsigned qh0[2], qh1[2], s0[2], s1[2];  // both 16-byte halves' high bits; the half's 8 scales
#pragma unroll
            for (int i = 0; i < 2; i++) {
                qh0[i] = v0.word(128 + 32 * half + 16 * i);
                qh1[i] = v1.word(128 + 32 * half + 16 * i);
                s0[i] = u0.word(192 + 8 * half + 4 * i);
                s1[i] = u1.word(192 + 8 * half + 4 * i);
            }
            if constexpr (NP < 8) {
#pragma unroll
                for (int i = 0; i < 2; i++) { s0[i] >>= 8 * e; s1[i] >>= 8 * e; }
            }
#pragma unroll
            for (int rl = 0; rl < 2; rl++) {
                unsigned q0[2], q1[2];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    q0[i] = v0.word(64 * half + 32 * rl + 16 * i);
                    q1[i] = v1.word(64 * half + 32 * rl + 16 * i);
                }
                unsigned b = 0;
                int k[4];
#pragma unroll
                for (int hi = 0; hi < 2; hi++) {
                    const int blk = 4 * half + 2 * hi + rl, sh = 2 * (2 * hi + rl);
                    unsigned x[4];  // rows g, g + 8 of the first 16 values, then of the last
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        x[2 * i] = ((q0[i] >> (4 * hi)) & 0x0F0F0F0Fu) | (((qh0[i] >> sh) & 0x03030303u) << 4);
                        x[2 * i + 1] = ((q1[i] >> (4 * hi)) & 0x0F0F0F0Fu) | (((qh1[i] >> sh) & 0x03030303u) << 4);
                    }
                    if constexpr (NP == 8) {
                        uint2 b2 = mv_ld<uint2>(bq + blk * L.bq_step);
                        b2.x &= L.mask[0]; b2.y &= L.mask[0];
                        const int2 ca = mv_ld<int2>(ci + 2 * blk * L.sc_step), cb = mv_ld<int2>(ci + (2 * blk + 1) * L.sc_step);
                        const float2 d = mv_ld<float2>(sc + blk * L.sc_step);
                        int c0[4] = {ca.x, ca.y, ca.x, ca.y}, c1[4] = {cb.x, cb.y, cb.x, cb.y};
                        mv_mma16(c0, x[0], x[1], b2.x);
                        mv_mma16(c1, x[2], x[3], b2.y);
                        // scales 2 (2 hi + rl) and + 1 of the half: word hi, bytes 2 rl and 2 rl + 1
                        const int a0 = mv_sbyte(s0[hi], 2 * rl), a1 = mv_sbyte(s0[hi], 2 * rl + 1), e0 = mv_sbyte(s1[hi], 2 * rl), e1 = mv_sbyte(s1[hi], 2 * rl + 1);
                        // (16 x 32 x 127 x 128 is above 2^22: this sum is converted)
                        sd[0] += d.x * (float)(c0[0] * a0 + c1[0] * a1);
                        sd[1] += d.y * (float)(c0[1] * a0 + c1[1] * a1);
                        sd[2] += d.x * (float)(c0[2] * e0 + c1[2] * e1);
                        sd[3] += d.y * (float)(c0[3] * e0 + c1[3] * e1);
                    } else {
                        const int set = NP == 2 ? 4 * half + rl : blk, mine = NP == 2 ? set + 2 * hs : blk;  // the set's first block; the block of this lane's sums
                        if (NP == 4 || hi == 0) b = mv_ld<unsigned>(bq + (NP == 2 ? set + 2 * hb : blk) * L.bq_step + 4 * eb);
                        const unsigned b0 = b & L.mask[NP == 2 ? 2 * hi : 0], b1 = b & L.mask[NP == 2 ? 2 * hi + 1 : 1];
                        if (NP == 4 || hi == 0) {
                            const int2 c = mv_ld<int2>(ci + (2 * mine + e) * L.sc_step);
                            const int start[4] = {c.x, c.y, c.x, c.y};
                            mv_mma32(k, x[0], x[1], x[2], x[3], b0, b1, start);
                        } else {
                            mv_mma32(k, x[0], x[1], x[2], x[3], b0, b1, k);
                        }
                        if (NP == 4 || hi == 1) {
                            const float2 d = mv_ld<float2>(sc + mine * L.sc_step);
                            const int a0 = mv_sbyte(NP == 2 ? (hs ? s0[1] : s0[0]) : s0[hi], 2 * rl), e0 = mv_sbyte(NP == 2 ? (hs ? s1[1] : s1[0]) : s1[hi], 2 * rl);
                            sd[0] += d.x * (float)(k[0] * a0);
                            sd[1] += d.y * (float)(k[1] * a0);
                            sd[2] += d.x * (float)(k[2] * e0);
                            sd[3] += d.y * (float)(k[3] * e0);
                        }
                    }
                }
            }
        }
        acc[0] += d0 * sd[0]; acc[1] += d0 * sd[1]; acc[2] += d1 * sd[2]; acc[3] += d1 * sd[3];
    } else if constexpr (mv_aligned(TYPE)) {
        constexpr int QS = TYPE == B200_TYPE_Q4_K ? 16 : 48;
        const uint4 h0 = mv_ld<uint4>(r0), h1 = mv_ld<uint4>(r1);
        // scales and minima of sub-blocks 0..3 and 4..7, one per byte (get_scale_min_k4); scales: from this lane's sub-block of a set on
        const int by = G == 1 ? 0 : 8 * L.sub;
        const unsigned sc0[2] = {(h0.y & 0x3f3f3f3fu) >> by, ((h0.w & 0x0f0f0f0fu) | ((h0.y >> 2) & 0x30303030u)) >> by};
        const unsigned sc1[2] = {(h1.y & 0x3f3f3f3fu) >> by, ((h1.w & 0x0f0f0f0fu) | ((h1.y >> 2) & 0x30303030u)) >> by};
        unsigned f[4] = {0u, 0u, 0u, 0u};  // q5_K: the fifth bits
        if constexpr (TYPE == B200_TYPE_Q5_K) {
            f[0] = mv_ld<unsigned>(r0 + 16 + 4 * t4); f[2] = mv_ld<unsigned>(r0 + 32 + 4 * t4);
            f[1] = mv_ld<unsigned>(r1 + 16 + 4 * t4); f[3] = mv_ld<unsigned>(r1 + 32 + 4 * t4);
        }
        float sd[4] = {0.f, 0.f, 0.f, 0.f};
        uint2 b = make_uint2(0u, 0u);
        int k[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            unsigned q[4];  // rows g, g + 8 of the chunk's first 16 bytes, then of its last
            q[0] = mv_ld<unsigned>(r0 + QS + 32 * c + 4 * t4); q[2] = mv_ld<unsigned>(r0 + QS + 32 * c + 16 + 4 * t4);
            q[1] = mv_ld<unsigned>(r1 + QS + 32 * c + 4 * t4); q[3] = mv_ld<unsigned>(r1 + QS + 32 * c + 16 + 4 * t4);
#pragma unroll
            for (int hi = 0; hi < 2; hi++) {
                const int blk = 2 * c + hi, j = blk % G, set = blk - j;
                unsigned x[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    x[i] = (q[i] >> (4 * hi)) & 0x0F0F0F0Fu;
                    if constexpr (TYPE == B200_TYPE_Q5_K) x[i] += ((f[i] >> blk) & 0x01010101u) * 16u;
                }
                if (j == 0) b = mv_ld<uint2>(bq + (set + (G == 1 ? 0 : L.gb)) * L.bq_step);
                if (j == 0) mv_mma32(k, x[0], x[1], x[2], x[3], b.x & L.mask[0], b.y & L.mask[0], magic);
                else mv_mma32(k, x[0], x[1], x[2], x[3], b.x & L.mask[j], b.y & L.mask[j], k);
                if (j == G - 1) {
                    const float2 d = mv_ld<float2>(sc + (set + (G == 1 ? 0 : L.sub)) * L.sc_step);
                    const float a = mv_byte(sc0[set >> 2], set & 3), e = mv_byte(sc1[set >> 2], set & 3), na = -12582912.0f * a, ne = -12582912.0f * e;
                    sd[0] += d.x * fmaf(__int_as_float(k[0]), a, na); sd[1] += d.y * fmaf(__int_as_float(k[1]), a, na);
                    sd[2] += d.x * fmaf(__int_as_float(k[2]), e, ne); sd[3] += d.y * fmaf(__int_as_float(k[3]), e, ne);
                }
            }
        }
        // minima 2 t4 and 2 t4 + 1 of both rows as f16 (1024 + m in the mantissa)
        const __half2 off = __half2half2(__ushort_as_half(0x6400));
        unsigned m[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const uint4 &h = i ? h1 : h0;
            const unsigned w = (t4 < 2 ? h.z & 0x3f3f3f3fu : ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u)) >> (16 * (t4 & 1));
            const unsigned x = __byte_perm(w, 0x64646464u, 0x4140);
            const __half2 y = __hsub2(*reinterpret_cast<const __half2 *>(&x), off);
            m[i] = *reinterpret_cast<const unsigned *>(&y);
        }
        float sm[4];
        mv_mma_f16(sm, m[0], m[1], mv_ld<unsigned>(L.su + (size_t)sb * (L.bq_step / 2)) & L.su_mask);
        const float d0 = h2f((unsigned short)(h0.x & 0xffff)), n0 = h2f((unsigned short)(h0.x >> 16)), d1 = h2f((unsigned short)(h1.x & 0xffff)), n1 = h2f((unsigned short)(h1.x >> 16));
        // (here and not behind the row: of activations of one sign two large sums would be left, of whose difference little remains)
        acc[0] = fmaf(-n0, sm[0], fmaf(d0, sd[0], acc[0])); acc[1] = fmaf(-n0, sm[1], fmaf(d0, sd[1], acc[1]));
        acc[2] = fmaf(-n1, sm[2], fmaf(d1, sd[2], acc[2])); acc[3] = fmaf(-n1, sm[3], fmaf(d1, sd[3], acc[3]));
    } else {
        constexpr int BB = type_block_bytes(TYPE);
        const MvRun e0(r0 + 2 + 4 * t4), e1(r1 + 2 + 4 * t4), o0(r0 + 2 + BB + 4 * t4), o1(r1 + 2 + BB + 4 * t4);  // quants of even and odd blocks
        uint2 b = make_uint2(0u, 0u);
        int k[4];
        float sd[4] = {0.f, 0.f, 0.f, 0.f};  // a block's sum by itself: chains of roundings are shorter (1.2e-7 off the exact sum of 5120 values at six columns -> 7.9e-8)
#pragma unroll
        for (int blk = 0; blk < 8; blk++) {
            const int j = blk % G, set = blk - j, at = 2 * BB * (blk / 2);
            const MvRun &w0 = blk & 1 ? o0 : e0, &w1 = blk & 1 ? o1 : e1;
            unsigned x[4];
            if constexpr (TYPE == B200_TYPE_Q4_0) {
                const unsigned q0 = w0.word(at), q1 = w1.word(at);
                x[0] = q0 & 0x0F0F0F0Fu; x[1] = q1 & 0x0F0F0F0Fu; x[2] = (q0 >> 4) & 0x0F0F0F0Fu; x[3] = (q1 >> 4) & 0x0F0F0F0Fu;
            } else {
                x[0] = w0.word(at); x[1] = w1.word(at);
                x[2] = w0.word(at + 16); x[3] = w1.word(at + 16);
            }
            if (j == 0) b = mv_ld<uint2>(bq + (set + (G == 1 ? 0 : L.gb)) * L.bq_step);
            if (j == 0) mv_mma32(k, x[0], x[1], x[2], x[3], b.x & L.mask[0], b.y & L.mask[0], magic);
            else mv_mma32(k, x[0], x[1], x[2], x[3], b.x & L.mask[j], b.y & L.mask[j], k);
            if (j == G - 1) {
                const int mine = set + (G == 1 ? 0 : L.sub);
                const float d0 = h2f(mv_ld<unsigned short>(r0 + BB * mine)), d1 = h2f(mv_ld<unsigned short>(r1 + BB * mine));
                if constexpr (TYPE == B200_TYPE_Q4_0) {
                    const float4 d = mv_ld<float4>(sc + mine * L.sc_step);  // d, -8 s of both columns
                    sd[0] += d0 * fmaf(d.x, mv_float(k[0]), d.y); sd[1] += d0 * fmaf(d.z, mv_float(k[1]), d.w);
                    sd[2] += d1 * fmaf(d.x, mv_float(k[2]), d.y); sd[3] += d1 * fmaf(d.z, mv_float(k[3]), d.w);
                } else {
                    const float2 d = mv_ld<float2>(sc + mine * L.sc_step);
                    sd[0] += d0 * d.x * mv_float(k[0]); sd[1] += d0 * d.y * mv_float(k[1]);
                    sd[2] += d1 * d.x * mv_float(k[2]); sd[3] += d1 * d.y * mv_float(k[3]);
                }
            }
        }
        acc[0] += sd[0]; acc[1] += sd[1]; acc[2] += sd[2]; acc[3] += sd[3];
    }
}

// NORM: there is a norm.  (A kernel of its own: in one for both, which needs all registers, its sums made the loop over the blocks 3 to 6 % slower.)
template <int TYPE, int NP, bool NORM>
__global__ void __launch_bounds__(MV_NW * 32, 1) mmvq_mma_kernel(const __grid_constant__ MvParams p) {
    constexpr int BB = mv_bytes<TYPE>(), PIECES = mv_pieces<TYPE>(), ROW = mv_row<TYPE>(), PER = (MV_ROWS * PIECES + 31) / 32;
    constexpr bool ALIGNED = mv_aligned(TYPE);
    unsigned char *smem = mv_smem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    const int N = p.n, NC = mv_cols(N), KS = p.ks, SLOTS = p.slots, nsb_all = (int)(p.m.K / 256);
    const int C = p.c, rank = C > 1 ? (int)mv_cluster_rank() : 0, cluster = (int)blockIdx.x / C, n_clusters = (int)gridDim.x / C;
    const int sbk = rank * nsb_all / C, nsb = (rank + 1) * nsb_all / C - sbk, nblk = nsb * 8;  // this CTA's part of K
    // scales: d [block][column] (q4_0: d, -8 s); q6_K: then the integer sums [block][half][column]; K-quants: s
    const int sc_step = NC * (TYPE == B200_TYPE_Q4_0 ? 8 : 4);
    unsigned char *aq = smem, *as = aq + (size_t)nblk * N * 32, *ai = as + (size_t)nblk * sc_step;
    float *part = reinterpret_cast<float *>(smem + (mv_act_bytes<TYPE>((nsb_all + C - 1) / C * 256, N) + 127) / 128 * 128);  // [2][MV_NW][16 rows x 8 columns]
    float *sums = part + 2 * MV_NW * 128;                                       // C > 1: [batch][N][16 rows]
    unsigned char *ring = reinterpret_cast<unsigned char *>(sums + p.batch * N * MV_ROWS) + (size_t)warp * SLOTS * MV_ROWS * ROW;

    const int groups = MV_NW / KS, grp = warp / KS, kp = warp - grp * KS;       // this warp's group of KS, its part of K
    const int sb0 = kp * nsb / KS, nb = (kp + 1) * nsb / KS - sb0;
    const int step = n_clusters * groups, first = cluster + grp * n_clusters;
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
                src[j] = ti.W + (size_t)row * p.m.w_row_bytes + (size_t)(sbk + sb0) * BB + (ALIGNED ? i % PIECES * 16 : 0);
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
    if (!p.m.in_order) copy_block();
    pdl_wait();
    pdl_trigger();

    // ---- the columns as q8_1, once per CTA: word w (4 values) of a block lies at 2 (w & 3) + (w >> 2), so that a lane's two words are neighbours.  Their loads
    // go out in front of the weights: behind some 100 KB of those they would wait for a microsecond.
    {
        const int64_t k0 = (int64_t)sbk * 256;
        const float *X = behind(p.m.jobs[0].X) + k0, *norm_w = NORM ? behind(p.m.norm_w) + k0 : nullptr;
        // 32 neighbouring lanes take 256 values of a column, 8 each: row w of [column][256-value block]; 4 lanes hold a block of 32
        const int rows = N * nsb, uwarp = __shfl_sync(0xffffffffu, warp, 0);
        __shared__ float nscale[8];
        const bool keep = cluster == 0;
        const unsigned div_nsb = p.div_nsb[rank];
        const int q_lane = (lane >> 2) * N * 32 + 16 * (lane & 1) + 4 * ((lane >> 1) & 1);  // words 2 q and 2 q + 1 of a block lie at 2 (w & 3) + (w >> 2), q = lane & 3
        constexpr int CHUNK = MV_U * MV_NW;
        float4 v[MV_U][2];
        auto load = [&](int base) {
#pragma unroll
            for (int u = 0; u < MV_U; u++) {
                const int w = base + u * MV_NW + uwarp, n = nsb == 1 ? w : (int)__umulhi((unsigned)w, div_nsb);
                v[u][0] = v[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (w < rows) {
                    const float4 *x = reinterpret_cast<const float4 *>(X + (int64_t)n * p.m.x_stride + (w - n * nsb) * 256) + 2 * lane;
                    v[u][0] = mv_ldcg(x);
                    v[u][1] = mv_ldcg(x + 1);
                }
            }
        };
        load(0);
        for (int i = p.m.in_order ? 0 : 1; i < SLOTS - 1; i++) copy_block();
        if constexpr (NORM) {
            // The sum of squares in the order of rms_scale, so that a column's norm, and with it its quants, is the same whichever kernel takes it: squares of four values
            // each, in aq ([column][four values], the quants come later), then thread t adds those of t, t + 512, ...  With two CTAs: of both.
            float *sq = reinterpret_cast<float *>(aq);
            for (int base = 0;;) {
#pragma unroll
                for (int u = 0; u < MV_U; u++) {
                    const int w = base + u * MV_NW + uwarp;
                    if (w < rows) reinterpret_cast<float2 *>(sq)[w * 32 + lane] = make_float2(square4(v[u][0]), square4(v[u][1]));
                }
                base += CHUNK;
                if (base >= rows) break;
                load(base);
            }
            if (C > 1) mv_cluster_meet();
            else __syncthreads();
            auto add_up = [&](auto square) {
                float ss[NP];
#pragma unroll
                for (int n = 0; n < NP; n++) ss[n] = 0.f;
#pragma unroll 2
                for (int i4 = threadIdx.x; i4 < nsb_all * 64; i4 += MV_NW * 32) {
#pragma unroll
                    for (int n = 0; n < NP; n++) ss[n] += square(n < N ? n : 0, i4);  // (of columns that do not exist: another's, for nobody)
                }
#pragma unroll
                for (int n = 0; n < NP; n++) {
                    const float s = warp_sum(ss[n]);
                    if (lane == 0) part[n * MV_NW + warp] = s;
                }
            };
            const int first4 = nsb_all / 2 * 64;  // where the second CTA's part begins
            if (C == 1) add_up([&](int n, int i4) { return sq[n * nsb * 64 + i4]; });
            else add_up([&](int n, int i4) { const bool far = i4 >= first4; return mv_cluster_ld(sq + n * (far ? nsb_all * 64 - first4 : first4) + (far ? i4 - first4 : i4), far); });
            if (C > 1) mv_cluster_meet();  // (and both have read the squares)
            else __syncthreads();
            if (warp < N) {
                const float s = warp_sum(lane < MV_NW ? part[warp * MV_NW + lane] : 0.f);
                if (lane == 0) nscale[warp] = rsqrtf(s / (float)p.m.K + p.m.norm_eps);
            }
            __syncthreads();
            if (rows > CHUNK) load(0);
        }
        for (int base = 0; base < rows; base += CHUNK) {
            if (base > 0) load(base);
#pragma unroll
            for (int u = 0; u < MV_U; u++) {
                const int w = base + u * MV_NW + uwarp, n = nsb == 1 ? w : (int)__umulhi((unsigned)w, div_nsb), sb = w - n * nsb;
                if (w >= rows) continue;
                if constexpr (NORM) {
                    const float s = nscale[n];
                    const int i4 = sb * 64 + 2 * lane;
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const float4 g4 = ld_behind(reinterpret_cast<const float4 *>(norm_w) + i4 + h);
                        float4 &x = v[u][h];
                        x.x = x.x * s; x.y = x.y * s; x.z = x.z * s; x.w = x.w * s;
                        if (keep && p.m.norm_out) reinterpret_cast<float4 *>(p.m.norm_out + (int64_t)n * p.m.K + k0)[i4 + h] = x;
                        x.x = x.x * g4.x; x.y = x.y * g4.y; x.z = x.z * g4.z; x.w = x.w * g4.w;
                        if (keep && p.m.norm_mul_out) reinterpret_cast<float4 *>(p.m.norm_mul_out + (int64_t)n * p.m.K + k0)[i4 + h] = x;
                    }
                }
                float d, s;
                int lo, hi, sum16;
                mv_quantize(v[u][0], v[u][1], lo, hi, d, s, sum16);
                const int hi16 = __shfl_xor_sync(0xffffffffu, sum16, 2);
                int *q = reinterpret_cast<int *>(mv_smem + ((sb * 8 * N + n) * 32 + q_lane));
                q[0] = lo;
                q[2] = hi;
                if ((lane & 3) == 0) {
                    const int blk = sb * 8 + (lane >> 2);
                    float *sc = reinterpret_cast<float *>(as + blk * sc_step);
                    if constexpr (TYPE == B200_TYPE_Q4_0) reinterpret_cast<float2 *>(sc)[n] = make_float2(d, -8.0f * s);
                    else sc[n] = d;
                    if constexpr (TYPE == B200_TYPE_Q6_K) {
                        int *sums32 = reinterpret_cast<int *>(ai + blk * 2 * sc_step);
                        sums32[n] = -32 * sum16;
                        sums32[NC + n] = -32 * hi16;
                    }
                    if constexpr (ALIGNED) reinterpret_cast<__half *>(ai)[(sb * N + n) * 8 + (lane >> 2)] = __float2half_rn(s);  // (s is an f16 value)
                }
            }
        }
    }
    __syncthreads();

    MvLane<NP> L;
    const int ncol = g % NP, c2 = 2 * t4 % NP, cp2 = c2 < NC ? c2 : NC - 2;  // (lanes of columns that do not exist read others' scales; their sums are not stored)
    L.t4 = t4;
    L.gb = g / NP;
    L.sub = 2 * t4 / NP;
#pragma unroll
    for (int j = 0; j < MvLane<NP>::G; j++) L.mask[j] = ncol < N && j == L.gb ? 0xffffffffu : 0u;
    L.bq = (unsigned)(aq - smem) + (ncol < N ? ncol : 0) * 32 + 8 * t4;
    L.bq_step = N * 32;
    L.sc = (unsigned)(as - smem) + cp2 * (TYPE == B200_TYPE_Q4_0 ? 8 : 4);
    L.sc_step = sc_step;
    L.ai = (unsigned)(ai - as);
    L.su = (unsigned)(ai - smem) + (ncol < N ? ncol : 0) * 16 + 4 * t4;
    // of the sub-blocks 2 t4 and 2 t4 + 1, those whose sums this column of the tile holds
    L.su_mask = ncol >= N || (NP == 2 && L.gb >> 1 != (t4 & 1)) ? 0u : NP == 8 ? 0xffffffffu : L.gb & 1 ? 0xffff0000u : 0x0000ffffu;
    auto store = [&](const Tile &ti, int r, int n, float v) {
        const int64_t o = (int64_t)n * p.m.dst_stride + ti.row + r;
        if (p.m.raw_dst[ti.job]) p.m.raw_dst[ti.job][o] = v;
        p.m.jobs[ti.job].dst[o] = p.m.residual[ti.job] ? v + p.m.residual[ti.job][o] : v;
    };
    int slot = 0, buf = 0, t = first;
    for (int t0 = cluster; t0 < p.n_tiles; t0 += p.batch * n_clusters) {
    const int t1 = C > 1 && t0 + p.batch * n_clusters < p.n_tiles ? t0 + p.batch * n_clusters : p.n_tiles;  // (one CTA: all at once)
    for (; t < t1; t += step) {
        const Tile ti = tile(t);
        const int64_t M = p.m.jobs[ti.job].M, last = M - 1;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        unsigned at0 = 0, at1 = 0;  // where in its slot row the block starts
        if constexpr (!ALIGNED) {
            const uintptr_t base = (uintptr_t)ti.W + (size_t)(sbk + sb0) * BB;
            at0 = (unsigned)(base + (size_t)(ti.row + g < M ? ti.row + g : last) * p.m.w_row_bytes) & 15u;
            at1 = (unsigned)(base + (size_t)(ti.row + g + 8 < M ? ti.row + g + 8 : last) * p.m.w_row_bytes) & 15u;
        }
        for (int b = 0; b < nb; b++) {
            if (SLOTS == 4) cp_async_wait<2>(); else if (SLOTS == 3) cp_async_wait<1>(); else cp_async_wait<0>();
            __syncwarp();  // the block has landed for all lanes, and all have left the one before
            copy_block();
            __syncwarp();  // (mma.sync and bar.sync want a warp that is together: nothing but this promises it behind a branch that lanes take differently)
            const unsigned rows = (unsigned)(ring - smem) + slot * MV_ROWS * ROW;
            mv_block<TYPE, NP>(rows + g * ROW + at0, rows + (g + 8) * ROW + at1, L, sb0 + b, acc);
            if constexpr (!ALIGNED) { at0 = (at0 + BB) & 15u; at1 = (at1 + BB) & 15u; }
            slot = slot + 1 == SLOTS ? 0 : slot + 1;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (NP <= 2) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 1);
            if (NP <= 4) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 2);
        }
        // ---- the group's sums meet in a fixed order: part[buf][warp][row][column]
        float *mine = part + ((size_t)buf * MV_NW + warp) * 128;
        if (2 * t4 < NP) {
            *reinterpret_cast<float2 *>(mine + g * 8 + 2 * t4) = make_float2(acc[0], acc[1]);
            *reinterpret_cast<float2 *>(mine + (g + 8) * 8 + 2 * t4) = make_float2(acc[2], acc[3]);
        }
        __syncwarp();
        if (KS > 1) asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(KS * 32) : "memory");
        const float *all = part + ((size_t)buf * MV_NW + grp * KS) * 128;
        for (int i = kp * 32 + lane; i < 128; i += KS * 32) {
            const int r = i & 15, n = i >> 4;
            if (n >= N || ti.row + r >= M) continue;
            // K-quants in pairs, which rounds less.  (For the others a chain: what pairs do to the registers of their kernels makes 32000 x 1024 q8_0 with two to four columns 6 to 8 %
            // slower; what the chain does to those of K-quants, 32000 x 8192 q4_K with three and four 10 %.)
            const float *x = all + r * 8 + n;
            float v = x[0];
            if constexpr (type_block_values(TYPE) == 256) {
                if (KS == 2) v += x[128];
                else if (KS >= 4) {
                    v = (v + x[128]) + (x[256] + x[384]);
                    for (int k = 4; k < KS; k += 4) v += (x[k * 128] + x[k * 128 + 128]) + (x[k * 128 + 256] + x[k * 128 + 384]);
                }
            } else {
                for (int k = 1; k < KS; k++) v += x[k * 128];
            }
            if (C > 1) sums[((t - t0) / n_clusters * N + n) * MV_ROWS + r] = v;
            else store(ti, r, n, v);
        }
        __syncwarp();
        buf ^= 1;
    }
    if (C == 1) break;
    // ---- the halves of K meet: each CTA stores half of the batch's columns of 16 rows
    mv_cluster_meet();
    const int cols = (t1 - t0 + n_clusters - 1) / n_clusters * N, end = (rank + 1) * cols / 2;
    for (int i = rank * cols / 2 + (int)threadIdx.x / MV_ROWS; i < end; i += MV_NW * 32 / MV_ROWS) {
        const int li = i / N, n = i - li * N, r = threadIdx.x % MV_ROWS;
        const Tile ti = tile(t0 + li * n_clusters);
        if (ti.row + r >= p.m.jobs[ti.job].M) continue;
        const float *at = sums + i * MV_ROWS + r;
        store(ti, r, n, mv_cluster_ld(at, 0) + mv_cluster_ld(at, 1));
    }
    mv_cluster_meet();
    }
    cp_async_wait<0>();
}

// -1000: not for this kernel (shared memory)
template <int TYPE, int NP, bool NORM = false>
static int launch_mmvq_mma(const MmvqParams &m, int N, cudaStream_t st, bool pdl) {
    if constexpr (!NORM) {
        if (m.norm_w) return launch_mmvq_mma<TYPE, NP, true>(m, N, st, pdl);
    }
    MvParams p;
    p.m = m;
    p.m.in_order = !pdl;
    p.n = N;
    int64_t tiles = 0;
    for (int j = 0; j < m.n_jobs; j++) { p.tile0[j] = (int)tiles; tiles += (m.jobs[j].M + MV_ROWS - 1) / MV_ROWS; }
    p.n_tiles = (int)tiles;
    const int rc = device_props();
    if (rc) return rc;
    const int nsb = (int)(m.K / 256);
    // How K is cut, into halves for two CTAs and among warps.  With two and three columns it follows from K and the columns alone, so that a row's bits do not depend on the
    // launch it is part of; with more, where few rows leave most of the device idle, from the rows too.  Two CTAs share row tiles where the columns are many enough to quantise
    // that half the work makes up for the meeting (about 1 us): 5120 x 13824 q6_K at 4 columns 32.3 -> 27.8 us, 4096 x 11008 q4_K 17.0 -> 15.8; 4096 x 4096 q4_0 at 4 columns
    // 8.4 -> 8.6, 22016 x 4096 q4_K 21.8 -> 23.4.  (The line is not sharp: between 20000 and 33000 values two CTAs are 0.94 .. 1.07 times as fast from 4096 rows on, and 0.95 .. 1.23 at
    // 1536 and 2400 rows; at 16400 values 0.90 .. 0.98 and 0.97 .. 1.09.)  Where half of the SMs would have no tile, from fewer values on: 512 rows, one CTA -> two with all warps on a tile, 4 columns,
    // 4096 q8_0 8.7 -> 6.6, 5120 q6_K 10.5 -> 8.9; 3072 q4_0 (12288 values) 5.2 -> 5.3.  Two and three columns over 16000 values: level
    // where rows are many (22016 x 8192 q4_K at 2 columns 1.11 and 1.07 of dp4a's speed), 512 x 8192 q6_K at 2 columns 8.6 -> 7.3, q4_0 at 3 8.5 -> 7.0.
    const bool by_rows = N >= 4;
    p.c = nsb >= 2 && m.K * N >= (!by_rows ? 16000 : tiles > g_sm_count / 2 ? 26000 : m.K >= 4096 ? 12000 : 13000) ? 2 : 1;
    const int per = (nsb + p.c - 1) / p.c;
    // (warps a tile: more of them help where rows are few, and meet more often where they are many.  One CTA, 2 columns, with 1, 2, 4, 8 warps: 4096 x 4096 q4_0 9.8,
    // 7.4, 7.1, 7.2 us, 22016 x 4096 q4_K 18.3, 19.3, 19.5, 20.8; two CTAs, 4 columns, 5120 x 13824 q6_K 32.6, 27.8, 29.3, 28.2)
    p.ks = p.c == 2 ? (per >= 24 ? 8 : per >= 16 ? 4 : 2) : per >= 32 ? 8 : per >= 8 ? 4 : per >= 4 ? 2 : 1;
    // Few tiles leave warps idle that could take a part: with rows of up to 1792 values (1024 x 512 q5_K at 4 columns 4.6 -> 4.0), and with two CTAs.  One CTA's longer rows are
    // level or slower so (512 x 5120 q4_0 at 4 columns 7.3 -> 8.2): what they wait for is the quantisation.
    const int64_t at_once = g_sm_count / p.c, tiles_each = (tiles + at_once - 1) / at_once;
    if (by_rows && (per < 8 || p.c == 2)) {
        for (int ks = MV_NW / (tiles_each <= 1 ? 1 : tiles_each <= 2 ? 2 : tiles_each <= 4 ? 4 : MV_NW); ks > p.ks; ks /= 2)
            if (ks <= per) p.ks = ks;
    }
    for (int r = 0; r < 2; r++) {
        const unsigned each = (unsigned)((r + 1) * nsb / p.c - r * nsb / p.c);
        p.div_nsb[r] = each > 1 ? (unsigned)(((1ull << 32) + each - 1) / each) : 0;
    }
    p.batch = p.c == 1 ? 0 : (int)((tiles_each < 64 ? tiles_each : 64) + MV_NW - 1) / MV_NW * MV_NW;  // (a multiple of the groups: a group's tiles follow one another)
    const size_t slot = (size_t)MV_NW * MV_ROWS * mv_row<TYPE>(), cap = g_smem_optin - 2048;
    auto beside = [&]() { return (mv_act_bytes<TYPE>((int64_t)per * 256, N) + 127) / 128 * 128 + (2 * MV_NW * 128 + p.batch * N * MV_ROWS) * sizeof(float); };  // the ring
    while (p.batch > MV_NW && beside() + 2 * slot > cap) p.batch -= MV_NW;
    const size_t acts = beside();
    p.slots = acts + 4 * slot <= cap ? 4 : acts + 3 * slot <= cap ? 3 : 2;
    if (acts + p.slots * slot > cap) return -1000;
    const size_t smem = acts + p.slots * slot;
    const auto kern = mmvq_mma_kernel<TYPE, NP, NORM>;
    static bool attr_set_dev[16] = {};  // cudaFuncSetAttribute is per device
    int cur_dev = 0;
    B200_CUDA_TRY(cudaGetDevice(&cur_dev));
    bool &attr_set = attr_set_dev[cur_dev & 15];
    if (!attr_set) {
        B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
        attr_set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(p.c * (tiles < at_once ? tiles : at_once)));
    cfg.blockDim = dim3(MV_NW * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)p.c;
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = p.c > 1 ? 2 : 1;
    B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, p));
    return B200_OK;
}

}  // namespace b200
