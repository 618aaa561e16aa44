// mmq_pair.cuh -- the prompt GEMM on pairs of SMs (tcgen05 cta_group::2), persistent over its tiles.  Included by mmq.cu, which holds the
// block formats and the entry points.
//
//   dst[n][m] = sum_k W[m][k] * X[n][k]     W quantised (or dense bf16), X bf16 rows in the workspace, dst f32
//
// What bounds it: the tensor pipe once the weights are unpacked fast enough, and before that the L2.  One CTA with a 128 x 256 tile
// fetches 32 KB of activations per K step of 64 (512 tensor cycles): 64 B per cycle and SM, more than the L2 gives 148 SMs.  So two CTAs
// share a 256 x BN tile: each unpacks its own 128 weight rows into its shared memory and fetches HALF of the activation rows, and the
// pair's one MMA reads both halves.
//   * 16 producer warps a CTA, 8 weight rows each: a warp copies the raw blocks of its rows (256 values of each, contiguous 16-byte cp.async) into
//     a ring of its own, one or two groups ahead, and unpacks them with packed f32 arithmetic, lane = (K step, half, row), two K
//     steps at a time into the 128-byte-swizzled operand tiles.  No barrier among the warps.
//   * a stage holds those two K steps (dense weights: one).  Waiting, passing on and committing cost each warp about 60 instructions among 20 warps, per
//     stage: with a stage of one step q4_K took 0.324 us a step of 64 values at 64 columns and 0.331 at 128, with two 0.288 and 0.295; a
//     launch's start and end went from 10.6 .. 16 to 8.3 .. 11 us.
//   * the MMA warp walks through its loop as a whole and elects a lane for the tcgen05 instructions only: loop counters and descriptors then
//     live in uniform registers.  (With one lane in the loop every MMA needed a dozen vector instructions, each of which waits its turn
//     among the producers: 190 cycles an MMA whatever its width.)
//   * the accumulators are double-buffered in TMEM (2 x 256 columns): four epilogue warps store tile i while tile i + 1 is computed.  The last tile, with
//     nothing behind it, is stored by all that are left, twenty warps (dense weights: twelve): 6144 x 4096 bf16 over 512 columns 28 -> 22 us,
//     11008 x 4096 q4_K 55.5 -> 49.1.
//   * where the tiles leave pairs idle, a cluster of up to eight pairs takes one tile, each a part of K; the parts meet in distributed shared memory and are
//     added in the order of K (pair_merge).  5120 x 5120 over 199 columns, 20 tiles in three parts: q5_K 32.4 -> 21.9 us, q6_K 43 -> 24; 1024 x 4096 q4_K over
//     300 columns, 12 in four, 19.4 -> 13.6; 256 x 5120 q6_K over 400, 5 in seven, 24.7 -> 13.5.  Rows whose tiles are left over behind whole waves are a launch of their own
//     where that is shorter (mmq_pair_whole_waves).
//   * BN is chosen on the host so that the tiles fill the pairs evenly (mmq_pair_plan): 512 columns are 2 x 256 or 3 x 176, whichever leaves
//     the last wave fuller.  In the grouped form (routed experts) the width of every tile follows its rows.
// Every wait has a limit (MmqParams::wait_limit).  A role whose wait runs out sets `failed` of its CTA and leaves its loop: no store, copy or MMA, and no
// arrival (an arrival that no wait stands before could find a phase whose arrivals are all there, waiting for bytes only).  Whoever
// waits for it, in either CTA, gives up in turn.  An accumulator is announced when the operands of all its K steps had arrived, so what is
// stored is right (of several parts of K nothing is stored unless all of them are there); the rest of the result stays as it was, *timeout is set, and the CTA stays until
// copies and MMAs in flight have ended.
#pragma once

namespace b200 {

constexpr int PAIR_PRODUCERS = 16;                   // warps that unpack, 8 rows of the CTA's 128 each
constexpr int PAIR_MAX_STAGES = 8;
constexpr int PAIR_MAX_SPLIT = 8;                    // parts of K: a cluster of 16 CTAs at most
constexpr int PAIR_SMEM = 232448 - 1024 - 1024;      // dynamic shared memory: what a CTA can have, less static data and alignment

// 256-value groups of 128 rows as they lie in memory: 16-byte pieces a row (a 2-byte aligned row starts up to 14 bytes into its first one)
__host__ __device__ constexpr bool raw_aligned(int t) { return t == B200_TYPE_Q4_K || t == B200_TYPE_Q5_K; }
__host__ __device__ constexpr int raw_pieces(int t) { return (group256_bytes(t) + (raw_aligned(t) ? 0 : 14) + 15) / 16; }
__host__ __device__ constexpr int raw_row(int t) { return (raw_pieces(t) | 1) * 16; }  // odd: rows start in different 16-byte bank groups
__host__ __device__ constexpr int raw_slots(int t) { return t == B200_TYPE_BF16 ? 0 : raw_row(t) <= 192 ? 3 : 2; }
__host__ __device__ constexpr int raw_bytes(int t) { return t == B200_TYPE_BF16 ? 0 : raw_slots(t) * MQ_BM * raw_row(t); }

struct PairParams {
    MmqParams q;
    int64_t w_rows_per_product;  // dense weights by TMA: rows from one product (batch, expert) to the next
    int bn;                      // columns of a tile (grouped: at most), a multiple of 16; grouped: of 32
    int box;                     // activation rows of one TMA box: all of the CTA's, grouped: 16
    int stages;
    int share;                   // the last tile of a pair is stored by all warps (of tiles of up to 32 columns, one step of a warp, there is nothing to share; a part of K meets the others)
    int n_tiles_n, n_tiles_m;    // n_tiles_n of the grouped form: read from the tile table
    int *timeout;
};

// ---------------------------------------------------------------- the pair's wrappers
__device__ __forceinline__ unsigned cluster_rank() { unsigned r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void pair_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void pair_await() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc2(unsigned *smem_dst, unsigned ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(unsigned taddr, unsigned ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_mma2_bf16(unsigned tmem_d, unsigned long long adesc, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives on `bar` of both CTAs (a bit each in `both`) when the MMAs issued so far have retired
__device__ __forceinline__ void tc_commit2(unsigned bar, unsigned short both) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(both) : "memory");
}
// CTA `rank`'s copy of a shared variable, and an arrival there.  (The default semantics: what the barrier guards is in shared memory or TMEM
// and complete when the arrival is issued; a release at cluster scope would wait for the thread's outstanding memory operations, about 1000
// cycles a K step.)
__device__ __forceinline__ unsigned cluster_addr(unsigned local, int rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
// what another CTA has written before the cluster barrier in front of the load
__device__ __forceinline__ int ld_cluster(unsigned at) { int v; asm volatile("ld.shared::cluster.b32 %0, [%1];" : "=r"(v) : "r"(at) : "memory"); return v; }
__device__ __forceinline__ float4 ld_cluster4(unsigned at) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void mbar_arrive_remote(unsigned bar) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory"); }
// ---------------------------------------------------------------- 32 values of a row out of shared memory -> 16 packed bf16 pairs
// Two values at a time (packed f32: one issue slot for both): four small unsigned integers, one per byte of x, become d * q + c as two bf16
// pairs.  Integers below 128 take the upper mantissa bits of 128 (0x43qq0000 = 128 + q), so that PRMT alone makes the float and the 128
// goes into the constant, c - 128 d.  Without a minimum that constant is exact; with one (q4_K, q5_K, q2_K, q4_1, q5_1) it is rounded to f32, off by
// 2^-17 d at most: small beside d, whatever is left of d q + c near 0.
struct Scale2 { unsigned long long d, c; };
__device__ __forceinline__ unsigned long long pack_f2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ unsigned fma2_bf16(unsigned long long x, const Scale2 &s) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(s.d), "l"(s.c));
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(r));
    return pack_bf16(lo, hi);
}
__device__ __forceinline__ Scale2 scale_q7(float d, float c) {
    const float c128 = fmaf(-128.0f, d, c);
    return {pack_f2(d, d), pack_f2(c128, c128)};
}
__device__ __forceinline__ void unpack_q7x4(unsigned x, const Scale2 &s, unsigned *o) {
    const float a = __uint_as_float(__byte_perm(x, 0x43000000u, 0x7044)), b = __uint_as_float(__byte_perm(x, 0x43000000u, 0x7144));
    const float e = __uint_as_float(__byte_perm(x, 0x43000000u, 0x7244)), f = __uint_as_float(__byte_perm(x, 0x43000000u, 0x7344));
    o[0] = fma2_bf16(pack_f2(a, b), s);
    o[1] = fma2_bf16(pack_f2(e, f), s);
}
// bytes 0..255: float(byte) first, exact
__device__ __forceinline__ void unpack_u8x4(unsigned x, const Scale2 &s, unsigned *o) {
    o[0] = fma2_bf16(pack_f2(byte_f<0>(x), byte_f<1>(x)), s);
    o[1] = fma2_bf16(pack_f2(byte_f<2>(x), byte_f<3>(x)), s);
}
// N consecutive words at a 2-byte aligned shared address: 8-byte loads from the aligned-down one, a word select and a 16-bit funnel shift
template <int N>
__device__ __forceinline__ void lds_run(const unsigned char *at, unsigned (&w)[N]) {
    const unsigned a = smem_u32(at);
    const uint2 *p = reinterpret_cast<const uint2 *>(at - (a & 7u));
    const bool odd = (a & 4u) != 0;
    const unsigned sh = (a & 2u) * 8u;
    constexpr int NP = (N + 3) / 2;
    unsigned u[2 * NP];
#pragma unroll
    for (int i = 0; i < NP; i++) { const uint2 v = p[i]; u[2 * i] = v.x; u[2 * i + 1] = v.y; }
#pragma unroll
    for (int i = 0; i < N; i++) w[i] = __funnelshift_r(odd ? u[i + 1] : u[i], odd ? u[i + 2] : u[i + 1], sh);
}

// run(g, c, h, o): g -> first byte of the 256-value group, c = 64-value chunk 0..3 of it, h = which half of the chunk's bytes (c and h differ between the
// lanes).  o[0..7] are the 16 values from unpack_first(TYPE, h) on, o[8..15] those from unpack_second on.  Formats as at Dequant64: in a K-quant's
// chunk 16 bytes hold values 16h.. (low bits) and 32 + 16h.. (high bits), in a 32-value block low and high nibbles are neighbouring values.
__host__ __device__ constexpr bool unpack_block32(int t) { return t != B200_TYPE_Q4_K && t != B200_TYPE_Q5_K && t != B200_TYPE_Q6_K && t != B200_TYPE_Q2_K && t != B200_TYPE_Q3_K; }
__host__ __device__ constexpr int unpack_first(int t, int h) { return unpack_block32(t) ? 32 * h : 16 * h; }
__host__ __device__ constexpr int unpack_second(int t, int h) { return unpack_block32(t) ? 32 * h + 16 : 32 + 16 * h; }
template <int TYPE> struct Unpack32;

// four words of nibbles: low ones with scale a, high ones with scale b
__device__ __forceinline__ void unpack_nibbles(const unsigned (&q)[4], const Scale2 &a, const Scale2 &b, unsigned (&o)[16]) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        unpack_q7x4(q[i] & 0x0F0F0F0Fu, a, o + 2 * i);
        unpack_q7x4((q[i] >> 4) & 0x0F0F0F0Fu, b, o + 8 + 2 * i);
    }
}
__device__ __forceinline__ unsigned spread4(unsigned b) { return ((b & 15u) * 0x00204081u) & 0x01010101u; }  // four bits, one to each byte

template <int TYPE>
struct UnpackK45 {
    static __device__ __forceinline__ void run(const unsigned char *g, int c, int h, unsigned (&o)[16]) {
        const uint4 hdr = *reinterpret_cast<const uint4 *>(g);
        const uint4 qv = *reinterpret_cast<const uint4 *>(g + (TYPE == B200_TYPE_Q4_K ? 16 : 48) + 32 * c + 16 * h);
        // 6-bit scales and minima of sub-blocks 2c and 2c + 1: two neighbouring bytes of the 12 (get_scale_min_k4)
        const unsigned sh = 16u * (c & 1), y = hdr.y >> sh, z = hdr.z >> sh, w = hdr.w >> sh;
        const unsigned sc = c < 2 ? y & 0x3F3Fu : (w & 0x0F0Fu) | ((y >> 2) & 0x3030u), mn = c < 2 ? z & 0x3F3Fu : ((w >> 4) & 0x0F0Fu) | ((z >> 2) & 0x3030u);
        const float d = f16lo(hdr.x), dmin = f16hi(hdr.x);
        const Scale2 a = scale_q7(d * byte_f<0>(sc), -(dmin * byte_f<0>(mn))), b = scale_q7(d * byte_f<1>(sc), -(dmin * byte_f<1>(mn)));
        const unsigned q[4] = {qv.x, qv.y, qv.z, qv.w};
        if constexpr (TYPE == B200_TYPE_Q4_K) {
            unpack_nibbles(q, a, b, o);
        } else {
            const uint4 hv = *reinterpret_cast<const uint4 *>(g + 16 + 16 * h);
            const unsigned f[4] = {hv.x >> (2 * c), hv.y >> (2 * c), hv.z >> (2 * c), hv.w >> (2 * c)};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                unpack_q7x4((q[i] & 0x0F0F0F0Fu) + (f[i] & 0x01010101u) * 16u, a, o + 2 * i);
                unpack_q7x4(((q[i] >> 4) & 0x0F0F0F0Fu) + (f[i] & 0x02020202u) * 8u, b, o + 8 + 2 * i);
            }
        }
    }
};
template <> struct Unpack32<B200_TYPE_Q4_K> : UnpackK45<B200_TYPE_Q4_K> {};
template <> struct Unpack32<B200_TYPE_Q5_K> : UnpackK45<B200_TYPE_Q5_K> {};

template <> struct Unpack32<B200_TYPE_Q6_K> {  // bytes 16h.. of both 32-byte rows of the half, nibbles c & 1
    static __device__ __forceinline__ void run(const unsigned char *g, int c, int h, unsigned (&o)[16]) {
        unsigned qa[4], qb[4], qh[4];
        lds_run<4>(g + 64 * (c >> 1) + 16 * h, qa);
        lds_run<4>(g + 64 * (c >> 1) + 32 + 16 * h, qb);
        lds_run<4>(g + 128 + 32 * (c >> 1) + 16 * h, qh);
        const float d = h2f(*reinterpret_cast<const unsigned short *>(g + 208));
        const signed char *sc = reinterpret_cast<const signed char *>(g + 192 + 4 * c + h);
        const float da = d * (float)sc[0], db = d * (float)sc[2];
        const Scale2 a = scale_q7(da, -32.0f * da), b = scale_q7(db, -32.0f * db);
        const int n = 4 * (c & 1);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const unsigned f = qh[i] >> n;
            unpack_q7x4(((qa[i] >> n) & 0x0F0F0F0Fu) + (f & 0x03030303u) * 16u, a, o + 2 * i);
            unpack_q7x4(((qb[i] >> n) & 0x0F0F0F0Fu) + (f & 0x0C0C0C0Cu) * 4u, b, o + 8 + 2 * i);
        }
    }
};
template <> struct Unpack32<B200_TYPE_Q4_0> {
    static __device__ __forceinline__ void run(const unsigned char *g, int c, int h, unsigned (&o)[16]) {
        const unsigned char *blk = g + 36 * c + 18 * h;
        const float d = h2f(*reinterpret_cast<const unsigned short *>(blk));
        const Scale2 s = scale_q7(d, -8.0f * d);
        unsigned q[4];
        lds_run<4>(blk + 2, q);
        unpack_nibbles(q, s, s, o);
    }
};
template <> struct Unpack32<B200_TYPE_Q8_0> {
    static __device__ __forceinline__ void run(const unsigned char *g, int c, int h, unsigned (&o)[16]) {
        const unsigned char *blk = g + 68 * c + 34 * h;
        const float d = h2f(*reinterpret_cast<const unsigned short *>(blk));
        const Scale2 s = {pack_f2(d, d), pack_f2(-128.0f * d, -128.0f * d)};
        unsigned q[8];
        lds_run<8>(blk + 2, q);
#pragma unroll
        for (int i = 0; i < 8; i++) unpack_u8x4(q[i] ^ 0x80808080u, s, o + 2 * i);  // int8 + 128
    }
};
template <int TYPE>
struct UnpackLegacy {  // q4_1, q5_0, q5_1: as q4_0, with a minimum and / or the fifth bits in qh
    static __device__ __forceinline__ void run(const unsigned char *g, int c, int h, unsigned (&o)[16]) {
        using L = LegacyLayout<TYPE>;
        const unsigned char *blk = g + 2 * L::BB * c + L::BB * h;
        const float d = h2f(*reinterpret_cast<const unsigned short *>(blk));
        const Scale2 s = scale_q7(d, L::HAS_M ? h2f(*reinterpret_cast<const unsigned short *>(blk + 2)) : d * -16.0f);
        unsigned q[4];
        lds_run<4>(blk + L::QS, q);
        if constexpr (L::HAS_H) {
            const unsigned fl = *reinterpret_cast<const unsigned short *>(blk + L::QH), fh = *reinterpret_cast<const unsigned short *>(blk + L::QH + 2);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                unpack_q7x4((q[i] & 0x0F0F0F0Fu) + spread4(fl >> (4 * i)) * 16u, s, o + 2 * i);
                unpack_q7x4(((q[i] >> 4) & 0x0F0F0F0Fu) + spread4(fh >> (4 * i)) * 16u, s, o + 8 + 2 * i);
            }
        } else {
            unpack_nibbles(q, s, s, o);
        }
    }
};
template <> struct Unpack32<B200_TYPE_Q4_1> : UnpackLegacy<B200_TYPE_Q4_1> {};
template <> struct Unpack32<B200_TYPE_Q5_0> : UnpackLegacy<B200_TYPE_Q5_0> {};
template <> struct Unpack32<B200_TYPE_Q5_1> : UnpackLegacy<B200_TYPE_Q5_1> {};

// an iq4 sub-block of 32: levels + 128
__device__ __forceinline__ void unpack_iq4x32(const unsigned (&q)[4], float dl, unsigned (&o)[16]) {
    const Scale2 s = {pack_f2(dl, dl), pack_f2(-128.0f * dl, -128.0f * dl)};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        unsigned lo, hi;
        iq4_levels(q[i], lo, hi);
        unpack_u8x4(lo ^ 0x80808080u, s, o + 2 * i);
        unpack_u8x4(hi ^ 0x80808080u, s, o + 8 + 2 * i);
    }
}
template <> struct Unpack32<B200_TYPE_IQ4_NL> {
    static __device__ __forceinline__ void run(const unsigned char *g, int c, int h, unsigned (&o)[16]) {
        const unsigned char *blk = g + 36 * c + 18 * h;
        unsigned q[4];
        lds_run<4>(blk + 2, q);
        unpack_iq4x32(q, h2f(*reinterpret_cast<const unsigned short *>(blk)), o);
    }
};
template <> struct Unpack32<B200_TYPE_IQ4_XS> {
    static __device__ __forceinline__ void run(const unsigned char *g, int c, int h, unsigned (&o)[16]) {
        unsigned hdr[2], q[4];
        lds_run<2>(g, hdr);
        lds_run<4>(g + 8 + 32 * c + 16 * h, q);
        unpack_iq4x32(q, f16lo(hdr[0]) * iq4xs_scale(hdr[1], hdr[0] >> 16, 2 * c + h), o);
    }
};
// q2_K / q3_K: chunk c is bit fields 2 (c & 1) and 2 (c & 1) + 1 of half c >> 1; its four scales are bytes 4c .. 4c + 3 of the 16
template <> struct Unpack32<B200_TYPE_Q2_K> {
    static __device__ __forceinline__ void run(const unsigned char *g, int c, int h, unsigned (&o)[16]) {
        unsigned q[4];
        lds_run<4>(g + 16 + 32 * (c >> 1) + 16 * h, q);
        const unsigned ba = g[4 * c + h], bb = g[4 * c + 2 + h];
        const float d = h2f(*reinterpret_cast<const unsigned short *>(g + 80)), dmin = h2f(*reinterpret_cast<const unsigned short *>(g + 82));
        const Scale2 a = scale_q7(d * (float)(ba & 15), -(dmin * (float)(ba >> 4))), b = scale_q7(d * (float)(bb & 15), -(dmin * (float)(bb >> 4)));
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const unsigned f = q[i] >> (4 * (c & 1));
            unpack_q7x4(f & 0x03030303u, a, o + 2 * i);
            unpack_q7x4((f >> 2) & 0x03030303u, b, o + 8 + 2 * i);
        }
    }
};
template <> struct Unpack32<B200_TYPE_Q3_K> {
    static __device__ __forceinline__ void run(const unsigned char *g, int c, int h, unsigned (&o)[16]) {
        unsigned q[4], m[4], sw[3];
        lds_run<4>(g + 32 + 32 * (c >> 1) + 16 * h, q);
        lds_run<4>(g + 16 * h, m);
        lds_run<3>(g + 96, sw);
        // word c of the 16 scales (q3k_scales)
        const unsigned sc = ((((c & 1) ? sw[1] : sw[0]) >> (c & 2 ? 4 : 0)) & 0x0f0f0f0fu) | (((sw[2] >> (2 * c)) & 0x03030303u) << 4);
        const float d = h2f(*reinterpret_cast<const unsigned short *>(g + 108));
        const float da = d * (float)((int)((sc >> (8 * h)) & 0xff) - 32), db = d * (float)((int)((sc >> (16 + 8 * h)) & 0xff) - 32);
        const Scale2 a = scale_q7(da, -4.0f * da), b = scale_q7(db, -4.0f * db);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const unsigned f = q[i] >> (4 * (c & 1)), k = m[i] >> (2 * c);
            unpack_q7x4((f & 0x03030303u) + (k & 0x01010101u) * 4u, a, o + 2 * i);
            unpack_q7x4(((f >> 2) & 0x03030303u) + (k & 0x02020202u) * 2u, b, o + 8 + 2 * i);
        }
    }
};

// words per 256-value group are read at up to 14 bytes behind the slot's row start: raw_row leaves room for the last 8-byte load
// ---------------------------------------------------------------- the tile that comes next
struct PairTile {
    int64_t m0;          // first weight row of the pair's tile
    int64_t n0, n_end;   // columns
    int64_t product;     // batch entry or expert
    int n;               // columns the MMA computes
    int kb0, nkb;        // K steps of 64
};
template <bool GROUPED>
__device__ __forceinline__ PairTile pair_tile(const PairParams &p, int t, int nt, int ksteps_unit, int split) {
    PairTile r;
    const int ni = t % nt;
    int rest = t / nt;
    r.m0 = (int64_t)(rest % p.n_tiles_m) * 256;
    rest /= p.n_tiles_m;
    r.kb0 = 0;
    r.nkb = (int)(p.q.K / MQ_BK);
    if constexpr (GROUPED) {
        const int *te = behind(p.q.tile_tab) + 1 + 3 * ni;
        r.product = ld_behind(te);
        r.n0 = ld_behind(te + 1);
        const int64_t end = ld_behind(te + 2);
        r.n_end = end < r.n0 + p.bn ? end : r.n0 + p.bn;
        r.n = ((int)(r.n_end - r.n0) + 31) / 32 * 32;
    } else {
        r.n0 = (int64_t)ni * p.bn;
        r.n_end = r.n0 + p.bn < p.q.N ? r.n0 + p.bn : p.q.N;
        r.n = p.bn;
        r.product = rest;
        const int units = r.nkb / ksteps_unit, u0 = split * units / p.q.ksplit, u1 = (split + 1) * units / p.q.ksplit;
        r.kb0 = u0 * ksteps_unit;
        r.nkb = (u1 - u0) * ksteps_unit;
    }
    return r;
}

template <int TYPE> __host__ __device__ constexpr int pair_steps() { return TYPE == B200_TYPE_BF16 ? 1 : 2; }  // K steps of 64 a stage
// warps: producers, MMAs, copies, four that store; of dense weights, which have no producers, eight more for the meeting of a tile's parts
template <int TYPE>
__host__ __device__ constexpr int pair_threads() { return 32 * (6 + (TYPE == B200_TYPE_BF16 ? 8 : PAIR_PRODUCERS)); }

// ===== 32 columns of an accumulator, and every `step`-th after them, to the result: a warp's 32 rows
template <bool GROUPED>
__device__ __forceinline__ void pair_store(const PairParams &p, const PairTile &ti, unsigned acc, int rank, int c0, int step, bool ok) {
    const int quarter = (int)(threadIdx.x >> 5) & 3, lane = threadIdx.x & 31, cols = (int)(ti.n_end - ti.n0);
    const int64_t m = ti.m0 + rank * MQ_BM + quarter * 32 + lane;
    const bool row_ok = m < p.q.M && ok;
    float *drow = p.q.dst + m + (GROUPED ? 0 : ti.product * p.q.dst_batch);
    const int *row_dst = behind(p.q.row_dst);
#pragma unroll 1
    for (; c0 < cols; c0 += step) {
        float v[32];
        // scatter: sorted row -> (token, slot).  A lane asks for one of the 32 columns' places: in front of each store a load would wait for its turn
        const int place = GROUPED && c0 + lane < cols ? ld_behind(row_dst + ti.n0 + c0 + lane) : 0;
        __syncwarp();
        tmem_ld32(acc + ((unsigned)(quarter * 32) << 16) + (unsigned)c0, v);
        if constexpr (GROUPED) {
#pragma unroll
            for (int j = 0; j < 32; j++) {
                const int to = __shfl_sync(0xffffffffu, place, j);
                if (row_ok && c0 + j < cols) drow[(int64_t)to] = v[j];
            }
        } else if (row_ok) {
#pragma unroll
            for (int j = 0; j < 32; j++) {
                if (c0 + j >= cols) continue;
                drow[(ti.n0 + c0 + j) * p.q.dst_stride] = v[j];
            }
        }
    }
}

// ===== the parts of a tile meet.  Each CTA lays its accumulators, [column][128 rows], over its operand ring, which its MMAs have left; behind the
// cluster's barrier CTA (split, rank) reads columns split / ksplit of them from every CTA with its rows and adds them in the order of K.
// All threads of the cluster come here.
template <int TYPE>
__device__ __forceinline__ void pair_merge(const PairParams &p, const PairTile &ti, unsigned char *smem, unsigned tmem_base, unsigned acc_full0, int rank, int split, volatile int *failed,
                                           volatile int *part_there) {
    constexpr int MW = pair_threads<TYPE>() / 128 * 4;  // warps that read TMEM: whole sets of its four quarters
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ks = p.q.ksplit, cols = (int)(ti.n_end - ti.n0);
    const bool ok = __all_sync(0xffffffffu, pair_wait<20>(acc_full0, 0, failed, p.q.wait_limit));
    tc_fence_after();
    if (ok && warp < MW) {
        const int quarter = warp & 3;
        float *mine = reinterpret_cast<float *>(smem) + quarter * 32 + lane;
#pragma unroll 1
        for (int c0 = 32 * (warp >> 2); c0 < cols; c0 += 8 * MW) {
            float v[32];
            tmem_ld32(tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)c0, v);
#pragma unroll
            for (int j = 0; j < 32; j++) if (c0 + j < cols) mine[(c0 + j) * MQ_BM] = v[j];
        }
    }
    const int all = __syncthreads_and(ok);
    if (threadIdx.x == 0) *part_there = all;
    __syncwarp();
    pair_arrive();
    pair_await();
    bool there = true;
#pragma unroll 1
    for (int s = 0; s < ks; s++) there = there && ld_cluster(cluster_addr(smem_u32(const_cast<int *>(part_there)), 2 * s + rank)) != 0;
    if (!there) return;
    const int per = (cols + ks - 1) / ks, c1 = min(cols, (split + 1) * per);
    const int64_t m = ti.m0 + rank * MQ_BM + 4 * lane;
    float *drow = p.q.dst + m + ti.product * p.q.dst_batch + ti.n0 * p.q.dst_stride;
    const bool whole = m + 3 < p.q.M && ((uintptr_t)p.q.dst & 15) == 0 && ((p.q.dst_stride | p.q.dst_batch) & 3) == 0;
    const unsigned here = smem_u32(smem) + 16u * lane;
#pragma unroll 1
    for (int c = split * per + warp; c < c1; c += pair_threads<TYPE>() / 32) {
        float4 v[4], sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int s0 = 0; s0 < ks; s0 += 4) {
#pragma unroll
            for (int s = 0; s < 4; s++) if (s0 + s < ks) v[s] = ld_cluster4(cluster_addr(here, 2 * (s0 + s) + rank) + (unsigned)c * (MQ_BM * 4));
#pragma unroll
            for (int s = 0; s < 4; s++) if (s0 + s < ks) { sum.x += v[s].x; sum.y += v[s].y; sum.z += v[s].z; sum.w += v[s].w; }
        }
        float *d = drow + c * p.q.dst_stride;
        if (whole) {
            *reinterpret_cast<float4 *>(d) = sum;
        } else {
            if (m < p.q.M) d[0] = sum.x;
            if (m + 1 < p.q.M) d[1] = sum.y;
            if (m + 2 < p.q.M) d[2] = sum.z;
            if (m + 3 < p.q.M) d[3] = sum.w;
        }
    }
}

// SHARE: p.share may be set.  (Experts of a few rows have a kernel without that code, in whose loops it cost 2 %: 10 tokens, 3 of 8 experts of 2048 x 7936 q4_K, 140.6 -> 143.6 us.)
template <int TYPE, bool GROUPED, bool SHARE>
__global__ void __launch_bounds__(pair_threads<TYPE>(), 1) mmq_pair_kernel(const __grid_constant__ TmapBytes tmA, const __grid_constant__ TmapBytes tmB, const __grid_constant__ PairParams p) {
    constexpr bool DENSE = TYPE == B200_TYPE_BF16;
    constexpr int NP = DENSE ? 0 : PAIR_PRODUCERS, SK = pair_steps<TYPE>(), A_STEP = MQ_BM * MQ_BK * 2, A_BYTES = SK * A_STEP, UNIT = DENSE ? 1 : 4;
    constexpr int G256 = DENSE ? 0 : group256_bytes(TYPE);
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) unsigned long long full_bar[PAIR_MAX_STAGES], peer_bar[PAIR_MAX_STAGES], empty_bar[PAIR_MAX_STAGES], acc_full[2], acc_empty[2];
    __shared__ unsigned tmem_base_s;
    __shared__ volatile int failed, part_there;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, tid = threadIdx.x;
    // a cluster is ksplit pairs: its pairs take parts of K of the same tile
    const int in_cluster = (int)cluster_rank(), rank = GROUPED ? in_cluster : in_cluster & 1, leader = GROUPED ? 0 : in_cluster & ~1, split = GROUPED ? 0 : in_cluster >> 1,
              ksplit = GROUPED ? 1 : p.q.ksplit;
    const int pair = (int)blockIdx.x / (2 * ksplit), n_pairs = (int)gridDim.x / (2 * ksplit);
    const unsigned short both = (unsigned short)(3u << leader);
    const long long limit = p.q.wait_limit;
    const int S = p.stages, b_step = p.bn * MQ_BK, stage_bytes = A_BYTES + SK * b_step;  // (a step: bn / 2 activation rows of 128 bytes)
    const unsigned full0 = smem_u32(full_bar), peer0 = smem_u32(peer_bar), empty0 = smem_u32(empty_bar), acc_full0 = smem_u32(acc_full), acc_empty0 = smem_u32(acc_empty);

    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full_bar[s], DENSE ? 1 : PAIR_PRODUCERS + 1);
            mbar_init(&peer_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; b++) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8); }
        failed = 0;
        part_there = 1;
        mbar_fence_init();
    }
    if (warp == NP) tmem_alloc2(&tmem_base_s, 512);
    tc_fence_before();
    __syncthreads();
    // producers and copies touch their own CTA only: they start at once, and wait for the other CTA to be there when they are done
    pair_arrive();
    if (warp == NP || warp >= NP + 2) pair_await();
    tc_fence_after();
    const unsigned tmem_base = tmem_base_s;
    pdl_enter();
    const int nt = GROUPED ? p.q.tile_tab[0] : p.n_tiles_n;
    const int n_tiles = nt * p.n_tiles_m * (GROUPED ? 1 : p.q.n_batch);

    if (warp < NP) {
        // ===== producers: rows 8 * warp .. 8 * warp + 7 of this CTA's 128
        if constexpr (!DENSE) {
            constexpr int PIECES = raw_pieces(TYPE), ROW = raw_row(TYPE), SLOTS = raw_slots(TYPE), PER = (8 * PIECES + 31) / 32;
            unsigned char *raw = smem + (size_t)S * stage_bytes + (size_t)warp * SLOTS * 8 * ROW;
            // first byte of row r (0..7) of this warp in the tile's first group; rows past the matrix read its last one (their results are not stored)
            auto row_base = [&](const PairTile &ti, int r) {
                const int64_t row = ti.m0 + rank * MQ_BM + 8 * warp + r;
                return p.q.W + (size_t)ti.product * (GROUPED ? p.q.expert_bytes : p.q.w_batch_bytes) + (size_t)(ti.kb0 / 4) * G256 + (size_t)(row < p.q.M ? row : p.q.M - 1) * p.q.w_row_bytes;
            };
            // the copy runs SLOTS - 1 groups ahead of the unpacking, over tile ends too
            int ct = pair, left = 0, slot_in = 0;
            const unsigned char *src[PER];
            unsigned to[PER];  // where piece j of this lane goes in slot 0
#pragma unroll
            for (int j = 0; j < PER; j++) to[j] = smem_u32(raw) + (unsigned)((lane + 32 * j) / PIECES * ROW + (lane + 32 * j) % PIECES * 16);
            auto copy_group = [&]() {
                if (left == 0 && ct < n_tiles) {
                    const PairTile ti = pair_tile<GROUPED>(p, ct, nt, UNIT, split);
                    left = ti.nkb / 4;
                    ct += n_pairs;
#pragma unroll
                    for (int j = 0; j < PER; j++) {
                        const int i = lane + 32 * j;
                        src[j] = row_base(ti, i / PIECES & 7) + (raw_aligned(TYPE) ? i % PIECES * 16 : 0);
                    }
                }
                if (left > 0) {
                    left--;
                    const unsigned slot_off = (unsigned)(slot_in * 8 * ROW);
#pragma unroll
                    for (int j = 0; j < PER; j++) {
                        const bool mine = 32 * (j + 1) <= 8 * PIECES || lane + 32 * j < 8 * PIECES;
                        if constexpr (raw_aligned(TYPE)) {
                            if (mine) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to[j] + slot_off), "l"(src[j]) : "memory");
                        } else {
                            const unsigned off = (unsigned)(uintptr_t)src[j] & 15u, at = (unsigned)((lane + 32 * j) % PIECES * 16);
                            if (mine && at < off + G256) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to[j] + slot_off), "l"(src[j] + (int)(at - off)) : "memory");
                        }
                        src[j] += G256;
                    }
                }
                cp_async_commit();
                slot_in = slot_in + 1 == SLOTS ? 0 : slot_in + 1;
            };
            for (int i = 0; i < SLOTS - 1; i++) copy_group();
            const int cc = lane >> 4, h = (lane >> 3) & 1, r = lane & 7;  // chunk of a pair of K steps, half of its bytes, row
            // the lane's four 16-byte pieces of row r, swizzled
            const unsigned a_row = smem_u32(smem) + (unsigned)(cc * A_STEP + warp * 1024 + r * 128);
            const int f0 = unpack_first(TYPE, h) / 8, f1 = unpack_second(TYPE, h) / 8;
            const unsigned p0 = a_row + (unsigned)((f0 ^ r) << 4), p1 = a_row + (unsigned)(((f0 + 1) ^ r) << 4), p2 = a_row + (unsigned)((f1 ^ r) << 4), p3 = a_row + (unsigned)(((f1 + 1) ^ r) << 4);
            int s = 0, slot = 0;
            unsigned ph = 1;            // parity of the stage's empty barrier: the first pass finds it free
            bool ok = true;  // (the same in all lanes)
            for (int t = pair; t < n_tiles && ok; t += n_pairs) {
                const PairTile ti = pair_tile<GROUPED>(p, t, nt, UNIT, split);
                unsigned at = raw_aligned(TYPE) ? 0u : (unsigned)(uintptr_t)row_base(ti, r) & 15u;  // where in its first piece the row's group starts
#pragma unroll 1
                for (int g = ti.nkb / 4; g > 0 && ok; g--) {
                    cp_async_wait<SLOTS - 2>();
                    __syncwarp();  // the group has landed for all lanes, and all have left the one before
                    copy_group();
                    const unsigned char *row = raw + (slot * 8 + r) * ROW + at;
                    if constexpr (!raw_aligned(TYPE)) at = (at + G256) & 15u;
                    slot = slot + 1 == SLOTS ? 0 : slot + 1;
#pragma unroll
                    for (int c2 = 0; c2 < 4; c2 += 2) {
                        unsigned o[16];
                        Unpack32<TYPE>::run(row, c2 + cc, h, o);
                        ok = __all_sync(0xffffffffu, pair_wait<20>(empty0 + 8u * s, ph, &failed, limit));
                        if (!ok) break;
                        const unsigned d = (unsigned)(s * stage_bytes);
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(p0 + d), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(p1 + d), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]) : "memory");
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(p2 + d), "r"(o[8]), "r"(o[9]), "r"(o[10]), "r"(o[11]) : "memory");
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(p3 + d), "r"(o[12]), "r"(o[13]), "r"(o[14]), "r"(o[15]) : "memory");
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full0 + 8u * s) : "memory");
                        if (++s == S) { s = 0; ph ^= 1u; }
                    }
                }
            }
            cp_async_wait<0>();
        }
    } else if (warp == NP) {
        // ===== the pair's MMAs (first CTA); the second CTA passes on that its half of a stage is ready
        const unsigned long long desc0 = umma_desc_sw128(smem_u32(smem));
        const bool elected = elect_lane();
        const unsigned peer_remote = cluster_addr(peer0, leader);
        int s = 0, buf = 0;
        unsigned ph = 0, aph = 1;
        bool ok = true;  // (the same in all lanes)
        for (int t = pair; t < n_tiles && ok; t += n_pairs) {
            const PairTile ti = pair_tile<GROUPED>(p, t, nt, UNIT, split);
            if (rank != 0) {
                for (int kb = 0; kb < ti.nkb; kb += SK) {
                    ok = __all_sync(0xffffffffu, pair_wait<0>(full0 + 8u * s, ph, &failed, limit));
                    if (!ok) break;
                    if (elected) mbar_arrive_remote(peer_remote + 8u * s);
                    __syncwarp();
                    if (++s == S) { s = 0; ph ^= 1u; }
                }
                continue;
            }
            const unsigned idesc = umma_idesc_bf16(256, 16) + ((unsigned)((ti.n - 16) >> 3) << 17), acc = tmem_base + (unsigned)buf * 256u;
            ok = __all_sync(0xffffffffu, pair_wait<0>(acc_empty0 + 8u * buf, aph, &failed, limit));
            if (!ok) break;
            tc_fence_after();
            unsigned accumulate = 0;
#pragma unroll 1
            for (int kb = 0; kb < ti.nkb; kb += SK) {
                const bool here = pair_wait<0>(full0 + 8u * s, ph, &failed, limit), there = pair_wait<0>(peer0 + 8u * s, ph, &failed, limit);
                ok = __all_sync(0xffffffffu, here && there);
                if (!ok) break;
                tc_fence_after();
                const unsigned long long ad = desc0 + (unsigned)(s * (stage_bytes >> 4)), bd = ad + (A_BYTES >> 4);
                if (elected) {
                    // 16 bf16 = 32 bytes further along K inside the swizzle atom: +2 in the (address >> 4) field
#pragma unroll
                    for (int j = 0; j < SK; j++) {
                        const unsigned long long aj = ad + (unsigned)(j * (A_STEP >> 4)), bj = bd + (unsigned)(j * (b_step >> 4));
#pragma unroll
                        for (int k = 0; k < MQ_BK / 16; k++) tc_mma2_bf16(acc, aj + 2u * k, bj + 2u * k, idesc, j + k ? 1u : accumulate);
                    }
                    tc_commit2(empty0 + 8u * s, both);
                }
                __syncwarp();
                accumulate = 1;
                if (++s == S) { s = 0; ph ^= 1u; }
            }
            if (!ok) break;
            if (elected) tc_commit2(acc_full0 + 8u * buf, both);
            __syncwarp();
            buf ^= 1;
            if (buf == 0) aph ^= 1u;
        }
    } else if (warp == NP + 1) {
        // ===== copies: this CTA's half of the activation rows (dense weights: its 128 weight rows too)
        // (the whole warp loops, as above)
        const bool elected = elect_lane();
        bool dead = false;
        int s = 0;
        unsigned ph = 1;
        for (int t = pair; t < n_tiles; t += n_pairs) {
            const PairTile ti = pair_tile<GROUPED>(p, t, nt, UNIT, split);
            const int half = ti.n / 2, row = (int)(ti.n0 + rank * half + (GROUPED ? 0 : ti.product * p.q.n_pad));
            const int a_row = DENSE ? (int)(ti.product * p.w_rows_per_product + ti.m0 + rank * MQ_BM) : 0;
            const unsigned tx = (unsigned)(SK * half * MQ_BK * 2 + (DENSE ? A_BYTES : 0));
            int k = ti.kb0 * MQ_BK;
#pragma unroll 1
            for (int kb = 0; kb < ti.nkb; kb += SK, k += SK * MQ_BK) {
                if (!dead && !pair_wait<20>(empty0 + 8u * s, ph, &failed, limit)) dead = true;
                if (elected && !dead) {  // no copy without a free stage
                    unsigned char *st = smem + (size_t)(s * stage_bytes);
                    mbar_expect_tx(&full_bar[s], tx);
                    if constexpr (DENSE) tma_load_2d(st, &tmA, k, a_row, &full_bar[s]);
#pragma unroll
                    for (int j = 0; j < SK; j++) {
                        unsigned char *sb = st + A_BYTES + j * b_step;
                        if constexpr (GROUPED) {
                            for (int r = 0; r < half; r += 16) tma_load_2d(sb + r * MQ_BK * 2, &tmB, k + j * MQ_BK, row + r, &full_bar[s]);
                        } else {
                            tma_load_2d(sb, &tmB, k + j * MQ_BK, row, &full_bar[s]);
                        }
                    }
                }
                __syncwarp();
                if (++s == S) { s = 0; ph ^= 1u; }
            }
        }
    } else if (warp < NP + 6 && ksplit == 1) {
        // ===== epilogue: TMEM lanes 32 * (warp % 4) .. of this CTA's 128 rows; of the last tile only the wait for it, if all share it
        bool ok = true;
        int buf = 0;
        unsigned ph = 0;
        const unsigned acc_remote = cluster_addr(acc_empty0, leader);
        for (int t = pair; t < n_tiles; t += n_pairs) {
            const PairTile ti = pair_tile<GROUPED>(p, t, nt, UNIT, split);
            ok = __all_sync(0xffffffffu, ok && pair_wait<200>(acc_full0 + 8u * buf, ph, &failed, limit));
            tc_fence_after();
            if (SHARE && p.share && t + n_pairs >= n_tiles) {
                if (!ok) part_there = 0;
                break;
            }
            pair_store<GROUPED>(p, ti, tmem_base + (unsigned)buf * 256u, rank, 0, 32, ok);
            tc_fence_before();
            __syncwarp();
            if (lane == 0 && ok) mbar_arrive_remote(acc_remote + 8u * buf);
            buf ^= 1;
            if (buf == 0) ph ^= 1u;
        }
    }
    // ===== the last tile, behind which nothing is left to do: its columns are shared by the epilogue and the producers (dense weights: the warps without another role)
    if (SHARE && p.share && warp != NP && warp != NP + 1 && pair < n_tiles) {
        constexpr int SETS = (pair_threads<TYPE>() / 32 - 2) / 4;
        const int before = (n_tiles - 1 - pair) / n_pairs;  // tiles of this pair in front of it
        const PairTile ti = pair_tile<GROUPED>(p, pair + before * n_pairs, nt, UNIT, split);
        __syncwarp();
        asm volatile("bar.sync 1, %0;" ::"n"(SETS * 128) : "memory");
        tc_fence_after();
        const int set = warp < NP ? 1 + warp / 4 : (warp - NP - 2) / 4;
        pair_store<GROUPED>(p, ti, *const_cast<volatile unsigned *>(&tmem_base_s) + (unsigned)(before & 1) * 256u, rank, 32 * set, 32 * SETS, part_there != 0);
    }
    __syncwarp();
    if (warp < NP || warp == NP + 1) pair_await();
    if (!GROUPED && ksplit > 1) pair_merge<TYPE>(p, pair_tile<GROUPED>(p, pair, nt, UNIT, split), smem, tmem_base, acc_full0, rank, split, &failed, &part_there);
    __syncthreads();
    if (failed) {  // copies and MMAs that were requested end within this time
        if (tid == 0) atomicExch(p.timeout, 1);
        for (const long long t0 = clock64(); clock64() - t0 < 4000000LL;) {}
    }
    tc_fence_before();
    pair_arrive();
    pair_await();
    if (warp == NP) {
        tc_fence_after();
        tmem_dealloc2(tmem_base, 512);
    }
}

// ---------------------------------------------------------------- host side
// Tile width and parts of K by the time of the longest pair's work, in microseconds.  A K step of 64 costs what the slower of producers and tensor cores
// takes, `unpack` or 1.83 ns a column, and a little more where they are level (sixth powers added: within 4 % of q4_K and q6_K at 64 .. 256
// columns); dense weights take 1.25 ns a column but 0.2 at least; a tile more costs about 1.  The last tile's values are stored with nothing
// behind them to hide it: 12 ns a column.  Parts of K meet for 1.6 + 0.2 a part + 8 ns a column (1024 x 4096 q4_K over 20 columns: 22.5 us in one part, 15.3, 13.0,
// 11.0, 10.8, 10.1, 10.2, 9.3 in two .. eight), and a cluster takes one tile, so that there are no more tiles than clusters.  Widths are N / 1, N / 2, ...
// rounded up to 16.

constexpr double PAIR_NEXT_US = 4;  // a launch behind another: its start, and the end of the one in front that is no longer hidden (3 .. 6 measured)
struct PairPlan { int bn, ksplit, n_tiles_n; double tile, cost; };  // microseconds of a tile, of all
static inline double pair_step_us(double a, double b) { const double a3 = a * a * a, b3 = b * b * b; return sqrt(cbrt(a3 * a3 + b3 * b3)); }
// stages of the ring beside `raw` bytes; a tile's parts lie in them when they meet
static inline int pair_stages(int bn, int steps, int raw) {
    const int n = (PAIR_SMEM - 1024 - raw) / (steps * (MQ_BM * MQ_BK * 2 + bn * MQ_BK));
    return n > PAIR_MAX_STAGES ? PAIR_MAX_STAGES : n;
}
static inline bool pair_parts_fit(int bn, int steps, int raw) { return pair_stages(bn, steps, raw) * steps * (MQ_BM * MQ_BK * 2 + bn * MQ_BK) >= bn * MQ_BM * 4; }
// clusters[ks]: clusters of ks pairs that the device holds at once, not more for a larger ks
static inline PairPlan mmq_pair_plan(int64_t M, int64_t N, int64_t K, int n_batch, const int *clusters, double unpack, int unit, int steps_stage, int raw) {
    PairPlan best = {256, 1, 1, 0, 0};
    double best_cost = -1;
    const unsigned mt = (unsigned)((M + 255) / 256), n = (unsigned)N, np = (unsigned)clusters[1];  // (32-bit: the divisions of every width, one for each 32 columns, are host time of each call)
    const int units = (int)(K / MQ_BK / unit);
    for (unsigned parts = (n + 255) / 256, last = (n + 31) / 32; parts <= last; parts++) {
        const unsigned even = ((n + parts - 1) / parts + 15) / 16 * 16, bn = even < 32 ? 32 : even, nt = (n + bn - 1) / bn;
        const double dense = 1.25e-3 * bn < 0.2 ? 0.2 : 1.25e-3 * bn, step = unpack > 0 ? pair_step_us(unpack, 1.83e-3 * bn) : dense;
        const uint64_t tiles = (uint64_t)mt * nt * n_batch;
        for (int ks = 1; ks <= PAIR_MAX_SPLIT && ks <= units; ks++) {
            if (ks > 1 && (tiles > (uint64_t)clusters[ks] || !pair_parts_fit((int)bn, steps_stage, raw))) break;  // (there are no more of the larger clusters)
            const double waves = tiles <= np ? 1.0 : (double)((tiles + np - 1) / np);
            const double tile = (units + ks - 1) / ks * unit * step + 1.0, cost = waves * tile + (ks == 1 ? 0.012 * bn : 1.6 + 0.2 * ks + 0.008 * bn);
            if (best_cost < 0 || cost < 0.98 * best_cost) { best_cost = cost; best = {(int)bn, ks, (int)nt, tile, cost}; }
        }
    }
    return best;
}

// Rows whose tiles are whole waves, if the rest is better off in a launch of its own, where its few tiles are taken in parts of K; else 0.  (Two halves of K, added into a zeroed
// result, once did this for products of a little more than a wave.  One launch -> two, us: 20480 x 2560 over 40 columns q6_K 42.8 -> 35.1, with the halves 39.1, q8_0 38.9 -> 32.9, 37.1;
// 11008 x 4096 q6_K over 280 69.6 -> 55.0, 65.1; 28672 x 4096 q4_K over 280 90.4 -> 79.8, 96.7.)  A rest of more tiles than there are clusters of two pairs stays: 13824 x 5120 q6_K over 280, 84.
static inline int64_t mmq_pair_whole_waves(const PairPlan &pl, int64_t M, int64_t N, int64_t K, const int *clusters, double unpack, int unit, int steps_stage, int raw) {
    const int64_t np = clusters[1], nt = pl.n_tiles_n, tiles = (M + 255) / 256 * nt, mt = tiles / np * np / nt;
    if (pl.ksplit > 1 || tiles <= np || tiles % np == 0 || mt <= 0 || mt * 256 >= M) return 0;
    const double whole = (double)((mt * nt + np - 1) / np) * pl.tile + 0.012 * pl.bn;
    if (whole + PAIR_NEXT_US > 0.93 * pl.cost) return 0;
    const PairPlan rest = mmq_pair_plan(M - mt * 256, N, K, 1, clusters, unpack, unit, steps_stage, raw);
    return whole + PAIR_NEXT_US + rest.cost < 0.93 * pl.cost ? mt * 256 : 0;
}

// what the device holds at once, one CTA an SM: clusters of 1 .. PAIR_MAX_SPLIT pairs
struct PairDevice { std::atomic<bool> known{false}; int clusters[PAIR_MAX_SPLIT + 1]; };

// microseconds a K step of 64 takes while unpacking is the slower side: one tile of 256 rows on each of 74 pairs, 64 columns, from the difference
// between 8192 and 4096 values a row
template <int TYPE> constexpr double pair_unpack_us() {
    switch (TYPE) {
        case B200_TYPE_BF16: return 0;
        case B200_TYPE_Q4_0: case B200_TYPE_Q4_1: case B200_TYPE_Q4_K: return 0.30;
        case B200_TYPE_Q5_K: return 0.32;
        case B200_TYPE_Q2_K: return 0.35;
        case B200_TYPE_Q8_0: return 0.37;
        case B200_TYPE_Q5_0: case B200_TYPE_Q5_1: return 0.38;
        case B200_TYPE_IQ4_NL: case B200_TYPE_IQ4_XS: return 0.47;
        default: return 0.44;  // q6_K, q3_K
    }
}

template <int TYPE, bool GROUPED, bool SHARE = true>
static int mmq_pair_launch(const MmqParams &q, int64_t n_pad, int64_t w_rows_per_product, int64_t max_tiles_n, int64_t grouped_bn, cudaStream_t st) {
    if constexpr (GROUPED && SHARE) {
        if (q.N <= 32 * (int64_t)q.n_expert) return mmq_pair_launch<TYPE, GROUPED, false>(q, n_pad, w_rows_per_product, max_tiles_n, grouped_bn, st);
    }
    const auto kern = mmq_pair_kernel<TYPE, GROUPED, SHARE>;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(pair_threads<TYPE>());
    cfg.dynamicSmemBytes = PAIR_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[2];  // (as launch_chained, in clusters)
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    static PairDevice devices[16];  // (attributes and what fits are a device's)
    static std::mutex first;
    int cur_dev = 0;
    B200_CUDA_TRY(cudaGetDevice(&cur_dev));
    PairDevice &dev = devices[cur_dev & 15];
    if (!dev.known.load(std::memory_order_acquire)) {
        // (one thread finds out and writes it down, once: another that comes meanwhile would plan with what is half written)
        std::lock_guard<std::mutex> lock(first);
        if (!dev.known.load(std::memory_order_relaxed)) {
            B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PAIR_SMEM));
            if (!GROUPED) B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            dev.clusters[1] = sm_count() / 2;
            for (int ks = 2; !GROUPED && ks <= PAIR_MAX_SPLIT; ks++) {  // (experts take no parts of K)
                cfg.gridDim = dim3((unsigned)(2 * ks));
                at[0].val.clusterDim.x = (unsigned)(2 * ks);
                cfg.numAttrs = 1;
                if (cudaOccupancyMaxActiveClusters(&dev.clusters[ks], kern, &cfg) != cudaSuccess) { dev.clusters[ks] = 0; cudaGetLastError(); }
                if (dev.clusters[ks] > dev.clusters[ks - 1]) dev.clusters[ks] = dev.clusters[ks - 1];
            }
            dev.known.store(true, std::memory_order_release);
        }
    }
    PairParams p;
    p.q = q;
    p.w_rows_per_product = w_rows_per_product;
    const int status_rc = gemm_status_prepare();
    if (status_rc != B200_OK) return status_rc;
    p.timeout = g_gemm_timeout.load(std::memory_order_acquire);
    p.n_tiles_m = (int)((q.M + 255) / 256);
    if (GROUPED) {
        p.bn = (int)grouped_bn;
        p.box = 16;
        p.n_tiles_n = 0;
        p.q.ksplit = 1;
        p.share = SHARE;
    } else {
        constexpr int UNIT = TYPE == B200_TYPE_BF16 ? 1 : 4;
        const PairPlan pl = mmq_pair_plan(q.M, q.N, q.K, q.n_batch, dev.clusters, pair_unpack_us<TYPE>(), UNIT, pair_steps<TYPE>(), raw_bytes(TYPE));
        const int64_t rows = q.n_batch > 1 ? 0 : mmq_pair_whole_waves(pl, q.M, q.N, q.K, dev.clusters, pair_unpack_us<TYPE>(), UNIT, pair_steps<TYPE>(), raw_bytes(TYPE));
        if (rows) {
            MmqParams part = q;
            part.M = rows;
            const int rc = mmq_pair_launch<TYPE, GROUPED, SHARE>(part, n_pad, w_rows_per_product, max_tiles_n, grouped_bn, st);
            if (rc != B200_OK) return rc;
            part.W += (size_t)rows * q.w_row_bytes;
            part.dst += rows;
            part.M = q.M - rows;
            return mmq_pair_launch<TYPE, GROUPED, SHARE>(part, n_pad, w_rows_per_product, max_tiles_n, grouped_bn, st);
        }
        p.bn = pl.bn;
        p.box = pl.bn / 2;
        p.n_tiles_n = pl.n_tiles_n;
        p.q.ksplit = pl.ksplit;
        p.share = pl.ksplit == 1 && pl.bn > 32;
    }
    p.stages = pair_stages(p.bn, pair_steps<TYPE>(), raw_bytes(TYPE));
    TmapBytes tmA = {}, tmB;
    if (TYPE == B200_TYPE_BF16) {
        const int64_t products = GROUPED ? q.n_expert : q.n_batch;
        const int rc = encode_rows(tmA, q.W, q.K, (products - 1) * w_rows_per_product + q.M, q.w_row_bytes, MQ_BM);
        if (rc != B200_OK) return rc;
    }
    const int rc = encode_rows(tmB, q.Xb, q.K, n_pad * (q.n_batch > 1 ? q.n_batch : 1), (size_t)q.K * 2, p.box);
    if (rc != B200_OK) return rc;
    const int64_t tiles = (int64_t)p.n_tiles_m * (GROUPED ? max_tiles_n : p.n_tiles_n * (int64_t)q.n_batch);
    if (tiles > 0x3fffffff) { set_error("b200_mul_mat_q: too many tiles"); return B200_ERR_UNSUPPORTED; }
    const int clusters = dev.clusters[p.q.ksplit];
    cfg.gridDim = dim3((unsigned)(2 * p.q.ksplit * (tiles < clusters ? tiles : clusters)));
    at[0].val.clusterDim.x = (unsigned)(2 * p.q.ksplit);
    cfg.numAttrs = 2;
    B200_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tmA, tmB, p));
    return B200_OK;
}

}  // namespace b200
