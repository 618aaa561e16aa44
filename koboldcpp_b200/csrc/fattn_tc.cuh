// fattn_tc.cuh -- prompt attention over an f16 cache on the 5th-generation tensor cores (heads of 64 and 128).  Included by fattn.cu.
//
// A CTA serves 128 query columns of one kv-head (tokens times the query heads that share the keys) and walks over tiles of 64 keys:
//   S = Q . K^T      tcgen05, both operands in shared memory (K by TMA, Q converted once), into TMEM
//   P = 2^(c S - m)  a thread a column: no exchange between lanes; P goes back to TMEM as f16, in place of S
//   O += P . V       tcgen05, A = P from TMEM, B = V as it lies in the cache (keys are the strided side: MN-major), O stays in TMEM
// Two groups of four softmax warps take the tiles in turn, each with a maximum, a sum and an O of its own (merged at the end), and with two S, so that
// products run while a group is busy with the tile before: 4 x 64 columns of S and 2 x 128 of O fill TMEM at 128 dims.
//   * warp 8 issues the first products, warp 9 the second ones, warp 10 copies K, warp 11 V (one warp for both products took 1560 cycles a tile to issue
//     them, one for both copies 1270; the two softmax groups want a tile each 650), warps 12 to 15 read the mask ahead: per 32 columns a tile is 0
//     throughout, mixed, or hidden (-inf throughout), and which groups of 16 keys anybody sees.  Tiles that no column sees are not loaded, groups that
//     none sees stay out of P . V whatever they hold.
//   * the maximum that the exponent subtracts follows the true one only when that has grown by 8 (a factor of 256, which f16 and the f32 sums hold
//     without loss), so O is hardly ever rescaled (at every growth: 41 us below instead of 34).  The largest weight is then no power of two and is rounded
//     like the others, 4 % of the error against 64 bits (2.83e-4 -> 2.94e-4).  So a quarter of Q's dims also brings what its f16 leaves over, two more MMAs
//     a tile: those blocks of 16 dims, of all the CTA's columns, that leave over most (a fixed quarter does nothing for queries that lie in the others: 2.84e-4 -> 2.96e-4).
//     White queries 2.73e-4, queries in three of four dims 2.6e-4; a column's last bits thus depend on the columns beside it.  For all dims it would be 2.04e-4,
//     for 42 us; the weights as two f16 each 2.1e-4, for 38.
//   * a key that is hidden from one column and visible to another of the CTA takes part with weight 0.  If its values are not finite, that column's
//     result is not either: such columns are computed again, key by key over what they see (ft_column_alone).
// What bounds it: K, V and mask on their way from L2 (32 KB a tile and CTA, 1150 cycles) and the softmax (940 cycles a tile for both groups: exponentials at 16 a
// cycle and SM), and start and end of a CTA.  32 heads of 128, 512 tokens behind 1536: 82 us with mma.sync (fattn_mma_prefill_kernel, which keeps the
// other head sizes and masks at odd places); 41.5 with tiles of 128 keys and one S a group (a group then waits for its own products: 4700 cycles for two
// tiles), 38 with tiles of 64, 34.3 with the mask read once (ft_mask_kernel), 32.1 .. 32.8 with all of Q asked for at once.
// Waits have a limit, as in the prompt GEMM: a role that gives up sets `failed`, the others follow, and the status word is set.  Rows are stored only where no softmax
// warp had given up when the sums met.
#pragma once
#include "tcgen05.cuh"

namespace b200 {

constexpr int FT_COLS = 128, FT_KEYS = 64, FT_NB = 4;  // columns and keys of a tile; buffers of S, K and V: tile i is in number i % 4 of each
constexpr int FT_SOFTMAX = 8, FT_MASK = 4, FT_WARPS = FT_SOFTMAX + 4 + FT_MASK;
constexpr int FT_Q_PANEL = FT_COLS * 128, FT_PANEL = FT_KEYS * 128;  // rows of 64 values, 128-byte swizzle
constexpr int FT_MAX_TILES = 4096;
constexpr float FT_SLACK = 8.0f;
template <int D> constexpr int ft_tile_bytes() { return D / 64 * FT_PANEL; }
template <int D> constexpr size_t ft_smem(int n_tiles) { return 1024 + (size_t)((D / 64 + 1) * FT_Q_PANEL) + (size_t)(2 * FT_NB) * ft_tile_bytes<D>() + (size_t)n_tiles * 4 + (size_t)(n_tiles + 2) * 4; }

__device__ __forceinline__ void tmem_st32(unsigned taddr, const unsigned (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
        "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
        "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D (TMEM) += A . B: A in TMEM (16-bit values, two a column), B in shared memory
__device__ __forceinline__ void ft_mma_ts(unsigned d, unsigned a, unsigned long long b, unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d),
        "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 32 accumulator columns without waiting for them (tmem_wait_ld)
__device__ __forceinline__ void tmem_ld32_async(unsigned taddr, float *v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]),
          "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]),
          "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(taddr)
        : "memory");
}
template <int N>
__device__ __forceinline__ void tmem_wait_ld(float (&v)[N]) {  // (v: nothing that reads it may move in front of the wait)
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; i++) asm volatile("" : "+f"(v[i]));
}
// operand whose 64-value rows run along the other dimension (MN-major): panels of 64 values FT_PANEL apart, groups of 8 rows 1024 bytes apart
__device__ __forceinline__ unsigned long long ft_desc_mn(unsigned smem_addr) {
    unsigned long long d = 0;
    d |= (unsigned long long)((smem_addr & 0x3FFFFu) >> 4);
    d |= (unsigned long long)(FT_PANEL >> 4) << 16;
    d |= (unsigned long long)(1024 >> 4) << 32;
    d |= (unsigned long long)1 << 46;
    d |= (unsigned long long)2 << 61;
    return d;
}
// f16 operands, f32 results, 128 rows; B along K (K-major) or not
__host__ __device__ constexpr unsigned ft_idesc(int n, bool b_mn) { return (1u << 4) | (b_mn ? 1u << 16 : 0u) | ((unsigned)(n >> 3) << 17) | ((unsigned)(FT_COLS >> 4) << 24); }
__device__ __forceinline__ float ft_slope(const FaParams &p, int h) {
    return p.max_bias > 0.0f ? (h < p.n_head_log2 ? powf(p.m0, (float)(h + 1)) : powf(p.m1, (float)(2 * (h - p.n_head_log2) + 1))) : 1.0f;
}
// two f32 at a time: one issue slot for both
__device__ __forceinline__ float2 ft_fma2(float2 x, float2 y, float2 z) {
    float2 r;
    asm("{\n.reg .b64 a, b, c;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %7};\nfma.rn.f32x2 a, a, b, c;\nmov.b64 {%0, %1}, a;\n}\n"
        : "=f"(r.x), "=f"(r.y) : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y), "f"(z.x), "f"(z.y));
    return r;
}
__device__ __forceinline__ float2 ft_add2(float2 x, float2 y) {
    float2 r;
    asm("{\n.reg .b64 a, b;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nadd.rn.f32x2 a, a, b;\nmov.b64 {%0, %1}, a;\n}\n" : "=f"(r.x), "=f"(r.y) : "f"(x.x), "f"(x.y), "f"(y.x), "f"(y.y));
    return r;
}
// what two pairs of f16 leave over of four floats; its square is added to energy
__device__ __forceinline__ void ft_rest(float4 &x, unsigned h0, unsigned h1, float2 &energy) {
    const float2 minus = make_float2(-1.0f, -1.0f);
    const float2 a = ft_fma2(__half22float2(*reinterpret_cast<const __half2 *>(&h0)), minus, make_float2(x.x, x.y));
    const float2 b = ft_fma2(__half22float2(*reinterpret_cast<const __half2 *>(&h1)), minus, make_float2(x.z, x.w));
    energy = ft_fma2(a, a, ft_fma2(b, b, energy));
    x = make_float4(a.x, a.y, b.x, b.y);
}

// one column by one warp, touching the keys that it sees and no others
template <int D>
__device__ __noinline__ void ft_column_alone(const FaParams &p, int hk, int col, int lane) {
    constexpr float LOG2E = 1.4426950408889634f;
    constexpr int R = D / 32;
    const int n = col / p.gqa, h = hk * p.gqa + col % p.gqa;
    const float *qrow = reinterpret_cast<const float *>(p.q + (size_t)n * p.q_nb1 + (size_t)h * p.q_nb2);
    const unsigned char *mrow = p.mask != nullptr ? p.mask + (size_t)n * p.mask_nb1 : nullptr;
    const float slope = ft_slope(p, h), scale = p.softcap != 0.0f ? p.scale / p.softcap : p.scale;
    float q[R], o[R], m = -INFINITY, l = 0.f;
#pragma unroll
    for (int j = 0; j < R; j++) { q[j] = __half2float(__float2half_rn(qrow[lane + 32 * j])); o[j] = 0.f; }
    for (int key = 0; key < p.n_kv; key++) {
        const float mf = mrow != nullptr ? __half2float(*reinterpret_cast<const __half *>(mrow + 2 * (size_t)key)) : 0.f;
        if (mf == -INFINITY) continue;
        const __half *k = reinterpret_cast<const __half *>(p.k + (size_t)hk * p.k_nb2 + (size_t)key * p.k_nb1), *v = reinterpret_cast<const __half *>(p.v + (size_t)hk * p.v_nb2 + (size_t)key * p.v_nb1);
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < R; j++) s = fmaf(q[j], __half2float(k[lane + 32 * j]), s);
        s = warp_sum(s) * scale;
        if (p.softcap != 0.0f) s = p.softcap * tanhf(s);
        s = (mrow != nullptr ? s + slope * mf : s) * LOG2E;
        const float mn = fmaxf(m, s), mb = mn == -INFINITY ? 0.f : mn, a = mn == -INFINITY ? 1.0f : ex2(m - mb), w = ex2(s - mb), wh = __half2float(__float2half_rn(w));
        m = mn;
        l = l * a + w;
#pragma unroll
        for (int j = 0; j < R; j++) o[j] = o[j] * a + wh * __half2float(v[lane + 32 * j]);
    }
    float *orow = p.dst + ((size_t)n * p.n_head + h) * D;
#pragma unroll
    for (int j = 0; j < R; j++) orow[lane + 32 * j] = o[j] * (1.0f / l);
}

// scores of 64 keys from key0 on: scaled, capped, with the mask, times log2 e
__device__ __forceinline__ void ft_scores(float (&v)[64], const FaParams &p, const unsigned char *mrow, float slope, float scale, int key0, bool mixed) {
    constexpr float LOG2E = 1.4426950408889634f;
    const bool masked = mixed && mrow != nullptr;
    uint4 mu[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {  // (a mask's keys come in eights)
        mu[i] = make_uint4(0u, 0u, 0u, 0u);
        if (masked && key0 + 8 * i + 8 <= p.n_kv) mu[i] = ld_behind(reinterpret_cast<const uint4 *>(mrow + 2 * (size_t)(key0 + 8 * i)));
    }
#pragma unroll
    for (int i = 0; i < 64; i++) v[i] *= scale;
    if (p.softcap != 0.0f) {
#pragma unroll
        for (int i = 0; i < 64; i++) v[i] = p.softcap * tanhf(v[i]);
    }
    if (masked) {
#pragma unroll
        for (int i = 0; i < 64; i++) {
            const unsigned word = (i & 7) < 2 ? mu[i / 8].x : (i & 7) < 4 ? mu[i / 8].y : (i & 7) < 6 ? mu[i / 8].z : mu[i / 8].w;
            const float mf = __half2float(__ushort_as_half((unsigned short)(word >> (16 * (i & 1)))));
            v[i] = mf == -INFINITY ? -INFINITY : v[i] + slope * mf;  // (whatever a hidden key's row holds)
        }
    }
#pragma unroll
    for (int i = 0; i < 64; i++) v[i] = key0 + i < p.n_kv ? v[i] * LOG2E : -INFINITY;
}
template <int D>
__device__ __noinline__ void ft_rescale(unsigned o_at, float alpha) {
#pragma unroll 1
    for (int ch = 0; ch < D / 32; ch++) {
        float v[32];
        unsigned x[32];
        tmem_ld32(o_at + 32 * ch, v);
#pragma unroll
        for (int i = 0; i < 32; i++) x[i] = __float_as_uint(v[i] * alpha);
        tmem_st32(o_at + 32 * ch, x);
    }
}

// The mask once for all heads: [tile][token] bytes, bit 0: some key's value is not 0, bits 2 .. 5: groups of 16 keys of which one is seen.  A warp takes a token,
// 8 lanes one of its tiles.  Without it the CTAs of all kv-heads read the mask from L2 beside their keys and values (512 tokens x 2048 cells, 32
// heads: 64 MB), which costs 5 of 38 us.
constexpr int FT_MASK_TILES = 32;  // a CTA's
__global__ void __launch_bounds__(256) ft_mask_kernel(const unsigned char *mask, size_t nb1, int n_tok, int n_kv, int n_tiles, unsigned char *table) {
    pdl_enter(mask);
    const int n = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, j = lane >> 3;
    if (n >= n_tok) return;
    const unsigned char *row = mask + (size_t)n * nb1 + (size_t)(lane & 7) * 16;
    const int t0 = blockIdx.y * FT_MASK_TILES, t1 = min(t0 + FT_MASK_TILES, n_tiles);
#pragma unroll 4
    for (int t = t0; t < t1; t += 4) {
        const int key = (t + j) * FT_KEYS + (lane & 7) * 8;
        uint4 u = make_uint4(0xfc00fc00u, 0xfc00fc00u, 0xfc00fc00u, 0xfc00fc00u);  // (keys behind the last: hidden)
        if (key + 8 <= n_kv) u = *reinterpret_cast<const uint4 *>(row + (size_t)(t + j) * FT_KEYS * 2);
        const unsigned o = u.x | u.y | u.z | u.w, all = u.x & u.y & u.z & u.w;
        const unsigned any = __ballot_sync(0xffffffffu, o != 0u) >> (8 * j), seen = __ballot_sync(0xffffffffu, o != 0xfc00fc00u || all != 0xfc00fc00u) >> (8 * j);
        unsigned groups = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) groups |= (seen >> (2 * i) & 3u) != 0u ? 4u << i : 0u;
        if ((lane & 7) == 0 && t + j < t1) table[(size_t)(t + j) * n_tok + n] = (unsigned char)(groups | ((any & 0xffu) != 0u ? 1u : 0u));
    }
}

// waits of the copying lanes that did not succeed at once
__device__ __noinline__ bool ft_wait_slow(unsigned bar, unsigned parity, volatile int *failed, long long limit) { return pair_wait<0>(bar, parity, failed, limit); }
// by a whole warp
__device__ __forceinline__ bool ft_wait(unsigned bar, unsigned parity, volatile int *failed, long long limit) {
    return __all_sync(0xffffffffu, mbar_try(bar, parity)) || __all_sync(0xffffffffu, ft_wait_slow(bar, parity, failed, limit));
}
// tiles whose mask has been read, once tile t is among them (t or less: somebody gave up)
__device__ __noinline__ int ft_wait_mask(const volatile int *scanned, int t, volatile int *failed, long long limit) {
    const long long t0 = clock64();
    int known;
    while ((known = min(min(scanned[0], scanned[1]), min(scanned[2], scanned[3]))) <= t && !*failed) {
        if (clock64() - t0 > limit) *failed = 1;
        __nanosleep(40);
    }
    __threadfence_block();
    return known;
}
// an entry of the list once it is there (-2: somebody gave up)
__device__ __noinline__ int ft_wait_list(const volatile int *at, volatile int *failed, long long limit) {
    const long long t0 = clock64();
    int ti;
    while ((ti = *at) == -2 && !*failed) {
        if (clock64() - t0 > limit) *failed = 1;
        __nanosleep(40);
    }
    return ti;
}
// a tile's rows of all panels, and the arrival that expects them
__device__ __forceinline__ void ft_copy(unsigned dst, const void *tmap, int row, int slice, unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %2, %4}], [%5];" ::"r"(dst), "l"(tmap), "r"(0), "r"(row), "r"(slice),
                 "r"(bar)
                 : "memory");
}
// the second products of the last tiles before number `count` of the list (done in order; the list may end at count or at count - 1)
__device__ __forceinline__ bool ft_wait_last(const volatile int *act, unsigned long long *o_done, int count, volatile int *failed, long long limit) {
    bool ok = true;
    for (int i = max(count - 3, 0); i < count; i++) if (act[i] >= 0) ok = ok && pair_wait<20>(smem_u32(&o_done[i % FT_NB]), (i / FT_NB) & 1, failed, limit);
    return ok;
}

template <int D>
__global__ void __launch_bounds__(FT_WARPS * 32, 1) fattn_tc_kernel(const __grid_constant__ TmapBytes tmK, const __grid_constant__ TmapBytes tmV, const __grid_constant__ FaParams p, unsigned gqa_div,
                                                                  const unsigned char *table, long long limit, int *timeout) {
    constexpr int TILE = ft_tile_bytes<D>();
    constexpr float LOG2E = 1.4426950408889634f;
    enum { ZERO = 0, MIXED = 1, HIDDEN = 2 };
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    // of buffer b: K there, V there, first product done (K free), weights there, second product done (V and S free)
    __shared__ __align__(8) unsigned long long k_full[FT_NB], v_full[FT_NB], s_full[FT_NB], p_full[FT_NB], o_done[FT_NB];
    __shared__ unsigned tmem_base_s, again[4];
    __shared__ volatile int failed, scanned[FT_MASK];
    __shared__ float top[2][FT_COLS], total[2][FT_COLS];
    __shared__ int rest_of[2];  // blocks of 16 dims whose remainder the last panel of Q holds
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, tid = threadIdx.x;
    const int hk = blockIdx.y, col0 = (int)(gridDim.x - 1 - blockIdx.x) * FT_COLS, ncol = min(FT_COLS, p.n_cols - col0);  // (long causal walks first)
    const int n_tiles = (p.n_kv + FT_KEYS - 1) / FT_KEYS;
    unsigned char *sq = smem, *sk = sq + (D / 64 + 1) * FT_Q_PANEL, *sv = sk + FT_NB * TILE;
    volatile unsigned char *kinds = sv + FT_NB * TILE;                                         // [tile][32 columns]: kind | groups of 16 keys << 2
    volatile int *act = reinterpret_cast<int *>(sv + FT_NB * TILE + (size_t)n_tiles * 4);       // the tiles that are worked on: tile << 4 | groups of any column; then -1 -1, and -2 as long as that is not known

    if (tid == 0) {
        for (int i = 0; i < FT_NB; i++) { mbar_init(&k_full[i], 1); mbar_init(&v_full[i], 1); mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); mbar_init(&o_done[i], 1); }
        mbar_fence_init();
        failed = 0;
        for (int i = 0; i < 4; i++) { again[i] = 0; scanned[i] = 0; }
    }
    for (int i = tid; i < n_tiles + 2; i += FT_WARPS * 32) act[i] = -2;
    if (warp == FT_SOFTMAX) tmem_alloc(&tmem_base_s, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_base_s, tmem_o = tmem + FT_NB * FT_KEYS;  // S number i at 64 i, O of group w at 256 + D w
    pdl_enter();

    auto token = [&](int c) { return p.gqa == 1 ? c : (int)__umulhi((unsigned)c, gqa_div); };  // column / gqa (ft_launch)
    // what is known of a tile without a mask: keys behind the last one are not there
    auto plain_kind = [&](int t) -> unsigned { const int left = p.n_kv - t * FT_KEYS; return left >= FT_KEYS ? (unsigned)ZERO | 0x3cu : (unsigned)MIXED | ((1u << ((left + 15) / 16)) - 1) << 2; };

    if (warp < FT_SOFTMAX) {
        // ===== Q as f16, swizzled; then every second tile, a thread a column
        const int w = warp >> 2, quarter = warp & 3, row = quarter * 32 + lane;
        const unsigned char *q_at = behind(p.q);
        constexpr int CH = D / 8, ROWS = FT_SOFTMAX * 32 / CH;  // a thread takes 8 dims, number c of a row, of every ROWS-th column
        const int c = tid % CH;
        float4 qv[FT_COLS / ROWS][2];
        uint4 qh[FT_COLS / ROWS];
#pragma unroll
        for (int i = 0; i < FT_COLS / ROWS; i++) {
            const int r = tid / CH + i * ROWS, qc = min(col0 + r, p.n_cols - 1), n = token(qc), h = hk * p.gqa + qc - n * p.gqa;  // (columns behind the last: not stored)
            const float4 *src = reinterpret_cast<const float4 *>(q_at + (size_t)n * p.q_nb1 + (size_t)h * p.q_nb2) + 2 * c;
            qv[i][0] = __ldcg(src);
            qv[i][1] = __ldcg(src + 1);
        }
#pragma unroll
        for (int i = 0; i < FT_COLS / ROWS; i++) {
            const int r = tid / CH + i * ROWS;
            const float4 a = qv[i][0], b = qv[i][1];
            qh[i] = make_uint4(pack_h2(a.x, a.y), pack_h2(a.z, a.w), pack_h2(b.x, b.y), pack_h2(b.z, b.w));
            *reinterpret_cast<uint4 *>(sq + c / 8 * FT_Q_PANEL + r * 128 + ((c % 8) ^ (r & 7)) * 16) = qh[i];
        }
        // the D / 64 blocks that leave over most go to the last panel (sums in a fixed order, equal ones by number: the same choice every time).  It takes 0.1 .. 0.2 us of a
        // CTA's start (32 heads, 73 tokens alone 9.06 -> 9.27 us, 8 on one kv-head 8.88 -> 8.98); all loads of Q in flight at once give more back
        // where Q comes from HBM (512 tokens behind 1536: 34.3 -> 32.1 .. 32.8).  A first product that begins without the panel is no faster.
        float2 energy2 = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < FT_COLS / ROWS; i++) {
            ft_rest(qv[i][0], qh[i].x, qh[i].y, energy2);
            ft_rest(qv[i][1], qh[i].z, qh[i].w, energy2);
        }
        float energy = energy2.x + energy2.y;
        float *sums = reinterpret_cast<float *>(top);  // (not in use yet)
        sums[tid] = energy;
        asm volatile("bar.sync 3, %0;" ::"n"(FT_SOFTMAX * 32) : "memory");
        energy = 0.f;
#pragma unroll
        for (int i = 0; i < FT_SOFTMAX; i++) energy += sums[32 * i + lane];
#pragma unroll
        for (int off = CH; off < 32; off *= 2) energy += __shfl_xor_sync(0xffffffffu, energy, off);
        energy += __shfl_xor_sync(0xffffffffu, energy, 1);
        energy = energy < 1e30f ? energy : 1e30f;  // (also what is not a number)
        int rank = 0;
#pragma unroll
        for (int b = 0; b < D / 16; b++) {
            const float e = __shfl_sync(0xffffffffu, energy, 2 * b);
            rank += e > energy || (e == energy && b < c / 2) ? 1 : 0;
        }
        if (rank < D / 64) {
            if (tid < CH) rest_of[rank] = c / 2;  // (the two threads of a block write the same)
#pragma unroll
            for (int i = 0; i < FT_COLS / ROWS; i++) {
                const int r = tid / CH + i * ROWS;
                *reinterpret_cast<uint4 *>(sq + D / 64 * FT_Q_PANEL + r * 128 + ((2 * rank + (c & 1)) ^ (r & 7)) * 16) = make_uint4(pack_h2(qv[i][0].x, qv[i][0].y), pack_h2(qv[i][0].z, qv[i][0].w), pack_h2(qv[i][1].x, qv[i][1].y), pack_h2(qv[i][1].z, qv[i][1].w));
            }
        }
        fence_proxy_async_smem();
        asm volatile("bar.arrive 2, %0;" ::"n"(FT_SOFTMAX * 32 + 32) : "memory");

        const int col = min(col0 + row, p.n_cols - 1), tok = token(col);
        const float slope = ft_slope(p, hk * p.gqa + col - tok * p.gqa), scale = p.softcap != 0.0f ? p.scale / p.softcap : p.scale;
        const unsigned char *mrow = p.mask != nullptr ? behind(p.mask) + (size_t)tok * p.mask_nb1 : nullptr;
        const unsigned lanes = (unsigned)(quarter * 32) << 16, o_at = tmem_o + (unsigned)(w * D) + lanes;
        float m = -INFINITY, l = 0.f;  // what the exponent subtracts (times log2 e), the sum
        bool ok = true;
        int count = 0;  // tiles of both groups, or one more
        for (int n = 0;; n++) {
            const int buf = 2 * (n & 1) + w;
            const unsigned s_at = tmem + (unsigned)(buf * FT_KEYS) + lanes;
            ok = __all_sync(0xffffffffu, pair_wait<20>(smem_u32(&s_full[buf]), (n >> 1) & 1, &failed, limit));
            if (!ok) break;
            const int t = act[2 * n + w] >> 4;
            if (t < 0) { count = 2 * n + w; break; }
            tc_fence_after();
            const unsigned what = p.mask != nullptr ? kinds[4 * t + quarter] : plain_kind(t);
            const int kind = what & 3;
            unsigned x[32];
            if (kind == HIDDEN) {
#pragma unroll
                for (int i = 0; i < 32; i++) x[i] = 0u;
            } else {
                float v[64], c = scale * LOG2E;  // the common tile keeps the raw products, c takes them to scaled scores times log2 e
                tmem_ld32_async(s_at, v);
                tmem_ld32_async(s_at + 32, v + 32);
                tmem_wait_ld(v);
                if (kind == MIXED || p.softcap != 0.0f || !(scale > 0.f)) {
                    ft_scores(v, p, mrow, slope, scale, t * FT_KEYS, kind == MIXED);
                    c = 1.0f;
                }
                float mx[4] = {v[0], v[1], v[2], v[3]};
#pragma unroll
                for (int i = 4; i < 64; i++) mx[i & 3] = fmaxf(mx[i & 3], v[i]);
                const float top_now = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * c;
                const bool grown = top_now > m + FT_SLACK;  // (m = -inf: as soon as a key is seen)
                if (__any_sync(0xffffffffu, grown)) {
                    const float alpha = grown ? ex2(m - top_now) : 1.0f;
                    if (grown) { m = top_now; l *= alpha; }
                    if (n > 0) {  // (S of this tile stood behind the second product of the group's tile before the last; the last one's may be under way)
                        ok = __all_sync(0xffffffffu, pair_wait<20>(smem_u32(&o_done[buf ^ 2]), ((n - 1) >> 1) & 1, &failed, limit));
                        if (!ok) break;
                        tc_fence_after();
                        ft_rescale<D>(o_at, alpha);
                    }
                }
                const float mb = m == -INFINITY ? 0.f : m;  // (nothing seen yet: 2^-inf = 0 throughout)
                const float2 c2 = make_float2(c, c), mb2 = make_float2(-mb, -mb);
                float2 sum[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                for (int i = 0; i < 64; i += 2) {
                    const float2 e = ft_fma2(make_float2(v[i], v[i + 1]), c2, mb2);
                    v[i] = ex2(e.x);
                    v[i + 1] = ex2(e.y);
                }
#pragma unroll
                for (int i = 0; i < 64; i += 2) sum[i / 2 & 1] = ft_add2(sum[i / 2 & 1], make_float2(v[i], v[i + 1]));
#pragma unroll
                for (int i = 0; i < 32; i++) x[i] = pack_h2(v[2 * i], v[2 * i + 1]);
                l += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
            }
            tmem_st32(s_at, x);  // (over scores that have been read)
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[buf]);
        }
        // ===== both groups' sums meet; this one takes half of the dims, into shared memory so that rows can be stored whole
        top[w][row] = m;
        total[w][row] = l;
        // (the second products of all tiles are done, K and V have been read: those of the last tiles end last)
        ok = ok && __all_sync(0xffffffffu, ft_wait_last(act, o_done, count, &failed, limit));
        tc_fence_after();
        asm volatile("bar.sync 3, %0;" ::"n"(FT_SOFTMAX * 32) : "memory");
        ok = __all_sync(0xffffffffu, ok && !failed);  // (whoever of the eight warps gave up had set it by now; a role that gives up later takes rows with it that were right)
        constexpr int OROW = D + 4;
        float *so = reinterpret_cast<float *>(sk);
        static_assert(FT_COLS * OROW * 4 <= 2 * FT_NB * TILE, "results lie where K and V were");
        if (ok) {
            const float m0 = top[0][row], m1 = top[1][row], mm = fmaxf(m0, m1), f0 = m0 == -INFINITY ? 0.f : ex2(m0 - mm), f1 = m1 == -INFINITY ? 0.f : ex2(m1 - mm);
            const float sum = total[0][row] * f0 + total[1][row] * f1, inv = 1.0f / sum;
            const bool any0 = __any_sync(0xffffffffu, f0 != 0.f), any1 = __any_sync(0xffffffffu, f1 != 0.f), both = __all_sync(0xffffffffu, f0 != 0.f && f1 != 0.f);
            const float g0 = f0 * inv, g1 = f1 * inv;
            float check = 0.f;  // 0 as long as every result is finite
#pragma unroll
            for (int ch = 0; ch < D / 64; ch++) {
                float a[32], b[32];
                const unsigned at = tmem_o + (unsigned)(w * (D / 2) + 32 * ch) + lanes;
#pragma unroll
                for (int i = 0; i < 32; i++) a[i] = b[i] = 0.f;
                if (any0) tmem_ld32_async(at, a);
                if (any1) tmem_ld32_async(at + D, b);
                tmem_wait_ld(a);
                tmem_wait_ld(b);
                if (!both) {  // (an O that nothing was added to holds anything)
#pragma unroll
                    for (int i = 0; i < 32; i++) { a[i] = f0 != 0.f ? a[i] : 0.f; b[i] = f1 != 0.f ? b[i] : 0.f; }
                }
#pragma unroll
                for (int i = 0; i < 32; i++) { a[i] = fmaf(a[i], g0, b[i] * g1); check = fmaf(a[i], 0.f, check); }
#pragma unroll
                for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4 *>(so + row * OROW + w * (D / 2) + 32 * ch + i) = make_float4(a[i], a[i + 1], a[i + 2], a[i + 3]);
            }
            if (row < ncol && !(check == 0.f) && !(sum == 0.f)) atomicOr(&again[quarter], 1u << lane);
        }
        tc_fence_before();
        asm volatile("bar.sync 3, %0;" ::"n"(FT_SOFTMAX * 32) : "memory");
        ok = __all_sync(0xffffffffu, ok && !failed);  // (all of a row has been put down, or nothing of it is stored)
        if (ok) {
#pragma unroll 4
            for (int i = tid; i < ncol * (D / 4); i += FT_SOFTMAX * 32) {
                const int r = i / (D / 4), c = i % (D / 4), oc = col0 + r, n = token(oc);
                reinterpret_cast<float4 *>(p.dst + ((size_t)n * p.n_head + hk * p.gqa + oc - n * p.gqa) * D)[c] = *reinterpret_cast<const float4 *>(so + r * OROW + 4 * c);
            }
        }
        if (again[0] | again[1] | again[2] | again[3]) {  // (the same for all threads)
            asm volatile("bar.sync 3, %0;" ::"n"(FT_SOFTMAX * 32) : "memory");  // (the rows are stored)
            for (int r = warp; ok && r < ncol; r += FT_SOFTMAX) if (again[r >> 5] >> (r & 31) & 1u) ft_column_alone<D>(p, hk, col0 + r, lane);
        }
    } else if (warp == FT_SOFTMAX) {
        // ===== first products: S of tile i goes where the weights of tile i - 4 were
        asm volatile("bar.sync 2, %0;" ::"n"(FT_SOFTMAX * 32 + 32) : "memory");
        const bool elected = elect_lane();
        const unsigned long long qd = umma_desc_sw128(smem_u32(sq)), kd0 = umma_desc_sw128(smem_u32(sk));
        const unsigned kf = smem_u32(k_full), od = smem_u32(o_done);
        unsigned rest_at[D / 64];  // (a reduction over the warp leaves it where the descriptors want it, the same in all lanes: through a shuffle every tile paid for it)
#pragma unroll
        for (int j = 0; j < D / 64; j++) {
            const int kk = (int)__reduce_or_sync(0xffffffffu, (unsigned)rest_of[j]);
            rest_at[j] = (unsigned)(kk / 4 * (FT_PANEL >> 4) + 2 * (kk % 4));
        }
        bool ok = true;
        for (int i = 0;; i++) {
            const unsigned b = i % FT_NB, ph = (i / FT_NB) & 1;
            ok = ft_wait(kf + 8 * b, ph, &failed, limit) && (i < FT_NB || ft_wait(od + 8 * b, ph ^ 1u, &failed, limit));
            if (!ok) break;
            if (act[i] < 0) {  // both groups look once more
                if (elected) mbar_arrive(&s_full[b]);
                const unsigned b1 = (i + 1) % FT_NB;
                ok = i + 1 < FT_NB || ft_wait(od + 8 * b1, (((i + 1) / FT_NB) & 1) ^ 1u, &failed, limit);
                if (ok && elected) mbar_arrive(&s_full[b1]);
                break;
            }
            tc_fence_after();
            const unsigned long long kd = kd0 + b * (TILE >> 4);
            const unsigned sd = tmem + b * FT_KEYS;
            if (elected) {
#pragma unroll
                for (int k = 0; k < D / 16 + D / 64; k++) {  // all of Q, then what it leaves over of two blocks (one with 64 dims; the panel behind the others)
                    const unsigned at = k < D / 16 ? (unsigned)(k / 4 * (FT_PANEL >> 4) + 2 * (k % 4)) : rest_at[k < D / 16 ? 0 : k - D / 16];
                    tc_mma_bf16(sd, qd + (unsigned)(k / 4 * (FT_Q_PANEL >> 4) + 2 * (k % 4)), kd + at, ft_idesc(FT_KEYS, false), k != 0);
                }
                tc_commit(&s_full[b]);
            }
            __syncwarp();
        }
        __syncwarp();
    } else if (warp == FT_SOFTMAX + 1) {
        // ===== second products
        const bool elected = elect_lane();
        const unsigned long long vd0 = ft_desc_mn(smem_u32(sv));
        const unsigned pf = smem_u32(p_full), vf = smem_u32(v_full);
        unsigned begun = 0;
        for (int i = 0;; i++) {
            const unsigned b = i % FT_NB, ph = (i / FT_NB) & 1, w = i & 1;
            if (!ft_wait(vf + 8 * b, ph, &failed, limit)) break;  // (behind the last tile: an arrival without a copy)
            const int ti = act[i];
            if (ti < 0) break;
            if (!ft_wait(pf + 8 * b, ph, &failed, limit)) break;
            tc_fence_after();
            if (elected) {
                const unsigned long long vd = vd0 + b * (TILE >> 4);
                const unsigned pd = tmem + b * FT_KEYS, out = tmem_o + w * D;
                unsigned acc = begun >> w & 1u;
#pragma unroll
                for (int k = 0; k < FT_KEYS / 16; k++) {
                    if (ti >> k & 1) {
                        ft_mma_ts(out, pd + 8 * k, vd + (unsigned)(k * (2048 >> 4)), ft_idesc(D, true), acc);
                        acc = 1u;
                    }
                }
                tc_commit(&o_done[b]);
            }
            __syncwarp();
            begun |= 1u << w;
        }
        __syncwarp();
    } else if (warp == FT_SOFTMAX + 2) {
        // ===== K, and the list of the tiles that somebody sees.  (An instruction of a lone warp takes about 12 cycles beside the others, so the copies' loops do
        // no more than they must: one lane, addresses made ahead, the slow side of the waits elsewhere)
        if (lane == 0) {
            const unsigned sf = smem_u32(s_full), kf = smem_u32(k_full), dst = smem_u32(sk);
            volatile const unsigned *what = reinterpret_cast<volatile const unsigned *>(kinds);
            volatile int *to = act;
            int known = p.mask != nullptr ? 0 : n_tiles;  // tiles whose mask has been read
            unsigned b = 0, ph = 1;
            bool ok = true, first = true;  // first: the buffers' first round, nothing to wait for
            for (int t = 0; t < n_tiles; t++) {
                if (t >= known) {
                    known = ft_wait_mask(scanned, t, &failed, limit);
                    if (t >= known) { ok = false; break; }
                }
                unsigned groups;
                if (p.mask != nullptr) {
                    const unsigned four = what[t];
                    groups = (four >> 2 | four >> 10 | four >> 18 | four >> 26) & 15u;
                    if (groups == 0) continue;
                } else {
                    groups = plain_kind(t) >> 2;
                }
                if (!first && !mbar_try(sf + 8 * b, ph) && !ft_wait_slow(sf + 8 * b, ph, &failed, limit)) { ok = false; break; }
                *to++ = t << 4 | (int)groups;
                ft_copy(dst + b * TILE, &tmK, t * FT_KEYS, hk, kf + 8 * b, TILE);
                if (++b == FT_NB) { b = 0; ph ^= 1u; first = false; }
            }
            if (ok && (first || ft_wait_slow(sf + 8 * b, ph, &failed, limit))) {
                to[0] = to[1] = -1;
                __threadfence_block();
                mbar_arrive(&k_full[b]);
            }
        }
        __syncwarp();
    } else if (warp == FT_SOFTMAX + 3) {
        // ===== V of the listed tiles
        if (lane == 0) {
            const unsigned od = smem_u32(o_done), vf = smem_u32(v_full), dst = smem_u32(sv);
            const volatile int *from = act;
            unsigned b = 0, ph = 1;
            bool first = true;
            for (;;) {
                int ti = *from++;
                if (ti == -2) ti = ft_wait_list(from - 1, &failed, limit);
                if (ti == -2) break;
                if (!first && !mbar_try(od + 8 * b, ph) && !ft_wait_slow(od + 8 * b, ph, &failed, limit)) break;
                if (ti < 0) {
                    mbar_arrive(&v_full[b]);
                    break;
                }
                ft_copy(dst + b * TILE, &tmV, ti >> 4 << 6, hk, vf + 8 * b, TILE);
                if (++b == FT_NB) { b = 0; ph ^= 1u; first = false; }
            }
        }
        __syncwarp();
    } else if (p.mask != nullptr) {
        // ===== the mask of 32 columns, tile by tile
        const int q = warp - FT_SOFTMAX - 4, r0 = 32 * q, r1 = min(r0 + 31, ncol - 1);
        auto post = [&](int t, bool mixed, unsigned groups) {
            if (lane == 0) {
                kinds[4 * t + q] = (unsigned char)((!mixed ? ZERO : groups == 0u ? HIDDEN : MIXED) | groups << 2);
                __threadfence_block();
                scanned[q] = t + 1;
            }
        };
        if (table != nullptr) {  // a byte of every token's (ft_mask_kernel)
            const unsigned char *mine = behind(table) + token(min(col0 + r0 + lane, p.n_cols - 1));
            const bool none = r1 < r0;
#pragma unroll 1
            for (int t = 0; t < n_tiles; t += 4) {
                unsigned v[4];
#pragma unroll
                for (int j = 0; j < 4; j++) v[j] = t + j < n_tiles ? __ldcg(mine + (size_t)(t + j) * p.N) : 0u;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const unsigned all = none ? 1u : __reduce_or_sync(0xffffffffu, v[j]);
                    if (t + j < n_tiles) post(t + j, all & 1u, all >> 2);
                }
            }
        } else {  // 8 lanes take a token's 64 keys
            const int n0 = token(min(col0 + r0, p.n_cols - 1)), n1 = r1 < r0 ? n0 : token(col0 + r1), fours = r1 < r0 ? 0 : (n1 - n0) / 4 + 1;
            const unsigned char *at = behind(p.mask) + (size_t)(lane & 7) * 16;
            for (int t = 0; t < n_tiles; t++) {
                unsigned any = 0, inf = 0, all = 0xffffffffu;
                if (t * FT_KEYS + (lane & 7) * 8 + 8 <= p.n_kv) {
#pragma unroll 8
                    for (int i = 0; i < fours; i++) {
                        const uint4 u = ld_behind(reinterpret_cast<const uint4 *>(at + (size_t)min(n0 + 4 * i + (lane >> 3), n1) * p.mask_nb1 + (size_t)t * FT_KEYS * 2));
                        const unsigned o = u.x | u.y | u.z | u.w;
                        any |= o;
                        inf |= o ^ 0xfc00fc00u;
                        all &= u.x & u.y & u.z & u.w;
                    }
                } else {
                    any = 1;
                    all = 0xfc00fc00u;
                }
                if (fours == 0) { any = 1; inf = 0; all = 0xfc00fc00u; }
                const bool mixed = __any_sync(0xffffffffu, any != 0u);
                unsigned seen = __ballot_sync(0xffffffffu, inf != 0u || all != 0xfc00fc00u), groups = 0;
                seen |= seen >> 16;
                seen |= seen >> 8;
#pragma unroll
                for (int i = 0; i < 4; i++) groups |= (seen >> (2 * i) & 3u) != 0u ? 1u << i : 0u;
                post(t, mixed, groups);
            }
        }
    }
    __syncwarp();
    __syncthreads();
    if (failed) {  // copies and MMAs that were requested end within this time
        if (tid == 0) atomicExch(timeout, 1);
        for (const long long t0 = clock64(); clock64() - t0 < 4000000LL;) {}
    }
    tc_fence_before();
    __syncthreads();
    if (warp == FT_SOFTMAX) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// host side: false where the other kernel is to serve the call
static bool ft_fits(const b200_fattn_args *a) {
    const uint64_t gqa = (uint64_t)(a->n_head / a->n_head_kv);
    const bool mask_ok = !a->mask || ((((uintptr_t)a->mask | a->mask_nb1) & 15) == 0 && a->n_kv % 8 == 0);
    const bool rows_ok = a->k_nb1 >= 2 * (size_t)a->D && a->v_nb1 >= 2 * (size_t)a->D && (a->n_head_kv == 1 || (a->k_nb2 > 0 && a->v_nb2 > 0));
    return (a->D == 64 || a->D == 128) && a->type_k == B200_TYPE_F16 && mask_ok && rows_ok && ((uintptr_t)a->dst & 15) == 0 && a->n_kv >= FT_KEYS && (uint64_t)a->N * gqa * gqa < (1ull << 31) &&
           a->n_kv <= (int64_t)FT_KEYS * FT_MAX_TILES;
}
static bool ft_encode(TmapBytes &tm, const void *base, int64_t D, int64_t rows, int64_t heads, size_t row_bytes, size_t head_bytes) {
    const EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return false;
    // a row as panels of 64 values: all panels of a tile in one copy
    const unsigned long long gdim[4] = {64, (unsigned long long)rows, (unsigned long long)(D / 64), (unsigned long long)heads};
    const unsigned long long gstr[3] = {(unsigned long long)row_bytes, 128, (unsigned long long)(heads == 1 ? row_bytes : head_bytes)};
    const unsigned box[4] = {64, FT_KEYS, (unsigned)(D / 64), 1}, estr[4] = {1, 1, 1, 1};
    // CU_TENSOR_MAP_DATA_TYPE_FLOAT16 = 6, INTERLEAVE_NONE = 0, SWIZZLE_128B = 3, L2_PROMOTION_L2_256B = 3, FLOAT_OOB_FILL_NONE = 0 (zeros)
    return enc(&tm, 6, 4, (void *)base, gdim, gstr, box, estr, 0, 3, 3, 0) == 0;
}
// Scratch for ft_mask_kernel's result.  Its launch (1.3 us) pays where a CTA would read the mask of many tokens for many tiles: 34 heads of 128, 52 tokens behind 912
// 26.4 -> 16.6 us, 16 heads, 213 tokens alone 12.9 -> 10.7; over 8 tiles with 8 heads a kv-head 8.9 -> 10.1, and still 22.5 -> 24.8 over 31.
constexpr size_t FT_TABLE_BYTES = 512 * 1024;
static size_t ft_table_bytes(const b200_fattn_args *a) { return (size_t)a->N * (size_t)((a->n_kv + FT_KEYS - 1) / FT_KEYS); }
static bool ft_mask_once(const b200_fattn_args *a, size_t room) {
    return a->mask && room >= ft_table_bytes(a) && (a->n_kv + FT_KEYS - 1) / FT_KEYS >= 6 * (a->n_head / a->n_head_kv);
}
// -1000: the other kernel's
template <int D>
static int ft_launch(const b200_fattn_args *a, const FaParams &p, unsigned char *ws, size_t ws_bytes, long long limit, cudaStream_t st) {
    TmapBytes tk, tv;
    if (!ft_encode(tk, a->k, D, a->n_kv, a->n_head_kv, a->k_nb1, a->k_nb2) || !ft_encode(tv, a->v, D, a->n_kv, a->n_head_kv, a->v_nb1, a->v_nb2)) return -1000;
    int *status = nullptr;
    const int rc = gemm_status_word(&status);
    if (rc != B200_OK) return rc;
    static bool attr_set_dev[16] = {};  // cudaFuncSetAttribute is per device
    int cur_dev = 0;
    B200_CUDA_TRY(cudaGetDevice(&cur_dev));
    if (!attr_set_dev[cur_dev & 15]) {
        B200_CUDA_TRY(cudaFuncSetAttribute(fattn_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ft_smem<D>(FT_MAX_TILES)));
        attr_set_dev[cur_dev & 15] = true;
    }
    const unsigned div = (unsigned)(((1ull << 32) + p.gqa - 1) / p.gqa);  // (exact while columns x gqa < 2^32: ft_fits)
    const int n_tiles = (p.n_kv + FT_KEYS - 1) / FT_KEYS;
    unsigned char *table = nullptr;
    if (ws != nullptr && ft_mask_once(a, ws_bytes)) {
        table = ws;
        B200_CUDA_TRY(launch_chained(ft_mask_kernel, dim3((unsigned)((p.N + 7) / 8), (unsigned)((n_tiles + FT_MASK_TILES - 1) / FT_MASK_TILES)), 256, 0, st, p.mask, p.mask_nb1, p.N, p.n_kv, n_tiles, table));
    }
    const dim3 grid((unsigned)((p.n_cols + FT_COLS - 1) / FT_COLS), (unsigned)p.n_head_kv);
    B200_CUDA_TRY(launch_chained(fattn_tc_kernel<D>, grid, FT_WARPS * 32, ft_smem<D>(n_tiles), st, tk, tv, p, div, (const unsigned char *)table, limit, status));
    return B200_OK;
}

}  // namespace b200
