// sink_tile.cuh -- prompt attention over f32 caches with bf16 products when a workspace is given.  Included by gattn.cu.
//
// Two launches: the cache rows become bf16 once (sink_rows_bf16_kernel: [kv head][cell][dim padded to 16], zeros for free cells), then
// sink_attn_tile_kernel works on tiles of 64 cells that arrive by cp.async.  A CTA serves 64 columns of one kv head, a column being a token and
// one of the query heads that share the keys, 16 columns a warp.  sink_attn_mma_kernel, which needs no workspace, converts every tile for every query head
// and block of 64 tokens, with its loads in front of its products: 214 us for 512 tokens behind 512, 32 heads over 8 of 128; both launches here
// take 56.  Bound by the latency of a tile's steps, of which two warps a scheduler (248 registers a thread) hide little, and by fetching their instructions: an instruction
// a scheduler every 4.4 cycles.  What a tile's cells are is asked for a tile ahead, and comes to shared memory as the rows do: 58.4 us with both read where they are
// needed; 32 heads over 4 of 64, 100 tokens behind 1400, 48.7 -> 42.1.
// Whether half a tile is seen wholly, partly or not at all follows from the positions of the warp's tokens (their smallest and largest) when they
// belong to one sequence, else token by token; only partly seen halves, and those with a soft cap or a distance bias, go value by value.
// A softmax step is 32 cells, half a tile: the running maximum and with it the bf16 roundings of the weights are those of sink_attn_mma_kernel,
// and cells of a half that none of the warp's tokens sees stay out of its products, whatever they hold.
#pragma once

namespace b200 {

constexpr int ST_CELLS = 64, ST_STEP = 32, ST_COLS = 64, ST_WARPS = 4, ST_NBUF = 3;

__device__ __forceinline__ float st_ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

static inline int64_t st_cells(const b200_sink_attn_args *a) { return ((int64_t)a->n_kv + ST_CELLS - 1) / ST_CELLS * ST_CELLS; }
// head sizes in steps of 16 as the kernels are instantiated
static inline int st_steps(int d) { const int s = (d + 15) / 16; return s <= 2 ? 2 : s <= 4 ? 4 : s <= 6 ? 6 : 8; }
static inline size_t st_workspace(const b200_sink_attn_args *a) { return (size_t)a->n_head_kv * st_cells(a) * (st_steps(a->dim) + st_steps(a->vdim)) * 32; }

// one CTA a cell: all kv heads' rows, four values a thread and step
__global__ void __launch_bounds__(256) sink_rows_bf16_kernel(const b200_sink_attn_args a, int ks, int vs, int64_t cells, uint2 *__restrict__ kd, uint2 *__restrict__ vd) {
    pdl_enter();
    const int64_t c = blockIdx.x;
    const bool used = c < a.n_kv && a.cell_seq[c] >= 0;
    const bool k4 = a.dim % 4 == 0 && a.k_cache_stride % 4 == 0 && ((uintptr_t)a.k_cache & 15) == 0, v4 = a.vdim % 4 == 0 && a.v_cache_stride % 4 == 0 && ((uintptr_t)a.v_cache & 15) == 0;
    const int gk = ks * 4, gv = vs * 4;  // groups of four values a padded row
    for (int i = threadIdx.x; i < a.n_head_kv * (gk + gv); i += blockDim.x) {
        const bool key = i < a.n_head_kv * gk;
        const int e = key ? i : i - a.n_head_kv * gk, per = key ? gk : gv, h = e / per, j = (e - h * per) * 4, width = key ? a.dim : a.vdim;
        const float *src = key ? a.k_cache + c * a.k_cache_stride + (int64_t)h * a.dim : a.v_cache + c * a.v_cache_stride + (int64_t)h * a.vdim;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (used) {
            if ((key ? k4 : v4) && j + 3 < width) {
                x = *reinterpret_cast<const float4 *>(src + j);
            } else {
                if (j < width) x.x = src[j];
                if (j + 1 < width) x.y = src[j + 1];
                if (j + 2 < width) x.z = src[j + 2];
                if (j + 3 < width) x.w = src[j + 3];
            }
        }
        (key ? kd : vd)[((int64_t)h * cells + c) * per + j / 4] = make_uint2(gm_pack_bf2(x.x, x.y), gm_pack_bf2(x.z, x.w));
    }
}

template <int KS, int VS>
__global__ void __launch_bounds__(ST_WARPS * 32, 2) sink_attn_tile_kernel(const b200_sink_attn_args a, const unsigned char *__restrict__ kd, const unsigned char *__restrict__ vd, int64_t cells) {
    pdl_enter(kd, vd);
    constexpr int KROW = KS * 32, VROW = VS * 32, KSTRIDE = KROW + 16, VSTRIDE = VROW + 16, KTILE = ST_CELLS * KSTRIDE, STAGE = KTILE + ST_CELLS * VSTRIDE, NB = ST_STEP / 8;
    constexpr float LOG2E = 1.4426950408889634f;
    extern __shared__ __align__(128) unsigned char st_smem[];
    __shared__ int cseq[ST_NBUF][ST_CELLS], cpos[ST_NBUF][ST_CELLS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int hk = blockIdx.y, gqa = a.n_head / a.n_head_kv, n_cols = a.n_tokens * gqa, col0 = blockIdx.x * ST_COLS + warp * 16, ncol = max(0, min(16, n_cols - col0));
    const int D = a.dim, V = a.vdim;
    kd += (size_t)hk * cells * KROW;
    vd += (size_t)hk * cells * VROW;
    const int n_tiles = (int)(cells / ST_CELLS);

    // the columns' tokens: lane i < 16 holds column i; the warp's one sequence (or not) and its range of positions
    int my_seq = -2, my_pos = 0;
    if (lane < ncol) { const int t = (col0 + lane) / gqa; my_seq = a.tok_seq[t]; my_pos = a.tok_pos[t]; }
    const int my_start = sa_chunk_start(my_pos, a.chunk);
    const int seq0 = __shfl_sync(0xffffffffu, my_seq, 0);
    const bool uniform = __all_sync(0xffffffffu, lane >= ncol || my_seq == seq0);
    int lo_pos = lane < ncol ? my_pos : 0x7fffffff, hi_pos = lane < ncol ? my_pos : -0x7fffffff;
#pragma unroll
    for (int s = 8; s > 0; s >>= 1) { lo_pos = min(lo_pos, __shfl_xor_sync(0xffffffffu, lo_pos, s)); hi_pos = max(hi_pos, __shfl_xor_sync(0xffffffffu, hi_pos, s)); }
    lo_pos = __shfl_sync(0xffffffffu, lo_pos, 0); hi_pos = __shfl_sync(0xffffffffu, hi_pos, 0);
    const int lo_start = sa_chunk_start(lo_pos, a.chunk), hi_start = sa_chunk_start(hi_pos, a.chunk);
    const int rs0 = __shfl_sync(0xffffffffu, my_seq, g), rp0 = __shfl_sync(0xffffffffu, my_pos, g), rl0 = sa_chunk_start(rp0, a.chunk);
    const int rs1 = __shfl_sync(0xffffffffu, my_seq, g + 8), rp1 = __shfl_sync(0xffffffffu, my_pos, g + 8), rl1 = sa_chunk_start(rp1, a.chunk);
    enum { WHOLE = 0, PART = 1, HIDDEN = 2, BOTH_HIDDEN = HIDDEN | HIDDEN << 2 };
    // the cells of the tile to be looked at next, lane and lane + 32 of it: asked for a tile ahead
    int look_seq[2], look_pos[2];
    auto look_at = [&](int t) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int64_t c = (int64_t)t * ST_CELLS + lane + 32 * i;
            look_seq[i] = -1; look_pos[i] = 0;
            if (c < a.n_kv) { look_seq[i] = a.cell_seq[c]; look_pos[i] = a.cell_pos[c]; }
        }
    };
    auto tile_kinds = [&]() {  // of that tile's halves, two bits each
        int kinds = 0;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int cs = look_seq[i], cp = look_pos[i];
            bool all, none;
            if (!uniform) {  // token by token: its columns follow one another
                all = none = true;
                for (int i = 0; i < ncol; i += gqa - (col0 + i) % gqa) {
                    const int ts = __shfl_sync(0xffffffffu, my_seq, i), tp = __shfl_sync(0xffffffffu, my_pos, i), tl = __shfl_sync(0xffffffffu, my_start, i);
                    const bool v = cs >= 0 && sa_visible(cs, cp, ts, tp, a.window, a.keep_first, tl);
                    all = all && v;
                    none = none && !v;
                }
            } else {
                all = cs == seq0 && cs >= 0 && cp <= lo_pos && cp >= hi_start && (a.window <= 0 || hi_pos - cp < a.window || cp < a.keep_first);
                none = cs != seq0 || cs < 0 || cp > hi_pos || cp < lo_start || (a.window > 0 && lo_pos - cp >= a.window && cp >= a.keep_first);
            }
            const bool hidden = __all_sync(0xffffffffu, none), whole = __all_sync(0xffffffffu, all);
            kinds |= (hidden ? HIDDEN : whole ? WHOLE : PART) << (2 * i);
        }
        return ncol > 0 ? kinds : (int)BOTH_HIDDEN;
    };

    // the CTA's next tile that one of its warps sees: the same for all threads; what this warp sees of it
    int next = 0;
    look_at(0);
    auto advance = [&](int &kinds) {
        for (; next < n_tiles; next++) {
            kinds = tile_kinds();
            look_at(next + 1);
            if (__syncthreads_or(kinds != BOTH_HIDDEN)) return next++;
        }
        return -1;
    };
    auto load_stage = [&](int t, int st) {
        if (t >= 0) {
            unsigned char *base = st_smem + (size_t)st * STAGE;
            const unsigned char *kt = kd + (size_t)t * ST_CELLS * KROW, *vt = vd + (size_t)t * ST_CELLS * VROW;
#pragma unroll 4
            for (int i = tid; i < ST_CELLS * (KROW / 16); i += ST_WARPS * 32) cp_async16(base + i / (KROW / 16) * KSTRIDE + i % (KROW / 16) * 16, kt + (size_t)i * 16);
#pragma unroll 4
            for (int i = tid; i < ST_CELLS * (VROW / 16); i += ST_WARPS * 32) cp_async16(base + KTILE + i / (VROW / 16) * VSTRIDE + i % (VROW / 16) * 16, vt + (size_t)i * 16);
            if (tid < ST_CELLS) {
                const int64_t c = (int64_t)t * ST_CELLS + tid;
                if (c < a.n_kv) {
                    cp_async4(&cseq[st][tid], a.cell_seq + c);
                    cp_async4(&cpos[st][tid], a.cell_pos + c);
                } else {
                    cseq[st][tid] = -1;
                    cpos[st][tid] = 0;
                }
            }
        }
        cp_async_commit();
    };
    int ahead[ST_NBUF], seen[ST_NBUF];  // tiles in the ring, oldest first, and their kinds
#pragma unroll
    for (int i = 0; i < ST_NBUF - 1; i++) { ahead[i] = advance(seen[i]); load_stage(ahead[i], i); }

    // queries as bf16 A fragments, straight from the f32 rows
    unsigned qa[KS][4];
    float lin[2];
    int hd[2];
#pragma unroll
    for (int hh = 0; hh < 2; hh++) {
        const bool ok = g + 8 * hh < ncol;
        const int col = ok ? col0 + g + 8 * hh : 0, t = col / gqa;
        hd[hh] = hk * gqa + col % gqa;
        lin[hh] = sa_dist_slope(a, hd[hh]);
        const float *qr = a.q + (int64_t)t * a.q_stride + (int64_t)hd[hh] * D;
#pragma unroll
        for (int s = 0; s < KS; s++) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int d = 16 * s + 8 * e + 2 * t4;
                qa[s][hh + 2 * e] = gm_pack_bf2(ok && d < D ? qr[d] : 0.f, ok && d + 1 < D ? qr[d + 1] : 0.f);
            }
        }
    }
    float o[2 * VS][4];
#pragma unroll
    for (int j = 0; j < 2 * VS; j++) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};  // maximum (times log2 e) and this lane's share of the sum
    const bool sig = a.weights == B200_ATTN_SIGMOID, plain = !sig && a.softcap <= 0.f && !a.dist_bias && a.scale > 0.f;
    const float two_over_cap = a.softcap > 0.f ? 2.0f / a.softcap : 0.f;
    const int mi = lane >> 3, mr = lane & 7;
    const unsigned k_off = (unsigned)(((mi >> 1) * 8 + mr) * KSTRIDE + (mi & 1) * 16), v_off = (unsigned)(((mi & 1) * 8 + mr) * VSTRIDE + (mi >> 1) * 16);

    int stage = 0;
    for (;;) {
        if (ahead[0] < 0) break;
        const int kinds = seen[0];
        int kinds_n = BOTH_HIDDEN;
        cp_async_wait<ST_NBUF - 2>();
        const int tn = advance(kinds_n);  // (its barriers: the tile has landed for everybody, and everybody is done with the one before)
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ST_NBUF - 2; i++) { ahead[i] = ahead[i + 1]; seen[i] = seen[i + 1]; }
        ahead[ST_NBUF - 2] = tn;
        seen[ST_NBUF - 2] = kinds_n;
        load_stage(tn, stage == 0 ? ST_NBUF - 1 : stage - 1);
        const int st = stage;
        stage = stage + 1 == ST_NBUF ? 0 : stage + 1;
#pragma unroll 1
        for (int half = 0; half < ST_CELLS / ST_STEP; half++) {
            const int kind = kinds >> (2 * half) & 3, x0 = half * ST_STEP;
            if (kind == HIDDEN) continue;
            const unsigned kt = smem_u32(st_smem + (size_t)st * STAGE) + (unsigned)(x0 * KSTRIDE), vt = smem_u32(st_smem + (size_t)st * STAGE) + KTILE + (unsigned)(x0 * VSTRIDE);
            float s[NB][4];
#pragma unroll
            for (int j = 0; j < NB; j++) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
            for (int ks = 0; ks < KS; ks++) {
#pragma unroll
                for (int j = 0; j < NB / 2; j++) {
                    unsigned b0, b1, b2, b3;
                    gm_ldsm4(kt + k_off + (unsigned)(j * 16 * KSTRIDE) + ks * 32, b0, b1, b2, b3);
                    gm_mma_bf16(s[2 * j], qa[ks], b0, b1);
                    gm_mma_bf16(s[2 * j + 1], qa[ks], b2, b3);
                }
            }
            // s[j][2 hh + e]: column g + 8 hh, cell x0 + 8 j + 2 t4 + e.  `c` takes raw products to scaled scores times log2 e inside the exponent's FMA
            float c = a.scale * LOG2E;
            if (kind == PART || !plain) {
#pragma unroll
                for (int j = 0; j < NB; j++) {
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        const int x = x0 + 8 * j + 2 * t4 + e, xs = cseq[st][x], xp = cpos[st][x];
                        const bool v0 = xs >= 0 && sa_visible(xs, xp, rs0, rp0, a.window, a.keep_first, rl0), v1 = xs >= 0 && sa_visible(xs, xp, rs1, rp1, a.window, a.keep_first, rl1);
                        float s0 = s[j][e] * a.scale, s1 = s[j][2 + e] * a.scale;
                        if (a.softcap > 0.f) { s0 = sa_cap_fast(s0, a.softcap, two_over_cap); s1 = sa_cap_fast(s1, a.softcap, two_over_cap); }
                        if (a.dist_bias) {
                            if (v0) s0 += sa_dist_bias(a, rp0 - xp, hd[0], lin[0]);
                            if (v1) s1 += sa_dist_bias(a, rp1 - xp, hd[1], lin[1]);
                        }
                        s[j][e] = v0 ? (sig ? s0 : s0 * LOG2E) : -INFINITY;
                        s[j][2 + e] = v1 ? (sig ? s1 : s1 * LOG2E) : -INFINITY;
                    }
                }
                c = 1.0f;
            }
            if (sig) {  // every visible key's weight is the sigmoid of its own score (0 for the others: the sigmoid of -inf)
#pragma unroll
                for (int j = 0; j < NB; j++) {
#pragma unroll
                    for (int e = 0; e < 4; e++) s[j][e] = sa_sigmoid_fast(s[j][e]);
                }
            } else {
                float alpha[2];
#pragma unroll
                for (int hh = 0; hh < 2; hh++) {
                    float mx = fmaxf(s[0][2 * hh], s[0][2 * hh + 1]);
#pragma unroll
                    for (int j = 1; j < NB; j++) mx = fmaxf(mx, fmaxf(s[j][2 * hh], s[j][2 * hh + 1]));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                    const float mn = fmaxf(m[hh], mx * c), mb = mn == -INFINITY ? 0.f : mn;  // (nothing seen yet: 2^-inf = 0 throughout)
                    alpha[hh] = mn == -INFINITY ? 1.0f : st_ex2(m[hh] - mb);
                    m[hh] = mn;
                    float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
                    for (int j = 0; j < NB; j++) {
                        s[j][2 * hh] = st_ex2(fmaf(s[j][2 * hh], c, -mb));
                        s[j][2 * hh + 1] = st_ex2(fmaf(s[j][2 * hh + 1], c, -mb));
                        sum0 += s[j][2 * hh];
                        sum1 += s[j][2 * hh + 1];
                    }
                    l[hh] = l[hh] * alpha[hh] + (sum0 + sum1);
                }
                if (__any_sync(0xffffffffu, alpha[0] != 1.0f || alpha[1] != 1.0f)) {
#pragma unroll
                    for (int i = 0; i < 2 * VS; i++) {
                        o[i][0] *= alpha[0]; o[i][1] *= alpha[0];
                        o[i][2] *= alpha[1]; o[i][3] *= alpha[1];
                    }
                }
            }
#pragma unroll
            for (int kk = 0; kk < ST_STEP / 16; kk++) {
                const unsigned pa[4] = {gm_pack_bf2(s[2 * kk][0], s[2 * kk][1]), gm_pack_bf2(s[2 * kk][2], s[2 * kk][3]), gm_pack_bf2(s[2 * kk + 1][0], s[2 * kk + 1][1]),
                                        gm_pack_bf2(s[2 * kk + 1][2], s[2 * kk + 1][3])};
#pragma unroll
                for (int j = 0; j < VS; j++) {
                    unsigned b0, b1, b2, b3;
                    gm_ldsm4_t(vt + v_off + (unsigned)(kk * 16 * VSTRIDE) + j * 32, b0, b1, b2, b3);
                    gm_mma_bf16(o[2 * j], pa, b0, b1);
                    gm_mma_bf16(o[2 * j + 1], pa, b2, b3);
                }
            }
        }
    }
    cp_async_wait<0>();
#pragma unroll
    for (int hh = 0; hh < 2; hh++) {
        l[hh] += __shfl_xor_sync(0xffffffffu, l[hh], 1);
        l[hh] += __shfl_xor_sync(0xffffffffu, l[hh], 2);
        if (g + 8 * hh >= ncol) continue;
        const int col = col0 + g + 8 * hh, t = col / gqa, h = hd[hh];
        float w = 1.0f;
        if (!sig) {  // the sink joins the denominator
            const float sink = a.sink ? a.sink[h] * LOG2E : -INFINITY, M = fmaxf(m[hh], sink), f = m[hh] == -INFINITY ? 0.f : st_ex2(m[hh] - M);
            const float d = l[hh] * f + (a.sink ? st_ex2(sink - M) : 0.f);
            w = d > 0.f ? f / d : 0.f;
        }
        w *= sa_head_gate(a, t, h);
        float *out = a.dst + (int64_t)t * a.dst_stride + (int64_t)h * V;
#pragma unroll
        for (int j = 0; j < 2 * VS; j++) {
            const int x = 8 * j + 2 * t4;
            if (x < V) out[x] = o[j][2 * hh] * w * sa_value_gate(a, t, h, x);
            if (x + 1 < V) out[x + 1] = o[j][2 * hh + 1] * w * sa_value_gate(a, t, h, x + 1);
        }
    }
}

template <int KS, int VS>
static int st_launch2(const b200_sink_attn_args *a, unsigned char *ws, cudaStream_t st) {
    const int64_t cells = st_cells(a);
    unsigned char *kd = ws, *vd = ws + (size_t)a->n_head_kv * cells * KS * 32;
    B200_CUDA_TRY(launch_chained(sink_rows_bf16_kernel, (unsigned)cells, 256, 0, st, *a, KS, VS, cells, (uint2 *)kd, (uint2 *)vd));
    constexpr int smem = ST_NBUF * ST_CELLS * ((KS + VS) * 32 + 32);
    static bool attr_set_dev[16] = {};  // cudaFuncSetAttribute is per device
    int cur_dev = 0;
    B200_CUDA_TRY(cudaGetDevice(&cur_dev));
    bool &attr_set = attr_set_dev[cur_dev & 15];
    if (!attr_set) {
        B200_CUDA_TRY(cudaFuncSetAttribute(sink_attn_tile_kernel<KS, VS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attr_set = true;
    }
    const dim3 grid((unsigned)(((int64_t)a->n_tokens * (a->n_head / a->n_head_kv) + ST_COLS - 1) / ST_COLS), (unsigned)a->n_head_kv);
    B200_CUDA_TRY(launch_chained(sink_attn_tile_kernel<KS, VS>, grid, ST_WARPS * 32, smem, st, *a, kd, vd, cells));
    return B200_OK;
}
template <int KS>
static int st_launch1(const b200_sink_attn_args *a, unsigned char *ws, cudaStream_t st) {
    switch (st_steps(a->vdim)) {
        case 2: return st_launch2<KS, 2>(a, ws, st);
        case 4: return st_launch2<KS, 4>(a, ws, st);
        case 6: return st_launch2<KS, 6>(a, ws, st);
        default: return st_launch2<KS, 8>(a, ws, st);
    }
}
static int st_launch(const b200_sink_attn_args *a, void *workspace, cudaStream_t st) {
    unsigned char *ws = (unsigned char *)workspace;
    switch (st_steps(a->dim)) {
        case 2: return st_launch1<2>(a, ws, st);
        case 4: return st_launch1<4>(a, ws, st);
        case 6: return st_launch1<6>(a, ws, st);
        default: return st_launch1<8>(a, ws, st);
    }
}
// worth its extra launch where the columns make enough CTAs to fill a good part of the device; with fewer, the kernel with a CTA per query
// head has more of them
static bool st_wanted(const b200_sink_attn_args *a) {
    return a->n_kv > 0 && ((int64_t)a->n_tokens * (a->n_head / a->n_head_kv) + ST_COLS - 1) / ST_COLS * a->n_head_kv >= 48 && a->n_head_kv <= 65535;
}

}  // namespace b200
