// recur.cu -- mixers that carry a fixed-size state per sequence instead of a cache row per token (include/b200_ggml_ops.h:
// b200_op_short_conv, b200_op_delta_rule_scan, b200_op_mingru_scan, b200_op_token_shift, b200_op_time_mix_scan).  A batch names its sequences through seq_info (first token,
// token count, state slot, fresh); a fresh sequence starts from zeros whatever its slot held before.  Everything is f32.
#include "ops_util.cuh"

namespace b200 {
using namespace opx;

__device__ __forceinline__ float silu_f(float x) { return x / (1.0f + expf(-x)); }
// ln(1 + e^x) without overflow for large x and without cancellation for very negative x
__device__ __forceinline__ float softplus_f(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }

// ------------------------------------------------------------------------------------------------ short causal convolution
// A thread takes VEC channels, a CTA 128 threads' channels of SC_TOK tokens of one sequence.  Input i of a sequence's portion is x[first + i]
// (+ bias) for i >= 0 and the tail's entry taps - 1 + i before that; only the CTA of the portion's first tokens reads the tail, and
// it alone rewrites it afterwards (each channel by one thread, so nobody else touches the same values): the new tail is the last taps - 1
// inputs, which are old tail entries shifted down where the portion is shorter than the tail.
// KMAX >= taps is the compile-time window: the weights are padded with zeros in front, the SC_TOK + KMAX - 1 inputs of the CTA's
// tokens travel to registers with all loads in flight at once, and every output is KMAX multiply-adds on registers.  KMAX == 0 is
// the general form for longer filters (every input read where it is used).
// Two channels a thread where all rows start on 8 bytes, one channel a thread would be more CTAs than the device holds at once, and few of them begin a sequence (whose
// loads from two places are slower so): 512 tokens of 12288 channels 16.0 -> 13.6 us.  (40 tokens of 1920 channels 4.7 -> 6.6.)
constexpr int SC_TOK = 16, SC_MAX_TAPS = SC_TOK + 1;
template <int KMAX, int VEC>
__global__ void __launch_bounds__(128) short_conv_kernel(const b200_short_conv_args a) {
    pdl_enter();
    const int c = (blockIdx.x * 128 + threadIdx.x) * VEC, s = blockIdx.z;
    const int first = a.seq_info[s], count = a.seq_info[a.n_seq + s], slot = a.seq_info[2 * a.n_seq + s], fresh = a.seq_info[3 * a.n_seq + s];
    const int t0 = blockIdx.y * SC_TOK;
    if (c >= a.channels || t0 >= count) return;
    const int taps = a.taps, nt = min(SC_TOK, count - t0);
    float bias[VEC];
#pragma unroll
    for (int e = 0; e < VEC; e++) bias[e] = a.bias ? a.bias[c + e] : 0.f;
    float *tail = a.tail + (int64_t)slot * a.slot_stride + c;  // entry j at tail[j * channels]
    const float *w = a.w + (int64_t)c * taps;
    auto input = [&](int i, int e) -> float {
        if (i >= 0) return a.x[(int64_t)(first + i) * a.x_stride + c + e] + bias[e];
        return (fresh || i < -(taps - 1)) ? 0.f : tail[(int64_t)(taps - 1 + i) * a.channels + e];
    };
    if (KMAX > 0) {
        float wp[KMAX > 0 ? KMAX : 1][VEC], win[SC_TOK + (KMAX > 0 ? KMAX : 1) - 1][VEC];  // win[i] = input t0 + i - (KMAX - 1)
#pragma unroll
        for (int j = 0; j < KMAX; j++) {
#pragma unroll
            for (int e = 0; e < VEC; e++) wp[j][e] = j >= KMAX - taps ? w[e * taps + j - (KMAX - taps)] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < SC_TOK + KMAX - 1; i++) {
#pragma unroll
            for (int e = 0; e < VEC; e++) win[i][e] = 0.f;
        }
        if (t0 > 0) {  // every input is a value of x (KMAX - 1 <= SC_TOK): no test between the loads but the end of the portion
            const float *xp = a.x + (int64_t)(first + t0 - (KMAX - 1)) * a.x_stride + c;
#pragma unroll
            for (int i = 0; i < SC_TOK + KMAX - 1; i++) {
                if (i - (KMAX - 1) >= nt) continue;
                if constexpr (VEC == 2) {
                    const float2 v = *reinterpret_cast<const float2 *>(xp + (int64_t)i * a.x_stride);
                    win[i][0] = v.x; win[i][1] = v.y;
                } else {
                    win[i][0] = xp[(int64_t)i * a.x_stride];
                }
            }
#pragma unroll
            for (int i = 0; i < SC_TOK + KMAX - 1; i++) {
#pragma unroll
                for (int e = 0; e < VEC; e++) win[i][e] += bias[e];  // (beyond the portion's end nobody reads it)
            }
        } else {
#pragma unroll
            for (int i = 0; i < SC_TOK + KMAX - 1; i++) {
#pragma unroll
                for (int e = 0; e < VEC; e++) if (i - (KMAX - 1) < nt) win[i][e] = input(t0 + i - (KMAX - 1), e);
            }
        }
#pragma unroll
        for (int t = 0; t < SC_TOK; t++) {
            float y[VEC];
#pragma unroll
            for (int e = 0; e < VEC; e++) {
                y[e] = 0.f;
#pragma unroll
                for (int j = 0; j < KMAX; j++) y[e] += wp[j][e] * win[t + j][e];
            }
            if (t < nt) {
#pragma unroll
                for (int e = 0; e < VEC; e++) if (a.act) y[e] = silu_f(y[e]);
                float *d = a.dst + (int64_t)(first + t0 + t) * a.dst_stride + c;
                if constexpr (VEC == 2) *reinterpret_cast<float2 *>(d) = make_float2(y[0], y[1]);
                else d[0] = y[0];
            }
        }
    } else {
        for (int t = t0; t < t0 + nt; t++) {
            for (int e = 0; e < VEC; e++) {
                float y = 0.f;
                for (int j = 0; j < taps; j++) y += w[e * taps + j] * input(t - taps + 1 + j, e);
                a.dst[(int64_t)(first + t) * a.dst_stride + c + e] = a.act ? silu_f(y) : y;
            }
        }
    }
    if (t0 == 0) {
        // entry j of the new tail is input count - (taps - 1) + j: an old entry of higher index, or a value of x; ascending j never
        // reads what it has written
        for (int j = 0; j < taps - 1; j++) {
#pragma unroll
            for (int e = 0; e < VEC; e++) tail[(int64_t)j * a.channels + e] = input(count - (taps - 1) + j, e);
        }
    }
}

// ------------------------------------------------------------------------------------------------ gated delta rule
// The columns of the state never interact: column j of S [dim, vdim] sees  S_j <- g S_j + k u_j  with  u_j = beta (v_j - g k.S_j),
// and the read-out is  o_j = q.S_j(new).  Token by token that is a chain S -> sums over the column -> u -> S of about 500 cycles, most of it latency.
// So four tokens are taken at once.  With S0 in front of them and G(t, j) = g_(j+1) ... g_t (products: nothing is divided),
//   u_t = beta_t (v_t - G(t, -1) k_t.S0 - sum_(j < t) G(t, j) (k_t.k_j) u_j),   o_t = G(t, -1) q_t.S0 + sum_(j <= t) G(t, j) (q_t.k_j) u_j,
//   S <- G(3, -1) S0 + sum_j G(3, j) k_j u_j:
// the eight sums over a column all read S0 and travel together, the dot products among the tokens do not depend on S and are made ahead, and what is left
// in a chain is a triangle of four.  The tokens behind the last whole group of four go through the same steps one by one.
//   * A warp carries 8 columns: LR lanes share CPL of them, lane r of them keeping rows 4 (r + LR i) .. + 3 in registers.  Rows are worked on two
//     at a time (packed f32).  16 lanes and 4 columns: a 16-byte load of k or q, four cycles of the shared-memory pipe, serves 16 products;
//     the sums of the four columns are exchanged so that four lanes end up with one column (halving: 16 + 8 values, then 11).  Column c of lane r is
//     number c ^ (r / 4) of the group: what a lane gives away in that exchange has the same names in all lanes.
//   * Four warps carry the state and do nothing else; four more prepare the next chunk meanwhile, a group of four tokens each: q and k as unit vectors
//     (q scaled), their dot products, decays and beta.
// What bounds it: issue (about 570 instructions a warp for four tokens, 208 of them packed multiply-adds of two to three cycles each) and the latency of
// the exchanges; with a decay per channel the staging warps' exponentials.  512 tokens, 32 heads of 128 x 128: 136 us token by token, 87 us here;
// 312 tokens, 22 heads of 64 x 64 with decays per channel 80 -> 53 us with the convolution in front.
// CHAN: the decay is one factor per key channel (row of S) instead of one per head: G is a vector, and what is staged are G(t, -1) k_t and G(t, -1) q_t for
// the sums, G(3, j) k_j for the update and G(3, -1) itself; the dot products are taken with G between their factors.
constexpr int DR_T = 4, DR_WARPS = 4, DR_COLS = 8 * DR_WARPS;
template <int DQ, bool CHAN> constexpr int dr_chunk() { return DQ * (CHAN ? 2 : 1) <= 8 ? 16 : 8; }  // tokens staged at once: DR_T for each staging warp, if two chunks fit 64 KB
// coefficients of a group of tokens, in floats from the group's row: beta_t | beta_t G(t, -1) | beta_t G(t, j) k_t.k_j for (1, 0) (2, 0) (2, 1) (3, 0) .. |
// G(3, j) | G(t, -1) | G(t, j) q_t.k_j, four a token.  Of an incomplete group every token is a group of its own.
constexpr int DR_BETA = 0, DR_BG = 4, DR_KK = 8, DR_LAST = 16, DR_G = 20, DR_QK = 24, DR_COEF = 40;
// a sequence shorter than this goes token by token: with a decay per channel the exponentials of a group, which one warp stages, take longer than four steps
template <bool CHAN> constexpr int dr_grouped() { return CHAN ? 16 : DR_T; }
template <int DQ, bool CHAN> constexpr int dr_smem() {
    constexpr int C = dr_chunk<DQ, CHAN>();
    return 4 * 2 * C * (32 * DQ * (CHAN ? 4 : 2) + DR_COLS + DR_COEF / DR_T);
}
__device__ __forceinline__ unsigned long long dr_pack(float lo, float hi) { unsigned long long r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ float2 dr_unpack(unsigned long long x) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x)); return r; }
__device__ __forceinline__ unsigned long long dr_fma(unsigned long long x, unsigned long long y, unsigned long long z) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
    return r;
}
__device__ __forceinline__ unsigned long long dr_mul(unsigned long long x, unsigned long long y) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return r;
}
__device__ __forceinline__ unsigned long long dr_add(unsigned long long x, unsigned long long y) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    return r;
}
// the meeting of both roles: all warps of the CTA, from whichever branch they come (__syncthreads() wants one place for all threads)
__device__ __forceinline__ void dr_meet() { asm volatile("bar.sync 1, %0;" ::"n"(DR_WARPS * 64) : "memory"); }
// sums over lanes that differ in bit `off`: N values become N / 2, the lanes with the bit set keep the upper half
template <int N>
__device__ __forceinline__ void dr_halve(float *v, bool upper, int off) {
#pragma unroll
    for (int i = 0; i < N / 2; i++) {
        const float send = upper ? v[i] : v[i + N / 2], keep = upper ? v[i + N / 2] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
}
template <int DQ, bool CHAN>
struct DrSmem {  // of one of the two buffers
    static constexpr int C = dr_chunk<DQ, CHAN>(), DP = 32 * DQ;
    float *k, *q, *kd, *g, *v, *coef;  // k, q [C][DP] for the sums; CHAN: kd [C][DP] for the update, g [C][DP]; v [C / 4][DR_COLS][4]; coef [C / 4][DR_COEF]
    __device__ __forceinline__ DrSmem(float *base, int buf) {
        base += buf * (dr_smem<DQ, CHAN>() / 8);
        k = base;
        q = k + C * DP;
        kd = CHAN ? q + C * DP : k;
        g = CHAN ? kd + C * DP : q;
        v = (CHAN ? g : q) + C * DP;
        coef = v + C * DR_COLS;
    }
};

// products of the lane's pieces of a row vector with its columns.  The columns are the inner loop: an instruction that reads the same register pair in the same
// place as the one before it issues in two cycles, with three new pairs it takes three.
template <int CPL, int NR>
__device__ __forceinline__ void dr_dots(const unsigned long long (&x)[NR][2], const unsigned long long (&y)[CPL][NR][2], float *to, int stride) {
    unsigned long long s[CPL][2];
#pragma unroll
    for (int i = 0; i < NR; i++) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
#pragma unroll
            for (int c = 0; c < CPL; c++) s[c][e] = i == 0 ? dr_mul(x[0][e], y[c][0][e]) : dr_fma(x[i][e], y[c][i][e], s[c][e]);
        }
    }
#pragma unroll
    for (int c = 0; c < CPL; c++) {
        const float2 z = dr_unpack(dr_add(s[c][0], s[c][1]));
        to[c * stride] = z.x + z.y;
    }
}

// ===== T tokens of a chunk, tok .. tok + T - 1 (T == DR_T: a whole group), against the columns that the warp carries
template <int DQ, bool CHAN, int T>
__device__ __forceinline__ void dr_step(unsigned long long (&S)[DQ == 1 ? 2 : 4][DQ == 1 ? 1 : DQ / 2][2], const DrSmem<DQ, CHAN> &sm, int tok, int warp, int lane, float *out, int64_t out_stride,
                                        bool col_ok) {
    constexpr int LR = DQ == 1 ? 8 : 16, CPL = LR / 4, NR = DQ == 1 ? 1 : DQ / 2, DP = 32 * DQ;
    const int r = lane & (LR - 1), cg = lane / LR;
    unsigned long long kk[T][NR][2];
    float ks[CPL * T], qs[CPL * T];  // [column][token]
    // the k sums travel while the q sums are made, the q sums while S moves on
#pragma unroll
    for (int t = 0; t < T; t++) {
#pragma unroll
        for (int i = 0; i < NR; i++) {
            const ulonglong2 kv = *reinterpret_cast<const ulonglong2 *>(sm.k + (tok + t) * DP + 4 * (r + LR * i));
            kk[t][i][0] = kv.x; kk[t][i][1] = kv.y;
        }
        dr_dots<CPL, NR>(kk[t], S, ks + t, T);
    }
    // one column for each four lanes: the lane's column 0 (columns are numbered from there: what a lane gives away are always the upper ones)
#pragma unroll
    for (int n = CPL / 2; n >= 1; n >>= 1) {
#pragma unroll
        for (int i = 0; i < T * n; i++) ks[i] += __shfl_xor_sync(0xffffffffu, ks[i + T * n], 4 * n);
    }
#pragma unroll
    for (int t = 0; t < T; t++) ks[t] += __shfl_xor_sync(0xffffffffu, ks[t], 2);
#pragma unroll
    for (int t = 0; t < T; t++) ks[t] += __shfl_xor_sync(0xffffffffu, ks[t], 1);
#pragma unroll
    for (int t = 0; t < T; t++) {
        unsigned long long qq[NR][2];
#pragma unroll
        for (int i = 0; i < NR; i++) {
            const ulonglong2 qv = *reinterpret_cast<const ulonglong2 *>(sm.q + (tok + t) * DP + 4 * (r + LR * i));
            qq[i][0] = qv.x; qq[i][1] = qv.y;
        }
        dr_dots<CPL, NR>(qq, S, qs + t, T);
    }
    const int col = warp * 8 + cg * CPL + (r >> 2);
    const int group = tok / DR_T, i0 = tok % DR_T;
    const float *co = sm.coef + group * DR_COEF;
    float u[T], last, o;
    if constexpr (T == 4) {
        const float4 v = *reinterpret_cast<const float4 *>(sm.v + (group * DR_COLS + col) * 4), be = *reinterpret_cast<const float4 *>(co + DR_BETA), bg = *reinterpret_cast<const float4 *>(co + DR_BG);
        const float4 a = *reinterpret_cast<const float4 *>(co + DR_KK), w = *reinterpret_cast<const float4 *>(co + DR_LAST), qk = *reinterpret_cast<const float4 *>(co + DR_QK + 4 * (r & 3));
        const float2 a2 = *reinterpret_cast<const float2 *>(co + DR_KK + 4);
        u[0] = be.x * v.x - bg.x * ks[0];
        u[1] = (be.y * v.y - bg.y * ks[1]) - a.x * u[0];
        u[2] = ((be.z * v.z - bg.z * ks[2]) - a.y * u[0]) - a.z * u[1];
        u[3] = (((be.w * v.w - bg.w * ks[3]) - a.w * u[0]) - a2.x * u[1]) - a2.y * u[2];
        o = qk.x * u[0];  // (of the tokens behind the lane's nothing enters, not even as 0 times it)
        if ((r & 3) > 0) o += qk.y * u[1];
        if ((r & 3) > 1) o += qk.z * u[2];
        if ((r & 3) > 2) o += qk.w * u[3];
        if (!CHAN) { u[0] *= w.x; u[1] *= w.y; u[2] *= w.z; u[3] *= w.w; }
        last = co[DR_G + 3];
    } else {
        u[0] = co[DR_BETA + i0] * sm.v[(group * DR_COLS + col) * 4 + i0] - co[DR_BG + i0] * ks[0];
        last = co[DR_G + i0];
        o = co[DR_QK + 4 * i0] * u[0];
    }
    if (CHAN) {
#pragma unroll
        for (int t = 0; t < T; t++) {
#pragma unroll
            for (int i = 0; i < NR; i++) {
                const ulonglong2 kv = *reinterpret_cast<const ulonglong2 *>(sm.kd + (tok + t) * DP + 4 * (r + LR * i));
                kk[t][i][0] = kv.x; kk[t][i][1] = kv.y;
            }
        }
    }
    unsigned long long gv[NR][2];
#pragma unroll
    for (int i = 0; i < NR; i++) {
        if (CHAN) {
            const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(sm.g + tok * DP + 4 * (r + LR * i));
            gv[i][0] = x.x; gv[i][1] = x.y;
        } else {
            gv[i][0] = gv[i][1] = dr_pack(last, last);
        }
    }
    unsigned long long u2[CPL][T];
#pragma unroll
    for (int c = 0; c < CPL; c++) {
#pragma unroll
        for (int t = 0; t < T; t++) {
            const float x = c == 0 ? u[t] : __shfl_xor_sync(0xffffffffu, u[t], 4 * c);
            u2[c][t] = dr_pack(x, x);
        }
    }
#pragma unroll
    for (int i = 0; i < NR; i++) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
            unsigned long long add[CPL];  // (the small terms k u are the ones that are rounded first)
#pragma unroll
            for (int t = 0; t < T; t++) {
#pragma unroll
                for (int c = 0; c < CPL; c++) add[c] = t == 0 ? dr_mul(kk[0][i][e], u2[c][0]) : dr_fma(kk[t][i][e], u2[c][t], add[c]);
            }
#pragma unroll
            for (int c = 0; c < CPL; c++) S[c][i][e] = dr_fma(S[c][i][e], gv[i][e], add[c]);
        }
    }
    // the read-out of token r & 3
#pragma unroll
    for (int n = CPL / 2; n >= 1; n >>= 1) {
#pragma unroll
        for (int i = 0; i < T * n; i++) qs[i] += __shfl_xor_sync(0xffffffffu, qs[i + T * n], 4 * n);
    }
    if constexpr (T == 4) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const float send = r & 2 ? qs[i] : qs[i + 2], keep = r & 2 ? qs[i + 2] : qs[i];
            qs[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
        }
        const float send = r & 1 ? qs[0] : qs[1], keep = r & 1 ? qs[1] : qs[0];
        qs[0] = keep + __shfl_xor_sync(0xffffffffu, send, 1);
        if (col_ok) out[(r & 3) * out_stride] = co[DR_G + (r & 3)] * qs[0] + o;
    } else {
        qs[0] += __shfl_xor_sync(0xffffffffu, qs[0], 2);
        qs[0] += __shfl_xor_sync(0xffffffffu, qs[0], 1);
        if (col_ok && (r & 3) == 0) out[0] = last * qs[0] + o;
    }
}

// ===== staging: T tokens (a whole group, or one by itself) from token t0 of the sequence on, tok of the chunk, by one warp; all loads in flight at once
template <int DQ, bool CHAN, int T>
__device__ __forceinline__ void dr_stage(const b200_delta_rule_args &a, const DrSmem<DQ, CHAN> &sm, int64_t t0, int tok, int h, int kvh, int cb, int lane, float decay_rate, float dtb,
                                         const float (&bias)[CHAN ? DQ : 1]) {
    constexpr int DP = 32 * DQ;
    const int D = a.dim, V = a.vdim;
    const int t4 = T == 1 ? 0 : lane & 3;
    float q[T][DQ], k[T][DQ], z[CHAN ? T : 1][CHAN ? DQ : 1], v[T];
    const float ga = CHAN ? 0.f : a.a[(t0 + t4) * a.a_stride + h], be = a.b[(t0 + t4) * a.b_stride + h];
#pragma unroll
    for (int t = 0; t < T; t++) {
#pragma unroll
        for (int j = 0; j < DQ; j++) {
            const int d = lane + 32 * j;
            q[t][j] = d < D ? a.q[(t0 + t) * a.q_stride + (int64_t)kvh * D + d] : 0.f;
            k[t][j] = d < D ? a.k[(t0 + t) * a.k_stride + (int64_t)kvh * D + d] : 0.f;
            if (CHAN) z[CHAN ? t : 0][CHAN ? j : 0] = d < D ? a.a[(t0 + t) * a.a_stride + (int64_t)h * D + d] : 0.f;
        }
        v[t] = cb + lane < V ? a.v[(t0 + t) * a.v_stride + (int64_t)h * V + cb + lane] : 0.f;
    }
    // unit vectors.  Of the 2 T sums of squares number i (q of the tokens, then k) ends up in the lanes from 4 i (T = 4) or 16 i (T = 1) on.
    float len[2 * T];
#pragma unroll
    for (int t = 0; t < T; t++) {
        len[t] = len[T + t] = 0.f;
#pragma unroll
        for (int j = 0; j < DQ; j++) { len[t] += q[t][j] * q[t][j]; len[T + t] += k[t][j] * k[t][j]; }
    }
    dr_halve<2 * T>(len, (lane & 16) != 0, 16);
    if constexpr (T == 4) {
        dr_halve<4>(len, (lane & 8) != 0, 8);
        dr_halve<2>(len, (lane & 4) != 0, 4);
    } else {
        len[0] += __shfl_xor_sync(0xffffffffu, len[0], 8);
        len[0] += __shfl_xor_sync(0xffffffffu, len[0], 4);
    }
    len[0] += __shfl_xor_sync(0xffffffffu, len[0], 2);
    len[0] += __shfl_xor_sync(0xffffffffu, len[0], 1);
    const float f = (a.unit_qk ? 1.0f / sqrtf(len[0] + a.unit_eps) : 1.0f) * (lane < 16 ? a.q_scale : 1.0f);
#pragma unroll
    for (int t = 0; t < T; t++) {
        const float fq = __shfl_sync(0xffffffffu, f, 4 * t), fk = __shfl_sync(0xffffffffu, f, 16 + 4 * t);
#pragma unroll
        for (int j = 0; j < DQ; j++) { q[t][j] *= fq; k[t][j] *= fk; }
    }
    // dot products q_t.k_j, j <= t, then k_t.k_j, j < t, with the channels' decays between them
    float dot[T == 4 ? 16 : 1];
#pragma unroll
    for (int i = 0; i < (T == 4 ? 16 : 1); i++) dot[i] = 0.f;
    float *row = sm.k + tok * DP + lane;
    const int64_t to_q = sm.q - sm.k, to_kd = sm.kd - sm.k, to_g = sm.g - sm.k;
#pragma unroll
    for (int j = 0; j < DQ; j++) {
        float gc[T];
        if (CHAN) {
#pragma unroll
            for (int t = 0; t < T; t++) gc[t] = expf(-decay_rate * softplus_f(z[CHAN ? t : 0][CHAN ? j : 0] + bias[CHAN ? j : 0]));
        }
#pragma unroll
        for (int jj = 0; jj < T; jj++) {
            float x = k[jj][j];
#pragma unroll
            for (int t = jj; t < T; t++) {
                if (CHAN && t > jj) x *= gc[t];
                dot[t * (t + 1) / 2 + jj] += q[t][j] * x;
                if (t > jj) dot[10 + t * (t - 1) / 2 + jj] += k[t][j] * x;
            }
            if (CHAN) row[to_kd + jj * DP + 32 * j] = x;
        }
        float all = 1.0f;
#pragma unroll
        for (int t = 0; t < T; t++) {
            if (CHAN) all *= gc[t];
            row[t * DP + 32 * j] = CHAN ? k[t][j] * all : k[t][j];
            row[to_q + t * DP + 32 * j] = CHAN ? q[t][j] * all : q[t][j];
        }
        if (CHAN) row[to_g + 32 * j] = all;
    }
    const float g_mine = CHAN ? 1.0f : expf(-decay_rate * softplus_f(ga + dtb)), beta = sigmoidf_(be);
    float *co = sm.coef + tok / DR_T * DR_COEF, *vs = sm.v + (tok / DR_T * DR_COLS + lane) * 4;
    if constexpr (T == 1) {
        const int i = tok % DR_T;
        vs[i] = v[0];
        const float qk = warp_sum(dot[0]);
        if (lane == 0) {
            co[DR_BETA + i] = beta;
            co[DR_BG + i] = beta * g_mine;
            co[DR_G + i] = g_mine;
            co[DR_QK + 4 * i] = qk;
        }
    } else {
        *reinterpret_cast<float4 *>(vs) = make_float4(v[0], v[1], v[2], v[3]);
        // value i ends up in lanes 2 i and 2 i + 1
        dr_halve<16>(dot, (lane & 16) != 0, 16);
        dr_halve<8>(dot, (lane & 8) != 0, 8);
        dr_halve<4>(dot, (lane & 4) != 0, 4);
        dr_halve<2>(dot, (lane & 2) != 0, 2);
        dot[0] += __shfl_xor_sync(0xffffffffu, dot[0], 1);
        const int i = lane >> 1, t = (int)(0xFE9FFA94u >> (2 * i)) & 3, j = (int)(0x910E4910u >> (2 * i)) & 3;  // its t and j, two bits each
        float between = 1.0f, upto = 1.0f, after = 1.0f;  // G(t, j); G(t4, -1); G(3, t4)
#pragma unroll
        for (int e = 0; e < DR_T; e++) {
            const float g = CHAN ? 1.0f : __shfl_sync(0xffffffffu, g_mine, e);
            if (e > j && e <= t) between *= g;
            if (e <= t4) upto *= g;
            else after *= g;
        }
        const float beta_t = __shfl_sync(0xffffffffu, beta, t);
        if ((lane & 1) == 0) co[i >= 10 ? DR_KK + t * (t - 1) / 2 + j : DR_QK + 4 * t + j] = (i >= 10 ? beta_t : 1.0f) * (between * dot[0]);
        if (lane < DR_T) {
            co[DR_BETA + lane] = beta;
            co[DR_BG + lane] = beta * upto;
            co[DR_LAST + lane] = after;
            co[DR_G + lane] = upto;
        }
    }
}

template <int DQ, bool CHAN, int CTAS>  // dim <= 32 DQ; CTAs that an SM is to hold
__global__ void __launch_bounds__(DR_WARPS * 64, CTAS) delta_rule_scan_kernel(const b200_delta_rule_args a) {
    constexpr int DR_CHUNK = dr_chunk<DQ, CHAN>();
    extern __shared__ __align__(16) float dr_shared[];
    pdl_enter();
    const int h = blockIdx.y, s = blockIdx.z, kvh = h / (a.heads / a.kv_heads);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int D = a.dim, V = a.vdim;
    const int first = a.seq_info[s], count = a.seq_info[a.n_seq + s], slot = a.seq_info[2 * a.n_seq + s], fresh = a.seq_info[3 * a.n_seq + s];
    if (count <= 0) return;
    const int cb = blockIdx.x * DR_COLS, n_chunks = (count + DR_CHUNK - 1) / DR_CHUNK;
    const int grouped = count >= dr_grouped<CHAN>() ? ~(DR_T - 1) : 0;  // tokens of a chunk in groups: all but the remainder, or none
    if (warp >= DR_WARPS) {
        // ===== staging: a warp takes a group of tokens of every chunk, or single tokens
        const int w = warp - DR_WARPS;
        const float decay_rate = expf(a.a_log[h]), dtb = !CHAN && a.dt_bias ? a.dt_bias[h] : 0.f;
        float bias[CHAN ? DQ : 1];
        if (CHAN) {
#pragma unroll
            for (int j = 0; j < DQ; j++) bias[CHAN ? j : 0] = a.dt_bias && lane + 32 * j < D ? a.dt_bias[(int64_t)h * D + lane + 32 * j] : 0.f;
        }
        for (int c = 0; c < n_chunks; c++) {
            const DrSmem<DQ, CHAN> sm(dr_shared, c & 1);
            const int nt = min(DR_CHUNK, count - c * DR_CHUNK), in_groups = nt & grouped;
            const int64_t t0 = first + c * DR_CHUNK;
            if (DR_T * w < in_groups) dr_stage<DQ, CHAN, DR_T>(a, sm, t0 + DR_T * w, DR_T * w, h, kvh, cb, lane, decay_rate, dtb, bias);
#pragma unroll 1
            for (int tok = in_groups + ((w - in_groups / DR_T) & (DR_WARPS - 1)); tok < nt; tok += DR_WARPS)
                dr_stage<DQ, CHAN, 1>(a, sm, t0 + tok, tok, h, kvh, cb, lane, decay_rate, dtb, bias);
            dr_meet();  // chunk c is ready; chunk c - 1, whose room the next one takes, has been read
        }
        return;
    }
    // ===== the state
    constexpr int LR = DQ == 1 ? 8 : 16, CPL = LR / 4, NR = DQ == 1 ? 1 : DQ / 2;
    const int r = lane & (LR - 1), c0 = cb + warp * 8 + lane / LR * CPL;  // the lane's columns are c0 + (c ^ (r / 4))
    float *Sp = a.state + (int64_t)slot * a.slot_stride + ((int64_t)h * V + c0) * D;
    const bool pieces = ((D | (int)a.slot_stride) & 3) == 0 && ((uintptr_t)a.state & 15) == 0;  // every column starts on 16 bytes
    unsigned long long S[CPL][NR][2];
#pragma unroll
    for (int c = 0; c < CPL; c++) {
#pragma unroll
        for (int i = 0; i < NR; i++) {
            const int d = 4 * (r + LR * i), cc = c ^ (r >> 2);
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!fresh && c0 + cc < V) {
                const float *p = Sp + (int64_t)cc * D + d;
                if (pieces) {
                    if (d < D) x = *reinterpret_cast<const float4 *>(p);
                } else {
                    if (d < D) x.x = p[0];
                    if (d + 1 < D) x.y = p[1];
                    if (d + 2 < D) x.z = p[2];
                    if (d + 3 < D) x.w = p[3];
                }
            }
            S[c][i][0] = dr_pack(x.x, x.y);
            S[c][i][1] = dr_pack(x.z, x.w);
        }
    }
    const int out_col = c0 + (r >> 2);
    const bool col_ok = out_col < V;
    float *out = a.dst + (int64_t)first * a.dst_stride + (int64_t)h * V + out_col;
    for (int ch = 0; ch < n_chunks; ch++) {
        const int nt = min(DR_CHUNK, count - ch * DR_CHUNK);
        const DrSmem<DQ, CHAN> sm(dr_shared, ch & 1);
        dr_meet();
        const int in_groups = nt & grouped;
#pragma unroll 1
        for (int tt = 0; tt < in_groups; tt += DR_T, out += DR_T * a.dst_stride) dr_step<DQ, CHAN, DR_T>(S, sm, tt, warp, lane, out, a.dst_stride, col_ok);
#pragma unroll 1
        for (int tt = in_groups; tt < nt; tt++, out += a.dst_stride) dr_step<DQ, CHAN, 1>(S, sm, tt, warp, lane, out, a.dst_stride, col_ok);
    }
#pragma unroll
    for (int c = 0; c < CPL; c++) {
#pragma unroll
        for (int i = 0; i < NR; i++) {
            const int d = 4 * (r + LR * i), cc = c ^ (r >> 2);
            const float2 x = dr_unpack(S[c][i][0]), y = dr_unpack(S[c][i][1]);
            if (c0 + cc < V) {
                float *p = Sp + (int64_t)cc * D + d;
                if (pieces) {
                    if (d < D) *reinterpret_cast<float4 *>(p) = make_float4(x.x, x.y, y.x, y.y);
                } else {
                    if (d < D) p[0] = x.x;
                    if (d + 1 < D) p[1] = x.y;
                    if (d + 2 < D) p[2] = y.x;
                    if (d + 3 < D) p[3] = y.y;
                }
            }
        }
    }
}

template <int DQ, bool CHAN, int CTAS>
static int launch_delta_rule3(const b200_delta_rule_args *a, dim3 grid, cudaStream_t st) {
    constexpr int SMEM = dr_smem<DQ, CHAN>();
    const auto kern = delta_rule_scan_kernel<DQ, CHAN, CTAS>;
    if (SMEM > 48 * 1024) {
        static bool attr_set_dev[16] = {};  // cudaFuncSetAttribute is per device
        int dev = 0;
        B200_CUDA_TRY(cudaGetDevice(&dev));
        if (!attr_set_dev[dev & 15]) {
            B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
            attr_set_dev[dev & 15] = true;
        }
    }
    B200_CUDA_TRY(launch_chained(kern, grid, DR_WARPS * 64, SMEM, st, *a));
    return B200_OK;
}
// Up to a CTA an SM: all the registers it wants (512 tokens, 32 heads of 128 x 128: 87 us, 97 with the registers of two).  More CTAs than that:
// two an SM, whose waiting the other fills.
template <int DQ, bool CHAN>
static int launch_delta_rule2(const b200_delta_rule_args *a, cudaStream_t st) {
    const dim3 grid((unsigned)((a->vdim + DR_COLS - 1) / DR_COLS), (unsigned)a->heads, (unsigned)a->n_seq);
    return (int64_t)grid.x * grid.y * grid.z <= sm_count() ? launch_delta_rule3<DQ, CHAN, 1>(a, grid, st) : launch_delta_rule3<DQ, CHAN, 2>(a, grid, st);
}

template <int DQ>
static int launch_delta_rule(const b200_delta_rule_args *a, cudaStream_t st) { return a->channel_decay ? launch_delta_rule2<DQ, true>(a, st) : launch_delta_rule2<DQ, false>(a, st); }

// ------------------------------------------------------------------------------------------------ minGRU
// S_t = (1 - z_t) S_(t-1) + z_t c_t is linear in S, so a stretch of tokens acts on the state as S -> A S + B.  A CTA takes 32
// channels of one sequence (a warp row reads 128 contiguous bytes of a token) and blockDim.y stretches of MG_TPT tokens at a time:
// every thread loads its stretch with all loads in flight, turns the pre-activations into gates once, finds its (A, B), reads the
// state in front of its stretch off the earlier stretches' (A, B) in shared memory, and runs its tokens again from registers to
// write the outputs.  With few tokens (decoding) the launch has one stretch per CTA and the middle step is empty.
constexpr int MG_TPT = 8, MG_SEG_MAX = 32;
__global__ void __launch_bounds__(32 * MG_SEG_MAX) mingru_scan_kernel(const b200_mingru_args a) {
    __shared__ float sA[MG_SEG_MAX][32], sB[MG_SEG_MAX][32], sS[32];
    const int lane = threadIdx.x, seg = threadIdx.y, n_seg = blockDim.y, c = blockIdx.x * 32 + lane, s = blockIdx.y;
    const int first = a.seq_info[s], count = a.seq_info[a.n_seq + s], slot = a.seq_info[2 * a.n_seq + s], fresh = a.seq_info[3 * a.n_seq + s];
    if (count <= 0) return;
    const bool live = c < a.width;
    const float zb = (a.z_bias && live) ? a.z_bias[c] : 0.f, xb = (a.x_bias && live) ? a.x_bias[c] : 0.f;
    float *Sp = a.state + (int64_t)slot * a.slot_stride + c;
    if (seg == 0) sS[lane] = (live && !fresh) ? *Sp : 0.f;
    for (int base = 0; base < count; base += n_seg * MG_TPT) {
        const int t_lo = base + seg * MG_TPT;
        float z[MG_TPT], cand[MG_TPT], g[MG_TPT];
#pragma unroll
        for (int u = 0; u < MG_TPT; u++) {
            const bool ok = live && t_lo + u < count;
            const int64_t tok = first + t_lo + u;
            z[u] = ok ? a.z[tok * a.z_stride + c] : 0.f;
            cand[u] = ok ? a.x[tok * a.x_stride + c] : 0.f;
            g[u] = (ok && a.g) ? a.g[tok * a.g_stride + c] : 0.f;
        }
        float A = 1.f, B = 0.f;
#pragma unroll
        for (int u = 0; u < MG_TPT; u++) {
            const bool ok = t_lo + u < count;
            const float zz = ok ? sigmoidf_(z[u] + zb) : 0.f, uu = cand[u] + xb;  // a token beyond the end leaves the state as it is
            z[u] = zz; cand[u] = uu >= 0.f ? uu + 0.5f : sigmoidf_(uu);
            A *= 1.f - zz; B = (1.f - zz) * B + zz * cand[u];
        }
        sA[seg][lane] = A; sB[seg][lane] = B;
        __syncthreads();  // (also: sS holds the state in front of these stretches)
        float S = sS[lane];
        for (int j = 0; j < seg; j++) S = sA[j][lane] * S + sB[j][lane];
#pragma unroll
        for (int u = 0; u < MG_TPT; u++) {
            S = (1.f - z[u]) * S + z[u] * cand[u];
            if (live && t_lo + u < count) a.dst[(int64_t)(first + t_lo + u) * a.dst_stride + c] = a.g ? S * silu_f(g[u]) : S;
        }
        __syncthreads();  // everybody has read sS, sA, sB
        if (seg == n_seg - 1) sS[lane] = S;
    }
    __syncthreads();
    if (seg == 0 && live) *Sp = sS[lane];
}

// ------------------------------------------------------------------------------------------------ token shift
// A thread per channel, a CTA per (128 channels, TS_TOK tokens of one sequence): the TS_TOK + 1 inputs travel to registers at once and
// serve all mixes.  Only the CTA of a portion's first tokens reads the slot, and it alone rewrites it (thread = channel).
constexpr int TS_TOK = 16;
__global__ void __launch_bounds__(128) token_shift_kernel(const b200_token_shift_args a) {
    const int c = blockIdx.x * 128 + threadIdx.x, s = blockIdx.z;
    const int first = a.seq_info[s], count = a.seq_info[a.n_seq + s], slot = a.seq_info[2 * a.n_seq + s], fresh = a.seq_info[3 * a.n_seq + s];
    const int t0 = blockIdx.y * TS_TOK;
    if (c >= a.width || t0 >= count) return;
    const int nt = min(TS_TOK, count - t0);
    float *prev = a.prev + (int64_t)slot * a.slot_stride + c;
    float win[TS_TOK + 1];
    win[0] = t0 > 0 ? a.h[(int64_t)(first + t0 - 1) * a.h_stride + c] : (fresh ? 0.f : *prev);
#pragma unroll
    for (int i = 0; i < TS_TOK; i++) win[i + 1] = i < nt ? a.h[(int64_t)(first + t0 + i) * a.h_stride + c] : 0.f;
    if (t0 == 0) *prev = a.h[(int64_t)(first + count - 1) * a.h_stride + c];
    for (int m = 0; m < a.n_mix; m++) {
        const float mu = a.mu[(int64_t)m * a.width + c];
        float *dst = a.dst + (int64_t)m * a.dst_s_mix + (int64_t)(first + t0) * a.dst_s_tok + c;
#pragma unroll
        for (int i = 0; i < TS_TOK; i++) if (i < nt) dst[(int64_t)i * a.dst_s_tok] = win[i + 1] + (win[i] - win[i + 1]) * mu;
    }
}

// ------------------------------------------------------------------------------------------------ time mixing
// The columns of the state never interact: a warp owns TM_CW columns of one (sequence, head) and keeps them in registers over the
// whole token loop, a lane the key channels d = lane, lane + 32, ...  Column j sees  o_j = sum_d r_d S_dj + (sum_d r_d u_d k_d) v_j
// and  S_dj <- w_d S_dj + k_d v_j;  the bracket is the same for every column, so a lane adds its share of it once per token.  The
// inputs of CHUNK tokens are staged in shared memory (decays computed there once per CTA) while the next chunk travels to registers.
// The read-outs do not feed the recurrence: 8 tokens x 4 columns of partial sums per lane are added up across the warp in one
// halving exchange.
constexpr int TM_CW = 4, TM_WARPS = 4, TM_COLS = TM_CW * TM_WARPS, TM_RG = 8;
static_assert(TM_RG * TM_CW == 32 && TM_CW == 4, "one partial sum per lane");
template <int DPL>
__global__ void __launch_bounds__(TM_WARPS * 32) time_mix_scan_kernel(const b200_time_mix_args a) {
    constexpr int CHUNK = DPL <= 4 ? 16 : 8, DP = 32 * DPL, NT = TM_WARPS * 32;
    __shared__ float sr[CHUNK * DP], sk[CHUNK * DP], sw[CHUNK * DP], sv[CHUNK * TM_COLS];
    const int h = blockIdx.y, s = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const int D = a.dim;
    const int first = a.seq_info[s], count = a.seq_info[a.n_seq + s], slot = a.seq_info[2 * a.n_seq + s], fresh = a.seq_info[3 * a.n_seq + s];
    if (count <= 0) return;
    const int cb = blockIdx.x * TM_COLS, col0 = cb + warp * TM_CW;
    float *Sp = a.state + (int64_t)slot * a.slot_stride + ((int64_t)h * D + col0) * D;
    float S[TM_CW][DPL], u[DPL];
#pragma unroll
    for (int i = 0; i < DPL; i++) {
        const int d = lane + 32 * i;
        u[i] = d < D ? a.u[h * D + d] : 0.f;
#pragma unroll
        for (int c = 0; c < TM_CW; c++) S[c][i] = (!fresh && d < D && col0 + c < D) ? Sp[(int64_t)c * D + d] : 0.f;
    }
    constexpr int NQ = CHUNK * DP / NT, NV = CHUNK * TM_COLS / NT;
    float pr[NQ], pk[NQ], pz[NQ], pv[NV];
    auto fetch = [&](int t0) {
        const int nt = min(CHUNK, count - t0);
#pragma unroll
        for (int j = 0; j < NQ; j++) {
            const int idx = tid + j * NT, tt = idx / DP, d = idx - tt * DP;
            const bool ok = tt < nt && d < D;
            const int64_t tok = first + t0 + tt;
            pr[j] = ok ? a.r[tok * a.r_stride + (int64_t)h * D + d] : 0.f;
            pk[j] = ok ? a.k[tok * a.k_stride + (int64_t)h * D + d] : 0.f;
            pz[j] = ok ? a.z[tok * a.z_stride + (int64_t)h * D + d] + a.w0[h * D + d] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < NV; j++) {
            const int idx = tid + j * NT, tt = idx / TM_COLS, c = idx - tt * TM_COLS;
            pv[j] = (tt < nt && cb + c < D) ? a.v[(int64_t)(first + t0 + tt) * a.v_stride + (int64_t)h * D + cb + c] : 0.f;
        }
    };
    fetch(0);
    for (int t0 = 0; t0 < count; t0 += CHUNK) {
        const int nt = min(CHUNK, count - t0);
        __syncthreads();  // the previous chunk has been read
#pragma unroll
        for (int j = 0; j < NQ; j++) { sr[tid + j * NT] = pr[j]; sk[tid + j * NT] = pk[j]; sw[tid + j * NT] = expf(-expf(pz[j])); }
#pragma unroll
        for (int j = 0; j < NV; j++) sv[tid + j * NT] = pv[j];
        __syncthreads();
        if (t0 + CHUNK < count) fetch(t0 + CHUNK);
        for (int tt0 = 0; tt0 < nt; tt0 += TM_RG) {
            float part[TM_RG * TM_CW];
#pragma unroll
            for (int g = 0; g < TM_RG; g++) {
                const int tt = tt0 + g;
                if (tt < nt) {  // warp-uniform
                    float rv[DPL], kv[DPL], wv[DPL], bonus = 0.f;
#pragma unroll
                    for (int i = 0; i < DPL; i++) {
                        const int d = tt * DP + lane + 32 * i;
                        rv[i] = sr[d]; kv[i] = sk[d]; wv[i] = sw[d];
                        bonus += rv[i] * (u[i] * kv[i]);
                    }
#pragma unroll
                    for (int c = 0; c < TM_CW; c++) {
                        const float vc = sv[tt * TM_COLS + warp * TM_CW + c];
                        float acc = bonus * vc;
#pragma unroll
                        for (int i = 0; i < DPL; i++) { acc += S[c][i] * rv[i]; S[c][i] = wv[i] * S[c][i] + kv[i] * vc; }
                        part[g * TM_CW + c] = acc;
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < TM_CW; c++) part[g * TM_CW + c] = 0.f;
                }
            }
#pragma unroll
            for (int off = 16, n = 32; off >= 1; off >>= 1, n >>= 1) {
                const bool upper = (lane & off) != 0;
#pragma unroll
                for (int i = 0; i < n / 2; i++) {
                    const float send = upper ? part[i] : part[i + n / 2], keep = upper ? part[i + n / 2] : part[i];
                    part[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
            }
            const int tt = tt0 + (lane >> 2), c = lane & 3;  // TM_CW == 4
            if (tt < nt && col0 + c < D) a.dst[(int64_t)(first + t0 + tt) * a.dst_stride + (int64_t)h * D + col0 + c] = part[0];
        }
    }
#pragma unroll
    for (int i = 0; i < DPL; i++) {
        const int d = lane + 32 * i;
#pragma unroll
        for (int c = 0; c < TM_CW; c++) if (d < D && col0 + c < D) Sp[(int64_t)c * D + d] = S[c][i];
    }
}

template <int DPL>
static int launch_time_mix(const b200_time_mix_args *a, cudaStream_t st) {
    const dim3 grid((unsigned)((a->dim + TM_COLS - 1) / TM_COLS), (unsigned)a->heads, (unsigned)a->n_seq);
    time_mix_scan_kernel<DPL><<<grid, TM_WARPS * 32, 0, st>>>(*a);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

}  // namespace b200

using namespace b200;

extern "C" int b200_op_token_shift(const b200_token_shift_args *a, b200_stream_t stream) {
    OPX_REQUIRE(a && a->h && a->mu && a->seq_info && a->prev && a->dst, B200_ERR_INVALID, "b200_op_token_shift: NULL argument");
    OPX_REQUIRE(a->width > 0 && a->n_mix > 0 && a->n_seq >= 0 && a->n_seq <= 65535 && a->n_tokens >= 0 && a->n_tokens <= 65535 * TS_TOK && a->slot_stride >= a->width, B200_ERR_INVALID,
                "b200_op_token_shift: bad sizes");
    if (a->n_seq == 0 || a->n_tokens == 0) return B200_OK;
    const dim3 grid((unsigned)((a->width + 127) / 128), (unsigned)((a->n_tokens + TS_TOK - 1) / TS_TOK), (unsigned)a->n_seq);
    token_shift_kernel<<<grid, 128, 0, (cudaStream_t)stream>>>(*a);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}

extern "C" int b200_op_time_mix_scan(const b200_time_mix_args *a, b200_stream_t stream) {
    OPX_REQUIRE(a && a->r && a->k && a->v && a->z && a->w0 && a->u && a->seq_info && a->state && a->dst, B200_ERR_INVALID, "b200_op_time_mix_scan: NULL argument");
    OPX_REQUIRE(a->heads > 0 && a->heads <= 65535 && a->dim > 0 && a->dim <= 256 && a->n_seq >= 0 && a->n_seq <= 65535 && a->slot_stride >= (int64_t)a->heads * a->dim * a->dim,
                B200_ERR_UNSUPPORTED, "b200_op_time_mix_scan: dim up to 256");
    if (a->n_seq == 0) return B200_OK;
    const cudaStream_t st = (cudaStream_t)stream;
    const int dpl = (a->dim + 31) / 32;
    if (dpl <= 1) return launch_time_mix<1>(a, st);
    if (dpl <= 2) return launch_time_mix<2>(a, st);
    if (dpl <= 4) return launch_time_mix<4>(a, st);
    return launch_time_mix<8>(a, st);
}

extern "C" int b200_op_short_conv(const b200_short_conv_args *a, b200_stream_t stream) {
    OPX_REQUIRE(a && a->x && a->w && a->seq_info && a->dst && (a->tail || a->taps <= 1), B200_ERR_INVALID, "b200_op_short_conv: NULL argument");
    OPX_REQUIRE(a->channels > 0 && a->taps >= 1 && a->taps <= SC_MAX_TAPS && a->n_seq >= 0 && a->n_seq <= 65535 && a->n_tokens >= 0 &&
                (a->taps <= 1 || a->slot_stride >= (int64_t)(a->taps - 1) * a->channels), B200_ERR_UNSUPPORTED, "b200_op_short_conv: at most %d taps", SC_MAX_TAPS);
    OPX_REQUIRE(a->x != a->dst, B200_ERR_INVALID, "b200_op_short_conv: not in place");
    if (a->n_seq == 0 || a->n_tokens == 0) return B200_OK;
    // (the general form reads every input where it is used: one channel a thread)
    const int64_t ctas = (int64_t)((a->channels + 127) / 128) * ((a->n_tokens + SC_TOK - 1) / SC_TOK);
    const bool two = a->taps <= 8 && ctas >= 8 * (int64_t)sm_count() && a->n_tokens >= 8 * SC_TOK * (int64_t)a->n_seq && ((a->channels | a->x_stride | a->dst_stride) & 1) == 0 && (((uintptr_t)a->x | (uintptr_t)a->dst) & 7) == 0;
    const int each = two ? 256 : 128;
    const dim3 grid((unsigned)((a->channels + each - 1) / each), (unsigned)((a->n_tokens + SC_TOK - 1) / SC_TOK), (unsigned)a->n_seq);
    OPX_REQUIRE(grid.y <= 65535, B200_ERR_UNSUPPORTED, "b200_op_short_conv: at most %d tokens in a batch", 65535 * SC_TOK);
    B200_CUDA_TRY(launch_chained(a->taps <= 4 ? (two ? short_conv_kernel<4, 2> : short_conv_kernel<4, 1>) : a->taps <= 8 ? (two ? short_conv_kernel<8, 2> : short_conv_kernel<8, 1>)
                                                                                                          : short_conv_kernel<0, 1>, grid, 128, 0, (cudaStream_t)stream, *a));
    return B200_OK;
}

extern "C" int b200_op_delta_rule_scan(const b200_delta_rule_args *a, b200_stream_t stream) {
    OPX_REQUIRE(a && a->q && a->k && a->v && a->a && a->b && a->a_log && a->seq_info && a->state && a->dst, B200_ERR_INVALID, "b200_op_delta_rule_scan: NULL argument");
    OPX_REQUIRE(a->heads > 0 && a->heads <= 65535 && a->kv_heads > 0 && a->heads % a->kv_heads == 0 && a->dim > 0 && a->dim <= 256 && a->vdim > 0 && a->n_seq >= 0 &&
                a->n_seq <= 65535 && a->slot_stride >= (int64_t)a->heads * a->dim * a->vdim, B200_ERR_UNSUPPORTED, "b200_op_delta_rule_scan: dim up to 256");
    if (a->n_seq == 0) return B200_OK;
    const cudaStream_t st = (cudaStream_t)stream;
    const int dq = (a->dim + 31) / 32;
    if (dq <= 1) return launch_delta_rule<1>(a, st);
    if (dq <= 2) return launch_delta_rule<2>(a, st);
    if (dq <= 4) return launch_delta_rule<4>(a, st);
    return launch_delta_rule<8>(a, st);
}

extern "C" int b200_op_mingru_scan(const b200_mingru_args *a, b200_stream_t stream) {
    OPX_REQUIRE(a && a->z && a->x && a->seq_info && a->state && a->dst, B200_ERR_INVALID, "b200_op_mingru_scan: NULL argument");
    OPX_REQUIRE(a->width > 0 && a->n_seq >= 0 && a->n_seq <= 65535 && a->slot_stride >= a->width, B200_ERR_INVALID, "b200_op_mingru_scan: bad sizes");
    if (a->n_seq == 0) return B200_OK;
    const dim3 grid((unsigned)((a->width + 31) / 32), (unsigned)a->n_seq);
    // stretches per CTA: as many as the longest sequence of the batch can fill (a sequence has at most n_tokens tokens)
    int segs = (a->n_tokens + MG_TPT - 1) / MG_TPT;
    segs = a->n_tokens <= 0 ? MG_SEG_MAX : segs < 1 ? 1 : segs > MG_SEG_MAX ? MG_SEG_MAX : segs;
    mingru_scan_kernel<<<grid, dim3(32, (unsigned)segs), 0, (cudaStream_t)stream>>>(*a);
    B200_CUDA_TRY(cudaGetLastError());
    return B200_OK;
}
