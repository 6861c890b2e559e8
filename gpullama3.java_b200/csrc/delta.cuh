// delta.cuh -- device kernels of the two mixers of pre-norm layered plans (B200_BLOCK_PRENORM).  First user: Lerosun.
//
//   * k_rope_mix_prep   windowed attention with rotated, head-mixed scores: projection biases, value rows = the keys BEFORE the
//                       rotation (or a value projection of their own), table-driven rotation of the leading entries of every
//                       query / key head, key / value rows into the window ring, and the head mixing FOLDED INTO THE QUERY:
//                           e'_h(i, j) = sum_m T[h][m] t_m <q_i^m, k_j^g(m)> = < q'_i^h , [k_j^0 | k_j^1 | ...] >,
//                           q'_i^h = [ sum_{m in group 0} T[h][m] t_m q_i^m | sum_{m in group 1} ... | ... ]
//                       so every head attends with ONE query of (key heads x key size) entries over the whole key row and the
//                       attention kernels of layered.cuh need no mixing pass (WindowAttn::k_heads = 1).  Without a mixing
//                       matrix the query is only scaled by its head's temperature;
//   * k_delta_prep      gated delta rule, everything in front of the recurrence: causal convolution of the q | k | v channels over
//                       a ring of earlier inputs, SiLU, unit vectors per q / k head, beta = sigmoid, decay = exp(-exp(A) softplus);
//   * k_delta_rule_reg  the recurrence S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q with the state in registers: eight
//                       lanes share a state column, the rows of a chunk run in sequence, columns in parallel over warps and CTAs;
//   * k_delta_rule_blocks (+ k_delta_coef)   the same, four tokens per step of the chain: prefill chunks;
//   * k_delta_rule      the same for key sizes above 128: one thread per state column, the state tile in shared memory;
//   * k_head_norm_gate  per-head RMS norm of the read-out (optionally divided by a denominator per head first), weight, SiLU or sigmoid gate.
// Rotation, scores, decays, gates, unit norms and the state are FP32 in both compute modes; fmaf is explicit because the
// translation unit is compiled with -fmad=false.
#pragma once
#include "latent.cuh"

namespace ly {

struct RopeMixArgs {
    int heads, kv_heads, dk, dv; // query heads, key/value heads, key size, value size (value_from_key: dv == dk)
    int rope_dims, rope_layout;  // the first rope_dims entries of every head turn (0: none)
    const float *cs;             // [position][rope_dims / 2][2] = (cos, sin)
    const float *temp;           // [heads] (nullable)
    const float *talk;           // [heads][heads] (nullable): mixing matrix T
    int value_from_key;
    int ring;                    // position j lives in slot j % ring
};

// grid (rows, ceil(heads / hpc) + 1), 128 threads (hpc = query heads per CTA: ROPE_MIX_HEADS for a chunk of rows, 1 for the decode step's single row); dynamic shared memory: max(heads, kv_heads) * dk floats.  P row:
// [q: heads*dk | k: kv_heads*dk | v: kv_heads*dv (absent with value_from_key) | ...].  A query-side CTA biases and rotates ALL query heads
// of the row into shared memory (every mixed query needs them all; the row in P stays as projected) and writes the queries of its
// hpc heads: heads * (talk ? kv_heads * dk : dk) entries per Q row (ldq).  The last CTA of a row owns the key side: bias,
// value row = unrotated key (or the value projection), rotation, key row.
#define ROPE_MIX_THREADS 128
#define ROPE_MIX_HEADS 4
__global__ void __launch_bounds__(ROPE_MIX_THREADS) k_rope_mix_prep(const float *__restrict__ P, int ldp, RopeMixArgs a, const float *__restrict__ bias, float *__restrict__ Q, int ldq,
                                                                    float *__restrict__ kc, float *__restrict__ vc, bf16 *__restrict__ kc16, bf16 *__restrict__ vc16,
                                                                    const StepState *__restrict__ st, int hpc) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float xs[];
    const int r = blockIdx.x, tid = threadIdx.x;
    const int qd = a.heads * a.dk, kd = a.kv_heads * a.dk, vd = a.kv_heads * a.dv;
    const float *p = P + (size_t)r * ldp;
    const int pos = st->pos + r, slot = pos % a.ring, half = a.rope_dims / 2;
    const float *cs = a.cs + (size_t)pos * half * 2;
    const bool key_side = blockIdx.y == gridDim.y - 1;
    // this CTA's vectors, biased: all query heads, or all key heads
    const int off = key_side ? qd : 0, len = key_side ? kd : qd, nh = key_side ? a.kv_heads : a.heads;
    for (int i = tid; i < len; i += ROPE_MIX_THREADS) xs[i] = p[off + i] + (bias ? bias[off + i] : 0.0f);
    __syncthreads();
    if (key_side) {
        for (int i = tid; i < vd; i += ROPE_MIX_THREADS) {
            const float v = a.value_from_key ? xs[i] : p[qd + kd + i] + (bias ? bias[qd + kd + i] : 0.0f);
            vc[(size_t)slot * vd + i] = v;
            if (vc16) vc16[(size_t)slot * vd + i] = __float2bfloat16_rn(v);
        }
        __syncthreads(); // the values above are the unrotated keys
    }
    for (int e = tid; e < nh * half; e += ROPE_MIX_THREADS) {
        const int hd = e / half, i = e % half;
        int u, w;
        rope_pair_index(i, a.rope_dims, a.rope_layout, u, w);
        float *x = xs + (size_t)hd * a.dk;
        const float co = cs[2 * i], si = cs[2 * i + 1];
        const float xu = x[u], xw = x[w];
        x[u] = fmaf(xu, co, -(xw * si));
        x[w] = fmaf(xw, co, xu * si);
    }
    __syncthreads();
    if (key_side) {
        for (int i = tid; i < kd; i += ROPE_MIX_THREADS) {
            kc[(size_t)slot * kd + i] = xs[i];
            if (kc16) kc16[(size_t)slot * kd + i] = __float2bfloat16_rn(xs[i]);
        }
        return;
    }
    const int h0 = blockIdx.y * hpc, h1 = h0 + hpc < a.heads ? h0 + hpc : a.heads;
    if (a.talk) {
        const int group = a.heads / a.kv_heads;
        float *qo = Q + (size_t)r * ldq + (size_t)h0 * kd;
        for (int e = tid; e < (h1 - h0) * kd; e += ROPE_MIX_THREADS) {
            const int h = h0 + e / kd, c = e % kd, kv = c / a.dk, d = c % a.dk;
            float s = 0.0f;
            for (int m = kv * group; m < (kv + 1) * group; m++) s = fmaf(a.talk[h * a.heads + m] * (a.temp ? a.temp[m] : 1.0f), xs[(size_t)m * a.dk + d], s);
            qo[e] = s;
        }
    } else {
        float *qo = Q + (size_t)r * ldq;
        for (int e = h0 * a.dk + tid; e < h1 * a.dk; e += ROPE_MIX_THREADS) qo[e] = a.temp ? xs[e] * a.temp[e / a.dk] : xs[e];
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Gated delta rule.
// ---------------------------------------------------------------------------------------------------------------------
struct DeltaArgs {
    int heads, kv_heads, dk, dv; // value heads, query/key heads, key size, value size
    int taps;                    // convolution taps; tap taps - 1 belongs to the current token
    int cring;                   // slots of the ring of convolution inputs: position j in slot j % cring (cring >= taps - 1 + rows of a step)
    const float *conv_w;         // [2 * kv_heads * dk + heads * dv][taps]: q | k | v channels
    const float *a_log, *dt_bias; // [heads]
    float unit_eps;              // inside the root of the unit-vector normalisation
};
// Row layout of the fused projection: [q: kv_heads*dk | k: kv_heads*dk | v: heads*dv | b: heads | a: heads | g: heads*dv]
// Row layout of the prepared buffer D (ldd): [q unit / sqrt(dk) | k unit | v | beta: heads | decay: heads]
__host__ __device__ inline int delta_channels(const DeltaArgs &a) { return 2 * a.kv_heads * a.dk + a.heads * a.dv; }

// grid (rows, 2 * kv_heads + heads + 1), 128 threads; dynamic shared memory: max(dk, dv) floats.  CTA (r, u) owns one unit of the row:
// a query head, a key head (convolution, SiLU, unit vector), a value head (convolution, SiLU), or -- the last unit -- beta and decay
// of all heads.  A row at position p reads the inputs of positions p - taps + 1 .. p: from the rows of this launch where they belong
// to it, else from the ring (written by earlier launches; positions before the start of the sequence count as zero).  Every unit
// leaves its own input channels in the ring.
#define DELTA_PREP_THREADS 128
__global__ void __launch_bounds__(DELTA_PREP_THREADS) k_delta_prep(const float *__restrict__ P, int ldp, DeltaArgs a, float *__restrict__ cstate, float *__restrict__ D, int ldd,
                                                                   const StepState *__restrict__ st) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float row[];
    __shared__ float red[32];
    const int r = blockIdx.x, u = blockIdx.y, tid = threadIdx.x;
    const int C = delta_channels(a), qk = a.kv_heads * a.dk;
    const int pos = st->pos + r;
    const float *p = P + (size_t)r * ldp;
    float *d = D + (size_t)r * ldd;
    if (u == 2 * a.kv_heads + a.heads) {
        for (int h = tid; h < a.heads; h += DELTA_PREP_THREADS) {
            d[C + h] = 1.0f / (1.0f + expf(-p[C + h]));
            const float z = p[C + a.heads + h] + a.dt_bias[h];
            const float sp = fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z)));
            d[C + a.heads + h] = expf(-expf(a.a_log[h]) * sp);
        }
        return;
    }
    const bool unit_vec = u < 2 * a.kv_heads;
    const int c0 = unit_vec ? u * a.dk : 2 * qk + (u - 2 * a.kv_heads) * a.dv, len = unit_vec ? a.dk : a.dv;
    float ss = 0.0f;
    for (int i = tid; i < len; i += DELTA_PREP_THREADS) {
        const int c = c0 + i;
        float acc = 0.0f;
        for (int m = 0; m < a.taps; m++) {
            const int back = a.taps - 1 - m;
            if (pos - back < 0) continue;
            const float x = back <= r ? P[(size_t)(r - back) * ldp + c] : cstate[(size_t)((pos - back) % a.cring) * C + c];
            acc = fmaf(a.conv_w[(size_t)c * a.taps + m], x, acc);
        }
        cstate[(size_t)(pos % a.cring) * C + c] = p[c];
        const float y = acc / (1.0f + expf(-acc));
        if (unit_vec) { row[i] = y; ss = fmaf(y, y, ss); }
        else d[c] = y;
    }
    if (!unit_vec) return;
    ss = block_sum(ss, red);
    float inv = 1.0f / sqrtf(ss + a.unit_eps);
    if (u < a.kv_heads) inv *= 1.0f / sqrtf((float)a.dk);
    for (int i = tid; i < len; i += DELTA_PREP_THREADS) d[c0 + i] = row[i] * inv;
}

// grid (heads, column tiles), DELTA_COLS threads: thread j owns column j of the head's state S [dk][dv]; the tile S[:, cols] stays
// in shared memory over the n rows of the launch.  Dynamic shared memory: (dk * DELTA_COLS + 4 * dk) floats.  pos == 0 starts
// from a zero state whatever the buffer holds (a new sequence needs no clearing).
#define DELTA_COLS 64
__host__ __device__ inline size_t delta_rule_smem_floats(int dk) { return (size_t)dk * DELTA_COLS + 4 * (size_t)dk; }

__global__ void __launch_bounds__(DELTA_COLS) k_delta_rule(const float *__restrict__ D, int ldd, DeltaArgs a, float *__restrict__ S, int n, float *__restrict__ O, int ldo,
                                                           const StepState *__restrict__ st) {
    pdl_launch_dependents();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    const int h = blockIdx.x, j0 = blockIdx.y * DELTA_COLS, tid = threadIdx.x, j = j0 + tid;
    const int dk = a.dk, dv = a.dv, g = h / (a.heads / a.kv_heads), C = delta_channels(a);
    float *Ss = sm, *kq = sm + (size_t)dk * DELTA_COLS; // kq: two buffers of [k (dk) | q (dk)]
    float *Sg = S + (size_t)h * dk * dv;
    const bool live = j < dv;
    const bool fresh = st->pos == 0;
    for (int i = 0; i < dk; i++) Ss[i * DELTA_COLS + tid] = (live && !fresh) ? Sg[(size_t)i * dv + j] : 0.0f;
    auto stage = [&](int t, int buf) {
        const float *d = D + (size_t)t * ldd;
        float *dst = kq + (size_t)buf * 2 * dk;
        for (int i = tid; i < dk; i += DELTA_COLS) {
            dst[i] = d[(size_t)(a.kv_heads + g) * dk + i];
            dst[dk + i] = d[(size_t)g * dk + i];
        }
    };
    stage(0, 0);
    __syncthreads();
    for (int t = 0; t < n; t++) {
        const int buf = t & 1;
        if (t + 1 < n) stage(t + 1, buf ^ 1); // the other buffer was last read in iteration t - 1, before its closing barrier
        const float *ks = kq + (size_t)buf * 2 * dk, *qs = ks + dk;
        const float *d = D + (size_t)t * ldd;
        const float beta = d[C + h], decay = d[C + a.heads + h];
        const float vj = live ? d[2 * a.kv_heads * dk + (size_t)h * dv + j] : 0.0f;
        float rd = 0.0f;
        for (int i = 0; i < dk; i++) rd = fmaf(Ss[i * DELTA_COLS + tid], ks[i], rd);
        const float u = beta * (vj - decay * rd);
        float o = 0.0f;
        for (int i = 0; i < dk; i++) {
            const float s = fmaf(ks[i], u, decay * Ss[i * DELTA_COLS + tid]);
            Ss[i * DELTA_COLS + tid] = s;
            o = fmaf(s, qs[i], o);
        }
        if (live) O[(size_t)t * ldo + (size_t)h * dv + j] = o;
        __syncthreads();
    }
    if (live)
        for (int i = 0; i < dk; i++) Sg[(size_t)i * dv + j] = Ss[i * DELTA_COLS + tid];
}

// The same recurrence with the state in REGISTERS (key sizes up to 16 * R, R = 1, 2, 4 or 8): grid (heads, column tiles of DR_COLS),
// DR_THREADS threads.  A column of S is shared by DR_SLICES = 16 neighbouring lanes, lane s holding rows s * R .. s * R + R - 1; the two
// products S^T k and S^T q are R multiply-adds per lane (four partial sums) and a four-step shuffle.  Columns are independent and a
// warp owns two of them completely, so the only block-wide step is staging DR_TB tokens of k, q, v, beta and decay in shared memory
// at a time (cp.async, double buffered: the next block lands while this one is computed; slices of eight padded by four floats: the
// 128-bit reads of a quarter warp fall on distinct banks) and writing their read-outs back coalesced.  Within a token the chain
// S^T k -> shuffles -> u -> S is what the next token waits for; the read-out's shuffles ride one token behind, interleaved with it.
// Sixteen lanes per column rather than eight: the per-token chain gets shorter and every scheduler has two warps to alternate
// between.  The state buffer is private to this kernel: [head][tile][R][thread].
#define DR_COLS 16
#define DR_SLICES 16
#define DR_THREADS (DR_COLS * DR_SLICES)
#define DR_TB 8
__host__ __device__ inline int delta_reg_rows(int dk) { return dk <= 16 ? 1 : dk <= 32 ? 2 : dk <= 64 ? 4 : dk <= 128 ? 8 : 0; } // 0: the shared-memory kernel
__host__ __device__ inline size_t delta_state_floats(int heads, int dk, int dv) {
    const int R = delta_reg_rows(dk);
    return R ? (size_t)heads * ((dv + DR_COLS - 1) / DR_COLS) * R * DR_THREADS : (size_t)heads * dk * dv;
}

__device__ __forceinline__ void cp_async4(void *dst, const void *src, bool valid) { // 4 bytes, zero-filled when !valid
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int nbytes = valid ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(nbytes) : "memory");
}

template <int R>
__global__ void __launch_bounds__(DR_THREADS) k_delta_rule_reg(const float *__restrict__ D, int ldd, DeltaArgs a, float *__restrict__ S, int n, float *__restrict__ O, int ldo,
                                                               const StepState *__restrict__ st) {
    pdl_launch_dependents();
    pdl_wait();
    constexpr int RP = R > 4 ? R + 4 : R, KR = DR_SLICES * RP; // floats per slice / per token in shared memory
    __shared__ __align__(16) float ks[2][DR_TB][KR], qs[2][DR_TB][KR];
    __shared__ float vs[2][DR_TB][DR_COLS], bd[2][DR_TB][2], os[DR_TB][DR_COLS];
    const int h = blockIdx.x, tile = blockIdx.y, j0 = tile * DR_COLS, tid = threadIdx.x, lane = tid & 31;
    const int c = (tid >> 5) * (32 / DR_SLICES) + lane / DR_SLICES, s = lane % DR_SLICES;
    const int dk = a.dk, dv = a.dv, g = h / (a.heads / a.kv_heads), C = delta_channels(a);
    float *Sg = S + ((size_t)h * gridDim.y + tile) * R * DR_THREADS + tid;
    float Sr[R];
    const bool fresh = st->pos == 0;
    // the tokens of block t0 travel global -> shared asynchronously while the previous block is computed
    auto stage = [&](int buf, int t0) {
        const int nb = n - t0 < DR_TB ? n - t0 : DR_TB;
        for (int e = tid; e < nb * DR_SLICES * R; e += DR_THREADS) {
            const int t = e / (DR_SLICES * R), i = e % (DR_SLICES * R); // key row i belongs to slice i / R
            const float *d = D + (size_t)(t0 + t) * ldd;
            const int at = (i / R) * RP + i % R;
            const bool ok = i < dk;
            cp_async4(&ks[buf][t][at], ok ? d + (size_t)(a.kv_heads + g) * dk + i : D, ok);
            cp_async4(&qs[buf][t][at], ok ? d + (size_t)g * dk + i : D, ok);
        }
        for (int e = tid; e < nb * DR_COLS; e += DR_THREADS) {
            const int t = e / DR_COLS, cc = e % DR_COLS;
            const bool ok = j0 + cc < dv;
            cp_async4(&vs[buf][t][cc], ok ? D + (size_t)(t0 + t) * ldd + 2 * a.kv_heads * dk + (size_t)h * dv + j0 + cc : D, ok);
        }
        if (tid < nb * 2) cp_async4(&bd[buf][tid >> 1][tid & 1], D + (size_t)(t0 + (tid >> 1)) * ldd + C + (tid & 1) * a.heads + h, true);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    stage(0, 0);
#pragma unroll
    for (int i = 0; i < R; i++) Sr[i] = fresh ? 0.0f : Sg[(size_t)i * DR_THREADS];
    int buf = 0;
    for (int t0 = 0; t0 < n; t0 += DR_TB, buf ^= 1) {
        const int nb = n - t0 < DR_TB ? n - t0 : DR_TB;
        if (t0 + DR_TB < n) {
            stage(buf ^ 1, t0 + DR_TB); // that buffer was last read before the barrier that ended the previous iteration
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        auto load = [&](int t, float (&kr)[R], float (&qr)[R]) {
            if (R >= 4) {
#pragma unroll
                for (int i = 0; i < R; i += 4) {
                    *reinterpret_cast<float4 *>(&kr[i]) = *reinterpret_cast<const float4 *>(&ks[buf][t][s * RP + i]);
                    *reinterpret_cast<float4 *>(&qr[i]) = *reinterpret_cast<const float4 *>(&qs[buf][t][s * RP + i]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < R; i++) { kr[i] = ks[buf][t][s * RP + i]; qr[i] = qs[buf][t][s * RP + i]; }
            }
        };
        float ka[R], qa[R], kb[R], qb[R]; // two register sets: the next token's k and q load while the current one's shuffles run
        load(0, ka, qa);
        float op = 0.0f; // read-out of the previous token, summed over the slices one shuffle step behind the current token's S^T k
        auto token = [&](int t, const float (&kr)[R], const float (&qr)[R], float (&kn)[R], float (&qn)[R]) {
            const float beta = bd[buf][t][0], decay = bd[buf][t][1], v = vs[buf][t][c];
            float r4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < R; i++) r4[i & 3] = fmaf(Sr[i], kr[i], r4[i & 3]);
            if (t + 1 < nb) load(t + 1, kn, qn); // in flight during the shuffles below
            float rd = (r4[0] + r4[1]) + (r4[2] + r4[3]);
#pragma unroll
            for (int m = 1; m < DR_SLICES; m <<= 1) {
                const float x = __shfl_xor_sync(0xffffffffu, rd, m), y = __shfl_xor_sync(0xffffffffu, op, m);
                rd += x;
                op += y;
            }
            if (s == 0 && t > 0) os[t - 1][c] = op;
            const float u = beta * (v - decay * rd);
            float o4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < R; i++) {
                Sr[i] = fmaf(kr[i], u, decay * Sr[i]);
                o4[i & 3] = fmaf(Sr[i], qr[i], o4[i & 3]);
            }
            op = (o4[0] + o4[1]) + (o4[2] + o4[3]);
        };
        for (int t = 0; t < nb; t += 2) {
            token(t, ka, qa, kb, qb);
            if (t + 1 < nb) token(t + 1, kb, qb, ka, qa);
        }
#pragma unroll
        for (int m = 1; m < DR_SLICES; m <<= 1) op += __shfl_xor_sync(0xffffffffu, op, m);
        if (s == 0) os[nb - 1][c] = op;
        __syncthreads();
        for (int e = tid; e < nb * DR_COLS; e += DR_THREADS) {
            const int t = e / DR_COLS, cc = e % DR_COLS;
            if (j0 + cc < dv) O[(size_t)(t0 + t) * ldo + (size_t)h * dv + j0 + cc] = os[t][cc];
        }
        // os is rewritten only after the barrier that follows the next block's wait
    }
#pragma unroll
    for (int i = 0; i < R; i++) Sg[(size_t)i * DR_THREADS] = Sr[i];
}

// ---- four tokens at a time -------------------------------------------------------------------------------------------------------------
// With S the state before four tokens, G_i the product of their first i decays and g(j, i) = G_i / G_j (formed as products, never divided), the recurrence is
//     u_i = beta_i v_i - beta_i G_i <S, k_i> - sum_{j < i} beta_i g(j, i) <k_j, k_i> u_j          (each per state column)
//     o_i = G_i <S, q_i> + sum_{j <= i} g(j, i) <k_j, q_i> u_j
//     S <- G_4 S + sum_j g(j, 4) k_j u_j
// so the eight products with S do not wait for one another and a column pays for ONE reduction over its lanes and one short triangular solve per four
// tokens: the chain per token drops from a shuffle tree to a quarter of one.  What the sums over j need (products of keys and queries, decays) is the same for all
// columns of a head: k_delta_coef computes it for the whole launch beforehand, 40 floats per (four tokens, head).  All of it is FP32.
// 16 heads of 128 x 128, 512 tokens: 130 us token by token (k_delta_rule_reg: 418 cycles per token), 101 us here and 7.6 us for the coefficients.
#define DC_FLOATS 40 // [0, 4) beta_i G_i | [4, 8) beta_i | [8, 14) beta_i g(j, i) <k_j, k_i> of (j, i) = 12 13 23 14 24 34 | [16, 32) g(j, i) <k_j, q_i> at 16 + 4 i + j | [32, 36) G_i | [36, 40) g(j, 4)
__host__ __device__ inline size_t delta_coef_floats(int rows, int heads) { return (size_t)((rows + 3) / 4) * heads * DC_FLOATS; }

// grid (ceil(n / 4), ceil(heads / 4)), 128 threads: a warp per (four tokens, head).  Tokens behind the last one count as beta = 0, decay = 1.
__global__ void __launch_bounds__(128) k_delta_coef(const float *__restrict__ D, int ldd, DeltaArgs a, int n, float *__restrict__ coef) {
    pdl_launch_dependents();
    pdl_wait();
    const int b = blockIdx.x, lane = threadIdx.x & 31, h = blockIdx.y * 4 + (threadIdx.x >> 5);
    if (h >= a.heads) return;
    const int dk = a.dk, g = h / (a.heads / a.kv_heads), C = delta_channels(a), t0 = 4 * b;
    float kk[6], kq[10]; // (j, i): 12 13 23 14 24 34 | 11 12 22 13 23 33 14 24 34 44
#pragma unroll
    for (int e = 0; e < 6; e++) kk[e] = 0.0f;
#pragma unroll
    for (int e = 0; e < 10; e++) kq[e] = 0.0f;
    for (int e = lane; e < dk; e += 32) {
        float k[4], q[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const bool ok = t0 + i < n;
            const float *d = D + (size_t)(ok ? t0 + i : t0) * ldd;
            k[i] = ok ? d[(size_t)(a.kv_heads + g) * dk + e] : 0.0f;
            q[i] = ok ? d[(size_t)g * dk + e] : 0.0f;
        }
#pragma unroll
        for (int i = 0, x = 0, y = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j <= i; j++) {
                if (j < i) { kk[x] = fmaf(k[j], k[i], kk[x]); x++; }
                kq[y] = fmaf(k[j], q[i], kq[y]);
                y++;
            }
    }
#pragma unroll
    for (int e = 0; e < 6; e++) kk[e] = warp_sum(kk[e]);
#pragma unroll
    for (int e = 0; e < 10; e++) kq[e] = warp_sum(kq[e]);
    if (lane) return;
    float beta[4], dec[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const bool ok = t0 + i < n;
        const float *d = D + (size_t)(ok ? t0 + i : t0) * ldd + C;
        beta[i] = ok ? d[h] : 0.0f;
        dec[i] = ok ? d[a.heads + h] : 1.0f;
    }
    float *o = coef + ((size_t)b * a.heads + h) * DC_FLOATS;
    float G = 1.0f;
#pragma unroll
    for (int i = 0, x = 0, y = 0; i < 4; i++) {
        G *= dec[i];
        o[i] = beta[i] * G;
        o[4 + i] = beta[i];
        o[32 + i] = G;
        float gj[4]; // g(j, i)
        gj[i] = 1.0f;
#pragma unroll
        for (int j = i - 1; j >= 0; j--) gj[j] = gj[j + 1] * dec[j + 1];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (j < i) { o[8 + x] = beta[i] * gj[j] * kk[x]; x++; }
            o[16 + 4 * i + j] = j <= i ? gj[j] * kq[y] : 0.0f;
            if (j <= i) y++;
            if (i == 3) o[36 + j] = gj[j];
        }
    }
    o[14] = o[15] = 0.0f;
}

// The layout of the state is k_delta_rule_reg's (16 lanes a column); a lane serves columns c and c + 8, so that a loaded key or query entry is used for both
// (one column a lane, eight warps: 110 us instead of 101).  The sixteen products of a lane's slices are reduced over the 16 lanes by halving:
// fifteen shuffles leave one complete product in every lane, eight more hand <S, k_i> to all of them.  Bound by the latency of that chain: one warp per scheduler, so
// the keys and queries of the next four tokens are loaded before the solve of these.
#define DB_THREADS (DR_THREADS / 2)
template <int R>
__global__ void __launch_bounds__(DB_THREADS) k_delta_rule_blocks(const float *__restrict__ D, int ldd, DeltaArgs a, const float *__restrict__ coef, float *__restrict__ S, int n,
                                                                  float *__restrict__ O, int ldo, const StepState *__restrict__ st) {
    static_assert(DR_SLICES == 16 && DR_COLS == 16, "two columns a lane, sixteen products over sixteen lanes");
    constexpr int RP = R > 4 ? R + 4 : R, KR = DR_SLICES * RP;
    __shared__ __align__(16) float ks[3][DR_TB][KR], qs[3][DR_TB][KR], cf[3][DR_TB / 4][DC_FLOATS];
    __shared__ float vs[3][DR_TB][DR_COLS], os[2][DR_TB][DR_COLS];
    const int h = blockIdx.x, tile = blockIdx.y, j0 = tile * DR_COLS, tid = threadIdx.x, lane = tid & 31;
    const int c = tid / DR_SLICES, s = lane % DR_SLICES; // columns c and c + 8
    const int dk = a.dk, dv = a.dv, g = h / (a.heads / a.kv_heads);
    float *Sg = S + ((size_t)h * gridDim.y + tile) * R * DR_THREADS + tid;
    float S0[R], S1[R];
    pdl_launch_dependents();
    pdl_wait();
    const bool fresh = st->pos == 0;
    const bool wide = R >= 4 && dk % 4 == 0 && ldd % 4 == 0 && (reinterpret_cast<uintptr_t>(D) & 15) == 0; // rows of whole, aligned 16-byte pieces
    auto stage = [&](int i) { // tokens behind the last one are zero
        const int buf = i % 3, t0 = i * DR_TB;
        if (t0 >= n) return;
        if (wide) {
            for (int e = tid; e < DR_TB * DR_SLICES * R / 4; e += DB_THREADS) {
                const int t = e / (DR_SLICES * R / 4), i = e % (DR_SLICES * R / 4) * 4;
                const bool ok = i < dk && t0 + t < n;
                const float *d = D + (size_t)(ok ? t0 + t : 0) * ldd;
                const int at = (i / R) * RP + i % R;
                cp_async16(&ks[buf][t][at], ok ? d + (size_t)(a.kv_heads + g) * dk + i : D, ok);
                cp_async16(&qs[buf][t][at], ok ? d + (size_t)g * dk + i : D, ok);
            }
        } else
            for (int e = tid; e < DR_TB * DR_SLICES * R; e += DB_THREADS) {
                const int t = e / (DR_SLICES * R), i = e % (DR_SLICES * R);
                const bool ok = i < dk && t0 + t < n;
                const float *d = D + (size_t)(ok ? t0 + t : 0) * ldd;
                const int at = (i / R) * RP + i % R;
                cp_async4(&ks[buf][t][at], ok ? d + (size_t)(a.kv_heads + g) * dk + i : D, ok);
                cp_async4(&qs[buf][t][at], ok ? d + (size_t)g * dk + i : D, ok);
            }
        for (int e = tid; e < DR_TB * DR_COLS; e += DB_THREADS) {
            const int t = e / DR_COLS, cc = e % DR_COLS;
            const bool ok = j0 + cc < dv && t0 + t < n;
            cp_async4(&vs[buf][t][cc], ok ? D + (size_t)(t0 + t) * ldd + 2 * a.kv_heads * dk + (size_t)h * dv + j0 + cc : D, ok);
        }
        for (int e = tid; e < DR_TB / 4 * DC_FLOATS; e += DB_THREADS) {
            const int b = e / DC_FLOATS;
            const bool ok = t0 + 4 * b < n;
            cp_async4(&cf[buf][b][e % DC_FLOATS], ok ? coef + ((size_t)(t0 / 4 + b) * a.heads + h) * DC_FLOATS + e % DC_FLOATS : coef, ok);
        }
    };
    auto flush = [&](int i) { // the outputs of staged block i
        for (int e = tid; e < DR_TB * DR_COLS; e += DB_THREADS) {
            const int t = i * DR_TB + e / DR_COLS, cc = e % DR_COLS;
            if (t < n && j0 + cc < dv) O[(size_t)t * ldo + (size_t)h * dv + j0 + cc] = os[i & 1][e / DR_COLS][cc];
        }
    };
    stage(0);
    asm volatile("cp.async.commit_group;" ::: "memory");
    stage(1);
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
    for (int i = 0; i < R; i++) {
        S0[i] = fresh ? 0.0f : Sg[(size_t)i * DR_THREADS];
        S1[i] = fresh ? 0.0f : Sg[(size_t)i * DR_THREADS + DB_THREADS];
    }
    auto load = [&](const float *row, float (&x)[R]) {
        if (R >= 4) {
#pragma unroll
            for (int i = 0; i < R; i += 4) *reinterpret_cast<float4 *>(&x[i]) = *reinterpret_cast<const float4 *>(row + s * RP + i);
        } else {
#pragma unroll
            for (int i = 0; i < R; i++) x[i] = row[s * RP + i];
        }
    };
    const bool b3 = s & 8, b2 = s & 4, b1 = s & 2, b0 = s & 1;
    const int own = (s >> 1) & 3; // lanes 0 .. 7 end up with <S, k_own>, lanes 8 .. 15 with <S, q_own>; odd lanes of column c + 8
    const int blocks = (n + DR_TB - 1) / DR_TB;
    for (int it = 0; it < blocks; it++) { // one barrier per staged block: behind it block it has arrived everywhere and nobody reads block it - 1 any more
        const int t0 = it * DR_TB, buf = it % 3;
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        stage(it + 2);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (it > 0) flush(it - 1);
        float k[4][R], q[4][R];
#pragma unroll
        for (int i = 0; i < 4; i++) { load(ks[buf][i], k[i]); load(qs[buf][i], q[i]); }
#pragma unroll 1
        for (int b = 0; b < DR_TB / 4; b++) {
            if (t0 + 4 * b >= n) break;
            const float *w = cf[buf][b];
            float x[16]; // [column][key products 0 .. 3, query products 0 .. 3]
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float d0 = 0.0f, d1 = 0.0f, e0 = 0.0f, e1 = 0.0f, f0 = 0.0f, f1 = 0.0f, g0 = 0.0f, g1 = 0.0f;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (r & 1) { d1 = fmaf(S0[r], k[i][r], d1); e1 = fmaf(S0[r], q[i][r], e1); f1 = fmaf(S1[r], k[i][r], f1); g1 = fmaf(S1[r], q[i][r], g1); }
                    else { d0 = fmaf(S0[r], k[i][r], d0); e0 = fmaf(S0[r], q[i][r], e0); f0 = fmaf(S1[r], k[i][r], f0); g0 = fmaf(S1[r], q[i][r], g0); }
                }
                x[i] = d0 + d1; x[4 + i] = e0 + e1; x[8 + i] = f0 + f1; x[12 + i] = g0 + g1;
            }
            if (b + 1 < DR_TB / 4) // the queries are used up: the next four tokens' (zero behind the last one)
#pragma unroll
                for (int i = 0; i < 4; i++) load(qs[buf][4 * b + 4 + i], q[i]);
            float y[8], z[4], m2[2], m;
#pragma unroll
            for (int i = 0; i < 8; i++) { // (i >> 2: column) lanes with bit 3 keep the queries' products, the others the keys'
                const int at = (i >> 2) * 8 + (i & 3);
                const float keep = b3 ? x[at + 4] : x[at], send = b3 ? x[at] : x[at + 4];
                y[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) { // (i >> 1: column) bit 2: tokens 2, 3 or 0, 1
                const int at = (i >> 1) * 4 + (i & 1);
                const float keep = b2 ? y[at + 2] : y[at], send = b2 ? y[at] : y[at + 2];
                z[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
            }
#pragma unroll
            for (int i = 0; i < 2; i++) { // bit 1: the odd or the even one
                const float keep = b1 ? z[2 * i + 1] : z[2 * i], send = b1 ? z[2 * i] : z[2 * i + 1];
                m2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
            }
            m = (b0 ? m2[1] : m2[0]) + __shfl_xor_sync(0xffffffffu, b0 ? m2[0] : m2[1], 1); // bit 0: the column
            const int base = lane & ~(DR_SLICES - 1);
            const float4 A = *reinterpret_cast<const float4 *>(w), B = *reinterpret_cast<const float4 *>(w + 4), L = *reinterpret_cast<const float4 *>(w + 8), Lr = *reinterpret_cast<const float4 *>(w + 12);
            const float4 gl = *reinterpret_cast<const float4 *>(w + 36);
            const float4 M = *reinterpret_cast<const float4 *>(w + 16 + 4 * own);
            const float Gown = w[32 + own], G4 = w[35];
            float u[2][4];
#pragma unroll
            for (int cc = 0; cc < 2; cc++) {
                const float a0 = __shfl_sync(0xffffffffu, m, base + cc), a1 = __shfl_sync(0xffffffffu, m, base + 2 + cc), a2 = __shfl_sync(0xffffffffu, m, base + 4 + cc),
                            a3 = __shfl_sync(0xffffffffu, m, base + 6 + cc);
                const float *v = &vs[buf][4 * b][c + 8 * cc];
                const float u0 = fmaf(-A.x, a0, B.x * v[0]);
                const float r1 = fmaf(-A.y, a1, B.y * v[DR_COLS]), r2 = fmaf(-A.z, a2, B.z * v[2 * DR_COLS]), r3 = fmaf(-A.w, a3, B.w * v[3 * DR_COLS]);
                const float u1 = fmaf(-L.x, u0, r1);
                const float u2 = fmaf(-L.z, u1, fmaf(-L.y, u0, r2));
                u[cc][0] = u0; u[cc][1] = u1; u[cc][2] = u2;
                u[cc][3] = fmaf(-Lr.y, u2, fmaf(-Lr.x, u1, fmaf(-L.w, u0, r3)));
            }
            if (b3) { // (a later token's update stays out by selection, not by its zero factor: it may be infinite)
                float o = fmaf(M.x, b0 ? u[1][0] : u[0][0], Gown * m);
                if (own >= 1) o = fmaf(M.y, b0 ? u[1][1] : u[0][1], o);
                if (own >= 2) o = fmaf(M.z, b0 ? u[1][2] : u[0][2], o);
                if (own >= 3) o = fmaf(M.w, b0 ? u[1][3] : u[0][3], o);
                os[it & 1][4 * b + own][b0 ? c + 8 : c] = o;
            }
            auto update = [&](float (&Sr)[R], const float (&uu)[4]) {
                const float w0 = gl.x * uu[0], w1 = gl.y * uu[1], w2 = gl.z * uu[2];
#pragma unroll
                for (int r = 0; r < R; r++) Sr[r] = fmaf(k[3][r], uu[3], fmaf(k[2][r], w2, fmaf(k[1][r], w1, fmaf(k[0][r], w0, G4 * Sr[r]))));
            };
            update(S0, u[0]);
            update(S1, u[1]);
            if (b + 1 < DR_TB / 4)
#pragma unroll
                for (int i = 0; i < 4; i++) load(ks[buf][4 * b + 4 + i], k[i]);
        }
    }
    __syncthreads();
    flush(blocks - 1);
#pragma unroll
    for (int i = 0; i < R; i++) {
        Sg[(size_t)i * DR_THREADS] = S0[i];
        Sg[(size_t)i * DR_THREADS + DB_THREADS] = S1[i];
    }
}

// One CTA per row, one warp per head: y = o / sqrt(mean(o^2) + eps) * w[h * w_stride + d] * gate(g[h][d]), gate = silu (sigmoid_gate: sigmoid).
// w_stride: 0 = one weight of size dv for all heads, dv = a weight per head.  den (nullable, row stride ldo): o is O / den[h].
struct HeadNormArgs {
    const float *w;
    int w_stride, sigmoid_gate;
    const float *den;
    int heads, dv;
    float eps;
};
__global__ void __launch_bounds__(256) k_head_norm_gate(const float *__restrict__ O, int ldo, const float *__restrict__ G, int ldg, HeadNormArgs a, float *__restrict__ out32,
                                                        bf16 *__restrict__ out16, int ldout) {
    pdl_launch_dependents();
    pdl_wait();
    const int r = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, heads = a.heads, dv = a.dv;
    const float eps = a.eps;
    for (int h = blockIdx.y * 8 + warp; h < heads; h += 8 * gridDim.y) {
        const float *w = a.w + (size_t)h * a.w_stride;
        const float rden = a.den ? 1.0f / a.den[(size_t)r * ldo + h] : 1.0f;
        const float *o = O + (size_t)r * ldo + (size_t)h * dv, *g = G + (size_t)r * ldg + (size_t)h * dv;
        float ss = 0.0f;
        for (int i = lane; i < dv; i += 32) { const float v = o[i] * rden; ss = fmaf(v, v, ss); }
        ss = warp_sum(ss);
        const float inv = rden / sqrtf(ss / (float)dv + eps);
        for (int i = lane; i < dv; i += 32) {
            const float z = g[i];
            const float y = o[i] * inv * w[i] * ((a.sigmoid_gate ? 1.0f : z) / (1.0f + expf(-z)));
            if (out32) out32[(size_t)r * ldout + (size_t)h * dv + i] = y;
            if (out16) out16[(size_t)r * ldout + (size_t)h * dv + i] = __float2bfloat16_rn(y);
        }
    }
}

} // namespace ly
