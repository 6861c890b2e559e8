// exact_prefill.cuh -- batched prefill of Q8_0 plans that leaves the KV cache bit-identical to the token-by-token path.
//
// A chunk of n tokens goes through every layer together, so a weight is read once per chunk and not once per token, and every float is
// still evaluated in the CPU path's order: the tokens of a chunk are independent of one another everywhere except in the attention, and
// there token i only reads the cache rows that the earlier tokens of the same layer have written.  Per layer:
//
//   AQ <- Q8_0(rmsnorm(X) * w)                 k_xp_norm       a CTA per token
//   QKV <- AQ [Wq;Wk;Wv]^T                     k_xp_gemm<XP_STORE>
//   q, k <- (Qwen3 head norm,) rotation; k, v -> cache     k_xp_rope_kv
//   AQ <- Q8_0(softmax(q k^T / sqrt(hs)) v)    k_xp_attention  a CTA per (64, 32 or 8 tokens, head)
//   X += AQ Wo^T                               k_xp_gemm<XP_RESID>
//   AQ <- Q8_0(rmsnorm(X) * w)                 k_xp_norm
//   HQ <- Q8_0(silu(AQ W1^T) * (AQ W3^T))      k_xp_gemm<XP_GATEUP>
//   X += HQ W2^T                               k_xp_gemm<XP_RESID>
//
// Measured on two layers of the 8B geometry, 512 tokens and the decode step behind them: 109.8 ms token by token, 2.68 ms here; two layers of the 4B
// Qwen3 geometry, 36 tokens: 5.36 ms and 0.54 ms.
#pragma once
#include "stream_matvec.cuh"

enum { XP_STORE = 0, XP_RESID = 1, XP_GATEUP = 2 };

__device__ __forceinline__ void xp_cp16(unsigned dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void xp_cp8(unsigned dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void xp_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void xp_cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void xp_ldsm4(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// two floats per instruction, each rounded like the scalar operation (round to nearest, subnormals kept)
typedef unsigned long long xp_f2;
__device__ __forceinline__ xp_f2 xp_pack(float a, float b) {
    xp_f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void xp_unpack(xp_f2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ xp_f2 xp_add2(xp_f2 a, xp_f2 b) {
    xp_f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ xp_f2 xp_mul2(xp_f2 a, xp_f2 b) {
    xp_f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// ---- RMSNorm + Q8_0 quantisation of one token's row (InferenceCore.rmsnorm, InferenceCore.java:39-48) ------------------------------
// One CTA per token, E entries per thread in registers, the sum of squares by seqsum3.cuh (a literal chain by one thread, the rows of a chunk side by
// side, took 22 us at dim 4096).  EMBED: the row is gathered from the embedding table first.
// The single-token buffers: every kernel leaves the last token's results there too, in the order of that token's own step (the attention's quantised output and the
// norms' share xq / xs), so that a read-back behind the chunk finds what it finds behind single steps.
struct XpLast {
    int8_t *xq, *hq;
    float *xs, *hs, *hb;
};
struct XpSync { __device__ __forceinline__ void operator()() const { __syncthreads(); } };
template <bool EMBED, int E>
__global__ void __launch_bounds__(256) k_xp_norm(float *__restrict__ X, const int *__restrict__ tok, DevMat emb, const float *__restrict__ w, float eps, int dim,
                                                 int8_t *__restrict__ AQ, float *__restrict__ AS, int lds, XpLast out1) {
    __shared__ __align__(16) float sq[256 * E];
    __shared__ SeqSum3Scratch scratch;
    constexpr int TPB = 32 / E; // threads of a quantisation block
    const int b = blockIdx.x, tid = threadIdx.x, base = tid * E;
    const bool live = base < dim;
    float *x = X + (size_t)b * dim;
    float v[E], t[E];
#pragma unroll
    for (int k = 0; k < E; k += 4) {
        float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
        if (live) {
            if (EMBED) {
                const int token = tok[b];
                q = make_float4(emb_get(emb, token, base + k), emb_get(emb, token, base + k + 1), emb_get(emb, token, base + k + 2), emb_get(emb, token, base + k + 3));
                *reinterpret_cast<float4 *>(x + base + k) = q;
            } else q = *reinterpret_cast<const float4 *>(x + base + k);
        }
        v[k] = q.x; v[k + 1] = q.y; v[k + 2] = q.z; v[k + 3] = q.w;
        t[k] = __fmul_rn(q.x, q.x); t[k + 1] = __fmul_rn(q.y, q.y); t[k + 2] = __fmul_rn(q.z, q.z); t[k + 3] = __fmul_rn(q.w, q.w);
        *reinterpret_cast<float4 *>(sq + base + k) = make_float4(t[k], t[k + 1], t[k + 2], t[k + 3]);
    }
    float ss = block_seqsum3<E>(t, sq, scratch, tid, XpSync());
    ss = __fdiv_rn(ss, (float)dim);
    ss = __fadd_rn(ss, eps);
    ss = (float)(1.0 / sqrt((double)ss));
    float amax = 0.0f;
#pragma unroll
    for (int k = 0; k < E; k += 4) {
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
        if (live) g = *reinterpret_cast<const float4 *>(w + base + k);
        v[k] = __fmul_rn(g.x, __fmul_rn(ss, v[k])); v[k + 1] = __fmul_rn(g.y, __fmul_rn(ss, v[k + 1]));
        v[k + 2] = __fmul_rn(g.z, __fmul_rn(ss, v[k + 2])); v[k + 3] = __fmul_rn(g.w, __fmul_rn(ss, v[k + 3]));
#pragma unroll
        for (int u = 0; u < 4; u++) amax = fmaxf(amax, fabsf(v[k + u]));
    }
#pragma unroll
    for (int o = TPB / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (!live) return;
    const float qs = __fdiv_rn(amax, 127.0f), as = __half2float(__float2half_rn(qs)), ainv = qs != 0.0f ? __fdiv_rn(1.0f, qs) : 0.0f; // quant_block_lane's arithmetic
    const bool last = b == (int)gridDim.x - 1;
#pragma unroll
    for (int k = 0; k < E; k += 4) {
        unsigned p = 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const float s = __fmul_rn(v[k + u], ainv);
            p |= ((unsigned)__float2int_rz(__fadd_rn(s, copysignf(0.5f, s))) & 0xffu) << (8 * u);
        }
        *reinterpret_cast<unsigned *>(AQ + (size_t)b * dim + base + k) = p;
        if (last) *reinterpret_cast<unsigned *>(out1.xq + base + k) = p;
    }
    if (tid % TPB == 0) {
        AS[(size_t)(base / 32) * lds + b] = as;
        if (last) out1.xs[base / 32] = as;
    }
}

// ---- the product -----------------------------------------------------------------------------------------------------------------
// out[token][row] = sum over 32-blocks, strictly in block order, of (float)isum * (wScale * aScale)   (Q8_0FloatTensor.java:90-123).
// isum of a block is one mma.sync.m16n8k32 (int8, exact).  The tensor pipe is not what bounds this: every (row, token, block) costs four
// FP32 operations (int to float, scale product, term, ordered add), the order of the adds is fixed, and those run on the CUDA cores.  So: the
// accumulator of each mma starts at the integer 0x4B400000, whose bit pattern plus isum IS the float 12582912 + isum (|isum| <= 520,192), and one
// exact subtraction replaces the conversion; the subtraction and the products are issued two values at a time (f32x2).  The ordered add is a scalar
// __fadd_rn: a packed add behind a packed product comes out as one fused operation (measured: results differ in the last bits), the scalar one never.
// Half of the row tiles take the conversion instruction after all: it runs beside the FP32 pipe (2799 -> 2746 us for the 512-token prompt above).
// Bound by latency, not by a pipe: the gate/up product of 512 tokens takes 41.5 cycles of a scheduler per (16 x 8 tile, block), of which the FP32 operations need 16;
// issue slots are used in 58 % of the cycles, the FMA pipe in 38 %.  128 registers allow four warps a scheduler, and a block's ldmatrix, mma, conversion, products and
// ordered add follow one another in each.
// A CTA is 4 warps: 64 weight rows (16 groups of the tile-major layout) x 8 * NJ tokens; with 32 tokens and more a warp owns 32 rows and half of the tokens
// (every B fragment and activation scale serves two row tiles), else 16 rows and all of them.  Three stages of 128 columns come in by cp.async; rows of 128 bytes are swizzled in 16-byte chunks so that ldmatrix is conflict-free.
// NJ (tokens per tile) is the largest that still gives every SM a CTA: a chunk of a few tokens is bound by the length of the column chain.
#define XP_STAGES 3
#define XP_ROWS 64
#define XP_THREADS 128
template <int NJ> struct XpTile {
    static constexpr int TOK = 8 * NJ;
    static constexpr int A_Q = 0, A_S = XP_ROWS * 128, B_Q = A_S + XP_ROWS * 8, B_S = B_Q + TOK * 128, STAGE = (B_S + 4 * TOK * 4 + 127) & ~127;
    static constexpr int HV = 33 * TOK * 4; // gate/up: the tile's 32 hidden units (+ 1: no bank conflicts) per token
    static constexpr int BYTES = XP_STAGES * STAGE > HV ? XP_STAGES * STAGE : HV;
};

template <int MODE, int NJ>
__global__ void __launch_bounds__(XP_THREADS, 4) k_xp_gemm(TileMat W, const int8_t *__restrict__ AQ, const float *__restrict__ AS, int lds, int n, float *__restrict__ out, int ldo,
                                                        int8_t *__restrict__ HQ, float *__restrict__ HS, XpLast last) {
    using T = XpTile<NJ>;
    constexpr int TOK = T::TOK, MI = NJ >= 4 ? 2 : 1, NW = NJ / MI; // a warp's tile: 16 MI rows x 8 NW tokens
    extern __shared__ __align__(128) unsigned char smraw[];
    const unsigned smb = smem_u32(smraw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = blockIdx.x * XP_ROWS, tok0 = blockIdx.y * TOK;
    const int nbs = W.seg >> 5, cps = (nbs + 3) >> 2, n_chunks = W.nseg * cps; // blocks per segment, chunks of <= 4 blocks per segment

    // what this thread fetches of a stage: A chunks c = tid + 128 u -> row c / 8, 16-byte piece c % 8 (4 of them)
    const int piece = tid & 7;
    const unsigned char *arow[4];
    unsigned adst[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int r = (tid >> 3) + 16 * u;
        const int row = min(row0 + r, W.rows - 1);
        arow[u] = W.base + ((size_t)(row >> 2) * W.nseg * 4 + (row & 3)) * (size_t)W.unit_bytes;
        adst[u] = T::A_Q + r * 128 + ((piece ^ (r & 7)) << 4);
    }
    const int srow = min(row0 + (tid & 63), W.rows - 1);
    const unsigned char *asrc = W.base + ((size_t)(srow >> 2) * W.nseg * 4 + (srow & 3)) * (size_t)W.unit_bytes + W.seg;
    constexpr int BU = (TOK + 15) / 16;
    const int8_t *brow[BU];
    unsigned bdst[BU];
#pragma unroll
    for (int u = 0; u < BU; u++) {
        const int t = (tid >> 3) + 16 * u;
        brow[u] = AQ + (size_t)(tok0 + t) * W.cols + piece * 16; // (TOK == 8: rows 8 .. 15 belong to nobody and are not fetched)
        bdst[u] = T::B_Q + t * 128 + ((piece ^ (t & 7)) << 4);
    }
#pragma unroll
    for (int u = 0; u < 4; u++) arow[u] += piece * 16;
    const float *bsrc = AS + (size_t)((tid - 64) / (TOK / 4)) * lds + tok0 + (tid - 64) % (TOK / 4) * 4; // scales of block (tid - 64) / (TOK / 4) of a stage
    const unsigned seg_step = 4u * (unsigned)W.unit_bytes;
    unsigned a_off = 0, s_off = 0, b_off = 0, f_c = 0, seg_off = 0; // byte offsets of the next chunk: weights, weight scales, activations; chunk in the segment
    size_t bs_off = 0;                                              // activation scales (floats)

    auto fetch = [&](int stage) {
        const int blocks = min(4, nbs - 4 * (int)f_c);
        const unsigned s = smb + stage * T::STAGE;
        if (piece < 2 * blocks) {
#pragma unroll
            for (int u = 0; u < 4; u++) xp_cp16(s + adst[u], arow[u] + a_off);
#pragma unroll
            for (int u = 0; u < BU; u++)
                if (TOK >= 16 || (tid >> 3) < TOK) xp_cp16(s + bdst[u], brow[u] + b_off);
        }
        if (tid < 64) xp_cp8(s + T::A_S + tid * 8, asrc + s_off); // the scale area of a unit is padded to 16 bytes
        else if (tid - 64 < blocks * (TOK / 4)) xp_cp16(s + T::B_S + (tid - 64) * 16, bsrc + bs_off);
        a_off += 128; s_off += 8;
        b_off += 32 * blocks;
        bs_off += (size_t)blocks * lds;
        if (++f_c == (unsigned)cps) { f_c = 0; seg_off += seg_step; a_off = s_off = seg_off; }
    };
#pragma unroll
    for (int s = 0; s < XP_STAGES - 1; s++) {
        if (s < n_chunks) fetch(s);
        xp_cp_commit();
    }

    float acc[MI][NW][2][2]; // [row tile][token tile][row lane/4 | row lane/4 + 8][token 2 (lane % 4) | + 1]
#pragma unroll
    for (int i = 0; i < MI; i++)
#pragma unroll
        for (int j = 0; j < NW; j++) acc[i][j][0][0] = acc[i][j][0][1] = acc[i][j][1][0] = acc[i][j][1][1] = 0.0f;
    const xp_f2 minus_magic = xp_pack(-12582912.0f, -12582912.0f);
    const int wrow = (warp % (4 / MI)) * 16 * MI, wtok = (warp / (4 / MI)) * 8 * NW; // the warp's first row and token in the tile
    const int ar = wrow + (lane & 15), ap = lane >> 4;                              // ldmatrix: A row, 16-byte half
    const int bt = wtok + (NW > 1 ? ((lane >> 4) << 3) + (lane & 7) : (lane & 7)), bp = (lane >> 3) & 1; // B token (of 16), half
    int stage = 0, c_in_seg = 0;
    for (int c = 0; c < n_chunks; c++) {
        xp_cp_wait<XP_STAGES - 2>();
        __syncthreads();
        {
            int fs = stage + XP_STAGES - 1;
            if (fs >= XP_STAGES) fs -= XP_STAGES;
            if (c + XP_STAGES - 1 < n_chunks) fetch(fs);
            xp_cp_commit();
        }
        const unsigned s = smb + stage * T::STAGE;
        const unsigned char *sp = smraw + stage * T::STAGE;
        uint2 ws[MI][2];
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int h = 0; h < 2; h++) ws[i][h] = *reinterpret_cast<const uint2 *>(sp + T::A_S + (wrow + 16 * i + 8 * h + (lane >> 2)) * 8);
        const int blocks = min(4, nbs - 4 * c_in_seg);
        auto block = [&](int k) {
            unsigned a[MI][4];
            xp_f2 wp[MI][2];
#pragma unroll
            for (int i = 0; i < MI; i++) {
                xp_ldsm4(a[i], s + T::A_Q + (ar + 16 * i) * 128 + (((2 * k + ap) ^ (ar & 7)) << 4));
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const unsigned hw = k < 2 ? ws[i][h].x : ws[i][h].y;
                    const float w = __half2float(__ushort_as_half((unsigned short)(k & 1 ? hw >> 16 : hw & 0xffffu)));
                    wp[i][h] = xp_pack(w, w);
                }
            }
#pragma unroll
            for (int j = 0; j < NW; j += 2) {
                unsigned b[4]; // two token tiles (NW == 1: the second one is the first again)
                const int t = bt + j * 8;
                xp_ldsm4(b, s + T::B_Q + t * 128 + (((2 * k + bp) ^ (t & 7)) << 4));
#pragma unroll
                for (int jj = 0; jj < (NW > 1 ? 2 : 1); jj++) {
                    const xp_f2 as = *reinterpret_cast<const xp_f2 *>(sp + T::B_S + (k * TOK + wtok + (j + jj) * 8 + 2 * (lane & 3)) * 4);
#pragma unroll
                    for (int i = 0; i < MI; i++) {
                        // one row tile turns its integers to floats by the subtraction above, the other by conversions: they run beside the FP32 pipe
                        const bool cvt = i == 1;
                        int d0, d1, d2, d3;
                        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                                     : "=r"(d0), "=r"(d1), "=r"(d2), "=r"(d3)
                                     : "r"(a[i][0]), "r"(a[i][1]), "r"(a[i][2]), "r"(a[i][3]), "r"(b[2 * jj]), "r"(b[2 * jj + 1]), "r"(cvt ? 0 : 0x4B400000));
                        const xp_f2 f0 = cvt ? xp_pack((float)d0, (float)d1) : xp_add2(xp_pack(__int_as_float(d0), __int_as_float(d1)), minus_magic);
                        const xp_f2 f1 = cvt ? xp_pack((float)d2, (float)d3) : xp_add2(xp_pack(__int_as_float(d2), __int_as_float(d3)), minus_magic);
                        float t0, t1, t2, t3;
                        xp_unpack(xp_mul2(f0, xp_mul2(wp[i][0], as)), t0, t1);
                        xp_unpack(xp_mul2(f1, xp_mul2(wp[i][1], as)), t2, t3);
                        float(&ac)[2][2] = acc[i][j + jj];
                        ac[0][0] = __fadd_rn(ac[0][0], t0); ac[0][1] = __fadd_rn(ac[0][1], t1);
                        ac[1][0] = __fadd_rn(ac[1][0], t2); ac[1][1] = __fadd_rn(ac[1][1], t3);
                    }
                }
            }
        };
        if (blocks == 4) {
#pragma unroll
            for (int k = 0; k < 4; k++) block(k);
        } else {
#pragma unroll
            for (int k = 0; k < 3; k++)
                if (k < blocks) block(k);
        }
        if (++stage == XP_STAGES) stage = 0;
        if (++c_in_seg == cps) c_in_seg = 0;
    }

    const int r0 = wrow + (lane >> 2), t0 = wtok + 2 * (lane & 3);
    if (MODE == XP_GATEUP) { // rows of a group: gate 2G, gate 2G + 1, up 2G, up 2G + 1; the CTA's 64 rows are one 32-unit block of the hidden row
        xp_cp_wait<0>();
        __syncthreads();
        float *hv = reinterpret_cast<float *>(smraw);
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int j = 0; j < NW; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const float g0 = acc[i][j][h][0], g1 = acc[i][j][h][1];
                    const float u0 = __shfl_down_sync(0xffffffffu, g0, 8), u1 = __shfl_down_sync(0xffffffffu, g1, 8);
                    if (!((lane >> 2) & 2)) {
                        const int row = r0 + 16 * i + 8 * h, unit = (row >> 2) * 2 + (row & 1), t = t0 + j * 8;
                        hv[t * 33 + unit] = swiglu_exact(g0, u0);
                        hv[(t + 1) * 33 + unit] = swiglu_exact(g1, u1);
                    }
                }
        __syncthreads();
        const int hidden = W.rows >> 1;
        for (int t = warp; t < TOK && tok0 + t < n; t += XP_THREADS / 32) {
            const float v = hv[t * 33 + lane];
            float as;
            const int q = quant_block_lane(v, as);
            HQ[(size_t)(tok0 + t) * hidden + blockIdx.x * 32 + lane] = (int8_t)q;
            if (lane == 0) HS[(size_t)blockIdx.x * lds + tok0 + t] = as;
            if (tok0 + t == n - 1) {
                last.hb[blockIdx.x * 32 + lane] = v;
                last.hq[blockIdx.x * 32 + lane] = (int8_t)q;
                if (lane == 0) last.hs[blockIdx.x] = as;
            }
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < MI; i++)
#pragma unroll
        for (int j = 0; j < NW; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int row = row0 + r0 + 16 * i + 8 * h, t = tok0 + t0 + j * 8;
                const float v0 = acc[i][j][h][0], v1 = acc[i][j][h][1];
                if (row < W.rows) {
                    float *o = out + (size_t)t * ldo + row;
                    if (t < n) o[0] = MODE == XP_RESID ? __fadd_rn(o[0], v0) : v0;
                    if (t + 1 < n) o[ldo] = MODE == XP_RESID ? __fadd_rn(o[ldo], v1) : v1;
                }
            }
}

// ---- head norm, rotation, cache rows of one token (k_attention's prologue for a whole row) ------------------------------------------
__global__ void __launch_bounds__(256) k_xp_rope_kv(float *__restrict__ QKV, float *__restrict__ kc, float *__restrict__ vc, int hs, int n_heads, int n_kv_heads, int flags,
                                                    const float *__restrict__ qnw, const float *__restrict__ knw, float eps, const float *__restrict__ cr,
                                                    const float *__restrict__ ci, int start_pos) {
    extern __shared__ __align__(16) float sm[];
    float *row = sm; // [q heads | k heads][hs + 1]
    __shared__ float scale[256];
    const int b = blockIdx.x, tid = threadIdx.x, pos = start_pos + b, half = hs / 2;
    const int nh = n_heads + n_kv_heads, qd = n_heads * hs, kvd = n_kv_heads * hs;
    float *src = QKV + (size_t)b * (qd + 2 * kvd);
    for (int i = tid; i < nh * hs; i += 256) row[(i / hs) * (hs + 1) + i % hs] = src[i];
    for (int i = tid; i < kvd; i += 256) vc[(size_t)pos * kvd + i] = src[qd + kvd + i];
    __syncthreads();
    for (int h0 = 0; h0 < nh; h0 += 256) { // (one pass: up to 256 query and key heads)
        if ((flags & KF_QKNORM) && h0 + tid < nh) { // literal sequential sum over the head
            const float *v = row + (h0 + tid) * (hs + 1);
            float ss = 0.0f;
            for (int i = 0; i < hs; i++) ss = __fadd_rn(ss, __fmul_rn(v[i], v[i]));
            ss = __fdiv_rn(ss, (float)hs);
            ss = __fadd_rn(ss, eps);
            scale[tid] = (float)(1.0 / sqrt((double)ss));
        }
        __syncthreads();
        const int h1 = min(h0 + 256, nh);
        for (int i = tid; i < (h1 - h0) * half; i += 256) {
            const int h = h0 + i / half, p = i % half;
            const bool is_q = h < n_heads;
            const int i0 = flags & KF_NEOX ? p : 2 * p, i1 = flags & KF_NEOX ? p + half : 2 * p + 1;
            float v0 = row[h * (hs + 1) + i0], v1 = row[h * (hs + 1) + i1];
            if (flags & KF_QKNORM) {
                const float *nw = is_q ? qnw : knw;
                const float ss = scale[h - h0];
                v0 = __fmul_rn(nw[i0], __fmul_rn(ss, v0));
                v1 = __fmul_rn(nw[i1], __fmul_rn(ss, v1));
            }
            const float fcr = cr[(size_t)pos * half + p], fci = ci[(size_t)pos * half + p];
            const float r0 = __fsub_rn(__fmul_rn(v0, fcr), __fmul_rn(v1, fci));
            const float r1 = __fadd_rn(__fmul_rn(v0, fci), __fmul_rn(v1, fcr));
            float *dst = is_q ? src + h * hs : kc + (size_t)pos * kvd + (h - n_heads) * hs;
            dst[i0] = r0;
            dst[i1] = r1;
        }
        __syncthreads();
    }
}

// ---- attention of QT tokens and one head, every sum in the CPU path's order ----------------------------------------------------------
// score = sequential sum over the head of q * k, / sqrt(hs); softmax with a sequential sum; out = sequential sum over the positions of a * v.
// A warp owns QI tokens and a lane two keys of the staged tile: QI x 2 chains per thread in the score pass, QI x 4 (token, element) chains in the
// value pass, so that a 16-byte shared load feeds several multiply and add pairs; the next tile comes in by cp.async meanwhile.  The rows of scores live in shared memory, or in the CTA's
// own slot of a global scratch for long contexts.  One work item = (tile of QT = warps x QI tokens, head); CTAs walk the items, the latest tiles (the
// longest rows) first.
#define XP_KT 64 // keys / values per staged tile (two tiles: the next one is on its way while one is worked on)
__host__ __device__ inline int xp_score_stride(int nt) { return (nt + 31) / 32 * 32 + 4; } // rows start four banks apart
__host__ __device__ inline size_t xp_att_smem_bytes(int hs, int qt, int nt, bool scratch) {
    return ((size_t)qt * (hs + 4) + (size_t)2 * XP_KT * (hs + 4) + (scratch ? 0 : (size_t)qt * xp_score_stride(nt)) + 2 * 64) * 4;
}
template <int HS, int QI, int XP_ATT_THREADS>
__global__ void __launch_bounds__(XP_ATT_THREADS) k_xp_attention(const float *__restrict__ QKV, const float *__restrict__ kc, const float *__restrict__ vc, int n_heads, int n_kv_heads,
                                                                 int n, int start_pos, float sqrt_hs, int8_t *__restrict__ AQ, float *__restrict__ AS, int lds, float *scratch, XpLast last) {
    extern __shared__ __align__(16) float sm[];
    constexpr int LD = HS + 4, QG = XP_ATT_THREADS / 32, QT = QG * QI;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int stride = xp_score_stride(start_pos + n), qd = n_heads * HS, kvd = n_kv_heads * HS, kv_mul = n_heads / n_kv_heads;
    float *sq = sm, *st = sq + QT * LD, *red = st + 2 * XP_KT * LD; // q tile | two key or value tiles | row maxima, row sums
    float *S = scratch ? scratch + (size_t)blockIdx.x * QT * stride : red + 128;
    const int tiles = (n + QT - 1) / QT;
    constexpr int KU = XP_KT / 32; // keys per lane
    constexpr int DG = HS / 4; // value pass: QG x DG threads, QI tokens x 4 neighbouring elements each
    constexpr int PV_PASSES = (QG * DG + XP_ATT_THREADS - 1) / XP_ATT_THREADS;
    for (int item = blockIdx.x; item < tiles * n_heads; item += gridDim.x) {
        const int h = item % n_heads, q0 = (tiles - 1 - item / n_heads) * QT, kvh = h / kv_mul;
        const int rows = min(QT, n - q0), nt = start_pos + q0 + rows; // keys the tile's last row sees
        const float *kb = kc + kvh * HS, *vb = vc + kvh * HS;
        __syncthreads(); // the previous item's readers are done
        for (int i = tid; i < QT * (HS / 4); i += XP_ATT_THREADS) {
            const int r = i / (HS / 4), d4 = i % (HS / 4);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < rows) v = *reinterpret_cast<const float4 *>(QKV + (size_t)(q0 + r) * (qd + 2 * kvd) + h * HS + 4 * d4);
            *reinterpret_cast<float4 *>(sq + r * LD + 4 * d4) = v;
        }
        auto load_tile = [&](const float *base, int tile) { // asynchronous; rows behind the last key stay as they are and are never used
            float *dst = st + (tile & 1) * XP_KT * LD;
            const int t0 = tile * XP_KT;
            for (int i = tid; i < XP_KT * (HS / 4); i += XP_ATT_THREADS) {
                const int t = i / (HS / 4), d4 = i % (HS / 4);
                if (t0 + t < nt) xp_cp16(smem_u32(dst + t * LD + 4 * d4), base + (size_t)(t0 + t) * kvd + 4 * d4);
            }
            xp_cp_commit();
        };
        const int n_tiles = (nt + XP_KT - 1) / XP_KT;
        load_tile(kb, 0);
        // ---- scores
        float mx[QI];
#pragma unroll
        for (int i = 0; i < QI; i++) mx[i] = -INFINITY;
        for (int tile = 0; tile < n_tiles; tile++) {
            const int t0 = tile * XP_KT;
            xp_cp_wait<0>();
            __syncthreads(); // the tile has landed for every thread, and the tile before it is done with
            if (tile + 1 < n_tiles) load_tile(kb, tile + 1);
            const float *sk = st + (tile & 1) * XP_KT * LD;
            if (warp * QI < rows) {
                float a[QI][KU];
#pragma unroll
                for (int i = 0; i < QI; i++)
#pragma unroll
                    for (int u = 0; u < KU; u++) a[i][u] = 0.0f;
#pragma unroll 4
                for (int d = 0; d < HS; d += 4) {
                    float4 q[QI], k[KU];
#pragma unroll
                    for (int i = 0; i < QI; i++) q[i] = *reinterpret_cast<const float4 *>(sq + (warp * QI + i) * LD + d);
#pragma unroll
                    for (int u = 0; u < KU; u++) k[u] = *reinterpret_cast<const float4 *>(sk + (lane + 32 * u) * LD + d);
#pragma unroll
                    for (int i = 0; i < QI; i++)
#pragma unroll
                        for (int u = 0; u < KU; u++) {
                            a[i][u] = __fadd_rn(a[i][u], __fmul_rn(q[i].x, k[u].x));
                            a[i][u] = __fadd_rn(a[i][u], __fmul_rn(q[i].y, k[u].y));
                            a[i][u] = __fadd_rn(a[i][u], __fmul_rn(q[i].z, k[u].z));
                            a[i][u] = __fadd_rn(a[i][u], __fmul_rn(q[i].w, k[u].w));
                        }
                }
#pragma unroll
                for (int i = 0; i < QI; i++) {
                    const int r = warp * QI + i, last = start_pos + q0 + r;
#pragma unroll
                    for (int u = 0; u < KU; u++) {
                        const int t = t0 + lane + 32 * u;
                        if (r < rows && t <= last) {
                            const float s = __fdiv_rn(a[i][u], sqrt_hs);
                            S[(size_t)r * stride + t] = s;
                            mx[i] = fmaxf(mx[i], s);
                        }
                    }
                }
            }
        }
        __syncthreads(); // the last key tile is done with
        load_tile(vb, 0); // in flight through the softmax
        // ---- softmax
#pragma unroll
        for (int i = 0; i < QI; i++) {
            const float m = warp_max_f(mx[i]);
            if (lane == 0) red[warp * QI + i] = m;
        }
        __syncthreads();
        for (int r = warp; r < rows; r += XP_ATT_THREADS / 32) {
            float *s = S + (size_t)r * stride;
            const int cnt = start_pos + q0 + r + 1;
            const float m = red[r];
            for (int t = lane; t < cnt; t += 32) s[t] = (float)exp((double)__fsub_rn(s[t], m));
        }
        __syncthreads();
        if (tid < rows) red[64 + tid] = pd_walk_terms(0.0f, S + (size_t)tid * stride, start_pos + q0 + tid + 1);
        __syncthreads();
        for (int r = warp; r < rows; r += XP_ATT_THREADS / 32) {
            float *s = S + (size_t)r * stride;
            const int cnt = start_pos + q0 + r + 1;
            const float sum = red[64 + r];
            for (int t = lane; t < cnt; t += 32) s[t] = __fdiv_rn(s[t], sum);
        }
        // ---- values
        float o[PV_PASSES][QI][4];
#pragma unroll
        for (int ps = 0; ps < PV_PASSES; ps++)
#pragma unroll
            for (int i = 0; i < QI; i++)
#pragma unroll
                for (int u = 0; u < 4; u++) o[ps][i][u] = 0.0f;
        for (int tile = 0; tile < n_tiles; tile++) {
            const int t0 = tile * XP_KT;
            xp_cp_wait<0>();
            __syncthreads();
            if (tile + 1 < n_tiles) load_tile(vb, tile + 1);
            const float *sv = st + (tile & 1) * XP_KT * LD;
#pragma unroll
            for (int ps = 0; ps < PV_PASSES; ps++) {
                const int w = tid + ps * XP_ATT_THREADS, g = w / DG, dg = w % DG;
                if (w < QG * DG && g * QI < rows) { // (a group behind the last row sees positions that its score rows have no room for)
                    const float *a0 = S + (size_t)(g * QI) * stride + t0;
                    const int full = start_pos + q0 + g * QI + 1 - t0; // positions of this tile that the group's first row sees
                    if (full >= XP_KT) { // ... all of them: so do the later rows
#pragma unroll 2
                        for (int t = 0; t < XP_KT; t += 4) {
                            float4 a[QI];
#pragma unroll
                            for (int i = 0; i < QI; i++) a[i] = *reinterpret_cast<const float4 *>(a0 + (size_t)i * stride + t);
#pragma unroll
                            for (int k = 0; k < 4; k++) {
                                const float4 v = *reinterpret_cast<const float4 *>(sv + (t + k) * LD + dg * 4);
#pragma unroll
                                for (int i = 0; i < QI; i++) {
                                    const float x = k == 0 ? a[i].x : k == 1 ? a[i].y : k == 2 ? a[i].z : a[i].w;
                                    o[ps][i][0] = __fadd_rn(__fmul_rn(x, v.x), o[ps][i][0]);
                                    o[ps][i][1] = __fadd_rn(__fmul_rn(x, v.y), o[ps][i][1]);
                                    o[ps][i][2] = __fadd_rn(__fmul_rn(x, v.z), o[ps][i][2]);
                                    o[ps][i][3] = __fadd_rn(__fmul_rn(x, v.w), o[ps][i][3]);
                                }
                            }
                        }
                    } else {
                        for (int t = 0; t < XP_KT && t < full + QI - 1; t++) {
                            const float4 v = *reinterpret_cast<const float4 *>(sv + t * LD + dg * 4);
#pragma unroll
                            for (int i = 0; i < QI; i++)
                                if (t < full + i && g * QI + i < rows) {
                                    const float x = a0[(size_t)i * stride + t];
                                    o[ps][i][0] = __fadd_rn(__fmul_rn(x, v.x), o[ps][i][0]);
                                    o[ps][i][1] = __fadd_rn(__fmul_rn(x, v.y), o[ps][i][1]);
                                    o[ps][i][2] = __fadd_rn(__fmul_rn(x, v.z), o[ps][i][2]);
                                    o[ps][i][3] = __fadd_rn(__fmul_rn(x, v.w), o[ps][i][3]);
                                }
                        }
                    }
                }
            }
        }
        __syncthreads(); // the q tile becomes the output tile
#pragma unroll
        for (int ps = 0; ps < PV_PASSES; ps++) {
            const int w = tid + ps * XP_ATT_THREADS, g = w / DG, dg = w % DG;
            if (w < QG * DG)
#pragma unroll
                for (int i = 0; i < QI; i++) *reinterpret_cast<float4 *>(sq + (g * QI + i) * LD + dg * 4) = make_float4(o[ps][i][0], o[ps][i][1], o[ps][i][2], o[ps][i][3]);
        }
        __syncthreads();
        for (int k = warp; k < rows * (HS / 32); k += XP_ATT_THREADS / 32) { // Q8_0 blocks of the output projection's activation
            const int r = k / (HS / 32), blk = k % (HS / 32);
            float as;
            const int q = quant_block_lane(sq[r * LD + blk * 32 + lane], as);
            AQ[(size_t)(q0 + r) * qd + h * HS + blk * 32 + lane] = (int8_t)q;
            if (lane == 0) AS[(size_t)(h * (HS / 32) + blk) * lds + q0 + r] = as;
            if (q0 + r == n - 1) {
                last.xq[h * HS + blk * 32 + lane] = (int8_t)q;
                if (lane == 0) last.xs[h * (HS / 32) + blk] = as;
            }
        }
    }
}
