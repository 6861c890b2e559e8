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
//   HQ <- Q8_0(silu(AQ W1^T) * (AQ W3^T))      k_xp_gemm<XP_GATEUP>, or k_xp_gemm<XP_STORE> and k_xt_swiglu (exact_prefill_umma.cuh) where there is much of it
//   X += HQ W2^T                               k_xp_gemm<XP_RESID>
//
// Each of the four products is k_xt_gemm's (exact_prefill_umma.cuh, tcgen05) where the host's time model says so: long chunks.  Its operands are FP16 numbers, AH
// and HH in AQ's and HQ's place.
//
// Measured on two layers of the 8B geometry, 512 tokens and the decode step behind them: 109.8 ms token by token, 1.94 ms here; two layers of the 4B
// Qwen3 geometry, 36 tokens: 5.36 ms and 0.44 ms.
#pragma once
#include "prefill_gemm.cuh"
#include "stream_matvec.cuh"

enum { XP_STORE = 0, XP_RESID = 1, XP_GATEUP = 2 };

__device__ __forceinline__ void xp_cp16(unsigned dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
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
__device__ __forceinline__ xp_f2 xp_mul2(xp_f2 a, xp_f2 b) {
    xp_f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ xp_f2 xp_fma2(xp_f2 a, xp_f2 b, xp_f2 c) {
    xp_f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// four quants as bytes, and four bytes as FP16 numbers (1024 + 128 + q has q + 128 in its low byte)
__device__ __forceinline__ unsigned xp_bytes(const int (&q)[4]) { return (q[0] & 0xff) | (q[1] & 0xff) << 8 | (q[2] & 0xff) << 16 | (unsigned)q[3] << 24; }
__device__ __forceinline__ void xp_halves(unsigned q, unsigned &lo, unsigned &hi) {
    const __half2 bias = __floats2half2_rn(1152.0f, 1152.0f);
    q ^= 0x80808080u;
    lo = __byte_perm(q, 0x64646464u, 0x4140);
    hi = __byte_perm(q, 0x64646464u, 0x4342);
    const __half2 a = __hsub2(*reinterpret_cast<__half2 *>(&lo), bias), b = __hsub2(*reinterpret_cast<__half2 *>(&hi), bias);
    lo = *reinterpret_cast<const unsigned *>(&a);
    hi = *reinterpret_cast<const unsigned *>(&b);
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
__global__ void __launch_bounds__(256, E <= 16 ? 4 : 1) k_xp_norm(float *__restrict__ X, const int *__restrict__ tok, DevMat emb, const float *__restrict__ w, float eps, int dim,
                                                 int8_t *__restrict__ AQ, __half *__restrict__ AH, float *__restrict__ AS, int lds, XpLast out1) {
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
    unsigned q[E / 4];
#pragma unroll
    for (int k = 0; k < E; k += 4) {
        int u[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float s = __fmul_rn(v[k + j], ainv);
            u[j] = __float2int_rz(__fadd_rn(s, copysignf(0.5f, s)));
        }
        q[k / 4] = xp_bytes(u);
        if (last) *reinterpret_cast<unsigned *>(out1.xq + base + k) = q[k / 4];
    }
    if (AH) {
#pragma unroll
        for (int k = 0; k < E; k += E >= 8 ? 8 : 4) {
            uint4 h;
            xp_halves(q[k / 4], h.x, h.y);
            if (E >= 8) {
                xp_halves(q[E >= 8 ? k / 4 + 1 : 0], h.z, h.w);
                *reinterpret_cast<uint4 *>(AH + (size_t)b * dim + base + k) = h;
            } else *reinterpret_cast<uint2 *>(AH + (size_t)b * dim + base + k) = make_uint2(h.x, h.y);
        }
    } else {
#pragma unroll
        for (int k = 0; k < E; k += E >= 16 ? 16 : E) {
            int8_t *dst = AQ + (size_t)b * dim + base + k;
            if (E >= 16) *reinterpret_cast<uint4 *>(dst) = make_uint4(q[k / 4], q[E >= 16 ? k / 4 + 1 : 0], q[E >= 16 ? k / 4 + 2 : 0], q[E >= 16 ? k / 4 + 3 : 0]);
            else if (E >= 8) *reinterpret_cast<uint2 *>(dst) = make_uint2(q[0], q[E >= 8 ? 1 : 0]);
            else *reinterpret_cast<unsigned *>(dst) = q[0];
        }
    }
    if (tid % TPB == 0) {
        AS[(size_t)(base / 32) * lds + b] = as;
        if (last) out1.xs[base / 32] = as;
    }
}

// ---- the product -----------------------------------------------------------------------------------------------------------------
// out[token][row] = sum over 32-blocks, strictly in block order, of (float)isum * (wScale * aScale)   (Q8_0FloatTensor.java:90-123).
// isum of a block is one mma.sync.m16n8k32 (int8, exact).  The tensor pipe is not what bounds this: every (row, token, block) costs a conversion, two
// products and an ordered add, and those run on the CUDA cores, two values at a time (f32x2).  The ordered add is fma(acc, 1, term), which rounds like the
// add: a packed add behind a packed product comes out as ONE fused operation (measured; also where the 1 is a constant of the kernel, so it is an argument).
// Integers are converted by the conversion instruction: accumulators that start at 0x4B400000 and a subtraction cost four register moves for every mma (gate/up
// product 411 against 392 us).
// A CTA is 4 warps that multiply: 64 weight rows (16 groups of the tile-major layout) x 8 * NJ tokens; with 32 tokens and more a warp owns 32 rows and half of the tokens
// (every B fragment and activation scale serves two row tiles), else 16 rows and all of them; and one that fetches: a ring of stages of 128 columns comes in by TMA (weights and
// their scales straight out of the tile-major layout by a 4-D map), rows of 128 bytes swizzled so that ldmatrix is conflict-free.  A multiplying warp that waited for the others and
// issued the fetches between its chunks held the whole CTA up by half of its time: gate/up of 512 tokens, 8B layer, 388 us against 328 us so; W2 of 36 tokens, 4B layer, 43 against 28 us (a
// deeper ring alone 43, all operands of a chunk in registers ahead 46).  Issue slots: 15.7 warp instructions per 16 x 8 tile and block, 10 of them the conversions, products and
// adds (65 % of the slots, FMA pipe 57 %).
// Long chunks' products are exact_prefill_umma.cuh's.
#define XP_STAGES 3      // of a ring, at least;
#define XP_STAGES_MAX 8  // and at most: as many as the CTAs of an SM have room for
#define XP_ROWS 64
#define XP_THREADS 128 // that multiply; a fifth warp fetches
struct XpMaps { CUtensorMap q, s; }; // quants; scales
template <int NJ> struct XpTile {
    static constexpr int TOK = 8 * NJ;
    static constexpr int A_Q = 0, B_Q = XP_ROWS * 128, A_S = B_Q + TOK * 128, B_S = A_S + XP_ROWS * 16, BYTES_IN = B_S + 4 * TOK * 4, STAGE = (BYTES_IN + 1023) & ~1023;
    static constexpr int HV = 33 * TOK * 4; // gate/up: the tile's 32 hidden units (+ 1: no bank conflicts) per token
    static constexpr int RESIDENT = NJ == 8 ? 3 : 4; // CTAs of an SM (registers)
    static constexpr int bytes(int stages) { return 1024 + stages * STAGE + 16 * stages; }
};
// Bounded: false = given up, after a second or once a wait has given up anywhere (the host's error word).  The clock is looked at every 256th time: read every time it
// cost a prompt of 512 tokens 26 of 2226 us.
#define XP_WAIT_NS 1000000000ull
__device__ __forceinline__ bool xp_wait(unsigned bar, unsigned parity, const unsigned *err) {
    unsigned long long t0 = 0;
    for (unsigned i = 1;; i++) {
        unsigned ok;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (i & 255u) continue;
        const unsigned long long t = gtime_ns();
        if (!t0) t0 = t;
        if (t - t0 > XP_WAIT_NS || *reinterpret_cast<const volatile unsigned *>(err)) return false;
    }
}
__device__ __forceinline__ void xp_load4(unsigned dst, const CUtensorMap *map, int x, int seg, int group, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst), "l"(map), "r"(x), "r"(0), "r"(seg),
                 "r"(group), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ xp_f2 xp_lds64(unsigned a) {
    xp_f2 r;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(r) : "r"(a));
    return r;
}

template <int MODE, int NJ>
__global__ void __launch_bounds__(XP_THREADS + 32, XpTile<NJ>::RESIDENT) k_xp_gemm(const __grid_constant__ XpMaps map_w, const __grid_constant__ XpMaps map_a, TileMat W, int lds, int n, float *__restrict__ out, int ldo,
                                                        int8_t *__restrict__ HQ, __half *__restrict__ HH, float *__restrict__ HS, XpLast last, float one_f, int stages, unsigned *err) {
    using T = XpTile<NJ>;
    static_assert(T::HV <= XP_STAGES * T::STAGE, "the gate/up epilogue's rows take the ring's place");
    constexpr int TOK = T::TOK, MI = NJ >= 4 ? 2 : 1, NW = NJ / MI; // a warp's tile: 16 MI rows x 8 NW tokens
    extern __shared__ unsigned char smraw[];
    unsigned char *const ring = reinterpret_cast<unsigned char *>(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023); // (the swizzle is by address)
    const unsigned smb = smem_u32(ring), full0 = smb + stages * T::STAGE, empty0 = full0 + 8 * stages;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = blockIdx.x * XP_ROWS, tok0 = blockIdx.y * TOK;
    const int nbs = W.seg >> 5, cps = (nbs + 3) >> 2, n_chunks = W.nseg * cps; // blocks per segment, chunks of <= 4 blocks per segment
    if (tid == 0) {
        for (int s = 0; s < stages; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, XP_THREADS / 32); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == XP_THREADS / 32) { // ---- fetches, by a warp of their own: one of the others that waited for the rest and issued them held the whole CTA up
        if (lane == 0) {
            int c = 0, stage = 0;
            unsigned ph = 1; // (a fresh stage is empty: the wait for the phase before the first one returns at once)
            bool ok = true;
            for (int seg = 0; ok && seg < W.nseg; seg++)
                for (int cs = 0; cs < cps; cs++, c++) {
                    if (!(ok = xp_wait(empty0 + 8 * stage, ph, err))) break;
                    const unsigned s = smb + stage * T::STAGE, bar = full0 + 8 * stage;
                    mbar_expect_tx(bar, T::BYTES_IN);
                    xp_load4(s + T::A_Q, &map_w.q, 128 * cs, seg, row0 >> 2, bar);
                    pg::tma_load_2d(s + T::B_Q, &map_a.q, seg * W.seg + 128 * cs, tok0, bar);
                    xp_load4(s + T::A_S, &map_w.s, W.seg + ((8 * cs) & ~15), seg, row0 >> 2, bar); // 8 scales of a row, 16 bytes
                    pg::tma_load_2d(s + T::B_S, &map_a.s, tok0, seg * nbs + 4 * cs, bar);
                    if (++stage == stages) { stage = 0; ph ^= 1u; }
                }
            // Nothing leaves with its copies in flight, whoever gave up: a multiplying warp whose wait did goes on without looking at its stages, and all chunks may be under way by then.
            for (c = min(c, stages); c > 0; c--) { // (the newest first: behind it the others have landed too, as a rule)
                if (stage == 0) { stage = stages; ph ^= 1u; }
                xp_wait(full0 + 8 * --stage, ph ^ 1u, err);
            }
        } // (the other lanes are gone, or at the barrier below: held at one of the warp's instead they made the product 1 - 2 % slower)
        if (MODE == XP_GATEUP) { __syncthreads(); __syncthreads(); } // (the epilogue's)
        return;
    }

    xp_f2 acc[MI][NW][2]; // [row tile][token tile][row lane/4 | row lane/4 + 8], tokens 2 (lane % 4), + 1
#pragma unroll
    for (int i = 0; i < MI; i++)
#pragma unroll
        for (int j = 0; j < NW; j++) acc[i][j][0] = acc[i][j][1] = 0ull;
    const xp_f2 one = xp_pack(one_f, one_f);
    const int wrow = (warp % (4 / MI)) * 16 * MI, wtok = (warp / (4 / MI)) * 8 * NW; // the warp's first row and token in the tile
    const int ar = wrow + (lane & 15), ap = lane >> 4;                              // ldmatrix: A row, 16-byte half
    const int bt = wtok + (NW > 1 ? ((lane >> 4) << 3) + (lane & 7) : (lane & 7)), bp = (lane >> 3) & 1; // B token (of 16), half
    const unsigned a_base = T::A_Q + ar * 128, b_base = T::B_Q + bt * 128, as_base = T::B_S + (wtok + 2 * (lane & 3)) * 4, ws_base = T::A_S + (wrow + (lane >> 2)) * 16;
    int stage = 0, c_in_seg = 0;
    unsigned ph = 0;
    bool ok = true;
    for (int c = 0; c < n_chunks; c++) {
        if (!(ok = __all_sync(0xffffffffu, xp_wait(full0 + 8 * stage, ph, err)))) break;
        const unsigned s = smb + stage * T::STAGE;
        __half2 ws[MI][2][2]; // scales of blocks {0, 1}, {2, 3}
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const xp_f2 v = xp_lds64(s + ws_base + (16 * i + 8 * h) * 16 + 8 * (c_in_seg & 1));
                const unsigned lo = (unsigned)v, hi = (unsigned)(v >> 32);
                ws[i][h][0] = *reinterpret_cast<const __half2 *>(&lo);
                ws[i][h][1] = *reinterpret_cast<const __half2 *>(&hi);
            }
        const int blocks = min(4, nbs - 4 * c_in_seg);
        auto block = [&](const int k) {
            unsigned a[MI][4];
            xp_f2 wp[MI][2];
#pragma unroll
            for (int i = 0; i < MI; i++) {
                xp_ldsm4(a[i], s + a_base + i * 2048 + (((2 * k + ap) ^ (ar & 7)) << 4));
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const float w = k & 1 ? __high2float(ws[i][h][k >> 1]) : __low2float(ws[i][h][k >> 1]);
                    wp[i][h] = xp_pack(w, w);
                }
            }
#pragma unroll
            for (int j = 0; j < NW; j += 2) {
                unsigned b[4]; // two token tiles (NW == 1: the second one is the first again)
                xp_ldsm4(b, s + b_base + j * 1024 + (((2 * k + bp) ^ (bt & 7)) << 4));
#pragma unroll
                for (int jj = 0; jj < (NW > 1 ? 2 : 1); jj++) {
                    const xp_f2 as = xp_lds64(s + as_base + (k * TOK + (j + jj) * 8) * 4);
#pragma unroll
                    for (int i = 0; i < MI; i++) {
                        int d0, d1, d2, d3;
                        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                                     : "=r"(d0), "=r"(d1), "=r"(d2), "=r"(d3)
                                     : "r"(a[i][0]), "r"(a[i][1]), "r"(a[i][2]), "r"(a[i][3]), "r"(b[2 * jj]), "r"(b[2 * jj + 1]), "r"(0));
                        const xp_f2 f0 = xp_pack((float)d0, (float)d1), f1 = xp_pack((float)d2, (float)d3);
                        xp_f2(&ac)[2] = acc[i][j + jj];
                        ac[0] = xp_fma2(ac[0], one, xp_mul2(f0, xp_mul2(wp[i][0], as)));
                        ac[1] = xp_fma2(ac[1], one, xp_mul2(f1, xp_mul2(wp[i][1], as)));
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
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + 8 * stage);
        if (++stage == stages) { stage = 0; ph ^= 1u; }
        if (++c_in_seg == cps) c_in_seg = 0;
    }
    if (!ok && lane == 0) *reinterpret_cast<volatile unsigned *>(err) = 200u; // (a wait gave up: the host is told)

    const int r0 = wrow + (lane >> 2), t0 = wtok + 2 * (lane & 3);
    if (MODE == XP_GATEUP) { // rows of a group: gate 2G, gate 2G + 1, up 2G, up 2G + 1; the CTA's 64 rows are one 32-unit block of the hidden row
        __syncthreads(); // (every fetch has landed: the fetching warp is here behind its last one)
        float *hv = reinterpret_cast<float *>(ring);
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int j = 0; j < NW; j++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float v0, v1; // lanes with a gate row finish the first token, those with its up row the second
                    xp_unpack(acc[i][j][h], v0, v1);
                    const bool up = (lane >> 2) & 2;
                    const float o = __shfl_xor_sync(0xffffffffu, up ? v0 : v1, 8);
                    const int row = r0 + 16 * i + 8 * h, unit = (row >> 2) * 2 + (row & 1), t = t0 + j * 8 + (up ? 1 : 0);
                    hv[t * 33 + unit] = swiglu_exact(up ? o : v0, up ? v1 : o);
                }
        __syncthreads();
        const int hidden = W.rows >> 1;
        for (int t = warp; t < TOK && tok0 + t < n; t += XP_THREADS / 32) {
            const float v = hv[t * 33 + lane];
            float as;
            const int q = quant_block_lane(v, as);
            if (HH) HH[(size_t)(tok0 + t) * hidden + blockIdx.x * 32 + lane] = __int2half_rn((int8_t)q);
            else HQ[(size_t)(tok0 + t) * hidden + blockIdx.x * 32 + lane] = (int8_t)q;
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
                float v0, v1;
                xp_unpack(acc[i][j][h], v0, v1);
                if (row < W.rows) {
                    float *o = out + (size_t)t * ldo + row;
                    if (t < n) o[0] = MODE == XP_RESID ? __fadd_rn(o[0], v0) : v0;
                    if (t + 1 < n) o[ldo] = MODE == XP_RESID ? __fadd_rn(o[ldo], v1) : v1;
                }
            }
}

// The tile-major matrix as {column of a segment, slot of a group, segment, group}: a box is 128 bytes of quants, or 16 of scales, of one segment in `rows`
// rows.  Behind the segment's last column a box of quants holds scales: blocks that are not multiplied.
inline int xp_map_weights(XpMaps *maps, const TileMat &W, int rows) {
    pg::EncodeTiledFn fn = pg::encode_fn();
    if (!fn) return -1;
    cuuint64_t dims[4] = {(cuuint64_t)W.unit_bytes, 4, (cuuint64_t)W.nseg, (cuuint64_t)(W.rows / 4)};
    cuuint64_t strides[3] = {(cuuint64_t)W.unit_bytes, (cuuint64_t)W.unit_bytes * 4, (cuuint64_t)W.unit_bytes * 4 * W.nseg};
    cuuint32_t box[4] = {128, 4, 1, (cuuint32_t)rows / 4}, sbox[4] = {16, 4, 1, (cuuint32_t)rows / 4}, estr[4] = {1, 1, 1, 1};
    void *base = const_cast<unsigned char *>(W.base);
    const CUresult q = fn(&maps->q, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    const CUresult s = fn(&maps->s, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, base, dims, strides, sbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return q == CUDA_SUCCESS && s == CUDA_SUCCESS ? 0 : -2;
}
// activations [rows][cols] (int8: boxes of 128 columns x the tile's tokens; FP16: of 64 columns) and their scales [blocks][lds] (boxes of the tile's tokens x 4
// blocks), from token `first` on
inline int xp_map_acts(XpMaps *maps, const void *q, bool halves, const float *s, int lds, int cols, int nt, int first = 0) {
    const int rows = lds - first;
    q = static_cast<const int8_t *>(q) + (size_t)first * cols * (halves ? 2 : 1);
    s += first;
    pg::EncodeTiledFn fn = pg::encode_fn();
    if (!fn) return -1;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)cols * (halves ? 2 : 1)}, sdims[2] = {(cuuint64_t)rows, (cuuint64_t)cols / 32}, sstrides[1] = {(cuuint64_t)lds * 4};
    cuuint32_t box[2] = {halves ? 64u : 128u, (cuuint32_t)nt}, sbox[2] = {(cuuint32_t)nt, 4}, estr[2] = {1, 1};
    const CUresult rq = fn(&maps->q, halves ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(q), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    const CUresult rs = fn(&maps->s, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(s), sdims, sstrides, sbox, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return rq == CUDA_SUCCESS && rs == CUDA_SUCCESS ? 0 : -2;
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
                                                                 int n, int start_pos, float sqrt_hs, int8_t *__restrict__ AQ, __half *__restrict__ AH, float *__restrict__ AS, int lds, float *scratch, XpLast last) {
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
            if (AH) AH[(size_t)(q0 + r) * qd + h * HS + blk * 32 + lane] = __int2half_rn((int8_t)q);
            else AQ[(size_t)(q0 + r) * qd + h * HS + blk * 32 + lane] = (int8_t)q;
            if (lane == 0) AS[(size_t)(h * (HS / 32) + blk) * lds + q0 + r] = as;
            if (q0 + r == n - 1) {
                last.xq[h * HS + blk * 32 + lane] = (int8_t)q;
                if (lane == 0) last.xs[h * (HS / 32) + blk] = as;
            }
        }
    }
}
