// exact_prefill_umma.cuh -- the product of the exact Q8_0 prefill (exact_prefill.cuh) for chunks of many tokens, on tcgen05.
//
// out[token][row] = sum over 32-blocks, strictly in block order, of (float)isum * (wScale * aScale), each operation rounded (Q8_0FloatTensor.java:90-123).  Both factors of a
// block come out of the tensor cores as floats, for 128 tokens (TMEM lanes) x N weight rows (TMEM columns) at a time:
//   F = (float)isum      kind::f16, K = 2 x 16: quants are FP16 numbers, their products and the sum (at most 32 * 128 * 127 < 2^19) are exact in FP32;
//   S = wScale * aScale  kind::f16, K = 16 of which one column is not zero: a single product of two 11-bit numbers, exact in FP32.
// The CUDA cores are left with a product and an ordered add for every (token, row, block).  F and S of a block are 2 N of the 512 columns: while eight warps add up one block,
// the tensor cores are on the next.
//
// Bound by: the sums.  Two warps a scheduler; a step of 16 columns (two tcgen05.ld, a wait, 8 packed products and 8 packed adds) takes 95 cycles and a block about 220 besides, in
// which its barrier is waited for and handed back: 600 cycles for N = 128 (FMA pipe 50 %, tensor pipe 32 %).  Measured, 512 tokens, 8B layer: W2 149 us, Wo 53, QKV 82,
// gate/up 303 (185, 60, 86 and 328 us with mma.sync, k_xp_gemm, which converts, multiplies twice and adds).  Without effect (gate/up 296 - 360 us): 12 and 16 warps of
// 32 columns, 8 or 32 columns a step, the next step's columns loaded ahead, all columns loaded at once (setmaxnreg), neither conversion nor scale products; kind::i8 and a
// conversion in the sums 335 us; one warp that did not walk together for the products 434 us.
//
// Warps: 0-7 sums (warp w: lanes 32 (w % 4) .., columns (w / 4) N / 2 ..), 8-11 turn a stage's bytes into FP16 operands (thread = weight row) and its scales into S's operands
// (one column of a zeroed tile), 12 TMA, 13 MMA.
#pragma once
#include "exact_prefill.cuh"

#define XT_SUM_WARPS 8
#define XT_THREADS (32 * (XT_SUM_WARPS + 6))
#define XT_TOK 128
#define XT_BOX 16     // weight rows of a fetch
#define XT_W_STAGES 3 // weights as bytes and both scales, 128 columns; activations (FP16): two stages of 128 columns; weights as FP16: two of 64 columns
template <int N> struct XtSmem {
    static constexpr int W_Q = 0, W_S = N * 128, A_S = W_S + N * 16, W_BYTES = A_S + 4 * XT_TOK * 4, W_STAGE = (W_BYTES + 1023) & ~1023;
    static constexpr int A_TILE = XT_TOK * 128, A_STAGE = 2 * A_TILE, H_STAGE = N * 128, S_STAGE = (XT_TOK + N) * 128; // tiles of 64 FP16 columns; S: four blocks of 16 columns
    static constexpr int O_W = 0, O_A = O_W + XT_W_STAGES * W_STAGE, O_H = O_A + 2 * A_STAGE, O_S = O_H + 2 * H_STAGE, BYTES = 1024 + O_S + 2 * S_STAGE;
    static_assert(N % 32 == 0 && N <= 128 && H_STAGE % 1024 == 0 && BYTES <= 227 * 1024, "tiles are swizzled by address");
};

__device__ __forceinline__ void xt_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
                   "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void xt_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// xp_wait for a whole warp
__device__ __forceinline__ bool xt_wait(unsigned bar, unsigned parity, const unsigned *err) {
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
    if (__all_sync(0xffffffffu, ok)) return true;
    return __all_sync(0xffffffffu, xp_wait(bar, parity, err));
}

template <int MODE, int N>
__global__ void __launch_bounds__(XT_THREADS, 1) k_xt_gemm(const __grid_constant__ XpMaps map_w, const __grid_constant__ XpMaps map_a, TileMat W, int n, float *__restrict__ out, int ldo,
                                                           float one_f, unsigned *err) {
    using T = XtSmem<N>;
    constexpr int C = N / 2; // a summing warp's columns
    extern __shared__ unsigned char smraw[];
    unsigned char *const sm = reinterpret_cast<unsigned char *>(((uintptr_t)smraw + 1023) & ~(uintptr_t)1023);
    const unsigned smb = smem_u32(sm);
    __shared__ __align__(8) unsigned long long bars[2 * XT_W_STAGES + 13];
    __shared__ uint32_t tmem_slot;
    const unsigned wfull0 = smem_u32(bars), wempty0 = wfull0 + 8 * XT_W_STAGES, afull0 = wempty0 + 8 * XT_W_STAGES, aempty0 = afull0 + 16, hfull0 = aempty0 + 16, hempty0 = hfull0 + 16,
                   tfull0 = hempty0 + 16, tempty0 = tfull0 + 16, fin = tempty0 + 16;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0); // (the same in every lane: so are the addresses made from it)
    const int nbs = W.seg >> 5, cps = (nbs + 3) >> 2, n_chunks = W.nseg * cps; // blocks per segment, chunks of <= 4 blocks
    const int m_tiles = (n + XT_TOK - 1) / XT_TOK, tiles = m_tiles * ((W.rows + N - 1) / N);

    if (tid == 0) {
        for (int s = 0; s < XT_W_STAGES; s++) { mbar_init(wfull0 + 8 * s, 1); mbar_init(wempty0 + 8 * s, 4); }
        for (int s = 0; s < 2; s++) {
            mbar_init(afull0 + 8 * s, 1); mbar_init(aempty0 + 8 * s, 1);
            mbar_init(hfull0 + 8 * s, 4); mbar_init(hempty0 + 8 * s, 1);
            mbar_init(tfull0 + 8 * s, 1); mbar_init(tempty0 + 8 * s, XT_SUM_WARPS);
        }
        mbar_init(fin, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == XT_SUM_WARPS + 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < 2 * T::S_STAGE / 16; i += XT_THREADS) reinterpret_cast<uint4 *>(sm + T::O_S)[i] = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    if (warp < XT_SUM_WARPS) { // ---- ordered sums
        const int quarter = warp & 3, cg = warp >> 2, n_blocks = nbs * W.nseg;
        const uint32_t tb = tmem + ((uint32_t)(quarter * 32) << 16) + cg * C;
        const xp_f2 one = xp_pack(one_f, one_f);
        int buf = 0;
        unsigned ph = 0;
        bool ok = true;
        auto block_ready = [&]() {
            ok = xt_wait(tfull0 + 8 * buf, ph, err);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            return ok;
        };
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
            const int t = tile % m_tiles * XT_TOK + quarter * 32 + lane, row0 = tile / m_tiles * N + cg * C;
            xp_f2 acc[C / 2];
#pragma unroll
            for (int i = 0; i < C / 2; i++) acc[i] = 0ull;
            for (int b = 0; b < n_blocks; b++) {
                if (!block_ready()) break;
                const uint32_t at = tb + buf * 2 * N;
#pragma unroll
                for (int c = 0; c < C; c += 16) {
                    uint32_t F[16], S[16];
                    xt_ld16(at + c, F);
                    xt_ld16(at + N + c, S);
                    xt_wait_ld();
                    if (c + 16 == C) { // the columns go back before the last of the sums
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(tempty0 + 8 * buf);
                        if (++buf == 2) { buf = 0; ph ^= 1u; }
                    }
#pragma unroll
                    for (int i = 0; i < 8; i++)
                        acc[c / 2 + i] = xp_fma2(acc[c / 2 + i], one, xp_mul2(xp_pack(__uint_as_float(F[2 * i]), __uint_as_float(F[2 * i + 1])),
                                                                              xp_pack(__uint_as_float(S[2 * i]), __uint_as_float(S[2 * i + 1]))));
                }
            }
            if (!ok) break;
            if (t < n) {
#pragma unroll
                for (int i = 0; i < C; i += 4) {
                    const int row = row0 + i;
                    if (row >= W.rows) break;
                    float4 v, *o = reinterpret_cast<float4 *>(out + (size_t)t * ldo + row);
                    xp_unpack(acc[i / 2], v.x, v.y);
                    xp_unpack(acc[i / 2 + 1], v.z, v.w);
                    if (MODE == XP_RESID) {
                        const float4 x = *o;
                        v = make_float4(__fadd_rn(x.x, v.x), __fadd_rn(x.y, v.y), __fadd_rn(x.z, v.z), __fadd_rn(x.w, v.w));
                    }
                    *o = v;
                }
            }
        }
        if (!ok && lane == 0) *reinterpret_cast<volatile unsigned *>(err) = 200u;
    } else {
        if (warp == XT_SUM_WARPS + 4) { // ---- fetches
            if (lane == 0) {
                int it = 0, n_w = 0, n_a = 0; // the chunk; chunks whose weights, whose activations are under way or there
                bool ok = true;
                for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
                    const int tok0 = tile % m_tiles * XT_TOK, row0 = tile / m_tiles * N;
                    for (int c = 0, seg = 0, cs = 0; c < n_chunks; c++, it++) {
                        const int ws = it % XT_W_STAGES, as = it & 1;
                        if (it >= XT_W_STAGES && !(ok = xp_wait(wempty0 + 8 * ws, (it / XT_W_STAGES - 1) & 1, err))) break;
                        const unsigned w = smb + T::O_W + ws * T::W_STAGE, wbar = wfull0 + 8 * ws, a = smb + T::O_A + as * T::A_STAGE, abar = afull0 + 8 * as;
                        mbar_expect_tx(wbar, T::W_BYTES);
                        pg::tma_load_2d(w + T::A_S, &map_a.s, tok0, seg * nbs + 4 * cs, wbar);
#pragma unroll
                        for (int r = 0; r < N; r += XT_BOX) {
                            xp_load4(w + T::W_Q + r * 128, &map_w.q, 128 * cs, seg, (row0 + r) >> 2, wbar);
                            xp_load4(w + T::W_S + r * 16, &map_w.s, W.seg + ((8 * cs) & ~15), seg, (row0 + r) >> 2, wbar); // 8 scales of a row, 16 bytes
                        }
                        n_w = it + 1;
                        if (it >= 2 && !(ok = xp_wait(aempty0 + 8 * as, ((it >> 1) - 1) & 1, err))) break;
                        mbar_expect_tx(abar, T::A_STAGE);
                        pg::tma_load_2d(a, &map_a.q, seg * W.seg + 128 * cs, tok0, abar);
                        pg::tma_load_2d(a + T::A_TILE, &map_a.q, seg * W.seg + 128 * cs + 64, tok0, abar);
                        n_a = it + 1;
                        if (++cs == cps) { cs = 0; seg++; }
                    }
                }
                // Nothing leaves with its copies in flight, whoever gave up: the others go to the block's last barrier without looking at their stages.
                for (int q = max(0, n_w - XT_W_STAGES); q < n_w; q++) xp_wait(wfull0 + 8 * (q % XT_W_STAGES), (q / XT_W_STAGES) & 1, err);
                for (int q = max(0, n_a - 2); q < n_a; q++) xp_wait(afull0 + 8 * (q & 1), (q >> 1) & 1, err);
            }
        } else if (warp == XT_SUM_WARPS + 5) { // ---- products: the warp walks together (addresses and phases stay in uniform registers), one lane issues
            constexpr uint32_t idesc = pg::umma_idesc_f16(XT_TOK, N);
            uint32_t lead;
            asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(lead));
            int as = 0, h = 0, buf = 0;
            unsigned ph_a = 0, ph_h = 0, ph_t = 1; // (a fresh buffer is empty: the wait for the phase before the first one returns at once)
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x)
                for (int c = 0, cs = 0; ok && c < n_chunks; c++) {
                    const int blocks = min(4, nbs - 4 * cs);
                    if (!(ok = xt_wait(afull0 + 8 * as, ph_a, err))) break;
                    const unsigned sc = smb + T::O_S + as * T::S_STAGE; // (a chunk's S operands sit in the buffer of the same parity as its activations)
                    const uint64_t s_a = pg::umma_desc_sw128(sc), s_w = pg::umma_desc_sw128(sc + XT_TOK * 128);
#pragma unroll
                    for (int half = 0; half < 2; half++) {
                        if (2 * half >= blocks) break;
                        if (!(ok = xt_wait(hfull0 + 8 * h, ph_h, err))) break;
                        const uint64_t f_a = pg::umma_desc_sw128(smb + T::O_A + as * T::A_STAGE + half * T::A_TILE), f_w = pg::umma_desc_sw128(smb + T::O_H + h * T::H_STAGE);
#pragma unroll
                        for (int i = 0; i < 2; i++) {
                            const int b = 2 * half + i;
                            if (b >= blocks) break;
                            if (!(ok = xt_wait(tempty0 + 8 * buf, ph_t, err))) break;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            const uint32_t d = tmem + buf * 2 * N;
                            if (lead) {
                                pg::umma_f16(d, f_a + 4 * i, f_w + 4 * i, idesc, 0u);
                                pg::umma_f16(d, f_a + 4 * i + 2, f_w + 4 * i + 2, idesc, 1u);
                                pg::umma_f16(d + N, s_a + 2 * b, s_w + 2 * b, idesc, 0u);
                                pg::umma_commit(tfull0 + 8 * buf);
                            }
                            if (++buf == 2) { buf = 0; ph_t ^= 1u; }
                        }
                        if (!ok) break;
                        if (lead) pg::umma_commit(hempty0 + 8 * h);
                        if (++h == 2) { h = 0; ph_h ^= 1u; }
                    }
                    if (!ok) break;
                    if (lead) pg::umma_commit(aempty0 + 8 * as);
                    if (++as == 2) { as = 0; ph_a ^= 1u; }
                    if (++cs == cps) cs = 0;
                }
            if (lead) { // no columns go back with products in flight, whoever gave up
                if (!ok) *reinterpret_cast<volatile unsigned *>(err) = 200u;
                pg::umma_commit(fin);
                xp_wait(fin, 0, err);
            }
            __syncwarp();
        } else if (warp < XT_SUM_WARPS + 4) { // ---- operands
            const int r = tid - XT_SUM_WARPS * 32; // weight row, and token
            int ws = 0, h = 0, sb = 0;
            unsigned ph_w = 0, ph_h = 1;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x)
                for (int c = 0, cs = 0; ok && c < n_chunks; c++) {
                    const int blocks = min(4, nbs - 4 * cs);
                    if (!(ok = xt_wait(wfull0 + 8 * ws, ph_w, err))) break;
                    const unsigned char *src = sm + T::O_W + ws * T::W_STAGE;
#pragma unroll
                    for (int half = 0; half < 2; half++) {
                        if (2 * half >= blocks) break;
                        uint4 q[4];
#pragma unroll
                        for (int i = 0; i < 4; i++)
                            if (r < N) q[i] = *reinterpret_cast<const uint4 *>(src + T::W_Q + r * 128 + (((4 * half + i) ^ (r & 7)) << 4));
                        if (!(ok = xt_wait(hempty0 + 8 * h, ph_h, err))) break;
                        unsigned char *dst = sm + T::O_H + h * T::H_STAGE + r * 128;
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            if (r >= N) break;
                            uint4 lo, hi;
                            xp_halves(q[i].x, lo.x, lo.y);
                            xp_halves(q[i].y, lo.z, lo.w);
                            xp_halves(q[i].z, hi.x, hi.y);
                            xp_halves(q[i].w, hi.z, hi.w);
                            *reinterpret_cast<uint4 *>(dst + (((2 * i) ^ (r & 7)) << 4)) = lo;
                            *reinterpret_cast<uint4 *>(dst + (((2 * i + 1) ^ (r & 7)) << 4)) = hi;
                        }
                        if (half == 0) { // the chunk's scales (products of the chunk before the last one, which had this buffer, are done: so are those of the half before the last)
                            unsigned char *a = sm + T::O_S + sb * T::S_STAGE + r * 128, *w = a + XT_TOK * 128;
                            const float *as = reinterpret_cast<const float *>(src + T::A_S) + r;
                            uint2 v = make_uint2(0u, 0u);
                            if (r < N) v = *reinterpret_cast<const uint2 *>(src + T::W_S + r * 16 + 8 * (cs & 1));
#pragma unroll
                            for (int b = 0; b < 4; b++) {
                                const int at = ((2 * b) ^ (r & 7)) << 4;
                                *reinterpret_cast<__half *>(a + at) = __float2half_rn(as[b * XT_TOK]); // (the scales are FP16 numbers)
                                if (r < N) *reinterpret_cast<unsigned short *>(w + at) = (unsigned short)((b < 2 ? v.x : v.y) >> (16 * (b & 1)));
                            }
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(hfull0 + 8 * h);
                        if (++h == 2) { h = 0; ph_h ^= 1u; }
                    }
                    if (!ok) break;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(wempty0 + 8 * ws);
                    if (++ws == XT_W_STAGES) { ws = 0; ph_w ^= 1u; }
                    sb ^= 1;
                    if (++cs == cps) cs = 0;
                }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == XT_SUM_WARPS + 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

// ---- hidden units behind the gate/up product: Q8_0(silu(gate) * up), FP16 quants (or bytes) and scales -------------------------------
// A warp takes two blocks of 32 units of a token, a lane two units: G's columns come in groups gate 2g, gate 2g + 1, up 2g, up 2g + 1.  A launch of its own because the double
// precision of the activation would stand between the tiles of the product: 360 us in its epilogue against 303 + 30 us, 512 tokens, 8B layer.  Tokens are the grid's x: y ends at 65535.
__global__ void __launch_bounds__(256) k_xt_swiglu(const float *__restrict__ G, int hidden, int n, int8_t *__restrict__ HQ, __half *__restrict__ HH, float *__restrict__ HS, int lds, XpLast last) {
    const int lane = threadIdx.x & 31, pair = blockIdx.y * 8 + (threadIdx.x >> 5), t = blockIdx.x, unit = pair * 64 + 2 * lane;
    if (pair * 64 >= hidden) return;
    const bool live = unit < hidden; // (an odd number of blocks)
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
    if (live) g = *reinterpret_cast<const float4 *>(G + (size_t)t * 2 * hidden + 2 * unit);
    const float v0 = swiglu_exact(g.x, g.z), v1 = swiglu_exact(g.y, g.w);
    float amax = fmaxf(fabsf(v0), fabsf(v1));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (!live) return;
    const float qs = __fdiv_rn(amax, 127.0f), as = __half2float(__float2half_rn(qs)), ainv = qs != 0.0f ? __fdiv_rn(1.0f, qs) : 0.0f; // quant_block_lane's arithmetic
    const float s0 = __fmul_rn(v0, ainv), s1 = __fmul_rn(v1, ainv);
    const int q0 = __float2int_rz(__fadd_rn(s0, copysignf(0.5f, s0))), q1 = __float2int_rz(__fadd_rn(s1, copysignf(0.5f, s1)));
    const char2 q = make_char2((char)q0, (char)q1);
    if (HH) *reinterpret_cast<__half2 *>(HH + (size_t)t * hidden + unit) = __halves2half2(__int2half_rn(q.x), __int2half_rn(q.y));
    else *reinterpret_cast<char2 *>(HQ + (size_t)t * hidden + unit) = q;
    if ((lane & 15) == 0) HS[(size_t)(unit >> 5) * lds + t] = as;
    if (t == n - 1) {
        *reinterpret_cast<float2 *>(last.hb + unit) = make_float2(v0, v1);
        *reinterpret_cast<char2 *>(last.hq + unit) = q;
        if ((lane & 15) == 0) last.hs[unit >> 5] = as;
    }
}
