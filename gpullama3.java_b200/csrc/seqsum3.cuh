// seqsum3.cuh -- the exact sequential float sum of the norms that the decode matvecs compute themselves (same contract as seqsum.cuh and
// seqsum2.cuh: the bit-exact value of  s = 0; for (i) s = s + t[i]  for non-negative float terms, InferenceCore.java:39-48).
//
// 256 threads with E consecutive terms each, the terms in registers (and, for the replays, in shared memory).  What is different from
// seqsum2.cuh, whose 1024 threads spend most of their time in barriers and in the scan of composed pairs:
//   * inside one binade a term that is not an exact tie adds the same integer whatever the parity of the sum, so a thread without ties needs ONE
//     integer (the sum of its rounded terms) and the scan over a run is an integer prefix sum; a thread with a tie is replayed literally (a few
//     of 256: a tie needs the dropped bits to be exactly 100..0);
//   * the walk works on the float's bits: within a binade they ARE the integer, and one shift-compare checks that the binade was not left; the items and the terms
//     of literal threads are fetched one and two items ahead, so that an item costs its own few dependent operations and no shared-memory round trip
//     (without that a walk of 32 items took 9,360 of 13,900 cycles).
// The predictions (a float prefix, margin 2^-9 against n * 2^-24 <= 2^-11 for n <= 8192) decide speed and never the result: a run that does not
// start or end in its binade is replayed literally.
// Measured at 4096 terms (SM cycles): a literal chain 16,400, seqsum2.cuh about 13,000, here 5,900 of which the walk of 32 items is 4,100.
#pragma once
#include "seqsum.cuh"

#define SEQSUM3_THREADS 256
#define SEQSUM3_WARPS 8
struct SeqSum3Scratch {
    float wsum[SEQSUM3_WARPS];
    int wcnt[SEQSUM3_WARPS];
    float result;
    int info[2];               // {items walked, runs replayed}
    int pad;
    int2 items[SEQSUM3_THREADS + 2]; // in order; x = first thread << 16 | last thread << 8 | biased exponent (0: one literal thread), y = the run's integer
};
template <int E> struct SeqSumTerms { static constexpr int value = E; };
// Shared copy of the terms: thread t's E terms start at t * E; a thread's 16-byte pieces are read by one lane at a time (broadcast), so the layout needs no padding.

// t: this thread's E terms (zero behind the last one); sq: all terms in shared memory, written by the caller BEFORE the call (a barrier inside
// orders them); s0: where the sum starts (a long sum comes in pieces); sync: a barrier over the 256 threads.  Every thread returns the sum.
template <int E, class Sync>
__device__ __forceinline__ float block_seqsum3(const float (&t)[E], const float *sq, SeqSum3Scratch &sc, int tid, Sync sync, float s0 = 0.0f) {
    static_assert(E % 4 == 0, "terms move in 16-byte pieces");
    const int lane = tid & 31, warp = tid >> 5;
    // ---- a float prefix over the threads' own sums predicts the binade of every thread
    float loc = 0.0f;
#pragma unroll
    for (int k = 0; k < E; k++) loc += t[k];
    float inc = loc;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const float u = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= d) inc += u;
    }
    if (lane == 31) sc.wsum[warp] = inc;
    sync();
    float before = s0;
#pragma unroll
    for (int w = 0; w < SEQSUM3_WARPS - 1; w++)
        if (w < warp) before += sc.wsum[w];
    const float p_end = before + inc, p_start = before + (inc - loc);
    // ---- the thread's integer inside its binade; no binade: literal
    int be = 0, sum = 0; // biased exponent, integer
    {
        const int e = f32_exponent(p_start);
        if (p_start > 0.0f && e > -100 && e < 127 && f32_exponent(p_end) == e) {
            const float b = __uint_as_float((unsigned)(e + 127) << 23);
            if (p_start >= b * (1.0f + 0x1p-9f) && p_end <= 2.0f * b * (1.0f - 0x1p-9f)) {
                const float scale = __uint_as_float((unsigned)(150 - e) << 23); // 2^(23 - e): a term in units of the sum's last place
                bool ok = true;
#pragma unroll
                for (int k = 0; k < E; k++) {
                    const float f = __fmul_rn(t[k], scale);
                    const float r = __fadd_rn(f, 8388608.0f); // f < 2^23: rounded to the nearest integer, ties to even
                    ok = ok && fabsf(__fsub_rn(f, __fsub_rn(r, 8388608.0f))) != 0.5f;
                    sum += __float_as_int(r) - 0x4B000000;
                }
                if (ok) be = e + 127;
            }
        }
    }
    // ---- items: one per literal thread, one per run of threads of a binade inside a warp
    int prev = __shfl_up_sync(0xffffffffu, be, 1), next = __shfl_down_sync(0xffffffffu, be, 1);
    if (lane == 0) prev = -1;
    if (lane == 31) next = -1;
    int scan = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, scan, d);
        if (lane >= d) scan += u;
    }
    const unsigned starts = __ballot_sync(0xffffffffu, be == 0 || prev != be);
    const bool is_item = be == 0 || next != be;
    const unsigned ends = __ballot_sync(0xffffffffu, is_item);
    const int first = 31 - __clz(starts & (0xffffffffu >> (31 - lane)));
    const int start_excl = __shfl_sync(0xffffffffu, scan - sum, first);
    if (lane == 0) sc.wcnt[warp] = __popc(ends);
    sync();
    int off = 0, n_items = 0;
#pragma unroll
    for (int w = 0; w < SEQSUM3_WARPS; w++) {
        const int c = sc.wcnt[w];
        if (w < warp) off += c;
        n_items += c;
    }
    if (is_item) {
        int2 it;
        it.x = ((warp * 32 + first) << 16) | (tid << 8) | be;
        it.y = scan - start_excl;
        sc.items[off + __popc(ends & ((1u << lane) - 1u))] = it;
    }
    sync();
    // ---- the walk: warp 0, every lane the same (shared-memory broadcasts)
    if (warp == 0) {
        float s = s0;
        int replays = 0;
        int2 it = sc.items[0], nx = sc.items[min(1, n_items - 1)];
        float4 v[E / 4];
        auto terms = [&](const int2 &i, float4 (&q)[E / 4]) {
#pragma unroll
            for (int k = 0; k < E / 4; k++) q[k] = *reinterpret_cast<const float4 *>(sq + (i.x >> 16) * E + 4 * k);
        };
        terms(it, v);
#pragma unroll 2
        for (int i = 0; i < n_items; i++) {
            float4 vn[E / 4];
            terms(nx, vn);
            const int2 nn = sc.items[min(i + 2, n_items - 1)];
            const unsigned sb = __float_as_uint(s), mb = sb + (unsigned)it.y, xe = (unsigned)it.x & 0xffu;
            if (xe != 0u && (sb >> 23) == xe && (mb >> 23) == xe) s = __uint_as_float(mb);
            else if (xe == 0u) { // a literal thread
#pragma unroll
                for (int k = 0; k < E / 4; k++) { s = __fadd_rn(s, v[k].x); s = __fadd_rn(s, v[k].y); s = __fadd_rn(s, v[k].z); s = __fadd_rn(s, v[k].w); }
            } else { // a run that did not stay in its binade: literally
                const float4 *q = reinterpret_cast<const float4 *>(sq + (it.x >> 16) * E);
                const int n4 = (((it.x >> 8) & 0xff) - (it.x >> 16) + 1) * (E / 4);
                replays++;
#pragma unroll 1
                for (int k = 0; k < n4; k++) {
                    const float4 c = q[k];
                    s = __fadd_rn(s, c.x); s = __fadd_rn(s, c.y); s = __fadd_rn(s, c.z); s = __fadd_rn(s, c.w);
                }
            }
            it = nx;
            nx = nn;
#pragma unroll
            for (int k = 0; k < E / 4; k++) v[k] = vn[k];
        }
        if (lane == 0) { sc.result = s; sc.info[0] = n_items; sc.info[1] = replays; }
    }
    sync();
    return sc.result;
}
