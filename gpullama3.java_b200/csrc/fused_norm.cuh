// fused_norm.cuh -- the RMSNorm in front of a decode matvec, computed by every CTA of the matvec for itself.
//
// As a kernel of its own (k_rmsnorm_quant) the norm was one CTA on an otherwise waiting GPU: 11.3 us at 4096 entries, 65 times per token of an 8B
// model, plus a kernel boundary and the round trip of the normalised row through L2.  Inside the matvec its rows of weights are already on
// their way into the shared-memory ring meanwhile, the 16 KB of x come from L2, the row goes straight to the shared memory that the products read,
// and the sum is seqsum3.cuh's.  What bounds it is the latency of its chain (load 1,300, prefix and classes
// 1,900, walk 4,100, square root 300, quantisation 700 SM cycles at 4096 entries).  Decode step of two layers: 8B Q8_0 249 -> 212 us, 1B FP16 223 -> 200 us, a toy model
// 123 -> 100 us.
//
// InferenceCore.rmsnorm (InferenceCore.java:39-48): ss = sequential sum of x*x; ss = ss / size + eps; ss = (float)(1.0 / Math.sqrt(ss)); out = w * (ss * x).
#pragma once
#include "decode_kernels.cuh"

struct NormIn { // x == nullptr: the kernel takes a finished activation
    const float *x;      // residual stream
    const float *w;
    float eps;
    int embed;           // 1: the row is the embedding of st->token, and CTA 0 leaves it in x_out
    float *x_out;
    DevMat emb;
    const StepState *st;
    int8_t *xq;          // CTA 0's copy of the result, for read-back (Q8_0: quants and scales; FP16: floats)
    float *xs, *xb;
};
// Terms per thread of the 256: a power of two, so that a quantisation block of 32 is 32 / E neighbouring lanes.
__host__ __device__ constexpr int norm_terms(int dim) { return dim <= 1024 ? 4 : dim <= 2048 ? 8 : dim <= 4096 ? 16 : 32; }

// Threads [0, 256); tid * E is the thread's first entry.  Returns the scale in every thread and the entries in x; sq: 256 * E floats of shared memory.
// w (immutable) is requested before the wait for the kernel in front when the registers allow it.
template <int E, class Sync>
__device__ __forceinline__ float norm_scale(const NormIn &in, int dim, float (&x)[E], float *sq, SeqSum3Scratch &sc, int tid, Sync sync) {
    const int base = tid * E;
    const bool live = base < dim; // dim is a multiple of 32
    if (in.embed) {
        const int token = in.st->token;
#pragma unroll
        for (int k = 0; k < E; k++) {
            x[k] = live ? emb_get(in.emb, token, base + k) : 0.0f;
            if (live && blockIdx.x == 0) in.x_out[base + k] = x[k];
        }
    } else {
#pragma unroll
        for (int k = 0; k < E; k += 4) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live) v = __ldcg(reinterpret_cast<const float4 *>(in.x + base + k));
            x[k] = v.x; x[k + 1] = v.y; x[k + 2] = v.z; x[k + 3] = v.w;
        }
    }
    float t[E];
#pragma unroll
    for (int k = 0; k < E; k++) t[k] = __fmul_rn(x[k], x[k]);
#pragma unroll
    for (int k = 0; k < E; k += 4) *reinterpret_cast<float4 *>(sq + base + k) = make_float4(t[k], t[k + 1], t[k + 2], t[k + 3]);
    float ss = block_seqsum3<E>(t, sq, sc, tid, sync);
    ss = __fdiv_rn(ss, (float)dim);
    ss = __fadd_rn(ss, in.eps);
    return (float)(1.0 / sqrt((double)ss));
}
template <int E> __device__ __forceinline__ void norm_weights(const NormIn &in, int dim, float (&w)[E], int tid) {
#pragma unroll
    for (int k = 0; k < E; k += 4) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tid * E < dim) v = __ldg(reinterpret_cast<const float4 *>(in.w + tid * E + k));
        w[k] = v.x; w[k + 1] = v.y; w[k + 2] = v.z; w[k + 3] = v.w;
    }
}
// Q8_0 quantisation of the thread's E entries (quant_block_lane's arithmetic); a block is 32 / E neighbouring lanes.  dq / ds: shared memory.
template <int E> __device__ __forceinline__ void norm_quantise(const NormIn &in, int dim, const float (&v)[E], int8_t *dq, float *ds, int tid) {
    constexpr int TPB = 32 / E;
    float amax = 0.0f;
#pragma unroll
    for (int k = 0; k < E; k++) amax = fmaxf(amax, fabsf(v[k]));
#pragma unroll
    for (int o = TPB / 2; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float qs = __fdiv_rn(amax, 127.0f);
    const float as = __half2float(__float2half_rn(qs));
    const float ainv = qs != 0.0f ? __fdiv_rn(1.0f, qs) : 0.0f;
    const int base = tid * E;
    if (base >= dim) return;
    unsigned pk[E / 4];
#pragma unroll
    for (int k = 0; k < E; k += 4) {
        unsigned p = 0;
#pragma unroll
        for (int b = 0; b < 4; b++) {
            const float s = __fmul_rn(v[k + b], ainv);
            p |= ((unsigned)__float2int_rz(__fadd_rn(s, copysignf(0.5f, s))) & 0xffu) << (8 * b);
        }
        pk[k / 4] = p;
    }
#pragma unroll
    for (int k = 0; k < E / 4; k++) reinterpret_cast<unsigned *>(dq + base)[k] = pk[k];
    if (tid % TPB == 0) ds[base / 32] = as;
    if (blockIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < E / 4; k++) reinterpret_cast<unsigned *>(in.xq + base)[k] = pk[k];
        if (tid % TPB == 0) in.xs[base / 32] = as;
    }
}

// Test hook: the sum alone, on arbitrary non-negative terms.
struct NormTestSync { __device__ __forceinline__ void operator()() const { __syncthreads(); } };
template <int E>
__global__ void __launch_bounds__(SEQSUM3_THREADS) k_test_seqsum3(const float *__restrict__ terms, int n, float *__restrict__ out, int *__restrict__ info) {
    __shared__ __align__(16) float sq[SEQSUM3_THREADS * E];
    __shared__ SeqSum3Scratch scratch;
    const int tid = threadIdx.x;
    float t[E];
#pragma unroll
    for (int k = 0; k < E; k++) {
        const int i = tid * E + k;
        t[k] = i < n ? terms[i] : 0.0f;
        sq[i] = t[k];
    }
    const float s = block_seqsum3<E>(t, sq, scratch, tid, NormTestSync());
    if (tid == 0) { out[0] = s; info[0] = scratch.info[0]; info[1] = scratch.info[1]; }
}
