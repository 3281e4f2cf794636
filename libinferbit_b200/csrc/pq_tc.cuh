// The product-quantised matvec on the tensor cores (pq_tc.cu), as pq.cu calls it.
#pragma once
#include "common.cuh"

constexpr int IBCU_PQ_TC_ERR = 200;            // error codes of a launch that gave up a bounded wait: this + the wait; its accumulators are not zero then

// acc, arrive: as the kernels of pq.cu leave them (zero between calls); max_counters: how many counters arrive has; amax_bits: room
// for 32 words; image: ibcu_pq_tc_image_bytes(t, B) bytes for the activations' operand image, 16-byte aligned. IBCU_DECLINED:
// not a tensor for this kernel, nothing has been launched.
int ibcu_pq_tc(ibcu_ctx* ctx, const ibcu_pq_t* t, const float* x, float* out, int out_stride, int B, bool l1_only, unsigned long long* acc, unsigned* arrive, int max_counters,
               unsigned* amax_bits, void* image);
size_t ibcu_pq_tc_image_bytes(const ibcu_pq_t* t, int B);

// Largest bit pattern of |x| that thread `tid` of T meets among n values (patterns of non-negative floats order like the floats,
// NaN and Inf sort last). U loads travel together whatever n is: a loop left to the compiler's unrolling takes what is over
// its multiple of eight one by one, and 14336 values are seven rounds of 512 threads.
template <int T, int U = 8>
__device__ __forceinline__ unsigned pq_absmax_bits(const float* xb, const int* inner, int n, bool vec, int tid) {
    unsigned m = 0u;
    if (vec) {
        const uint4* x4 = reinterpret_cast<const uint4*>(xb);
        for (int j0 = tid; j0 < (n >> 2); j0 += U * T) {
            uint4 v[U];
#pragma unroll
            for (int u = 0; u < U; u++) v[u] = j0 + u * T < (n >> 2) ? x4[j0 + u * T] : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int u = 0; u < U; u++) m = max(max(m, v[u].x & 0x7fffffffu), max(max(v[u].y & 0x7fffffffu, v[u].z & 0x7fffffffu), v[u].w & 0x7fffffffu));
        }
        return m;
    }
    for (int j0 = tid; j0 < n; j0 += U * T) {
        unsigned v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {                         // past the end: the last value again, so that no load waits for a test
            const int j = min(j0 + u * T, n - 1);
            v[u] = __float_as_uint(xb[inner ? inner[j] : j]) & 0x7fffffffu;
        }
#pragma unroll
        for (int u = 0; u < U; u++) m = max(m, v[u]);
    }
    return m;
}
