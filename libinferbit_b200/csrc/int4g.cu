// Group-scaled INT4 matvec (the INT4 tensors of the reference's session engine, src/pq_decode.c:3474-3483 for the
// layout, :3565-3651 for the arithmetic): two columns per byte (low nibble = even column, value = nibble - 8), one FP16
// scale per row and group of G columns,
//   out[m] = sum over groups g of scale[m][g] * (sum over the group's columns of (nibble - 8) * x[col])
//          + sum over k < K_out of outl_val[m][k] * x[outl_idx[m][k]]          (optional per-row outlier columns),
// with groups whose largest |x| is at most eps * max|x| left out when eps > 0 (build_skip_mask, :3854-3882; off by
// default there). HBM-bound: N/2 bytes of weights and 2 N/G bytes of scales per row, read once.
//
// Both kernels for N and G multiples of 32 use integer arithmetic; int4g_mma_kernel below takes the tensor cores and most calls, int4g_kernel dp4a: outlier
// columns, the skip rule, groups of any other multiple of 32 columns, rows beyond 16384 columns, and what im_pays leaves it.
// int4g_kernel: the activation becomes 32-bit fixed point (2^sh max|x| in
// [2^29, 2^30)), split into four balanced base-256 digits per column ("limbs"), and a row's 32-column chunk is 32 dp4a
// instructions: nibbles as bytes (even columns w & 0x0F0F0F0F, odd columns (w >> 4) & 0x0F0F0F0F) times the limb words of
// the same columns, one int32 sum per limb, exact. The chunk's value sum_k 256^k a_k - 8 sum(X) goes to FP32, times the
// group's scale into the row's sum. Against FP32 FMAs on unpacked nibbles (the first form of this kernel: four
// instructions per weight, 25 us for 14336 x 4096) this is 1.7 instructions per weight.
// The limb words sit in shared memory per chunk as eight 16-byte pieces (piece 2 j + e: limbs 0..3 of the even (e = 0)
// or odd columns of the chunk's j-th group of eight), rotated by chunk % 8 so that lanes reading consecutive chunks hit
// different banks. A warp owns two rows at a time; lane l takes chunks l, l + 32, ...; weights and scales come through a
// ring of asynchronous copies per warp, STAGES - 1 steps ahead of their use. A fixed butterfly adds the lanes. Sums are ordered differently from the
// reference's scalar loop and the activation is rounded to 2^-30 of its largest magnitude: equal to the reference within
// the float bar, not bit for bit; f(2x) = 2 f(x) exactly.
#include "common.cuh"
#include <algorithm>
#include <mutex>

namespace {

constexpr int I4G_THREADS = 256;
constexpr int I4G_WARPS = I4G_THREADS / 32;
constexpr int I4G_ROWS = 2;                                  // rows a warp carries through a pass over the columns
constexpr int I4G_STAGES = 4;                                // steps of a warp's ring of weights in shared memory (a power of two)

struct I4gParams {
    int M, N, G, K_out;
    const uint8_t* q; const __half* s; const uint16_t* outl_idx; const __half* outl_val;
    const float* x; float* out;
    float eps;                                               // > 0: groups with max|x| <= eps * max|x| are left out
};

__device__ __forceinline__ void transpose4x4_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t* o) {
    const uint32_t t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(a, b, 0x7362);
    const uint32_t t2 = __byte_perm(c, d, 0x5140), t3 = __byte_perm(c, d, 0x7362);
    o[0] = __byte_perm(t0, t2, 0x5410); o[1] = __byte_perm(t0, t2, 0x7632);
    o[2] = __byte_perm(t1, t3, 0x5410); o[3] = __byte_perm(t1, t3, 0x7632);
}

template <int ROWS, int STAGES, int HELD>
__global__ void __launch_bounds__(I4G_THREADS) int4g_kernel(const I4gParams p) {
    extern __shared__ __align__(16) uint32_t xl[];           // [N/32 chunks][8 pieces][4 limb words], then chunk sums (float), then skip flags
    __shared__ float red[I4G_WARPS];
    __shared__ float s_mul, s_back;
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nchunk = p.N >> 5, ng = p.N / p.G, cpg = p.G >> 5;     // chunks per group
    // group of a chunk: a shift when a group is a power-of-two number of chunks (runtime divisions in the step loop cost
    // as many instructions as the dot products they index)
    const int cpg_sh = (cpg & (cpg - 1)) == 0 ? 31 - __clz(cpg) : -1;
    auto group_of = [&](int c) { return cpg_sh >= 0 ? c >> cpg_sh : c / cpg; };
    float* sxs = reinterpret_cast<float*>(xl + p.N);
    unsigned char* skip = reinterpret_cast<unsigned char*>(sxs + ((nchunk + 3) & ~3));     // keeps the ring behind it 16-byte aligned
    // ── rows: a warp walks its tiles of ROWS rows, lane l the chunks l, l + 32, ...; (tile, pass over 32 chunks) form one
    //    sequence of steps, and the weights (16 bytes per lane and row) and scales of step q + STAGES - 1 are on their way
    //    into the warp's ring in shared memory while step q is worked on ──
    const uint4* wq = reinterpret_cast<const uint4*>(p.q);
    constexpr int STAGE_WORDS = ROWS * 32 * 5;                // per row 32 lanes x (16 bytes of weights + 4 bytes holding the scale)
    uint32_t* ring = reinterpret_cast<uint32_t*>(skip + ((ng + 15) & ~15)) + (size_t)warp * STAGES * STAGE_WORDS;
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring);
    const int npass = (nchunk + 31) >> 5;
    const int tile0 = blockIdx.x * I4G_WARPS + warp, tstride = gridDim.x * I4G_WARPS;
    const int ntile = (p.M + ROWS - 1) / ROWS;
    const int my_tiles = tile0 < ntile ? (ntile - tile0 + tstride - 1) / tstride : 0;
    const int nstep = my_tiles * npass;
    int iq = 0, ipass = 0, itile = tile0;                     // the step to request next, its pass and its tile
    auto issue = [&]() {                                      // requests the next step (nothing beyond the last: an empty group keeps the count)
        const int q = iq++;
        if (q < nstep) {
            const int tile = itile, c = lane + 32 * ipass;
            if (++ipass == npass) { ipass = 0; itile += tstride; }
            const int g = group_of(c < nchunk ? c : 0);
            const bool on = c < nchunk && !(p.eps > 0.0f && skip[g]);
            const uint32_t dst = ring_s + (uint32_t)((q & (STAGES - 1)) * STAGE_WORDS) * 4u;
#pragma unroll
            for (int u = 0; u < ROWS; u++) {
                const int r = min(tile * ROWS + u, p.M - 1);  // rows past the end repeat the last one and are not stored
                const int cc = on ? c : 0;
                const unsigned nb = on ? 16u : 0u;            // a chunk that is off is filled with zeros: scale 0 times 0
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst + (uint32_t)(u * 32 + lane) * 16u), "l"(wq + (size_t)r * nchunk + cc), "r"(nb) : "memory");
                const uintptr_t sa = (uintptr_t)(p.s + (size_t)r * ng + (on ? g : 0)) & ~(uintptr_t)3;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"(dst + (uint32_t)(ROWS * 32 * 4 + u * 32 + lane) * 4u), "l"(sa), "r"(on ? 4u : 0u) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // weights and scales do not depend on the kernel ahead: without the skip rule the first steps are requested before the wait
    // for it, and travel while the activation is converted
    const bool early = !(p.eps > 0.0f);
    if (early) {
#pragma unroll
        for (int q = 0; q < STAGES - 1; q++) issue();
    }
    pdl_wait();
    // max |x|, then the fixed-point scale: 2^sh max|x| in [2^29, 2^30)
    // Up to HELD groups of eight columns per thread stay in registers from here to the conversion, all loads in flight at once: the
    // block pays one round trip to L2 for its activation instead of one per loop iteration and pass (14336 x 4096: 13.9 -> 13.5 us,
    // 12021 x 3072: 14.1 -> 10.2 us).
    const bool held = (p.N >> 3) <= HELD * I4G_THREADS;
    float4 xa[HELD], xb[HELD];
    float amax = 0.0f;
    if (held) {
#pragma unroll
        for (int u = 0; u < HELD; u++) {
            const int i8 = tid + u * I4G_THREADS;
            xa[u] = xb[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i8 < (p.N >> 3)) { xa[u] = __ldcg(reinterpret_cast<const float4*>(p.x) + 2 * i8); xb[u] = __ldcg(reinterpret_cast<const float4*>(p.x) + 2 * i8 + 1); }
        }
#pragma unroll
        for (int u = 0; u < HELD; u++)
            amax = fmaxf(amax, fmaxf(fmaxf(fmaxf(fabsf(xa[u].x), fabsf(xa[u].y)), fmaxf(fabsf(xa[u].z), fabsf(xa[u].w))),
                                     fmaxf(fmaxf(fabsf(xb[u].x), fabsf(xb[u].y)), fmaxf(fabsf(xb[u].z), fabsf(xb[u].w)))));
    } else {
        for (int i = tid; i < (p.N >> 2); i += I4G_THREADS) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(p.x) + i);
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
        }
    }
    amax = warp_max(amax);
    if (lane == 0) red[warp] = amax;
    __syncthreads();
    amax = red[0];
#pragma unroll
    for (int w = 1; w < I4G_WARPS; w++) amax = fmaxf(amax, red[w]);
    if (tid == 0) {
        const int e = (int)((__float_as_uint(amax) >> 23) & 0xFF);   // amax in [2^(e-127), 2^(e-126))
        int sh = (amax > 0.0f && e != 255) ? 156 - e : 0;
        sh = max(-126, min(126, sh));
        s_mul = __uint_as_float((uint32_t)(127 + sh) << 23);
        s_back = __uint_as_float((uint32_t)(127 - sh) << 23);
    }
    if (p.eps > 0.0f) {
        const float thr = p.eps * amax;
        for (int g = tid; g < ng; g += I4G_THREADS) {
            float gm = 0.0f;
            for (int j = 0; j < p.G; j++) gm = fmaxf(gm, fabsf(__ldcg(p.x + g * p.G + j)));
            skip[g] = gm <= thr;
        }
    }
    __syncthreads();
    const float mul = s_mul, back = s_back;
    // eight columns per thread: group j of chunk c. Every lane of a warp comes here the same number of times: the shuffles take all 32
    auto convert = [&](int i8, const float4& a, const float4& b) {
        const bool on = i8 < (p.N >> 3);
        const int c = i8 >> 2, j = i8 & 3;
        const int X[8] = { __float2int_rn(a.x * mul), __float2int_rn(a.y * mul), __float2int_rn(a.z * mul), __float2int_rn(a.w * mul),
                           __float2int_rn(b.x * mul), __float2int_rn(b.y * mul), __float2int_rn(b.z * mul), __float2int_rn(b.w * mul) };
        uint32_t D[8], ev[4], od[4];
        long long sum = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) { D[i] = ((uint32_t)X[i] + 0x00808080u) ^ 0x00808080u; sum += X[i]; }   // the four balanced digits of X as bytes
        transpose4x4_bytes(D[0], D[2], D[4], D[6], ev);      // ev[k]: limb k of columns 0, 2, 4, 6
        transpose4x4_bytes(D[1], D[3], D[5], D[7], od);
        if (on) {
            reinterpret_cast<uint4*>(xl)[c * 8 + ((2 * j + c) & 7)] = make_uint4(ev[0], ev[1], ev[2], ev[3]);
            reinterpret_cast<uint4*>(xl)[c * 8 + ((2 * j + 1 + c) & 7)] = make_uint4(od[0], od[1], od[2], od[3]);
        }
        float fs = (float)sum;                                // the four groups of a chunk sit in four neighbouring lanes
        fs += __shfl_xor_sync(0xffffffffu, fs, 1);
        fs += __shfl_xor_sync(0xffffffffu, fs, 2);
        if (on && j == 0) sxs[c] = fs;
    };
    if (held) {
#pragma unroll
        for (int u = 0; u < HELD; u++)
            if (u * I4G_THREADS < (p.N >> 3)) convert(tid + u * I4G_THREADS, xa[u], xb[u]);
    } else {
        for (int i8 = tid; i8 - tid < (p.N >> 3); i8 += I4G_THREADS) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
            if (i8 < (p.N >> 3)) { a = __ldcg(reinterpret_cast<const float4*>(p.x) + 2 * i8); b = __ldcg(reinterpret_cast<const float4*>(p.x) + 2 * i8 + 1); }
            convert(i8, a, b);
        }
    }
    __syncthreads();
    if (!early) {
#pragma unroll
        for (int q = 0; q < STAGES - 1; q++) issue();
    }
    float acc[ROWS];
    int pass = 0, tile = tile0, stage = 0;
    for (int q = 0; q < nstep; q++) {
        const int r0 = tile * ROWS;
        if (pass == 0) {
#pragma unroll
            for (int u = 0; u < ROWS; u++) acc[u] = 0.0f;
        }
        asm volatile("cp.async.wait_group %0;" :: "n"(STAGES - 2) : "memory");
        __syncwarp();
        const int c = lane + 32 * pass;
        const uint32_t* st = ring + stage * STAGE_WORDS;
        uint4 w[ROWS];
        float sc[ROWS];
#pragma unroll
        for (int u = 0; u < ROWS; u++) {
            w[u] = reinterpret_cast<const uint4*>(st)[u * 32 + lane];
            const uint32_t pair = st[ROWS * 32 * 4 + u * 32 + lane];
            const int r = min(r0 + u, p.M - 1);
            const bool hi = (((uintptr_t)(p.s + (size_t)r * ng + group_of(c < nchunk ? c : 0))) & 2) != 0;
            sc[u] = __half2float(__ushort_as_half((unsigned short)(hi ? pair >> 16 : pair & 0xffffu)));
        }
        __syncwarp();                                         // every lane has taken its words: the stage may be refilled
        issue();
        if (c < nchunk) {
            uint32_t xw[32];
#pragma unroll
            for (int piece = 0; piece < 8; piece++) {
                const uint4 v = reinterpret_cast<const uint4*>(xl)[c * 8 + ((piece + c) & 7)];
                xw[4 * piece] = v.x; xw[4 * piece + 1] = v.y; xw[4 * piece + 2] = v.z; xw[4 * piece + 3] = v.w;
            }
            const float m8s = -8.0f * sxs[c];
#pragma unroll
            for (int u = 0; u < ROWS; u++) {
                const uint32_t ww[4] = { w[u].x, w[u].y, w[u].z, w[u].w };
                int a[4] = { 0, 0, 0, 0 };
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int we = (int)(ww[j] & 0x0F0F0F0Fu), wo = (int)((ww[j] >> 4) & 0x0F0F0F0Fu);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        a[k] = __dp4a(we, (int)xw[(2 * j) * 4 + k], a[k]);
                        a[k] = __dp4a(wo, (int)xw[(2 * j + 1) * 4 + k], a[k]);
                    }
                }
                const float v = fmaf((float)a[3], 16777216.0f, fmaf((float)a[2], 65536.0f, fmaf((float)a[1], 256.0f, (float)a[0])));
                acc[u] = fmaf(sc[u], v + m8s, acc[u]);       // sum (nibble - 8) X = sum nibble X - 8 sum X
            }
        }
        if (pass == npass - 1) {
#pragma unroll
            for (int u = 0; u < ROWS; u++) {
                float t = acc[u] * back;
                if (p.K_out > 0) {                            // per-row outlier columns: FP16 value times the activation of the listed column
                    const int r = min(r0 + u, p.M - 1);
                    for (int k = lane; k < p.K_out; k += 32)
                        t = fmaf(__half2float(p.outl_val[(size_t)r * p.K_out + k]), __ldcg(p.x + p.outl_idx[(size_t)r * p.K_out + k]), t);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (lane == 0 && r0 + u < p.M) p.out[r0 + u] = t;
            }
        }
        if (++pass == npass) { pass = 0; tile += tstride; }
        stage = (stage + 1) & (STAGES - 1);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ── tensor-core kernel ──────────────────────────────────────────────────────────────────
// The same integer arithmetic on mma.sync.m16n8k32 (u8 x s8 -> s32), for groups of 32, 64 or a multiple of 128 columns and no outliers or
// skipped groups. Weights stream through a cp.async ring of (16 RT rows x 512 bytes, and the scales of those rows and columns) stages,
// a warp instruction per 512 contiguous bytes; warp w takes 64-byte k-block w (128 columns) of every stage: raw & 0x0F0F0F0F against the
// limbs of the even columns, raw & 0xF0F0F0F0 (sixteen times the nibble; shifted back exactly) against those of the odd ones. The limbs
// are the MMA's columns: four of the eight, so a k-block of two groups (G = 64) has the limbs of the first in columns 0 .. 3, zero where
// the other group's columns are, and those of the second in 4 .. 7; four groups (G = 32) take two sets of MMAs. A thread then holds limbs
// 0 and 1 or 2 and 3 of a row and group: their exact sum (limb a + 256 limb b, less 8 times the activations' own) goes to FP32, times the
// group's scale into the row's sum. Sums of a row meet over lanes and warps once per tile of rows.
// Against 32 dp4a per row and 32 columns (int4g_kernel), us per call: 14336 x 4096, G = 128: 13.7 -> 9.3, G = 64: 13.6 -> 9.8, G = 32: 13.6 ->
// 12.4; 4096 x 14336: 17.0 -> 12.0; 4096 x 4096: 6.3 -> 4.8. What is left is the chain of a launch: the dependency, the activation, which
// every block converts for itself, and the first weights.
constexpr int IM_LD = I4G_WARPS * 64 + 64;                   // bytes per row of a stage, padded: conflict-free fragment reads
struct I4gMma {
    const uint8_t* q; const __half* s; const float* x; float* out;
    int M, N, ng, gsh, rows_per, xs_ld;                      // groups per row; group of a k-block: k >> gsh (G >= 128); rows per block; bytes per limb row
};
// words of a row's scales in a stage (1024 columns): its halves may start in the middle of a word
__host__ __device__ constexpr int im_sw(int G) { return 1024 / G / 2 + 1; }
__host__ __device__ constexpr size_t im_stage(int RT, int G) { return (size_t)RT * 16 * (IM_LD + im_sw(G) * 4); }

__device__ __forceinline__ void im_mma(int* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t im_word(const uint4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

// Shared memory: stage ring | limbs [4][xs_ld] | 32 zero bytes | per group (limb 0 + 256 limb 1, limb 2 + 256 limb 3 sums, times 8) | row sums [2][8][16 RT]
template <int G, int RT, int STAGES, int HELD>
__global__ void __launch_bounds__(I4G_THREADS) int4g_mma_kernel(const I4gMma p) {
    constexpr int R = 16 * RT, SW = im_sw(G), SETS = G == 32 ? 2 : 1, SUB = 128 / G;     // column sets, groups per k-block
    constexpr size_t STAGE = im_stage(RT, G);
    extern __shared__ __align__(128) unsigned char im_smem[];
    __shared__ float s_amax[I4G_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    pdl_launch_dependents();
    const int row_begin = blockIdx.x * p.rows_per, row_end = min(p.M, row_begin + p.rows_per);
    const int rowbytes = p.N >> 1, nkb = (p.N + 127) >> 7, nst = (nkb + I4G_WARPS - 1) / I4G_WARPS;
    unsigned char* xs = im_smem + STAGES * STAGE;
    unsigned char* zero = xs + 4 * (size_t)p.xs_ld;
    int* bias = reinterpret_cast<int*>(zero + 32);
    float* red = reinterpret_cast<float*>(bias + 2 * SUB * nkb);

    // producer: this thread owns 16-byte piece lane of rows warp + 8 i of every stage, and its share of the scales
    int pf_row = row_begin, pf_it = 0, pf_slot = 0;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(im_smem);
    auto issue = [&]() {
        if (pf_row < row_end) {
            const int rows = min(R, row_end - pf_row), col = pf_it * 512 + lane * 16;
            const uint32_t d = ring + (uint32_t)(pf_slot * STAGE);
#pragma unroll
            for (int i = 0; i < 2 * RT; i++) {
                const int r = warp + 8 * i;
                const bool on = r < rows && col < rowbytes;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(d + r * IM_LD + lane * 16),
                             "l"(p.q + (size_t)(pf_row + (on ? r : 0)) * rowbytes + (on ? col : 0)), "r"(on ? 16 : 0) : "memory");
            }
            // The scales of group j of G columns; of a group longer than a k-block only once, at its place among the k-blocks. (Where the number of
            // scales is odd the last word's other half lies behind them, in the same aligned word, and is not used; here and in int4g_kernel. Copies
            // that stop before it took G = 32 3 to 8 % longer.)
            for (int e = tid; e < R * SW; e += I4G_THREADS) {
                const int r = e / SW, w = e - r * SW;
                const size_t first = (size_t)(pf_row + r) * p.ng + ((size_t)(pf_it * I4G_WARPS * SUB) >> p.gsh);
                const size_t at = (first & ~(size_t)1) + 2 * w;
                const bool on = r < rows && at < (size_t)p.M * p.ng;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"(d + R * IM_LD + e * 4), "l"(p.s + (on ? at : 0)), "r"(on ? 4 : 0) : "memory");
            }
            pf_slot = pf_slot + 1 == STAGES ? 0 : pf_slot + 1;
            if (++pf_it == nst) { pf_it = 0; pf_row += rows; }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int q = 0; q < STAGES - 1; q++) issue();             // weights and scales do not depend on the kernel ahead
    if (tid < 8) reinterpret_cast<int*>(zero)[tid] = 0;
    pdl_wait();

    // ── activation: max |x|, fixed point, limbs, and the limb sums of every group ──
    const int n8 = p.N >> 3, n8p = nkb << 4;                  // groups of eight columns; with the padding of the last k-block
    float4 xa[HELD], xb[HELD];
    float amax = 0.0f;
#pragma unroll
    for (int u = 0; u < HELD; u++) {
        const int i8 = tid + u * I4G_THREADS;
        xa[u] = xb[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i8 < n8) { xa[u] = __ldcg(reinterpret_cast<const float4*>(p.x) + 2 * i8); xb[u] = __ldcg(reinterpret_cast<const float4*>(p.x) + 2 * i8 + 1); }
    }
#pragma unroll
    for (int u = 0; u < HELD; u++)
        amax = fmaxf(amax, fmaxf(fmaxf(fmaxf(fabsf(xa[u].x), fabsf(xa[u].y)), fmaxf(fabsf(xa[u].z), fabsf(xa[u].w))),
                                 fmaxf(fmaxf(fabsf(xb[u].x), fabsf(xb[u].y)), fmaxf(fabsf(xb[u].z), fabsf(xb[u].w)))));
    amax = warp_max(amax);
    if (lane == 0) s_amax[warp] = amax;
    __syncthreads();
    amax = s_amax[0];
#pragma unroll
    for (int w = 1; w < I4G_WARPS; w++) amax = fmaxf(amax, s_amax[w]);
    const int ex = (int)((__float_as_uint(amax) >> 23) & 0xFF);      // amax in [2^(ex-127), 2^(ex-126))
    const int sh = max(-126, min(126, (amax > 0.0f && ex != 255) ? 156 - ex : 0));
    const float mul = __uint_as_float((uint32_t)(127 + sh) << 23), back = __uint_as_float((uint32_t)(127 - sh) << 23);
#pragma unroll
    for (int u = 0; u < HELD; u++) {
        const int i8 = tid + u * I4G_THREADS;
        if (i8 - lane >= n8p) break;                          // whole warps: the shuffles take all lanes
        const int X[8] = { __float2int_rn(xa[u].x * mul), __float2int_rn(xa[u].y * mul), __float2int_rn(xa[u].z * mul), __float2int_rn(xa[u].w * mul),
                           __float2int_rn(xb[u].x * mul), __float2int_rn(xb[u].y * mul), __float2int_rn(xb[u].z * mul), __float2int_rn(xb[u].w * mul) };
        uint32_t D[8], ev[4], od[4];
#pragma unroll
        for (int i = 0; i < 8; i++) D[i] = ((uint32_t)X[i] + 0x00808080u) ^ 0x00808080u;     // the four balanced digits of X as bytes
        transpose4x4_bytes(D[0], D[2], D[4], D[6], ev);       // ev[k]: limb k of columns 0, 2, 4, 6
        transpose4x4_bytes(D[1], D[3], D[5], D[7], od);
        int l[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (i8 < n8p) *reinterpret_cast<uint2*>(xs + (size_t)k * p.xs_ld + (size_t)i8 * 8) = make_uint2(ev[k], od[k]);
            l[k] = __dp4a((int)ev[k], 0x01010101, __dp4a((int)od[k], 0x01010101, 0));
        }
        int s01 = l[0] + 256 * l[1], s23 = l[2] + 256 * l[3];
#pragma unroll
        for (int o = 1; o < G / 8; o <<= 1) { s01 += __shfl_xor_sync(0xffffffffu, s01, o); s23 += __shfl_xor_sync(0xffffffffu, s23, o); }
        if (i8 < n8p && (i8 & (G / 8 - 1)) == 0) *reinterpret_cast<int2*>(bias + 2 * (i8 / (G / 8))) = make_int2(8 * s01, 8 * s23);
    }
    __syncthreads();

    // B operand: limb g % 4 of the columns this lane's k positions stand for; zeros where they belong to another group's set
    const unsigned char* xcol[SETS];
    int kstep[SETS], xoff[SETS];
#pragma unroll
    for (int c = 0; c < SETS; c++) {
        const bool mine = G == 128 || (G == 64 ? (t >> 1) == (g >> 2) : t == 2 * c + (g >> 2));
        xcol[c] = mine ? xs + (size_t)(g & 3) * p.xs_ld + 32 * t : zero;
        kstep[c] = mine ? 128 : 0;
        xoff[c] = mine ? 16 : 0;
    }
    int slot = 0, buf = 0, tile_rows = 0;
    for (int row0 = row_begin; row0 < row_end; row0 += tile_rows) {
        tile_rows = min(R, row_end - row0);
        float acc[RT][2];
        int odd[RT][2];                                       // the row's first scale is the upper half of its word
#pragma unroll
        for (int i = 0; i < RT; i++)
#pragma unroll
            for (int h = 0; h < 2; h++) { acc[i][h] = 0.0f; odd[i][h] = (row0 + i * 16 + 8 * h + g) & p.ng & 1; }
        for (int it = 0; it < nst; it++) {
            asm volatile("cp.async.wait_group %0;" :: "n"(STAGES - 2) : "memory");
            __syncthreads();                                  // this stage has landed for everyone; the previous one is free
            issue();
            const int k = it * I4G_WARPS + warp;
            if (k < nkb) {
                const unsigned char* st = im_smem + slot * STAGE;
                const unsigned char* sw = st + warp * 64 + 16 * t;
                const __half* sc = reinterpret_cast<const __half*>(st + R * IM_LD);
                const int g0 = (it * I4G_WARPS * SUB) >> p.gsh;                         // first group of the stage
                uint4 cur[RT * 2];
#pragma unroll
                for (int j = 0; j < RT * 2; j++) cur[j] = *reinterpret_cast<const uint4*>(sw + ((j >> 1) * 16 + (j & 1) * 8 + g) * IM_LD);
#pragma unroll
                for (int c = 0; c < SETS; c++) {
                    uint4 xf[2];
#pragma unroll
                    for (int h = 0; h < 2; h++) xf[h] = *reinterpret_cast<const uint4*>(xcol[c] + (size_t)k * kstep[c] + h * xoff[c]);
                    const int grp = G == 128 ? k >> p.gsh : k * SUB + 2 * c + (t >> 1);
                    const int b8 = bias[2 * (G == 128 ? k : grp) + (t & 1)], gl = grp - g0;
                    const bool on = grp < p.ng;               // the padding of the last k-block has no scale
#pragma unroll
                    for (int i = 0; i < RT; i++) {
                        int lo[4] = { 0, 0, 0, 0 }, hi[4] = { 0, 0, 0, 0 };
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const uint32_t r0a = im_word(cur[2 * i], 2 * h), r0b = im_word(cur[2 * i], 2 * h + 1);
                            const uint32_t r1a = im_word(cur[2 * i + 1], 2 * h), r1b = im_word(cur[2 * i + 1], 2 * h + 1);
                            im_mma(lo, r0a & 0x0F0F0F0Fu, r1a & 0x0F0F0F0Fu, r0b & 0x0F0F0F0Fu, r1b & 0x0F0F0F0Fu, xf[h].x, xf[h].z);
                            im_mma(hi, r0a & 0xF0F0F0F0u, r1a & 0xF0F0F0F0u, r0b & 0xF0F0F0F0u, r1b & 0xF0F0F0F0u, xf[h].y, xf[h].w);
                        }
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const int v = lo[2 * h] + (hi[2 * h] >> 4) + 256 * (lo[2 * h + 1] + (hi[2 * h + 1] >> 4)) - b8;
                            const __half w = sc[(i * 16 + 8 * h + g) * (2 * SW) + (odd[i][h] ^ (g0 & 1)) + gl];
                            acc[i][h] = fmaf(on ? __half2float(w) : 0.0f, (float)v, acc[i][h]);
                        }
                    }
                }
            }
            slot = slot + 1 == STAGES ? 0 : slot + 1;
        }
        float* rw = red + (size_t)buf * I4G_WARPS * R;
#pragma unroll
        for (int i = 0; i < RT; i++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float v = G == 128 && t >= 2 ? 0.0f : (t & 1 ? 65536.0f * acc[i][h] : acc[i][h]);       // G >= 128: columns 4 .. 7 repeat 0 .. 3
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if (t == 0) rw[warp * R + i * 16 + 8 * h + g] = v;
            }
        __syncthreads();
        if (tid < tile_rows) {
            float v = rw[tid];
#pragma unroll
            for (int w = 1; w < I4G_WARPS; w++) v += rw[w * R + tid];
            p.out[row0 + tid] = v * back;
        }
        buf ^= 1;                                             // the next tile's sums do not wait for these reads
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <int G, int RT, int STAGES>
int im_launch(ibcu_ctx* ctx, const I4gMma& p, size_t smem) {
    static SmemOptIn opt4, opt8;
    const dim3 grid((p.M + p.rows_per - 1) / p.rows_per), block(I4G_THREADS);
    if (p.N <= 4 * 8 * I4G_THREADS) {
        if (int rc = ibcu_allow_smem(ctx, opt4, int4g_mma_kernel<G, RT, STAGES, 4>, smem)) return rc;
        return ibcu_launch(ctx, int4g_mma_kernel<G, RT, STAGES, 4>, grid, block, smem, 1, true, p);
    }
    if (int rc = ibcu_allow_smem(ctx, opt8, int4g_mma_kernel<G, RT, STAGES, 8>, smem)) return rc;
    return ibcu_launch(ctx, int4g_mma_kernel<G, RT, STAGES, 8>, grid, block, smem, 1, true, p);
}

// Rows in equal runs over two blocks per SM, but at least a tile of 16 each: with fewer rows a block more blocks convert the whole activation, and
// that is what they take their time for (256 x 16384, G = 128: 13.1 us with a row a block, 12.5 with 8, 8.8 with 16; 1024 x 4096 4.1 and 3.4).
// Tiles of 32 rows where a run is longer than 16 and three stages still fit beside the limbs, else of 16, with as many stages as fit. Five
// stages of 32 rows / three / eight stages of 16 / four, us, G = 128: 14336 x 4096 8.9 / 11.7 / 10.7 / 14.5; 14336 x 8192 - / 16.1 / 19.3 / 26.6;
// 4096 x 4096 (14 rows a block) 5.2 / 7.0 / 4.3 / 6.5. Up to four groups of eight columns per thread held instead of eight: 16 to 35 registers.
template <int G>
int im_dispatch(ibcu_ctx* ctx, I4gMma& p) {
    const int nkb = (p.N + 127) / 128;
    const size_t tail = 4 * (size_t)p.xs_ld + 32 + (size_t)nkb * (128 / G) * 8, room = 112 * 1024;
    p.rows_per = std::max(16, (p.M + 2 * ctx->sm_count - 1) / (2 * ctx->sm_count));
    auto total = [&](int rt, int stages) { return stages * im_stage(rt, G) + tail + 2 * (size_t)I4G_WARPS * 16 * rt * sizeof(float); };
    if (p.rows_per > 16 && total(2, 5) <= room) return im_launch<G, 2, 5>(ctx, p, total(2, 5));
    if (p.rows_per > 16 && total(2, 3) <= room) return im_launch<G, 2, 3>(ctx, p, total(2, 3));
    if (total(1, 8) <= room) return im_launch<G, 1, 8>(ctx, p, total(1, 8));
    return im_launch<G, 1, 4>(ctx, p, total(1, 4));
}

// Whether such a call goes to the tensor cores. dp4a / tensor cores, us: few short rows are all launch, and dp4a's is the shorter: 4096 x 1024 3.0 / 3.3,
// 8192 x 1024 4.1 / 3.4, 1024 x 2048 3.0 / 3.4, 2048 x 2048 3.6 / 3.3, 64 x 4096 4.1 / 3.3 (G = 32 to 256 alike). Groups of 32 in long rows leave room
// for tiles of 16 rows only, and a run of 49 rows then pays for 64: 14336 x 14336 42.7 / 48.8, 8192 x 14336 (28 rows) 27.5 / 26.7.
bool im_pays(const ibcu_ctx* ctx, int M, int N, int G) {
    const int slots = 2 * ctx->sm_count;
    if (N <= 1024 ? M <= 16 * slots : (N <= 2048 && M <= 4 * slots)) return false;
    return !(G == 32 && N > 12288 && M > 48 * slots);
}

// Any N, G (even): a warp per row, lanes over the groups, columns in order inside a group; activations from global memory.
__global__ void __launch_bounds__(I4G_THREADS) int4g_generic_kernel(const I4gParams p, const unsigned char* skip) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, ng = p.N / p.G;
    for (int r = blockIdx.x * I4G_WARPS + warp; r < p.M; r += gridDim.x * I4G_WARPS) {
        const uint8_t* qrow = p.q + (size_t)r * (p.N / 2);
        float acc = 0.0f;
        for (int g = lane; g < ng; g += 32) {
            if (skip && __ldcg(skip + g)) continue;          // written by the kernel just ahead
            float gs = 0.0f;
            for (int j = 0; j < p.G; j += 2) {
                const uint32_t b = qrow[(g * p.G + j) >> 1];
                gs = fmaf((float)((int)(b & 15u) - 8), __ldcg(p.x + g * p.G + j), gs);
                gs = fmaf((float)((int)(b >> 4) - 8), __ldcg(p.x + g * p.G + j + 1), gs);
            }
            acc = fmaf(__half2float(p.s[(size_t)r * ng + g]), gs, acc);
        }
        for (int k = lane; k < p.K_out; k += 32)
            acc = fmaf(__half2float(p.outl_val[(size_t)r * p.K_out + k]), __ldcg(p.x + p.outl_idx[(size_t)r * p.K_out + k]), acc);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) p.out[r] = acc;
    }
}

// skip[g] = max|x over group g| <= eps * max|x| (one block; for the generic kernel)
__global__ void __launch_bounds__(1024) int4g_skip_kernel(const float* x, int N, int G, float eps, unsigned char* __restrict__ skip) {
    __shared__ float red[32];
    pdl_launch_dependents();
    pdl_wait();
    float m = 0.0f;
    for (int i = threadIdx.x; i < N; i += 1024) m = fmaxf(m, fabsf(__ldcg(x + i)));
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = red[0];
    for (int w = 1; w < 32; w++) m = fmaxf(m, red[w]);
    const float thr = eps * m;
    for (int g = threadIdx.x; g < N / G; g += 1024) {
        float gm = 0.0f;
        for (int j = 0; j < G; j++) gm = fmaxf(gm, fabsf(__ldcg(x + g * G + j)));
        skip[g] = gm <= thr;
    }
}

}  // namespace

extern "C" int ibcu_int4g_matmul_fp32(ibcu_ctx* ctx, const ibcu_int4g_t* t, const float* x, float* out, float eps_act_rel) {
    IBCU_CHECK_CTX(ctx);
    IBCU_REQUIRE(ctx, t && x && out && t->q && t->s, "ibcu_int4g_matmul_fp32: null pointer");
    IBCU_REQUIRE(ctx, t->M > 0 && t->N > 0 && t->G > 0 && (t->G & 1) == 0 && t->N % t->G == 0 && t->K_out >= 0 && t->N <= 65536,
                 "ibcu_int4g_matmul_fp32: bad shape M=%d N=%d G=%d K_out=%d", t->M, t->N, t->G, t->K_out);
    IBCU_REQUIRE(ctx, t->K_out == 0 || (t->outl_idx && t->outl_val), "ibcu_int4g_matmul_fp32: outlier arrays missing");
    IBCU_REQUIRE(ctx, !(eps_act_rel < 0.0f) && eps_act_rel == eps_act_rel, "ibcu_int4g_matmul_fp32: eps_act_rel must be >= 0");
    I4gParams p;
    p.M = t->M; p.N = t->N; p.G = t->G; p.K_out = t->K_out;
    p.q = t->q; p.s = (const __half*)t->s; p.outl_idx = t->outl_idx; p.outl_val = (const __half*)t->outl_val;
    p.x = x; p.out = out; p.eps = eps_act_rel;
    // groups of 32, 64 or a power-of-two multiple of 128 columns, nothing left out and nothing beside the groups: the tensor cores. Up to
    // 16384 columns are held in registers while they are converted.
    const int per128 = t->G / 128;
    if (p.eps == 0.0f && t->K_out == 0 && (t->N & 31) == 0 && t->N <= 8 * 8 * I4G_THREADS && (t->G == 32 || t->G == 64 || (t->G % 128 == 0 && (per128 & (per128 - 1)) == 0)) && im_pays(ctx, t->M, t->N, t->G) &&
        (((uintptr_t)t->q | (uintptr_t)x) & 15) == 0 && ((uintptr_t)t->s & 3) == 0) {
        I4gMma m = { t->q, (const __half*)t->s, x, out, t->M, t->N, t->N / t->G, 0, 0, (t->N + 127) / 128 * 128 + 16 };
        while ((128 << m.gsh) < t->G) m.gsh++;
        return t->G == 32 ? im_dispatch<32>(ctx, m) : (t->G == 64 ? im_dispatch<64>(ctx, m) : im_dispatch<128>(ctx, m));
    }
    const size_t xbytes = (size_t)t->N * sizeof(float) + (((size_t)(t->N / 32) + 3) & ~(size_t)3) * sizeof(float) + (((size_t)(t->N / t->G) + 15) & ~(size_t)15);
    const size_t smem = xbytes + (size_t)I4G_WARPS * I4G_STAGES * I4G_ROWS * 32 * 5 * sizeof(uint32_t);
    const bool fast = (t->N & 31) == 0 && (t->G & 31) == 0 && smem <= 200 * 1024 &&
                      (((uintptr_t)t->q | (uintptr_t)x) & 15) == 0 && ((uintptr_t)t->s & 3) == 0;
    if (fast) {
        static std::once_flag once[64];                      // dynamic shared memory beyond 48 KB: opt in once per device
        cudaError_t e = cudaSuccess;
        std::call_once(once[ctx->device & 63], [&] {
            e = cudaFuncSetAttribute(int4g_kernel<I4G_ROWS, I4G_STAGES, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(int4g_kernel<I4G_ROWS, I4G_STAGES, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        });
        if (e != cudaSuccess) return ibcu_fail(ctx, IBCU_ERR_CUDA, "cudaFuncSetAttribute(int4g_kernel): %s", cudaGetErrorString(e));
        // Two rows per warp (four measured slower on both benchmark shapes: 9.1 against 6.9 us and 15.0 against 14.3 us).
        // With more tiles than two blocks per SM can take, three blocks share an SM; with fewer, the launch asks for more
        // shared memory than it needs so that at most two do and the blocks spread over the SMs (256 blocks packed three
        // to an SM: 8.3 us; two to an SM: 6.9 us).
        const size_t ring = (size_t)I4G_WARPS * I4G_STAGES * I4G_ROWS * 32 * 5 * sizeof(uint32_t);
        const size_t need = xbytes + ring;
        const int tiles = (t->M + I4G_WARPS * I4G_ROWS - 1) / (I4G_WARPS * I4G_ROWS);
        const bool crowd = tiles > 2 * ctx->sm_count && need <= 70 * 1024;
        const size_t ask = crowd ? need : (need > 100 * 1024 ? need : 100 * 1024);
        const int per_sm = crowd ? 3 : (ask <= 110 * 1024 ? 2 : 1);
        const int slots = ctx->sm_count * per_sm;
        // up to 8192 columns held in registers leave room for three blocks per SM; longer rows have two at most anyway
        auto kern = t->N <= 8 * 4 * I4G_THREADS ? int4g_kernel<I4G_ROWS, I4G_STAGES, 4> : int4g_kernel<I4G_ROWS, I4G_STAGES, 8>;
        return ibcu_launch(ctx, kern, dim3(tiles < slots ? tiles : slots), dim3(I4G_THREADS), ask, 1, true, p);
    }
    unsigned char* skip = nullptr;
    if (eps_act_rel > 0.0f) {
        int rc = ibcu_reserve(ctx, &ctx->scratch, &ctx->scratch_bytes, (size_t)(t->N / t->G) + 16);
        if (rc) return rc;
        skip = (unsigned char*)ctx->scratch;
        rc = ibcu_launch(ctx, int4g_skip_kernel, dim3(1), dim3(1024), 0, 1, true, x, t->N, t->G, eps_act_rel, skip);
        if (rc) return rc;
    }
    const int blocks = (t->M + I4G_WARPS - 1) / I4G_WARPS;
    return ibcu_launch(ctx, int4g_generic_kernel, dim3(blocks < 4 * ctx->sm_count ? blocks : 4 * ctx->sm_count), dim3(I4G_THREADS), 0, 1, true, p,
                       (const unsigned char*)skip);
}
