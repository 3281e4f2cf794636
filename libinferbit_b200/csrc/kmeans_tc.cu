// k-means assignment for D = 4, 8 or 16 and up to 256 centroids on the fifth-generation tensor cores (tcgen05.mma, accumulators in TMEM).
//
// Scores s_k = x.c_k - |c_k|^2 / 2 (the nearest centroid maximises s_k) for a tile of 128 points against up to 128 centroids are one
// accumulator in tensor memory (a unit; a tile has one or two). x and c, scaled by a power of two that brings the largest |c| to 8 .. 16,
// are split into two FP16 terms each (x = xh + xl to 2^-22 of it), -|c|^2 / 2 into three, and everything rides in one contraction over
// xh.ch + xl.ch + xh.cl + [1 1 1].[n0 n1 n2]: 3 D + 3 columns, that is one, two or four tcgen05.mma steps of K = 16 for D = 4, 8, 16.
// Operands sit in shared memory in the canonical K-major layout without swizzle (8 rows x 16 bytes core matrices); the centroid operand
// is built once per block, the point operand per tile. Centroids are padded to a multiple of 32 with rows that score -1.8e5.
//
// Three roles, joined by mbarriers, so that every scheduler has several independent chains to issue from. Four pipelines, each a
// loader, an operand stage, an accumulator and four scanning warps, take tiles in turn:
//   loaders (4 warps)      raw rows by cp.async, split into the two FP16 terms, into the operand stage; then one elected lane issues the
//                          steps of a unit as soon as the accumulator has been scanned
//   scan (16 warps)        tcgen05.ld (32x32b: a thread owns one point) and the best and second-best maxima over groups of 8 centroids
//                          (three-input max; the group's number rides in the four low bits of its maximum), handed on per tile
//   finish (12 warps)      the best group in the exact form, results, and the point into its cluster's sums
// A Lloyd iteration over 4 Mi points of 8 with 256 centroids: 183 us (285 with scan and finish in the same eight warps, whose chains of
// TMEM loads, exact step and turns of equal clusters two warps per scheduler did not hide; 202 with eight finishing warps, 209 with votes
// in place of match); 4 Mi of 4: 152 (652 on the CUDA cores, with a second pass to accumulate); 1 Mi of 16: 100 (582). What bounds it now
// is the pipe for comparisons and logic, some 500 instructions per scheduler and tile, with issue slots close behind.
//
// The scores only FILTER. If the best group leads by more than 1.25 * 2^-16 (|x|^2 + max |c|^2), the reference's nearest centroid lies in
// that group, and its 8 centroids are evaluated in the reference binary's exact order and rounding, lowest index winning ties. Otherwise
// (near ties, NaN, Inf, points 500 times longer than the longest centroid, magnitudes whose squares leave FP32's range) the warp evaluates
// all centroids in that exact form. Codes and distances are therefore bit-identical to the reference, as with the other kernels.
// Bound, in units of 10^-6 (|x|^2 + max |c|^2): xl.cl and what two FP16 terms do not hold 0.4, -|c|^2 / 2 0.5, accumulation in at most
// four steps of 17 terms each cut at 2^-24 of the largest 3.8, the group's number in the maximum 1.9: 6.6 for a score, 13.2 for a gap;
// the reference's own FP32 distances 2.2; in all 15.4 against a margin of 19.1. (FP16's smallest step, 2^-24 at a scale where the
// longest centroid is 8 or more, adds nothing that shows. Where the scale is held at 2^60, a point with |x|^2 + max |c|^2 of at least
// 1e-30 is as long when scaled.)
//
// Every wait (mbarrier) is bounded: when one runs out the block raises a flag in shared memory, every role
// leaves its loop, tensor memory is released and a host-visible error word is set; nothing spins for ever.
#include "common.cuh"
#include "tc_common.cuh"
#include "kmeans_ref.cuh"

namespace {

constexpr int TC_TILE = 128;                 // points per accumulator tile
constexpr int TC_PIPES = 4;                  // pipelines: tile i goes through pipeline i % 4
constexpr int TC_ACC_COLS = 128;             // columns of a pipeline's accumulator: the centroids of a unit
constexpr int TC_SCAN_WARPS = 4 * TC_PIPES;  // warp w scans for pipeline w / 4, rows 32 (w % 4) .. + 31
constexpr int TC_FIN_WARPS = 12;             // three per quarter of a tile's rows: warp f of the role takes tiles f / 4, f / 4 + 3, ...
constexpr int TC_SLOTS = 3;                  // tiles a scan warp may be ahead of the warp that finishes its rows
constexpr int TC_BLOCKS = 148;               // the most blocks of a launch: one per SM; a number of its own, so that sums depend on the points alone
constexpr int TC_CHUNK = 16 * 128;           // one 16-byte K chunk of 128 rows: 16 core matrices of 128 bytes

// What the number of dimensions decides. Chunks are 16 bytes (8 FP16 values) of every row.
//   D = 4:  A [xh xl | xh 1 1 1 0]                                 B [ch ch | cl n0 n1 n2 0]
//   D = 8:  A [xh | xl], [xh | aug]                                B [ch | ch], [cl | n]
//   D = 16: A [xh xh'], [xl xl'], [xh xh'], [aug | 0]              B [ch ch'], [ch ch'], [cl cl'], [n | 0]
template <int D> struct Shape {
    static constexpr int a_chunks = D == 16 ? 4 : 2, b_chunks = D == 4 ? 2 : D == 8 ? 4 : 6, aug_chunks = D == 4 ? 0 : D == 8 ? 1 : 2;
    static constexpr int raws = D == 16 ? 1 : 2;                  // raw tiles on their way per loader
    static constexpr int a_stage = a_chunks * TC_CHUNK, raw_stage = TC_TILE * D * 4;
    // Exact centroids by group: the 8 values of a dimension are two 16-byte halves. For D = 4 and 8 there are four copies, copy c in banks
    // 8 c .. 8 c + 7: lane l reads copy l % 4, lanes with bit 2 set the halves in the other order, so that eight lanes with eight
    // different groups meet no conflict (one copy: 2.6 wavefronts for each). D = 16 has no room for them: one copy, groups skewed.
    static constexpr int copies = D == 16 ? 1 : 4;
    static constexpr int dim_stride = 8 * copies;                 // floats
    static constexpr int group_stride = dim_stride * D + (copies == 1 ? 4 : 0);
    static constexpr int each_lane = D == 4 ? 10 : 16;            // undecided rows of a warp from which every lane does its own
    static constexpr int row_stride = D == 16 ? 20 : D;           // floats per cluster in a table of sums (16: skewed, or all clusters' pieces would share two places in the banks)
};

__device__ __forceinline__ uint32_t f16x2_of(float lo, float hi) { uint32_t r; asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo)); return r; }
__device__ __forceinline__ float f16_lo(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)v)); }
__device__ __forceinline__ float f16_hi(uint32_t v) { return __half2float(__ushort_as_half((unsigned short)(v >> 16))); }
// N values times scale as two FP16 terms: h[i] and l[i] hold values 2 i and 2 i + 1
template <int N>
__device__ __forceinline__ void split_f16(const float* v, float scale, uint32_t* h, uint32_t* l) {
#pragma unroll
    for (int i = 0; i < N / 2; i++) {
        const float a = v[2 * i] * scale, b = v[2 * i + 1] * scale;
        h[i] = f16x2_of(a, b);
        l[i] = f16x2_of(a - f16_lo(h[i]), b - f16_hi(h[i]));
    }
}
__device__ __forceinline__ void mma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                 :: "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) { float r; asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r; }

// two FP32 lanes per instruction (round to nearest, each lane rounded like the scalar operation)
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) { unsigned long long r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) { unsigned long long r; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) { unsigned long long r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }

struct TcShared {
    unsigned long long empty_a[TC_PIPES];                          // MMAs have read the operand stage
    unsigned long long full_acc[TC_PIPES], empty_acc[TC_PIPES];    // MMA -> scan, scan -> MMA
    unsigned long long full_h[TC_SCAN_WARPS][TC_SLOTS], empty_h[TC_SCAN_WARPS][TC_SLOTS];   // scan -> finish, finish -> scan
    unsigned long long turn[4][TC_FIN_WARPS / 4];                  // warps that share a table -> the next of them
    unsigned long long drained;                                    // every MMA of the block has completed
    float2 found[TC_SCAN_WARPS][TC_SLOTS][32];                     // per point: gap between the best and the second-best group; the best group (an int)
    uint32_t tmem_base;
    int abort_flag;
    unsigned cmax2_bits;
    double inert[TC_FIN_WARPS];
};

// Best and second-best of the maxima over groups of 8 scores, two groups (16 scores) at a time. The group's number within the unit
// replaces the four low bits of its maximum.
struct Top2 { float m1, m2; };
__device__ __forceinline__ float group_max(const float* v, int gid) {
    float g = max3(v[0], v[1], v[2]);
    g = max3(g, v[3], v[4]);
    g = max3(g, v[5], v[6]);
    g = fmaxf(g, v[7]);
    return __uint_as_float((__float_as_uint(g) & ~15u) | (uint32_t)gid);
}
__device__ __forceinline__ void top2_groups(const uint32_t* r, int gid0, Top2& t) {
    const float* v = reinterpret_cast<const float*>(r);
    const float a = group_max(v, gid0), b = group_max(v + 8, gid0 + 1);
    const float hi = fmaxf(a, b), lo = fminf(a, b);
    t.m2 = max3(t.m2, fminf(t.m1, hi), lo);
    t.m1 = fmaxf(t.m1, hi);
}

// Read past L1 and not as a read-only load: the kernel just ahead may have written the row (centroids of the last iteration).
template <int D> __device__ __forceinline__ void load_row(const float* X, long row, bool have, float* x) {
#pragma unroll
    for (int d = 0; d < D; d += 4) {
        const float4 v = have ? __ldcg(reinterpret_cast<const float4*>(X + row * D + d)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        x[d] = v.x; x[d + 1] = v.y; x[d + 2] = v.z; x[d + 3] = v.w;
    }
}

// the reference's squared distance to centroid k, read from the table of groups (neighbouring groups from different copies)
template <int D> __device__ __forceinline__ float group_sqdist(const float* x, const float* cgrp, int k) {
    using S = Shape<D>;
    const float* c = cgrp + (k >> 3) * S::group_stride + ((k >> 3) % S::copies) * 8 + (k & 7);
    float s = 0.0f;
#pragma unroll
    for (int d = 0; d < D; d++) {
        const float v = __fsub_rn(x[d], c[d * S::dim_stride]);
        s = __fadd_rn(s, __fmul_rn(v, v));
    }
    return s;
}

// Dynamic shared memory: centroid operand [b_chunks][Kp rows x 16 B] | stages of the point operand | constant chunks of the point
// operand (behind the stages: a step of D = 8 takes its second chunk from here) | stages of raw points | exact centroids by group
// [Kp / 8][D dims][copies][8] | ACC: a table of K sums per finishing warp, then [warp][K] counts | TcShared
// ACC: the finishing warps also add every point into the table of its cluster (points of a warp in index order), and the block leaves
// the sum of its tables, its counts and its share of the inertia in part_*[blockIdx.x]: the accumulate pass over X of a Lloyd iteration
// then needs no kernel and no second read of X. The order of the adds is fixed by the grid. TAB tables: one per
// finishing warp, or, where twelve do not fit, one for the three warps of a quarter, which take turns tile by tile.
template <int D, bool ACC, int TAB>
__global__ void __launch_bounds__((TC_SCAN_WARPS + TC_FIN_WARPS + TC_PIPES) * 32, 1)
assign_tc_kernel(const float* X, long N, const float* C, int K, int32_t* __restrict__ idx, float* __restrict__ dist,
                 int* __restrict__ err, float* __restrict__ part_sums, int32_t* __restrict__ part_counts, double* __restrict__ part_inertia) {
    using S = Shape<D>;
    constexpr int FIN = TC_FIN_WARPS, THREADS = (TC_SCAN_WARPS + FIN + TC_PIPES) * 32;
    constexpr int STEP = FIN / 4, SHARE = FIN / TAB;             // tiles from one of a finishing warp to its next; warps that share a table
    constexpr int FIN0 = TC_SCAN_WARPS, LOAD0 = FIN0 + FIN, PP = D / 4;
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Kp = (K + 31) & ~31, halves = Kp > TC_ACC_COLS ? 2 : 1;          // units per tile
    const uint32_t b_chunk = (uint32_t)Kp * 16u;
    unsigned char* sB = tc_smem;
    unsigned char* sA = sB + S::b_chunks * b_chunk;
    unsigned char* sAug = sA + TC_PIPES * S::a_stage;
    unsigned char* sRaw = sAug + S::aug_chunks * TC_CHUNK;
    float* cgrp = reinterpret_cast<float*>(sRaw + TC_PIPES * S::raws * S::raw_stage);
    float* wtab = cgrp + (size_t)(Kp / 8) * S::group_stride;
    int* wcnt = reinterpret_cast<int*>(wtab + (ACC ? (size_t)TAB * K * S::row_stride : 0));
    TcShared* sh = reinterpret_cast<TcShared*>(((uintptr_t)(wcnt + (ACC ? (size_t)TAB * K : 0)) + 15) & ~(uintptr_t)15);
    volatile int* abort_flag = &sh->abort_flag;

    if (tid == 0) {
        for (int b = 0; b < TC_PIPES; b++) { mbar_init(smem_u32(&sh->empty_a[b]), 1); mbar_init(smem_u32(&sh->full_acc[b]), 1); mbar_init(smem_u32(&sh->empty_acc[b]), 4); }
        for (int w = 0; w < TC_SCAN_WARPS; w++)
            for (int s = 0; s < TC_SLOTS; s++) { mbar_init(smem_u32(&sh->full_h[w][s]), 1); mbar_init(smem_u32(&sh->empty_h[w][s]), 1); }
        for (int t = 0; t < FIN; t++) mbar_init(smem_u32(&sh->turn[t & 3][t >> 2]), 1);
        mbar_init(smem_u32(&sh->drained), TC_PIPES);
        sh->abort_flag = 0;
        sh->cmax2_bits = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == LOAD0) {                     // all 512 columns of tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&sh->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        // Not before: a block of a later launch that moves in beside this one may allocate tensor memory too and keeps it until
        // this launch has ended, so every block of this launch must hold its own first.
        pdl_launch_dependents();
    }
    if (ACC) {
        for (int e = tid; e < TAB * K * S::row_stride; e += THREADS) wtab[e] = 0.0f;
        for (int e = tid; e < TAB * K; e += THREADS) wcnt[e] = 0;
    }
    if (D > 4) {                             // constant chunks of the point operand: row e = (1 1 1 0 0 0 0 0 | zeros)
        for (int e = tid; e < 128 * S::aug_chunks; e += THREADS)
            *reinterpret_cast<uint4*>(sAug + e * 16) = e < 128 ? make_uint4(0x3C003C00u, 0x00003C00u, 0u, 0u) : make_uint4(0u, 0u, 0u, 0u);
    }
    __syncthreads();
    pdl_wait();

    const long ntile = (N + TC_TILE - 1) / TC_TILE;
    const int n_my = (long)blockIdx.x < ntile ? (int)((ntile - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0;      // tiles blockIdx.x + i gridDim.x
    auto tile_row = [&](int i) { return ((long)blockIdx.x + (long)i * gridDim.x) * TC_TILE; };

    // raw rows of a tile into a loader's own buffers (pieces of a row permuted so that eight rows read at once lie on all banks); the
    // first ones travel while the centroids are prepared
    unsigned char* const raws = sRaw + max(warp - LOAD0, 0) * (S::raws * S::raw_stage);
    auto piece_at = [](int r, int p) { return r * PP + (p ^ ((r / (8 / PP)) & (PP - 1))); };
    auto issue = [&](int i) {
        if (i < n_my) {
            const long p0 = tile_row(i);
            const uint32_t dst = smem_u32(raws + (i / TC_PIPES) % S::raws * S::raw_stage);
#pragma unroll
            for (int j = 0; j < 4 * PP; j++) {
                const int e = lane + 32 * j, r = e / PP, p = e % PP;
                const long pt = p0 + r;
                const int nbytes = pt < N ? 16 : 0;              // points past the end read as zeros
                const float* src = X + (pt < N ? pt : 0) * D + p * 4;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst + piece_at(r, p) * 16), "l"(src), "r"(nbytes) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (warp >= LOAD0) for (int t = 0; t < S::raws; t++) issue(warp - LOAD0 + t * TC_PIPES);

    // ── centroids: exact copies by group (padding is NaN: never nearer than anything), max |c|^2 ──
    static_assert(THREADS >= 256, "a thread per centroid");
    unsigned cm_bits = 0u;
    const int n = tid;
    float c[D], nn = 0.0f;
    if (n < Kp) {
        if (((uintptr_t)C & 15) == 0) load_row<D>(C, n, n < K, c);
        else {
#pragma unroll
            for (int d = 0; d < D; d++) c[d] = n < K ? __ldcg(C + n * D + d) : 0.0f;
        }
#pragma unroll
        for (int d = 0; d < D; d++) {
#pragma unroll
            for (int j = 0; j < S::copies; j++)                          // neighbouring groups write different copies: no bank conflict
                cgrp[(n >> 3) * S::group_stride + d * S::dim_stride + (j + (n >> 3)) % S::copies * 8 + (n & 7)] = n < K ? c[d] : __uint_as_float(0x7FFFFFFFu);
            nn = fmaf(c[d], c[d], nn);
        }
        cm_bits = __float_as_uint(nn);                       // nn >= 0 or NaN: NaN and Inf sort above everything finite
    }
    cm_bits = __reduce_max_sync(0xffffffffu, cm_bits);
    if (lane == 0) atomicMax(&sh->cmax2_bits, cm_bits);
    __syncthreads();
    // the scale of points and centroids, 2^(3 - e) for the largest |c| in [2^e, 2^(e + 1)): 8 .. 16 when scaled
    const float cm2 = __uint_as_float(sh->cmax2_bits);
    const int cexp = ((int)(sh->cmax2_bits >> 23) - 127) >> 1;                 // -64 for zero, 64 for Inf and NaN (where everything goes the exact way)
    const float scale = __uint_as_float((uint32_t)(min(max(3 - cexp, -60), 60) + 127) << 23);
    if (n < Kp) {
        nn = 0.0f;
#pragma unroll
        for (int d = 0; d < D; d++) nn = fmaf(c[d] * scale, c[d] * scale, nn);
        uint32_t h[D / 2], l[D / 2], t[2];
        split_f16<D>(c, scale, h, l);
        const float nh = n < K ? -0.5f * nn : -60000.0f;
        const uint32_t n0 = f16x2_of(nh, 0.0f);
        const float r1 = nh - f16_lo(n0);
        const uint32_t n1 = f16x2_of(r1, 0.0f);
        t[0] = n < K ? (n0 & 0xFFFFu) | (n1 << 16) : n0 * 0x10001u;
        t[1] = n < K ? f16x2_of(r1 - f16_lo(n1), 0.0f) : n0;
        unsigned char* dst = sB + (uint32_t)(n >> 3) * 128u + (uint32_t)(n & 7) * 16u;
        auto put = [&](int chunk, uint32_t a, uint32_t b, uint32_t c2, uint32_t d2) { *reinterpret_cast<uint4*>(dst + chunk * b_chunk) = make_uint4(a, b, c2, d2); };
        if (D == 4) {
            put(0, h[0], h[1], h[0], h[1]);
            put(1, l[0], l[1], t[0], t[1]);
        } else if (D == 8) {
            put(0, h[0], h[1], h[2], h[3]);
            put(1, h[0], h[1], h[2], h[3]);
            put(2, l[0], l[1], l[2], l[3]);
            put(3, t[0], t[1], 0u, 0u);
        } else {
            put(0, h[0], h[1], h[2], h[3]);
            put(1, h[D / 2 - 4], h[D / 2 - 3], h[D / 2 - 2], h[D / 2 - 1]);
            put(2, l[0], l[1], l[2], l[3]);
            put(3, l[D / 2 - 4], l[D / 2 - 3], l[D / 2 - 2], l[D / 2 - 1]);
            put(4, t[0], t[1], 0u, 0u);
            put(5, 0u, 0u, 0u, 0u);
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the operands written above are read by the tensor cores
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = sh->tmem_base;

    if (warp >= LOAD0) {
        // ── loaders: warp lw owns pipeline lw: raw rows by cp.async (one or two of its tiles ahead), the two FP16 terms into the operand
        //    stage, and the MMAs. (One warp issuing for all accumulators was a chain of 1000 cycles per tile: two waits, two issues and
        //    three commits one after the other.) ──
        const int lw = warp - LOAD0;
        const uint32_t a0 = smem_u32(sA + lw * S::a_stage), b0 = smem_u32(sB), aug = smem_u32(sAug), acc = tmem_base + (uint32_t)(lw * TC_ACC_COLS);
        bool ok = true;
        for (int i = lw, use = 0; i < n_my && ok; i += TC_PIPES) {
            asm volatile("cp.async.wait_group %0;" :: "n"(S::raws - 1) : "memory");
            __syncwarp();
            ok = __all_sync(0xffffffffu, mbar_wait<false>(smem_u32(&sh->empty_a[lw]), (uint32_t)(((i / TC_PIPES) & 1) ^ 1), abort_flag, 1));   // the whole warp leaves or stays
            if (!ok) break;
            const unsigned char* raw = raws + (i / TC_PIPES) % S::raws * S::raw_stage;
#pragma unroll 1
            for (int t = 0; t < 4; t++) {
                const int r = 32 * t + lane;
                float v[D];
#pragma unroll
                for (int p = 0; p < PP; p++) {
                    const float4 f = *reinterpret_cast<const float4*>(raw + piece_at(r, p) * 16);
                    v[4 * p] = f.x; v[4 * p + 1] = f.y; v[4 * p + 2] = f.z; v[4 * p + 3] = f.w;
                }
                uint32_t h[D / 2], l[D / 2];
                split_f16<D>(v, scale, h, l);
                unsigned char* dst = sA + lw * S::a_stage + (uint32_t)(r >> 3) * 128u + (uint32_t)(r & 7) * 16u;
                if (D == 4) {
                    *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], l[0], l[1]);
                    *reinterpret_cast<uint4*>(dst + TC_CHUNK) = make_uint4(h[0], h[1], 0x3C003C00u, 0x00003C00u);
                } else {
#pragma unroll
                    for (int j = 0; j < D / 8; j++) {
                        *reinterpret_cast<uint4*>(dst + j * TC_CHUNK) = make_uint4(h[4 * j], h[4 * j + 1], h[4 * j + 2], h[4 * j + 3]);
                        *reinterpret_cast<uint4*>(dst + (D / 8 + j) * TC_CHUNK) = make_uint4(l[4 * j], l[4 * j + 1], l[4 * j + 2], l[4 * j + 3]);
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();                                            // the raw rows about to be refilled have been read by every lane
            issue(i + S::raws * TC_PIPES);
            for (int p = 0; p < halves; p++, use++) {
                ok = __all_sync(0xffffffffu, mbar_wait<false>(smem_u32(&sh->empty_acc[lw]), (uint32_t)((use & 1) ^ 1), abort_flag, 3));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int cols = min(Kp - p * TC_ACC_COLS, TC_ACC_COLS);
                const uint32_t idesc = (1u << 4) | ((uint32_t)(cols >> 3) << 17) | ((uint32_t)(TC_TILE >> 4) << 24);   // F16 x F16 -> F32
                const uint32_t bp = b0 + (uint32_t)p * (TC_ACC_COLS * 16u);
                if (elect_one()) {
                    mma_f16_ss(acc, smem_desc(a0, TC_CHUNK, 128), smem_desc(bp, b_chunk, 128), idesc, 0u);
                    if (D == 8) mma_f16_ss(acc, smem_desc(a0, aug - a0, 128), smem_desc(bp + 2 * b_chunk, b_chunk, 128), idesc, 1u);
                    if (D == 16) {
                        mma_f16_ss(acc, smem_desc(a0 + 2 * TC_CHUNK, TC_CHUNK, 128), smem_desc(bp, b_chunk, 128), idesc, 1u);
                        mma_f16_ss(acc, smem_desc(a0, TC_CHUNK, 128), smem_desc(bp + 2 * b_chunk, b_chunk, 128), idesc, 1u);
                        mma_f16_ss(acc, smem_desc(aug, TC_CHUNK, 128), smem_desc(bp + 4 * b_chunk, b_chunk, 128), idesc, 1u);
                    }
                    mma_commit(smem_u32(&sh->full_acc[lw]));                         // the accumulator is complete
                    if (p == halves - 1) mma_commit(smem_u32(&sh->empty_a[lw]));     // and the operand stage is free
                }
                __syncwarp();
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (elect_one()) mma_commit(smem_u32(&sh->drained));
        __syncwarp();
        mbar_wait<false>(smem_u32(&sh->drained), 0u, abort_flag, 4);            // nothing of this block is left in the tensor pipe
    } else if (warp < FIN0) {
        // ── scan ──
        const int q = warp & 3, b = warp >> 2;
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * TC_ACC_COLS);
        bool ok = true;
        for (int i = b, j = 0, use = 0; i < n_my; i += TC_PIPES, j++) {
            float m1 = -INFINITY, m2 = -INFINITY;
            int g1 = 0;
            for (int p = 0; p < halves; p++, use++) {
                ok = __all_sync(0xffffffffu, mbar_wait<false>(smem_u32(&sh->full_acc[b]), (uint32_t)(use & 1), abort_flag, 5));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int cols = min(Kp - p * TC_ACC_COLS, TC_ACC_COLS);
                Top2 ta = { -INFINITY, -INFINITY }, tb = { -INFINITY, -INFINITY };
                for (int c0 = 0; c0 < cols; c0 += 32) {              // the other warps of the scheduler hide the load
                    uint32_t r[32];
                    tmem_ld32(taddr + c0, r);
                    tmem_wait_ld(r);
                    top2_groups(r, c0 >> 3, ta);
                    top2_groups(r + 16, (c0 >> 3) + 2, tb);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sh->empty_acc[b]));      // the tensor cores may overwrite this accumulator
                const float u1 = fmaxf(ta.m1, tb.m1), u2 = max3(ta.m2, tb.m2, fminf(ta.m1, tb.m1));
                m2 = max3(m2, u2, fminf(m1, u1));
                if (u1 > m1) g1 = p * (TC_ACC_COLS / 8) + (int)(__float_as_uint(u1) & 15u);
                m1 = fmaxf(m1, u1);
            }
            const int slot = j % TC_SLOTS;
            ok = ok && __all_sync(0xffffffffu, mbar_wait<false>(smem_u32(&sh->empty_h[warp][slot]), (uint32_t)(((j / TC_SLOTS) & 1) ^ 1), abort_flag, 6));
            if (!ok) break;
            sh->found[warp][slot][lane] = make_float2(m1 - m2, __int_as_float(g1));
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sh->full_h[warp][slot]));
        }
    } else {
        // ── finish ──
        // A slot's tiles are TC_PIPES * TC_SLOTS apart and must all be one warp's: were they several warps', one could wait for a phase of
        // full_h while another has yet to take the one two before it, which has the same parity.
        static_assert(TC_PIPES * TC_SLOTS % STEP == 0, "the tiles of a slot go to one finishing warp");
        const int f = warp - FIN0, q = f & 3;
        float* mytab = wtab + (size_t)(f % TAB) * K * S::row_stride;
        int* mycnt = wcnt + (size_t)(f % TAB) * K;
        double inert = 0.0;
        constexpr bool AHEAD = D <= 8;                               // the next row is fetched while this one is worked on (D = 16 lacks the registers)
        float xnext[AHEAD ? D : 4];
        if (AHEAD) {
            const long row = tile_row(f >> 2) + q * 32 + lane;
            load_row<AHEAD ? D : 4>(X, row, row < N && (f >> 2) < n_my, xnext);
        }
        const int swap = S::copies == 4 ? (lane >> 2) & 1 : 0;
        const float* const mygrp = cgrp + (S::copies == 4 ? (lane & 3) * 8 : 0);
        for (int i = f >> 2; i < n_my; i += STEP) {
            const long row = tile_row(i) + q * 32 + lane;
            const bool have = row < N;
            float xr[D], xn = 0.0f;
            if (AHEAD) {
#pragma unroll
                for (int d = 0; d < D; d++) xr[d] = xnext[AHEAD ? d : 0];
                const long next = tile_row(i + STEP) + q * 32 + lane;
                load_row<AHEAD ? D : 4>(X, next, next < N && i + STEP < n_my, xnext);
            } else load_row<D>(X, row, have, xr);
#pragma unroll
            for (int d = 0; d < D; d++) xn = fmaf(xr[d], xr[d], xn);
            const int from = i % TC_PIPES * 4 + q, j = i / TC_PIPES, slot = j % TC_SLOTS;
            if (!__all_sync(0xffffffffu, mbar_wait<false>(smem_u32(&sh->full_h[from][slot]), (uint32_t)((j / TC_SLOTS) & 1), abort_flag, 7))) break;
            const float2 w = sh->found[from][slot][lane];
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sh->empty_h[from][slot]));
            const int g1 = __float_as_int(w.y);
            // the margin that makes the filter safe: false for NaN / Inf, where squares overflow or vanish, and for points so long
            // (2^13 when scaled) that a centroid might score below the padding
            const float mag = xn + cm2, smag = mag * scale * scale;
            const bool sure = w.x > 1.9073486328125e-5f * smag && smag < 6.7108864e7f && mag < 1e37f && mag > 1e-30f;
            // the best group in the exact form (subtract, multiply, add, each rounded, in dimension order), then ascending
            // with strict '<': the lowest index wins ties as in the reference
            int win;
            float best;
            {
                const float* ca = mygrp + g1 * S::group_stride + 4 * swap;
                const float* cb = mygrp + g1 * S::group_stride + 4 * (swap ^ 1);
                // subtract and multiply go two centroids at a time; the add stays scalar, because the assembler contracts
                // a packed multiply followed by a packed add into a fused multiply-add, which rounds differently
                float dk[8] = { 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f };
#pragma unroll
                for (int d = 0; d < D; d++) {
                    const ulonglong2 va = *reinterpret_cast<const ulonglong2*>(ca + d * S::dim_stride), vb = *reinterpret_cast<const ulonglong2*>(cb + d * S::dim_stride);
                    const unsigned long long xx = pack2(xr[d], xr[d]);
                    const unsigned long long c2[4] = { va.x, va.y, vb.x, vb.y };
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const unsigned long long v = sub2(xx, c2[k]);
                        float p0, p1;
                        unpack2(mul2(v, v), p0, p1);
                        dk[2 * k] = __fadd_rn(dk[2 * k], p0);
                        dk[2 * k + 1] = __fadd_rn(dk[2 * k + 1], p1);
                    }
                }
                const float m0 = fminf(fminf(dk[0], dk[1]), fminf(dk[2], dk[3])), m4 = fminf(fminf(dk[4], dk[5]), fminf(dk[6], dk[7]));
                best = fminf(m0, m4);
                int at0 = 3, at4 = 3;                                // lowest index of the minimum in the half read first, in the second
#pragma unroll
                for (int k = 2; k >= 0; k--) { if (dk[k] == best) at0 = k; if (dk[4 + k] == best) at4 = k; }
                // the lower half wins a tie between the two (with the halves exchanged it is the second one read)
                const bool second = swap ? m4 == best : m0 != best;
                win = g1 * 8 + (second ? at4 : at0) + (second != (swap != 0) ? 4 : 0);
            }
            // Rows the filter could not decide: all centroids in the exact form, by the whole warp for one row after another, or, where they
            // are many (equal centroids, points on a grid), by every lane for its own row. 1 Mi points that are all undecided, 256 centroids:
            // 479 -> 181 us for 4 dimensions, 595 -> 288 for 8, 1241 -> 508 for 16 (assign_exact_kernel: 144, 256, 467). As turns of the
            // loop that evaluates the best group it would save the code, but took 204 us instead of 183 per iteration without ties.
            unsigned todo = __ballot_sync(0xffffffffu, have && !sure);
            if (todo == 0u) {
                // nearly always: one test on the way
            } else if (__popc(todo) > S::each_lane) {
                win = 0;
                best = group_sqdist<D>(xr, cgrp, 0);                 // the reference's seed whatever its distance
#pragma unroll 1
                for (int k = 0; k < Kp; k += 4) {                    // four centroids at a time, the same for all lanes; padding is NaN
                    const float* c4 = cgrp + (k >> 3) * S::group_stride + (k & 4);
                    float dk[4] = { 0.0f, 0.0f, 0.0f, 0.0f };
#pragma unroll
                    for (int d = 0; d < D; d++) {
                        const ulonglong2 c2 = *reinterpret_cast<const ulonglong2*>(c4 + d * S::dim_stride);
                        const unsigned long long xx = pack2(xr[d], xr[d]), va = sub2(xx, c2.x), vb = sub2(xx, c2.y);
                        float p0, p1, p2, p3;
                        unpack2(mul2(va, va), p0, p1);
                        unpack2(mul2(vb, vb), p2, p3);
                        dk[0] = __fadd_rn(dk[0], p0); dk[1] = __fadd_rn(dk[1], p1); dk[2] = __fadd_rn(dk[2], p2); dk[3] = __fadd_rn(dk[3], p3);
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) if (dk[j] < best) { best = dk[j]; win = k + j; }      // ascending and strict, as the reference goes
                }
            }
            else do {
                const int rl = __ffs(todo) - 1;
                todo &= todo - 1;
                float xq[D];
#pragma unroll
                for (int d = 0; d < D; d++) xq[d] = __shfl_sync(0xffffffffu, xr[d], rl);
                float bd = INFINITY; int bk = 0x7fffffff;
#pragma unroll 1                                              // rare: short code rather than short chains (ten iterations of 4 Mi x 8 1859 -> 1833 us)
                for (int k = lane; k < K; k += 32) {
                    const float dk = group_sqdist<D>(xq, cgrp, k);
                    if (dk < bd || k == 0) { bd = dk; bk = k; }      // centroid 0 is the reference's seed whatever its distance
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {                   // lexicographic (distance, index) minimum; lane 0 keeps a seed that is NaN
                    const float od = __shfl_xor_sync(0xffffffffu, bd, o);
                    const int ok = __shfl_xor_sync(0xffffffffu, bk, o);
                    if (od < bd || (od == bd && ok < bk)) { bd = od; bk = ok; }
                }
                bd = __shfl_sync(0xffffffffu, bd, 0);
                bk = __shfl_sync(0xffffffffu, bk, 0);
                if (lane == rl) { win = bk; best = bd; }
            } while (todo);
            if (have) { idx[row] = win; if (dist) dist[row] = best; }
            if (ACC) {
                // Points of the warp that share a cluster: the first of them fetches the others' rows, adds them behind its own, in index
                // order, and their sum to the table: an entry receives one value per tile, so that its error grows with the number of
                // tiles of the table (74 at 4 Mi points) and not with that of points. Different clusters go together. (Equal clusters bit by bit with votes: eight votes and thirty-odd more
                // instructions for the pipe that bounds the kernel.)
                const unsigned grp = __match_any_sync(0xffffffffu, have ? win : -1 - lane);
                if (SHARE > 1 && i > 0) {                    // the warp with the tile before has added its points
                    if (!__all_sync(0xffffffffu, mbar_wait<false>(smem_u32(&sh->turn[q][f >> 2]), (uint32_t)(((i - 1) / SHARE) & 1), abort_flag, 8))) break;
                }
                const bool first = have && (grp & ((1u << lane) - 1u)) == 0;
                const int turns = __reduce_max_sync(0xffffffffu, (unsigned)__popc(grp));
                float4* t = reinterpret_cast<float4*>(mytab + (size_t)win * S::row_stride);
                float4 sum[PP];
#pragma unroll
                for (int p = 0; p < PP; p++) sum[p] = make_float4(xr[4 * p], xr[4 * p + 1], xr[4 * p + 2], xr[4 * p + 3]);
                unsigned rest = grp & (grp - 1u);
                for (int r = 1; r < turns; r++) {
                    const int src = rest ? __ffs(rest) - 1 : lane;
                    const bool add = rest != 0u;
                    rest &= rest - 1u;
#pragma unroll
                    for (int p = 0; p < PP; p++) {
                        const float a0 = __shfl_sync(0xffffffffu, xr[4 * p], src), a1 = __shfl_sync(0xffffffffu, xr[4 * p + 1], src);
                        const float a2 = __shfl_sync(0xffffffffu, xr[4 * p + 2], src), a3 = __shfl_sync(0xffffffffu, xr[4 * p + 3], src);
                        if (add) { sum[p].x += a0; sum[p].y += a1; sum[p].z += a2; sum[p].w += a3; }
                    }
                }
                if (first) {
                    mycnt[win] += __popc(grp);
#pragma unroll
                    for (int p = 0; p < PP; p++) {
                        const float4 v = t[p];
                        t[p] = make_float4(v.x + sum[p].x, v.y + sum[p].y, v.z + sum[p].z, v.w + sum[p].w);
                    }
                }
                __syncwarp();
                if (SHARE > 1 && lane == 0) mbar_arrive(smem_u32(&sh->turn[q][((f >> 2) + 1) % SHARE]));
                if (have) inert += (double)best;
            }
        }
        if (ACC) {
            // the tables of the block, added in warp order; every finishing warp gets here, also after a wait ran out
            const int ft = tid - FIN0 * 32, used = min(TAB, 4 * n_my);       // tables that had a tile
            for (int o = 16; o > 0; o >>= 1) inert += __shfl_xor_sync(0xffffffffu, inert, o);
            if (lane == 0) sh->inert[f] = inert;
            asm volatile("bar.sync 1, %0;" :: "n"(FIN * 32) : "memory");
            for (int e = ft; e < K * D; e += FIN * 32) {
                const float* t = wtab + (e / D) * S::row_stride + e % D;
                double v = (double)t[0];
#pragma unroll 4
                for (int w = 1; w < used; w++) v += (double)t[(size_t)w * K * S::row_stride];
                part_sums[(size_t)blockIdx.x * K * D + e] = (float)v;
            }
            for (int e = ft; e < K; e += FIN * 32) {
                int v = wcnt[e];
#pragma unroll 4
                for (int w = 1; w < used; w++) v += wcnt[(size_t)w * K + e];
                part_counts[(size_t)blockIdx.x * K + e] = v;
            }
            if (ft == 0) {
                double t = 0.0;
                for (int w = 0; w < FIN; w++) t += sh->inert[w];
                part_inertia[blockIdx.x] = t;
            }
        }
    }
    // ── teardown: every role is out of its loop (all waits are bounded); release tensor memory ──
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == LOAD0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"(512u) : "memory");
    }
    if (tid == 0 && sh->abort_flag) *err = 100 + sh->abort_flag;
}

template <int D>
size_t tc_smem_bytes(int K, bool acc, int tab) {
    using S = Shape<D>;
    const size_t Kp = (size_t)((K + 31) & ~31);
    return S::b_chunks * Kp * 16 + TC_PIPES * (size_t)(S::a_stage + S::raws * S::raw_stage) + S::aug_chunks * TC_CHUNK + Kp / 8 * S::group_stride * sizeof(float) +
           (acc ? (size_t)tab * K * (S::row_stride + 1) * sizeof(float) : 0) + sizeof(TcShared) + 16;
}

template <int D, bool ACC, int TAB>
int tc_launch(ibcu_ctx* ctx, long blocks, const float* X, long N, const float* C, int K, int32_t* idx, float* dist,
              float* part_sums, int32_t* part_counts, double* part_inertia) {
    const size_t smem = tc_smem_bytes<D>(K, ACC, TAB);
    static SmemOptIn opt;
    if (int rc = ibcu_allow_smem(ctx, opt, assign_tc_kernel<D, ACC, TAB>, smem)) return rc;
    return ibcu_launch(ctx, assign_tc_kernel<D, ACC, TAB>, dim3((unsigned)blocks), dim3((TC_SCAN_WARPS + TC_FIN_WARPS + TC_PIPES) * 32), smem, 1, true,
                       X, N, C, K, idx, dist, ctx->kern_err, part_sums, part_counts, part_inertia);
}

constexpr size_t TC_SMEM_MAX = 227 * 1024;

}  // namespace

// The calls the tensor-memory kernel takes: 4, 8 or 16 dimensions, up to 256 centroids, points at 16 bytes (their rows then are
// too). Tiles are counted in an int.
bool ibcu_kmeans_tc_takes(const float* X, long N, int D, int K) {
    return (D == 4 || D == 8 || D == 16) && K >= 1 && K <= 256 && ((uintptr_t)X & 15) == 0 && N <= (1L << 37);
}
long ibcu_kmeans_tc_blocks(long N) {
    const long ntile = (N + TC_TILE - 1) / TC_TILE;
    return ntile < TC_BLOCKS ? ntile : TC_BLOCKS;
}

// Returns IBCU_DECLINED without touching the context's error when the call is not its own (the caller takes another kernel).
int ibcu_kmeans_assign_tc(ibcu_ctx* ctx, const float* X, long N, int D, const float* C, int K, int32_t* idx, float* dist) {
    if (!ibcu_kmeans_tc_takes(X, N, D, K)) return IBCU_DECLINED;
    const long blocks = ibcu_kmeans_tc_blocks(N);
    switch (D) {
        case 4: return tc_launch<4, false, 12>(ctx, blocks, X, N, C, K, idx, dist, nullptr, nullptr, nullptr);
        case 8: return tc_launch<8, false, 12>(ctx, blocks, X, N, C, K, idx, dist, nullptr, nullptr, nullptr);
        default: return tc_launch<16, false, 12>(ctx, blocks, X, N, C, K, idx, dist, nullptr, nullptr, nullptr);
    }
}

// The assignment and the accumulate pass of a Lloyd iteration in one launch of ibcu_kmeans_tc_blocks blocks: per-block partial tables
// go to part_* (K * D sums, K counts and one inertia per block), which accumulate_finish_kernel then adds up. Same conditions
// and return convention as above.
int ibcu_kmeans_assign_accumulate_tc(ibcu_ctx* ctx, const float* X, long N, int D, const float* C, int K, int32_t* idx, float* dist,
                                     float* part_sums, int32_t* part_counts, double* part_inertia) {
    if (!ibcu_kmeans_tc_takes(X, N, D, K)) return IBCU_DECLINED;
    const long blocks = ibcu_kmeans_tc_blocks(N);
    switch (D) {
        case 4: return tc_launch<4, true, 12>(ctx, blocks, X, N, C, K, idx, dist, part_sums, part_counts, part_inertia);
        case 8: return tc_launch<8, true, 12>(ctx, blocks, X, N, C, K, idx, dist, part_sums, part_counts, part_inertia);
        // Twelve tables fit up to 125 clusters or so. Beyond, the three warps of a quarter share one: 1 Mi points, ten iterations, 256
        // clusters 1014 us (1152 with four finishing warps and a table each), 200 clusters 964 (1108), 128 clusters 820 (804 with eight).
        default:
            if (tc_smem_bytes<16>(K, true, 12) <= TC_SMEM_MAX) return tc_launch<16, true, 12>(ctx, blocks, X, N, C, K, idx, dist, part_sums, part_counts, part_inertia);
            return tc_launch<16, true, 4>(ctx, blocks, X, N, C, K, idx, dist, part_sums, part_counts, part_inertia);
    }
}
