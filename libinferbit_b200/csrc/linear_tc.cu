// Linear layers for several activations on the fifth-generation tensor cores (tcgen05.mma kind::i8, accumulators in
// tensor memory): the exact integer arithmetic of linear.cu as a GEMM, weights [rows x columns] times the four base-256
// digits ("limbs") of every activation, 4 B columns.
//
// xprep_tc_kernel, or xprep_tc_cluster_kernel with a cluster of blocks per activation (tq_prep), turns the activations into digits once, with one
// power-of-two scale per activation, and lays them out as the operand image: per block of 128 columns NC rows of 128 bytes, swizzled. linear_tc_kernel is a cluster of S blocks per
// run of up to 256 weight rows; block r of the cluster takes the r-th part of the columns. Per 128-column block of its part
// TMA brings the weights of all rows of the run (one box, rows the tensor lacks are not fetched) and one bulk copy the
// digits. INT8 weights are the A operand as they land. INT4 nibbles go to tensor memory as bytes (worker warps: four
// 16-byte shared-memory reads, two masks per word, one tcgen05.st per row and block) and the MMA takes A from there: writing
// the widened bytes back to shared memory for the MMA to read again would cost four times the bytes of the nibbles there,
// and shared-memory bandwidth is what an M = 128 integer MMA of 128 columns uses up first.
// All digit sums are exact int32, recombined to one int64 per (row, activation); the S parts of a run meet in the blocks'
// shared memory (distributed shared memory, every block finishes the activations b = rank mod S), are added as integers and
// converted once: the result does not depend on S or on how the rows are dealt.
// No warp polls a barrier while it would have to poll until the kernel ahead has ended: everyone sleeps in the dependency wait.
// (When the warps of weights and MMAs polled their barriers meanwhile, with suspended tries, the end of the kernel ahead was in
// rare cases - once in tens of thousands of launches - not delivered until they gave up.)
// Workers (INT4 widening, then epilogue): four warps per tile of 128 rows and team; the teams take the blocks of columns in turn;
// then one warp each for the weights (TMA), the digits (bulk copies) and the MMAs. What a block of columns costs a warp is waits
// and latencies one behind the other, not work: with two teams instead of one, gate and up of 14336 x 4096 INT4 at eight
// activations went from 22.0 to 18.0 us and 4096 x 14336 from 19.3 to 16.4. No single pipe bounds it: 4096 x 14336 at 32 activations took 19.9 us, 19.8 without the
// transfer of the digits (which every SM reads from L2, 56 MB of them), 19.1 without three of four MMAs, 19.2 without the weights, 9.9 with one block of columns. Four teams for some runs of one tile (tq_teams): 4096 x 4096 INT4 at 4, 16 and 32 activations 8.3 -> 7.5, 9.2 -> 8.9,
// 12.4 -> 11.5, 2560 x 6400 at 32 14.3 -> 13.3, 4096 x 14336 at 32 20.7 -> 19.8.
// The weights do not depend on the kernel ahead: their ring fills before the dependency wait.
#include "common.cuh"
#include "tc_common.cuh"
#include "xconvert.cuh"
#include <cudaTypedefs.h>

bool ibcu_push_match(ibcu_ctx* ctx, float* const* outs, int n);      // comm.cu
void ibcu_push_fill(ibcu_ctx* ctx, GatherPush* gp, size_t bytes);

namespace {

// Warps of a block whose runs have T tiles: Q teams of 4 T workers, then one each for the weights, the digits and the MMAs.
template <int T, int Q> struct Tq { static constexpr int WORKERS = 4 * T * Q, A_WARP = WORKERS, B_WARP = WORKERS + 1, MMA_WARP = WORKERS + 2, THREADS = (WORKERS + 3) * 32; };
constexpr int TQ_MAX_STAGES = 12;
constexpr int TQ_MAX_B = 32;

struct alignas(64) TqMaps { CUtensorMap m[4]; };

struct TqParams {
    LinTensor t[4];
    int n_tensors, run_start[5];               // runs of tensor i are [run_start[i], run_start[i + 1])
    int R, NC, B, nkb, S;                      // rows per run (a multiple of 8), MMA columns, activations, 128-column blocks per row, cluster size
    int sa, sb, a_stage;                       // ring depths (weights; digits), bytes of a weight stage (one block of columns)
    int gb;                                    // blocks of columns per digit stage
    int recv_off;                              // where the parts of a run meet in shared memory; 0: in the rings, once they are free
    int tmem_cols, xparts;
    const int8_t* xtiles;                      // digit image [nkb][NC][128]
    const float* xscale;                       // [B][xparts], equal over the parts
    const int* xsum;                           // [B][xparts][4] digit sums (INT4 bias)
    GatherPush gp;
    int* err;
};

struct TqShared {
    unsigned long long full_a[TQ_MAX_STAGES], empty_a[TQ_MAX_STAGES];    // weights -> MMA (INT8) or widening warps (INT4), and back
    unsigned long long full_b[TQ_MAX_STAGES], empty_b[TQ_MAX_STAGES];    // digits -> MMA, and back
    unsigned long long full_t[4], empty_t[4];                            // INT4: widened blocks in tensor memory -> MMA, and back
    unsigned long long full_acc, empty_acc, drained;
    uint32_t tmem_base;
    int abort_flag;
    float back[TQ_MAX_B];
    long long bias[TQ_MAX_B];
};

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 :: "r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void mma_i8_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
                 :: "r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void mma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                 :: "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// the four digit sums of one (row, activation) as one integer
__device__ __forceinline__ long long join_limbs(const uint32_t* a) {
    return (((long long)(int)a[3] * 256 + (int)a[2]) * 256 + (int)a[1]) * 256 + (int)a[0];
}
__device__ __forceinline__ float row_scale(const LinTensor& W, int row) {
    return W.scales_fp32 ? reinterpret_cast<const float*>(W.scales)[row] : __half2float(reinterpret_cast<const __half*>(W.scales)[row]);
}

// grid (parts, B): digits of one activation (or of one part of its columns when the caller knows the maximum)
template <int T, bool MG>       // MG: see linear.cu
__global__ void __launch_bounds__(T) xprep_tc_kernel(const XSource src, int N, int part_cols, int all_cols, int nc, int perm8, int8_t* __restrict__ xtiles,
                                                     float* __restrict__ xscale, int* __restrict__ xsum, const GatherWait gw) {
    __shared__ XScratch sc;
    pdl_launch_dependents();
    pdl_wait();
    if (MG) gather_wait(gw);
    const int part = blockIdx.x, b = blockIdx.y, c0 = part * part_cols;
    const XTiles dst = { xtiles, nc, b * LIN_LIMBS, c0 };
    xconvert_any(src, N, b, c0, min(part_cols, all_cols - c0), dst, perm8, sc, xscale + b * gridDim.x + part, xsum + ((size_t)b * gridDim.x + part) * LIN_LIMBS);
}

// The same by a cluster of blocks per activation, a part of its columns each and eight columns a thread: one round trip to memory, and the parts' maxima and
// sums of squares meet in shared memory. Rows of up to IBCU_PREPARED_COLUMNS columns. src.op: none, RMSNorm or silu(x) * x2.
constexpr int XCL_PARTS = 8, XCL_COLS = IBCU_PREPARED_COLUMNS / XCL_PARTS;
template <bool MG>       // MG: see linear.cu
__global__ void __launch_bounds__(XCL_COLS / 8) xprep_tc_cluster_kernel(const XSource src, int N, int part_cols, int all_cols, int nc, int perm8, int8_t* __restrict__ xtiles,
                                                                        float* __restrict__ xscale, int* __restrict__ xsum, const GatherWait gw) {
    constexpr int WARPS = XCL_COLS / 256;
    __shared__ float2 warps[WARPS], parts[XCL_PARTS];         // max, sum of squares
    __shared__ int sums[WARPS][LIN_LIMBS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, part = blockIdx.x, nparts = gridDim.x, b = blockIdx.y;
    const int col = part * part_cols + tid * 8;
    const bool mine = tid * 8 < part_cols && col < all_cols, have = mine && col < N;
    pdl_launch_dependents();
    // Waited for before the first store into a peer's shared memory: by then every block has started. Nothing has been written yet, so nothing is
    // released (with a release, ahead of the line above, 2048 x 5632 with silu at 6 activations took 8.7 us instead of 8.4).
    cluster_arrive_relaxed();
    float4 w0 = make_float4(1.0f, 1.0f, 1.0f, 1.0f), w1 = w0;
    if (src.op == IBCU_PRO_RMSNORM && have) {                 // weights: the kernel ahead does not write them
        const __half2* h = reinterpret_cast<const __half2*>(src.norm_w + col);                          // 4-byte aligned at least
        const float2 p0 = __half22float2(h[0]), p1 = __half22float2(h[1]), p2 = __half22float2(h[2]), p3 = __half22float2(h[3]);
        w0 = make_float4(p0.x, p0.y, p1.x, p1.y); w1 = make_float4(p2.x, p2.y, p3.x, p3.y);
    }
    pdl_wait();
    if (MG) gather_wait(gw);
    float4 u = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v = u;
    if (have) {
        const float4* x = reinterpret_cast<const float4*>(src.x + (size_t)b * N + col);
        u = __ldcg(x); v = __ldcg(x + 1);
        if (src.op == IBCU_PRO_SILU_MUL) {
            const float4* x2 = reinterpret_cast<const float4*>(src.x2 + (size_t)b * N + col);
            const float4 p = __ldcg(x2), q = __ldcg(x2 + 1);
            u.x = u.x / (1.0f + expf(-u.x)) * p.x; u.y = u.y / (1.0f + expf(-u.y)) * p.y; u.z = u.z / (1.0f + expf(-u.z)) * p.z; u.w = u.w / (1.0f + expf(-u.w)) * p.w;
            v.x = v.x / (1.0f + expf(-v.x)) * q.x; v.y = v.y / (1.0f + expf(-v.y)) * q.y; v.z = v.z / (1.0f + expf(-v.z)) * q.z; v.w = v.w / (1.0f + expf(-v.w)) * q.w;
        }
    }
    float ss = fmaf(u.x, u.x, fmaf(u.y, u.y, fmaf(u.z, u.z, u.w * u.w)));
    ss = warp_sum(fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss)))));
    float mx = fmaxf(fmaxf(fabsf(u.x * w0.x), fabsf(u.y * w0.y)), fmaxf(fabsf(u.z * w0.z), fabsf(u.w * w0.w)));
    mx = warp_max(fmaxf(mx, fmaxf(fmaxf(fabsf(v.x * w1.x), fabsf(v.y * w1.y)), fmaxf(fabsf(v.z * w1.z), fabsf(v.w * w1.w)))));
    if (lane == 0) warps[warp] = make_float2(mx, ss);
    __syncthreads();
    cluster_wait();
    if (tid < nparts) {                                       // this part's into every block of the cluster
        float2 m = warps[0];
#pragma unroll
        for (int q = 1; q < WARPS; q++) { m.x = fmaxf(m.x, warps[q].x); m.y += warps[q].y; }
        uint32_t remote;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(&parts[part])), "r"(tid));
        asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" :: "r"(remote), "f"(m.x), "f"(m.y) : "memory");
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    float vmax = 0.0f, t = 0.0f, r = 1.0f;
    for (int q = 0; q < nparts; q++) { vmax = fmaxf(vmax, parts[q].x); t += parts[q].y; }
    if (src.op == IBCU_PRO_RMSNORM) {                         // 1/sqrt(mean(x^2) + eps) (src/kernels/scalar.c:126-138)
        r = 1.0f / sqrtf(t / (float)N + src.eps);
        vmax *= r;                                            // within a rounding of the largest magnitude: the digits have a bit to spare
    }
    const int e = (int)((__float_as_uint(vmax) >> 23) & 0xFF);
    int sh = (vmax > 0.0f && e != 255) ? 156 - e : 0;         // 2^sh vmax in [2^29, 2^30)
    sh = max(-126, min(126, sh));
    const float mul = __uint_as_float((uint32_t)(127 + sh) << 23);
    if (tid == 0) xscale[b * nparts + part] = __uint_as_float((uint32_t)(127 - sh) << 23);
    int lsum[LIN_LIMBS] = { 0, 0, 0, 0 };
    if (mine) {
        int X[8];
        X[0] = __float2int_rn(u.x * r * w0.x * mul); X[1] = __float2int_rn(u.y * r * w0.y * mul); X[2] = __float2int_rn(u.z * r * w0.z * mul); X[3] = __float2int_rn(u.w * r * w0.w * mul);
        X[4] = __float2int_rn(v.x * r * w1.x * mul); X[5] = __float2int_rn(v.y * r * w1.y * mul); X[6] = __float2int_rn(v.z * r * w1.z * mul); X[7] = __float2int_rn(v.w * r * w1.w * mul);
        uint2 pk[LIN_LIMBS];
        limbs8(X, perm8, pk, lsum);
        const XTiles dst = { xtiles, nc, b * LIN_LIMBS, part * part_cols };
#pragma unroll
        for (int l = 0; l < LIN_LIMBS; l++) dst.put(l, tid * 8, pk[l]);
    }
    if (!perm8) return;                                       // the digits' sums only take the bias off INT4 nibbles
#pragma unroll
    for (int l = 0; l < LIN_LIMBS; l++) {
        const int s = __reduce_add_sync(0xffffffffu, lsum[l]);
        if (lane == 0) sums[warp][l] = s;
    }
    __syncthreads();
    if (tid < LIN_LIMBS) {
        int s = 0;
#pragma unroll
        for (int q = 0; q < WARPS; q++) s += sums[q][tid];
        xsum[((size_t)b * nparts + part) * LIN_LIMBS + tid] = s;
    }
}

// BITS 4 or 8; T: 128-row tiles per run; Q: teams of workers; MG: see linear.cu
template <int BITS, int T, int Q, bool MG>
__global__ void __launch_bounds__(Tq<T, Q>::THREADS, T * Q == 2 ? 2 : 1) linear_tc_kernel(const __grid_constant__ TqMaps maps, const __grid_constant__ TqParams p) {
    extern __shared__ __align__(1024) unsigned char tq_smem[];
    constexpr int NT = 4;                                      // INT4: widened blocks in tensor memory
    using W = Tq<T, Q>;
    constexpr int TQ_WORKERS = W::WORKERS, TQ_A_WARP = W::A_WARP, TQ_B_WARP = W::B_WARP, TQ_MMA_WARP = W::MMA_WARP, TQ_THREADS = W::THREADS;
    // INT4: Q teams of workers, a warp per 32 rows, widen every Q-th block of columns. A warp's way from the nibbles to the MMA is
    // a chain of waits and latencies (about 1300 cycles measured, a few hundred of them work), and Q chains run side by side.
    constexpr int TW = TQ_WORKERS / Q;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int S = p.S, rank = (int)blockIdx.x % S, cl = (int)blockIdx.x / S, ncl = (int)gridDim.x / S;
    const int nruns = p.run_start[p.n_tensors];
    const int k0 = (int)((long)p.nkb * rank / S), k1 = (int)((long)p.nkb * (rank + 1) / S);
    unsigned char* ringA = tq_smem;
    unsigned char* ringB = tq_smem + (((size_t)p.sa * p.a_stage + 1023) & ~(size_t)1023);
    const int b_block = p.NC * 128, b_stage = p.gb * b_block;
    size_t ring_bytes = (size_t)(ringB - tq_smem) + (size_t)p.sb * b_stage;
    if (BITS == 8 && ring_bytes < (size_t)p.sa * p.a_stage + T * 16384) ring_bytes = (size_t)p.sa * p.a_stage + T * 16384;   // an MMA reads 128 rows whatever the run has
    if (p.recv_off) ring_bytes = p.recv_off + (size_t)S * ((p.B + S - 1) / S) * T * 1024;
    TqShared* sh = reinterpret_cast<TqShared*>(tq_smem + ((ring_bytes + 15) & ~(size_t)15));
    volatile int* abort_flag = &sh->abort_flag;

    if (tid == 0) {
        for (int s = 0; s < TQ_MAX_STAGES; s++) {
            mbar_init(smem_u32(&sh->full_a[s]), 1); mbar_init(smem_u32(&sh->empty_a[s]), BITS == 8 ? 1 : TW);
            mbar_init(smem_u32(&sh->full_b[s]), 1); mbar_init(smem_u32(&sh->empty_b[s]), 1);
        }
        for (int s = 0; s < NT; s++) { mbar_init(smem_u32(&sh->full_t[s]), TW); mbar_init(smem_u32(&sh->empty_t[s]), 1); }
        mbar_init(smem_u32(&sh->full_acc), 1); mbar_init(smem_u32(&sh->empty_acc), TQ_WORKERS); mbar_init(smem_u32(&sh->drained), 1);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (S > 1) cluster_arrive();                               // waited for before the first store into a peer's shared memory: by then every block has started

    // Blocks of a launch start at different blocks of columns: all of them read the same digits, fresh from the preparation
    // kernel, and reading the same lines at the same moment they queue for them. (Integer sums: the order is free.)
    const int nk = k1 - k0, rot = nk % p.gb == 0 ? (cl * p.gb) % nk : 0;
    auto column_block = [&](int i) { const int k = i + rot; return k0 + (k < nk ? k : k - nk); };
    auto tensor_of = [&](int run, int& ti, int& row0) {
        ti = 0;
#pragma unroll
        for (int i = 1; i < 4; i++) if (i < p.n_tensors && run >= p.run_start[i]) ti = i;
        row0 = (run - p.run_start[ti]) * p.R;
    };

    // weights: the ring fills at once, before tensor memory is there and before the kernel ahead has ended
    if (warp == TQ_A_WARP) {
        const bool one = elect_one();
        int s = 0; uint32_t ph = 1;                             // a fresh ring is free
        bool ok = true;
        long n = 0;
        for (int run = cl; run < nruns && ok; run += ncl) {
            int ti, row0;
            tensor_of(run, ti, row0);
            for (int i = 0; i < nk; i++, n++) {
                const int kb = column_block(i);
                if (n == p.sa) pdl_wait();                      // see below: nobody polls a barrier while the kernel ahead runs
                if (one) {
                    ok = mbar_wait(smem_u32(&sh->empty_a[s]), ph, abort_flag, 1);
                    if (ok) {
                        mbar_expect_tx(smem_u32(&sh->full_a[s]), (uint32_t)p.R * (BITS == 8 ? 128u : 64u));
                        tma_load_2d(smem_u32(ringA + (size_t)s * p.a_stage), &maps.m[ti], kb * (BITS == 8 ? 128 : 64), row0, smem_u32(&sh->full_a[s]));
                    }
                }
                ok = __any_sync(0xffffffffu, one && ok);
                if (!ok) break;
                if (++s == p.sa) { s = 0; ph ^= 1; }
            }
        }
        __syncwarp();
    }
    if (warp == TQ_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&sh->tmem_base)), "r"((uint32_t)p.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        // Only now may the launches behind this one start: their blocks allocate tensor memory too and keep it until this launch
        // has ended, so every block of this launch must hold its own first.
        pdl_launch_dependents();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    // everyone but the weight warp, which is still filling its ring, needs the tensor-memory address
    if (warp != TQ_A_WARP) asm volatile("bar.sync 1, %0;" :: "n"(TQ_THREADS - 32) : "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = warp == TQ_A_WARP ? 0u : sh->tmem_base;
    const uint32_t tmem_a = tmem_base + (uint32_t)(T * p.NC);                          // INT4: NT blocks of T x 32 columns

    if (warp == TQ_B_WARP) {
        pdl_wait();
        if (elect_one()) {
            int s = 0; uint32_t ph = 1;
            bool ok = true;
            for (int run = cl; run < nruns && ok; run += ncl)
                for (int i = 0; i < nk; i += p.gb) {
                    const int kb = column_block(i);
                    ok = mbar_wait(smem_u32(&sh->empty_b[s]), ph, abort_flag, 2);
                    if (!ok) break;
                    const uint32_t bytes = (uint32_t)(min(p.gb, nk - i) * b_block);
                    mbar_expect_tx(smem_u32(&sh->full_b[s]), bytes);
                    bulk_load(smem_u32(ringB + (size_t)s * b_stage), p.xtiles + (size_t)kb * b_block, bytes, smem_u32(&sh->full_b[s]));
                    if (++s == p.sb) { s = 0; ph ^= 1; }
                }
        }
        __syncwarp();
    } else if (warp == TQ_MMA_WARP) {
        pdl_wait();
        if (elect_one()) {
            // s32 accumulators; A unsigned bytes for widened nibbles, signed for INT8; B signed digits
            const uint32_t idesc = (2u << 4) | ((BITS == 8 ? 1u : 0u) << 7) | (1u << 10) | ((uint32_t)(p.NC >> 3) << 17) | (8u << 24);
            const uint32_t ra = smem_u32(ringA), rb = smem_u32(ringB);
            const int na = BITS == 8 ? p.sa : NT;                                       // weight stages, or widened blocks
            unsigned long long* full_a = BITS == 8 ? sh->full_a : sh->full_t;
            unsigned long long* empty_a = BITS == 8 ? sh->empty_a : sh->empty_t;
            int sa = 0, sb = 0, j = 0;
            uint32_t pha = 0, phb = 0;
            bool ok = true;
            for (int run = cl; run < nruns && ok; run += ncl, j++) {
                ok = mbar_wait(smem_u32(&sh->empty_acc), (uint32_t)((j & 1) ^ 1), abort_flag, 3);
                for (int i = 0; i < nk && ok;) {
                    ok = mbar_wait(smem_u32(&sh->full_b[sb]), phb, abort_flag, 4);
                    const int ie = min(i + p.gb, nk);
                    uint64_t bd = smem_desc_sw128(rb + (uint32_t)(sb * b_stage));
                    for (; i < ie && ok; i++, bd += (uint64_t)(b_block >> 4)) {
                        ok = mbar_wait(smem_u32(&full_a[sa]), pha, abort_flag, 5);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint64_t ad = smem_desc_sw128(ra + (uint32_t)(sa * p.a_stage));
#pragma unroll
                        for (int m = 0; m < 4; m++) {                                  // 32 columns each: descriptors count 16-byte units
#pragma unroll
                            for (int tt = 0; tt < T; tt++) {
                                const uint32_t d = tmem_base + (uint32_t)(tt * p.NC);
                                if (BITS == 8) mma_i8_ss(d, ad + tt * 1024 + m * 2, bd + m * 2, idesc, (i | m) ? 1u : 0u);
                                else mma_i8_ts(d, tmem_a + (uint32_t)((sa * T + tt) * 32 + m * 8), bd + m * 2, idesc, (i | m) ? 1u : 0u);
                            }
                        }
                        mma_commit(smem_u32(&empty_a[sa]));
                        if (++sa == na) { sa = 0; pha ^= 1; }
                    }
                    if (ok) mma_commit(smem_u32(&sh->empty_b[sb]));
                    if (++sb == p.sb) { sb = 0; phb ^= 1; }
                }
                if (ok) mma_commit(smem_u32(&sh->full_acc));
            }
            mma_commit(smem_u32(&sh->drained));
            mbar_wait(smem_u32(&sh->drained), 0u, abort_flag, 7);                      // nothing of this block is left in the tensor pipe
        }
        __syncwarp();
    } else if (warp < TQ_WORKERS) {
        const int q = warp & 3, rt = (warp >> 2) % T, team = warp / (4 * T);           // tensor-memory quarter, tile, and which blocks (INT4) / groups of activations
        int s = team, sT = team, j = 0, next = team;                                   // next: this team's next block of columns, counted from the run's first
        uint32_t phA = 0, phT = 1;
        bool alive = true, staged = false, waited = false;
        for (int run = cl; run < nruns && alive; run += ncl, j++) {
            int ti, row0;
            tensor_of(run, ti, row0);
            const LinTensor& W = p.t[ti];
            const int rows = min(p.R, W.M - row0);
            const int rl = rt * 128 + q * 32 + lane;                                    // this thread's row of the run
            if (BITS == 4) {
                const uint32_t rawrow = (uint32_t)rl * 64u, sw = (uint32_t)((rl >> 1) & 3);
                const bool have = rt * 128 + q * 32 < p.R;                              // the box has rows for this warp
                for (; next < nk; next += Q) {
                    if (!waited && next >= NT) { pdl_wait(); waited = true; }           // the first widened blocks do not need the digits; the next wait for them to be used
                    if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->full_a[s]), phA, abort_flag, 8))) { alive = false; break; }
                    uint32_t o[32];
                    if (have) {
                        const unsigned char* raw = ringA + (size_t)s * p.a_stage + (rl < p.R ? rawrow : 0u);
#pragma unroll
                        for (int c = 0; c < 4; c++) {                                  // the 64-byte swizzle: piece c of row r at piece c ^ (r / 2 % 4)
                            const uint4 v = *reinterpret_cast<const uint4*>(raw + (((uint32_t)c ^ sw) << 4));
                            const uint32_t w[4] = { v.x, v.y, v.z, v.w };
#pragma unroll
                            for (int u = 0; u < 4; u++) { o[c * 8 + 2 * u] = w[u] & 0x0F0F0F0Fu; o[c * 8 + 2 * u + 1] = (w[u] >> 4) & 0x0F0F0F0Fu; }
                        }
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&sh->empty_a[s]));              // the nibbles are in registers
                    if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->empty_t[sT]), phT, abort_flag, 9))) { alive = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (have) {
                        tmem_st32(tmem_a + ((uint32_t)(q * 32) << 16) + (uint32_t)((sT * T + rt) * 32), o);
                        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&sh->full_t[sT]));
                    s += Q;
                    if (s >= p.sa) { s -= p.sa; phA ^= 1; }
                    sT += Q;
                    if (sT >= NT) { sT -= NT; phT ^= 1; }
                }
                next -= nk;
                if (!alive) break;
            }
            if (!staged) {
                // what the preparation kernel left: 2^-s and 8 x the digit sum of every activation
                pdl_wait();
                if (tid < p.B) {
                    sh->back[tid] = p.xscale[tid * p.xparts];
                    long long sum = 0;
                    if (BITS == 4)
                        for (int part = 0; part < p.xparts; part++) sum += join_limbs(reinterpret_cast<const uint32_t*>(p.xsum) + ((size_t)tid * p.xparts + part) * LIN_LIMBS);
                    sh->bias[tid] = 8 * sum;
                }
                asm volatile("bar.sync 2, %0;" :: "n"(TQ_WORKERS * 32) : "memory");
                staged = true;
            }
            if (S == 1) {
                const bool have = rl < rows;
                const int row = row0 + rl;
                const float sc = have ? row_scale(W, row) : 0.0f;
                const unsigned tag = MG ? tag_current(p.gp) : 0u;
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->full_acc), (uint32_t)(j & 1), abort_flag, 10))) { alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int g = team; g * 4 < p.B; g += Q) {
                    uint32_t acc[16];
                    tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(rt * p.NC + g * 16), acc);
                    float* o = W.out + (size_t)(g * 4) * W.out_stride + row;
                    float old[4] = { 0.0f, 0.0f, 0.0f, 0.0f };
                    if (W.epilogue == IBCU_EPI_ADD) {
#pragma unroll
                        for (int u = 0; u < 4; u++) if (have && g * 4 + u < p.B) old[u] = o[(size_t)u * W.out_stride];
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int b = g * 4 + u;
                        if (b >= p.B || !have) continue;
                        const long long V = join_limbs(acc + 4 * u) - (BITS == 4 ? sh->bias[b] : 0ll);
                        const float y = (float)((double)V * (double)sh->back[b]);
                        const float v = W.epilogue == IBCU_EPI_ADD ? old[u] + y * sc : y * sc;
                        o[(size_t)u * W.out_stride] = v;
                        if (MG) tag_push(p.gp, (size_t)W.win_off + ((size_t)b * W.out_stride + row) * sizeof(float), v, tag);
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sh->empty_acc));                   // the tensor cores may overwrite the accumulators
            } else {
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->full_acc), 0u, abort_flag, 10))) { alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
        }
        if (!staged) asm volatile("bar.sync 2, %0;" :: "n"(TQ_WORKERS * 32) : "memory");    // a warp that gave up: the others may be waiting there
    }
    if (S > 1) {
        // One run per cluster: the parts of the columns meet; block b mod S takes activation b. A meeting place inside the rings
        // is free once every block's MMAs are done; one of its own only needs the peers to have started.
        __syncwarp();
        cluster_wait();
        if (!p.recv_off) { cluster_arrive(); cluster_wait(); }
        const int BL = (p.B + S - 1) / S;                                               // activations per block
        constexpr int RP = T * 128;
        int ti, row0;
        tensor_of(cl, ti, row0);
        const LinTensor& W = p.t[ti];
        const int rows = min(p.R, W.M - row0);
        const uint32_t recv = smem_u32(tq_smem + p.recv_off);                           // [source block][activation][row] int64
        if (warp < TQ_WORKERS && !*abort_flag) {
            const int q = warp & 3, rt = (warp >> 2) % T, team = warp / (4 * T), rl = rt * 128 + q * 32 + lane;
            if (rt * 128 + q * 32 < rows) {
                for (int g = team; g * 4 < p.B; g += Q) {
                    uint32_t acc[16];
                    tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(rt * p.NC + g * 16), acc);
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int b = g * 4 + u;
                        if (b >= p.B) continue;
                        const uint32_t mine = recv + (uint32_t)(((rank * BL + b / S) * RP + rl) * 8);
                        uint32_t remote;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(mine), "r"(b % S));
                        asm volatile("st.shared::cluster.u64 [%0], %1;" :: "r"(remote), "l"(join_limbs(acc + 4 * u)) : "memory");
                    }
                }
            }
        }
        __syncwarp();
        cluster_arrive();
        // a thread finishes one row; what it needs from memory is under way while the parts arrive
        const int frl = tid % RP, row = row0 + frl;
        const bool mine = warp < TQ_WORKERS && frl < rows;
        const int nb = (p.B - rank + S - 1) / S, bl0 = tid / RP;
        constexpr int BSTEP = TQ_WORKERS * 32 / RP;
        const float sc = mine ? row_scale(W, row) : 0.0f;
        float old = mine && bl0 < nb && W.epilogue == IBCU_EPI_ADD ? W.out[(size_t)(bl0 * S + rank) * W.out_stride + row] : 0.0f;
        cluster_wait();
        if (mine && !*abort_flag) {
            const unsigned tag = MG ? tag_current(p.gp) : 0u;
            const long long* rv = reinterpret_cast<const long long*>(tq_smem + p.recv_off);
            for (int bl = bl0; bl < nb; bl += BSTEP) {
                const int b = bl * S + rank;
                float* o = W.out + (size_t)b * W.out_stride + row;
                const float next = bl + BSTEP < nb && W.epilogue == IBCU_EPI_ADD ? W.out[(size_t)((bl + BSTEP) * S + rank) * W.out_stride + row] : 0.0f;
                long long V = BITS == 4 ? -sh->bias[b] : 0ll;
                for (int k = 0; k < S; k++) V += rv[(size_t)(k * BL + bl) * RP + frl];
                const float y = (float)((double)V * (double)sh->back[b]);
                const float v = W.epilogue == IBCU_EPI_ADD ? old + y * sc : y * sc;
                *o = v;
                if (MG) tag_push(p.gp, (size_t)W.win_off + ((size_t)b * W.out_stride + row) * sizeof(float), v, tag);
                old = next;
            }
        }
    }
    // ── the end: tensor memory back, a wait that ran out reported ──
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == TQ_MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem_base), "r"((uint32_t)p.tmem_cols) : "memory");
    }
    if (tid == 0 && sh->abort_flag) {
        *p.err = 100 + sh->abort_flag;
        for (int i = 0; i < 1000; i++) __nanosleep(1000);      // copies still on their way into this block's shared memory land before it goes
    }
}

// ── host ──
using EncodeFn = PFN_cuTensorMapEncodeTiled_v12000;
EncodeFn encode_fn() {
    static EncodeFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult r;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess) { cudaGetLastError(); f = nullptr; }
        return (EncodeFn)f;
    }();
    return fn;
}

// How a call's digits are prepared: parts blocks of part_kb blocks of columns each per activation, as a cluster or not.
struct TqPrep { bool clustered; int parts, part_kb; };
TqPrep tq_prep(const TqCut& cut, int bits, int B, int op) {
    TqPrep x = { false, 1, cut.nkb };
    int blocks = 1;                                           // of a cluster
    while (blocks * XCL_COLS < cut.nkb * 128) blocks *= 2;
    // Clusters of INT4 runs of two tiles in clusters of four (19 warps of 96 registers on 132 SMs) leave clusters of four and eight blocks no room.
    const bool crowded = bits == 4 && cut.T == 2 && cut.S == 4 && blocks >= 4;
    // A cluster per activation, us, one block and a cluster. silu(x) * x2: always (936 calls: 0.73 of the time on the mean, 1.01 at most).
    // RMSNorm: 4096 x 4096 INT8 at 8, 16 and 32 8.9 and 8.2, 10.5 and 10.1, 12.8 and 11.9, 4096 x 14336 at 32 22.1 and 21.1; crowded: 5120 x 5120 at 8, 20 and 32 10.1 and 11.3,
    // 13.3 and 14.9, 16.7 and 16.6; clusters of eight ahead of runs of two tiles: 935 + 8677 x 10848 INT4 at 4 and 8 20.7 and 22.4, 23.4 and 22.7, 4463 + 279 x 13120 INT8 at 4 17.2 and 18.5, 4500 x 9600 INT8 at 6 14.5 and 13.8. Without a prologue there is no sum to wait for: beyond 16 activations, INT4 3072 + 1024 + 1024 x 3072 at 20 12.2 and 10.7,
    // 3072 + 3072 x 1024 at 32 10.2 and 8.6, 4096 x 4096 INT8 at 20 and 32 10.7 and 11.1, 11.9 and 11.8; but INT4 2560 x 6400 at 17 11.3 and 13.0, INT8 6400 + 6400 x 2560 at 24
    // 14.4 and 15.6, 10000 x 2560 at 24 15.4 and 16.2, 2048 x 6144 INT4, in clusters of eight, at 32 11.6 and 12.3.
    if (cut.nkb * 128L <= IBCU_PREPARED_COLUMNS) {
        if (op == IBCU_PRO_SILU_MUL) x.clustered = true;
        if (op == IBCU_PRO_RMSNORM) x.clustered = (!crowded || B > 20) && (cut.T == 1 || cut.S == 1 || blocks < 8 || B >= (bits == 8 ? 5 : 8));
        if (op == IBCU_PRO_NONE) x.clustered = B > 16 && ((cut.S == 4 && !crowded && (B > 20 || (bits == 4 && blocks <= 2))) || (cut.S == 2 && blocks == 1));
    }
    // otherwise a block per activation, or several when the maximum is known
    if (op == IBCU_PRO_KNOWN_MAX) { x.parts = (cut.nkb + 15) / 16; if (x.parts > 8) x.parts = 8; }
    if (x.clustered) x.parts = blocks;
    x.part_kb = (cut.nkb + x.parts - 1) / x.parts;
    if (!x.clustered) x.parts = (cut.nkb + x.part_kb - 1) / x.part_kb;                 // a cluster may end with empty parts
    return x;
}

// Teams of widening warps (INT4). Runs of one tile have room for four (16 workers); two tiles fill the block with two, and INT8 weights need none. Clusters of eight keep
// to half an SM a block: sixteen of them with an SM to each block do not find room at once (2048 x 6144 INT8 at 4 and 32 activations 7.3 and 12.6, 12.1 and 17.8 us); that is two
// teams, with 80 registers, of which 32 bytes spill.
// Beside a block of four teams, 19 warps of 96 registers, no block of the next call's preparation finds registers (with 72 or 80 it does, but the block
// spills). Where that preparation does not fit on the SMs this launch leaves idle either, it starts late and two teams are the faster: us, two and four,
// 8192 x 2048 (none idle) at 6 8.7 and 9.6, 2560 x 6400 with RMSNorm at 8 9.3 and 11.0, 16384 x 2048 at 8 9.3 and 10.2; where it fits, or finds no room beside two teams
// either (rows of more than 2048 columns by one block), 4096 x 4096 with RMSNorm at 3 8.1 and 7.2, 8192 x 8192 at 4 16.9 and 15.8. Short parts of a row need more than eight
// activations to have work for four in the epilogue (3072 + 3072 x 1024 at 4 5.8 and 6.2, at 16 8.4 and 7.3), and beyond 24 that work weighs more than the late start.
// Against two teams with half an SM, 1296 calls: 0.854 of the time on the mean, 8 behind by more than 3 %, at most 10 %; four teams everywhere 0.871, 93, 14 %.
int tq_teams(int sm_count, int bits, const TqCut& cut, int B, int op, const TqPrep& x) {
    if (bits == 8 || cut.T == 2 || cut.S == 8) return 2;
    const int nk = (cut.nkb + cut.S - 1) / cut.S, idle = sm_count - cut.S * (cut.nruns < cut.slots ? cut.nruns : cut.slots);
    const int per_sm = x.clustered ? 5 : (x.part_kb * 128 <= 2048 ? 3 : 1);             // blocks of the preparation on an idle SM, by their registers
    if (B > 24 || (per_sm == 1 && nk >= 5)) return 4;
    if (op == IBCU_PRO_KNOWN_MAX && B > 4 && B <= 8) return 2;                          // at 8 3000 x 3008 6.5 and 7.2, 4096 x 4096 7.4 and 7.9
    if (x.parts * B > idle * per_sm) return 2;
    if (x.clustered && x.parts >= 4 && (x.parts > 4 || B > 4 || idle < 8)) return 2;    // clusters need their places in one group of SMs
    return nk >= 5 || B > 8 ? 4 : 2;
}

template <int BITS, int T, int Q, bool MG>
int launch_tc_mg(ibcu_ctx* ctx, const TqMaps& maps, const TqParams& p, int grid, size_t smem) {
    auto kern = linear_tc_kernel<BITS, T, Q, MG>;
    static SmemOptIn opt;
    if (int rc = ibcu_allow_smem(ctx, opt, kern, smem)) return rc;
    return ibcu_launch(ctx, kern, dim3(grid), dim3(Tq<T, Q>::THREADS), smem, p.S, true, maps, p);
}

template <int BITS, int T>
int launch_tc(ibcu_ctx* ctx, const TqMaps& maps, const TqParams& p, int teams, int grid, size_t smem) {
    if constexpr (BITS == 4 && T == 1) {
        if (teams == 4) return p.gp.world ? launch_tc_mg<4, 1, 4, true>(ctx, maps, p, grid, smem) : launch_tc_mg<4, 1, 4, false>(ctx, maps, p, grid, smem);
    }
    return p.gp.world ? launch_tc_mg<BITS, T, 2, true>(ctx, maps, p, grid, smem) : launch_tc_mg<BITS, T, 2, false>(ctx, maps, p, grid, smem);
}

}  // namespace

TqCut ibcu_linear_tc_cut(int sm_count, const ibcu_linear_t* tensors, int n_tensors, int N, int B) {
    TqCut c;
    long total_rows = 0;
    for (int i = 0; i < n_tensors; i++) total_rows += tensors[i].M;
    c.nkb = (N + 127) / 128;
    c.NC = (B * LIN_LIMBS + 15) / 16 * 16;
    // Columns over S blocks of a cluster: enough rows per block that the digits every block fetches stay few against the
    // weights, and no more than 256 of them.
    const int slots_of[4] = { sm_count, sm_count / 2, sm_count * 9 / 40, sm_count / 9 };
    int lg = 0;
    while (lg < 3 && total_rows / slots_of[lg] < 80 && c.nkb >= (4 << lg)) lg++;
    while (lg > 0 && (c.nkb < (1 << lg) || total_rows > 256L * slots_of[lg])) lg--;
    // A cluster of eight blocks of two tiles, an SM each, does not find room for all sixteen clusters at once: 2280 rows of 2048 columns at
    // four activations took 11.8 us, rows of 3840 at sixteen 16.4; four blocks of one tile take over there.
    for (;; lg--) {
        c.S = 1 << lg;
        c.slots = slots_of[lg];
        const long per = (total_rows + c.slots - 1) / c.slots;
        c.R = per > 256 ? 256 : (int)(per + 7) & ~7;
        for (;; c.R += 8) {
            c.nruns = 0;
            for (int i = 0; i < n_tensors; i++) c.nruns += (tensors[i].M + c.R - 1) / c.R;
            if (c.R >= 256 || c.nruns <= c.slots) break;
        }
        if (lg < 3 || c.R <= 128) break;
    }
    c.T = c.R > 128 ? 2 : 1;
    return c;
}

// The call as the preparation kernel and the tcgen05 kernel. Returns IBCU_DECLINED without touching the context's error when
// the call is not its own (the caller takes the other kernels).
int ibcu_linear_tc(ibcu_ctx* ctx, const ibcu_linear_t* tensors, int n_tensors, const float* x, int N, int B, int bits, const ibcu_prologue_t* pro, int op) {
    EncodeFn encode = encode_fn();
    const int rowbytes = bits == 8 ? N : N / 2;
    if (!encode || rowbytes % 16 || B > TQ_MAX_B) return IBCU_DECLINED;
    long total_rows = 0;
    for (int i = 0; i < n_tensors; i++) total_rows += tensors[i].M;
    if (total_rows == 0) return IBCU_OK;
    const TqCut cut = ibcu_linear_tc_cut(ctx->sm_count, tensors, n_tensors, N, B);
    const int S = cut.S, R = cut.R, T = cut.T, slots = cut.slots;
    TqParams p;
    memset(&p, 0, sizeof p);
    p.n_tensors = n_tensors; p.B = B; p.nkb = cut.nkb; p.NC = cut.NC;
    p.R = R; p.S = S;
    int nruns = 0;
    for (int i = 0, row = 0; i < n_tensors; i++) {
        p.t[i] = { (const uint8_t*)tensors[i].w, tensors[i].scales, tensors[i].out, tensors[i].M,
                   tensors[i].out_stride, tensors[i].scales_fp32, tensors[i].epilogue, row, 0, 0, -1 };
        p.run_start[i] = nruns;
        nruns += (tensors[i].M + R - 1) / R;
        row += tensors[i].M;
    }
    for (int i = n_tensors; i <= 4; i++) p.run_start[i] = nruns;
    if (S > 1 && nruns > slots) return IBCU_DECLINED;
    // a block adds up its part of the columns in s32: weights of up to 128 (INT4, before the bias is taken off: 15) times digits of
    // up to 128 stay exact for 131071 (1118481) columns; rows with longer parts go to the kernel that cuts them into slices
    const long part_cols = (long)((p.nkb + S - 1) / S) * 128;
    if ((part_cols < N ? part_cols : N) * (bits == 8 ? 128L : 15L) * 128L > 0x7fffffffL) return IBCU_DECLINED;
    // Shared memory: the rings take what an SM has. A block of runs of one tile used to keep to half, so that the next launch's blocks move in beside
    // it, but what a block of columns costs is the way of its weights and digits from L2, and with twice the ring twice as many are on it:
    // 4096 x 14336 INT4 at 4, 16 and 32 activations 15.0 -> 13.1, 18.1 -> 17.2, 25.3 -> 20.7 us, 6144 x 4096 INT8 at 4 and 32 9.9 -> 9.2,
    // 17.6 -> 16.0. INT8 at 9 to 20 activations keeps the overlap: an SM's ring against half of one, without a prologue, runs alone, in clusters of two and of four: at 8 0.98, 0.99, 0.96,
    // at 9 1.02, 1.00, 0.99, at 12 1.00, 1.00, 0.98, at 16 1.00, 0.99, 0.98, at 20 0.99, 1.00, 0.97, at 24 0.98, 0.95, 0.94 (22 shapes). So do clusters of eight (tq_teams).
    const int tcols = T * (p.NC + (bits == 4 ? 128 : 0));
    p.tmem_cols = 32;
    while (p.tmem_cols < tcols) p.tmem_cols *= 2;
    const size_t cap = (T == 1 && (S == 8 || (bits == 8 && p.NC > 32 && p.NC <= 80)) ? 111 : 200) * 1024 - sizeof(TqShared) - 2048;
    const size_t b_block = (size_t)p.NC * 128;
    p.a_stage = R * (bits == 8 ? 128 : 64);
    const int nk = (p.nkb + S - 1) / S;
    const TqPrep prep = tq_prep(cut, bits, B, op);
    const int teams = tq_teams(ctx->sm_count, bits, cut, B, op, prep);
    const size_t recv = S > 1 ? (size_t)S * ((B + S - 1) / S) * T * 128 * 8 : 0;
    const size_t spare = bits == 8 ? 16384 * T : 0;                                      // an MMA reads 128 rows whatever the run has
    // digit stages of at least 8 KB; the rings share the room in the proportion of what a block of columns takes of each
    p.gb = p.NC <= 16 ? 4 : (p.NC <= 32 ? 2 : 1);
    const size_t b_stage = p.gb * b_block;
    auto plan = [&](long room) {
        long n = room / (long)(p.a_stage + b_block);                                     // blocks of columns in flight
        if (n > nk && nruns <= slots) n = nk;
        p.sb = (int)((n + p.gb - 1) / p.gb);
        if (p.sb > TQ_MAX_STAGES) p.sb = TQ_MAX_STAGES;
        if (p.sb < 1) p.sb = 1;
        n = (room - (long)(p.sb * b_stage)) / p.a_stage;
        if (n > nk && nruns <= slots) n = nk;
        p.sa = n > TQ_MAX_STAGES ? TQ_MAX_STAGES : (int)n;
    };
    auto ring_of = [&]() {
        const size_t a = ((size_t)p.sa * p.a_stage + 1023) & ~(size_t)1023, r = a + (size_t)p.sb * b_stage;
        return spare && r < (size_t)p.sa * p.a_stage + spare ? (size_t)p.sa * p.a_stage + spare : r;
    };
    plan((long)cap - (long)recv - 1024);
    size_t smem;
    if (recv && p.sa >= (nk < 3 ? nk : 3) && ring_of() + recv + 1024 <= cap) {           // the meeting place beside the rings
        p.recv_off = (int)((ring_of() + 1023) & ~(size_t)1023);
        smem = p.recv_off + recv;
    } else {
        plan((long)cap);
        while (p.sa > 1 && ring_of() > cap) p.sa--;
        while (p.sa < TQ_MAX_STAGES && recv > ring_of()) p.sa++;
        if (recv > ring_of() || p.sa < 1) return IBCU_DECLINED;
        smem = ring_of();
    }
    if (bits == 4 && (p.sa < nk || nruns > slots)) {
        // a ring that is used again: a multiple of the teams, so that a stage always belongs to the same team of widening warps (a warp that
        // misses every other phase of a barrier cannot tell a phase from the next but one)
        if (p.sa < teams) return IBCU_DECLINED;
        p.sa -= p.sa % teams;
        if (!p.recv_off && recv > ring_of()) return IBCU_DECLINED;
        smem = p.recv_off ? smem : ring_of();
    }
    smem = ((smem + 15) & ~(size_t)15) + sizeof(TqShared);
    TqMaps maps;
    memset(&maps, 0, sizeof maps);
    for (int i = 0; i < n_tensors; i++) {
        if (tensors[i].M == 0) continue;
        const cuuint64_t dims[2] = { (cuuint64_t)rowbytes, (cuuint64_t)tensors[i].M };
        const cuuint64_t strides[1] = { (cuuint64_t)rowbytes };
        const cuuint32_t box[2] = { bits == 8 ? 128u : 64u, (cuuint32_t)R }, es[2] = { 1, 1 };
        if (encode(&maps.m[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(tensors[i].w), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   bits == 8 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return IBCU_DECLINED;
    }
    // The digits' room is there before a pending gather is taken: growing it may fail (under capture), and the call must then leave the gather to the next one.
    const int parts = prep.parts;
    p.xparts = parts;
    const size_t tiles = (size_t)p.nkb * b_block, scales = (((size_t)B * parts * sizeof(float)) + 255) & ~(size_t)255;
    int rc = ibcu_reserve(ctx, &ctx->xpack, &ctx->xpack_bytes, tiles + scales + (size_t)B * parts * LIN_LIMBS * sizeof(int));
    if (rc) return rc;
    GatherWait gw;
    ibcu_take_gather_wait_x(ctx, &gw, x, (size_t)B * N * sizeof(float));
    if (pro && pro->x2) ibcu_gather_wait_mark(ctx, &gw, pro->x2, (size_t)B * N * sizeof(float));
    ibcu_gather_wait_settle(ctx, &gw);
    {
        float* outs[4];
        for (int i = 0; i < n_tensors; i++) outs[i] = tensors[i].out;
        if (ibcu_push_match(ctx, outs, n_tensors)) {
            size_t bytes = 0;
            for (int i = 0; i < n_tensors; i++) bytes += (size_t)tensors[i].M * B * sizeof(float);
            ibcu_push_fill(ctx, &p.gp, bytes);
            for (int i = 0; i < n_tensors; i++) p.t[i].win_off = (long)((const char*)tensors[i].out - ctx->win_base);
        }
    }
    int8_t* xtiles = (int8_t*)ctx->xpack;
    float* xscale = (float*)((char*)ctx->xpack + tiles);
    int* xsum = (int*)((char*)ctx->xpack + tiles + scales);
    p.xtiles = xtiles; p.xscale = xscale; p.xsum = xsum; p.err = ctx->kern_err;
    const XSource xsrc = { x, pro ? pro->x2 : nullptr, pro ? (const __half*)pro->norm_w : nullptr, pro ? pro->eps : 0.0f, op,
                           op == IBCU_PRO_KNOWN_MAX ? pro->amax : nullptr, op == IBCU_PRO_KNOWN_MAX ? pro->n_amax : 0 };
    const dim3 xg(parts, B);
    const int perm8 = bits == 4 ? 1 : 0, cols = prep.part_kb * 128, all = p.nkb * 128;
    const bool mg = gw.flags || gw.tag.n;
    if (prep.clustered) {
        rc = ibcu_launch(ctx, mg ? xprep_tc_cluster_kernel<true> : xprep_tc_cluster_kernel<false>, xg, dim3(XCL_COLS / 8), 0, parts, true, xsrc, N, cols, all, p.NC, perm8, xtiles, xscale, xsum, gw);
    } else {
        auto kern = cols > 2048 ? (mg ? xprep_tc_kernel<512, true> : xprep_tc_kernel<512, false>) : (mg ? xprep_tc_kernel<256, true> : xprep_tc_kernel<256, false>);
        rc = ibcu_launch(ctx, kern, xg, dim3(cols > 2048 ? 512 : 256), 0, 1, true, xsrc, N, cols, all, p.NC, perm8, xtiles, xscale, xsum, gw);
    }
    if (rc) return rc;
    const int grid = S * (nruns < slots ? nruns : slots);
    if (bits == 8) return T == 1 ? launch_tc<8, 1>(ctx, maps, p, teams, grid, smem) : launch_tc<8, 2>(ctx, maps, p, teams, grid, smem);
    return T == 1 ? launch_tc<4, 1>(ctx, maps, p, teams, grid, smem) : launch_tc<4, 2>(ctx, maps, p, teams, grid, smem);
}
