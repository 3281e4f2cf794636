// Product-quantised matvec on the fifth-generation tensor cores (tcgen05.mma kind::f16, accumulators in tensor memory): the
// codebook entries themselves are the A operand, looked up 16 bytes at a time, and the activations are the columns of B.
//
// A lookup table per activation (pq.cu) costs one shared-memory word per code and activation, plus the table. An entry costs
// the four words of its eight weights once, whatever the number of activations, and the tensor cores do the rest.
//
// pq_xprep_kernel: max |x|, the 1 % rule, and every activation as three FP16 pieces of x 2^s (11 + 11 + 11 bits: an FP32
// significand fits with room; piece p is scaled by 2^(11 p)), laid out as the operand image: per 64 columns NC rows of 128 bytes,
// swizzled; rows 0 - 15 first pieces, then the other two of every activation. Entries are FP16 already, so every product is exact.
// pq_tc_kernel: the list of (tile of 128 rows) x (slab of 32 subspaces) is cut into equal contiguous pieces, one per block, and
// worked off in units of up to 256 columns:
//   warps 0-15   two teams of workers that take units in turn. Thread = row: code byte from the staged slab, entry from the
//                block's copy of the codebooks (held eight times, copy = lane mod 8, so that the eight lanes that shared memory
//                serves at once never meet in a bank), its weights into tensor memory
//   warps 16-23  two teams that take the sums out. Tensor cores cut off low bits when they add: first pieces are summed over
//                64 columns at a time (four MMAs), joined in FP32 outside, and units are added with compensation. Parts of a row
//                meet in the fixed-point accumulators of pq.cu. (Over 256 columns at a time the error was 3.4e-7 of the result's
//                root mean square, over 128 1.9e-7, now 1.25e-7; the tables' 1.0e-7.)
//   warps 24-26  codes (cp.async), operand image (bulk copies), MMA issue; a 28th warp fills their warpgroup
// What bounds it: the latency of every role's chain of waits, not a pipe, and what lies around the units: launches, the preparation, staging the codebooks, and the
// meeting of the parts. 4096 rows of entries of eight, 4096, 8192 and 14336 columns (4, 7 and 13 units a block at most): eight activations 12.8, 14.8 and 18.1 us, sixteen 16.8, 19.4
// and 23.7, so a unit takes about 0.58 us (1150 cycles, of which the entries keep the shared-memory pipe busy for 740 and the MMAs the tensor cores for 500) and all
// around the units 10.5. 4096 x 14336, entries of eight, 24 tensors in turn: eight activations 28.1 -> 18 us, sixteen 46 -> 24; 4096 x 8192 with entries
// of four at eight 49 -> 17, of sixteen 37 -> 15, with a second level 45 -> 19.
#include "tc_common.cuh"
#include "common.cuh"
#include "pq_tc.cuh"

namespace {

constexpr int PT_TEAM = 8, PT_WORKERS = 2 * PT_TEAM, PT_SUMMERS = 8, PT_SUM_WARP = 16, PT_CODE_WARP = 24, PT_X_WARP = 25, PT_MMA_WARP = 26, PT_THREADS = 28 * 32;       // the last warp only completes a warpgroup
// Registers a thread by role (launched with PT_REGS each). With the same for all, every instance spilled 36 to 364 bytes of stores in its loops, and with
// an SM's shared memory full there is little L1 to spill to. The helpers give up what the sums or, for entries of eight and up to eight
// activations, the workers are short of (4 to 72 bytes are left, the most in entries of four): 4096 x 14336 at 3, 8 and 16 activations 18.4 -> 16.3, 20.4 -> 18.0, 26.7 -> 24.0 us, 4096 x 8192
// with entries of sixteen at 1, 8 and 16 16.9 -> 12.3, 22.0 -> 15.1, 23.5 -> 19.0, with a second level 23.7 -> 19.1. Entries of four keep the even split (17.3;
// 18.6 with 80 for workers and sums and 24 for the helpers).
constexpr int PT_REGS = 72;
template <int HALF, int NG> struct PtRegs {
    static constexpr bool NARROW = HALF == 8 && NG == 1;
    static constexpr int WORKER = HALF != 4 && NARROW ? 80 : 72, SUMMER = HALF == 4 ? 72 : (NARROW ? 64 : 88), HELPER = HALF == 4 ? 72 : (NARROW ? 56 : 40);
    static_assert(PT_WORKERS * WORKER + PT_SUMMERS * SUMMER + 4 * HELPER == 28 * PT_REGS, "what the block is launched with");
};
template <int N> __device__ __forceinline__ void pt_set_regs() {
    if constexpr (N > PT_REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(N));
    if constexpr (N < PT_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(N));
}
// The codebooks' copies are written and tensor memory is allocated: every warp but that of the codes, which reads neither, comes here once.
__device__ __forceinline__ void pt_staged() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("bar.sync 1, %0;" :: "n"(PT_THREADS - 32) : "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
constexpr int PT_GROUP = 528;                                // bytes of a staged group of 16 rows x 32 codes: 16 more than it has, so that the two groups of a warp sit in different banks
constexpr int PT_SLAB = 8 * PT_GROUP;
constexpr int PT_MAX_X = 6, PT_MAX_C = 6, PT_MAXSEG = 8;
constexpr int PT_MAXB = 16;                                  // activations of a launch: 16 MMA columns for their first pieces, two columns each for the others
constexpr int PT_CHAIN = 64;                                 // columns whose products the tensor cores add up (first pieces) before FP32 additions outside take over

struct PtParams {
    int M, M_pad, N, K, K2, rows2, B, NC, nslab1, nslab, tiles;
    int sx, sc, tab_off, tab2_off, code_off, sh_off, tmem_cols;
    const __half* cb_l; const __half* cb_r; const __half* cb2_l; const __half* cb2_r;
    const uint8_t* idx_t;
    const float* cbmax;
    const __half* row_scale;
    const unsigned char* ximg;                 // [column blocks][2][NC][128]
    const unsigned* amax_bits;                 // [B]
    float* out; int out_stride;
    unsigned long long* acc;                   // [B][M_pad] fixed-point sums, zero between calls
    unsigned* arrive;                          // [tiles][4], zero between calls: one counter per 32 rows
    int* err;
};

struct PtShared {
    unsigned long long full_x[PT_MAX_X], empty_x[PT_MAX_X], full_c[PT_MAX_C], empty_c[PT_MAX_C], full_t[2], full_d[2], drained, met;
    uint32_t tmem_base;
    int abort_flag;
    double to_fix[PT_MAXB], to_out[PT_MAXB];        // a sum of scaled pieces -> fixed point; fixed point -> result (NaN: an activation held NaN or Inf)
    int seg_tile[PT_SUMMERS][PT_MAXSEG], seg_n[PT_SUMMERS][PT_MAXSEG];
};

// exponent of the power of two that takes max|x| to [2^14, 2^15), as the pieces are scaled by it
__device__ __forceinline__ int pt_shift(unsigned amax_bits) { return 14 - max((int)(amax_bits >> 23) - 127, -100); }
// exponent ex with N max|entry| max|x| < 2^ex: the quantum of the fixed-point sums is 2^(ex - 62) (as in pq.cu)
__device__ __forceinline__ int pt_bound(int N, float cbmax, unsigned amax_bits) {
    const float bound = (float)N * cbmax * __uint_as_float(amax_bits);
    return max(-60, min(120, (int)((__float_as_uint(bound) >> 23) & 0xFF) - 126));
}
__device__ __forceinline__ double pt_pow2(int e) { return __longlong_as_double((long long)(1023 + e) << 52); }

// grid (parts, B), 512 threads: a block takes max |x| of its activation and makes the pieces of its part of the columns
__global__ void __launch_bounds__(512) pq_xprep_kernel(const float* __restrict__ x, int N, const int* __restrict__ inner, int n_inner, int cols, int part_cols,
                                                       int G, int no_skip, int NC, unsigned char* __restrict__ ximg, unsigned* __restrict__ amax_out) {
    __shared__ unsigned red[16];
    pdl_launch_dependents();
    pdl_wait();
    const int b = blockIdx.y, tid = threadIdx.x;
    const float* xb = x + (size_t)b * N;
    const bool vec = !inner && (N & 3) == 0 && ((uintptr_t)x & 15) == 0;
    unsigned m = pq_absmax_bits<512>(xb, inner, n_inner, vec, tid);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((tid & 31) == 0) red[tid >> 5] = m;
    __syncthreads();
    m = __reduce_max_sync(0xffffffffu, red[tid & 15]);
    if (blockIdx.x == 0 && tid == 0) amax_out[b] = m;
    const float amax = __uint_as_float(m);
    const bool bad = m > 0x7f7fffffu;                         // the result is NaN then, whatever the pieces
    const float sc = __uint_as_float((unsigned)(127 + pt_shift(m)) << 23);
    const int c_lo = blockIdx.x * part_cols, c_hi = min(cols, c_lo + part_cols);
    for (int c0 = c_lo + (tid & ~31) * 8; c0 < c_hi; c0 += 512 * 8) {          // eight columns a thread; a warp stays together for the chunk maxima
        const int c = c0 + (tid & 31) * 8;
        float v[8];
        if (vec && c + 8 <= n_inner) {
            const float4 a0 = *reinterpret_cast<const float4*>(xb + c), a1 = *reinterpret_cast<const float4*>(xb + c + 4);
            v[0] = a0.x; v[1] = a0.y; v[2] = a0.z; v[3] = a0.w; v[4] = a1.x; v[5] = a1.y; v[6] = a1.z; v[7] = a1.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = c + i < n_inner ? xb[inner ? inner[c + i] : c + i] : 0.0f;
        }
        // the reference drops a chunk whose largest |x| is under 1 % of the largest overall
        float cm = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; i++) cm = fmaxf(cm, fabsf(v[i]));
        for (int o = 1; o < (G >> 3); o <<= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, o));
        const bool dead = bad || (amax > 0.0f && !no_skip && !(cm >= amax * 0.01f));
        if (c >= c_hi) continue;
        __half h[3][8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            float r = dead ? 0.0f : v[i] * sc;
#pragma unroll
            for (int p = 0; p < 3; p++) {
                h[p][i] = __float2half_rn(r);
                r = (r - __half2float(h[p][i])) * 2048.0f;   // exact
            }
        }
        unsigned char* half = ximg + (size_t)(c >> 6) * NC * 128;
#pragma unroll
        for (int p = 0; p < 3; p++) {
            const int row = p ? 15 + 2 * b + p : b;
            *reinterpret_cast<uint4*>(half + row * 128 + ((((c & 63) >> 3) ^ (row & 7)) << 4)) = *reinterpret_cast<const uint4*>(h[p]);
        }
    }
}

__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 :: "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

// HALF: values of an entry (4, 8, 16); NG: activations, in eights
template <int HALF, int NG>
__global__ void __launch_bounds__(PT_THREADS, 1) pq_tc_kernel(const __grid_constant__ PtParams p) {
    extern __shared__ __align__(1024) unsigned char pt_smem[];
    constexpr int CB = HALF == 4 ? 128 : 256;                 // columns of a unit of work: a slab, or half of one with 16-wide entries
    constexpr int NB = 32 * HALF / CB, ND = CB / PT_CHAIN;    // units of a slab; sums of first pieces in a unit
    constexpr int NC = 16 + 16 * NG, DC = 16 * ND + 16 * NG;  // rows of the operand image (MMA columns); tensor-memory columns of a unit's sums
    constexpr int SPW = CB / 2 / HALF;                        // subspaces of a unit that a worker warp looks up
    constexpr int PLANES = HALF == 16 ? 2 : 1;                // 16-byte planes of an entry
    constexpr int ROW = 256 * PLANES;                         // bytes of an entry's row of the table: [side][plane][copies, 128 bytes]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    PtShared* sh = reinterpret_cast<PtShared*>(pt_smem + p.sh_off);
    volatile int* abort_flag = &sh->abort_flag;
    const int G16 = p.M_pad >> 4;
    const int total = p.tiles * p.nslab;
    const int lo = (int)((long)total * blockIdx.x / gridDim.x), hi = (int)((long)total * (blockIdx.x + 1) / gridDim.x);
    constexpr uint32_t x_stage = NC * 2u * CB;
    const int nunit = (hi - lo) * NB;                         // units of this piece

    if (tid == 0) {
        for (int s = 0; s < PT_MAX_X; s++) { mbar_init(smem_u32(&sh->full_x[s]), 1); mbar_init(smem_u32(&sh->empty_x[s]), 1); }
        for (int s = 0; s < PT_MAX_C; s++) { mbar_init(smem_u32(&sh->full_c[s]), 32); mbar_init(smem_u32(&sh->empty_c[s]), NB * PT_TEAM); }
        for (int s = 0; s < 2; s++) { mbar_init(smem_u32(&sh->full_t[s]), PT_TEAM + PT_SUMMERS / 2); mbar_init(smem_u32(&sh->full_d[s]), 1); }
        mbar_init(smem_u32(&sh->drained), 1); mbar_init(smem_u32(&sh->met), PT_SUMMERS);
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp >= PT_CODE_WARP) {
        pt_set_regs<PtRegs<HALF, NG>::HELPER>();
        if (warp == PT_CODE_WARP) {
            // the codes do not depend on the kernel ahead: the ring fills at once
            int s = 0; uint32_t ph = 1;
            for (int item = lo; item < hi; item++) {
                if (item == lo + p.sc) pdl_wait();                // nobody polls a barrier for long while the kernel ahead runs
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->empty_c[s]), ph, abort_flag, 1))) break;
                const int tile = item / p.nslab, slab = item - tile * p.nslab;
                const uint32_t dst = smem_u32(pt_smem + p.code_off + s * PT_SLAB) + lane * 16;
                const unsigned char* src = p.idx_t + ((size_t)slab * G16 + (size_t)tile * 8) * 512 + lane * 16;
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const bool in = tile * 8 + u < G16;           // rows past the last group: zeros
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst + u * PT_GROUP), "l"(in ? src + u * 512 : p.idx_t), "r"(in ? 16 : 0) : "memory");
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" :: "r"(smem_u32(&sh->full_c[s])) : "memory");
                if (++s == p.sc) { s = 0; ph ^= 1; }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
        } else {
            if (warp == PT_MMA_WARP) {
                asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&sh->tmem_base)), "r"((uint32_t)p.tmem_cols) : "memory");
                asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
                pdl_launch_dependents();                          // not before: the blocks behind allocate too, and every block of this launch must hold its own first
            }
            pt_staged();
            const uint32_t tmem_base = sh->tmem_base, tmem_a = tmem_base + 2 * DC;
            if (warp == PT_X_WARP) {
                pdl_wait();
                if (elect_one()) {
                    int s = 0; uint32_t ph = 1;
                    bool ok = true;
                    for (int item = lo; item < hi && ok; item++) {
                        int slab = item % p.nslab;
                        if (slab >= p.nslab1) slab -= p.nslab1;       // the second level runs over the same activations
                        for (int hb = 0; hb < NB; hb++) {
                            ok = mbar_wait(smem_u32(&sh->empty_x[s]), ph, abort_flag, 2);
                            if (!ok) break;
                            mbar_expect_tx(smem_u32(&sh->full_x[s]), x_stage);
                            bulk_load(smem_u32(pt_smem + (size_t)s * x_stage), p.ximg + (size_t)(slab * NB + hb) * x_stage, x_stage, smem_u32(&sh->full_x[s]));
                            if (++s == p.sx) { s = 0; ph ^= 1; }
                        }
                    }
                }
                __syncwarp();
            } else if (warp == PT_MMA_WARP) {
                pdl_wait();
                if (elect_one()) {
                    constexpr uint32_t idesc = (1u << 4) | (8u << 24);    // FP32 accumulators, FP16 operands, 128 rows
                    constexpr uint32_t idesc_a = idesc | (2u << 17), idesc_b = idesc | ((uint32_t)(2 * NG) << 17);     // 16 columns; 16 NG columns
                    int s = 0; uint32_t ph = 0;
                    bool ok = true;
                    for (int n = 0; n < nunit; n++) {
                        ok = mbar_wait(smem_u32(&sh->full_x[s]), ph, abort_flag, 3) && mbar_wait(smem_u32(&sh->full_t[n & 1]), (uint32_t)(n >> 1) & 1u, abort_flag, 4);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint64_t bd = smem_desc_sw128(smem_u32(pt_smem) + (uint32_t)s * x_stage);
                        const uint32_t a = tmem_a + (uint32_t)(n & 1) * (CB / 2), d = tmem_base + (uint32_t)((n & 1) * DC);
#pragma unroll
                        for (int m = 0; m < CB / 16; m++) {           // 16 columns each; the image has NC * 128 bytes per 64 columns
                            const uint64_t b = bd + (uint64_t)((m >> 2) * (NC * 8) + (m & 3) * 2);
                            mma_f16_ts(d + (m / (PT_CHAIN / 16)) * 16, a + m * 8, b, idesc_a, m % (PT_CHAIN / 16) ? 1u : 0u);
                            mma_f16_ts(d + ND * 16, a + m * 8, b + 128, idesc_b, m ? 1u : 0u);
                        }
                        mma_commit(smem_u32(&sh->full_d[n & 1]));
                        mma_commit(smem_u32(&sh->empty_x[s]));
                        if (++s == p.sx) { s = 0; ph ^= 1; }
                    }
                    mma_commit(smem_u32(&sh->drained));
                    mbar_wait(smem_u32(&sh->drained), 0u, abort_flag, 5);
                }
                __syncwarp();
            }
        }
    } else {
        // the codebooks into the copies
        const int t0 = tid;
        constexpr int NT = PT_CODE_WARP * 32;
        auto stage = [&](const __half* l, const __half* r, int k_have, int rows, int off) {
            for (int e = t0; e < rows * 2 * PLANES; e += NT) {
                const int k = e / (2 * PLANES), side = (e / PLANES) & 1, plane = e % PLANES;
                const __half* src = (side ? r : l) + (size_t)k * HALF + plane * 8;
                uint4 v = make_uint4(0, 0, 0, 0);
                if (k < k_have) {
                    if constexpr (HALF == 4) { const uint2 w = *reinterpret_cast<const uint2*>(src); v = make_uint4(w.x, w.y, w.x, w.y); }
                    else v = *reinterpret_cast<const uint4*>(src);
                }
                uint4* dst = reinterpret_cast<uint4*>(pt_smem + off + (size_t)k * ROW + side * 128 * PLANES + plane * 128);
#pragma unroll
                for (int c = 0; c < 8; c++) dst[(c + t0) & 7] = v;              // lanes start at different copies: 128 bytes apart they would share banks
            }
        };
        stage(p.cb_l, p.cb_r, p.K, 256, p.tab_off);
        if (p.rows2) stage(p.cb2_l, p.cb2_r, p.K2, p.rows2, p.tab2_off);
        pt_staged();
        const uint32_t tmem_base = sh->tmem_base, tmem_a = tmem_base + 2 * DC;                   // two units of CB / 2 columns
        if (warp < PT_WORKERS) {
            pt_set_regs<PtRegs<HALF, NG>::WORKER>();
            // ── entries into tensor memory: the two teams take units in turn, each into its own half ──
            const int q = warp & 3, h = (warp >> 2) & 1, team = warp >> 3, rl = q * 32 + lane;
            const uint32_t at = tmem_a + ((uint32_t)(q * 32) << 16) + (uint32_t)(team * (CB / 2) + h * (CB / 4));
            const uint32_t lane_off = HALF == 4 ? (lane & 15) * 8 : (lane & 7) * 16;
            const uint32_t tab1 = smem_u32(pt_smem + p.tab_off) + lane_off, tab2 = smem_u32(pt_smem + p.tab2_off) + lane_off;
            // row i of a group keeps the code of subspace l at byte i ^ (l >> 1); the warp's subspaces: l0 .. l0 + SPW - 1 of the slab
            const int l0 = (NB == 2 ? team * 2 * SPW : 0) + h * SPW;
            const uint32_t crow = smem_u32(pt_smem + p.code_off) + (rl >> 4) * PT_GROUP + l0 * 16, ib = (uint32_t)((rl & 15) ^ (l0 >> 1));
            uint32_t code[SPW];
            int s = NB == 1 ? team : 0;
            uint32_t ph = 0;
            auto load_codes = [&]() {
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->full_c[s]), ph, abort_flag, 7))) return false;
#pragma unroll
                for (int j = 0; j < SPW; j++) asm volatile("ld.shared.u8 %0, [%1];" : "=r"(code[j]) : "r"(crow + s * PT_SLAB + j * 16 + (ib ^ (j >> 1))) : "memory");
                return true;
            };
            int slab = (lo + (NB == 1 ? team : 0)) % p.nslab;
            uint32_t dph = 1;                                     // the first wait passes: nothing has used the team's half yet
            bool alive = team < nunit && load_codes();
            for (int n = team; n < nunit && alive; n += 2) {
                const uint32_t tab = slab >= p.nslab1 ? tab2 : tab1;
                // sixteen words at a time, the next ones on their way while these are stored: every warp's whole share at once kept the
                // shared-memory pipe's queue so long that the other warps' barrier tests took 500 cycles
                constexpr int CH = CB / 64, PER = SPW / CH;       // chunks; lookups of a chunk
                uint32_t o[2][16];
                auto lookup = [&](int c) {
#pragma unroll
                    for (int i = 0; i < PER; i++) {
                        const int j = c * PER + i;
                        uint32_t* r = o[c & 1] + i * (16 / PER);
                        const uint32_t e = tab + code[j] * ROW + (j & 1) * 128 * PLANES;
                        if constexpr (HALF == 4) asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(e) : "memory");
                        else {
#pragma unroll
                            for (int pl = 0; pl < PLANES; pl++)
                                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r[4 * pl]), "=r"(r[4 * pl + 1]), "=r"(r[4 * pl + 2]), "=r"(r[4 * pl + 3]) : "r"(e + pl * 128) : "memory");
                        }
                    }
                };
                lookup(0);
                if (n >= 2 && n < 4) pdl_wait();                  // nobody polls a barrier for long while the kernel ahead runs
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->full_d[team]), dph, abort_flag, 6))) break;
                dph ^= 1;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int c = 0; c < CH; c++) {
                    if (c + 1 < CH) lookup(c + 1);
                    tmem_st16(at + 16 * c, o[c & 1]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sh->empty_c[s]));              // the codes have become addresses
                if (NB == 1) {
                    s += 2; slab += 2;
                    while (slab >= p.nslab) slab -= p.nslab;
                } else { s++; if (++slab == p.nslab) slab = 0; }
                if (s >= p.sc) { s -= p.sc; ph ^= 1; }
                if (n + 2 < nunit) { alive = load_codes(); if (!alive) break; }    // the next unit's codes travel while this one's entries are stored
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sh->full_t[team]));
            }
        } else if (warp < PT_SUM_WARP + PT_SUMMERS) {
            pt_set_regs<PtRegs<HALF, NG>::SUMMER>();
            // ── sums out of the accumulators ──
            const int q = warp & 3, rl = q * 32 + lane, st = tid - PT_SUM_WARP * 32, w = warp - PT_SUM_WARP, team = w >> 2;
            const uint32_t dq = tmem_base + ((uint32_t)(q * 32) << 16);
            const float cbmax = *p.cbmax;
            float acc[NG * 8], low[NG * 8];         // a sum and what its roundings lost
#pragma unroll
            for (int i = 0; i < NG * 8; i++) acc[i] = low[i] = 0.0f;
            bool alive = true;
            int nseg = 0, seg_n = 0;
            uint32_t met_ph = 0;
            auto meet = [&]() {                                   // these warps' own barrier, bounded like every other wait
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sh->met));
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->met), met_ph, abort_flag, 8))) alive = false;
                met_ph ^= 1;
                return alive;
            };
            auto flush = [&](int tile) {                          // the sums of a tile into the fixed-point accumulators
                const int r = tile * 128 + rl;
#pragma unroll
                for (int b = 0; b < NG * 8; b++) {
                    if (b < p.B && r < p.M) atomicAdd(p.acc + (size_t)b * p.M_pad + r, (unsigned long long)__double2ll_rn(((double)acc[b] + (double)low[b]) * sh->to_fix[b]));
                    acc[b] = low[b] = 0.0f;
                }
            };
            // this warp's arrivals for the tiles met since the last time; 32 rows to which all parts have come become results
            auto settle = [&]() {
                __threadfence();
                __syncwarp();
                bool last = false;
                if (lane < nseg) {
                    unsigned* cnt = p.arrive + sh->seg_tile[w][lane] * 4 + q;
                    const unsigned old = atomicAdd(cnt, (unsigned)sh->seg_n[w][lane]);
                    last = old + (unsigned)sh->seg_n[w][lane] == (unsigned)(p.nslab * NB);
                    if (last) *cnt = 0;
                }
                unsigned todo = __ballot_sync(0xffffffffu, last);
                if (todo) __threadfence();                        // every part has arrived, each behind its warp's fence: loads past L1 read the sums
                for (; todo; todo &= todo - 1) {
                    const int r = sh->seg_tile[w][__ffs(todo) - 1] * 128 + rl;
                    if (r >= p.M) continue;
                    const float sc = __half2float(p.row_scale[r]);
                    long long sum[NG * 8];
#pragma unroll
                    for (int b = 0; b < NG * 8; b++) sum[b] = b < p.B ? (long long)__ldcg(p.acc + (size_t)b * p.M_pad + r) : 0;
#pragma unroll
                    for (int b = 0; b < NG * 8; b++) {
                        if (b >= p.B) break;
                        p.acc[(size_t)b * p.M_pad + r] = 0ull;
                        p.out[(size_t)b * p.out_stride + r] = (float)((double)sum[b] * sh->to_out[b]) * sc;
                    }
                }
                __syncwarp();
                nseg = 0;
            };
            auto close_tile = [&](int tile) {
                if (!seg_n) return;                               // all of it was the other team's
                flush(tile);
                if (lane == 0) { sh->seg_tile[w][nseg] = tile; sh->seg_n[w][nseg] = seg_n; }
                seg_n = 0;
                if (++nseg == PT_MAXSEG) settle();
            };
            if (lane == 0)
                mbar_arrive(smem_u32(&sh->full_t[team]));         // the accumulators start free
            pdl_wait();
            if (st < p.B) {
                const unsigned ab = __ldcg(p.amax_bits + st);
                sh->to_fix[st] = pt_pow2(62 - pt_bound(p.N, cbmax, ab) - pt_shift(ab));
                sh->to_out[st] = ab > 0x7f7fffffu ? __longlong_as_double(0x7ff8000000000000ll) : pt_pow2(pt_bound(p.N, cbmax, ab) - 62);
            }
            meet();
            int cur = lo / p.nslab, left = (cur + 1) * p.nslab - lo;           // left: slabs of the tile from this piece's first on
            uint32_t ph = 0;
            for (int n = team; n < nunit && alive; n += 2, ph ^= 1) {
                if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&sh->full_d[team]), ph, abort_flag, 9))) { alive = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                while (n / NB >= left) { close_tile(cur); cur++; left += p.nslab; }
                const uint32_t d = dq + (uint32_t)(team * DC);
                float f[16];
                {
                    uint32_t u[16], v[16];
                    tmem_ld16(d, u); tmem_ld16(d + 16, v);
#pragma unroll
                    for (int b = 0; b < NG * 8; b++) f[b] = __uint_as_float(u[b]) + __uint_as_float(v[b]);
                    if constexpr (ND == 4) {
                        tmem_ld16(d + 32, u); tmem_ld16(d + 48, v);
#pragma unroll
                        for (int b = 0; b < NG * 8; b++) f[b] += __uint_as_float(u[b]) + __uint_as_float(v[b]);
                    }
                }
#pragma unroll
                for (int g = 0; g < NG; g++) {
                    uint32_t u[16];
                    tmem_ld16(d + ND * 16 + 16 * g, u);
#pragma unroll
                    for (int i = 0; i < 8; i++) {                 // piece p counts 2^(-11 p)
                        const int b = 8 * g + i;
                        const float v = fmaf(__uint_as_float(u[2 * i + 1]), 0x1p-22f, fmaf(__uint_as_float(u[2 * i]), 0x1p-11f, f[b]));
                        const float a = acc[b], sum = __fadd_rn(a, v), fr = __fsub_rn(sum, a);
                        low[b] += __fadd_rn(__fsub_rn(a, __fsub_rn(sum, fr)), __fsub_rn(v, fr));
                        acc[b] = sum;
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&sh->full_t[team]));
                seg_n++;
            }
            if (alive) close_tile(cur);
            if (alive && nseg) settle();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == PT_MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(sh->tmem_base), "r"((uint32_t)p.tmem_cols) : "memory");
    }
    if (tid == 0 && sh->abort_flag) {
        *p.err = IBCU_PQ_TC_ERR + sh->abort_flag;
        for (int i = 0; i < 1000; i++) __nanosleep(1000);     // copies still on their way into this block's shared memory land before it goes
    }
}

template <int HALF, int NG>
int launch_pt(ibcu_ctx* ctx, const PtParams& p, int grid, size_t smem) {
    auto kern = pq_tc_kernel<HALF, NG>;
    static SmemOptIn opt;
    if (int rc = ibcu_allow_smem(ctx, opt, kern, smem)) return rc;
    return ibcu_launch(ctx, kern, dim3(grid), dim3(PT_THREADS), smem, 1, true, p);
}
// setmaxnreg.inc waits for registers out of those that the block was launched with. A build that gives a thread fewer than PT_REGS (a debug build, a register
// limit) would wait for good: its calls take the tables.
template <int HALF, int NG>
bool pt_regs_suffice() {
    static const bool ok = [] { cudaFuncAttributes a; return cudaFuncGetAttributes(&a, pq_tc_kernel<HALF, NG>) == cudaSuccess ? a.numRegs >= PT_REGS : (cudaGetLastError(), false); }();
    return ok;
}
template <int HALF>
bool pt_regs_suffice(int B) { return B <= 8 ? pt_regs_suffice<HALF, 1>() : pt_regs_suffice<HALF, 2>(); }
template <int HALF>
int launch_half(ibcu_ctx* ctx, const PtParams& p, int grid, size_t smem) {
    return p.B <= 8 ? launch_pt<HALF, 1>(ctx, p, grid, smem) : launch_pt<HALF, 2>(ctx, p, grid, smem);
}
int pt_rows(int B) { return 16 + 16 * ((B + 7) / 8); }       // rows of the operand image

}  // namespace

size_t ibcu_pq_tc_image_bytes(const ibcu_pq_t* t, int B) {
    const size_t slabs = (2 * (size_t)((t->N - t->n_outlier) / t->G) + 31) / 32;
    return slabs * 32 * (t->G / 2) * 2 * pt_rows(B > PT_MAXB ? (B + 1) / 2 : B);
}

// Returns IBCU_DECLINED without touching the context's error when the tensor is not one for this kernel.
int ibcu_pq_tc(ibcu_ctx* ctx, const ibcu_pq_t* t, const float* x, float* out, int out_stride, int B, bool l1_only, unsigned long long* acc, unsigned* arrive, int max_counters,
               unsigned* amax_bits, void* image) {
    const int half = t->G >> 1;
    const bool two = t->K_l2 > 0 && !l1_only;
    const uintptr_t align = half == 4 ? 7 : 15;
    if ((half != 4 && half != 8 && half != 16) || t->cb_chunk_stride || B > 32 || (((uintptr_t)t->codebook_l | (uintptr_t)t->codebook_r) & align)) return IBCU_DECLINED;
    if (two && (((uintptr_t)t->codebook2_l | (uintptr_t)t->codebook2_r) & align)) return IBCU_DECLINED;
    const int b_launch = B > PT_MAXB ? (B + 1) / 2 : B;
    if (!(half == 4 ? pt_regs_suffice<4>(b_launch) : half == 8 ? pt_regs_suffice<8>(b_launch) : pt_regs_suffice<16>(b_launch))) return IBCU_DECLINED;
    if (B > PT_MAXB) {
        const int b0 = (B + 1) / 2;
        const int rc = ibcu_pq_tc(ctx, t, x, out, out_stride, b0, l1_only, acc, arrive, max_counters, amax_bits, image);
        return rc ? rc : ibcu_pq_tc(ctx, t, x + (size_t)b0 * t->N, out + (size_t)b0 * out_stride, out_stride, B - b0, l1_only, acc, arrive, max_counters, amax_bits, image);
    }
    PtParams p;
    memset(&p, 0, sizeof p);
    const int n_inner = t->N - t->n_outlier, C = n_inner / t->G;
    p.M = t->M; p.M_pad = t->M_pad; p.N = t->N; p.K = t->K; p.K2 = t->K_l2; p.B = B;
    p.nslab1 = (2 * C + 31) / 32;
    p.nslab = two ? 2 * p.nslab1 : p.nslab1;
    p.tiles = (t->M + 127) / 128;
    if (4 * p.tiles > max_counters || (long)p.tiles * p.nslab > (1l << 28)) return IBCU_DECLINED;
    p.rows2 = two ? (t->K_l2 == 16 ? 16 : 256) : 0;          // one-byte codes may be any, 4-bit ones not above 15
    p.NC = pt_rows(B);
    // Tensor memory: two units of 128 columns of entries and two times up to 96 of sums. Shared memory: the codebook
    // copies, a ring of codes (an even number of slabs: the teams take them in turn), a ring of activations.
    p.tmem_cols = 512;
    const int row = half == 16 ? 512 : 256, nd = half == 4 ? 1 : 2;
    const size_t x_stage = (size_t)p.NC * 256 * nd, tab = (size_t)256 * row, tab2 = (size_t)p.rows2 * row, fixed = tab + tab2 + sizeof(PtShared) + 16, cap = 226 * 1024;
    auto fits = [&]() { return fixed + p.sc * PT_SLAB + 2 * x_stage <= cap; };
    p.sc = PT_MAX_C;
    if (!fits()) p.sc = 4;
    if (!fits()) return IBCU_DECLINED;
    p.sx = (int)((cap - fixed - p.sc * PT_SLAB) / x_stage);
    if (p.sx > PT_MAX_X) p.sx = PT_MAX_X;
    p.tab_off = (int)(p.sx * x_stage);
    p.tab2_off = (int)(p.tab_off + tab);
    p.code_off = (int)(p.tab2_off + tab2);
    p.sh_off = (p.code_off + p.sc * PT_SLAB + 15) & ~15;
    const size_t smem = p.sh_off + sizeof(PtShared);
    const int cols = p.nslab1 * 32 * half;
    p.cb_l = (const __half*)t->codebook_l; p.cb_r = (const __half*)t->codebook_r; p.cb2_l = (const __half*)t->codebook2_l; p.cb2_r = (const __half*)t->codebook2_r;
    p.idx_t = t->idx_t;
    const int slabs_all = t->K_l2 > 0 ? 2 * p.nslab1 : p.nslab1;
    p.cbmax = reinterpret_cast<const float*>(t->idx_t + (size_t)slabs_all * 32 * t->M_pad);
    p.row_scale = (const __half*)t->row_scale; p.ximg = (const unsigned char*)image; p.amax_bits = amax_bits;
    p.out = out; p.out_stride = out_stride; p.acc = acc; p.arrive = arrive; p.err = ctx->kern_err;
    // parts of at least 1024 columns: every part reads the whole activation for its maximum
    int parts = cols / 1024;
    parts = parts < 1 ? 1 : (parts > 8 ? 8 : parts);
    const int part_cols = ((cols + parts - 1) / parts + 255) & ~255;                 // whole warps of eight columns a lane
    parts = (cols + part_cols - 1) / part_cols;
    const int rc = ibcu_launch(ctx, pq_xprep_kernel, dim3(parts, B), dim3(512), 0, 1, true, x, t->N, (const int*)(t->n_outlier > 0 ? t->inner_cols : nullptr), n_inner,
                               cols, part_cols, t->G, l1_only ? 1 : 0, p.NC, (unsigned char*)image, amax_bits);
    if (rc) return rc;
    const int total = p.tiles * p.nslab, grid = total < ctx->sm_count ? total : ctx->sm_count;
    return half == 4 ? launch_half<4>(ctx, p, grid, smem) : half == 8 ? launch_half<8>(ctx, p, grid, smem) : launch_half<16>(ctx, p, grid, smem);
}
