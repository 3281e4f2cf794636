// Per-row-scaled INT4 / INT8 linear layers for 1..32 FP32 activations.
//
// Data in HBM: weights keep the reference layout bit for bit (INT8 row-major; INT4 two columns per
// byte, low nibble first, bias 8), scales are FP16 (or FP32) per output row.
//
// Arithmetic of the fast path: integer tensor cores, exactly. Every slice of an FP32 activation becomes
// a 32-bit fixed-point integer X = rint(x * 2^s) (s per slice, so that the slice maximum sits just
// under 2^30), split into four signed base-256 digits (int8 "limbs").
// linear_mma_kernel feeds the weights - INT8 bytes as they are, INT4 nibbles masked in place with
// one LOP3 per four weights - and the limbs to mma.sync.m16n8k32 (s8/u8 x s8 -> s32): every product
// and every sum is an exact integer. The four limb sums are recombined in 64-bit, converted to
// floating point once, scaled back by 2^-s and multiplied by the row scale. The result is the
// correctly rounded dot product of the weights with x rounded to 2^-32 of its slice maximum: closer
// to the true value than the reference's own FP32 running sum, and independent of summation order.
// Because a dot product is invariant under a permutation of k applied to both operands, each lane
// simply owns 16 contiguous bytes of a row; no transpose or ldmatrix is needed for the weights.
//
// Activation conversion (xconvert_*): short rows are converted by every block of linear_mma_kernel for
// itself, straight into shared memory, with all of the block's loads issued before the first is used;
// long rows once, by xprep_kernel (one block per activation and column slice), into a scratch buffer
// the blocks copy from. RMSNorm and silu(x)*x2 can be folded into the conversion; a caller that knows
// max|x| (IBCU_PRO_KNOWN_MAX) spares the blocks their reduction.
//
// Work split: linear_mma_kernel is persistent, one wave of blocks. A block is bound to one column slice,
// whose limbs it holds in shared memory, and to one tensor of the launch, of which it owns one contiguous
// run of rows; the runs are equal to within a row (blocks are allotted to the tensors in proportion to
// their rows), so every SM streams the same number of bytes. A run is walked in tiles of up to RT*16
// rows; rows a tile lacks are zero-filled without fetching anything. Weights reach shared memory through
// a cp.async ring whose stages are (tile rows) x 64*W bytes, written in row-linear order (every warp
// instruction covers contiguous bytes of one row, which is what HBM wants; lane-owns-a-row-fragment
// register loads measured 2-3 TB/s, this pattern 6+ TB/s). The W warps of a block take one 64-byte
// k-block of each stage each and meet in a shared-memory reduction per tile. When the columns are split
// over several blocks (only when a row's limbs do not fit shared memory), each writes its integer partial
// sums to scratch and linear_finalize_kernel recombines them (a fence + arrival-counter epilogue
// inside the main kernel cost ~3 us per tile and slice, a second small launch costs ~2 us once).
//
// Portable path (linear_generic_kernel): one warp per output row, plain FP32 FMAs; used for shapes
// the fast path does not take (row bytes not a multiple of 16, unaligned pointers) and by tests.
#include "common.cuh"
#include "xconvert.cuh"

int ibcu_linear_tc(ibcu_ctx* ctx, const ibcu_linear_t* tensors, int n_tensors, const float* x, int N, int B, int bits, const ibcu_prologue_t* pro, int op);      // linear_tc.cu
bool ibcu_push_match(ibcu_ctx* ctx, float* const* outs, int n);      // comm.cu
void ibcu_push_fill(ibcu_ctx* ctx, GatherPush* gp, size_t bytes);  // bytes this launch pushes to each peer

namespace {

struct LinearParams {
    LinTensor t[4];
    int n_tensors;
    int total_rows;                // rows over all tensors
    int rowbytes;                  // bytes per weight row
    int nkb;                       // 64-byte k-blocks per row
    int N, B, ncols;               // columns, activations, limb columns (4 per activation)
    int slice_kb;                  // k-blocks per column slice (a multiple of the stage width)
    int nks;                       // column slices
    int xs_ld;                     // bytes per limb row: slice columns + pad
    const int8_t* xpack;           // [nks][ncols][xs_ld] limbs in fragment order
    const float* xscale;           // [B][nks] 2^-s of each slice
    const int* xsum;               // [B][nks][4] sum of each limb over the slice (INT4 bias term)
    int* partial;                  // [slice][B*4][total_rows] when nks > 1
    XSource xsrc;                  // FP32 source of the activations when the block converts them itself
    int fused_x;                   // 1: convert in the block, 0: limbs were prepared by xprep_kernel
    GatherWait gw;                 // the activations may be rows that peers pushed: wait for them (flags == NULL: nothing to wait for)
    GatherPush gp;                 // world > 0: this rank's output rows also go into the peers' copies (row-sharded output of a gather)
};

// Row length of the reduction buffer in words. With more than one group of 8 columns the rows are padded by 4 words:
// rows then start 4 banks apart and the 128-bit reads of a (row, activation)'s four limbs never collide. One group keeps
// its 8 words (a two-way collision there costs less than the shared memory the padding would take from the ring).
__host__ __device__ constexpr int lin_rld(int ncg) { return ncg == 1 ? 8 : ncg * 8 + 4; }

// ── activation split (xconvert.cuh) ─────────────────────────────────────────────────────
// grid (nks, B): the conversion as a kernel of its own, used when doing it inside every block of the
// main kernel would cost more than a launch (several activations, long rows, the SiLU prologue).
template <int T>
__global__ void __launch_bounds__(T) xprep_kernel(const XSource src, int N, int slice_cols, int xs_ld, int perm8,
                                                     int nks, int xregs, int8_t* __restrict__ xpack, float* __restrict__ xscale, int* __restrict__ xsum,
                                                     const GatherWait gw) {
    __shared__ XScratch sc;
    pdl_launch_dependents();
    pdl_wait();
    gather_wait(gw);
    const int ks = blockIdx.x, b = blockIdx.y;
    int8_t* dst = xpack + ((size_t)ks * (gridDim.y * LIN_LIMBS) + (size_t)b * LIN_LIMBS) * xs_ld;
    xconvert_any(src, N, b, ks * slice_cols, slice_cols, XRows{dst, xs_ld}, perm8, sc, xscale + b * nks + ks, xsum + ((size_t)b * nks + ks) * LIN_LIMBS, xregs);
}

__device__ __forceinline__ void imma_s8(int* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void imma_u8(int* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t u4_get(const uint4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

// ── fast path ───────────────────────────────────────────────────────────────────────────
// BITS: 4 or 8. NCG: groups of 8 MMA columns (ceil(4B/8)). RT: 16-row MMA tiles per tile of rows.
// W: warps per block. STAGES: shared-memory ring depth.
// MMA operands (m16n8k32, lane = 4g + t): A regs a0/a2 = row g, a1/a3 = row g+8, four bytes of k each;
// B regs b0/b1 = column g. INT8: a 16-byte lane chunk is four words w0..w3 -> two MMAs (w0,w1), (w2,w3)
// against 16 consecutive limb bytes. INT4: a raw word holds eight nibbles; raw & 0x0F0F0F0F are
// columns c0,c2,c4,c6 and raw & 0xF0F0F0F0 are 16 x columns c1,c3,c5,c7, so low and high nibbles go to
// separate accumulators (the high one is divided by 16 at the end, exactly) and no shift is needed.
// The nibble bias of 8 is removed once per output as 8 * (sum of the limb over the slice).
// Dynamic shared memory: stage ring [STAGES][R][LIN_LD] | reduction buffer [W][R][NCG*8] ints (x2 for
// INT4) | limbs [ncols][xs_ld] | scale-back factors [32] | limb sums [32][4].
__host__ __device__ constexpr int lin_sk(int W) { return W * 64; }                // bytes per row per stage: one 64-byte k-block per warp
__host__ __device__ constexpr int lin_ld(int W) { return W * 64 + 64; }           // padded row stride: conflict-free fragment reads

__device__ __forceinline__ void cp_async16(uint32_t smem_dst, const void* gsrc, bool valid) {
    const int n = valid ? 16 : 0;                             // 0 source bytes -> 16 zero bytes
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(smem_dst), "l"(gsrc), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// XV: 4 XV columns of an activation per thread are held in registers while the block converts it. Up to 4096 columns the instance with 4
// is enough (76 registers; the one with 8 takes 120): hidden size 4096, one token, 8-bit projections of 12 layers 171.8 -> 161.1 us; 2048:
// 128.1 -> 115.6. Two blocks fill an SM's shared memory with either, so it is not room for a third; what else it is was not measured apart.
// MG: the launch waits for rows of peers or pushes its own to them. Without that code, which a single GPU never runs, projections of a
// 7B shape took 204 us instead of 214 (INT8, one activation, sixteen layers), a decode step 1779 instead of 1819.
template <int BITS, int NCG, int RT, int W, int STAGES, int XV, bool MG>
__global__ void __launch_bounds__(W * 32) linear_mma_kernel(const LinearParams p) {
    constexpr int R = RT * 16;                                // most rows per tile
    constexpr int RLD = lin_rld(NCG);                         // words per row of the reduction buffer
    constexpr int NACC = BITS == 4 ? 2 : 1;                   // INT4 keeps low- and high-nibble sums apart
    constexpr int XB = BITS == 8 ? 64 : 128;                  // limb bytes (= columns) per k-block
    constexpr int KBS = W;                                    // k-blocks per stage: one per warp
    constexpr int LIN_SK = lin_sk(W), LIN_LD = lin_ld(W);
    constexpr int CPR = LIN_SK / 16;                          // 16-byte chunks per row per stage; the block copies 8 rows per pass
    static_assert(W == 8, "8 warps");
    constexpr int STAGE_BYTES = R * LIN_LD;
    constexpr int NCP = RT * 2;                               // 16-byte chunks per thread per stage
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    pdl_launch_dependents();

    const int ks = blockIdx.x % p.nks;                        // this block's column slice, fixed
    const int cb = blockIdx.x / p.nks;                        // a block works on one tensor: a contiguous run of its rows, in tiles of up to R
    int ti = 0;
#pragma unroll
    for (int i = 1; i < 4; i++) if (i < p.n_tensors && cb >= p.t[i].blk_start) ti = i;
    const LinTensor& T = p.t[ti];
    const int row_begin = (cb - T.blk_start) * T.rows_per;
    const int row_end = min(T.M, row_begin + T.rows_per);
    const int kb_begin = ks * p.slice_kb;
    const int nk = min(p.nkb, kb_begin + p.slice_kb) - kb_begin;
    const int nst = (nk + KBS - 1) / KBS;

    unsigned char* ring = smem_raw;
    int* red = reinterpret_cast<int*>(smem_raw + STAGES * STAGE_BYTES);
    int8_t* xs = reinterpret_cast<int8_t*>(smem_raw + STAGES * STAGE_BYTES + NACC * W * R * RLD * 4);
    float* s_back = reinterpret_cast<float*>(xs + (((size_t)p.ncols * p.xs_ld + 15) & ~(size_t)15));
    int* s_xsum = reinterpret_cast<int*>(s_back + 32);

    // ── producer side: thread owns chunk column cc of rows pr + 8i of every stage ──
    const int cc = threadIdx.x % CPR, pr = threadIdx.x / CPR;
    const uint32_t ring_u32 = (uint32_t)__cvta_generic_to_shared(ring) + pr * LIN_LD + cc * 16;
    const uint8_t* src[NCP];
    // A tile is up to R consecutive rows; rows of the tile that do not exist are zero-filled.
    int pf_row = row_begin, pf_rows = 0, pf_it = 0, pf_slot = 0;
    unsigned pf_mask = 0;                                     // bit i: row pr + 8i exists in the tile
    auto pf_setup = [&]() {                                   // row pointers for the tile at pf_row
        pf_rows = min(R, row_end - pf_row);
        const int r0 = pr;
        pf_mask = 0;
#pragma unroll
        for (int i = 0; i < NCP; i++) {
            const bool has = r0 + 8 * i < pf_rows;
            pf_mask |= has ? 1u << i : 0u;
            src[i] = T.w + (size_t)(pf_row + (has ? r0 + 8 * i : 0)) * p.rowbytes + (size_t)kb_begin * 64 + cc * 16;
        }
    };
    auto pf_issue = [&]() {                                   // next stage of the prefetch stream, if any
        if (pf_row < row_end) {
            const bool valid = (kb_begin + pf_it * KBS) * 64 + cc * 16 < p.rowbytes && pf_it * KBS + (cc >> 2) < nk;
            const uint32_t d = ring_u32 + pf_slot * STAGE_BYTES;
#pragma unroll
            for (int i = 0; i < NCP; i++) {
                const bool v = valid && ((pf_mask >> i) & 1u);
                cp_async16(d + i * 8 * LIN_LD, v ? src[i] + pf_it * LIN_SK : src[i], v);
            }
            pf_slot = pf_slot + 1 == STAGES ? 0 : pf_slot + 1;
            if (++pf_it == nst) { pf_it = 0; pf_row += pf_rows; if (pf_row < row_end) pf_setup(); }
        }
        cp_async_commit();
    };
    if (pf_row < row_end) pf_setup();
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) pf_issue();          // weights first: they do not depend on x
    pdl_wait();
    const unsigned recv_tag = MG ? gather_wait(p.gw) : 0u;   // not 0: this launch received a tagged gather; its own pushes then carry the next tag

    // ── this slice's limbs, scale-back factors and limb sums ──
    if (p.fused_x) {
        __shared__ XScratch xsc;
        for (int b = 0; b < p.B; b++)
            xconvert_any<XV>(p.xsrc, p.N, b, kb_begin * XB, p.slice_kb * XB, XRows{xs + (size_t)b * LIN_LIMBS * p.xs_ld, p.xs_ld}, BITS == 4 ? 1 : 0,
                         xsc, s_back + b, s_xsum + b * LIN_LIMBS);
    } else {
        const uint4* gsrc = reinterpret_cast<const uint4*>(p.xpack + (size_t)ks * p.ncols * p.xs_ld);
        const uint32_t d0 = (uint32_t)__cvta_generic_to_shared(xs);
        const int nchunk = p.ncols * p.xs_ld / 16;
        for (int c = threadIdx.x; c < nchunk; c += W * 32) cp_async16(d0 + c * 16, gsrc + c, true);
        cp_async_commit();
        if (threadIdx.x < p.B) s_back[threadIdx.x] = p.xscale[threadIdx.x * p.nks + ks];
        if (threadIdx.x < p.B * LIN_LIMBS)
            s_xsum[threadIdx.x] = p.xsum[((size_t)(threadIdx.x / LIN_LIMBS) * p.nks + ks) * LIN_LIMBS + (threadIdx.x % LIN_LIMBS)];
    }
    cp_async_wait<0>();
    __syncthreads();

    const int8_t* xcol[NCG];
#pragma unroll
    for (int c = 0; c < NCG; c++) {
        int col = c * 8 + g;
        col = col < p.ncols ? col : 0;                        // spare MMA columns reread column 0
        xcol[c] = xs + (size_t)col * p.xs_ld + (XB / 4) * t;
    }

    int slot = 0;
    int tile_rows = 0;
    for (int row0 = row_begin; row0 < row_end; row0 += tile_rows) {
        tile_rows = min(R, row_end - row0);
        int acc[NACC][RT][NCG][4];
#pragma unroll
        for (int a = 0; a < NACC; a++)
#pragma unroll
            for (int i = 0; i < RT; i++)
#pragma unroll
                for (int c = 0; c < NCG; c++) { acc[a][i][c][0] = acc[a][i][c][1] = acc[a][i][c][2] = acc[a][i][c][3] = 0; }

        for (int it = 0; it < nst; it++) {
            cp_async_wait<STAGES - 2>();
            __syncthreads();                                  // this stage has landed for everyone; the previous one is free
            pf_issue();
            const int k = it * KBS + warp;                    // this warp's k-block within the slice
            if (k < nk) {
                const unsigned char* sw = ring + slot * STAGE_BYTES + warp * 64 + 16 * t;
                uint4 cur[RT * 2];
#pragma unroll
                for (int j = 0; j < RT * 2; j++)
                    cur[j] = *reinterpret_cast<const uint4*>(sw + ((j >> 1) * 16 + (j & 1) * 8 + g) * LIN_LD);
                if (BITS == 8) {
                    uint4 xf[NCG];
#pragma unroll
                    for (int c = 0; c < NCG; c++) xf[c] = *reinterpret_cast<const uint4*>(xcol[c] + (size_t)k * XB);
#pragma unroll
                    for (int i = 0; i < RT; i++)
#pragma unroll
                        for (int c = 0; c < NCG; c++) {
                            imma_s8(acc[0][i][c], cur[2 * i].x, cur[2 * i + 1].x, cur[2 * i].y, cur[2 * i + 1].y, xf[c].x, xf[c].y);
                            imma_s8(acc[0][i][c], cur[2 * i].z, cur[2 * i + 1].z, cur[2 * i].w, cur[2 * i + 1].w, xf[c].z, xf[c].w);
                        }
                } else {
#pragma unroll
                    for (int h = 0; h < 2; h++) {             // two raw words (16 columns... 8 each) per half
                        uint4 xf[NCG];
#pragma unroll
                        for (int c = 0; c < NCG; c++) xf[c] = *reinterpret_cast<const uint4*>(xcol[c] + (size_t)k * XB + 16 * h);
#pragma unroll
                        for (int i = 0; i < RT; i++) {
                            const uint32_t r0a = u4_get(cur[2 * i], 2 * h), r0b = u4_get(cur[2 * i], 2 * h + 1);
                            const uint32_t r1a = u4_get(cur[2 * i + 1], 2 * h), r1b = u4_get(cur[2 * i + 1], 2 * h + 1);
#pragma unroll
                            for (int c = 0; c < NCG; c++) {
                                // low nibbles of words a, b against columns c0,c2,c4,c6 of each word
                                imma_u8(acc[0][i][c], r0a & 0x0F0F0F0Fu, r1a & 0x0F0F0F0Fu, r0b & 0x0F0F0F0Fu, r1b & 0x0F0F0F0Fu, xf[c].x, xf[c].z);
                                // high nibbles (x16) against columns c1,c3,c5,c7
                                imma_u8(acc[1][i][c], r0a & 0xF0F0F0F0u, r1a & 0xF0F0F0F0u, r0b & 0xF0F0F0F0u, r1b & 0xF0F0F0F0u, xf[c].y, xf[c].w);
                            }
                        }
                    }
                }
            }
            slot = slot + 1 == STAGES ? 0 : slot + 1;
        }
        // ── tile done: every warp holds integer partial sums of all R rows over its k-blocks ──
#pragma unroll
        for (int a = 0; a < NACC; a++) {
            int* mine = red + ((size_t)a * W + warp) * R * RLD;
#pragma unroll
            for (int i = 0; i < RT; i++)
#pragma unroll
                for (int c = 0; c < NCG; c++) {
                    *reinterpret_cast<int2*>(mine + (i * 16 + g) * RLD + c * 8 + 2 * t) = make_int2(acc[a][i][c][0], acc[a][i][c][1]);
                    *reinterpret_cast<int2*>(mine + (i * 16 + g + 8) * RLD + c * 8 + 2 * t) = make_int2(acc[a][i][c][2], acc[a][i][c][3]);
                }
        }
        __syncthreads();
        const int B = p.B;
        const unsigned tag = MG && p.gp.world ? (recv_tag ? recv_tag + 1u : tag_current(p.gp)) : 0u;
        // one thread per (row, activation): limb sums over the warps, bias, recombination
        for (int e = threadIdx.x; e < R * B; e += W * 32) {
            const int r = e % R, b = e / R;
            if (r >= tile_rows) continue;
            const int row = row0 + r;
            int limb[LIN_LIMBS];
            {                                                 // the four limbs of (row, activation) sit side by side: one 128-bit read per warp
                int4 lo = make_int4(0, 0, 0, 0);
#pragma unroll
                for (int w = 0; w < W; w++) {
                    const int4 v = *reinterpret_cast<const int4*>(red + ((size_t)w * R + r) * RLD + b * LIN_LIMBS);
                    lo.x += v.x; lo.y += v.y; lo.z += v.z; lo.w += v.w;
                }
                if (BITS == 4) {
                    int4 hi = make_int4(0, 0, 0, 0);
#pragma unroll
                    for (int w = 0; w < W; w++) {
                        const int4 v = *reinterpret_cast<const int4*>(red + ((size_t)(W + w) * R + r) * RLD + b * LIN_LIMBS);
                        hi.x += v.x; hi.y += v.y; hi.z += v.z; hi.w += v.w;
                    }
                    lo.x += (hi.x >> 4) - 8 * s_xsum[b * LIN_LIMBS + 0];
                    lo.y += (hi.y >> 4) - 8 * s_xsum[b * LIN_LIMBS + 1];
                    lo.z += (hi.z >> 4) - 8 * s_xsum[b * LIN_LIMBS + 2];
                    lo.w += (hi.w >> 4) - 8 * s_xsum[b * LIN_LIMBS + 3];
                }
                limb[0] = lo.x; limb[1] = lo.y; limb[2] = lo.z; limb[3] = lo.w;
            }
            if (p.nks == 1) {
                {
                    const long long V = (((long long)limb[3] * 256 + limb[2]) * 256 + limb[1]) * 256 + limb[0];
                    const float y = (float)((double)V * (double)s_back[b]);
                    const float sc = T.scales_fp32 ? reinterpret_cast<const float*>(T.scales)[row]
                                                   : __half2float(reinterpret_cast<const __half*>(T.scales)[row]);
                    float* o = T.out + (size_t)b * T.out_stride + row;
                    const float v = T.epilogue == IBCU_EPI_ADD ? *o + y * sc : y * sc;
                    *o = v;
                    if (MG && p.gp.world) tag_push(p.gp, (size_t)T.win_off + ((size_t)b * T.out_stride + row) * sizeof(float), v, tag);
                }
            } else {
#pragma unroll
                for (int l = 0; l < LIN_LIMBS; l++)
                    p.partial[((size_t)ks * (B * LIN_LIMBS) + b * LIN_LIMBS + l) * p.total_rows + T.row_start + row] = limb[l];
            }
        }
    }
    cp_async_wait<0>();
}

// When the columns are split over several blocks: one thread per (row, activation) recombines the
// integer partial sums of all slices, each with its own 2^-s, in slice order.
__global__ void __launch_bounds__(256) linear_finalize_kernel(const LinearParams p) {
    pdl_launch_dependents();
    pdl_wait();
    const int B = p.B;
    const long total = (long)p.total_rows * B;
    const unsigned tag = p.gp.world ? tag_current(p.gp) : 0u;
    for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
        const int vrow = (int)(e % p.total_rows);
        const int b = (int)(e / p.total_rows);
        int ti = 0;
#pragma unroll
        for (int i = 1; i < 4; i++) if (i < p.n_tensors && vrow >= p.t[i].row_start) ti = i;
        const LinTensor& T = p.t[ti];
        const int row = vrow - T.row_start;
        double y = 0.0;
        for (int k = 0; k < p.nks; k++) {
            const int* src_p = p.partial + ((size_t)k * (B * LIN_LIMBS) + b * LIN_LIMBS) * p.total_rows + vrow;
            const size_t st = p.total_rows;
            const long long V = (((long long)src_p[3 * st] * 256 + src_p[2 * st]) * 256 + src_p[st]) * 256 + src_p[0];
            y += (double)V * (double)p.xscale[b * p.nks + k];
        }
        const float sc = T.scales_fp32 ? reinterpret_cast<const float*>(T.scales)[row]
                                       : __half2float(reinterpret_cast<const __half*>(T.scales)[row]);
        float* o = T.out + (size_t)b * T.out_stride + row;
        const float v = T.epilogue == IBCU_EPI_ADD ? *o + (float)y * sc : (float)y * sc;
        *o = v;
        if (p.gp.world) tag_push(p.gp, (size_t)T.win_off + ((size_t)b * T.out_stride + row) * sizeof(float), v, tag);
    }
}

// ── portable path ───────────────────────────────────────────────────────────────────────
// One warp per output row; lanes stride over the columns; FP32 FMAs; activations straight from x.
template <int BITS>
__global__ void __launch_bounds__(256) linear_generic_kernel(LinTensor T, const float* __restrict__ x, int N, int B) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= T.M) return;
    const size_t rowbytes = BITS == 8 ? (size_t)N : (size_t)(N / 2);
    const uint8_t* wr = T.w + (size_t)row * rowbytes;
    const float sc = T.scales_fp32 ? reinterpret_cast<const float*>(T.scales)[row]
                                   : __half2float(reinterpret_cast<const __half*>(T.scales)[row]);
    for (int b = 0; b < B; b++) {
        const float* xb = x + (size_t)b * N;
        float s = 0.0f;
        if (BITS == 8) {
            for (int j = lane; j < N; j += 32) s = fmaf((float)(int8_t)wr[j], xb[j], s);
        } else {
            for (int j = 2 * lane; j < N; j += 64) {
                uint8_t v = wr[j >> 1];
                s = fmaf((float)((int)(v & 15) - 8), xb[j], s);
                if (j + 1 < N) s = fmaf((float)((int)(v >> 4) - 8), xb[j + 1], s);
            }
        }
        s = warp_sum(s);
        if (lane == 0) {
            float y = s * sc;
            float* o = T.out + (size_t)b * T.out_stride + row;
            *o = T.epilogue == IBCU_EPI_ADD ? *o + y : y;
        }
    }
}

template <int BITS, int NCG, int RT, int W, int STAGES, int XV, bool MG>
int launch_mma_mg(ibcu_ctx* ctx, const LinearParams& p, int grid, size_t smem_tail) {
    auto kern = linear_mma_kernel<BITS, NCG, RT, W, STAGES, XV, MG>;
    const size_t smem = (size_t)STAGES * RT * 16 * lin_ld(W) + (size_t)(BITS == 4 ? 2 : 1) * W * RT * 16 * lin_rld(NCG) * 4 + smem_tail;   // ring + reduction buffer + limbs
    static SmemOptIn opt;
    if (int rc = ibcu_allow_smem(ctx, opt, kern, smem)) return rc;
    return ibcu_launch(ctx, kern, dim3(grid), dim3(W * 32), smem, 1, true, p);
}

template <int BITS, int NCG, int RT, int W, int STAGES, int XV>
int launch_mma_x(ibcu_ctx* ctx, const LinearParams& p, int grid, size_t smem_tail) {
    if (p.gp.world || p.gw.flags || p.gw.tag.n) return launch_mma_mg<BITS, NCG, RT, W, STAGES, XV, true>(ctx, p, grid, smem_tail);
    return launch_mma_mg<BITS, NCG, RT, W, STAGES, XV, false>(ctx, p, grid, smem_tail);
}

// a block that converts more than 4096 columns itself, and has to find their maximum first, holds up to 8192 (one activation: see lin_plan)
template <int BITS, int NCG, int RT, int W, int STAGES>
int launch_mma(ibcu_ctx* ctx, const LinearParams& p, int grid, size_t smem_tail) {
    if constexpr (NCG == 1) {
        const bool longer = p.fused_x && p.xsrc.op != IBCU_PRO_KNOWN_MAX && p.slice_kb * (BITS == 8 ? 64 : 128) > 4 * 4 * W * 32;
        if (longer) return launch_mma_x<BITS, NCG, RT, W, STAGES, 8>(ctx, p, grid, smem_tail);
    }
    return launch_mma_x<BITS, NCG, RT, W, STAGES, 4>(ctx, p, grid, smem_tail);
}

// Eight warps and 512-byte stages; the ring is as deep as two resident blocks per SM allow.
template <int BITS, int NCG>
int dispatch_shape(ibcu_ctx* ctx, const LinearParams& p, int grid, int rt, int stages, size_t smem_tail) {
    if constexpr (NCG <= 2) {                                  // more groups of columns take tiles of 16 rows
        if (rt == 2) return stages >= 6 ? launch_mma<BITS, NCG, 2, 8, 6>(ctx, p, grid, smem_tail) : launch_mma<BITS, NCG, 2, 8, 4>(ctx, p, grid, smem_tail);
    }
    if (stages >= 8) return launch_mma<BITS, NCG, 1, 8, 8>(ctx, p, grid, smem_tail);
    return launch_mma<BITS, NCG, 1, 8, 4>(ctx, p, grid, smem_tail);
}

// How linear_mma_kernel takes a call of up to 16 activations.
struct LinPlan {
    int ncols, ncg, nkb, rt, stages;           // limb columns and groups of eight of them, 64-byte k-blocks per row, 16-row MMA tiles per tile of rows, ring depth
    int slice_kb, nks, xs_ld;                  // k-blocks per column slice, slices, bytes per limb row
    size_t piece_smem;                         // bytes of a slice's limbs
    int fit, rows_per_block, nblk;             // blocks per SM, longest run of rows, blocks per slice
    int blk_start[4], rows_per[4];             // of every tensor
    bool fused;                                // every block converts the activations for itself
};

LinPlan lin_plan(const ibcu_ctx* ctx, const ibcu_linear_t* tensors, int n_tensors, long total_rows, int N, int B, int bits, int op) {
    LinPlan pl;
    const int rowbytes = bits == 8 ? N : N / 2;
    pl.ncols = B * LIN_LIMBS;
    const int groups = (pl.ncols + 7) / 8;
    pl.ncg = groups <= 1 ? 1 : (groups <= 2 ? 2 : (groups <= 4 ? 4 : 8));
    pl.nkb = (rowbytes + 63) / 64;
    const int xk = bits == 8 ? 64 : 128;
    const int xpad = bits == 8 ? 64 : 16;                     // keeps limb rows of neighbouring columns on different banks
    // Rows are dealt out evenly: every block of the persistent grid owns one contiguous run of rows and
    // walks it in tiles of up to R = 16 or 32 rows. 32-row tiles once a block's run is longer than 16.
    const int w = 8;                                          // warps per block; two blocks share an SM
    pl.rt = (pl.ncg >= 4 || total_rows <= 16L * 2 * ctx->sm_count) ? 1 : 2;
    const int R = 16 * pl.rt;
    // Shared memory per block: stage ring + reduction buffer + the slice's limbs. Columns are
    // split over several blocks only when the limbs of a whole row do not fit.
    const int kbs = w;
    const int LIN_LD = lin_ld(w);
    // ring depth: the deeper ring when two blocks per SM still fit with it, else the shallower one
    const size_t red_bytes = (size_t)(bits == 4 ? 2 : 1) * w * R * lin_rld(pl.ncg) * 4;
    const size_t whole_row_pieces = (size_t)pl.ncols * ((size_t)pl.nkb * xk + xpad);
    pl.stages = pl.rt == 2 ? 6 : 8;
    if (2 * ((size_t)pl.stages * R * LIN_LD + red_bytes + whole_row_pieces + 2048) > 227 * 1024) pl.stages = 4;
    const size_t fixed_smem = (size_t)pl.stages * R * LIN_LD + red_bytes + 1024;
    const size_t smem_cap = 200 * 1024;
    long piece_budget = (long)smem_cap - (long)fixed_smem;
    int max_slice_kb = (int)((piece_budget / pl.ncols - xpad) / xk) / kbs * kbs;
    if (max_slice_kb < kbs) max_slice_kb = kbs;
    pl.slice_kb = (pl.nkb + kbs - 1) / kbs * kbs;             // whole stages per slice
    if (pl.slice_kb > max_slice_kb) pl.slice_kb = max_slice_kb;
    pl.nks = (pl.nkb + pl.slice_kb - 1) / pl.slice_kb;
    pl.xs_ld = pl.slice_kb * xk + xpad;
    pl.piece_smem = (((size_t)pl.ncols * pl.xs_ld) + 15) & ~(size_t)15;
    // persistent grid: as many blocks as fit on the machine at once, a multiple of nks, at most one per item
    pl.fit = (int)((227 * 1024) / (fixed_smem + pl.piece_smem + 1024));
    if (pl.fit < 1) pl.fit = 1;
    if (pl.fit > 4) pl.fit = 4;
    const int slots = pl.fit * ctx->sm_count;
    int per_slice = slots / pl.nks;
    if (per_slice < 1) per_slice = 1;
    // every tensor gets blocks in proportion to its rows, and its rows are dealt out evenly among them;
    // the run length grows until all blocks are resident at once
    pl.rows_per_block = (int)((total_rows + per_slice - 1) / per_slice);
    if (pl.rows_per_block < 4) pl.rows_per_block = 4;
    for (;; pl.rows_per_block++) {
        pl.nblk = 0;
        for (int i = 0; i < n_tensors; i++) pl.nblk += (tensors[i].M + pl.rows_per_block - 1) / pl.rows_per_block;
        if (pl.nblk <= per_slice || pl.rows_per_block >= total_rows) break;
    }
    pl.nblk = 0;
    for (int i = 0; i < n_tensors; i++) {
        const int n = (tensors[i].M + pl.rows_per_block - 1) / pl.rows_per_block;
        pl.blk_start[i] = pl.nblk;
        pl.rows_per[i] = n ? (tensors[i].M + n - 1) / n : 0;
        pl.nblk += n;
    }
    // Cheap conversions are done by every block of the main kernel for itself (no extra launch, no
    // dependency chain); expensive ones (SiLU, several activations, long rows) once, by xprep_kernel.
    pl.fused = op != IBCU_PRO_SILU_MUL && (long)B * pl.slice_kb * xk <= 8192 && pl.nks == 1;
    if (op == IBCU_PRO_KNOWN_MAX && pl.nks == 1 && B <= 2) pl.fused = true;          // no reduction: cheap at any row length
    return pl;
}

// Which kernel takes a call of 2 to 16 activations: the time of either, in us, from what it does. The coefficients are least squares
// (relative error 6 %) over 2296 calls on a B200, direct and in graphs: 2, 3, 4, 5, 6, 8, 12 and 16 activations, 512 to 14336 columns, 512
// to 32000 rows in one to three tensors, 4 and 8 bits. The choice was 0.2 % behind the better kernel on the mean and more than 5 % behind
// it in one call of 60; choosing by the number of activations and the bytes of the weights was 2.2 % behind, up to 95 %.
// The fit is older than the tcgen05 kernel's full rings and its digits by clusters, which took 2 to 20 % off its times: now the choice is 1.1 % behind the better kernel on the mean
// of 2592 calls (0.4 % without a prologue, 1.7 % with RMSNorm), more than 5 % in one of 15, up to 60 % (INT4 856 x 1440 with RMSNorm at 4 activations 8.9 against 5.5),
// nearly always by staying with mma.sync.
// mma.sync kernel: per block the MMAs of its tiles, the weights, and a reduction per tile; the conversion in the block, or a launch ahead.
double lin_mma_us(const LinPlan& pl, int N, int B, int bits) {
    const int R = 16 * pl.rt, tiles = (pl.rows_per_block + R - 1) / R, stages = ((pl.slice_kb < pl.nkb ? pl.slice_kb : pl.nkb) + 7) / 8;
    const double i4 = bits == 4 ? 1.0 : 0.0;
    double us = 1.73 + (pl.fused ? 0.69 * B + 0.171e-3 * N * B : 2.03 + 0.345e-3 * N);
    us += pl.fit * (tiles * stages * pl.ncg * pl.rt * (0.045 + 0.037 * i4) + 0.168e-4 * pl.rows_per_block * stages * 512 + 0.043 * tiles * B * pl.rt * (1.0 + i4));
    return us + (pl.nks > 1 ? 1.1 : 0.0) + (pl.fit == 1 ? 0.6 : 0.0);
}
// tcgen05 kernel: a preparation launch, and per block of 128 columns the weights and the digits, which hardly grow with the activations.
double lin_tc_us(const TqCut& c, int N, int bits) {
    const int per_block = (c.nruns + c.slots - 1) / c.slots * ((c.nkb + c.S - 1) / c.S);
    return 6.3 + 0.16e-3 * N + per_block * ((bits == 4 ? 0.084 : 0.0) + 0.151e-4 * c.R * bits * 16 + 0.317e-4 * c.NC * 128);
}

}  // namespace

extern "C" void ibcu_linear_force_generic(ibcu_ctx* ctx, int on) { if (ctx) ctx->force_generic = on; }
extern "C" void ibcu_linear_use_tcgen05(ibcu_ctx* ctx, int on) { if (ctx) ctx->linear_tc = on; }

extern "C" int ibcu_linear(ibcu_ctx* ctx, const ibcu_linear_t* tensors, int n_tensors,
                           const float* x, int N, int B, int bits) {
    return ibcu_linear_ex(ctx, tensors, n_tensors, x, N, B, bits, nullptr);
}

extern "C" int ibcu_linear_ex(ibcu_ctx* ctx, const ibcu_linear_t* tensors, int n_tensors,
                              const float* x, int N, int B, int bits, const ibcu_prologue_t* pro) {
    IBCU_CHECK_CTX(ctx);
    const int op = pro ? pro->op : IBCU_PRO_NONE;
    IBCU_REQUIRE(ctx, op == IBCU_PRO_NONE || (op == IBCU_PRO_RMSNORM && pro->norm_w) || (op == IBCU_PRO_SILU_MUL && pro->x2) ||
                      (op == IBCU_PRO_KNOWN_MAX && pro->amax && pro->n_amax >= 1),
                 "ibcu_linear_ex: prologue %d lacks its operand", op);
    IBCU_REQUIRE(ctx, tensors && x, "ibcu_linear: null pointer");
    IBCU_REQUIRE(ctx, n_tensors >= 1 && n_tensors <= 4, "ibcu_linear: n_tensors=%d not in 1..4", n_tensors);
    IBCU_REQUIRE(ctx, bits == 4 || bits == 8, "ibcu_linear: bits=%d (4 or 8 supported)", bits);
    IBCU_REQUIRE(ctx, B >= 1 && B <= 32, "ibcu_linear: B=%d not in 1..32", B);
    IBCU_REQUIRE(ctx, N >= 1 && (bits == 8 || (N & 1) == 0), "ibcu_linear: N=%d invalid for %d-bit rows", N, bits);
    for (int i = 0; i < n_tensors; i++) {
        IBCU_REQUIRE(ctx, tensors[i].w && tensors[i].scales && tensors[i].out, "ibcu_linear: tensor %d has a null pointer", i);
        IBCU_REQUIRE(ctx, tensors[i].M >= 0 && tensors[i].out_stride >= tensors[i].M, "ibcu_linear: tensor %d M=%d stride=%d", i, tensors[i].M, tensors[i].out_stride);
    }
    const int rowbytes = bits == 8 ? N : N / 2;
    bool fast = !ctx->force_generic && (rowbytes % 16 == 0) && ((uintptr_t)x & 15) == 0 &&
                (!pro || ((((uintptr_t)pro->x2) & 15) == 0 && (((uintptr_t)pro->norm_w) & 3) == 0));
    for (int i = 0; i < n_tensors; i++) if (((uintptr_t)tensors[i].w & 15) != 0) fast = false;

    if (!fast) {
        if (op == IBCU_PRO_RMSNORM || op == IBCU_PRO_SILU_MUL) {
            // portable path: apply the prologue with the element-wise kernels into the context's activation buffer
            int rc0 = ibcu_reserve(ctx, &ctx->xpack, &ctx->xpack_bytes, (size_t)B * N * sizeof(float));
            if (rc0) return rc0;
            float* tmp = (float*)ctx->xpack;
            rc0 = op == IBCU_PRO_RMSNORM ? ibcu_rmsnorm_fp16w(ctx, tmp, x, pro->norm_w, pro->eps, N, B)
                                         : ibcu_silu_mul(ctx, tmp, x, pro->x2, (size_t)B * N);
            if (rc0) return rc0;
            x = tmp;
        }
        for (int i = 0; i < n_tensors; i++) {
            if (tensors[i].M == 0) continue;
            LinTensor T = { (const uint8_t*)tensors[i].w, tensors[i].scales, tensors[i].out, tensors[i].M,
                            tensors[i].out_stride, tensors[i].scales_fp32, tensors[i].epilogue, 0 };
            dim3 grid((tensors[i].M + 7) / 8);
            int rc = bits == 8 ? ibcu_launch(ctx, linear_generic_kernel<8>, grid, dim3(256), 0, 1, true, T, x, N, B)
                               : ibcu_launch(ctx, linear_generic_kernel<4>, grid, dim3(256), 0, 1, true, T, x, N, B);
            if (rc) return rc;
        }
        return IBCU_OK;
    }

    long total_rows = 0;
    for (int i = 0; i < n_tensors; i++) total_rows += tensors[i].M;
    if (total_rows == 0) return IBCU_OK;
    const LinPlan pl = lin_plan(ctx, tensors, n_tensors, total_rows, N, B < 16 ? B : 16, bits, op);
    bool tc = ctx->linear_tc > 0 && (bits == 4 || ctx->linear_tc > 1);
    // See lin_mma_us; beyond 16 activations the mma.sync kernel goes over the weights twice. The estimates know nothing of silu(x) * x2, which one block per
    // activation forms ahead of the mma.sync kernel: 5.3 to 6.5 us more than digits of a known maximum, behind the tcgen05 kernel in all of 656 calls
    // (1024 x 3072 INT8 at 4 activations 12.0 against 6.8 us, 4096 x 28672 48.6 against 41.0).
    if (ctx->linear_tc == 0)
        tc = B > 16 || (B > 1 && (op == IBCU_PRO_SILU_MUL || lin_tc_us(ibcu_linear_tc_cut(ctx->sm_count, tensors, n_tensors, N, B), N, bits) < lin_mma_us(pl, N, B, bits)));
    if (tc) {
        const int rc_tc = ibcu_linear_tc(ctx, tensors, n_tensors, x, N, B, bits, pro, op);
        if (rc_tc != IBCU_DECLINED) return rc_tc;
    }
    if (B > 16) {
        // sixteen activations fill the eight column groups of one pass; more go in a second pass
        ibcu_linear_t part[4];
        for (int b0 = 0; b0 < B; b0 += 16) {
            for (int i = 0; i < n_tensors; i++) { part[i] = tensors[i]; part[i].out = tensors[i].out + (size_t)b0 * tensors[i].out_stride; }
            ibcu_prologue_t pp; if (pro) { pp = *pro; if (pp.x2) pp.x2 += (size_t)b0 * N; if (pp.amax) pp.amax += (size_t)b0 * pp.n_amax; }
            int rc2 = ibcu_linear_ex(ctx, part, n_tensors, x + (size_t)b0 * N, N, B - b0 < 16 ? B - b0 : 16, bits, pro ? &pp : nullptr);
            if (rc2) return rc2;
        }
        return IBCU_OK;
    }
    const int ncols = pl.ncols, ncg = pl.ncg, nks = pl.nks, slice_kb = pl.slice_kb, xs_ld = pl.xs_ld, rt = pl.rt, stages = pl.stages;
    const int xk = bits == 8 ? 64 : 128;
    LinearParams p;
    memset(&p, 0, sizeof p);
    {
        int row_start = 0;
        for (int i = 0; i < n_tensors; i++) {
            p.t[i] = { (const uint8_t*)tensors[i].w, tensors[i].scales, tensors[i].out, tensors[i].M,
                       tensors[i].out_stride, tensors[i].scales_fp32, tensors[i].epilogue, row_start, pl.blk_start[i], pl.rows_per[i], -1 };
            row_start += tensors[i].M;
        }
    }
    // multi-GPU: a windowed exchange may be pending (wait in the first kernel of this call), and the outputs may be this
    // rank's slices of an announced gather (every result also goes, tagged, into the peers' windows from the epilogue)
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
    const int grid = pl.nblk * nks;

    const size_t xpack_bytes = (((size_t)nks * ncols * xs_ld) + 255) & ~(size_t)255;
    const size_t xscale_bytes = (((size_t)B * nks * sizeof(float)) + 255) & ~(size_t)255;
    int rc = ibcu_reserve(ctx, &ctx->xpack, &ctx->xpack_bytes, xpack_bytes + xscale_bytes + (size_t)B * nks * LIN_LIMBS * sizeof(int));
    if (rc) return rc;
    int8_t* xpack = (int8_t*)ctx->xpack;
    float* xscale = (float*)((char*)ctx->xpack + xpack_bytes);
    int* xsum = (int*)((char*)ctx->xpack + xpack_bytes + xscale_bytes);
    p.n_tensors = n_tensors; p.total_rows = (int)total_rows; p.rowbytes = rowbytes; p.nkb = pl.nkb; p.N = N; p.B = B; p.ncols = ncols;
    p.slice_kb = slice_kb; p.nks = nks; p.xs_ld = xs_ld;
    p.xpack = xpack; p.xscale = xscale; p.xsum = xsum;
    if (nks > 1) {
        const size_t part_bytes = (size_t)total_rows * nks * B * LIN_LIMBS * sizeof(int);
        rc = ibcu_reserve(ctx, &ctx->scratch, &ctx->scratch_bytes, part_bytes);
        if (rc) return rc;
        p.partial = (int*)ctx->scratch;
    }
    XSource xsrc = { x, pro ? pro->x2 : nullptr, pro ? (const __half*)pro->norm_w : nullptr, pro ? pro->eps : 0.0f, op,
                     op == IBCU_PRO_KNOWN_MAX ? pro->amax : nullptr, op == IBCU_PRO_KNOWN_MAX ? pro->n_amax : 0 };
    const bool fused = pl.fused;
    p.xsrc = xsrc; p.fused_x = fused ? 1 : 0;
    // 512 threads hold up to 16384 columns in registers; longer slices take 1024 threads and the looping conversion
    const int xthreads = slice_kb * xk > XREG_V * 4 * 512 ? 1024 : (slice_kb * xk >= 2048 ? 512 : 256);
    if (!fused) {
        const dim3 xg(nks, B);
        const int perm8 = bits == 4 ? 1 : 0, cols = slice_kb * xk;
        rc = xthreads == 1024 ? ibcu_launch(ctx, xprep_kernel<1024>, xg, dim3(1024), 0, 1, true, xsrc, N, cols, xs_ld, perm8, nks, 0, xpack, xscale, xsum, gw)
           : xthreads == 512  ? ibcu_launch(ctx, xprep_kernel<512>, xg, dim3(512), 0, 1, true, xsrc, N, cols, xs_ld, perm8, nks, 1, xpack, xscale, xsum, gw)
                              : ibcu_launch(ctx, xprep_kernel<256>, xg, dim3(256), 0, 1, true, xsrc, N, cols, xs_ld, perm8, nks, 1, xpack, xscale, xsum, gw);
        gw.flags = nullptr; gw.tag.n = 0;                     // the conversion kernel has waited and received; the main kernel follows it
    }
    p.gw = gw;
    if (rc) return rc;
    const size_t smem = pl.piece_smem + 32 * sizeof(float) + 32 * LIN_LIMBS * sizeof(int);
#define IBCU_DISPATCH(BITS) \
    switch (ncg) { \
        case 1: rc = dispatch_shape<BITS, 1>(ctx, p, grid, rt, stages, smem); break; \
        case 2: rc = dispatch_shape<BITS, 2>(ctx, p, grid, rt, stages, smem); break; \
        case 4: rc = dispatch_shape<BITS, 4>(ctx, p, grid, rt, stages, smem); break; \
        default: rc = dispatch_shape<BITS, 8>(ctx, p, grid, rt, stages, smem); break; \
    }
    if (bits == 8) { IBCU_DISPATCH(8) } else { IBCU_DISPATCH(4) }
#undef IBCU_DISPATCH
    if (rc) return rc;
    if (nks == 1) return rc;
    long outs = total_rows * B;
    int fgrid = (int)((outs + 255) / 256);
    if (fgrid > 4 * ctx->sm_count) fgrid = 4 * ctx->sm_count;
    return ibcu_launch(ctx, linear_finalize_kernel, dim3(fgrid), dim3(256), 0, 1, true, p);
}

// v1: the two projections in one launch, then the element-wise kernel over gate.out.
extern "C" int ibcu_linear_gate_up_silu(ibcu_ctx* ctx, const ibcu_linear_t* gate_up, const float* x, int N, int B, int bits) {
    IBCU_CHECK_CTX(ctx);
    IBCU_REQUIRE(ctx, gate_up && gate_up[0].M == gate_up[1].M && gate_up[0].out_stride == gate_up[1].out_stride,
                 "ibcu_linear_gate_up_silu: gate and up must have equal shapes");
    IBCU_REQUIRE(ctx, gate_up[0].epilogue == IBCU_EPI_STORE && gate_up[1].epilogue == IBCU_EPI_STORE, "ibcu_linear_gate_up_silu: store epilogue only");
    int rc = ibcu_linear(ctx, gate_up, 2, x, N, B, bits);
    if (rc) return rc;
    return ibcu_silu_mul(ctx, gate_up[0].out, gate_up[0].out, gate_up[1].out,
                         (size_t)(B - 1) * gate_up[0].out_stride + gate_up[0].M);
}
