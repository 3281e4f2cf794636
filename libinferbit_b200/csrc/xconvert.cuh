// Activations of the linear kernels as integer digits: X = rint(x * 2^s) per slice, four balanced base-256 digits
// ("limbs") per value. Shared by the mma.sync kernels (linear.cu) and the tcgen05 kernel (linear_tc.cu), which differ in
// where a digit lies: the destination is a type with put(limb, column, eight digits).
#pragma once
#include "common.cuh"

struct LinTensor {
    const uint8_t* w;
    const void* scales;
    float* out;
    int M, out_stride, scales_fp32, epilogue;
    int row_start;                 // first row of this tensor in the launch's concatenated row space
    int blk_start, rows_per;       // its blocks (per column slice) start at blk_start; each owns rows_per contiguous rows
    long win_off;                  // byte offset of `out` inside the peer window when the launch pushes its rows to the peers
};

struct XSource {                   // where an activation value comes from
    const float* x;                // [B][N]
    const float* x2;               // second operand of silu(x)*x2, or NULL
    const __half* norm_w;          // RMSNorm weights, or NULL
    float eps;
    int op;                        // IBCU_PRO_*
    const float* amax;             // IBCU_PRO_KNOWN_MAX: [B][n_amax] pieces of max|x[b]|
    int n_amax;
};

constexpr int LIN_LIMBS = 4;

// How the tcgen05 kernel cuts a call: runs of R rows in T tiles of 128, each by a cluster of S blocks that share its nkb blocks of 128
// columns; slots clusters are resident at once.
struct TqCut { int S, R, T, nkb, slots, nruns, NC; };
TqCut ibcu_linear_tc_cut(int sm_count, const ibcu_linear_t* tensors, int n_tensors, int N, int B);      // linear_tc.cu

// rows of digits, one per limb, ld bytes apart (mma.sync kernels)
struct XRows {
    int8_t* p; int ld;
    __device__ __forceinline__ void put(int l, int j, uint2 v) const { *reinterpret_cast<uint2*>(p + (size_t)l * ld + j) = v; }
};
// The operand image of the tcgen05 kernel: per block of 128 columns nc rows of 128 bytes (row = 4 * activation + limb) in the
// 128-byte swizzle, 16-byte piece c of row n at piece c ^ (n % 8); a block is one contiguous copy into shared memory.
struct XTiles {
    int8_t* base; int nc, row0, col0;
    __device__ __forceinline__ void put(int l, int j, uint2 v) const {
        const int col = col0 + j, n = row0 + l;
        *reinterpret_cast<uint2*>(base + (size_t)(col >> 7) * (nc * 128) + n * 128 + ((((col >> 4) & 7) ^ (n & 7)) << 4) + (col & 15)) = v;
    }
};

// ── activation split ────────────────────────────────────────────────────────────────────
// grid (nks, B), one block per slice of one activation: X = rint(x * 2^s) with 2^s * max|x| in
// [2^29, 2^30), then X = d0 + 256 d1 + 65536 d2 + 2^24 d3 with every digit in [-128, 127].
// Eight columns at a time: INT8 consumers get them in natural order, INT4 consumers as
// c0,c2,c4,c6,c1,c3,c5,c7 (low nibbles of four bytes, then high nibbles).

// four consecutive transformed activation values starting at column j of activation row xb
__device__ __forceinline__ float4 xsrc_load4(const XSource& s, const float* xb, const float* x2b, int col, float r) {
    float4 v = *reinterpret_cast<const float4*>(xb + col);
    if (s.op == IBCU_PRO_RMSNORM) {
        const __half2 w01 = *reinterpret_cast<const __half2*>(s.norm_w + col), w23 = *reinterpret_cast<const __half2*>(s.norm_w + col + 2);
        v.x = v.x * r * __low2float(w01); v.y = v.y * r * __high2float(w01);
        v.z = v.z * r * __low2float(w23); v.w = v.w * r * __high2float(w23);
    } else if (s.op == IBCU_PRO_SILU_MUL) {
        const float4 u = *reinterpret_cast<const float4*>(x2b + col);
        v.x = v.x / (1.0f + expf(-v.x)) * u.x; v.y = v.y / (1.0f + expf(-v.y)) * u.y;
        v.z = v.z / (1.0f + expf(-v.z)) * u.z; v.w = v.w / (1.0f + expf(-v.w)) * u.w;
    }
    return v;
}

// Balanced base-256 digits of eight fixed-point values, as limb words. With Y = X + 0x00808080 the
// unsigned bytes u_l of Y satisfy X = sum (u_l - 128) 256^l (l < 3) + (Y >> 24) 2^24, and u_l - 128 as
// a signed byte is u_l ^ 0x80: so the four digits of X are the four bytes of Y ^ 0x00808080. Two 4x4
// byte transposes turn eight such words into limb-major words; bit 0 of perm8 picks the INT4 column order of the
// mma.sync kernel, any non-zero perm8 also asks for the limb sums (perm8 == 2: natural order with sums).
__device__ __forceinline__ void transpose4x4_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t* o) {
    const uint32_t t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(a, b, 0x7362);
    const uint32_t t2 = __byte_perm(c, d, 0x5140), t3 = __byte_perm(c, d, 0x7362);
    o[0] = __byte_perm(t0, t2, 0x5410); o[1] = __byte_perm(t0, t2, 0x7632);
    o[2] = __byte_perm(t1, t3, 0x5410); o[3] = __byte_perm(t1, t3, 0x7632);
}
__device__ __forceinline__ void limbs8(const int* X, int perm8, uint2* pk, int* lsum) {
    uint32_t D[8], lo[4], hi[4];
#pragma unroll
    for (int i = 0; i < 8; i++) D[i] = ((uint32_t)X[i] + 0x00808080u) ^ 0x00808080u;
    if (perm8 & 1) { transpose4x4_bytes(D[0], D[2], D[4], D[6], lo); transpose4x4_bytes(D[1], D[3], D[5], D[7], hi); }
    else       { transpose4x4_bytes(D[0], D[1], D[2], D[3], lo); transpose4x4_bytes(D[4], D[5], D[6], D[7], hi); }
#pragma unroll
    for (int l = 0; l < LIN_LIMBS; l++) {
        pk[l] = make_uint2(lo[l], hi[l]);
        lsum[l] = __dp4a((int)lo[l], 0x01010101, __dp4a((int)hi[l], 0x01010101, lsum[l]));
    }
}

// Converts columns [c0, c0 + slice_cols) of activation b to limbs. Called by every thread of a block
// (it synchronises); dst takes the limbs of this activation and slice, in global or shared memory. Thread 0 stores 2^-s to *back_out, threads 0..3 the limb sums to sum_out.
struct XScratch { float red[32]; int sred[32][LIN_LIMBS]; float mul, r; };

template <class D>
__device__ __forceinline__ void xconvert(const XSource& src, int N, int b, int c0, int slice_cols, const D& dst,
                                         int perm8, XScratch& sc, float* back_out, int* sum_out) {
    const int nth = blockDim.x, nwarp = nth >> 5;
    const int valid = max(0, min(slice_cols, N - c0));       // N and c0 are multiples of 16
    const float* xrow = src.x + (size_t)b * N;
    const float* xb = xrow + c0;
    const float* x2b = src.x2 ? src.x2 + (size_t)b * N + c0 : nullptr;
    float r = 1.0f;
    if (src.op == IBCU_PRO_RMSNORM) {                         // 1/sqrt(mean(x^2) + eps) over the whole row (src/kernels/scalar.c:126-138)
        float ss = 0.0f;
        for (int j = threadIdx.x * 4; j < N; j += nth * 4) {
            const float4 v = *reinterpret_cast<const float4*>(xrow + j);
            ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
        }
        ss = warp_sum(ss);
        __syncthreads();
        if ((threadIdx.x & 31) == 0) sc.red[threadIdx.x >> 5] = ss;
        __syncthreads();
        if (threadIdx.x == 0) {
            float t = 0.0f;
            for (int w = 0; w < nwarp; w++) t += sc.red[w];
            sc.r = 1.0f / sqrtf(t / (float)N + src.eps);
        }
        __syncthreads();
        r = sc.r;
    }
    XSource sl = src;
    sl.norm_w = src.norm_w ? src.norm_w + c0 : nullptr;
    float amax = 0.0f;
    for (int j = threadIdx.x * 4; j < valid; j += nth * 4) {
        const float4 v = xsrc_load4(sl, xb, x2b, j, r);
        amax = fmaxf(fmaxf(amax, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));
    }
    amax = warp_max(amax);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sc.red[threadIdx.x >> 5] = amax;
    __syncthreads();
    if (threadIdx.x == 0) {
        float v = sc.red[0];
        for (int w = 1; w < nwarp; w++) v = fmaxf(v, sc.red[w]);
        const int e = (int)((__float_as_uint(v) >> 23) & 0xFF);      // v in [2^(e-127), 2^(e-126))
        int sh = (v > 0.0f && e != 255) ? 156 - e : 0;               // 2^sh * v in [2^29, 2^30)
        sh = max(-126, min(126, sh));
        sc.mul = __uint_as_float((uint32_t)(127 + sh) << 23);
        *back_out = __uint_as_float((uint32_t)(127 - sh) << 23);
    }
    __syncthreads();
    const float mul = sc.mul;
    int lsum[LIN_LIMBS] = {0, 0, 0, 0};
    for (int j = threadIdx.x * 8; j < slice_cols; j += nth * 8) {
        int X[8];
        if (j < valid) {
            const float4 a = xsrc_load4(sl, xb, x2b, j, r), c = xsrc_load4(sl, xb, x2b, j + 4, r);
            X[0] = __float2int_rn(a.x * mul); X[1] = __float2int_rn(a.y * mul); X[2] = __float2int_rn(a.z * mul); X[3] = __float2int_rn(a.w * mul);
            X[4] = __float2int_rn(c.x * mul); X[5] = __float2int_rn(c.y * mul); X[6] = __float2int_rn(c.z * mul); X[7] = __float2int_rn(c.w * mul);
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) X[i] = 0;
        }
        uint2 pk[LIN_LIMBS];
        limbs8(X, perm8, pk, lsum);
#pragma unroll
        for (int l = 0; l < LIN_LIMBS; l++) dst.put(l, j, pk[l]);
    }
#pragma unroll
    for (int l = 0; l < LIN_LIMBS; l++) {
        int v = lsum[l];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) sc.sred[threadIdx.x >> 5][l] = v;
    }
    __syncthreads();
    if (threadIdx.x < LIN_LIMBS) {
        int v = 0;
        for (int w = 0; w < nwarp; w++) v += sc.sred[w][threadIdx.x];
        sum_out[threadIdx.x] = v;
    }
}

// The same conversion with the whole slice held in registers (up to V float4 per thread): every global
// load of the block is issued before the first one is used, so the block pays one memory round trip
// instead of one per loop iteration. Values, digits and sums are those of xconvert.
template <int V, class D>
__device__ __forceinline__ void xconvert_regs(const XSource& src, int N, int b, int c0, int slice_cols, const D& dst,
                                              int perm8, XScratch& sc, float* back_out, int* sum_out) {
    constexpr int P = V / 2;                                  // groups of 8 columns per thread
    const int nth = blockDim.x, nwarp = nth >> 5;
    const int valid = max(0, min(slice_cols, N - c0));       // N and c0 are multiples of 16
    const float* xrow = src.x + (size_t)b * N;
    const float* xb = xrow + c0;
    float4 va[P], vc[P];
#pragma unroll
    for (int i = 0; i < P; i++) {
        const int j = (threadIdx.x + i * nth) * 8;
        va[i] = vc[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (j < valid) { va[i] = *reinterpret_cast<const float4*>(xb + j); vc[i] = *reinterpret_cast<const float4*>(xb + j + 4); }
    }
    if (src.op == IBCU_PRO_SILU_MUL) {
        const float* x2b = src.x2 + (size_t)b * N + c0;
        float4 ua[P], uc[P];
#pragma unroll
        for (int i = 0; i < P; i++) {
            const int j = (threadIdx.x + i * nth) * 8;
            ua[i] = uc[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (j < valid) { ua[i] = *reinterpret_cast<const float4*>(x2b + j); uc[i] = *reinterpret_cast<const float4*>(x2b + j + 4); }
        }
#pragma unroll
        for (int i = 0; i < P; i++) {
            float4& a = va[i]; float4& c = vc[i];
            a.x = a.x / (1.0f + expf(-a.x)) * ua[i].x; a.y = a.y / (1.0f + expf(-a.y)) * ua[i].y;
            a.z = a.z / (1.0f + expf(-a.z)) * ua[i].z; a.w = a.w / (1.0f + expf(-a.w)) * ua[i].w;
            c.x = c.x / (1.0f + expf(-c.x)) * uc[i].x; c.y = c.y / (1.0f + expf(-c.y)) * uc[i].y;
            c.z = c.z / (1.0f + expf(-c.z)) * uc[i].z; c.w = c.w / (1.0f + expf(-c.w)) * uc[i].w;
        }
    } else if (src.op == IBCU_PRO_RMSNORM) {                  // 1/sqrt(mean(x^2) + eps) over the whole row (src/kernels/scalar.c:126-138)
        __half2 w[P][4];
        const bool w16 = ((uintptr_t)(src.norm_w + c0) & 15) == 0;
#pragma unroll
        for (int i = 0; i < P; i++) {
            const int j = (threadIdx.x + i * nth) * 8;
            if (j < valid && w16) {
                const uint4 raw = *reinterpret_cast<const uint4*>(src.norm_w + c0 + j);
                w[i][0] = *reinterpret_cast<const __half2*>(&raw.x); w[i][1] = *reinterpret_cast<const __half2*>(&raw.y);
                w[i][2] = *reinterpret_cast<const __half2*>(&raw.z); w[i][3] = *reinterpret_cast<const __half2*>(&raw.w);
            } else {
#pragma unroll
                for (int q = 0; q < 4; q++)
                    w[i][q] = j < valid ? *reinterpret_cast<const __half2*>(src.norm_w + c0 + j + 2 * q) : __floats2half2_rn(0.0f, 0.0f);
            }
        }
        float ss = 0.0f;
        if (c0 == 0 && valid == N) {
#pragma unroll
            for (int i = 0; i < P; i++) {
                ss = fmaf(va[i].x, va[i].x, fmaf(va[i].y, va[i].y, fmaf(va[i].z, va[i].z, fmaf(va[i].w, va[i].w, ss))));
                ss = fmaf(vc[i].x, vc[i].x, fmaf(vc[i].y, vc[i].y, fmaf(vc[i].z, vc[i].z, fmaf(vc[i].w, vc[i].w, ss))));
            }
        } else {
            for (int j = threadIdx.x * 4; j < N; j += nth * 4) {
                const float4 v = *reinterpret_cast<const float4*>(xrow + j);
                ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
            }
        }
        ss = warp_sum(ss);
        __syncthreads();
        if ((threadIdx.x & 31) == 0) sc.red[threadIdx.x >> 5] = ss;
        __syncthreads();
        float t = 0.0f;
        for (int q = 0; q < nwarp; q++) t += sc.red[q];       // every thread adds in the same order: no broadcast step
        const float r = 1.0f / sqrtf(t / (float)N + src.eps);
#pragma unroll
        for (int i = 0; i < P; i++) {
            va[i].x = va[i].x * r * __low2float(w[i][0]); va[i].y = va[i].y * r * __high2float(w[i][0]);
            va[i].z = va[i].z * r * __low2float(w[i][1]); va[i].w = va[i].w * r * __high2float(w[i][1]);
            vc[i].x = vc[i].x * r * __low2float(w[i][2]); vc[i].y = vc[i].y * r * __high2float(w[i][2]);
            vc[i].z = vc[i].z * r * __low2float(w[i][3]); vc[i].w = vc[i].w * r * __high2float(w[i][3]);
        }
    }
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < P; i++) {
        amax = fmaxf(fmaxf(amax, fmaxf(fabsf(va[i].x), fabsf(va[i].y))), fmaxf(fabsf(va[i].z), fabsf(va[i].w)));
        amax = fmaxf(fmaxf(amax, fmaxf(fabsf(vc[i].x), fabsf(vc[i].y))), fmaxf(fabsf(vc[i].z), fabsf(vc[i].w)));
    }
    amax = warp_max(amax);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sc.red[threadIdx.x >> 5] = amax;
    __syncthreads();
    float vmax = sc.red[0];
    for (int q = 1; q < nwarp; q++) vmax = fmaxf(vmax, sc.red[q]);
    const int e = (int)((__float_as_uint(vmax) >> 23) & 0xFF);       // vmax in [2^(e-127), 2^(e-126))
    int sh = (vmax > 0.0f && e != 255) ? 156 - e : 0;                // 2^sh * vmax in [2^29, 2^30)
    sh = max(-126, min(126, sh));
    const float mul = __uint_as_float((uint32_t)(127 + sh) << 23);
    if (threadIdx.x == 0) *back_out = __uint_as_float((uint32_t)(127 - sh) << 23);
    int lsum[LIN_LIMBS] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < P; i++) {
        const int j = (threadIdx.x + i * nth) * 8;
        if (j >= slice_cols) continue;
        int X[8];
        X[0] = __float2int_rn(va[i].x * mul); X[1] = __float2int_rn(va[i].y * mul); X[2] = __float2int_rn(va[i].z * mul); X[3] = __float2int_rn(va[i].w * mul);
        X[4] = __float2int_rn(vc[i].x * mul); X[5] = __float2int_rn(vc[i].y * mul); X[6] = __float2int_rn(vc[i].z * mul); X[7] = __float2int_rn(vc[i].w * mul);
        uint2 pk[LIN_LIMBS];
        limbs8(X, perm8, pk, lsum);
#pragma unroll
        for (int l = 0; l < LIN_LIMBS; l++) dst.put(l, j, pk[l]);
    }
    if (!perm8) return;                                       // the limb sums only remove the nibble bias of INT4 weights
#pragma unroll
    for (int l = 0; l < LIN_LIMBS; l++) {
        int v = lsum[l];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) sc.sred[threadIdx.x >> 5][l] = v;
    }
    __syncthreads();
    if (threadIdx.x < LIN_LIMBS) {
        int v = 0;
        for (int q = 0; q < nwarp; q++) v += sc.sred[q][threadIdx.x];
        sum_out[threadIdx.x] = v;
    }
}

// Groups of 8 columns in flight per thread. One: every block of a launch converts the same row while its weights are on their way, and
// more requests for the same lines at once only queue in front of them (step of a 7B shape: one 1929, two 1972, four 1975, eight 2040 us).
constexpr int XKNOWN_U = 1;
// The conversion when the caller knows max|x[b]| (IBCU_PRO_KNOWN_MAX): no reduction before the digits, so
// rows of any length stream through in one pass.
template <class D>
__device__ __forceinline__ void xconvert_known(const XSource& src, int N, int b, int c0, int slice_cols, const D& dst,
                                               int perm8, XScratch& sc, float* back_out, int* sum_out) {
    const int nth = blockDim.x, nwarp = nth >> 5;
    const int valid = max(0, min(slice_cols, N - c0));
    const float* xb = src.x + (size_t)b * N + c0;
    // the pieces of the maximum, a lane each, and the first columns are on their way together
    float vmax = 0.0f;
    for (int q = threadIdx.x & 31; q < src.n_amax; q += 32) vmax = fmaxf(vmax, src.amax[(size_t)b * src.n_amax + q]);
    int lsum[LIN_LIMBS] = {0, 0, 0, 0};
    constexpr int U = XKNOWN_U;
    float4 va[U], vc[U];
    auto load = [&](int j0) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int j = j0 + u * nth * 8;
            va[u] = vc[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (j < valid) { va[u] = *reinterpret_cast<const float4*>(xb + j); vc[u] = *reinterpret_cast<const float4*>(xb + j + 4); }
        }
    };
    load(threadIdx.x * 8);
    vmax = warp_max(vmax);
    const int e = (int)((__float_as_uint(vmax) >> 23) & 0xFF);
    int sh = (vmax > 0.0f && e != 255) ? 156 - e : 0;
    sh = max(-126, min(126, sh));
    const float mul = __uint_as_float((uint32_t)(127 + sh) << 23);
    if (threadIdx.x == 0) *back_out = __uint_as_float((uint32_t)(127 - sh) << 23);
    for (int j0 = threadIdx.x * 8; j0 < slice_cols; j0 += nth * 8 * U) {
        if (j0 != threadIdx.x * 8) load(j0);
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int j = j0 + u * nth * 8;
            if (j >= slice_cols) continue;
            int X[8];
            X[0] = __float2int_rn(va[u].x * mul); X[1] = __float2int_rn(va[u].y * mul); X[2] = __float2int_rn(va[u].z * mul); X[3] = __float2int_rn(va[u].w * mul);
            X[4] = __float2int_rn(vc[u].x * mul); X[5] = __float2int_rn(vc[u].y * mul); X[6] = __float2int_rn(vc[u].z * mul); X[7] = __float2int_rn(vc[u].w * mul);
            uint2 pk[LIN_LIMBS];
            limbs8(X, perm8, pk, lsum);
#pragma unroll
            for (int l = 0; l < LIN_LIMBS; l++) dst.put(l, j, pk[l]);
        }
    }
    if (!perm8) return;                                       // the limb sums only remove the nibble bias of INT4 weights
    if (b > 0) __syncthreads();                               // a block that converts several in turn: threads 0..3 may still be adding up the sums of the one before
#pragma unroll
    for (int l = 0; l < LIN_LIMBS; l++) {
        int v = lsum[l];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) sc.sred[threadIdx.x >> 5][l] = v;
    }
    __syncthreads();
    if (threadIdx.x < LIN_LIMBS) {
        int v = 0;
        for (int q = 0; q < nwarp; q++) v += sc.sred[q][threadIdx.x];
        sum_out[threadIdx.x] = v;
    }
}

constexpr int XREG_V = 8;                                     // 32 columns per thread in registers
template <int V = XREG_V, class D>
__device__ __forceinline__ void xconvert_any(const XSource& src, int N, int b, int c0, int slice_cols, const D& dst,
                                             int perm8, XScratch& sc, float* back_out, int* sum_out, int xregs = 1) {
    if (src.op == IBCU_PRO_KNOWN_MAX) { xconvert_known(src, N, b, c0, slice_cols, dst, perm8, sc, back_out, sum_out); return; }
    if (xregs && slice_cols <= V * 4 * (int)blockDim.x) xconvert_regs<V>(src, N, b, c0, slice_cols, dst, perm8, sc, back_out, sum_out);
    else xconvert(src, N, b, c0, slice_cols, dst, perm8, sc, back_out, sum_out);
}
