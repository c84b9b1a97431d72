// recon.cu -- reconstruction of the transform-block records of a batch of
// pictures: dequantisation + inverse DCT/DST / transform skip / transquant
// bypass (transform.rs), intra prediction (intra.rs) and residual add + clip
// (reconstruct.rs), in the decode order of decode.rs:3478-5426.
//
// Two kernels:
//
//  k_residual -- every coded TB of every picture, fully parallel (a lane, eight
//     lanes or a warp per TB by its size).  The TBs of prediction-in-plane
//     pictures are added and clipped into the plane right away; all others
//     leave an int16 residual in a residual plane, which k_recon adds to intra
//     and motion compensation to inter samples (so the residuals of a sequence
//     wait for nothing and stay off its frame-to-frame chain).
//     (for 8-bit the reference itself truncates to i16, transform.rs:55-63;
//     then every residual is clamped to +-(2^bd - 1), which the clip of the
//     sum to [0, 2^bd - 1] cannot tell from the full value.)
//
//  k_recon -- the intra wavefront.  One CTA reconstructs one CTU at a time;
//     CTUs are claimed from a global queue sorted by wavefront index
//     (x + 2y) across all pictures, so a CTU is only claimed after every CTU
//     it depends on (left, above-left, above, above-right) was claimed by a
//     running CTA: no deadlock for any grid size.  Per CTU all warps turn the
//     records into walk entries, residuals are staged with cp.async and a
//     blend table is filled, all in shared memory; then luma, Cb and Cr are
//     walked by warps of their own in parallel (chroma availability only
//     depends on the luma `decoded` map, which the records give beforehand).
//     Neighbours synchronise per TB: a walking warp writes the samples of its
//     CTU's right column and bottom row into edge words as each TB is done,
//     and the CTA's last warp moves the neighbours' words into shared memory,
//     where a walking warp looks before a TB on the CTU's top or left edge
//     (waits bounded).  So a CTU starts while its left and above-right
//     neighbours are still being walked.  Finally the whole CTU is written out
//     for the filters.
#include <mutex>
#include <climits>

#include "common.cuh"

namespace hpvcd {

// intra.rs:30-38 (H.265 Tables 8-4 / 8-5)
__constant__ int8_t c_intra_angle[33] = {32,  26,  21,  17,  13,  9,  5,  2,  0,  -2, -5,
                                         -9,  -13, -17, -21, -26, -32, -26, -21, -17, -13, -9,
                                         -5,  -2,  0,   2,   5,   9,   13,  17,  21,  26,  32};
__constant__ int16_t c_inv_angle[15] = {-4096, -1638, -910, -630, -482, -390, -315, -256,
                                        -315,  -390,  -482, -630, -910, -1638, -4096};
// transform.rs:37
__constant__ int32_t c_dequant_scale[6] = {40, 45, 51, 57, 64, 72};
// transform.rs:30 DST4
__constant__ int8_t c_dst4[4][4] = {{29, 55, 74, 84}, {74, 74, 0, -74}, {84, -29, -74, 55}, {55, -84, 74, -29}};
constexpr int kScr = 33;  // padded row stride of the transform scratch
// Inverse-transform variants of k_residual (schedule knob; pixels identical).
constexpr int kIdctMatrix = 0;     // matrix product, all-zero rows / columns skipped
constexpr int kIdctButterfly = 1;  // even-odd butterflies for 16x16 and 32x32 TBs
constexpr int kIdctTensor = 2;     // integer tensor-core products (int8 halves) for 16x16 and 32x32 TBs

__device__ __forceinline__ int sat16(int v) { return v < -32768 ? -32768 : (v > 32767 ? 32767 : v); }

// A residual as the residual planes hold it, mx the largest sample: clip(pred
// + r, 0, mx) is the same for r clamped to [-mx, mx], and the sum of a sample
// and a clamped residual fits 16 bits.
__device__ __forceinline__ int16_t res_store(int v, int mx) { return (int16_t)clamp3i(v, -mx, mx); }

// Entry (k, m) of the n-point H.265 DCT basis as a compile-time constant (the
// multipliers of the unrolled butterflies, the tables below); mag: the basis
// magnitudes by angle j, in units of pi/64.
__host__ __device__ constexpr int dct_c(int n, int k, int m) {
    constexpr int8_t mag[33] = {64, 90, 90, 90, 89, 88, 87, 85, 83, 82, 80, 78, 75, 73, 70, 67, 64,
                                61, 57, 54, 50, 46, 43, 38, 36, 31, 25, 22, 18, 13, 9,  4,  0};
    if (k == 0) return 64;
    int j = (k * (32 / n) * (2 * m + 1)) & 127;
    int sign = 1;
    if (j > 64) j = 128 - j;
    if (j > 32) {
        j = 64 - j;
        sign = -1;
    }
    return sign * mag[j];
}

// Even-odd (partial butterfly) N-point inverse: out[m] = sum_{k < KMAX}
// T_N[k][m] * in[k * S].  Rows of the basis are symmetric for even k and
// antisymmetric for odd k, and T_N[2j][m] = T_{N/2}[j][m], so the even
// coefficients form an N/2-point inverse and out[N-1-m] = E[m] - O[m].
// Integer sums in any order are identical, so the result equals the matrix
// product bit for bit (the clip follows the complete sum in both forms).
template <int N, int S, int KMAX>
__device__ __forceinline__ void inv_butterfly(const int* in, int* out) {
    if constexpr (N == 1) {
        out[0] = KMAX > 0 ? 64 * in[0] : 0;
    } else {
        int e[N / 2];
        inv_butterfly<N / 2, 2 * S, (KMAX + 1) / 2>(in, e);
#pragma unroll
        for (int m = 0; m < N / 2; ++m) {
            int o = 0;
#pragma unroll
            for (int k = 1; k < KMAX && k < N; k += 2) o += dct_c(N, k, m) * in[k * S];
            out[m] = e[m] + o;
            out[N - 1 - m] = e[m] - o;
        }
    }
}

// One stage of a 16- or 32-point inverse by butterflies, lane = line:
// line l reads in[k] = src[l * ls + k * ks] for k < KMAX (the rest are zero)
// and writes dst[l * ld + m * md] = fin(out[m]).
template <int N, int KMAX, typename Fin>
__device__ __forceinline__ void bf_stage(const int16_t* src, int ls, int ks, int16_t* dst, int ld, int md, int lane,
                                         Fin fin) {
    if (lane >= N) return;
    int in[KMAX], out[N];
#pragma unroll
    for (int k = 0; k < KMAX; ++k) in[k] = src[lane * ls + k * ks];
    inv_butterfly<N, 1, KMAX>(in, out);
#pragma unroll
    for (int m = 0; m < N; ++m) dst[lane * ld + m * md] = (int16_t)fin(out[m]);
}

template <int N, typename Fin>
__device__ __forceinline__ void bf_stage_k(int kcount, const int16_t* src, int ls, int ks, int16_t* dst, int ld,
                                           int md, int lane, Fin fin) {
    if (kcount <= 4)
        bf_stage<N, 4>(src, ls, ks, dst, ld, md, lane, fin);
    else if (kcount <= 8)
        bf_stage<N, 8>(src, ls, ks, dst, ld, md, lane, fin);
    else if (N == 16 || kcount <= 16)
        bf_stage<N, (N < 16 ? N : 16)>(src, ls, ks, dst, ld, md, lane, fin);
    else
        bf_stage<N, N>(src, ls, ks, dst, ld, md, lane, fin);
}

// ===========================================================================
// Integer tensor-core inverse transform of 16x16 and 32x32 TBs.
//
// Both stages are products with the H.265 basis T (entries in [-90, 90], an
// s8 value): stage 1 tmp = T^T * D over the dequantised coefficients D,
// stage 2 out = tmp * T.  The int16 operand X of each product is split
// exactly into a signed high byte and an unsigned low byte, X = 256 * hi +
// lo, and the product is 256 * (T * hi) + (T * lo): two mma.sync products
// with s32 accumulation.  No sum overflows (|sum| <= 32 * 90 * 32768 <
// 2^31), so the result is the reference's integer sum bit for bit; the
// rounding, shift and clip of each stage are applied to it unchanged.
// Fragments follow the PTX layouts of mma.m16n8k32 (32x32 TBs) and
// mma.m16n8k16 (16x16 TBs) with 8-bit operands: lane = 4 * group + t; an A
// register holds four consecutive K entries of one row (row group or group
// + 8), a B register four consecutive K entries of one column (group), a
// C/D register pair two adjacent columns (2t, 2t + 1) of one row.
// ===========================================================================
__device__ __forceinline__ void mma32(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, bool a_u8,
                                      bool b_u8) {
    // D += A * B, A 16x32 (row), B 32x8 (col), 8-bit operands, s32 accumulation
    if (!a_u8 && !b_u8)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                     "{%0,%1,%2,%3};"
                     : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else if (!a_u8)
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                     "{%0,%1,%2,%3};"
                     : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                     "{%0,%1,%2,%3};"
                     : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, bool a_u8, bool b_u8) {
    // D += A * B, A 16x16 (row), B 16x8 (col), 8-bit operands, s32 accumulation
    if (!a_u8 && !b_u8)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                     : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                     : "r"(a0), "r"(a1), "r"(b0));
    else if (!a_u8)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                     : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                     : "r"(a0), "r"(a1), "r"(b0));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
                     : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                     : "r"(a0), "r"(a1), "r"(b0));
}

// Basis fragments, per lane (index [entry][lane]):
//   s1a32: T^T as the A operand of stage 1, 32x32: 2 row tiles x 4 registers
//   s2b32: T as the B operand of stage 2, 32x32: 4 column tiles x 2 registers
//   s1a16: T^T, 16x16: 2 registers;  s2b16: T, 16x16: 2 column tiles x 1 register
// Stage 2 takes stage 1's accumulators as its A operand without moving them
// between lanes: byte i of lane t's register holds column 8 * (i / 2) + 2t +
// (i & 1) of its half instead of column 4t + i, and the rows of the stage-2
// basis are permuted the same way (a sum over K in another order).
constexpr int kFragS1A32 = 0, kFragS2B32 = 8, kFragS1A16 = 16, kFragS2B16 = 18, kFragEntries = 20;

// The basis as the kernels stage it into shared memory, computed at compile
// time (building it in every CTA cost a launch several microseconds of
// serialised constant reads).
struct BasisTables {
    uint32_t frags[kFragEntries * 32];
    int16_t dct[32 * 32];
};
constexpr BasisTables make_basis() {
    BasisTables B{};
    for (int i = 0; i < 32 * 32; ++i) B.dct[i] = (int16_t)dct_c(32, i / 32, i % 32);
    for (int e = 0; e < kFragEntries * 32; ++e) {
        const int entry = e >> 5, lane = e & 31, g = lane >> 2, t = lane & 3;
        uint32_t w = 0;
        for (int i = 0; i < 4; ++i) {
            int n = 0, k = 0, m = 0;
            if (entry < kFragS2B32) {  // A of stage 1, n = 32: A[m][k] = T[k][m]
                const int mt = entry >> 2, reg = entry & 3;
                n = 32, m = mt * 16 + g + (reg & 1) * 8, k = (reg >> 1) * 16 + 4 * t + i;
            } else if (entry < kFragS1A16) {  // B of stage 2, n = 32 (permuted rows)
                const int nt = (entry - kFragS2B32) >> 1, reg = (entry - kFragS2B32) & 1;
                n = 32, m = nt * 8 + g, k = reg * 16 + (i >> 1) * 8 + 2 * t + (i & 1);
            } else if (entry < kFragS2B16) {  // A of stage 1, n = 16
                n = 16, m = g + (entry - kFragS1A16) * 8, k = 4 * t + i;
            } else {  // B of stage 2, n = 16 (permuted rows)
                n = 16, m = (entry - kFragS2B16) * 8 + g, k = (i >> 1) * 8 + 2 * t + (i & 1);
            }
            w |= (uint32_t)(dct_c(n, k, m) & 0xff) << (8 * i);
        }
        B.frags[e] = w;
    }
    return B;
}
__device__ const __align__(16) BasisTables g_basis = make_basis();

// Copies `bytes` (a multiple of 16) of a table into shared memory.
__device__ __forceinline__ void stage_table(void* dst, const void* src, int bytes) {
    for (int i = threadIdx.x; i < bytes / 16; i += blockDim.x) ((uint4*)dst)[i] = ((const uint4*)src)[i];
}

// Four int16 values (each in the low half of its word) split into their high
// bytes (s8) and low bytes (u8).
__device__ __forceinline__ void split4(int a, int b, int c, int d, uint32_t& hi, uint32_t& lo) {
    const uint32_t ab = __byte_perm((uint32_t)a, (uint32_t)b, 0x5410), cd = __byte_perm((uint32_t)c, (uint32_t)d, 0x5410);
    lo = __byte_perm(ab, cd, 0x6420);
    hi = __byte_perm(ab, cd, 0x7531);
}

// Four 8x8 matrices of 16-bit entries from shared memory, transposed: lane l
// passes the address of row l % 8 of matrix l / 8 and receives entries
// (2t, g) and (2t + 1, g) of each.
__device__ __forceinline__ void ldmatrix_x4_trans(const int16_t* row, uint32_t (&r)[4]) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(row);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a)
                 : "memory");
}

// Row stride of the dequantised block in shared memory: rows stay 16-byte
// aligned and eight consecutive rows of a column block fall into different
// banks.
__host__ __device__ constexpr int tensor_stride(int n) { return n == 32 ? 40 : 24; }

// Both stages of an n x n (16 or 32) inverse DCT by one warp: buf holds the
// dequantised coefficients (row k, column c, stride tensor_stride(n));
// emit(mt, out) gets, per 16-row tile, out[nt][e] = row mt * 16 + g + 8 *
// (e / 2), column nt * 8 + 2t + (e & 1), before the storage wrap.  The row
// tiles are a rolled loop: the kernel's tasks of every size run side by side on
// an SM, and its warps waited for instructions before anything else.  Stage 1's
// operand fragments are four rows of one column: two transposed 8x8 loads
// whose row addresses interleave rows 4t, 4t + 1 and 4t + 2, 4t + 3.
template <int N, typename Emit>
__device__ __forceinline__ void idct_tensor(const int16_t* buf, const uint32_t* frags, int bd, int lane, Emit emit) {
    constexpr int MT = N / 16, NT = N / 8;  // row tiles, column tiles
    constexpr int STR = tensor_stride(N);
    // ---- stage 1: tmp[m][c] = clip((sum_k T[k][m] D[k][c] + 64) >> 7) ----
    const int mat = lane >> 3, li = lane & 7;
    const int row = 4 * (li >> 1) + (li & 1) + 2 * (mat & 1);
    uint32_t bh[NT][N / 16], bl[NT][N / 16];
#pragma unroll
    for (int q = 0; q < NT * (N / 16) / 2; ++q) {
        // N = 16: one load covers both column tiles; N = 32: one column tile,
        // both 16-row halves
        uint32_t r[4];
        if constexpr (N == 16)
            ldmatrix_x4_trans(buf + row * STR + 8 * (mat >> 1), r);
        else
            ldmatrix_x4_trans(buf + (row + 16 * (mat >> 1)) * STR + 8 * q, r);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int nt = N == 16 ? h : q, reg = N == 16 ? 0 : h;
            bl[nt][reg] = __byte_perm(r[2 * h], r[2 * h + 1], 0x6420);
            bh[nt][reg] = __byte_perm(r[2 * h], r[2 * h + 1], 0x7531);
        }
    }
    const int shift2 = 20 - bd;
    const int add2 = 1 << (shift2 - 1);
#pragma unroll 1
    for (int mt = 0; mt < MT; ++mt) {
        uint32_t tmp[NT][2];  // two int16 per word: columns 2t, 2t + 1 of rows g and g + 8
        uint32_t a[4];
#pragma unroll
        for (int i = 0; i < (N == 32 ? 4 : 2); ++i)
            a[i] = frags[((N == 32 ? kFragS1A32 + mt * 4 : kFragS1A16) + i) * 32 + lane];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            int dh[4] = {0, 0, 0, 0}, dl[4] = {0, 0, 0, 0};
            if constexpr (N == 32) {
                mma32(dh, a, bh[nt][0], bh[nt][1], false, false);
                mma32(dl, a, bl[nt][0], bl[nt][1], false, true);
            } else {
                mma16(dh, a[0], a[1], bh[nt][0], false, false);
                mma16(dl, a[0], a[1], bl[nt][0], false, true);
            }
            int v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = clamp3i((dh[e] * 256 + dl[e] + 64) >> 7, -32768, 32767);
            tmp[nt][0] = __byte_perm((uint32_t)v[0], (uint32_t)v[1], 0x5410);
            tmp[nt][1] = __byte_perm((uint32_t)v[2], (uint32_t)v[3], 0x5410);
        }
        // ---- stage 2: out[r][m] = (sum_k tmp[r][k] T[k][m] + add2) >> shift2 ----
        uint32_t ah[4], al[4];
#pragma unroll
        for (int half = 0; half < N / 16; ++half)
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
                const uint32_t p = tmp[2 * half][rr], q = tmp[2 * half + 1][rr];
                al[2 * half + rr] = __byte_perm(p, q, 0x6420);
                ah[2 * half + rr] = __byte_perm(p, q, 0x7531);
            }
        int out[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            int dh[4] = {0, 0, 0, 0}, dl[4] = {0, 0, 0, 0};
            if constexpr (N == 32) {
                const uint32_t b0 = frags[(kFragS2B32 + nt * 2 + 0) * 32 + lane], b1 = frags[(kFragS2B32 + nt * 2 + 1) * 32 + lane];
                mma32(dh, ah, b0, b1, false, false);
                mma32(dl, al, b0, b1, true, false);
            } else {
                const uint32_t b0 = frags[(kFragS2B16 + nt) * 32 + lane];
                mma16(dh, ah[0], ah[1], b0, false, false);
                mma16(dl, al[0], al[1], b0, true, false);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) out[nt][e] = (dh[e] * 256 + dl[e] + add2) >> shift2;
        }
        emit(mt, out);
    }
}

// ===========================================================================
// k_residual
// ===========================================================================
constexpr int kResWarps = 8;

// Residual of one coded TB by one warp (transform.rs:489-858, decode.rs
// :4754-4903 luma, :5313-5417 chroma).  `emit(r, m, v)` receives every
// residual sample (row r, column m) in the reference's storage semantics.
// `allow16` false keeps 8-bit residuals in i32 storage (the reference's
// path for chroma TBs with cross-component prediction, decode.rs:5313-5316).
template <int kIdct, typename Emit>
__device__ void tb_residual_warp(const DevPic& P, const hpvcd_tu& t, const int16_t* dct, int16_t* buf,
                                 int16_t* tmp, int lane, Emit emit, bool allow16 = true) {
    const int n = 1 << t.log2n;
    const bool luma = t.comp == 0;
    const int bd = luma ? P.bd : P.bd_c;
    const bool i16s = bd <= 8 && allow16;
    // levels: int16, or int8 when the host narrowed the picture's pool
    const bool c8 = (P.flags & HPVCD_PIC_COEFF8) != 0;
    const int16_t* lv16 = P.coeffs + t.coeff_off;
    const int8_t* lv8 = (const int8_t*)P.coeffs + t.coeff_off;
    auto lv = [&](int i) -> int { return c8 ? (int)lv8[i] : (int)lv16[i]; };
    const uint32_t rext = t.flags & (HPVCD_TU_ROTATE | HPVCD_TU_RDPCM_H | HPVCD_TU_RDPCM_V);
    // decode.rs:4754-4757 / :4830-4834: residual = levels (transquant bypass);
    // an I_PCM record's levels are its samples (decode.rs:2768-2839)
    if ((t.flags & (HPVCD_TU_TQB | HPVCD_TU_PCM)) && !rext) {
        for (int i = lane; i < n * n; i += 32) emit(i / n, i % n, (int)lv(i));
        return;
    }
    int qpp;
    if (luma) {
        qpp = qp_prime(t.qp_y, bd);
    } else {
        const int pps_off = t.comp == 1 ? P.pps_cb_qp_offset : P.pps_cr_qp_offset;
        qpp = qp_prime(qpc_map(t.qp_y + pps_off + t.cqp_off, P.idc, bd), bd);
    }
    // transform.rs:701-725 dequant_params (non-extended precision: range 15)
    const int bd_shift = bd + t.log2n + 10 - 15;
    const int qs = clamp3i(qpp, 0, 51 + 6 * (bd - 8));
    const long long base = (long long)c_dequant_scale[qs % 6] * (1ll << (qs / 6));
    const long long add = 1ll << (bd_shift - 1);
    // Scaling lists (decode.rs:5874-5899, transform.rs:668-683): the factor
    // of coefficient (r, c) is base * m(r, c) instead of base * 16; 4x4
    // lists index the 4x4 raster, larger TBs the 8x8 list upsampled, with
    // the DC entry for 16x16 and 32x32.  Transform-skip TBs above 4x4 stay
    // flat.
    const uint8_t* sm = nullptr;
    int sdc = 16;
    if (P.scaling && (!(t.flags & HPVCD_TU_TSKIP) || n == 4)) {
        const int size_id = t.log2n - 2;
        const int matrix_id = min((int)t.comp, 2) + ((t.flags & HPVCD_TU_INTRA) ? 0 : 3);
        sm = P.scaling->m[size_id][matrix_id];
        sdc = P.scaling->dc[size_id][matrix_id];
    }
    const int down = t.log2n > 3 ? t.log2n - 3 : 0;
    auto factor_at = [&](int r, int c) -> long long {
        if (!sm) return base * 16;
        if (n == 4) return base * sm[r * 4 + c];
        if (n >= 16 && r == 0 && c == 0) return base * sdc;
        return base * sm[(r >> down) * 8 + (c >> down)];
    };
    if (rext && (t.flags & (HPVCD_TU_TSKIP | HPVCD_TU_TQB))) {
        // RExt residual modification (decode.rs:8418-8446): the TS / TQB
        // residual goes to int32 scratch (rotated: sample i from n*n-1-i),
        // then one lane per column (vertical RDPCM) or row (horizontal)
        // accumulates it.  At 8 bits the reference adds in wrapping i16;
        // the int32 sums wrapped once at the end are the same values.
        int32_t* r32 = reinterpret_cast<int32_t*>(buf);  // buf + tmp: 32 * kScr int32
        const int tr_shift = 15 - bd - t.log2n;
        const int tr_add = tr_shift > 0 ? 1 << (tr_shift - 1) : 0;
        const bool rot = (rext & HPVCD_TU_ROTATE) != 0;
        for (int i = lane; i < n * n; i += 32) {
            int r;
            if (t.flags & HPVCD_TU_TQB) {
                r = lv(i);
            } else {
                long long v = ((long long)lv(i) * factor_at(i / n, i % n) + add) >> bd_shift;
                v = v < -32768 ? -32768 : (v > 32767 ? 32767 : v);
                r = tr_shift >= 0 ? ((int)v + tr_add) >> tr_shift : (int)((unsigned)v << (-tr_shift));
            }
            r32[rot ? n * n - 1 - i : i] = r;
        }
        __syncwarp();
        if (lane < n) {
            if (rext & HPVCD_TU_RDPCM_V) {
                int acc = 0;
                for (int y = 0; y < n; ++y) r32[y * n + lane] = acc += r32[y * n + lane];
            } else if (rext & HPVCD_TU_RDPCM_H) {
                int acc = 0;
                for (int x = 0; x < n; ++x) r32[lane * n + x] = acc += r32[lane * n + x];
            }
        }
        __syncwarp();
        for (int i = lane; i < n * n; i += 32) {
            const int r = r32[i];
            emit(i / n, i % n, i16s ? (int)(int16_t)r : r);
        }
        __syncwarp();
        return;
    }
    if (t.flags & HPVCD_TU_TSKIP) {  // transform.rs:728-792
        const int tr_shift = 15 - bd - t.log2n;
        const int tr_add = tr_shift > 0 ? 1 << (tr_shift - 1) : 0;
        for (int i = lane; i < n * n; i += 32) {
            long long v = ((long long)lv(i) * factor_at(i / n, i % n) + add) >> bd_shift;
            v = v < -32768 ? -32768 : (v > 32767 ? 32767 : v);
            const int r = tr_shift >= 0 ? ((int)v + tr_add) >> tr_shift : (int)((unsigned)v << (-tr_shift));
            emit(i / n, i % n, i16s ? (int)(int16_t)r : r);
        }
        return;
    }
    const int nx = (t.nx == 0 || t.nx > n) ? n : t.nx;
    if (n == 4) {
        // 4x4 in registers: lane l < 16 holds coefficient (l / 4, l % 4); both
        // stages gather their four inputs by shuffles.  The same integer sums
        // as the shared-memory path, clipped after the complete sum.
        const bool dst = luma && (t.flags & HPVCD_TU_INTRA);
        const int l = lane & 15, r = l >> 2, c = l & 3;
        int d = 0;
        if (lane < 16 && c < nx) {
            const long long v = ((long long)lv(l) * factor_at(r, c) + add) >> bd_shift;
            d = (int)(v < -32768 ? -32768 : (v > 32767 ? 32767 : v));
        }
        // basis entry T[k][m] of the 4-point DCT (rows 64 / 83,36 / 64 / 36,83
        // with the H.265 signs) or of the DST
        auto basis = [dst](int k, int m) -> int {
            if (dst) return c_dst4[k][m];
            switch (k) {  // dct_c(4, k, m) without a lookup table
                case 0: return 64;
                case 1: return m == 0 ? 83 : (m == 1 ? 36 : (m == 2 ? -36 : -83));
                case 2: return (m == 0 || m == 3) ? 64 : -64;
                default: return m == 0 ? 36 : (m == 1 ? -83 : (m == 2 ? 83 : -36));
            }
        };
        // stage 1: tmp[r][c] = clip((sum_k T[k][r] d[k][c] + 64) >> 7)
        int acc = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) acc += basis(k, r) * __shfl_sync(0xffffffffu, d, k * 4 + c);
        const int tmp = clamp3i((acc + 64) >> 7, -32768, 32767);
        // stage 2: out[r][c] = (sum_k T[k][c] tmp[r][k] + add2) >> shift2
        const int shift2 = 20 - bd;
        int acc2 = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) acc2 += basis(k, c) * __shfl_sync(0xffffffffu, tmp, r * 4 + k);
        const int v = (acc2 + (1 << (shift2 - 1))) >> shift2;
        if (lane < 16) emit(r, c, i16s ? (int)(int16_t)v : v);
        __syncwarp();
        return;
    }
    // dequantise into buf; columns >= nx are zero (transform.rs:510-511);
    // track the last non-zero row so stage 1 skips all-zero rows.
    int my_rows = 0;
    for (int i = lane; i < n * n; i += 32) {
        const int r = i / n, c = i % n;
        int v = 0;
        if (c < nx) {
            const long long d = ((long long)lv(i) * factor_at(r, c) + add) >> bd_shift;
            v = (int)(d < -32768 ? -32768 : (d > 32767 ? 32767 : d));
        }
        buf[r * kScr + c] = (int16_t)v;
        if (v) my_rows = r + 1;
    }
    int rows = my_rows;
#pragma unroll
    for (int o = 16; o; o >>= 1) rows = max(rows, __shfl_xor_sync(0xffffffffu, rows, o));
    __syncwarp();
    const bool dst = luma && n == 4 && (t.flags & HPVCD_TU_INTRA);
    if (kIdct == kIdctButterfly && n >= 16) {
        // stage 1, lane = column: rows >= `rows` are zero
        auto st1 = [](int acc) { return clamp3i((acc + 64) >> 7, -32768, 32767); };
        // stage 2, lane = row: columns >= nx are zero.  The output is kept
        // as int16 in buf: wrapped at 8 bits (the reference's i16 storage),
        // saturated above 8 bits (exact: a saturated residual clips a
        // sample to the same bound as the full value).
        const int shift2 = 20 - bd;
        const int add2 = 1 << (shift2 - 1);
        auto st2 = [=](int acc) {
            const int v = (acc + add2) >> shift2;
            return i16s ? (int)(int16_t)v : sat16(v);
        };
        if (n == 16) {
            bf_stage_k<16>(rows, buf, 1, kScr, tmp, 1, kScr, lane, st1);
            __syncwarp();
            bf_stage_k<16>(nx, tmp, kScr, 1, buf, kScr, 1, lane, st2);
        } else {
            bf_stage_k<32>(rows, buf, 1, kScr, tmp, 1, kScr, lane, st1);
            __syncwarp();
            bf_stage_k<32>(nx, tmp, kScr, 1, buf, kScr, 1, lane, st2);
        }
        __syncwarp();
        for (int i = lane; i < n * n; i += 32) {
            const int r = i / n, m = i % n;
            emit(r, m, (int)buf[r * kScr + m]);
        }
        __syncwarp();
        return;
    }
    const int step = 32 / n;
    // stage 1 (columns): tmp[m][c] = clip((sum_k T[k][m] * buf[k][c] + 64) >> 7)
    for (int i = lane; i < n * n; i += 32) {
        const int m = i / n, c = i % n;
        int acc = 0;
        if (dst) {
#pragma unroll
            for (int k = 0; k < 4; ++k) acc += c_dst4[k][m] * buf[k * kScr + c];
        } else {
            for (int k = 0; k < rows; ++k) acc += dct[(k * step) * 32 + m] * buf[k * kScr + c];
        }
        tmp[m * kScr + c] = (int16_t)clamp3i((acc + 64) >> 7, -32768, 32767);
    }
    __syncwarp();
    // stage 2 (rows): out[r][m] = (sum_k T[k][m] * tmp[r][k] + add2) >> shift2
    const int shift2 = 20 - bd;
    const int add2 = 1 << (shift2 - 1);
    const int kmax = dst ? 4 : nx;
    for (int i = lane; i < n * n; i += 32) {
        const int r = i / n, m = i % n;
        int acc = 0;
        if (dst) {
#pragma unroll
            for (int k = 0; k < 4; ++k) acc += c_dst4[k][m] * tmp[r * kScr + k];
        } else {
            for (int k = 0; k < kmax; ++k) acc += dct[(k * step) * 32 + m] * tmp[r * kScr + k];
        }
        const int v = (acc + add2) >> shift2;
        emit(r, m, i16s ? (int)(int16_t)v : v);
    }
    __syncwarp();
}

// Dequantisation scale m_levelScale[qs % 6] (transform.rs:701-725) without a
// table: lanes of one warp index it differently, which a constant-bank read
// would serialise.
__device__ __forceinline__ int level_scale(int r) {
    return r == 0 ? 40 : (r == 1 ? 45 : (r == 2 ? 51 : (r == 3 ? 57 : (r == 4 ? 64 : 72))));
}

// Dequantisation of one TB in 32-bit arithmetic (transform.rs:764-858):
// clip((l * (s << q) * m + 2^(b - 1)) >> b) to int16 with s = levelScale, q =
// qP / 6, m the scaling factor (16 when flat) and b = bd + log2n - 5.  The
// common factor 2^min(q, b) cancels exactly: with b > q the result is (l s m
// + 2^(b - q - 1)) >> (b - q), else (l s m) << (q - b).  |l s m| <= 32768 *
// 72 * 255 < 2^30; before a left shift the product is clamped to +-32768,
// which the final clip cannot tell from the full value.
struct Dequant {
    int s, lim, left, right, rnd;
    __device__ __forceinline__ Dequant(const DevPic& P, const hpvcd_tu& t, int log2n) {
        const int c = t.comp, bd = c ? P.bd_c : P.bd;
        int qpp;
        if (c == 0) {
            qpp = qp_prime(t.qp_y, bd);
        } else {
            const int pps_off = c == 1 ? P.pps_cb_qp_offset : P.pps_cr_qp_offset;
            qpp = qp_prime(qpc_map(t.qp_y + pps_off + t.cqp_off, P.idc, bd), bd);
        }
        const int qs = clamp3i(qpp, 0, 51 + 6 * (bd - 8));
        const int q = qs / 6, b = bd + log2n - 5;
        s = level_scale(qs - 6 * q);
        left = max(q - b, 0);
        right = max(b - q, 0);
        rnd = right ? 1 << (right - 1) : 0;
        lim = left ? 32768 : 0x7fffffff;
    }
    __device__ __forceinline__ int operator()(int l, int m) const {
        const int x = min(max(l * (s * m), -lim), lim);
        return clamp3i(((x << left) + rnd) >> right, -32768, 32767);
    }
};

// Scaling list of a TB (transform.rs:668-683), NULL when flat.
__device__ __forceinline__ const uint8_t* scaling_of(const DevPic& P, const hpvcd_tu& t, int log2n) {
    if (!P.scaling) return nullptr;
    return P.scaling->m[log2n - 2][min((int)t.comp, 2) + ((t.flags & HPVCD_TU_INTRA) ? 0 : 3)];
}

// One 4-point inverse transform, DST-VII (kDst) or DCT, with the basis as
// immediates: o[m] = sum_k T[k][m] * in[k] (transform.rs:535-603 for the
// DST, :406-533 for the DCT; the H.265 matrices).
template <bool kDst>
__device__ __forceinline__ void inv4(int i0, int i1, int i2, int i3, int& o0, int& o1, int& o2, int& o3) {
    if (kDst) {
        o0 = 29 * i0 + 74 * i1 + 84 * i2 + 55 * i3;
        o1 = 55 * i0 + 74 * i1 - 29 * i2 - 84 * i3;
        o2 = 74 * i0 - 74 * i2 + 74 * i3;
        o3 = 84 * i0 - 74 * i1 + 55 * i2 - 29 * i3;
    } else {
        const int e0 = 64 * (i0 + i2), e1 = 64 * (i0 - i2);
        const int q0 = 83 * i1 + 36 * i3, q1 = 36 * i1 - 83 * i3;
        o0 = e0 + q0;
        o1 = e1 + q1;
        o2 = e1 - q1;
        o3 = e0 - q0;
    }
}

// Both stages of a 4x4 inverse transform in one thread's registers: d is
// the dequantised block (row k, column c at d[4k + c]); on return d holds
// the residual before the storage wrap.  Stage 1 (columns) clips
// (sum + 64) >> 7 to int16, stage 2 (rows) adds 2^(shift2 - 1) and shifts
// by shift2, the same sums as the warp path of tb_residual_warp.
template <bool kDst>
__device__ __forceinline__ void idct4_thread(int (&d)[16], int shift2) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        int o0, o1, o2, o3;
        inv4<kDst>(d[c], d[4 + c], d[8 + c], d[12 + c], o0, o1, o2, o3);
        d[c] = clamp3i((o0 + 64) >> 7, -32768, 32767);
        d[4 + c] = clamp3i((o1 + 64) >> 7, -32768, 32767);
        d[8 + c] = clamp3i((o2 + 64) >> 7, -32768, 32767);
        d[12 + c] = clamp3i((o3 + 64) >> 7, -32768, 32767);
    }
    const int add2 = 1 << (shift2 - 1);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        int o0, o1, o2, o3;
        inv4<kDst>(d[4 * r], d[4 * r + 1], d[4 * r + 2], d[4 * r + 3], o0, o1, o2, o3);
        d[4 * r] = (o0 + add2) >> shift2;
        d[4 * r + 1] = (o1 + add2) >> shift2;
        d[4 * r + 2] = (o2 + add2) >> shift2;
        d[4 * r + 3] = (o3 + add2) >> shift2;
    }
}

// Four horizontally adjacent samples of a plane at an address aligned to
// four samples.
__device__ __forceinline__ void ld_row4(const void* plane, int bps, size_t idx, int (&v)[4]) {
    if (bps == 1) {
        const uint32_t w = *(const uint32_t*)((const uint8_t*)plane + idx);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = (w >> (8 * i)) & 0xff;
    } else {
        const uint2 w = *(const uint2*)((const uint16_t*)plane + idx);
        v[0] = w.x & 0xffff; v[1] = w.x >> 16; v[2] = w.y & 0xffff; v[3] = w.y >> 16;
    }
}
__device__ __forceinline__ void st_row4(void* plane, int bps, size_t idx, const int (&v)[4]) {
    if (bps == 1)
        *(uint32_t*)((uint8_t*)plane + idx) =
            (uint32_t)v[0] | ((uint32_t)v[1] << 8) | ((uint32_t)v[2] << 16) | ((uint32_t)v[3] << 24);
    else
        *(uint2*)((uint16_t*)plane + idx) =
            make_uint2((uint32_t)v[0] | ((uint32_t)v[1] << 16), (uint32_t)v[2] | ((uint32_t)v[3] << 16));
}

// A plain coded TB of size 2^log2n: valid, with a transform (no transform
// skip, bypass, I_PCM or RExt residual tool) and a residual that is not
// k_ccp's.
__device__ __forceinline__ bool tb_plain(const DevPic& P, const hpvcd_tu& t) {
    constexpr uint32_t kOther = HPVCD_TU_TSKIP | HPVCD_TU_TQB | HPVCD_TU_ROTATE | HPVCD_TU_RDPCM_H |
                                HPVCD_TU_RDPCM_V | HPVCD_TU_PCM;
    if (!(t.flags & HPVCD_TU_CBF) || (t.flags & kOther) || t.log2n < 2 || t.log2n > 5) return false;
    if ((P.flags & HPVCD_PIC_CROSS_COMPONENT) && t.comp && t.res_scale) return false;
    const int ncomp = P.idc ? 3 : 1;
    if (t.comp >= ncomp) return false;
    const int pw = t.comp ? P.cw : P.w, ph = t.comp ? P.ch : P.h;
    return (int)t.x < pw && (int)t.y < ph && (uint64_t)t.coeff_off + (1u << (2 * t.log2n)) <= P.n_coeffs;
}

// Whether a picture's prediction is already in its planes: its TBs are added
// there.  Every other TB leaves its residual in the int16 residual plane,
// which motion compensation (inter TBs) or k_recon (intra TBs) adds.
__device__ __forceinline__ bool in_plane_of(const DevPic& P) { return (P.flags & HPVCD_PIC_PRED_IN_PLANE) != 0; }

// Residual of one plain 4x4 TB by one thread (the 4x4 case of
// tb_residual_warp), stored where the warp path stores it: added to the plane
// and clipped where the prediction is in it, else into the int16 residual
// plane.
__device__ void tb4_thread(const DevPic& P, const hpvcd_tu& t) {
    const int c = t.comp;
    const int bd = c ? P.bd_c : P.bd;
    const int pw = c ? P.cw : P.w, ph = c ? P.ch : P.h;
    const int x0 = t.x, y0 = t.y;
    const bool in_plane = in_plane_of(P);
    // the plane's rows are read up front, beside the levels
    int pv[4][4];
    void* pl = P.rec[c];
    const size_t p0 = (size_t)y0 * pw + x0;
    const bool pvec = in_plane && x0 + 4 <= pw && y0 + 4 <= ph && (p0 & 3) == 0 && (pw & 3) == 0;
    if (pvec) {
#pragma unroll
        for (int r = 0; r < 4; ++r) ld_row4(pl, P.bps, p0 + (size_t)r * pw, pv[r]);
    }
    int d[16];
    const bool c8 = (P.flags & HPVCD_PIC_COEFF8) != 0;
    if (c8) {
        const int8_t* lv = (const int8_t*)P.coeffs + t.coeff_off;
        if (((uintptr_t)lv & 15) == 0) {
            const int4 w = *(const int4*)lv;
            const int ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int i = 0; i < 16; ++i) d[i] = (int)(int8_t)(ws[i >> 2] >> (8 * (i & 3)));
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) d[i] = lv[i];
        }
    } else {
        const int16_t* lv = P.coeffs + t.coeff_off;
        if (((uintptr_t)lv & 15) == 0) {
            const int4 w0 = *(const int4*)lv, w1 = *(const int4*)(lv + 8);
            const int ws[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
            for (int i = 0; i < 16; ++i) d[i] = (int)(int16_t)(ws[i >> 1] >> (16 * (i & 1)));
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) d[i] = lv[i];
        }
    }
    const Dequant dq(P, t, 2);
    const int nx = (t.nx == 0 || t.nx > 4) ? 4 : t.nx;
    uint32_t m4[4] = {0x10101010u, 0x10101010u, 0x10101010u, 0x10101010u};  // factors of row r
    if (const uint8_t* sm = scaling_of(P, t, 2)) {
#pragma unroll 1
        for (int r = 0; r < 4; ++r) {
            const uint32_t w = (uint32_t)sm[4 * r] | ((uint32_t)sm[4 * r + 1] << 8) | ((uint32_t)sm[4 * r + 2] << 16) |
                               ((uint32_t)sm[4 * r + 3] << 24);
            if (r == 0) m4[0] = w;
            if (r == 1) m4[1] = w;
            if (r == 2) m4[2] = w;
            if (r == 3) m4[3] = w;
        }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) d[i] = (i & 3) < nx ? dq(d[i], (int)((m4[i >> 2] >> (8 * (i & 3))) & 0xffu)) : 0;
    const int shift2 = 20 - bd;
    if (c == 0 && (t.flags & HPVCD_TU_INTRA))
        idct4_thread<true>(d, shift2);
    else
        idct4_thread<false>(d, shift2);
    if (bd <= 8) {  // the reference's int16 storage
#pragma unroll
        for (int i = 0; i < 16; ++i) d[i] = (int)(int16_t)d[i];
    }
    if (in_plane) {  // reconstruct.rs:214-251: add and clip into the plane
        const int mx = (1 << bd) - 1;
        if (pvec) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
#pragma unroll
                for (int m = 0; m < 4; ++m) pv[r][m] = clamp3i(pv[r][m] + d[4 * r + m], 0, mx);
                st_row4(pl, P.bps, p0 + (size_t)r * pw, pv[r]);
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int x = x0 + (i & 3), y = y0 + (i >> 2);
                if (x < pw && y < ph) {
                    const size_t idx = (size_t)y * pw + x;
                    store_sample(pl, P.bps, idx, clamp3i(load_sample(pl, P.bps, idx) + d[i], 0, mx));
                }
            }
        }
    } else {  // the int16 residual plane k_recon adds to its prediction
        int16_t* rp = P.res[c];
        const int rs = P.res_stride[c];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int y = y0 + r;
            if (y >= ph) break;
            int16_t* row = rp + (size_t)y * rs + x0;
            int16_t v4[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) v4[m] = res_store(d[4 * r + m], (1 << bd) - 1);
            if (x0 + 4 <= pw && ((uintptr_t)row & 7) == 0) {
                *(uint2*)row = make_uint2((uint32_t)(uint16_t)v4[0] | ((uint32_t)(uint16_t)v4[1] << 16),
                                          (uint32_t)(uint16_t)v4[2] | ((uint32_t)(uint16_t)v4[3] << 16));
            } else {
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    if (x0 + m < pw) row[m] = v4[m];
            }
        }
    }
}

// 8-point inverse DCT with the basis as immediates, even-odd form:
// o[m] = sum_k T8[k][m] * in[k] (transform.rs:406-533, the H.265 matrix).
__device__ __forceinline__ void inv8(const int (&in)[8], int (&o)[8]) {
    const int ee0 = 64 * (in[0] + in[4]), ee1 = 64 * (in[0] - in[4]);
    const int eo0 = 83 * in[2] + 36 * in[6], eo1 = 36 * in[2] - 83 * in[6];
    const int e0 = ee0 + eo0, e3 = ee0 - eo0, e1 = ee1 + eo1, e2 = ee1 - eo1;
    const int o0 = 89 * in[1] + 75 * in[3] + 50 * in[5] + 18 * in[7];
    const int o1 = 75 * in[1] - 18 * in[3] - 89 * in[5] - 50 * in[7];
    const int o2 = 50 * in[1] - 89 * in[3] + 18 * in[5] + 75 * in[7];
    const int o3 = 18 * in[1] - 50 * in[3] + 75 * in[5] - 89 * in[7];
    o[0] = e0 + o0; o[7] = e0 - o0;
    o[1] = e1 + o1; o[6] = e1 - o1;
    o[2] = e2 + o2; o[5] = e2 - o2;
    o[3] = e3 + o3; o[4] = e3 - o3;
}

// Stage 1 of a plain 8x8 TB by lane q (0..7) of its group of eight: column q
// dequantised (the 8x8 case of tb_residual_warp, columns >= nx zero) and
// inverse transformed, (sum + 64) >> 7 clipped to int16 into the group's
// scratch S[m * 9 + q].
__device__ __forceinline__ void tb8_cols(const DevPic& P, const hpvcd_tu& t, int q, int16_t* S) {
    const bool c8 = (P.flags & HPVCD_PIC_COEFF8) != 0;
    int in[8];
    if (c8) {
        const int8_t* lv = (const int8_t*)P.coeffs + t.coeff_off + q;
#pragma unroll
        for (int r = 0; r < 8; ++r) in[r] = lv[r * 8];
    } else {
        const int16_t* lv = P.coeffs + t.coeff_off + q;
#pragma unroll
        for (int r = 0; r < 8; ++r) in[r] = lv[r * 8];
    }
    const Dequant dq(P, t, 3);
    const uint8_t* sm = scaling_of(P, t, 3);
    const int nx = (t.nx == 0 || t.nx > 8) ? 8 : t.nx;
#pragma unroll
    for (int r = 0; r < 8; ++r) in[r] = q < nx ? dq(in[r], sm ? sm[r * 8 + q] : 16) : 0;
    int o[8];
    inv8(in, o);
#pragma unroll
    for (int m = 0; m < 8; ++m) S[m * 9 + q] = (int16_t)clamp3i((o[m] + 64) >> 7, -32768, 32767);
}

// Stage 2 of the same TB by lane q: row q of the stage-1 result, inverse
// transformed, + 2^(shift2 - 1) >> shift2, stored as tb4_thread stores
// (added to the plane, or into the int16 residual plane).
__device__ __forceinline__ void tb8_rows(const DevPic& P, const hpvcd_tu& t, int q, const int16_t* S) {
    const int c = t.comp;
    const int bd = c ? P.bd_c : P.bd;
    const int pw = c ? P.cw : P.w, ph = c ? P.ch : P.h;
    const int x0 = t.x, y = t.y + q;
    if (y >= ph) return;
    const bool in_plane = in_plane_of(P);
    void* pl = P.rec[c];
    const size_t p0 = (size_t)y * pw + x0;
    const bool pvec = in_plane && x0 + 8 <= pw && (p0 & 3) == 0;
    int pv[2][4];
    if (pvec) {
        ld_row4(pl, P.bps, p0, pv[0]);
        ld_row4(pl, P.bps, p0 + 4, pv[1]);
    }
    const int shift2 = 20 - bd, add2 = 1 << (shift2 - 1);
    const bool i16s = bd <= 8;
    int in[8], o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) in[k] = S[q * 9 + k];
    inv8(in, o);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        const int v = (o[m] + add2) >> shift2;
        o[m] = i16s ? (int)(int16_t)v : v;
    }
    if (in_plane) {  // reconstruct.rs:214-251: add and clip into the plane
        const int mx = (1 << bd) - 1;
        if (pvec) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int m = 0; m < 4; ++m) pv[h][m] = clamp3i(pv[h][m] + o[4 * h + m], 0, mx);
                st_row4(pl, P.bps, p0 + 4 * h, pv[h]);
            }
        } else {
#pragma unroll
            for (int m = 0; m < 8; ++m)
                if (x0 + m < pw)
                    store_sample(pl, P.bps, p0 + m, clamp3i(load_sample(pl, P.bps, p0 + m) + o[m], 0, mx));
        }
    } else {
        int16_t* row = P.res[c] + (size_t)y * P.res_stride[c] + x0;
        if (x0 + 8 <= pw && ((uintptr_t)row & 15) == 0) {
            uint32_t w[4];
#pragma unroll
            for (int h = 0; h < 4; ++h)
                w[h] = (uint32_t)(uint16_t)res_store(o[2 * h], (1 << bd) - 1) |
                       ((uint32_t)(uint16_t)res_store(o[2 * h + 1], (1 << bd) - 1) << 16);
            *(uint4*)row = make_uint4(w[0], w[1], w[2], w[3]);
        } else {
#pragma unroll
            for (int m = 0; m < 8; ++m)
                if (x0 + m < pw) row[m] = res_store(o[m], (1 << bd) - 1);
        }
    }
}

// Residual of one plain 16x16 or 32x32 TB by one warp on the integer tensor
// pipe: eight levels per lane and load (all loads in flight together),
// dequantised into shared memory, both stages in registers (idct_tensor),
// two adjacent samples per store.  x0 is even (the caller's class test).
template <int N>
__device__ __forceinline__ void tb_tensor(const DevPic& P, const hpvcd_tu& t, int16_t* buf, const uint32_t* frags,
                                          int lane) {
    constexpr int LOG2N = N == 32 ? 5 : 4, STR = tensor_stride(N), PASS = N * N / 256;
    const int c = t.comp;
    const int bd = c ? P.bd_c : P.bd;
    const bool c8 = (P.flags & HPVCD_PIC_COEFF8) != 0;
    uint4 raw[PASS];  // eight levels: four words of two int16, or two words of four int8
    if (c8) {
        const int8_t* lv = (const int8_t*)P.coeffs + t.coeff_off;
        const bool al = ((uintptr_t)lv & 7) == 0;
#pragma unroll
        for (int p = 0; p < PASS; ++p) {
            const int8_t* q = lv + (p * 32 + lane) * 8;
            uint2 w;
            if (al) {
                w = *(const uint2*)q;
            } else {
                memcpy(&w, q, 8);  // byte loads
            }
            raw[p] = make_uint4(w.x, w.y, 0u, 0u);
        }
    } else {
        const int16_t* lv = P.coeffs + t.coeff_off;
        const bool al = ((uintptr_t)lv & 15) == 0;
#pragma unroll
        for (int p = 0; p < PASS; ++p) {
            const int16_t* q = lv + (p * 32 + lane) * 8;
            if (al) {
                raw[p] = *(const uint4*)q;
            } else {
                uint32_t w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    w[i] = (uint32_t)(uint16_t)q[2 * i] | ((uint32_t)(uint16_t)q[2 * i + 1] << 16);
                raw[p] = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
    }
    const Dequant dq(P, t, LOG2N);
    const uint8_t* sm = scaling_of(P, t, LOG2N);
    const int nx = (t.nx == 0 || t.nx > N) ? N : t.nx;
    // factors of the lane's eight columns: the 8x8 list upsampled (its row
    // changes with the pass), a byte each, two words
    auto level = [&](const uint4& q, int j) {
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
        return c8 ? (int)(int8_t)(w[j >> 2] >> (8 * (j & 3))) : (int)(int16_t)(w[j >> 1] >> (16 * (j & 1)));
    };
    const int col = (lane * 8) & (N - 1);
    if (!sm) {
#pragma unroll
        for (int p = 0; p < PASS; ++p) {
            const int r = ((p * 32 + lane) * 8) >> LOG2N;
            uint32_t o[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int d0 = col + 2 * h < nx ? dq(level(raw[p], 2 * h), 16) : 0;
                const int d1 = col + 2 * h + 1 < nx ? dq(level(raw[p], 2 * h + 1), 16) : 0;
                o[h] = __byte_perm((uint32_t)d0, (uint32_t)d1, 0x5410);
            }
            *(uint4*)(buf + r * STR + col) = make_uint4(o[0], o[1], o[2], o[3]);
        }
    } else {
        const int dc = P.scaling->dc[LOG2N - 2][min(c, 2) + ((t.flags & HPVCD_TU_INTRA) ? 0 : 3)];
#pragma unroll
        for (int p = 0; p < PASS; ++p) *(uint4*)(buf + (((p * 32 + lane) * 8) >> LOG2N) * STR + col) = raw[p];
        __syncwarp();
#pragma unroll 1
        for (int p = 0; p < PASS; ++p) {
            const int i0 = (p * 32 + lane) * 8, r = i0 >> LOG2N;
            int16_t* q = buf + r * STR + col;
            const uint4 w = *(const uint4*)q;  // this lane's levels
#pragma unroll 1
            for (int j = 0; j < 8; ++j) {
                const uint32_t pair = c8 ? (j < 4 ? w.x : w.y) : (j < 2 ? w.x : (j < 4 ? w.y : (j < 6 ? w.z : w.w)));
                const int l = c8 ? (int)(int8_t)(pair >> (8 * (j & 3))) : (int)(int16_t)(pair >> (16 * (j & 1)));
                const int m = i0 + j == 0 ? dc : sm[(r >> (LOG2N - 3)) * 8 + ((col + j) >> (LOG2N - 3))];
                q[j] = (int16_t)(col + j < nx ? dq(l, m) : 0);
            }
        }
    }
    __syncwarp();
    const int pw = c ? P.cw : P.w, ph = c ? P.ch : P.h;
    const int x0 = t.x, y0 = t.y;
    const int g = lane >> 2, tq = lane & 3;
    const bool in_plane = in_plane_of(P);
    const bool i16s = bd <= 8;
    const int mx = (1 << bd) - 1, bps = P.bps;
    void* pl = P.rec[c];
    int16_t* rp = P.res[c];
    const int rs = P.res_stride[c];
    // plane widths are even, so a pair starting at an even column is inside
    // or outside as a whole
    idct_tensor<N>(buf, frags, bd, lane, [&](int mt, int (&out)[N / 8][4]) {
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            const int y = y0 + mt * 16 + g + 8 * rr;
            if (y >= ph) continue;
            if (in_plane) {  // reconstruct.rs:214-251: add and clip into the plane
                uint32_t pv[N / 8];
                const size_t row = (size_t)y * pw;
#pragma unroll
                for (int nt = 0; nt < N / 8; ++nt) {
                    const int x = x0 + nt * 8 + 2 * tq;
                    pv[nt] = 0u;
                    if (x < pw)
                        pv[nt] = bps == 1 ? (uint32_t) * (const uint16_t*)((const uint8_t*)pl + row + x)
                                          : *(const uint32_t*)((const uint16_t*)pl + row + x);
                }
#pragma unroll
                for (int nt = 0; nt < N / 8; ++nt) {
                    const int x = x0 + nt * 8 + 2 * tq;
                    int v0 = out[nt][2 * rr], v1 = out[nt][2 * rr + 1];
                    if (i16s) v0 = (int)(int16_t)v0, v1 = (int)(int16_t)v1;
                    if (x >= pw) continue;
                    if (bps == 1) {
                        const uint32_t a = (uint32_t)clamp3i((int)(pv[nt] & 0xff) + v0, 0, mx);
                        const uint32_t b = (uint32_t)clamp3i((int)(pv[nt] >> 8) + v1, 0, mx);
                        *(uint16_t*)((uint8_t*)pl + row + x) = (uint16_t)(a | (b << 8));
                    } else {
                        const uint32_t a = (uint32_t)clamp3i((int)(pv[nt] & 0xffff) + v0, 0, mx);
                        const uint32_t b = (uint32_t)clamp3i((int)(pv[nt] >> 16) + v1, 0, mx);
                        *(uint32_t*)((uint16_t*)pl + row + x) = a | (b << 16);
                    }
                }
            } else {
                int16_t* row = rp + (size_t)y * rs + x0;
#pragma unroll
                for (int nt = 0; nt < N / 8; ++nt) {
                    const int x = nt * 8 + 2 * tq;
                    int v0 = out[nt][2 * rr], v1 = out[nt][2 * rr + 1];
                    if (i16s) v0 = (int)(int16_t)v0, v1 = (int)(int16_t)v1;
                    if (x0 + x < pw)
                        *(uint32_t*)(row + x) =
                            (uint32_t)(uint16_t)res_store(v0, mx) | ((uint32_t)(uint16_t)res_store(v1, mx) << 16);
                }
            }
        }
    });
    __syncwarp();
}

// Residual of any other coded TB (transform skip, bypass, I_PCM, RExt tools;
// every 16x16 / 32x32 TB of the matrix and butterfly schedules) by one warp.
template <int kIdct>
__device__ __noinline__ void tb_general(const DevPic& P, const hpvcd_tu& t, const int16_t* dct, int16_t* scr,
                                        uint32_t* dev_err, int lane) {
    if ((P.flags & HPVCD_PIC_CROSS_COMPONENT) && t.comp && t.res_scale) return;  // k_ccp's
    const int c = t.comp;
    const int ncomp = P.idc ? 3 : 1;
    const int n = 1 << t.log2n;
    const int pw = c < 3 && c ? P.cw : P.w, ph = c < 3 && c ? P.ch : P.h;
    if (c >= ncomp || t.log2n < 2 || t.log2n > 5 || (int)t.x >= pw || (int)t.y >= ph ||
        (uint64_t)t.coeff_off + (uint64_t)n * n > P.n_coeffs) {
        if (lane == 0) atomicOr(dev_err, DEV_ERR_BITSTREAM);
        return;
    }
    const int x0 = t.x, y0 = t.y;
    if (in_plane_of(P)) {  // prediction already in the plane: add + clip (reconstruct.rs:214-251)
        void* pl = P.rec[c];
        const int mx = (1 << (c ? P.bd_c : P.bd)) - 1;
        const int keep = (t.flags & HPVCD_TU_PCM) ? 0 : 1;  // I_PCM samples replace the plane's
        tb_residual_warp<kIdct>(P, t, dct, scr, scr + 32 * kScr, lane, [&](int r, int m, int v) {
            const int x = x0 + m, y = y0 + r;
            if (x < pw && y < ph) {
                const size_t idx = (size_t)y * pw + x;
                store_sample(pl, P.bps, idx, clamp3i(keep * load_sample(pl, P.bps, idx) + v, 0, mx));
            }
        });
    } else {
        int16_t* rp = P.res[c];
        const int rs = P.res_stride[c], mx = (1 << (c ? P.bd_c : P.bd)) - 1;
        tb_residual_warp<kIdct>(P, t, dct, scr, scr + 32 * kScr, lane, [&](int r, int m, int v) {
            const int x = x0 + m, y = y0 + r;
            if (x < pw && y < ph) rp[(size_t)y * rs + x] = res_store(v, mx);
        });
    }
    __syncwarp();
}

// Classes of coded records, in the order their warp tasks are taken: the
// longest first, so that the last tasks of a CTA are short.
constexpr int kCls32 = 0, kCls16 = 1, kClsGeneral = 2, kCls8 = 3, kCls4 = 4, kClasses = 5;
constexpr uint32_t kResMaxChunk = 1024;  // records of a CTA step

// One CTA takes `chunk` consecutive records at a time and sorts them by class
// (the picture of the first by one search, of the others by a short walk from
// it); the warps then take tasks off the sorted list: one 32x32, 16x16 or
// general TB, four 8x8 (eight lanes each) or thirty-two 4x4 (one lane each).
// What bounds a launch on a small picture is the latency of its longest chain
// of tasks, so the chunk is chosen by the record count (hpvcd_launch_residual)
// to spread it over all SMs; on a large one the warps wait for instructions
// first (the stall before any other at 256 records a step), and a long sorted
// list keeps the warps of an SM in the same code: up to 1024 records a step
// instead of 256 took the whole call on 24 mixed pictures from 4115 to 3940 us
// and the 1920x1080 sequence from 2480 to 2421, and left the residual-only
// 512x512 picture at 41 (40 before: one phase more).  One warp taking 32
// consecutive records one after another, one sample per lane and step, took
// 150 us on any picture of 512x512 and up (whole call 185 us).
template <int kIdct>
__global__ void __launch_bounds__(kResWarps * 32, 4)
k_residual(const DevPic* __restrict__ pics, const uint32_t* __restrict__ rec_prefix, uint32_t n_pics,
           uint32_t* dev_err, uint32_t chunk) {
    __shared__ __align__(16) BasisTables basis;
    __shared__ __align__(16) int16_t scr[kResWarps][2 * 32 * kScr];  // per warp
    __shared__ uint32_t s_pic[kResMaxChunk];   // picture of a record
    __shared__ uint16_t s_list[kResMaxChunk];  // records by class
    __shared__ uint32_t s_cnt[kClasses], s_next;
    constexpr int kPerThread = kResMaxChunk / (kResWarps * 32);
    static_assert(tensor_stride(32) * 32 <= 2 * 32 * kScr, "the tensor path's block fits the scratch");
    stage_table(&basis, &g_basis, (int)sizeof(basis));
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t first = rec_prefix[0], total = rec_prefix[n_pics];
    for (uint32_t g0 = first + blockIdx.x * chunk; g0 < total; g0 += gridDim.x * chunk) {
        __syncthreads();  // the previous step's lists are done with (and, first, the tables staged)
        if (threadIdx.x < kClasses) s_cnt[threadIdx.x] = 0u;
        if (threadIdx.x == kClasses) s_next = 0u;
        __syncthreads();
        uint32_t pic = 0;
        for (uint32_t hi = n_pics; hi - pic > 1;) {  // the picture of the step's first record (uniform)
            const uint32_t mid = (pic + hi) >> 1;
            if (rec_prefix[mid] <= g0) pic = mid; else hi = mid;
        }
        uint32_t cls[kPerThread], place[kPerThread];  // a record's class and its place there
#pragma unroll
        for (int u = 0; u < kPerThread; ++u) {
            const uint32_t i = u * (kResWarps * 32) + threadIdx.x, gl = g0 + i;
            cls[u] = kClasses;
            if (i >= chunk || gl >= total) continue;
            while (rec_prefix[pic + 1] <= gl) ++pic;
            const DevPic& P = pics[pic];
            const uint4 r4 = *(const uint4*)(P.tus + (gl - rec_prefix[pic]));  // records are 16-byte aligned
            hpvcd_tu t;
            memcpy(&t, &r4, sizeof(t));
            if (!(t.flags & HPVCD_TU_CBF)) continue;
            cls[u] = kClsGeneral;
            if (tb_plain(P, t)) {
                if (t.log2n <= 3)
                    cls[u] = t.log2n == 2 ? kCls4 : kCls8;
                else if (kIdct == kIdctTensor && (t.x & 1) == 0)
                    cls[u] = t.log2n == 4 ? kCls16 : kCls32;
            }
            s_pic[i] = pic;
            place[u] = atomicAdd(&s_cnt[cls[u]], 1u);
        }
        __syncthreads();
        const uint32_t e32 = s_cnt[kCls32], e16 = e32 + s_cnt[kCls16], eg = e16 + s_cnt[kClsGeneral];
        const uint32_t n8 = s_cnt[kCls8], n4 = s_cnt[kCls4];
        const uint32_t e8 = eg + (n8 + 3) / 4, e4 = e8 + (n4 + 31) / 32;
#pragma unroll
        for (int u = 0; u < kPerThread; ++u) {
            if (cls[u] == kClasses) continue;
            place[u] += cls[u] == kCls32 ? 0u : cls[u] == kCls16 ? e32 : cls[u] == kClsGeneral ? e16 : cls[u] == kCls8 ? eg : eg + n8;
            s_list[place[u]] = (uint16_t)(u * (kResWarps * 32) + threadIdx.x);
        }
        __syncthreads();
        // the record at place k of the sorted list, and its picture
        auto record = [&](uint32_t k, hpvcd_tu& t) -> const DevPic& {
            const uint32_t i = s_list[k], pi = s_pic[i];
            const DevPic& P = pics[pi];
            const uint4 r4 = *(const uint4*)(P.tus + (g0 + i - rec_prefix[pi]));
            memcpy(&t, &r4, sizeof(t));
            return P;
        };
        for (;;) {
            uint32_t task = 0;
            if (lane == 0) task = atomicAdd(&s_next, 1u);
            task = __shfl_sync(kAll, task, 0);
            if (task >= e4) break;
            hpvcd_tu t;
            if (task < eg) {
                const DevPic& P = record(task, t);
                if (kIdct == kIdctTensor && task < e32)
                    tb_tensor<32>(P, t, scr[warp], basis.frags, lane);
                else if (kIdct == kIdctTensor && task < e16)
                    tb_tensor<16>(P, t, scr[warp], basis.frags, lane);
                else
                    tb_general<kIdct == kIdctButterfly ? kIdctButterfly : kIdctMatrix>(P, t, basis.dct, scr[warp],
                                                                                       dev_err, lane);
            } else if (task < e8) {
                const uint32_t k = (task - eg) * 4 + (lane >> 3);
                const int q = lane & 7;
                const DevPic& P = record(eg + min(k, n8 - 1), t);
                int16_t* S = scr[warp] + (lane >> 3) * 72;
                if (k < n8) tb8_cols(P, t, q, S);
                __syncwarp();
                if (k < n8) tb8_rows(P, t, q, S);
                __syncwarp();
            } else {
                const uint32_t k = (task - e8) * 32 + lane;
                if (k < n4) {
                    const DevPic& P = record(eg + n8 + k, t);
                    tb4_thread(P, t);
                }
                __syncwarp();
            }
        }
    }
}

// ===========================================================================
// k_ccp -- chroma TBs with cross-component prediction (RExt 4:4:4)
// ===========================================================================
// One warp per chroma TB with res_scale != 0 of a HPVCD_PIC_CROSS_COMPONENT
// picture: it recomputes its TU's luma residual rY (the matrix inverse
// transform, which keeps i32 values above 8 bits), then the chroma residual
// in i32 storage (decode.rs:5286-5426; zero without coded residual,
// :5428-5466), adds (res_scale * ((rY << BitDepthC) >> BitDepthY)) >> 3
// (decode.rs:5488-5504) and writes it where k_residual would.
constexpr int kCcpWarps = 4;

__global__ void __launch_bounds__(kCcpWarps * 32)
k_ccp(const DevPic* __restrict__ pics, const uint32_t* __restrict__ rec_prefix, uint32_t n_pics,
      uint32_t* dev_err) {
    __shared__ __align__(16) int16_t dct[32 * 32];
    __shared__ __align__(16) int16_t scr[kCcpWarps][2][32 * kScr];
    __shared__ int32_t ry_all[kCcpWarps][32 * 32];
    stage_table(dct, g_basis.dct, (int)sizeof(dct));
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t* ry = ry_all[warp];
    const uint32_t total = rec_prefix[n_pics];
    for (uint32_t g = rec_prefix[0] + blockIdx.x * kCcpWarps + warp; g < total; g += gridDim.x * kCcpWarps) {
        uint32_t lo = 0, hi = n_pics;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (rec_prefix[mid] <= g) lo = mid; else hi = mid;
        }
        const DevPic& P = pics[lo];
        if (!(P.flags & HPVCD_PIC_CROSS_COMPONENT)) continue;
        const uint32_t gl = g - rec_prefix[lo];
        const hpvcd_tu t = P.tus[gl];
        if (t.comp == 0 || t.res_scale == 0) continue;
        const int n = 1 << t.log2n;
        bool bad = P.idc != 3 || t.comp > 2 || t.log2n < 2 || t.log2n > 5 || (int)t.x >= P.cw ||
                   (int)t.y >= P.ch ||
                   ((t.flags & HPVCD_TU_CBF) && (uint64_t)t.coeff_off + (uint64_t)n * n > P.n_coeffs);
        // the TU's luma TB: same place and size, among the three records before
        hpvcd_tu lt{};
        bool found = false;
        for (uint32_t k = 1; k <= 3 && k <= gl && !found; ++k) {
            lt = P.tus[gl - k];
            found = lt.comp == 0 && lt.x == t.x && lt.y == t.y && lt.log2n == t.log2n;
        }
        bad = bad || !found || !(lt.flags & HPVCD_TU_CBF) ||
              (uint64_t)lt.coeff_off + (uint64_t)n * n > P.n_coeffs;
        if (bad) {
            if (lane == 0) atomicOr(dev_err, DEV_ERR_BITSTREAM);
            continue;
        }
        tb_residual_warp<kIdctMatrix>(P, lt, dct, scr[warp][0], scr[warp][1], lane,
                                      [&](int r, int m, int v) { ry[r * n + m] = v; });
        __syncwarp();
        const int c = t.comp, x0 = t.x, y0 = t.y, pw = P.cw, ph = P.ch;
        const int bdy = P.bd, bdc = P.bd_c, rs = t.res_scale;
        const bool in_plane = in_plane_of(P);
        const int mx = (1 << bdc) - 1;
        auto out = [&](int r, int m, long long v) {
            const long long sy = ((long long)ry[r * n + m] << bdc) >> bdy;
            v += (rs * sy) >> 3;
            const int vv = (int)(v < INT_MIN ? INT_MIN : (v > INT_MAX ? INT_MAX : v));
            const int x = x0 + m, y = y0 + r;
            if (x >= pw || y >= ph) return;
            if (in_plane) {
                const size_t idx = (size_t)y * pw + x;
                const long long s = (long long)load_sample(P.rec[c], P.bps, idx) + vv;
                store_sample(P.rec[c], P.bps, idx, (int)(s < 0 ? 0 : (s > mx ? mx : s)));
            } else {
                P.res[c][(size_t)y * P.res_stride[c] + x] = res_store(vv, mx);
            }
        };
        if (t.flags & HPVCD_TU_CBF)
            tb_residual_warp<kIdctMatrix>(P, t, dct, scr[warp][0], scr[warp][1], lane,
                                          [&](int r, int m, int v) { out(r, m, v); }, false);
        else
            for (int i = lane; i < n * n; i += 32) out(i / n, i % n, 0);
        __syncwarp();
    }
}

// ===========================================================================
// k_recon
// ===========================================================================
constexpr unsigned kFull = 0xffffffffu;

// Per-warp scratch of the decode-order walk.
struct WalkScratch {
    uint16_t s[132];  // the substituted line of a gathered TB, position i at s[i]
    // its available samples before substitution; the references of a 16x16 /
    // 32x32 TB, each with the next one (angular) or on its own (planar)
    union {
        uint16_t f[132];
        uint32_t pairs[66];
    };
};
constexpr size_t kWsBytes = (sizeof(WalkScratch) + 15) & ~(size_t)15;

// One bordered canvas per component of a CTU S x Sh: the row above the CTU
// first (x = -1 .. 2S-1 at index x + 8), then the CTU's Sh rows of S + 8
// entries (index 7 = the column left of the CTU, x at x + 8).  Both row
// lengths are multiples of 8 entries, so every interior row starts 16-byte
// aligned.
__host__ __device__ constexpr int can_top(int S) { return 2 * S + 8; }
__host__ __device__ constexpr int can_row(int S) { return S + 8; }
__host__ __device__ constexpr int can_size(int S, int Sh) { return can_top(S) + Sh * can_row(S); }
__device__ __forceinline__ int can_at(int S, int x, int y) {
    return y < 0 ? x + 8 : can_top(S) + y * can_row(S) + x + 8;
}
// The same index for a sample of the CTU's own rows (y >= 0), without the
// test for the row above.
__device__ __forceinline__ int can_in(int S, int x, int y) { return can_top(S) + y * can_row(S) + x + 8; }

// Shared-memory layout of one CTA: the canvases, one walk scratch per
// walking warp, the walk entries, the blend table, the 16x16 stamp map.
// Records of one CTU staged at once: up to 256 luma TBs, one "mark decoded"
// record per inter CU (64 at most) and the chroma TBs (64 per component at
// 4:2:0, 128 at 4:2:2, 256 at 4:4:4).  A CTU with more records is malformed.
// Chroma formats of a layout: kFmt420 (also 4:0:0), kFmt444, kFmt422; the
// 4:4:4 layout holds every format, the 4:2:2 one also 4:2:0.
constexpr int kFmt420 = 0, kFmt444 = 1, kFmt422 = 2;
constexpr int kRecCap420 = 256 + 64 + 2 * 64;
constexpr int kRecCap422 = 256 + 64 + 2 * 128;
constexpr int kRecCap444 = 256 + 64 + 2 * 256;
constexpr int kListCap = 256;  // intra TBs of luma in one CTU (all 4x4)
constexpr uint32_t kNoStamp = 0xffffffffu;

struct ReconLayout {
    int cs_w, cs_h;  // chroma canvas width and height (CTU interior)
    int rec_cap;     // staged records
    int list_c;      // intra TBs per chroma component
    size_t off_can_y, off_can_c, off_ws, off_ents, off_tab, off_stamp, off_misc, total;
    __host__ __device__ ReconLayout(int cfmt, int walkers) {
        cs_w = cfmt == kFmt444 ? 64 : 32;
        cs_h = cfmt == kFmt420 ? 32 : 64;
        rec_cap = cfmt == kFmt444 ? kRecCap444 : (cfmt == kFmt422 ? kRecCap422 : kRecCap420);
        list_c = cfmt == kFmt444 ? 256 : (cfmt == kFmt422 ? 128 : 64);
        size_t o = 0;
        off_can_y = o; o += (size_t)can_size(64, 64) * sizeof(uint16_t);
        o = (o + 15) & ~(size_t)15;
        off_can_c = o; o += 2 * (size_t)can_size(cs_w, cs_h) * sizeof(uint16_t);
        o = (o + 15) & ~(size_t)15;
        off_ws = o;    o += (size_t)walkers * kWsBytes;
        off_ents = o;  o += (size_t)(kListCap + 2 * list_c) * sizeof(uint4);
        off_tab = o;   o += (size_t)(64 * 64 + cs_w * cs_h) * sizeof(uint32_t);
        off_stamp = o; o += 256 * sizeof(uint32_t);
        off_misc = o;  o += 128;  // claimed item, have bits, covered words, done flags, TB counts
        total = o;
    }
    __host__ __device__ int ent_off(int c) const { return c == 0 ? 0 : kListCap + (c - 1) * list_c; }
    __host__ __device__ int ent_cap(int c) const { return c == 0 ? kListCap : list_c; }
    __host__ __device__ int tab_off(int c) const { return c == 0 ? 0 : 64 * 64; }
};
// The CTU's records are staged in the canvases: they are done with (turned
// into walk entries) before any sample or residual is put there.
static_assert(kRecCap420 * sizeof(hpvcd_tu) <= (can_size(64, 64) + 2 * can_size(32, 32)) * sizeof(uint16_t) &&
                  kRecCap422 * sizeof(hpvcd_tu) <= (can_size(64, 64) + 2 * can_size(32, 64)) * sizeof(uint16_t) &&
                  kRecCap444 * sizeof(hpvcd_tu) <= (can_size(64, 64) + 2 * can_size(64, 64)) * sizeof(uint16_t),
              "records fit the canvases");
// (a gathered line is addressed from its component's canvas on)
static_assert(3 * can_size(64, 64) + 3 * kWsBytes / sizeof(uint16_t) < 0x4000, "line positions fit the walk entries");

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Everything one warp needs about one component of the current CTU.
struct Comp {
    int ox, oy;   // CTU origin in component samples
    int pw, ph;   // plane size
    int S, Sh;    // CTU width and height in component samples
    int sw, sh;   // luma samples per component sample (1 or 2)
    uint32_t nb_ok;  // neighbour CTUs of the same slice and tile: 1 left, 2 above-left, 4 above, 8 above-right
    const hpvcd_cell* ci_cells;  // constrained intra prediction: cells whose INTER samples are unusable
    int gw;                      // cells per row
    bool restricted;             // nb_ok != 0xf or ci_cells: gather_ref runs restricted_ok
    bool ccp;                    // chroma of a cross-component picture: res_scale gives a residual
    int bd, max_v;
    bool luma, filt, smoothing, strong;
    uint16_t* can;       // bordered canvas
    const int16_t* res;  // int16 residual plane (k_residual) at the CTU origin
    int rs;              // its row stride in samples (a multiple of 16)
};

__device__ __forceinline__ int cidx(const Comp& k, int x, int y) { return can_at(k.S, x, y); }
__device__ __forceinline__ int cin(const Comp& k, int x, int y) { return can_in(k.S, x, y); }

// Reference sample i of the line (i < 2n: left column bottom-up, 2n: the
// corner, > 2n: above row) with its availability (decode.rs:4651-4690
// luma_avail / chroma_avail restricted to this CTU and its already
// reconstructed neighbours of the same slice and tile).  Inside the
// CTU a sample is available when the luma record that marked its 4x4 cell
// decoded comes before the current record `jrec` in decode order: `stamp`
// holds, per cell, the index of the first luma record covering it
// (decode.rs:3170-3189 marks cells as records complete).
// Slices, tiles and constrained intra prediction: a sample of a neighbour CTU
// of another slice or tile (decode.rs:4651-4690 same_slice / same_tile) or
// of an inter cell under constrained_intra_pred (decode.rs:4641-4649) is not
// available.  (x, y) relative to the CTU, (ax, ay) in the plane.
__device__ __forceinline__ bool restricted_ok(const Comp& k, int x, int y, int ax, int ay) {
    uint32_t bit = 0;  // 1 left, 2 above-left, 4 above, 8 above-right, 0 this CTU
    if (x < 0)
        bit = y < 0 ? 2u : 1u;
    else if (y < 0)
        bit = x < k.S ? 4u : 8u;
    if (bit && !(k.nb_ok & bit)) return false;
    if (k.ci_cells && (k.ci_cells[(size_t)((ay * k.sh) >> 2) * k.gw + ((ax * k.sw) >> 2)].flags & HPVCD_CELL_INTER))
        return false;
    return true;
}

__device__ __forceinline__ bool gather_ref(const Comp& k, const uint32_t* stamp, uint32_t jrec, int n2, int x0,
                                           int y0, int i, int* v) {
    const bool left_side = i < n2;
    const int x = left_side ? x0 - 1 : x0 + (i - n2 - 1);
    const int y = left_side ? y0 + (n2 - 1 - i) : y0 - 1;
    const int ax = k.ox + x, ay = k.oy + y;
    // both loads from clamped (always valid) positions, issued together;
    // the availability test picks the result
    const int ys = min(max(y, 0), k.Sh - 1), xs = min(max(x, 0), k.S - 1);
    const uint32_t st = stamp[((ys * k.sh) >> 2) * 16 + ((xs * k.sw) >> 2)];
    const int cv = k.can[cidx(k, y < 0 ? x : min(x, k.S - 1), min(y, k.Sh - 1))];
    bool a = ax >= 0 && ay >= 0 && ax < k.pw && ay < k.ph;
    if (y >= 0) {
        if (x < 0)
            a = a && y < k.Sh;  // left CTU (below-left CTU is not reconstructed yet)
        else
            a = a && x < k.S && y < k.Sh && st < jrec;
    }
    if (k.restricted && a) a = restricted_ok(k, x, y, ax, ay);  // warp-uniform branch
    *v = a ? cv : 0;
    return a;
}

// The angular reference projection of intra.rs:305-318: position in the
// reference line of refs[k] (k in [-n, 2n]).
__device__ __forceinline__ int ref_pos(int k, bool vertical, int n2, int inv) {
    if (k >= 0) return vertical ? n2 + k : n2 - k;
    const int idx = max(min((k * inv + 128) >> 8, n2), 0);
    return vertical ? n2 - idx : n2 + idx;
}

// I_PCM block (decode.rs:2768-2839): its samples, written to the residual
// plane by k_residual, go to the canvas unchanged.
__device__ __forceinline__ void pcm_tb(const Comp& k, int log2n, int x0, int y0, int lane) {
    const int n = 1 << log2n;
    const int vw = min(n, k.pw - (k.ox + x0)), vh = min(n, k.ph - (k.oy + y0));
    for (int i = lane; i < n * n; i += 32) {
        const int yy = i >> log2n, xx = i & (n - 1);
        if (xx < vw && yy < vh)
            k.can[cin(k, x0 + xx, y0 + yy)] =
                (uint16_t)clamp3i(k.res[(size_t)(y0 + yy) * k.rs + x0 + xx], 0, k.max_v);
    }
    __syncwarp();
}

// Whether the reference line of an n x n intra TB is filtered
// (intra.rs:151-219: luma, or 4:4:4 chroma, with smoothing on and a mode
// far enough from the horizontal / vertical).
__device__ __forceinline__ bool ref_filtered(const Comp& k, int n, int mode) {
    if (!(k.filt && k.smoothing && mode != 1)) return false;
    const int md = min(abs(mode - 26), abs(mode - 10));
    const int thresh = n == 8 ? 7 : (n == 16 ? 1 : 0);
    return mode == 0 || md > thresh;
}

__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s), "l"(gmem) : "memory");
}

// Stages the visible part of a coded n x n TB's residual (written by
// k_residual) into the TB's own canvas area with asynchronous copies, the
// lanes of a warp side by side: 16 bytes per copy, 8 for 4x4 TBs.  Every coded
// TB of a CTU is staged before its walk starts.  The area of a TB not yet
// reconstructed is never an available reference sample of an earlier TB (its
// stamp is later), so the staged values are never read as samples; each lane
// predicting a sample reads its residual in place.
__device__ __forceinline__ void stage_residual(const Comp& k, int n, int x0, int y0, int lane) {
    const int vw = min(n, k.pw - (k.ox + x0)), vh = min(n, k.ph - (k.oy + y0));
    const int16_t* src = k.res + (size_t)y0 * k.rs + x0;
    uint16_t* dst = k.can + cin(k, x0, y0);
    const int cr = can_row(k.S);
    if (n == 4) {
        if (lane < vh) cp_async8(dst + lane * cr, src + (size_t)lane * k.rs);
        return;
    }
    const int lq = 28 - __clz(n);  // 8-sample chunks of a row
    for (int i = lane; i < vh << lq; i += 32) {
        const int r = i >> lq, q = 8 * (i & ((1 << lq) - 1));
        if (q < vw) cp_async16(dst + r * cr + q, src + (size_t)r * k.rs + q);
    }
}

// ---- edges between neighbouring CTUs ----
// Other CTUs only read a CTU's right column and bottom row.  A CTU publishes
// them as 64-bit edge words of four samples (common.cuh), each word as soon
// as the TB that covers it is reconstructed: plain stores, nothing to wait
// for.  The CTA's edge warp polls the words of the left, above-left, above
// and above-right CTUs, unpacks them into the canvases and sets a bit per
// word in shared memory, where the walking warps look before a TB on the
// CTU's top or left edge.  So a CTU's lag behind its neighbours is a few TBs
// and a walking warp never waits for a round trip to L2.
//
// Have bits of a component: word 0, bit i: row above, samples 4i .. 4i + 3
// (i < 2S / 4); word 1, bit i < 16: left column, rows 4i .. 4i + 3, bit 16:
// the corner.  Words outside the picture count as present.
constexpr uint32_t kHaveCorner = 1u << 16;

// The right-column and bottom-row words of component c of CTU (cx, cy).
__device__ __forceinline__ unsigned long long* edge_words(const DevPic& P, int cx, int cy, int c) {
    const int ctb = 1 << P.log2_ctb;
    const int per = edge_words_per_ctu(ctb, P.idc, P.sub_w, P.sub_h);
    unsigned long long* w = P.edges + ((size_t)cy * P.ctb_cols + cx) * per;
    return c ? w + edge_words_of(ctb, P.sub_w, P.sub_h, 0) + (c - 1) * edge_words_of(ctb, P.sub_w, P.sub_h, 1) : w;
}
constexpr unsigned long long kEdgeTags = 0x8000800080008000ull;
__device__ __forceinline__ void put_edge(unsigned long long* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    st_edge(p, a | 0x8000u, b | 0x8000u, c | 0x8000u, d | 0x8000u);
}

// Publishes the edge words a finished n x n TB at (x0, y0) covers, from the
// canvas: lanes 0..15 the right column, lanes 16..31 the bottom row.
__device__ __forceinline__ void publish_tb(const uint16_t* can, int row, int S, int Sh, int x0, int y0, int n,
                                           unsigned long long* words, int lane) {
    const bool bottom = lane >= 16;
    const int i = lane & 15;
    if (i < (n >> 2) && (bottom ? y0 + n == Sh : x0 + n == S)) {
        const int x = bottom ? x0 + 4 * i : S - 1, y = bottom ? Sh - 1 : y0 + 4 * i, st = bottom ? 1 : row;
        const uint16_t* q = can + can_in(S, x, y);
        put_edge(words + (bottom ? (Sh >> 2) + (x >> 2) : y >> 2), q[0], q[st], q[2 * st], q[3 * st]);
    }
}

// One component's place in the CTU, for the edge warp.
struct EdgeGeo {
    int ox, oy, S, Sh, pw, ph;
};
__device__ __forceinline__ EdgeGeo edge_geo(const DevPic& P, int c, int cx, int cy) {
    const int ctb = 1 << P.log2_ctb;
    EdgeGeo e;
    e.S = c ? ctb / P.sub_w : ctb;
    e.Sh = c ? ctb / P.sub_h : ctb;
    e.ox = cx * e.S;
    e.oy = cy * e.Sh;
    e.pw = c ? P.cw : P.w;
    e.ph = c ? P.ch : P.h;
    return e;
}
// Whether this lane's word of the row above / of the left column (lane 16:
// the corner) lies inside the picture.
__device__ __forceinline__ bool edge_top_in(const EdgeGeo& e, int lane) {
    return e.oy > 0 && 4 * lane < 2 * e.S && e.ox + 4 * lane < e.pw;
}
__device__ __forceinline__ bool edge_left_in(const EdgeGeo& e, int lane) {
    if (lane == 16) return e.ox > 0 && e.oy > 0;
    return e.ox > 0 && 4 * lane < e.Sh && e.oy + 4 * lane < e.ph;
}

// The edge warp of a CTU: first publishes the edge words no intra TB covers
// (inter samples, final in the canvas), then receives the neighbours' words
// until every one has arrived or the walking warps are done.  A wait here
// cannot outlast them: theirs are bounded.
template <class CanOf>
__device__ void edge_service(const DevPic& P, int cx, int cy, int ncomp, CanOf can_of, const uint32_t* cov,
                             volatile uint32_t* s_have, volatile uint32_t* s_done, int walkers, int lane) {
    const unsigned long long* tp[3];
    const unsigned long long* lp[3];
    uint32_t pend = 0;  // bit 2c: this lane's word above, 2c + 1: left / corner
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        tp[c] = lp[c] = nullptr;
        if (c >= ncomp) continue;
        const EdgeGeo e = edge_geo(P, c, cx, cy);
        const uint32_t full = ((1u << (e.Sh >> 2)) - 1u) | (((1u << (e.S >> 2)) - 1u) << 16);
        const uint32_t miss = full & ~cov[c];
        if (miss >> lane & 1u) {
            const uint16_t* can = can_of(c);
            const bool bottom = lane >= 16;
            const int i = lane & 15, st = bottom ? 1 : can_row(e.S);
            const uint16_t* q = can + (bottom ? can_in(e.S, 4 * i, e.Sh - 1) : can_in(e.S, e.S - 1, 4 * i));
            put_edge(edge_words(P, cx, cy, c) + (bottom ? (e.Sh >> 2) + i : i), q[0], q[st], q[2 * st], q[3 * st]);
        }
        if (edge_top_in(e, lane)) {
            const int w = e.S >> 2;
            tp[c] = (lane < w ? edge_words(P, cx, cy - 1, c) + lane : edge_words(P, cx + 1, cy - 1, c) + lane - w) + (e.Sh >> 2);
            pend |= 1u << (2 * c);
        }
        if (edge_left_in(e, lane)) {
            lp[c] = lane == 16 ? edge_words(P, cx - 1, cy - 1, c) + (e.Sh >> 2) + (e.S >> 2) - 1
                               : edge_words(P, cx - 1, cy, c) + lane;
            pend |= 2u << (2 * c);
        }
    }
    uint32_t nap = 32;
    for (;;) {
        unsigned long long t[3], l[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            t[c] = l[c] = 0ull;
            if (pend >> (2 * c) & 1u) t[c] = ld_edge(tp[c]);
            if (pend >> (2 * c) & 2u) l[c] = ld_edge(lp[c]);
        }
        bool news = false;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (c >= ncomp) continue;
            const int S = c ? (1 << P.log2_ctb) / P.sub_w : 1 << P.log2_ctb;
            uint16_t* can = can_of(c);
            const bool gt = (t[c] & kEdgeTags) == kEdgeTags, gl = (l[c] & kEdgeTags) == kEdgeTags;
            if (gt) {  // can_at(S, 4 * lane, -1): 8-byte aligned
                t[c] &= ~kEdgeTags;
                *(uint2*)(can + 8 + 4 * lane) = make_uint2((uint32_t)t[c], (uint32_t)(t[c] >> 32));
            }
            if (gl) {
                l[c] &= ~kEdgeTags;
                if (lane == 16) {
                    can[7] = (uint16_t)(l[c] >> 48);  // can_at(S, -1, -1)
                } else {
                    uint16_t* q = can + can_in(S, -1, 4 * lane);
                    const int row = can_row(S);
                    q[0] = (uint16_t)l[c];
                    q[row] = (uint16_t)(l[c] >> 16);
                    q[2 * row] = (uint16_t)(l[c] >> 32);
                    q[3 * row] = (uint16_t)(l[c] >> 48);
                }
            }
            const uint32_t bt = __ballot_sync(kFull, gt), bl = __ballot_sync(kFull, gl);
            if (gt) pend &= ~(1u << (2 * c));
            if (gl) pend &= ~(2u << (2 * c));
            if (bt | bl) {
                news = true;
                __threadfence_block();  // the samples before their bits
                __syncwarp();
                if (lane == 0) {
                    s_have[2 * c] = s_have[2 * c] | bt;
                    s_have[2 * c + 1] = s_have[2 * c + 1] | bl;
                }
            }
        }
        if (!__any_sync(kFull, pend != 0u)) break;
        int done = 0;
        for (int w = 0; w < walkers; ++w) done += s_done[w] != 0u;
        if (done == walkers) break;
        if (news) {
            nap = 32;
        } else {
            __nanosleep(nap);
            nap = min(2 * nap, 256u);
        }
    }
}

// Waits (bounded, in shared memory) until the words a TB needs are in the
// canvas; after a wait that ran out every word counts as present.
struct Have {
    uint32_t top, left;
};
__device__ __noinline__ Have wait_edges(Have h, uint32_t need_top, uint32_t need_left, const volatile uint32_t* s_have,
                                        uint32_t spin_limit, uint32_t* dev_err, int lane) {
    uint32_t spins = 0;
    for (;;) {
        h.top = s_have[0];
        h.left = s_have[1];
        if (!((need_top & ~h.top) | (need_left & ~h.left))) break;
        if (++spins > spin_limit) {
            if (lane == 0) atomicOr(dev_err, DEV_ERR_TIMEOUT);
            h.top = h.left = 0xffffffffu;
            break;
        }
        if (spins > 16) __nanosleep(spins > 1024 ? 64 : 16);
    }
    // one lane may have seen a later state than another
    h.top = __reduce_and_sync(kFull, h.top);
    h.left = __reduce_and_sync(kFull, h.left);
    __threadfence_block();
    return h;
}

// ---- walk entries: everything about an intra TB that does not depend on
// sample values, worked out for all TBs of a CTU in parallel before its walk
// (overwriting the TB's staged record), so that the serial walk only loads
// reference samples, predicts and adds the residual ----
//
// The reference line of an n x n TB has 4n + 1 positions: i < 2n the left
// column bottom-up, 2n the corner, > 2n the row above.  Substitution
// (intra.rs:84-148) replaces an unavailable sample by the nearest available
// one below it in the line, or by the first available one.  The available
// positions of a TB in z-order are one run [lo, hi] around the corner, so
// substitution is a clamp of the position to [lo, hi]; a TB whose positions
// are not one run (possible at slice boundaries and under constrained intra
// prediction), or that has none, is flagged kTbGather and its line is gathered
// sample by sample first.
//   x: canvas offset of the TB | of line position 0 << 16 | plain << 30 |
//      coded << 31
//   y: canvas offset of the corner | blend table offset of a plain TB << 16
//   z: lo | hi << 8 | 2n << 16 | mode << 24 | kTbFilt
//   w: x (6 bits) | kHow* << 6 | y << 8 (in the CTU) | kHow* << 14 |
//      record index (< 1024) << 16 | kTb* flags << 26
// Measured when the entries came in (4032x3024 grid, 70 luma TBs a CTU): the
// walk's chain went from ~87k to ~46k cycles a CTU (4x4 700 -> 500, 16x16 5100
// -> 1650, 32x32 10700 -> 3300 cycles); 512x512 tile 1004 -> 649 us.
constexpr uint32_t kTbCoded = 1u << 31, kTbPlainX = 1u << 30 /* of x */, kTbFilt = 1u << 31 /* of z */;
// the TB reads neighbour CTUs, its line must be gathered, it is an I_PCM
// block, it covers edge words, line position 32 is available, it is a 4x4 or
// 8x8 TB of an angular mode without line or edge filter and with one run of
// available samples (each sample is a blend of two line samples)
constexpr uint32_t kTbEdge = 1u, kTbGather = 2u, kTbPcm = 4u, kTbPub = 8u, kTbHi32 = 16u, kTbPlain = 32u;

struct TbEntry {
    uint4 w;
    __device__ __forceinline__ int org() const { return (int)(w.x & 0xffffu); }
    __device__ __forceinline__ int line0() const { return (int)((w.x >> 16) & 0x3fffu); }
    __device__ __forceinline__ bool coded() const { return (w.x & kTbCoded) != 0u; }
    __device__ __forceinline__ bool plain() const { return (w.x & kTbPlainX) != 0u; }
    __device__ __forceinline__ int corner() const { return (int)(w.y & 0xffffu); }
    __device__ __forceinline__ uint32_t tab() const { return w.y >> 16; }
    __device__ __forceinline__ int lo() const { return (int)(w.z & 0xffu); }
    __device__ __forceinline__ int hi() const { return (int)((w.z >> 8) & 0xffu); }
    __device__ __forceinline__ int n2() const { return (int)((w.z >> 16) & 0xffu); }
    __device__ __forceinline__ int mode() const { return (int)((w.z >> 24) & 0x3fu); }
    __device__ __forceinline__ int x() const { return (int)(w.w & 0x3fu); }
    __device__ __forceinline__ int y() const { return (int)((w.w >> 8) & 0x3fu); }
    __device__ __forceinline__ uint32_t jrec() const { return (w.w >> 16) & 0x3ffu; }
    __device__ __forceinline__ uint32_t flags() const { return w.w >> 26; }
};

// An entry whose owner may be adding the walk's kHow* bits to word w at the
// same time: w is read (and written by set_how) by strong accesses of its own,
// not as a part of the vector; the bits that are read never change.  (Two
// barriers around the additions instead: 24 mixed pictures 4146 us for 3946,
// 4032x3024 grid 579 for 557.)
__device__ __forceinline__ TbEntry shared_entry(const uint4* e) {
    const uint2 xy = *(const uint2*)e;
    return TbEntry{make_uint4(xy.x, xy.y, e->z, *(const volatile uint32_t*)&e->w)};
}
// The same without w.
__device__ __forceinline__ TbEntry line_entry(const uint4* e) {
    const uint2 xy = *(const uint2*)e;
    return TbEntry{make_uint4(xy.x, xy.y, e->z, 0u)};
}
__device__ __forceinline__ void set_how(uint4* e, uint32_t w) { *(volatile uint32_t*)&e->w = w; }

// The walk entry of intra record j (t, at (x0, y0) of the CTU); `flags` gives
// kTbPcm and kTbPub, the others are added here.
__device__ __forceinline__ uint4 make_entry(const Comp& k, const hpvcd_tu& t, int x0, int y0, uint32_t jrec,
                                            const uint32_t* stamp, bool coded, uint32_t flags) {
    const int n = 1 << t.log2n, n2 = 2 * n;
    auto decoded = [&](int x, int y) { return stamp[((y * k.sh) >> 2) * 16 + ((x * k.sw) >> 2)] < jrec; };
    auto allowed = [&](int x, int y) { return !k.restricted || restricted_ok(k, x, y, k.ox + x, k.oy + y); };
    // Availability is per cell, but an n x n block aligned to its size is one
    // run of the decode order, so the first and last cell of each side's n
    // samples (the row above, above-right, left, below-left) speak for it.
    // Where they differ, and where slices, tiles or constrained intra
    // prediction decide per cell, every cell is looked at.
    const int yend = min(min(y0 + n2, k.Sh), k.ph - k.oy), xend = min(y0 == 0 ? x0 + n2 : min(x0 + n2, k.S), k.pw - k.ox);
    const bool any_l = k.ox + x0 > 0, any_a = k.oy + y0 > 0;
    bool one_run = true, cells = k.restricted;
    int al = 0, ar = 0;  // samples available downwards from the top left, rightwards from the left above
    if (any_l && !cells) {
        if (x0 == 0) {
            al = n2;
        } else {
            const bool a = decoded(x0 - 1, y0), b = decoded(x0 - 1, min(y0 + n, yend) - 1);
            const bool low = y0 + n < yend;
            const bool d = low && decoded(x0 - 1, y0 + n), e = low && decoded(x0 - 1, yend - 1);
            cells = a != b || d != e || (d && !a);
            al = a ? (d ? n2 : n) : 0;
        }
    }
    if (any_a && !cells) {
        if (y0 == 0) {
            ar = n2;
        } else {
            const bool a = decoded(x0, y0 - 1), b = decoded(min(x0 + n, xend) - 1, y0 - 1);
            const bool right = x0 + n < xend;
            const bool d = right && decoded(x0 + n, y0 - 1), e = right && decoded(xend - 1, y0 - 1);
            cells = a != b || d != e || (d && !a);
            ar = a ? (d ? n2 : n) : 0;
        }
    }
    if (cells) {
        const int uw = 4 / k.sw, uh = 4 / k.sh;  // a cell in this component's samples
        al = ar = 0;
        bool open = true;
        for (int y = y0; any_l && y < yend; y += uh) {
            const bool a = (x0 == 0 || decoded(x0 - 1, y)) && allowed(x0 - 1, y);
            if (a && open) al = y + uh - y0;
            if (a && !open) one_run = false;
            open = open && a;
        }
        open = true;
        for (int x = x0; any_a && x < xend; x += uw) {
            const bool a = (y0 == 0 || decoded(x, y0 - 1)) && allowed(x, y0 - 1);
            if (a && open) ar = x + uw - x0;
            if (a && !open) one_run = false;
            open = open && a;
        }
    }
    al = min(al, max(yend - y0, 0));
    ar = min(ar, max(xend - x0, 0));
    bool corner = any_l && any_a && allowed(x0 - 1, y0 - 1);
    if (corner && x0 > 0 && y0 > 0) corner = decoded(x0 - 1, y0 - 1);
    int lo = n2 - al, hi = n2 + ar;
    if (!corner) {
        if (al && ar) one_run = false;
        if (al)
            hi = n2 - 1;
        else
            lo = n2 + 1;
    }
    if (lo > hi) one_run = false;  // nothing available
    if (!one_run) lo = 0, hi = 4 * n, flags |= kTbGather;
    if (x0 == 0 || y0 == 0) flags |= kTbEdge;
    if (hi == 32) flags |= kTbHi32;
    const bool filt = n > 4 && ref_filtered(k, n, t.mode);
    if (n <= 8 && t.mode >= 2 && one_run && !filt && !(flags & kTbPcm) && !(k.luma && (t.mode == 10 || t.mode == 26)))
        flags |= kTbPlain;
    const uint32_t tab = flags & kTbPlain ? (uint32_t)((y0 >> 2) * (k.S >> 2) + (x0 >> 2)) * 16u : 0u;
    uint4 w;
    w.x = (uint32_t)cin(k, x0, y0) | ((uint32_t)cin(k, x0 - 1, y0 + n2 - 1) << 16);
    w.y = (uint32_t)cidx(k, x0 - 1, y0 - 1) | (tab << 16);
    w.z = (uint32_t)lo | ((uint32_t)hi << 8) | ((uint32_t)n2 << 16) | ((uint32_t)t.mode << 24);
    if (coded) w.x |= kTbCoded;
    if (flags & kTbPlain) w.x |= kTbPlainX;
    if (filt) w.z |= kTbFilt;
    w.w = (uint32_t)x0 | ((uint32_t)y0 << 8) | (jrec << 16) | (flags << 26);
    return w;
}

// Angular prediction of 4x4 and 8x8 TBs as data: for every mode and sample
// the two line positions it interpolates (intra.rs:305-318, the projection
// of negative angles included) and their weights: p0 | p1 << 8 | weight of
// p1 << 16 | weight of p0 << 24.
struct AngularTables {
    uint32_t t4[33][16], t8[33][64];
};
constexpr uint32_t angular_entry(int mode, int n, int x, int y) {
    constexpr int ang[33] = {32,  26,  21,  17,  13,  9,  5,  2,  0,  -2, -5, -9, -13, -17, -21, -26, -32,
                             -26, -21, -17, -13, -9,  -5, -2, 0,  2,  5,  9,  13, 17,  21,  26,  32};
    constexpr int inva[15] = {-4096, -1638, -910, -630, -482, -390, -315, -256, -315, -390, -482, -630, -910, -1638, -4096};
    const int angle = ang[mode - 2], n2 = 2 * n;
    const bool vertical = mode >= 18;
    const int inv = angle < 0 ? inva[mode - 11] : 0;
    const int a = vertical ? y : x, b = vertical ? x : y, pos = (a + 1) * angle;
    const int whole = pos >= 0 ? pos / 32 : -((31 - pos) / 32), frac = pos - 32 * whole;
    uint32_t p[2] = {0, 0};
    for (int h = 0; h < 2; ++h) {
        int k = b + whole + 1 + h;
        if (k > n2) k = n2;
        if (k >= 0) {
            p[h] = (uint32_t)(vertical ? n2 + k : n2 - k);
        } else {
            int idx = (k * inv + 128) / 256;  // k and inv are negative
            idx = idx < 0 ? 0 : (idx > n2 ? n2 : idx);
            p[h] = (uint32_t)(vertical ? n2 - idx : n2 + idx);
        }
    }
    return p[0] | (p[1] << 8) | ((uint32_t)frac << 16) | ((uint32_t)(32 - frac) << 24);
}
constexpr AngularTables make_angular() {
    AngularTables T{};
    for (int m = 0; m < 33; ++m) {
        for (int i = 0; i < 16; ++i) T.t4[m][i] = angular_entry(m + 2, 4, i & 3, i >> 2);
        for (int i = 0; i < 64; ++i) T.t8[m][i] = angular_entry(m + 2, 8, i & 7, i >> 3);
    }
    return T;
}
__device__ const __align__(16) AngularTables g_angular = make_angular();

// The line of a TB as the walk addresses it: position i is at canvas offset
// l0 - i * ls below the corner and c0 + i from it on, after the clamp to
// [lo, hi] that substitutes unavailable samples.
struct Line {
    int l0, ls, c0, lo, hi, n2;
    __device__ __forceinline__ Line(const TbEntry& E, int stride) {
        n2 = E.n2();
        l0 = E.line0();
        ls = stride;
        c0 = E.corner() - n2;
        lo = E.lo();
        hi = E.hi();
    }
    __device__ __forceinline__ int at(int i) const {
        i = min(max(i, lo), hi);
        return i < n2 ? l0 - i * ls : c0 + i;
    }
};

// Blend table of a CTU component: one word per sample of its plain TBs, by
// 4x4 blocks in raster order: canvas byte offsets of the two line samples
// (even, < 2^14) << 0 and << 13 | weight of the second (of 32) << 27.
// With it the walk neither looks anything up nor clamps: it was 270 cycles a
// 4x4 TB and 850 an 8x8 one with the table of modes and the line in the loop.
constexpr uint32_t kBlendAdr = 0x3ffeu;
static_assert(2 * can_size(64, 64) < 0x4000, "canvas byte offsets fit the blend words");
__device__ __forceinline__ uint32_t blend_word(const Line& L, uint32_t ang) {
    return (uint32_t)(2 * L.at((int)(ang & 0xffu))) | ((uint32_t)(2 * L.at((int)((ang >> 8) & 0xffu))) << 13) |
           ((ang & 0x1f0000u) << 11);
}
__device__ __forceinline__ int blend_of(const uint16_t* can, uint32_t w) {
    const int a = *(const uint16_t*)((const char*)can + (w & kBlendAdr));
    const int b = *(const uint16_t*)((const char*)can + ((w >> 13) & kBlendAdr));
    return (32 * a + (int)(w >> 27) * (b - a) + 16) >> 5;
}

// Residual add + clip (reconstruct.rs:214-251) of two samples in 16-bit halves.
__device__ __forceinline__ uint32_t add_clip2(uint32_t pred, uint32_t res, int max_v) {
    return __viaddmin_s16x2_relu(pred, res, (uint32_t)max_v * 0x10001u);
}

// 4x4 intra TB that is not plain: v is line position `lane` (lanes 0..16;
// prediction intra.rs:257-372, no filtering of 4x4
// lines, intra.rs:174), lanes 0..15 one sample each, at px.
__device__ __forceinline__ void walk_tb4(uint16_t* px, int mode, bool coded, bool luma, int max_v, int v, int lane) {
    constexpr int n = 4, n2 = 8;
    const int yy = (lane >> 2) & 3, xx = lane & 3;
    const int rv = coded ? (int)(int16_t)*px : 0;
    int pred;
    if (mode >= 2) {
        if (luma && (mode == 26 || mode == 10)) {  // straight, with the vertical / horizontal edge filter (n < 32)
            pred = __shfl_sync(kFull, v, mode == 26 ? n2 + xx + 1 : n2 - yy - 1);
            const int c0 = __shfl_sync(kFull, v, n2);
            const int a0 = __shfl_sync(kFull, v, mode == 26 ? n2 + 1 : n2 - 1);
            const int e = __shfl_sync(kFull, v, mode == 26 ? n2 - (yy + 1) : n2 + xx + 1);
            if (mode == 26 ? xx == 0 : yy == 0) pred = clamp3i(a0 + ((e - c0) >> 1), 0, max_v);
        } else {  // a gathered line
            const uint32_t lut = g_angular.t4[mode - 2][lane & 15];
            const int r0 = __shfl_sync(kFull, v, (int)lut), r1 = __shfl_sync(kFull, v, (int)(lut >> 8));
            pred = (int)((lut >> 24) * (uint32_t)r0 + ((lut >> 16) & 0xffu) * (uint32_t)r1 + 16u) >> 5;
        }
    } else if (mode == 1) {  // DC
        const int part = ((lane >= n2 - n && lane < n2) || (lane > n2 && lane <= n2 + n)) ? v : 0;
        const int dc = ((int)__reduce_add_sync(kFull, (unsigned)part) + n) >> 3;
        pred = dc;
        if (luma) {
            const int l1 = __shfl_sync(kFull, v, n2 - 1), a1 = __shfl_sync(kFull, v, n2 + 1);
            const int e = __shfl_sync(kFull, v, yy == 0 ? n2 + xx + 1 : n2 - yy - 1);
            if (xx == 0 && yy == 0)
                pred = (l1 + 2 * dc + a1 + 2) >> 2;
            else if (yy == 0 || xx == 0)
                pred = (e + 3 * dc + 2) >> 2;
        }
    } else {  // planar
        const int lft = __shfl_sync(kFull, v, n2 - yy - 1), abv = __shfl_sync(kFull, v, n2 + xx + 1);
        const int tr = __shfl_sync(kFull, v, n2 + n + 1), bl = __shfl_sync(kFull, v, n2 - n - 1);
        pred = ((n - 1 - xx) * lft + (xx + 1) * tr + (n - 1 - yy) * abv + (yy + 1) * bl + n) >> 3;
    }
    if (lane < 16) *px = (uint16_t)__viaddmin_s32_relu(pred, rv, max_v);
    __syncwarp();
}

// 8x8 intra TB that is not plain: v is line position `lane`, v_hi position 32 where it is
// available (the same in every lane; else position 31 stands in for it);
// [1 2 1] filtering (intra.rs:151-219; no strong filter below
// 32x32) and prediction (intra.rs:257-372) by shuffles, two horizontally
// adjacent samples per lane, at px (canvas rows and TB columns are even).
__device__ __forceinline__ void walk_tb8(uint32_t* px, int mode, bool coded, bool filt, bool luma, int max_v, int v,
                                         int v_hi, bool hi_ok, uint2 lut, int lane) {
    constexpr int n = 8, n2 = 16;
    const int v31 = __shfl_sync(kFull, v, 31);
    v_hi = hi_ok ? v_hi : v31;
    const int yy = lane >> 2, xx = 2 * (lane & 3);
    const uint32_t rv = coded ? *px : 0u;
    if (filt) {
        const int up = __shfl_up_sync(kFull, v, 1);
        const int dn = __shfl_down_sync(kFull, v, 1);
        const int f = (up + 2 * v + (lane == 31 ? v_hi : dn) + 2) >> 2;
        v = lane == 0 ? v : f;
    }
    int out[2];
    if (mode >= 2) {
        const uint32_t w[2] = {lut.x, lut.y};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            int r0 = __shfl_sync(kFull, v, (int)w[h]);
            const int r1 = __shfl_sync(kFull, v, (int)(w[h] >> 8));
            if (h == 1 && (w[h] & 32u)) r0 = v_hi;  // position 32 (mode 34, the last sample)
            out[h] = (int)((w[h] >> 24) * (uint32_t)r0 + ((w[h] >> 16) & 0xffu) * (uint32_t)r1 + 16u) >> 5;
        }
        if (luma && (mode == 26 || mode == 10)) {
            const int c0 = __shfl_sync(kFull, v, n2);
            const int a0 = __shfl_sync(kFull, v, mode == 26 ? n2 + 1 : n2 - 1);
            const int e0 = __shfl_sync(kFull, v, mode == 26 ? n2 - (yy + 1) : n2 + xx + 1);
            const int e1 = __shfl_sync(kFull, v, n2 + xx + 2);
            if (mode == 26 ? xx == 0 : yy == 0) out[0] = clamp3i(a0 + ((e0 - c0) >> 1), 0, max_v);
            if (mode == 10 && yy == 0) out[1] = clamp3i(a0 + ((e1 - c0) >> 1), 0, max_v);
        }
    } else if (mode == 1) {  // DC
        const int part = ((lane >= n2 - n && lane < n2) || (lane > n2 && lane <= n2 + n)) ? v : 0;
        const int dc = ((int)__reduce_add_sync(kFull, (unsigned)part) + n) >> 4;
        out[0] = out[1] = dc;
        if (luma) {
            const int l1 = __shfl_sync(kFull, v, n2 - 1), a1 = __shfl_sync(kFull, v, n2 + 1);
            const int e0 = __shfl_sync(kFull, v, yy == 0 ? n2 + xx + 1 : n2 - yy - 1);
            const int e1 = __shfl_sync(kFull, v, n2 + xx + 2);
            if (xx == 0 && yy == 0)
                out[0] = (l1 + 2 * dc + a1 + 2) >> 2;
            else if (yy == 0 || xx == 0)
                out[0] = (e0 + 3 * dc + 2) >> 2;
            if (yy == 0) out[1] = (e1 + 3 * dc + 2) >> 2;
        }
    } else {  // planar
        const int tr = __shfl_sync(kFull, v, n2 + n + 1), bl = __shfl_sync(kFull, v, n2 - n - 1);
        const int lft = __shfl_sync(kFull, v, n2 - yy - 1);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int abv = __shfl_sync(kFull, v, n2 + xx + h + 1);
            out[h] = ((n - 1 - xx - h) * lft + (xx + h + 1) * tr + (n - 1 - yy) * abv + (yy + 1) * bl + n) >> 4;
        }
    }
    *px = add_clip2((uint32_t)out[0] | ((uint32_t)out[1] << 16), rv, max_v);
    __syncwarp();
}

// Two horizontally adjacent samples of a plain 8x8 TB per lane.
__device__ __forceinline__ void walk_plain8(const uint16_t* can, uint32_t* px, uint2 w, bool coded, int max_v) {
    const uint32_t rv = coded ? *px : 0u;
    const uint32_t p0 = (uint32_t)blend_of(can, w.x), p1 = (uint32_t)blend_of(can, w.y);
    *px = add_clip2(p0 | (p1 << 16), rv, max_v);
    __syncwarp();
}

// 16x16 or 32x32 intra TB by one warp, four horizontally adjacent samples per
// lane and row step.  First the line samples the prediction reads, filtered
// (intra.rs:151-219), go to the scratch: the projected references, each with
// the next one, or for planar and DC the line from the sample below the left
// column to the one right of the row above.  Then one rolled row loop per kind
// of prediction: the loops are kept small because on a loaded SM the walks
// wait for instructions first (unrolled by four the same batch took 8 % more).
__device__ __forceinline__ void walk_tb_big(uint16_t* can, int row, const Line& L, int org, int mode, bool coded,
                                            bool filt, bool luma, bool strong_on, int bd, WalkScratch& ws, int lane) {
    const int n2 = L.n2, n = n2 >> 1, hl = 29 - __clz(n);  // hl: log2 of the lanes per row
    const int max_v = (1 << bd) - 1;
    auto raw = [&](int i) { return (int)can[L.at(i)]; };
    const bool angular = mode >= 2, vertical = mode >= 18;
    const int angle = angular ? (int)c_intra_angle[mode - 2] : 0;
    const int inv = angle < 0 ? (int)c_inv_angle[mode - 11] : 0;
    const int k0 = angle < 0 ? 1 - n : 1;  // references k0 .. k0 + 2n - 1 are all a TB reads with a weight
    bool strong = false;
    int tl = 0, tr = 0, bl = 0;
    if (filt && luma && strong_on && n == 32) {  // intra.rs:176-196
        tl = raw(n2), tr = raw(2 * n2), bl = raw(0);
        const int thr = 1 << (bd - 5);
        strong = abs(bl + tl - 2 * raw(n2 - n)) < thr && abs(tr + tl - 2 * raw(n2 + n)) < thr;
    }
    uint16_t* const halves = (uint16_t*)ws.pairs;
    const int count = angular ? n2 : n2 + 3;
#pragma unroll 1
    for (int q = lane; q < count; q += 32) {
        const int i = angular ? ref_pos(k0 + q, vertical, n2, inv) : n2 - n - 1 + q;
        int v = raw(i);
        if (filt && i != 0 && i != 2 * n2) {
            if (!strong) {
                v = (raw(i - 1) + 2 * v + raw(i + 1) + 2) >> 2;
            } else if (i != n2) {
                const int d = abs(i - n2);
                v = ((n2 - d) * tl + d * (i > n2 ? tr : bl) + n) >> 6;
            }
        }
        if (angular) {  // reference q in its own pair and the one before
            halves[2 * q] = (uint16_t)v;
            if (q) halves[2 * q - 1] = (uint16_t)v;
        } else {
            ws.f[q] = (uint16_t)v;
        }
    }
    // this lane's columns, first row and rows per step
    const int x = 4 * (lane & ((1 << hl) - 1)), y0 = lane >> hl, ys = 32 >> hl;
    const bool edge = luma && n < 32;
    uint2* px = (uint2*)(can + org + y0 * row + x);  // canvas rows and TB columns are multiples of four
    const int step = (ys * row) >> 2;
    auto put = [&](int p0, int p1, int p2, int p3) {
        const uint2 r = coded ? *px : make_uint2(0u, 0u);
        *px = make_uint2(add_clip2(__byte_perm((uint32_t)p0, (uint32_t)p1, 0x5410), r.x, max_v),
                         add_clip2(__byte_perm((uint32_t)p2, (uint32_t)p3, 0x5410), r.y, max_v));
        px += step;
    };
    __syncwarp();
    if (angular) {
        // Sample (x, y) blends references idx and idx + 1 by frac, idx * 32 +
        // frac = 32 b + (a + 1) angle, b along the edge and a away from it.
        auto blend = [](uint32_t pair, int weights) { return __dp2a_lo((int)pair, weights, 16) >> 5; };
        auto weights = [](int pos) { return 32 + (pos & 31) * 255; };  // 32 - f | f << 8
        const uint32_t* const refs = ws.pairs + 1 - k0;
        if (edge && angle == 0) {  // modes 10 and 26: the first row / column is filtered
            const int c0 = raw(n2), a0 = raw(vertical ? n2 + 1 : n2 - 1);
#pragma unroll 1
            for (int y = y0; y < n; y += ys) {
                int p[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const bool first = vertical ? x + u == 0 : y == 0;
                    p[u] = (int)(refs[vertical ? x + u : y] & 0xffffu);
                    if (first) p[u] = clamp3i(a0 + ((raw(vertical ? n2 - (y + 1) : n2 + x + u + 1) - c0) >> 1), 0, max_v);
                }
                put(p[0], p[1], p[2], p[3]);
            }
        } else if (vertical) {
            int pos = (y0 + 1) * angle;
#pragma unroll 1
            for (int y = y0; y < n; y += ys, pos += ys * angle) {
                const uint32_t* r = refs + x + (pos >> 5);
                const int w = weights(pos);
                put(blend(r[0], w), blend(r[1], w), blend(r[2], w), blend(r[3], w));
            }
        } else {
            const int pa = (x + 1) * angle, pb = pa + angle, pc = pb + angle, pd = pc + angle;
            const int wa = weights(pa), wb = weights(pb), wc = weights(pc), wd = weights(pd);
            const uint32_t* r = refs + y0;
            const int ia = pa >> 5, ib = pb >> 5, ic = pc >> 5, id = pd >> 5;
#pragma unroll 1
            for (int y = y0; y < n; y += ys, r += ys) put(blend(r[ia], wa), blend(r[ib], wb), blend(r[ic], wc), blend(r[id], wd));
        }
    } else {
        // ws.f: below-left, left column upwards, corner, row above, above-right
        const uint16_t* const left = ws.f + n;       // left[-y]
        const uint16_t* const above = ws.f + n + 2;  // above[x]
        const int dc = mode == 1 ? (int)(__reduce_add_sync(kFull, lane < n ? (unsigned)above[lane] + left[-lane] : 0u) + n) >> (hl + 3)
                                 : 0;
        const int rt = above[n], lb = left[-n];
        int ab[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) ab[u] = above[x + u];
#pragma unroll 1
        for (int y = y0; y < n; y += ys) {
            const int lf = left[-y];
            int q[4] = {dc, dc, dc, dc};
            if (mode == 0) {  // planar
                const int vb = (y + 1) * lb + n, up = n - 1 - y;
#pragma unroll
                for (int u = 0; u < 4; ++u) q[u] = ((n - 1 - x - u) * lf + (x + u + 1) * rt + up * ab[u] + vb) >> (hl + 3);
            } else if (edge) {
                if (y == 0) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) q[u] = (ab[u] + 3 * dc + 2) >> 2;
                    if (x == 0) q[0] = (lf + 2 * dc + ab[0] + 2) >> 2;
                } else if (x == 0) {
                    q[0] = (lf + 3 * dc + 2) >> 2;
                }
            }
            put(q[0], q[1], q[2], q[3]);
        }
    }
    __syncwarp();
}

// The substituted line of a TB whose available positions are not one run
// (kTbGather): gathered sample by sample, then substituted (intra.rs:84-148)
// into ws.s.
__device__ __noinline__ void gather_line(const Comp& k, int log2n, int x0, int y0, const uint32_t* stamp, uint32_t jrec,
                                         WalkScratch& ws, int lane) {
    const int total = (4 << log2n) + 1, n2 = 2 << log2n;
    const int nw = (total + 31) >> 5;
    uint32_t my_mask = 0u;  // lane w: availability of positions 32w .. 32w + 31
    int first = -1;         // first available position
    for (int wd = 0; wd < nw; ++wd) {
        const int i = wd * 32 + lane;
        int v = 0;
        bool a = gather_ref(k, stamp, jrec, n2, x0, y0, min(i, total - 1), &v);
        a = a && i < total;
        if (a) ws.f[i] = (uint16_t)v;
        const uint32_t m = __ballot_sync(kFull, a);
        if (lane == wd) my_mask = m;
        if (first < 0 && m) first = wd * 32 + __ffs(m) - 1;
    }
    __syncwarp();
    int run = -1;  // last available position of the words before
    for (int wd = 0; wd < nw; ++wd) {
        const int i = wd * 32 + lane;
        const uint32_t m = __shfl_sync(kFull, my_mask, wd);
        if (i < total) {
            int v = 1 << (k.bd - 1);
            if (first >= 0) {
                const uint32_t m0 = m & ((2u << lane) - 1u);
                int j = m0 ? wd * 32 + 31 - __clz(m0) : run;
                if (j < 0) j = first;
                v = ws.f[j];
            }
            ws.s[i] = (uint16_t)v;
        }
        if (m) run = wd * 32 + 31 - __clz(m);
    }
    __syncwarp();
}

// Warps of a k_recon CTA: warp 0 walks luma, chroma is walked by warps 1 and 2
// (one component each: kCW = 2, the default) or by warp 1 (Cb, then Cr: kCW =
// 1), and the last warp moves edge words.  At 4:2:0 a CTU's two chroma walks
// together are shorter than its luma walk, so a picture alone takes as long
// either way; 24 mixed pictures took 4305 us with kCW = 2 and 4597 with kCW = 1,
// and at 4:2:2 and 4:4:4 one warp for both would be the longer chain.
__host__ __device__ constexpr int recon_warps(int kCW) { return 2 + kCW; }

// kFeat: some picture of the launch has slices / tiles, constrained intra
// prediction, cross-component prediction or I_PCM blocks; without them the
// availability, coded and PCM tests compile to the plain form.  fine: a TB
// waits for the edge words it reads; otherwise a CTU waits for all of its
// neighbours' words before its walk.
// How the walk takes the TB at an entry (bits of its word w): it is a plain
// 4x4 TB (kHowTwo: the next one too), it (or the pair) reads neighbour CTUs /
// covers edge words.
constexpr uint32_t kHowTwo = 1u << 6, kHowEdge = 1u << 7, kHowPub = 1u << 14, kHowPlain4 = 1u << 15;
constexpr uint32_t kHowPlain = kTbPlain << 26;

template <int kCW, bool kFeat>
__global__ void __launch_bounds__(32 * recon_warps(kCW), kCW == 1 ? 5 : 4)
k_recon(const DevPic* __restrict__ pics, const CtuItem* __restrict__ items, uint32_t n_items,
        uint32_t* work_counter, uint32_t* dev_err, int cfmt, uint32_t spin_limit, int fine) {
    static_assert(kCW == 1 || kCW == 2, "one or two chroma warps");
    constexpr int kWarps = recon_warps(kCW), kThreads = 32 * kWarps, kWalkers = kWarps - 1;
    extern __shared__ __align__(16) unsigned char smem[];
    const ReconLayout lay(cfmt, kWalkers);
    uint32_t* s_item = (uint32_t*)(smem + lay.off_misc);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // components walked (and listed) by this warp: [c_lo, c_hi], none for the edge warp
    const int c_lo = warp == kWalkers ? 3 : (warp == 0 ? 0 : (kCW == 1 ? 1 : warp));
    const int c_hi = warp == 0 ? 0 : (kCW == 1 ? 2 : warp);
    for (;;) {
        __syncthreads();
        if (tid == 0) *s_item = atomicAdd(work_counter, 1u);
        __syncthreads();
        const uint32_t item = *s_item;
        if (item >= n_items) break;
        const CtuItem it = items[item];
        const DevPic& P = pics[it.pic];
        const int ctb = 1 << P.log2_ctb;
        const int ncomp = P.idc ? 3 : 1;
        const int oxl = it.cx * ctb, oyl = it.cy * ctb;
        // chroma CTU: Scw x Sch samples (4:2:2: half as wide as tall)
        const int ocx = oxl / P.sub_w, ocy = oyl / P.sub_h, Scw = ctb / P.sub_w, Sch = ctb / P.sub_h;
        const uint32_t ci = (uint32_t)it.cy * P.ctb_cols + it.cx;
        uint32_t r0 = P.ctu_start[ci], r1 = P.ctu_start[ci + 1];
        if (r1 > P.n_tus || r0 > r1) {  // malformed CTU range: report, reconstruct nothing
            if (tid == 0) atomicOr(dev_err, DEV_ERR_BITSTREAM);
            r1 = min(r1, P.n_tus);
            r0 = min(r0, r1);
        }
        uint32_t nrec = r1 - r0;
        if (nrec > (uint32_t)lay.rec_cap) {  // more records than a CTU can hold
            if (tid == 0) atomicOr(dev_err, DEV_ERR_BITSTREAM);
            nrec = (uint32_t)lay.rec_cap;
        }
        uint4* recs = (uint4*)(smem + lay.off_can_y);  // until the walk entries are built
        uint4* ents = (uint4*)(smem + lay.off_ents);
        uint32_t* stamp = (uint32_t*)(smem + lay.off_stamp);
        uint32_t* s_have = (uint32_t*)(smem + lay.off_misc) + 1;  // have bits, two words per component
        uint32_t* s_cov = s_have + 6;                             // edge words covered by intra TBs
        uint32_t* s_done = s_cov + 3;                             // walking warps that are done
        uint32_t* s_diff = s_done + 3;                            // the Cb and Cr TBs differ in more than their residual
        uint32_t* s_wcnt = s_diff + 1;                            // TBs found per warp and component
        auto can_of = [&](int c) -> uint16_t* {
            return c == 0 ? (uint16_t*)(smem + lay.off_can_y)
                          : (uint16_t*)(smem + lay.off_can_c) + (size_t)(c - 1) * can_size(lay.cs_w, lay.cs_h);
        };
        // the CTU's records (16 bytes each; the record array is 16-byte aligned)
        for (uint32_t i = tid; i < nrec; i += kThreads) cp_async16(recs + i, P.tus + r0 + i);
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (int i = tid; i < 256; i += kThreads) stamp[i] = kNoStamp;
        if (tid < 3) s_cov[tid] = s_done[tid] = 0u;
        if (tid == 3) *s_diff = 0u;
        if (warp == kWalkers)  // words outside the picture count as present
            for (int c = 0; c < ncomp; ++c) {
                const EdgeGeo e = edge_geo(P, c, it.cx, it.cy);
                const uint32_t t = __ballot_sync(kFull, edge_top_in(e, lane));
                const uint32_t l = __ballot_sync(kFull, edge_left_in(e, lane));
                if (lane == 0) s_have[2 * c] = ~t, s_have[2 * c + 1] = ~l;
            }
        // the CTU's own records have arrived: the decode-order build below
        // runs before the neighbour wait, off the critical path
        cp_async_wait_all();
        __syncthreads();
        // ---- decode order, in parallel: every luma record stamps the 4x4
        // cells it marks decoded (decode.rs:3170-3189; cells outside the
        // picture stay unmarked) ----
        const int vis_w = min(64, P.w - oxl), vis_h = min(64, P.h - oyl);
        const bool intra_pred_ok = !(P.flags & HPVCD_PIC_PRED_IN_PLANE);
        // validity of record i for component tc: -1 skip silently, 0 invalid
        // (reported), 1 usable; (x, y) relative to the CTU
        auto rec_check = [&](const hpvcd_tu& t, int& x, int& y) -> int {
            const int tc = t.comp;
            if (tc >= ncomp || t.log2n < 2 || t.log2n > 6) return -1;
            const int n = 1 << t.log2n;
            x = (int)t.x - (tc ? ocx : oxl);
            y = (int)t.y - (tc ? ocy : oyl);
            const int Sw = tc ? Scw : ctb, Sh = tc ? Sch : ctb;
            return (x < 0 || y < 0 || x + n > Sw || y + n > Sh) ? 0 : 1;
        };
        for (uint32_t base = 32 * warp; base < nrec; base += kThreads) {
            const uint32_t i = base + lane;
            // cell rectangle of a luma record: x | y << 8 | width << 16 | height << 24
            uint32_t rect = 0u;
            if (i < nrec) {
                hpvcd_tu t;
                memcpy(&t, &recs[i], sizeof(t));
                int x, y;
                const int ok = rec_check(t, x, y);
                if (ok == 0) atomicOr(dev_err, DEV_ERR_BITSTREAM);
                if (ok == 1 && t.comp == 0) {
                    const int n = 1 << t.log2n;
                    const int cx = x >> 2, cy = y >> 2;
                    const int w = ((min(x + n, vis_w) + 3) >> 2) - cx, h = ((min(y + n, vis_h) + 3) >> 2) - cy;
                    if (w > 0 && h > 0) {
                        if (w * h <= 4) {
                            for (int u = 0; u < w * h; ++u) {
                                const int yy = u >= w ? (u - w >= w ? (u - 2 * w >= w ? 3 : 2) : 1) : 0;
                                atomicMin(&stamp[(cy + yy) * 16 + cx + u - yy * w], i);
                            }
                        } else {
                            rect = (uint32_t)cx | ((uint32_t)cy << 8) | ((uint32_t)w << 16) | ((uint32_t)h << 24);
                        }
                    }
                }
            }
            // larger blocks by the whole warp
            for (uint32_t m = __ballot_sync(kFull, rect != 0u); m; m &= m - 1u) {
                const int src = __ffs(m) - 1;
                const uint32_t r = __shfl_sync(kFull, rect, src);
                const int cx = (int)(r & 0xffu), cy = (int)((r >> 8) & 0xffu), w = (int)((r >> 16) & 0xffu), h = (int)(r >> 24);
                for (int u = lane; u < 16 * h; u += 32)
                    if ((u & 15) < w) atomicMin(&stamp[(cy + (u >> 4)) * 16 + cx + (u & 15)], base + src);
            }
        }
        // neighbour CTUs that intra prediction may read: same slice and tile
        // (decode.rs:4651-4690)
        uint32_t nb_ok = 0xfu;
        if (kFeat && P.ctb_region) {
            const uint16_t me = P.ctb_region[ci];
            const int cx = it.cx, cy = it.cy;
            auto same = [&](int nx, int ny) {
                return nx >= 0 && ny >= 0 && nx < P.ctb_cols && P.ctb_region[(size_t)ny * P.ctb_cols + nx] == me;
            };
            nb_ok = (same(cx - 1, cy) ? 1u : 0u) | (same(cx - 1, cy - 1) ? 2u : 0u) | (same(cx, cy - 1) ? 4u : 0u) |
                    (same(cx + 1, cy - 1) ? 8u : 0u);
        }
        // Everything one walking warp needs about component c of this CTU.
        auto comp_of = [&](int c) -> Comp {
            Comp k;
            k.S = c ? Scw : ctb;
            k.Sh = c ? Sch : ctb;
            k.ox = c ? ocx : oxl;
            k.oy = c ? ocy : oyl;
            k.pw = c ? P.cw : P.w;
            k.ph = c ? P.ch : P.h;
            k.sw = c ? P.sub_w : 1;
            k.sh = c ? P.sub_h : 1;
            k.nb_ok = nb_ok;
            k.ci_cells = kFeat && (P.flags & HPVCD_PIC_CONSTRAINED_INTRA) ? P.cells : nullptr;
            k.gw = P.gw;
            k.restricted = kFeat && (nb_ok != 0xfu || k.ci_cells != nullptr);
            k.ccp = kFeat && c && (P.flags & HPVCD_PIC_CROSS_COMPONENT);
            k.bd = c ? P.bd_c : P.bd;
            k.max_v = (1 << k.bd) - 1;
            k.luma = c == 0;
            k.filt = c == 0 || P.idc == 3;
            k.smoothing = !(P.flags & HPVCD_PIC_SMOOTHING_DISABLED);
            k.strong = (P.flags & HPVCD_PIC_STRONG_SMOOTHING) != 0;
            k.can = can_of(c);
            k.rs = P.res_stride[c];
            k.res = P.res[c] + (size_t)k.oy * k.rs + k.ox;
            return k;
        };
        __syncthreads();
        // ---- the intra TBs become walk entries, listed per component in decode
        // order: one record per thread, its place from ballots within the
        // warp and the other warps' counts ----
        uint32_t listed[3] = {0u, 0u, 0u};
        for (uint32_t base = 0; base < nrec; base += kThreads) {
            const uint32_t i = base + tid;
            int tc = -1;
            uint4 w = make_uint4(0u, 0u, 0u, 0u);
            if (i < nrec) {
                hpvcd_tu t;
                memcpy(&t, &recs[i], sizeof(t));
                int x, y;
                if ((t.flags & HPVCD_TU_INTRA) && intra_pred_ok && rec_check(t, x, y) == 1) {
                    // The walk stages, reads and writes a TB's samples in words
                    // of up to 16 bytes, and its edge words four samples at a
                    // time: only a TB at a multiple of its size (the only places
                    // a coding quadtree has) is listed.
                    if (t.mode > 34 || t.log2n > 5 || ((x | y) & ((1 << t.log2n) - 1))) {
                        atomicOr(dev_err, DEV_ERR_BITSTREAM);
                    } else {
                        tc = t.comp;
                        const Comp k = comp_of(tc);
                        // a chroma TB with cross-component prediction has a
                        // residual (written by k_ccp) even without coded coefficients
                        const bool coded = (t.flags & HPVCD_TU_CBF) != 0 || (k.ccp && t.res_scale);
                        uint32_t f = kFeat && (t.flags & HPVCD_TU_PCM) ? kTbPcm : 0u;
                        const int n = 1 << t.log2n;
                        const uint32_t run = (1u << (n >> 2)) - 1u;
                        uint32_t cov = 0;
                        if (x + n == k.S) cov |= run << (y >> 2);
                        if (y + n == k.Sh) cov |= run << (16 + (x >> 2));
                        if (cov) {
                            f |= kTbPub;
                            atomicOr(&s_cov[tc], cov);
                        }
                        w = make_entry(k, t, x, y, i, stamp, coded, f);
                    }
                }
            }
            uint32_t pos = 0;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const uint32_t m = __ballot_sync(kFull, tc == c);
                if (tc == c) pos = listed[c] + __popc(m & ((1u << lane) - 1u));
                if (lane == 0) s_wcnt[3 * warp + c] = (uint32_t)__popc(m);
            }
            __syncthreads();
            for (int v = 0; v < kWarps; ++v)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const uint32_t nv = s_wcnt[3 * v + c];
                    if (tc == c && v < warp) pos += nv;
                    listed[c] += nv;
                }
            if (tc >= 0 && pos < (uint32_t)lay.ent_cap(tc)) ents[lay.ent_off(tc) + pos] = w;
            __syncthreads();  // the counts are read, the entries written
        }
#pragma unroll
        for (int c = 0; c < 3; ++c)
            if (listed[c] > (uint32_t)lay.ent_cap(c)) {
                if (tid == 0) atomicOr(dev_err, DEV_ERR_BITSTREAM);
                listed[c] = (uint32_t)lay.ent_cap(c);
            }
        // A CTU without intra TBs (inter pictures) has its final samples in the
        // plane already: it neither waits for its neighbours nor rewrites
        // anything, it only publishes its edge words.
        if (!(listed[0] | listed[1] | listed[2])) {
            for (int c = 0; c < ncomp; ++c) {
                const EdgeGeo e = edge_geo(P, c, it.cx, it.cy);
                const int nr = e.Sh >> 2, nw = nr + (e.S >> 2);
                unsigned long long* words = edge_words(P, it.cx, it.cy, c);
                for (int i = tid; i < nw; i += kThreads) {
                    uint32_t v[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int ax = e.ox + (i < nr ? e.S - 1 : 4 * (i - nr) + u);
                        const int ay = e.oy + (i < nr ? 4 * i + u : e.Sh - 1);
                        v[u] = ax < e.pw && ay < e.ph ? (uint32_t)load_sample(P.rec[c], P.bps, (size_t)ay * e.pw + ax) : 0u;
                    }
                    put_edge(words + i, v[0], v[1], v[2], v[3]);
                }
            }
            continue;
        }
        // Inter pictures: the plane holds motion-compensated + residual
        // samples; load the CTU interior so intra TBs can predict from it.
        if (P.flags & HPVCD_PIC_INTER) {
            for (int c = 0; c < ncomp; ++c) {
                const int S = c ? Scw : ctb, Sh = c ? Sch : ctb, ox = c ? ocx : oxl, oy = c ? ocy : oyl;
                const int pw = c ? P.cw : P.w, ph = c ? P.ch : P.h;
                uint16_t* can = can_of(c);
                const int lq = 28 - __clz(S);  // 8-sample chunks of a row; plane widths are multiples of four
                for (int i = tid; i < Sh << lq; i += kThreads) {
                    const int y = i >> lq, x = 8 * (i & ((1 << lq) - 1));
                    const int ax = ox + x, ay = oy + y;
                    int v[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
                    if (ay < ph) {
                        const size_t at = (size_t)ay * pw + ax;
                        if (ax < pw) ld_row4(P.rec[c], P.bps, at, v[0]);
                        if (ax + 4 < pw) ld_row4(P.rec[c], P.bps, at + 4, v[1]);
                    }
                    *(uint4*)(can + can_in(S, x, y)) =
                        make_uint4((uint32_t)(v[0][0] | (v[0][1] << 16)), (uint32_t)(v[0][2] | (v[0][3] << 16)),
                                   (uint32_t)(v[1][0] | (v[1][1] << 16)), (uint32_t)(v[1][2] | (v[1][3] << 16)));
                }
            }
        }
        if (P.flags & HPVCD_PIC_INTER) __syncthreads();  // the interior before the residuals staged over it
        // ---- residuals into the canvas, before the walk.  In an intra picture
        // every sample of the CTU comes from the walk, so the whole visible
        // residual block of each component is copied by all threads (the areas
        // of uncoded TBs are never read); in an inter picture the canvas holds
        // inter samples, so only the areas of coded intra TBs are staged (a warp
        // each) ----
        if (!(P.flags & HPVCD_PIC_INTER)) {
            for (int c = 0; c < ncomp; ++c) {
                const int S = c ? Scw : ctb, Sh = c ? Sch : ctb, ox = c ? ocx : oxl, oy = c ? ocy : oyl;
                const int rows = min(Sh, (c ? P.ch : P.h) - oy), cols = min(S, (c ? P.cw : P.w) - ox);
                const int lq = 28 - __clz(S);  // 8-sample chunks of a whole CTU row
                const int rs = P.res_stride[c];
                const int16_t* res = P.res[c] + (size_t)oy * rs + ox;
                uint16_t* can = can_of(c);
                for (int i = tid; i < rows << lq; i += kThreads) {
                    const int r = i >> lq, q = i & ((1 << lq) - 1);
                    if (8 * q < cols) cp_async16(can + can_in(S, 8 * q, r), res + (size_t)r * rs + 8 * q);
                }
            }
        } else {
            for (int c = 0; c < ncomp; ++c) {
                const Comp k = comp_of(c);
                const uint4* list = ents + lay.ent_off(c);
                const uint32_t cnt = c == 0 ? listed[0] : (c == 1 ? listed[1] : listed[2]);
                for (uint32_t e = warp; e < cnt; e += kWarps) {
                    const TbEntry E = shared_entry(&list[e]);
                    if (E.coded() && !(E.flags() & kTbPcm)) stage_residual(k, E.n2() >> 1, E.x(), E.y(), lane);
                }
            }
        }
        // ---- how the walk takes each entry, one thread each.  Cb and Cr share a
        // blend table: their TBs have the same places, modes and available
        // lines (a CTU where they do not walks its Cr without the table) ----
        if (tid == 0 && listed[1] != listed[2]) *s_diff = 1u;
        for (int c = 0; c < ncomp; ++c) {
            uint4* list = ents + lay.ent_off(c);
            const uint4* cb_list = ents + lay.ent_off(1);
            const uint32_t cnt = c == 0 ? listed[0] : (c == 1 ? listed[1] : listed[2]);
            for (uint32_t e = tid; e < cnt; e += kThreads) {
                const TbEntry E{list[e]}, F = shared_entry(&list[min(e + 1, cnt - 1)]);
                const uint32_t f = E.flags();
                const bool four = (f & kTbPlain) && E.n2() == 8;
                const bool pair = e + 1 < cnt && four && (F.flags() & kTbPlain) && F.n2() == 8;
                const uint32_t g = pair ? f | F.flags() : f;
                set_how(&list[e], E.w.w | (four ? kHowPlain4 : 0u) | (pair ? kHowTwo : 0u) |
                                      (g & kTbEdge ? kHowEdge : 0u) | (g & kTbPub ? kHowPub : 0u));
                if (c == 2) {
                    const uint4 b = line_entry(&cb_list[min(e, listed[1] ? listed[1] - 1 : 0u)]).w;
                    if (((b.x ^ E.w.x) & ~kTbCoded) | (b.y ^ E.w.y) | (b.z ^ E.w.z)) *s_diff = 1u;
                }
            }
        }
        // ---- the blend tables, by all warps, two TBs at a time ----
        const int half = lane >> 4, l15 = lane & 15;
        for (int c = 0; c < min(ncomp, 2); ++c) {
            const int S = c ? Scw : ctb, row = can_row(S);
            uint32_t* tab = (uint32_t*)(smem + lay.off_tab) + lay.tab_off(c);
            const uint4* list = ents + lay.ent_off(c);
            const uint32_t cnt = c == 0 ? listed[0] : listed[1];
            // the angular words of the next TB are on their way while one is done
            auto angles = [&](const TbEntry& E, uint32_t (&ang)[4]) {
                if (!E.plain()) return;
                const bool four = E.n2() == 8;
                const uint32_t* a = (four ? g_angular.t4[E.mode() - 2] : g_angular.t8[E.mode() - 2]) + l15;
                ang[0] = a[0];
                if (!four) ang[1] = a[16], ang[2] = a[32], ang[3] = a[48];
            };
            uint32_t e = 2 * warp + half;
            TbEntry E{};
            uint32_t ang[4] = {0u, 0u, 0u, 0u};
            if (e < cnt) {
                E = line_entry(&list[e]);
                angles(E, ang);
            }
            while (e < cnt) {
                const uint32_t en = e + 2 * kWarps;
                TbEntry N{};
                uint32_t ang_n[4] = {0u, 0u, 0u, 0u};
                if (en < cnt) {
                    N = line_entry(&list[en]);
                    angles(N, ang_n);
                }
                if (E.plain()) {
                    const Line L(E, row);
                    uint32_t* t = tab + E.tab();
                    if (E.n2() == 8) {
                        t[l15] = blend_word(L, ang[0]);
                    } else {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int x = l15 & 7, y = 2 * u + (l15 >> 3);
                            t[((y >> 2) * (S >> 2) + (x >> 2)) * 16 + (y & 3) * 4 + (x & 3)] = blend_word(L, ang[u]);
                        }
                    }
                }
                E = N;
                e = en;
#pragma unroll
                for (int u = 0; u < 4; ++u) ang[u] = ang_n[u];
            }
        }
        cp_async_wait_all();  // this thread's residual copies; the barrier publishes them
        __syncthreads();
        if (warp == kWalkers)
            edge_service(P, it.cx, it.cy, ncomp, can_of, s_cov, s_have, s_done, kWalkers, lane);
        // ---- decode-order walk: each warp reconstructs its components ----
        WalkScratch& ws = *(WalkScratch*)(smem + lay.off_ws + (size_t)min(warp, kWalkers - 1) * kWsBytes);
        for (int c = c_lo; c <= c_hi && c < ncomp; ++c) {
            const Comp k = comp_of(c);
            const uint32_t cnt = c == 0 ? listed[0] : (c == 1 ? listed[1] : listed[2]), last = cnt ? cnt - 1 : 0u;
            const uint4* list = ents + lay.ent_off(c);
            // (a walk without the table takes every TB by its line)
            const uint32_t how_mask = c == 2 && *s_diff ? ~(kHowPlain | kHowPlain4 | kHowTwo) : 0xffffffffu;
            const uint32_t* tab = (const uint32_t*)(smem + lay.off_tab) + lay.tab_off(c);
            uint16_t* const can = k.can;
            const int row = can_row(k.S), max_v = k.max_v;
            const bool luma = c == 0;
            unsigned long long* const words = edge_words(P, it.cx, it.cy, c);
            const int px4 = ((lane >> 2) & 3) * row + (lane & 3), px8 = (lane >> 2) * row + 2 * (lane & 3);
            // this lane's pair of samples in the blend table of an 8x8 TB
            const int tab8 = ((lane >> 4) * (k.S >> 2) + ((lane >> 1) & 1)) * 16 + ((lane >> 2) & 3) * 4 + 2 * (lane & 1);
            Have have{0u, 0u};
            if (!fine && cnt) have = wait_edges(have, 0xffffffffu, 0xffffffffu, s_have + 2 * c, spin_limit, dev_err, lane);
            // The edge words a TB reads: with x = 0 the left column from row
            // y - 1 on, with y = 0 the row above from sample x - 1 on.
            auto await = [&](const TbEntry& E) {
                const int x = E.x(), y = E.y(), n2 = E.n2();
                uint32_t need_top = 0u, need_left = 0u;
                if (y == 0) {
                    const int lo = max(x - 1, 0) >> 2, hi = (x + n2) >> 2;
                    need_top = (0xffffffffu >> (32 - (hi - lo))) << lo;
                }
                if (x == 0) {
                    const int lo = max(y - 1, 0) >> 2, hi = min(y + n2, k.Sh) >> 2;
                    need_left = ((1u << (hi - lo)) - 1u) << lo;
                    if (y == 0) need_left |= kHaveCorner;
                }
                need_top = __reduce_or_sync(kFull, need_top & ~have.top);
                need_left = __reduce_or_sync(kFull, need_left & ~have.left);
                if (need_top | need_left)
                    have = wait_edges(have, need_top, need_left, s_have + 2 * c, spin_limit, dev_err, lane);
            };
            // Plain 4x4 TBs are taken in pairs: lanes 0..15 hold TB e, lanes
            // 16..31 TB e + 1, predicted after TB e is stored.  The pair's
            // blend words and place are loaded an iteration ahead.
            uint32_t how = 0, bw = 0, place = 0;  // flags, blend word, word x of the entry
            auto fetch = [&](uint32_t e) { return *(const uint2*)&list[min(e + half, last)]; };
            auto how_of = [&](uint32_t e) { return list[min(e, last)].w & how_mask; };
            if (cnt) {
                const uint2 h = fetch(0);
                place = h.x;
                bw = tab[(h.y >> 16) + l15];
                how = how_of(0);
            }
            // Samples s of the half-warps' 4x4 TBs that lie on the CTU's right
            // column or bottom row.
            auto publish4 = [&](int s, uint32_t entry) {
                const TbEntry E{list[entry]};
                uint16_t* const w16 = (uint16_t*)words;
                const int x = E.x() + (lane & 3), y = E.y() + (l15 >> 2);
                const uint16_t t = (uint16_t)(s | 0x8000);
                if (x == k.S - 1) st_edge16(w16 + y, t);
                if (y == k.Sh - 1) st_edge16(w16 + k.Sh + x, t);
            };
            for (uint32_t e = 0; e < cnt;) {
                if (how & kHowTwo) {
                    if (how & kHowEdge) await(TbEntry{list[e + half]});
                    uint16_t* const px = can + (place & 0xffffu) + px4;
                    const int rv = (place & kTbCoded) ? (int)(int16_t)*px : 0;
                    int s = __viaddmin_s32_relu(blend_of(can, bw), rv, max_v);
                    if (half == 0) *px = (uint16_t)s;
                    const uint2 h = fetch(e + 2);
                    const uint32_t hn = how_of(e + 2);
                    __syncwarp();
                    s = __viaddmin_s32_relu(blend_of(can, bw), rv, max_v);  // (the first TB's lanes: the same again)
                    if (half) *px = (uint16_t)s;
                    place = h.x;
                    bw = tab[(h.y >> 16) + l15];
                    if (how & kHowPub) publish4(s, e + half);
                    how = hn;
                    e += 2;
                    __syncwarp();
                    continue;
                }
                const uint2 h = fetch(e + 1);
                const uint32_t hn = how_of(e + 1);
                TbEntry E{list[e]};
                if (how & kHowEdge) await(E);
                const int n2 = E.n2();
                if ((how & kHowPlain) && !(how & kHowPlain4)) {
                    walk_plain8(can, (uint32_t*)(can + E.org() + px8), *(const uint2*)(tab + E.tab() + tab8), E.coded(),
                                max_v);
                } else {
                    const uint32_t f = E.flags();
                    const int mode = E.mode();
                    int stride = row;
                    if (f & kTbGather) {
                        gather_line(k, 31 - __clz(n2) - 1, E.x(), E.y(), stamp, E.jrec(), ws, lane);
                        const uint32_t at = (uint32_t)(ws.s - can);  // position i at canvas offset at + i
                        E.w.x = (E.w.x & (0xffffu | kTbCoded)) | (at << 16);
                        E.w.y = (E.w.y & 0xffff0000u) | (at + (uint32_t)n2);
                        stride = -1;
                    }
                    const Line L(E, stride);
                    const bool coded = E.coded(), filt = (E.w.z & kTbFilt) != 0u;
                    if (kFeat && (f & kTbPcm)) {
                        pcm_tb(k, 31 - __clz(n2) - 1, E.x(), E.y(), lane);
                    } else if (n2 == 8) {
                        // positions past the line clamp to its last one
                        walk_tb4(can + E.org() + px4, mode, coded, luma, max_v, can[L.at(lane)], lane);
                    } else if (n2 == 16) {
                        const bool hi_ok = (f & kTbHi32) != 0u;
                        walk_tb8((uint32_t*)(can + E.org() + px8), mode, coded, filt, luma, max_v, can[L.at(lane)],
                                 hi_ok ? can[E.corner() + 16] : 0, hi_ok,
                                 *(const uint2*)&g_angular.t8[max(mode - 2, 0)][2 * lane], lane);
                    } else {
                        walk_tb_big(can, row, L, E.org(), mode, coded, filt, luma, k.strong, k.bd, ws, lane);
                    }
                }
                const uint32_t was = how;
                ++e;
                how = hn;
                place = h.x;
                bw = tab[(h.y >> 16) + l15];
                if (was & kHowPub) publish_tb(can, row, k.S, k.Sh, E.x(), E.y(), n2 >> 1, words, lane);
            }
        }
        if (warp < kWalkers && lane == 0) *(volatile uint32_t*)&s_done[warp] = 1u;
        __syncthreads();
        // ---- write the CTU out for the filters (8 samples per store when
        // rows allow); the kernel boundary orders it before them ----
        for (int c = 0; c < ncomp; ++c) {
            const int S = c ? Scw : ctb, Sh = c ? Sch : ctb, ox = c ? ocx : oxl, oy = c ? ocy : oyl;
            const int pw = c ? P.cw : P.w, ph = c ? P.ch : P.h;
            const uint16_t* can = can_of(c);
            const int rows = min(Sh, ph - oy), cols = min(S, pw - ox);
            if ((pw & 7) == 0 && (cols & 7) == 0) {
                const int lq = 28 - __clz(S);
                for (int i = tid; i < rows << lq; i += kThreads) {
                    const int y = i >> lq, q = i & ((1 << lq) - 1);
                    if (8 * q >= cols) continue;
                    const uint4 v = *(const uint4*)(can + can_in(S, 8 * q, y));
                    const size_t off = (size_t)(oy + y) * pw + ox + 8 * q;
                    if (P.bps == 2) {
                        *(uint4*)((uint16_t*)P.rec[c] + off) = v;
                    } else {
                        const uint32_t lo = (v.x & 0xffu) | ((v.x >> 8) & 0xff00u) | ((v.y & 0xffu) << 16) |
                                            ((v.y & 0xff0000u) << 8);
                        const uint32_t hi = (v.z & 0xffu) | ((v.z >> 8) & 0xff00u) | ((v.w & 0xffu) << 16) |
                                            ((v.w & 0xff0000u) << 8);
                        *(uint2*)((uint8_t*)P.rec[c] + off) = make_uint2(lo, hi);
                    }
                }
            } else {
                for (int i = tid; i < rows * cols; i += kThreads) {
                    const int y = i / cols, x = i % cols;
                    store_sample(P.rec[c], P.bps, (size_t)(oy + y) * pw + ox + x, can[can_in(S, x, y)]);
                }
            }
        }
    }
}

}  // namespace hpvcd

extern "C" size_t hpvcd_recon_smem_bytes(int cfmt, int chroma_warps) {
    return hpvcd::ReconLayout(cfmt, hpvcd::recon_warps(chroma_warps == 1 ? 1 : 2) - 1).total;
}

extern "C" cudaError_t hpvcd_launch_residual(const hpvcd::DevPic* pics, const uint32_t* rec_prefix,
                                             uint32_t n_pics, uint32_t total_records, uint32_t* dev_err,
                                             int sms, int idct, cudaStream_t stream) {
    if (total_records == 0) return cudaSuccess;
    // Records of a CTA step: at least kResMinChunk (a warp's worth), doubled
    // while twice as many still give every SM a step, so that a small picture
    // spreads over the whole chip and a large one fills the lanes of its 4x4
    // tasks and keeps to one class for long (4032x3024 grid, whole call: 559
    // us, 571 with two steps per SM and 604 with four; 24 mixed pictures
    // 3937 to 3951 in all three).
    constexpr uint32_t kResMinChunk = 32;
    uint32_t chunk = kResMinChunk;
    while (chunk < hpvcd::kResMaxChunk && total_records / (2 * chunk) >= (uint32_t)sms) chunk *= 2;
    const uint32_t steps = (total_records + chunk - 1) / chunk;
    const uint32_t cap = (uint32_t)sms * 4u;  // resident CTAs
    const int grid = (int)(steps < cap ? steps : cap), threads = hpvcd::kResWarps * 32;
    // schedule value: 0 integer tensor cores (the default), 1 butterflies, 2 matrix product
    if (idct == 0)
        hpvcd::k_residual<hpvcd::kIdctTensor><<<grid, threads, 0, stream>>>(pics, rec_prefix, n_pics, dev_err, chunk);
    else if (idct == 1)
        hpvcd::k_residual<hpvcd::kIdctButterfly><<<grid, threads, 0, stream>>>(pics, rec_prefix, n_pics, dev_err,
                                                                             chunk);
    else
        hpvcd::k_residual<hpvcd::kIdctMatrix><<<grid, threads, 0, stream>>>(pics, rec_prefix, n_pics, dev_err, chunk);
    hpvcd_note_launches(1);
    return cudaGetLastError();
}

extern "C" cudaError_t hpvcd_launch_ccp(const hpvcd::DevPic* pics, const uint32_t* rec_prefix, uint32_t n_pics,
                                        uint32_t total_records, uint32_t* dev_err, int sms, cudaStream_t stream) {
    if (total_records == 0) return cudaSuccess;
    const uint32_t blocks_needed = (total_records + hpvcd::kCcpWarps - 1) / hpvcd::kCcpWarps;
    const uint32_t cap = (uint32_t)sms * 8u;
    const int grid = (int)(blocks_needed < cap ? blocks_needed : cap);
    hpvcd::k_ccp<<<grid, hpvcd::kCcpWarps * 32, 0, stream>>>(pics, rec_prefix, n_pics, dev_err);
    hpvcd_note_launches(1);
    return cudaGetLastError();
}

extern "C" cudaError_t hpvcd_launch_recon(const hpvcd::DevPic* pics, const hpvcd::CtuItem* items,
                                          uint32_t n_items, uint32_t* work_counter, uint32_t* dev_err,
                                          int cfmt, int grid, int chroma_warps, int feat, int fine, uint32_t spin,
                                          cudaStream_t stream) {
    if (n_items == 0) return cudaSuccess;
    // the dynamic shared-memory limit was raised by hpvcd_recon_occupancy()
    // when the plan was built (no non-stream API call here, so launches can
    // be captured into CUDA graphs)
    const int cw = chroma_warps == 1 ? 1 : 2;  // walking warps for chroma
    const size_t smem = hpvcd::ReconLayout(cfmt, hpvcd::recon_warps(cw) - 1).total;
    const int threads = 32 * hpvcd::recon_warps(cw);
    // default: 2^22 polls of up to 64 ns each bound one wait to a few hundred ms
    if (spin == 0) spin = 1u << 22;
    if (cw == 2 && feat)
        hpvcd::k_recon<2, true><<<grid, threads, smem, stream>>>(pics, items, n_items, work_counter, dev_err, cfmt,
                                                                 spin, fine);
    else if (cw == 2)
        hpvcd::k_recon<2, false><<<grid, threads, smem, stream>>>(pics, items, n_items, work_counter, dev_err, cfmt,
                                                                  spin, fine);
    else if (feat)
        hpvcd::k_recon<1, true><<<grid, threads, smem, stream>>>(pics, items, n_items, work_counter, dev_err, cfmt,
                                                                 spin, fine);
    else
        hpvcd::k_recon<1, false><<<grid, threads, smem, stream>>>(pics, items, n_items, work_counter, dev_err, cfmt,
                                                                  spin, fine);
    hpvcd_note_launches(1);
    return cudaGetLastError();
}

namespace {
// Every instantiation: the shared-memory limit of the 4:4:4 layout of three
// warps (the largest) and the whole unified L1 / shared array as shared
// memory.  The common carveout matters when waves of different layouts
// (4:2:0 and 4:4:4, one stream per concurrent group of a batch) follow each
// other on the SMs: an SM changes its L1 / shared split only when it holds
// no CTA, so a wave that wanted a larger split than the one running could
// start only once the other groups' waves had drained every SM.
template <int kCW, bool kFeat>
void recon_attrs(int lim) {
    cudaFuncSetAttribute(hpvcd::k_recon<kCW, kFeat>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
    cudaFuncSetAttribute(hpvcd::k_recon<kCW, kFeat>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxShared);
}

// Occupancy of one build with the layout of `cfmt` (attributes already set).
int recon_occupancy_of(int cfmt, int cw) {
    int blocks = 0;
    const size_t smem = hpvcd::ReconLayout(cfmt, hpvcd::recon_warps(cw) - 1).total;
    if (cw == 2)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, hpvcd::k_recon<2, false>, 32 * hpvcd::recon_warps(2),
                                                      smem);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, hpvcd::k_recon<1, false>, 32 * hpvcd::recon_warps(1),
                                                      smem);
    return blocks;
}

// Attributes and occupancies are set up once per device: every plan build
// asks for them, and a serving loop builds a plan for every new batch
// layout (setting the attributes of every instantiation each time cost
// milliseconds per plan).  Like the no-allocation entry point's per-device
// set-up, this assumes the device's primary context lives until the process
// exits (no cudaDeviceReset while the library is in use).
constexpr int kAttrDevices = 64;
std::mutex g_attr_mu;
bool g_attr_done[kAttrDevices];
int g_attr_occ[kAttrDevices][3][2];
}  // namespace

// CTAs per SM of the wavefront kernel with the layout of `cfmt` and
// `chroma_warps` (1 or 2) walking warps for chroma; the first call on a device
// sets the attributes of every instantiation (recon_attrs) and of the residual
// kernel.
extern "C" int hpvcd_recon_occupancy(int cfmt, int chroma_warps) {
    const int cw = chroma_warps == 1 ? 1 : 2;
    const int cf = cfmt >= 0 && cfmt <= 2 ? cfmt : 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kAttrDevices) {
        cudaGetLastError();
        dev = -1;
    }
    std::lock_guard<std::mutex> lock(g_attr_mu);
    if (dev >= 0 && g_attr_done[dev]) return g_attr_occ[dev][cf][cw - 1];
    const int lim = (int)hpvcd::ReconLayout(hpvcd::kFmt444, hpvcd::recon_warps(2) - 1).total;
    recon_attrs<1, false>(lim);
    recon_attrs<2, false>(lim);
    recon_attrs<1, true>(lim);
    recon_attrs<2, true>(lim);
    // the residual pre-pass of one group runs beside another group's waves
    cudaFuncSetAttribute(hpvcd::k_residual<hpvcd::kIdctMatrix>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxShared);
    cudaFuncSetAttribute(hpvcd::k_residual<hpvcd::kIdctButterfly>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxShared);
    cudaFuncSetAttribute(hpvcd::k_residual<hpvcd::kIdctTensor>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxShared);
    if (dev < 0) return recon_occupancy_of(cf, cw);
    for (int f = 0; f < 3; ++f)
        for (int b = 1; b <= 2; ++b) g_attr_occ[dev][f][b - 1] = recon_occupancy_of(f, b);
    g_attr_done[dev] = true;
    return g_attr_occ[dev][cf][cw - 1];
}
