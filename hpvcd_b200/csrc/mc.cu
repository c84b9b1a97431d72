// mc.cu -- motion compensation (mc.rs + decode.rs:7000-7488 motion_compensate).
//
// PUs are cut into 8x8 luma tiles (and the chroma they cover).  Eight lanes
// take a tile: together they copy the reference blocks of both lists to shared
// memory in 16-byte chunks (asynchronously, so that a tile waits for memory
// once), then one column each, a lane filters its column's rows horizontally
// (8-tap luma quarter-pel, 4-tap chroma eighth-pel, mc.rs:351-530) and adds
// each row's 14-bit intermediate to the outputs it reaches vertically, so a
// tile needs 15 horizontal sums a column instead of 64 and every sum is two
// (8-bit) or four (above) packed dot products.  Then the uni / bi / explicitly
// weighted combination with clipping (mc.rs:538-736), plus the residual,
// written into the current picture's plane.  Bound by memory latency at 32
// warps an SM, then by instruction issue (0.52 a cycle).  A 1920x1080 frame of
// the synthetic GOP: 135 us with one thread per output sample filtering 64
// loads, 55 with each lane loading its own rows, 43 with the shared blocks.
#include "common.cuh"

namespace hpvcd {

// mc.rs:30-45, four taps per word
__constant__ uint32_t c_luma_filter[4][2] = {{0x40000000u, 0x00000000u},   // 0 0 0 64, 0 0 0 0
                                             {0x3af604ffu, 0x0001fb11u},   // -1 4 -10 58, 17 -5 1 0
                                             {0x28f504ffu, 0xff04f528u},   // -1 4 -11 40, 40 -11 4 -1
                                             {0x11fb0100u, 0xff04f63au}};  // 0 1 -5 17, 58 -10 4 -1
__constant__ uint32_t c_chroma_filter[8] = {0x00004000u, 0xfe0a3afeu, 0xfe1036fcu, 0xfc1c2efau,
                                            0xfc2424fcu, 0xfa2e1cfcu, 0xfc3610feu, 0xfe3a0afeu};

__device__ __forceinline__ int tap(uint32_t w, int t) { return (int)(int8_t)(w >> (8 * t)); }
__device__ __forceinline__ int dot4(uint32_t a, uint32_t b, int c) {  // unsigned samples x signed taps
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ int dot2lo(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp2a.lo.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ int dot2hi(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp2a.hi.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// The reference block of a tile of LANES columns: every row as the 16-byte
// chunks that hold its LANES + TAPS - 1 samples, kept at their own alignment.
template <int TAPS, int LANES, int BPS>
struct Block {
    static constexpr int kCols = LANES + TAPS - 1, kChunks = (kCols * BPS + 15 - BPS) / 16 + 1;
    static constexpr int kRowBytes = 16 * kChunks;
};
// bytes of an eight-lane group's block of one list (16-bit luma: 15 rows of
// 48; 16-bit 4:2:2 chroma: two components of 11 rows of 32); the groups of a
// warp start in different banks
constexpr int kBlockBytes = 720, kHalfBlock = 352, kMcWarps = 8;
constexpr int kListBytes = 4 * kMcWarps * kBlockBytes;  // all groups' blocks of one list

// Start to fetch the block's rows from (x, y), column 0 of lane 0 with its
// taps, by its LANES lanes together; outside the picture sample by sample, the
// first and last row and column repeated (mc.rs:310).
template <int TAPS, int ROWS, int LANES, int BPS>
__device__ __forceinline__ void fetch_block(const void* plane, int pw, int ph, int x, int y, char* buf, int q) {
    using B = Block<TAPS, LANES, BPS>;
    constexpr int kRows = ROWS + TAPS - 1, kLoads = (kRows * B::kChunks + LANES - 1) / LANES;
    const uintptr_t col = (uintptr_t)plane + (intptr_t)x * BPS;
    if (x >= 0 && x + B::kCols <= pw) {
#pragma unroll
        for (int k = 0; k < kLoads; ++k) {
            const int i = q + k * LANES, r = i / B::kChunks, j = i - r * B::kChunks;
            const uintptr_t a = col + (size_t)clamp3i(y + r, 0, ph - 1) * pw * BPS;
            // an aligned chunk that holds a sample of the plane lies in its allocation
            if (r < kRows && 16 * j < (int)(a & 15) + B::kCols * BPS) {
                const uint32_t d = (uint32_t)__cvta_generic_to_shared(buf + 16 * i);
                const uintptr_t from = (a & ~(uintptr_t)15) + 16 * j;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(from) : "memory");
            }
        }
    } else {
#pragma unroll 1
        for (int i = q; i < kRows * B::kCols; i += LANES) {
            const int r = i / B::kCols, c = i - r * B::kCols;
            const size_t row = (size_t)clamp3i(y + r, 0, ph - 1) * pw;
            char* d = buf + r * B::kRowBytes + (int)((col + row * BPS) & 15) + c * BPS;
            const int smp = load_sample(plane, BPS, row + clamp3i(x + c, 0, pw - 1));
            if (BPS == 1) *(uint8_t*)d = (uint8_t)smp; else *(uint16_t*)d = (uint16_t)smp;
        }
    }
}

// The 14-bit intermediates (int16) of ROWS vertically adjacent samples of lane
// q's column; (x, y) is the reference sample of lane 0's first.  A zero
// fraction is the tap 64 alone, which gives the reference's unfiltered cases
// exactly: (64 r) >> (bd - 8) loses no bit for bd <= 14, and (64 h) >> 6 = h.
template <int TAPS, int ROWS, int LANES, int BPS>
__device__ __forceinline__ void interp_column(const void* plane, int pw, int ph, int x, int y, int fx, int fy, int bd,
                                              const char* buf, int q, int (&out)[ROWS]) {
    using B = Block<TAPS, LANES, BPS>;
    constexpr int back = TAPS / 2 - 1, W = TAPS * BPS / 4;
    const int s1 = bd - 8;
    const uint32_t h0 = TAPS == 8 ? c_luma_filter[fx][0] : c_chroma_filter[fx], h1 = TAPS == 8 ? c_luma_filter[fx][1] : 0u;
    const uint32_t v0 = TAPS == 8 ? c_luma_filter[fy][0] : c_chroma_filter[fy], v1 = TAPS == 8 ? c_luma_filter[fy][1] : 0u;
    int vt[TAPS];
#pragma unroll
    for (int t = 0; t < TAPS; ++t) vt[t] = t < 4 ? tap(v0, t) : tap(v1, t & 3);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) out[r] = 0;
    const uint32_t col = (uint32_t)(uintptr_t)plane + (uint32_t)((x - back) * BPS), pitch = (uint32_t)(pw * BPS);
#pragma unroll
    for (int r = 0; r < ROWS + TAPS - 1; ++r) {
        const uint32_t at = ((col + (uint32_t)clamp3i(y - back + r, 0, ph - 1) * pitch) & 15u) + q * BPS;
        const uint32_t* src = (const uint32_t*)(buf + r * B::kRowBytes) + (at >> 2);
        uint32_t w[W + 1];
#pragma unroll
        for (int i = 0; i <= W; ++i) w[i] = src[i];
#pragma unroll
        for (int i = 0; i < W; ++i) w[i] = __funnelshift_r(w[i], w[i + 1], 8 * (at & 3));
        int h;
        if constexpr (BPS == 1) {
            h = dot4(w[0], h0, 0);
            if constexpr (TAPS == 8) h = dot4(w[1], h1, h);
        } else {
            h = dot2hi(w[1], h0, dot2lo(w[0], h0, 0));
            if constexpr (TAPS == 8) h = dot2hi(w[3], h1, dot2lo(w[2], h1, h));
        }
        h >>= s1;  // intermediate kept in i32 (mc.rs:408-418)
#pragma unroll
        for (int t = 0; t < TAPS; ++t)
            if (r - t >= 0 && r - t < ROWS) out[r - t] += vt[t] * h;
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) out[r] = (int)(int16_t)(out[r] >> 6);
}

// Lane q's column of a tile of component c whose first sample is (x, y): ROWS
// samples, of which `rows` are written (none by a lane outside the PU).  The
// eight lanes of a group come here together, one tile of eight lanes or two of
// four.
template <int TAPS, int ROWS, int LANES, int BPS>
__device__ __forceinline__ void mc_column(const DevPic& P, const hpvcd_pu& u, const void* const (*refs)[3], int c, int x, int y,
                                          int rows, char* buf) {
    const int q = threadIdx.x & (LANES - 1);
    const unsigned group = ((1u << LANES) - 1) << (threadIdx.x & 31 & ~(LANES - 1));
    const unsigned owners = 0xffu << (threadIdx.x & 24);  // the eight lanes whose tiles share buf
    static_assert((ROWS + TAPS - 1) * Block<TAPS, LANES, BPS>::kRowBytes <= (LANES == 8 ? kBlockBytes : kHalfBlock),
                  "the block fits its group's bytes");
    constexpr bool luma = TAPS == 8;
    constexpr int back = TAPS / 2 - 1;
    const int pw = luma ? P.w : P.cw, ph = luma ? P.h : P.ch;
    const int bd = luma ? P.bd : P.bd_c;
    const int mx = (1 << bd) - 1;
    auto vector = [&](int l, int& ix, int& iy, int& fx, int& fy) {
        if (luma) {
            ix = u.mv[l][0] >> 2, iy = u.mv[l][1] >> 2;
            fx = u.mv[l][0] & 3, fy = u.mv[l][1] & 3;
        } else {  // decode.rs:7282-7287, Rust `/` truncates toward zero like C
            const int mvcx = u.mv[l][0] * 2 / P.sub_w, mvcy = u.mv[l][1] * 2 / P.sub_h;
            ix = mvcx >> 3, iy = mvcy >> 3;
            fx = mvcx & 7, fy = mvcy & 7;
        }
    };
    // The blocks before are read, by every lane that shares the bytes: a chroma
    // tile's four lanes write where all eight read a luma block.
    __syncwarp(owners);
#pragma unroll 1
    for (int l = 0; l < 2; ++l) {
        const void* const ref = refs[l][c];
        if (!ref) continue;
        int ix, iy, fx, fy;
        vector(l, ix, iy, fx, fy);
        fetch_block<TAPS, ROWS, LANES, BPS>(ref, pw, ph, x + ix - back, y + iy - back, buf + l * kListBytes, q);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp(group);
    int a[ROWS], b[ROWS];  // the lists found, in turn
    int have = 0;
#pragma unroll 1
    for (int l = 0; l < 2; ++l) {
        const void* const ref = refs[l][c];
        if (!ref) continue;
        have |= 1 << l;
        int ix, iy, fx, fy;
        vector(l, ix, iy, fx, fy);
        int t[ROWS];
        interp_column<TAPS, ROWS, LANES, BPS>(ref, pw, ph, x + ix, y + iy, fx, fy, bd, buf + l * kListBytes, q, t);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            b[r] = t[r];
            if (l == 0) a[r] = t[r];
        }
    }
    const int denom = P.has_wp ? (luma ? P.wp.luma_log2_denom : P.wp.chroma_log2_denom) : 0;
    auto wpair = [&](int l, int& wgt, int& off) {
        const hpvcd_wp_entry& e = P.wp.e[l][max((int)u.ref_idx[l], 0)];
        wgt = luma ? e.luma_w : (c == 1 ? e.cb_w : e.cr_w);
        off = luma ? e.luma_o : (c == 1 ? e.cb_o : e.cr_o);
    };
    int v[ROWS];
    if (have == 3) {
        if (P.has_wp) {  // mc.rs:682-736
            int w0, o0, w1, o1;
            wpair(0, w0, o0);
            wpair(1, w1, o1);
            const int log2_wd = denom + 14 - bd;
            const long long rnd = ((long long)o0 + o1 + 1) << log2_wd;
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const long long t = ((long long)a[r] * w0 + (long long)b[r] * w1 + rnd) >> (log2_wd + 1);
                v[r] = (int)(t < 0 ? 0 : (t > mx ? mx : t));
            }
        } else {  // mc.rs:579-629
            const int shift = 15 - bd;
#pragma unroll
            for (int r = 0; r < ROWS; ++r) v[r] = clamp3i((a[r] + b[r] + (1 << (shift - 1))) >> shift, 0, mx);
        }
    } else if (have) {
        if (have == 2) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) a[r] = b[r];
        }
        if (P.has_wp) {  // mc.rs:631-680
            int wg, of;
            wpair(have == 1 ? 0 : 1, wg, of);
            const int log2_wd = denom + 14 - bd;
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const int t = log2_wd >= 1 ? ((a[r] * wg + (1 << (log2_wd - 1))) >> log2_wd) + of : a[r] * wg + of;
                v[r] = clamp3i(t, 0, mx);
            }
        } else {  // mc.rs:538-577
            const int shift = 14 - bd;
#pragma unroll
            for (int r = 0; r < ROWS; ++r) v[r] = clamp3i((a[r] + (shift > 0 ? 1 << (shift - 1) : 0)) >> shift, 0, mx);
        }
    } else {  // decode.rs:7206-7216: missing reference -> mid-grey
#pragma unroll
        for (int r = 0; r < ROWS; ++r) v[r] = 1 << (bd - 1);
    }
    // the residual (k_residual; zero without one) is added here, reconstruct.rs:214-251
    void* dst = P.rec[c];
    const int rs = P.res_stride[c];
    const int16_t* res = P.res[c] + (size_t)y * rs + x + q;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) a[r] = r < rows ? (int)res[(size_t)r * rs] : 0;
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
        if (r < rows) store_sample(dst, BPS, (size_t)(y + r) * pw + x + q, clamp3i(v[r] + a[r], 0, mx));
}

// A CTA takes kMcPus consecutive PUs; blockIdx.y = its share of their tiles
// (kMcSplit CTAs interleave, so that a run of large PUs does not end up on one
// SM).  A warp takes four tiles of luma, or of both chroma components, at a
// time.
constexpr int kMcPus = 32, kMcSplit = 12;

template <int BPS>
__device__ __forceinline__ void mc_tiles(const DevPic& P, const hpvcd_pu* s_pu, const uint32_t* s_pre,
                                         const void* const (*s_ref)[2][3], char* block) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 3, l = lane & 7;
    const uint32_t tiles = s_pre[kMcPus], groups = (tiles + 3) / 4;
    const uint32_t tasks = P.idc ? 2 * groups : groups;
    char* buf = block + (threadIdx.x >> 3) * kBlockBytes;
    for (uint32_t t = blockIdx.y * kMcWarps + warp; t < tasks; t += kMcSplit * kMcWarps) {
        const bool luma = t < groups;
        const uint32_t tile = (luma ? t : t - groups) * 4 + g;
        if (tile >= tiles) continue;
        int j = 0;
#pragma unroll
        for (int step = kMcPus / 2; step; step >>= 1)
            if (s_pre[j + step] <= tile) j += step;
        const hpvcd_pu u = s_pu[j];
        const int k = (int)(tile - s_pre[j]), tw = (u.w + 7) >> 3;
        const int ty = k / tw, tx = k - ty * tw;
        if (luma) {
            const int x = u.x + 8 * tx, y = u.y + 8 * ty;
            const int rows = 8 * tx + l < u.w && x + l < P.w ? min(min((int)u.h - 8 * ty, 8), P.h - y) : 0;
            mc_column<8, 8, 8, BPS>(P, u, s_ref[j], 0, x, y, rows, buf);
        } else {
            const int sw = P.sub_w, sh = P.sub_h, cols = 8 / sw, q = l & (cols - 1);
            const int ox = cols * tx, oy = 8 / sh * ty;
            const int x = u.x / sw + ox, y = u.y / sh + oy;
            const int rows = ox + q < u.w / sw && x + q < P.cw ? min(min(u.h / sh - oy, 8 / sh), P.ch - y) : 0;
            char* half = buf + (l >> 2) * kHalfBlock;
            if (sw == 1) {  // 4:4:4: both components by every lane
                for (int c = 1; c < 3; ++c) mc_column<4, 8, 8, BPS>(P, u, s_ref[j], c, x, y, rows, buf);
            } else if (sh == 1) {
                mc_column<4, 8, 4, BPS>(P, u, s_ref[j], 1 + (l >> 2), x, y, rows, half);
            } else {
                mc_column<4, 4, 4, BPS>(P, u, s_ref[j], 1 + (l >> 2), x, y, rows, half);
            }
        }
    }
}

__global__ void __launch_bounds__(32 * kMcWarps, 4) k_mc(const DevPic* __restrict__ pics, int pic_index) {
    __shared__ __align__(16) char block[2 * kListBytes];
    __shared__ hpvcd_pu s_pu[kMcPus];
    __shared__ uint32_t s_pre[kMcPus + 1];  // tiles of the PUs before
    // reference planes of the PUs by list and component, NULL where there is
    // none (looked up here once: in the tasks it was two dependent loads before
    // the first sample)
    __shared__ const void* s_ref[kMcPus][2][3];
    static_assert(kMcPus == 32, "one PU per lane");
    const DevPic& P = pics[pic_index];
    const uint32_t first = blockIdx.x * kMcPus;
    if (threadIdx.x < 32) {
        uint32_t n = 0;
        if (threadIdx.x < kMcPus && first + threadIdx.x < P.n_pus) {
            const hpvcd_pu u = P.pus[first + threadIdx.x];
            s_pu[threadIdx.x] = u;
            n = ((u.w + 7u) >> 3) * ((u.h + 7u) >> 3);
#pragma unroll
            for (int l = 0; l < 2; ++l) {  // reference views per list (decode.rs:7040-7120 ref_frame_for_lists)
                const int ri = u.ref_idx[l];
                int rp = -1;
                if ((u.flags & (l ? HPVCD_PU_L1 : HPVCD_PU_L0)) && ri >= 0 && ri < HPVCD_MAX_REFS) rp = P.ref_pic[l][ri];
                // the host maps references to earlier pictures of the batch (< pic_index)
                // or to DPB pictures appended after the batch's own; -1 is none
                if (rp == pic_index) rp = -1;
#pragma unroll
                for (int c = 0; c < 3; ++c) s_ref[threadIdx.x][l][c] = rp >= 0 ? pics[rp].fin[c] : nullptr;
            }
        }
        for (int d = 1; d < kMcPus; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, n, d);
            if ((int)threadIdx.x >= d) n += o;
        }
        if (threadIdx.x < kMcPus) s_pre[threadIdx.x + 1] = n;
        if (threadIdx.x == 0) s_pre[0] = 0u;
    }
    __syncthreads();
    if (P.bps == 1)
        mc_tiles<1>(P, s_pu, s_pre, s_ref, block);
    else
        mc_tiles<2>(P, s_pu, s_pre, s_ref, block);
}

}  // namespace hpvcd

extern "C" cudaError_t hpvcd_launch_mc(const hpvcd::DevPic* pics, int pic_index, int n_pus, cudaStream_t stream) {
    if (n_pus <= 0) return cudaSuccess;
    dim3 grid((n_pus + hpvcd::kMcPus - 1) / hpvcd::kMcPus, hpvcd::kMcSplit);
    hpvcd::k_mc<<<grid, 32 * hpvcd::kMcWarps, 0, stream>>>(pics, pic_index);
    hpvcd_note_launches(1);
    return cudaGetLastError();
}
