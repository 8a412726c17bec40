// deblock.cu — §7.14 deblocking filter, both passes fused per tile.
//
// Replaces loop_filter_frame (src/loop_filter.rs:271) as driven by
// loop_filter_frame_from_grid (src/cdf.rs:20449).  The reference walks every
// 4-sample edge segment in raster order, vertical pass then horizontal pass,
// filtering in place.  Within one pass no two edges touch the same samples:
// an edge's filter length is capped by the smaller of the two adjoining
// transform dimensions (loop_filter.rs:434-443) and its taps reach at most 7
// samples back and 6 forward (loop_filter.rs:643-671, 800-821), so every edge
// of a pass is independent and the sequential order is immaterial.
//
// B200 mapping: one CTA owns a 64x64 output tile of one plane and stages a
// 96x96 window (16-sample halo: an output sample can be moved by an edge up to
// 6 samples away whose taps reach 7 further) in shared memory.  It computes
// the per-4x4 edge parameters (filter length, limit, blimit, thresh) for the
// window from the mi grid, runs the vertical pass over all window rows, then
// the horizontal pass over the tile's columns, and writes the tile.  The
// frame is filtered out of place (recon -> deblocked) so halo reads never
// observe another tile's output.
#include "common.cuh"
#include "av1_spec_tables.h"

namespace av1g {

__constant__ AV1T_SUBSAMPLED_SIZE_TYPE c_subsampled AV1T_SUBSAMPLED_SIZE_DIMS = AV1T_SUBSAMPLED_SIZE_INIT;
__constant__ AV1T_MAX_TX_SIZE_RECT_TYPE c_max_tx_rect AV1T_MAX_TX_SIZE_RECT_DIMS = AV1T_MAX_TX_SIZE_RECT_INIT;
__constant__ AV1T_NUM_4X4_BLOCKS_WIDE_TYPE c_n4w AV1T_NUM_4X4_BLOCKS_WIDE_DIMS = AV1T_NUM_4X4_BLOCKS_WIDE_INIT;
__constant__ AV1T_NUM_4X4_BLOCKS_HIGH_TYPE c_n4h AV1T_NUM_4X4_BLOCKS_HIGH_DIMS = AV1T_NUM_4X4_BLOCKS_HIGH_INIT;
__constant__ AV1T_TX_WIDTH_TYPE c_txw AV1T_TX_WIDTH_DIMS = AV1T_TX_WIDTH_INIT;
__constant__ AV1T_TX_HEIGHT_TYPE c_txh AV1T_TX_HEIGHT_DIMS = AV1T_TX_HEIGHT_INIT;

namespace {

// window rows hold u16 samples at an odd number of 32-bit words per row
// (49), so a warp walking down a column touches 32 distinct banks; a row
// starts on a 4-byte (not always 8-byte) boundary, so the window is moved in
// 32-bit words
constexpr int TILE = 64, HALO = 16, WIN = TILE + 2 * HALO, PITCH = WIN + 2, CELLS = WIN / 4;
constexpr int kDbThreads = 256;  // deblock_kernel's CTA size
static_assert(WIN * (WIN / 4) % kDbThreads == 0, "window groups split evenly over the CTA");
constexpr int BLOCK_SIZES = 22, BLOCK_INVALID = 22;

// ---- edge codes ---------------------------------------------------------------
// u16 per 4x4 cell of every deblocked plane: the code of the cell's vertical
// (left) edge in the low byte, of its horizontal (top) edge in the high one; a code
// is the filter length class (1: 4, 2: 8 or chroma 6, 3: 16) << 6 | level (1..63),
// 0 for an edge that is not filtered.
//
// A code needs the grid entries of two cells (loop_filter_edge,
// loop_filter.rs:302-423, up to the sample loop), so a CTA derives what an
// edge needs of each cell once — levels, transform dimensions, whether each of
// its edges is one — for 64 x 16 luma cells, a row above and a column to the
// left, in shared memory, and then joins neighbours.  A thread takes 2 x 2 luma
// cells, whose grid entries it loads in pairs, and the chroma cells they make.
// Bound by instruction issue: 145 us per 64 x 1080p 8-bit (289 us when every
// edge gathered and derived both its cells).

constexpr int PW = 32, PH = 8;  // 2 x 2-cell groups per CTA (+ the halo)

// What an edge needs of a cell: level of its vertical edge | of its horizontal
// edge << 6 | (log2 transform width - 2) << 12 | height << 15 | whether the left
// / top border of the cell is an edge to filter << 18 / 19.
__device__ __forceinline__ uint32_t cell_info(int lv, int lh, int tw, int th, bool av, bool ah) {
    return (uint32_t)(lv | lh << 6 | tw << 12 | th << 15 | (av ? 1 << 18 : 0) | (ah ? 1 << 19 : 0));
}

// log2 of a transform dimension, minus 2 (3 bits each, TX_4X4 first)
constexpr unsigned long long pack_tx(const uint8_t* t) {
    unsigned long long v = 0;
    for (int k = 0; k < 19; k++) {
        int l = 0;
        while ((4 << l) < t[k]) l++;
        v |= (unsigned long long)l << (3 * k);
    }
    return v;
}
constexpr uint8_t kTxWidths[19] = AV1T_TX_WIDTH_INIT;
constexpr uint8_t kTxHeights[19] = AV1T_TX_HEIGHT_INIT;
constexpr unsigned long long kTxwBits = pack_tx(kTxWidths), kTxhBits = pack_tx(kTxHeights);
__device__ __forceinline__ int tx_w(int tx) { return (int)(kTxwBits >> (3 * tx)) & 7; }
__device__ __forceinline__ int tx_h(int tx) { return (int)(kTxhBits >> (3 * tx)) & 7; }

struct PrepShared {
    uint32_t y[2 * PH + 1][2 * PW + 2], uv[2 * PH + 1][2 * PW + 2];  // uv: u's level | v's << 6, else as y
    int seg[8][4];   // SEG_LVL_ALT_LF_* data, or kNoSeg
    int delta[8][2]; // reference (+ mode) delta by ref_frame0 and mode type
    // per block size: its cell-grid masks in the luma and in the chroma plane,
    // the chroma transform's dimensions
    struct {
        uint8_t yw, yh, uw, uh, tw, th;
    } bs[BLOCK_SIZES + 1];
};
constexpr int kNoSeg = 1 << 20;

// adaptive_filter_strength(_selection) (loop_filter.rs:465-580): the level for
// loop-filter index i (0 / 1: luma vertical / horizontal, 2 / 3: u / v).
__device__ __forceinline__ int cell_level(const PrepShared& S, const av1g_frame_header& h, int i, int dl, int seg,
                                          int delta) {
    int lvl = clip3(0, 63, dl + h.lf_level[i]);
    if (seg >= 0 && seg < 8 && S.seg[seg][i] != kNoSeg) lvl = clip3(0, 63, S.seg[seg][i] + lvl);
    return clip3(0, 63, lvl + delta * (1 << (lvl >> 5)));
}

// Two adjacent grid entries (a low, b high byte); idx is even.
__device__ __forceinline__ int ld2(const void* base, int idx, bool pairs) {
    const uint8_t* p = static_cast<const uint8_t*>(base) + idx;
    return pairs ? *reinterpret_cast<const uint16_t*>(p) : p[0] | p[1] << 8;
}

// An edge's code from its cell and the one before it.  sh: 0 vertical, 1
// horizontal edges; lsh: where the level lies; most: the longest filter's class.
__device__ __forceinline__ uint32_t edge_code(uint32_t cur, uint32_t prev, int sh, int lsh, int most) {
    if (!((cur >> (18 + sh)) & 1)) return 0;
    int lvl = (cur >> lsh) & 63;
    if (lvl == 0) lvl = (prev >> lsh) & 63;
    if (lvl == 0) return 0;
    const int d = 12 + 3 * sh, base = min((cur >> d) & 7, (prev >> d) & 7);
    return (uint32_t)(min(base + 1, most) << 6 | lvl);
}

__global__ void __launch_bounds__(256) lf_prep_kernel(const FrameDev* __restrict__ frames) {
    __shared__ PrepShared S;
    const FrameDev& F = frames[blockIdx.y];
    const av1g_frame_header& h = F.h;
    if (!F.do_stage[ST_DEBLOCK]) return;
    const int mr = h.mi_rows, mc = h.mi_cols;
    const int ntx = (mc + 2 * PW - 1) / (2 * PW), nty = (mr + 2 * PH - 1) / (2 * PH);
    if ((int)blockIdx.x >= ntx * nty) return;
    const int r0 = (int)blockIdx.x / ntx * 2 * PH, c0 = (int)blockIdx.x % ntx * 2 * PW;
    const int np = h.num_planes, ssx = np > 1 ? h.subsampling_x : 0, ssy = np > 1 ? h.subsampling_y : 0;
    if (threadIdx.x < 32) {
        const int sg = threadIdx.x >> 2, i = threadIdx.x & 3;
        S.seg[sg][i] = h.seg_lf_active[sg][i] ? h.seg_lf_data[sg][i] : kNoSeg;
    } else if (threadIdx.x < 48) {
        const int ref = (threadIdx.x - 32) >> 1, mt = threadIdx.x & 1;
        S.delta[ref][mt] = !h.lf_delta_enabled ? 0 : ref == 0 ? h.lf_ref_deltas[0] : h.lf_ref_deltas[ref] + h.lf_mode_deltas[mt];
    } else if (threadIdx.x >= 64 && threadIdx.x <= 64 + BLOCK_SIZES) {
        const int ms = threadIdx.x - 64;
        auto& b = S.bs[ms];
        b.yw = b.yh = b.uw = b.uh = b.tw = b.th = 0;
        if (ms < BLOCK_SIZES) {
            b.yw = c_n4w[ms] - 1;
            b.yh = c_n4h[ms] - 1;
            const int psz = c_subsampled[ms][ssx][ssy], es = psz == BLOCK_INVALID ? ms : psz;
            b.uw = c_n4w[es] - 1;
            b.uh = c_n4h[es] - 1;
            if (psz != BLOCK_INVALID) {  // loopfilter_tx_size_at (cdf.rs:20559-20594)
                const int uv = c_max_tx_rect[psz], w = c_txw[uv], hh = c_txh[uv];
                const int tx = (w == 64 || hh == 64) ? (w == 16 ? 9 : (hh == 16 ? 10 : 3)) : uv;
                b.tw = tx_w(tx);
                b.th = tx_h(tx);
            }
        }
    }
    const av1g_mi_grid& g = F.g;
    const bool pairs = !(((uintptr_t)g.mi_size | (uintptr_t)g.skip | (uintptr_t)g.is_inter | (uintptr_t)g.ref_frame0 |
                          (uintptr_t)g.y_mode | (uintptr_t)g.segment_id | (uintptr_t)g.tx_size |
                          (uintptr_t)g.inter_tx_size) & 1);
    const bool quads = !((uintptr_t)g.delta_lf & 7);
    const bool chroma = np > 1;
    const int iu = h.delta_lf_multi;
    __syncthreads();
    for (int q = threadIdx.x; q < (PW + 1) * (PH + 1); q += blockDim.x) {
        const int py = q / (PW + 1) - 1, px = q - (py + 1) * (PW + 1) - 1;
        const int r = r0 + 2 * py, c = c0 + 2 * px;
        if (r < 0 || c < 0 || r >= mr || c >= mc) continue;
        int even = BLOCK_SIZES;  // block size of the group's first row (chroma transforms are read there)
#pragma unroll
        for (int rr = 0; rr < 2; rr++) {
            const int idx = (r + rr) * mc + c;
            const int ms2 = ld2(g.mi_size, idx, pairs), sk2 = ld2(g.skip, idx, pairs), in2 = ld2(g.is_inter, idx, pairs);
            const int rf2 = ld2(g.ref_frame0, idx, pairs), ym2 = ld2(g.y_mode, idx, pairs);
            const int sg2 = ld2(g.segment_id, idx, pairs);
            const int tx2 = ld2(g.tx_size, idx, pairs), it2 = ld2(g.inter_tx_size, idx, pairs);
            uint2 dl;
            if (quads) {
                dl = *reinterpret_cast<const uint2*>(g.delta_lf + 4 * (size_t)idx);
            } else {
                const uint8_t* d = reinterpret_cast<const uint8_t*>(g.delta_lf) + 4 * (size_t)idx;
                dl = make_uint2(d[0] | d[1] << 8 | d[2] << 16 | (uint32_t)d[3] << 24,
                                d[4] | d[5] << 8 | d[6] << 16 | (uint32_t)d[7] << 24);
            }
            const int ms0 = min(ms2 & 0xff, BLOCK_SIZES), ms1 = min(ms2 >> 8, BLOCK_SIZES);
            if (rr == 0) even = ms0;
#pragma unroll
            for (int cc = 0; cc < 2; cc++) {
                const int ms = cc ? ms1 : ms0, sh = 8 * cc;
                const int ref = min(max((int)(int8_t)(rf2 >> sh), 0), 7), seg = (int8_t)(sg2 >> sh);
                const int m = (ym2 >> sh) & 0xff, mt = (m >= 14 && m != 16 && m != 24) ? 1 : 0;
                const int delta = S.delta[ref][mt];
                const bool inner = ((sk2 >> sh) & 0xff) && (int8_t)(rf2 >> sh) > 0;  // only block edges are filtered
                const uint32_t d4 = cc ? dl.y : dl.x;
                auto dlf = [&](int i) { return (int)(int8_t)(d4 >> (iu ? 8 * i : 0)); };
                int tx = (((in2 >> sh) & 0xff) ? it2 >> sh : tx2 >> sh) & 0xff;
                if (tx >= 19) tx = 0;  // not a TX_* ordinal: malformed grid, filtered as TX_4X4
                const int row = r + rr, col = c + cc;
                const auto& b = S.bs[ms];
                if (2 * py + rr >= -1 && 2 * px + cc >= -1) {
                    const int tw = tx_w(tx), th = tx_h(tx);
                    const bool in = col * 4 < h.frame_width && row * 4 < h.frame_height;
                    S.y[2 * py + rr + 1][2 * px + cc + 1] = cell_info(
                        cell_level(S, h, 0, dlf(0), seg, delta), cell_level(S, h, 1, dlf(1), seg, delta), tw, th,
                        in && col > 0 && !(col & ((1 << tw) - 1)) && (!inner || !(col & b.yw)),
                        in && row > 0 && !(row & ((1 << th) - 1)) && (!inner || !(row & b.yh)));
                }
                // a chroma cell takes its last luma cell's entries and its
                // transform from the first one's block size
                if (chroma && rr >= ssy && cc >= ssx) {
                    const int cy = row >> ssy, cx = col >> ssx, ey = cy - (r0 >> ssy), ex = cx - (c0 >> ssx);
                    if (ey >= -1 && ex >= -1) {
                        // the first luma cell: this one's column pair's first, and the
                        // group's first row when rows are shared too
                        const int first = ssy ? even : (ssx ? ms0 : ms);
                        const int tw = S.bs[first].tw, th = S.bs[first].th;
                        const bool in = (cx << ssx) * 4 < h.frame_width && (cy << ssy) * 4 < h.frame_height;
                        S.uv[ey + 1][ex + 1] = cell_info(
                            cell_level(S, h, 2, dlf(2), seg, delta), cell_level(S, h, 3, dlf(3), seg, delta), tw, th,
                            in && cx > 0 && !(cx & ((1 << tw) - 1)) && (!inner || !(cx & b.uw)),
                            in && cy > 0 && !(cy & ((1 << th) - 1)) && (!inner || !(cy & b.uh)));
                    }
                }
            }
        }
    }
    __syncthreads();
    // luma: a pair of cells per thread and round, one 32-bit store
    uint32_t* out = reinterpret_cast<uint32_t*>(F.lf_codes[0]);
    for (int k = threadIdx.x; k < 2 * PH * PW; k += blockDim.x) {
        const int y = k / PW, x = 2 * (k - y * PW), r = r0 + y, c = c0 + x;
        if (r >= mr || c >= mc) continue;
        const uint32_t a = S.y[y + 1][x], b = S.y[y + 1][x + 1], d = S.y[y + 1][x + 2];
        const uint32_t v0 = edge_code(b, a, 0, 0, 3) | edge_code(b, S.y[y][x + 1], 1, 6, 3) << 8;
        const uint32_t v1 = edge_code(d, b, 0, 0, 3) | edge_code(d, S.y[y][x + 2], 1, 6, 3) << 8;
        out[(r * mc + c) >> 1] = v0 | v1 << 16;
    }
    if (!chroma) return;
    const int cw = mc >> ssx, ch = mr >> ssy, tw = (2 * PW) >> ssx, th = (2 * PH) >> ssy;
    for (int k = threadIdx.x; k < tw * th; k += blockDim.x) {
        const int y = k / tw, x = k - y * tw, cy = (r0 >> ssy) + y, cx = (c0 >> ssx) + x;
        if (cy >= ch || cx >= cw) continue;
        const uint32_t b = S.uv[y + 1][x + 1], a = S.uv[y + 1][x], t = S.uv[y][x + 1];
#pragma unroll
        for (int p = 1; p <= 2; p++)
            if (h.lf_level[1 + p])
                F.lf_codes[p][cy * cw + cx] =
                    (uint16_t)(edge_code(b, a, 0, 6 * (p - 1), 2) | edge_code(b, t, 1, 6 * (p - 1), 2) << 8);
    }
}

// Unpacks a cell code into filter length | limit << 8 | blimit << 16 |
// thresh << 24 (adaptive_filter_strength, loop_filter.rs:500-525).
__device__ __forceinline__ uint32_t decode_code(uint32_t code, int sharp) {
    if (code == 0) return 0;
    int lvl = code & 63, fsc = code >> 6;
    int fsize = fsc == 1 ? 4 : (fsc == 2 ? 8 : 16);
    int sh = sharp > 4 ? 2 : (sharp > 0 ? 1 : 0);
    int limit = sharp > 0 ? clip3(1, 9 - sharp, lvl >> sh) : max(lvl >> sh, 1);
    int blimit = (2 * (lvl + 2) + limit) & 0xff;
    return (uint32_t)fsize | ((uint32_t)limit << 8) | ((uint32_t)blimit << 16) | ((uint32_t)(lvl >> 4) << 24);
}

__device__ __forceinline__ int f4clamp(int v, int bd) { return clip3(-(1 << (bd - 1)), (1 << (bd - 1)) - 1, v); }

// wide_filter (loop_filter.rs:789-822) for one (n, log2Size) case: outputs
// i in [-n, n) from taps j in [-n, n] weighted 2 for |j| <= n2 else 1, source
// positions clamped to [-(n + 1), n].  All indices are compile-time.
template <int N, int LOG2, int N2>
__device__ __forceinline__ void wide(uint16_t* b, int st) {
    int v[2 * N + 2];
#pragma unroll
    for (int k = 0; k < 2 * N + 2; k++) v[k] = b[(k - N - 1) * st];
    int o[2 * N];
#pragma unroll
    for (int i = -N; i < N; i++) {
        int t = 0;
#pragma unroll
        for (int j = -N; j <= N; j++) {
            int pp = i + j < -(N + 1) ? -(N + 1) : (i + j > N ? N : i + j);
            t += v[pp + N + 1] * ((j <= N2 && j >= -N2) ? 2 : 1);
        }
        o[i + N] = (t + (1 << (LOG2 - 1))) >> LOG2;
    }
#pragma unroll
    for (int i = -N; i < N; i++) b[i * st] = (uint16_t)o[i + N];
}

// sample_filtering + filter_mask + narrow/wide filters (loop_filter.rs:582-822)
// on a line of shared-memory samples; b points at q0, st is the step.
__device__ void filter_line(uint16_t* b, int st, uint32_t prm, int plane, int bd) {
    int fs = prm & 0xff;
    int limit = (prm >> 8) & 0xff, blimit = (prm >> 16) & 0xff, thresh = prm >> 24;
    int bds = bd - 8;
    int q0 = b[0], q1 = b[st], q2 = b[2 * st], q3 = b[3 * st];
    int p0 = b[-st], p1 = b[-2 * st], p2 = b[-3 * st], p3 = b[-4 * st];
    // every test below is "some |difference| > bound": the largest
    // difference against the bound, the shared ones computed once
    const int d1 = max(abs(p1 - p0), abs(q1 - q0));
    int thr = thresh << bds;
    bool hev = d1 > thr;
    int flen = fs == 4 ? 4 : (plane ? 6 : (fs == 8 ? 8 : 16));
    int lim = limit << bds, blim = blimit << bds;
    int dl = d1;
    if (flen >= 6) dl = __vimax3_s32(dl, abs(p2 - p1), abs(q2 - q1));
    if (flen >= 8) dl = __vimax3_s32(dl, abs(p3 - p2), abs(q3 - q2));
    if (dl > lim || abs(p0 - q0) * 2 + abs(p1 - q1) / 2 > blim) return;
    int one = 1 << bds;
    bool flat = false, flat2 = false;
    if (fs >= 8) {
        int df = __vimax3_s32(d1, abs(p2 - p0), abs(q2 - q0));
        if (flen >= 8) df = __vimax3_s32(df, abs(p3 - p0), abs(q3 - q0));
        flat = df <= one;
    }
    if (fs >= 16 && flat) {
        int q4 = b[4 * st], q5 = b[5 * st], q6 = b[6 * st];
        int p4 = b[-5 * st], p5 = b[-6 * st], p6 = b[-7 * st];
        const int d2 = __vimax3_s32(__vimax3_s32(abs(p6 - p0), abs(q6 - q0), abs(p5 - p0)),
                                    __vimax3_s32(abs(q5 - q0), abs(p4 - p0), abs(q4 - q0)), 0);
        flat2 = d2 <= one;
    }
    if (fs == 4 || !flat) {
        int half = 0x80 << bds;
        int ps1 = p1 - half, ps0 = p0 - half, qs0 = q0 - half, qs1 = q1 - half;
        int f = hev ? f4clamp(ps1 - qs1, bd) : 0;
        f = f4clamp(f + 3 * (qs0 - ps0), bd);
        int f1 = f4clamp(f + 4, bd) >> 3;
        int f2 = f4clamp(f + 3, bd) >> 3;
        b[0] = (uint16_t)(f4clamp(qs0 - f1, bd) + half);
        b[-st] = (uint16_t)(f4clamp(ps0 + f2, bd) + half);
        if (!hev) {
            int ff = (f1 + 1) >> 1;
            b[st] = (uint16_t)(f4clamp(qs1 - ff, bd) + half);
            b[-2 * st] = (uint16_t)(f4clamp(ps1 + ff, bd) + half);
        }
        return;
    }
    if (fs == 8 || !flat2) {
        if (plane == 0) wide<3, 3, 0>(b, st);
        else wide<2, 3, 1>(b, st);
    } else {
        wide<6, 4, 1>(b, st);
    }
}

__global__ void __launch_bounds__(kDbThreads, 6) deblock_kernel(const FrameDev* __restrict__ frames,
                                                      const int32_t* __restrict__ starts, int n, int total) {
    __shared__ __align__(16) uint16_t win[WIN * PITCH];
    __shared__ uint32_t ev[CELLS * CELLS], eh[CELLS * CELLS];
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        int f = find_frame(starts, n, t);
        const FrameDev& F = frames[f];
        int local = t - starts[f];
        // tile -> (plane, ty, tx); planes with no deblock work have no tiles
        int plane = 0, tx = 0, ty = 0;
        for (int p = 0; p < F.h.num_planes; p++) {
            if (p > 0 && F.h.lf_level[1 + p] == 0) continue;
            int ntx = (F.recon[p].w + TILE - 1) / TILE, nty = (F.recon[p].h + TILE - 1) / TILE;
            if (local < ntx * nty) { plane = p; ty = local / ntx; tx = local % ntx; break; }
            local -= ntx * nty;
        }
        const PlaneDev& S = F.recon[plane];
        const PlaneDev& D = F.deb[plane];
        const int hbd = F.hbd, bd = F.h.bit_depth;
        const int gx0 = tx * TILE - HALO, gy0 = ty * TILE - HALO;
        __syncthreads();  // previous tile done with shared memory
        // window: 4 consecutive samples per thread, one vector load when the
        // group lies inside the plane (rows are 4-sample aligned: gx0 % 4 == 0).
        // A window inside the plane horizontally (almost every tile) issues
        // all of a thread's loads before it unpacks any, so their latencies
        // overlap instead of adding up.
        if (gx0 >= 0 && gx0 + WIN <= S.w) {
            constexpr int G = WIN / 4, PER = WIN * G / kDbThreads;
            const uint8_t* base = S.p + (size_t)(hbd ? 2 : 1) * gx0;
            if (hbd) {
                uint2 v[PER];
#pragma unroll
                for (int q = 0; q < PER; q++) {
                    const int i = threadIdx.x + q * kDbThreads, r = i / G, c = (i - r * G) * 4;
                    v[q] = *reinterpret_cast<const uint2*>(base + (size_t)clip3(0, S.h - 1, gy0 + r) * S.stride + 2 * c);
                }
#pragma unroll
                for (int q = 0; q < PER; q++) {
                    const int i = threadIdx.x + q * kDbThreads, r = i / G, c = (i - r * G) * 4;
                    uint32_t* w = reinterpret_cast<uint32_t*>(&win[r * PITCH + c]);  // 4-byte aligned
                    w[0] = v[q].x;
                    w[1] = v[q].y;
                }
            } else {
                uint32_t v[PER];
#pragma unroll
                for (int q = 0; q < PER; q++) {
                    const int i = threadIdx.x + q * kDbThreads, r = i / G, c = (i - r * G) * 4;
                    v[q] = *reinterpret_cast<const uint32_t*>(base + (size_t)clip3(0, S.h - 1, gy0 + r) * S.stride + c);
                }
#pragma unroll
                for (int q = 0; q < PER; q++) {
                    const int i = threadIdx.x + q * kDbThreads, r = i / G, c = (i - r * G) * 4;
                    uint32_t* w = reinterpret_cast<uint32_t*>(&win[r * PITCH + c]);  // 4-byte aligned
                    w[0] = __byte_perm(v[q], 0u, 0x4140);
                    w[1] = __byte_perm(v[q], 0u, 0x4342);
                }
            }
        } else
        for (int i = threadIdx.x; i < WIN * (WIN / 4); i += blockDim.x) {
            int r = i / (WIN / 4), c = (i % (WIN / 4)) * 4;
            int gy = clip3(0, S.h - 1, gy0 + r), gx = gx0 + c;
            uint16_t* w = &win[r * PITCH + c];
            const uint8_t* row = S.p + (size_t)gy * S.stride;
            if (gx >= 0 && gx + 3 < S.w) {
                uint32_t* w32 = reinterpret_cast<uint32_t*>(w);  // 4-byte aligned
                if (hbd) {
                    const uint2 v = *reinterpret_cast<const uint2*>(row + 2 * gx);
                    w32[0] = v.x;
                    w32[1] = v.y;
                } else {
                    const uint32_t v = *reinterpret_cast<const uint32_t*>(row + gx);
                    w32[0] = __byte_perm(v, 0u, 0x4140);
                    w32[1] = __byte_perm(v, 0u, 0x4342);
                }
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) w[k] = (uint16_t)ld_px(S, hbd, gy, clip3(0, S.w - 1, gx + k));
            }
        }
        const int cy0 = gy0 / 4, cx0 = gx0 / 4;  // gx0,gy0 are multiples of 4 (may be negative)
        const int cw = S.w >> 2, ch = S.h >> 2, sharp = F.h.lf_sharpness;
        const uint16_t* codes = F.lf_codes[plane];
        {
            // the edge codes: a thread's (at most 3) loads first, then the decodes
            constexpr int PER = (CELLS * CELLS + kDbThreads - 1) / kDbThreads;
            uint32_t code[PER];
#pragma unroll
            for (int q = 0; q < PER; q++) {
                const int i = threadIdx.x + q * kDbThreads, cr = i / CELLS, cc = i - cr * CELLS;
                const int cy = cy0 + cr, cx = cx0 + cc;
                code[q] = (i < CELLS * CELLS && cy >= 0 && cx >= 0 && cy < ch && cx < cw) ? codes[cy * cw + cx] : 0;
            }
#pragma unroll
            for (int q = 0; q < PER; q++) {
                const int i = threadIdx.x + q * kDbThreads;
                if (i >= CELLS * CELLS) break;
                ev[i] = decode_code(code[q] & 0xff, sharp);
                eh[i] = decode_code(code[q] >> 8, sharp);
            }
        }
        __syncthreads();
        // vertical pass: window rows x edge columns 12..84 (cells 3..21: a
        // filter moves at most 6 samples from its edge, so only those edges
        // move tile columns; all window rows keep each warp's rows aligned to
        // the 4-row cells)
        constexpr int VR = WIN, VE = CELLS - 5;
        for (int i = threadIdx.x; i < VR * VE; i += blockDim.x) {
            int r = i % VR, cc = 3 + i / VR;
            uint32_t prm = ev[(r >> 2) * CELLS + cc];
            if (prm & 0xff) filter_line(&win[r * PITCH + cc * 4], 1, prm, plane, bd);
        }
        __syncthreads();
        // horizontal pass: tile columns x edge rows 12..84
        constexpr int HE = CELLS - 5;  // cells 3..21
        for (int i = threadIdx.x; i < TILE * HE; i += blockDim.x) {
            int c = HALO + i % TILE, cr = 3 + i / TILE;
            uint32_t prm = eh[cr * CELLS + (c >> 2)];
            if (prm & 0xff) filter_line(&win[cr * 4 * PITCH + c], PITCH, prm, plane, bd);
        }
        __syncthreads();
        // write the tile, four samples per thread (one vector store inside the plane)
        const int dh = min(D.h, S.h), dw = min(D.w, S.w);
        for (int i = threadIdx.x; i < TILE * (TILE / 4); i += blockDim.x) {
            int r = i / (TILE / 4), c = (i % (TILE / 4)) * 4;
            int gy = ty * TILE + r, gx = tx * TILE + c;
            if (gy >= dh) continue;
            const uint16_t* w = &win[(r + HALO) * PITCH + c + HALO];
            uint8_t* row = D.p + (size_t)gy * D.stride;
            if (gx + 3 < dw) {
                const uint32_t* w32 = reinterpret_cast<const uint32_t*>(w);  // 4-byte aligned
                const uint2 v = make_uint2(w32[0], w32[1]);
                if (hbd) *reinterpret_cast<uint2*>(row + 2 * gx) = v;
                else *reinterpret_cast<uint32_t*>(row + gx) = __byte_perm(v.x, v.y, 0x6420);
            } else {
                for (int k = 0; k < 4 && gx + k < dw; k++) st_px(D, hbd, gy, gx + k, w[k]);
            }
        }
    }
}

}  // namespace

int tiles_deblock(const FrameDev& f) {
    int n = 0;
    for (int p = 0; p < f.h.num_planes; p++) {
        if (p > 0 && f.h.lf_level[1 + p] == 0) continue;
        n += ((f.recon[p].w + TILE - 1) / TILE) * ((f.recon[p].h + TILE - 1) / TILE);
    }
    return n;
}

int cells_deblock(const FrameDev& f) {
    int n = 0;
    for (int p = 0; p < f.h.num_planes; p++) n += (f.recon[p].w >> 2) * (f.recon[p].h >> 2);
    return n;
}

int tiles_lf_prep(const FrameDev& f) {
    return ((f.h.mi_cols + 2 * PW - 1) / (2 * PW)) * ((f.h.mi_rows + 2 * PH - 1) / (2 * PH));
}

void launch_deblock(const FrameDev* frames, const int32_t* starts, int n, int total, int max_prep,
                    const StageShape& sh, cudaStream_t s) {
    if (total <= 0) return;
    lf_prep_kernel<<<dim3(max_prep, n), 256, 0, s>>>(frames);
    deblock_kernel<<<shape_grid(sh, total), kDbThreads, 0, s>>>(frames, starts, n, total);
}

}  // namespace av1g
