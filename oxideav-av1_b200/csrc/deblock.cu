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
// 96x88 window (16- and 12-sample halos: an output sample can be moved by an edge up
// to 6 samples away whose taps reach 7 further) in shared memory with the edge
// codes of its cells.  It runs the vertical pass over all window rows, then
// the horizontal pass over the tile's columns, and writes the tile.  The
// frame is filtered out of place (recon -> deblocked) so halo reads never
// observe another tile's output.
//
// A thread filters two lines at a time, the halves of a word, in
// half-precision differences and 16-bit sums that are exact for 8 and 10 bits
// (12-bit lines go one by one, and so do the lines of a 10-bit tile with a sample above
// 1023, which a valid stream does not have); both passes read two lines' samples as
// pairs of words without bank conflicts, and the filters that few edges take are calls
// of their own.  Bound by issue, and by warps whose edges take different filters: 500 us for 64
// 1080p 8-bit frames and 89 us for four 3840x2160 10-bit ones (1.4 TB/s of planes read
// and written), against 713 and 119 us with a line per thread.
#include <cuda_fp16.h>
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

// Window rows hold u16 samples two to a word, a pair of rows kPair words apart and
// its second row kRow words after the first: two rows of a line pair are one offset
// apart, and 8-byte accesses of 16 consecutive pairs touch 32 distinct banks.
constexpr int TILE = 64, HALO = 16, WIN = TILE + 2 * HALO, CELLS = WIN / 4;
constexpr int kRow = WIN / 2, kPair = 2 * kRow + 2;
static_assert(kPair % 32 == 2, "pairs of rows two banks apart");
// The horizontal pass reads at most 7 samples above and 6 below its edges, which
// lie in rows 12 to 84: no other row of the window is loaded or filtered.
constexpr int kRow0 = 4, kRow1 = 92;
constexpr int kDbThreads = 256;  // deblock_kernel's CTA size
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
    chain_wait();
    chain_next();
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

// limit, blimit and thresh of a level (adaptive_filter_strength,
// loop_filter.rs:500-525), before the scaling by bit depth.
struct Strength {
    int limit, blimit, thresh;
};
__device__ __forceinline__ Strength strength(int lvl, int sharp) {
    const int sh = sharp > 4 ? 2 : (sharp > 0 ? 1 : 0);
    const int limit = sharp > 0 ? clip3(1, 9 - sharp, lvl >> sh) : max(lvl >> sh, 1);
    return Strength{limit, (2 * (lvl + 2) + limit) & 0xff, lvl >> 4};
}

__device__ __forceinline__ int f4clamp(int v, int bd) { return clip3(-(1 << (bd - 1)), (1 << (bd - 1)) - 1, v); }

// wide_filter (loop_filter.rs:789-822) for one (n, log2Size) case: outputs
// i in [-n, n) from taps j in [-n, n] weighted 2 for |j| <= n2 else 1, source
// positions clamped to [-(n + 1), n].  PAIR: two lines at a time, one per half of a
// word: at 10 bits no sum passes 16 bits (16 times 1023, plus the rounding).
template <bool PAIR, int N, int LOG2, int N2>
__device__ __forceinline__ void wide(const uint32_t (&v)[2 * N + 2], uint32_t (&o)[2 * N]) {
    auto at = [&](int k) { return v[(k < -(N + 1) ? -(N + 1) : (k > N ? N : k)) + N + 1]; };
    uint32_t box = (1u << (LOG2 - 1)) * (PAIR ? 0x10001u : 1u);
#pragma unroll
    for (int j = -N; j <= N; j++) box += at(j - N);
#pragma unroll
    for (int i = -N; i < N; i++) {
        uint32_t t = box + at(i);
        if (N2) t += at(i - 1) + at(i + 1);
        o[i + N] = PAIR ? (t >> LOG2) & 0x0fff0fffu : t >> LOG2;
        box += at(i + N + 1) - at(i - N);
    }
}

// ---- two lines at a time, 8 and 10 bits -------------------------------------
// A sample v is the half 1024 + v (0x6400 | v): the differences of two are exact,
// and so is all that decides or makes a result below; what is larger than
// that is rounded only where it is beyond a bound or a clamp already.
constexpr uint32_t kBias = 0x64006400u, kSample = 0x03ff03ffu;

__device__ __forceinline__ __half2 h2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }
__device__ __forceinline__ uint32_t u32(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 dup(float x) { return __float2half2_rn(x); }
// max(m, |a - b|)
__device__ __forceinline__ __half2 far(__half2 m, uint32_t a, uint32_t b) {
    return __hmax2(m, __habs2(__hsub2(h2(a), h2(b))));
}
__device__ __forceinline__ uint32_t pick(uint32_t mask, uint32_t a, uint32_t b) { return (a & mask) | (b & ~mask); }

struct HalfConsts {
    __half2 one, lo, hi, top;  // 1 << (bd - 8), the clamp's ends, 1024 + the largest sample
};

// Samples 2j and 2j + 1 of both lines of a pair, counted from q0: the vertical
// pass's lines are the two rows of a pair, the horizontal pass's two adjacent columns.
template <bool VERT>
__device__ __forceinline__ void ld_pair(const uint32_t* m, int j, uint32_t& a, uint32_t& b) {
    if (VERT) {
        const uint32_t u = m[j], v = m[j + kRow];
        a = __byte_perm(u, v, 0x5410);
        b = __byte_perm(u, v, 0x7632);
    } else {
        a = m[j * kPair];
        b = m[j * kPair + kRow];
    }
}
template <bool VERT>
__device__ __forceinline__ void st_pair(uint32_t* m, int j, uint32_t a, uint32_t b) {
    if (VERT) {
        m[j] = __byte_perm(a, b, 0x5410);
        m[j + kRow] = __byte_perm(a, b, 0x7632);
    } else {
        m[j * kPair] = a;
        m[j * kPair + kRow] = b;
    }
}

// The 13-tap filter on the lines of `on`, which are unchanged so far: a call of its
// own that reads its samples again, so that the path most edges take fits the
// 40 registers that six CTAs per SM leave.
template <bool VERT>
__device__ __noinline__ void filter_wide(uint32_t* m, uint32_t on) {
    uint32_t v[16];
#pragma unroll
    for (int j = 0; j < 8; j++) ld_pair<VERT>(m, j - 4, v[2 * j], v[2 * j + 1]);
    uint32_t x[14], o[12];
#pragma unroll
    for (int k = 0; k < 14; k++) x[k] = v[k + 1] & kSample;
    wide<true, 6, 4, 1>(x, o);
#pragma unroll
    for (int j = 0; j < 6; j++)
        st_pair<VERT>(m, j - 3, pick(on, o[2 * j] | kBias, v[2 * j + 2]), pick(on, o[2 * j + 1] | kBias, v[2 * j + 3]));
}

// The same for the 7-tap (luma) and 5-tap (chroma) ones.
template <bool VERT>
__device__ __noinline__ void filter_flat(uint32_t* m, uint32_t on, int plane) {
    uint32_t v[8];
#pragma unroll
    for (int j = 0; j < 4; j++) ld_pair<VERT>(m, j - 2, v[2 * j], v[2 * j + 1]);
    uint32_t x[8];
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = v[k] & kSample;
    if (plane) {
        const uint32_t y[6] = {x[1], x[2], x[3], x[4], x[5], x[6]};
        uint32_t o[4];
        wide<true, 2, 3, 1>(y, o);
#pragma unroll
        for (int k = 0; k < 4; k++) v[k + 2] = pick(on, o[k] | kBias, v[k + 2]);
    } else {
        uint32_t o[6];
        wide<true, 3, 3, 0>(x, o);
#pragma unroll
        for (int k = 0; k < 6; k++) v[k + 1] = pick(on, o[k] | kBias, v[k + 1]);
        st_pair<VERT>(m, -2, v[0], v[1]);
        st_pair<VERT>(m, 1, v[6], v[7]);
    }
    st_pair<VERT>(m, -1, v[2], v[3]);
    st_pair<VERT>(m, 0, v[4], v[5]);
}

// sample_filtering + filter_mask + narrow/wide filters (loop_filter.rs:582-822).
// The edges of one pass share no samples, but two 4-sample edges share the
// 8 bytes between them: only words with changed samples are written.
template <bool VERT>
__device__ __forceinline__ void filter_pair(uint32_t* m, int cls, uint2 st, int plane, const HalfConsts& K) {
    uint32_t p3 = 0, p2 = 0, p1, p0, q0, q1, q2 = 0, q3 = 0;
    ld_pair<VERT>(m, -1, p1, p0);
    ld_pair<VERT>(m, 0, q0, q1);
    const __half2 dp = __hsub2(h2(p1), h2(q1)), dq = __hsub2(h2(q0), h2(p0));
    const __half2 d1 = far(__habs2(__hsub2(h2(p1), h2(p0))), q1, q0);
    __half2 dl = d1;
    if (cls >= 2) {
        ld_pair<VERT>(m, -2, p3, p2);
        ld_pair<VERT>(m, 1, q2, q3);
        dl = far(far(dl, p2, p1), q2, q1);
        if (!plane) dl = far(far(dl, p3, p2), q3, q2);
    }
    // 2 |p0 - q0| + |p1 - q1| / 2 <= blimit with the half kept: st holds blimit + 1/2
    const __half2 step = __hfma2(__habs2(dq), dup(2.f), __hmul2(__habs2(dp), dup(0.5f)));
    const uint32_t on = __hle2_mask(dl, h2(__byte_perm(st.x, 0u, 0x1010))) &
                        __hle2_mask(step, h2(__byte_perm(st.x, 0u, 0x3232)));
    if (!on) return;
    uint32_t flat = 0;
    if (cls >= 2) {
        __half2 df = far(far(d1, p2, p0), q2, q0);
        if (!plane) df = far(far(df, p3, p0), q3, q0);
        flat = on & __hle2_mask(df, K.one);
    }
    if (const uint32_t narrow = on & ~flat) {
        const uint32_t hev = __hgt2_mask(d1, h2(__byte_perm(st.y, 0u, 0x1010)));
        __half2 f = h2(u32(__hmin2(__hmax2(dp, K.lo), K.hi)) & hev);
        f = __hmin2(__hmax2(__hfma2(dq, dup(3.f), f), K.lo), K.hi);
        // min(f + 4, hi) >> 3 and min(f + 3, hi) >> 3: less 3.5, an eighth, to the nearest whole number
        const __half2 cap = __hsub2(K.hi, dup(3.5f)), big = dup(1536.f);
        const __half2 f1 = __hsub2(__hfma2(__hmin2(__hadd2(f, dup(0.5f)), cap), dup(0.125f), big), big);
        const __half2 f2 = __hsub2(__hfma2(__hmin2(__hsub2(f, dup(0.5f)), cap), dup(0.125f), big), big);
        const __half2 zero = dup(1024.f);
        const uint32_t r0 = pick(narrow, u32(__hmin2(__hmax2(__hsub2(h2(q0), f1), zero), K.top)), q0);
        const uint32_t n0 = pick(narrow, u32(__hmin2(__hmax2(__hadd2(h2(p0), f2), zero), K.top)), p0);
        // (f1 + 1) >> 1
        const __half2 ff = __hsub2(__hadd2(__hfma2(f1, dup(0.5f), dup(0.25f)), big), big);
        const uint32_t outer = narrow & ~hev;
        const uint32_t r1 = pick(outer, u32(__hmin2(__hmax2(__hsub2(h2(q1), ff), zero), K.top)), q1);
        const uint32_t n1 = pick(outer, u32(__hmin2(__hmax2(__hadd2(h2(p1), ff), zero), K.top)), p1);
        st_pair<VERT>(m, -1, n1, n0);
        st_pair<VERT>(m, 0, r0, r1);
    }
    if (!flat) return;
    if (cls == 3) {
        uint32_t p4, p5, p6, p7, q4, q5, q6, q7;
        ld_pair<VERT>(m, -3, p5, p4);
        ld_pair<VERT>(m, 2, q4, q5);
        ld_pair<VERT>(m, -4, p7, p6);
        ld_pair<VERT>(m, 3, q6, q7);
        __half2 d2 = far(far(__habs2(__hsub2(h2(p6), h2(p0))), q6, q0), p5, p0);
        d2 = far(far(far(d2, q5, q0), p4, p0), q4, q0);
        const uint32_t flat2 = flat & __hle2_mask(d2, K.one);
        if (flat2) filter_wide<VERT>(m, flat2);
        flat &= ~flat2;
    }
    if (flat) filter_flat<VERT>(m, flat, plane);
}

// ---- one line at a time, any 16-bit samples: 12 bits (a difference of two 12-bit
// samples is no half), and 10-bit tiles in which a sample has more than 10 bits ----
// Line `e` (0 or 1) of a pair; position k counts from q0.
template <bool VERT, int bd>
__device__ void filter_line(uint16_t* b, int e, int cls, uint32_t st, int plane) {
    auto at = [&](int k) -> uint16_t& {
        return VERT ? b[2 * kRow * e + k] : b[2 * (kPair * (k >> 1) + kRow * (k & 1)) + e];
    };
    const int limit = st & 0xff, blimit = (st >> 8) & 0xff, thresh = st >> 16;
    int bds = bd - 8;
    int q0 = at(0), q1 = at(1), q2 = at(2), q3 = at(3);
    int p0 = at(-1), p1 = at(-2), p2 = at(-3), p3 = at(-4);
    // every test below is "some |difference| > bound": the largest
    // difference against the bound, the shared ones computed once
    const int d1 = max(abs(p1 - p0), abs(q1 - q0));
    int thr = thresh << bds;
    bool hev = d1 > thr;
    int flen = cls == 1 ? 4 : (plane ? 6 : (cls == 2 ? 8 : 16));
    int lim = limit << bds, blim = blimit << bds;
    int dl = d1;
    if (flen >= 6) dl = __vimax3_s32(dl, abs(p2 - p1), abs(q2 - q1));
    if (flen >= 8) dl = __vimax3_s32(dl, abs(p3 - p2), abs(q3 - q2));
    if (dl > lim || abs(p0 - q0) * 2 + abs(p1 - q1) / 2 > blim) return;
    int one = 1 << bds;
    bool flat = false, flat2 = false;
    if (cls >= 2) {
        int df = __vimax3_s32(d1, abs(p2 - p0), abs(q2 - q0));
        if (flen >= 8) df = __vimax3_s32(df, abs(p3 - p0), abs(q3 - q0));
        flat = df <= one;
    }
    int p4 = 0, p5 = 0, p6 = 0, q4 = 0, q5 = 0, q6 = 0;
    if (cls >= 3 && flat) {
        q4 = at(4), q5 = at(5), q6 = at(6);
        p4 = at(-5), p5 = at(-6), p6 = at(-7);
        const int d2 = __vimax3_s32(__vimax3_s32(abs(p6 - p0), abs(q6 - q0), abs(p5 - p0)),
                                    __vimax3_s32(abs(q5 - q0), abs(p4 - p0), abs(q4 - q0)), 0);
        flat2 = d2 <= one;
    }
    if (!flat) {
        int half = 0x80 << bds;
        int ps1 = p1 - half, ps0 = p0 - half, qs0 = q0 - half, qs1 = q1 - half;
        int f = hev ? f4clamp(ps1 - qs1, bd) : 0;
        f = f4clamp(f + 3 * (qs0 - ps0), bd);
        int f1 = f4clamp(f + 4, bd) >> 3;
        int f2 = f4clamp(f + 3, bd) >> 3;
        at(0) = (uint16_t)(f4clamp(qs0 - f1, bd) + half);
        at(-1) = (uint16_t)(f4clamp(ps0 + f2, bd) + half);
        if (!hev) {
            int ff = (f1 + 1) >> 1;
            at(1) = (uint16_t)(f4clamp(qs1 - ff, bd) + half);
            at(-2) = (uint16_t)(f4clamp(ps1 + ff, bd) + half);
        }
        return;
    }
    if (!flat2) {
        if (plane == 0) {
            const uint32_t v[8] = {(uint32_t)p3, (uint32_t)p2, (uint32_t)p1, (uint32_t)p0,
                                   (uint32_t)q0, (uint32_t)q1, (uint32_t)q2, (uint32_t)q3};
            uint32_t o[6];
            wide<false, 3, 3, 0>(v, o);
#pragma unroll
            for (int i = -3; i < 3; i++) at(i) = (uint16_t)o[i + 3];
        } else {
            const uint32_t v[6] = {(uint32_t)p2, (uint32_t)p1, (uint32_t)p0, (uint32_t)q0, (uint32_t)q1, (uint32_t)q2};
            uint32_t o[4];
            wide<false, 2, 3, 1>(v, o);
#pragma unroll
            for (int i = -2; i < 2; i++) at(i) = (uint16_t)o[i + 2];
        }
    } else {
        const uint32_t v[14] = {(uint32_t)p6, (uint32_t)p5, (uint32_t)p4, (uint32_t)p3, (uint32_t)p2,
                                (uint32_t)p1, (uint32_t)p0, (uint32_t)q0, (uint32_t)q1, (uint32_t)q2,
                                (uint32_t)q3, (uint32_t)q4, (uint32_t)q5, (uint32_t)q6};
        uint32_t o[12];
        wide<false, 6, 4, 1>(v, o);
#pragma unroll
        for (int i = -6; i < 6; i++) at(i) = (uint16_t)o[i + 6];
    }
}

template <bool VERT, int BD>
__device__ __forceinline__ void filter_lines(uint32_t* m, int cls, uint32_t st, int plane) {
    uint16_t* b = reinterpret_cast<uint16_t*>(m);
    filter_line<VERT, BD>(b, 0, cls, st, plane);
    filter_line<VERT, BD>(b, 1, cls, st, plane);
}

// What the CTA needs of a tile, worked out by one thread while the previous tile
// is filtered.
struct DbTile {
    const uint8_t* src;
    uint8_t* dst;
    const uint16_t* codes;
    int src_stride, dst_stride, w, h, dw, dh, x, y;  // (x, y): the tile's first sample
    int plane, hbd, bd, sharp;
    int lines;  // filtered line by line: 12 bits, or samples of more than ten found while staging
};

__device__ __noinline__ void plan_tile(const FrameDev* __restrict__ frames, const int32_t* __restrict__ starts, int n,
                                       int t, DbTile& T) {
    const int f = find_frame(starts, n, t);
    const FrameDev& F = frames[f];
    int local = t - starts[f], plane = 0, tx = 0, ty = 0;
    // planes with no deblock work have no tiles
    for (int p = 0; p < F.h.num_planes; p++) {
        if (p > 0 && F.h.lf_level[1 + p] == 0) continue;
        const int ntx = (F.recon[p].w + TILE - 1) / TILE, nty = (F.recon[p].h + TILE - 1) / TILE;
        if (local < ntx * nty) { plane = p; ty = local / ntx; tx = local - ty * ntx; break; }
        local -= ntx * nty;
    }
    const PlaneDev& S = F.recon[plane];
    const PlaneDev& D = F.deb[plane];
    T = DbTile{S.p, D.p, F.lf_codes[plane], S.stride, D.stride, S.w, S.h, min(D.w, S.w), min(D.h, S.h),
               tx * TILE, ty * TILE, plane, F.hbd, F.h.bit_depth, F.h.lf_sharpness,
               F.h.bit_depth == 12};
}

// Writes the tile, the bits `keep` of its samples, eight per thread (one vector store
// inside the plane).
__device__ __forceinline__ void write_tile(const DbTile& T, const uint32_t* __restrict__ win, uint32_t keep) {
    const int dh = T.dh, dw = T.dw, dst_stride = T.dst_stride, hbd = T.hbd;
    uint8_t* dst = T.dst;
#pragma unroll
    for (int q = 0; q < TILE * TILE / 8 / kDbThreads; q++) {
        const int i = threadIdx.x + q * kDbThreads, r = i / (TILE / 8), c = i % (TILE / 8);
        const int gy = T.y + r, gx = T.x + 8 * c;
        if (gy >= dh) continue;
        const int wr = r + HALO;
        const uint32_t* w = win + (wr >> 1) * kPair + (wr & 1) * kRow + HALO / 2 + 4 * c;
        const uint2 a = *reinterpret_cast<const uint2*>(w), b = *reinterpret_cast<const uint2*>(w + 2);
        uint8_t* row = dst + (size_t)gy * dst_stride;
        if (gx + 7 < dw) {
            if (hbd)
                *reinterpret_cast<uint4*>(row + 2 * gx) = make_uint4(a.x & keep, a.y & keep, b.x & keep, b.y & keep);
            else
                *reinterpret_cast<uint2*>(row + gx) =
                    make_uint2(__byte_perm(a.x, a.y, 0x6420), __byte_perm(b.x, b.y, 0x6420));
        } else {
            const uint32_t v[4] = {a.x & keep, a.y & keep, b.x & keep, b.y & keep};
#pragma unroll
            for (int e = 0; e < 8; e++) {
                const uint32_t px = (v[e / 2] >> (16 * (e & 1))) & 0xffff;
                if (gx + e >= dw) continue;
                if (hbd) reinterpret_cast<uint16_t*>(row)[gx + e] = (uint16_t)px;
                else row[gx + e] = (uint8_t)px;
            }
        }
    }
}

// The passes over pairs of window rows (vertical edges) and of tile columns (horizontal
// ones), edge columns and rows 12..84 (cells 3..21: a filter moves at most 6 samples from
// its edge, so only those edges move tile samples).
constexpr int VP = (kRow1 - kRow0) / 2, HP = TILE / 2, EDGES = CELLS - 5;

__device__ __forceinline__ uint2 line_strength(int lvl, int sharp) {
    const Strength s = strength(lvl, sharp);
    return make_uint2((uint32_t)s.limit | (uint32_t)s.blimit << 8 | (uint32_t)s.thresh << 16, 0u);
}

// A staged tile of any 16-bit samples, line by line: 12 bits, and 10-bit tiles with a
// sample of more than 10 bits, whose bias comes off first.  A call of its own, so that
// it costs the other tiles no registers: 32 1080p frames take 348 us at 8 bits and 365
// at 10 (376 and 393 with the choice made at each edge; 346 and 362 with none).
template <int BD>
__device__ __noinline__ void filter_tile_by_lines(const DbTile& T, uint32_t* win, const uint16_t* code, uint2* strengths) {
    if (BD != 12) {
        for (int i = threadIdx.x; i < (kRow1 - kRow0) * kRow; i += kDbThreads) {
            const int r = kRow0 + i / kRow;
            win[(r >> 1) * kPair + (r & 1) * kRow + i % kRow] -= kBias;
        }
        if (threadIdx.x < 64) strengths[threadIdx.x] = line_strength(threadIdx.x, T.sharp);
        __syncthreads();
    }
    for (int i = threadIdx.x; i < VP * EDGES; i += kDbThreads) {
        const int e = i / VP, r = kRow0 / 2 + i - e * VP, cc = 3 + e;
        const int c = code[(r >> 1) * CELLS + cc] & 0xff;
        if (c) filter_lines<true, BD>(win + r * kPair + cc * 2, c >> 6, strengths[c & 63].x, T.plane);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < HP * EDGES; i += kDbThreads) {
        const int x = HALO / 2 + i % HP, cr = 3 + i / HP;
        const int c = code[cr * CELLS + (x >> 1)] >> 8;
        if (c) filter_lines<false, BD>(win + cr * 2 * kPair + x, c >> 6, strengths[c & 63].x, T.plane);
    }
    __syncthreads();
    write_tile(T, win, 0xffffffffu);
}

constexpr int kDbCtas = 6;

__global__ void __launch_bounds__(kDbThreads, kDbCtas) deblock_kernel(const FrameDev* __restrict__ frames,
                                                      const int32_t* __restrict__ starts, int n, int total) {
    chain_wait();
    chain_next();
    __shared__ __align__(16) uint32_t win[WIN / 2 * kPair];
    __shared__ uint16_t code[CELLS * CELLS];
    __shared__ uint2 strengths[64];  // by level: halves limit, blimit + 1/2, thresh; by lines: bytes
    __shared__ DbTile plan[2];
    if (threadIdx.x == 0 && (int)blockIdx.x < total) plan_tile(frames, starts, n, blockIdx.x, plan[0]);
    int k = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x, k ^= 1) {
        __syncthreads();  // the plan is there, and the previous tile done with shared memory
        const DbTile& T = plan[k];
        const int hbd = T.hbd, bd = T.bd, plane = T.plane;
        const int gx0 = T.x - HALO, gy0 = T.y - HALO;
        // added, so that it comes off again whatever the samples are
        const uint32_t bias = bd == 12 ? 0u : kBias;
        uint32_t seen = 0;  // high bit depths: the bits of the samples staged
        {
            // window: 8 consecutive samples per thread.  A window inside the
            // plane horizontally (almost every tile) issues three loads before it
            // stores any, so that their latencies overlap (all five at once cost the
            // filters' loop its registers: 531 against 497 us).
            constexpr int G = WIN / 8, ITEMS = (kRow1 - kRow0) * G, PER = 3;
            const uint8_t* src = T.src;
            const int stride = T.src_stride, h1 = T.h - 1, w = T.w;
            if (gx0 >= 0 && gx0 + WIN <= w) {
#pragma unroll 1
                for (int i0 = threadIdx.x; i0 < ITEMS; i0 += PER * kDbThreads) {
                    uint4 v[PER];
#pragma unroll
                    for (int q = 0; q < PER; q++) {
                        const int i = i0 + q * kDbThreads, r = kRow0 + i / G, c = i - (i / G) * G;
                        if (i >= ITEMS) continue;
                        const uint8_t* row = src + (size_t)clip3(0, h1, gy0 + r) * stride;
                        if (hbd) v[q] = *reinterpret_cast<const uint4*>(row + 2 * gx0 + 16 * c);
                        else *reinterpret_cast<uint2*>(&v[q]) = *reinterpret_cast<const uint2*>(row + gx0 + 8 * c);
                    }
#pragma unroll
                    for (int q = 0; q < PER; q++) {
                        const int i = i0 + q * kDbThreads, r = kRow0 + i / G, c = i - (i / G) * G;
                        if (i >= ITEMS) continue;
                        uint4 o;
                        if (hbd) {
                            seen |= (v[q].x | v[q].y) | (v[q].z | v[q].w);
                            o = make_uint4(v[q].x + bias, v[q].y + bias, v[q].z + bias, v[q].w + bias);
                        } else {
                            o = make_uint4(__byte_perm(v[q].x, kBias, 0x7170), __byte_perm(v[q].x, kBias, 0x7372),
                                           __byte_perm(v[q].y, kBias, 0x7170), __byte_perm(v[q].y, kBias, 0x7372));
                        }
                        uint2* d = reinterpret_cast<uint2*>(win + (r >> 1) * kPair + (r & 1) * kRow + 4 * c);
                        d[0] = make_uint2(o.x, o.y);
                        d[1] = make_uint2(o.z, o.w);
                    }
                }
            } else {
                for (int i = threadIdx.x; i < (kRow1 - kRow0) * kRow; i += kDbThreads) {
                    const int r = kRow0 + i / kRow, c = i % kRow;
                    const uint8_t* row = src + (size_t)clip3(0, h1, gy0 + r) * stride;
                    const int xa = clip3(0, w - 1, gx0 + 2 * c), xb = clip3(0, w - 1, gx0 + 2 * c + 1);
                    const uint32_t a = hbd ? reinterpret_cast<const uint16_t*>(row)[xa] : row[xa];
                    const uint32_t b = hbd ? reinterpret_cast<const uint16_t*>(row)[xb] : row[xb];
                    seen |= a | b << 16;
                    win[(r >> 1) * kPair + (r & 1) * kRow + c] = (a | b << 16) + bias;
                }
            }
        }
        {
            const int cy0 = gy0 / 4, cx0 = gx0 / 4;  // gx0,gy0 are multiples of 4 (may be negative)
            const int cw = T.w >> 2, ch = T.h >> 2;
            for (int i = threadIdx.x; i < CELLS * CELLS; i += kDbThreads) {
                const int cr = i / CELLS, cy = cy0 + cr, cx = cx0 + i - cr * CELLS;
                code[i] = cy >= 0 && cx >= 0 && cy < ch && cx < cw ? T.codes[cy * cw + cx] : (uint16_t)0;
            }
        }
        if (threadIdx.x < 64) {
            uint2 e;
            if (bd == 12) {
                e = line_strength(threadIdx.x, T.sharp);
            } else {
                const Strength s = strength(threadIdx.x, T.sharp);
                const float scale = bd == 8 ? 1.f : 4.f;
                const __half2 a = __floats2half2_rn(scale * s.limit, scale * s.blimit + 0.5f);
                e = make_uint2(u32(a), u32(__float2half2_rn(scale * s.thresh)));
            }
            strengths[threadIdx.x] = e;
        }
        if (__builtin_expect(seen & ~kSample, 0)) plan[k].lines = 1;
        __syncthreads();
        if (threadIdx.x == kDbThreads - 1 && t + (int)gridDim.x < total)
            plan_tile(frames, starts, n, t + gridDim.x, plan[k ^ 1]);
        if (__builtin_expect(T.lines, 0)) {
            if (bd == 12) filter_tile_by_lines<12>(T, win, code, strengths);
            else filter_tile_by_lines<10>(T, win, code, strengths);
            continue;
        }
        HalfConsts K;
        K.one = dup(bd == 8 ? 1.f : 4.f);
        K.lo = dup(bd == 8 ? -128.f : -512.f);
        K.hi = dup(bd == 8 ? 127.f : 511.f);
        K.top = dup(bd == 8 ? 1279.f : 2047.f);
        // vertical pass
        for (int i = threadIdx.x; i < VP * EDGES; i += kDbThreads) {
            const int e = i / VP, r = kRow0 / 2 + i - e * VP, cc = 3 + e;
            const int c = code[(r >> 1) * CELLS + cc] & 0xff;
            if (!c) continue;
            uint32_t* m = win + r * kPair + cc * 2;
            filter_pair<true>(m, c >> 6, strengths[c & 63], plane, K);
        }
        __syncthreads();
        // horizontal pass
        for (int i = threadIdx.x; i < HP * EDGES; i += kDbThreads) {
            const int x = HALO / 2 + i % HP, cr = 3 + i / HP;
            const int c = code[cr * CELLS + (x >> 1)] >> 8;
            if (!c) continue;
            uint32_t* m = win + cr * 2 * kPair + x;
            filter_pair<false>(m, c >> 6, strengths[c & 63], plane, K);
        }
        __syncthreads();
        write_tile(T, win, kSample);
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
    launch_chained(lf_prep_kernel, dim3(max_prep, n), 256, 0, s, frames);
    launch_chained(deblock_kernel, shape_grid(sh, total), kDbThreads, 0, s, frames, starts, n, total);
}

}  // namespace av1g
