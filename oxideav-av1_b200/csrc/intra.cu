// intra.cu — §7.11.2 intra prediction, §7.11.5 chroma from luma and intra
// reconstruction as one persistent superblock-wavefront launch.
//
// Replaces predict_intra_into_curr_frame (src/cdf.rs:16789),
// intra_predict_block_samples (cdf.rs:16990-17250), the mode kernels
// (cdf.rs:1348-3120) and predict_chroma_from_luma_into_curr_frame
// (cdf.rs:17256) in the order transform_block_emit runs them per TU
// (cdf.rs:32540-32910): predict, CfL, dequant + inverse transform + merge.
//
// Dependencies.  An intra TU reads final samples of the row above and the
// column to its left (up to twice its size), the co-located luma for CfL and,
// for intra block copy, a window of the frame.  The host walks each frame's
// TUs in decode order and records every area a TU reads:
//  - between superblocks, B waits for A when a TU of one of them reads the
//    other's area and A comes first in decode order (a read of a later
//    superblock's area orders the later one after the reader, as sequential
//    decoding does), so the waits form a DAG ordered by decode order;
//  - inside a superblock, a TU's level is one above the last writer of each
//    4x4 cell it reads or writes and the last reader of each cell it writes,
//    so the TUs of one level are independent of one another.
// One persistent launch covers the batch.  A CTA claims superblocks from an
// atomic counter in a topological order (dependency depth, frame, decode
// order), stages the superblock's samples, a border of its neighbours and its TU
// records in shared memory and runs the levels: small TUs one per warp, large
// ones with a group of warps.  A CTA only waits for superblocks claimed before
// its own, by CTAs that are running, so every wait ends; the time bound only
// guards against a broken invariant: a wait that runs out sets its frame's
// abort word in the launch's control block, the superblocks of that frame then
// no longer wait (they still run and publish their levels, so no wait of the
// launch is left hanging, but their samples are not to be used), and the host
// reports that frame of that launch as AV1G_EDEVICE.  Other frames of the batch
// are not affected: waits never cross frames.
//
// What bounds it is the chain of levels: a 1920x1080 key frame's longest one has
// about 2,200, nearly all with one to four TUs of at most 256 samples.  Measured
// on that frame (one launch, B200): 8.5 ms with a body per transform size and
// every level on one barrier, 2.2 ms in this form; 3840x2160 10-bit in 2 x 2
// tiles 10.0 against 2.3 ms, eight 640x360 frames 2.7 against 0.78 ms.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "common.cuh"
#include "host_pool.h"
#include "intra_plan.h"
#include "itx.cuh"
#include "wedge.cuh"

namespace av1g {

namespace {

using namespace itx;

constexpr int kT = 128;             // threads per CTA of intra_pre_kernel
constexpr int kNW = kT / 32;
constexpr int kGroups = 3;          // worker groups of intra_kernel, which take levels in turn
constexpr int kGW = 4;              // warps per group
constexpr int kGT = kGW * 32;
constexpr int kWW = kGroups * kGW;  // worker warps
constexpr int kIT = kWW * 32 + 64;  // + the publishing warp and the waiting warp
constexpr int kSmallPx = kIntraSmallPx;
constexpr int kLvStage = 512;       // level-table entries staged per superblock (more: read from HBM)
constexpr int kTuStage = 512;       // TU records staged per superblock (more: read from HBM)
constexpr long long kWaitNs = 2000000000LL;  // the bound of one dependency wait
// Readings of a shared word by one wait inside a CTA.  The workers wait for the waiting
// warp, whose own waits are bounded by time, and the publishing warp for the workers: both
// end well before this many (20 s and more), which mark the frame as a wait that ran out.
constexpr int kSpins = 1 << 30;

__constant__ AV1T_TX_WIDTH_TYPE c_txw_d AV1T_TX_WIDTH_DIMS = AV1T_TX_WIDTH_INIT;
__constant__ AV1T_TX_HEIGHT_TYPE c_txh_d AV1T_TX_HEIGHT_DIMS = AV1T_TX_HEIGHT_INIT;
__constant__ AV1T_MODE_TO_ANGLE_TYPE c_mode_angle AV1T_MODE_TO_ANGLE_DIMS = AV1T_MODE_TO_ANGLE_INIT;
__constant__ AV1T_DR_INTRA_DERIVATIVE_TYPE c_dr AV1T_DR_INTRA_DERIVATIVE_DIMS = AV1T_DR_INTRA_DERIVATIVE_INIT;
__constant__ AV1T_INTRA_FILTER_TAPS_TYPE c_fi_taps AV1T_INTRA_FILTER_TAPS_DIMS = AV1T_INTRA_FILTER_TAPS_INIT;
__constant__ AV1T_SM_WEIGHTS_TX_4X4_TYPE c_sm4 AV1T_SM_WEIGHTS_TX_4X4_DIMS = AV1T_SM_WEIGHTS_TX_4X4_INIT;
__constant__ AV1T_SM_WEIGHTS_TX_8X8_TYPE c_sm8 AV1T_SM_WEIGHTS_TX_8X8_DIMS = AV1T_SM_WEIGHTS_TX_8X8_INIT;
__constant__ AV1T_SM_WEIGHTS_TX_16X16_TYPE c_sm16 AV1T_SM_WEIGHTS_TX_16X16_DIMS = AV1T_SM_WEIGHTS_TX_16X16_INIT;
__constant__ AV1T_SM_WEIGHTS_TX_32X32_TYPE c_sm32 AV1T_SM_WEIGHTS_TX_32X32_DIMS = AV1T_SM_WEIGHTS_TX_32X32_INIT;
__constant__ AV1T_SM_WEIGHTS_TX_64X64_TYPE c_sm64 AV1T_SM_WEIGHTS_TX_64X64_DIMS = AV1T_SM_WEIGHTS_TX_64X64_INIT;
__constant__ AV1T_SUBPEL_FILTERS_TYPE c_subpel AV1T_SUBPEL_FILTERS_DIMS = AV1T_SUBPEL_FILTERS_INIT;

// The superblock's copy in shared memory: per plane its area {x0, y0, w, h}
// with one row above (running on past the right edge, for above-right edges)
// and one column to the left, so that an edge is read the same way inside the
// superblock and across its border.  off: the index of the area's first
// sample; cs: the row pitch in samples, a multiple of four (four-sample groups
// are 8-byte aligned) whose 32-bit words advance two banks per row, so that
// the 16 rows of a left edge fall on 16 banks.
struct SbCtx {
    int4 rect[3];
    int off[3], cs[3];
};
__device__ __forceinline__ int copy_pitch(int log2sb, int ssx) { return intra_copy_pitch((1 << log2sb) >> ssx); }
__device__ __forceinline__ int copy_off(int log2sb, int ssx, int ssy, int p) {
    int o = copy_pitch(log2sb, p ? ssx : 0) + 4;
    if (p > 0) o += intra_copy_samples(1 << log2sb, 1 << log2sb);
    if (p > 1) o += intra_copy_samples((1 << log2sb) >> ssx, (1 << log2sb) >> ssy);
    return o;
}

__device__ const AV1T_II_WEIGHTS_1D_TYPE g_ii_w AV1T_II_WEIGHTS_1D_DIMS = AV1T_II_WEIGHTS_1D_INIT;
__device__ const wedge::Master g_wmaster = wedge::kMaster;
// The wait bound in effect (kWaitNs unless a test shortens it, see
// av1g_test_intra_wait_fault).
__device__ long long g_wait_ns = kWaitNs;

// ---- TU records -------------------------------------------------------------
// intra_pre_kernel turns every av1g_intra_tu of the launch, in place, into the
// form the wavefront reads: all that follows from the descriptor, the frame
// and the superblock (class, angles, edge lengths and filters, the place in
// the superblock's copy) is worked out there, in parallel, so that the serial
// chain of TUs holds only what depends on samples.

enum Cls : uint8_t {
    C_NONE, C_DC, C_V, C_H, C_SMOOTH, C_SMOOTH_V, C_SMOOTH_H, C_PAETH,
    C_D1,  // directional, angle below 90: the above edge only
    C_D2,  // between 90 and 180: both edges
    C_D3,  // from 180: the left edge only
    C_FI, C_PAL, C_BC
};
enum : uint8_t {  // TuHead::bits
    R_ABOVE = 1, R_LEFT = 2, R_RES = 4, R_CFL = 8,
    R_EDGE = 16,     // an edge is filtered or upsampled, or the corner is
    R_CORNER = 32, R_UPA = 64, R_UPL = 128
};
enum : uint8_t {  // TuHead::where
    W_COPY = 1,      // every edge sample lies in the superblock's copy
    W_DIRECT = 2,    // and the prediction reads both edges there, in place
    W_CFL = 4,       // CfL's luma lies in the copy, in aligned pairs
    W_ALIGNED = 8,   // x and the plane's width are multiples of four: a group of four samples
                     // lies wholly inside or outside the plane
    W_FAST = 16      // a small TU that fast_decode / fast_run take
};

struct TuHead {
    uint32_t res;          // its residual block (R_RES)
    uint16_t x, y;         // plane sample position
    uint32_t coff;         // its first sample in the superblock's copy
    uint8_t dims;          // log2 width | log2 height << 4
    uint8_t cls, plane, bits;
    uint8_t strength;      // edge filter strength above | left << 4
    uint8_t misc;          // filter intra mode | interintra << 4
    int8_t alpha;
    uint8_t where;
    uint16_t na, nl;       // samples the above / left edge has before it repeats the last
    uint16_t ea, el;       // edge samples the prediction uses
    uint16_t fa, fl;       // edge filter lengths (corner included)
    int16_t dx, dy;
    uint16_t cx, cy;       // CfL: the last luma position averaged
    uint32_t map;          // palette map, wedge window of an inter-intra block, or the copy's vector (row << 16 | column)
    uint16_t stride;       // palette map
    uint8_t ii_mode, pad;
};
struct alignas(16) TuRec {
    TuHead h;
    union {
        uint16_t colors[8];
        uint32_t recip;    // DC: ceil(2^32 / edge samples)
    };
};
static_assert(sizeof(TuHead) == 48 && sizeof(TuRec) == sizeof(av1g_intra_tu), "records are converted in place");

// The intra half of an inter-intra block: blend of the intra prediction
// with the inter half (mask_blend_interintra, src/inter_pred.rs:3272).  The
// mask is the §7.11.3.13 smooth mask on the plane block (read at [i][j]
// directly) or the §7.11.3.11 wedge mask on the luma grid (orientation
// resolved by the host into map).
__device__ int interintra_px(const IntraFrame& F, const TuHead& t, int kind, int i, int j, int intra, int inter,
                             int maxv) {
    int m;
    if (kind == 2) {
        const uint32_t o = t.map;
        const wedge::Orient w{(uint8_t)(o & 0xff), (uint8_t)((o >> 8) & 0xff), (uint8_t)((o >> 16) & 0xff),
                              (uint8_t)(o >> 24)};
        m = wedge::mask_px(g_wmaster, w, t.plane ? F.ssx : 0, t.plane ? F.ssy : 0, i, j);
    } else {
        const int sh = 7 - max(t.dims & 15, t.dims >> 4);  // 128 / max(w, h)
        const int mode = t.ii_mode;
        m = mode == 1 ? __ldg(&g_ii_w[i << sh]) : mode == 2 ? __ldg(&g_ii_w[j << sh])
          : mode == 3 ? __ldg(&g_ii_w[min(i, j) << sh]) : 32;
    }
    return min(max((m * intra + (64 - m) * inter + 32) >> 6, 0), maxv);
}

// A TU is run either by one warp or by the whole CTA; both expose a rank,
// a size and a barrier over exactly the threads that run the TU.
struct WarpG {
    static constexpr int N = 32;
    int r;
    __device__ __forceinline__ void sync() const { __syncwarp(); }
};
struct CtaG {  // intra_pre_kernel's CTA
    static constexpr int N = kT;
    int r;
    __device__ __forceinline__ void sync() const { __syncthreads(); }
};
// Hardware barriers of intra_kernel: 0 the CTA, 1..3 the end of a level (the
// group that ran it arrives, the group of the next level waits), 4..6 within a
// group.
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}
struct WorkG {  // a worker group
    static constexpr int N = kGT;
    int r, id;
    __device__ __forceinline__ void sync() const { bar_sync(id, kGT); }
};

// Per-group scratch.  The edge arrays hold position k of an edge at [4 + k]
// (the corner, position -1, at [3]; an upsampled edge starts at position -2):
// [0, E) above, [E, 2 E) left, as gathered (raw) and after the edge filter or
// upsampling (fin).
template <int EN, int PX>
struct Scr {
    static constexpr int E = EN;
    alignas(16) uint16_t raw[2 * EN];
    alignas(16) uint16_t fin[2 * EN];
    alignas(16) uint16_t buf[PX];  // CfL luma, intra block copy
    int red[kGW];
};
using WScr = Scr<48, kSmallPx>;  // W + H <= 40 for the small sizes
using CScr = Scr<136, 64 * 64>;  // W + H <= 128

constexpr int kNoWait = 0x7fffffff;

struct Tables {
    alignas(8) int8_t fi[5][8][8];  // filter intra taps
    alignas(4) uint8_t sm[124];     // smooth weights, length n at n - 4
};

struct alignas(16) Shared {
    union {
        WScr w[kGW];
        CScr c;
    } s[kGroups];
    IntraFrame fr;  // the superblock's frame record
    Tables tb;
    int2 lv[kLvStage];
    SbCtx sb;
    int idx;
    int done;   // levels finished, as far as they are published (workers -> publishing warp)
    int ready;  // levels below this one may run (waiting warp -> workers)
    int stuck;  // a wait inside the CTA ran out (-> publishing warp)
};
static_assert(sizeof(IntraFrame) % 4 == 0, "frame record copied as words");
constexpr size_t kSharedBytes = (sizeof(Shared) + 15) & ~(size_t)15;

// Sum over the group (every thread of it calls).
template <class G, class S>
__device__ __forceinline__ int gsum(const G& g, S& s, int v) {
    v = __reduce_add_sync(0xffffffffu, v);
    if constexpr (G::N > 32) {
        if ((g.r & 31) == 0) s.red[g.r >> 5] = v;
        g.sync();
        int t = 0;
#pragma unroll
        for (int k = 0; k < G::N / 32; k++) t += s.red[k];
        g.sync();
        return t;
    } else {
        return v;
    }
}

// A sample of plane p at (y, x), inside the plane: from the shared-memory
// copy when it lies in the current superblock, else from HBM (an earlier
// superblock's final samples, published by its progress word; read past L1).
__device__ __forceinline__ int rdp(const IntraFrame& F, const SbCtx& c, const uint16_t* cache, int p, int y, int x) {
    const int4 r = c.rect[p];
    const int ly = y - r.y, lx = x - r.x;
    if ((unsigned)ly < (unsigned)r.w && (unsigned)lx < (unsigned)r.z) return cache[c.off[p] + ly * c.cs[p] + lx];
    const PlaneDev& P = F.planes[p];
    const uint8_t* row = P.p + (size_t)y * P.stride;
    return F.hbd ? (int)__ldcg(reinterpret_cast<const unsigned short*>(row) + x) : (int)__ldcg(row + x);
}

// intra_edge_filter_strength_selection (cdf.rs:2610)
__device__ int strength_sel(int w, int h, int ft, int delta) {
    int d = abs(delta), wh = w + h, st = 0;
    if (ft == 0) {
        if (wh <= 8) { if (d >= 56) st = 1; }
        else if (wh <= 16) { if (d >= 40) st = 1; }
        else if (wh <= 24) { if (d >= 8) st = 1; if (d >= 16) st = 2; if (d >= 32) st = 3; }
        else if (wh <= 32) { st = 1; if (d >= 4) st = 2; if (d >= 32) st = 3; }
        else st = 3;
    } else {
        if (wh <= 8) { if (d >= 40) st = 1; if (d >= 64) st = 2; }
        else if (wh <= 16) { if (d >= 20) st = 1; if (d >= 48) st = 2; }
        else if (wh <= 24) { if (d >= 4) st = 3; }
        else st = 3;
    }
    return st;
}
// intra_edge_upsample_selection (cdf.rs:2588)
__device__ int upsample_sel(int w, int h, int ft, int delta) {
    int d = abs(delta);
    if (d == 0 || d >= 40) return 0;
    return ft == 0 ? (w + h <= 16) : (w + h <= 8);
}

// The record of one TU (see TuHead).
__device__ void prep_tu(const IntraFrame& F, int log2sb, const av1g_intra_tu& t, TuRec& o) {
    TuHead r{};
    const int pl = t.plane, ssx = pl ? F.ssx : 0, ssy = pl ? F.ssy : 0;
    const int W = c_txw_d[t.tx_size], H = c_txh_d[t.tx_size];
    const int sx = t.x, sy = t.y;
    const int max_x = F.planes[pl].w - 1, max_y = F.planes[pl].h - 1;
    const int sbw = (1 << log2sb) >> ssx, sbh = (1 << log2sb) >> ssy;
    const int lx = sx & (sbw - 1), ly = sy & (sbh - 1);
    uint32_t recip = 0;
    r.x = t.x;
    r.y = t.y;
    r.coff = (uint32_t)(copy_off(log2sb, F.ssx, F.ssy, pl) + ly * copy_pitch(log2sb, ssx) + lx);
    r.dims = (uint8_t)((31 - __clz(W)) | (31 - __clz(H)) << 4);
    r.plane = t.plane;
    r.res = t.res.coeff_offset;
    if (!(sx & 3) && !(F.planes[pl].w & 3)) r.where |= W_ALIGNED;
    if (t.flags & AV1G_INTRA_RESIDUAL) r.bits |= R_RES;
    if ((t.flags & AV1G_INTRA_CFL) && pl > 0) {
        r.bits |= R_CFL;
        const int cx = max((int)t.max_luma_w - (1 << F.ssx), 0), cy = max((int)t.max_luma_h - (1 << F.ssy), 0);
        r.cx = (uint16_t)cx;
        r.cy = (uint16_t)cy;
        r.alpha = t.cfl_alpha;
        const int x0 = (sx - lx) << ssx, y0 = (sy - ly) << ssy, sb = 1 << log2sb;
        if (cx >= x0 && cy >= y0 && min((sx + W - 1) << ssx, cx) + ssx < x0 + sb &&
            min((sy + H - 1) << ssy, cy) + ssy < y0 + sb && !(ssx && (cx & 1)))
            r.where |= W_CFL;
    }
    const int fim = (pl == 0 && t.filter_intra_mode < 5) ? t.filter_intra_mode : -1;
    r.misc = (uint8_t)((fim >= 0 ? fim : 0) | (t.mode < 13 && fim < 0 ? t.interintra << 4 : 0));
    r.ii_mode = t.interintra_mode;
    r.stride = t.palette_stride;
    r.map = t.mode == AV1G_INTRA_MODE_INTRABC ? (uint32_t)(uint16_t)t.mv[0] << 16 | (uint16_t)t.mv[1] : t.palette_map;
    if (t.mode < 13) {
        const bool ha = (t.flags & AV1G_INTRA_HAVE_ABOVE) && sy > 0;
        const bool hl = (t.flags & AV1G_INTRA_HAVE_LEFT) && sx > 0;
        const int ft = (t.flags & AV1G_INTRA_FILTER_TYPE) ? 1 : 0;
        if (ha) r.bits |= R_ABOVE;
        if (hl) r.bits |= R_LEFT;
        // intra_predict_block_samples' edge limits (cdf.rs:17030-17075)
        r.na = (uint16_t)(min(max_x, sx + ((t.flags & AV1G_INTRA_HAVE_ABOVE_RIGHT) ? 2 * W : W) - 1) - sx + 1);
        r.nl = (uint16_t)(min(max_y, sy + ((t.flags & AV1G_INTRA_HAVE_BELOW_LEFT) ? 2 * H : H) - 1) - sy + 1);
        int ea = W, el = H;
        const bool copy_v = t.mode == 1 && t.angle_delta == 0, copy_h = t.mode == 2 && t.angle_delta == 0;
        const bool dir = t.mode >= 1 && t.mode <= 8 && !copy_v && !copy_h;
        if (dir) {
            const int pa = c_mode_angle[t.mode] + t.angle_delta * 3;
            auto dr = [](int k) { return k >= 0 && k < 90 ? c_dr[k] : (int16_t)0; };
            r.dx = pa < 90 ? dr(pa) : (pa < 180 ? dr(180 - pa) : (int16_t)0);
            r.dy = (pa >= 90 && pa < 180) ? dr(pa - 90) : (pa > 180 ? dr(270 - pa) : (int16_t)0);
            r.cls = pa < 90 ? C_D1 : pa < 180 ? C_D2 : C_D3;
            ea = pa < 90 ? W + H : (pa < 180 || fim >= 0) ? W : 0;
            el = pa > 180 ? W + H : pa == 180 ? W + H : (pa >= 90 || fim >= 0) ? H : 0;
            if ((t.flags & AV1G_INTRA_EDGE_FILTER) && pa != 90 && pa != 180) {
                if (pa > 90 && pa < 180 && W + H >= 24) r.bits |= R_EDGE | R_CORNER;
                r.fa = (uint16_t)(min(W, max_x - sx + 1) + (pa < 90 ? H : 0) + 1);
                r.fl = (uint16_t)(min(H, max_y - sy + 1) + (pa > 180 ? W : 0) + 1);
                const int sa = ha ? strength_sel(W, H, ft, pa - 90) : 0;
                const int sl = hl ? strength_sel(W, H, ft, pa - 180) : 0;
                r.strength = (uint8_t)(sa | sl << 4);
                if (r.strength) r.bits |= R_EDGE;
                if (upsample_sel(W, H, ft, pa - 90)) r.bits |= R_EDGE | R_UPA;
                if (upsample_sel(W, H, ft, pa - 180)) r.bits |= R_EDGE | R_UPL;
            }
        } else if (copy_v) {
            r.cls = C_V;
            el = 0;
        } else if (copy_h) {
            r.cls = C_H;
            ea = 0;
        } else if (t.mode == 0) {
            r.cls = C_DC;
            if (!ha) ea = 0;
            if (!hl) el = 0;
        } else {
            r.cls = t.mode == 9 ? C_SMOOTH : t.mode == 10 ? C_SMOOTH_V : t.mode == 11 ? C_SMOOTH_H : C_PAETH;
        }
        if (fim >= 0) {
            r.cls = C_FI;
            ea = max(ea, W);
            el = max(el, H);
        }
        r.ea = (uint16_t)ea;
        r.el = (uint16_t)el;
        if (r.cls == C_DC && ea + el) recip = (uint32_t)(((1ull << 32) + ea + el - 1) / (ea + el));
        // the copy holds the row above up to intra_copy_ext samples past the
        // superblock, and otherwise the superblock's own columns
        const int wide = ly == 0 ? sbw + intra_copy_ext(sbw) : sbw;
        if (lx + min(ea, (int)r.na) <= wide && ly + min(el, (int)r.nl) <= sbh) {
            r.where |= W_COPY;
            const bool a_ok = ha && r.na >= W, l_ok = hl && r.nl >= H;
            const bool in_place = r.cls == C_V ? a_ok : r.cls == C_H ? l_ok
                                : r.cls == C_DC ? (!ha || a_ok) && (!hl || l_ok)
                                : (r.cls >= C_SMOOTH && r.cls <= C_PAETH) || (r.cls == C_FI && !(r.bits & R_EDGE)) ? a_ok && l_ok
                                : false;
            if (in_place && !(sx & 3)) r.where |= W_DIRECT;
        }
    } else if (t.mode == AV1G_INTRA_MODE_PALETTE) {
        r.cls = C_PAL;
    } else if (t.mode == AV1G_INTRA_MODE_INTRABC) {
        r.cls = C_BC;
    }
    const bool cfl = r.bits & R_CFL, direct = r.where & W_DIRECT;
    bool fast = W * H <= kSmallPx && (r.where & W_ALIGNED) && !(r.misc >> 4);
    switch (r.cls) {
        case C_NONE:
        case C_PAL: fast = fast && !cfl; break;
        case C_DC: fast = fast && direct && (!cfl || (r.where & W_CFL)); break;
        case C_D1:
        case C_D2:
        case C_D3: fast = fast && !cfl && (r.where & W_COPY) && (r.bits & (R_ABOVE | R_LEFT)); break;
        case C_BC: fast = false; break;
        default: fast = fast && direct && !cfl; break;
    }
    if (fast) r.where |= W_FAST;
    o.h = r;
    for (int k = 0; k < 8; k++) o.colors[k] = t.palette_colors[k];
    if (r.cls == C_DC) o.recip = recip;
}

// Scratch of one residual block.
template <int PX>
struct ResScr {
    int buf[PX];
};

// Dequantize (dequantize_step1, cdf.rs:13655-13703) and inverse transform
// (transform.rs:707-789) one TU's residual, stored as w*h int32 in sample
// orientation (the FLIPADST flips of curr_frame_step3_merge, cdf.rs:17398-17470,
// already applied).  cf holds the compact levels, cf[q] == level[g.r + q * G::N].
template <int TX, class G, class S>
__device__ __forceinline__ void residual_store(const G& g, S& s, const IntraFrame& R, const av1g_tu& tu, const int* cf,
                                               int32_t* out) {
    constexpr int W = kTxW[TX], H = kTxH[TX];
    constexpr int LW = ilog2<W>(), LH = ilog2<H>();
    constexpr int TW = W < 32 ? W : 32, TH = H < 32 ? H : 32, NC = TW * TH, K = (NC + G::N - 1) / G::N;
    constexpr int ABS_D = LW > LH ? LW - LH : LH - LW;
    const int bd = R.bd;
    const int seg = tu.segment_id > 7 ? 7 : tu.segment_id;
    const bool lossless = R.q.lossless[seg] != 0;
    for (int k = g.r; k < W * H; k += G::N) s.buf[k] = 0;
    g.sync();
    {
        const av1g_quant_params& q = R.q;
        int qidx;
        if (q.segmentation_enabled && q.seg_alt_q_active[seg]) {
            int data = q.seg_alt_q_data[seg];
            qidx = clip3(0, 255, (q.delta_q_present ? tu.current_q_index : q.base_q_idx) + data);
        } else {
            qidx = q.delta_q_present ? tu.current_q_index : q.base_q_idx;
        }
        const int p = tu.plane;
        const int ddc = p == 0 ? q.delta_q_y_dc : (p == 1 ? q.delta_q_u_dc : q.delta_q_v_dc);
        const int dac = p == 0 ? 0 : (p == 1 ? q.delta_q_u_ac : q.delta_q_v_ac);
        const int row = min((max(bd, 8) - 8) >> 1, 2);
        const int dcq = c_dcq[row][clip3(0, 255, qidx + ddc)], acq = c_acq[row][clip3(0, 255, qidx + dac)];
        const int qml = q.seg_qm_level[p][seg];
        const bool qm = q.using_qmatrix && tu.tx_type < 9 && qml < 15;
        constexpr int denom_sh = (TX == 3 || TX == 9 || TX == 10 || TX == 17 || TX == 18) ? 1
                               : (TX == 4 || TX == 11 || TX == 12) ? 2 : 0;
        const long long cmax = (1LL << (7 + bd)) - 1, cmin = -(1LL << (7 + bd));
#pragma unroll
        for (int qq = 0; qq < K; qq++) {
            const int k = g.r + qq * G::N;
            if (NC % G::N == 0 || k < NC) {
                const int i = k / TW, j = k % TW;
                long long qv = k == 0 ? dcq : acq;
                if (qm) qv = (qv * g_qm[qml][p > 0][c_qm_off[TX] + k] + 16) >> 5;
                const long long dq = (long long)cf[qq] * qv;
                const long long mag = (dq < 0 ? -dq : dq) & 0xFFFFFF;
                const long long v = (dq < 0 ? -mag : mag) / (1 << denom_sh);  // truncating division, as the reference
                s.buf[i * W + j] = (int)min(max(v, cmin), cmax);
            }
        }
    }
    g.sync();
    const Clamp rr{-(1 << (bd + 7)), (1 << (bd + 7)) - 1};
    const int crb = bd + 6 > 16 ? bd + 6 : 16;
    const Clamp cr{-(1 << (crb - 1)), (1 << (crb - 1)) - 1};
    if (g.r < H && g.r < 32) {
        int t[W];
        int* rowp = s.buf + g.r * W;
#pragma unroll
        for (int j = 0; j < W; j++) t[j] = j < 32 ? rowp[j] : 0;
        if constexpr (ABS_D == 1) {
#pragma unroll
            for (int j = 0; j < W; j++) t[j] = rnd12((long long)t[j] * 2896);
        }
        constexpr int kRs = kRowShift[TX];
        const int rsh = lossless ? 0 : kRs;
        if (lossless) {
            if constexpr (W == 4) iwht4(t, 2);
        } else {
            tx1d<LW>(t, row_kind(tu.tx_type), rr);
        }
#pragma unroll
        for (int j = 0; j < W; j++) {
            int v = rsh ? (t[j] + (1 << (rsh - 1))) >> rsh : t[j];
            rowp[j] = min(max(v, cr.lo), cr.hi);
        }
    }
    g.sync();
    if (g.r < W) {
        const int lane = g.r;
        int t[H];
#pragma unroll
        for (int i = 0; i < H; i++) t[i] = s.buf[i * W + lane];
        if (lossless) {
            if constexpr (H == 4) iwht4(t, 0);
        } else {
            tx1d<LH>(t, col_kind(tu.tx_type), cr);
        }
        const int csh = lossless ? 0 : 4;
        const int tt = tu.tx_type;
        const bool fud = tt == 4 || tt == 8 || tt == 14 || tt == 6;
        const bool flr = tt == 5 || tt == 7 || tt == 15 || tt == 6;
        const int x = flr ? W - 1 - lane : lane;
#pragma unroll
        for (int i = 0; i < H; i++) {
            const int y = fud ? H - 1 - i : i;
            out[y * W + x] = csh ? (t[i] + (1 << (csh - 1))) >> csh : t[i];
        }
    }
    g.sync();
}

// One residual task: its compact levels, then residual_store.
template <int TX, class G, class S>
__device__ __forceinline__ void residual_task(const G& g, S& s, const IntraFrame& F, const av1g_tu& tu, int32_t* out) {
    constexpr int W = kTxW[TX], H = kTxH[TX];
    constexpr int TW = W < 32 ? W : 32, TH = H < 32 ? H : 32, NC = TW * TH, K = (NC + G::N - 1) / G::N;
    int cf[K];
    const int32_t* lv = F.coeffs + tu.coeff_offset;
#pragma unroll
    for (int q = 0; q < K; q++) {
        const int k = g.r + q * G::N;
        cf[q] = k < NC ? __ldg(lv + k) : 0;
    }
    residual_store<TX>(g, s, F, tu, cf, out);
}

// ---- small TUs of the common kinds -------------------------------------------
// What bounds a TU is latency: it is a chain of shared-memory round trips on
// the wavefront's critical path, run by a single warp at the issue latency of
// dependent instructions.  So all that does not depend on samples is worked
// out ahead, while other groups run earlier levels (fast_decode): where each
// lane's edge samples, filter taps, prediction taps, residual and destination
// lie.  What is left (fast_run) is loads, a few multiplications and stores.

struct Prog {
    int cls, bits;
    // places in the copy are kept as indexes: a pointer carried through a
    // record would be a 64-bit generic one
    int cp;             // the lane's first four samples in the copy
    uint8_t* out;       // and in HBM
    int cs, cstep, ostep;  // copy row pitch; from the first four samples to the second
    int ok;             // bit 0 / 1: the first / second four exist; bit 2 / 3: and lie inside the plane
    int4 r0, r1;        // their residual, 0 where none applies
    // directional: per edge element of the lane, its place from the TU's first
    // sample (low half, signed) and in the raw edge arrays (bits 16-23); its
    // taps in them; coefficients and places after the edge filter
    // DC: element places in src; recip and edge length in px
    int two;            // directional: some lanes have a second edge element; copied edges: rows between the groups
    int src[2];
    uint32_t tap[2], flt[2];
    // prediction taps of the two groups: places in the edge arrays, weights
    uint32_t px[2], wt[2];
    int tp;             // the TU's first sample in the copy
};

// flt: k0 | k1 << 4 | k2 << 8 | (place << 16) | bits 13 / 14: tap -2 / -1 is
// the corner | bit 15: upsampled (place holds the interpolated sample, the
// next one the sample itself) | bit 31: the element exists
__device__ __forceinline__ void fast_decode(Prog& d, const TuRec* rec, const IntraFrame& F, const SbCtx& c,
                                            const int32_t* __restrict__ pool, int lane) {
    constexpr int E = WScr::E;
    const TuHead t = rec->h;
    const PlaneDev& P = F.planes[t.plane];
    const int LW = t.dims & 15, LH = t.dims >> 4, W = 1 << LW, H = 1 << LH, Q = 1 << (LW + LH - 2);
    const int hbd = F.hbd, cs = c.cs[t.plane];
    const int q = lane < Q ? lane : 0, i = q >> (LW - 2), j = (q << 2) & (W - 1), rows = 128 >> LW;
    d.cls = t.cls;
    d.bits = t.bits;
    d.tp = t.coff;
    d.cp = t.coff + i * cs + j;
    d.cs = cs;
    d.cstep = rows * cs;
    d.ostep = rows * P.stride;
    d.out = P.p + (size_t)(t.y + i) * P.stride + ((size_t)(t.x + j) << hbd);
    const bool a0 = lane < Q, a1 = lane + 32 < Q;
    const bool in0 = a0 && t.y + i < P.h && t.x + j < P.w, in1 = a1 && t.y + i + rows < P.h && t.x + j < P.w;
    d.ok = (a0 ? 1 : 0) | (a1 ? 2 : 0) | (in0 ? 4 : 0) | (in1 ? 8 : 0) | (Q > 32 ? 16 : 0);
    d.r0 = d.r1 = make_int4(0, 0, 0, 0);
    if (t.bits & R_RES) {
        // chroma past the plane is not merged (luma is: chroma from luma reads it)
        const int4* rp = reinterpret_cast<const int4*>(pool + t.res);
        if (t.plane == 0 ? a0 : in0) d.r0 = __ldg(rp + lane);
        if (t.plane == 0 ? a1 : in1) d.r1 = __ldg(rp + lane + 32);
    }
    if (t.cls >= C_D1 && t.cls <= C_D3) {
        const bool ha = t.bits & R_ABOVE, hl = t.bits & R_LEFT, edge = t.bits & R_EDGE;
        const int ea = t.ea, total = ea + 1 + t.el;
        d.two = total > 32;
#pragma unroll
        for (int x = 0; x < 2; x++) {
            const int k = lane + 32 * x;
            if (x && !d.two) break;
            const bool above = k <= ea;
            const int kk = above ? k : k - ea, p = kk - 1;  // position along its edge
            const bool from_row = above ? ha : !hl;
            const int xo = from_row ? (!above ? 0 : p < 0 ? (hl ? -1 : 0) : min(p, t.na - 1)) : -1;
            const int yo = from_row ? -1 : above ? 0 : min(p, t.nl - 1);
            const int bs = above ? 3 : E + 3;  // place of the edge's corner
            const bool live = k < total;
            d.src[x] = ((yo * cs + xo) & 0xffff) | (bs + kk) << 16;
            if (!live) d.src[x] = 0;
            d.flt[x] = live ? 0x80000000u : 0u;
            if (edge) {
                const int st = above ? t.strength & 15 : t.strength >> 4, sz = above ? t.fa : t.fl;
                const int n = above ? ea : t.el;
                const bool up = t.bits & (above ? R_UPA : R_UPL);
                const int hi = up ? n : sz - 1;
                const bool filt = st && kk && kk < sz;
                const uint32_t tm2 = bs + max(kk - 2, 0), tm1 = bs + max(kk - 1, 0), tp1 = bs + min(kk + 1, max(hi, 0)),
                               tp2 = bs + min(kk + 2, max(hi, 0));
                d.tap[x] = tm2 | tm1 << 8 | tp1 << 16 | tp2 << 24;
                const uint32_t k0 = filt && st == 3 ? 2 : 0, k1 = filt ? (st == 2 ? 5 : 4) : 0,
                               k2 = filt ? (st == 1 ? 8 : st == 2 ? 6 : 4) : 16;
                const bool ups = up && kk;
                // position -1, or -2 of an upsampled edge, for the corner
                const uint32_t place = ups ? bs + 2 * kk - 2 : bs + kk - (up ? 1 : 0);
                d.flt[x] |= k0 | k1 << 4 | k2 << 8 | (kk <= 2 && kk ? 1u << 13 : 0) | (kk == 1 ? 1u << 14 : 0) |
                            (ups ? 1u << 15 : 0) | place << 16;
                if (!live) d.flt[x] = 0;
            }
        }
        // prediction taps (predict_intra_directional, cdf.rs:2879-3010)
        const int ua = t.bits & R_UPA ? 1 : 0, ul = t.bits & R_UPL ? 1 : 0;
#pragma unroll
        for (int x = 0; x < 2; x++) {
            if (x && Q <= 32) break;
            const int ii = i + x * rows;
            uint32_t pa = 0, wa = 0;
#pragma unroll
            for (int e = 0; e < 4; e++) {
                int at, sh;
                if (t.cls == C_D2) {
                    const int ix = ((j + e) << 6) - (ii + 1) * t.dx, bx = ix >> (6 - ua);
                    const int iy = (ii << 6) - (j + e + 1) * t.dy, by = max(iy >> (6 - ul), -(1 << ul));
                    const bool fa = bx >= -(1 << ua);
                    at = fa ? 4 + bx : E + 4 + by;
                    sh = ((fa ? ix << ua : iy << ul) >> 1) & 0x1F;
                } else {
                    const bool d3 = t.cls == C_D3;
                    const int up = d3 ? ul : ua, maxb = (W + H - 1) << up;
                    const int idx = ((d3 ? j + e : ii) + 1) * (d3 ? t.dy : t.dx);
                    const int base = (idx >> (6 - up)) + ((d3 ? ii : j + e) << up);
                    at = (d3 ? E + 4 : 4) + min(base, maxb);
                    sh = base < maxb ? ((idx << up) >> 1) & 0x1F : 0;  // past the end: its last sample
                }
                pa |= (uint32_t)at << (8 * e);
                wa |= (uint32_t)sh << (8 * e);
            }
            d.px[x] = pa;
            d.wt[x] = wa;
        }
    } else if (t.cls == C_DC) {
        const int ea = t.ea, n = ea + t.el;
#pragma unroll
        for (int x = 0; x < 2; x++) {
            const int k = lane + 32 * x;
            d.src[x] = k < ea ? k - cs : k < n ? (k - ea) * cs - 1 : -0x8000;
        }
        d.px[0] = rec->recip;
        d.px[1] = n;
        if (t.bits & R_CFL) {
            // luma of the lane's samples: the place of the first group's row
            // and column, limits and alpha
            d.tap[0] = t.x + j;
            d.tap[1] = t.y + i;
            d.flt[0] = t.cx | (uint32_t)t.cy << 16;
            d.flt[1] = (uint32_t)(int)t.alpha;
            d.wt[0] = LW + LH;
            d.wt[1] = rows;
        }
    } else if (t.cls == C_PAL) {
        const uint8_t* m = F.maps + t.map + i * t.stride + j;
#pragma unroll
        for (int x = 0; x < 2; x++) {
            if (x && Q <= 32) break;
            const uint8_t* mm = m + x * (a1 ? rows : 0) * t.stride;
            uint32_t v[4];
#pragma unroll
            for (int e = 0; e < 4; e++) v[e] = rec->colors[mm[e] & 7];
            d.px[x] = v[0] | v[1] << 16;
            d.wt[x] = v[2] | v[3] << 16;
        }
    } else if (t.cls == C_FI) {
        d.px[0] = t.misc & 7;
        d.px[1] = W >> 2;
        d.wt[0] = H >> 1;
    } else {
        d.px[0] = W;
        d.px[1] = H;
        d.wt[0] = j;
        d.wt[1] = i;
        d.two = rows;
    }
}

// Four predicted samples: curr_frame_step3_merge (cdf.rs:17398-17470),
// Clip1(pred + residual), to the copy and to HBM (other superblocks read them
// once this level is published).  ok: bit 0 they exist, bit 2 they lie inside
// the plane.
__device__ __forceinline__ void put4(int v0, int v1, int v2, int v3, const int4& r, int maxv, uint16_t* cache, int cp,
                                     uint8_t* out, int ok, int hbd) {
    v0 = __viaddmin_s32_relu(v0, r.x, maxv);
    v1 = __viaddmin_s32_relu(v1, r.y, maxv);
    v2 = __viaddmin_s32_relu(v2, r.z, maxv);
    v3 = __viaddmin_s32_relu(v3, r.w, maxv);
    const uint2 pk = make_uint2(__byte_perm(v0, v1, 0x5410), __byte_perm(v2, v3, 0x5410));
    if (ok & 1) *reinterpret_cast<uint2*>(cache + cp) = pk;
    if (ok & 4) {
        if (hbd) *reinterpret_cast<uint2*>(out) = pk;
        else *reinterpret_cast<uint32_t*>(out) = __byte_perm(pk.x, pk.y, 0x6420);
    }
}

// Each kind is one straight path to its stores: a branch costs a lone warp more
// than the instructions it skips.
__device__ __forceinline__ void fast_run(const Prog& d, WScr& s, const IntraFrame& F, const SbCtx& c, uint16_t* cache,
                                         const Tables& tb, int lane) {
    constexpr int E = WScr::E;
    const int maxv = (1 << F.bd) - 1, hbd = F.hbd, cs = d.cs, tp = d.tp;
    const bool second = d.ok & 16;
    if (d.cls >= C_D1 && d.cls <= C_D3) {
        const int v0 = cache[tp + (int16_t)(d.src[0] & 0xffff)];
        int v1 = 0;
        if (d.two) v1 = cache[tp + (int16_t)(d.src[1] & 0xffff)];
        if (d.flt[0] >> 31) s.raw[d.src[0] >> 16] = (uint16_t)v0;
        if (d.two && d.flt[1] >> 31) s.raw[d.src[1] >> 16] = (uint16_t)v1;
        if (lane == 0) s.raw[E + 3] = (uint16_t)v0;
        __syncwarp();
        int ed = 0;  // raw, or fin 2 E further
        if (d.bits & R_EDGE) {
            // corner filter, intra_edge_filter (cdf.rs:2760) or
            // intra_edge_upsample (cdf.rs:2700) of both edges at once
            int fc = 0;
            if (d.bits & R_CORNER) fc = (s.raw[E + 4] * 5 + s.raw[3] * 6 + s.raw[4] * 5 + 8) >> 4;
#pragma unroll
            for (int x = 0; x < 2; x++) {
                if (x && !d.two) break;
                const uint32_t ta = d.tap[x], fl = d.flt[x];
                int m2 = s.raw[ta & 0xff], m1 = s.raw[(ta >> 8) & 0xff], p1 = s.raw[(ta >> 16) & 0xff], p2 = s.raw[ta >> 24];
                int v = x ? v1 : v0;
                if (d.bits & R_CORNER) {
                    m2 = fl & (1u << 13) ? fc : m2;
                    m1 = fl & (1u << 14) ? fc : m1;
                    if (x == 0) v = lane == 0 ? fc : v;
                }
                const bool up = fl & (1u << 15);
                const int k0 = up ? -1 : (int)(fl & 15), k1 = up ? 9 : (int)(fl >> 4) & 15, k2 = up ? 9 : (int)(fl >> 8) & 31;
                const int k3 = up ? -1 : k1, k4 = up ? 0 : k0;
                const int f = __vimin_s32_relu((k0 * m2 + k1 * m1 + k2 * v + (k3 * p1 + k4 * p2 + 8)) >> 4, maxv);
                const int place = (fl >> 16) & 0x7fff;
                if (fl >> 31) s.fin[place] = (uint16_t)f;
                if (up) s.fin[place + 1] = (uint16_t)v;
                if (x == 0 && lane == 0) s.fin[E + (d.bits & R_UPL ? 2 : 3)] = (uint16_t)v;  // the left edge's corner
            }
            ed = (int)(s.fin - s.raw);
            __syncwarp();
        }
        const uint16_t* e0 = s.raw + ed;
#pragma unroll
        for (int x = 0; x < 2; x++) {
            if (x && !second) break;
            const uint32_t px = d.px[x], wt = d.wt[x];
            int v[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const uint16_t* a = e0 + ((px >> (8 * e)) & 0xff);
                const int lo = a[0], hi = a[1], w = (wt >> (8 * e)) & 0xff;
                v[e] = lo + (((hi - lo) * w + 16) >> 5);
            }
            put4(v[0], v[1], v[2], v[3], x ? d.r1 : d.r0, maxv, cache, d.cp + x * d.cstep, d.out + (x ? d.ostep : 0),
                 d.ok >> x, hbd);
        }
    } else if (d.cls == C_DC) {
        // predict_intra_dc_pred (cdf.rs:1348); a missing edge has length 0.
        // The quotient by the reciprocal is exact: sum + n / 2 < 2^20, n <= 128.
        int part = 0;
        if (d.src[0] != -0x8000) part = cache[tp + d.src[0]];
        if (d.src[1] != -0x8000) part += cache[tp + d.src[1]];
        const unsigned n = d.px[1], sum = __reduce_add_sync(0xffffffffu, part);
        const int dc = n == 0 ? (maxv + 1) >> 1 : __umulhi(sum + (n >> 1), d.px[0]);
        if (!(d.bits & R_CFL)) {
            put4(dc, dc, dc, dc, d.r0, maxv, cache, d.cp, d.out, d.ok, hbd);
            if (second) put4(dc, dc, dc, dc, d.r1, maxv, cache, d.cp + d.cstep, d.out + d.ostep, d.ok >> 1, hbd);
        } else {
            // predict_chroma_from_luma_into_curr_frame (cdf.rs:17256-17340)
            const int ssx = F.ssx, ssy = F.ssy, ycs = c.cs[0];
            const int cx = d.flt[0] & 0xffff, cy = d.flt[0] >> 16;
            const int Y = c.off[0] - c.rect[0].y * ycs - c.rect[0].x;
            int xs[4], l[2][4] = {};
#pragma unroll
            for (int e = 0; e < 4; e++) xs[e] = min((int)(d.tap[0] + e) << ssx, cx);
            part = 0;
#pragma unroll
            for (int x = 0; x < 2; x++) {
                if (x && !second) break;
                const int yp = Y + min((int)(d.tap[1] + x * d.wt[1]) << ssy, cy) * ycs;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const uint16_t* p = cache + yp + xs[e];
                    if (ssx) {
                        uint32_t w = *reinterpret_cast<const uint32_t*>(p);  // two samples below 4096: no carry
                        if (ssy) w += *reinterpret_cast<const uint32_t*>(p + ycs);
                        l[x][e] = (int)((w & 0xffff) + (w >> 16)) << (2 - ssy);
                    } else {
                        l[x][e] = ssy ? (p[0] + p[ycs]) << 2 : p[0] << 3;
                    }
                    part += l[x][e];
                }
            }
            if (!(d.ok & 1)) part = 0;  // this lane repeats another's samples
            const unsigned lsum = __reduce_add_sync(0xffffffffu, part);
            const int avg = (int)((lsum + (1u << (d.wt[0] - 1))) >> d.wt[0]);
#pragma unroll
            for (int x = 0; x < 2; x++) {
                if (x && !second) break;
                int v[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int al = (int)d.flt[1] * (l[x][e] - avg);
                    const int sc = (al + 32 - (al < 0)) >> 6;  // rounds halves away from zero
                    v[e] = (d.ok >> (2 + x)) & 1 ? min(max(dc + sc, 0), maxv) : dc;
                }
                put4(v[0], v[1], v[2], v[3], x ? d.r1 : d.r0, maxv, cache, d.cp + x * d.cstep,
                     d.out + (x ? d.ostep : 0), d.ok >> x, hbd);
            }
        }
    } else if (d.cls >= C_V && d.cls <= C_PAETH) {
        const int j = d.wt[0], W = d.px[0], H = d.px[1];
        const uint2 aw = *reinterpret_cast<const uint2*>(cache + tp - cs + j);
        const int l0 = cache[tp + (int)d.wt[1] * cs - 1];
        const int l1 = second ? cache[tp + (int)(d.wt[1] + d.two) * cs - 1] : 0;
        const int a[4] = {(int)(aw.x & 0xffff), (int)(aw.x >> 16), (int)(aw.y & 0xffff), (int)(aw.y >> 16)};
        const int corner = cache[tp - cs - 1], ar = cache[tp + W - 1 - cs], lb = cache[tp + (H - 1) * cs - 1];
        const uint32_t wx = *reinterpret_cast<const uint32_t*>(tb.sm + W - 4 + j);
        const int wy0 = tb.sm[H - 4 + d.wt[1]], wy1 = second ? tb.sm[H - 4 + d.wt[1] + d.two] : 0;
#pragma unroll
        for (int x = 0; x < 2; x++) {
            if (x && !second) break;
            const int l = x ? l1 : l0, wy = x ? wy1 : wy0;
            int v[4];
            if (d.cls >= C_SMOOTH && d.cls <= C_SMOOTH_H) {  // SMOOTH (cdf.rs:2267), SMOOTH_V, SMOOTH_H
                // weights of the two directions, 0 for the one a mode leaves out
                const int kv = d.cls != C_SMOOTH_H, kh = d.cls != C_SMOOTH_V, sh = 7 + kv + kh;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int w = (wx >> (8 * e)) & 0xff;
                    const int vv = wy * (a[e] - lb) + 256 * lb, vh = w * (l - ar) + 256 * ar;
                    v[e] = ((kv ? vv : 0) + (kh ? vh : 0) + (1 << (sh - 1))) >> sh;
                }
            } else if (d.cls == C_PAETH) {  // cdf.rs:2077
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int base = a[e] + l - corner;
                    const int dl = abs(base - l), dt = abs(base - a[e]), dtl = abs(base - corner);
                    v[e] = (dl <= dt && dl <= dtl) ? l : (dt <= dtl ? a[e] : corner);
                }
            } else {
#pragma unroll
                for (int e = 0; e < 4; e++) v[e] = d.cls == C_V ? a[e] : l;
            }
            put4(v[0], v[1], v[2], v[3], x ? d.r1 : d.r0, maxv, cache, d.cp + x * d.cstep, d.out + (x ? d.ostep : 0),
                 d.ok >> x, hbd);
        }
    } else if (d.cls == C_PAL) {  // predict_palette (cdf.rs:11907); indices checked on the host
        put4(d.px[0] & 0xffff, d.px[0] >> 16, d.wt[0] & 0xffff, d.wt[0] >> 16, d.r0, maxv, cache, d.cp, d.out, d.ok, hbd);
        if (second)
            put4(d.px[1] & 0xffff, d.px[1] >> 16, d.wt[1] & 0xffff, d.wt[1] >> 16, d.r1, maxv, cache, d.cp + d.cstep,
                 d.out + d.ostep, d.ok >> 1, hbd);
    } else {
        if (d.cls == C_FI) {
            // predict_intra_recursive (cdf.rs:2145): 4x2 cells, wavefront over
            // i2 + j4; eight lanes per cell and a column of cells per eight
            // lanes (two for 32 wide).  The edges lie in place around the
            // block, so every cell reads the same way.
            const int W4 = d.px[1], H2 = d.wt[0], o = lane & 7;
            const uint2 tw = *reinterpret_cast<const uint2*>(tb.fi[d.px[0]][o]);
            auto tap = [&](int q) { return (int)(int8_t)((q < 4 ? tw.x : tw.y) >> (8 * (q & 3))); };
            const int w0 = tap(0), w1 = tap(1), w2 = tap(2), w3 = tap(3), w4 = tap(4), w5 = tap(5), w6 = tap(6);
            const int oo = (o >> 2) * cs + (o & 3), j4 = lane >> 3;
            int up = tp + (4 - 2 * cs) * j4 - cs;  // the row above the lane's cell, whose row is dd - j4
#pragma unroll 1
            for (int dd = 0; dd < W4 + H2 - 1; dd++) {
                auto cell = [&](int at) {  // at: the row above it
                    const uint16_t* q = cache + at;
                    const int lo = w0 * q[-1] + w1 * q[0] + w2 * q[1] + 8;
                    const int hi = w3 * q[2] + w4 * q[3] + w5 * q[cs - 1] + w6 * q[2 * cs - 1];
                    cache[at + cs + oo] = (uint16_t)__vimin_s32_relu((lo + hi) >> 4, maxv);
                };
                if (j4 < W4 && (unsigned)(dd - j4) < (unsigned)H2) cell(up);
                if (W4 > 4 && (unsigned)(dd - j4 - 4) < (unsigned)H2) cell(up + 16 - 8 * cs);
                up += 2 * cs;
                __syncwarp();
            }
        }
        // in the copy already
        const uint2 p0 = *reinterpret_cast<const uint2*>(cache + d.cp);
        put4(p0.x & 0xffff, p0.x >> 16, p0.y & 0xffff, p0.y >> 16, d.r0, maxv, cache, d.cp, d.out, d.ok, hbd);
        if (second) {
            const uint2 p1 = *reinterpret_cast<const uint2*>(cache + d.cp + d.cstep);
            put4(p1.x & 0xffff, p1.x >> 16, p1.y & 0xffff, p1.y >> 16, d.r1, maxv, cache, d.cp + d.cstep,
                 d.out + d.ostep, d.ok >> 1, hbd);
        }
    }
}

// The first four residual samples of the thread of rank r in a TU.
__device__ __forceinline__ int4 first_res(const TuRec* rec, const int32_t* __restrict__ pool, int r) {
    const int Q = 1 << ((rec->h.dims & 15) + (rec->h.dims >> 4) - 2);
    if (!(rec->h.bits & R_RES) || r >= Q) return make_int4(0, 0, 0, 0);
    return __ldg(reinterpret_cast<const int4*>(pool + rec->h.res) + r);
}

// The general form, for any TU: the large ones (a group of warps each) and what
// fast_decode does not take (edges past the copy or cut off by the frame's edge,
// inter-intra blocks, intra block copies, unaligned positions).  One body
// that takes the size at run time keeps the code inside the instruction cache,
// which a body per transform size missed on almost every TU.
template <class G, class S>
__device__ __forceinline__ void run_tu(const G& g, S& s, const TuRec* rec, const IntraFrame& F, const SbCtx& c,
                                       uint16_t* cache, const Tables& tb, const int32_t* __restrict__ pool,
                                       int4 rv) {
    const TuHead t = rec->h;
    const int tid = g.r, pl = t.plane, bd = F.bd, hbd = F.hbd, maxv = (1 << bd) - 1;
    const int LW = t.dims & 15, LH = t.dims >> 4, W = 1 << LW, H = 1 << LH, Q = 1 << (LW + LH - 2);
    const PlaneDev P = F.planes[pl];
    const int sx = t.x, sy = t.y, cs = c.cs[pl], wlim = P.w - sx, hlim = P.h - sy;
    uint16_t* tp = cache + t.coff;
    uint8_t* dst = P.p + (size_t)sy * P.stride + ((size_t)sx << hbd);
    constexpr int E = S::E;
    // A[k] == AboveRow[k], Lc[k * ls] == LeftCol[k]
    const uint16_t* A = tp - cs;
    const uint16_t* Lc = tp - 1;
    int ls = cs;
    if (t.cls >= C_DC && t.cls <= C_FI && !(t.where & W_DIRECT)) {
        // edge arrays (intra_predict_block_samples, cdf.rs:17030-17075)
        const bool ha = t.bits & R_ABOVE, hl = t.bits & R_LEFT;
        const int ea = t.ea, total = ea + 1 + t.el;
        const int mid = 1 << (bd - 1);
        for (int k = tid; k < total; k += G::N) {
            const bool above = k <= ea;
            const int i = above ? k - 1 : k - ea - 1;
            int v;
            // a missing row repeats the left column's first sample, a missing column the row's
            const bool from_row = above ? ha : !hl;
            const int xo = from_row ? (!above ? 0 : i < 0 ? (hl ? -1 : 0) : min(i, t.na - 1)) : -1;
            const int yo = from_row ? -1 : above ? 0 : min(i, t.nl - 1);
            if (!ha && !hl) v = above ? (i < 0 ? mid : mid - 1) : mid + 1;
            else if (t.where & W_COPY) v = tp[yo * cs + xo];
            else v = rdp(F, c, cache, pl, sy + yo, sx + xo);
            s.raw[(above ? 4 : E + 4) + i] = (uint16_t)v;
            if (k == 0) s.raw[E + 3] = (uint16_t)v;
        }
        A = s.raw + 4;
        Lc = s.raw + E + 4;
        ls = 1;
        g.sync();
        if (t.bits & R_EDGE) {
            // corner filter, intra_edge_filter (cdf.rs:2760) or
            // intra_edge_upsample (cdf.rs:2700) of both edges at once
            const int nA = ea + 1, nT = nA + t.el + 1;
            int fc = s.raw[3];
            if (t.bits & R_CORNER) fc = (s.raw[E + 4] * 5 + fc * 6 + s.raw[4] * 5 + 8) >> 4;
            for (int k = tid; k < nT; k += G::N) {
                const bool left = k >= nA;
                const int kk = left ? k - nA : k;  // position kk - 1
                const uint16_t* R = s.raw + (left ? E + 3 : 3);
                uint16_t* D = s.fin + (left ? E + 3 : 3);
                if (t.bits & (left ? R_UPL : R_UPA)) {
                    const int n = left ? t.el : ea;
                    if (kk == 0) {
                        D[-1] = R[0];
                    } else {
                        const int sum = -R[max(kk - 2, 0)] + 9 * R[kk - 1] + 9 * R[kk] - R[min(kk + 1, n)];
                        D[2 * kk - 2] = (uint16_t)clip3(0, maxv, (sum + 8) >> 4);
                        D[2 * kk - 1] = (uint16_t)min((int)R[kk], maxv);
                    }
                } else {
                    const int st = left ? t.strength >> 4 : t.strength & 15, sz = left ? t.fl : t.fa;
                    int v = kk ? R[kk] : fc;
                    if (st && kk && kk < sz) {
                        const int k0 = st == 3 ? 2 : 0, k1 = st == 2 ? 5 : 4, k2 = st == 1 ? 8 : st == 2 ? 6 : 4;
                        auto tap = [&](int q) { return q <= 0 ? fc : (int)R[min(q, sz - 1)]; };
                        v = (k0 * (tap(kk - 2) + tap(kk + 2)) + k1 * (tap(kk - 1) + tap(kk + 1)) + k2 * v + 8) >> 4;
                    }
                    D[kk] = (uint16_t)v;
                }
            }
            A = s.fin + 4;
            Lc = s.fin + E + 4;
            g.sync();
        }
    }
    int dc = 0;
    if (t.cls == C_DC) {
        // predict_intra_dc_pred (cdf.rs:1348); a missing edge has length 0
        int part = 0;
        for (int i = tid; i < t.ea + t.el; i += G::N) part += i < t.ea ? A[i] : Lc[(i - t.ea) * ls];
        const unsigned n = t.ea + t.el, sum = gsum(g, s, part);
        // the quotient by the reciprocal is exact: sum + n / 2 < 2^20, n <= 128
        dc = n == 0 ? 1 << (bd - 1) : __umulhi(sum + (n >> 1), rec->recip);
    } else if (t.cls == C_FI) {
        // predict_intra_recursive (cdf.rs:2145): 4x2 cells, wavefront over
        // i2 + j4, reading earlier cells back from the copy
        const int W4 = W >> 2, H2 = H >> 1, o = tid & 7, i1 = o >> 2, j1 = o & 3;
        const uint2 tw = *reinterpret_cast<const uint2*>(tb.fi[t.misc & 7][o]);
        auto tap = [&](int i) { return (int)(int8_t)((i < 4 ? tw.x : tw.y) >> (8 * (i & 3))); };
        for (int dd = 0; dd < W4 + H2 - 1; dd++) {
            for (int bb = tid >> 3;; bb += G::N >> 3) {
                const int i2 = max(0, dd - (W4 - 1)) + bb, j4 = dd - i2;
                if (i2 >= H2 || j4 < 0) break;
                const uint16_t* up = i2 == 0 ? A + (j4 << 2) : tp + ((i2 << 1) - 1) * cs + (j4 << 2);
                const int ps = j4 == 0 ? ls : cs;
                const uint16_t* lf = j4 == 0 ? Lc + (i2 << 1) * ls : tp + (i2 << 1) * cs + (j4 << 2) - 1;
                int acc = tap(0) * (j4 == 0 && i2 > 0 ? lf[-ps] : up[-1]);
#pragma unroll
                for (int i = 1; i < 5; i++) acc += tap(i) * up[i - 1];
                acc += tap(5) * lf[0] + tap(6) * lf[ps];
                const int v = acc >= 0 ? (acc + 8) >> 4 : -(((-acc) + 8) >> 4);
                tp[((i2 << 1) + i1) * cs + (j4 << 2) + j1] = (uint16_t)clip3(0, maxv, v);
            }
            g.sync();
        }
    } else if (t.cls == C_BC) {
        // predict_intrabc_leaf_into_curr_frame (cdf.rs:19235): BILINEAR
        // block_inter_prediction from the pre-filter plane at unit scale,
        // start = (x << 10) + (((2 * mv) >> ss) << 6) + 32, clamped to the
        // mi-padded plane (the reference's window clamp is the same set).
        // The whole block is predicted before any of it is stored.
        const int pss_x = pl ? F.ssx : 0, pss_y = pl ? F.ssy : 0;
        const int stx = (sx << 10) + ((2 * (int16_t)(t.map & 0xffff)) >> pss_x) * 64 + 32;
        const int sty = (sy << 10) + ((2 * (int16_t)(t.map >> 16)) >> pss_y) * 64 + 32;
        const int b0 = bd == 12 ? 5 : 3, b1 = bd == 12 ? 9 : 11;
        const int hph = (stx >> 6) & 15, vph = (sty >> 6) & 15;
#pragma unroll 1
        for (int k = tid; k < W * H; k += G::N) {
            const int i = k >> LW, j = k & (W - 1);
            const int xi = ((stx >> 10) + j) - 3, yi = ((sty >> 10) + i) - 3;
            int acc = 0;
#pragma unroll 1
            for (int tt = 0; tt < 8; tt++) {
                const int vc = c_subpel[3][vph][tt];
                if (!vc) continue;
                const int yy = min(max(yi + tt, 0), P.h - 1);
                int hsum = 0;
#pragma unroll 1
                for (int u = 0; u < 8; u++) {
                    const int hc = c_subpel[3][hph][u];
                    if (hc) hsum += hc * rdp(F, c, cache, pl, yy, min(max(xi + u, 0), P.w - 1));
                }
                acc += vc * ((hsum + ((1 << b0) >> 1)) >> b0);
            }
            s.buf[k] = (uint16_t)min(max((acc + (1 << (b1 - 1))) >> b1, 0), maxv);
        }
        g.sync();
        for (int k = tid; k < W * H; k += G::N) tp[(k >> LW) * cs + (k & (W - 1))] = s.buf[k];
        g.sync();
    }
    int cfl_avg = 0;
    if (t.bits & R_CFL) {
        // predict_chroma_from_luma_into_curr_frame (cdf.rs:17256-17340).  The
        // block's luma transforms may run past the mi-grid plane; their
        // samples there stay in the superblock's staged copy (the reference's
        // LumaOverhang side store, cdf.rs:15938, read at cdf.rs:17292-17305),
        // which spans the whole superblock.  Luma neither in the plane nor in
        // that copy reads as 0.
        const int ssx = F.ssx, ssy = F.ssy;
        int part = 0;
        if (t.where & W_CFL) {
            const uint16_t* Y = cache + c.off[0] - c.rect[0].y * c.cs[0] - c.rect[0].x;
            const int ycs = c.cs[0];
#pragma unroll 1
            for (int q = tid; q < Q; q += G::N) {
                const int i = q >> (LW - 2), j = (q << 2) & (W - 1);
                const uint16_t* yp = Y + min((sy + i) << ssy, (int)t.cy) * ycs;
                int v[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const uint16_t* p = yp + min((sx + j + e) << ssx, (int)t.cx);
                    if (ssx) {
                        uint32_t w = *reinterpret_cast<const uint32_t*>(p);  // two samples below 4096: no carry
                        if (ssy) w += *reinterpret_cast<const uint32_t*>(p + ycs);
                        v[e] = (int)((w & 0xffff) + (w >> 16)) << (2 - ssy);
                    } else {
                        v[e] = ssy ? (p[0] + p[ycs]) << 2 : p[0] << 3;
                    }
                    part += v[e];
                }
                *reinterpret_cast<uint2*>(s.buf + 4 * q) =
                    make_uint2((uint32_t)v[0] | (uint32_t)v[1] << 16, (uint32_t)v[2] | (uint32_t)v[3] << 16);
            }
        } else {
            const PlaneDev& Y = F.planes[0];
            const int4 yr = c.rect[0];
#pragma unroll 1
            for (int k = tid; k < W * H; k += G::N) {
                const int i = k >> LW, j = k & (W - 1);
                const int ly = min((sy + i) << ssy, (int)t.cy), lx = min((sx + j) << ssx, (int)t.cx);
                int acc = 0;
                for (int ddy = 0; ddy <= ssy; ddy++)
                    for (int ddx = 0; ddx <= ssx; ddx++) {
                        const int yy = ly + ddy, xx = lx + ddx;
                        const bool staged =
                            (unsigned)(yy - yr.y) < (unsigned)yr.w && (unsigned)(xx - yr.x) < (unsigned)yr.z;
                        acc += (staged || (yy < Y.h && xx < Y.w)) ? rdp(F, c, cache, 0, yy, xx) : 0;
                    }
                const int v = acc << (3 - ssx - ssy);  // at most 4 * 4095 * 2
                s.buf[k] = (uint16_t)v;
                part += v;
            }
        }
        const int sum = gsum(g, s, part);  // at most 4096 * 32760, never negative
        cfl_avg = (int)(((unsigned)sum + (1u << (LW + LH - 1))) >> (LW + LH));
        g.sync();
    }
    const int ii = t.misc >> 4;
    const int4* rp = reinterpret_cast<const int4*>(pool + t.res);
#pragma unroll 1
    for (int q = tid; q < Q; q += G::N) {
        const int i = q >> (LW - 2), j = (q << 2) & (W - 1);
        int4 rn = rv;  // the next round's residual
        if ((t.bits & R_RES) && q + G::N < Q) rn = __ldg(rp + q + G::N);
        uint16_t* cp = tp + i * cs + j;
        int v[4];
        switch (t.cls) {
            case C_DC:
#pragma unroll
                for (int e = 0; e < 4; e++) v[e] = dc;
                break;
            case C_H:
#pragma unroll
                for (int e = 0; e < 4; e++) v[e] = Lc[i * ls];
                break;
            case C_V:
            case C_SMOOTH:
            case C_SMOOTH_V:
            case C_SMOOTH_H:
            case C_PAETH: {
                const uint2 aw = *reinterpret_cast<const uint2*>(A + j);
                const int a[4] = {(int)(aw.x & 0xffff), (int)(aw.x >> 16), (int)(aw.y & 0xffff), (int)(aw.y >> 16)};
                if (t.cls == C_V) {
#pragma unroll
                    for (int e = 0; e < 4; e++) v[e] = a[e];
                    break;
                }
                const int l = Lc[i * ls];
                if (t.cls == C_PAETH) {  // cdf.rs:2077
                    const int corner = A[-1];
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int base = a[e] + l - corner;
                        const int dl = abs(base - l), dt = abs(base - a[e]), dtl = abs(base - corner);
                        v[e] = (dl <= dt && dl <= dtl) ? l : (dt <= dtl ? a[e] : corner);
                    }
                    break;
                }
                // SMOOTH (cdf.rs:2267), SMOOTH_V, SMOOTH_H
                const uint32_t wx = *reinterpret_cast<const uint32_t*>(tb.sm + W - 4 + j);
                const int wy = tb.sm[H - 4 + i], ar = A[W - 1], lb = Lc[(H - 1) * ls];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int w = (wx >> (8 * e)) & 0xff;
                    const int vv = wy * a[e] + (256 - wy) * lb, vh = w * l + (256 - w) * ar;
                    v[e] = t.cls == C_SMOOTH ? (vv + vh + 256) >> 9 : ((t.cls == C_SMOOTH_V ? vv : vh) + 128) >> 8;
                }
                break;
            }
            case C_D1:
            case C_D3: {
                // predict_intra_directional (cdf.rs:2879-3010) along one edge
                const bool d3 = t.cls == C_D3;
                const uint16_t* edge = d3 ? Lc : A;
                const int up = t.bits & (d3 ? R_UPL : R_UPA) ? 1 : 0, maxb = (W + H - 1) << up;
                const int step = d3 ? t.dy : t.dx;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int idx = ((d3 ? j + e : i) + 1) * step;
                    const int base = (idx >> (6 - up)) + ((d3 ? i : j + e) << up);
                    const int sh = ((idx << up) >> 1) & 0x1F;
                    v[e] = base < maxb ? (edge[base] * (32 - sh) + edge[base + 1] * sh + 16) >> 5 : edge[maxb];
                }
                break;
            }
            case C_D2: {
                const int ua = t.bits & R_UPA ? 1 : 0, ul = t.bits & R_UPL ? 1 : 0;
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int ix = ((j + e) << 6) - (i + 1) * t.dx, bx = ix >> (6 - ua);
                    const int iy = (i << 6) - (j + e + 1) * t.dy, by = max(iy >> (6 - ul), -(1 << ul));
                    const bool fa = bx >= -(1 << ua);
                    const uint16_t* ed = fa ? A + bx : Lc + by;
                    const int sh = ((fa ? ix << ua : iy << ul) >> 1) & 0x1F;
                    v[e] = (ed[0] * (32 - sh) + ed[1] * sh + 16) >> 5;
                }
                break;
            }
            case C_PAL: {  // predict_palette (cdf.rs:11907); indices checked on the host
                const uint8_t* m = F.maps + t.map + i * t.stride + j;
#pragma unroll
                for (int e = 0; e < 4; e++) v[e] = rec->colors[m[e] & 7];
                break;
            }
            default:  // in the copy already: filter intra, intra block copy, no prediction
#pragma unroll
                for (int e = 0; e < 4; e++) v[e] = cp[e];
                break;
        }
        const bool row_in = i < hlim;
        if (ii) {
            // the intra half of an inter-intra block is blended as it is stored
            // (only inside the plane: the side plane has the plane's extent)
#pragma unroll 1
            for (int e = 0; e < 4; e++)
                if (row_in && j + e < wlim) {
                    const int w = interintra_px(F, t, ii, i, j + e, e == 0 ? v[0] : e == 1 ? v[1] : e == 2 ? v[2] : v[3],
                                                ld_px(F.side[pl], hbd, sy + i, sx + j + e), maxv);
                    if (e == 0) v[0] = w;
                    else if (e == 1) v[1] = w;
                    else if (e == 2) v[2] = w;
                    else v[3] = w;
                }
        }
        if (t.bits & R_CFL) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int al = t.alpha * ((int)s.buf[4 * q + e] - cfl_avg);
                const int sc = al >= 0 ? (al + 32) >> 6 : -(((-al) + 32) >> 6);
                if (row_in && j + e < wlim) v[e] = min(max(v[e] + sc, 0), maxv);
            }
        }
        if (t.bits & R_RES) {
            // curr_frame_step3_merge (cdf.rs:17398-17470): Clip1(pred + residual);
            // luma past the plane is merged too, in the staged copy only (the
            // overhang chroma from luma reads)
            const int r[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (pl == 0 || (row_in && j + e < wlim)) v[e] = min(max(v[e] + r[e], 0), maxv);
        }
        // the final samples to the copy and to HBM: other superblocks read
        // them once this level is published.
        uint8_t* out = dst + (size_t)i * P.stride + (j << hbd);
        if (t.where & W_ALIGNED) {
            const uint2 pk = make_uint2((uint32_t)v[0] | (uint32_t)v[1] << 16, (uint32_t)v[2] | (uint32_t)v[3] << 16);
            *reinterpret_cast<uint2*>(cp) = pk;
            if (row_in && j < wlim) {
                if (hbd) *reinterpret_cast<uint2*>(out) = pk;
                else *reinterpret_cast<uint32_t*>(out) = __byte_perm(pk.x, pk.y, 0x6420);
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                cp[e] = (uint16_t)v[e];
                if (row_in && j + e < wlim) {
                    if (hbd) reinterpret_cast<uint16_t*>(out)[e] = (uint16_t)v[e];
                    else out[e] = (uint8_t)v[e];
                }
            }
        }
        rv = rn;
    }
}

__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ long long gtimer() {
    long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Four samples at column x of a row, as u16 pairs.
__device__ __forceinline__ uint2 ld_quad(const uint8_t* row, int hbd, int x) {
    if (hbd) return __ldcg(reinterpret_cast<const uint2*>(row + 2 * x));
    const uint32_t u = __ldcg(reinterpret_cast<const uint32_t*>(row + x));
    return make_uint2(__byte_perm(u, 0u, 0x4140), __byte_perm(u, 0u, 0x4342));
}

// HBM -> the superblock's area of the copy, four samples per thread (superblock
// origins and row pitches are multiples of four samples).  Subsampled planes of an odd
// number of mode info columns end half a group short: the group's rest is row
// padding, which nothing reads from the copy.
__device__ void load_area(const IntraFrame& F, const SbCtx& c, uint16_t* cache) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int p = 0; p < F.np; p++) {
        const PlaneDev& P = F.planes[p];
        const int4 r = c.rect[p];
        const int rows = min(r.w, P.h - r.y), quads = (min(r.z, P.w - r.x) + 3) >> 2;
        uint16_t* cp = cache + c.off[p];
        for (int k = warp; k < rows; k += kIT / 32) {
            const uint8_t* row = P.p + (size_t)(r.y + k) * P.stride;
            for (int q = lane; q < quads; q += 32)
                *reinterpret_cast<uint2*>(cp + k * c.cs[p] + 4 * q) = ld_quad(row, F.hbd, r.x + 4 * q);
        }
    }
}

// HBM -> the copy's row above and column to the left, by n threads of rank r;
// a thread's loads are in flight together.  What neighbours have not finished
// yet is loaded too and loaded again once a wait on it is over; no TU reads it
// before that.
__device__ void load_border(const IntraFrame& F, const SbCtx& c, uint16_t* cache, int r, int n) {
    constexpr int B = 4;
    auto items = [&](int p) { return (4 + c.rect[p].z + intra_copy_ext(c.rect[p].z)) / 4 + c.rect[p].w; };
    const int n0 = items(0), n1 = F.np > 1 ? items(1) : 0, total = n0 + 2 * n1;
#pragma unroll 1
    for (int base = r; base < total; base += B * n) {
        uint2 v[B];
        int at[B];  // where it goes; the low bit of a group of four's marks it
#pragma unroll
        for (int e = 0; e < B; e++) {
            const int k = base + e * n;
            at[e] = -1;
            if (k >= total) continue;
            const int p = k < n0 ? 0 : k < n0 + n1 ? 1 : 2, q = k - (p == 0 ? 0 : p == 1 ? n0 : n0 + n1);
            const PlaneDev& P = F.planes[p];
            const int4 a = c.rect[p];
            const int groups = (4 + a.z + intra_copy_ext(a.z)) / 4;
            if (q < groups) {
                const int x = a.x - 4 + 4 * q, y = a.y - 1;
                if (y < 0 || x < 0 || x >= P.w) continue;
                v[e] = ld_quad(P.p + (size_t)y * P.stride, F.hbd, x);
                at[e] = 2 * (c.off[p] - c.cs[p] - 4 + 4 * q) + 1;
            } else {
                const int x = a.x - 1, y = a.y + q - groups;
                if (x < 0 || y >= P.h) continue;
                const uint8_t* row = P.p + (size_t)y * P.stride;
                v[e].x = F.hbd ? __ldcg(reinterpret_cast<const unsigned short*>(row) + x) : __ldcg(row + x);
                at[e] = 2 * (c.off[p] + (q - groups) * c.cs[p] - 1);
            }
        }
#pragma unroll
        for (int e = 0; e < B; e++) {
            if (at[e] < 0) continue;
            uint16_t* o = cache + (at[e] >> 1);
            if (at[e] & 1) *reinterpret_cast<uint2*>(o) = v[e];
            else *o = (uint16_t)v[e].x;
        }
    }
}

// One residual block to compute: the TU, its frame, where its block goes.
struct ResTask {
    av1g_tu tu;
    int32_t frame;
    int32_t out;
};

// Ahead of the wavefront, what depends on the descriptors and coefficients
// only: the TU records (blocks [0, prep_blocks), a superblock per warp) and the
// residual blocks of every intra TU of the batch (the next small_blocks run
// the small TUs one per warp, the others the large TUs with the whole CTA).
__global__ void __launch_bounds__(kT) intra_pre_kernel(const IntraFrame* __restrict__ frames,
                                                       const SbItem* __restrict__ items, int nitems, TuRec* tus,
                                                       const ResTask* __restrict__ small, int n_small,
                                                       const ResTask* __restrict__ large, int n_large,
                                                       int32_t* __restrict__ res, int prep_blocks, int small_blocks) {
    __shared__ union {
        ResScr<kSmallPx> w[kNW];
        ResScr<64 * 64> c;
    } u;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if ((int)blockIdx.x < prep_blocks) {
        for (int q = blockIdx.x * kNW + warp; q < nitems; q += prep_blocks * kNW) {
            const SbItem it = items[q];
            const IntraFrame& F = frames[it.frame];
            for (int k = it.tu_first + lane; k < it.tu_end; k += 32) {
                const av1g_intra_tu t = *reinterpret_cast<const av1g_intra_tu*>(tus + k);
                TuRec r;
                prep_tu(F, it.log2sb, t, r);
                tus[k] = r;
            }
        }
    } else if ((int)blockIdx.x < prep_blocks + small_blocks) {
        for (int q = (blockIdx.x - prep_blocks) * kNW + warp; q < n_small; q += small_blocks * kNW) {
            const ResTask tk = small[q];
            const IntraFrame& F = frames[tk.frame];
            const WarpG g{lane};
            int32_t* out = res + tk.out;
            switch (tk.tu.tx_size) {
                case 0: residual_task<0>(g, u.w[warp], F, tk.tu, out); break;
                case 1: residual_task<1>(g, u.w[warp], F, tk.tu, out); break;
                case 2: residual_task<2>(g, u.w[warp], F, tk.tu, out); break;
                case 5: residual_task<5>(g, u.w[warp], F, tk.tu, out); break;
                case 6: residual_task<6>(g, u.w[warp], F, tk.tu, out); break;
                case 7: residual_task<7>(g, u.w[warp], F, tk.tu, out); break;
                case 8: residual_task<8>(g, u.w[warp], F, tk.tu, out); break;
                case 13: residual_task<13>(g, u.w[warp], F, tk.tu, out); break;
                case 14: residual_task<14>(g, u.w[warp], F, tk.tu, out); break;
                case 15: residual_task<15>(g, u.w[warp], F, tk.tu, out); break;
                default: residual_task<16>(g, u.w[warp], F, tk.tu, out); break;
            }
        }
    } else {
        const int first = prep_blocks + small_blocks;
        for (int q = blockIdx.x - first; q < n_large; q += gridDim.x - first) {
            const ResTask tk = large[q];
            const IntraFrame& F = frames[tk.frame];
            const CtaG g{tid};
            int32_t* out = res + tk.out;
            switch (tk.tu.tx_size) {
                case 3: residual_task<3>(g, u.c, F, tk.tu, out); break;
                case 4: residual_task<4>(g, u.c, F, tk.tu, out); break;
                case 9: residual_task<9>(g, u.c, F, tk.tu, out); break;
                case 10: residual_task<10>(g, u.c, F, tk.tu, out); break;
                case 11: residual_task<11>(g, u.c, F, tk.tu, out); break;
                case 12: residual_task<12>(g, u.c, F, tk.tu, out); break;
                case 17: residual_task<17>(g, u.c, F, tk.tu, out); break;
                default: residual_task<18>(g, u.c, F, tk.tu, out); break;
            }
        }
    }
}

// The waits of a superblock, by one warp: polls the progress words its next
// waits name, and after each that is over reloads the copy's border and lets
// the workers on up to the level of the first wait that is not.  A wait that
// runs out of time sets the frame's abort word; from then on the frame's
// superblocks no longer wait (their samples are incomplete, and the host
// reports the frame).
__device__ void wait_warp(Shared& S, uint16_t* cache, const int4* __restrict__ waits, const SbItem& it, int* prog,
                          int* abort_word, int lane) {
    long long t0 = gtimer();
    const long long bound = *(volatile long long*)&g_wait_ns;
    int wq = 0;
    while (wq < it.nwait) {
        const int q = wq + lane;
        bool over = false;
        if (q < it.nwait) {
            const int4 w = __ldg(waits + it.wait_first + q);
            over = *(volatile int*)(prog + w.y) >= w.z;
            if (over) ld_acquire(prog + w.y);
        }
        // the waits are in level order: only the ones before the first open one count
        const unsigned open = __ballot_sync(0xffffffffu, !over);
        const int n = open ? __ffs(open) - 1 : 32;
        if (n > 0) {
            wq += n;
            __syncwarp();
            load_border(S.fr, S.sb, cache, lane, 32);
            __syncwarp();
            __threadfence_block();
            if (lane == 0) *(volatile int*)&S.ready = wq < it.nwait ? __ldg(waits + it.wait_first + wq).x : kNoWait;
            t0 = gtimer();
            continue;
        }
        int stop = 0;
        if (lane == 0) {
            stop = *(volatile int*)abort_word;
            if (!stop && gtimer() - t0 > bound) {
                atomicExch(abort_word, 1);
                stop = 1;
            }
        }
        if (__shfl_sync(0xffffffffu, stop, 0)) {
            if (lane == 0) *(volatile int*)&S.ready = kNoWait;
            return;
        }
        __nanosleep(20);
    }
}

// One persistent launch.  A CTA claims superblocks in claim order.  Its worker
// warps run a superblock's levels, in three groups of four warps that take the
// levels in turn: a group decodes its TUs (fast_decode) while the other two
// run the levels before its own, and only the group of the next level waits for
// the end of a level.  Another warp publishes finished levels (its fence waits for
// their samples to reach L2 without holding up the next level), and another waits
// for other superblocks' levels and brings the border samples in ahead of the
// level that reads them.
__global__ void __launch_bounds__(kIT, 1) intra_kernel(const IntraFrame* __restrict__ frames,
                                                       const TuRec* __restrict__ tus,
                                                       const SbItem* __restrict__ items, const int2* __restrict__ lvs,
                                                       const int4* __restrict__ waits, int* prog, int* ctl, int nitems,
                                                       const int32_t* __restrict__ res) {
    // ctl[0]: the claim counter; ctl[1 + f]: frame f's abort word
    // dynamic shared memory: Shared | TU records | superblock copy
    extern __shared__ __align__(16) uint8_t dsm[];
    Shared& S = *reinterpret_cast<Shared*>(dsm);
    TuRec* win = reinterpret_cast<TuRec*>(dsm + kSharedBytes);
    uint16_t* cache = reinterpret_cast<uint16_t*>(dsm + kSharedBytes + kTuStage * sizeof(TuRec));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const IntraFrame& F = S.fr;
    // the tables that lanes index by different entries: shared, not constant, memory
    for (int q = tid; q < 5 * 8 * 8; q += kIT) {
        const int m = q >> 6, o = (q >> 3) & 7, i = q & 7;
        S.tb.fi[m][o][i] = i < 7 ? (int8_t)c_fi_taps[m][o][i] : (int8_t)0;
    }
    if (tid < 124)
        S.tb.sm[tid] = tid < 4 ? c_sm4[tid] : tid < 12 ? c_sm8[tid - 4] : tid < 28 ? c_sm16[tid - 12]
                     : tid < 60 ? c_sm32[tid - 28] : c_sm64[tid - 60];
    for (;;) {
        __syncthreads();
        if (tid == 0) S.idx = atomicAdd(&ctl[0], 1);
        __syncthreads();
        const int idx = S.idx;
        if (idx >= nitems) return;
        const SbItem it = items[idx];
        {
            const uint32_t* src = reinterpret_cast<const uint32_t*>(frames + it.frame);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&S.fr);
            for (int q = tid; q < (int)(sizeof(IntraFrame) / 4); q += kIT) dst[q] = __ldg(src + q);
        }
        __syncthreads();
        if (tid < 3) {
            const int p = tid, ssx = p ? F.ssx : 0, ssy = p ? F.ssy : 0;
            S.sb.rect[p] = make_int4(it.x0 >> ssx, it.y0 >> ssy, (1 << it.log2sb) >> ssx, (1 << it.log2sb) >> ssy);
            S.sb.cs[p] = copy_pitch(it.log2sb, ssx);
            S.sb.off[p] = copy_off(it.log2sb, F.ssx, F.ssy, p);
        }
        if (tid == 3) {
            S.done = 0;
            S.stuck = 0;
            S.ready = it.nwait > 0 ? __ldg(waits + it.wait_first).x : kNoWait;
        }
        __syncthreads();
        // the superblock's own area is written only by its own TUs, and its
        // TU records are inputs: stage both before any wait
        load_area(F, S.sb, cache);
        load_border(F, S.sb, cache, tid, kIT);
        {
            const uint4* src = reinterpret_cast<const uint4*>(tus + it.tu_first);
            uint4* dst = reinterpret_cast<uint4*>(win);
            const int n = min(it.tu_end - it.tu_first, kTuStage) * 4;
            for (int q = tid; q < n; q += kIT) dst[q] = __ldg(src + q);
        }
        for (int q = tid; q <= it.nlv && q < kLvStage; q += kIT) S.lv[q] = __ldg(lvs + it.lv_first + q);
        __syncthreads();
        if (warp == kWW) {
            if (lane == 0)
                for (int last = 0, spins = 0; last < it.nlv;) {
                    int done = *(volatile int*)&S.done;
                    if (done == last) {
                        __nanosleep(20);
                        if (spins++ < kSpins) continue;
                        S.stuck = 1;
                        done = it.nlv;
                    }
                    if (*(volatile int*)&S.stuck) atomicExch(ctl + 1 + it.frame, 1);
                    __threadfence();
                    atomicExch(prog + idx, done);
                    last = done;
                    spins = 0;
                }
            continue;
        }
        if (warp == kWW + 1) {
            wait_warp(S, cache, waits, it, prog, ctl + 1 + it.frame, lane);
            continue;
        }
        const int grp = warp / kGW, wi = warp % kGW;
        auto level = [&](int q) { return q < kLvStage ? S.lv[q] : __ldg(lvs + it.lv_first + q); };
        auto record = [&](int k) { return k - it.tu_first < kTuStage ? win + (k - it.tu_first) : tus + k; };
        int ready = 0;
        int lg = grp;
        for (; lg <= it.nlv; lg += kGroups) {
            const int2 prev = lg > 0 ? level(lg - 1) : make_int2(0, 0);
            int b = 0, m = 0, e = 0;
            Prog d;
            bool fast = false;
            int4 big = make_int4(0, 0, 0, 0);  // the first large TU's residual
            if (lg < it.nlv) {
                const int2 cur = level(lg);
                b = cur.x;
                m = cur.y & ~kLevelPublished;
                e = level(lg + 1).x;
                if (m < e) big = first_res(record(m), res, tid - grp * kGT);
                if (b + wi < m) {
                    const TuRec* rec = record(b + wi);
                    fast = rec->h.where & W_FAST;
                    if (fast) fast_decode(d, rec, F, S.sb, res, lane);
                }
            }
            if (lg > 0) {
                bar_sync(1 + (lg - 1) % kGroups, 2 * kGT);
                // "lg levels done", when another superblock waits for it or
                // the superblock is finished
                if (wi == 0 && lane == 0 && ((prev.y & kLevelPublished) || lg == it.nlv)) {
                    __threadfence_block();
                    *(volatile int*)&S.done = lg;
                }
            }
            if (lg == it.nlv) break;
            if (ready <= lg) {
                int k = kSpins;
                while ((ready = *(volatile int*)&S.ready) <= lg && --k) {}
                if (!k) S.stuck = 1;
                __threadfence_block();
            }
            WScr& ws = S.s[grp].w[wi];
            for (int k = b + wi; k < m; k += kGW) {
                if (k > b + wi) {
                    const TuRec* rec = record(k);
                    fast = rec->h.where & W_FAST;
                    if (fast) fast_decode(d, rec, F, S.sb, res, lane);
                }
                if (fast) fast_run(d, ws, F, S.sb, cache, S.tb, lane);
                else run_tu(WarpG{lane}, ws, record(k), F, S.sb, cache, S.tb, res, first_res(record(k), res, lane));
                __syncwarp();
            }
            if (m < e) {
                const WorkG g{tid - grp * kGT, 4 + grp};
                for (int k = m; k < e; k++) {
                    if (k > b) g.sync();
                    if (k > m) big = first_res(record(k), res, g.r);
                    run_tu(g, S.s[grp].c, record(k), F, S.sb, cache, S.tb, res, big);
                }
            }
            bar_arrive(1 + lg % kGroups, 2 * kGT);
        }
    }
}

// Test hook state: a never-satisfied wait is planned into the first
// superblock of every job whose frame is this wide (0: none).
std::atomic<int> g_fault_width{0};

// Before its first level, the first superblock of job f waits for its own
// progress to reach a value it never reaches.
void plan_fault_wait(IntraPlan& plan, int f) {
    for (size_t i = 0; i < plan.items.size(); i++) {
        SbItem& it = plan.items[i];
        if (it.frame != f) continue;
        plan.waits.insert(plan.waits.begin() + it.wait_first, int4{0, (int)i, 0x3fffffff, 0});
        it.nwait++;
        for (size_t k = 0; k < plan.items.size(); k++)
            if (k != i && plan.items[k].wait_first >= it.wait_first) plan.items[k].wait_first++;
        return;
    }
}

// The most dynamic shared memory any launch asks for: the fixed part, the TU
// window and the largest superblock copy (128x128, three full planes, u16).
constexpr size_t kMaxDynSmem =
    kSharedBytes + kTuStage * sizeof(TuRec) + 3 * intra_copy_samples(128, 128) * sizeof(uint16_t);
static_assert(kMaxDynSmem <= 227 * 1024, "intra_kernel's shared memory exceeds an SM's");

// The kernel's dynamic shared memory limit is a per-device attribute that
// every launch on the device shares, and engine lanes launch concurrently
// with different sizes: it is raised once per device to the largest size,
// so no launch can find it lowered by another thread between its own
// setting and its launch.
cudaError_t ensure_intra_smem_limit(int dev) {
    static std::mutex mu;
    static bool done[256];
    std::lock_guard<std::mutex> lk(mu);
    if (dev >= 0 && dev < 256 && done[dev]) return cudaSuccess;
    const cudaError_t e =
        cudaFuncSetAttribute(intra_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDynSmem);
    if (e == cudaSuccess && dev >= 0 && dev < 256) done[dev] = true;
    return e;
}
}  // namespace

// Host side of av1g_run_intra: the plan (intra_plan.cu), its upload, one
// launch.  frame_status (pinned host memory of n words, or null) receives,
// in stream order after the launch, each job's abort word: non-zero when a
// dependency wait of that frame ran out of time.
av1g_status intra_run_status(const av1g_intra_job* jobs, int n, cudaStream_t st, std::string& err,
                             int32_t* frame_status) {
    int dev = 0;
    cudaGetDevice(&dev);
    IntraPlan plan;
    av1g_status rc = intra_plan(jobs, n, plan, err);
    if (rc != AV1G_OK || plan.items.empty()) {
        if (rc == AV1G_OK && frame_status) memset(frame_status, 0, sizeof(int32_t) * n);
        return rc;
    }
    if (int fw = g_fault_width.load(); fw > 0)
        for (int i = 0; i < n; i++)
            if (jobs[i].hdr->frame_width == fw) plan_fault_wait(plan, i);
    const int nitems = (int)plan.items.size();
    // residual tasks, counted by part of the superblocks: each TU's device
    // record will point at its residual block
    const int parts = std::min(nitems, parallel_parts((long long)plan.ntus, 4096));
    struct Count {
        size_t small = 0, large = 0;
        long long ints = 0;
    };
    std::vector<Count> at(parts + 1);
    auto span = [&](int u, int& i0, int& i1) {
        i0 = (int)((long long)nitems * u / parts);
        i1 = (int)((long long)nitems * (u + 1) / parts);
    };
    // TU k of a superblock's range, in decode order (its records take the same range)
    auto source = [&](const SbItem& it, int k) -> const av1g_intra_tu& {
        return jobs[it.frame].tus[k - plan.tu_base[it.frame]];
    };
    parallel_for(parts, (long long)plan.ntus, [&](int u) {
        Count c;
        int i0, i1;
        span(u, i0, i1);
        for (int i = i0; i < i1; i++)
            for (int k = plan.items[i].tu_first; k < plan.items[i].tu_end; k++) {
                const av1g_intra_tu& t = source(plan.items[i], k);
                if (!(t.flags & AV1G_INTRA_RESIDUAL)) continue;
                const int px = kTxW[t.tx_size] * kTxH[t.tx_size];
                (px > kSmallPx ? c.large : c.small)++;
                c.ints += px;
            }
        at[u + 1] = c;
    });
    for (int u = 0; u < parts; u++) {
        at[u + 1].small += at[u].small;
        at[u + 1].large += at[u].large;
        at[u + 1].ints += at[u].ints;
    }
    const size_t n_rs = at[parts].small, n_rl = at[parts].large;
    const long long res_ints = at[parts].ints;
    if (res_ints >= (1LL << 31)) {
        err = "intra batch: more than 2^31 residual samples";
        return AV1G_EINVAL;
    }
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t off_tus = al(sizeof(IntraFrame) * n);
    const size_t off_items = al(off_tus + sizeof(av1g_intra_tu) * plan.ntus);
    const size_t off_lv = al(off_items + sizeof(SbItem) * plan.items.size());
    const size_t off_waits = al(off_lv + sizeof(int2) * plan.lvtab.size());
    const size_t off_done = al(off_waits + sizeof(int4) * plan.waits.size());
    const size_t off_ctl = al(off_done + sizeof(int) * plan.items.size());
    const size_t off_rs = al(off_ctl + (1 + (size_t)n) * sizeof(int));
    const size_t off_rl = al(off_rs + sizeof(ResTask) * n_rs);
    const size_t off_maps = al(off_rl + sizeof(ResTask) * n_rl);
    const size_t bytes = off_maps + plan.maps.size();  // uploaded
    const size_t off_res = al(bytes);
    const size_t total = off_res + sizeof(int32_t) * (size_t)res_ints;
    uint8_t* dev_buf = nullptr;
    cudaError_t e = workspace_alloc(&dev_buf, total, st);
    if (e != cudaSuccess) {
        err = std::string("cudaMallocAsync: ") + cudaGetErrorString(e);
        return AV1G_EDEVICE;
    }
    for (int i = 0; i < n; i++) plan.frames[i].maps = dev_buf + off_maps + plan.map_base[i];
    e = upload_with(dev_buf, bytes, st, [&](uint8_t* host) {
        memcpy(host, plan.frames.data(), sizeof(IntraFrame) * n);
        av1g_intra_tu* tus = reinterpret_cast<av1g_intra_tu*>(host + off_tus);
        ResTask* small = reinterpret_cast<ResTask*>(host + off_rs);
        ResTask* large = reinterpret_cast<ResTask*>(host + off_rl);
        parallel_for(parts, (long long)plan.ntus, [&](int u) {
            Count c = at[u];
            int i0, i1;
            span(u, i0, i1);
            for (int i = i0; i < i1; i++) {
                const SbItem& it = plan.items[i];
                for (int k = it.tu_first; k < it.tu_end; k++) {
                    const av1g_intra_tu& t = source(it, k);
                    av1g_intra_tu& r = tus[plan.order[k]];
                    r = t;
                    if (t.interintra) r.palette_map = plan.wedge[k];
                    if (!(t.flags & AV1G_INTRA_RESIDUAL)) continue;
                    const int px = kTxW[t.tx_size] * kTxH[t.tx_size];
                    (px > kSmallPx ? large[c.large++] : small[c.small++]) = ResTask{t.res, it.frame, (int32_t)c.ints};
                    r.res.coeff_offset = (uint32_t)c.ints;
                    c.ints += px;
                }
                if (parts > 1) write_back(tus + it.tu_first, sizeof(av1g_intra_tu) * (size_t)(it.tu_end - it.tu_first));
            }
            if (parts > 1) {
                write_back(small + at[u].small, sizeof(ResTask) * (c.small - at[u].small));
                write_back(large + at[u].large, sizeof(ResTask) * (c.large - at[u].large));
            }
        });
        memcpy(host + off_items, plan.items.data(), sizeof(SbItem) * plan.items.size());
        memcpy(host + off_lv, plan.lvtab.data(), sizeof(int2) * plan.lvtab.size());
        if (!plan.waits.empty()) memcpy(host + off_waits, plan.waits.data(), sizeof(int4) * plan.waits.size());
        memset(host + off_done, 0, off_rs - off_done);  // progress, claim counter, abort flag
        if (!plan.maps.empty()) memcpy(host + off_maps, plan.maps.data(), plan.maps.size());
    });
    const IntraFrame* dframes = (const IntraFrame*)dev_buf;
    int32_t* dres = (int32_t*)(dev_buf + off_res);
    int sms = 0;
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) {
        const int pb_blocks = (int)std::min<long long>(((long long)nitems + kNW - 1) / kNW, 8LL * sms);
        const int sb_blocks = (int)std::min<long long>(((long long)n_rs + kNW - 1) / kNW, 16LL * sms);
        const int lb_blocks = (int)std::min<long long>((long long)n_rl, 4LL * sms);
        intra_pre_kernel<<<pb_blocks + sb_blocks + lb_blocks, kT, 0, st>>>(
            dframes, (const SbItem*)(dev_buf + off_items), nitems, (TuRec*)(dev_buf + off_tus),
            (const ResTask*)(dev_buf + off_rs), (int)n_rs, (const ResTask*)(dev_buf + off_rl), (int)n_rl, dres,
            pb_blocks, sb_blocks);
        e = cudaGetLastError();
    }
    const size_t smem = kSharedBytes + kTuStage * sizeof(TuRec) + plan.cache_bytes;
    if (e == cudaSuccess && smem > kMaxDynSmem) e = cudaErrorInvalidValue;  // cannot happen: cache_bytes is bounded
    if (e == cudaSuccess) e = ensure_intra_smem_limit(dev);
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, intra_kernel, kIT, smem);
    if (e == cudaSuccess) {
        // as many CTAs as the wavefront can keep busy (the superblocks of
        // one depth, twice over since level-granular waits let the next depth
        // start early), not the whole GPU: idle CTAs would only poll while
        // other streams' kernels wait for SMs
        const int grid = std::max(1, std::min({nitems, std::max(per_sm, 1) * sms, 2 * plan.width + 2}));
        intra_kernel<<<grid, kIT, smem, st>>>(
            dframes, (const TuRec*)(dev_buf + off_tus), (const SbItem*)(dev_buf + off_items),
            (const int2*)(dev_buf + off_lv), (const int4*)(dev_buf + off_waits), (int*)(dev_buf + off_done),
            (int*)(dev_buf + off_ctl), nitems, dres);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess && frame_status)
        e = cudaMemcpyAsync(frame_status, dev_buf + off_ctl + sizeof(int), sizeof(int32_t) * n,
                            cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(dev_buf, st);
    if (e != cudaSuccess) {
        err = std::string("intra launch: ") + cudaGetErrorString(e);
        return AV1G_EDEVICE;
    }
    return AV1G_OK;
}

av1g_status intra_run(const av1g_intra_job* jobs, int n, cudaStream_t st, std::string& err) {
    return intra_run_status(jobs, n, st, err, nullptr);
}

}  // namespace av1g

extern "C" av1g_status av1g_intra_plan_stats_get(const av1g_intra_job* jobs, int32_t n,
                                                  av1g_intra_plan_stats* out) {
    if (!out || n < 0 || (n > 0 && !jobs)) return AV1G_EINVAL;
    av1g::IntraPlan plan;
    std::string err;
    av1g_status rc = av1g::intra_plan(jobs, n, plan, err);
    if (rc != AV1G_OK) return rc;
    *out = av1g_intra_plan_stats{(int32_t)plan.items.size(), (int32_t)plan.ntus, (int32_t)plan.waits.size(),
                                 plan.depth, plan.width, 0};
    return AV1G_OK;
}

extern "C" av1g_status av1g_test_intra_wait_fault(int64_t wait_ns, int32_t frame_width) {
    long long ns = wait_ns > 0 ? (long long)wait_ns : av1g::kWaitNs;
    cudaError_t e = cudaMemcpyToSymbol(av1g::g_wait_ns, &ns, sizeof ns);
    if (e != cudaSuccess) return AV1G_EDEVICE;
    av1g::g_fault_width.store(frame_width > 0 ? frame_width : 0);
    return AV1G_OK;
}
