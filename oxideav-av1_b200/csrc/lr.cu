// lr.cu — §7.17 loop restoration (Wiener and self-guided filters).
//
// Replaces loop_restoration_frame / loop_restore_block / wiener_filter /
// self_guided_filter / box_filter / get_source_sample
// (src/loop_restoration.rs:268-883) as driven by loop_restore_frame_from_grid
// (src/cdf.rs:20624).
//
// The reference filters 4x4 blocks (MI_SIZE walk), each recomputing its
// 7-tap Wiener rows and its (2r+1)^2 box sums over a halo.  Every quantity it
// computes is a function of the sample position, the restoration unit and the
// 64-row stripe only (stripe boundaries fall on 4x4 block boundaries and unit
// boundaries on stripe boundaries), so the kernel computes each quantity once
// per position.  One CTA owns (plane, stripe, 32-row half of the stripe,
// column tile) where the column tile, min(unit size, 64) wide, lies inside a
// single restoration unit.  The CTA stages the source window with a 3-sample
// halo in shared memory — rows inside the stripe from the CDEF frame, up to 2
// rows beyond it from the deblocked frame, clamped to the plane, exactly
// get_source_sample — then:
//  * Wiener: 7-tap horizontal pass into an intermediate array, 7-tap vertical
//    pass to the output (loop_restoration.rs:742-857);
//  * self-guided: per radius, separable box sums (column sums of the samples
//    and their squares, then row sums), the a/b coefficients with the
//    1/(z+1) term from a 256-entry table, the 3x3 weighting, and the
//    projection (loop_restoration.rs:485-736).  For the r0 pass the
//    reference's weights are zero on even rows of the A/B grid, so those rows
//    are not computed.
// Units of type RESTORE_NONE copy the CDEF samples through.
//
// Bound by instruction issue: 64 x 1080p 8-bit take 1.29 ms at 127 thread instructions
// per sample, with one thread working out the next tile, the scales in a table, a and b
// in one word and the 3x3 weighting of a pair of rows from one reading of them (three
// loads per output, not nine), against 1.67 ms at 198 without any of these.  Four CTAs
// per SM: five leave 48 registers and are slower.
#include <cstddef>

#include "common.cuh"

namespace av1g {

namespace {

constexpr int TW = 64, TH = 32, H3 = 3;
constexpr int kLrThreads = 256;  // lr_kernel's CTA size
constexpr int SW = TW + 2 * H3, SP = SW + 2;  // source window row pitch (u16)
constexpr int SH = TH + 2 * H3;
constexpr int VW = TW + 2 * H3 + 1;           // column-sum row pitch (odd: rows fall on distinct banks)
constexpr int AR = TH + 2, AP = TW + 2 + 1;   // A/B grid rows / pitch

constexpr int8_t kSgrParams[16][4] = {
    {2, 12, 1, 4}, {2, 15, 1, 6}, {2, 18, 1, 8}, {2, 21, 1, 9}, {2, 24, 1, 10}, {2, 29, 1, 11},
    {2, 36, 1, 12}, {2, 45, 1, 13}, {2, 56, 1, 14}, {2, 68, 1, 15}, {0, 0, 1, 5}, {0, 0, 1, 8},
    {0, 0, 1, 11}, {0, 0, 1, 14}, {2, 30, 0, 0}, {2, 75, 0, 0}};

// box_filter's scale of one pass of a self-guided set: the radius, the rounded
// 2^20 / (n^2 eps), n the box's samples, and the p from which
// z = (p * scale + 2^19) >> 20 reaches 255 (a2 = 256): clamping p to it keeps every
// product below 2^32 (zsat + scale) and leaves a2 unchanged, so z is computed in
// 32 bits.
struct SgrPass {
    uint32_t r, scale, pcap;
};
struct SgrSets {
    SgrPass pass[16][2];
};
constexpr SgrSets make_sgr() {
    SgrSets t{};
    for (int s = 0; s < 16; s++)
        for (int k = 0; k < 2; k++) {
            const int r = kSgrParams[s][2 * k], eps = kSgrParams[s][2 * k + 1];
            if (r == 0) continue;
            const long long n = (2 * r + 1) * (2 * r + 1), n2e = n * n * eps;
            const uint32_t scale = (uint32_t)(((1LL << 20) + n2e / 2) / n2e), zsat = (255u << 20) - (1u << 19);
            t.pass[s][k] = SgrPass{(uint32_t)r, scale, (zsat + scale - 1) / scale};
        }
    return t;
}
__constant__ SgrSets c_sgr = make_sgr();

// A tile: what every thread of its CTA needs, worked out once.  Deriving it
// takes a few dozen divisions, as many instructions as 40 of the thread's
// outputs when each of the 256 threads did it for its own 8.
struct Tile {
    int frame, plane, x0, y0, tw, th, sstart, send, pw, ph;
    av1g_lr_unit u;
    int packed;  // a and b share a word: not at 12 bits, nor with samples of more than ten
};

struct Smem {
    uint16_t src[SH * SP];
    int v1[AR * VW];      // column sums; the Wiener intermediate reuses v1/v2
    int v2[AR * VW];
    uint32_t AB[AR * AP];  // packed: b << kABits | a; else b alone
    uint16_t A[AR * AP];   // not packed: a
    uint16_t a2lut[256];
    Tile tile[2];  // the current one, and the next one while it is worked out
};
// The Wiener intermediate ((TH + 6) x TW ints) spans the adjacent v1 and v2 arrays.
static_assert((TH + 6) * TW <= 2 * AR * VW, "Wiener intermediate does not fit");
static_assert(offsetof(Smem, v2) == offsetof(Smem, v1) + sizeof(int) * AR * VW, "v1/v2 must be adjacent");

__device__ __forceinline__ int r2u(int x, int n) { return n ? (x + (1 << (n - 1))) >> n : x; }

__device__ __forceinline__ int tile_w(const av1g_frame_header& h, int p) {
    int us = h.lr_unit_size[p] > 0 ? h.lr_unit_size[p] : 1;
    return us < TW ? us : TW;
}

__device__ __forceinline__ int n_stripes(const av1g_frame_header& h, int p) {
    int ssy = p ? h.subsampling_y : 0;
    int ph = r2u(h.frame_height, ssy);
    return ((((ph - 1) << ssy) + 8) >> 6) + 1;
}

__device__ __forceinline__ int count_units(int us, int sz) {
    int n = (sz + (us >> 1)) / us;
    return n > 1 ? n : 1;
}

// At 8 and 10 bits the coefficients a (at most 256) and b (at most 261,120) share a
// word, and the sums of up to five of them that the 3x3 weighting needs do too
// (1,280 below 2^11, 1,305,600 below 2^21).  Not packed: 12 bits, and 10-bit tiles in
// whose window a sample has more than 10 bits.
constexpr int kABits = 11;
constexpr uint32_t kAMask = (1u << kABits) - 1;

// Box sums, a/b coefficients (box_filter, loop_restoration.rs:594-700) for
// radius R over the A/B grid rows i in [-1, th] (stored at i + 1), columns
// j in [-1, tw].  The self-guided sets use R = 2 only for the first pass,
// which needs only the rows whose plane row is odd; their column sums are
// stored compactly (grid row i + 1 at i + 1 >> 1).  Column sums slide down
// the rows and row sums slide along the columns, so each sum costs two loads
// instead of 2R + 1; the runs have fixed lengths so the loops unroll and the
// coefficient arithmetic of neighbouring positions overlaps.
template <int R, int BD, bool PACK>
__device__ void box_coeffs(Smem& s, int th, int tw, const SgrPass& ps, int y0) {
    constexpr bool ODD = R == 2;
    constexpr int n = (2 * R + 1) * (2 * R + 1);
    const unsigned sm = ps.scale, pcap = ps.pcap;
    constexpr int one_over_n = ((1 << 12) + n / 2) / n;
    constexpr int sa = 2 * (BD - 8), sb = BD - 8;
    const int vw = tw + 2 * H3;
    const int rows = th + 2;
    // column sums: one thread per (column, run of 12 grid rows): 3 x 71
    // items, one round of the 256 threads
    constexpr int RUN = 12;
    const int runs = (rows + RUN - 1) / RUN;
    for (int k = threadIdx.x; k < runs * VW; k += blockDim.x) {
        const int ru = k / VW, jj = k - ru * VW;
        if (jj >= vw) continue;
        const int ra = ru * RUN;
        const uint16_t* c = s.src + jj + (ra - 1 + H3 - R) * SP;  // first source row of grid row ra's window
        int s1 = 0, s2 = 0;
#pragma unroll
        for (int d = 0; d <= 2 * R; d++) {
            const int v = c[d * SP];
            s1 += v;
            s2 += v * v;
        }
#pragma unroll
        for (int t = 0; t < RUN; t++) {
            const int row = ra + t;
            if (row >= rows) break;
            if (!ODD || ((y0 + row - 1) & 1)) {
                const int cr = ODD ? row >> 1 : row;
                s.v1[cr * VW + jj] = s1;
                s.v2[cr * VW + jj] = s2;
            }
            const int vo = c[t * SP], vn = c[(t + 2 * R + 1) * SP];
            s1 += vn - vo;
            s2 += vn * vn - vo * vo;
        }
    }
    __syncthreads();
    // row sums and coefficients: one thread per (grid row, run of columns),
    // consecutive threads on consecutive rows of one run, so their column-sum
    // loads are an odd pitch apart (distinct banks); with ODD the work list
    // holds only the odd-plane-row grid rows, so no lane of a warp idles on a
    // skipped row.  Runs of 11 columns (34 rows x 6) or, odd rows only, 5
    // columns (17 rows x 14): one round of the 256 threads either way.
    constexpr int CRUN = ODD ? 5 : 11;
    constexpr int SEGS = (TW + 2 + CRUN - 1) / CRUN;
    const int first = ODD ? ((y0 & 1) ? 1 : 0) : 0;  // grid row r holds plane row y0 + r - 1
    constexpr int STEP = ODD ? 2 : 1;
    const int nrows = (rows - first + STEP - 1) / STEP;
    for (int k = threadIdx.x; k < nrows * SEGS; k += blockDim.x) {
        const int sg = k / nrows, rk = k - sg * nrows;
        const int row = first + rk * STEP;
        const int ja = sg * CRUN - 1, jb = min(tw + 1, ja + CRUN);  // j in [ja, jb)
        if (ja >= jb) continue;
        const int cr = ODD ? rk : row;  // rk == row >> 1 for the odd-only rows
        const int* c1 = s.v1 + cr * VW + ja + H3 - R;
        const int* c2 = s.v2 + cr * VW + ja + H3 - R;
        int b = 0, a = 0;
#pragma unroll
        for (int d = 0; d <= 2 * R; d++) {
            b += c1[d];
            a += c2[d];
        }
        uint16_t* ao = s.A + row * AP + ja + 1;
        uint32_t* bo = s.AB + row * AP + ja + 1;
#pragma unroll
        for (int t = 0; t < CRUN; t++) {
            if (ja + t >= jb) break;
            // 8-bit: both shifts are 0
            const int ar = BD > 8 ? (a + ((1 << sa) >> 1)) >> sa : a;
            const int dr = BD > 8 ? (b + ((1 << sb) >> 1)) >> sb : b;
            int p = ar * n - dr * dr;
            if (p < 0) p = 0;
            const unsigned z = (min((unsigned)p, pcap) * sm + (1u << 19)) >> 20;
            int a2 = z >= 255 ? 256 : s.a2lut[z];
            // b2 uses the raw box sum b, as the reference does
            // (loop_restoration.rs:660-661); (256 - a2) * b * one_over_n
            // stays below 2^32 at every bit depth (b <= 25 * 4095)
            const unsigned b2 = (unsigned)(256 - a2) * (unsigned)b * (unsigned)one_over_n;
            const uint32_t bq = (b2 + (1u << 11)) >> 12;
            if (!PACK) ao[t] = (uint16_t)a2;
            bo[t] = PACK ? (bq << kABits | (uint32_t)a2) : bq;
            b += c1[t + 2 * R + 1] - c1[t];
            a += c2[t + 2 * R + 1] - c2[t];
        }
    }
    __syncthreads();
}

// 3x3 weighting of A/B (loop_restoration.rs:700-736) for the outputs (i, j0 .. j0 + 3)
// and (i + 1, j0 .. j0 + 3), i even, reading each A/B entry once.  y0 is even (stripes
// and their halves start on even rows), so i + 1 is an odd plane row.  Weights: first pass,
// even rows 5 6 5 above and below, odd rows 5 6 5 in their own row; second pass 4 in the
// cross, 3 in the corners.
__device__ __forceinline__ int weigh(int wk, uint32_t k, int wc, uint32_t c, int u, int sh) {
    const int as = wk * (int)(k & kAMask) + wc * (int)(c & kAMask);
    const int bs = wk * (int)(k >> kABits) + wc * (int)(c >> kABits);
    return (as * u + bs + (1 << (sh - 1))) >> sh;
}
template <int PASS>
__device__ __forceinline__ void weight_pair(const Smem& s, int i, int j0, const int (&u)[2][4], int (&out)[2][4]) {
    const uint32_t* g = s.AB + i * AP + j0;  // top-left of the first 3x3 window
    uint32_t top[6], mid[6], low[6];
    if (PASS == 0) {
#pragma unroll
        for (int c = 0; c < 6; c++) {
            low[c] = g[2 * AP + c];
            top[c] = g[c] + low[c];
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            out[0][e] = weigh(5, top[e] + top[e + 2], 6, top[e + 1], u[0][e], 9);
            out[1][e] = weigh(5, low[e] + low[e + 2], 6, low[e + 1], u[1][e], 8);
        }
    } else {
#pragma unroll
        for (int c = 0; c < 6; c++) {
            const uint32_t r1 = g[AP + c], r2 = g[2 * AP + c];
            top[c] = g[c] + r2;         // rows above and below the first output
            mid[c] = r1;
            low[c] = r2;
        }
#pragma unroll
        for (int e = 0; e < 4; e++)
            out[0][e] = weigh(3, top[e] + top[e + 2], 4, top[e + 1] + mid[e] + mid[e + 1] + mid[e + 2], u[0][e], 9);
#pragma unroll
        for (int c = 0; c < 6; c++) top[c] = mid[c] + g[3 * AP + c];
#pragma unroll
        for (int e = 0; e < 4; e++)
            out[1][e] = weigh(3, top[e] + top[e + 2], 4, top[e + 1] + low[e] + low[e + 1] + low[e + 2], u[1][e], 9);
    }
}

// The same from the two arrays, one row at a time.
template <int PASS>
__device__ __noinline__ int4 weight_row(const Smem& s, int i, int j0, int4 uq) {
    const uint16_t* a = s.A + i * AP + j0;
    const uint32_t* b = s.AB + i * AP + j0;
    const bool odd = i & 1;
    // weights of the three rows' side and middle columns
    const int ws[3] = {PASS ? 3 : (odd ? 0 : 5), PASS ? 4 : (odd ? 5 : 0), PASS ? 3 : (odd ? 0 : 5)};
    const int wm[3] = {PASS ? 4 : (odd ? 0 : 6), PASS ? 4 : (odd ? 6 : 0), PASS ? 4 : (odd ? 0 : 6)};
    const int sh = PASS || !odd ? 9 : 8;
    const int u[4] = {uq.x, uq.y, uq.z, uq.w};
    int out[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        int as = 0, bs = 0;
        for (int r = 0; r < 3; r++) {
            if (!wm[r]) continue;  // the first pass has no other rows' entries
            const int o = r * AP + e;
            as += ws[r] * (a[o] + a[o + 2]) + wm[r] * a[o + 1];
            bs += ws[r] * (int)(b[o] + b[o + 2]) + wm[r] * (int)b[o + 1];
        }
        out[e] = (as * u[e] + bs + (1 << (sh - 1))) >> sh;
    }
    return make_int4(out[0], out[1], out[2], out[3]);
}
template <int PASS>
__device__ __forceinline__ void weight_pair(const Smem& s, bool packed, int i, int j0, const int (&u)[2][4], int (&out)[2][4]) {
    if (!packed) {
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int4 v = weight_row<PASS>(s, i + e, j0, make_int4(u[e][0], u[e][1], u[e][2], u[e][3]));
            out[e][0] = v.x, out[e][1] = v.y, out[e][2] = v.z, out[e][3] = v.w;
        }
    } else {
        weight_pair<PASS>(s, i, j0, u, out);
    }
}
template <int R>
__device__ __forceinline__ void box_coeffs(Smem& s, int th, int tw, int bd, bool packed, const SgrPass& ps, int y0) {
    if (bd == 8) box_coeffs<R, 8, true>(s, th, tw, ps, y0);
    else if (bd == 12) box_coeffs<R, 12, false>(s, th, tw, ps, y0);
    else if (packed) box_coeffs<R, 10, true>(s, th, tw, ps, y0);
    else box_coeffs<R, 10, false>(s, th, tw, ps, y0);
}

// Tile t of the batch: its frame, plane, stripe half, column tile and
// restoration unit (derive_block_geometry, loop_restoration.rs:370-428).
__device__ void plan_tile(Tile& T, const FrameDev* __restrict__ frames, const int32_t* __restrict__ starts, int n,
                          int t) {
    const int f = find_frame(starts, n, t);
    const FrameDev& F = frames[f];
    const av1g_frame_header& h = F.h;
    int local = t - starts[f];
    int plane = 0, stripe = 0, half = 0, ct = 0;
    for (int p = 0; p < h.num_planes; p++) {
        if (h.lr_type[p] == 0) continue;
        const int pw = r2u(h.upscaled_width, p ? h.subsampling_x : 0);
        const int nct = (pw + tile_w(h, p) - 1) / tile_w(h, p);
        const int halves = 2 >> (p ? h.subsampling_y : 0);
        const int cnt = nct * halves * n_stripes(h, p);
        if (local < cnt) {
            plane = p;
            ct = local % nct;
            half = (local / nct) % halves;
            stripe = local / (nct * halves);
            break;
        }
        local -= cnt;
    }
    const int ssx = plane ? h.subsampling_x : 0, ssy = plane ? h.subsampling_y : 0;
    const int pw = r2u(h.upscaled_width, ssx), ph = r2u(h.frame_height, ssy);
    const int tw = tile_w(h, plane), x0 = ct * tw;
    const int sstart = (-8 + stripe * 64) >> ssy, send = sstart + (64 >> ssy) - 1;
    const int y0 = max(0, sstart + half * TH), y1 = min(min(ph, send + 1), sstart + half * TH + TH);
    const int us = h.lr_unit_size[plane] > 0 ? h.lr_unit_size[plane] : 1;
    const int ur = min(count_units(us, ph) - 1, (((max(0, sstart) << ssy) + 8) >> ssy) / us);
    const int uc = min(count_units(us, pw) - 1, x0 / us);
    av1g_lr_unit u{};
    if (F.lr_units[plane] && ur < F.lr_unit_rows[plane] && uc < F.lr_unit_cols[plane])
        u = F.lr_units[plane][ur * F.lr_unit_cols[plane] + uc];
    T = Tile{f, plane, x0, y0, min(x0 + tw, pw) - x0, y1 - y0, sstart, send, pw, ph, u, h.bit_depth != 12};
}

__global__ void __launch_bounds__(kLrThreads, 4) lr_kernel(const FrameDev* __restrict__ frames,
                                                 const int32_t* __restrict__ starts, int n, int total) {
    chain_wait();
    chain_next();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& s = *reinterpret_cast<Smem*>(smem_raw);
    for (int z = threadIdx.x; z < 256; z += blockDim.x)
        s.a2lut[z] = (uint16_t)(z == 0 ? 1 : ((z << 8) + z / 2) / (z + 1));
    // the next tile is worked out by one thread while the CTA filters the
    // current one (the first by the same thread ahead of the loop)
    const bool planner = threadIdx.x == kLrThreads - 32;
    if (planner && (int)blockIdx.x < total) plan_tile(s.tile[0], frames, starts, n, blockIdx.x);
    int cur = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x, cur ^= 1) {
        __syncthreads();  // the tile is worked out; the previous one is done with shared memory
        if (planner && t + (int)gridDim.x < total) plan_tile(s.tile[cur ^ 1], frames, starts, n, t + gridDim.x);
        const Tile& T = s.tile[cur];
        const FrameDev& F = frames[T.frame];
        const int plane = T.plane, pw = T.pw, ph = T.ph, x0 = T.x0, y0 = T.y0, tw = T.tw, th = T.th;
        const int sstart = T.sstart, send = T.send;
        if (th <= 0) continue;  // uniform across the CTA
        const int hbd = F.hbd, bd = F.h.bit_depth;
        const PlaneDev& C = F.upcdef[plane];
        const PlaneDev& Dq = F.updeb[plane];
        const PlaneDev& O = F.lr[plane];
        const av1g_lr_unit& u = T.u;
        if (u.type != 1 && u.type != 2) {
            // RESTORE_NONE: copied through, four samples per thread (x0 is a
            // multiple of 32 and plane rows start on 16-byte boundaries, so
            // each group of four is one aligned load and store)
            for (int k = threadIdx.x; k < th * (TW / 4); k += blockDim.x) {
                const int i = k >> 4, j0 = (k & 15) * 4;
                if (j0 >= tw) continue;
                const int y = y0 + i, x = x0 + j0;
                if (j0 + 4 <= tw) {
                    const uint8_t* src = C.p + (size_t)y * C.stride;
                    uint8_t* dst = O.p + (size_t)y * O.stride;
                    if (hbd) *reinterpret_cast<uint2*>(dst + 2 * x) = *reinterpret_cast<const uint2*>(src + 2 * x);
                    else *reinterpret_cast<uint32_t*>(dst + x) = *reinterpret_cast<const uint32_t*>(src + x);
                } else {
                    for (int e = 0; e < 4 && j0 + e < tw; e++) st_px(O, hbd, y, x + e, ld_px(C, hbd, y, x + e));
                }
            }
            continue;
        }
        // source window: get_source_sample (loop_restoration.rs:862-883)
        const int sw = tw + 2 * H3;
        uint32_t seen = 0;  // high bit depths: the bits of the samples staged
        if (x0 >= 4 && x0 + tw + 4 <= pw && !(x0 & 3) && !(tw & 3)) {
            // columns [x0 - 4, x0 + tw + 4) lie inside the plane (and inside
            // both source planes, which are at least pw wide): aligned
            // 4-sample loads, the row routed once per load
            // every thread issues its (at most 3) loads before it unpacks
            // any, so their latencies overlap
            const int ng = (tw + 8) >> 2, items = (th + 2 * H3) * ng;
            // k / ng for k < 38 * ng
            const unsigned mag = ng == (TW + 8) / 4 ? (1u << 16) / ((TW + 8) / 4) + 1 : (1u << 16) / ng + 1;
            constexpr int PER = (SH * ((TW + 8) >> 2) + kLrThreads - 1) / kLrThreads;
            uint2 q[PER];
#pragma unroll
            for (int e = 0; e < PER; e++) {
                const int k = threadIdx.x + e * kLrThreads;
                if (k >= items) break;
                const int i = (int)(((unsigned)k * mag) >> 16), g = k - i * ng;
                const int y = clip3(0, ph - 1, y0 - H3 + i);
                const PlaneDev* P;
                int yy;
                if (y < sstart) {
                    P = &Dq;
                    yy = clip3(0, Dq.h - 1, max(y, sstart - 2));
                } else if (y > send) {
                    P = &Dq;
                    yy = clip3(0, Dq.h - 1, min(y, send + 2));
                } else {
                    P = &C;
                    yy = min(y, C.h - 1);
                }
                const uint8_t* row = P->p + (size_t)yy * P->stride;
                const int xs = x0 - 4 + 4 * g;
                if (hbd) q[e] = *reinterpret_cast<const uint2*>(row + 2 * xs);
                else q[e].x = *reinterpret_cast<const uint32_t*>(row + xs);
            }
#pragma unroll
            for (int e = 0; e < PER; e++) {
                const int k = threadIdx.x + e * kLrThreads;
                if (k >= items) break;
                const int i = (int)(((unsigned)k * mag) >> 16), g = k - i * ng;
                int v[4];
                if (hbd) {
                    seen |= q[e].x | q[e].y;
                    v[0] = q[e].x & 0xffff;
                    v[1] = q[e].x >> 16;
                    v[2] = q[e].y & 0xffff;
                    v[3] = q[e].y >> 16;
                } else {
                    v[0] = q[e].x & 0xff;
                    v[1] = (q[e].x >> 8) & 0xff;
                    v[2] = (q[e].x >> 16) & 0xff;
                    v[3] = q[e].x >> 24;
                }
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const int j = 4 * g + t - 1;
                    if (j >= 0 && j < sw) s.src[i * SP + j] = (uint16_t)v[t];
                }
            }
        } else {
            for (int k = threadIdx.x; k < (th + 2 * H3) * SW; k += blockDim.x) {
                int i = k / SW, j = k - i * SW;
                if (j >= sw) continue;
                int x = clip3(0, pw - 1, x0 - H3 + j), y = clip3(0, ph - 1, y0 - H3 + i);
                int v;
                if (y < sstart) v = ld_px(Dq, hbd, clip3(0, Dq.h - 1, max(y, sstart - 2)), min(x, Dq.w - 1));
                else if (y > send) v = ld_px(Dq, hbd, clip3(0, Dq.h - 1, min(y, send + 2)), min(x, Dq.w - 1));
                else v = ld_px(C, hbd, min(y, C.h - 1), min(x, C.w - 1));
                seen |= (uint32_t)v;
                s.src[i * SP + j] = (uint16_t)v;
            }
        }
        if (seen & 0xfc00fc00u) s.tile[cur].packed = 0;
        __syncthreads();
        const bool packed = bd == 8 || __builtin_expect(T.packed, 1);
        const int maxv = (1 << bd) - 1;
        if (u.type == 1) {
            int hf[7], vf[7];
            hf[3] = vf[3] = 128;
#pragma unroll
            for (int i = 0; i < 3; i++) {
                vf[i] = vf[6 - i] = u.wiener[0][i];
                vf[3] -= 2 * u.wiener[0][i];
                hf[i] = hf[6 - i] = u.wiener[1][i];
                hf[3] -= 2 * u.wiener[1][i];
            }
            const int rr0 = bd == 12 ? 5 : 3, rr1 = bd == 12 ? 9 : 11;
            const int off = 1 << (bd + 7 - rr0 - 1);
            const int lim = (1 << (bd + 1 + 7 - rr0)) - 1;
            // four adjacent outputs per thread in both passes: the source
            // samples and intermediate rows they share are loaded once, as
            // vectors (source and intermediate rows start on 16-byte
            // boundaries; columns past tw are computed and not stored)
            int* inter = s.v1;  // (th + 6) x TW
            constexpr int Q4 = TW / 4;
            for (int k = threadIdx.x; k < (th + 6) * Q4; k += blockDim.x) {
                const int i = k / Q4, j0 = (k - i * Q4) * 4;
                if (j0 >= tw) continue;
                const uint2* w2 = reinterpret_cast<const uint2*>(s.src + i * SP + j0);
                int w[12];
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    const uint2 v = w2[q];
                    w[4 * q] = v.x & 0xffff;
                    w[4 * q + 1] = v.x >> 16;
                    w[4 * q + 2] = v.y & 0xffff;
                    w[4 * q + 3] = v.y >> 16;
                }
                int o[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int acc = hf[3] * w[e + 3] + hf[0] * (w[e] + w[e + 6]) + hf[1] * (w[e + 1] + w[e + 5]) +
                                    hf[2] * (w[e + 2] + w[e + 4]);
                    o[e] = clip3(-off, lim - off, (acc + (1 << (rr0 - 1))) >> rr0);
                }
                *reinterpret_cast<int4*>(inter + i * TW + j0) = make_int4(o[0], o[1], o[2], o[3]);
            }
            __syncthreads();
            for (int k = threadIdx.x; k < th * Q4; k += blockDim.x) {
                const int i = k / Q4, j0 = (k - i * Q4) * 4;
                if (j0 >= tw) continue;
                int4 r[7];
#pragma unroll
                for (int d = 0; d < 7; d++) r[d] = *reinterpret_cast<const int4*>(inter + (i + d) * TW + j0);
                int o[4];
#define LR_VTAP(F) (vf[3] * r[3].F + vf[0] * (r[0].F + r[6].F) + vf[1] * (r[1].F + r[5].F) + vf[2] * (r[2].F + r[4].F))
                const int acc[4] = {LR_VTAP(x), LR_VTAP(y), LR_VTAP(z), LR_VTAP(w)};
#undef LR_VTAP
#pragma unroll
                for (int e = 0; e < 4; e++) o[e] = clip3(0, maxv, (acc[e] + (1 << (rr1 - 1))) >> rr1);
                if (j0 + 4 <= tw && !((x0 + j0) & 3)) {  // one aligned vector store
                    uint8_t* row = O.p + (size_t)(y0 + i) * O.stride;
                    if (hbd)
                        *reinterpret_cast<uint2*>(row + 2 * (x0 + j0)) =
                            make_uint2((uint32_t)o[0] | (uint32_t)o[1] << 16, (uint32_t)o[2] | (uint32_t)o[3] << 16);
                    else
                        *reinterpret_cast<uint32_t*>(row + x0 + j0) =
                            (uint32_t)o[0] | (uint32_t)o[1] << 8 | (uint32_t)o[2] << 16 | (uint32_t)o[3] << 24;
                } else {
                    for (int e = 0; e < 4 && j0 + e < tw; e++) st_px(O, hbd, y0 + i, x0 + j0 + e, o[e]);
                }
            }
            continue;
        }
        // self-guided (loop_restoration.rs:485-588)
        const int set = u.sgr_set < 16 ? u.sgr_set : 15;
        const SgrPass &p0 = c_sgr.pass[set][0], &p1 = c_sgr.pass[set][1];
        const int r0 = p0.r, r1 = p1.r;
        const int w0 = u.sgr_xqd[0], w1 = u.sgr_xqd[1], w2 = 128 - w0 - w1;
        // a thread's outputs: four along a row in a pair of rows, the same in both
        // passes, so that the first pass's outputs stay in registers and the rows of
        // the A/B grid that the two share are read once
        constexpr int Q = TW / 4;
        static_assert(TH / 2 * Q == kLrThreads, "one run of four in a pair of rows per thread");
        const int i0 = 2 * (threadIdx.x / Q), j0 = (threadIdx.x % Q) * 4;
        const bool mine = i0 < th && j0 < tw;
        int f0[2][4] = {}, uq[2][4];
        auto load_u = [&] {
#pragma unroll
            for (int e = 0; e < 2; e++)
#pragma unroll
                for (int q = 0; q < 4; q++) uq[e][q] = s.src[(i0 + e + H3) * SP + j0 + q + H3];
        };
        if (r0) {  // r0 is 2 in every set that has it
            box_coeffs<2>(s, th, tw, bd, packed, p0, y0);
            if (mine) {
                load_u();
                weight_pair<0>(s, packed, i0, j0, uq, f0);
            }
            __syncthreads();
        }
        if (r1) box_coeffs<1>(s, th, tw, bd, packed, p1, y0);  // r1 is 1 in every set that has it
        if (!mine) continue;
        int f1[2][4];
        load_u();
        if (r1) weight_pair<1>(s, packed, i0, j0, uq, f1);
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int i = i0 + e;
            if (i >= th) break;
            int o[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int uu = uq[e][q] << 4;
                const int v = w1 * uu + w0 * (r0 ? f0[e][q] : uu) + w2 * (r1 ? f1[e][q] : uu);
                o[q] = clip3(0, maxv, (v + (1 << 10)) >> 11);
            }
            if (j0 + 4 <= tw && !((x0 + j0) & 3)) {  // one aligned vector store
                uint8_t* row = O.p + (size_t)(y0 + i) * O.stride;
                if (hbd)
                    *reinterpret_cast<uint2*>(row + 2 * (x0 + j0)) =
                        make_uint2((uint32_t)o[0] | (uint32_t)o[1] << 16, (uint32_t)o[2] | (uint32_t)o[3] << 16);
                else
                    *reinterpret_cast<uint32_t*>(row + x0 + j0) =
                        (uint32_t)o[0] | (uint32_t)o[1] << 8 | (uint32_t)o[2] << 16 | (uint32_t)o[3] << 24;
            } else {
                for (int q = 0; q < 4 && j0 + q < tw; q++) st_px(O, hbd, y0 + i, x0 + j0 + q, o[q]);
            }
        }
    }
}

}  // namespace

size_t lr_smem_bytes() { return sizeof(Smem); }

int tiles_lr(const FrameDev& f) {
    const av1g_frame_header& h = f.h;
    int n = 0;
    for (int p = 0; p < h.num_planes; p++) {
        if (h.lr_type[p] == 0) continue;
        int ssx = p ? h.subsampling_x : 0, ssy = p ? h.subsampling_y : 0;
        int pw = ssx ? (h.upscaled_width + 1) >> 1 : h.upscaled_width;
        int ph = ssy ? (h.frame_height + 1) >> 1 : h.frame_height;
        int us = h.lr_unit_size[p] > 0 ? h.lr_unit_size[p] : 1;
        int tw = us < TW ? us : TW;
        int ns = ((((ph - 1) << ssy) + 8) >> 6) + 1;
        n += ((pw + tw - 1) / tw) * ns * (2 >> ssy);
    }
    return n;
}

void launch_lr(const FrameDev* frames, const int32_t* starts, int n, int total, const StageShape& sh,
               cudaStream_t s) {
    if (total <= 0) return;
    size_t bytes = lr_smem_bytes();
    cudaFuncSetAttribute(lr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    launch_chained(lr_kernel, shape_grid(sh, total), kLrThreads, bytes, s, frames, starts, n, total);
}

}  // namespace av1g
