// filmgrain.cu — §7.18.3 film grain synthesis.
//
// Replaces film_grain_synthesis / generate_grain / scaling_lookup_init /
// add_noise_synthesis (src/film_grain.rs:100-873) as called at
// frame_driver.rs:1060-1096.
//
// Two kernels:
//  * grain_template_kernel — one CTA per frame builds the 82x73 luma and the
//    chroma grain templates, the three scaling LUTs and the per-stripe random
//    block offsets into a per-frame scratch area.  The reference draws the
//    white noise from one 16-bit LFSR in raster order; the LFSR is linear over
//    GF(2), so the state at the start of row y is M^(W*y) applied to the seed
//    and every row is generated by its own thread after a jump of at most
//    seven precomputed matrix-vector products.  The auto-regressive filter
//    (lag <= 3) reads only earlier rows and earlier samples of the same row,
//    so samples with equal x + 4y are independent and one warp sweeps the
//    template in ~370 wavefront steps, the two chroma templates' warps a little
//    behind the luma one's.  The chain of those steps bounds the kernel: 56 us
//    for any batch of frames (190 us for twelve 4:4:4 frames, 171 us for four
//    4:2:0 ones with all taps read from shared memory and chroma after luma).
//  * grain_blend_kernel — a tile is a noise stripe (32 luma rows) by 256 luma
//    columns; a warp takes a chroma-resolution row of it at a time, a lane eight
//    luma columns.  Those lie in one noise block, so a lane reads its random
//    offsets once per tile.  The noise value of a sample is evaluated in closed
//    form from the template, the offsets of the (at most two) blocks that wrote
//    it in each direction and the 27/17, 17/27 and 23/22 overlap blends, which is
//    exactly what the reference's materialised noise stripes and noise image hold
//    (film_grain.rs:599-760).  Chroma is blended first from the un-noised
//    luma, then luma, as the reference orders it (film_grain.rs:758-828).
//    A CTA lays the frame's templates out in shared memory, with a scaling table
//    of one entry per sample value, and asks for all of a row's samples at once.
//    Bound by issue and the latency of the samples' loads: 89 us for four 3840x2160
//    10-bit 4:2:0 frames and 67 us for twelve 718p 4:4:4 ones (2.2 TB/s and 2.3 TB/s of
//    planes read and written), against 193 and 170 us when a thread took four columns,
//    interpolated each scaling value and reread the frame's parameters after every store.
#include "common.cuh"
#include "av1_spec_tables.h"

namespace av1g {

__device__ const AV1T_GAUSSIAN_SEQUENCE_TYPE g_gauss AV1T_GAUSSIAN_SEQUENCE_DIMS = AV1T_GAUSSIAN_SEQUENCE_INIT;

namespace {

constexpr int LW = 82, LH = 73;
constexpr int kSpins = 1 << 22;  // readings of a progress word by one wait, some 30 cycles each

// ---- LFSR jump tables: M^(w * 2^b) for row widths 82 and 44 ---------------
struct Jumps {
    uint16_t m[2][7][16];  // [width 82 / 44][bit][column]
};

constexpr uint16_t mat_apply(const uint16_t* cols, uint16_t v) {
    uint16_t r = 0;
    for (int k = 0; k < 16; k++)
        if ((v >> k) & 1) r ^= cols[k];
    return r;
}

constexpr uint16_t lfsr_step(uint16_t r) {
    unsigned bit = (r ^ (r >> 1) ^ (r >> 3) ^ (r >> 12)) & 1;
    return (uint16_t)((r >> 1) | (bit << 15));
}

constexpr Jumps make_jumps() {
    Jumps j{};
    const int widths[2] = {LW, 44};
    for (int wi = 0; wi < 2; wi++) {
        // M^w by stepping each basis vector w times
        for (int k = 0; k < 16; k++) {
            uint16_t v = (uint16_t)(1u << k);
            for (int s = 0; s < widths[wi]; s++) v = lfsr_step(v);
            j.m[wi][0][k] = v;
        }
        for (int b = 1; b < 7; b++)
            for (int k = 0; k < 16; k++)
                j.m[wi][b][k] = mat_apply(j.m[wi][b - 1], j.m[wi][b - 1][k]);
    }
    return j;
}

__constant__ Jumps c_jumps = make_jumps();

__device__ __forceinline__ uint16_t row_state(uint16_t seed, int row, int wi) {
    uint16_t s = seed;
    for (int b = 0; b < 7; b++)
        if ((row >> b) & 1) s = mat_apply(c_jumps.m[wi][b], s);
    return s;
}

__device__ __forceinline__ int r2(int x, int n) { return n ? (x + (1 << (n - 1))) >> n : x; }

// scaling_lookup_fill (film_grain.rs:490-540) at one value: the first point's
// scaling below it, the last one's from it on, and between two points the
// interpolation of the last segment (of positive length) that holds the value
__device__ int scaling_at(int v, int np, const uint8_t* xv, const uint8_t* yv) {
    if (np == 0) return 0;
    if (v >= xv[np - 1]) return yv[np - 1];
    int r = v < xv[0] ? yv[0] : 0;
    for (int i = 0; i + 1 < np; i++) {
        const int dx = xv[i + 1] - xv[i], x = v - xv[i];
        if (dx <= 0 || x < 0 || x >= dx) continue;
        const int delta = (yv[i + 1] - yv[i]) * ((65536 + (dx >> 1)) / dx);
        r = clip3(0, 255, yv[i] + ((x * delta + 32768) >> 16));
    }
    return r;
}

// AR filter of a w x h template by one warp, in place: a wavefront over
// T = x + 4y in which lane y % 32 walks row y (a row takes w <= 82 steps and
// starts four steps after the row above, so a lane is done with row y before
// row y + 32 starts).  A sample's neighbours stay in registers: the three
// samples to its left, and for each of the LAG rows above a window of 2 LAG + 1
// samples that takes in one more per step, shuffled from the lane of the row
// above: its last output is row y - 1 at x + 3, and its own windows hold row
// y - 2 and y - 3 there.  So a step's chain is a shuffle and a row's
// multiplications, 240 cycles at lag 3; reading all taps from shared memory at
// each step took 600.  The filter leaves the first three rows and
// the outer three columns as they are; they pass through the same chain unchanged.
//
// The chroma warps follow the luma warp through `prog`, the luma steps whose
// samples are in shared memory: chroma step T weighs luma samples of at most
// luma step 2 T with 4:2:0, T + w with 4:2:2 and T with 4:4:4.
// SS: -1 the luma template, else a chroma template, subsampled in SS directions.
template <int LAG, int SS>
__device__ void ar_filter(int16_t* C, const int16_t* L, const uint8_t* coef, const av1g_film_grain& fg, int gmin,
                          int gmax, volatile int* prog) {
    constexpr bool CHROMA = SS >= 0;
    constexpr int ssx = SS >= 1, ssy = SS == 2;
    constexpr int w = ssx ? 44 : LW, h = ssy ? 38 : LH;
    constexpr int NC = 2 * LAG * (LAG + 1);  // of chroma, coefficient NC weighs the co-located luma
    constexpr int WN = 2 * LAG + 1, R = LAG > 0 ? LAG : 1, D = LAG > 0 ? 3 - LAG : 0;
    int c[NC + 1];
#pragma unroll
    for (int i = 0; i < NC; i++) c[i] = coef[i] - 128;
    c[NC] = CHROMA ? coef[NC] - 128 : 0;
    const bool luma = CHROMA && fg.num_y_points > 0;
    const int shift = fg.ar_coeff_shift, half = shift ? 1 << (shift - 1) : 0, lane = threadIdx.x & 31;
    int win[R][WN];  // win[r][k]: row y - 1 - r at x - LAG + k
    int left[R];     // left[k]: this row at x - 1 - k
    // The newest sample of each window comes from the lane above, whose last
    // step was x + 3 of row y - 1: its output there, and the middle of its windows
    // (rows y - 2 and y - 3 there).  LAG < 3 windows end at x + LAG and take that
    // sample D = 3 - LAG steps later.
    int keep[R][D + 1];  // arrived, not yet in the window
#pragma unroll
    for (int r = 0; r < R; r++) {
        left[r] = 0;
#pragma unroll
        for (int k = 0; k < WN; k++) win[r][k] = 0;
#pragma unroll
        for (int k = 0; k < D; k++) keep[r][k] = 0;
    }
    constexpr int last = w - 1 + 4 * (h - 1);
    int out = 0, y = lane, x = -4 * lane, seen = 0;
    // the step's noise and the luma around it, read one step ahead
    int g = 0, l[4] = {0, 0, 0, 0};
    // (outside the template some sample is read that nothing uses: no branch)
    auto fetch = [&](int yy, int xx) {
        const int yi = min(yy, h - 1), xi = max(xx, 0);
        g = C[yi * w + xi];
        if (CHROMA) {
            const int yl = max(yi, 3), xl = min(max(xi, 3), w - 4);
            const int16_t* p = L + (ssy ? 2 * yl - 3 : yl) * LW + (ssx ? 2 * xl - 3 : xl);
            l[0] = p[0];
            if (ssx) l[1] = p[1];
            if (ssy) {
                l[2] = p[LW];
                l[3] = p[LW + 1];
            }
        }
    };
    fetch(y, x);
    // seven steps per round: a window's samples come round to the same registers
#pragma unroll 7
    for (int T = 0; T <= last; T++) {
        const int gc = g;
        const int lc = !luma ? 0 : (SS == 2 ? (l[0] + l[1] + l[2] + l[3] + 2) >> 2 : SS == 1 ? (l[0] + l[1] + 1) >> 1 : l[0]) * c[NC];
        if (luma) {
            const int need = min(ssy ? 2 * (T + 1) : ssx ? T + 1 + w : T + 1, LW - 1 + 4 * (LH - 1));
            if (seen <= need) {
                // the luma warp waits for nothing, so this ends within its few hundred steps; the
                // bound, a thousand times that, only guards against a broken invariant
                for (int k = 0; (seen = *prog) <= need && k < kSpins; k++) {}
                __threadfence_block();
            }
        }
        // the lane's next step: the next sample, or its next row once that starts
        const bool end = x + 1 >= w;
        const int yn = end ? y + 32 : y, xn = end ? T + 1 - 4 * (y + 32) : x + 1;
        fetch(yn, xn);
        const bool filt = y >= 3 && x >= 3 && x < w - 3;
        int s = lc + half;
        if constexpr (LAG > 0) {
            int in[R];
            in[0] = __shfl_sync(0xffffffffu, out, (lane + 31) & 31);
#pragma unroll
            for (int r = 1; r < LAG; r++) in[r] = __shfl_sync(0xffffffffu, win[r - 1][LAG], (lane + 31) & 31);
#pragma unroll
            for (int r = 0; r < LAG; r++) {
#pragma unroll
                for (int k = 0; k + 1 < WN; k++) win[r][k] = win[r][k + 1];
                if constexpr (D == 0) {
                    win[r][WN - 1] = in[r];
                } else {
                    win[r][WN - 1] = keep[r][0];
#pragma unroll
                    for (int k = 0; k + 1 < D; k++) keep[r][k] = keep[r][k + 1];
                    keep[r][D - 1] = in[r];
                }
            }
            // a chain of multiplications per row; the left samples end the last
#pragma unroll
            for (int r = LAG - 1; r >= 0; r--) {
                int q = 0;
#pragma unroll
                for (int k = 0; k < WN; k++) q += win[r][k] * c[(LAG - 1 - r) * WN + k];
                s += q;
            }
#pragma unroll
            for (int k = LAG - 1; k >= 0; k--) s += left[k] * c[LAG * WN + LAG - 1 - k];
        }
        out = filt ? clip3(gmin, gmax, gc + (s >> shift)) : gc;
        if constexpr (LAG > 0) {
#pragma unroll
            for (int k = LAG - 1; k > 0; k--) left[k] = left[k - 1];
            left[0] = out;
        }
        if (x >= 0 && y < h) C[y * w + x] = (int16_t)out;
        if (!CHROMA && (T & 3) == 3) {
            __threadfence_block();
            __syncwarp();
            if (lane == 0) *prog = T + 1;
        }
        x = xn;
        y = yn;
    }
    if (!CHROMA) {
        __threadfence_block();
        __syncwarp();
        if (lane == 0) *prog = last + 1;
    }
}

template <int SS>
__device__ void ar_filter_lag(int16_t* C, const int16_t* L, const uint8_t* coef, const av1g_film_grain& fg, int gmin,
                              int gmax, volatile int* prog) {
    switch (fg.ar_coeff_lag) {
        case 0: ar_filter<0, SS>(C, L, coef, fg, gmin, gmax, prog); break;
        case 1: ar_filter<1, SS>(C, L, coef, fg, gmin, gmax, prog); break;
        case 2: ar_filter<2, SS>(C, L, coef, fg, gmin, gmax, prog); break;
        default: ar_filter<3, SS>(C, L, coef, fg, gmin, gmax, prog); break;
    }
}

constexpr int kTmplThreads = 256;

__global__ void __launch_bounds__(kTmplThreads) grain_template_kernel(const FrameDev* __restrict__ frames,
                                                             const int32_t* __restrict__ starts, int n, int total) {
    chain_wait();
    chain_next();
    __shared__ int16_t T[3][LH * LW];
    __shared__ int prog;
    __shared__ int16_t gauss[2048];  // the lanes draw different entries: shared, not constant, memory
    for (int i = threadIdx.x; i < 2048; i += blockDim.x) gauss[i] = (int16_t)__ldg(&g_gauss[i]);
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        int f = find_frame(starts, n, t);
        const FrameDev& F = frames[f];
        const av1g_film_grain& fg = F.h.film_grain;
        const int bd = F.h.bit_depth, ssx = F.h.subsampling_x, ssy = F.h.subsampling_y;
        const int center = 128 << (bd - 8), gmin = -center, gmax = (256 << (bd - 8)) - 1 - center;
        const int shift = 12 - bd + fg.grain_scale_shift;
        const int cw = ssx ? 44 : 82, ch = ssy ? 38 : 73;
        __syncthreads();
        for (int i = threadIdx.x; i < 3 * 256; i += blockDim.x) {
            const int p = i >> 8, v = i & 255;
            int r = 0;
            if (p < F.h.num_planes) {
                if (p == 0 || fg.chroma_scaling_from_luma) r = scaling_at(v, fg.num_y_points, fg.point_y_value, fg.point_y_scaling);
                else if (p == 1) r = scaling_at(v, fg.num_cb_points, fg.point_cb_value, fg.point_cb_scaling);
                else r = scaling_at(v, fg.num_cr_points, fg.point_cr_value, fg.point_cr_scaling);
            }
            F.grain_lut[i] = (uint8_t)r;
        }
        if (threadIdx.x == 0) prog = 0;
        // white noise (generate_grain, film_grain.rs:245-300)
        for (int job = threadIdx.x; job < LH + 2 * ch; job += blockDim.x) {
            int p = job < LH ? 0 : (job < LH + ch ? 1 : 2);
            int y = p == 0 ? job : (p == 1 ? job - LH : job - LH - ch);
            int w = p == 0 ? LW : cw;
            bool on = p == 0 ? fg.num_y_points > 0
                             : (p == 1 ? (fg.num_cb_points > 0 || fg.chroma_scaling_from_luma)
                                       : (fg.num_cr_points > 0 || fg.chroma_scaling_from_luma));
            uint16_t seed = p == 0 ? fg.grain_seed : (uint16_t)(fg.grain_seed ^ (p == 1 ? 0xb524 : 0x49d8));
            uint16_t s = on ? row_state(seed, y, (p == 0 || cw == LW) ? 0 : 1) : 0;
            int16_t* row = &T[p][y * w];
            for (int x = 0; x < w; x++) {
                int g = 0;
                if (on) {
                    s = lfsr_step(s);
                    g = gauss[(s >> 5) & 2047];
                }
                row[x] = (int16_t)r2(g, shift);
            }
        }
        __syncthreads();
        const int warp = threadIdx.x >> 5;
        if (warp == 0) {
            if (fg.num_y_points > 0)
                ar_filter_lag<-1>(T[0], nullptr, fg.ar_coeffs_y_plus_128, fg, gmin, gmax, &prog);
        } else if (warp < 3) {
            if (fg.chroma_scaling_from_luma || fg.num_cb_points > 0 || fg.num_cr_points > 0) {
                const uint8_t* cf = warp == 1 ? fg.ar_coeffs_cb_plus_128 : fg.ar_coeffs_cr_plus_128;
                if (ssy) ar_filter_lag<2>(T[warp], T[0], cf, fg, gmin, gmax, &prog);
                else if (ssx) ar_filter_lag<1>(T[warp], T[0], cf, fg, gmin, gmax, &prog);
                else ar_filter_lag<0>(T[warp], T[0], cf, fg, gmin, gmax, &prog);
            }
        } else {
            // meanwhile the per-stripe block offsets (add_noise_synthesis,
            // film_grain.rs:604-615)
            const int h = F.out[0].h;
            const int nstripes = ((h + 1) / 2 + 15) / 16, nblocks = F.grain_nblocks;
            for (int s = threadIdx.x - 96; s < nstripes; s += blockDim.x - 96) {
                uint16_t st = fg.grain_seed;
                st ^= (uint16_t)((((unsigned)s * 37 + 178) & 255) << 8);
                st ^= (uint16_t)(((unsigned)s * 173 + 105) & 255);
                for (int k = 0; k < nblocks; k++) {
                    st = lfsr_step(st);
                    F.grain_offs[s * nblocks + k] = (uint8_t)(st >> 8);
                }
            }
        }
        __syncthreads();
        int16_t* out = F.grain_tmpl;
        for (int i = threadIdx.x; i < LH * LW; i += blockDim.x) out[i] = T[0][i];
        for (int i = threadIdx.x; i < ch * cw; i += blockDim.x) {
            out[LH * LW + i] = T[1][i];
            out[2 * LH * LW + i] = T[2][i];
        }
    }
}

// ---- blend ------------------------------------------------------------------
constexpr int kBlendThreads = 256;
constexpr int kLumaCols = 8;    // luma columns of a thread: 16 bytes of a high-bit-depth row
constexpr int kTileGroups = 32;  // threads across a tile: 256 luma columns
constexpr int kStripe = 32;      // luma rows of a tile, the height of a noise stripe
constexpr int kWarps = kBlendThreads / 32;
static_assert(kTileGroups == 32, "a warp is one row of groups");

// What the CTA needs of the frame whose tiles it works on.
struct BlendPlan {
    PlaneDev in[3], out[3];
    const uint8_t* offs;
    int nblocks, hbd, bd, np, ssx, ssy, tcols;
    int gmin, gmax, overlap, scaling, rnd;
    int noise[3];             // the plane gets grain
    int minv, maxv[3];        // clip of the result
    int luma[3], self[3], add[3];  // the scaling index of a chroma sample
};

struct BlendShared {
    BlendPlan P;
    uint32_t tmpl[3][LH * LW / 2];
    uint8_t lut[3 << 12];  // scaling by sample value, 1 << bit depth entries per plane
};

// N template samples from sample `at` on, which may be odd.
template <int N>
__device__ __forceinline__ void template_row(const uint32_t* __restrict__ t, int at, int (&v)[N]) {
    const uint32_t* w = t + (at >> 1);
    const unsigned sel = (at & 1) ? 0x5432u : 0x3210u;
    uint32_t a = w[0];
#pragma unroll
    for (int e = 0; e < N; e += 2) {
        const uint32_t b = w[e / 2 + 1];
        const uint32_t u = __byte_perm(a, b, sel);
        v[e] = (int16_t)u;
        v[e + 1] = (int)u >> 16;
        a = b;
    }
}

// Noise of N adjacent samples of a plane subsampled by SX and SY: the
// materialised noiseImage of the reference (film_grain.rs:599-760) in closed
// form.  The samples lie in one block of one stripe, from column j on, in the
// stripe's row i.  `o` holds the random offsets of the block (byte 0), the block
// to its left (1) and the same two of the stripe above (2, 3).
template <int N, int SX>
__device__ __forceinline__ void stripe_row(const BlendPlan& P, const uint32_t* t, int o, bool left, int sy, int i, int j,
                                           int (&v)[N]) {
    const int tw = SX ? 44 : LW;
    const int ox = (o >> 4) & 15, oy = o & 15;
    template_row<N>(t, ((sy ? 6 + oy : 9 + oy * 2) + i) * tw + (SX ? 6 + ox : 9 + ox * 2) + j, v);
    if (left && j == 0) {  // the left block's last columns blend into the first ones
        const int px = (o >> 12) & 15, py = (o >> 8) & 15;
        const int16_t* old = reinterpret_cast<const int16_t*>(t) + ((sy ? 6 + py : 9 + py * 2) + i) * tw +
                             (SX ? 6 + px + 16 : 9 + px * 2 + 32);
        if (SX) {
            v[0] = clip3(P.gmin, P.gmax, r2(old[0] * 23 + v[0] * 22, 5));
        } else {
            v[0] = clip3(P.gmin, P.gmax, r2(old[0] * 27 + v[0] * 17, 5));
            v[1] = clip3(P.gmin, P.gmax, r2(old[1] * 17 + v[1] * 27, 5));
        }
    }
}
template <int N, int SX>
__device__ __forceinline__ void noise_row(const BlendPlan& P, const uint32_t* t, uint32_t o, bool left, bool above, int sy,
                                          int i, int j, int (&v)[N]) {
    stripe_row<N, SX>(P, t, o & 0xffff, left, sy, i, j, v);
    if (above && (sy ? i == 0 : i < 2)) {  // the stripe above's last rows blend into the first ones
        int old[N];
        stripe_row<N, SX>(P, t, o >> 16, left, sy, sy ? 16 : i + 32, j, old);
        const int a = sy ? 23 : (i == 0 ? 27 : 17), b = sy ? 22 : (i == 0 ? 17 : 27);
#pragma unroll
        for (int e = 0; e < N; e++) v[e] = clip3(P.gmin, P.gmax, r2(old[e] * a + v[e] * b, 5));
    }
}

// N samples of a row at x0, two to a word: one vector access when the group is
// whole (rows start on 16-byte boundaries), else sample by sample (x < w only).
template <int N>
__device__ __forceinline__ void ld_n(const PlaneDev& P, int hbd, int y, int x0, int w, uint32_t (&u)[N / 2]) {
    const uint8_t* row = P.p + (size_t)y * P.stride;
    if (x0 + N <= w) {
        if (hbd) {
            if constexpr (N == 8) {
                const uint4 q = *reinterpret_cast<const uint4*>(row + 2 * x0);
                u[0] = q.x, u[1] = q.y, u[2] = q.z, u[3] = q.w;
            } else {
                const uint2 q = *reinterpret_cast<const uint2*>(row + 2 * x0);
                u[0] = q.x, u[1] = q.y;
            }
        } else {
            uint32_t b[N / 4];
            if constexpr (N == 8) {
                const uint2 q = *reinterpret_cast<const uint2*>(row + x0);
                b[0] = q.x, b[1] = q.y;
            } else {
                b[0] = *reinterpret_cast<const uint32_t*>(row + x0);
            }
#pragma unroll
            for (int e = 0; e < N / 4; e++) {
                u[2 * e] = __byte_perm(b[e], 0u, 0x4140);
                u[2 * e + 1] = __byte_perm(b[e], 0u, 0x4342);
            }
        }
        return;
    }
#pragma unroll
    for (int e = 0; e < N; e += 2)
        u[e / 2] = (x0 + e < w ? (uint32_t)ld_px(P, hbd, y, x0 + e) : 0u) |
                   (x0 + e + 1 < w ? (uint32_t)ld_px(P, hbd, y, x0 + e + 1) << 16 : 0u);
}
template <int N>
__device__ __forceinline__ void unpack(const uint32_t (&u)[N / 2], int (&v)[N]) {
#pragma unroll
    for (int e = 0; e < N; e += 2) {
        v[e] = (int)(u[e / 2] & 0xffff);
        v[e + 1] = (int)(u[e / 2] >> 16);
    }
}
template <int N>
__device__ __forceinline__ void st_n(const PlaneDev& P, int hbd, int y, int x0, int w, const int (&v)[N]) {
    uint8_t* row = P.p + (size_t)y * P.stride;
    if (x0 + N <= w) {
        uint32_t u[N / 2];
#pragma unroll
        for (int e = 0; e < N / 2; e++) u[e] = (uint32_t)v[2 * e] | (uint32_t)v[2 * e + 1] << 16;
        if (hbd) {
            if constexpr (N == 8) *reinterpret_cast<uint4*>(row + 2 * x0) = make_uint4(u[0], u[1], u[2], u[3]);
            else *reinterpret_cast<uint2*>(row + 2 * x0) = make_uint2(u[0], u[1]);
        } else {
            const uint32_t a = __byte_perm(u[0], u[1], 0x6420);
            if constexpr (N == 8) *reinterpret_cast<uint2*>(row + x0) = make_uint2(a, __byte_perm(u[2], u[3], 0x6420));
            else *reinterpret_cast<uint32_t*>(row + x0) = a;
        }
        return;
    }
#pragma unroll
    for (int e = 0; e < N; e++)
        if (x0 + e < w) st_px(P, hbd, y, x0 + e, v[e]);
}

// One chroma-resolution row yc of a thread's columns: CQ chroma samples of each
// chroma plane (blended from the un-noised luma first), then the luma samples
// they cover, as the reference orders it (film_grain.rs:758-828).
template <int CQ>
__device__ __forceinline__ void blend_row(const BlendShared& S, uint32_t offs, bool left, bool above, int x0, int yc,
                                          int ly0) {
    constexpr int SX = CQ < kLumaCols;
    const BlendPlan& P = S.P;
    const int hbd = P.hbd, bd = P.bd, ssy = P.ssy, scaling = P.scaling, rnd = P.rnd, minv = P.minv;
    const int w = P.out[0].w, h = P.out[0].h, top = (1 << bd) - 1;
    const int ly = yc << ssy;
    // all the row's samples are asked for before the first is needed
    uint32_t lu[2][kLumaCols / 2], cu[2][CQ / 2];
    ld_n<kLumaCols>(P.in[0], hbd, ly, x0, w, lu[0]);
    const bool two = ssy && ly + 1 < h;
    if (two) ld_n<kLumaCols>(P.in[0], hbd, ly + 1, x0, w, lu[1]);
    if (P.np >= 3) {
        const int xc0 = x0 >> SX, gw = (w + SX) >> SX;
        ld_n<CQ>(P.in[1], hbd, yc, xc0, gw, cu[0]);
        ld_n<CQ>(P.in[2], hbd, yc, xc0, gw, cu[1]);
#pragma unroll
        for (int p = 1; p <= 2; p++) {
            int v[CQ];
            unpack<CQ>(cu[p - 1], v);
            if (P.noise[p]) {
                int l[kLumaCols], nz[CQ];
                unpack<kLumaCols>(lu[0], l);
                noise_row<CQ, SX>(P, S.tmpl[p], offs, left, above, ssy, yc - (ly0 >> ssy), xc0 & (SX ? 15 : 31), nz);
                const int a = P.luma[p], b = P.self[p], add = P.add[p], maxc = P.maxv[p];
                const uint8_t* lut = S.lut + (p << bd);
#pragma unroll
                for (int c = 0; c < CQ; c++) {
                    // average of the two luma columns, the right one clamped to the plane
                    const int avg = SX ? (l[2 * c] + (x0 + 2 * c + 1 < w ? l[2 * c + 1] : l[2 * c]) + 1) >> 1 : l[c];
                    // with scaling from luma the index is the average alone
                    const int at = clip3(0, top, ((avg * a + v[c] * b) >> 6) + add);
                    v[c] = clip3(minv, maxc, v[c] + ((lut[at] * nz[c] + rnd) >> scaling));
                }
            }
            st_n<CQ>(P.out[p], hbd, yc, xc0, gw, v);
        }
    }
#pragma unroll
    for (int dy = 0; dy < (SX ? 2 : 1); dy++) {
        if (dy && !two) break;
        int v[kLumaCols];
        unpack<kLumaCols>(lu[dy], v);
        if (P.noise[0]) {
            int nz[kLumaCols];
            noise_row<kLumaCols, 0>(P, S.tmpl[0], offs, left, above, 0, ly + dy - ly0, x0 & 31, nz);
            const int maxl = P.maxv[0];
#pragma unroll
            for (int e = 0; e < kLumaCols; e++)
                v[e] = clip3(minv, maxl, v[e] + ((S.lut[min(v[e], top)] * nz[e] + rnd) >> scaling));
        }
        st_n<kLumaCols>(P.out[0], hbd, ly + dy, x0, w, v);
    }
}

__device__ __noinline__ void plan_blend(const FrameDev& F, BlendPlan& P) {
    const av1g_frame_header& h = F.h;
    const av1g_film_grain& fg = h.film_grain;
    const int bd = h.bit_depth, np = h.num_planes, center = 128 << (bd - 8);
    for (int p = 0; p < 3; p++) {
        P.in[p] = F.lr[p];
        P.out[p] = F.out[p];
    }
    P.offs = F.grain_offs;
    P.nblocks = F.grain_nblocks;
    P.hbd = F.hbd;
    P.bd = bd;
    P.np = np;
    P.ssx = np > 1 ? h.subsampling_x : 0;
    P.ssy = np > 1 ? h.subsampling_y : 0;
    P.tcols = (F.out[0].w + kTileGroups * kLumaCols - 1) / (kTileGroups * kLumaCols);
    P.gmin = -center;
    P.gmax = (256 << (bd - 8)) - 1 - center;
    P.overlap = fg.overlap_flag;
    P.scaling = fg.grain_scaling;
    P.rnd = fg.grain_scaling ? 1 << (fg.grain_scaling - 1) : 0;
    const bool cfl = fg.chroma_scaling_from_luma;
    P.noise[0] = fg.num_y_points > 0;
    P.noise[1] = np > 1 && (cfl || fg.num_cb_points > 0);
    P.noise[2] = np > 1 && (cfl || fg.num_cr_points > 0);
    const bool clip = fg.clip_to_restricted_range;
    P.minv = clip ? 16 << (bd - 8) : 0;
    P.maxv[0] = clip ? 235 << (bd - 8) : (256 << (bd - 8)) - 1;
    P.maxv[1] = P.maxv[2] = clip && h.matrix_coefficients != 0 ? 240 << (bd - 8) : P.maxv[0];
    // (avg * luma + sample * self) >> 6, plus add; from luma: the average itself
    P.luma[1] = cfl ? 64 : fg.cb_luma_mult - 128;
    P.luma[2] = cfl ? 64 : fg.cr_luma_mult - 128;
    P.self[1] = cfl ? 0 : fg.cb_mult - 128;
    P.self[2] = cfl ? 0 : fg.cr_mult - 128;
    P.add[1] = cfl ? 0 : (fg.cb_offset - 256) * (1 << (bd - 8));
    P.add[2] = cfl ? 0 : (fg.cr_offset - 256) * (1 << (bd - 8));
}

__global__ void __launch_bounds__(kBlendThreads, 4) grain_blend_kernel(const FrameDev* __restrict__ frames,
                                                                   const int32_t* __restrict__ starts, int n, int total) {
    chain_wait();
    chain_next();
    __shared__ BlendShared S;
    const BlendPlan& P = S.P;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // each CTA walks a contiguous run of tiles, so it lays out a frame's
    // templates and tables once
    const int per = (total + gridDim.x - 1) / gridDim.x;
    const int t_end = min(total, ((int)blockIdx.x + 1) * per);
    int end = -1, first = 0;
    for (int t = blockIdx.x * per; t < t_end; t++) {
        if (t >= end) {
            const int f = find_frame(starts, n, t);
            const FrameDev& F = frames[f];
            first = starts[f];
            end = starts[f + 1];
            __syncthreads();  // the previous frame's are no longer read
            if (threadIdx.x == 0) plan_blend(F, S.P);
            const int np = F.h.num_planes, bd = F.h.bit_depth, sub = bd - 8;
            const int cw = F.h.subsampling_x ? 44 : LW, ch = F.h.subsampling_y ? 38 : LH;
            for (int p = 0; p < np; p++) {
                const uint32_t* src = reinterpret_cast<const uint32_t*>(F.grain_tmpl) + p * (LH * LW / 2);
                const int words = p ? cw * ch / 2 : LH * LW / 2;
                for (int i = threadIdx.x; i < words; i += kBlendThreads) S.tmpl[p][i] = __ldg(src + i);
                // between two of the 256 entries the table is linear; above the last, flat
                for (int x = threadIdx.x; x < 256; x += kBlendThreads) {
                    const int a = F.grain_lut[p * 256 + x], d = x < 255 ? F.grain_lut[p * 256 + x + 1] - a : 0;
                    for (int k = 0; k < 1 << sub; k++) S.lut[(p << bd) + (x << sub) + k] = (uint8_t)(a + r2(d * k, sub));
                }
            }
            __syncthreads();
        }
        const int stripe = (t - first) / P.tcols, col = (t - first) - stripe * P.tcols;
        const int x0 = (col * kTileGroups + lane) * kLumaCols, ly0 = stripe * kStripe;
        if (x0 >= P.out[0].w) continue;
        const int k = x0 >> 5;
        const bool left = P.overlap && k > 0, above = P.overlap && stripe > 0;
        const uint8_t* o = P.offs + stripe * P.nblocks + k;
        uint32_t offs = o[0];
        if (left) offs |= (uint32_t)o[-1] << 8;
        if (above) {
            offs |= (uint32_t)o[-P.nblocks] << 16;
            if (left) offs |= (uint32_t)o[-P.nblocks - 1] << 24;
        }
        const int gh = (P.out[0].h + P.ssy) >> P.ssy, yc1 = min(gh, (ly0 + kStripe) >> P.ssy);
        for (int yc = (ly0 >> P.ssy) + warp; yc < yc1; yc += kWarps) {
            if (P.ssx) blend_row<kLumaCols / 2>(S, offs, left, above, x0, yc, ly0);
            else blend_row<kLumaCols>(S, offs, left, above, x0, yc, ly0);
        }
    }
}

}  // namespace

int tiles_grain_blend(const FrameDev& f) {
    const int cols = kTileGroups * kLumaCols;
    return ((f.out[0].h + kStripe - 1) / kStripe) * ((f.out[0].w + cols - 1) / cols);
}

void launch_grain(const FrameDev* frames, const int32_t* starts_tmpl, const int32_t* starts_blend, int n,
                  int total_tmpl, int total_blend, const StageShape& sh, cudaStream_t s) {
    if (total_tmpl > 0)
        launch_chained(grain_template_kernel, total_tmpl, kTmplThreads, 0, s, frames, starts_tmpl, n, total_tmpl);
    if (total_blend <= 0) return;
    launch_chained(grain_blend_kernel, shape_grid(sh, total_blend), kBlendThreads, 0, s, frames, starts_blend, n, total_blend);
}

}  // namespace av1g
