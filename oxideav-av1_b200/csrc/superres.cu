// superres.cu — §7.16 horizontal super-resolution upscaling.
//
// Replaces upscale_frame / upscale_plane / upscale_sample
// (src/superres.rs:282-445) as called at frame_driver.rs:906-966: both the
// CDEF output and (when loop restoration is on) the deblocked frame are
// upscaled from the padded FrameWidth-wide planes to exact UpscaledWidth x
// FrameHeight planes.  A tile is 256, 512 or 1024 output samples (the launch
// shape's tile width) of eight rows of one plane of one source set, whose source
// window (clamped to the mi-padded width exactly as the reference clamps every
// tap) the CTA stages in shared memory.  A thread makes four adjacent outputs of
// a row from the six words of two samples that their taps span, as two-way dot
// products: each output's eight taps are placed among the twelve samples once
// for a whole column of tiles, since positions and phases do not depend on the row.
// The next tile's samples are in registers while this one is filtered, so a tile
// costs one barrier.
//
// Both source sets of four 3840x2160 10-bit 4:2:0 frames at denominator 12: 128 us,
// against 402 us with tiles of one row and each tap a load and a multiply-add of its
// own.  That is 40 % of the copy rate on the planes read and written; what
// remains is the dot products and the window's way through shared memory.
#include "common.cuh"
#include "av1_spec_tables.h"

namespace av1g {

namespace {

__device__ __forceinline__ int r2u(int x, int n) { return n ? (x + (1 << (n - 1))) >> n : x; }

constexpr int kSrThreads = 256;
constexpr int kSrRows = 8;               // rows per tile
constexpr int kSrPad = 24;               // the step is below 1; 8 taps, and both ends rounded outwards
constexpr __host__ __device__ int sr_pitch(int tile) { return tile + kSrPad; }

// The filters as bytes, four taps per word.  The centre taps, 3 and 4, reach
// 128, which a byte does not hold: both are stored less 64, and the two samples
// are added 64 times by themselves.
constexpr int kCentre = 64;
constexpr int filter_byte(int c, int k) { return k == 3 || k == 4 ? c - kCentre : c; }
struct SrFilters {
    uint32_t w[64][2];
};
constexpr SrFilters make_filters() {
    constexpr int f[64][8] = AV1T_UPSCALE_FILTER_INIT;
    SrFilters o{};
    for (int s = 0; s < 64; s++)
        for (int k = 0; k < 8; k++)
            o.w[s][k >> 2] |= (uint32_t)(filter_byte(f[s][k], k) & 0xff) << (8 * (k & 3));
    return o;
}
__device__ const SrFilters g_filters = make_filters();
constexpr bool filters_fit() {
    constexpr int f[64][8] = AV1T_UPSCALE_FILTER_INIT;
    for (int s = 0; s < 64; s++)
        for (int k = 0; k < 8; k++)
            if (filter_byte(f[s][k], k) < -128 || filter_byte(f[s][k], k) > 127) return false;
    return true;
}
static_assert(filters_fit(), "every tap is a signed byte");

// Output segments of a plane row.
__device__ __host__ __forceinline__ int sr_segs(int uw, int tile) { return (uw + tile - 1) / tile; }

// A plane of one source set, as a run of tiles: column of tiles by column.
struct SrPlane {
    const uint8_t* src;
    uint8_t* dst;
    int src_stride, dst_stride;
    int t0, end, groups;  // tiles [t0, end); a column is `groups` groups of kSrRows rows
    int rows, step_x, init, lim, uw, maxv, hbd;
};

__device__ __noinline__ void plan_plane(const FrameDev* __restrict__ frames, const int32_t* __restrict__ starts, int n,
                                        int t, int tile, SrPlane& P) {
    const int f = find_frame(starts, n, t);
    const FrameDev& F = frames[f];
    const av1g_frame_header& h = F.h;
    const int nsets = h.uses_lr ? 2 : 1;
    int first = starts[f];
    for (int s = 0; s < nsets; s++)
        for (int p = 0; p < h.num_planes; p++) {
            const int ssx = p ? h.subsampling_x : 0;
            const int rows = r2u(h.frame_height, p ? h.subsampling_y : 0), groups = (rows + kSrRows - 1) / kSrRows;
            const int uw = r2u(h.upscaled_width, ssx), end = first + groups * sr_segs(uw, tile);
            if (t < end) {
                // upscale_plane's step and start (superres.rs:363-377)
                const int dw = r2u(h.frame_width, ssx);
                const long long stepx_num = ((long long)dw << 14) + uw / 2;
                const int step_x = (int)(stepx_num / uw);
                const int err = (int)((long long)uw * step_x - ((long long)dw << 14));
                const long long num = -(((long long)uw - dw) << 13) + uw / 2;
                const int init = (int)(num / uw) + (1 << 7) - err / 2;
                const int max_x = (h.mi_cols >> ssx) * 4 - 1;
                const PlaneDev& S = s == 0 ? F.cdef[p] : F.deb[p];
                const PlaneDev& D = s == 0 ? F.upcdef[p] : F.updeb[p];
                P = SrPlane{S.p, D.p, S.stride, D.stride, first, end, groups, rows, step_x, init & ((1 << 14) - 1),
                            min(max_x, S.w - 1), uw, (1 << h.bit_depth) - 1, F.hbd};
                return;
            }
            first = end;
        }
}

// Four samples from x on, the row's ends repeated.
__device__ __forceinline__ uint2 load4(const uint8_t* __restrict__ row, int hbd, int x, int lim) {
    if (x >= 0 && x + 3 <= lim) {
        if (hbd) return *reinterpret_cast<const uint2*>(row + 2 * x);
        const uint32_t u = *reinterpret_cast<const uint32_t*>(row + x);
        return make_uint2(__byte_perm(u, 0u, 0x4140), __byte_perm(u, 0u, 0x4342));
    }
    uint32_t q[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
        const int sx = clip3(0, lim, x + e);
        q[e] = hbd ? reinterpret_cast<const uint16_t*>(row)[sx] : row[sx];
    }
    return make_uint2(q[0] | q[1] << 16, q[2] | q[3] << 16);
}

template <int N>
__device__ __forceinline__ void load_row(uint2 (&v)[N], const SrPlane& P, int hbd, int y, int lo, int ng, int lane) {
    if (y >= P.rows) return;
    const uint8_t* row = P.src + (size_t)y * P.src_stride;
#pragma unroll
    for (int k = 0; k < N; k++)
        if (lane + 32 * k < ng) v[k] = load4(row, hbd, lo + 4 * (lane + 32 * k), P.lim);
}

// Eight taps moved up by `by` samples (0 to 4) of a window of twelve.
struct Taps {
    int w[3];
};
__device__ __forceinline__ Taps place_taps(uint32_t lo, uint32_t hi, int by) {
    return Taps{{(int)__funnelshift_lc(0u, lo, 8 * by), (int)__funnelshift_lc(lo, hi, 8 * by),
                 (int)__funnelshift_lc(hi, 0u, 8 * by)}};
}

// sum + two products of an unsigned 16-bit sample and a signed byte: the samples of x
// (low, high half) with the lower (dp_lo) or upper (dp_hi) two bytes of w.  (__dp2a
// takes both operands' signs alike, and samples may use all 16 bits.)
__device__ __forceinline__ int dp_lo(int x, int w, int sum) {
    int d;
    asm("dp2a.lo.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "r"(w), "r"(sum));
    return d;
}
__device__ __forceinline__ int dp_hi(int x, int w, int sum) {
    int d;
    asm("dp2a.hi.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(x), "r"(w), "r"(sum));
    return d;
}

// Output J of a quad: its window starts at most J + 1 samples after the quad's first word.
template <int J>
__device__ __forceinline__ int dot(const int (&x)[6], const Taps& c, const Taps& m, int maxv) {
    int sum = dp_hi(x[1], m.w[0], 64);  // round2 by 7 bits
    sum = dp_lo(x[2], m.w[1], sum);
    if (J >= 1) sum = dp_hi(x[3], m.w[1], sum);
    if (J >= 3) sum = dp_lo(x[4], m.w[2], sum);
    sum = dp_lo(x[0], c.w[0], sum);
    sum = dp_hi(x[1], c.w[0], sum);
    sum = dp_lo(x[2], c.w[1], sum);
    sum = dp_hi(x[3], c.w[1], sum);
    sum = dp_lo(x[4], c.w[2], sum);
    if (J >= 2) sum = dp_hi(x[5], c.w[2], sum);
    return __vimin_s32_relu(sum >> 7, maxv);
}

// Four CTAs per SM: 128 us against 140 us for the three that fit unasked.
template <int TILE>
__global__ void __launch_bounds__(kSrThreads, 4) superres_kernel(const FrameDev* __restrict__ frames,
                                                              const int32_t* __restrict__ starts, int n, int total) {
    chain_wait();
    chain_next();
    constexpr int kPitch = sr_pitch(TILE);
    constexpr int kGroups = (TILE + kSrPad - 8) / 4;  // groups of four source samples at most
    constexpr int kLoads = (kGroups + 31) / 32;       // a lane's
    __shared__ __align__(16) uint16_t win[2][kSrRows * kPitch];
    __shared__ uint2 filt[64];
    __shared__ SrPlane plan;
    if (threadIdx.x < 64) filt[threadIdx.x] = make_uint2(g_filters.w[threadIdx.x][0], g_filters.w[threadIdx.x][1]);
    // a thread's columns and rows: four adjacent outputs, every parts-th row
    constexpr int kQuads = TILE / 4, kParts = kSrThreads / kQuads;
    const int quad = threadIdx.x % kQuads, part = threadIdx.x / kQuads, lane = threadIdx.x & 31, wrow = threadIdx.x >> 5;
    // each CTA walks a contiguous run of tiles, down the columns: a thread's
    // taps stay the same until the next column
    const int per = (total + gridDim.x - 1) / gridDim.x;
    const int t_end = min(total, ((int)blockIdx.x + 1) * per);
    int plan_end = -1, group = 0, seg = 0;
    int xb = 0, x1 = 0, at = 0, lo = 0, ng = 0;
    bool fresh = true, held = false;  // a column begins; `ahead` holds tile t
    Taps c[4], m[4];
    uint2 ahead[kLoads];  // the next tile's samples of this lane
    int buf = 0;
    for (int t = blockIdx.x * per; t < t_end; t++) {
        if (t >= plan_end) {
            __syncthreads();  // the previous plan is no longer read
            if (threadIdx.x == 0) plan_plane(frames, starts, n, t, TILE, plan);
            __syncthreads();
            plan_end = plan.end;
            seg = (t - plan.t0) / plan.groups;
            group = (t - plan.t0) - seg * plan.groups;
            fresh = true;
        }
        if (fresh) {
            const int start = -(1 << 14) + plan.init, step = plan.step_x, x0 = seg * TILE;
            x1 = min(plan.uw, x0 + TILE);
            xb = x0 + 4 * quad;
            // window position 0 is a multiple of four, so groups of four are aligned
            lo = (((start + x0 * step) >> 14) - 3) & ~3;
            ng = (((start + (x1 - 1) * step) >> 14) + 4 - lo) / 4 + 1;
            const int first = ((start + min(xb, x1 - 1) * step) >> 14) - 3 - lo;
            at = first & ~1;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int src_x = start + min(xb + j, x1 - 1) * step;
                const int by = (src_x >> 14) - 3 - lo - at;
                const uint2 fl = filt[(src_x >> 8) & 63];
                c[j] = place_taps(fl.x, fl.y, by);
                m[j] = place_taps((uint32_t)kCentre << 24, (uint32_t)kCentre, by);
            }
            fresh = false;
            held = false;
        }
        const int hbd = plan.hbd, y0 = group * kSrRows, rows = min(kSrRows, plan.rows - y0);
        if (!held) load_row(ahead, plan, hbd, y0 + wrow, lo, ng, lane);
#pragma unroll
        for (int k = 0; k < kLoads; k++)
            if (lane + 32 * k < ng)
                *reinterpret_cast<uint2*>(win[buf] + wrow * kPitch + 4 * (lane + 32 * k)) = ahead[k];
        __syncthreads();  // this window is whole, and the other is no longer read
        held = group + 1 < plan.groups && t + 1 < t_end;
        if (held) load_row(ahead, plan, hbd, y0 + kSrRows + wrow, lo, ng, lane);
        if (xb < x1) {
            const int maxv = plan.maxv;
            // rows start on 16-byte boundaries and xb is a multiple of four
            uint8_t* drow = plan.dst + (size_t)(y0 + part) * plan.dst_stride + (xb << hbd);
            for (int r = part; r < rows; r += kParts, drow += (size_t)kParts * plan.dst_stride) {
                const int* row = reinterpret_cast<const int*>(win[buf] + r * kPitch + at);
                const int x[6] = {row[0], row[1], row[2], row[3], row[4], row[5]};
                const int v[4] = {dot<0>(x, c[0], m[0], maxv), dot<1>(x, c[1], m[1], maxv), dot<2>(x, c[2], m[2], maxv),
                                  dot<3>(x, c[3], m[3], maxv)};
                if (xb + 4 <= x1) {
                    const uint32_t a = (uint32_t)v[0] | (uint32_t)v[1] << 16, b = (uint32_t)v[2] | (uint32_t)v[3] << 16;
                    if (hbd) *reinterpret_cast<uint2*>(drow) = make_uint2(a, b);
                    else *reinterpret_cast<uint32_t*>(drow) = __byte_perm(a, b, 0x6420);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (xb + j < x1) {
                            if (hbd) reinterpret_cast<uint16_t*>(drow)[j] = (uint16_t)v[j];
                            else drow[j] = (uint8_t)v[j];
                        }
                }
            }
        }
        buf ^= 1;
        if (++group == plan.groups) {
            group = 0;
            seg++;
            fresh = true;
        }
    }
}

}  // namespace

int tiles_superres(const FrameDev& f, int tile) {
    int tiles = 0;
    for (int p = 0; p < f.h.num_planes; p++) {
        const int ssy = p ? f.h.subsampling_y : 0, ssx = p ? f.h.subsampling_x : 0;
        const int rows = ssy ? (f.h.frame_height + 1) >> 1 : f.h.frame_height;
        const int uw = ssx ? (f.h.upscaled_width + 1) >> 1 : f.h.upscaled_width;
        tiles += (rows + kSrRows - 1) / kSrRows * sr_segs(uw, tile);
    }
    return tiles * (f.h.uses_lr ? 2 : 1);
}

void launch_superres(const FrameDev* frames, const int32_t* starts, int n, int total, const StageShape& sh,
                     cudaStream_t s) {
    if (total <= 0) return;
    const auto kernel = sh.tile == 256 ? superres_kernel<256> : sh.tile == 512 ? superres_kernel<512> : superres_kernel<1024>;
    launch_chained(kernel, shape_grid(sh, total), kSrThreads, 0, s, frames, starts, n, total);
}

}  // namespace av1g
