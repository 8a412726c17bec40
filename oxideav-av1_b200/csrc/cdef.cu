// cdef.cu — §7.15 constrained directional enhancement filter.
//
// Replaces cdef_frame / cdef_block / cdef_direction / cdef_filter_block
// (src/cdef.rs:180-606) as driven by cdef_frame_from_idx (src/cdf.rs:20300).
// One CTA owns one 64x64 filter block (the cdef_idx granularity), or some of its
// rows, across all planes.  It stages the deblocked samples of the block plus a 2-sample halo
// (the furthest tap of Cdef_Directions) for every plane in shared memory,
// marking samples outside the plane as unavailable (the reference's
// CdefAvailable == 0 arm, cdef.rs:564-590).
//
// Direction search (cdef.rs:366-456): a warp per direction and a lane per pair
// of 8x8 luma blocks, whose bins are added in packed 16-bit halves (the cost's
// bin pattern is fixed at compile time per direction, so a warp never
// diverges); the block's direction is then the arg-max over the eight costs with
// the lowest index winning ties, exactly the reference's first-strictly-greater
// scan.
// Filtering (cdef.rs:465-590): two horizontally adjacent samples per thread with
// the block's tap offsets read from a per-direction table; tiles whose halo lies
// inside the plane take a path without availability tests.
// Samples of skipped blocks (cdef_idx == -1, or all four 4x4 cells skipped)
// are copied through, as cdef_block does (cdef.rs:229-262).
//
// 8- and 10-bit frames filter two horizontally adjacent samples per thread in
// packed half-precision registers, so each add / fma / min / max serves both
// samples.  The window holds 1024 + v as half-precision bits (0x6400 | v;
// unavailable samples are NaN), every difference, threshold, weighted sum
// and clip bound is an integer below 2048 (exact in half precision), and the
// two roundings the reference asks for — floor(|d| >> damping) inside
// constrain and the (8 + sum - (sum < 0)) >> 4 of the tap sum — are each one
// round-to-nearest addition of 1536 to an exactly computed value whose
// fraction cannot be a tie.  The maximum with zero that ends constrain turns
// a NaN (unavailable) tap into a zero contribution and the clip range's min
// / max skip NaNs, which is the reference's CdefAvailable == 0 arm.  A tap is
// one aligned 32-bit load from the plane's window or from a copy of it shifted
// by one sample.  12-bit frames keep the 32-bit integer path (their sums pass
// 2048).
#include <cuda_fp16.h>

#include "common.cuh"

namespace av1g {

namespace {

constexpr int FB = 64, H2 = 2;
// A window row: 4 samples of halo, of which 2 are used, on either side of up to
// 64 samples, so that staged groups of four and pairs stay aligned.
constexpr int HX = 4, WP = FB + 2 * HX;
constexpr int kCdefThreads = 256;  // cdef_kernel's CTA size
constexpr int16_t NA = -32768;

__constant__ int8_t c_cdef_dirs[8][2][2] = {
    {{-1, 1}, {-2, 2}}, {{0, 1}, {-1, 2}}, {{0, 1}, {0, 2}}, {{0, 1}, {1, 2}},
    {{1, 1}, {2, 2}},   {{1, 0}, {2, 1}},  {{1, 0}, {2, 0}}, {{1, 0}, {2, -1}}};
__constant__ uint8_t c_uv_dir[2][2][8] = {{{0, 1, 2, 3, 4, 5, 6, 7}, {1, 2, 2, 2, 3, 4, 6, 0}},
                                          {{7, 0, 2, 4, 5, 6, 6, 6}, {0, 1, 2, 3, 4, 5, 6, 7}}};

// Costs of direction D for two 8x8 blocks at once (cdef.rs:366-440), bins fixed
// at compile time.  blk: the blocks' 64 samples, row-major, block A in the low
// halves and block B in the high ones, shifted to 8 bits and centred
// ((v >> (bitDepth - 8)) - 128), 16-byte aligned; a bin's sum is at most 8 * 128.
template <int D>
__device__ __forceinline__ void dir_cost(const uint32_t* blk, int& costa, int& costb) {
    constexpr int NB = (D == 2 || D == 6) ? 8 : ((D & 1) ? 11 : 15);
    uint32_t p[NB];
#pragma unroll
    for (int k = 0; k < NB; k++) p[k] = 0;
    const uint4* q = reinterpret_cast<const uint4*>(blk);
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
            const uint4 w = q[i * 2 + hh];
            const uint32_t xs[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int j = hh * 4 + e;
                const int b = D == 0 ? i + j : D == 1 ? i + j / 2 : D == 2 ? i : D == 3 ? 3 + i - j / 2
                            : D == 4 ? 7 + i - j : D == 5 ? 3 - i / 2 + j : D == 6 ? j : i / 2 + j;
                p[b] = __vadd2(p[b], xs[e]);
            }
        }
    auto total = [&](auto val) {
        int cost = 0;
        if (D == 2 || D == 6) {
#pragma unroll
            for (int k = 0; k < 8; k++) cost += val(k) * val(k);
            cost *= 105;
        } else if (D == 0 || D == 4) {
            constexpr int div[8] = {840, 420, 280, 210, 168, 140, 120, 105};
#pragma unroll
            for (int k = 0; k < 7; k++) cost += (val(k) * val(k) + val(14 - k) * val(14 - k)) * div[k];
            cost += val(7) * val(7) * 105;
        } else {
            constexpr int div2[3] = {420, 210, 140};
#pragma unroll
            for (int k = 0; k < 5; k++) cost += val(3 + k) * val(3 + k);
            cost *= 105;
#pragma unroll
            for (int k = 0; k < 3; k++) cost += (val(k) * val(k) + val(10 - k) * val(10 - k)) * div2[k];
        }
        return cost;
    };
    costa = total([&](int k) { return (int)(int16_t)(p[k] & 0xffff); });
    costb = total([&](int k) { return (int)p[k] >> 16; });
}

__device__ __forceinline__ int constrain_adj(int diff, int threshold, int adj) {
    // constrain (cdef.rs:592-606) with dampingAdj precomputed:
    // min(|d|, max(t - (|d| >> adj), 0)) == max(min(|d|, t - (|d| >> adj)), 0) as |d| >= 0
    int ad = abs(diff);
    int v = __vimin_s32_relu(ad, threshold - (ad >> adj));
    return diff < 0 ? -v : v;
}

// Tap offsets of one direction: primary (k = 0, 1), then the two secondary
// directions (dir + 2, dir - 2) for k = 0, 1.
struct Taps {
    int p0, p1, a0, a1, b0, b1;
};

__device__ __forceinline__ Taps taps_of(const int* toff, int dir) {
    const int da = (dir + 2) & 7, db = (dir + 6) & 7;
    return Taps{toff[dir * 2], toff[dir * 2 + 1], toff[da * 2], toff[da * 2 + 1], toff[db * 2], toff[db * 2 + 1]};
}

// One tap pair (+o and -o) of weight w: constrain (cdef.rs:592-606) with the
// damping shift precomputed, accumulated into sum; with MINMAX, min / max of
// the samples taken (the reference's clip range, cdef.rs:540-560).
template <bool BORDER, bool MINMAX>
__device__ __forceinline__ void tap2(const int16_t* c, int o, int xv, int w, int thr, int adj, int& sum, int& mn,
                                     int& mx) {
    if (!BORDER) {  // both taps available: one weight product, three-input min / max
        const int x0 = c[o], x1 = c[-o];
        sum += w * (constrain_adj(x0 - xv, thr, adj) + constrain_adj(x1 - xv, thr, adj));
        if (MINMAX) {
            mx = __vimax3_s32(mx, x0, x1);
            mn = __vimin3_s32(mn, x0, x1);
        }
        return;
    }
#pragma unroll
    for (int s = 0; s < 2; s++) {
        const int x = s ? c[-o] : c[o];
        if (x == NA) continue;
        sum += w * constrain_adj(x - xv, thr, adj);
        if (MINMAX) {
            mx = max(mx, x);
            mn = min(mn, x);
        }
    }
}

// One sample of cdef_filter (cdef.rs:465-590).  MODE 3: primary and
// secondary taps, clipped to the taps' range as the reference always does.
// MODE 1 / 2: only the primary / only the secondary strength is non-zero;
// the taps of a zero strength add nothing (constrain with threshold 0 is 0)
// and the clip is the identity, so both are left out: the remaining taps'
// weights sum to 12 (2 x (4 + 2), 2 x (3 + 3), or 2 x 2 x (2 + 1)), each
// constrained difference has its tap's sign and at most its magnitude, so
// with D the largest positive difference sum <= 12 D and
// (8 + sum) >> 4 <= D (and symmetrically below): x + offset stays inside
// [min, max] of the taps, and the unclipped value is the clipped one.
template <bool BORDER, int MODE>
__device__ __forceinline__ int filter_px(const int16_t* c, int xv, const Taps& T, int pri, int sec, int padj,
                                         int sadj, int pt0, int pt1) {
    constexpr bool MM = MODE == 3;
    int sum = 0, mx = xv, mn = xv;
    if (MODE & 1) {
        tap2<BORDER, MM>(c, T.p0, xv, pt0, pri, padj, sum, mn, mx);
        tap2<BORDER, MM>(c, T.p1, xv, pt1, pri, padj, sum, mn, mx);
    }
    if (MODE & 2) {
        tap2<BORDER, MM>(c, T.a0, xv, 2, sec, sadj, sum, mn, mx);
        tap2<BORDER, MM>(c, T.b0, xv, 2, sec, sadj, sum, mn, mx);
        tap2<BORDER, MM>(c, T.a1, xv, 1, sec, sadj, sum, mn, mx);
        tap2<BORDER, MM>(c, T.b1, xv, 1, sec, sadj, sum, mn, mx);
    }
    const int y = xv + ((8 + sum - (sum < 0)) >> 4);
    return MM ? clip3(mn, mx, y) : y;
}

// ---- half-precision path (8- and 10-bit) ---------------------------------

constexpr uint16_t kHalfNA = 0x7E00;        // NaN: a tap outside the plane
constexpr uint32_t kH1536 = 0x66006600u;    // 1536, 1536
constexpr uint32_t kHNeg1 = 0xBC00BC00u;    // -1, -1
constexpr uint32_t kH1_16 = 0x2C002C00u;    // 1/16, 1/16
constexpr uint32_t kH1_32 = 0x28002800u;    // 1/32, 1/32
constexpr uint32_t kSign2 = 0x80008000u;

__device__ __forceinline__ __half2 u2h(uint32_t u) {
    __half2 h;
    memcpy(&h, &u, 4);
    return h;
}
__device__ __forceinline__ uint32_t h2u(__half2 h) {
    uint32_t u;
    memcpy(&u, &h, 4);
    return u;
}

// Half-precision constants of one strength: 1536 + t, 2^-adj and
// -(2^adj - 1) / 2^(adj + 1), each in both lanes.
struct HalfStrength {
    uint32_t tb, k, c;
};

__device__ __forceinline__ HalfStrength half_strength(int t, int adj) {
    const uint32_t tb = __half_as_ushort(__int2half_rn(1536 + t));
    const uint32_t k = (uint32_t)(15 - adj) << 10;  // 2^-adj (adj <= 9)
    const uint32_t c = __half_as_ushort(__float2half_rn(-(float)((1 << adj) - 1) / (float)(2 << adj)));
    return HalfStrength{tb * 0x10001u, k * 0x10001u, c * 0x10001u};
}

// constrain (cdef.rs:592-606) of two taps against two centres, both
// biased by 1024: |d| * 2^-adj - (2^adj - 1) / 2^(adj+1) is exact, adding
// 1536 rounds it to 1536 + (|d| >> adj), the threshold minus that is exact,
// and the result takes d's sign bit.  BORDER: NaN taps (outside the plane)
// give 0 through the NaN-skipping maximum with zero.
template <bool BORDER>
__device__ __forceinline__ __half2 constrain_h(__half2 x, __half2 xv, const HalfStrength& S) {
    const __half2 d = __hsub2(x, xv);
    const __half2 ad = __habs2(d);
    const __half2 v2 = __hadd2(__hfma2(ad, u2h(S.k), u2h(S.c)), u2h(kH1536));
    const __half2 m = BORDER ? __hmax2(__hsub2(u2h(S.tb), v2), u2h(0u)) : __hfma2_relu(v2, u2h(kHNeg1), u2h(S.tb));
    return u2h(h2u(__hmin2(ad, m)) | (h2u(d) & kSign2));
}

// One pair of taps (bytes from the centre pair; an odd column offset points
// into the shifted window, so every tap is one aligned 32-bit load) of weight w
// for two samples, with the clip range.
__device__ __forceinline__ __half2 ld_at(const uint16_t* cp, int byteoff) {
    return u2h(*reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(cp) + byteoff));
}
template <bool BORDER, bool MINMAX>
__device__ __forceinline__ void tap2_h(const uint16_t* cp, int e0, int e1, __half2 xv, uint32_t w, const HalfStrength& S,
                                       __half2& sum, __half2& mn, __half2& mx) {
    const __half2 x0 = ld_at(cp, e0), x1 = ld_at(cp, e1);
    sum = __hfma2(u2h(w), __hadd2(constrain_h<BORDER>(x0, xv, S), constrain_h<BORDER>(x1, xv, S)), sum);
    if (MINMAX) {
        mx = __hmax2(mx, __hmax2(x0, x1));
        mn = __hmin2(mn, __hmin2(x0, x1));
    }
}

// cdef_filter (cdef.rs:465-590) of two adjacent samples; MODE as filter_px; eo:
// the direction's tap offsets: primary k = 0, 1, secondary (dir + 2) k = 0, 1,
// secondary (dir - 2) k = 0, 1, each +offset then -offset.  Returns the two
// filtered samples as half-precision bits 0x6400 | value.
template <bool BORDER, int MODE>
__device__ __forceinline__ uint32_t filter_pair_h(const uint16_t* cp, __half2 xv, const int* eo, const HalfStrength& P,
                                                  uint32_t pw0, uint32_t pw1, const HalfStrength& Sc) {
    constexpr bool MM = MODE == 3;
    __half2 sum = u2h(0u), mn = xv, mx = xv;
    const int4* e4 = reinterpret_cast<const int4*>(eo);
    if (MODE & 1) {
        const int4 e = e4[0];
        tap2_h<BORDER, MM>(cp, e.x, e.y, xv, pw0, P, sum, mn, mx);
        tap2_h<BORDER, MM>(cp, e.z, e.w, xv, pw1, P, sum, mn, mx);
    }
    if (MODE & 2) {
        const int4 a = e4[1], b = e4[2];
        tap2_h<BORDER, MM>(cp, a.x, a.y, xv, 0x40004000u, Sc, sum, mn, mx);  // weight 2
        tap2_h<BORDER, MM>(cp, b.x, b.y, xv, 0x40004000u, Sc, sum, mn, mx);
        tap2_h<BORDER, MM>(cp, a.z, a.w, xv, 0x3C003C00u, Sc, sum, mn, mx);  // weight 1
        tap2_h<BORDER, MM>(cp, b.z, b.w, xv, 0x3C003C00u, Sc, sum, mn, mx);
    }
    // (8 + sum - (sum < 0)) >> 4: sum / 16 + copysign(1/32, sum) is exact and
    // never a half-integer; adding 1536 rounds it to the reference's offset
    const __half2 g = __hfma2(sum, u2h(kH1_16), u2h((h2u(sum) & kSign2) | kH1_32));
    __half2 y = __hadd2(__hadd2(g, u2h(kH1536)), __hsub2(xv, u2h(kH1536)));
    if (MM) y = __hmin2(__hmax2(y, mn), mx);
    return h2u(y);
}

template <bool BORDER>
__device__ __forceinline__ void filter_two(const int16_t* cp, int xv0, int xv1, const Taps& T, int pri, int sec,
                                           int padj, int sadj, int pt0, int pt1, int& out0, int& out1) {
    if (pri && sec) {
        out0 = filter_px<BORDER, 3>(cp, xv0, T, pri, sec, padj, sadj, pt0, pt1);
        out1 = filter_px<BORDER, 3>(cp + 1, xv1, T, pri, sec, padj, sadj, pt0, pt1);
    } else if (pri) {
        out0 = filter_px<BORDER, 1>(cp, xv0, T, pri, sec, padj, sadj, pt0, pt1);
        out1 = filter_px<BORDER, 1>(cp + 1, xv1, T, pri, sec, padj, sadj, pt0, pt1);
    } else if (sec) {
        out0 = filter_px<BORDER, 2>(cp, xv0, T, pri, sec, padj, sadj, pt0, pt1);
        out1 = filter_px<BORDER, 2>(cp + 1, xv1, T, pri, sec, padj, sadj, pt0, pt1);
    }
}

// A tile: RB rows of a 64x64 filter block, and the strengths its frame and block
// select, worked out once by one thread while the CTA filters the tile before.
struct Tile {
    int frame, fbr, fbc, row0, idx;  // row0: its first luma row inside the block
    int border;                      // some luma tap lies outside the plane
    HalfStrength sec[2], pri_uv;     // luma / chroma secondary, chroma primary
    int sec_v[2], sadj[2], pri_uv_v, padj_uv;
};

__device__ void plan_tile(Tile& T, const FrameDev* __restrict__ frames, const int32_t* __restrict__ starts, int n,
                          int t, int rb) {
    const int sub = t % (FB / rb);
    t /= FB / rb;
    const int f = find_frame(starts, n, t);
    const FrameDev& F = frames[f];
    const av1g_frame_header& h = F.h;
    const int local = t - starts[f], fcols = (h.mi_cols + 15) >> 4;
    T.frame = f;
    T.fbr = local / fcols;
    T.fbc = local - T.fbr * fcols;
    T.row0 = sub * rb;
    int idx = F.cdef_idx[local];
    if (idx > 7) idx = -1;  // not a strength-set index: malformed, copied through
    T.idx = idx;
    const int lx0 = T.fbc * FB, ly0 = T.fbr * FB + T.row0;
    T.border = lx0 < H2 || ly0 < H2 || lx0 + FB + H2 > F.deb[0].w || ly0 + rb + H2 > F.deb[0].h;
    const int cs = h.bit_depth - 8;
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const int sec = idx >= 0 ? (c ? h.cdef_uv_sec[idx] : h.cdef_y_sec[idx]) << cs : 0;
        T.sec_v[c] = sec;
        T.sadj[c] = sec ? max(h.cdef_damping + cs - c - floor_log2u((unsigned)sec), 0) : 0;
        T.sec[c] = half_strength(sec, T.sadj[c]);
    }
    const int pri = idx >= 0 ? h.cdef_uv_pri[idx] << cs : 0;
    T.pri_uv_v = pri;
    T.padj_uv = pri ? max(h.cdef_damping + cs - 1 - floor_log2u((unsigned)pri), 0) : 0;
    T.pri_uv = half_strength(pri, T.padj_uv);
}

// Per 8x8 luma block: the luma primary strength's half-precision constants, and
// the direction | chroma direction << 4 | filtered << 8 | odd primary row
// (Cdef_Pri_Taps) << 9 | luma primary strength non-zero << 10.
struct alignas(16) BlockParams {
    uint32_t tb, k, c, misc;
};

template <int RB>
struct CdefShared {
    static constexpr int BR = RB / 8, NB = BR * 8, NP = NB / 2;  // block rows, blocks, pairs of blocks
    // luma of the 8x8 blocks b (low halves) and b + NP (high halves), four words
    // of padding per pair, so that lanes reading 16 bytes of successive pairs spread over the banks
    alignas(16) uint32_t pair[NP][68];
    alignas(16) int deo[8][12];  // tap byte offsets by direction (see filter_pair_h)
    BlockParams bp[NB];
    int2 bpi[NB];  // 12-bit: luma primary strength, its damping shift
    int costs[NB][9];
    int toff[16];
    uint8_t blive[NB];  // 8x8 luma block filtered (inside the mi grid, not all skip)
    Tile tile[2];
};

// Samples of the three planes' windows: RB (+ halo) luma rows, chroma rows by
// whether any frame of the batch keeps full vertical chroma.
template <int RB>
constexpr __host__ __device__ int window_samples(bool full_chroma) {
    return (RB + 2 * H2) * WP + 2 * ((full_chroma ? RB : RB / 2) + 2 * H2) * WP;
}
template <int RB>
constexpr size_t cdef_smem(bool full_chroma) {
    return sizeof(CdefShared<RB>) + 2 * 2 * (size_t)window_samples<RB>(full_chroma);
}

// One CTA per tile.  Shared memory: CdefShared, the planes' windows, and a copy
// of the windows shifted by one sample (copy[i] = window[i + 1]), so that a pair
// of samples that starts at an odd column is one aligned word too.
//
// Bound by instruction issue: 64 x 1080p 8-bit 1.21 ms (1.53 ms when every
// thread derived the tile and its strengths, a direction lane took one block, and
// chroma taps were two loads and a permute).  RB = 64 is one CTA per filter
// block; smaller ones serve batches of few blocks (launch_cdef).
template <int RB>
__global__ void __launch_bounds__(kCdefThreads, 4) cdef_kernel(const FrameDev* __restrict__ frames,
                                                      const int32_t* __restrict__ starts, int n, int total,
                                                      int full_chroma) {
    chain_wait();
    chain_next();
    extern __shared__ __align__(16) unsigned char cdef_raw[];
    using SM = CdefShared<RB>;
    SM& S = *reinterpret_cast<SM*>(cdef_raw);
    uint16_t* const win = reinterpret_cast<uint16_t*>(cdef_raw + sizeof(SM));
    const int shift = window_samples<RB>(full_chroma);  // from a window to its shifted copy
    const int cwin = ((full_chroma ? RB : RB / 2) + 2 * H2) * WP;
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid < 16) S.toff[tid] = c_cdef_dirs[tid >> 1][tid & 1][0] * WP + c_cdef_dirs[tid >> 1][tid & 1][1];
    if (tid >= 32 && tid < 32 + 96) {
        const int dir = (tid - 32) / 12, q = (tid - 32) % 12, t = q >> 1;  // t: primary 0-1, dir + 2, dir - 2
        const int d2 = t < 2 ? dir : t < 4 ? (dir + 2) & 7 : (dir + 6) & 7;
        const int o = c_cdef_dirs[d2][t & 1][0] * WP + c_cdef_dirs[d2][t & 1][1], v = (q & 1) ? -o : o;
        S.deo[dir][q] = 2 * ((v & 1) ? v - 1 + shift : v);
    }
    const bool planner = tid == kCdefThreads - 32;
    if (planner && (int)blockIdx.x < total) plan_tile(S.tile[0], frames, starts, n, blockIdx.x, RB);
    int cur = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x, cur ^= 1) {
        __syncthreads();  // the tile is worked out; the previous one is done with shared memory
        if (planner && t + (int)gridDim.x < total) plan_tile(S.tile[cur ^ 1], frames, starts, n, t + gridDim.x, RB);
        const Tile& T = S.tile[cur];
        const FrameDev& F = frames[T.frame];
        const av1g_frame_header& h = F.h;
        const int idx = T.idx, hbd = F.hbd, np = h.num_planes;
        const int ssx = h.subsampling_x, ssy = h.subsampling_y, cs = h.bit_depth - 8;
        const bool half = h.bit_depth <= 10;  // the half-precision filter path
        const int lx0 = T.fbc * FB, ly0 = T.fbr * FB + T.row0;
        if (ly0 >= F.deb[0].h) continue;  // rows of the block past the plane (uniform)
        for (int p = 0; p < np; p++) {
            const int px = p ? ssx : 0, py = p ? ssy : 0;
            const int bw = FB >> px, wh = (RB >> py) + 2 * H2;
            const int x0 = lx0 >> px, y0 = ly0 >> py;
            const PlaneDev& D = F.deb[p];
            uint16_t* const w = win + (p == 0 ? 0 : (RB + 2 * H2) * WP + (p - 1) * cwin);
            // 8-bit centred luma of the direction search
            auto put_dir = [&](int sr, int sc, int v) {
                const int blk = ((sr >> 3) << 3) + (sc >> 3), hi = blk >= SM::NP;
                reinterpret_cast<int16_t*>(&S.pair[blk - (hi ? SM::NP : 0)][((sr & 7) << 3) + (sc & 7)])[hi] =
                    (int16_t)((v >> cs) - 128);
            };
            if (x0 >= HX && y0 >= H2 && x0 + bw + HX <= D.w && y0 + wh - H2 <= D.h) {
                // interior: aligned 4-sample loads over [x0 - 4, x0 + bw + 4),
                // every one inside the plane; a thread's loads are issued
                // before it unpacks any, so their latencies overlap
                const bool full = bw == FB;
                const int ng = full ? (FB + 8) / 4 : (FB / 2 + 8) / 4, items = wh * ng;
                const unsigned mag = full ? (1u << 16) / ((FB + 8) / 4) + 1 : (1u << 16) / ((FB / 2 + 8) / 4) + 1;
                constexpr int PER = ((RB + 2 * H2) * ((FB + 8) / 4) + kCdefThreads - 1) / kCdefThreads;
                const uint8_t* base = D.p + (size_t)(y0 - H2) * D.stride + ((x0 - HX) << hbd);
                uint2 q[PER];
                uint32_t nx[PER];  // the first samples of the next group
#pragma unroll
                for (int k = 0; k < PER; k++) {
                    const int i = tid + k * kCdefThreads;
                    q[k] = make_uint2(0u, 0u);
                    nx[k] = 0;
                    if (i < items) {
                        const int r = (int)(((unsigned)i * mag) >> 16), g = i - r * ng;
                        const uint8_t* a = base + (size_t)r * D.stride + ((4 * g) << hbd);
                        if (hbd) q[k] = *reinterpret_cast<const uint2*>(a);
                        else q[k].x = *reinterpret_cast<const uint32_t*>(a);
                        // the last lane has no neighbour in its warp
                        if (lane == 31 && g + 1 < ng) nx[k] = *reinterpret_cast<const uint32_t*>(a + (4 << hbd));
                    }
                }
#pragma unroll
                for (int k = 0; k < PER; k++) {
                    const int i = tid + k * kCdefThreads;
                    const uint32_t nl = __shfl_down_sync(0xffffffffu, q[k].x, 1);
                    if (i >= items) continue;
                    const uint32_t nxt = lane == 31 ? nx[k] : nl;  // (garbage past a row's end, which no tap reads)
                    const int r = (int)(((unsigned)i * mag) >> 16), g = i - r * ng;
                    // the group as pairs of u16, and the pairs one sample on
                    uint32_t lo, hi, s0, s1;
                    if (hbd) {
                        lo = q[k].x;
                        hi = q[k].y;
                        s0 = __byte_perm(lo, hi, 0x5432);
                        s1 = __byte_perm(hi, nxt, 0x5432);
                    } else {
                        lo = __byte_perm(q[k].x, 0u, 0x4140);
                        hi = __byte_perm(q[k].x, 0u, 0x4342);
                        s0 = __byte_perm(q[k].x, 0u, 0x4241);
                        s1 = (q[k].x >> 24) | ((nxt & 0xff) << 16);
                    }
                    if (p == 0 && r >= H2 && r < H2 + RB && g >= 1 && g <= FB / 4) {
                        const int sr = r - H2, sc = 4 * g - HX;
                        put_dir(sr, sc, lo & 0xffff);
                        put_dir(sr, sc + 1, lo >> 16);
                        put_dir(sr, sc + 2, hi & 0xffff);
                        put_dir(sr, sc + 3, hi >> 16);
                    }
                    const uint32_t bias = half ? 0x64006400u : 0u;  // biased half-precision samples
                    uint16_t* o = w + r * WP + 4 * g;
                    *reinterpret_cast<uint2*>(o) = make_uint2(lo | bias, hi | bias);
                    *reinterpret_cast<uint2*>(o + shift) = make_uint2(s0 | bias, s1 | bias);
                }
            } else {
                for (int i = tid; i < WP * wh; i += kCdefThreads) {
                    const int r = i / WP, c = i - r * WP;
                    const int gy = y0 - H2 + r, gx = x0 - HX + c;
                    const bool in = gy >= 0 && gy < D.h && gx >= 0 && gx < D.w;
                    const int v = in ? ld_px(D, hbd, gy, gx) : 0;
                    const uint16_t o = half ? (uint16_t)(in ? 0x6400 | v : kHalfNA) : (uint16_t)(in ? v : NA);
                    w[i] = o;
                    if (i > 0) w[i - 1 + shift] = o;
                    if (p == 0 && r >= H2 && r < H2 + RB && c >= HX && c < HX + FB) put_dir(r - H2, c - HX, v);
                }
            }
        }
        // which 8x8 blocks are filtered (cdef_block's skip test, cdef.rs:229-262):
        // the four mi skip flags loaded together, out-of-grid ones read as skip
        if (tid < SM::NB) {
            const int r = (ly0 >> 2) + (tid >> 3) * 2, c = T.fbc * 16 + (tid & 7) * 2;
            bool live = idx >= 0 && r < h.mi_rows && c < h.mi_cols;
            if (live) {
                const uint8_t* sk = F.g.skip;
                const int mc = h.mi_cols;
                const bool rn = r + 1 < h.mi_rows, cn = c + 1 < mc;
                const int s00 = sk[r * mc + c];
                const int s10 = rn ? sk[(r + 1) * mc + c] : 1;
                const int s01 = cn ? sk[r * mc + c + 1] : 1;
                const int s11 = rn && cn ? sk[(r + 1) * mc + c + 1] : 1;
                live = !(s00 && s10 && s01 && s11);
            }
            S.blive[tid] = live;
        }
        __syncthreads();
        // direction search: a warp per direction, a lane per pair of blocks; one
        // thread per block then takes the arg-max
        if (lane < SM::NP && (S.blive[lane] || S.blive[lane + SM::NP])) {
            int ca, cb;
            const uint32_t* w = S.pair[lane];
            switch (tid >> 5) {
                case 0: dir_cost<0>(w, ca, cb); break;
                case 1: dir_cost<1>(w, ca, cb); break;
                case 2: dir_cost<2>(w, ca, cb); break;
                case 3: dir_cost<3>(w, ca, cb); break;
                case 4: dir_cost<4>(w, ca, cb); break;
                case 5: dir_cost<5>(w, ca, cb); break;
                case 6: dir_cost<6>(w, ca, cb); break;
                default: dir_cost<7>(w, ca, cb); break;
            }
            S.costs[lane][tid >> 5] = ca;
            S.costs[lane + SM::NP][tid >> 5] = cb;
        }
        __syncthreads();
        if (tid < SM::NB) {
            BlockParams b{0, 0, 0, 0};
            int2 bi = make_int2(0, 0);
            if (S.blive[tid]) {
                // first strictly greater wins (cdef.rs:440-456)
                int best = S.costs[tid][0], bd = 0;
#pragma unroll
                for (int d = 1; d < 8; d++)
                    if (S.costs[tid][d] > best) {
                        best = S.costs[tid][d];
                        bd = d;
                    }
                const int var = (best - S.costs[tid][(bd + 4) & 7]) >> 10;
                const int pri = h.cdef_y_pri[idx] << cs;
                const int vs = (var >> 6) > 0 ? min(floor_log2u((unsigned)(var >> 6)), 12) : 0;
                const int pri_y = var != 0 ? (pri * (4 + vs) + 8) >> 4 : 0;
                const int padj = pri_y ? max(h.cdef_damping + cs - floor_log2u((unsigned)pri_y), 0) : 0;
                const int ydir = pri == 0 ? 0 : bd, uvdir = T.pri_uv_v == 0 ? 0 : c_uv_dir[ssx][ssy][bd];
                bi = make_int2(pri_y, padj);
                if (half) {
                    const HalfStrength hs = half_strength(pri_y, padj);
                    b.tb = hs.tb;
                    b.k = hs.k;
                    b.c = hs.c;
                }
                b.misc = (uint32_t)(ydir | uvdir << 4 | 1 << 8 | ((pri_y >> cs) & 1) << 9 | (pri_y ? 1 : 0) << 10);
            }
            S.bp[tid] = b;
            S.bpi[tid] = bi;
        }
        __syncthreads();
        const bool border = T.border;
        for (int p = 0; p < np; p++) {
            const int px = p ? ssx : 0, py = p ? ssy : 0, ch = p ? 1 : 0;
            const int bh = RB >> py, lbw = 6 - px;
            const int x0 = lx0 >> px, y0 = ly0 >> py;
            const PlaneDev& D = F.cdef[p];
            const int dh = min(D.h, F.deb[p].h), dw = min(D.w, F.deb[p].w);
            const int rows = min(bh, dh - y0);
            // a thread takes a pair of columns, every rstep-th row
            const int c = (2 * tid) & ((FB >> px) - 1), rstep = (2 * kCdefThreads) >> lbw, gx = x0 + c;
            if (gx >= dw) continue;
            int r = (2 * tid) >> lbw;
            const uint16_t* cp = win + (p == 0 ? 0 : (RB + 2 * H2) * WP + (p - 1) * cwin) + (r + H2) * WP + c + HX;
            uint8_t* out = D.p + (size_t)(y0 + r) * D.stride + (gx << hbd);
            const bool both = gx + 1 < dw;  // gx is even: one aligned 2- or 4-byte store
            const int bc = c >> (3 - px);
            if (half) {
                const HalfStrength Sc = T.sec[ch];
                const int sec = T.sec_v[ch] ? 2 : 0;
                HalfStrength P = T.pri_uv;
                bool prow = (T.pri_uv_v >> cs) & 1;
                int pri = T.pri_uv_v ? 1 : 0;
                for (; r < rows; r += rstep, cp += rstep * WP, out += (size_t)rstep * D.stride) {
                    const BlockParams b = S.bp[(r >> (3 - py)) * 8 + bc];
                    const __half2 xv = u2h(*reinterpret_cast<const uint32_t*>(cp));
                    uint32_t o = h2u(xv);
                    if (p == 0) {
                        P = HalfStrength{b.tb, b.k, b.c};
                        prow = b.misc & (1 << 9);
                        pri = (b.misc >> 10) & 1;
                    }
                    const int mode = pri | sec;
                    if ((b.misc & (1 << 8)) && mode) {
                        const int* eo = S.deo[(p ? b.misc >> 4 : b.misc) & 7];
                        const uint32_t pw0 = prow ? 0x42004200u : 0x44004400u;  // 3 : 4
                        const uint32_t pw1 = prow ? 0x42004200u : 0x40004000u;  // 3 : 2
                        // in border tiles the taps of a zero strength run too:
                        // they add nothing and the clip is the identity
                        if (border || mode == 3) {
                            o = border ? filter_pair_h<true, 3>(cp, xv, eo, P, pw0, pw1, Sc)
                                       : filter_pair_h<false, 3>(cp, xv, eo, P, pw0, pw1, Sc);
                        } else if (mode == 1) {
                            o = filter_pair_h<false, 1>(cp, xv, eo, P, pw0, pw1, Sc);
                        } else {
                            o = filter_pair_h<false, 2>(cp, xv, eo, P, pw0, pw1, Sc);
                        }
                    }
                    // o holds 0x6400 | value per lane
                    if (both) {
                        if (hbd) *reinterpret_cast<uint32_t*>(out) = o & 0x03FF03FFu;
                        else *reinterpret_cast<uint16_t*>(out) = (uint16_t)__byte_perm(o, 0u, 0x0020);
                    } else {
                        st_px(D, hbd, y0 + r, gx, (int)(o & 0x3FFu));
                    }
                }
                continue;
            }
            // 12-bit: 32-bit integers, as the reference states it
            for (; r < rows; r += rstep, cp += rstep * WP, out += (size_t)rstep * D.stride) {
                const int blk = (r >> (3 - py)) * 8 + bc;
                const int16_t* cw = reinterpret_cast<const int16_t*>(cp);
                const int xv0 = cw[0], xv1 = cw[1];
                const uint32_t misc = S.bp[blk].misc;
                int out0 = xv0, out1 = xv1;
                if (misc & (1 << 8)) {
                    const int pri = p ? T.pri_uv_v : S.bpi[blk].x, padj = p ? T.padj_uv : S.bpi[blk].y;
                    const Taps tp = taps_of(S.toff, (p ? misc >> 4 : misc) & 7);
                    const int prow = (pri >> cs) & 1, pt0 = prow ? 3 : 4, pt1 = prow ? 3 : 2;
                    if (border) filter_two<true>(cw, xv0, xv1, tp, pri, T.sec_v[ch], padj, T.sadj[ch], pt0, pt1, out0, out1);
                    else filter_two<false>(cw, xv0, xv1, tp, pri, T.sec_v[ch], padj, T.sadj[ch], pt0, pt1, out0, out1);
                }
                if (both) *reinterpret_cast<uint32_t*>(out) = (uint32_t)out0 | (uint32_t)out1 << 16;
                else st_px(D, hbd, y0 + r, gx, out0);
            }
        }
    }
}

template <int RB>
void launch(const FrameDev* frames, const int32_t* starts, int n, int total, bool full_chroma, const StageShape& sh,
            cudaStream_t s) {
    const size_t bytes = cdef_smem<RB>(full_chroma);
    // the largest size either way, so that no concurrent launch finds it lowered
    cudaFuncSetAttribute(cdef_kernel<RB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cdef_smem<RB>(true));
    total *= FB / RB;
    launch_chained(cdef_kernel<RB>, shape_grid(sh, total), kCdefThreads, bytes, s, frames, starts, n, total, full_chroma);
}

}  // namespace

int tiles_cdef(const FrameDev& f) { return ((f.h.mi_rows + 15) >> 4) * ((f.h.mi_cols + 15) >> 4); }

void launch_cdef(const FrameDev* frames, const int32_t* starts, int n, int total, bool full_chroma,
                 const StageShape& sh, cudaStream_t s) {
    if (total <= 0) return;
    // A launch of few blocks takes as long as one tile: quarter tiles up to a
    // block per SM (640x360: 12.2 us, 15.6 with halves, 24.1 with whole blocks),
    // half tiles up to the blocks that are resident at once (1280x720: 19.4, 23.1
    // with quarters, 26.9 with whole ones) and where three full-size windows
    // would leave room for three CTAs (4:4:4, 12 x 718p: 199, 212 with whole
    // ones); above, whole blocks stage the least halo (64 x 1080p: 1.21 ms, 1.50
    // with halves).
    if (total <= kSMs) launch<16>(frames, starts, n, total, full_chroma, sh, s);
    else if (total <= kSMs * 4 || full_chroma) launch<32>(frames, starts, n, total, full_chroma, sh, s);
    else launch<64>(frames, starts, n, total, full_chroma, sh, s);
}

}  // namespace av1g
