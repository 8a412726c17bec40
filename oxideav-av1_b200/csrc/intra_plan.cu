// intra_plan.cu — host side of the intra wavefront: validation of the jobs
// and the dependency analysis behind one persistent launch (intra.cu).
//
// Walks each frame's TUs in decode order (transform_block_emit,
// src/cdf.rs:32540-32910) and records the areas every TU reads: the row above
// and the column to its left that intra_predict_block_samples gathers
// (cdf.rs:17030-17075, availability from the TU's flags), the co-located luma
// of chroma from luma (cdf.rs:17256-17340) and the window of an intra block
// copy (cdf.rs:19235).  Inside a superblock each TU gets a level one above
// the last writer of every 4x4 cell it reads or writes and the last reader of
// every cell it writes; across superblocks a read of another superblock's
// area orders the two in decode order.  Replaying the levels and the waits
// therefore reproduces the reference's sequential decode sample for sample.
#include <algorithm>
#include <cstring>
#include <string>
#include <unordered_map>
#include <utility>
#include <vector>

#include "av1_spec_tables.h"
#include "host_pool.h"
#include "intra_plan.h"
#include "wedge.cuh"

namespace av1g {

namespace {

constexpr int kW[19] = AV1T_TX_WIDTH_INIT;
constexpr int kH[19] = AV1T_TX_HEIGHT_INIT;

// An area of one plane, inclusive, in that plane's sample coordinates.
struct Rect {
    int p, x0, y0, x1, y1;
};

// A rect's 4x4 cells inside the current superblock (empty when cx1 < cx0 or cy1 < cy0).
struct Cells {
    int base, stride, cx0, cx1, cy0, cy1;
};

// One job's part of the plan.
struct JobPlan {
    const av1g_intra_job* j;
    int pw[3] = {}, ph[3] = {};
    int sb = 64, log2sb = 6, ssx = 0, ssy = 0, sb_cols = 0, sb_rows = 0;
    struct Sb {
        int sbx, sby, first, count;
    };
    std::vector<Sb> sbs;             // in decode order
    std::vector<int> sb_index;       // superblock grid -> decode-order index
    std::vector<int> lvl;            // per TU: its level within its superblock
    std::vector<int> fwl;            // per 4x4 cell of the frame: the level of its last writer
    int fgw[3] = {}, fgh[3] = {}, fbase[3] = {};
    int gw[3] = {}, gh[3] = {}, cbase[3] = {}, ncell = 0;  // cells of one superblock
    int gbase = 0;                   // its first superblock and TU in the batch
    size_t tbase = 0;
};

// A problem of one TU, to be reported for the first such TU of its job.
struct Problem {
    int at = -1;
    const char* before = nullptr;  // "intra job i: <before> k<after>"
    const char* after = nullptr;
};

// The areas a TU reads, inside the plane (the kernel clamps every coordinate
// the same way); returns how many.
int reads_of(const JobPlan& J, const av1g_intra_tu& t, Rect* out) {
    int m = 0;
    const int ssx = J.ssx, ssy = J.ssy;
    const int p = t.plane, W = kW[t.tx_size], H = kH[t.tx_size];
    const int sx = t.x, sy = t.y, mx = J.pw[p] - 1, my = J.ph[p] - 1;
    if (t.mode < 13) {
        const bool ha = (t.flags & AV1G_INTRA_HAVE_ABOVE) && sy > 0;
        const bool hl = (t.flags & AV1G_INTRA_HAVE_LEFT) && sx > 0;
        const bool har = t.flags & AV1G_INTRA_HAVE_ABOVE_RIGHT, hbl = t.flags & AV1G_INTRA_HAVE_BELOW_LEFT;
        if (ha)
            out[m++] = Rect{p, std::min(hl ? sx - 1 : sx, mx), std::min(sy - 1, my),
                            std::min(mx, sx + (har ? 2 * W : W) - 1), std::min(sy - 1, my)};
        if (hl)
            out[m++] = Rect{p, std::min(sx - 1, mx), std::min(ha ? sy - 1 : sy, my), std::min(sx - 1, mx),
                            std::min(my, sy + (hbl ? 2 * H : H) - 1)};
    }
    if (t.mode == AV1G_INTRA_MODE_INTRABC) {
        const int pss_x = p ? ssx : 0, pss_y = p ? ssy : 0;
        const int stx = (sx << 10) + ((2 * t.mv[1]) >> pss_x) * 64 + 32;
        const int sty = (sy << 10) + ((2 * t.mv[0]) >> pss_y) * 64 + 32;
        out[m++] = Rect{p, std::min(std::max((stx >> 10) - 3, 0), mx), std::min(std::max((sty >> 10) - 3, 0), my),
                        std::min(std::max((stx >> 10) + W - 1 + 4, 0), mx),
                        std::min(std::max((sty >> 10) + H - 1 + 4, 0), my)};
    }
    if ((t.flags & AV1G_INTRA_CFL) && p > 0) {
        const int cx = std::max((int)t.max_luma_w - (1 << ssx), 0), cy = std::max((int)t.max_luma_h - (1 << ssy), 0);
        const int y0 = std::min(sy << ssy, cy), y1 = std::min(std::min((sy + H - 1) << ssy, cy) + ssy, J.ph[0] - 1);
        const int x0 = std::min(sx << ssx, cx), x1 = std::min(std::min((sx + W - 1) << ssx, cx) + ssx, J.pw[0] - 1);
        if (y0 <= y1 && x0 <= x1) out[m++] = Rect{0, x0, y0, x1, y1};
    }
    return m;
}

// Checks TUs [k0, k1) of a job, fills their wedge windows and lists the runs of
// TUs of one superblock {superblock key, first TU}; stops at the first problem.
void check_tus(const JobPlan& J, const IntraFrame& F, PlaneDev side[3], uint32_t* wedge_of, int k0, int k1,
               std::vector<std::pair<int, int>>& runs, Problem& bad) {
    const av1g_intra_job& j = *J.j;
    const av1g_frame_header& h = *j.hdr;
    int prev = -1;
    for (int k = k0; k < k1; k++) {
        const av1g_intra_tu& t = j.tus[k];
        const bool res = t.flags & AV1G_INTRA_RESIDUAL;
        const bool fi_ok = !(t.plane == 0 && t.filter_intra_mode < 5) ||
                           (t.tx_size != 4 && t.tx_size != 11 && t.tx_size != 12 && t.tx_size != 17 && t.tx_size != 18);
        if (t.tx_size >= 19 || t.plane >= h.num_planes || !fi_ok ||
            (res && (t.res.tx_size != t.tx_size || t.res.plane != t.plane || t.res.x != t.x || t.res.y != t.y ||
                     t.res.tx_type >= 16 || !j.coeffs))) {
            bad = Problem{k, "TU ", " is malformed"};
            return;
        }
        const int tw = kW[t.tx_size], th = kH[t.tx_size];
        const int pss_x = t.plane ? J.ssx : 0, pss_y = t.plane ? J.ssy : 0;
        const int sbx = (t.x << pss_x) >> J.log2sb, sby = (t.y << pss_y) >> J.log2sb;
        // a TU lies inside its superblock (the superblock's copy holds all it writes)
        if (t.x + tw > ((sbx + 1) << J.log2sb) >> pss_x || t.y + th > ((sby + 1) << J.log2sb) >> pss_y ||
            t.x >= J.pw[t.plane] || t.y >= J.ph[t.plane]) {
            bad = Problem{k, "TU ", " leaves its superblock or the plane"};
            return;
        }
        if (t.interintra) {
            // the intra half of an inter-intra block: an II mode's intra
            // mode (DC, V, H, SMOOTH) over the whole block, then the blend
            static const uint8_t ii_to_intra[4] = {0, 1, 2, 9};
            const av1g_plane& sp = j.interintra_in[t.plane];
            wedge::Orient o{};
            bool ok = t.interintra <= 2 && t.interintra_mode <= 3 && t.mode == ii_to_intra[t.interintra_mode] &&
                      t.filter_intra_mode >= 5 && !(t.flags & AV1G_INTRA_CFL) && sp.data &&
                      sp.width >= J.pw[t.plane] && sp.height >= J.ph[t.plane] &&
                      sp.stride >= J.pw[t.plane] * (F.hbd ? 2 : 1) && !(sp.stride & 15);
            if (ok && t.interintra == 2) ok = wedge::orient(t.mi_size, t.wedge_index, 0, tw, th, pss_x, pss_y, o);
            if (!ok) {
                bad = Problem{k, "inter-intra TU ", " is malformed"};
                return;
            }
            side[t.plane] = PlaneDev{(uint8_t*)sp.data, sp.stride, J.pw[t.plane], J.ph[t.plane]};
            // the device copy of the TU carries the wedge window in
            // palette_map (an inter-intra TU has no palette)
            wedge_of[k] = (uint32_t)o.dir | ((uint32_t)o.xoff << 8) | ((uint32_t)o.yoff << 16) |
                          ((uint32_t)o.invert << 24);
        }
        if (t.mode == AV1G_INTRA_MODE_PALETTE) {
            // predict_palette's checks (cdf.rs:11907-11960)
            const long long last = (long long)t.palette_map + (long long)(th - 1) * t.palette_stride + (tw - 1);
            bool ok = t.palette_size >= 1 && t.palette_size <= 8 && t.palette_stride >= tw && last < j.palette_map_bytes;
            if (ok) {
                uint8_t most = 0;
                for (int r = 0; r < th; r++) {
                    const uint8_t* m = j.palette_maps + t.palette_map + (long long)r * t.palette_stride;
                    for (int c = 0; c < tw; c++) most = std::max(most, m[c]);
                }
                ok = most < t.palette_size;
            }
            if (!ok) {
                bad = Problem{k, "palette TU ", " is malformed"};
                return;
            }
        }
        if (t.mode == AV1G_INTRA_MODE_INTRABC &&
            (std::abs((int)t.mv[0]) >= (1 << 14) || std::abs((int)t.mv[1]) >= (1 << 14))) {
            bad = Problem{k, "intra block copy TU ", " has a motion vector out of range"};
            return;
        }
        const int key = sby * J.sb_cols + sbx;
        if (key != prev) {
            runs.emplace_back(key, k);
            prev = key;
        }
    }
}

// 4x4-cell hazard maps of one superblock, reused from one to the next: the last
// writer's and the last reader's level plus `epoch`; entries of earlier
// superblocks lie below epoch and so count as no constraint.
struct Hazards {
    std::vector<int> hw, hr;
    int epoch = 0;
};

// The cells of an area inside the superblock whose first samples are (ox, oy).
Cells cells_of(const JobPlan& J, const int ox[3], const int oy[3], const Rect& r) {
    const int p = r.p;
    const int x0 = std::max(r.x0 - ox[p], 0), x1 = std::min(r.x1 - ox[p], 4 * J.gw[p] - 1);
    const int y0 = std::max(r.y0 - oy[p], 0), y1 = std::min(r.y1 - oy[p], 4 * J.gh[p] - 1);
    return Cells{J.cbase[p], J.gw[p], x0 >> 2, x1 < x0 ? -1 : x1 >> 2, y0 >> 2, y1 < y0 ? -1 : y1 >> 2};
}

void sb_origin(const JobPlan& J, const JobPlan::Sb& b, int ox[3], int oy[3]) {
    for (int p = 0; p < 3; p++) {
        ox[p] = (b.sbx << J.log2sb) >> (p ? J.ssx : 0);
        oy[p] = (b.sby << J.log2sb) >> (p ? J.ssy : 0);
    }
}

// The levels of superblock q's TUs, and of its cells' last writers; returns
// how many levels it has.  Touches nothing of other superblocks.
int sb_levels(JobPlan& J, int q, Hazards& hz) {
    const JobPlan::Sb& b = J.sbs[q];
    if ((int)hz.hw.size() != J.ncell || hz.epoch > (1 << 30)) {
        hz.hw.assign(J.ncell, -1);
        hz.hr.assign(J.ncell, -1);
        hz.epoch = 0;
    }
    int* const hw = hz.hw.data();
    int* const hr = hz.hr.data();
    const int epoch = hz.epoch;
    int ox[3], oy[3], nlv = 0;
    sb_origin(J, b, ox, oy);
    for (int k = b.first; k < b.first + b.count; k++) {
        const av1g_intra_tu& t = J.j->tus[k];
        Rect rr[4];
        const int nr = reads_of(J, t, rr);
        Cells rc[4];
        int L = 0;
        for (int u = 0; u < nr; u++) {
            const Cells c = rc[u] = cells_of(J, ox, oy, rr[u]);
            for (int cy = c.cy0; cy <= c.cy1; cy++)
                for (int cx = c.cx0; cx <= c.cx1; cx++) L = std::max(L, hw[c.base + cy * c.stride + cx] - epoch + 1);
        }
        const Cells wc = cells_of(J, ox, oy, Rect{t.plane, t.x, t.y, t.x + kW[t.tx_size] - 1, t.y + kH[t.tx_size] - 1});
        for (int cy = wc.cy0; cy <= wc.cy1; cy++)
            for (int cx = wc.cx0; cx <= wc.cx1; cx++) {
                const int c = wc.base + cy * wc.stride + cx;
                L = std::max(L, std::max(hw[c], hr[c]) - epoch + 1);
            }
        for (int u = 0; u < nr; u++) {
            const Cells& c = rc[u];
            for (int cy = c.cy0; cy <= c.cy1; cy++)
                for (int cx = c.cx0; cx <= c.cx1; cx++) {
                    int& v = hr[c.base + cy * c.stride + cx];
                    v = std::max(v, epoch + L);
                }
        }
        for (int cy = wc.cy0; cy <= wc.cy1; cy++)
            for (int cx = wc.cx0; cx <= wc.cx1; cx++) hw[wc.base + cy * wc.stride + cx] = epoch + L;
        J.lvl[k] = L;
        nlv = std::max(nlv, L + 1);
    }
    // the frame-wide writers, from the superblock's own map
    for (int p = 0; p < J.j->hdr->num_planes; p++) {
        const int fx = ox[p] >> 2, fy = oy[p] >> 2;
        const int w = std::min(J.gw[p], J.fgw[p] - fx), hh = std::min(J.gh[p], J.fgh[p] - fy);
        for (int cy = 0; cy < hh; cy++) {
            int* o = J.fwl.data() + J.fbase[p] + (size_t)(fy + cy) * J.fgw[p] + fx;
            const int* w0 = hw + J.cbase[p] + cy * J.gw[p];
            for (int cx = 0; cx < w; cx++) o[cx] = std::max(w0[cx] - epoch, -1);
        }
    }
    hz.epoch += b.count + 1;
    return nlv;
}

// A read of a cell of a later superblock: that superblock's first writer of
// the cell waits for the reader.
struct Pend {
    int owner, cell, sb, level;  // owner: decode-order index; sb: the reader's index in the batch
};

// Superblock q's waits for earlier superblocks {level, superblock, progress},
// once all levels are known.
void sb_waits(const JobPlan& J, int q, std::vector<int3>& waits, std::vector<Pend>& pend) {
    const JobPlan::Sb& b = J.sbs[q];
    const int sb = J.sb;
    int ox[3], oy[3];
    sb_origin(J, b, ox, oy);
    for (int k = b.first; k < b.first + b.count; k++) {
        const av1g_intra_tu& t = J.j->tus[k];
        Rect rr[4];
        const int nr = reads_of(J, t, rr), L = J.lvl[k];
        int3 tw[8];  // this TU's waits, one per superblock
        int ntw = 0;
        for (int u = 0; u < nr; u++) {
            const Rect& r = rr[u];
            const int p = r.p, sw = sb >> (p ? J.ssx : 0), shh = sb >> (p ? J.ssy : 0);
            if (r.x0 >= ox[p] && r.x1 < ox[p] + sw && r.y0 >= oy[p] && r.y1 < oy[p] + shh) continue;
            for (int cy = r.y0 >> 2; cy <= r.y1 >> 2; cy++) {
                const int py = cy << 2;
                const bool row_in = py >= oy[p] && py < oy[p] + shh;
                const int by = (py << (p ? J.ssy : 0)) >> J.log2sb;
                for (int cx = r.x0 >> 2; cx <= r.x1 >> 2; cx++) {
                    const int px = cx << 2;
                    if (row_in && px >= ox[p] && px < ox[p] + sw) continue;
                    const int o = J.sb_index[(size_t)by * J.sb_cols + ((px << (p ? J.ssx : 0)) >> J.log2sb)];
                    if (o < 0) continue;
                    const int fc = J.fbase[p] + cy * J.fgw[p] + cx;
                    if (o < q) {
                        const int need = J.fwl[fc] + 1;
                        if (need <= 0) continue;
                        int a = 0;
                        while (a < ntw && tw[a].y != J.gbase + o) a++;
                        if (a == ntw) {
                            if (ntw == 8) {
                                waits.push_back(int3{L, J.gbase + o, need});
                                continue;
                            }
                            tw[ntw++] = int3{L, J.gbase + o, need};
                        } else {
                            tw[a].z = std::max(tw[a].z, need);
                        }
                    } else {
                        pend.push_back(Pend{o, fc, J.gbase + q, L});
                    }
                }
            }
        }
        waits.insert(waits.end(), tw, tw + ntw);
    }
}

// The waits that reads of later superblocks make: for each such cell, the
// owner's first TU (in decode order) that writes it waits for every reader.
// `pend` is sorted by owner.
void pend_waits(const JobPlan& J, const std::vector<Pend>& pend, std::vector<std::vector<int3>>& waits) {
    std::unordered_map<int, std::vector<const Pend*>> cells;
    for (size_t u = 0; u < pend.size();) {
        const int o = pend[u].owner;
        cells.clear();
        for (; u < pend.size() && pend[u].owner == o; u++) cells[pend[u].cell].push_back(&pend[u]);
        const JobPlan::Sb& b = J.sbs[o];
        for (int k = b.first; k < b.first + b.count && !cells.empty(); k++) {
            const av1g_intra_tu& t = J.j->tus[k];
            const int p = t.plane;
            const int cx1 = std::min((t.x + kW[t.tx_size] - 1) >> 2, J.fgw[p] - 1);
            const int cy1 = std::min((t.y + kH[t.tx_size] - 1) >> 2, J.fgh[p] - 1);
            for (int cy = t.y >> 2; cy <= cy1; cy++)
                for (int cx = t.x >> 2; cx <= cx1; cx++) {
                    auto c = cells.find(J.fbase[p] + cy * J.fgw[p] + cx);
                    if (c == cells.end()) continue;
                    for (const Pend* e : c->second) waits[J.gbase + o].push_back(int3{J.lvl[k], e->sb, e->level + 1});
                    cells.erase(c);
                }
        }
    }
}

// Of a superblock's waits, the strongest per (level, superblock), and only
// those a smaller level does not already imply; in level order.
void reduce_waits(std::vector<int3>& waits) {
    std::sort(waits.begin(), waits.end(), [](const int3& a, const int3& c) {
        return a.y != c.y ? a.y < c.y : (a.x != c.x ? a.x < c.x : a.z > c.z);
    });
    size_t o = 0;
    int cur = -1, best = 0;
    for (size_t u = 0; u < waits.size(); u++) {
        const int3 w = waits[u];
        if (w.y != cur) {
            cur = w.y;
            best = 0;
        }
        if (w.z > best) {
            best = w.z;
            waits[o++] = w;
        }
    }
    waits.resize(o);
    std::sort(waits.begin(), waits.end(), [](const int3& a, const int3& c) { return a.x < c.x; });
}

}  // namespace

// The analysis is cut into parts that helper threads share (host_pool.h): TU
// ranges for the checks, superblocks for the levels and then, with all
// levels known, for the waits and the records.  A 1080p key frame (43,740 TUs)
// took 4.8 ms of host time per call on one thread of a B200 host.
av1g_status intra_plan(const av1g_intra_job* jobs, int n, IntraPlan& plan, std::string& err) {
    plan = IntraPlan{};
    plan.frames.resize(n);
    plan.map_base.assign(n, 0);
    std::vector<JobPlan> J(n);
    size_t total_tus = 0;
    int total_sbs = 0;
    for (int i = 0; i < n; i++) {
        const av1g_intra_job& j = jobs[i];
        if (!j.hdr || !j.quant || j.num_tus < 0 || (j.num_tus > 0 && !j.tus) || (j.sb_size != 64 && j.sb_size != 128) ||
            j.palette_map_bytes < 0 || (j.palette_map_bytes > 0 && !j.palette_maps)) {
            err = "intra job " + std::to_string(i) + ": missing header/quantizer/TUs/maps or superblock size not 64/128";
            return AV1G_EINVAL;
        }
        const av1g_frame_header& h = *j.hdr;
        if (h.bit_depth != 8 && h.bit_depth != 10 && h.bit_depth != 12) {
            err = "intra job " + std::to_string(i) + ": bit depth";
            return AV1G_EINVAL;
        }
        if (h.num_planes != 1 && h.num_planes != 3) {
            err = "intra job " + std::to_string(i) + ": plane count";
            return AV1G_EINVAL;
        }
        IntraFrame& F = plan.frames[i];
        memset(&F, 0, sizeof F);
        F.bd = h.bit_depth;
        F.hbd = h.bit_depth > 8;
        F.q = *j.quant;
        F.coeffs = j.coeffs;
        F.ssx = h.subsampling_x;
        F.ssy = h.subsampling_y;
        F.np = h.num_planes;
        JobPlan& P = J[i];
        P.j = &j;
        P.sb = j.sb_size;
        P.log2sb = P.sb == 128 ? 7 : 6;
        P.ssx = h.subsampling_x;
        P.ssy = h.subsampling_y;
        int nf = 0;
        for (int p = 0; p < h.num_planes; p++) {
            int sx = p ? h.subsampling_x : 0, sy = p ? h.subsampling_y : 0;
            P.pw[p] = (h.mi_cols * 4) >> sx;
            P.ph[p] = (h.mi_rows * 4) >> sy;
            const av1g_plane& pl = j.planes[p];
            if (!pl.data || pl.width < P.pw[p] || pl.height < P.ph[p] || pl.stride < P.pw[p] * (F.hbd ? 2 : 1) ||
                (pl.stride & 15) || ((uintptr_t)pl.data & 15)) {
                err = "intra job " + std::to_string(i) + ": plane " + std::to_string(p);
                return AV1G_EINVAL;
            }
            F.planes[p] = PlaneDev{(uint8_t*)pl.data, pl.stride, P.pw[p], P.ph[p]};
            P.fgw[p] = (P.pw[p] + 3) >> 2;
            P.fgh[p] = (P.ph[p] + 3) >> 2;
            P.fbase[p] = nf;
            nf += P.fgw[p] * P.fgh[p];
        }
        for (int p = 0; p < 3; p++) {
            P.gw[p] = (P.sb >> (p ? P.ssx : 0)) >> 2;
            P.gh[p] = (P.sb >> (p ? P.ssy : 0)) >> 2;
            P.cbase[p] = P.ncell;
            if (p < h.num_planes) P.ncell += P.gw[p] * P.gh[p];
        }
        {
            size_t cb = intra_copy_samples(P.sb, P.sb);
            if (h.num_planes > 1) cb += 2 * (size_t)intra_copy_samples(P.sb >> P.ssx, P.sb >> P.ssy);
            plan.cache_bytes = std::max(plan.cache_bytes, cb * sizeof(uint16_t));
        }
        plan.map_base[i] = plan.maps.size();
        if (j.palette_map_bytes > 0) plan.maps.insert(plan.maps.end(), j.palette_maps, j.palette_maps + j.palette_map_bytes);
        P.sb_cols = (h.mi_cols * 4 + P.sb - 1) >> P.log2sb;
        P.sb_rows = (h.mi_rows * 4 + P.sb - 1) >> P.log2sb;
        P.sb_index.assign((size_t)P.sb_cols * P.sb_rows, -1);
        plan.wedge.resize(total_tus + j.num_tus);
        P.lvl.resize(j.num_tus);
        P.fwl.assign(nf, -1);
        P.tbase = total_tus;
        plan.tu_base.push_back(total_tus);
        total_tus += j.num_tus;

        // --- validation, and the superblocks in decode order ---
        const int parts = parallel_parts(j.num_tus, 2048);
        struct Part {
            std::vector<std::pair<int, int>> runs;
            Problem bad;
            PlaneDev side[3] = {};
        };
        std::vector<Part> part(parts);
        parallel_for(parts, j.num_tus, [&](int u) {
            check_tus(P, F, part[u].side, plan.wedge.data() + P.tbase, (int)((long long)j.num_tus * u / parts),
                      (int)((long long)j.num_tus * (u + 1) / parts), part[u].runs, part[u].bad);
        });
        int prev = -1;
        for (Part& pt : part) {
            for (const auto& r : pt.runs) {
                if (r.first == prev) continue;  // continues across parts
                if (P.sb_index[r.first] >= 0) {
                    err = "intra job " + std::to_string(i) + ": TUs of a superblock are not contiguous in decode order";
                    return AV1G_EINVAL;
                }
                P.sb_index[r.first] = (int)P.sbs.size();
                if (!P.sbs.empty()) P.sbs.back().count = r.second - P.sbs.back().first;
                P.sbs.push_back(JobPlan::Sb{r.first % P.sb_cols, r.first / P.sb_cols, r.second, 0});
                prev = r.first;
            }
            if (pt.bad.at >= 0) {
                err = "intra job " + std::to_string(i) + ": " + pt.bad.before + std::to_string(pt.bad.at) + pt.bad.after;
                return AV1G_EINVAL;
            }
            for (int p = 0; p < 3; p++)
                if (pt.side[p].p) F.side[p] = pt.side[p];
        }
        if (!P.sbs.empty()) P.sbs.back().count = j.num_tus - P.sbs.back().first;
        P.gbase = total_sbs;
        total_sbs += (int)P.sbs.size();
    }
    if (total_sbs == 0) return AV1G_OK;

    // --- levels inside each superblock, then waits between superblocks ---
    std::vector<std::pair<int, int>> where(total_sbs);  // (job, superblock)
    for (int i = 0; i < n; i++)
        for (size_t q = 0; q < J[i].sbs.size(); q++) where[J[i].gbase + q] = {i, (int)q};
    std::vector<int> nlv(total_sbs);
    const int parts = std::min(total_sbs, parallel_parts((long long)total_tus, 1024));
    auto span = [&](int u, int& q0, int& q1) {
        q0 = (int)((long long)total_sbs * u / parts);
        q1 = (int)((long long)total_sbs * (u + 1) / parts);
    };
    parallel_for(parts, (long long)total_tus, [&](int u) {
        Hazards hz;
        int q0, q1;
        span(u, q0, q1);
        for (int q = q0; q < q1; q++) nlv[q] = sb_levels(J[where[q].first], where[q].second, hz);
    });
    std::vector<int> lv_first(total_sbs);
    int lv_total = 0;
    for (int q = 0; q < total_sbs; q++) {
        lv_first[q] = lv_total;
        lv_total += nlv[q] + 1;
    }
    plan.lvtab.resize(lv_total);
    plan.ntus = total_tus;
    plan.order.reset(new uint32_t[total_tus]);
    std::vector<std::vector<int3>> waits(total_sbs);
    std::vector<std::vector<Pend>> pends(parts);
    parallel_for(parts, (long long)total_tus, [&](int u) {
        std::vector<int> bucket;
        int q0, q1;
        span(u, q0, q1);
        for (int g = q0; g < q1; g++) {
            const JobPlan& P = J[where[g].first];
            const int q = where[g].second;
            sb_waits(P, q, waits[g], pends[u]);
            // the TUs by level, a level's small TUs before its large ones (a
            // counting sort on 2 * level + large, stable in decode order)
            const JobPlan::Sb& b = P.sbs[q];
            auto key = [&](int k) {
                const int tx = P.j->tus[k].tx_size;
                return 2 * P.lvl[k] + (kW[tx] * kH[tx] > kIntraSmallPx ? 1 : 0);
            };
            bucket.assign(2 * nlv[g] + 1, 0);
            for (int k = b.first; k < b.first + b.count; k++) bucket[key(k) + 1]++;
            for (int v = 1; v <= 2 * nlv[g]; v++) bucket[v] += bucket[v - 1];
            const int base = (int)P.tbase + b.first;
            for (int L = 0; L < nlv[g]; L++)
                plan.lvtab[lv_first[g] + L] = int2{base + bucket[2 * L], base + bucket[2 * L + 1]};
            plan.lvtab[lv_first[g] + nlv[g]] = int2{base + b.count, base + b.count};
            for (int k = b.first; k < b.first + b.count; k++)
                plan.order[P.tbase + k] = (uint32_t)(base + bucket[key(k)]++);
        }
    });
    for (int i = 0; i < n; i++) {  // reads of superblocks decoded later: none in most streams
        std::vector<Pend> pend;
        for (const auto& v : pends)
            for (const Pend& e : v)
                if (where[e.sb].first == i) pend.push_back(e);
        if (pend.empty()) continue;
        std::stable_sort(pend.begin(), pend.end(), [](const Pend& a, const Pend& b) { return a.owner < b.owner; });
        pend_waits(J[i], pend, waits);
    }
    parallel_for(parts, (long long)total_tus, [&](int u) {
        int q0, q1;
        span(u, q0, q1);
        for (int q = q0; q < q1; q++) reduce_waits(waits[q]);
    });
    // dependency depth (every wait points to a superblock earlier in decode order)
    std::vector<int> depth(total_sbs, 0);
    size_t nwaits = 0;
    for (int q = 0; q < total_sbs; q++) {
        for (const int3& w : waits[q]) depth[q] = std::max(depth[q], depth[w.y] + 1);
        plan.depth = std::max(plan.depth, depth[q] + 1);
        nwaits += waits[q].size();
    }
    // claim order: depth, then frame, then decode order (a counting sort) — a
    // topological order of the waits, so a CTA only ever waits for superblocks
    // claimed earlier
    std::vector<int> start(plan.depth + 1, 0), claim(total_sbs), pos(total_sbs);
    for (int q = 0; q < total_sbs; q++) start[depth[q] + 1]++;
    for (int v = 0; v < plan.depth; v++) {
        plan.width = std::max(plan.width, start[v + 1]);
        start[v + 1] += start[v];
    }
    for (int q = 0; q < total_sbs; q++) {
        pos[q] = start[depth[q]]++;
        claim[pos[q]] = q;
    }
    // the levels some superblock waits for are published (progress z means
    // z levels done: published after level z - 1)
    for (int q = 0; q < total_sbs; q++)
        for (const int3& w : waits[q]) plan.lvtab[lv_first[w.y] + w.z - 1].y |= kLevelPublished;
    plan.items.resize(total_sbs);
    plan.waits.reserve(nwaits);
    for (int c = 0; c < total_sbs; c++) {
        const int q = claim[c];
        const JobPlan& P = J[where[q].first];
        const JobPlan::Sb& b = P.sbs[where[q].second];
        const int first = (int)P.tbase + b.first;
        plan.items[c] = SbItem{where[q].first, lv_first[q], nlv[q], (int)plan.waits.size(), (int)waits[q].size(),
                               b.sbx << P.log2sb, b.sby << P.log2sb, P.log2sb, first, first + b.count};
        for (const int3& w : waits[q]) plan.waits.push_back(int4{w.x, pos[w.y], w.z, 0});
    }
    return AV1G_OK;
}

}  // namespace av1g
