// plane_copy.cu — copies of whole planes, any number of them in one launch.
//
// A finished frame's reference payload goes to its slot and its output, packed, to
// pinned host memory: six planes of one 4:2:0 frame, and a step holds many frames.
// One strided copy per plane took 4.4 us of the enqueuing thread each, more than
// the device took for a small frame's planes (1.6 us to a slot, 3.3 us to the host).
// The descriptors travel as kernel parameters.
//
// Sixteen bytes per thread.  Rows that start on 16-byte boundaries on both sides are
// moved as they are; a packed destination whose rows do not is cut by its own 16-byte
// units, so that the stores to host memory stay whole.
#include "common.cuh"

namespace av1g {

namespace {

constexpr int kCopyThreads = 256;
constexpr int kUnits = 4;             // 16-byte units per thread
constexpr int kPerLaunch = 80;        // descriptors in the 4 KB of parameters

struct Chunk {
    PlaneCopy c[kPerLaunch];
    int first[kPerLaunch];  // the copy's first block
    int n;
};
static_assert(sizeof(Chunk) <= 4096, "parameters of one launch");

__host__ __device__ bool by_rows(const PlaneCopy& P) {
    return (((uintptr_t)P.dst | (unsigned)P.dst_stride) & 15) == 0;
}
__host__ __device__ int units(const PlaneCopy& P) {
    if (by_rows(P)) return (P.row + 15) / 16 * P.height;
    return (int)((((uintptr_t)P.dst & 15) + (size_t)P.row * P.height + 15) / 16);
}

__global__ void __launch_bounds__(kCopyThreads) plane_copy_kernel(const __grid_constant__ Chunk C) {
    int p = 0;
    for (int step = 64; step; step >>= 1)
        if (p + step < C.n && C.first[p + step] <= (int)blockIdx.x) p += step;
    const PlaneCopy P = C.c[p];
    const bool rows = by_rows(P);
    const int n = units(P), u0 = ((int)blockIdx.x - C.first[p]) * (kCopyThreads * kUnits) + threadIdx.x;
#pragma unroll
    for (int k = 0; k < kUnits; k++) {
        const int u = u0 + k * kCopyThreads;
        if (u >= n) break;
        int r, c, bytes;
        uint8_t* d;
        if (rows) {
            const int per = (P.row + 15) / 16;
            r = u / per;
            c = (u - r * per) * 16;
            bytes = min(16, P.row - c);
            d = P.dst + (size_t)r * P.dst_stride + c;
        } else {  // packed: dst_stride == row
            const int at = u * 16 - (int)((uintptr_t)P.dst & 15), lo = max(at, 0), hi = min(at + 16, P.row * P.height);
            r = lo / P.row;
            c = lo - r * P.row;
            bytes = hi - lo;
            d = P.dst + lo;
        }
        const uint8_t* s = P.src + (size_t)r * P.src_stride + c;
        if (bytes == 16 && c + 16 <= P.row) {
            uint4 v;
            const int sh = 8 * (c & 3);
            if (!(c & 15)) {  // source rows start on 16-byte boundaries
                v = *reinterpret_cast<const uint4*>(s);
            } else {
                const uint32_t* w = reinterpret_cast<const uint32_t*>(s - (c & 3));
                const uint32_t e = sh ? w[4] : 0u;
                v = make_uint4(__funnelshift_r(w[0], w[1], sh), __funnelshift_r(w[1], w[2], sh),
                               __funnelshift_r(w[2], w[3], sh), __funnelshift_r(w[3], e, sh));
            }
            *reinterpret_cast<uint4*>(d) = v;
        } else {
            for (int b = 0; b < bytes; b++) {
                d[b] = *s++;
                if (++c == P.row) {
                    c = 0;
                    r++;
                    s = P.src + (size_t)r * P.src_stride;
                }
            }
        }
    }
}

}  // namespace

cudaError_t launch_plane_copies(const PlaneCopy* copies, int n, cudaStream_t s, int* done) {
    *done = 0;
    for (int i = 0; i < n;) {
        Chunk C;
        int blocks = 0;
        C.n = 0;
        for (; i < n && C.n < kPerLaunch; i++) {
            if (copies[i].row <= 0 || copies[i].height <= 0) continue;
            C.c[C.n] = copies[i];
            C.first[C.n++] = blocks;
            blocks += (units(copies[i]) + kCopyThreads * kUnits - 1) / (kCopyThreads * kUnits);
        }
        if (blocks) {
            plane_copy_kernel<<<blocks, kCopyThreads, 0, s>>>(C);
            const cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess) return e;
        }
        *done = i;
    }
    return cudaSuccess;
}

}  // namespace av1g
