// quality_kernels.cu -- the codec's quality measure on the GPU: the symmetric
// nearest-neighbour geometry and Y/U/V errors of two coloured clouds,
// restating common::MSE::Compute (src/registration/registration_base.cc:
// 168-223), from which the decoder reports PSNR (pvvc_decompression.cc:
// 151-171).
//
// Every kernel takes both clouds (blockIdx.y):
//   k_q_bbox    bounding box of a cloud; its last block lays a uniform grid
//               over it (cell edge h, at most qcap(n) cells)
//   k_q_count / k_q_scatter  counting sort of the cloud's points by cell
//               (float4 x, y, z, input index)
//   k_q_sums / k_q_scan  exclusive prefix sum of the cell counts
//   k_q_query   per query point: the exact nearest neighbour in the other
//               cloud; FP32 squared distance accumulated x, y, z; among equal
//               distances the lower input index (the reference's k-d tree
//               leaves that order open); the squared Y/U/V differences of the
//               two points' BT.601 colours (common.h:94-98); per-block sums in
//               double, added by the last block in a fixed order
//
// Two clouds of 800k points: 1.39 ms with a kernel per cloud and step, 0.32 ms now:
// boxes by six atomics a block (2 x 97 -> 12 us), searches that visit the rows of
// cells inside the ball to the best point instead of whole rings (2 x 345 -> 173
// us), the final sums in parallel (2 x 235 us by one warp).  What is left is the
// queries' instructions, some 2,500 a warp, lanes diverging over rows.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstdint>

#include "decode_internal.h"
#include "pvvc_gb300.h"

namespace pvvc {
namespace {

constexpr int kQThreads = 256;
constexpr int kScanPer = 16;                       // cells per thread of a scan block
constexpr int kScanBlock = kQThreads * kScanPer;   // cells per scan block
constexpr uint32_t kQMaxCells = 1u << 24;

struct QGrid {
    float lo[3];
    float h;
    int dim[3];
    int ncells;
    float eps;  // bounds how far rounding can put a point outside its cell's box
};

// what a call zeroes, per cloud: the box (order-preserving codes of -min and
// max), and the counts of finished blocks
struct QZero {
    uint32_t box[6];
    uint32_t done_bbox, done_query;
};

struct QCloud {
    const float* xyz;
    const uint8_t* rgb;
    uint32_t n, cap;
    QGrid* grid;
    QZero* zero;
    uint32_t* cell;    // cell[0] = 0; cell[c + 1]: cell c's count, then its first point, then its end
    uint32_t* totals;  // of the scan blocks
    float4* sorted;
    double* partial;   // 4 sums per block of the cloud's queries
};
struct QPair {
    QCloud c[2];
};

__device__ __forceinline__ uint32_t f2ord(float f) {  // order-preserving float -> unsigned, above 0
    const uint32_t u = __float_as_uint(f);
    return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float ord2f(uint32_t u) { return __uint_as_float(u & 0x80000000u ? u & 0x7FFFFFFFu : ~u); }

// Box of a cloud; its last block derives the grid: about `cap` cells of edge
// h >= 0.5 spread over the box's own shape, grown until the cell count fits.
__global__ void __launch_bounds__(kQThreads) k_q_bbox(QPair pr) {
    __shared__ float s_red[kQThreads / 32][6];
    __shared__ bool s_last;
    const QCloud& c = pr.c[blockIdx.y];
    float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.n; i += gridDim.x * blockDim.x)
        for (int k = 0; k < 3; ++k) {
            const float v = c.xyz[3ull * i + k];
            mn[k] = fminf(mn[k], v);
            mx[k] = fmaxf(mx[k], v);
        }
    for (int o = 16; o; o >>= 1)
        for (int k = 0; k < 3; ++k) {
            mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
            mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
        }
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 3; ++k) {
            s_red[threadIdx.x >> 5][k] = -mn[k];
            s_red[threadIdx.x >> 5][3 + k] = mx[k];
        }
    __syncthreads();
    if (threadIdx.x < 6) {
        float v = s_red[0][threadIdx.x];
        for (int w = 1; w < kQThreads / 32; ++w) v = fmaxf(v, s_red[w][threadIdx.x]);
        atomicMax(&c.zero->box[threadIdx.x], f2ord(v));
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&c.zero->done_bbox, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    __threadfence();
    QGrid q;
    float e[3], ext = 0.f;
    q.eps = 0.f;
    for (int k = 0; k < 3; ++k) {
        const float hi = ord2f(atomicMax(&c.zero->box[3 + k], 0u));
        q.lo[k] = -ord2f(atomicMax(&c.zero->box[k], 0u));
        e[k] = hi - q.lo[k];
        if (!(e[k] >= 0.f) || !(e[k] < 1e30f)) e[k] = 0.f;  // non-finite coordinates: one cell along that axis
        ext = fmaxf(ext, e[k]);
        q.eps = fmaxf(q.eps, 1e-6f * (fabsf(q.lo[k]) + e[k]));
    }
    const float fl = fmaxf(ext / 1024.f, 1e-3f);
    const float vol = fmaxf(e[0], fl) * fmaxf(e[1], fl) * fmaxf(e[2], fl);
    float h = fmaxf(cbrtf(vol / (float)c.cap), 0.5f);
    long long cells = 0;
    for (int guard = 0; guard < 400; ++guard) {
        cells = 1;
        for (int k = 0; k < 3; ++k) cells *= (long long)floorf(e[k] / h) + 1;
        if (cells <= (long long)c.cap) break;
        h *= 1.05f;
    }
    q.h = h;
    for (int k = 0; k < 3; ++k) q.dim[k] = (int)floorf(e[k] / h) + 1;
    if (cells > (long long)c.cap || cells < 1) {  // absurd extents: one cell
        q.h = FLT_MAX;
        q.dim[0] = q.dim[1] = q.dim[2] = 1;
        cells = 1;
    }
    q.ncells = (int)cells;
    *c.grid = q;
}

__device__ __forceinline__ int qcell(const QGrid& g, float v, int k) {
    const int c = (int)floorf(__fdiv_rn(v - g.lo[k], g.h));
    return min(max(c, 0), g.dim[k] - 1);
}
__device__ __forceinline__ uint32_t qcell3(const QGrid& g, float x, float y, float z) {
    return ((uint32_t)qcell(g, z, 2) * g.dim[1] + qcell(g, y, 1)) * g.dim[0] + qcell(g, x, 0);
}

__global__ void __launch_bounds__(kQThreads) k_q_count(QPair pr) {
    const QCloud& c = pr.c[blockIdx.y];
    const QGrid g = *c.grid;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.n; i += gridDim.x * blockDim.x)
        atomicAdd(c.cell + 1 + qcell3(g, c.xyz[3ull * i], c.xyz[3ull * i + 1], c.xyz[3ull * i + 2]), 1u);
}

// sum of v over the block, in every thread
__device__ __forceinline__ uint32_t block_total(uint32_t v, uint32_t* s_w) {
    v = __reduce_add_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t t = 0;
    for (int w = 0; w < kQThreads / 32; ++w) t += s_w[w];
    return t;
}

// total of each scan block's cells
__global__ void __launch_bounds__(kQThreads) k_q_sums(QPair pr) {
    __shared__ uint32_t s_w[kQThreads / 32];
    const QCloud& c = pr.c[blockIdx.y];
    const uint32_t m = (uint32_t)c.grid->ncells, first = blockIdx.x * kScanBlock;
    if (first >= m) return;
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        const uint32_t i = first + k * kQThreads + threadIdx.x;
        if (i < m) sum += c.cell[1 + i];
    }
    sum = block_total(sum, s_w);
    if (threadIdx.x == 0) c.totals[blockIdx.x] = sum;
}

// exclusive scan of the counts: the totals before the block, then its cells,
// kScanPer consecutive ones per thread through shared memory
__global__ void __launch_bounds__(kQThreads) k_q_scan(QPair pr) {
    __shared__ uint32_t s_w[kQThreads / 32], s_v[kScanBlock + kScanBlock / 16];
    const QCloud& c = pr.c[blockIdx.y];
    const uint32_t m = (uint32_t)c.grid->ncells, first = blockIdx.x * kScanBlock;
    if (first >= m) return;
    uint32_t before = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += kQThreads) before += c.totals[b];
    before = block_total(before, s_w);
    auto at = [](uint32_t i) { return i + (i >> 4); };  // a thread's 16 lie in 17 banks' steps
    for (int k = 0; k < kScanPer; ++k) {
        const uint32_t i = k * kQThreads + threadIdx.x;
        s_v[at(i)] = first + i < m ? c.cell[1 + first + i] : 0u;
    }
    __syncthreads();
    uint32_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) sum += s_v[at(threadIdx.x * kScanPer + k)];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) s_w[wid] = x;
    __syncthreads();
    uint32_t run = before + x - sum;
    for (int w = 0; w < wid; ++w) run += s_w[w];
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        uint32_t& v = s_v[at(threadIdx.x * kScanPer + k)];
        const uint32_t t = v;
        v = run;
        run += t;
    }
    __syncthreads();
    for (int k = 0; k < kScanPer; ++k) {
        const uint32_t i = k * kQThreads + threadIdx.x;
        if (first + i < m) c.cell[1 + first + i] = s_v[at(i)];
    }
}

// the points into their cells: cell[c + 1] ends as the end of cell c, which is
// the start of cell c + 1
__global__ void __launch_bounds__(kQThreads) k_q_scatter(QPair pr) {
    const QCloud& c = pr.c[blockIdx.y];
    const QGrid g = *c.grid;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < c.n; i += gridDim.x * blockDim.x) {
        const float x = c.xyz[3ull * i], y = c.xyz[3ull * i + 1], z = c.xyz[3ull * i + 2];
        c.sorted[atomicAdd(c.cell + 1 + qcell3(g, x, y, z), 1u)] = make_float4(x, y, z, __int_as_float((int)i));
    }
}

// BT.601 YUV of an RGB point (ColorYUV(const pcl::PointXYZRGB&), common.h:94-98)
__device__ __forceinline__ void yuv601(const uint8_t* c, float* o) {
    const float r = c[0], g = c[1], b = c[2];
    o[0] = __fadd_rn(__fadd_rn(__fmul_rn(r, 0.299f), __fmul_rn(g, 0.587f)), __fmul_rn(b, 0.114f));
    o[1] = __fadd_rn(__fadd_rn(__fsub_rn(__fmul_rn(r, -0.168736f), __fmul_rn(g, 0.331264f)), __fmul_rn(b, 0.5f)), 128.0f);
    o[2] = __fadd_rn(__fsub_rn(__fsub_rn(__fmul_rn(r, 0.5f), __fmul_rn(g, 0.418688f)), __fmul_rn(b, 0.081312f)), 128.0f);
}

// Four sums over the warp: at each exchange a lane keeps half of its values, so
// six additions instead of twenty; the sums are a butterfly's (16, 8, 4, 2, 1).
// Lane l's result is sum number 2 * (l >> 4) + (l >> 3 & 1).
__device__ __forceinline__ double warp_sums4(const double (&v)[4], int lane) {
    const bool h16 = lane & 16, h8 = lane & 8;
    const double a0 = (h16 ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, h16 ? v[0] : v[2], 16);
    const double a1 = (h16 ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, h16 ? v[1] : v[3], 16);
    double s = (h8 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, h8 ? a0 : a1, 8);
    for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// One thread per query point of cloud blockIdx.y against the other cloud.
__global__ void __launch_bounds__(kQThreads) k_q_query(QPair pr, double* __restrict__ out) {
    __shared__ double s_sum[kQThreads / 32][4];
    __shared__ bool s_last;
    const QCloud& c = pr.c[blockIdx.y];
    const QCloud& t = pr.c[1 - blockIdx.y];
    const uint32_t blocks = (c.n + kQThreads - 1) / kQThreads;
    if (blockIdx.x >= blocks) return;
    const QGrid g = *t.grid;
    const uint32_t* __restrict__ cell = t.cell;
    const float4* __restrict__ sorted = t.sorted;
    double acc[4] = {0, 0, 0, 0};
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (i < c.n) {
        const float x = c.xyz[3ull * i], y = c.xyz[3ull * i + 1], z = c.xyz[3ull * i + 2];
        float best = FLT_MAX;
        int bi = 0x7FFFFFFF;
        auto run = [&](uint32_t row, int x0, int x1) {  // the points of cells [x0, x1] of a row
            const uint32_t e = __ldg(cell + row + x1 + 1);
            for (uint32_t k = __ldg(cell + row + x0); k < e; ++k) {
                const float4 p = __ldg(sorted + k);
                const float ex = __fsub_rn(x, p.x), ey = __fsub_rn(y, p.y), ez = __fsub_rn(z, p.z);
                const float d = __fadd_rn(__fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)), __fmul_rn(ez, ez));
                const int pi = __float_as_int(p.w);
                if (d < best || (d == best && pi < bi)) {
                    best = d;
                    bi = pi;
                }
            }
        };
        const float inv = 1.0f / g.h, pad = 0.001f * g.h + g.eps;
        auto cells = [&](float v, int k) { return min(max((int)floorf((v - g.lo[k]) * inv), 0), g.dim[k] - 1); };
        // Distance from q to cell a's extent along an axis, the ends open; cells
        // are widened by pad (rounding of the cell assignment), and squared bounds
        // keep a margin of 1e-4, so that no point that could win is skipped.
        auto gap = [&](int a, float q, int k) {
            const float lo = g.lo[k] + (float)a * g.h;
            const float d = q < lo ? (a > 0 ? lo - q : 0.f) : (q > lo + g.h && a < g.dim[k] - 1 ? q - (lo + g.h) : 0.f);
            return fmaxf(d - pad, 0.f);
        };
        // a first point from the query's own cell, or boxes of growing size; then
        // the rows of cells inside the ball to the best one
        const int cx = qcell(g, x, 0), cy = qcell(g, y, 1), cz = qcell(g, z, 2);
        run(((uint32_t)cz * g.dim[1] + cy) * g.dim[0], cx, cx);
        float rad = 0.5f * g.h;
        for (bool last = false; !last; rad *= 4.f) {
            const bool bounded = bi != 0x7FFFFFFF;
            if (bounded) rad = sqrtf(best) * 1.0001f;
            const float o = rad + pad;
            const int x0 = cells(x - o, 0), x1 = cells(x + o, 0), y0 = cells(y - o, 1), y1 = cells(y + o, 1),
                      z0 = cells(z - o, 2), z1 = cells(z + o, 2);
            last = bounded || !(rad < FLT_MAX) ||
                   (x0 == 0 && y0 == 0 && z0 == 0 && x1 == g.dim[0] - 1 && y1 == g.dim[1] - 1 && z1 == g.dim[2] - 1);
            // the ball within the query's own cell: done.  (A far outlier makes cells of
            // very many points, which cost twice as much when they were gone through
            // again: 200k points in one, 99 ms, 48 now.)
            if (bounded && x0 == x1 && y0 == y1 && z0 == z1) break;
            for (int zz = z0; zz <= z1; ++zz) {
                const float gz = gap(zz, z, 2), gz2 = gz * gz * 0.9999f;
                if (gz2 > best) continue;
                for (int yy = y0; yy <= y1; ++yy) {
                    const float gy = gap(yy, y, 1);
                    if (gz2 + gy * gy * 0.9999f > best) continue;
                    run(((uint32_t)zz * g.dim[1] + yy) * g.dim[0], x0, x1);
                }
            }
        }
        float qc[3], tc[3];
        yuv601(c.rgb + 3ull * i, qc);
        yuv601(t.rgb + 3ull * (bi != 0x7FFFFFFF ? bi : 0), tc);  // (none: no distance was a number)
        acc[0] = (double)best;
        for (int k = 0; k < 3; ++k) {
            const double e = (double)__fsub_rn(qc[k], tc[k]);
            acc[1 + k] = e * e;
        }
    }
    const double s = warp_sums4(acc, lane);
    if ((lane & 7) == 0) s_sum[wid][2 * (lane >> 4) + (lane >> 3 & 1)] = s;
    __syncthreads();
    if (threadIdx.x < 4) {
        double v = 0;
        for (int w = 0; w < kQThreads / 32; ++w) v += s_sum[w][threadIdx.x];
        c.partial[4ull * blockIdx.x + threadIdx.x] = v;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&c.zero->done_query, 1u) == blocks - 1;
    __syncthreads();
    if (!s_last) return;
    // the last block: out[2k + dir] = the blocks' sums, strided over the threads
    // and then as above (the order does not depend on the launch), / query count
    __threadfence();
    double v[4] = {0, 0, 0, 0};
    for (uint32_t b = threadIdx.x; b < blocks; b += kQThreads)
        for (int k = 0; k < 4; ++k) v[k] += __ldcg(c.partial + 4ull * b + k);
    const double r = warp_sums4(v, lane);
    if ((lane & 7) == 0) s_sum[wid][2 * (lane >> 4) + (lane >> 3 & 1)] = r;
    __syncthreads();
    if (threadIdx.x < 4) {
        double a = 0;
        for (int w = 0; w < kQThreads / 32; ++w) a += s_sum[w][threadIdx.x];
        out[2 * threadIdx.x + blockIdx.y] = a / (double)c.n;
    }
}

// an empty cloud: MSE::Compute sets that side's errors to -1 and returns
// without computing the other (registration_base.cc:168-177)
__global__ void k_q_empty(double* __restrict__ out, int a_empty, int b_empty) {
    if (threadIdx.x < 4) {
        out[2 * threadIdx.x] = a_empty ? -1.0 : 0.0;
        out[2 * threadIdx.x + 1] = b_empty ? -1.0 : 0.0;
    }
}

uint32_t qcap(uint64_t n) {
    const uint64_t c = 8 * n;  // 4, 8, 16 n: 358, 333, 346 us for the clouds above
    return (uint32_t)(c < 64 ? 64 : (c > kQMaxCells ? kQMaxCells : c));
}
uint64_t al(uint64_t v) { return (v + 255) / 256 * 256; }

// The workspace of two clouds: what a call zeroes comes first (both QZero, both
// cell arrays), then the rest.  Returns its size; with ws, the pointers.
struct QLayout {
    uint64_t zeroed, bytes;
};
QLayout qlayout(QPair* pr, const uint64_t n[2], uint8_t* ws) {
    uint64_t o = 0;
    auto take = [&](uint64_t b) {
        const uint64_t r = o;
        o = al(o + b);
        return ws ? ws + r : nullptr;
    };
    QPair dummy;
    QPair& p = pr ? *pr : dummy;
    for (int k = 0; k < 2; ++k) p.c[k].zero = reinterpret_cast<QZero*>(take(sizeof(QZero)));
    for (int k = 0; k < 2; ++k) {
        p.c[k].cap = qcap(n[k]);
        p.c[k].cell = reinterpret_cast<uint32_t*>(take(4 * ((uint64_t)p.c[k].cap + 1)));
    }
    QLayout l;
    l.zeroed = o;
    for (int k = 0; k < 2; ++k) {
        p.c[k].grid = reinterpret_cast<QGrid*>(take(sizeof(QGrid)));
        p.c[k].totals = reinterpret_cast<uint32_t*>(take(4 * ((p.c[k].cap + kScanBlock - 1) / kScanBlock)));
        p.c[k].sorted = reinterpret_cast<float4*>(take(16 * std::max<uint64_t>(n[k], 1)));
        p.c[k].partial = reinterpret_cast<double*>(take(32 * std::max<uint64_t>((n[k] + kQThreads - 1) / kQThreads, 1)));
    }
    l.bytes = o;
    return l;
}

}  // namespace
}  // namespace pvvc

using namespace pvvc;

extern "C" int pvvc_cloud_quality_workspace_size(uint64_t npoints_a, uint64_t npoints_b, uint64_t* bytes) {
    if (!bytes) return PVVC_ERR_ARG;
    const uint64_t n[2] = {npoints_a, npoints_b};
    *bytes = qlayout(nullptr, n, nullptr).bytes;
    return PVVC_OK;
}

extern "C" int pvvc_cloud_quality(uint64_t npoints_a, const float* xyz_a, const uint8_t* rgb_a, uint64_t npoints_b,
                                  const float* xyz_b, const uint8_t* rgb_b, double* mse_out, void* workspace,
                                  uint64_t workspace_bytes, void* stream) {
    if (!mse_out || !workspace || (npoints_a && (!xyz_a || !rgb_a)) || (npoints_b && (!xyz_b || !rgb_b))) return PVVC_ERR_ARG;
    if (npoints_a > 0x7FFFFFFFull || npoints_b > 0x7FFFFFFFull) return PVVC_ERR_ARG;
    if (reinterpret_cast<uintptr_t>(workspace) & 255u) return PVVC_ERR_ARG;
    uint64_t need = 0;
    pvvc_cloud_quality_workspace_size(npoints_a, npoints_b, &need);
    if (workspace_bytes < need) return PVVC_ERR_CAPACITY;
    cudaStream_t s = (cudaStream_t)stream;
    if (npoints_a == 0 || npoints_b == 0) {
        k_q_empty<<<1, 32, 0, s>>>(mse_out, npoints_a == 0, npoints_b == 0);
        return cudaGetLastError() == cudaSuccess ? PVVC_OK : PVVC_ERR_CUDA;
    }
    QPair pr;
    const uint64_t n[2] = {npoints_a, npoints_b};
    const QLayout l = qlayout(&pr, n, static_cast<uint8_t*>(workspace));
    pr.c[0].xyz = xyz_a;
    pr.c[0].rgb = rgb_a;
    pr.c[1].xyz = xyz_b;
    pr.c[1].rgb = rgb_b;
    for (int k = 0; k < 2; ++k) pr.c[k].n = (uint32_t)n[k];
    const uint64_t most = std::max(n[0], n[1]);
    const uint32_t blocks = (uint32_t)((most + kQThreads - 1) / kQThreads);
    const uint32_t passes = std::min<uint32_t>(blocks, 4096);
    const uint32_t boxes = std::min<uint32_t>(blocks, 4 * (uint32_t)sm_count());  // one atomic each
    const uint32_t scans = (std::max(pr.c[0].cap, pr.c[1].cap) + kScanBlock - 1) / kScanBlock;
    if (cudaMemsetAsync(workspace, 0, l.zeroed, s) != cudaSuccess) return PVVC_ERR_CUDA;
    k_q_bbox<<<dim3(boxes, 2), kQThreads, 0, s>>>(pr);
    k_q_count<<<dim3(passes, 2), kQThreads, 0, s>>>(pr);
    k_q_sums<<<dim3(scans, 2), kQThreads, 0, s>>>(pr);
    k_q_scan<<<dim3(scans, 2), kQThreads, 0, s>>>(pr);
    k_q_scatter<<<dim3(passes, 2), kQThreads, 0, s>>>(pr);
    // direction 0: every point of A against B's grid (MSE's .first); 1: B against A
    k_q_query<<<dim3(blocks, 2), kQThreads, 0, s>>>(pr, mse_out);
    return cudaGetLastError() == cudaSuccess ? PVVC_OK : PVVC_ERR_CUDA;
}
