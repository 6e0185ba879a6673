// fitting.cu -- the encoder's fitting cloud on the GPU: PatchFitting::Compute
// with the direct clustering every reference config selects
// (src/patch/patch_fitting.cc:92-136 Compute, :138-236 Clustering, :238-381
// Split; octree_base.cc:102-162).
//
// Host: the octree descent over the GoP's registered patches (Split), which
// ends in clustering cells -- a cell where some octant would hold points of
// only some patches, or one at the threshold height.  A cell's points are
// its patches' points, patch by patch, in input order; its k is the mean
// point count per patch, rounded.
//
// Device: k_kmeans, one to sixteen CTAs per cell: the reference's seeding (a partial
// Fisher-Yates shuffle from the back, drawing rand() % (i + 1)), then up to
// max_iter rounds of exact nearest-centroid assignment (FP32 squared
// distance accumulated x, y, z; the lower centroid index among equal
// distances, as the exact k-d tree the reference is pinned with), centroid
// sums in point order in FP32, an empty cluster replaced by a random point,
// and the mean centroid shift (square roots in double, summed into a float)
// against clustering_err_ths.
//
// Random numbers.  The reference draws from the process-wide rand(); a call
// here gives every GoP its own generator -- glibc's rand() algorithm seeded
// like srand(seed), through random_r -- so a GoP's fitting cloud equals the
// reference's Compute after srand(seed).  A cell's draws are the next ones
// of its GoP's sequence after the cells before it, which consumed k draws
// each plus one per empty cluster.  Empty clusters are rare, so every cell is
// first run with its draws placed as if none occurred; a cell whose position
// in the sequence turns out different (a cell before it had empty clusters),
// or that used up its window, runs again with the right draws.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <new>
#include <numeric>
#include <thread>
#include <vector>

#include "decode_internal.h"
#include "pvvc_gb300.h"

namespace pvvc {
namespace {

struct FitCell {
    uint32_t first;   // first point (into the points' order)
    uint32_t n;       // points
    uint32_t k;       // centroids
    uint32_t out;     // first centroid of the GoP's fitting clouds (output index)
    uint64_t draw;    // this cell's window in the draw array
    uint32_t window;  // draws in the window
    int32_t pad;
};

constexpr int kFitThreads = 512;
constexpr uint32_t kFitSlack = 8;  // extra draws per window for empty clusters
constexpr int kFitTile = 1024;     // centroids staged in shared memory at a time
constexpr int kFitList = 256;      // members of a centroid sorted in shared memory (per warp)

// What the CTAs of a cell's cluster share in global memory.
struct FitCtl {
    double shift[16];  // each CTA's sum of centroid shifts
    uint32_t used;     // draws consumed
    int32_t done, empty;
    int32_t pad;
};

// Barrier over the CTAs of a cluster (their global and shared writes before it
// are visible after it).
template <int CL>
__device__ __forceinline__ void cell_sync() {
    if constexpr (CL == 1) {
        __syncthreads();
    } else {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
    }
}

// sum of v over the block, in thread 0
__device__ __forceinline__ double block_sum(double v, double* s_w) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kFitThreads / 32; ++w) t += s_w[w];
    __syncthreads();
    return t;
}

// k_kmeans: a cluster of CL CTAs per cell of `todo`.  used[c] = draws consumed,
// or window + 1 when the window ran out (the cell must run again).
//
// The reference's sums run over the points in order, in FP32, so each centroid's
// sum is a chain; but the centroids are independent.  An iteration:
//   1. every point's nearest centroid (four points a thread, centroids staged in
//      shared memory) and the centroids' member counts,
//   2. the points' indices bucketed by centroid (scan of the counts, atomics),
//   3. a warp per centroid: its members sorted by index and added in that order,
//   4. empty centroids redrawn in centroid order, the mean shift, the decision.
// The shift's reference value is a float sum in centroid order; a double sum in
// any order decides against the threshold unless it lies within the float sum's
// rounding of it, and only then the chain is added up.
//
// Cells differ: of 1,375 cells of 40 patches over 30 frames the median has 550
// points, the largest 57,500 (1,900 centroids: 110M distances an iteration).
// One CTA each, one thread adding and deciding, took 99 ms, set by the largest.
// With the steps above one CTA a cell takes 25 ms; with clusters for the large
// cells the launches take 2.2, 0.6 and 0.4 ms side by side.  Bound by the largest
// cells' distances (FP32 pipe) and the barriers of the others' iterations.
template <int CL>
__global__ void __launch_bounds__(kFitThreads, 2) k_kmeans(const float* __restrict__ xyz, const uint32_t* __restrict__ order,
                                                        const FitCell* __restrict__ cells,
                                                        const int32_t* __restrict__ todo, const uint32_t* __restrict__ draws,
                                                        float* work, float* cbuf, float* nbuf, uint32_t* cnt, uint32_t* start,
                                                        int32_t* asg, uint32_t* mem, FitCtl* ctls, float err_ths, int max_iter,
                                                        float* __restrict__ out, uint32_t* __restrict__ used,
                                                        int32_t* __restrict__ iters) {
    __shared__ float4 s_ctr[kFitTile];
    __shared__ uint32_t s_list[kFitThreads / 32][kFitList];
    __shared__ double s_w[kFitThreads / 32];
    __shared__ uint32_t s_scan[kFitThreads / 32];
    const int ci = todo[blockIdx.x / CL], rank = blockIdx.x % CL;
    const FitCell c = cells[ci];
    const uint32_t n = c.n, k = c.k;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const uint32_t gtid = rank * kFitThreads + tid, gthreads = CL * kFitThreads;
    if (k == 0) {  // no centroid: the shift is never below the threshold
        if (gtid == 0) {
            used[ci] = 0;
            iters[ci] = max_iter;
        }
        return;
    }
    float* const w = work + 3ull * c.first;
    float* const ctr = cbuf + 3ull * c.first;
    float* const nxt = nbuf + 3ull * c.first;
    uint32_t* const cc = cnt + c.first;
    uint32_t* const st = start + c.first;
    int32_t* const as = asg + c.first;
    uint32_t* const mb = mem + c.first;
    FitCtl* const ctl = ctls + blockIdx.x / CL;
    const uint32_t* const dr = draws + c.draw;
    for (uint32_t i = gtid; i < n; i += gthreads) {
        const float* p = xyz + 3ull * order[c.first + i];
        for (int d = 0; d < 3; ++d) w[3ull * i + d] = p[d];
    }
    for (uint32_t q = gtid; q < k; q += gthreads) cc[q] = 0;
    cell_sync<CL>();
    if (gtid < 32) {
        // seeds (patch_fitting.cc:160-165): for i = n - 1 down, point i swapped
        // with point draw % (i + 1), 32 swaps at a time where no two of them
        // touch the same point, else one after another
        for (uint32_t t0 = 0; t0 < k; t0 += 32) {
            const uint32_t t = t0 + lane, lo = n - min(t0 + 32, k);  // this batch's i: [lo, n - t0)
            const bool on = t < k;
            const uint32_t i = n - 1 - t, j = on ? (t < c.window ? dr[t] : 0u) % (i + 1) : 0u;
            const uint32_t same = __match_any_sync(0xffffffffu, on ? j : 0x80000000u + lane);
            const bool clash = on && (__popc(same) > 1 || (j >= lo && j != i));
            if (!__any_sync(0xffffffffu, clash)) {
                if (on) {
                    float a[3], b[3];
                    for (int d = 0; d < 3; ++d) {
                        a[d] = w[3ull * i + d];
                        b[d] = w[3ull * j + d];
                    }
                    for (int d = 0; d < 3; ++d) {
                        w[3ull * j + d] = a[d];
                        w[3ull * i + d] = b[d];
                        ctr[3ull * t + d] = b[d];
                    }
                }
            } else {
                for (uint32_t u = t0; u < min(t0 + 32, k); ++u) {
                    const uint32_t iu = n - 1 - u, ju = __shfl_sync(0xffffffffu, j, u - t0);
                    if (lane < 3) {
                        const float a = w[3ull * iu + lane], b = w[3ull * ju + lane];
                        w[3ull * ju + lane] = a;
                        w[3ull * iu + lane] = b;
                        ctr[3ull * u + lane] = b;
                    }
                }
            }
            __syncwarp();
        }
        if (lane == 0) {
            ctl->used = k;
            ctl->done = 0;
            ctl->empty = 0;
        }
    }
    cell_sync<CL>();
    int iter = 1;
    for (; iter <= max_iter; ++iter) {
        // 1. nearest centroid of every point (:179-189)
        for (uint32_t j0 = 4 * kFitThreads * rank; j0 < n; j0 += 4 * gthreads) {  // (the same for the whole CTA)
            float px[4], py[4], pz[4], best[4];
            int bi[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t j = min(j0 + u * kFitThreads + tid, n - 1);
                px[u] = w[3ull * j];
                py[u] = w[3ull * j + 1];
                pz[u] = w[3ull * j + 2];
                best[u] = FLT_MAX;
                bi[u] = 0;
            }
            for (uint32_t q0 = 0; q0 < k; q0 += kFitTile) {
                const uint32_t qn = min((uint32_t)kFitTile, k - q0);
                __syncthreads();
                for (uint32_t q = tid; q < qn; q += kFitThreads)
                    s_ctr[q] = make_float4(ctr[3ull * (q0 + q)], ctr[3ull * (q0 + q) + 1], ctr[3ull * (q0 + q) + 2], 0.f);
                __syncthreads();
#pragma unroll 2
                for (uint32_t q = 0; q < qn; ++q) {
                    const float4 s = s_ctr[q];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const float dx = __fsub_rn(s.x, px[u]), dy = __fsub_rn(s.y, py[u]), dz = __fsub_rn(s.z, pz[u]);
                        const float d = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
                        if (d < best[u]) {
                            best[u] = d;
                            bi[u] = (int)(q0 + q);
                        }
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t j = j0 + u * kFitThreads + tid;
                if (j < n) {
                    as[j] = bi[u];
                    atomicAdd(cc + bi[u], 1u);
                }
            }
        }
        cell_sync<CL>();
        // 2. members bucketed by centroid
        if (rank == 0) {
            const uint32_t per = (k + kFitThreads - 1) / kFitThreads, q0 = min(k, tid * per), q1 = min(k, q0 + per);
            uint32_t sum = 0;
            for (uint32_t q = q0; q < q1; ++q) sum += cc[q];
            uint32_t x = sum;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) s_scan[wid] = x;
            __syncthreads();
            uint32_t run = x - sum;
            for (int v = 0; v < wid; ++v) run += s_scan[v];
            for (uint32_t q = q0; q < q1; ++q) {
                st[q] = run;
                run += cc[q];
            }
        }
        cell_sync<CL>();
        for (uint32_t j = gtid; j < n; j += gthreads) mb[atomicAdd(st + as[j], 1u)] = j;
        cell_sync<CL>();
        // 3. sums in point order, FP32 (:184-188), and the means
        for (uint32_t q = rank * (kFitThreads / 32) + wid; q < k; q += CL * (kFitThreads / 32)) {
            const uint32_t m = cc[q], s0 = st[q] - m;  // st: the bucket's end by now
            if (m == 0) {
                if (lane == 0) atomicExch(&ctl->empty, 1);
                continue;
            }
            float sx = 0.f, sy = 0.f, sz = 0.f;
            auto add = [&](uint32_t j, uint32_t count) {  // lanes' points j, in lane order
                const float x = w[3ull * j], y = w[3ull * j + 1], z = w[3ull * j + 2];
                for (uint32_t t = 0; t < count; ++t) {
                    sx = __fadd_rn(sx, __shfl_sync(0xffffffffu, x, t));
                    sy = __fadd_rn(sy, __shfl_sync(0xffffffffu, y, t));
                    sz = __fadd_rn(sz, __shfl_sync(0xffffffffu, z, t));
                }
            };
            if (m <= 32) {
                uint32_t j = (uint32_t)lane < m ? mb[s0 + lane] : 0xFFFFFFFFu;
#pragma unroll
                for (int size = 2; size <= 32; size <<= 1)  // bitonic sort over the lanes
#pragma unroll
                    for (int o = size >> 1; o; o >>= 1) {
                        const uint32_t y = __shfl_xor_sync(0xffffffffu, j, o);
                        const bool up = (lane & size) == 0, low = (lane & o) == 0;
                        j = (up == low) ? min(j, y) : max(j, y);
                    }
                add(min(j, n - 1), m);
            } else if (m <= (uint32_t)kFitList) {
                uint32_t* const l = s_list[wid];
                uint32_t v[kFitList / 32], at[kFitList / 32];
#pragma unroll
                for (int u = 0; u < kFitList / 32; ++u) {
                    const uint32_t e = u * 32 + lane;
                    v[u] = e < m ? mb[s0 + e] : 0xFFFFFFFFu;
                    l[e] = v[u];
                    at[u] = 0;
                }
                __syncwarp();
                for (uint32_t e = 0; e < m; ++e) {
                    const uint32_t y = l[e];
#pragma unroll
                    for (int u = 0; u < kFitList / 32; ++u) at[u] += y < v[u] ? 1u : 0u;
                }
                __syncwarp();
#pragma unroll
                for (int u = 0; u < kFitList / 32; ++u)
                    if ((uint32_t)(u * 32 + lane) < m) l[at[u]] = v[u];
                __syncwarp();
                for (uint32_t e = 0; e < m; e += 32) add(l[min(e + lane, m - 1)], min(32u, m - e));
                __syncwarp();
            } else {  // many members: a scan over all points, in order
                for (uint32_t j0 = 0; j0 < n; j0 += 32) {
                    const uint32_t j = j0 + lane;
                    uint32_t in = __ballot_sync(0xffffffffu, j < n && as[j] == (int32_t)q);
                    if (!in) continue;
                    const uint32_t jj = min(j, n - 1);
                    const float x = w[3ull * jj], y = w[3ull * jj + 1], z = w[3ull * jj + 2];
                    for (; in; in &= in - 1) {
                        const int t = __ffs(in) - 1;
                        sx = __fadd_rn(sx, __shfl_sync(0xffffffffu, x, t));
                        sy = __fadd_rn(sy, __shfl_sync(0xffffffffu, y, t));
                        sz = __fadd_rn(sz, __shfl_sync(0xffffffffu, z, t));
                    }
                }
            }
            if (lane < 3) nxt[3ull * q + lane] = __fdiv_rn(lane == 0 ? sx : lane == 1 ? sy : sz, (float)m);
        }
        cell_sync<CL>();
        // 4. empty centroids drawn at random, in order (:191-204)
        if (__ldcg(&ctl->empty)) {
            if (gtid < 32) {
                uint32_t d = ctl->used;
                for (uint32_t q0 = 0; q0 < k; q0 += 32) {
                    const uint32_t q = q0 + lane;
                    const bool e = q < k && cc[q] == 0;
                    const uint32_t bal = __ballot_sync(0xffffffffu, e);
                    if (e) {
                        const uint32_t t = d + __popc(bal & ((1u << lane) - 1u));
                        const uint32_t j = (t < c.window ? dr[t] : 0u) % n;
                        for (int a = 0; a < 3; ++a) nxt[3ull * q + a] = w[3ull * j + a];
                    }
                    d += __popc(bal);
                }
                __syncwarp();
                if (lane == 0) ctl->used = d;
            }
            cell_sync<CL>();
        }
        // the mean shift (:205-214)
        auto shift = [&](uint32_t q) {
            const double ex = (double)__fsub_rn(nxt[3ull * q], ctr[3ull * q]);
            const double ey = (double)__fsub_rn(nxt[3ull * q + 1], ctr[3ull * q + 1]);
            const double ez = (double)__fsub_rn(nxt[3ull * q + 2], ctr[3ull * q + 2]);
            return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)), __dmul_rn(ez, ez)));
        };
        double mine = 0;
        for (uint32_t q = gtid; q < k; q += gthreads) mine += shift(q);
        mine = block_sum(mine, s_w);
        if (tid == 0) ctl->shift[rank] = mine;
        cell_sync<CL>();
        if (gtid == 0) {
            double total = 0;
            for (int v = 0; v < CL; ++v) total += ctl->shift[v];
            // the float sum is within k roundings of the total (while it stays
            // in range), the mean in two more
            const double mean = total / (double)k, slack = mean * (double)(k + 4) * 0x1p-23 + 0x1p-126;
            bool less;
            if (mean + slack < (double)err_ths && total < 1e38) {
                less = true;
            } else if (mean - slack > (double)err_ths) {
                less = false;
            } else {
                float error = 0.f;
                for (uint32_t q = 0; q < k; ++q) error = (float)__dadd_rn((double)error, shift(q));
                less = __fdiv_rn(error, (float)k) < err_ths;
            }
            ctl->done = less;
            ctl->empty = 0;
        }
        cell_sync<CL>();
        const bool done = __ldcg(&ctl->done) != 0;
        // the new centroids become current (:215-217)
        for (uint32_t i = gtid; i < 3 * k; i += gthreads) ctr[i] = nxt[i];
        for (uint32_t q = gtid; q < k; q += gthreads) cc[q] = 0;
        cell_sync<CL>();
        if (done) break;
    }
    for (uint32_t i = gtid; i < 3 * k; i += gthreads) out[3ull * c.out + i] = ctr[i];
    if (gtid == 0) {
        used[ci] = ctl->used > c.window ? c.window + 1 : ctl->used;
        iters[ci] = iter > max_iter ? max_iter : iter;
    }
}

// Cells of more than kFitWide points run on clusters of 16 CTAs, of more than
// kFitMid on 4, the others on one CTA.  Over the cells above, by (wide, mid):
// (6144, 1536) 2.8 + 0.6 + 0.3 ms for the three launches, (12288, 3072) 2.2 + 0.6 +
// 0.4, (24576, 6144) 2.2 + 1.3 + 0.6; all on one CTA 25 ms.
constexpr uint32_t kFitWide = 12288, kFitMid = 3072;
inline int fit_class(uint32_t n) { return n > kFitWide ? 0 : n > kFitMid ? 1 : 2; }

struct Vec3 {
    float x, y, z;
};

// The octree descent of one GoP (Split, patch_fitting.cc:238-381, with direct
// clustering): cells appended to `cells`, their points' indices to `order`.
struct Splitter {
    const float* xyz;              // the call's points (of its first patch on)
    uint32_t first;                // the first one's index in the caller's array
    const uint32_t* poff;          // patch point ranges (indices in the caller's array)
    int p0, np;                    // the GoP's patches
    int max_height;
    uint32_t *idx, *tmp;           // point indices, patch by patch, partitioned in place; scratch
    uint8_t* oct;
    uint32_t* order;               // the cells' point indices, cell after cell
    uint32_t base;                 // where the GoP's begin in the call's order
    uint32_t nord = 0;
    std::vector<FitCell>* cells;
    uint32_t out_base;             // the GoP's first output centroid
    uint32_t nout = 0;

    void emit(const std::vector<uint32_t>& a, const std::vector<uint32_t>& b) {
        uint64_t total = 0;
        for (int i = 0; i < np; ++i) total += b[i] - a[i];
        FitCell c{};
        c.first = base + nord;
        c.n = (uint32_t)total;
        c.k = (uint32_t)std::max(0.0f, std::round((float)total / (float)np));
        c.out = out_base + nout;
        nout += c.k;
        for (int i = 0; i < np; ++i) {
            std::copy(idx + a[i], idx + b[i], order + nord);
            nord += b[i] - a[i];
        }
        cells->push_back(c);
    }
    void split(const std::vector<uint32_t>& a, const std::vector<uint32_t>& b, Vec3 ctr, Vec3 rng, int h) {
        bool empty = true;
        for (int i = 0; i < np; ++i) empty &= a[i] == b[i];
        if (empty) return;
        if (h >= max_height) {
            emit(a, b);
            return;
        }
        // octant of every point: bit 2 x <= cx, bit 1 y <= cy, bit 0 z <= cz
        std::vector<uint32_t> cnt(8 * (size_t)np, 0);
        for (int i = 0; i < np; ++i)
            for (uint32_t t = a[i]; t < b[i]; ++t) {
                const float* p = xyz + 3ull * idx[t];
                const uint8_t o = (uint8_t)(((p[0] > ctr.x ? 0 : 1) << 2) | ((p[1] > ctr.y ? 0 : 1) << 1) | (p[2] > ctr.z ? 0 : 1));
                oct[t] = o;
                ++cnt[8 * (size_t)i + o];
            }
        // CheckSubSpace: every octant holds points of all patches or of none
        for (int s = 0; s < 8; ++s) {
            int nonempty = 0;
            for (int i = 0; i < np; ++i) nonempty += cnt[8 * (size_t)i + s] ? 1 : 0;
            if (nonempty != 0 && nonempty != np) {
                emit(a, b);
                return;
            }
        }
        // stable partition of each patch's range by octant
        std::vector<uint32_t> ca(8 * (size_t)np), cb(8 * (size_t)np);
        for (int i = 0; i < np; ++i) {
            uint32_t at = a[i];
            uint32_t pos[8];
            for (int s = 0; s < 8; ++s) {
                ca[(size_t)s * np + i] = at;
                pos[s] = at;
                at += cnt[8 * (size_t)i + s];
                cb[(size_t)s * np + i] = at;
            }
            for (uint32_t t = a[i]; t < b[i]; ++t) tmp[pos[oct[t]]++] = idx[t];
            std::copy(tmp + a[i], tmp + b[i], idx + a[i]);
        }
        const Vec3 sr{rng.x / 2.0f, rng.y / 2.0f, rng.z / 2.0f};
        for (int s = 0; s < 8; ++s) {
            // SubSpaceCenter (octree_base.cc:102-120)
            const Vec3 sc{(s & 4) ? ctr.x - sr.x / 2.0f : ctr.x + sr.x / 2.0f, (s & 2) ? ctr.y - sr.y / 2.0f : ctr.y + sr.y / 2.0f,
                          (s & 1) ? ctr.z - sr.z / 2.0f : ctr.z + sr.z / 2.0f};
            std::vector<uint32_t> sa(ca.begin() + (size_t)s * np, ca.begin() + (size_t)(s + 1) * np);
            std::vector<uint32_t> sb(cb.begin() + (size_t)s * np, cb.begin() + (size_t)(s + 1) * np);
            split(sa, sb, sc, sr, h + 1);
        }
    }
    // Compute (patch_fitting.cc:92-136)
    void run(float clustering_ths) {
        float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {FLT_TRUE_MIN, FLT_TRUE_MIN, FLT_TRUE_MIN};
        std::vector<uint32_t> a(np), b(np);
        uint32_t at = 0;
        for (int i = 0; i < np; ++i) {
            a[i] = at;
            for (uint32_t j = poff[p0 + i]; j < poff[p0 + i + 1]; ++j) {
                idx[at++] = j - first;
                for (int d = 0; d < 3; ++d) {
                    const float v = xyz[3ull * (j - first) + d];
                    mn[d] = v < mn[d] ? v : mn[d];
                    mx[d] = v > mx[d] ? v : mx[d];
                }
            }
            b[i] = at;
        }
        const Vec3 ctr{(mx[0] + mn[0]) / 2.0f, (mx[1] + mn[1]) / 2.0f, (mx[2] + mn[2]) / 2.0f};
        const Vec3 rng{mx[0] - mn[0], mx[1] - mn[1], mx[2] - mn[2]};
        const int range_height = (int)std::ceil(std::log2(std::max(rng.x, std::max(rng.y, rng.z))));
        const int ths_height = (int)std::ceil(std::log2(clustering_ths));
        max_height = range_height - ths_height;
        split(a, b, ctr, rng, 0);
    }
};

}  // namespace
}  // namespace pvvc

struct pvvc_fitter {
    pvvc::DevBuf pts, d_order, cells, todo, draws, work, cbuf, nbuf, cnt, asg, out, used, iters, start, mem, ctl;
    pvvc::HostBuf order;           // page-locked: the points' order, uploaded
    std::vector<uint32_t> idx, tmp;  // the descent's
    std::vector<uint8_t> oct;
    pvvc::SideStream side[2];  // the launches of the smaller cells, beside the largest ones'
};

using namespace pvvc;

extern "C" int pvvc_fitter_create(pvvc_fitter** out) {
    if (!out) return PVVC_ERR_ARG;
    *out = new (std::nothrow) pvvc_fitter();
    return *out ? PVVC_OK : PVVC_ERR_NOMEM;
}

extern "C" int pvvc_fitter_destroy(pvvc_fitter* f) {
    if (!f) return PVVC_ERR_ARG;
    delete f;
    return PVVC_OK;
}

extern "C" int pvvc_fitting_clouds(pvvc_fitter* f, int32_t ngops, const int32_t* gop_patch, const uint32_t* patch_off,
                                   const float* xyz, const uint32_t* seeds, float clustering_ths, float clustering_err_ths,
                                   int32_t max_iter, float* out_xyz, uint64_t out_cap, uint64_t* out_off, int32_t* stats,
                                   void* stream) {
    if (!f || ngops < 0 || (ngops && (!gop_patch || !patch_off || !xyz || !seeds || !out_off))) return PVVC_ERR_ARG;
    if (!(clustering_ths > 0.f) || max_iter < 1) return PVVC_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    // ---- the octree descent of every GoP (host threads, one GoP each, the largest first) ----
    for (int g = 0; g < ngops; ++g)
        if (gop_patch[g + 1] - gop_patch[g] < 1 || gop_patch[g] < 0) return PVVC_ERR_ARG;
    // The points go up as the caller has them, their order by cell beside them:
    // k_kmeans gathers.  (Copying every cell's points together, GoP by GoP and
    // then into one array, took 6 of the 13 ms of a call of 2.1M points.)
    uint64_t N = 0;
    for (int g = 0; g < ngops; ++g) N += patch_off[gop_patch[g + 1]] - patch_off[gop_patch[g]];
    if (N > 0xFFFFFFFFull) return PVVC_ERR_CAPACITY;
    const uint32_t p_first = ngops ? patch_off[gop_patch[0]] : 0;
    try {
        f->idx.resize(N);
        f->tmp.resize(N);
        f->oct.resize(N);
    } catch (const std::bad_alloc&) {
        return PVVC_ERR_NOMEM;
    }
    if (N && f->order.ensure(4 * N) != cudaSuccess) return PVVC_ERR_NOMEM;
    std::vector<std::vector<FitCell>> gcells(ngops);
    std::vector<uint32_t> gout(ngops, 0);
    {
        std::vector<int> by_size(ngops);
        std::iota(by_size.begin(), by_size.end(), 0);
        auto points = [&](int g) { return patch_off[gop_patch[g + 1]] - patch_off[gop_patch[g]]; };
        std::stable_sort(by_size.begin(), by_size.end(), [&](int a, int b) { return points(a) > points(b); });
        std::atomic<int> next{0};
        auto work = [&] {
            for (int i; (i = next.fetch_add(1)) < ngops;) {
                const int g = by_size[i];
                Splitter sp;
                sp.xyz = xyz + 3ull * p_first;
                sp.first = p_first;
                sp.poff = patch_off;
                sp.p0 = gop_patch[g];
                sp.np = gop_patch[g + 1] - gop_patch[g];
                sp.base = patch_off[sp.p0] - p_first;
                sp.idx = f->idx.data() + sp.base;
                sp.tmp = f->tmp.data() + sp.base;
                sp.oct = f->oct.data() + sp.base;
                sp.order = static_cast<uint32_t*>(f->order.p) + sp.base;
                sp.cells = &gcells[g];
                sp.out_base = 0;
                sp.run(clustering_ths);
                gout[g] = sp.nout;
            }
        };
        const int nt = (int)std::min<unsigned>(16, std::max(1u, std::thread::hardware_concurrency()));
        std::vector<std::thread> pool;
        for (int t = 1; t < std::min(nt, ngops); ++t) pool.emplace_back(work);
        work();
        for (auto& t : pool) t.join();
    }
    // the GoPs' cells one after another: output ranges and cell lists
    std::vector<FitCell> cells;
    std::vector<uint32_t> gop_first_cell(ngops + 1, 0);
    out_off[0] = 0;
    for (int g = 0; g < ngops; ++g) {
        for (FitCell c : gcells[g]) {
            c.out += (uint32_t)out_off[g];
            cells.push_back(c);
        }
        out_off[g + 1] = out_off[g] + gout[g];
        gop_first_cell[g + 1] = (uint32_t)cells.size();
    }
    const uint64_t total_out = out_off[ngops];
    if (stats) {
        stats[0] = (int32_t)cells.size();
        stats[1] = stats[2] = stats[3] = 0;
    }
    if (total_out > out_cap) return PVVC_ERR_CAPACITY;
    if (cells.empty()) return PVVC_OK;
    if (!out_xyz) return PVVC_ERR_ARG;
    // ---- device buffers ----
    if (f->pts.ensure(12 * N) || f->d_order.ensure(4 * N) || f->cells.ensure(sizeof(FitCell) * cells.size()) || f->todo.ensure(4 * cells.size()) ||
        f->work.ensure(12 * N) || f->cbuf.ensure(12 * N) || f->nbuf.ensure(12 * N) || f->cnt.ensure(4 * N) ||
        f->asg.ensure(4 * N) || f->out.ensure(12 * std::max<uint64_t>(total_out, 1)) || f->used.ensure(4 * cells.size()) ||
        f->iters.ensure(4 * cells.size()) || f->start.ensure(4 * N) || f->mem.ensure(4 * N) ||
        f->ctl.ensure(sizeof(FitCtl) * cells.size()) || f->side[0].ensure() || f->side[1].ensure())
        return PVVC_ERR_NOMEM;
    // An error from here on leaves with nothing of the call under way: its copies
    // read the fitter's host arrays and its launches, on three streams, the device
    // ones, which the next call fills again.
    struct Settle {
        pvvc_fitter* f;
        cudaStream_t s;
        ~Settle() {
            if (!f) return;
            cudaStreamSynchronize(s);
            for (SideStream& sd : f->side) cudaStreamSynchronize(sd.s);
        }
    } settle{f, s};
    if (cudaMemcpyAsync(f->pts.p, xyz + 3ull * p_first, 12 * N, cudaMemcpyHostToDevice, s) != cudaSuccess ||
        cudaMemcpyAsync(f->d_order.p, f->order.p, 4 * N, cudaMemcpyHostToDevice, s) != cudaSuccess)
        return PVVC_ERR_CUDA;
    // ---- draws: every GoP's generator, cells placed by the draws before them ----
    std::vector<uint32_t> extra(cells.size(), 0), window(cells.size(), kFitSlack), used(cells.size(), 0);
    std::vector<int32_t> iters(cells.size(), 0);
    std::vector<uint64_t> placed(cells.size(), ~0ull);  // sequence position each cell last ran with
    std::vector<uint8_t> done(cells.size(), 0);
    int rounds = 0;
    for (;;) {
        // positions in each GoP's sequence, from the extra draws known so far
        std::vector<uint64_t> pos(cells.size());
        std::vector<int32_t> todo;
        uint64_t ndraws = 0;
        std::vector<uint64_t> seq_need(ngops, 0);
        for (int g = 0; g < ngops; ++g) {
            uint64_t at = 0;
            for (uint32_t c = gop_first_cell[g]; c < gop_first_cell[g + 1]; ++c) {
                pos[c] = at;
                at += cells[c].k + extra[c];
                if (!done[c] || placed[c] != pos[c]) todo.push_back((int32_t)c);
                seq_need[g] = std::max<uint64_t>(seq_need[g], pos[c] + cells[c].k + window[c]);
            }
        }
        if (todo.empty()) break;
        // largest cells first, so that each launch starts with its longest work
        std::stable_sort(todo.begin(), todo.end(), [&](int32_t x, int32_t y) { return cells[x].n > cells[y].n; });
        if (++rounds > 64) return PVVC_ERR_CUDA;  // cannot happen: each round settles the first unsettled cell of a GoP
        // the draw windows of the cells to run
        std::vector<uint64_t> seq_base(ngops + 1, 0);
        for (int g = 0; g < ngops; ++g) seq_base[g + 1] = seq_base[g] + seq_need[g];
        std::vector<uint32_t> draws(std::max<uint64_t>(seq_base[ngops], 1));
        for (int g = 0; g < ngops; ++g) {
            struct random_data rd;
            char state[128];
            std::memset(&rd, 0, sizeof(rd));
            if (initstate_r(seeds[g], state, sizeof(state), &rd) != 0) return PVVC_ERR_ARG;
            for (uint64_t t = 0; t < seq_need[g]; ++t) {
                int32_t r = 0;
                random_r(&rd, &r);
                draws[seq_base[g] + t] = (uint32_t)r;
            }
        }
        for (int g = 0; g < ngops; ++g)
            for (uint32_t c = gop_first_cell[g]; c < gop_first_cell[g + 1]; ++c) {
                cells[c].draw = seq_base[g] + pos[c];
                cells[c].window = cells[c].k + window[c];
            }
        ndraws = draws.size();
        if (f->draws.ensure(4 * ndraws) != cudaSuccess ||
            cudaMemcpyAsync(f->draws.p, draws.data(), 4 * ndraws, cudaMemcpyHostToDevice, s) != cudaSuccess ||
            cudaMemcpyAsync(f->cells.p, cells.data(), sizeof(FitCell) * cells.size(), cudaMemcpyHostToDevice, s) != cudaSuccess ||
            cudaMemcpyAsync(f->todo.p, todo.data(), 4 * todo.size(), cudaMemcpyHostToDevice, s) != cudaSuccess)
            return PVVC_ERR_CUDA;
        int first[4] = {0, 0, 0, (int)todo.size()};
        for (int t = 0; t < 3; ++t)
            while (first[t] < (int)todo.size() && fit_class(cells[todo[first[t]]].n) < t) ++first[t];
        for (int t = 0; t < 3; ++t) {
            const int count = first[t + 1] - first[t];
            if (count <= 0) continue;
            cudaStream_t on = s;
            if (t > 0) {
                SideStream& sd = f->side[t - 1];
                if (cudaEventRecord(sd.fork, s) != cudaSuccess || cudaStreamWaitEvent(sd.s, sd.fork, 0) != cudaSuccess)
                    return PVVC_ERR_CUDA;
                on = sd.s;
            }
            const float* a_pts = static_cast<const float*>(f->pts.p);
            const FitCell* a_cells = static_cast<const FitCell*>(f->cells.p);
            const int32_t* a_todo = static_cast<const int32_t*>(f->todo.p) + first[t];
            const uint32_t* a_draws = static_cast<const uint32_t*>(f->draws.p);
            FitCtl* a_ctl = static_cast<FitCtl*>(f->ctl.p) + first[t];
            auto launch = [&](auto kernel, int cl) -> bool {
                cudaLaunchConfig_t cfg{};
                cfg.gridDim = dim3((unsigned)(count * cl));
                cfg.blockDim = dim3(kFitThreads);
                cfg.stream = on;
                cudaLaunchAttribute at[1];
                at[0].id = cudaLaunchAttributeClusterDimension;
                at[0].val.clusterDim.x = (unsigned)cl;
                at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
                cfg.attrs = at;
                cfg.numAttrs = cl > 1 ? 1 : 0;
                if (cl > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
                    return false;
                return cudaLaunchKernelEx(&cfg, kernel, a_pts, static_cast<const uint32_t*>(f->d_order.p), a_cells, a_todo, a_draws, static_cast<float*>(f->work.p),
                                          static_cast<float*>(f->cbuf.p), static_cast<float*>(f->nbuf.p),
                                          static_cast<uint32_t*>(f->cnt.p), static_cast<uint32_t*>(f->start.p),
                                          static_cast<int32_t*>(f->asg.p), static_cast<uint32_t*>(f->mem.p), a_ctl,
                                          clustering_err_ths, max_iter, static_cast<float*>(f->out.p),
                                          static_cast<uint32_t*>(f->used.p), static_cast<int32_t*>(f->iters.p)) == cudaSuccess;
            };
            if (!(t == 0 ? launch(k_kmeans<16>, 16) : t == 1 ? launch(k_kmeans<4>, 4) : launch(k_kmeans<1>, 1)))
                return PVVC_ERR_CUDA;
        }
        for (int t = 1; t < 3; ++t)
            if (first[t + 1] > first[t] && (cudaEventRecord(f->side[t - 1].join, f->side[t - 1].s) != cudaSuccess ||
                                            cudaStreamWaitEvent(s, f->side[t - 1].join, 0) != cudaSuccess))
                return PVVC_ERR_CUDA;
        if (cudaGetLastError() != cudaSuccess ||
            cudaMemcpyAsync(used.data(), f->used.p, 4 * cells.size(), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaMemcpyAsync(iters.data(), f->iters.p, 4 * cells.size(), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            return PVVC_ERR_CUDA;
        for (int32_t c : todo) {
            placed[c] = pos[c];
            if (used[c] > cells[c].window) {  // the window ran out: widen it and run again
                window[c] *= 4;
                done[c] = 0;
                placed[c] = ~0ull;
            } else {
                extra[c] = used[c] - std::min(used[c], cells[c].k);
                done[c] = 1;
            }
        }
    }
    if (cudaMemcpyAsync(out_xyz, f->out.p, 12 * total_out, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return PVVC_ERR_CUDA;
    settle.f = nullptr;
    if (stats) {
        int64_t it = 0, ex = 0;
        for (size_t c = 0; c < cells.size(); ++c) {
            it += iters[c];
            ex += extra[c];
        }
        stats[1] = (int32_t)std::min<int64_t>(it, INT32_MAX);
        stats[2] = (int32_t)ex;
        stats[3] = rounds;
    }
    return PVVC_OK;
}
