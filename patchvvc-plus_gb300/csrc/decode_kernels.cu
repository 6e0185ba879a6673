// decode_kernels.cu -- GB300 (sm_103a) kernels of the patchVVC decode path.
//
//   k_tree  one CTA per intra slice: occupancy bytes -> BFS octree tables
//           (child bases by block scans of popcounts), subtree weights,
//           butterfly coefficients, coefficient offsets, node and leaf
//           centres.  Restates InvertRAHTOctree::MakeTree/AddPoints
//           (src/octree/invert_raht_octree.cc:122-254) level-parallel.
//   k_rlgr  one thread per slice: adaptive run-length / Golomb-Rice decode
//           of 3N symbols with a 64-bit window and count-leading-ones,
//           fused dequantisation, written un-reversed as Y|U|V planes.
//           Restates RLGRDecoder::Decode (src/common/entropy_codec.cc:163-283)
//           and the dequantisation of invert_raht_octree.cc:63-69.
//   k_raht_slice, k_raht_few, k_raht_group  a slice or a group of slices that
//           share a tree: level-synchronous inverse RAHT (7 butterflies
//           per internal node, octree_base.cc:84-100,186-206), fused with the reference-colour add
//           (invert_raht_octree.cc:304-311), YUV->RGB (common.h:154-158) and
//           the rigid transform (pvvc_decompression.cc:141-150).
//
// Bit-exactness with the CPU decoder: every float operation is an explicitly
// rounded intrinsic (__fadd_rn/__fmul_rn/__fdiv_rn/__fsqrt_rn), evaluated in
// the reference's order, so nothing is contracted into an FMA.
#include <cuda_runtime.h>

#include <mutex>

#include <cstdint>

#include "decode_types.h"
#include "pvvc_gb300.h"

namespace pvvc {

// child slots of butterfly i (include/octree/octree.h:79); constexpr so that
// unrolled loops index the per-thread slot arrays with constants (registers)
__device__ __forceinline__ constexpr int pair0(int i) {
    return i == 1 ? 2 : i == 2 ? 4 : i == 3 ? 5 : i == 4 ? 8 : i == 5 ? 9 : i == 6 ? 10 : 11;
}
__device__ __forceinline__ constexpr int pair1(int i) {
    return i == 1 ? 3 : i == 2 ? 6 : i == 3 ? 7 : i == 4 ? 12 : i == 5 ? 13 : i == 6 ? 14 : 15;
}

// ---------------------------------------------------------------------------
// block-wide exclusive scan (T threads, T multiple of 32)
template <int T>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* total, uint32_t* s_warp) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t t = lane < T / 32 ? s_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < T / 32) s_warp[lane] = t;  // inclusive warp totals
    }
    __syncthreads();
    const uint32_t warp_base = wid ? s_warp[wid - 1] : 0;
    *total = s_warp[T / 32 - 1];
    __syncthreads();  // s_warp reused by the next call
    return warp_base + x - v;
}

__device__ __forceinline__ float load_be_float(const uint8_t* p) {
    const uint32_t t = ((uint32_t)p[0] << 24) | ((uint32_t)p[1] << 16) | ((uint32_t)p[2] << 8) | (uint32_t)p[3];
    return __uint_as_float(t);
}

// ---------------------------------------------------------------------------
// k_tree
template <int T>
__global__ void __launch_bounds__(T) k_tree(const SliceWork* __restrict__ work, const uint8_t* __restrict__ payload,
                                            StateView st, int32_t* __restrict__ tstatus) {
    __shared__ uint32_t s_warp[T / 32];
    __shared__ int s_err, s_H, s_lstart[kMaxLevels + 1];
    __shared__ float s_c[3], s_r[kMaxLevels + 1][3];
    const int item = blockIdx.x;
    const SliceWork& w = work[item];
    const int tid = threadIdx.x;
    SlotInfo* info = st.info + w.slot;
    const size_t nb = (size_t)w.slot * st.max_nodes;
    const size_t lb = (size_t)w.slot * st.max_leaves;
    const uint8_t* g = payload + w.geo_off;

    if (!(w.type & PVVC_TYPE_VALID)) {  // SetSlice rejects it before touching state (:25-27)
        if (tid == 0) tstatus[item] = PVVC_ERR_BAD_SLICE;
        return;
    }
    if (tid == 0) {
        int err = PVVC_OK, H = 0;
        info->valid = 0;
        if (w.gsz < 25) {
            err = PVVC_ERR_GEOMETRY;
        } else {
            for (int a = 0; a < 3; ++a) {
                s_c[a] = load_be_float(g + 4 * a);
                s_r[0][a] = load_be_float(g + 12 + 4 * a);
            }
            H = g[24];
            if (H < 1) err = PVVC_ERR_GEOMETRY;
            else if (H > kMaxLevels) err = PVVC_ERR_TREE;
            for (int l = 1; l <= H && l <= kMaxLevels; ++l)
                for (int a = 0; a < 3; ++a) s_r[l][a] = __fdiv_rn(s_r[l - 1][a], 2.0f);
        }
        s_err = err;
        s_H = H;
    }
    __syncthreads();
    if (s_err) {
        if (tid == 0) tstatus[item] = s_err;
        return;
    }
    const int H = s_H;

    // ---- level expansion (MakeTree, invert_raht_octree.cc:158-192) ----
    uint32_t pos = 25, count = 1, nbase = 0, max_w = 0;
    for (int l = 0; l < H - 1; ++l) {
        if (pos + count > w.gsz) { if (tid == 0) s_err = PVVC_ERR_GEOMETRY; }
        else if (nbase + count > (uint32_t)st.max_nodes) { if (tid == 0) s_err = PVVC_ERR_TREE; }
        __syncthreads();
        if (s_err) break;
        if (tid == 0) s_lstart[l] = (int)nbase;
        max_w = max(max_w, count);
        uint32_t running = 0;
        for (uint32_t c0 = 0; c0 < count; c0 += T) {
            const uint32_t j = c0 + tid;
            const uint32_t byte = j < count ? g[pos + j] : 0u;
            uint32_t tot;
            const uint32_t ex = block_excl_scan<T>(__popc(byte), &tot, s_warp);
            if (j < count) {
                st.occ[nb + nbase + j] = (uint8_t)byte;
                st.cbase[nb + nbase + j] = running + ex;
            }
            running += tot;
        }
        pos += count;
        nbase += count;
        count = running;
    }
    if (tid == 0 && !s_err) {
        s_lstart[H - 1] = (int)nbase;
        if (count != w.n) s_err = PVVC_ERR_SIZE;
        else if (count > (uint32_t)st.max_leaves) s_err = PVVC_ERR_TREE;
    }
    __syncthreads();
    if (s_err) {
        if (tid == 0) tstatus[item] = s_err;
        return;
    }
    __threadfence_block();

    // ---- subtree weights, bottom-up (AddPoints, :236-247) ----
    for (int l = H - 2; l >= 0; --l) {
        const int a = s_lstart[l], b = s_lstart[l + 1];
        for (int j = a + tid; j < b; j += T) {
            const uint32_t byte = st.occ[nb + j], cb = st.cbase[nb + j], k = __popc(byte);
            uint32_t tot = k;
            if (l < H - 2) {
                tot = 0;
                for (uint32_t c = 0; c < k; ++c) tot += st.wsum[nb + b + cb + c];
            }
            st.wsum[nb + j] = tot;
        }
        __syncthreads();
    }

    // ---- butterflies and coefficient counts per node ----
    // coefficient offsets need a BFS-order scan over all internal nodes
    uint32_t running = 1;  // coefficient 0 is the DC
    for (int l = 0; l < H - 1; ++l) {
        const int a = s_lstart[l], b = s_lstart[l + 1];
        for (int c0 = a; c0 < b; c0 += T) {
            const int j = c0 + tid;
            uint32_t cnt = 0;
            if (j < b) {
                const uint32_t byte = st.occ[nb + j], cb = st.cbase[nb + j];
                int wt[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) wt[i] = 0;
                uint32_t r = 0;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    if (byte & (0x80u >> c)) {
                        wt[8 + c] = (l == H - 2) ? 1 : (int)st.wsum[nb + b + cb + r];
                        ++r;
                    }
#pragma unroll
                for (int i = 7; i > 0; --i) wt[i] = wt[pair0(i)] + wt[pair1(i)];
                uint32_t m = 0;
#pragma unroll
                for (int i = 1; i < 8; ++i) {
                    const int w0 = wt[pair0(i)], w1 = wt[pair1(i)];
                    float av = 0.f, bv = 0.f;
                    if (w0 != 0 || w1 != 0) {
                        const float base = __fsqrt_rn(__int2float_rn(w0 + w1));
                        av = __fdiv_rn(__fsqrt_rn(__int2float_rn(w0)), base);
                        bv = __fdiv_rn(__fsqrt_rn(__int2float_rn(w1)), base);
                    }
                    if (w0 != 0 && w1 != 0) m |= 1u << i;
                    st.ab[(nb + j) * 7 + (i - 1)] = make_float2(av, bv);
                }
                st.mask[nb + j] = (uint8_t)m;
                cnt = __popc(m);
            }
            uint32_t tot;
            const uint32_t ex = block_excl_scan<T>(cnt, &tot, s_warp);
            if (j < b) st.coff[nb + j] = running + ex;
            running += tot;
        }
    }
    // A well-formed tree codes exactly one coefficient per leaf, and none of its
    // levels is wider than its leaves.  Empty occupancy bytes can break either:
    // reads would go past the planes, and writes past the level buffers, which
    // are sized by the leaves.
    if (running != count || max_w > count) {
        if (tid == 0) tstatus[item] = PVVC_ERR_GEOMETRY;
        return;
    }

    // ---- centres, top-down (SubSpaceCenter, octree_base.cc:102-120) ----
    if (tid == 0) {
        st.ctr[nb * 3 + 0] = s_c[0];
        st.ctr[nb * 3 + 1] = s_c[1];
        st.ctr[nb * 3 + 2] = s_c[2];
        if (H == 1) {
            st.xyz[lb * 3 + 0] = s_c[0];
            st.xyz[lb * 3 + 1] = s_c[1];
            st.xyz[lb * 3 + 2] = s_c[2];
        }
    }
    __syncthreads();
    for (int l = 0; l < H - 1; ++l) {
        const int a = s_lstart[l], b = s_lstart[l + 1];
        // child offset = (range_l / 2) / 2, per axis
        const float ox = __fdiv_rn(s_r[l + 1][0], 2.0f), oy = __fdiv_rn(s_r[l + 1][1], 2.0f), oz = __fdiv_rn(s_r[l + 1][2], 2.0f);
        for (int j = a + tid; j < b; j += T) {
            const uint32_t byte = st.occ[nb + j], cb = st.cbase[nb + j];
            const float cx = st.ctr[(nb + j) * 3 + 0], cy = st.ctr[(nb + j) * 3 + 1], cz = st.ctr[(nb + j) * 3 + 2];
            uint32_t r = 0;
            for (int c = 0; c < 8; ++c) {
                if (!(byte & (0x80u >> c))) continue;
                const float x = (c & 4) ? __fsub_rn(cx, ox) : __fadd_rn(cx, ox);
                const float y = (c & 2) ? __fsub_rn(cy, oy) : __fadd_rn(cy, oy);
                const float z = (c & 1) ? __fsub_rn(cz, oz) : __fadd_rn(cz, oz);
                float* dst = (l < H - 2) ? st.ctr + (nb + b + cb + r) * 3 : st.xyz + (lb + cb + r) * 3;
                dst[0] = x;
                dst[1] = y;
                dst[2] = z;
                ++r;
            }
        }
        __syncthreads();
    }

    if (tid == 0) {
        info->height = H;
        info->nodes = (int)nbase;
        info->leaves = (int)count;
        info->max_width = (int)max_w;
        for (int l = 0; l < H; ++l) info->level_start[l] = s_lstart[l];
        __threadfence();
        info->valid = 1;
        tstatus[item] = PVVC_OK;
    }
}

// ---------------------------------------------------------------------------
// k_rlgr
//
// Bit window: two words `hi:lo` of the stream, complemented, with the next bit
// at bit `o` (0..31, counted from the MSB) of `hi`, and the word after them,
// `nx`, as loaded: the next 32 bits are one funnel shift away, and the load of
// a word is issued when the one before it enters the window, a dozen
// iterations ahead of its use.
//
// Words come from 16-byte payload blocks staged in shared memory: each lane
// owns a ring of kRing blocks (kRing * 16 bytes, aligned to its size), filled
// by cp.async.  The copies are requested at a point the whole warp passes
// together (stage(), every kRlCheck iterations: as many blocks as those can
// take), never from inside a lane's own branch: with 32 slices in a warp, some
// lane needs a block in nearly every iteration, and each such branch cost the
// warp its instructions and a wait for copies that other lanes had just
// requested.  `landed` counts the blocks known to be in shared memory: those
// requested three stage() calls ago.  A lane that may run out of landed words
// before the next stage() -- only after codes longer than 32 bits -- refills its
// ring synchronously.  Blocks past the payload are zero.
constexpr int kRing = 8;             // 16-byte blocks per lane
constexpr uint32_t kRlCheck = 8;     // iterations between stage() calls (4: 5-10% slower, 16: no faster);
                                     // a fast iteration takes at most one word

struct BitReader {
    const uint4* first;  // the slice's first block
    uint32_t nblk;       // blocks holding payload bytes
    uint32_t ring;       // shared address of this lane's ring
    uint32_t hi, lo, nx, o;
    uint32_t wi;         // index of the word after nx
    uint32_t sp;         // blocks requested
    uint32_t s1, s2, s3;  // ... as of the last three stage() calls
    uint32_t landed;     // blocks that have landed (at most kRing of them still in the ring)

    __device__ __forceinline__ static uint32_t inv(uint32_t w) { return ~__byte_perm(w, 0, 0x0123); }
    __device__ __forceinline__ uint32_t slot(uint32_t blk) const { return ring | ((blk << 4) & (kRing * 16 - 1)); }
    __device__ __forceinline__ uint32_t ring_word(uint32_t w) const {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(ring | ((w << 2) & (kRing * 16 - 1))));
        return v;
    }
    __device__ __forceinline__ uint32_t payload_word(uint32_t w) const {  // straight from the payload
        return (w >> 2) < nblk ? __ldg(reinterpret_cast<const uint32_t*>(first) + w) : 0u;
    }
    __device__ __forceinline__ uint32_t base_block() const { return (wi - 1) >> 2; }  // nx's: the first still read
    __device__ __forceinline__ void request() {  // block sp into its slot
        const bool valid = sp < nblk;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(slot(sp)), "l"(first + (valid ? sp : 0u)),
                     "r"(valid ? 16 : 0)
                     : "memory");
        ++sp;
    }
    // every lane of the warp: the copies of three calls ago have landed; the
    // blocks of kRlCheck more iterations requested
    __device__ __forceinline__ void stage(bool active) {
        asm volatile("cp.async.wait_group 2;\n" ::: "memory");
        landed = s3;
        s3 = s2;
        s2 = s1;
#pragma unroll
        for (uint32_t j = 0; j < kRlCheck / 4; ++j)
            if (active && sp < base_block() + kRing) request();
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        s1 = sp;
    }
    // the words up to the next stage() may not all have landed
    __device__ __forceinline__ bool short_of_words() const { return 4 * landed < wi + kRlCheck; }
    __device__ __forceinline__ void refill() {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        sp = max(sp, base_block());
        for (; sp < base_block() + kRing; ++sp) {
            const uint4 b = sp < nblk ? __ldg(first + sp) : make_uint4(0, 0, 0, 0);
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(slot(sp)), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                         : "memory");
        }
        s1 = s2 = s3 = landed = sp;
    }
    // a lane without a slice: it takes part in stage(), and reads words of its
    // own ring that it never uses
    __device__ __forceinline__ void idle(const uint4* ring0) {
        first = nullptr;
        ring = (uint32_t)__cvta_generic_to_shared(ring0);
        nblk = hi = lo = nx = o = wi = sp = s1 = s2 = s3 = landed = 0;
    }
    __device__ __forceinline__ void init(const uint8_t* payload, uint64_t off, uint32_t nbytes, uint4* ring0) {
        first = reinterpret_cast<const uint4*>(payload + (off & ~15ull));
        nblk = (uint32_t)((((uint64_t)(off & 15) + nbytes) + 15) >> 4);
        ring = (uint32_t)__cvta_generic_to_shared(ring0);
        const uint32_t w0 = (uint32_t)(off & 15) >> 2;  // payload words before the slice's first byte
        hi = inv(payload_word(w0));
        lo = inv(payload_word(w0 + 1));
        nx = payload_word(w0 + 2);
        wi = w0 + 3;
        o = (uint32_t)(off & 3) * 8;
        sp = base_block();
        for (int j = 0; j < kRing; ++j) request();
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        s1 = s2 = s3 = landed = sp;
    }
    // the next 32 bits of the stream, complemented
    __device__ __forceinline__ uint32_t peek_inv() const { return __funnelshift_l(lo, hi, o); }
    __device__ __forceinline__ uint32_t peek() const { return ~peek_inv(); }
    // consume n <= 32 bits, the words landed (fast iterations); n = 0: nothing
    __device__ __forceinline__ void advance(uint32_t n) {
        o += n;
        const bool take = o >= 32;
        o &= 31u;
        hi = take ? lo : hi;
        lo = take ? inv(nx) : lo;
        wi += take ? 1u : 0u;
        nx = ring_word(wi - 1);
    }
    // consume n <= 32 bits, the words from the payload (outside the fast iterations)
    __device__ __forceinline__ void advance_slow(uint32_t n) {
        o += n;
        if (o >= 32) {
            hi = lo;
            lo = inv(nx);
            nx = payload_word(wi);
            ++wi;
            o &= 31u;
        }
    }
    // payload bits consumed: the words before hi plus o, minus the bytes
    // before the slice in its first block
    __device__ __forceinline__ int64_t consumed(uint64_t off) const {
        return ((int64_t)wi - 3) * 32 + (int64_t)o - (int64_t)(off & 15) * 8;
    }
    // no copy of this thread's left in flight (before the CTA ends)
    __device__ __forceinline__ void drain() const { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
};

constexpr uint32_t kRlU0 = 3, kRlU1 = 2, kRlD0 = 1, kRlD1 = 1, kRlMaxRP = 32 * 4;

// leading zeros of w; all ones (-1) for w = 0
__device__ __forceinline__ uint32_t lead0(uint32_t w) {
    uint32_t d;
    asm("bfind.shiftamt.u32 %0, %1;" : "=r"(d) : "r"(w));
    return d;
}

// One iteration of a slice's serial chain = an optional zero run (run mode,
// kP >= 4) followed by one Golomb-Rice symbol.  RlFast evaluates it on the
// next 32 bits in one branch-free line that every lane of a warp executes in
// step, whatever mode its slice is in (a lane outside run mode computes an
// empty run): the leading ones of the run code by one bit search, its length
// in closed form, the symbol's ones by a second bit search on the same bits,
// and one advance consumes both.
//
// Run length.  c ones read in run mode from state kP stand for
// sum_{i<c} 2^((kP + 2i) >> 2) zeros (entropy_codec.cc:228-233; kP grows by
// U1 = 2 per one).  With G(t) = (2 | (t & 1)) << (t >> 1), and t = kP >> 1
// before and t2 = t + c after the ones, that sum is G(t2) - G(t); k = t2 >> 1
// remainder bits follow.  Let z be the complemented bits of the zero and the
// remainder read together (k + 1 bits): the remainder is 2^(k+1) - 1 - z, and
// run + 1 = ((4 | (t2 & 1)) << k) - z - G(t).
//
// Symbol.  q ones, a zero and kR bits: with z the complemented zero and
// remainder, u = ((q + 2) << kR) - 1 - z.
//
// The iteration is fast when the codes lie within the 32 bits, kRP is small
// (kR <= 17, so that the symbol is below 2^23, and kRP + q - 1 needs no cap)
// and run + 1 <= left.  32 leading ones make c or q all ones: then r + q is
// either 32 or all ones, and the test fails.  Everything else (longer codes,
// the 32-ones escape, wide symbols) goes to RlSlow, about one lane-iteration
// in 4,000 at q = 8.
//
// kRlCheck iterations run without a branch: a lane whose iteration is not
// fast changes nothing until the check that follows them, so the compiler
// schedules one iteration's stores and adaptation into the next one's chain.
// What bounds the kernels is that chain and the ~80 instructions of an
// iteration on one or two warps per scheduler.  Longest slices of a GoP of 30
// frames of 800k points (8,200 iterations, 15 CTAs): 1.51 ms with the refills
// and the general path inside the loop, 0.96 ms now; windowed larger half of
// the medium tier 1.10 -> 0.59 ms, shorter half 0.75 -> 0.41, short tier
// 0.57 -> 0.34.
constexpr uint32_t kRlFastRP = 72;
struct RlFast {
    uint32_t kPn, kRPn, bits, m1, zz;
    bool ok;
    __device__ __forceinline__ RlFast(uint32_t vi, uint32_t kP, uint32_t kRP, uint32_t left) {
        const bool run = kP >= 4;
        const uint32_t nrun = run ? 0u : 0xFFFFFFFFu;
        const uint32_t c = lead0(vi | nrun);
        const uint32_t kP2 = kP + 2 * c;
        const uint32_t k = kP2 >> 2;
        const uint32_t r = c + k + (nrun + 1u);  // bits of the run code
        const uint32_t w = __funnelshift_lc(0xFFFFFFFFu, vi, r);
        const uint32_t q = lead0(w);
        const uint32_t kR = kRP >> 2, nR = 31u - kR, rq = r + q;
        bits = rq + (kR + 1u);
        const uint32_t G = (2u | ((kP >> 1) & 1u)) << (kP >> 2);
        const uint32_t z0 = __funnelshift_r(__funnelshift_l(0u, vi, c), 0u, ~k);  // >> 31 - k
        m1 = run ? (__funnelshift_l(0u, 4u | ((kP2 >> 1) & 1u), k) - z0 - G) : 1u;
        const uint32_t z1 = __funnelshift_r(__funnelshift_l(0u, w, q), 0u, nR);
        zz = __funnelshift_l(0u, q + 2u, kR) - z1 + nrun;  // u + run
        // outside run mode u = 0 when the zero and the remainder are all zeros
        const bool zero = !run && vi >= __funnelshift_l(0u, 0xFFFFFFFFu, nR);
        ok = rq <= nR && kRP < kRlFastRP && m1 <= left;
        // adaptation (entropy_codec.cc:245-281); here p = u >> kR = q
        kRPn = q ? kRP + q - 1u : max(kRP, 2u) - 2u;
        kPn = zero ? kP2 + kRlU0 : max(kP2, 1u) - 1u;  // D0 = D1 = 1
    }
    // float(Unsign2Sign(zz) * qp): x = ceil(zz / 2) is below 2^23 here (zz <=
    // 15 << 17), so it is the low mantissa of 2^23 + x and needs no conversion;
    // the float product rounds the exact one once, as the conversion of the
    // integer product does.  zz odd is negative (sign: 2^31, or 0 for qp = 0,
    // whose products are +0).
    __device__ __forceinline__ float value(float qp, uint32_t sign) const {
        const float x = __fmul_rn(__fsub_rn(__uint_as_float(0x4B000000u + ((zz + 1u) >> 1)), 8388608.0f), qp);
        return __uint_as_float(__float_as_uint(x) ^ ((zz << 31) & sign));
    }
};

// One iteration read piece by piece, as the reference does.  `left`: symbols
// of the slice still to come.  The run's zeros (at most `left`) in m; a symbol
// follows unless they end the slice or the code is malformed (err).
struct RlSlow {
    uint32_t m = 0;
    long long sym = 0;
    bool has = false;
    int err = PVVC_OK;
    __device__ __forceinline__ RlSlow(BitReader& br, uint32_t& kP, uint32_t& kRP, uint32_t left) {
        const bool run = kP >= 4;
        uint32_t kPr = kP;  // kP after the run's ones
        if (run) {
            // zero run (entropy_codec.cc:226-233): ones, a zero, k remainder bits
            uint64_t m64 = 0;
            uint32_t kk = kP >> 2;
            uint32_t cc;
            int guard = 0;
            do {
                cc = __clz(br.peek_inv());
                for (uint32_t i = 0; i < cc; ++i) {
                    m64 += 1ull << (kk & 31);
                    kPr += kRlU1;
                    kk = kPr >> 2;
                }
                br.advance_slow(cc);
            } while (cc == 32 && ++guard < 64);
            br.advance_slow(1);
            if (kk > 31) {
                err = PVVC_ERR_OVERRUN;
                return;
            }
            m64 += kk ? br.peek() >> (32 - kk) : 0u;
            br.advance_slow(kk);
            m = m64 > left ? left : (uint32_t)m64;
            if (m == left) return;
        }
        // Golomb-Rice symbol (GRRead, entropy_codec.cc:196-205)
        const uint32_t kR = kRP >> 2;
        const uint32_t qq = __clz(br.peek_inv());
        uint64_t uw;
        uint32_t pq;
        if (qq < 32) {
            br.advance_slow(qq + 1);
            uint32_t rr = 0;
            if (kR) {
                rr = kR >= 32 ? br.peek() : (br.peek() >> (32 - kR));
                br.advance_slow(kR >= 32 ? 32u : kR);
            }
            uw = ((uint64_t)qq << kR) | rr;
            pq = qq;
        } else {  // 32 ones: a raw 32-bit value follows
            br.advance_slow(32);
            const uint32_t raw = br.peek();
            br.advance_slow(32);
            uw = raw;
            // p may be far above the kRP cap; any p > kRlMaxRP saturates
            // kRP + p - 1 at the cap (kRP >= 0), so clamp p to kRlMaxRP + 1,
            // not kRlMaxRP (that would leave kRP one short when kRP = 0)
            const uint32_t t2 = kR >= 32 ? 0u : (raw >> kR);
            pq = t2 > kRlMaxRP ? kRlMaxRP + 1 : t2;
        }
        kRP = pq ? min(kRP + pq - 1, kRlMaxRP) : (kRP < 2 ? 0u : kRP - 2);
        kP = (run || uw) ? (kPr ? kPr - kRlD1 : 0u) : kPr + kRlU0;
        const uint64_t z = uw + (uint64_t)run;
        sym = (long long)(z >> 1) ^ -(long long)(z & 1);
        has = true;
    }
};

__device__ __forceinline__ void st_if(float* p, float v, bool c) {  // *p = v where c, without a branch
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p st.global.f32 [%0], %1;\n}\n" ::"l"(p), "f"(v),
                 "r"((uint32_t)c)
                 : "memory");
}
__device__ __forceinline__ void st_shared_if(uint32_t a, float v, bool c) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %2, 0;\n@p st.shared.f32 [%0], %1;\n}\n" ::"r"(a), "f"(v),
                 "r"((uint32_t)c)
                 : "memory");
}

// k_rlgr: one thread per slice.  The coefficient planes are zeroed before the
// launch, so a run of zeros only moves the output position; symbol j of a
// plane goes to coefficient N-1-j (the stream is reversed), which is also the
// number of the plane's symbols still to come after it.
//
// LANES < 32: only the first LANES lanes of each warp decode, so a warp
// executes the union of fewer lanes' paths per iteration.
template <int T, int LANES = 32>
__global__ void __launch_bounds__(T) k_rlgr(const SliceWork* __restrict__ work, const int32_t* __restrict__ order,
                                              int nslices, const uint8_t* __restrict__ payload, float* __restrict__ coef,
                                              int32_t* __restrict__ rstatus) {
    extern __shared__ __align__(128) uint4 s_ring[];  // kRing blocks per thread
    const int lane = threadIdx.x & 31;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    const int t = (g >> 5) * LANES + lane;
    BitReader br;
    br.idle(s_ring + threadIdx.x * kRing);
    uint32_t N = 0, rem = 0;   // symbols of a plane; left in the current plane
    uint32_t qp = 0;
    int plane = 0;
    int32_t item = -1;         // -1: no slice, or done
    uint32_t kP = 0, kRP = 8;
    float* dst = nullptr;      // the current plane
    uint32_t stride = 0;
    if (lane < LANES && t < nslices) {
        const int it = order[t];
        const SliceWork& wk = work[it];
        N = rem = wk.n;
        qp = wk.qp;
        dst = coef + wk.coef_off + wk.coef_lane;
        stride = wk.coef_stride;
        if (N == 0) rstatus[it] = PVVC_OK;
        else br.init(payload, wk.col_off, wk.csz, s_ring + threadIdx.x * kRing);
        if (N != 0) item = it;
    }
    auto finish = [&](int err) {
        const SliceWork& wk = work[item];
        // bits consumed vs the payload (the reference reads past it, which is undefined)
        if (!err && br.consumed(wk.col_off) > 8ll * wk.csz) err = PVVC_ERR_OVERRUN;
        rstatus[item] = err;
        rem = 0;
        item = -1;
    };
    auto next_plane = [&]() {
        if (plane == 2) {
            finish(PVVC_OK);
        } else {
            ++plane;
            dst += (uint64_t)N * stride;
            rem = N;
        }
    };
    const uint32_t sign = qp ? 0x80000000u : 0u;
    const float fqp = (float)qp;
    while (__any_sync(0xffffffffu, rem != 0)) {
        bool ok = true;
#pragma unroll
        for (uint32_t it = 0; it < kRlCheck; ++it) {
            const RlFast f(br.peek_inv(), kP, kRP, rem);
            ok = f.ok;  // a lane that is not stays where it is until the check below
            br.advance(ok ? f.bits : 0u);
            kP = ok ? f.kPn : kP;
            kRP = ok ? f.kRPn : kRP;
            rem -= ok ? f.m1 : 0u;
            st_if(dst + (uint64_t)rem * stride, f.value(fqp, sign), ok && f.zz != 0);
        }
        if (rem == 0 && item >= 0) next_plane();
        // general iterations until the next one is fast (a slice's first
        // coefficients, large ones, take some forty in a row)
        while (!ok && rem != 0) {
            ok = RlFast(br.peek_inv(), kP, kRP, rem).ok;
            if (ok) break;
            const RlSlow w(br, kP, kRP, rem + (uint32_t)(2 - plane) * N);
            if (w.err) {
                finish(w.err);
            } else {
                uint32_t z = w.m;  // zeros, possibly across planes
                while (rem != 0 && z >= rem) {
                    z -= rem;
                    rem = 0;
                    next_plane();
                }
                rem -= z;
                if (w.has) {
                    --rem;
                    if (w.sym) dst[(uint64_t)rem * stride] = __ll2float_rn(w.sym * (long long)(int32_t)qp);
                    if (rem == 0) next_plane();
                }
            }
        }
        br.stage(rem != 0);
        if (rem != 0 && br.short_of_words()) br.refill();
        __syncwarp();
    }
    br.drain();
}

// ---------------------------------------------------------------------------
// k_rlgr_win: RLGR of the slices of one group (the frames of one patch, all
// of the same size N), one warp per group, lane l decoding the group's slice
// l.  The group's coefficients live in its frame-interleaved region: stream
// position s of every lane's slice (plane s / N, coefficient N-1 - s % N)
// is one 128-byte line, lane l's word at offset l.
//
// Instead of scattered 4-byte stores into planes cleared beforehand, each
// lane stages its nonzero symbols in a shared-memory window of WROWS rows
// (row r = stream position r: the 32 lanes' words of that line, their eight
// 16-byte chunks XOR-swizzled by r & 7).  Every kRlCheck iterations the
// warp takes the smallest position any lane can still write
// (__reduce_min_sync); rows below it are final for every lane.  Each full
// unit of 32 final rows is written out with lane l taking row unit + l:
// eight 16-byte loads of its row (conflict-free thanks to the swizzle), eight
// 16-byte stores of the whole line, zeros included, and the row cleared.  A
// lane whose next symbol lands beyond the window keeps it pending and pauses
// until the window reaches it.  So the planes need no clear, every line is
// written once, in full, and no partially written line ever leaves L2.
//
// The decode loop is k_rlgr's with linear stream positions: the common path
// also takes runs that cross a plane boundary.  Every round of the loop
// either consumes a symbol in some lane or moves the window forward (a
// paused lane's position is at least WROWS rows ahead of the window, so the
// minimum has passed a whole unit), so the loop ends after at most 3N rounds
// per lane plus one flush per unit of rows.
constexpr uint32_t kWinUnit = 32;        // rows written out together (one per lane)
constexpr int kWinRows = 64;             // window rows (8 KB per warp)

// shared memory of a windowed CTA: rings and windows, at least 16 KB (with
// the 1 KB the SM keeps per CTA, more than the 15 KB a long per-slice CTA's
// SM has left)
constexpr int kWinMinSmem = 16 * 1024;
__host__ __device__ constexpr int win_smem(int warps, int rows) {
    return warps * (32 * kRing * 16 + rows * 32 * 4) > kWinMinSmem ? warps * (32 * kRing * 16 + rows * 32 * 4)
                                                                   : kWinMinSmem;
}

template <int WARPS, int WROWS>
__global__ void __launch_bounds__(32 * WARPS) k_rlgr_win(const SliceWork* __restrict__ work,
                                                         const GroupDesc* __restrict__ groups, int ngroups,
                                                         const int32_t* __restrict__ items,
                                                         const uint8_t* __restrict__ payload, float* __restrict__ coef,
                                                         int32_t* __restrict__ rstatus) {
    static_assert((WROWS & (WROWS - 1)) == 0 && WROWS >= 2 * (int)kWinUnit, "window rows: a power of two");
    extern __shared__ __align__(128) uint4 s_dyn[];  // [blockDim][kRing] payload blocks, then [WARPS][WROWS][32] floats
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int gi = blockIdx.x * WARPS + wid;
    if (gi >= ngroups) return;  // the whole warp
    float* const win = reinterpret_cast<float*>(s_dyn + kRing * blockDim.x) + (size_t)wid * WROWS * 32;
    // word of (row r, lane) in the window: chunk (lane / 4) ^ (r & 7), word lane % 4
    auto slot = [&](uint32_t r) { return ((r & (WROWS - 1)) << 5) + ((((uint32_t)lane >> 2) ^ (r & 7u)) << 2) + (lane & 3); };
    const GroupDesc G = groups[gi];
    const int item0 = items[G.first];
    const uint32_t N = work[item0].n;
    const uint32_t total = 3u * N;
    const uint64_t region = work[item0].coef_off;
    const int item = lane < G.count ? items[G.first + lane] : -1;
    for (int i = lane; i < WROWS * 8; i += 32) reinterpret_cast<float4*>(win)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncwarp();  // rows are cleared by all lanes, then written by their owners
    BitReader br;
    br.idle(s_dyn + threadIdx.x * kRing);
    bool live = false, pend = false;
    uint32_t qp = 0;
    uint32_t s = total;             // stream position of this lane's next symbol (total: done)
    if (item >= 0) {
        const SliceWork& wk = work[item];
        if (wk.n != N) {
            rstatus[item] = PVVC_ERR_SIZE;  // the planner keeps such slices out of window groups
        } else if (N == 0) {
            rstatus[item] = PVVC_OK;
        } else {
            qp = wk.qp;
            br.init(payload, wk.col_off, wk.csz, s_dyn + threadIdx.x * kRing);
            s = 0;
            live = true;
        }
    }
    auto finish = [&](int err) {
        const SliceWork& wk = work[item];
        // bits consumed vs the payload (the reference reads past it, which is undefined)
        if (!err && br.consumed(wk.col_off) > 8ll * wk.csz) err = PVVC_ERR_OVERRUN;
        rstatus[item] = err;
        s = total;
        live = false;
    };
    const uint32_t sign = qp ? 0x80000000u : 0u;
    const float fqp = (float)qp;
    const uint32_t win0 = (uint32_t)__cvta_generic_to_shared(win);
    uint32_t kP = 0, kRP = 8;
    uint32_t pend_q = 0;            // a pending symbol's position and value
    float pend_v = 0.f;
    uint32_t base = 0;              // rows below `base` are written out (warp-uniform)
    uint32_t bp = 0, bc = N - 1;    // plane and coefficient index of row `base`
    for (;;) {
        // rows this lane may fill before the next check: to the end of the
        // slice or of the window, none with a symbol pending
        const uint32_t lim = min(total, base + (uint32_t)WROWS);
        uint32_t room = pend || s >= lim ? 0u : lim - s;
        const uint32_t end = s + room;
        bool ok = true;
#pragma unroll
        for (uint32_t it = 0; it < kRlCheck; ++it) {
            const RlFast f(br.peek_inv(), kP, kRP, room);
            ok = f.ok;  // a lane that is not stays where it is until the check below
            br.advance(ok ? f.bits : 0u);
            kP = ok ? f.kPn : kP;
            kRP = ok ? f.kRPn : kRP;
            room -= ok ? f.m1 : 0u;
            st_shared_if(win0 + 4u * slot(end - room - 1u), f.value(fqp, sign), ok && f.zz != 0);
        }
        s = end - room;
        while (!ok && s < total && !pend) {
            // a symbol beyond the window (it stays pending), or general
            // iterations until the next one is fast
            float val = 0.f;
            bool has = false;
            const RlFast f(br.peek_inv(), kP, kRP, total - s);
            ok = f.ok;
            if (ok) {
                if (s + f.m1 <= lim) break;
                br.advance_slow(f.bits);
                kP = f.kPn;
                kRP = f.kRPn;
                s += f.m1;
                has = f.zz != 0;
                val = f.value(fqp, sign);
            } else {
                const RlSlow w(br, kP, kRP, total - s);
                if (w.err) {
                    finish(w.err);
                } else {
                    s += w.m + (uint32_t)w.has;
                    has = w.sym != 0;
                    val = __ll2float_rn(w.sym * (long long)(int32_t)qp);
                }
            }
            if (has) {
                if (s - 1u - base < (uint32_t)WROWS) {
                    win[slot(s - 1u)] = val;
                } else {
                    pend = true;
                    pend_q = s - 1u;
                    pend_v = val;
                }
            }
        }
        if (live && s >= total) finish(PVVC_OK);
        br.stage(live);
        if (live && br.short_of_words()) br.refill();
        __syncwarp();
        // ---- the window (warp-uniform) ----
        const uint32_t lb = pend ? pend_q : s;  // this lane writes no row below lb
        const uint32_t mn = __reduce_min_sync(0xffffffffu, lb);
        if (mn - base < kWinUnit && mn < total) continue;
        // write out whole units of final rows (and at the end the last,
        // partial one); rows from base + WROWS on were never staged: zeros
        const uint32_t top = base + WROWS;
        const uint32_t stop = mn == total ? total : base + (mn - base) / kWinUnit * kWinUnit;
        __syncwarp();  // every lane's staged words are visible to the row's owner
        while (base < stop) {
            const uint32_t r = base + (uint32_t)lane;  // this lane's row
            if (r < stop) {
                // its plane and coefficient, from row base's: lane rows down
                uint32_t p = bp, c = bc;
                uint32_t d = (uint32_t)lane;
                while (d > c) {  // past the plane's coefficient 0: to the top of the next
                    d -= c + 1;
                    c = N - 1;
                    ++p;
                }
                c -= d;
                float4* dst = reinterpret_cast<float4*>(coef + region + (((uint64_t)p * N + c) << 5));
                if (r < top) {
                    float4* row = reinterpret_cast<float4*>(win + ((r & (WROWS - 1)) << 5));
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) {
                        const uint32_t pj = j ^ (r & 7u);
                        dst[j] = row[pj];
                        row[pj] = make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) dst[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
            // row base += one unit (warp-uniform)
            uint32_t d = kWinUnit;
            while (d > bc) {
                d -= bc + 1;
                bc = N - 1;
                ++bp;
            }
            bc -= d;
            base += kWinUnit;
        }
        base = stop;
        __syncwarp();  // cleared rows before their owners' next writes
        if (pend && pend_q - base < (uint32_t)WROWS) {
            win[slot(pend_q)] = pend_v;
            pend = false;
        }
        if (mn == total) break;
    }
    br.drain();  // a lane that finished last has copies of its last two stage() calls in flight
}

// ---------------------------------------------------------------------------
// k_raht
struct OutPtrs {
    float* xyz;
    uint8_t* rgb;
    float* p24;
    int32_t* status;  // caller's status, indexed by SliceWork::orig (may be null)
};

// std::round (half away from zero), clamped to [0, 255].  Clamping first
// commutes with the rounding (it is monotone and 0 and 255 are integers);
// for a clamped c >= 0, round(c) = floor(c + 0.5), and the sum rounded
// toward -inf keeps that floor exact, since every integer is a float.  NaN
// clamps to 0, as fmaxf(roundf(NaN), 0) does.
__device__ __forceinline__ uint8_t to_u8(float v) {
    const float c = fminf(fmaxf(v, 0.0f), 255.0f);
    return (uint8_t)__float2uint_rd(__fadd_rd(c, 0.5f));
}

// one leaf: reference add / store, YUV->RGB, transform (rows m), output
__device__ __forceinline__ void emit_leaf(const float* m, uint64_t out_off, bool white, const StateView& st, size_t lb,
                                          uint32_t leaf, float y, float u, float v, bool predict, const OutPtrs& o) {
    float* ref = st.ref + (lb + leaf) * 3;
    if (predict) {
        y = __fadd_rn(y, ref[0]);
        u = __fadd_rn(u, ref[1]);
        v = __fadd_rn(v, ref[2]);
    } else {
        ref[0] = y;
        ref[1] = u;
        ref[2] = v;
    }
    const float* p = st.xyz + (lb + leaf) * 3;
    const float x0 = p[0], y0 = p[1], z0 = p[2];
    const float X = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(x0, m[0]), __fmul_rn(y0, m[1])), __fmul_rn(z0, m[2])), m[3]);
    const float Y = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(x0, m[4]), __fmul_rn(y0, m[5])), __fmul_rn(z0, m[6])), m[7]);
    const float Z = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(x0, m[8]), __fmul_rn(y0, m[9])), __fmul_rn(z0, m[10])), m[11]);
    const float du = __fsub_rn(u, 128.0f), dv = __fsub_rn(v, 128.0f);
    const float R = __fadd_rn(y, __fmul_rn(1.4020f, dv));
    const float G = __fsub_rn(__fsub_rn(y, __fmul_rn(0.3441f, du)), __fmul_rn(0.7141f, dv));
    const float B = __fadd_rn(y, __fmul_rn(1.7720f, du));
    const uint64_t oi = out_off + leaf;
    if (o.xyz) {
        o.xyz[oi * 3 + 0] = X;
        o.xyz[oi * 3 + 1] = Y;
        o.xyz[oi * 3 + 2] = Z;
    }
    if (o.rgb) {
        o.rgb[oi * 3 + 0] = to_u8(R);
        o.rgb[oi * 3 + 1] = to_u8(G);
        o.rgb[oi * 3 + 2] = to_u8(B);
    }
    if (o.p24) {  // CUDA2OpenGL.cu:44-58: unrounded /255, patches under 10 points white
        float* q = o.p24 + oi * 6;
        q[0] = X;
        q[1] = Y;
        q[2] = Z;
        q[3] = white ? 1.0f : __fdiv_rn(R, 255.0f);
        q[4] = white ? 1.0f : __fdiv_rn(G, 255.0f);
        q[5] = white ? 1.0f : __fdiv_rn(B, 255.0f);
    }
}

// Inverse hierarchical transform of one internal node (octree_base.cc:84-100):
// the node's DC `g` and its coded coefficients -> the 8 child slots (absent
// children's slots hold values nobody reads).
__device__ __forceinline__ void inverse_node(const StateView& st, size_t node, const float* __restrict__ cy,
                                             const float* __restrict__ cu, const float* __restrict__ cv, float gy, float gu,
                                             float gv, float (&oy)[8], float (&ou)[8], float (&ov)[8]) {
    const uint32_t m = st.mask[node];
    uint32_t ci = st.coff[node];
    const float2* ab = st.ab + node * 7;
    float sy[8], su[8], sv[8];  // slots 1..7 (index 0 unused)
    sy[1] = gy;
    su[1] = gu;
    sv[1] = gv;
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        const float2 t = ab[i - 1];
        float hy = 0.f, hu = 0.f, hv = 0.f;
        if (m & (1u << i)) {
            hy = cy[ci];
            hu = cu[ci];
            hv = cv[ci];
            ++ci;
        }
        const float ay = sy[i], au = su[i], av = sv[i];
        const float nbv = -t.y;
        // [G;H] = [[a,-b],[b,a]] [g;h]   (InvertHaarTransform, octree_base.cc:186-206)
        const float Gy = __fadd_rn(__fmul_rn(ay, t.x), __fmul_rn(hy, nbv));
        const float Gu = __fadd_rn(__fmul_rn(au, t.x), __fmul_rn(hu, nbv));
        const float Gv = __fadd_rn(__fmul_rn(av, t.x), __fmul_rn(hv, nbv));
        const float Hy = __fadd_rn(__fmul_rn(ay, t.y), __fmul_rn(hy, t.x));
        const float Hu = __fadd_rn(__fmul_rn(au, t.y), __fmul_rn(hu, t.x));
        const float Hv = __fadd_rn(__fmul_rn(av, t.y), __fmul_rn(hv, t.x));
        if (pair0(i) < 8) {
            sy[pair0(i)] = Gy; su[pair0(i)] = Gu; sv[pair0(i)] = Gv;
            sy[pair1(i)] = Hy; su[pair1(i)] = Hu; sv[pair1(i)] = Hv;
        } else {
            oy[pair0(i) - 8] = Gy; ou[pair0(i) - 8] = Gu; ov[pair0(i) - 8] = Gv;
            oy[pair1(i) - 8] = Hy; ou[pair1(i) - 8] = Hu; ov[pair1(i) - 8] = Hv;
        }
    }
}

// Status of one slice before its inverse RAHT.  Priority: slice type, then
// the tree (intra) or the reference (predictive), then the colour stream.
__device__ __forceinline__ int slice_status(const SliceWork& w, int item, const StateView& st, const int32_t* tstatus,
                                            const int32_t* rstatus) {
    const bool predict = (w.type & PVVC_TYPE_PREDICT) != 0;
    int err = PVVC_OK;
    if (!(w.type & PVVC_TYPE_VALID)) err = PVVC_ERR_BAD_SLICE;
    else if (!predict) err = tstatus[item];
    if (!err) {
        const SlotInfo* si = st.info + w.slot;
        if (!si->valid) err = PVVC_ERR_NO_REFERENCE;
        else if ((uint32_t)si->leaves != w.n) err = PVVC_ERR_SIZE;
    }
    if (!err) err = rstatus[item];
    return err;
}

// k_raht_slice: one CTA per slice, level-synchronous over all internal levels
// with the level signal in shared memory (global fallback for wide levels).
// Used for slices that share their tree with few others in the batch.
template <int T>
__global__ void __launch_bounds__(T) k_raht_slice(const SliceWork* __restrict__ work, const int32_t* __restrict__ list,
                                                  StateView st, const float* __restrict__ coef, float* __restrict__ fallback,
                                                  const int32_t* __restrict__ tstatus, const int32_t* __restrict__ rstatus,
                                                  int32_t* __restrict__ fstatus, OutPtrs o, int wcap) {
    extern __shared__ float s_g[];  // [2][wcap][3]
    __shared__ SlotInfo s_info;
    __shared__ int s_err;
    const int item = list[blockIdx.x];
    const SliceWork& w = work[item];
    const int tid = threadIdx.x;
    const bool predict = (w.type & PVVC_TYPE_PREDICT) != 0;
    if (tid == 0) {
        int err = slice_status(w, item, st, tstatus, rstatus);
        if (!err) {
            s_info = st.info[w.slot];
            if (s_info.max_width > wcap && (w.fb_off == ~0ull || s_info.max_width > (int)w.n)) err = PVVC_ERR_TREE;
        }
        // an intra slice that fails leaves its slot without a reference
        if (err && !predict && (w.type & PVVC_TYPE_VALID)) st.info[w.slot].valid = 0;
        s_err = err;
        fstatus[item] = err;
        if (o.status) o.status[w.orig] = err;
    }
    __syncthreads();
    if (s_err) return;
    const int H = s_info.height;
    const size_t nb = (size_t)w.slot * st.max_nodes;
    const size_t lb = (size_t)w.slot * st.max_leaves;
    const uint32_t N = w.n;
    const float* cy = coef + w.coef_off;
    const float* cu = cy + N;
    const float* cv = cu + N;
    if (H == 1) {
        if (tid == 0) emit_leaf(w.mv, w.out_off, w.n < 10, st, lb, 0, cy[0], cu[0], cv[0], predict, o);
        return;
    }
    float *gA, *gB;
    if (s_info.max_width <= wcap) {
        gA = s_g;
        gB = s_g + 3 * wcap;
    } else {
        gA = fallback + w.fb_off;
        gB = gA + 3ull * N;
    }
    if (tid == 0) {
        gA[0] = cy[0];
        gA[1] = cu[0];
        gA[2] = cv[0];
    }
    __syncthreads();
    for (int l = 0; l < H - 1; ++l) {
        const int a = s_info.level_start[l], b = s_info.level_start[l + 1];
        const bool last = (l == H - 2);
        for (int j = tid; j < b - a; j += T) {
            const size_t node = nb + a + j;
            const uint32_t byte = st.occ[node], cb = st.cbase[node];
            float oy[8], ou[8], ov[8];
            inverse_node(st, node, cy, cu, cv, gA[3 * j], gA[3 * j + 1], gA[3 * j + 2], oy, ou, ov);
            uint32_t r = 0;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                if (!(byte & (0x80u >> c))) continue;
                const uint32_t child = cb + r;
                ++r;
                if (!last) {
                    gB[3 * child] = oy[c];
                    gB[3 * child + 1] = ou[c];
                    gB[3 * child + 2] = ov[c];
                } else {
                    emit_leaf(w.mv, w.out_off, w.n < 10, st, lb, child, oy[c], ou[c], ov[c], predict, o);
                }
            }
        }
        __syncthreads();
        float* t = gA;
        gA = gB;
        gB = t;
    }
}

// inverse_node for a lane that may be inactive (no coefficient loads then),
// given the node's coded-slot mask `m`, first coefficient `ci` and butterfly
// pairs ab[i * AS] (AS = 1: the state's node record; 32: a warp's staged
// rows).  Coded slot i reads coefficient ci + (coded slots below i), so the
// node's coefficient loads are independent and issue together.
//
// `m` is the same in every lane (the lanes share the tree), so each slot's
// branch is uniform.  An uncoded butterfly has a zero weight on one side
// and h = 0: with (a, b) = (1, 0), G = g*1 + 0*(-0) = g exactly and H feeds
// only the empty side; with (0, 1), H = g*1 + 0*0 = g + 0 (+0 for g = -0)
// and G feeds only the empty side; with both weights zero neither is read.
// So G = g, H = g + 0 reproduce every value a child can see.
template <int S, int AS>  // coefficient stride (32 in frame-interleaved group regions), ab stride
__device__ __forceinline__ void lane_node_md(uint32_t m, uint32_t ci, const float2* ab, bool act, const float* cy,
                                             const float* cu, const float* cv, float gy, float gu, float gv,
                                             float (&oy)[8], float (&ou)[8], float (&ov)[8]) {
    float hy[8], hu[8], hv[8];
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        const bool coded = act && (m & (1u << i));
        const size_t k = (size_t)(ci + __popc(m & ((1u << i) - 2u))) * S;
        hy[i] = coded ? __ldg(cy + k) : 0.f;
        hu[i] = coded ? __ldg(cu + k) : 0.f;
        hv[i] = coded ? __ldg(cv + k) : 0.f;
    }
    float sy[8], su[8], sv[8];
    sy[1] = gy;
    su[1] = gu;
    sv[1] = gv;
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        const float ay = sy[i], au = su[i], av = sv[i];
        float Gy, Gu, Gv, Hy, Hu, Hv;
        if (m & (1u << i)) {
            const float2 t = ab[(i - 1) * AS];
            const float nbv = -t.y;
            // [G;H] = [[a,-b],[b,a]] [g;h]   (InvertHaarTransform, octree_base.cc:186-206)
            Gy = __fadd_rn(__fmul_rn(ay, t.x), __fmul_rn(hy[i], nbv));
            Gu = __fadd_rn(__fmul_rn(au, t.x), __fmul_rn(hu[i], nbv));
            Gv = __fadd_rn(__fmul_rn(av, t.x), __fmul_rn(hv[i], nbv));
            Hy = __fadd_rn(__fmul_rn(ay, t.y), __fmul_rn(hy[i], t.x));
            Hu = __fadd_rn(__fmul_rn(au, t.y), __fmul_rn(hu[i], t.x));
            Hv = __fadd_rn(__fmul_rn(av, t.y), __fmul_rn(hv[i], t.x));
        } else {
            Gy = ay;
            Gu = au;
            Gv = av;
            Hy = __fadd_rn(ay, 0.0f);
            Hu = __fadd_rn(au, 0.0f);
            Hv = __fadd_rn(av, 0.0f);
        }
        if (pair0(i) < 8) {
            sy[pair0(i)] = Gy; su[pair0(i)] = Gu; sv[pair0(i)] = Gv;
            sy[pair1(i)] = Hy; su[pair1(i)] = Hu; sv[pair1(i)] = Hv;
        } else {
            oy[pair0(i) - 8] = Gy; ou[pair0(i) - 8] = Gu; ov[pair0(i) - 8] = Gv;
            oy[pair1(i) - 8] = Hy; ou[pair1(i) - 8] = Hu; ov[pair1(i) - 8] = Hv;
        }
    }
}

template <int S>
__device__ __forceinline__ void lane_node(const StateView& st, size_t node, bool act, const float* cy, const float* cu,
                                          const float* cv, float gy, float gu, float gv, float (&oy)[8], float (&ou)[8],
                                          float (&ov)[8]) {
    lane_node_md<S, 1>(__ldg(st.mask + node), __ldg(st.coff + node), st.ab + node * 7, act, cy, cu, cv, gy, gu, gv, oy, ou,
                       ov);
}

// A warp's staged node records: kRowNodes consecutive nodes of one level.
constexpr int kRowNodes = 32;
struct NodeRows {
    uint32_t occ[kRowNodes], cb[kRowNodes], mask[kRowNodes], coff[kRowNodes];
    float2 ab[7][kRowNodes];
};

// k_raht_group (window groups: near 32 slices each, as many as the device has SMs
// or more; there its uniform control flow and line-wide accesses cost the least
// instructions a point): persistent CTAs; each takes the next group of slices that
// share a slot (the frames of one patch) from a queue.  Lane f of every warp
// owns frame f (same control flow in all lanes, node records are broadcast
// loads).  The intra slice, when the group has one, is lane 0 and hands its
// leaf colours to the predictive lanes by shuffle.
//
// Levels above the last two internal ones: the 8 warps split each level's
// nodes and the CTA synchronises per level.  The level signal lives in the
// CTA's own scratch region as [node][yuv][lane], so each warp access is one
// 128-byte line.
//
// The last two internal levels (most of the nodes) go without a barrier or
// a level buffer: warp w takes a contiguous range of last-level nodes, whose
// leaves are contiguous too, and walks their parents alongside -- each
// parent's children DCs go to the warp's shared-memory rows [yuv][child]
// [lane] (a lane reads back only its own column), the first parent found by
// a 32-way search of the parents' child offsets.  A parent whose children
// straddle two warps' ranges is transformed by both.  The warp stages its
// finished points in its own rows [frame][leaf]; when the next node's leaves
// would not fit, it writes the staged leaves of every frame as contiguous
// runs and goes on.  Against a level buffer in global memory for the last
// internal level too, this cut the kernel's DRAM bytes by a quarter.  The
// kernel needs 80 registers without spills: 3 CTAs of 8 warps per SM.
constexpr int kGrpWarps = 8;
constexpr int kWarpLeaves = 16;              // staged leaves per warp (a node adds <= 8)
constexpr int kStageRow = kWarpLeaves + 1;   // odd row length: the 32 lanes' column stores hit 32 banks
static_assert(kWarpLeaves == 16, "the flush maps a frame's staged leaves onto a half-warp");

// A warp stages colours only: leaf centres are the same in every frame of
// the group, and the flush transforms them with each frame's matrix.
template <bool P24>
struct WarpStage {
    uint32_t rgb[32][kStageRow];
};
template <>
struct WarpStage<true> {
    uint32_t rgb[32][kStageRow];
    float fr[32][kStageRow], fg[32][kStageRow], fb[32][kStageRow];  // points24 colours
};
template <bool P24>
struct GroupStage {
    WarpStage<P24> w[kGrpWarps];
};

template <bool P24>
__global__ void __launch_bounds__(32 * kGrpWarps, 3) k_raht_group(const SliceWork* __restrict__ work,
                                                               const GroupDesc* __restrict__ groups, int ngroups,
                                                               const int32_t* __restrict__ items, StateView st,
                                                               const float* __restrict__ coef,
                                                               const int32_t* __restrict__ tstatus,
                                                               const int32_t* __restrict__ rstatus,
                                                               int32_t* __restrict__ fstatus, OutPtrs o,
                                                               float* __restrict__ scratch, uint64_t scratch_floats,
                                                               int* __restrict__ counter) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    GroupStage<P24>& sg = *reinterpret_cast<GroupStage<P24>*>(s_raw);
    __shared__ int s_g, s_H, s_ls[kMaxLevels + 1];
    __shared__ uint64_t s_out[32];
    __shared__ int s_act[32], s_white[32];
    __shared__ float s_mv[32][13];  // each frame's transform rows (odd stride: the lanes' row fills hit 32 banks)
    __shared__ NodeRows s_nodes[kGrpWarps];
    __shared__ float s_dc[kGrpWarps][3][8][32];  // each warp's current parent: its children's DCs [yuv][child][lane]
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    WarpStage<P24>& ws = sg.w[wid];
    float* const bufA = scratch + (uint64_t)blockIdx.x * scratch_floats;
    float* const bufB = bufA + scratch_floats / 2;
    for (;;) {
        if (tid == 0) s_g = atomicAdd(counter, 1);
        __syncthreads();
        const int gi = s_g;
        if (gi >= ngroups) break;
        const GroupDesc G = groups[gi];
        const bool have = lane < G.count;
        const int item = have ? items[G.first + lane] : 0;
        const SliceWork& w = work[item];
        const bool intra_lane = have && G.intra && lane == 0;
        int err = have ? slice_status(w, item, st, tstatus, rstatus) : PVVC_OK;
        const int ierr = G.intra ? __shfl_sync(0xffffffffu, err, 0) : PVVC_OK;
        if (ierr && !intra_lane && have && !err) err = PVVC_ERR_NO_REFERENCE;
        const bool act = have && !err;
        if (wid == 0) {
            if (ierr && lane == 0) st.info[G.slot].valid = 0;  // a failed intra slice empties the slot
            if (have) {
                fstatus[item] = err;
                if (o.status) o.status[w.orig] = err;
            }
            s_act[lane] = act;
            s_out[lane] = act ? w.out_off : 0;
            s_white[lane] = act && w.n < 10;
#pragma unroll
            for (int i = 0; i < 12; ++i) s_mv[lane][i] = act ? w.mv[i] : 0.f;
        }
        const bool any = __any_sync(0xffffffffu, act);  // the same in every warp
        const bool ref_lane0 = G.intra && !ierr;
        if (tid == 0) {
            const SlotInfo* si = st.info + G.slot;
            s_H = si->height;
            for (int l = 0; l < kMaxLevels + 1; ++l) s_ls[l] = si->level_start[l];
        }
        __syncthreads();
        if (any) {
            const int H = s_H;
            const size_t nb = (size_t)G.slot * st.max_nodes;
            const size_t lb = (size_t)G.slot * st.max_leaves;
            const uint32_t N = act ? w.n : 0;
            // frame-interleaved region: coefficient i of plane p at (p*N + i)*32 + lane
            const float* cy = coef + (act ? w.coef_off + lane : 0);
            const float* cu = cy + (size_t)N * 32;
            const float* cv = cu + (size_t)N * 32;
            // one finished leaf of this lane's frame into the warp's stage
            auto finish = [&](uint32_t leaf, uint32_t slot_local, float y, float u, float v) {
                float ry, ru, rv;
                if (ref_lane0) {
                    ry = __shfl_sync(0xffffffffu, y, 0);
                    ru = __shfl_sync(0xffffffffu, u, 0);
                    rv = __shfl_sync(0xffffffffu, v, 0);
                } else {
                    const float* r = st.ref + (lb + leaf) * 3;
                    ry = __ldg(r);
                    ru = __ldg(r + 1);
                    rv = __ldg(r + 2);
                }
                if (!act) return;
                if (intra_lane) {
                    float* r = st.ref + (lb + leaf) * 3;
                    r[0] = y;
                    r[1] = u;
                    r[2] = v;
                } else {
                    y = __fadd_rn(y, ry);
                    u = __fadd_rn(u, ru);
                    v = __fadd_rn(v, rv);
                }
                const float du = __fsub_rn(u, 128.0f), dv = __fsub_rn(v, 128.0f);
                const float R = __fadd_rn(y, __fmul_rn(1.4020f, dv));
                const float Gc = __fsub_rn(__fsub_rn(y, __fmul_rn(0.3441f, du)), __fmul_rn(0.7141f, dv));
                const float B = __fadd_rn(y, __fmul_rn(1.7720f, du));
                ws.rgb[lane][slot_local] = (uint32_t)to_u8(R) | ((uint32_t)to_u8(Gc) << 8) | ((uint32_t)to_u8(B) << 16);
                if constexpr (P24) {
                    ws.fr[lane][slot_local] = __fdiv_rn(R, 255.0f);
                    ws.fg[lane][slot_local] = __fdiv_rn(Gc, 255.0f);
                    ws.fb[lane][slot_local] = __fdiv_rn(B, 255.0f);
                }
            };
            // the warp writes its staged leaves [base, base + cnt) of every active
            // frame, two frames per pass: half-warp h writes frame f0 + h, its
            // lanes consecutive points of that frame.  The leaf centre (read
            // once) goes through the frame's transform here.
            auto flush = [&](uint32_t base, uint32_t cnt) {
                __syncwarp();
                const uint32_t i = lane & 15, h = lane >> 4;
                float x0 = 0.f, y0 = 0.f, z0 = 0.f;
                if (i < cnt) {
                    const float* p = st.xyz + (lb + base + i) * 3;
                    x0 = __ldg(p);
                    y0 = __ldg(p + 1);
                    z0 = __ldg(p + 2);
                }
                for (uint32_t f0 = 0; f0 < 32; f0 += 2) {
                    const uint32_t f = f0 + h;
                    if (i >= cnt || !s_act[f]) continue;
                    const uint64_t oi = s_out[f] + base + i;
                    const float* m = s_mv[f];
                    const float X = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(x0, m[0]), __fmul_rn(y0, m[1])), __fmul_rn(z0, m[2])), m[3]);
                    const float Y = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(x0, m[4]), __fmul_rn(y0, m[5])), __fmul_rn(z0, m[6])), m[7]);
                    const float Z = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(x0, m[8]), __fmul_rn(y0, m[9])), __fmul_rn(z0, m[10])), m[11]);
                    if (o.xyz) {
                        o.xyz[oi * 3 + 0] = X;
                        o.xyz[oi * 3 + 1] = Y;
                        o.xyz[oi * 3 + 2] = Z;
                    }
                    const uint32_t c = ws.rgb[f][i];
                    if (o.rgb) {
                        o.rgb[oi * 3 + 0] = (uint8_t)c;
                        o.rgb[oi * 3 + 1] = (uint8_t)(c >> 8);
                        o.rgb[oi * 3 + 2] = (uint8_t)(c >> 16);
                    }
                    if constexpr (P24) {
                        float* q = o.p24 + oi * 6;
                        const bool white = s_white[f];
                        q[0] = X;
                        q[1] = Y;
                        q[2] = Z;
                        q[3] = white ? 1.0f : ws.fr[f][i];
                        q[4] = white ? 1.0f : ws.fg[f][i];
                        q[5] = white ? 1.0f : ws.fb[f][i];
                    }
                }
                __syncwarp();
            };
            if (H == 1) {
                if (wid == 0) {
                    const float gy = act ? cy[0] : 0.f, gu = act ? cu[0] : 0.f, gv = act ? cv[0] : 0.f;
                    finish(0, 0, gy, gu, gv);
                    flush(0, 1);
                }
            } else {
                float* gA = bufA;
                float* gB = bufB;
                if (wid == 0) {
                    gA[lane] = act ? cy[0] : 0.f;
                    gA[32 + lane] = act ? cu[0] : 0.f;
                    gA[64 + lane] = act ? cv[0] : 0.f;
                }
                __syncthreads();
                for (int l = 0; l < H - 3; ++l) {  // internal levels above the last two
                    const int a = s_ls[l], b = s_ls[l + 1];
                    for (int j = wid; j < b - a; j += kGrpWarps) {
                        const size_t node = nb + a + j;
                        const uint32_t byte = __ldg(st.occ + node), cb = __ldg(st.cbase + node);
                        const float* g3 = gA + (size_t)j * 96 + lane;
                        float oy[8], ou[8], ov[8];
                        lane_node<32>(st, node, act, cy, cu, cv, g3[0], g3[32], g3[64], oy, ou, ov);
                        uint32_t r = 0;
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            if (!(byte & (0x80u >> c))) continue;
                            float* go = gB + (size_t)(cb + r) * 96 + lane;
                            ++r;
                            go[0] = oy[c];
                            go[32] = ou[c];
                            go[64] = ov[c];
                        }
                    }
                    __syncthreads();
                    float* t = gA;
                    gA = gB;
                    gB = t;
                }
                // gA: the DCs of level H - 3 (the parents), or for H = 2 the root's
                const int a = s_ls[H - 2], cnt = s_ls[H - 1] - a;                       // last internal level
                const int pa = H >= 3 ? s_ls[H - 3] : 0, pcnt = H >= 3 ? s_ls[H - 2] - pa : 1;  // its parents
                float(&dc)[3][8][32] = s_dc[wid];
                uint32_t pc0 = 0, pc1 = 0;  // the current parent's children [pc0, pc1) of the last level
                // parent pj: its children's DCs into dc, compacted (child pc0 + r at row r)
                auto parent = [&](int pj) {
                    if (H == 2) {  // the root is the only last-level node: its DC as the one child
                        dc[0][0][lane] = gA[lane];
                        dc[1][0][lane] = gA[32 + lane];
                        dc[2][0][lane] = gA[64 + lane];
                        pc0 = 0;
                        pc1 = 1;
                        return;
                    }
                    const size_t node = nb + pa + pj;
                    const uint32_t byte = __ldg(st.occ + node), cb = __ldg(st.cbase + node);
                    const float* g3 = gA + (size_t)pj * 96 + lane;
                    float oy[8], ou[8], ov[8];
                    lane_node<32>(st, node, act, cy, cu, cv, g3[0], g3[32], g3[64], oy, ou, ov);
                    uint32_t r = 0;
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        if (!(byte & (0x80u >> c))) continue;
                        dc[0][r][lane] = oy[c];
                        dc[1][r][lane] = ou[c];
                        dc[2][r][lane] = ov[c];
                        ++r;
                    }
                    pc0 = cb;
                    pc1 = cb + r;
                };
                // the group's region (every lane's frame shares it) and plane
                // stride, from lane 0, which always holds a slice
                const uint64_t g_off = __shfl_sync(0xffffffffu, have ? w.coef_off : 0ull, 0);
                const uint32_t g_n = __shfl_sync(0xffffffffu, have ? w.n : 0u, 0);
                const float* const g_coef = coef + g_off;
                // Node t+1's coefficient lines into L1 while node t is
                // transformed: lane l < 21 takes line (plane l / 7, coded slot
                // l % 7).
                auto prefetch_node = [&](const NodeRows& r, int t) {
                    const uint32_t nc = __popc(r.mask[t] & 0xFEu);
                    if (lane < 21) {
                        const uint32_t k = (uint32_t)lane % 7u, pl = (uint32_t)lane / 7u;
                        if (k < nc) {
                            const float* line = g_coef + ((size_t)pl * g_n + r.coff[t] + k) * 32;
                            asm volatile("prefetch.global.L1 [%0];" ::"l"(line));
                        }
                    }
                };
                // this warp's share of the last-level nodes
                const int per = (cnt + kGrpWarps - 1) / kGrpWarps;
                const int j0 = min(cnt, wid * per), j1 = min(cnt, j0 + per);
                uint32_t base = 0, staged = 0;
                int pj = 0;
                if (j0 < j1) {
                    base = __ldg(st.cbase + nb + a + j0);
                    if (H >= 3) {
                        // the parent of node j0: the last parent whose first
                        // child is at or below j0 (child offsets ascend)
                        int lo = 0, hi = pcnt;
                        while (hi - lo > 1) {
                            const int step = (hi - lo + 31) >> 5;
                            const int idx = lo + lane * step;
                            const bool le = idx < hi && (int)__ldg(st.cbase + nb + pa + idx) <= j0;
                            const uint32_t bal = __ballot_sync(0xffffffffu, le);  // lanes 0.. k hold; lane 0 always
                            lo += (bal ? 31 - __clz(bal) : 0) * step;
                            hi = min(hi, lo + step);
                        }
                        pj = lo;
                    }
                    parent(pj);
                }
                NodeRows& nr = s_nodes[wid];
                for (int jb = j0; jb < j1; jb += kRowNodes) {
                    // the next node records, one node per lane, all loads in flight at once
                    const int nn = min(kRowNodes, j1 - jb);
                    __syncwarp();
                    if (lane < nn) {
                        const size_t node = nb + a + jb + lane;
                        nr.occ[lane] = __ldg(st.occ + node);
                        nr.cb[lane] = __ldg(st.cbase + node);
                        nr.mask[lane] = __ldg(st.mask + node);
                        nr.coff[lane] = __ldg(st.coff + node);
                        const float2* ab = st.ab + node * 7;
#pragma unroll
                        for (int i = 0; i < 7; ++i) nr.ab[i][lane] = __ldg(ab + i);
                    }
                    __syncwarp();
                    if (nn > 0) prefetch_node(nr, 0);
                    for (int t = 0; t < nn; ++t) {
                        if (t + 1 < nn) prefetch_node(nr, t + 1);
                        const uint32_t jc = (uint32_t)(jb + t);
                        while (jc >= pc1 && pj + 1 < pcnt) parent(++pj);  // the next parent with children
                        const uint32_t byte = nr.occ[t], cb = nr.cb[t];
                        const uint32_t k = __popc(byte);
                        if (staged + k > (uint32_t)kWarpLeaves) {
                            flush(base, staged);
                            base += staged;
                            staged = 0;
                        }
                        const uint32_t rc = jc - pc0 < 8u ? jc - pc0 : 0u;  // its row (in range for a well-formed tree)
                        float oy[8], ou[8], ov[8];
                        lane_node_md<32, kRowNodes>(nr.mask[t], nr.coff[t], &nr.ab[0][t], act, cy, cu, cv, dc[0][rc][lane],
                                                    dc[1][rc][lane], dc[2][rc][lane], oy, ou, ov);
                        uint32_t r = 0;
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            if (!(byte & (0x80u >> c))) continue;
                            finish(cb + r, cb + r - base, oy[c], ou[c], ov[c]);
                            ++r;
                        }
                        staged = cb + k - base;
                    }
                }
                if (staged) flush(base, staged);
            }
        }
        __syncthreads();
    }
}

// k_raht_few: groups of slices that share a slot, `parts` CTAs a group, each
// taking a range of the last internal level's nodes and their ancestors.  A warp
// takes 32 consecutive nodes of a level, a lane each, and holds their records
// while it goes through (some of) the slices, whose planes are contiguous: the
// lanes are as full as the level is wide, where k_raht_group's lane per slice
// leaves 32 - count of them idle, and there are 3 n floats a slice to clear
// instead of 96 n a group.  The level signal of the part's own nodes is
// [slice][node][yuv] in the CTA's scratch region, between kFewSlack rows for the
// children of its end nodes that belong to another part.  A part's range of a
// level is no wider than its range of the last one unless empty nodes lie between,
// and then the slices go through in chunks that fit.  The leaves of 32 nodes are
// contiguous: their colours go through the warp's shared rows, then a lane writes
// a point.  At the last internal level the intra slice, when the group has one,
// goes first: the others read its colours.
//
// 58 groups of 8 slices (0.8M points): k_raht_group took 275 us for its long tier
// (22 CTAs, 8 of 32 lanes), this 36 (110 CTAs); 1,023 groups of 2 (4M points): 728
// us for the medium tier, 81; the long tier of a 30-frame GoP (64 groups of 30,
// 8M points): 535 us over two CTAs a group, 350 here.  A pair of (slice, node) a
// thread writing its own leaves took 492 on that tier: 12-byte stores 48 bytes
// apart, half the lanes idle.  Bound by the instructions of the transform and the
// points (some 10 a point) at two CTAs an SM.
constexpr int kFewThreads = 256;
constexpr int kFewWarps = kFewThreads / 32;

// a node's record in a lane's registers (no children, no coefficients: idle)
struct LaneNode {
    uint32_t byte, cb, m, ci;
    float2 ab[7];
};

__device__ __forceinline__ void lane_inverse(const LaneNode& r, const float* cy, uint32_t N, float gy, float gu, float gv,
                                             float (&oy)[8], float (&ou)[8], float (&ov)[8]) {
    const float *cu = cy + N, *cv = cu + N;
    float hy[8], hu[8], hv[8];
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        const uint32_t k = r.ci + __popc(r.m & ((1u << i) - 2u));
        const bool coded = r.m & (1u << i);
        hy[i] = coded ? __ldg(cy + k) : 0.f;
        hu[i] = coded ? __ldg(cu + k) : 0.f;
        hv[i] = coded ? __ldg(cv + k) : 0.f;
    }
    float sy[8], su[8], sv[8];
    sy[1] = gy;
    su[1] = gu;
    sv[1] = gv;
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        const float2 t = r.ab[i - 1];
        const float ay = sy[i], au = su[i], av = sv[i], nbv = -t.y;
        // [G;H] = [[a,-b],[b,a]] [g;h]   (InvertHaarTransform, octree_base.cc:186-206)
        const float Gy = __fadd_rn(__fmul_rn(ay, t.x), __fmul_rn(hy[i], nbv));
        const float Gu = __fadd_rn(__fmul_rn(au, t.x), __fmul_rn(hu[i], nbv));
        const float Gv = __fadd_rn(__fmul_rn(av, t.x), __fmul_rn(hv[i], nbv));
        const float Hy = __fadd_rn(__fmul_rn(ay, t.y), __fmul_rn(hy[i], t.x));
        const float Hu = __fadd_rn(__fmul_rn(au, t.y), __fmul_rn(hu[i], t.x));
        const float Hv = __fadd_rn(__fmul_rn(av, t.y), __fmul_rn(hv[i], t.x));
        if (pair0(i) < 8) {
            sy[pair0(i)] = Gy; su[pair0(i)] = Gu; sv[pair0(i)] = Gv;
            sy[pair1(i)] = Hy; su[pair1(i)] = Hu; sv[pair1(i)] = Hv;
        } else {
            oy[pair0(i) - 8] = Gy; ou[pair0(i) - 8] = Gu; ov[pair0(i) - 8] = Gv;
            oy[pair1(i) - 8] = Hy; ou[pair1(i) - 8] = Hu; ov[pair1(i) - 8] = Hv;
        }
    }
}

__global__ void __launch_bounds__(kFewThreads, 2) k_raht_few(const SliceWork* __restrict__ work,
                                                             const GroupDesc* __restrict__ groups, int ngroups, int parts,
                                                             const int32_t* __restrict__ items, StateView st,
                                                             const float* __restrict__ coef,
                                                             const int32_t* __restrict__ tstatus,
                                                             const int32_t* __restrict__ rstatus,
                                                             int32_t* __restrict__ fstatus, OutPtrs o,
                                                             float* __restrict__ scratch, uint64_t scratch_floats,
                                                             int* __restrict__ counter) {
    __shared__ int s_q, s_n, s_intra, s_H, s_ls[kMaxLevels + 1];
    __shared__ uint32_t s_N, s_lo[kMaxLevels], s_hi[kMaxLevels];  // this part's nodes of each level
    __shared__ uint64_t s_out[32], s_coef[32];                    // of the slices without an error
    __shared__ float s_mv[32][12];
    __shared__ float s_leaf[kFewWarps][3][256];  // a warp's leaves: [yuv][leaf] (also keeps a CTA off a long RLGR CTA's SM)
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    float* const bufA = scratch + (uint64_t)blockIdx.x * scratch_floats;
    float* const bufB = bufA + scratch_floats / 2;
    for (;;) {
        if (tid == 0) s_q = atomicAdd(counter, 1);
        __syncthreads();
        const int q = s_q;
        if (q >= ngroups * parts) break;
        const GroupDesc G = groups[q / parts];
        const int part = q % parts;
        if (tid < 32) {
            const bool have = tid < G.count;
            const int item = have ? items[G.first + tid] : 0;
            const SliceWork& w = work[item];
            const bool intra_lane = have && G.intra && tid == 0;
            int err = have ? slice_status(w, item, st, tstatus, rstatus) : PVVC_OK;
            const int ierr = G.intra ? __shfl_sync(0xffffffffu, err, 0) : PVVC_OK;
            if (ierr && !intra_lane && have && !err) err = PVVC_ERR_NO_REFERENCE;
            if (part == 0) {
                if (ierr && tid == 0) st.info[G.slot].valid = 0;  // a failed intra slice empties the slot
                if (have) {
                    fstatus[item] = err;
                    if (o.status) o.status[w.orig] = err;
                }
            }
            const bool act = have && !err;
            const uint32_t bal = __ballot_sync(0xffffffffu, act);
            if (act) {
                const int f = __popc(bal & ((1u << tid) - 1u));
                s_out[f] = w.out_off;
                s_coef[f] = w.coef_off;
                for (int i = 0; i < 12; ++i) s_mv[f][i] = w.mv[i];
                s_N = w.n;  // every active slice's: the tree's leaves
            }
            if (tid == 0) {
                s_n = __popc(bal);
                s_intra = G.intra && !ierr;
            }
        } else if (tid == 32) {
            const SlotInfo* si = st.info + G.slot;
            s_H = si->height;
            for (int l = 0; l < kMaxLevels + 1; ++l) s_ls[l] = si->level_start[l];
        }
        __syncthreads();
        const int na = s_n;
        if (na > 0) {
            const int H = s_H, fi = s_intra ? 1 : 0;
            const uint32_t N = s_N;
            const size_t nb = (size_t)G.slot * st.max_nodes;
            const size_t lb = (size_t)G.slot * st.max_leaves;
            if (H == 1) {
                if (tid == 0 && part == 0)
                    for (int f = 0; f < na; ++f) {
                        const float* cy = coef + s_coef[f];
                        emit_leaf(s_mv[f], s_out[f], N < 10, st, lb, 0, cy[0], cy[N], cy[2ull * N], !(fi && f == 0), o);
                    }
            } else {
                if (wid < 2) {
                    // this part's range of each level, upwards: warp 0 its first
                    // node, warp 1 its last one (child offsets ascend: a node's
                    // parent is the last one whose first child is at or below it)
                    const int cnt = s_ls[H - 1] - s_ls[H - 2], per = (cnt + parts - 1) / parts;
                    const int j0 = min(cnt, part * per), j1 = min(cnt, j0 + per);
                    int at = wid == 0 ? j0 : max(j0, j1 - 1);
                    for (int l = H - 2;; --l) {
                        if (lane == 0) (wid == 0 ? s_lo : s_hi)[l] = wid == 0 ? at : j0 < j1 ? at + 1 : 0;
                        if (l == 0) break;
                        const uint32_t* cb = st.cbase + nb + s_ls[l - 1];
                        int lo = 0, hi = s_ls[l] - s_ls[l - 1];
                        while (hi - lo > 1) {
                            const int step = (hi - lo + 31) >> 5, idx = lo + lane * step;
                            const uint32_t bal = __ballot_sync(0xffffffffu, idx < hi && (int)__ldg(cb + idx) <= at);
                            lo += (bal ? 31 - __clz(bal) : 0) * step;
                            hi = min(hi, lo + step);
                        }
                        at = lo;
                    }
                }
                __syncthreads();
                auto width = [&](int l) { return max(s_hi[l], s_lo[l]) - s_lo[l]; };
                uint32_t widest = 0;
                for (int l = 0; l < H - 1; ++l) widest = max(widest, width(l));
                const size_t row = 3ull * (widest + 2 * kFewSlack);  // a slice's level signal
                // slices at a time: all, but for a range widened by empty nodes (the
                // buffers hold a slice of any width up to N, the widest level)
                const int chunk = widest ? (int)min((uint64_t)na, scratch_floats / 2 / row) : 0;
                float *gA, *gB;
                // this part's nodes of level l of the slices [f0, f0 + nf) of a chunk
                auto nodes = [&](int l, int first, int f0, int nf, bool predict) {
                    const bool last = l == H - 2;
                    const uint32_t lo = s_lo[l], nj = width(l), nbatch = (nj + 31) / 32;
                    const uint32_t clo = last ? 0u : s_lo[l + 1];
                    // the slices in chunks, so that every warp has two units or more
                    const int chunks = nbatch ? min(nf, (int)((2 * kFewWarps + nbatch - 1) / nbatch)) : 1;
                    const int per = (nf + chunks - 1) / max(chunks, 1);
                    for (uint32_t unit = wid; unit < nbatch * chunks; unit += kFewWarps) {
                        const uint32_t ch = unit / nbatch, j0 = (unit - ch * nbatch) * 32;
                        const int fa = f0 + (int)ch * per, fb = min(f0 + nf, fa + per);
                        const uint32_t nv = min(32u, nj - j0), j = lo + j0 + min((uint32_t)lane, nv - 1);
                        const size_t node = nb + s_ls[l] + j;
                        LaneNode rec;
                        rec.byte = (uint32_t)lane < nv ? st.occ[node] : 0u;
                        rec.m = (uint32_t)lane < nv ? st.mask[node] : 0u;
                        rec.cb = st.cbase[node];
                        rec.ci = st.coff[node];
#pragma unroll
                        for (int i = 0; i < 7; ++i) rec.ab[i] = __ldg(st.ab + node * 7 + i);
                        const uint32_t base = __shfl_sync(0xffffffffu, rec.cb, 0);
                        const uint32_t total = __shfl_sync(0xffffffffu, rec.cb + __popc(rec.byte), nv - 1) - base;
                        for (int f = fa; f < fb; ++f) {
                            const float* g = gA + (f - first) * row + 3ull * (j + kFewSlack - lo);
                            float oy[8], ou[8], ov[8];
                            lane_inverse(rec, coef + s_coef[f], N, g[0], g[1], g[2], oy, ou, ov);
                            if (!last) {
                                float* gb = gB + (f - first) * row;
                                gb += 3ull * (rec.cb + kFewSlack - clo);
#pragma unroll
                                for (int c = 0; c < 8; ++c) {
                                    if (!(rec.byte & (0x80u >> c))) continue;
                                    gb[0] = oy[c];
                                    gb[1] = ou[c];
                                    gb[2] = ov[c];
                                    gb += 3;
                                }
                                continue;
                            }
                            float(&lf)[3][256] = s_leaf[wid];
                            uint32_t at = rec.cb - base;
#pragma unroll
                            for (int c = 0; c < 8; ++c) {
                                if (!(rec.byte & (0x80u >> c))) continue;
                                lf[0][at] = oy[c];
                                lf[1][at] = ou[c];
                                lf[2][at] = ov[c];
                                ++at;
                            }
                            __syncwarp();
                            const uint64_t out = s_out[f];
                            for (uint32_t i = lane; i < total; i += 32)
                                emit_leaf(s_mv[f], out, N < 10, st, lb, base + i, lf[0][i], lf[1][i], lf[2][i], predict, o);
                            __syncwarp();
                        }
                    }
                };
                for (int first = 0; chunk && first < na; first += chunk) {
                    const int nf = min(chunk, na - first);
                    gA = bufA;
                    gB = bufB;
                    if (tid < nf) {
                        const float* cy = coef + s_coef[first + tid];
                        float* g = gA + tid * row + 3 * kFewSlack;
                        g[0] = cy[0];
                        g[1] = cy[N];
                        g[2] = cy[2ull * N];
                    }
                    __syncthreads();
                    for (int l = 0; l < H - 2; ++l) {
                        nodes(l, first, first, nf, true);
                        __syncthreads();
                        float* t = gA;
                        gA = gB;
                        gB = t;
                    }
                    const int f1 = first == 0 ? fi : 0;
                    if (f1) {
                        nodes(H - 2, 0, 0, 1, false);
                        __syncthreads();
                    }
                    nodes(H - 2, first, first + f1, nf - f1, true);
                    __syncthreads();
                }
            }
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// k_refresh: the per-call fields of a reused plan's records, gathered from
// the call's description arrays by each record's caller index.
__global__ void k_refresh(SliceWork* __restrict__ work, int n, CallFields f) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    SliceWork& w = work[q];
    const int i = w.orig;
    w.col_off = f.col_off[i];
    w.geo_off = f.geo_off[i];
    w.out_off = f.out_off[i];
    w.csz = f.csz[i];
    w.gsz = f.gsz[i];
    w.qp = f.qp[i];
#pragma unroll
    for (int k = 0; k < 12; ++k) w.mv[k] = f.mv[16ull * i + k];
}

// ---------------------------------------------------------------------------
// launchers (host)
constexpr int kTreeThreads = 256;
constexpr int kRahtThreads = 128;

// Dynamic shared-memory limits of the inverse-RAHT kernels, set once per
// device before any launch (and so before any stream capture: the launchers
// themselves make only capturable calls).
cudaError_t prepare_kernels() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> g(mu);
    if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
    e = cudaFuncSetAttribute(k_raht_slice<kRahtThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    // The tree kernel runs beside the RLGR launches on every SM.  An SM's split of
    // L1 and shared memory changes only while it is idle: with the tree kernel's
    // own small share, the RLGR CTAs found room for one or two CTAs on most SMs
    // and piled up on the others (a medium tier of a 30-frame GoP took 1.43 ms
    // instead of 0.6; the whole decode 1.98 ms, 1.35 with this).
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_tree<kTreeThreads>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_raht_group<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(GroupStage<false>));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_raht_group<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(GroupStage<true>));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rlgr<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRlgrLongSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rlgr<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRlgrLongSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rlgr<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRlgrLongSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_rlgr<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRlgrLongSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_rlgr<256, 16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRlgrLongSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_rlgr<512, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRlgrLongSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_rlgr_win<1, kWinRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, win_smem(1, kWinRows));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_rlgr_win<2, kWinRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, win_smem(2, kWinRows));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_rlgr_win<4, kWinRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, win_smem(4, kWinRows));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_rlgr_win<8, kWinRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, win_smem(8, kWinRows));
    if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
    return e;
}

cudaError_t launch_tree(const SliceWork* work, int nintra, const uint8_t* payload, const StateView& st, int32_t* tstatus,
                        cudaStream_t s) {
    if (nintra <= 0) return cudaSuccess;
    k_tree<kTreeThreads><<<nintra, kTreeThreads, 0, s>>>(work, payload, st, tstatus);
    return cudaGetLastError();
}

cudaError_t launch_refresh(SliceWork* work, int n, const CallFields& f, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_refresh<<<(n + 255) / 256, 256, 0, s>>>(work, n, f);
    return cudaGetLastError();
}

// smem: dynamic shared memory reserved per CTA (beyond the payload rings it
// limits which CTAs share an SM, see kRlgrLongSmem)
cudaError_t launch_rlgr(const SliceWork* work, const int32_t* order, int nslices, const uint8_t* payload, float* coef,
                        int32_t* rstatus, int block, int smem, cudaStream_t s) {
    if (nslices <= 0) return cudaSuccess;
    const int grid = (nslices + block - 1) / block;
    smem = smem > block * kRing * 16 ? smem : block * kRing * 16;  // at least the payload rings
    switch (block) {
        case 32: k_rlgr<32><<<grid, 32, smem, s>>>(work, order, nslices, payload, coef, rstatus); break;
        case 64: k_rlgr<64><<<grid, 64, smem, s>>>(work, order, nslices, payload, coef, rstatus); break;
        case 128: k_rlgr<128><<<grid, 128, smem, s>>>(work, order, nslices, payload, coef, rstatus); break;
        case 256: k_rlgr<256><<<grid, 256, smem, s>>>(work, order, nslices, payload, coef, rstatus); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// The long-slice launch: kRlgrLongBlock slices per CTA, `lanes` (8, 16, 32)
// of them per warp.
cudaError_t launch_rlgr_long(const SliceWork* work, const int32_t* order, int nslices, const uint8_t* payload, float* coef,
                             int32_t* rstatus, int lanes, int smem, cudaStream_t s) {
    if (nslices <= 0) return cudaSuccess;
    static_assert(kRlgrLongBlock == 128, "a long CTA holds 128 slices");
    static_assert(kRlgrLongSmem >= 512 * kRing * 16, "the long launch's reservation holds its payload rings");
    const int grid = (nslices + kRlgrLongBlock - 1) / kRlgrLongBlock;
    switch (lanes) {
        case 8: k_rlgr<512, 8><<<grid, 512, smem, s>>>(work, order, nslices, payload, coef, rstatus); break;
        case 16: k_rlgr<256, 16><<<grid, 256, smem, s>>>(work, order, nslices, payload, coef, rstatus); break;
        case 32: k_rlgr<128><<<grid, 128, smem, s>>>(work, order, nslices, payload, coef, rstatus); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// Windowed RLGR of `ngroups` groups, one warp each, `warps` per CTA; a
// warp's rings and window take 12 KB, a CTA at least kWinMinSmem, more than
// the SM of a long per-slice CTA has left.
cudaError_t launch_rlgr_win(const SliceWork* work, const GroupDesc* groups, int ngroups, const int32_t* items,
                            const uint8_t* payload, float* coef, int32_t* rstatus, int warps, cudaStream_t s) {
    if (ngroups <= 0) return cudaSuccess;
    static_assert(win_smem(1, kWinRows) + 1024 > 228 * 1024 - (kRlgrLongSmem + 1024),
                  "a windowed CTA must not fit beside a long CTA");
    const int grid = (ngroups + warps - 1) / warps;
    switch (warps) {
        case 1: k_rlgr_win<1, kWinRows><<<grid, 32, win_smem(1, kWinRows), s>>>(work, groups, ngroups, items, payload, coef, rstatus); break;
        case 2: k_rlgr_win<2, kWinRows><<<grid, 64, win_smem(2, kWinRows), s>>>(work, groups, ngroups, items, payload, coef, rstatus); break;
        case 4: k_rlgr_win<4, kWinRows><<<grid, 128, win_smem(4, kWinRows), s>>>(work, groups, ngroups, items, payload, coef, rstatus); break;
        case 8: k_rlgr_win<8, kWinRows><<<grid, 256, win_smem(8, kWinRows), s>>>(work, groups, ngroups, items, payload, coef, rstatus); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_raht_slice(const SliceWork* work, const int32_t* list, int count, const StateView& st, const float* coef,
                              float* fallback, const int32_t* tstatus, const int32_t* rstatus, int32_t* fstatus, float* xyz,
                              uint8_t* rgb, float* p24, int32_t* status, int wcap, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    const size_t smem = 2ull * wcap * 3 * sizeof(float);
    OutPtrs o{xyz, rgb, p24, status};
    k_raht_slice<kRahtThreads><<<count, kRahtThreads, smem, s>>>(work, list, st, coef, fallback, tstatus, rstatus, fstatus, o,
                                                                 wcap);
    return cudaGetLastError();
}

cudaError_t launch_raht_few(const SliceWork* work, const GroupDesc* groups, int ngroups, int parts, const int32_t* items,
                            const StateView& st, const float* coef, const int32_t* tstatus, const int32_t* rstatus,
                            int32_t* fstatus, float* xyz, uint8_t* rgb, float* p24, int32_t* status, float* scratch,
                            uint64_t scratch_floats, int nctas, int* counter, cudaStream_t s) {
    if (ngroups <= 0) return cudaSuccess;
    if (cudaMemsetAsync(counter, 0, sizeof(int), s) != cudaSuccess) return cudaGetLastError();
    OutPtrs o{xyz, rgb, p24, status};
    const int grid = ngroups * parts < nctas ? ngroups * parts : nctas;
    k_raht_few<<<grid, kFewThreads, 0, s>>>(work, groups, ngroups, parts, items, st, coef, tstatus, rstatus, fstatus, o, scratch,
                                            scratch_floats, counter);
    return cudaGetLastError();
}

cudaError_t launch_raht_group(const SliceWork* work, const GroupDesc* groups, int ngroups, const int32_t* items,
                              const StateView& st, const float* coef, const int32_t* tstatus, const int32_t* rstatus,
                              int32_t* fstatus, float* xyz, uint8_t* rgb, float* p24, int32_t* status, float* scratch,
                              uint64_t scratch_floats, int nctas, int* counter, cudaStream_t s) {
    if (ngroups <= 0) return cudaSuccess;
    if (cudaMemsetAsync(counter, 0, sizeof(int), s) != cudaSuccess) return cudaGetLastError();
    OutPtrs o{xyz, rgb, p24, status};
    const int grid = ngroups < nctas ? ngroups : nctas;
    if (p24)
        k_raht_group<true><<<grid, 32 * kGrpWarps, sizeof(GroupStage<true>), s>>>(
            work, groups, ngroups, items, st, coef, tstatus, rstatus, fstatus, o, scratch, scratch_floats, counter);
    else
        k_raht_group<false><<<grid, 32 * kGrpWarps, sizeof(GroupStage<false>), s>>>(
            work, groups, ngroups, items, st, coef, tstatus, rstatus, fstatus, o, scratch, scratch_floats, counter);
    return cudaGetLastError();
}

}  // namespace pvvc
