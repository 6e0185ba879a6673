// encode_kernels.cu -- GB300 (sm_103a) encoder back end of the colour path:
// forward RAHT, quantisation and RLGR coding of a batch of slices.
//
//   k_tree     (decode_kernels.cu) expands each intra slice's geometry
//              payload into its slot's tables, exactly as for decoding
//   k_fwd_raht one persistent CTA per group of slices that share a slot (the
//              frames of one patch as the 32 lanes of every warp): bottom-up
//              HierarchicalTransform (src/octree/octree_base.cc:65-82,
//              164-184) level by level, the coded high-pass coefficients
//              quantised (src/patch/GoP_encoding.cc:184-189) into the
//              slice's symbol planes in stream (reversed) order
//   k_rlgr_enc one CTA per group: RLGREncoder::Encode/GetResult
//              (src/common/entropy_codec.cc:65-159) into the caller's buffer
//
// Bit-exactness with the CPU encoder: the butterfly pairs come from k_tree
// (the decoder's own a = sqrt(w0)/base, b = sqrt(w1)/base); every FP32
// operation is an explicitly rounded intrinsic in the reference's order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <new>
#include <vector>

#include "decode_internal.h"

namespace pvvc {
namespace {

// warps of a k_fwd_raht CTA; one CTA runs per SM (113 groups of 30 frames, 6M
// points: 0.85 ms with 8 warps, 0.41 with 32)
constexpr int kEncWarps = 32;

__device__ __forceinline__ constexpr int epair0(int i) {
    return i == 1 ? 2 : i == 2 ? 4 : i == 3 ? 5 : i == 4 ? 8 : i == 5 ? 9 : i == 6 ? 10 : 11;
}
__device__ __forceinline__ constexpr int epair1(int i) {
    return i == 1 ? 3 : i == 2 ? 6 : i == 3 ? 7 : i == 4 ? 12 : i == 5 ? 13 : i == 6 ? 14 : 15;
}

// static_cast<FIX_DATA_INT>(std::round(c / QP)) (GoP_encoding.cc:186-188)
__device__ __forceinline__ int32_t quantise(float c, float qp) { return (int32_t)roundf(__fdiv_rn(c, qp)); }

// k_fwd_raht: lanes = the group's slices.  The level signal (children's DC)
// lives in the CTA's scratch as [node][yuv][lane]; levels run bottom-up with
// a CTA barrier each.  Symbol planes use the plan's frame-interleaved group
// regions: symbol j of plane p at coef_off + (p*N + j)*32 + lane.
__global__ void __launch_bounds__(32 * kEncWarps) k_fwd_raht(const SliceWork* __restrict__ work,
                                                             const GroupDesc* __restrict__ groups, int ngroups,
                                                             const int32_t* __restrict__ items, StateView st,
                                                             const float* __restrict__ leaf_yuv, int32_t* __restrict__ sym,
                                                             const int32_t* __restrict__ tstatus, int32_t* __restrict__ fstatus,
                                                             float* __restrict__ scratch, uint64_t scratch_floats,
                                                             int* __restrict__ counter) {
    __shared__ int s_g, s_H, s_ls[kMaxLevels + 1];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
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
        int err = PVVC_OK;
        if (have) {
            if (!(w.type & PVVC_TYPE_VALID)) err = PVVC_ERR_BAD_SLICE;
            else if (!(w.type & PVVC_TYPE_PREDICT)) err = tstatus[item];
            if (!err) {
                const SlotInfo* si = st.info + w.slot;
                if (!si->valid) err = PVVC_ERR_NO_REFERENCE;
                else if ((uint32_t)si->leaves != w.n) err = PVVC_ERR_SIZE;
            }
            if (wid == 0) fstatus[item] = err;
        }
        const bool act = have && !err;
        const bool any = __any_sync(0xffffffffu, act);
        if (tid == 0) {
            const SlotInfo* si = st.info + G.slot;
            s_H = si->height;
            for (int l = 0; l < kMaxLevels + 1; ++l) s_ls[l] = si->level_start[l];
        }
        __syncthreads();
        if (any) {
            const int H = s_H;
            const size_t nb = (size_t)G.slot * st.max_nodes;
            const uint32_t N = act ? w.n : 0;
            const float qp = act ? (float)w.qp : 1.f;
            const float* leaf = leaf_yuv + (act ? 3 * w.out_off : 0);
            int32_t* sy = sym + (act ? w.coef_off + lane : 0);
            // coefficient k (0 = DC, un-reversed order) -> symbol N-1-k of each plane
            auto put = [&](uint32_t k, float y, float u, float v) {
                if (!act) return;
                const size_t j = (size_t)(N - 1 - k);
                sy[j * 32] = quantise(y, qp);
                sy[((size_t)N + j) * 32] = quantise(u, qp);
                sy[((size_t)2 * N + j) * 32] = quantise(v, qp);
            };
            if (H == 1) {
                if (wid == 0 && act) put(0, leaf[0], leaf[1], leaf[2]);
            } else {
                float* gIn = bufA;   // children's DC of the level being transformed
                float* gOut = bufB;  // its nodes' DC
                for (int l = H - 2; l >= 0; --l) {
                    const int a = s_ls[l], b = s_ls[l + 1];
                    const bool last = l == H - 2;  // children are leaves
                    for (int j = wid; j < b - a; j += kEncWarps) {
                        const size_t node = nb + a + j;
                        const uint32_t byte = __ldg(st.occ + node), cb = __ldg(st.cbase + node);
                        const uint32_t m = __ldg(st.mask + node);
                        const uint32_t ci = __ldg(st.coff + node);
                        const float2* ab = st.ab + node * 7;
                        float sy8[16], su8[16], sv8[16];
#pragma unroll
                        for (int c = 0; c < 16; ++c) sy8[c] = su8[c] = sv8[c] = 0.f;
                        uint32_t r = 0;
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            if (!(byte & (0x80u >> c))) continue;
                            if (act) {
                                if (last) {
                                    const float* p = leaf + 3ull * (cb + r);
                                    sy8[8 + c] = p[0];
                                    su8[8 + c] = p[1];
                                    sv8[8 + c] = p[2];
                                } else {
                                    const float* p = gIn + (size_t)(cb + r) * 96 + lane;
                                    sy8[8 + c] = p[0];
                                    su8[8 + c] = p[32];
                                    sv8[8 + c] = p[64];
                                }
                            }
                            ++r;
                        }
                        // HaarTransform for i = 7..1: G = g0 a + g1 b, H = g0 (-b) + g1 a
                        float hy[8], hu[8], hv[8];
#pragma unroll
                        for (int i = 7; i > 0; --i) {
                            const float2 t = __ldg(ab + (i - 1));
                            const float nb2 = -t.y;
                            const float g0y = sy8[epair0(i)], g1y = sy8[epair1(i)];
                            const float g0u = su8[epair0(i)], g1u = su8[epair1(i)];
                            const float g0v = sv8[epair0(i)], g1v = sv8[epair1(i)];
                            sy8[i] = __fadd_rn(__fmul_rn(g0y, t.x), __fmul_rn(g1y, t.y));
                            su8[i] = __fadd_rn(__fmul_rn(g0u, t.x), __fmul_rn(g1u, t.y));
                            sv8[i] = __fadd_rn(__fmul_rn(g0v, t.x), __fmul_rn(g1v, t.y));
                            hy[i] = __fadd_rn(__fmul_rn(g0y, nb2), __fmul_rn(g1y, t.x));
                            hu[i] = __fadd_rn(__fmul_rn(g0u, nb2), __fmul_rn(g1u, t.x));
                            hv[i] = __fadd_rn(__fmul_rn(g0v, nb2), __fmul_rn(g1v, t.x));
                        }
                        // the node's DC to its parent (or the stream's coefficient 0)
                        if (l == 0) {
                            put(0, sy8[1], su8[1], sv8[1]);
                        } else {
                            float* q = gOut + (size_t)j * 96 + lane;
                            q[0] = sy8[1];
                            q[32] = su8[1];
                            q[64] = sv8[1];
                        }
                        // coded high-pass coefficients (both weights > 0) at the node's offsets
#pragma unroll
                        for (int i = 1; i < 8; ++i)
                            if (m & (1u << i)) put(ci + __popc(m & ((1u << i) - 2u)), hy[i], hu[i], hv[i]);
                    }
                    __syncthreads();
                    float* t = gIn;
                    gIn = gOut;
                    gOut = t;
                }
            }
        }
        __syncthreads();
    }
}

constexpr uint32_t kU0 = 3, kU1 = 2, kMaxRP = 32 * 4;

// k_rlgr_enc: RLGREncoder::Encode/GetResult, one CTA per group of slices (the
// frames of one patch, all of N points), 64 symbols of every slice at a time.
//
// Only the adaptive state (kP, kRP, and m, the zeros of the unfinished run) is
// serial.  Warp 0 steps it, lane f for slice f, branch-free, and leaves the
// state each symbol sees in shared memory.  The other warps turn the chunk
// before into bits meanwhile: a warp takes a slice, each lane builds the codes
// of its two symbols from the states, a warp scan places them, and they are
// ORed into the slice's bit buffer, whose full words go out.  The symbols of
// the chunk after come in by cp.async; one barrier per chunk.  A lane's two
// codes fit 32 bits nearly always; a slice's chunk where some lane's do not is
// coded 32 symbols at a time in 64 bits.
//
// What bounds it is warp 0, about 35 instructions and 80 cycles a symbol, over
// the longest slices.  3,390 slices of 18M symbols (longest 21,500): 11.0 ms as
// a thread per slice in divergent 64-bit code, 1.79 ms as a warp per slice that
// stepped its own state in every lane, 0.96 ms in this form (1.01 with 6 coders
// instead of 12).
constexpr int kEncWarpsR = 16;                // warp 0, three idle ones and the coders
constexpr int kEncCoders = kEncWarpsR / 4 * 3;
constexpr uint32_t kEncChunk = 64;            // symbols of a slice in a chunk, two per lane of its coder
// Symbol j of slice f at word j * kEncRow + f: a row's lanes hit 32 banks, a
// column's (a coder's lanes, two symbols apart) 16, and the stepper's addresses
// are one register plus constants.
constexpr uint32_t kEncRow = 33;
__device__ __forceinline__ uint32_t enc_at(uint32_t j, uint32_t f) { return j * kEncRow + f; }
// A symbol's state in one word, kP | kRP << 8 | (m & 0xFFFF) << 16.  m is below
// 2^(kP >> 2), and kP rises by at most 2 per 2^(kP >> 2) zeros in run mode: from
// below kEncWideP it stays below 68 for a chunk, so m's high half is zero.  A
// chunk that a slice enters above it keeps the high halves in a second array.
constexpr uint32_t kEncWideP = 60;
// The bit buffer: 32 symbols of at most 1 + 32 (the run's zero and remainder)
// + 64 bits (a Golomb-Rice code, escaped ones included) after up to 31 carried
// over, with two words of slack for a code's 96-bit placement; also holds 1,023
// bits kept and a chunk's 32 codes of 32 bits.
constexpr int kEncBufWords = (31 + 32 * 97) / 32 + 3;

struct EncShared {
    int32_t sym[3][kEncRow * kEncChunk];      // chunk i % 3: the symbols
    uint32_t st[2][kEncRow * kEncChunk];      // chunk i % 2: the state before each symbol
    uint16_t mhigh[2][kEncRow * kEncChunk];   // ... and m >> 16 in a wide chunk
    uint32_t wide[2];
    uint32_t buf[32][kEncBufWords];           // the slices' bit buffers
    uint32_t nbits[32];                       // bits in buf[f]: below 1024 between chunks
    uint64_t nwords[32], cap[32];             // words out, words that fit
    uint32_t* dst[32];
    uint32_t end_kp[32], end_m[32];           // the state after the last symbol
    uint8_t act[32], trail[32];               // has a slice; its last symbol was read in run mode and left u = 0
};

__device__ __forceinline__ uint32_t shr_clamp(uint32_t v, uint32_t n) {  // v >> n, 0 for n >= 32
    uint32_t d;
    asm("shr.u32 %0, %1, %2;" : "=r"(d) : "r"(v), "r"(n));
    return d;
}

// a symbol and the state it is coded in
struct EncSymbol {
    uint32_t uu, kr, k, m;
    bool run, skip, full;  // skip: a zero inside a run; full: it completes 2^k of them
    __device__ __forceinline__ EncSymbol(int32_t x, uint32_t st, uint32_t mhigh) {
        const uint32_t u = ((uint32_t)x << 1) ^ (uint32_t)(x >> 31);  // Sign2Unsign
        k = (st & 0xFFu) >> 2;
        kr = (st >> 10) & 0x3Fu;
        m = st >> 16 | mhigh << 16;
        run = k != 0;
        skip = run && u == 0;
        full = ((m + 1) >> (k & 31)) != 0;
        uu = u - (run && u != 0 ? 1u : 0u);
    }
    __device__ __forceinline__ uint32_t p() const { return shr_clamp(uu, kr); }
};

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// OR the low `len` (<= 64) bits of v into the MSB-first bit buffer at bit `at`
__device__ __forceinline__ void put_bits(uint32_t* buf, uint32_t at, uint64_t v, uint32_t len) {
    if (len == 0) return;
    v <<= 64 - len;
    const uint32_t w = at >> 5, s = at & 31;
    const uint32_t hi = (uint32_t)(v >> 32), lo = (uint32_t)v;
    const uint32_t a = hi >> s, b = __funnelshift_r(lo, hi, s), c = __funnelshift_r(0u, lo, s);
    if (a) atomicOr(buf + w, a);
    if (b) atomicOr(buf + w + 1, b);
    if (c) atomicOr(buf + w + 2, c);
}

__global__ void __launch_bounds__(32 * kEncWarpsR) k_rlgr_enc(const SliceWork* __restrict__ work,
                                                              const GroupDesc* __restrict__ groups,
                                                              const int32_t* __restrict__ items,
                                                              const int32_t* __restrict__ sym, uint8_t* __restrict__ out,
                                                              const uint64_t* __restrict__ out_off,
                                                              const uint32_t* __restrict__ out_cap,
                                                              uint32_t* __restrict__ out_len, int32_t* __restrict__ fstatus) {
    extern __shared__ __align__(16) unsigned char s_enc[];
    EncShared& e = *reinterpret_cast<EncShared*>(s_enc);
    __shared__ uint32_t s_n;
    __shared__ uint64_t s_region;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const GroupDesc G = groups[blockIdx.x];
    if (wid == 0) {
        bool act = false;
        uint32_t n = 0;
        uint64_t region = 0;
        if (lane < G.count) {
            const int item = items[G.first + lane];
            const SliceWork& w = work[item];
            act = fstatus[item] == PVVC_OK;
            e.dst[lane] = reinterpret_cast<uint32_t*>(out + out_off[w.orig]);
            e.cap[lane] = out_cap[w.orig] / 4;
            n = w.n;
            region = w.coef_off;
            if (!act) out_len[w.orig] = 0;
        }
        e.act[lane] = act;
        e.trail[lane] = 0;
        e.nbits[lane] = 0;
        e.nwords[lane] = 0;
        // the good slices of a group have their slot's leaf count
        const uint32_t bal = __ballot_sync(0xffffffffu, act);
        if (bal) {
            n = __shfl_sync(0xffffffffu, n, __ffs(bal) - 1);
            region = __shfl_sync(0xffffffffu, region, __ffs(bal) - 1);
        }
        if (lane == 0) {
            s_n = bal ? n : 0u;
            s_region = region;
        }
    }
    for (int i = tid; i < 32 * kEncBufWords; i += 32 * kEncWarpsR) e.buf[0][i] = 0;
    __syncthreads();
    const uint64_t total = 3ull * s_n;
    const uint64_t nch = (total + kEncChunk - 1) / kEncChunk;
    const int32_t* const src = sym + s_region;
    auto fetch = [&](uint64_t c) {  // chunk c's symbols (position j of the planes: 32 lanes at j * 32)
        if (c < nch) {
            int32_t* const to = e.sym[c % 3];
            for (uint32_t i = tid; i < 32 * kEncChunk; i += 32 * kEncWarpsR) {
                const uint64_t j = c * kEncChunk + (i >> 5);
                if (j < total)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(
                                     (uint32_t)__cvta_generic_to_shared(to + enc_at(i >> 5, i & 31))),
                                 "l"(src + j * 32 + (i & 31))
                                 : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // the full words of slice f's buffer (n bits) out, the rest carried to its front
    auto flush = [&](int f, uint32_t n) {
        uint32_t* const buf = e.buf[f];
        const uint32_t full = n >> 5;
        const uint64_t nw = e.nwords[f], cap = e.cap[f];
        __syncwarp();
        const uint32_t carry = buf[full];
        for (uint32_t i = lane; i < full; i += 32)
            if (nw + i < cap) e.dst[f][nw + i] = __byte_perm(buf[i], 0, 0x0123);
        __syncwarp();
        for (uint32_t i = lane; i <= full; i += 32) buf[i] = i == 0 ? carry : 0u;
        if (lane == 0) {
            e.nwords[f] = nw + full;
            e.nbits[f] = n & 31u;
        }
        __syncwarp();
    };
    uint32_t kP = 0, kRP = 8, m = 0;  // warp 0, lane f: slice f's state
    fetch(0);
    for (uint64_t i = 0; i <= nch; ++i) {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();  // chunk i is in, the states of chunk i - 1 are written, chunk i - 2 is coded
        fetch(i + 1);
        if (wid == 0) {
            if (i < nch) {
                const int32_t* const S = e.sym[i % 3];
                uint32_t* const T = e.st[i & 1];
                uint16_t* const M = e.mhigh[i & 1];
                const bool wide = __any_sync(0xffffffffu, kP >= kEncWideP);
                if (lane == 0) e.wide[i & 1] = wide;
                const uint32_t cnt = (uint32_t)min(total - i * kEncChunk, (uint64_t)kEncChunk);
                auto step = [&](uint32_t j, int32_t x) {
                    const uint32_t u = ((uint32_t)x << 1) ^ (uint32_t)(x >> 31);  // Sign2Unsign
                    T[enc_at(j, lane)] = (m << 16) + (kRP << 8) + kP;
                    const bool run = kP >= 4, zero = u == 0, skip = run && zero;
                    // p = (u - run) >> kR, capped (any p above kMaxRP saturates kRP);
                    // kRP + p - 1, or kRP - 2 for p = 0, without a predicate: this
                    // chain is the longest
                    const uint32_t p = min(shr_clamp(run ? max(u, 1u) - 1u : u, kRP >> 2), kMaxRP + 1);
                    const bool full = ((m + 1) >> (kP >> 2)) != 0;  // the run reaches 2^k zeros
                    const uint32_t rp = (uint32_t)max(min((int)(kRP + p + min(p, 1u)) - 2, (int)kMaxRP), 0);
                    const uint32_t zp = run ? (full ? kP + kU1 : kP) : kP + kU0;
                    kP = zero ? zp : max(kP, 1u) - 1u;
                    kRP = skip ? kRP : rp;
                    m = skip && !full ? m + 1 : 0u;
                };
                if (cnt == kEncChunk && !wide) {
                    // the symbols eight at a time, ahead of their steps: the
                    // compiler keeps loads behind the states' stores
                    int32_t x[8];
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j) x[j] = S[enc_at(j, lane)];
#pragma unroll
                    for (uint32_t j0 = 0; j0 < kEncChunk; j0 += 8) {
                        int32_t y[8];
#pragma unroll
                        for (uint32_t j = 0; j < 8; ++j) y[j] = j0 + 8 < kEncChunk ? S[enc_at(j0 + 8 + j, lane)] : 0;
#pragma unroll
                        for (uint32_t j = 0; j < 8; ++j) step(j0 + j, x[j]);
#pragma unroll
                        for (uint32_t j = 0; j < 8; ++j) x[j] = y[j];
                    }
                } else {
                    for (uint32_t j = 0; j < cnt; ++j) {
                        M[enc_at(j, lane)] = (uint16_t)(m >> 16);
                        step(j, S[enc_at(j, lane)]);
                    }
                }
                if (i + 1 == nch) {
                    e.end_kp[lane] = kP;
                    e.end_m[lane] = m;
                }
            }
        } else if (i > 0 && (wid & 3) != 0) {  // (warps 4, 8, .. would share warp 0's scheduler)
            const uint64_t c = i - 1;
            const uint32_t cnt = (uint32_t)min(total - c * kEncChunk, (uint64_t)kEncChunk);
            const int32_t* const S = e.sym[c % 3];
            const uint32_t* const T = e.st[c & 1];
            const uint16_t* const M = e.mhigh[c & 1];
            const bool wide_m = e.wide[c & 1] != 0;
            for (int f = wid - 1 - (wid >> 2); f < G.count; f += kEncCoders) {
                if (!e.act[f]) continue;
                uint32_t code = 0, len = 0;
                bool wide = false;
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    const uint32_t j = 2 * lane + h, at = enc_at(j, f);
                    if (j >= cnt) continue;
                    const EncSymbol y(S[at], T[at], wide_m ? M[at] : 0u);
                    const uint32_t p = y.p();
                    uint32_t n = p + 1 + y.kr + (y.run ? 1 + y.k : 0u);
                    uint32_t v = (((2u << (p & 31)) - 2u) << (y.kr & 31)) | (y.uu & ((1u << (y.kr & 31)) - 1u));
                    v |= y.run ? __funnelshift_lc(0u, y.m, p + 1 + y.kr) : 0u;
                    if (y.skip) n = v = y.full ? 1u : 0u;  // a completed run: a 1
                    wide |= n > 32 || p >= 32 || len + n > 32;
                    code = __funnelshift_lc(0u, code, n) | v;
                    len += n;
                    if (c + 1 == nch && j == cnt - 1) e.trail[f] = y.run && y.uu == 0;
                }
                if (__any_sync(0xffffffffu, wide)) {
                    flush(f, e.nbits[f]);
                    for (uint32_t h = 0; h < kEncChunk; h += 32) {
                        uint64_t head = 0, body = 0;
                        uint32_t hlen = 0, blen = 0;
                        if (h + lane < cnt) {
                            const uint32_t at = enc_at(h + lane, f);
                            const EncSymbol y(S[at], T[at], wide_m ? M[at] : 0u);
                            const uint32_t p = y.p();
                            if (y.skip) {
                                body = blen = y.full ? 1u : 0u;
                            } else {
                                if (y.run) {  // the run's end: a zero and its remainder
                                    head = y.m;
                                    hlen = 1 + y.k;
                                }
                                if (p < 32) {  // GRWrite: p ones, a zero, kR bits
                                    body = (((1ull << (p + 1)) - 2) << y.kr) | (y.uu & (uint32_t)((1ull << y.kr) - 1));
                                    blen = p + 1 + y.kr;
                                } else {
                                    body = 0xFFFFFFFF00000000ull | y.uu;
                                    blen = 64;
                                }
                            }
                        }
                        const uint32_t n = hlen + blen;
                        const uint32_t end = warp_incl_scan(n, lane), bits = __shfl_sync(0xffffffffu, end, 31);
                        if (bits == 0) continue;
                        const uint32_t nb = e.nbits[f], at = nb + end - n;
                        put_bits(e.buf[f], at, head, hlen);
                        put_bits(e.buf[f], at + hlen, body, blen);
                        flush(f, nb + bits);
                    }
                    continue;
                }
                const uint32_t end = warp_incl_scan(len, lane), bits = __shfl_sync(0xffffffffu, end, 31);
                if (bits == 0) continue;
                const uint32_t nb = e.nbits[f];
                if (len) {
                    const uint32_t at = nb + end - len, w = at >> 5, sh = at & 31, v = code << (32 - len);
                    atomicOr(&e.buf[f][w], v >> sh);
                    if (sh + len > 32) atomicOr(&e.buf[f][w + 1], __funnelshift_r(0u, v, sh));
                }
                // out once a line's worth of words is full
                if (nb + bits >= 1024) {
                    flush(f, nb + bits);
                } else {
                    __syncwarp();
                    if (lane == 0) e.nbits[f] = nb + bits;
                    __syncwarp();
                }
            }
        }
    }
    __syncthreads();
    for (int f = wid; f < G.count; f += kEncWarpsR) {
        if (!e.act[f]) continue;
        flush(f, e.nbits[f]);
        if (e.trail[f]) {  // trailing run (entropy_codec.cc:144-147)
            const uint32_t n = 1 + (e.end_kp[f] >> 2), nb = e.nbits[f];
            if (lane == 0) put_bits(e.buf[f], nb, e.end_m[f], n);
            flush(f, nb + n);
        }
        if (lane == 0) {  // zero bits up to the byte boundary
            const uint32_t nb = e.nbits[f];
            const uint64_t nw = e.nwords[f], cap = e.cap[f], nbytes = nw * 4 + ((nb + 7) >> 3);
            const int item = items[G.first + f];
            const SliceWork& w = work[item];
            if (nb && nw < cap) e.dst[f][nw] = __byte_perm(e.buf[f][0], 0, 0x0123);
            out_len[w.orig] = nbytes > cap * 4 ? 0u : (uint32_t)nbytes;
            if (nbytes > cap * 4) fstatus[item] = PVVC_ERR_CAPACITY;
        }
    }
}

__global__ void k_status_out(const SliceWork* __restrict__ work, int n, const int32_t* __restrict__ fstatus,
                             int32_t* __restrict__ status) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) status[work[t].orig] = fstatus[t];
}

}  // namespace
}  // namespace pvvc

using namespace pvvc;

struct pvvc_encoder {
    pvvc_plan plan;
    DevBuf ws, off, cap;
    HostBuf h_off, h_cap;
};

extern "C" int pvvc_encoder_create(pvvc_encoder** out) {
    if (!out) return PVVC_ERR_ARG;
    *out = new (std::nothrow) pvvc_encoder();
    return *out ? PVVC_OK : PVVC_ERR_NOMEM;
}

extern "C" int pvvc_encoder_destroy(pvvc_encoder* e) {
    if (!e) return PVVC_ERR_ARG;
    delete e;
    return PVVC_OK;
}

extern "C" int pvvc_encode_colors(pvvc_encoder* enc, const pvvc_batch_desc* desc, pvvc_state* st, const uint8_t* payload,
                                  const float* leaf_yuv, uint8_t* out, const uint64_t* out_byte_off, const uint32_t* out_cap,
                                  uint32_t* out_len, int32_t* status, void* stream) {
    if (!enc || !desc || !st || desc->nslices < 0) return PVVC_ERR_ARG;
    const int n = desc->nslices;
    if (n == 0) return PVVC_OK;
    if (!payload || !leaf_yuv || !out || !out_byte_off || !out_cap || !out_len || !status) return PVVC_ERR_ARG;
    if ((reinterpret_cast<uintptr_t>(payload) & 15u) || (reinterpret_cast<uintptr_t>(out) & 3u)) return PVVC_ERR_ARG;
    for (int i = 0; i < n; ++i)
        if ((out_byte_off[i] & 3u) || (out_cap[i] & 3u)) return PVVC_ERR_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    // every slot's slices in groups of up to 32 (no per-slice path), no RLGR split
    const pvvc_tune t{1, 1, 128, -1, -1, 32};
    pvvc_plan& p = enc->plan;
    p.wide_only = true;
    int rc = build_plan(desc, &p, &t, nullptr);
    if (rc) return rc;
    if (p.max_slot >= st->v.nslots) return PVVC_ERR_ARG;
    if (p.nlist_a || p.nlist_b) return PVVC_ERR_ARG;  // min_group 1 groups every slice
    const uint64_t sym_bytes = 4ull * p.coef_floats;  // int32 symbols in the planes' layout
    const uint64_t scratch_bytes = 4ull * p.grp_floats * std::max(p.grp_ctas, 1);
    const uint64_t o_sym = 0, o_scr = align_up(sym_bytes, 256), o_ts = align_up(o_scr + scratch_bytes, 256),
                   o_fs = align_up(o_ts + 4ull * n, 256), o_cnt = align_up(o_fs + 4ull * n, 256), total = o_cnt + 256;
    if (enc->ws.ensure(total) != cudaSuccess || enc->off.ensure(8ull * n) != cudaSuccess ||
        enc->cap.ensure(4ull * n) != cudaSuccess || enc->h_off.ensure(8ull * n) != cudaSuccess ||
        enc->h_cap.ensure(4ull * n) != cudaSuccess)
        return PVVC_ERR_NOMEM;
    std::memcpy(enc->h_off.p, out_byte_off, 8ull * n);
    std::memcpy(enc->h_cap.p, out_cap, 4ull * n);
    uint8_t* w = static_cast<uint8_t*>(enc->ws.p);
    int32_t* sym = reinterpret_cast<int32_t*>(w + o_sym);
    float* scr = reinterpret_cast<float*>(w + o_scr);
    int32_t* ts = reinterpret_cast<int32_t*>(w + o_ts);
    int32_t* fs = reinterpret_cast<int32_t*>(w + o_fs);
    int* cnt = reinterpret_cast<int*>(w + o_cnt);
    const SliceWork* dw = static_cast<const SliceWork*>(p.d_work.p);
    if (cudaMemcpyAsync(enc->off.p, enc->h_off.p, 8ull * n, cudaMemcpyHostToDevice, s) != cudaSuccess ||
        cudaMemcpyAsync(enc->cap.p, enc->h_cap.p, 4ull * n, cudaMemcpyHostToDevice, s) != cudaSuccess ||
        cudaMemsetAsync(cnt, 0, sizeof(int), s) != cudaSuccess)
        return PVVC_ERR_CUDA;
    if (launch_tree(dw, p.nintra, payload, st->v, ts, s) != cudaSuccess ||
        cudaFuncSetAttribute(k_rlgr_enc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(EncShared)) != cudaSuccess)
        return PVVC_ERR_CUDA;
    const int ng = p.ngroups_a + p.ngroups_b;
    const int grid = std::min(ng, std::max(p.grp_ctas, 1));
    k_fwd_raht<<<grid, 32 * kEncWarps, 0, s>>>(dw, static_cast<const GroupDesc*>(p.d_groups.p), ng,
                                               static_cast<const int32_t*>(p.d_idx.p), st->v, leaf_yuv, sym, ts, fs, scr,
                                               p.grp_floats, cnt);
    k_rlgr_enc<<<ng, 32 * kEncWarpsR, sizeof(EncShared), s>>>(
        dw, static_cast<const GroupDesc*>(p.d_groups.p), static_cast<const int32_t*>(p.d_idx.p), sym, out,
        static_cast<const uint64_t*>(enc->off.p), static_cast<const uint32_t*>(enc->cap.p), out_len, fs);
    k_status_out<<<(n + 255) / 256, 256, 0, s>>>(dw, n, fs, status);
    if (cudaGetLastError() != cudaSuccess) return PVVC_ERR_CUDA;
    // the host arrays above are reused by the next call: finish this one
    return cudaStreamSynchronize(s) == cudaSuccess ? PVVC_OK : PVVC_ERR_CUDA;
}
