// Chunk-indexed canonical Huffman coding of the quant codes on B200.
//
// The reference entropy-codes each residual stream with SZ3-ncp's
// HuffmanEncoder<int> and a per-chunk "marker" table of bit offsets
// (encode_marked_fast / decode_marked_transform / decode_marked_chunks_fast,
// call sites FD5:1264-1306, 1401-1413, 1512-1562, 1870-1875). That library is
// not available, so the byte format here is this project's own; the roles are
// the same: a codebook per stream, codes grouped in C^3 marker chunks with a
// word offset per chunk (the marker table), so any chunk decodes on its own.
//
// Parallel decomposition: every z-plane of a chunk (C^2 symbols, a
// "sub-chunk") has its bit offset inside the chunk in the stream header, so
// all planes of all chunks of all streams encode and decode independently.
// Inside a plane, the encode side shares the codes among a group of lanes
// (runs are the gaps between literal masks); the decode side shares the bits
// among one, or, in large launches of streams without runs, gives a plane a
// thread. Bits are packed MSB-first into 32-bit words; a chunk starts on a
// word boundary.
//
// Runs: inside a plane, a maximal run of r centre codes (code == radius) is
// coded with run symbols (run_geometry): while r > D, 2^k (the largest power
// of two <= r, k <= J) when k > LD, else D codes; then one symbol for the
// remaining 2..D codes, or the centre code itself for one. The run symbols
// occupy run_n code values the stream does not use (StreamDesc::run_base),
// so they share the codebook, the tables and the 16-bit symbol width with
// the codes; a well-predicted stream (mostly centre codes) then costs well
// under one bit per code.
#include <cuda_runtime.h>

#include "huffman.h"
#include "run_symbols.cuh"

namespace stz {
namespace {

// ---- encode side: a lane group per plane ----------------------------------------
// (Planes of up to 1024 codes take the literal lists below; this segment form
// serves larger planes.)
// Lane i of a group of W lanes (W = 32 for planes of 1024 codes and more,
// fewer for smaller planes, see lanes_per_plane) owns the codes [a_i, b_i) of
// the plane (W consecutive segments of S = ceil(plane / W) codes). A run of centre codes is coded by
// the lane holding the literal that follows it, or, for a run that reaches
// the plane's end, by the lane holding the plane's last code (`tail`): a
// warp max-scan of the lanes' last literal positions gives every lane the
// centre codes just before its segment (`lead`), which belong to the run
// leading into its first literal. The lanes' bit counts, an exclusive warp
// scan of them and the plane's bit offset place every lane's bits, so the
// bitstream is the one a sequential pass over the plane writes.
constexpr int kLaneThreads = 256;  // 8 warps per CTA, each one plane at a time
constexpr int kPlaneSlices = 4;    // CTAs per work item (gridDim.y)

// Lanes per plane: the largest power of two <= plane / 32, at most 32, so a
// lane holds about 32 codes; a warp takes 32 / W planes at a time (small
// planes of the coarser levels would otherwise leave each lane a few codes
// and the per-plane lane scans would dominate).
__host__ __device__ inline uint32_t lanes_per_plane(uint32_t P)
{
    uint32_t w = 1;
    while (w < 32 && 2 * w <= P / 32) w *= 2;
    return w;
}

// A lane group's view of one plane (a group without a plane has an empty
// segment but still takes part in the group's shuffles).
struct LaneSeg {
    uint32_t P, a, b;  // plane size; this lane's codes [a, b)
    uint32_t W, lane;  // lanes of the group; this lane's index in it
    bool vec;          // segments are whole 16-byte groups of 8 codes
};

__device__ __forceinline__ LaneSeg lane_seg(uint32_t C, const uint16_t* src, uint32_t W, bool active)
{
    LaneSeg g;
    g.P = C * C;
    g.W = W;
    g.lane = threadIdx.x & (W - 1);
    const uint32_t S = (g.P + W - 1) / W;
    g.a = active ? min(g.lane * S, g.P) : 0;
    g.b = active ? min(g.a + S, g.P) : 0;
    g.vec = g.P % (8 * W) == 0 && ((uintptr_t)src & 15) == 0;
    return g;
}

// Sum over a lane group of width W (a power of two).
__device__ __forceinline__ uint32_t group_sum(uint32_t v, uint32_t W)
{
    for (uint32_t o = W >> 1; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Inclusive prefix sum over a lane group of width W.
__device__ __forceinline__ uint32_t group_scan(uint32_t v, uint32_t W, uint32_t lane)
{
    for (uint32_t o = 1; o < W; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, v, o, W);
        if (lane >= o) v += u;
    }
    return v;
}

// The lane's codes in order (streams without runs): f(q) for each.
template <class G>
__device__ __forceinline__ void lane_codes(const uint16_t* __restrict__ src, const LaneSeg& g, G&& f)
{
    if (g.vec) {
        const uint4* v = reinterpret_cast<const uint4*>(src + g.a);
        for (uint32_t j = 0; j < (g.b - g.a) / 8; ++j) {
            const uint4 q = __ldg(v + j);
            f(q.x & 0xffffu), f(q.x >> 16), f(q.y & 0xffffu), f(q.y >> 16);
            f(q.z & 0xffffu), f(q.z >> 16), f(q.w & 0xffffu), f(q.w >> 16);
        }
    } else {
        for (uint32_t j = g.a; j < g.b; ++j) f(__ldg(src + j));
    }
}

// Bits 0 and 1 set for the 16-bit halves of w equal to those of R2.
__device__ __forceinline__ uint32_t pair_mask(uint32_t w, uint32_t R2)
{
    const uint32_t e = __vcmpeq2(w, R2);  // 0xffff per equal half
    return (e & 1u) | ((e >> 15) & 2u);
}

// Literal mask of the n <= 32 codes at plane position p: bit i set when code
// p + i is not the centre code R (with g.vec, p and n are multiples of 8).
__device__ __forceinline__ uint32_t literal_mask(const uint16_t* __restrict__ src, const LaneSeg& g, uint32_t p,
                                                 uint32_t n, uint32_t R)
{
    uint32_t m = 0;  // centre codes
    if (g.vec) {
        const uint4* v = reinterpret_cast<const uint4*>(src + p);
        const uint32_t R2 = R | (R << 16);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            if (j < n / 8) {
                const uint4 q = __ldg(v + j);
                m |= (pair_mask(q.x, R2) | pair_mask(q.y, R2) << 2 | pair_mask(q.z, R2) << 4 |
                      pair_mask(q.w, R2) << 6)
                     << (8 * j);
            }
    } else {
        for (uint32_t i = 0; i < n; ++i) m |= (uint32_t)(__ldg(src + p + i) == R) << i;
    }
    return ~m & (n == 32 ? ~0u : (1u << n) - 1);
}

// A lane's plane segment with runs, as 32-code blocks: the literal mask of
// the first block is kept (most segments are one block), later ones are
// rebuilt on each pass.
struct RunLane {
    uint32_t lit0 = 0;  // literal mask of the block at a
    uint32_t lead = 0;  // centre codes between the last literal before a and a
    bool tail = false;  // the lane holds the plane's last code

    template <class F>
    __device__ __forceinline__ void blocks(const uint16_t* __restrict__ src, const LaneSeg& g, uint32_t R, F&& fn) const
    {
        for (uint32_t p = g.a; p < g.b; p += 32) {
            const uint32_t n = min(32u, g.b - p);
            fn(p, n, p == g.a ? lit0 : literal_mask(src, g, p, n, R));
        }
    }

    // Literal masks, then a group max-scan of the lanes' last literal
    // positions for lead.
    __device__ __forceinline__ void init(const uint16_t* __restrict__ src, const LaneSeg& g, uint32_t R)
    {
        uint32_t last = 0;  // last literal + 1 (0: none)
        for (uint32_t p = g.a; p < g.b; p += 32) {
            const uint32_t n = min(32u, g.b - p);
            const uint32_t lit = literal_mask(src, g, p, n, R);
            if (p == g.a) lit0 = lit;
            if (lit) last = p + 32 - __clz(lit);
        }
        for (uint32_t o = 1; o < g.W; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, last, o, g.W);
            if (g.lane >= o) last = max(last, v);
        }
        uint32_t excl = __shfl_up_sync(0xffffffffu, last, 1, g.W);
        if (g.lane == 0) excl = 0;
        lead = g.a - excl;
        tail = g.a < g.b && g.b == g.P;
    }

    // The lane's symbols in order: f(sym). Between consecutive literals of a
    // block every code is a centre code, so the runs are the gaps.
    template <class F>
    __device__ __forceinline__ void symbols(const uint16_t* __restrict__ src, const LaneSeg& g, const StreamDesc& s,
                                            F&& f) const
    {
        uint32_t D, LD;
        const uint32_t J = run_geometry(g.P, D, LD);
        uint32_t run = lead;
        blocks(src, g, s.radius, [&](uint32_t p, uint32_t n, uint32_t lit) {
            uint32_t i = 0;
            while (lit) {
                const uint32_t j = __ffs(lit) - 1;
                run += j - i;
                if (run) {
                    run_symbols(run, s.radius, s.run_base, J, D, LD, f);
                    run = 0;
                }
                f((uint32_t)__ldg(src + p + j));
                i = j + 1;
                lit &= lit - 1;
            }
            run += n - i;
        });
        if (tail && run) run_symbols(run, s.radius, s.run_base, J, D, LD, f);
    }
};

// Planes of a work item for this lane group: warp i of the grid's
// (blockDim.x / 32) * gridDim.y warps on an item takes its planes
// [i * G, i * G + G), then every (warps * G)-th group of G after that (G =
// 32 / W planes per warp); p is this group's plane, valid when active (else
// pe, a valid plane of the same warp, stands in for reads).
#define STZ_GROUP_PLANES(nplanes, W)                                                                      \
    for (uint32_t base_ = (blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 / (W));            \
         base_ < (nplanes); base_ += (blockDim.x >> 5) * gridDim.y * (32 / (W)))
#define STZ_GROUP_PLANE(nplanes, W)                                     \
    const uint32_t p = base_ + (threadIdx.x & 31) / (W);               \
    const bool active = p < (nplanes);                                 \
    const uint32_t pe = active ? p : base_

// ---- literal lists: the symbols of a run-coded plane in warp-wide rounds ----
// A lane's literals vary in number from lane to lane, so a walk over each
// lane's own literals leaves most of the warp idle. Instead the group first
// lists the plane's literal positions in plane order in shared memory (a
// group scan of the lanes' literal counts places each lane's), then visits
// them in rounds of W: literal k (lane k mod W) with the run of centre codes
// before it (the gap to literal k - 1), then the run after the last literal.
// That is the symbol order of a sequential pass over the plane. Used where a
// lane holds at most 32 codes (planes of up to 1024 codes).
constexpr uint32_t kListPerWarp = 1024;  // list entries per warp: 32 / W groups of at most 32 W codes
constexpr uint32_t kStagePerWarp = 832;  // staging words per warp: groups of at most (32 W * 24 + 63) / 32

__device__ __forceinline__ bool lits_ok(uint32_t P, uint32_t W) { return (P + W - 1) / W <= 32; }

// The group's literal positions into list[0, L) in plane order; returns L.
__device__ __forceinline__ uint32_t plane_literals(const uint16_t* __restrict__ src, const LaneSeg& g, uint32_t R,
                                                   uint16_t* list)
{
    const uint32_t n = g.b - g.a;
    const uint32_t m = n ? literal_mask(src, g, g.a, n, R) : 0u;
    const uint32_t c = __popc(m);
    const uint32_t incl = group_scan(c, g.W, g.lane);
    const uint32_t L = __shfl_sync(0xffffffffu, incl, g.W - 1, g.W);
    uint32_t j = incl - c;
    for (uint32_t mm = m; mm; mm &= mm - 1) list[j++] = (uint16_t)(g.a + (__ffs(mm) - 1));
    __syncwarp();
    return L;
}

// Rounds over the group's literals with a warp-uniform trip count (every lane
// takes part in the shuffles f may make): f(valid, pos, run).
template <class F>
__device__ __forceinline__ void literal_rounds(const uint16_t* list, uint32_t L, const LaneSeg& g, F&& f)
{
    const uint32_t rounds = __reduce_max_sync(0xffffffffu, (L + g.W - 1) / g.W);
    for (uint32_t t = 0; t < rounds; ++t) {
        const uint32_t k = t * g.W + g.lane;
        const bool valid = k < L;
        uint32_t pos = 0, run = 0;
        if (valid) {
            pos = list[k];
            run = pos - (k ? list[k - 1] + 1u : 0u);
        }
        f(valid, pos, run);
    }
}

// The same, two consecutive literals per lane per round (2 lane, 2 lane + 1
// of the round's 2W): two independent load chains per lane.
template <class F>
__device__ __forceinline__ void literal_rounds2(const uint16_t* list, uint32_t L, const LaneSeg& g, F&& f)
{
    const uint32_t rounds = __reduce_max_sync(0xffffffffu, (L + 2 * g.W - 1) / (2 * g.W));
    for (uint32_t t = 0; t < rounds; ++t) {
        const uint32_t k = t * 2 * g.W + 2 * g.lane;
        const bool v0 = k < L, v1 = k + 1 < L;
        uint32_t pos0 = 0, run0 = 0, pos1 = 0, run1 = 0;
        if (v0) {
            pos0 = list[k];
            run0 = pos0 - (k ? list[k - 1] + 1u : 0u);
        }
        if (v1) {
            pos1 = list[k + 1];
            run1 = pos1 - pos0 - 1u;
        }
        f(v0, pos0, run0, v1, pos1, run1);
    }
}

// Centre codes after the plane's last literal.
__device__ __forceinline__ uint32_t tail_run(const uint16_t* list, uint32_t L, uint32_t P)
{
    return P - (L ? list[L - 1] + 1u : 0u);
}

// Run-symbol counts of every listed plane (streams with runs).
__global__ void __launch_bounds__(kLaneThreads) k_run_stats(const CtaWork* __restrict__ work,
                                                            const uint32_t* __restrict__ chunk_ids,
                                                            const StreamDesc* __restrict__ sd,
                                                            const uint16_t* __restrict__ codes,
                                                            unsigned long long* __restrict__ stats)
{
    __shared__ uint32_t cnt[kRunStats];
    const CtaWork w = work[blockIdx.x];
    const StreamDesc s = sd[w.stream];
    if (s.run_n == 0) return;  // uniform per block
    if (threadIdx.x < kRunStats) cnt[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t C = s.C, P = C * C, W = lanes_per_plane(P), np = w.count * C;
    uint32_t singles = 0;
    auto count = [&](uint32_t sym) {
        if (sym == s.radius) ++singles;
        else if (sym - s.run_base < s.run_n) atomicAdd(&cnt[sym - s.run_base + 1], 1u);
    };
    if (lits_ok(P, W)) {
        __shared__ uint16_t lists[kLaneThreads / 32][kListPerWarp];
        uint16_t* list = lists[threadIdx.x >> 5] + ((threadIdx.x & 31) / W) * 32 * W;
        uint32_t D, LD;
        const uint32_t J = run_geometry(P, D, LD);
        STZ_GROUP_PLANES(np, W)
        {
            STZ_GROUP_PLANE(np, W);
            const uint32_t c = chunk_ids[w.first + pe / C], lz = pe % C;
            const uint16_t* src = codes + s.code_off + (size_t)c * P * C + (size_t)lz * P;
            const LaneSeg g = lane_seg(C, src, W, active);
            const uint32_t L = plane_literals(src, g, s.radius, list);
            literal_rounds2(list, L, g, [&](bool v0, uint32_t, uint32_t run0, bool v1, uint32_t, uint32_t run1) {
                if (v0 && run0) run_symbols(run0, s.radius, s.run_base, J, D, LD, count);
                if (v1 && run1) run_symbols(run1, s.radius, s.run_base, J, D, LD, count);
            });
            if (active && g.lane == 0) run_symbols(tail_run(list, L, P), s.radius, s.run_base, J, D, LD, count);
            __syncwarp();  // the list is rewritten for the next plane
        }
    } else {
        STZ_GROUP_PLANES(np, W)
        {
            STZ_GROUP_PLANE(np, W);
            const uint32_t c = chunk_ids[w.first + pe / C], lz = pe % C;
            const uint16_t* src = codes + s.code_off + (size_t)c * P * C + (size_t)lz * P;
            const LaneSeg g = lane_seg(C, src, W, active);
            RunLane rl;
            rl.init(src, g, s.radius);
            rl.symbols(src, g, s, count);
        }
    }
    singles = group_sum(singles, 32);
    if ((threadIdx.x & 31) == 0 && singles) atomicAdd(&cnt[0], singles);
    __syncthreads();
    if (threadIdx.x < kRunStats && cnt[threadIdx.x])
        atomicAdd(&stats[(size_t)w.stream * kRunStats + threadIdx.x], cnt[threadIdx.x]);
}

// Bits of every plane.
__global__ void __launch_bounds__(kLaneThreads) k_sub_bits(const CtaWork* __restrict__ work,
                                                           const uint32_t* __restrict__ chunk_ids,
                                                           const StreamDesc* __restrict__ sd,
                                                           const uint16_t* __restrict__ codes,
                                                           const uint32_t* __restrict__ ctab,
                                                           const uint8_t* __restrict__ rbits,
                                                           uint32_t* __restrict__ sub_bits)
{
    const CtaWork w = work[blockIdx.x];
    const StreamDesc s = sd[w.stream];
    const uint32_t C = s.C, P = C * C, W = lanes_per_plane(P), np = w.count * C;
    const uint32_t* tab = ctab + (size_t)w.stream * 2 * s.radius;
    if (s.run_n && lits_ok(P, W)) {
        __shared__ uint16_t lists[kLaneThreads / 32][kListPerWarp];
        uint16_t* list = lists[threadIdx.x >> 5] + ((threadIdx.x & 31) / W) * 32 * W;
        const uint8_t* rb = rbits + (size_t)w.stream * kRunBitsStride;
        STZ_GROUP_PLANES(np, W)
        {
            STZ_GROUP_PLANE(np, W);
            const uint32_t c = chunk_ids[w.first + pe / C], lz = pe % C;
            const uint16_t* src = codes + s.code_off + (size_t)c * P * C + (size_t)lz * P;
            const LaneSeg g = lane_seg(C, src, W, active);
            const uint32_t L = plane_literals(src, g, s.radius, list);
            uint32_t bits = 0;
            literal_rounds2(list, L, g, [&](bool v0, uint32_t pos0, uint32_t run0, bool v1, uint32_t pos1, uint32_t run1) {
                const uint32_t q0 = v0 ? __ldg(src + pos0) : 0u, q1 = v1 ? __ldg(src + pos1) : 0u;
                if (v0) bits += __ldg(rb + run0) + (__ldg(tab + q0) & 31u);
                if (v1) bits += __ldg(rb + run1) + (__ldg(tab + q1) & 31u);
            });
            if (active && g.lane == 0) bits += __ldg(rb + tail_run(list, L, P));
            bits = group_sum(bits, W);
            if (active && g.lane == 0) sub_bits[s.sub_base + (size_t)c * C + lz] = bits;
            __syncwarp();  // the list is rewritten for the next plane
        }
        return;
    }
    STZ_GROUP_PLANES(np, W)
    {
        STZ_GROUP_PLANE(np, W);
        const uint32_t c = chunk_ids[w.first + pe / C], lz = pe % C;
        const uint16_t* src = codes + s.code_off + (size_t)c * P * C + (size_t)lz * P;
        const LaneSeg g = lane_seg(C, src, W, active);
        uint32_t bits = 0;
        auto add = [&](uint32_t sym) { bits += __ldg(tab + sym) & 31u; };
        if (s.run_n) {
            RunLane rl;
            rl.init(src, g, s.radius);
            rl.symbols(src, g, s, add);
        } else {
            lane_codes(src, g, add);
        }
        bits = group_sum(bits, W);
        if (active && g.lane == 0) sub_bits[s.sub_base + (size_t)c * C + lz] = bits;
    }
}

// Plane bit offsets inside each chunk (one warp per chunk: a scan of the
// planes' bit counts); the chunk's word count goes to chunk_word_off, which
// k_scan_stream then turns into offsets. Block (s, y) takes chunks 32y..32y+31
// of stream s.
__global__ void __launch_bounds__(1024) k_plane_offsets(const StreamDesc* __restrict__ sd,
                                                        const uint32_t* __restrict__ sub_bits,
                                                        uint32_t* __restrict__ sub_off,
                                                        uint64_t* __restrict__ chunk_word_off)
{
    const StreamDesc s = sd[blockIdx.x];
    const uint32_t c = blockIdx.y * 32 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (c >= s.nchunks) return;  // uniform per warp
    const size_t k0 = s.sub_base + (size_t)c * s.C;
    uint64_t carry = 0;
    for (uint32_t lz0 = 0; lz0 < s.C; lz0 += 32) {
        const uint32_t lz = lz0 + lane;
        const uint32_t bits = lz < s.C ? sub_bits[k0 + lz] : 0u;
        uint32_t incl = bits;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        if (lz < s.C) sub_off[k0 + lz] = (uint32_t)(carry + incl - bits);
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) chunk_word_off[s.chunk_base + c] = (carry + 31) / 32;
}

// Per stream: chunk word counts -> word offsets (the marker table) and the
// stream's word count; then the boundary words of every plane are cleared
// for the encoder's atomic ORs.
__global__ void __launch_bounds__(1024) k_scan_stream(const StreamDesc* __restrict__ sd,
                                                      const uint32_t* __restrict__ sub_bits,
                                                      const uint32_t* __restrict__ sub_off,
                                                      uint64_t* __restrict__ chunk_word_off,
                                                      uint64_t* __restrict__ stream_words,
                                                      uint32_t* __restrict__ payload)
{
    const StreamDesc s = sd[blockIdx.x];
    const uint32_t C = s.C;
    __shared__ uint64_t carry;
    __shared__ uint64_t wsum[32];
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < s.nchunks; base += blockDim.x) {
        const uint32_t c = base + threadIdx.x;
        const uint64_t words = c < s.nchunks ? chunk_word_off[s.chunk_base + c] : 0;
        uint64_t incl = words;
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if ((threadIdx.x & 31) >= o) incl += v;
        }
        if ((threadIdx.x & 31) == 31) wsum[threadIdx.x >> 5] = incl;
        __syncthreads();
        if (threadIdx.x < 32) {
            uint64_t v = wsum[threadIdx.x];
            for (int o = 1; o < 32; o <<= 1) {
                const uint64_t u = __shfl_up_sync(0xffffffffu, v, o);
                if (threadIdx.x >= o) v += u;
            }
            wsum[threadIdx.x] = v;
        }
        __syncthreads();
        const uint64_t pre = carry + ((threadIdx.x >> 5) ? wsum[(threadIdx.x >> 5) - 1] : 0) + incl - words;
        if (c < s.nchunks) chunk_word_off[s.chunk_base + c] = pre;
        __syncthreads();
        if (threadIdx.x == 0) carry += wsum[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        chunk_word_off[s.chunk_base + s.nchunks] = carry;
        stream_words[blockIdx.x] = carry;
    }
    __syncthreads();  // every chunk offset is written
    // four planes per thread in flight (one block per stream: the loop is
    // latency-bound)
    const uint64_t np = (uint64_t)s.nchunks * C;
    for (uint64_t p0 = threadIdx.x; p0 < np; p0 += 4 * (uint64_t)blockDim.x) {
        uint32_t b0[4], nb[4];
        uint64_t cw[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint64_t p = p0 + (uint64_t)j * blockDim.x;
            nb[j] = 0;
            if (p < np) {
                const size_t k = s.sub_base + p;
                b0[j] = sub_off[k];
                nb[j] = sub_bits[k];
                cw[j] = chunk_word_off[s.chunk_base + p / C];
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (nb[j]) {
                uint32_t* w = payload + s.word_base + cw[j];
                w[b0[j] >> 5] = 0;
                w[(b0[j] + nb[j] - 1) >> 5] = 0;
            }
    }
}

// Encode: a warp packs one plane MSB-first, each lane its own bits from the
// plane's offset plus the bits of the lanes before it. The plane's first and
// last words (shared with its neighbours, cleared by k_scan_stream) and each
// lane's first and last words are merged with atomicOr; the warp clears the
// plane's inner words first, and words inside one lane's range are stored.
__global__ void __launch_bounds__(kLaneThreads) k_encode(const CtaWork* __restrict__ work,
                                                         const uint32_t* __restrict__ chunk_ids,
                                                         const StreamDesc* __restrict__ sd,
                                                         const uint16_t* __restrict__ codes,
                                                         const uint32_t* __restrict__ ctab,
                                                         const uint8_t* __restrict__ rbits,
                                                         const uint32_t* __restrict__ sub_bits,
                                                         const uint32_t* __restrict__ sub_off,
                                                         const uint64_t* __restrict__ chunk_word_off,
                                                         uint32_t* __restrict__ payload)
{
    const CtaWork w = work[blockIdx.x];
    const StreamDesc s = sd[w.stream];
    const uint32_t C = s.C, P = C * C, W = lanes_per_plane(P), np = w.count * C;
    const uint32_t* tab = ctab + (size_t)w.stream * 2 * s.radius;
    if (s.run_n && lits_ok(P, W)) {
        // literal rounds: each literal's bits (its run's, then its own) placed
        // by a group scan, written into a shared staging copy of the plane's
        // words aligned as in the chunk; then the inner words are stored and
        // the first and last (shared with the neighbouring planes) merged
        __shared__ uint16_t lists[kLaneThreads / 32][kListPerWarp];
        __shared__ uint32_t stage[kLaneThreads / 32][kStagePerWarp];
        const uint32_t gi = (threadIdx.x & 31) / W;
        uint16_t* list = lists[threadIdx.x >> 5] + gi * 32 * W;
        uint32_t* stg = stage[threadIdx.x >> 5] + gi * (24 * W + 2);
        const uint8_t* rb = rbits + (size_t)w.stream * kRunBitsStride;
        uint32_t D, LD;
        const uint32_t J = run_geometry(P, D, LD);
        auto put = [&](uint32_t e, uint32_t& p) {  // e = code << 5 | length, MSB first at bit p
            const uint32_t l = e & 31u, v = e >> 5, o = p & 31u, wi = p >> 5;
            if (!l) return;
            if (o + l <= 32) {
                atomicOr(stg + wi, v << (32 - o - l));
            } else {
                atomicOr(stg + wi, v >> (o + l - 32));
                atomicOr(stg + wi + 1, v << (64 - o - l));
            }
            p += l;
        };
        STZ_GROUP_PLANES(np, W)
        {
            STZ_GROUP_PLANE(np, W);
            const uint32_t c = chunk_ids[w.first + pe / C], lz = pe % C;
            const uint16_t* src = codes + s.code_off + (size_t)c * P * C + (size_t)lz * P;
            const LaneSeg g = lane_seg(C, src, W, active);
            const uint32_t L = plane_literals(src, g, s.radius, list);
            const size_t k = s.sub_base + (size_t)c * C + lz;
            const uint32_t b0 = sub_off[k], nb = active ? sub_bits[k] : 0u;
            const uint32_t nw = ((b0 & 31u) + nb + 31u) >> 5;
            for (uint32_t x = g.lane; x < nw; x += W) stg[x] = 0;
            __syncwarp();
            uint32_t at = b0 & 31u;  // the group's next bit in the staging words
            literal_rounds2(list, L, g, [&](bool v0, uint32_t pos0, uint32_t run0, bool v1, uint32_t pos1, uint32_t run1) {
                const uint32_t q0 = v0 ? __ldg(src + pos0) : 0u, q1 = v1 ? __ldg(src + pos1) : 0u;
                uint32_t e0 = 0, e1 = 0, len0 = 0, len1 = 0;
                if (v0) {
                    e0 = __ldg(tab + q0);
                    len0 = __ldg(rb + run0) + (e0 & 31u);
                }
                if (v1) {
                    e1 = __ldg(tab + q1);
                    len1 = __ldg(rb + run1) + (e1 & 31u);
                }
                const uint32_t len = len0 + len1;
                const uint32_t incl = group_scan(len, W, g.lane);
                uint32_t p = at + incl - len;
                at += __shfl_sync(0xffffffffu, incl, W - 1, W);
                auto sym_put = [&](uint32_t sym) { put(__ldg(tab + sym), p); };
                if (v0) {
                    run_symbols(run0, s.radius, s.run_base, J, D, LD, sym_put);
                    put(e0, p);
                }
                if (v1) {
                    run_symbols(run1, s.radius, s.run_base, J, D, LD, sym_put);
                    put(e1, p);
                }
            });
            if (active && g.lane == 0) {
                uint32_t p = at;
                run_symbols(tail_run(list, L, P), s.radius, s.run_base, J, D, LD,
                            [&](uint32_t sym) { put(__ldg(tab + sym), p); });
            }
            __syncwarp();
            if (active && nb) {
                uint32_t* out = payload + s.word_base + chunk_word_off[s.chunk_base + c] + (b0 >> 5);
                for (uint32_t x = g.lane; x < nw; x += W) {
                    const uint32_t v = stg[x];
                    if (x == 0 || x == nw - 1) atomicOr(out + x, v);
                    else out[x] = v;
                }
            }
            __syncwarp();  // list and staging are rewritten for the next plane
        }
        return;
    }
    STZ_GROUP_PLANES(np, W)
    {
        STZ_GROUP_PLANE(np, W);
        const uint32_t c = chunk_ids[w.first + pe / C], lz = pe % C;
        const uint16_t* src = codes + s.code_off + (size_t)c * P * C + (size_t)lz * P;
        const LaneSeg g = lane_seg(C, src, W, active);
        RunLane rl;
        if (s.run_n) rl.init(src, g, s.radius);
        auto each = [&](auto&& f) {
            if (s.run_n) rl.symbols(src, g, s, f);
            else lane_codes(src, g, f);
        };
        uint32_t bits = 0;
        each([&](uint32_t sym) { bits += __ldg(tab + sym) & 31u; });
        uint32_t off = group_scan(bits, W, g.lane);  // inclusive -> this lane's first bit in the plane
        const uint32_t nb = __shfl_sync(0xffffffffu, off, W - 1, W);
        off -= bits;
        uint32_t* out = payload + s.word_base + chunk_word_off[s.chunk_base + c];
        const uint32_t b0 = sub_off[s.sub_base + (size_t)c * C + lz];
        if (active && nb)
            for (uint32_t x = (b0 >> 5) + 1 + g.lane; x < (b0 + nb - 1) >> 5; x += W) out[x] = 0;
        __syncwarp();
        if (active && bits) {
            const uint32_t pos = b0 + off;
            const uint32_t first_w = pos >> 5, last_w = (pos + bits - 1) >> 5;
            uint32_t wi = first_w;
            uint64_t acc = 0;            // pending bits, right-aligned
            int nacc = (int)(pos & 31);  // leading bits of the first word belong to earlier lanes (zeros here)
            each([&](uint32_t sym) {
                const uint32_t e = __ldg(tab + sym);
                const int l = e & 31;
                acc = (acc << l) | (e >> 5);
                nacc += l;
                if (nacc >= 32) {
                    const uint32_t word = (uint32_t)(acc >> (nacc - 32));
                    nacc -= 32;
                    if (wi == first_w || wi == last_w) atomicOr(out + wi, word);
                    else out[wi] = word;
                    ++wi;
                }
            });
            if (nacc > 0) atomicOr(out + wi, (uint32_t)(acc << (32 - nacc)));
        }
        __syncwarp();
    }
}

// ---- decode: a lane group per plane ----------------------------------------------
// Parallel Huffman decoding by self-synchronisation (Weissenberger & Schmidt,
// "Massively parallel Huffman decoding on GPUs", ICPP 2018): a plane's bits
// are cut into W slices; lane i decodes the codes that start in its slice,
// beginning at the slice start. A lane whose start is not where its left
// neighbour's last code ends decodes again from there, until no start moves
// (codes resynchronise within 5 to 20 symbols, so one to five rounds are
// usual). A scan of the lanes' code counts (a run symbol counts its run) then
// places each lane's literals.
// A symbol is decoded about three times, so the kernel is bound by the
// instructions and the latency of that step, and everything it reads lies in
// shared memory: the stream's table, the plane's payload words (copied there
// first, asynchronously), and the plane's codes, which start out as centre
// codes, take the literals, and are stored at the end, 16 bytes a lane.
//   * One lookup gives the length of any code but the few whose table prefix
//     spans two lengths: canonical codes of one length are one interval. A
//     code of up to kLutBits bits also gets its symbol or run length, a
//     longer one its canonical index. For those few the entry says where the
//     search through the lengths starts, which then ends within a step or two.
//   * The counting passes, two thirds of the steps, take only the length and
//     the run length from the entry.
//   * The symbols of longer codes are looked up when the plane is stored,
//     many at a time, so no lane waits for one in the middle of its chain.
//     Where long codes are common (DecodeTables::by_index) the plane holds
//     indexes only.
// Before, table, payload words and symbols were read through L1 in the chain,
// the length of a long code was searched there, and dense streams of large
// launches had one thread per plane (below, in today's form). Launch times on one
// B200, then and now (levels below the finest and its two halves together):
//   512^3 f32 at 1e-3          0.430 -> 0.338 ms
//   512^3 f32 at 1e-4          1.968 -> 0.687 ms
//   384x384x256 f64 at 1e-6    1.310 -> 0.464 ms (its halves stay below plane_items' line)
//   its boxes of 16-128 a side 0.156 -> 0.048 ms a box
// (With one step function for counting and placing, the search from kLutBits
// up and through L1, and one build for launches of all sizes: 0.41, 0.86, 0.56
// and 0.068 ms.)
// Tried as well: one lane per plane in lockstep for all streams (windows of
// codes in shared memory, payload rings filled by asynchronous copies), 0.17 /
// 0.62 / 0.42 ms at 1e-4 and a chain of 1024 symbols in every small launch; several symbols
// per lookup in the counting passes (fewer instructions, more table to load:
// even); four lanes' worth of planes per warp for all streams (fewer warps
// resident: slower); only the planes that a box needs, as work items of equal
// plane ranges (a box's decode is the chain of the one plane that each of its
// warps has, which fewer planes do not shorten: even).

// lut entry: code length in bits 0-4 (0: the prefix spans lengths, holds long
// run symbols, or no code; bits 16-31 then hold the shortest length above
// kLutBits that a code under it may have); kLutRun: a run symbol, its run length in
// bits 16-31; kLutLong: a longer code, its canonical index is its value plus
// bits 16-31 (mod 2^16); else the symbol in bits 16-31 (its canonical index
// where the stream decodes by index).
constexpr uint32_t kLutRun = 0x100u, kLutLong = 0x200u;
constexpr uint32_t kNoIndex = 0xffffu;  // a plane's entry without a literal, where the stream decodes by index
struct DecodeTables {
    uint32_t lut[1 << kLutBits];
    // per code length: limit (codes of up to that length lie below it, as
    // left-aligned kMaxCodeLen-bit numbers), the canonical index of a code
    // minus its value, the first index of its run symbols, and their count
    // (bits 0-15) and place in run (bits 16-31)
    uint4 len[kMaxCodeLen + 1];
    uint16_t run[64];   // run lengths, in canonical order
    uint32_t max_len;   // longest code
    uint32_t by_index;  // decode canonical indexes, look symbols up at the store
};

constexpr int kBuildThreads = 512;

// One CTA per stream.
__global__ void __launch_bounds__(kBuildThreads) k_build_tables(const StreamDesc* __restrict__ sd,
                                                                const uint16_t* __restrict__ cb_sym,
                                                                const uint8_t* __restrict__ cb_len,
                                                                DecodeTables* __restrict__ out)
{
    const StreamDesc s = sd[blockIdx.x];
    DecodeTables& t = out[blockIdx.x];
    __shared__ uint32_t cnt[kMaxCodeLen + 1], first_code[kMaxCodeLen + 1], first_idx[kMaxCodeLen + 1];
    __shared__ uint32_t start[kMaxCodeLen + 1];  // first index of each length (the list is in length order)
    __shared__ uint32_t rlo[kMaxCodeLen + 1], rcnt[kMaxCodeLen + 1], roff[kMaxCodeLen + 1];
    __shared__ uint32_t by_index, longest;
    const uint32_t tid = threadIdx.x;
    if (tid <= kMaxCodeLen) start[tid] = 0xffffffffu, rlo[tid] = 0xffffffffu, rcnt[tid] = 0;
    __syncthreads();
    uint32_t D, LD;
    run_geometry(s.C * s.C, D, LD);
    for (uint32_t i = tid; i < s.n_used; i += kBuildThreads) {
        const uint32_t l = cb_len[s.cb_off + i];
        if (i == 0 || cb_len[s.cb_off + i - 1] != l) start[l] = i;
        if ((uint32_t)cb_sym[s.cb_off + i] - s.run_base < s.run_n) {
            atomicMin(&rlo[l], i);
            atomicAdd(&rcnt[l], 1u);
        }
    }
    __syncthreads();
    if (tid == 0) {
        for (int l = kMaxCodeLen, end = (int)s.n_used; l >= 0; --l) {
            cnt[l] = start[l] == 0xffffffffu ? 0u : (uint32_t)end - start[l];
            if (cnt[l]) end = (int)start[l];
        }
        uint32_t code = 0, idx = cnt[0], ro = 0, mass = 0;
        longest = 0;
        first_code[0] = first_idx[0] = roff[0] = 0;
        for (int l = 1; l <= kMaxCodeLen; ++l) {
            code = (code + (l > 1 ? cnt[l - 1] : 0)) << 1;
            first_code[l] = code;
            first_idx[l] = idx;
            idx += cnt[l];
            roff[l] = ro;
            ro += rcnt[l];
            if (cnt[l]) longest = l;
            if (l <= kLutBits) mass += cnt[l] << (kLutBits - l);
        }
        t.max_len = longest;
        // more than one symbol in 128 has a long code; with run symbols an
        // entry can stay without a literal, so kNoIndex must not be an index
        by_index = t.by_index = (1u << kLutBits) - mass > (1u << kLutBits) / 128 && longest > kLutBits &&
                                (s.run_n == 0 || s.n_used <= kNoIndex);
    }
    __syncthreads();
    if (tid <= kMaxCodeLen)
        t.len[tid] = make_uint4(tid ? (first_code[tid] + cnt[tid]) << (kMaxCodeLen - tid) : 0u,
                                first_idx[tid] - first_code[tid], rlo[tid], rcnt[tid] | roff[tid] << 16);
    // run lengths in canonical order: run symbols of one length are consecutive
    for (uint32_t i = tid; i < s.n_used; i += kBuildThreads) {
        const uint32_t r = (uint32_t)cb_sym[s.cb_off + i] - s.run_base;
        if (r < s.run_n) {
            const uint32_t l = cb_len[s.cb_off + i];
            t.run[roff[l] + i - rlo[l]] = (uint16_t)run_length(r, D, LD);
        }
    }
    // the shortest length whose canonical range holds the entry's prefix, or
    // the one longer length all codes under the prefix have
    for (uint32_t j = tid; j < (1u << kLutBits); j += kBuildThreads) {
        uint32_t e = 0;
        for (uint32_t l = 1; l <= (uint32_t)kMaxCodeLen && !e; ++l) {
            if (l <= (uint32_t)kLutBits) {
                const uint32_t v = (j >> (kLutBits - l)) - first_code[l];
                if (v < cnt[l]) {
                    const uint32_t i = first_idx[l] + v, sym = cb_sym[s.cb_off + i], r = sym - s.run_base;
                    e = l | (r < s.run_n ? kLutRun | run_length(r, D, LD) << 16 : (by_index ? i : sym) << 16);
                }
            } else {
                const uint32_t sh = l - kLutBits, lo = j << sh, hi = lo + (1u << sh) - 1, b = first_idx[l] - first_code[l];
                if (lo >= first_code[l] && hi < first_code[l] + cnt[l] &&
                    (!rcnt[l] || hi + b < rlo[l] || lo + b >= rlo[l] + rcnt[l]))
                    e = l | kLutLong | b << 16;
            }
        }
        if (!e) {  // as DecodeCtx::slow looks for the prefix's first code
            uint32_t l = kLutBits + 1;
            while (l <= longest && j << (kMaxCodeLen - kLutBits) >= (first_code[l] + cnt[l]) << (kMaxCodeLen - l)) ++l;
            e = l << 16;
        }
        t.lut[j] = e;
    }
}

constexpr int kDecodeWarps = 8;
constexpr int kDecodeThreads = 32 * kDecodeWarps;
constexpr uint32_t kMaxPlane = 1024;    // planes of up to this many codes fit the shared buffers
constexpr uint32_t kStageWords = 512;   // payload words of the planes a warp decodes at a time

struct DecodeSmem {
    uint32_t lut[1 << kLutBits];
    uint4 out[kDecodeWarps][kMaxPlane / 8];
    uint4 stage[kDecodeWarps][kStageWords / 4];
    uint32_t late[kDecodeWarps][kMaxPlane / 32];  // entries that hold the index of a long code
    uint4 len[kMaxCodeLen + 1];                   // as DecodeTables
    uint32_t max_len;
};

// Symbol decoding from a stream's tables, those of each code in shared memory.
struct DecodeCtx {
    const uint32_t* lut;
    const uint4* len;
    uint32_t longest;
    const DecodeTables* __restrict__ t;
    __device__ __forceinline__ uint32_t entry(uint32_t bits) const
    {
        return lut[bits >> (32 - kLutBits)];
    }
    // The code at the top of bits: its length, and symbol or run length, or
    // canonical index (late).
    __device__ __forceinline__ void symbol(uint32_t bits, uint32_t& l, uint32_t& val, bool& run, bool& late) const
    {
        const uint32_t e = entry(bits);
        l = e & 31u, val = e >> 16, run = e & kLutRun, late = e & kLutLong;
        if (late) val = (bits >> (32 - l)) + val & 0xffffu;
        if (l == 0) slow(bits, l, val, run, late);
    }
    // Its length, and how many codes it stands for.
    __device__ __forceinline__ void count(uint32_t bits, uint32_t& l, uint32_t& n) const
    {
        const uint32_t e = entry(bits);
        l = e & 31u, n = e & kLutRun ? e >> 16 : 1u;
        if (l == 0) {
            uint32_t val = e >> 16;
            bool run, late;
            slow(bits, l, val, run, late);
            n = run ? val : 1u;
        }
    }
    // val: the length to start from.
    __device__ __forceinline__ void slow(uint32_t bits, uint32_t& l, uint32_t& val, bool& run, bool& late) const
    {
        const uint32_t v = bits >> (32 - kMaxCodeLen);
        l = val;
        while (l <= longest && v >= len[l].x) ++l;
        run = false, late = true;
        if (l > longest) {  // no code (corrupt stream): the codebook's first symbol, one bit
            l = 1;
            val = 0;
            return;
        }
        const uint4 e = len[l];
        const uint32_t i = (bits >> (32 - l)) + e.y, r = i - e.z;
        run = r < (e.w & 0xffffu);
        val = run ? __ldg(&t->run[(e.w >> 16) + r]) : i;
    }
};

// 32 bits of a plane from any bit position; the words lie in shared or in
// global memory, and at least two more follow every plane's in the same
// buffer (a stream keeps four words after its payload).
template <class Words>
__device__ __forceinline__ uint32_t peek(const Words& w, uint32_t pos)
{
    return __funnelshift_l(w((pos >> 5) + 1), w(pos >> 5), pos);
}

// Decode the plane of bits [r0, r1) by this lane's group of W lanes: the
// literals go to put(code, value, late).
template <class Words, class Put>
__device__ __forceinline__ void decode_plane(const DecodeCtx& dc, const Words& w, uint32_t r0, uint32_t r1, uint32_t W,
                                             uint32_t lane, Put&& put)
{
    const uint32_t nb = r1 - r0, L = (nb + W - 1) / W;
    const uint32_t stop = r0 + min(nb, (lane + 1) * L);
    uint32_t start = r0 + min(nb, lane * L), end = start, cnt = 0;
    auto count = [&]() {
        cnt = 0;
        while (end < stop) {
            uint32_t l, n;
            dc.count(peek(w, end), l, n);
            cnt += n;
            end += l;
        }
    };
    count();
    for (uint32_t round = 0; round < W; ++round) {
        uint32_t prev = __shfl_up_sync(0xffffffffu, end, 1, W);
        if (lane == 0) prev = r0;
        const bool moved = prev != start;
        if (!__any_sync(0xffffffffu, moved)) break;
        if (moved) {
            start = end = prev;
            count();
        }
    }
    uint32_t q = group_scan(cnt, W, lane) - cnt;  // first code of this lane
    while (start < stop) {
        uint32_t l, val;
        bool run, late;
        dc.symbol(peek(w, start), l, val, run, late);
        if (!run) put(q, val, late);
        q += run ? val : 1u;
        start += l;
    }
}

// Lanes per plane: as many as leave a lane about 32 codes.
__device__ __forceinline__ uint32_t decode_lanes(uint32_t P)
{
    uint32_t W = 1;
    while (W < 32 && 32 * W < P) W *= 2;
    return W;
}

// One plane's place: its bits in the payload words from the 16-byte group it
// starts in, and its codes.
struct PlaneAt {
    const uint32_t* src;
    uint16_t* dst;
    uint32_t r0, r1;
};
__device__ __forceinline__ PlaneAt plane_at(const StreamDesc& s, const uint32_t* __restrict__ chunks, uint32_t p,
                                            bool active, const uint32_t* __restrict__ sub_off,
                                            const uint64_t* __restrict__ chunk_word_off,
                                            const uint32_t* __restrict__ payload, uint16_t* __restrict__ codes)
{
    const uint32_t C = s.C, P = C * C, pc = p / C, lz = p - pc * C, c = chunks[pc];
    const uint64_t cw = chunk_word_off[s.chunk_base + c];
    const uint32_t b0 = sub_off[s.sub_base + (size_t)c * C + lz];
    const uint32_t b1 = lz + 1 < C ? sub_off[s.sub_base + (size_t)c * C + lz + 1]
                                   : (uint32_t)(32 * (chunk_word_off[s.chunk_base + c + 1] - cw));
    const uint64_t w0 = s.word_base + cw + (b0 >> 5);
    PlaneAt a;
    a.src = payload + (w0 & ~3ull);
    a.dst = codes + s.code_off + (size_t)c * P * C + (size_t)lz * P;
    a.r0 = ((uint32_t)(w0 & 3) << 5) + (b0 & 31);
    a.r1 = a.r0 + (active && s.n_used != 1 && b1 > b0 ? b1 - b0 : 0u);  // a lone symbol has no bits
    return a;
}

// Half a warp decodes a plane of a stream with fewer payload bits per plane
// than this on average, in launches of at least kHalfWarpItems items: each
// lane then takes twice the bits, and the rounds and scans cost half as much
// per symbol (512^3 f32 at 1e-3, ~600 bits per plane, the finest level's
// halves: 0.18 + 0.14 -> 0.16 + 0.12 ms). Two planes of 1024 codes do not fit
// the warp's buffer: centre codes go to global memory first and literals over
// them. Smaller launches are bound by latency and take all 32 lanes.
constexpr uint32_t kHalfWarpBits = 2048;
constexpr int kHalfWarpItems = 128;

// A code without a literal: the centre code; a lone symbol that is not a run
// fills the plane itself.
__device__ __forceinline__ uint32_t fill_code(const StreamDesc& s, const uint16_t* __restrict__ syms)
{
    return s.n_used == 1 && (uint32_t)syms[0] - s.run_base >= s.run_n ? (uint32_t)syms[0] : s.radius;
}

// Payload and table in shared memory, and the codes too where the warp's
// planes fit its buffer: then only final values are stored, each once.
__device__ __forceinline__ void decode_buffered(DecodeSmem& sm, const StreamDesc& s,
                                                const DecodeTables* __restrict__ t, uint32_t W,
                                                const uint32_t* __restrict__ chunks, uint32_t np, uint32_t first,
                                                uint32_t nwarps, const uint16_t* __restrict__ cb_sym,
                                                const uint32_t* __restrict__ sub_off,
                                                const uint64_t* __restrict__ chunk_word_off,
                                                const uint32_t* __restrict__ payload, uint16_t* __restrict__ codes)
{
    const uint32_t P = s.C * s.C, G = 32 / W, wid = threadIdx.x >> 5, all = threadIdx.x & 31;
    if (first * G >= np) return;  // uniform per warp; nothing below waits for the other warps
    const bool direct = G * P > kMaxPlane;
    const uint32_t lane = all & (W - 1), gi = all / W;
    const uint16_t* __restrict__ syms = cb_sym + s.cb_off;
    const bool by_index = t->by_index;
    const uint32_t f2 = (by_index && !direct ? kNoIndex : fill_code(s, syms)) * 0x10001u;
    const uint4 f4 = make_uint4(f2, f2, f2, f2);
    const uint32_t Pc = (P + 7) & ~7u;      // codes of a group's share of the buffer (G * Pc <= kMaxPlane)
    const uint32_t cap = kStageWords / G;   // payload words of it
    uint4* const out = sm.out[wid] + gi * (Pc / 8);
    uint16_t* const out16 = reinterpret_cast<uint16_t*>(out);
    uint4* const stage = sm.stage[wid] + gi * (cap / 4);
    uint32_t* const late = sm.late[wid];
    if (!direct) {
        for (uint32_t k = all; k < kMaxPlane / 8; k += 32) sm.out[wid][k] = f4;
        late[all] = 0;
    }
    __syncwarp();
    const DecodeCtx dc{sm.lut, sm.len, sm.max_len, t};
    for (uint32_t base = first * G; base < np; base += nwarps * G) {
        const bool active = base + gi < np;
        const PlaneAt a = plane_at(s, chunks, active ? base + gi : base, active, sub_off, chunk_word_off, payload, codes);
        bool any_late = false;
        auto put = [&](uint32_t q, uint32_t val, bool lt) {
            if (q >= P) return;  // corrupt stream
            if (direct) {
                a.dst[q] = lt || by_index ? __ldg(syms + val) : (uint16_t)val;
                return;
            }
            out16[q] = (uint16_t)val;
            if (lt && !by_index) {
                const uint32_t x = gi * Pc + q;
                atomicOr(&late[x >> 5], 1u << (x & 31));
                any_late = true;
            }
        };
        const uint32_t nw = a.r1 > a.r0 ? ((a.r1 + 31) >> 5) + 2 : 0u;
        const bool vec = P % 8 == 0 && ((uintptr_t)a.dst & 15) == 0;
        if (direct) {
            if (active && vec)
                for (uint32_t k = lane; k < P / 8; k += W) reinterpret_cast<uint4*>(a.dst)[k] = f4;
            else if (active)
                for (uint32_t k = lane; k < P; k += W) a.dst[k] = (uint16_t)f2;
            __syncwarp();
        }
        if (__all_sync(0xffffffffu, nw <= cap)) {
            const uint32_t at = (uint32_t)__cvta_generic_to_shared(stage);
            for (uint32_t k = lane; k < (nw + 3) / 4; k += W)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(at + k * 16), "l"(a.src + 4 * k)
                             : "memory");
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncwarp();
            const uint32_t* const sw = reinterpret_cast<const uint32_t*>(stage);
            decode_plane(dc, [&](uint32_t i) { return sw[i]; }, a.r0, a.r1, W, lane, put);
        } else {
            decode_plane(dc, [&](uint32_t i) { return __ldg(a.src + i); }, a.r0, a.r1, W, lane, put);
        }
        __syncwarp();
        if (direct) continue;
        any_late = __any_sync(0xffffffffu, any_late);
        // the planes to global memory, the buffer back to its empty state
        for (uint32_t k = lane; k < Pc / 8; k += W) {
            const uint4 v = out[k];
            out[k] = f4;
            if (!active) continue;
            uint32_t x[4] = {v.x, v.y, v.z, v.w};
            if (by_index) {
                auto sym = [&](uint32_t i) -> uint32_t { return i < s.n_used ? __ldg(syms + i) : s.radius; };
#pragma unroll
                for (int j = 0; j < 4; ++j) x[j] = sym(x[j] & 0xffffu) | sym(x[j] >> 16) << 16;
            } else if (any_late) {
                const uint32_t m = late[(gi * Pc + 8 * k) >> 5] >> ((gi * Pc + 8 * k) & 31) & 0xffu;
                if (m)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (m >> (2 * j) & 1u) x[j] = (x[j] & 0xffff0000u) | __ldg(syms + (x[j] & 0xffffu));
                        if (m >> (2 * j + 1) & 1u) x[j] = (x[j] & 0xffffu) | (uint32_t)__ldg(syms + (x[j] >> 16)) << 16;
                    }
            }
            if (vec) {
                *reinterpret_cast<uint4*>(a.dst + 8 * k) = make_uint4(x[0], x[1], x[2], x[3]);
            } else {
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j)
                    if (8 * k + j < P) a.dst[8 * k + j] = (uint16_t)(x[j >> 1] >> (16 * (j & 1)));
            }
        }
        __syncwarp();
        if (any_late) late[all] = 0;
        __syncwarp();
    }
}

// The stream's table into shared memory (the whole CTA; a barrier before the
// old one is overwritten and one after).
__device__ __forceinline__ void load_table(DecodeSmem& sm, const DecodeTables* __restrict__ t)
{
    __syncthreads();
    const uint4* __restrict__ src = reinterpret_cast<const uint4*>(t->lut);
    for (uint32_t i = threadIdx.x; i < (1u << kLutBits) / 4; i += kDecodeThreads)
        reinterpret_cast<uint4*>(sm.lut)[i] = __ldg(src + i);
    if (threadIdx.x <= kMaxCodeLen) sm.len[threadIdx.x] = __ldg(t->len + threadIdx.x);
    if (threadIdx.x == 0) sm.max_len = t->max_len;
    __syncthreads();
}

// ---- decode: a thread per plane ---------------------------------------------------
// In large launches a plane of a stream without run symbols is one thread's:
// it decodes each code once, where a lane group decodes it about three times,
// and the lanes of a warp write the same code of their planes in step. Bound by
// the instructions of that step, with the plane's chain of codes as the least
// time a launch takes, hence plane_items' rule on the number of items. The
// table and the payload words lie in shared memory as above; the words are
// fetched ahead by the same instruction for all lanes, since a load or a copy
// that only some lanes issue makes the warp wait for it at the next one's use
// (0.53 us a step with asynchronous copies per lane, 0.17 so). Where codes are
// indexes, eight symbols are looked up together when they are stored.
// k_decode, lane groups and now (levels below the finest and its two halves;
// everything in one launch): 512^3 f32 GRF at 1e-2 0.74 -> 0.43; 0.65 -> 0.35
// ms, at 1e-4 0.92 -> 0.70; 0.82 -> 0.57; 1024^3 at 1e-3 5.40 -> 2.65; 5.03 ->
// 2.40. (A thread per plane through L1, as before the lane groups took all:
// 0.98; 0.49, 1.18; 0.72, 3.63; 3.01.) Run symbols bring the lanes out of step:
// fields with them took 0.58 -> 0.74 (512^3 f32 lognormal at 1e-4, one launch).
constexpr int kPlaneThreads = kCoderThreads;
constexpr uint32_t kRingWords = 32;  // payload words at hand of each thread
struct PlaneSmem {
    uint32_t lut[1 << kLutBits];
    uint4 len[kMaxCodeLen + 1];
    uint32_t ring[kRingWords][kPlaneThreads];
    uint32_t max_len;
};

// A plane's bits in order. The words come through a ring in shared memory, two
// 16-byte groups at a time, fetched and put into it by refill() every eight
// symbols (which take six words at most): eleven words or more are always left.
struct PlaneBits {
    const uint4* __restrict__ src;
    uint32_t (*ring)[kPlaneThreads];
    uint32_t last;     // group that holds the word after the plane's last one
    uint32_t fetched;  // groups in the ring so far
    uint32_t wi;       // the word after next
    uint64_t buf;      // the next bits on top, `have` >= 32 of them; next follows them
    uint32_t next;
    int have;
    uint4 f0, f1;
    bool flying;

    __device__ __forceinline__ uint32_t word(uint32_t i) const { return ring[i % kRingWords][threadIdx.x]; }
    __device__ __forceinline__ void put(uint32_t k, const uint4& v)
    {
        const uint32_t i = 4 * k % kRingWords, t = threadIdx.x;
        ring[i][t] = v.x, ring[i + 1][t] = v.y, ring[i + 2][t] = v.z, ring[i + 3][t] = v.w;
    }
    __device__ __forceinline__ void init(const PlaneAt& a)
    {
        src = reinterpret_cast<const uint4*>(a.src);
        last = (((a.r1 + 31) >> 5) + 1) >> 2;
        fetched = kRingWords / 4 - 2;
#pragma unroll
        for (uint32_t k = 0; k < kRingWords / 4 - 2; ++k) put(k, __ldg(src + min(k, last)));
        wi = a.r0 >> 5;
        buf = ((uint64_t)word(wi) << 32 | word(wi + 1)) << (a.r0 & 31);
        next = word(wi + 2);
        wi += 3;
        have = 64 - (int)(a.r0 & 31);
        flying = false;
    }
    __device__ __forceinline__ void refill()
    {
        if (flying) {
            put(fetched, f0), put(fetched + 1, f1);
            fetched += 2;
        }
        flying = fetched <= last && fetched + 2 - (wi >> 2) <= kRingWords / 4;
        if (flying) f0 = __ldg(src + fetched), f1 = __ldg(src + min(fetched + 1, last));
    }
    __device__ __forceinline__ uint32_t top() const { return (uint32_t)(buf >> 32); }
    __device__ __forceinline__ void skip(uint32_t l)
    {
        buf <<= l;
        have -= (int)l;
        if (have < 32) {
            buf |= (uint64_t)next << (32 - have);
            have += 32;
            next = word(wi++);
        }
    }
};

// The symbols of those of eight codes that are indexes (bit j of m: code j).
__device__ __forceinline__ void look_up(uint32_t (&x)[4], uint32_t m, const uint16_t* __restrict__ syms)
{
    uint32_t y[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (m >> j & 1u) y[j] = __ldg(syms + (x[j >> 1] >> (16 * (j & 1)) & 0xffffu));
#pragma unroll
    for (int j = 0; j < 8; ++j)
        if (m >> j & 1u) x[j >> 1] = j & 1 ? (x[j >> 1] & 0xffffu) | y[j] << 16 : (x[j >> 1] & 0xffff0000u) | y[j];
}

// Planes of the listed chunks, a thread each; items of plane_items only.
__global__ void __launch_bounds__(kPlaneThreads, 6)
    k_decode_planes(const CtaWork* __restrict__ work, const uint32_t* __restrict__ chunk_ids,
                    const StreamDesc* __restrict__ sd, const DecodeTables* __restrict__ tabs,
                    const uint16_t* __restrict__ cb_sym, const uint32_t* __restrict__ sub_off,
                    const uint64_t* __restrict__ chunk_word_off, const uint32_t* __restrict__ payload,
                    uint16_t* __restrict__ codes)
{
    __shared__ __align__(16) PlaneSmem sm;
    const CtaWork w = work[blockIdx.x];
    const StreamDesc s = sd[w.stream];
    const DecodeTables* __restrict__ t = tabs + w.stream;
    {
        const uint4* __restrict__ src = reinterpret_cast<const uint4*>(t->lut);
        for (uint32_t i = threadIdx.x; i < (1u << kLutBits) / 4; i += kPlaneThreads)
            reinterpret_cast<uint4*>(sm.lut)[i] = __ldg(src + i);
        if (threadIdx.x <= kMaxCodeLen) sm.len[threadIdx.x] = __ldg(t->len + threadIdx.x);
        if (threadIdx.x == 0) sm.max_len = t->max_len;
    }
    const uint16_t* __restrict__ syms = cb_sym + s.cb_off;
    const uint32_t all = t->by_index ? 0xffu : 0u;
    const uint32_t f2 = fill_code(s, syms) * 0x10001u;
    const uint4 f4 = make_uint4(f2, f2, f2, f2);
    __syncthreads();
    const DecodeCtx dc{sm.lut, sm.len, sm.max_len, t};
    const uint32_t P = s.C * s.C;
    if (threadIdx.x >= w.count * s.C) return;
    const PlaneAt a = plane_at(s, chunk_ids + w.first, threadIdx.x, true, sub_off, chunk_word_off, payload, codes);
    uint4* const out = reinterpret_cast<uint4*>(a.dst);
    if (a.r1 == a.r0) {  // a lone symbol has no bits
        for (uint32_t g = 0; g < P / 8; ++g) out[g] = f4;
        return;
    }
    PlaneBits b;
    b.ring = sm.ring;
    b.init(a);
    for (uint32_t g = 0; g < P / 8; ++g) {
        b.refill();
        uint32_t x[4], m = all;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t top = b.top(), e = sm.lut[top >> (32 - kLutBits)];
            uint32_t l = e & 31u, val = e >> 16;
            if ((e & (kLutLong | 31u)) - 1u >= 31u) {  // no plain entry: an index
                bool run, late;
                if (l) val = (top >> (32 - l)) + val & 0xffffu;
                else dc.slow(top, l, val, run, late);
                m |= 1u << j;
            }
            b.skip(l);
            x[j >> 1] = j & 1 ? x[j >> 1] | val << 16 : val;
        }
        if (m) look_up(x, m, syms);
        out[g] = make_uint4(x[0], x[1], x[2], x[3]);
    }
}

// CTAs that share a work item: a plane per warp, down to a few per warp in
// the largest launches. Short CTAs balance better than they pay for loading
// the table (finest level's halves, 448 items, 512^3 f32 at 1e-4: 0.63 + 0.51
// ms with one CTA an item, 0.56 + 0.41 with four, 0.50 + 0.32 with eight).
__host__ __device__ inline uint32_t decode_slices(uint32_t nwork)
{
    uint32_t S = 16;
    while (S > 1 && (uint64_t)nwork * S > 148 * 48) S /= 2;
    return S;
}

// Planes of the listed chunks: CTA (x, y) takes the planes of item x that
// fall to its warps of the item's gridDim.y * kDecodeWarps; the tables of
// stream i at tabs[i].
// LARGE: of at least kHalfWarpItems items; bound by instructions, four CTAs per
// SM. Smaller launches are bound by latency and keep more in registers (72
// against 62 and, before, spills): boxes of 384x384x256 f64 0.058 -> 0.048 ms.
template <bool LARGE>
__global__ void __launch_bounds__(kDecodeThreads, LARGE ? 4 : 3)
    k_decode(const CtaWork* __restrict__ work, const uint32_t* __restrict__ chunk_ids,
             const StreamDesc* __restrict__ sd, const DecodeTables* __restrict__ tabs,
             const uint16_t* __restrict__ cb_sym, const uint32_t* __restrict__ sub_off,
             const uint64_t* __restrict__ chunk_word_off, const uint32_t* __restrict__ payload,
             uint16_t* __restrict__ codes)
{
    extern __shared__ __align__(16) uint8_t decode_smem[];
    DecodeSmem& sm = *reinterpret_cast<DecodeSmem*>(decode_smem);
    const CtaWork w = work[blockIdx.x];
    const StreamDesc s = sd[w.stream];
    const uint32_t P = s.C * s.C, np = w.count * s.C;
    uint32_t W = decode_lanes(P);
    if (LARGE && P == kMaxPlane && s.code_off % 8 == 0 &&
        32 * (s.word_cap - 4) < (uint64_t)kHalfWarpBits * s.nchunks * s.C)
        W = 16;
    if (blockIdx.y * kDecodeWarps * (32 / W) >= np) return;  // uniform per block
    const uint32_t first = blockIdx.y * kDecodeWarps + (threadIdx.x >> 5), nwarps = gridDim.y * kDecodeWarps;
    load_table(sm, tabs + w.stream);
    decode_buffered(sm, s, tabs + w.stream, W, chunk_ids + w.first, np, first, nwarps, cb_sym, sub_off, chunk_word_off,
                    payload, codes);
}

// Persistent variant: a fixed grid walks the work list of a batch held in
// device memory (BatchHdr at meta), so one captured launch serves any batch.
__global__ void __launch_bounds__(kDecodeThreads, 3) k_decode_dyn(const uint8_t* __restrict__ meta,
                                                               const StreamDesc* __restrict__ sd,
                                                               const DecodeTables* __restrict__ tabs,
                                                               const uint16_t* __restrict__ cb_sym,
                                                               const uint32_t* __restrict__ sub_off,
                                                               const uint64_t* __restrict__ chunk_word_off,
                                                               const uint32_t* __restrict__ payload,
                                                               uint16_t* __restrict__ codes)
{
    extern __shared__ __align__(16) uint8_t decode_smem[];
    DecodeSmem& sm = *reinterpret_cast<DecodeSmem*>(decode_smem);
    const BatchHdr* h = reinterpret_cast<const BatchHdr*>(meta);
    const uint32_t n = h->n_work;
    if (n == 0) return;
    const CtaWork* __restrict__ work = reinterpret_cast<const CtaWork*>(meta + h->o_work);
    const uint32_t* __restrict__ chunk_ids = reinterpret_cast<const uint32_t*>(meta + h->o_ids);
    const uint32_t S = decode_slices(n);
    uint32_t loaded = 0xffffffffu;  // stream whose table is in shared memory
    for (uint32_t i = blockIdx.x; i < n * S; i += gridDim.x) {
        const CtaWork w = work[i / S];
        const StreamDesc s = sd[w.stream];
        const uint32_t P = s.C * s.C, W = decode_lanes(P), np = w.count * s.C;
        if (i % S * kDecodeWarps * (32 / W) >= np) continue;  // uniform per block
        const uint32_t first = i % S * kDecodeWarps + (threadIdx.x >> 5);
        if (w.stream != loaded) load_table(sm, tabs + w.stream);
        loaded = w.stream;
        decode_buffered(sm, s, tabs + w.stream, W, chunk_ids + w.first, np, first, S * kDecodeWarps, cb_sym, sub_off,
                        chunk_word_off, payload, codes);
    }
}

// Unpredictable values: for each listed chunk, the positions of its zero codes
// in order, and a value moved for each between the dense per-position buffer
// and the chunk's slot of the compact list (gather on encode, scatter on
// decode). A thread turns 32 consecutive codes into a mask of zeros with four
// 16-byte loads, so the codes are read once. The positions go to a list in
// shared memory, so that the moves are spread over all threads wherever the
// zeros lie (along a front, most codes of a chunk are zero). Bound by latency.
// A launch takes a thread for every 32 codes of its largest chunk: a warp, four
// or 32 (in larger CTAs a chunk of up to 1024 codes is one warp's work, and a
// chunk of more than 32768 takes several spans). With one warp for chunks of up
// to 4096, a warp's lanes listed up to 128 zeros each: 128^3 f64 GRF at 1e-5,
// half resolution, 0.030 -> 0.012 ms; 256^3 f64 fronts with chunks of 16, 0.14
// -> 0.072. Before that (a thread read its 32 codes one by one, twice, and
// moved its own values) and now: 512^3 f32 at 1e-4, decode, 0.25 -> 0.059 ms;
// 384x384x256 f64 fronts at 1e-6, decode, 0.32 -> 0.096; a box of them 21 -> 11
// us; 336x272x208 f32 with chunks of 8, 0.14 -> 0.061 ms.
template <uint32_t THREADS>
struct UnpredShape {
    static constexpr uint32_t threads = THREADS;
    static constexpr uint32_t span = 32 * THREADS;  // codes the CTA holds
};
using UnpredBig = UnpredShape<1024>;
template <class S>
struct UnpredSmem {
    uint32_t wsum[S::threads / 32];
    uint16_t pos[S::span];
};

template <class S, typename T, bool GATHER>
__device__ __forceinline__ void unpred_move_one(const UnpredWork& uw, const StreamDesc* __restrict__ sd,
                                                const uint16_t* __restrict__ codes, T* __restrict__ dense,
                                                T* __restrict__ list, UnpredSmem<S>& sm)
{
    const StreamDesc s = sd[uw.stream];
    const uint32_t vol = s.C * s.C * s.C, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const bool alone = S::threads == 32 || vol <= 1024;  // one warp's work
    if (alone && wid) return;
    const uint32_t threads = alone ? 32u : S::threads;
    auto sync = [&]() {
        if (alone) __syncwarp();
        else __syncthreads();
    };
    const size_t base = s.code_off + (size_t)uw.chunk * vol;
    const uint16_t* __restrict__ src = codes + base;
    const bool vec = vol % 8 == 0 && ((uintptr_t)src & 15) == 0;
    uint64_t before = 0;  // zeros of the spans done
    for (uint32_t at = 0; at < vol && before < uw.count; at += S::span) {
        const uint32_t i = at + threadIdx.x * 32;
        uint32_t m = 0;
        if (vec) {
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (i + 8 * j < vol) {
                    const uint4 q = __ldg(reinterpret_cast<const uint4*>(src + i + 8 * j));
                    m |= (pair_mask(q.x, 0) | pair_mask(q.y, 0) << 2 | pair_mask(q.z, 0) << 4 | pair_mask(q.w, 0) << 6)
                         << (8 * j);
                }
        } else {
            for (uint32_t j = 0; j < 32 && i + j < vol; ++j) m |= (uint32_t)(src[i + j] == 0) << j;
        }
        const uint32_t c = __popc(m), incl = group_scan(c, 32, lane);
        const uint32_t n = __shfl_sync(0xffffffffu, incl, 31);
        uint32_t r0 = 0, all = n;  // zeros before this warp's in the span, and in the span
        if (!alone) {
            if (lane == 0) sm.wsum[wid] = n;
            __syncthreads();
            all = 0;
#pragma unroll
            for (uint32_t w = 0; w < S::threads / 32; ++w) {
                const uint32_t v = sm.wsum[w];
                if (w < wid) r0 += v;
                all += v;
            }
        }
        uint32_t r = r0 + incl - c;
        for (uint32_t mm = m; mm; mm &= mm - 1, ++r) sm.pos[r] = (uint16_t)(threadIdx.x * 32 + (__ffs(mm) - 1));
        sync();
        for (uint32_t k = threadIdx.x; k < all; k += threads) {
            const uint64_t v = before + k;
            if (v >= uw.count) break;
            const size_t d = base + at + sm.pos[k];
            if (GATHER) list[uw.list_off + v] = dense[d];
            else dense[d] = list[uw.list_off + v];
        }
        sync();  // the list and wsum are written again
        before += all;
    }
}

template <class S, typename T, bool GATHER>
__global__ void __launch_bounds__(S::threads) k_unpred_move(const UnpredWork* __restrict__ work,
                                                            const StreamDesc* __restrict__ sd,
                                                            const uint16_t* __restrict__ codes, T* __restrict__ dense,
                                                            T* __restrict__ list)
{
    extern __shared__ __align__(16) uint8_t unpred_smem[];
    unpred_move_one<S, T, GATHER>(work[blockIdx.x], sd, codes, dense, list,
                                  *reinterpret_cast<UnpredSmem<S>*>(unpred_smem));
}

// Persistent scatter (decode side) over the unpredictable-value list of a
// batch held in device memory (BatchHdr at meta).
template <typename T>
__global__ void __launch_bounds__(UnpredBig::threads) k_unpred_scatter_dyn(const uint8_t* __restrict__ meta,
                                                                           const StreamDesc* __restrict__ sd,
                                                                           const uint16_t* __restrict__ codes,
                                                                           T* __restrict__ dense, T* __restrict__ list)
{
    extern __shared__ __align__(16) uint8_t unpred_smem[];
    const BatchHdr* h = reinterpret_cast<const BatchHdr*>(meta);
    const uint32_t n = h->n_uwork;
    const UnpredWork* __restrict__ work = reinterpret_cast<const UnpredWork*>(meta + h->o_uwork);
    for (uint32_t wi = blockIdx.x; wi < n; wi += gridDim.x)
        unpred_move_one<UnpredBig, T, false>(work[wi], sd, codes, dense, list,
                                             *reinterpret_cast<UnpredSmem<UnpredBig>*>(unpred_smem));
}

__global__ void k_pack_streams(const StreamDesc* __restrict__ sd, const uint64_t* __restrict__ stream_words, int s0,
                               const uint32_t* __restrict__ payload, uint32_t* __restrict__ dst)
{
    const int s = s0 + (int)blockIdx.y;
    uint64_t b = 0;  // words of the streams before s in this group
    for (int i = s0; i < s; ++i) b += stream_words[i];
    const uint64_t n = stream_words[s], a = sd[s].word_base;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        dst[b + i] = payload[a + i];
}

}  // namespace

void launch_pack_streams(const StreamDesc* sd, const uint64_t* stream_words, int s0, int s1, const uint32_t* payload,
                         uint32_t* dst, cudaStream_t st)
{
    if (s1 > s0) k_pack_streams<<<dim3(16, s1 - s0), 256, 0, st>>>(sd, stream_words, s0, payload, dst);
}

void launch_run_stats(const CtaWork* work, const uint32_t* chunk_ids, int nwork, const StreamDesc* sd,
                      const uint16_t* codes, unsigned long long* stats, cudaStream_t st)
{
    if (nwork > 0) k_run_stats<<<dim3(nwork, kPlaneSlices), kLaneThreads, 0, st>>>(work, chunk_ids, sd, codes, stats);
}

void launch_sub_bits(const CtaWork* work, const uint32_t* chunk_ids, int nwork, const StreamDesc* sd,
                     const uint16_t* codes, const uint32_t* ctab, const uint8_t* rbits, uint32_t* sub_bits,
                     cudaStream_t st)
{
    if (nwork)
        k_sub_bits<<<dim3(nwork, kPlaneSlices), kLaneThreads, 0, st>>>(work, chunk_ids, sd, codes, ctab, rbits,
                                                                        sub_bits);
}

void launch_scan_streams(const StreamDesc* sd, int nstreams, uint32_t max_chunks, const uint32_t* sub_bits,
                         uint32_t* sub_off, uint64_t* chunk_word_off, uint64_t* stream_words, uint32_t* payload,
                         cudaStream_t st)
{
    if (!nstreams || !max_chunks) return;
    k_plane_offsets<<<dim3(nstreams, (max_chunks + 31) / 32), 1024, 0, st>>>(sd, sub_bits, sub_off, chunk_word_off);
    k_scan_stream<<<nstreams, 1024, 0, st>>>(sd, sub_bits, sub_off, chunk_word_off, stream_words, payload);
}

void launch_encode(const CtaWork* work, const uint32_t* chunk_ids, int nwork, const StreamDesc* sd,
                   const uint16_t* codes, const uint32_t* ctab, const uint8_t* rbits, const uint32_t* sub_bits,
                   const uint32_t* sub_off, const uint64_t* chunk_word_off, uint32_t* payload, cudaStream_t st)
{
    if (nwork)
        k_encode<<<dim3(nwork, kPlaneSlices), kLaneThreads, 0, st>>>(work, chunk_ids, sd, codes, ctab, rbits, sub_bits,
                                                                      sub_off, chunk_word_off, payload);
}

void launch_decode(const CtaWork* work, const uint32_t* chunk_ids, int nwork, const StreamDesc* sd,
                   const uint16_t* cb_sym, const void* tables, const uint32_t* sub_off, const uint64_t* chunk_word_off,
                   const uint32_t* payload, uint16_t* codes, cudaStream_t st)
{
    if (!nwork) return;
    auto* k = nwork >= kHalfWarpItems ? k_decode<true> : k_decode<false>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DecodeSmem));
    k<<<dim3(nwork, decode_slices((uint32_t)nwork)), kDecodeThreads, sizeof(DecodeSmem), st>>>(
        work, chunk_ids, sd, static_cast<const DecodeTables*>(tables), cb_sym, sub_off, chunk_word_off, payload, codes);
}

void launch_decode_planes(const CtaWork* work, const uint32_t* chunk_ids, int nwork, const StreamDesc* sd,
                          const uint16_t* cb_sym, const void* tables, const uint32_t* sub_off,
                          const uint64_t* chunk_word_off, const uint32_t* payload, uint16_t* codes, cudaStream_t st)
{
    if (nwork)
        k_decode_planes<<<nwork, kPlaneThreads, 0, st>>>(work, chunk_ids, sd, static_cast<const DecodeTables*>(tables),
                                                         cb_sym, sub_off, chunk_word_off, payload, codes);
}

size_t decode_tables_bytes() { return sizeof(DecodeTables); }

void launch_build_tables(const StreamDesc* sd, int nstreams, const uint16_t* cb_sym, const uint8_t* cb_len,
                         void* tables, cudaStream_t st)
{
    if (nstreams > 0)
        k_build_tables<<<nstreams, kBuildThreads, 0, st>>>(sd, cb_sym, cb_len, static_cast<DecodeTables*>(tables));
}

namespace {
template <class S, typename T>
void unpred_move(bool gather, const UnpredWork* work, int nwork, const StreamDesc* sd, const uint16_t* codes, T* dense,
                 T* list, cudaStream_t st)
{
    auto kern = gather ? k_unpred_move<S, T, true> : k_unpred_move<S, T, false>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(UnpredSmem<S>));
    kern<<<nwork, S::threads, sizeof(UnpredSmem<S>), st>>>(work, sd, codes, dense, list);
}
}  // namespace

template <typename T>
void launch_unpred_move(bool gather, uint32_t codes_most, const UnpredWork* work, int nwork, const StreamDesc* sd,
                        const uint16_t* codes, T* dense, T* list, cudaStream_t st)
{
    if (!nwork) return;
    if (codes_most <= 1024) unpred_move<UnpredShape<32>, T>(gather, work, nwork, sd, codes, dense, list, st);
    else if (codes_most <= 4096) unpred_move<UnpredShape<128>, T>(gather, work, nwork, sd, codes, dense, list, st);
    else unpred_move<UnpredBig, T>(gather, work, nwork, sd, codes, dense, list, st);
}

template void launch_unpred_move<float>(bool, uint32_t, const UnpredWork*, int, const StreamDesc*, const uint16_t*, float*,
                                        float*, cudaStream_t);
template void launch_unpred_move<double>(bool, uint32_t, const UnpredWork*, int, const StreamDesc*, const uint16_t*,
                                         double*, double*, cudaStream_t);

void launch_decode_dyn(int grid, const uint8_t* meta, const StreamDesc* sd, const uint16_t* cb_sym,
                       const void* tables, const uint32_t* sub_off, const uint64_t* chunk_word_off,
                       const uint32_t* payload, uint16_t* codes, cudaStream_t st)
{
    cudaFuncSetAttribute(k_decode_dyn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DecodeSmem));
    k_decode_dyn<<<grid, kDecodeThreads, sizeof(DecodeSmem), st>>>(meta, sd, static_cast<const DecodeTables*>(tables), cb_sym, sub_off,
                                                  chunk_word_off, payload, codes);
}

template <typename T>
void launch_unpred_scatter_dyn(int grid, const uint8_t* meta, const StreamDesc* sd, const uint16_t* codes, T* dense,
                               T* list, cudaStream_t st)
{
    cudaFuncSetAttribute(k_unpred_scatter_dyn<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(UnpredSmem<UnpredBig>));
    k_unpred_scatter_dyn<T><<<grid, UnpredBig::threads, sizeof(UnpredSmem<UnpredBig>), st>>>(meta, sd, codes, dense, list);
}

template void launch_unpred_scatter_dyn<float>(int, const uint8_t*, const StreamDesc*, const uint16_t*, float*, float*,
                                               cudaStream_t);
template void launch_unpred_scatter_dyn<double>(int, const uint8_t*, const StreamDesc*, const uint16_t*, double*,
                                                double*, cudaStream_t);

}  // namespace stz
