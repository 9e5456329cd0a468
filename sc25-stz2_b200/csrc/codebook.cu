// Huffman codebooks of a compress on the GPU.
//
// The rule is the container's (build_codebook in host.cpp states it for the
// host): symbols with a nonzero count, sorted by (count, symbol);
// minimum-redundancy code lengths of the two-queue construction (on equal
// weights a symbol is merged before an earlier merge); lengths capped at
// kMaxCodeLen; canonical codes in (length, symbol) order. Two codebooks are
// built per stream, one of the plain codes and one with run symbols, and the
// one with fewer payload bits is taken.
//
// On the host this ended the device's work for the longest part of a
// compress: the full histograms crossed PCIe (256 KB per stream with a code
// outside the window), and a codebook of tens of thousands of symbols took
// milliseconds of sorting and merging. Measured from the histograms to the
// code tables (one B200, 16 host cores), host before and both kernels here
// now: 64^3 f32 0.52 -> 0.058 ms, 512^3 f32 at rel 1e-3 0.25 -> 0.073 ms and
// at 1e-4 1.4 -> 0.11 ms, 384x384x256 f64 fronts at 1e-6 (codebooks of up to
// 65 K symbols) 12-14 -> 0.69 ms, 1.07 ms of it before the searches of a
// thread ran four side by side and the sort loaded four items ahead. The
// merges of up to kSmallBook symbols are one warp's work in shared memory:
// 0.085 -> 0.073 ms on the 512^3 field at 1e-3.
//
// The merging is sequential in the textbook form, but every weight not above
// the sum t of the two smallest is consumed before the first merge of that
// round is (merges weigh at least t and lose ties), so a round pairs all of
// them at once, in merged order. The smallest weight doubles every two
// rounds, so about 2 log2(codes) rounds of one CTA finish a stream. The
// kernel is bound by the latency of those rounds and of the sort's passes,
// not by bandwidth: a stream is one CTA of 1024 threads, all streams and
// both codebooks side by side.
#include <algorithm>

#include <cuda_runtime.h>

#include "huffman.h"
#include "run_symbols.cuh"

namespace stz {
namespace {

constexpr int kCbThreads = 1024;
constexpr int kCbWarps = kCbThreads / 32;
constexpr uint32_t kSmallBook = 512;  // symbols whose merges one warp makes (14 KB of lists)
constexpr int kMaxRounds = 192;  // rounds <= 2 log2(total count) + 2
constexpr int kMaxDepth = 80;    // depth <= 1.45 log2(total count) + 2

// What the first kernel leaves for the second, per stream and codebook.
struct BookRecord {
    uint64_t bits;     // payload bits with this codebook
    uint32_t n;        // symbols (0: not built)
    uint32_t run_base, run_n;
    uint32_t cnt[kMaxCodeLen + 1];  // symbols of each code length
};

// Scratch of one codebook of at most cap symbols (a multiple of 16).
struct BookScratch {
    uint64_t* key[2];  // count << 32 | index in symbol order; the sort's two buffers
    uint64_t* node;    // weights of the merges, in the order they are made
    uint32_t* up;      // their parents, then their depths
    uint16_t* sym;     // symbols in symbol order
    uint8_t* len;      // their code lengths
};
constexpr size_t kBookBytes = 8 + 8 + 8 + 4 + 2 + 1;  // per symbol

// Scratch of stream q's codebook ph: the streams' two codebooks of
// off[q + 1] - off[q] symbols each, back to back.
__device__ __forceinline__ BookScratch book_scratch(uint8_t* scratch, const uint64_t* off, uint32_t q, uint32_t ph)
{
    const size_t cap = (size_t)(off[q + 1] - off[q]);
    BookScratch b;
    b.key[0] = reinterpret_cast<uint64_t*>(scratch + (2 * (size_t)off[q] + ph * cap) * kBookBytes);
    b.key[1] = b.key[0] + cap;
    b.node = b.key[1] + cap;
    b.up = reinterpret_cast<uint32_t*>(b.node + cap);
    b.sym = reinterpret_cast<uint16_t*>(b.up + cap);
    b.len = reinterpret_cast<uint8_t*>(b.sym + cap);
    return b;
}

// Exclusive prefix of v over the CTA's threads; total in *sum. wsum: one word per warp.
__device__ __forceinline__ uint32_t block_prefix(uint32_t v, uint32_t* wsum, uint32_t* sum)
{
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += u;
    }
    __syncthreads();  // wsum may still be read from an earlier use
    if (lane == 31) wsum[w] = incl;
    __syncthreads();
    if (w == 0) {
        uint32_t x = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= (uint32_t)o) x += u;
        }
        wsum[lane] = x;
    }
    __syncthreads();
    *sum = wsum[kCbWarps - 1];
    return (w ? wsum[w - 1] : 0u) + incl - v;
}

// Stable counting sort of n items by an 8-bit digit: put(i, key, pos) for item
// i at its place. Every warp owns n / 32 consecutive items and a row of 256
// counters, so a pass has no barrier between its counting and its ranking
// steps; four items per lane are loaded ahead of both. cnt: kCbWarps x 256
// words of shared memory.
template <class Key, class Load, class Digit, class Put>
__device__ __forceinline__ void counting_pass(uint32_t n, uint32_t* cnt, uint32_t* wsum, Load&& load, Digit&& digit,
                                              Put&& put)
{
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t per = ((n + kCbThreads - 1) / kCbThreads) * 32;
    const uint32_t a = min(w * per, n), b = min(a + per, n);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kCbWarps * 256; i += kCbThreads) cnt[i] = 0;
    __syncthreads();
    for (uint32_t i0 = a; i0 < b; i0 += 128) {
        Key key[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i0 + 32 * j + lane < b) key[j] = load(i0 + 32 * j + lane);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (i0 + 32 * j >= b) break;  // uniform per warp
            const bool in = i0 + 32 * j + lane < b;
            const uint32_t d = in ? digit(key[j]) : 256u;
            const uint32_t same = __match_any_sync(0xffffffffu, d);
            if (in && (uint32_t)(__ffs(same) - 1) == lane) cnt[w * 256 + d] += __popc(same);
            __syncwarp();
        }
    }
    __syncthreads();
    // counters -> first places, digit by digit and warp by warp within one:
    // thread t holds digit t / 4, warps 8 (t % 4) .. + 7
    {
        const uint32_t d = threadIdx.x >> 2, r0 = (threadIdx.x & 3) * 8;
        uint32_t c[8], s = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) c[k] = cnt[(r0 + k) * 256 + d], s += c[k];
        uint32_t total;
        uint32_t at = block_prefix(s, wsum, &total);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            cnt[(r0 + k) * 256 + d] = at;
            at += c[k];
        }
    }
    __syncthreads();
    for (uint32_t i0 = a; i0 < b; i0 += 128) {
        Key key[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i0 + 32 * j + lane < b) key[j] = load(i0 + 32 * j + lane);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (i0 + 32 * j >= b) break;  // uniform per warp
            const uint32_t i = i0 + 32 * j + lane;
            const bool in = i < b;
            const uint32_t d = in ? digit(key[j]) : 256u;
            const uint32_t same = __match_any_sync(0xffffffffu, d);
            uint32_t first = 0;
            if (in) first = cnt[w * 256 + d];
            __syncwarp();
            if (in) {
                if ((uint32_t)(__ffs(same) - 1) == lane) cnt[w * 256 + d] = first + __popc(same);
                put(i, key[j], first + __popc(same & ((1u << lane) - 1u)));
            }
            __syncwarp();
        }
    }
    __syncthreads();
}

// The threads that merge one codebook: the CTA, or one warp for a small one,
// whose rounds cost the latency of their barriers.
struct WholeCta {
    static constexpr uint32_t size = kCbThreads;
    static __device__ __forceinline__ uint32_t id() { return threadIdx.x; }
    static __device__ __forceinline__ void sync() { __syncthreads(); }
    static __device__ __forceinline__ uint32_t count(bool p) { return (uint32_t)__syncthreads_count(p); }
};
struct OneWarp {
    static constexpr uint32_t size = 32;
    static __device__ __forceinline__ uint32_t id() { return threadIdx.x & 31; }
    static __device__ __forceinline__ void sync() { __syncwarp(); }
    static __device__ __forceinline__ uint32_t count(bool p) { return __popc(__ballot_sync(0xffffffffu, p)); }
};

// For items k < n: the number of the sorted list's first m entries that come
// before value(k), to done(k, value, rank). Up to four searches per thread
// side by side: the lists of a large codebook lie in L2, and a search is a
// chain of its latency.
template <class Group, class Value, class Before, class Done>
__device__ __forceinline__ void ranks(uint32_t n, uint32_t m, Value&& value, Before&& before, Done&& done)
{
    const uint32_t top = m ? 1u << (31 - __clz(m)) : 0u;
    uint32_t k0 = Group::id();
    if (Group::size == kCbThreads)
        for (; k0 + kCbThreads < n; k0 += 4 * kCbThreads) {
            uint64_t v[4];
            uint32_t pos[4] = {0, 0, 0, 0};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (k0 + j * kCbThreads < n) v[j] = value(k0 + j * kCbThreads);
            for (uint32_t step = top; step; step >>= 1)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (k0 + j * kCbThreads < n && pos[j] + step <= m && before(pos[j] + step - 1, v[j])) pos[j] += step;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (k0 + j * kCbThreads < n) done(k0 + j * kCbThreads, v[j], pos[j]);
        }
    for (; k0 < n; k0 += Group::size) {
        const uint64_t v = value(k0);
        uint32_t pos = 0;
        for (uint32_t step = top; step; step >>= 1)
            if (pos + step <= m && before(pos + step - 1, v)) pos += step;
        done(k0, v, pos);
    }
}

// All merges of n sorted symbols: weights to node, parents to up, the first
// merge of every round to first; returns the rounds, and the merges in m.
template <class Group>
__device__ __forceinline__ uint32_t merge_rounds(uint32_t n, const uint64_t* leaf, uint64_t* node, uint64_t* merged,
                                                 uint32_t* up, uint32_t* first, uint32_t& m)
{
    const uint32_t id = Group::id();
    uint32_t i = 0, j = 0, rounds = 0;  // first unmerged symbol, first unmerged merge
    m = 0;
    if (id == 0) first[0] = 0;
    while (n - i + (m - j) > 1) {
        const uint64_t none = ~0ull;
        const uint64_t l0 = i < n ? leaf[i] >> 32 : none, l1 = i + 1 < n ? leaf[i + 1] >> 32 : none;
        const uint64_t q0 = j < m ? node[j] : none, q1 = j + 1 < m ? node[j + 1] : none;
        // sum of the two smallest
        const uint64_t t = l0 <= q0 ? l0 + min(l1, q0) : q0 + min(l0, q1);
        // symbols and merges of weight <= t
        uint32_t a = 0, b = 0;
        for (;;) {
            const uint32_t k = i + a + id, c = Group::count(k < n && (leaf[k] >> 32) <= t);
            a += c;
            if (c < Group::size) break;
        }
        for (;;) {
            const uint32_t k = j + b + id, c = Group::count(k < m && node[k] <= t);
            b += c;
            if (c < Group::size) break;
        }
        if ((a + b) & 1) {  // the last of them waits for the next round (on equal weights the merge is last)
            if (b && (a == 0 || node[j + b - 1] >= (leaf[i + a - 1] >> 32))) --b;
            else --a;
        }
        // places in merged order (on equal weights the symbol is first); a
        // merge's pair is its parent
        ranks<Group>(a, b, [&](uint32_t k) { return leaf[i + k] >> 32; },
                     [&](uint32_t x, uint64_t w) { return node[j + x] < w; },
                     [&](uint32_t k, uint64_t w, uint32_t r) { merged[k + r] = w; });
        ranks<Group>(b, a, [&](uint32_t k) { return node[j + k]; },
                     [&](uint32_t x, uint64_t w) { return (leaf[i + x] >> 32) <= w; },
                     [&](uint32_t k, uint64_t w, uint32_t r) {
                         merged[k + r] = w;
                         up[j + k] = m + ((k + r) >> 1);
                     });
        Group::sync();
        const uint32_t pairs = (a + b) >> 1;
        for (uint32_t k = id; k < pairs; k += Group::size) node[m + k] = merged[2 * k] + merged[2 * k + 1];
        i += a, j += b, m += pairs;
        ++rounds;
        if (id == 0) first[rounds] = m;
        Group::sync();
        if (rounds == kMaxRounds) break;  // not reached: the smallest weight doubles every two rounds
    }
    return rounds;
}

// Code lengths of both codebooks of every stream: blockIdx.x the stream,
// blockIdx.y 0 without and 1 with run symbols.
__global__ void __launch_bounds__(kCbThreads) k_codebook(const StreamDesc* __restrict__ sd,
                                                         const uint32_t* __restrict__ hist,
                                                         const uint32_t* __restrict__ outside,
                                                         const unsigned long long* __restrict__ rstats,
                                                         const uint64_t* __restrict__ scratch_off, uint8_t* scratch,
                                                         BookRecord* __restrict__ rec)
{
    // the sort's counters; before it, the bitmap of used codes; after it, the lists of a small codebook
    __shared__ __align__(8) uint32_t cnt[kCbWarps * 256];
    __shared__ uint32_t wsum[kCbWarps];
    __shared__ uint32_t first[kMaxRounds + 1];  // first merge of every round
    __shared__ uint32_t icnt[kMaxDepth];
    __shared__ uint32_t s_val;
    __shared__ uint32_t lcnt[kMaxCodeLen + 1], lpos[kMaxCodeLen + 1];
    __shared__ unsigned long long s_bits;
    const StreamDesc s = sd[blockIdx.x];
    const bool runs = blockIdx.y != 0;
    const uint32_t tid = threadIdx.x, lane = tid & 31, R = s.radius, R2 = 2 * R;
    BookRecord& out = rec[2 * blockIdx.x + blockIdx.y];
    const uint32_t* h = hist + (size_t)blockIdx.x * R2;
    const unsigned long long* rs = rstats + (size_t)blockIdx.x * kRunStats;
    const uint32_t J = run_slot_count(s.C * s.C);
    if (runs && J == 0) {  // uniform
        if (tid == 0) out.n = 0, out.bits = ~0ull;
        return;
    }

    // ---- bitmap of the codes in use ----
    uint32_t* used = cnt;
    const uint32_t words = (R2 + 31) / 32;
    for (uint32_t i = tid; i < words + 2; i += kCbThreads) used[i] = 0;
    __syncthreads();
    uint32_t c0 = 0, c1 = R2;
    if (outside[blockIdx.x] == 0) {  // every code lies in the window
        c0 = R > (uint32_t)kHistWindow / 2 ? R - kHistWindow / 2 : 0u;
        c1 = min(R2, R + kHistWindow / 2);
    }
    for (uint32_t c = (c0 & ~31u) + tid; c < ((c1 + 31) & ~31u); c += 8 * kCbThreads) {
        uint32_t v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t x = c + j * kCbThreads;
            v[j] = x >= c0 && x < c1 ? h[x] : 0u;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t x = c + j * kCbThreads, m = __ballot_sync(0xffffffffu, v[j] != 0);
            if (lane == 0 && m) used[x >> 5] = m;
        }
    }
    __syncthreads();
    uint32_t run_base = 0;
    if (runs) {
        // the highest run of J free codes, at 1 or above
        if (tid == 0) s_val = 0;
        __syncthreads();
        for (uint32_t top = R2 > J ? R2 - J : 0; top >= 1;) {
            if (tid < top) {
                const uint32_t u = top - tid;  // codes [u, u + J), J <= 40
                const uint32_t wi = u >> 5, sh = u & 31;
                uint64_t v = ((uint64_t)used[wi + 1] << 32 | used[wi]) >> sh;
                if (sh) v |= (uint64_t)used[wi + 2] << (64 - sh);
                if ((v & ((1ull << J) - 1)) == 0) atomicMax(&s_val, u);
            }
            __syncthreads();
            run_base = s_val;
            __syncthreads();
            if (run_base || top <= kCbThreads) break;
            top -= kCbThreads;
        }
        if (run_base == 0) {  // uniform
            if (tid == 0) out.n = 0, out.bits = ~0ull;
            return;
        }
        // the run symbols, and the centre codes they leave
        if (tid == 0) {
            if (rs[0]) used[R >> 5] |= 1u << (R & 31);
            else used[R >> 5] &= ~(1u << (R & 31));
            for (uint32_t i = 0; i < J; ++i)
                if (rs[1 + i]) used[(run_base + i) >> 5] |= 1u << ((run_base + i) & 31);
        }
        __syncthreads();
    }
    auto count_of = [&](uint32_t c) -> uint32_t {
        if (runs) {
            if (c == R) return (uint32_t)rs[0];
            if (c - run_base < J) return (uint32_t)rs[1 + c - run_base];
        }
        return h[c];
    };

    // ---- symbols in order, with their counts ----
    const BookScratch B = book_scratch(scratch, scratch_off, blockIdx.x, blockIdx.y);
    uint32_t n;
    {
        constexpr uint32_t kPer = 65536 / 32 / kCbThreads;  // words per thread
        uint32_t m[kPer], c = 0;
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t wi = tid * kPer + k;
            m[k] = wi < words ? used[wi] : 0u;
            c += __popc(m[k]);
        }
        uint32_t at = block_prefix(c, wsum, &n);
        uint32_t mx = 0;
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k)
            for (uint32_t mm = m[k]; mm; mm &= mm - 1, ++at) {
                const uint32_t code = (tid * kPer + k) * 32 + __ffs(mm) - 1;
                const uint32_t w = count_of(code);
                B.sym[at] = (uint16_t)code;
                B.key[0][at] = (uint64_t)w << 32 | at;
                mx = max(mx, w);
            }
        if (tid == 0) s_val = 0;
        __syncthreads();
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) atomicMax(&s_val, mx);
        __syncthreads();
    }
    const uint32_t maxw = s_val;
    if (tid <= kMaxCodeLen) lcnt[tid] = 0;
    if (n <= 1) {  // uniform: a lone symbol has an empty code
        __syncthreads();
        if (tid == 0) {
            if (n) B.len[0] = 0;
            out.n = n, out.bits = n ? 0 : ~0ull, out.run_base = run_base, out.run_n = runs ? J : 0;
            for (int l = 0; l <= kMaxCodeLen; ++l) out.cnt[l] = l == 0 ? n : 0;
        }
        return;
    }

    // ---- sort by count, 8 bits a pass (stable: equal counts stay in symbol order) ----
    int cur = 0;
    for (uint32_t sh = 32; sh < 64 && (maxw >> (sh - 32)); sh += 8) {
        const uint64_t* src = B.key[cur];
        uint64_t* dst = B.key[cur ^ 1];
        counting_pass<uint64_t>(
            n, cnt, wsum, [&](uint32_t i) { return src[i]; },
            [&](uint64_t k) { return (uint32_t)(k >> sh) & 255u; },
            [&](uint32_t, uint64_t k, uint32_t p) { dst[p] = k; });
        cur ^= 1;
    }
    const uint64_t* leaf = B.key[cur];
    uint32_t* up = B.up;
    uint32_t m, rounds;
    if (n <= kSmallBook) {  // in shared memory, where the sort's counters were
        uint64_t* sl = reinterpret_cast<uint64_t*>(cnt);
        for (uint32_t k = tid; k < n; k += kCbThreads) sl[k] = leaf[k];
        leaf = sl;
        up = reinterpret_cast<uint32_t*>(sl + 3 * kSmallBook);
        __syncthreads();
        if (tid < 32) {
            rounds = merge_rounds<OneWarp>(n, leaf, sl + kSmallBook, sl + 2 * kSmallBook, up, first, m);
            if (tid == 0) wsum[0] = rounds, wsum[1] = m;
        }
        __syncthreads();
        rounds = wsum[0], m = wsum[1];
    } else {
        rounds = merge_rounds<WholeCta>(n, leaf, B.node, B.key[cur ^ 1], up, first, m);
    }

    // ---- depths of the merges, last round first; merges of each depth ----
    for (uint32_t k = tid; k < kMaxDepth; k += kCbThreads) icnt[k] = 0;
    if (tid == 0) s_bits = 0;
    __syncthreads();
    for (uint32_t r = rounds; r-- > 0;) {
        const uint32_t x1 = first[r + 1];
        uint32_t x0 = first[r];
        for (; x0 + kCbThreads < x1; x0 += 4 * kCbThreads) {
            uint32_t d[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t x = x0 + q * kCbThreads + tid;
                d[q] = x < x1 && x != m - 1 ? up[x] : m - 1;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t x = x0 + q * kCbThreads + tid;
                d[q] = x < x1 ? (x == m - 1 ? 0u : min(up[d[q]] + 1u, (uint32_t)kMaxDepth - 1)) : (uint32_t)kMaxDepth;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t x = x0 + q * kCbThreads + tid;
                const uint32_t same = __match_any_sync(0xffffffffu, d[q]);
                if (x < x1) {
                    if ((uint32_t)(__ffs(same) - 1) == lane) atomicAdd(&icnt[d[q]], __popc(same));
                    up[x] = d[q];
                }
            }
        }
        for (; x0 < x1; x0 += kCbThreads) {
            const uint32_t x = x0 + tid;
            uint32_t d = kMaxDepth;
            if (x < x1) d = x == m - 1 ? 0u : min(up[up[x]] + 1u, (uint32_t)kMaxDepth - 1);
            const uint32_t same = __match_any_sync(0xffffffffu, d);
            if (x < x1) {
                if ((uint32_t)(__ffs(same) - 1) == lane) atomicAdd(&icnt[d], __popc(same));
                up[x] = d;
            }
        }
        __syncthreads();
    }

    // ---- symbols of each length (the lightest have the longest codes), capped ----
    if (tid == 0) {
        uint32_t avail = 1;
        for (int d = 0; d < kMaxDepth; ++d) {
            const uint32_t leaves = avail - icnt[d];
            lcnt[min(d, kMaxCodeLen)] += leaves;
            avail = 2 * icnt[d];
        }
        uint64_t kraft = 0;
        for (int l = 0; l <= kMaxCodeLen; ++l) kraft += (uint64_t)lcnt[l] << (kMaxCodeLen - l);
        // lengthen, lightest first, the first code shorter than the cap until
        // the Kraft sum fits: a code of length l raised to the cap frees
        // 2^(cap - l) - 1 units
        uint64_t over = kraft > (1ull << kMaxCodeLen) ? kraft - (1ull << kMaxCodeLen) : 0;
        for (int l = kMaxCodeLen - 1; l >= 1 && over; --l) {
            const uint64_t full = (1ull << (kMaxCodeLen - l)) - 1;
            const uint32_t k = (uint32_t)min((uint64_t)lcnt[l], over / full);
            over -= k * full;
            lcnt[l] -= k;
            lcnt[kMaxCodeLen] += k;
            if (over && lcnt[l]) {  // one more, part of the way
                int to = l;
                while (over) {
                    const uint64_t unit = 1ull << (kMaxCodeLen - 1 - to);
                    over = over > unit ? over - unit : 0;
                    ++to;
                }
                --lcnt[l];
                ++lcnt[to];
            }
        }
        uint32_t at = 0;
        for (int l = kMaxCodeLen; l >= 0; --l) lpos[l] = at, at += lcnt[l];
    }
    __syncthreads();
    unsigned long long bits = 0;
    uint32_t l = kMaxCodeLen;  // lengths fall along the list
    for (uint32_t k = tid; k < n; k += kCbThreads) {
        while (l > 0 && k >= lpos[l] + lcnt[l]) --l;
        const uint64_t e = leaf[k];
        B.len[(uint32_t)e] = (uint8_t)l;
        bits += (e >> 32) * l;
    }
    for (int o = 16; o; o >>= 1) bits += __shfl_xor_sync(0xffffffffu, bits, o);
    if (lane == 0) atomicAdd(&s_bits, bits);
    __syncthreads();
    if (tid == 0) out.n = n, out.bits = s_bits, out.run_base = run_base, out.run_n = runs ? J : 0;
    if (tid <= kMaxCodeLen) out.cnt[tid] = lcnt[tid];
}

// The codebook each stream takes (run symbols only where they shorten its
// payload), in canonical order: the code table, the run bit counts, the
// stream's descriptor fields, and the (symbol, length) lists of all streams
// back to back for the stream headers.
__global__ void __launch_bounds__(kCbThreads) k_codebook_emit(StreamDesc* sd,
                                                              const uint64_t* __restrict__ scratch_off,
                                                              uint8_t* scratch, const BookRecord* __restrict__ rec,
                                                              uint32_t* __restrict__ ctab, uint8_t* __restrict__ rbits,
                                                              uint16_t* __restrict__ cb_sym,
                                                              uint8_t* __restrict__ cb_len,
                                                              CodebookInfo* __restrict__ info)
{
    __shared__ uint32_t cnt[kCbWarps * 256];
    __shared__ uint32_t wsum[kCbWarps];
    __shared__ uint32_t first_code[kMaxCodeLen + 1], first_idx[kMaxCodeLen + 1];
    const uint32_t tid = threadIdx.x;
    auto pick = [&](int q) { return rec[2 * q + 1].n && rec[2 * q + 1].bits < rec[2 * q].bits ? 1 : 0; };
    // symbols of the streams before this one
    uint32_t before = 0, off;
    for (uint32_t q = tid; q < blockIdx.x; q += kCbThreads) before += rec[2 * q + pick((int)q)].n;
    block_prefix(before, wsum, &off);
    const int ph = pick((int)blockIdx.x);
    const BookRecord r = rec[2 * blockIdx.x + ph];
    const uint32_t C = sd[blockIdx.x].C, R = sd[blockIdx.x].radius;
    const BookScratch B = book_scratch(scratch, scratch_off, blockIdx.x, ph);
    if (tid == 0) {
        uint32_t code = 0, idx = r.cnt[0];
        first_code[0] = first_idx[0] = 0;
        for (int l = 1; l <= kMaxCodeLen; ++l) {
            code = (code + (l > 1 ? r.cnt[l - 1] : 0)) << 1;
            first_code[l] = code;
            first_idx[l] = idx;
            idx += r.cnt[l];
        }
        StreamDesc& d = sd[blockIdx.x];
        d.cb_off = off, d.n_used = r.n;
        d.run_base = ph ? r.run_base : 0, d.run_n = ph ? r.run_n : 0;
        info[blockIdx.x] = {off, r.n, d.run_base, d.run_n};
    }
    uint32_t* tab = ctab + (size_t)blockIdx.x * 2 * R;
    counting_pass<uint32_t>(
        r.n, cnt, wsum, [&](uint32_t i) { return (uint32_t)B.len[i] << 16 | B.sym[i]; },
        [&](uint32_t k) { return k >> 16; },
        [&](uint32_t, uint32_t k, uint32_t p) {
            const uint32_t l = k >> 16;
            const uint16_t sym = (uint16_t)k;
            cb_sym[off + p] = sym;
            cb_len[off + p] = (uint8_t)l;
            tab[sym] = l ? (first_code[l] + (p - first_idx[l])) << 5 | l : 0u;
        });
    // (the pass ends with a barrier: the code table is complete)
    const uint32_t P = C * C;
    if (ph == 0 || P >= kRunBitsStride) return;
    // bits of a run of k centre codes (planes of up to 1024 codes)
    uint32_t D, LD;
    const uint32_t J = run_geometry(P, D, LD);
    for (uint32_t k = tid; k <= P; k += kCbThreads) {
        uint32_t b = 0;
        run_symbols(k, R, r.run_base, J, D, LD, [&](uint32_t sym) { b += tab[sym] & 31u; });
        rbits[(size_t)blockIdx.x * kRunBitsStride + k] = (uint8_t)b;
    }
}

}  // namespace

uint64_t codebook_items(const StreamDesc& s, uint64_t codes)
{
    // no more symbols than code values or codes (a run symbol stands for two codes or more)
    return (std::min<uint64_t>(2 * (uint64_t)s.radius, codes) + 15) & ~15ull;
}

size_t codebook_scratch_bytes(uint64_t items, int nstreams)
{
    return ((2 * (size_t)items * kBookBytes + 255) & ~(size_t)255) + 2 * (size_t)nstreams * sizeof(BookRecord);
}

void launch_codebooks(StreamDesc* sd, int nstreams, const uint32_t* hist, const uint32_t* outside,
                      const unsigned long long* rstats, const uint64_t* scratch_off, uint64_t items, void* scratch,
                      uint32_t* ctab, uint8_t* rbits, uint16_t* cb_sym, uint8_t* cb_len, CodebookInfo* info,
                      cudaStream_t st)
{
    if (nstreams <= 0) return;
    uint8_t* sp = static_cast<uint8_t*>(scratch);
    BookRecord* rec = reinterpret_cast<BookRecord*>(sp + ((2 * (size_t)items * kBookBytes + 255) & ~(size_t)255));
    k_codebook<<<dim3(nstreams, 2), kCbThreads, 0, st>>>(sd, hist, outside, rstats, scratch_off, sp, rec);
    k_codebook_emit<<<nstreams, kCbThreads, 0, st>>>(sd, scratch_off, sp, rec, ctab, rbits, cb_sym, cb_len, info);
}

}  // namespace stz
