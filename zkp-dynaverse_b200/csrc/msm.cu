// Pippenger MSM kernels and their launch sequence (see msm.cuh).
#include <algorithm>
#include <cstring>
#include <vector>

#include "host_curve.hpp"
#include "msm.cuh"

namespace dv {

namespace {

constexpr uint32_t NO_INDEX = 0xffffffffu;

// Bucket-reduction segment length 2^DV_SEG_LOG (buckets per thread in the
// first level; doubled for long G1 windows).
#ifndef DV_SEG_LOG
#define DV_SEG_LOG 3
#endif

DV_INL uint32_t window_raw(const uint32_t* s, int bit, int c) {
    if (bit >= 256) return 0;
    const int limb = bit >> 5, sh = bit & 31;
    uint32_t v = s[limb] >> sh;
    if (sh + c > 32 && limb + 1 < 8) v |= s[limb + 1] << (32 - sh);
    return v & ((1u << c) - 1u);
}

// Carry into window w of the signed recoding (digits in (-B, B], B =
// 2^(c-1); a window above B goes negative and carries): decided by the next
// lower window unless that is exactly B.
DV_INL uint32_t carry_into(const uint32_t* s, int w, int c) {
    const uint32_t B = 1u << (c - 1);
    for (int v = w - 1; v >= 0; --v) {
        const uint32_t d = window_raw(s, v * c, c);
        if (d != B) return d > B ? 1u : 0u;
    }
    return 0;
}

DV_INL void load_scalar(const uint32_t* scalars, uint32_t i, uint32_t* s) {
    const uint4* q = reinterpret_cast<const uint4*>(scalars + 8ull * i);
    const uint4 a = q[0], b = q[1];
    s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
    s[4] = b.x; s[5] = b.y; s[6] = b.z; s[7] = b.w;
}

DV_INL uint32_t set_of(const uint32_t* set_off, uint32_t count, uint32_t i) {
    // largest k with set_off[k] <= i
    uint32_t lo = 0, hi = count;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (set_off[mid] <= i) lo = mid; else hi = mid;
    }
    return lo;
}

// Where digit i of a launch comes from: its set, its scalar and its point.
DV_INL void locate(const SetMap& m, uint32_t i, uint32_t& set, uint32_t& sidx, uint32_t& pidx) {
    set = m.count > 1 ? set_of(m.off, m.count, i) : 0;
    const uint32_t rel = i - (m.count > 1 ? m.off[set] : 0u);
    sidx = m.term_scalar ? m.term_scalar[i] : m.src ? m.src[set] + rel : i;
    pidx = m.term_point ? m.term_point[i] : m.prefix ? rel : sidx;
}

// Windows [w0, w1) of this block: blockIdx.y of gridDim.y even shares.
DV_INL void window_share(int W, int& w0, int& w1) {
    const int per = (W + (int)gridDim.y - 1) / (int)gridDim.y;
    w0 = min(W, (int)blockIdx.y * per);
    w1 = min(W, w0 + per);
}

// 1. Histogram of signed digits.  Few scalars leave the GPU idle on W
// dependent atomics each, so their windows are shared among gridDim.y threads
// (the carry into a thread's first window is found by carry_into): 1000
// scalars of 32 windows, histogram and scatter, 39 us with one thread a
// scalar, 10 us with one a window.
template <bool PRE>
__global__ void k_hist(const uint32_t* __restrict__ scalars, uint32_t n, const SetMap m, int c, int W,
                       uint32_t* __restrict__ counts, uint32_t* __restrict__ first_bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t set, sidx, pidx;
    locate(m, i, set, sidx, pidx);
    uint32_t s[8];
    load_scalar(scalars, sidx, s);
    if (!Fr::is_canonical(s)) {
        atomicMin(first_bad, sidx);
        return;
    }
    const uint32_t B = 1u << (c - 1), full = 1u << c;
    // PRE: precomputed window multiples share one bucket set per MSM
    const uint32_t base = PRE ? set * B : set * (uint32_t)W * B;
    const uint32_t active = __activemask();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t* words = scalars + 8ull * sidx;
    int w0, w1;
    window_share(W, w0, w1);
    uint32_t carry = carry_into(words, w0, c);
    for (int w = w0; w < w1; ++w) {
        const uint32_t d = window_raw(words, w * c, c) + carry;
        const bool neg = d > B;
        const uint32_t mag = neg ? full - d : d;
        carry = neg ? 1u : 0u;
        // Warp-aggregated increment: lanes hitting the same bucket (skewed
        // digits, e.g. a top window with few bits) issue one atomic.
        const uint32_t key = mag ? base + (PRE ? 0u : (uint32_t)w * B) + mag - 1 : NO_INDEX;
        const uint32_t peers = __match_any_sync(active, key);
        if (key != NO_INDEX && lane == (uint32_t)(__ffs(peers) - 1)) atomicAdd(counts + key, (uint32_t)__popc(peers));
    }
}

// 2. Exclusive scan of the counts: tiles of 4096 (1024 threads x 4), three
// passes -- tile sums, scan of the tile sums, per-tile scan with its prefix.
constexpr uint32_t SCAN_TILE = 4096;

// Exclusive scan of one value per thread over a 1024-thread block.
DV_INL uint32_t block_exclusive_scan(uint32_t v, uint32_t* block_total) {
    __shared__ uint32_t warp_sums[32];
    const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= (uint32_t)d) x += y;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t s = warp_sums[lane];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= (uint32_t)d) s += y;
        }
        warp_sums[lane] = s;
    }
    __syncthreads();
    const uint32_t prefix = (wid ? warp_sums[wid - 1] : 0u) + x - v;
    if (block_total) *block_total = warp_sums[31];
    __syncthreads();
    return prefix;
}

DV_INL void load4(const uint32_t* counts, uint32_t nb, uint32_t i, uint32_t* v) {
    if (i + 3 < nb) {
        const uint4 q = *reinterpret_cast<const uint4*>(counts + i);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
        for (int k = 0; k < 4; ++k) v[k] = i + k < nb ? counts[i + k] : 0u;
    }
}

__global__ void __launch_bounds__(1024) k_scan_tiles(const uint32_t* __restrict__ counts, uint32_t nb,
                                                     uint32_t* __restrict__ tile_sums) {
    const uint32_t i = blockIdx.x * SCAN_TILE + threadIdx.x * 4;
    uint32_t v[4];
    load4(counts, nb, i, v);
    uint32_t total;
    block_exclusive_scan(v[0] + v[1] + v[2] + v[3], &total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) k_scan_top(uint32_t* __restrict__ tile_sums, uint32_t ntiles,
                                                   uint32_t* __restrict__ grand_total) {
    const uint32_t per = (ntiles + 1023) / 1024;
    const uint32_t lo = min(ntiles, threadIdx.x * per), hi = min(ntiles, lo + per);
    uint32_t local = 0;
    for (uint32_t i = lo; i < hi; ++i) local += tile_sums[i];
    uint32_t total;
    uint32_t run = block_exclusive_scan(local, &total);
    for (uint32_t i = lo; i < hi; ++i) {
        const uint32_t v = tile_sums[i];
        tile_sums[i] = run;
        run += v;
    }
    if (threadIdx.x == 0) *grand_total = total;
}

__global__ void __launch_bounds__(1024) k_scan_apply(const uint32_t* __restrict__ counts, uint32_t nb,
                                                     const uint32_t* __restrict__ tile_prefix,
                                                     uint32_t* __restrict__ offsets, uint32_t* __restrict__ cursor) {
    const uint32_t i = blockIdx.x * SCAN_TILE + threadIdx.x * 4;
    uint32_t v[4];
    load4(counts, nb, i, v);
    uint32_t run = tile_prefix[blockIdx.x] + block_exclusive_scan(v[0] + v[1] + v[2] + v[3], nullptr);
    for (int k = 0; k < 4; ++k) {
        if (i + k < nb) {
            offsets[i + k] = run;
            cursor[i + k] = run;
        }
        run += v[k];
    }
}

// The same by one block for few buckets, tile after tile: one launch of 4 to
// 7 us for three of 3 each.
constexpr uint32_t SCAN_ONE = 4 * SCAN_TILE;
__global__ void __launch_bounds__(1024) k_scan_one(const uint32_t* __restrict__ counts, uint32_t nb,
                                                   uint32_t* __restrict__ offsets, uint32_t* __restrict__ cursor) {
    uint32_t before = 0;
    for (uint32_t tile = 0; tile < nb; tile += SCAN_TILE) {
        const uint32_t i = tile + threadIdx.x * 4;
        uint32_t v[4], total;
        load4(counts, nb, i, v);
        uint32_t run = before + block_exclusive_scan(v[0] + v[1] + v[2] + v[3], &total);
        for (int k = 0; k < 4; ++k) {
            if (i + k < nb) {
                offsets[i + k] = run;
                cursor[i + k] = run;
            }
            run += v[k];
        }
        before += total;
    }
    if (threadIdx.x == 0) offsets[nb] = before;
}

// 3. Scatter (point index | sign << 31) into bucket order.
template <bool PRE>
__global__ void k_scatter(const uint32_t* __restrict__ scalars, uint32_t n, const SetMap m, int c, int W,
                          uint32_t* __restrict__ cursor, uint32_t* __restrict__ sorted) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t set, sidx, pidx;
    locate(m, i, set, sidx, pidx);
    uint32_t s[8];
    load_scalar(scalars, sidx, s);
    if (!Fr::is_canonical(s)) return;
    const uint32_t B = 1u << (c - 1), full = 1u << c;
    // PRE: precomputed window multiples share one bucket set per MSM
    const uint32_t base = PRE ? set * B : set * (uint32_t)W * B;
    const uint32_t active = __activemask();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t* words = scalars + 8ull * sidx;
    int w0, w1;
    window_share(W, w0, w1);
    uint32_t carry = carry_into(words, w0, c);
    for (int w = w0; w < w1; ++w) {
        const uint32_t d = window_raw(words, w * c, c) + carry;
        const bool neg = d > B;
        const uint32_t mag = neg ? full - d : d;
        carry = neg ? 1u : 0u;
        const uint32_t key = mag ? base + (PRE ? 0u : (uint32_t)w * B) + mag - 1 : NO_INDEX;
        const uint32_t peers = __match_any_sync(active, key);
        if (key != NO_INDEX) {
            // one atomic per group of lanes with the same bucket; each lane
            // takes its rank within the group
            const uint32_t leader = (uint32_t)(__ffs(peers) - 1);
            uint32_t pos = 0;
            if (lane == leader) pos = atomicAdd(cursor + key, (uint32_t)__popc(peers));
            pos = __shfl_sync(peers, pos, leader) + (uint32_t)__popc(peers & ((1u << lane) - 1u));
            const uint32_t idx = PRE ? pidx * (uint32_t)W + (uint32_t)w : pidx;  // PRE: table entry 2^(c w) P_i
            sorted[pos] = idx | (neg ? 0x80000000u : 0u);
        }
    }
}

// 4. Balanced accumulation over the sorted list.
// Resident blocks per SM: four for G1 (128 registers, which its accumulator
// and the paired products fit but for 250 bytes), two for G2, whose 255
// registers leave 290 bytes of spills where four blocks' 128 left 2.5 KB
// (G2 MSM of 2^16 points: 2.24 to 2.03 ms; three blocks 2.12 ms).
template <class F>
constexpr int ACCUM_BLOCKS = sizeof(F) == sizeof(Fq) ? 4 : 2;
// A chunk of the pairwise levels (below): buckets [b0, b1) of a launch, its
// first level's slots, and whether the levels run (else the chunk's buckets
// are accumulated from the sorted list itself).
struct AccumChunk {
    uint32_t b0, b1, slots, pairs;
};
// The points to sum: with sorted, pts[index] under the entry's sign; without, pts in order.
template <class F>
__global__ void __launch_bounds__(128, ACCUM_BLOCKS<F>) k_accum(const Affine<F>* __restrict__ pts, const uint32_t* __restrict__ sorted,
                                               const uint32_t* __restrict__ offsets, uint32_t nb,
                                               XYZZ<F>* __restrict__ buckets, int* __restrict__ pgid,
                                               XYZZ<F>* __restrict__ ppt, const AccumChunk* __restrict__ chunk,
                                               const Affine<F>* __restrict__ chunk_pts,
                                               const uint32_t* __restrict__ chunk_offsets) {
    if (chunk) {
        const AccumChunk c = *chunk;
        nb = c.b1 - c.b0;
        buckets += c.b0;
        offsets += c.b0;
        if (c.pairs) {
            pts = chunk_pts;
            sorted = nullptr;
            offsets = chunk_offsets;
        }
    }
    // buckets [0, nb) of this launch cover sorted positions [offsets[0], offsets[nb])
    const uint32_t T = gridDim.x * blockDim.x;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t M0 = offsets[0];
    const uint32_t M = offsets[nb] - M0;
    const uint32_t L = (M + T - 1) / T;
    int head_gid = -1, tail_gid = -1;
    XYZZ<F> head = XYZZ<F>::inf(), tail = XYZZ<F>::inf();
    const uint64_t rel64 = (uint64_t)t * L;
    if (L && rel64 < M) {
        const uint32_t start = M0 + (uint32_t)rel64;
        const uint32_t end = M0 + min(M, (uint32_t)rel64 + L);
        uint32_t lo = 0, hi = nb;  // offsets[lo] <= start < offsets[hi]
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (offsets[mid] <= start) lo = mid; else hi = mid;
        }
        uint32_t g = lo;
        uint32_t gbeg = offsets[g], gend = offsets[g + 1];
        XYZZ<F> acc = XYZZ<F>::inf();
        uint32_t run_start = start;
        for (uint32_t pos = start; pos < end; ++pos) {
            if (pos == gend) {
                // bucket g ended inside this slice: run [run_start, pos)
                if (gbeg < run_start) { head_gid = (int)g; head = acc; }
                else buckets[g] = acc;
                do { ++g; gbeg = gend; gend = offsets[g + 1]; } while (gend <= pos);
                acc = XYZZ<F>::inf();
                run_start = pos;
            }
            const uint32_t e = sorted ? sorted[pos] : pos;
            Affine<F> p = pts[e & 0x7fffffffu];
            if (e >> 31) p.y = F::neg(p.y);
            acc = XYZZ<F>::add_affine(acc, p);
        }
        const bool before = gbeg < run_start;
        const bool after = gend > end;
        if (before) { head_gid = (int)g; head = acc; }
        else if (after) { tail_gid = (int)g; tail = acc; }
        else buckets[g] = acc;
    }
    pgid[2 * t] = head_gid;
    pgid[2 * t + 1] = tail_gid;
    ppt[2 * t] = head;
    ppt[2 * t + 1] = tail;
}

// 4b. Pairwise levels before the accumulation, for long G1 lists: each level
// adds the points of every bucket in pairs, in affine coordinates, and halves
// the list; the accumulation then sums what is left.  An affine addition is
// six products (788 multiply-adds) where the mixed one is 1240, given
// 1 / (x2 - x1); a thread forms the running product of its K differences,
// inverts it once and walks back (Montgomery's trick), so the inversion
// (18 us) is paid once per K additions.
//
// Level k of bucket g starts at slot s_k(g), s_0 = its offset in the sorted
// list and s_k(g) = (s_(k-1)(g) + g) >> 1 = (s_0(g) + (2^k - 1) g) >> k, which leaves room for
// ceil(count / 2) points without a scan; the slots between hold no point (at
// most one a bucket and level).  A slot's descriptor names its one or two
// source points.  Slots are dealt to lanes in rows of 32, so that
// descriptors, running products and points (in planes of 16 bytes) are read
// and written in whole lines; only the first level gathers.
constexpr uint32_t PAIR_BIT = 0x80000000u, NO_POINT = 0xffffffffu;
constexpr int PAIR_LEVELS_MAX = 6;
struct PairDescs {
    uint2* first;  // level 1: two sorted entries (NO_POINT: none)
    uint32_t* next[PAIR_LEVELS_MAX];  // level k + 2: source slot | PAIR_BIT, NO_POINT
};
struct PairCaps {
    uint32_t slots[PAIR_LEVELS_MAX];  // room of level k + 1
};
DV_INL uint32_t pair_start(const uint32_t* offsets, uint32_t g) { return (uint32_t)(((uint64_t)offsets[g] + g) >> 1); }

// Chunks of about equal slots, cut at buckets; pairs = 0 where one does not
// fit its room (digits far from uniform) or holds next to nothing (scalars that
// are nearly all zero; 4096 entries are one addition a thread in k_accum, and
// in one bucket still only 64 merges in a row, less than the levels take).
constexpr uint32_t PAIR_LEAST = 4096;
__global__ void k_pair_chunks(const uint32_t* __restrict__ offsets, uint32_t nb, uint32_t chunks, int levels,
                              const PairCaps caps, AccumChunk* __restrict__ out) {
    const uint32_t c = threadIdx.x;
    if (c >= chunks) return;
    const uint64_t total = ((uint64_t)offsets[nb] + nb) >> 1, each = (total + chunks - 1) / chunks;
    uint32_t bound[2];
    for (int e = 0; e < 2; ++e) {
        const uint64_t want = each * (c + e);
        uint32_t lo = 0, hi = c + e == 0 || c + e == chunks ? 0 : nb;  // first bucket that starts at or past `want`
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (pair_start(offsets, mid) < want) lo = mid + 1; else hi = mid;
        }
        bound[e] = c + e == chunks ? nb : lo;
    }
    const uint32_t n = bound[1] - bound[0];
    uint64_t slots = offsets[bound[1]] - offsets[bound[0]];
    bool fits = n > 0 && slots >= PAIR_LEAST;
    uint32_t first = 0;
    for (int k = 0; k < levels; ++k) {
        slots = (slots + n) >> 1;
        if (k == 0) first = (uint32_t)slots;
        fits = fits && slots <= caps.slots[k];
    }
    out[c] = {bound[0], bound[1], first, fits ? 1u : 0u};
}

// Descriptors of level blockIdx.y + 1 (and, in the slice past the levels, the
// last level's bucket offsets).  A warp takes tiles of 32 rows of 32 slots: a binary
// search gives the tile's first bucket; then every row looks its slots up in
// the starts of the next 32 buckets, one a lane, so that neither many short
// buckets nor one long one cost more than their slots.
__global__ void __launch_bounds__(256) k_pair_descs(const AccumChunk* __restrict__ chunk,
                                                    const uint32_t* __restrict__ offsets,
                                                    const uint32_t* __restrict__ sorted, int levels,
                                                    const PairDescs d, uint32_t* __restrict__ last_offsets) {
    const AccumChunk ch = *chunk;
    if (!ch.pairs) return;
    const uint32_t nb = ch.b1 - ch.b0, base = offsets[ch.b0];
    const uint32_t* off = offsets + ch.b0;
    const auto start = [&](uint32_t g, int k) {
        return (uint32_t)(((uint64_t)(off[g] - base) + (uint64_t)g * ((1u << k) - 1)) >> k);
    };
    const uint32_t thread = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
    if ((int)blockIdx.y == levels) {
        for (uint32_t g = thread; g <= nb; g += threads) last_offsets[g] = start(g, levels);
        return;
    }
    const int k = (int)blockIdx.y + 1;
    const uint32_t n = start(nb, k), lane = threadIdx.x & 31;
    for (uint32_t tile = thread >> 5; (uint64_t)tile * 1024 < n; tile += threads >> 5) {
        uint32_t lo = 0, hi = nb;  // start(lo) <= the tile's first slot < start(hi)
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (start(mid, k) <= tile * 1024) lo = mid; else hi = mid;
        }
        uint32_t g0 = lo;
        for (uint32_t row = 0; row < 32 && tile * 1024 + row * 32 < n; ++row) {
            const uint32_t slot = tile * 1024 + row * 32 + lane;
            uint32_t g = 0;
            bool found = slot >= n;  // the last row's rest: any bucket
            for (uint32_t from = g0;; from += 32) {
                const uint32_t next = from + 1 + lane <= nb ? start(from + 1 + lane, k) : 0xffffffffu;
                uint32_t pos = 0;  // buckets of these 32 that end at or before the slot
#pragma unroll
                for (uint32_t step = 16; step; step >>= 1)
                    if (__shfl_sync(0xffffffffu, next, pos + step - 1) <= slot) pos += step;
                const bool past = __shfl_sync(0xffffffffu, next, pos) <= slot;  // pos = 31: all of them
                if (!found && !past) {
                    g = from + pos;
                    found = true;
                }
                if (__all_sync(0xffffffffu, found)) break;
            }
            const unsigned in = __ballot_sync(0xffffffffu, slot < n);
            g0 = __shfl_sync(0xffffffffu, g, 31 - __clz(in));
            if (slot >= n) continue;
            const uint32_t src = start(g, k - 1), cnt = (off[g + 1] - off[g] + (1u << (k - 1)) - 1) >> (k - 1);
            const uint32_t j = slot - start(g, k);
            const bool one = 2 * j < cnt, two = 2 * j + 1 < cnt;
            if (k == 1)
                d.first[slot] = {one ? sorted[base + src + 2 * j] : NO_POINT, two ? sorted[base + src + 2 * j + 1] : NO_POINT};
            else
                d.next[k - 2][slot] = one ? (src + 2 * j) | (two ? PAIR_BIT : 0u) : NO_POINT;
        }
    }
}

// What a pair gives: the sum, the double, one of the points, or infinity.
enum { PK_ADD, PK_DOUBLE, PK_FIRST, PK_SECOND, PK_NONE };
DV_INL int pair_kind(const G1A& a, const G1A& b) {
    const bool ai = a.is_inf(), bi = b.is_inf();
    if (ai || bi) return ai && bi ? PK_NONE : ai ? PK_SECOND : PK_FIRST;
    if (!(a.x == b.x)) return PK_ADD;
    return a.y == b.y && !a.y.is_zero() ? PK_DOUBLE : PK_NONE;
}
DV_INL Fq load_planes(const uint4* p, size_t stride, uint32_t i) {
    Fq r;
    const uint4 a = p[i], b = p[stride + i];
    r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
    r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
    return r;
}
DV_INL void store_planes(uint4* p, size_t stride, uint32_t i, const Fq& a) {
    p[i] = make_uint4(a.v[0], a.v[1], a.v[2], a.v[3]);
    p[stride + i] = make_uint4(a.v[4], a.v[5], a.v[6], a.v[7]);
}

// One level.  FIRST: sources are entries of the point table; else points in
// planes (four per point) of the level before.  LAST: results as whole points, with
// infinity in the slots that hold none, for the accumulation.
// Measured (MSM of 2^20 points, 17.8 M entries): 112 us per million additions
// and 60 us a level beside, against 171 us per million mixed additions; four
// blocks of 128 threads an SM (five with 96 registers 10 % slower, three 3 %).
// What bounds it is the multiply pipe, about three quarters busy; without the
// copies ahead, waiting for points took a third of the time.
constexpr int PAIR_BLOCKS = 4;
template <bool FIRST, bool LAST>
__global__ void __launch_bounds__(128, PAIR_BLOCKS) k_pair_level(const AccumChunk* __restrict__ chunk, int level,
                                                       const G1A* __restrict__ pts, const PairDescs descs,
                                                       const uint4* __restrict__ in, size_t in_stride,
                                                       uint4* __restrict__ prefix, size_t prefix_stride,
                                                       uint4* __restrict__ out, size_t out_stride) {
    const AccumChunk ch = *chunk;
    if (!ch.pairs) return;
    uint32_t n = ch.slots;
    for (int k = 1; k < level; ++k) n = (n + (ch.b1 - ch.b0)) >> 1;
    const uint32_t lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t rows = (n + 31) >> 5, each = (rows + warps - 1) / warps;
    const uint32_t r0 = min(rows, warp * each), r1 = min(rows, r0 + each);  // none: the warp only joins the barriers
    // sources of a slot: (a, b), NO_POINT where there is none
    const auto sources = [&](uint32_t slot) -> uint2 {
        if (slot >= n) return {NO_POINT, NO_POINT};
        if constexpr (FIRST) {
            return descs.first[slot];
        } else {
            const uint32_t d = descs.next[level - 2][slot];
            if (d == NO_POINT) return {NO_POINT, NO_POINT};
            const uint32_t s = d & ~PAIR_BIT;
            return {s, d & PAIR_BIT ? s + 1 : NO_POINT};
        }
    };
    // The next row's points are on their way to shared memory while a row is
    // worked on (each thread copies and reads its own: no barrier): x of both
    // at 0..3, y at 4..7, the running product at 8..9.
    __shared__ uint4 stage[2][10][128];
    const auto copy2 = [&](int buf, int at, const uint4* from, size_t step) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(
                             (uint32_t)__cvta_generic_to_shared(&stage[buf][at + h][threadIdx.x])),
                         "l"(from + h * step)
                         : "memory");
    };
    const auto copy_x = [&](int buf, int at, uint32_t e) {
        if constexpr (FIRST) copy2(buf, at, reinterpret_cast<const uint4*>(&pts[e & ~PAIR_BIT].x), 1);
        else copy2(buf, at, in + e, in_stride);
    };
    const auto copy_y = [&](int buf, int at, uint32_t e) {
        if constexpr (FIRST) copy2(buf, at, reinterpret_cast<const uint4*>(&pts[e & ~PAIR_BIT].y), 1);
        else copy2(buf, at, in + 2 * in_stride + e, in_stride);
    };
    const auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
    const auto arrived = [] { asm volatile("cp.async.wait_group 1;" ::: "memory"); };
    const auto staged = [&](int buf, int at) -> Fq {
        Fq r;
        const uint4 a = stage[buf][at][threadIdx.x], b = stage[buf][at + 1][threadIdx.x];
        r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
        r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
        return r;
    };
    const auto signed_y = [&](const Fq& y, uint32_t e) -> Fq {
        return FIRST && e >> 31 ? Fq::neg(y) : y;
    };
    const auto y_now = [&](uint32_t e) -> Fq {
        if constexpr (FIRST) return signed_y(pts[e & ~PAIR_BIT].y, e);
        else return load_planes(in + 2 * in_stride, in_stride, e);
    };
    const auto copy_xs = [&](int buf, const uint2& e) {
        if (e.y != NO_POINT) {
            copy_x(buf, 0, e.x);
            copy_x(buf, 2, e.y);
        }
        commit();
    };
    // running products of the denominators
    Fq acc = Fq::one();
    uint2 e = r0 < r1 ? sources(r0 * 32 + lane) : uint2{NO_POINT, NO_POINT};
    uint2 e1 = r0 + 1 < r1 ? sources(r0 * 32 + 32 + lane) : uint2{NO_POINT, NO_POINT};
    copy_xs(0, e);
#pragma unroll 1
    for (uint32_t r = r0; r < r1; ++r) {
        const uint32_t slot = r * 32 + lane;
        const int buf = (r - r0) & 1;
        copy_xs(buf ^ 1, e1);
        const uint2 e2 = r + 2 < r1 ? sources(slot + 64) : uint2{NO_POINT, NO_POINT};
        arrived();
        if (e.y != NO_POINT) {
            const Fq x1 = staged(buf, 0), x2 = staged(buf, 2);
            Fq d = Fq::sub(x2, x1);
            bool one = true;
            if (d.is_zero() || x1.is_zero() || x2.is_zero()) {
                const G1A a = {x1, y_now(e.x)}, b = {x2, y_now(e.y)};
                const int kind = pair_kind(a, b);
                one = kind <= PK_DOUBLE;
                if (kind == PK_DOUBLE) d = Fq::dbl(a.y);
            }
            if (one) {
                store_planes(prefix, prefix_stride, slot, acc);
                acc = Fq::mul_inl(acc, d);
            }
        }
        e = e1;
        e1 = e2;
    }
    // The block's 128 inverses from 32 inversions: warp 0 multiplies the four
    // warps' products lane by lane, inverts and splits.
    __shared__ Fq accs[128];
    accs[threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        const Fq a0 = accs[lane], a1 = accs[32 + lane], a2 = accs[64 + lane], a3 = accs[96 + lane];
        const Fq p1 = Fq::mul(a0, a1), p2 = Fq::mul(p1, a2);
        Fq i = Fq::inv(Fq::mul(p2, a3));
        accs[96 + lane] = Fq::mul(i, p2);
        i = Fq::mul(i, a3);
        accs[64 + lane] = Fq::mul(i, p1);
        i = Fq::mul(i, a2);
        accs[32 + lane] = Fq::mul(i, a0);
        accs[lane] = Fq::mul(i, a1);
    }
    __threadfence();  // the running products, before the copies that read them back
    __syncthreads();
    Fq inv = accs[threadIdx.x];
    if (r0 == r1) return;
    const auto copy_all = [&](int buf, const uint2& e, uint32_t slot) {
        if (e.x != NO_POINT) {
            copy_x(buf, 0, e.x);
            copy_y(buf, 4, e.x);
        }
        if (e.y != NO_POINT) {
            copy_x(buf, 2, e.y);
            copy_y(buf, 6, e.y);
            copy2(buf, 8, prefix + slot, prefix_stride);
        }
        commit();
    };
    // back: 1 / d of each pair, its sum, and the denominator taken out of inv
    const uint32_t last = (r1 - 1) * 32 + lane;
    e = sources(last);
    e1 = r1 - r0 > 1 ? sources(last - 32) : uint2{NO_POINT, NO_POINT};
    copy_all(0, e, last);
#pragma unroll 1
    for (uint32_t r = r1; r-- > r0;) {
        const uint32_t slot = r * 32 + lane;
        const int buf = (r1 - 1 - r) & 1;
        copy_all(buf ^ 1, e1, slot - 32);
        const uint2 e2 = r >= r0 + 2 ? sources(slot - 64) : uint2{NO_POINT, NO_POINT};
        arrived();
        G1A p = G1A::inf();
        if (e.x != NO_POINT) {
            p = {staged(buf, 0), signed_y(staged(buf, 4), e.x)};
            if (e.y != NO_POINT) {
                const G1A b = {staged(buf, 2), signed_y(staged(buf, 6), e.y)};
                Fq d = Fq::sub(b.x, p.x), num = Fq::sub(b.y, p.y);
                int kind = PK_ADD;
                if (d.is_zero() || p.x.is_zero() || b.x.is_zero()) {
                    kind = pair_kind(p, b);
                    if (kind == PK_DOUBLE) {
                        d = Fq::dbl(p.y);
                        const Fq xx = Fq::sqr(p.x);
                        num = Fq::add(Fq::dbl(xx), xx);
                    } else if (kind == PK_SECOND) {
                        p = b;
                    } else if (kind == PK_NONE) {
                        p = G1A::inf();
                    }
                }
                if (kind <= PK_DOUBLE) {
                    // inlined: a call moves its operands, on the multiply pipe too
                    const Fq lam = Fq::mul_inl(Fq::mul_inl(inv, staged(buf, 8)), num);
                    inv = Fq::mul_inl(inv, d);
                    const Fq x3 = Fq::sub(Fq::sub(Fq::sqr_inl(lam), p.x), b.x);
                    p.y = Fq::sub(Fq::mul_inl(lam, Fq::sub(p.x, x3)), p.y);
                    p.x = x3;
                }
            }
        }
        const bool some = e.x != NO_POINT;
        e = e1;
        e1 = e2;
        if constexpr (LAST) {
            if (slot < n) reinterpret_cast<G1A*>(out)[slot] = p;
        } else if (some) {
            store_planes(out, out_stride, slot, p.x);
            store_planes(out + 2 * out_stride, out_stride, slot, p.y);
        }
    }
}

// 5. Merge partials of buckets that span slices.  The owner of bucket g is
// the slice whose tail holds g; the following slices hold g in their heads.
// A lane quad per slice adds up to FIX_SHORT heads in turn (most buckets are
// cut once).  Longer chains (skewed digits, few buckets) are queued: k_fixup_long
// gives each a warp, eight quads and a three-step tree, and those of more
// than FIX_WARP heads a block.  A merge is 2.5 us (G2: 5) where a thread's
// took 6: 1000 points 33 -> 9 us; limits of 4, 8 and 16 measured the same.
// The queue is dealt to the blocks item by item, so that a skewed call's
// longest chains (a few windows' buckets: 10 to 130) run side by side; with eight
// neighbours to a block it took them in turn (one value everywhere, 30000 points
// over a c = 16 table, whole call: 2.41 ms, 0.58 so).
constexpr uint32_t FIX_SHORT = 8, FIX_WARP = 256;

template <class F>
__global__ void __launch_bounds__(256) k_fixup(const int* __restrict__ pgid, const XYZZ<F>* __restrict__ ppt, uint32_t T,
                        XYZZ<F>* __restrict__ buckets, uint32_t* __restrict__ long_list,
                        uint32_t* __restrict__ long_count, const AccumChunk* __restrict__ chunk) {
    if (chunk) buckets += chunk->b0;
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 2, r = threadIdx.x & 3;
    const int g = t < T ? pgid[2 * t + 1] : -1;
    uint32_t heads = 0;
    if (g >= 0)
        while (heads <= FIX_SHORT && t + 1 + heads < T && pgid[2 * (t + 1 + heads)] == g) ++heads;
    const bool queued = heads > FIX_SHORT;
    if (queued && r == 0) long_list[atomicAdd(long_count, 1u)] = t;
    if (queued || g < 0) heads = 0;
    const F* parts = reinterpret_cast<const F*>(ppt);
    F acc = g >= 0 ? parts[(size_t)(2 * t + 1) * 4 + r] : Quad<F>::inf();
    for (uint32_t k = 1; __any_sync(0xffffffffu, k <= heads); ++k)
        acc = Quad<F>::add(acc, k <= heads ? parts[(size_t)(2 * (t + k)) * 4 + r] : Quad<F>::inf());
    if (g >= 0 && !queued) reinterpret_cast<F*>(buckets)[(size_t)g * 4 + r] = acc;
}

// The sum over the quads of a group of lanes: quad 0 ends with it.
template <class F>
DV_INL F quads_sum_warp(F acc) {
#pragma unroll 1
    for (int d = 16; d >= 4; d >>= 1) acc = Quad<F>::add(acc, shfl_xor(acc, d));
    return acc;
}

template <class F>
__global__ void __launch_bounds__(256) k_fixup_long(const int* __restrict__ pgid, const XYZZ<F>* __restrict__ ppt,
                                                   uint32_t T, XYZZ<F>* __restrict__ buckets,
                                                   const uint32_t* __restrict__ long_list,
                                                   const uint32_t* __restrict__ long_count,
                                                   const AccumChunk* __restrict__ chunk) {
    __shared__ F warp_sum[8][4];
    __shared__ uint32_t huge[8];
    if (chunk) buckets += chunk->b0;
    const uint32_t nlong = *long_count, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = threadIdx.x & 3;
    const F* parts = reinterpret_cast<const F*>(ppt);
    F* out = reinterpret_cast<F*>(buckets);
    // heads of g at positions from + step k, while they are g's (contiguous from t0 + 1)
    const auto add_heads = [&](F acc, int g, uint32_t from, uint32_t step) {
        for (uint32_t k = from;; k += step) {
            const bool have = k < T && pgid[2 * k] == g;
            if (!__any_sync(0xffffffffu, have)) return acc;
            acc = Quad<F>::add(acc, have ? parts[(size_t)(2 * k) * 4 + r] : Quad<F>::inf());
        }
    };
    for (uint64_t base = blockIdx.x; base < nlong; base += 8ull * gridDim.x) {
        const uint64_t at = base + (uint64_t)gridDim.x * warp;
        const uint32_t item = at < nlong ? (uint32_t)at : nlong;
        bool is_huge = false;
        if (item < nlong) {
            const uint32_t t0 = long_list[item], far = t0 + 1 + FIX_WARP;
            const int g = pgid[2 * t0 + 1];
            is_huge = far < T && pgid[2 * far] == g;
            if (!is_huge) {
                F acc = lane < 4 ? parts[(size_t)(2 * t0 + 1) * 4 + r] : Quad<F>::inf();
                acc = quads_sum_warp<F>(add_heads(acc, g, t0 + 1 + (lane >> 2), 8));
                if (lane < 4) out[(size_t)g * 4 + r] = acc;
            }
        }
        if (lane == 0) huge[warp] = is_huge ? item : 0xffffffffu;
        __syncthreads();
        for (int h = 0; h < 8; ++h) {
            if (huge[h] == 0xffffffffu) continue;
            const uint32_t t0 = long_list[huge[h]];
            const int g = pgid[2 * t0 + 1];
            F acc = threadIdx.x < 4 ? parts[(size_t)(2 * t0 + 1) * 4 + r] : Quad<F>::inf();
            acc = quads_sum_warp<F>(add_heads(acc, g, t0 + 1 + (threadIdx.x >> 2), 64));
            if (lane < 4) warp_sum[warp][r] = acc;
            __syncthreads();
            if (warp == 0) {
                acc = quads_sum_warp<F>(warp_sum[lane >> 2][r]);
                if (lane < 4) out[(size_t)g * 4 + r] = acc;
            }
            __syncthreads();
        }
        __syncthreads();
    }
}

// 6. Bucket reduction.  Window (set, w) needs
//      S_w = sum_b (b + 1) B_b,   b < 2^(c-1).
// Every level carries a window as pairs (U_j, V_j) with
//      S_w = sum_j U_j + sum_j j V_j ,
// V_j already multiplied by the weight unit of its level.  Level 1:
// segment j holds buckets [j s, (j+1) s); a running sum from the top gives
//      U_j = sum_i (i + 1) B_{js+i},   V_j = s sum_i B_{js+i}.
// Grouping G consecutive pairs (j = G q + l) gives the next level:
//      U'_q = sum_l U_{Gq+l} + sum_l l V_{Gq+l} = sum_l (U_l + Suf_{l+1}),
//      V'_q = G sum_l V_{Gq+l},
// with Suf the group's suffix sums of V; the doublings for G apply to one
// sum per group, so the critical path holds log2(total weight) of them.

// Additions and doublings of the reduction: few threads per bucket set on a
// dependent chain, so over Fq the products go out in pairs.
template <class F>
DV_INL XYZZ<F> wadd(const XYZZ<F>& p, const XYZZ<F>& q) {
    if constexpr (sizeof(F) == sizeof(Fq)) return XYZZ<F>::add_paired(p, q);
    else return XYZZ<F>::add(p, q);
}
template <class F>
DV_INL XYZZ<F> wdbl(const XYZZ<F>& p) {
    if constexpr (sizeof(F) == sizeof(Fq)) return XYZZ<F>::dbl_paired(p);
    else return XYZZ<F>::dbl(p);
}
// Level 1: one segment of s buckets per thread.
template <class F>
__global__ void __launch_bounds__(128) k_segments(const XYZZ<F>* __restrict__ buckets, const uint32_t* __restrict__ offsets,
                                                  uint32_t B, uint32_t NW, int seg_log, XYZZ<F>* __restrict__ seg_u,
                                                  XYZZ<F>* __restrict__ seg_v) {
    const uint32_t S = B >> seg_log;
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
    if (tid >= NW * S) return;
    const uint32_t w = tid / S, j = tid % S;
    const uint32_t s = 1u << seg_log;
    XYZZ<F> R = XYZZ<F>::inf(), U = XYZZ<F>::inf();
    const size_t base = (size_t)w * B + (size_t)j * s;
    for (int b = (int)s - 1; b >= 0; --b) {
        const size_t g = base + b;
        if (offsets[g + 1] != offsets[g]) R = wadd<F>(R, buckets[g]);
        U = wadd<F>(U, R);
    }
    for (int i = 0; i < seg_log; ++i) R = wdbl<F>(R);  // V = s R
    seg_u[tid] = U;
    seg_v[tid] = R;
}

// Upper levels: blocks of WTREE pairs (G = WTREE), windows of S pairs; S <=
// WTREE is the last level (one block per window, its U' is S_w).  A binary
// tree: pairs 2j and 2j + 1 give
//      U = U_a + U_b + V_b,   V = 2 (V_a + V_b),
// one lane quad for each of the two, so a tree level is two dependent point
// operations whatever the number of pairs, and V ends multiplied by G.  A
// window of S pairs is the latency of 2 log2(S) operations of 2.5 us (G2: 5 us),
// where suffix scans by one lane a point took 26 operations of 6 us a level.
// All upper levels of one MSM: 2^18 buckets, 310 -> 158 us; 1000 points, 115 ->
// 49 us; G2, 2^16 points, 627 -> 392 us.
constexpr int WTREE = 64;
template <class F>
__global__ void __launch_bounds__(256) k_wtree(const XYZZ<F>* __restrict__ u_in, const XYZZ<F>* __restrict__ v_in,
                                               uint32_t S, XYZZ<F>* __restrict__ u_out, XYZZ<F>* __restrict__ v_out,
                                               const uint32_t* bad, const uint32_t* points_bad, uint32_t* host_bad) {
    __shared__ F sh[2 * WTREE][4];  // U, then V
    const uint32_t nblk = S > (uint32_t)WTREE ? S / WTREE : 1u;
    const uint32_t w = blockIdx.x / nblk, k = blockIdx.x % nblk;
    const uint32_t width = S < (uint32_t)WTREE ? S : (uint32_t)WTREE;
    const size_t first = ((size_t)w * S + (size_t)k * WTREE) * 4;
    for (uint32_t i = threadIdx.x; i < 4 * width; i += 256) {
        (&sh[0][0])[i] = reinterpret_cast<const F*>(u_in)[first + i];
        (&sh[WTREE][0])[i] = reinterpret_cast<const F*>(v_in)[first + i];
    }
    __syncthreads();
    const uint32_t quad = threadIdx.x >> 2, r = threadIdx.x & 3;
    for (uint32_t m = width / 2; m >= 1; m >>= 1) {
        // U on the first quads, V on the next, never both in one warp
        const uint32_t v0 = m < 8 ? 8 : m;
        const bool is_u = quad < m, is_v = quad >= v0 && quad < v0 + m;
        const uint32_t j = is_u ? quad : quad - v0;
        const bool warp_u = (threadIdx.x >> 5) * 8 < m;
        const bool warp_v = !warp_u && (threadIdx.x >> 5) * 8 < v0 + m;
        F s = Quad<F>::inf();
        if (warp_u || warp_v) {
            const F* x = &sh[is_v ? WTREE : 0][0];
            const bool live = is_u || is_v;
            s = Quad<F>::add(live ? x[(2 * j) * 4 + r] : Quad<F>::inf(), live ? x[(2 * j + 1) * 4 + r] : Quad<F>::inf());
            if (warp_u) s = Quad<F>::add(s, is_u ? sh[WTREE + 2 * j + 1][r] : Quad<F>::inf());
            else if (__any_sync(0xffffffffu, r == 2 && !s.is_zero())) s = Quad<F>::dbl(s);
        }
        __syncthreads();
        if (is_u) sh[j][r] = s;
        if (is_v) sh[WTREE + j][r] = s;
        __syncthreads();
    }
    if (threadIdx.x < 4) {
        reinterpret_cast<F*>(u_out)[(size_t)blockIdx.x * 4 + r] = sh[0][r];
        if (nblk > 1) reinterpret_cast<F*>(v_out)[(size_t)blockIdx.x * 4 + r] = sh[WTREE][r];
    }
    if (host_bad && blockIdx.x == 0 && threadIdx.x == 0) {
        host_bad[0] = *bad;
        host_bad[1] = points_bad ? *points_bad : NO_INDEX;
    }
}

// Window multiples of resident bases: table[i W + w] = 2^(c w) P_i (affine,
// Montgomery).  One thread per base, c doublings per window, normalised with
// one inversion per warp per window (warp_batch_inverse: every lane takes
// part, so lanes past n carry infinity).
template <class F>
__global__ void __launch_bounds__(128) k_precompute(const Affine<F>* __restrict__ bases, uint64_t n, int W, int c,
                                                    Affine<F>* __restrict__ table) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = i < n;
    XYZZ<F> acc = active ? XYZZ<F>::from_affine(bases[i]) : XYZZ<F>::inf();
    for (int w = 0; w < W; ++w) {
        const bool inf = acc.is_inf();
        const F d = warp_batch_inverse<F>(inf ? F::one() : F::mul(acc.zz, acc.zzz));
        if (active) {
            table[i * (uint64_t)W + w] =
                inf ? Affine<F>::inf()
                    : Affine<F>{F::mul(acc.x, F::mul(d, acc.zzz)), F::mul(acc.y, F::mul(d, acc.zz))};
        }
        if (w + 1 < W)
            for (int k = 0; k < c; ++k) acc = XYZZ<F>::dbl(acc);
    }
}

// Canonical -> Montgomery conversion with validation.
DV_INL bool all_zero_words(const uint32_t* w, int n) {
    uint32_t x = 0;
    for (int i = 0; i < n; ++i) x |= w[i];
    return x == 0;
}

__global__ void k_convert_g1(const uint8_t* __restrict__ canon, G1A* __restrict__ out, uint64_t n,
                             uint32_t* __restrict__ first_bad) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t x[8], y[8];
    load_words(canon + 64 * i, x);
    load_words(canon + 64 * i + 32, y);
    G1A p;
    if (all_zero_words(x, 8) && all_zero_words(y, 8)) {
        p = G1A::inf();
    } else {
        if (!Fq::is_canonical(x) || !Fq::is_canonical(y)) { atomicMin(first_bad, (uint32_t)i); return; }
        p.x = Fq::from_canonical(x);
        p.y = Fq::from_canonical(y);
        if (!CurveOps<Fq>::on_curve(p)) { atomicMin(first_bad, (uint32_t)i); return; }
    }
    out[i] = p;
}

__global__ void k_convert_g2(const uint8_t* __restrict__ canon, G2A* __restrict__ out, uint64_t n,
                             uint32_t* __restrict__ first_bad) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t w[4][8];
    bool zero = true;
    for (int j = 0; j < 4; ++j) {
        load_words(canon + 128 * i + 32 * j, w[j]);
        zero &= all_zero_words(w[j], 8);
    }
    G2A p;
    if (zero) {
        p = G2A::inf();
    } else {
        for (int j = 0; j < 4; ++j)
            if (!Fq::is_canonical(w[j])) { atomicMin(first_bad, (uint32_t)i); return; }
        p.x = {Fq::from_canonical(w[0]), Fq::from_canonical(w[1])};
        p.y = {Fq::from_canonical(w[2]), Fq::from_canonical(w[3])};
        if (!CurveOps<Fq2>::on_curve(p)) { atomicMin(first_bad, (uint32_t)i); return; }
    }
    out[i] = p;
}

template <class F>
__global__ void k_gather(const Affine<F>* __restrict__ bases, uint64_t nbases, int W, const uint64_t* __restrict__ idx,
                         uint64_t k, Affine<F>* __restrict__ out, uint32_t* __restrict__ first_bad) {
    // W entries per index: a table of window multiples (W = 1: the bases)
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= k * (uint64_t)W) return;
    const uint64_t j = t / (uint64_t)W, w = t % (uint64_t)W;
    const uint64_t i = idx[j];
    if (i >= nbases) { atomicMin(first_bad, (uint32_t)j); return; }
    out[t] = bases[i * W + w];
}

inline unsigned blocks_for(uint64_t n, unsigned threads) { return (unsigned)((n + threads - 1) / threads); }

// Host Horner over windows: sum_w 2^(c w) S_w.
template <class HF>
void horner(const dvh::XYZZ<HF>* win, int W, int c, uint8_t* out) {
    dvh::XYZZ<HF> acc = dvh::xyzz_inf<HF>();
    for (int w = W - 1; w >= 0; --w) {
        for (int k = 0; k < c; ++k) acc = dvh::xyzz_dbl(acc);
        acc = dvh::xyzz_add(acc, win[w]);
    }
    dvh::xyzz_to_affine_bytes(acc, out);
}

// Device tail of one MSM per thread: Horner over the set's window sums, then
// affine normalisation (infinity stays all-zero bytes).
template <class F>
__global__ void __launch_bounds__(64) k_msm_finish(const XYZZ<F>* __restrict__ win, uint32_t count, int W, int c,
                                                   const uint32_t* __restrict__ out_idx, uint8_t* __restrict__ out) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= count) return;
    const XYZZ<F>* w = win + (size_t)k * W;
    XYZZ<F> acc = w[W - 1];
    for (int j = W - 2; j >= 0; --j) {
        if (!acc.is_inf())
            for (int d = 0; d < c; ++d) acc = XYZZ<F>::dbl(acc);
        acc = XYZZ<F>::add(acc, w[j]);
    }
    uint8_t* o = out + (size_t)(out_idx ? out_idx[k] : k) * 2 * sizeof(F);
    if (acc.is_inf()) {
        const uint4 z = make_uint4(0, 0, 0, 0);
        for (size_t b = 0; b < 2 * sizeof(F); b += 16) *reinterpret_cast<uint4*>(o + b) = z;
        return;
    }
    const Affine<F> a = acc.to_affine();
    store_canonical(o, a.x);
    store_canonical(o + sizeof(F), a.y);
}

template <class F>
struct HostOf;
template <>
struct HostOf<Fq> { typedef dvh::Fq T; };
template <>
struct HostOf<Fq2> { typedef dvh::Fq2 T; };

}  // namespace

// Default window width by size class: the autotuner's choices on B200 over
// 2^8..2^22 points, G1 and G2 alike.  Widths whose ceil(255 / c) windows
// leave few spare bits (5, 8, 10, 15, 16) win, by up to a quarter against
// the cost model's choice (2^16 points: c = 15 in 0.96 ms against the model's
// 13 in 1.28 ms).  0 outside the measured classes.
static int measured_c(uint64_t n) {
    int k = 0;
    while (k < 63 && (1ull << k) < n) ++k;
    if (k >= 8 && k <= 9) return 5;
    if (k >= 10 && k <= 12) return 8;
    if (k >= 13 && k <= 15) return 10;
    if (k >= 16 && k <= 20) return 15;
    if (k >= 21 && k <= 22) return 16;
    return 0;
}

int msm_seg_log(uint64_t all_buckets, uint32_t buckets, int c, bool g1) {
    // Long windows (a precomputed table's single bucket set of 2^18 or more
    // G1 buckets) take 16-bucket segments: fewer upper-level entries for a
    // modest first level; shorter windows and G2, whose additions cost three
    // times as much, keep 8 (G1 2^20 points: 3.60 ms with 8 or 16, 3.69 with 4;
    // G2 2^16 points: 1.80 with 8 or 16, 2.12 with 4).
    int seg_want = (g1 && buckets >= (1u << 18)) ? DV_SEG_LOG + 1 : DV_SEG_LOG;
    // Few buckets in all (sparse updates over a precomputed table, small
    // MSMs): the reduction is a latency chain, so keep about 2^15 first-level
    // threads and shorten the segments (128 buckets: one bucket each).
    int room = 0;
    while ((all_buckets >> (room + 1)) >= (1u << 15)) ++room;
    // Many buckets in all (a batch of sets over one table, 2^21 buckets or
    // more): longer segments, up to 64 buckets, while at least 2^17
    // first-level threads remain (several waves of k_segments at two blocks
    // per SM).  A bucket costs two additions in a segment, a segment four
    // operations in the tree above.
    int wide = 0;
    while (wide < 6 && (all_buckets >> (wide + 1)) >= (1u << 17)) ++wide;
    seg_want = std::min(std::max(seg_want, wide), room);
    return std::min(seg_want, c - 1);
}

MsmPlan msm_plan(uint64_t n, int force_c) {
    MsmPlan p;
    int best_c = 4;
    double best = 1e300;
    for (int c = 4; c <= 20; ++c) {
        const double W = (255 + c - 1) / c;
        const double cost = W * (10.0 * (double)n + 28.0 * (double)(1u << (c - 1)));
        if (cost < best) { best = cost; best_c = c; }
    }
    if (const int m = measured_c(n)) best_c = m;
    p.c = force_c ? force_c : best_c;
    p.windows = (255 + p.c - 1) / p.c;
    p.buckets = 1u << (p.c - 1);
    p.seg_log = std::min(DV_SEG_LOG, p.c - 1);
    return p;
}

template <class F>
void convert_points(const uint8_t* d_canon, Affine<F>* d_out, uint64_t n, uint32_t* d_first_bad, cudaStream_t st) {
    if (!n) return;
    if constexpr (sizeof(F) == sizeof(Fq)) k_convert_g1<<<blocks_for(n, 128), 128, 0, st>>>(d_canon, d_out, n, d_first_bad);
    else k_convert_g2<<<blocks_for(n, 128), 128, 0, st>>>(d_canon, d_out, n, d_first_bad);
    DV_LAUNCH();
}

template <class F>
void gather_points(const Affine<F>* d_bases, uint64_t nbases, const uint64_t* d_idx, uint64_t k, Affine<F>* d_out,
                   uint32_t* d_first_bad, cudaStream_t st) {
    if (!k) return;
    k_gather<F><<<blocks_for(k, 256), 256, 0, st>>>(d_bases, nbases, 1, d_idx, k, d_out, d_first_bad);
    DV_LAUNCH();
}

template <class F>
void gather_table(const Affine<F>* d_table, uint64_t nbases, int W, const uint64_t* d_idx, uint64_t k,
                  Affine<F>* d_out, uint32_t* d_first_bad, cudaStream_t st) {
    if (!k) return;
    k_gather<F><<<blocks_for(k * (uint64_t)W, 256), 256, 0, st>>>(d_table, nbases, W, d_idx, k, d_out, d_first_bad);
    DV_LAUNCH();
}
template void gather_table<Fq>(const Affine<Fq>*, uint64_t, int, const uint64_t*, uint64_t, Affine<Fq>*, uint32_t*,
                               cudaStream_t);

template <class F>
MsmPlan msm_plan_batch(uint32_t count, uint32_t max_set, uint64_t total, int force_c, const MsmPrecomp<F>* pre) {
    MsmPlan plan = msm_plan(max_set, force_c);
    if (!force_c && !pre && count > 1) {
        // every set carries windows * 2^(c-1) buckets: minimise
        // windows * (10 total + 2 * 28 * count * 2^(c-1)) (the reduction
        // runs at about half the accumulation's efficiency)
        double best = 1e300;
        for (int c = 4; c <= 20; ++c) {
            const double W = (255 + c - 1) / c;
            const double cost = W * (10.0 * (double)total + 56.0 * (double)count * (double)(1u << (c - 1)));
            if (cost < best) { best = cost; plan.c = c; }
        }
        plan.windows = (255 + plan.c - 1) / plan.c;
        plan.buckets = 1u << (plan.c - 1);
        plan.seg_log = std::min(DV_SEG_LOG, plan.c - 1);
    }
    // Bound the bucket table of a batch: count * windows * buckets <= 2^26
    // (8 GB of G1 XYZZ buckets); smaller windows trade buckets for windows.
    while (plan.c > 4 && (uint64_t)count * plan.windows * plan.buckets > (1ull << 26)) {
        plan.c--;
        plan.windows = (255 + plan.c - 1) / plan.c;
        plan.buckets = 1u << (plan.c - 1);
        plan.seg_log = std::min(DV_SEG_LOG, plan.c - 1);
    }
    if (pre) {
        // precomputed window multiples: the table fixes c and the window count
        plan.c = pre->c;
        plan.windows = pre->windows;
        plan.buckets = 1u << (plan.c - 1);
        plan.seg_log = std::min(DV_SEG_LOG, plan.c - 1);
    }
    return plan;
}

// Steps 4 and 5: bucket sums of the sorted list of up to `entries` entries.
// Pairwise levels pay once a thread has enough additions for its inversion:
// level k runs while the list that it makes leaves PAIR_MIN_ROWS slots a
// lane and a bucket still holds about four points.  Long lists go in chunks
// of up to PAIR_CHUNK slots, so that the levels' room (about 150 bytes a
// slot: 1.43 GB for 2^20 points) stays below PAIR_ROOM bytes a workspace whatever
// the launch.  Where the device has no such room left, the list is accumulated
// without levels, and the room is given back to any other allocation of its owner.
// MSM of 2^20 points: 4.11 ms without levels, 3.57 with; 32 proofs of 65536 gates
// 34.9 and 33.5 ms.  The least slots a lane, over 18 lists of 200000 to 4 M points
// and 16 over tables of c = 16 and 13: 18 to 22 are within 1.5 % of each other at
// every size; 14 is up to 6 % slower (150000 points, c = 16), 28 and 36 gain up to
// 4 % at 200000 points and lose 4 to 9 % over the c = 13 table.  18, because lists
// with few full buckets gain by every level (300001 scalars 0 and 1: 1.06 ms, with
// 20 1.90).
constexpr uint64_t PAIR_MIN_ROWS = 18, PAIR_CHUNK = 12u << 20;
constexpr size_t PAIR_ROOM = 2100u << 20;

// The levels' room, or null.  A launch that is captured takes what an earlier one
// of its shapes left: nothing can be allocated then.
inline uint8_t* pair_room(MsmWorkspace& ws, size_t bytes, cudaStream_t st) {
    if (ws.pairs.cap < bytes) {
        cudaStreamCaptureStatus capture;
        DV_CUDA(cudaStreamIsCapturing(st, &capture));
        if (capture != cudaStreamCaptureStatusNone) return nullptr;
    }
    return static_cast<uint8_t*>(ws.pairs.try_get(bytes, PAIR_ROOM));
}

template <class F>
void accumulate(MsmWorkspace& ws, const Affine<F>* pts, const uint32_t* d_sorted, const uint32_t* d_offsets,
                uint32_t NB, uint64_t entries, XYZZ<F>* d_buckets, cudaStream_t st) {
    int per_sm = 0;
    DV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_accum<F>, 128, 0));
    per_sm = std::max(1, per_sm);
    uint32_t grid = (uint32_t)sm_count() * (uint32_t)per_sm;
    // small inputs: keep at least ~8 entries per thread
    grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(grid, (entries + 8 * 128 - 1) / (8 * 128)));
    const uint32_t T = grid * 128;
    int* d_pgid = ws.pgid.as<int>(2ull * T);
    XYZZ<F>* d_ppt = ws.ppt.as<XYZZ<F>>(2ull * T);
    uint32_t* d_fix_count = ws.fix_count.as<uint32_t>(1);
    uint32_t* d_fix_list = ws.fix_list.as<uint32_t>(T / FIX_SHORT + 1);
    const auto sum_and_merge = [&](const AccumChunk* chunk, const Affine<F>* chunk_pts, const uint32_t* chunk_off) {
        k_accum<F><<<grid, 128, 0, st>>>(pts, d_sorted, d_offsets, NB, d_buckets, d_pgid, d_ppt, chunk, chunk_pts,
                                         chunk_off);
        DV_LAUNCH();
        if (!chunk && ws.timeline.enabled) DV_CUDA(cudaEventRecord(ws.timeline.acc_ev[1], st));
        DV_CUDA(cudaMemsetAsync(d_fix_count, 0, sizeof(uint32_t), st));
        k_fixup<F><<<blocks_for(4ull * T, 256), 256, 0, st>>>(d_pgid, d_ppt, T, d_buckets, d_fix_list, d_fix_count,
                                                               chunk);
        DV_LAUNCH();
        // long chains are rare: a small grid loops over the queue
        k_fixup_long<F><<<std::min<uint32_t>(T / FIX_SHORT / 8 + 1, (uint32_t)sm_count() * 2), 256, 0, st>>>(
            d_pgid, d_ppt, T, d_buckets, d_fix_list, d_fix_count, chunk);
        DV_LAUNCH();
    };
    if constexpr (sizeof(F) == sizeof(Fq)) {
        const uint64_t lanes = (uint64_t)sm_count() * PAIR_BLOCKS * 128;
        const uint64_t chunks = std::max<uint64_t>(1, ((entries + NB) / 2 + PAIR_CHUNK - 1) / PAIR_CHUNK);
        // slots of each level for a chunk of even digits; its room is an eighth over
        const uint64_t e = entries / chunks, b = NB / chunks;
        PairCaps caps{};
        int levels = 0;
        uint64_t slots = e, room_slots = e + e / 8 + 1024;
        for (uint64_t per_bucket = entries / NB; levels < PAIR_LEVELS_MAX && per_bucket >= 4; per_bucket /= 2) {
            slots = (slots + b) / 2;
            if (slots < PAIR_MIN_ROWS * lanes) break;
            room_slots = (room_slots + b + b / 8 + 1024) / 2;
            caps.slots[levels++] = (uint32_t)room_slots;
        }
        AccumChunk* d_chunks = nullptr;
        uint32_t* d_last = nullptr;
        uint8_t* room = nullptr;
        if (levels && chunks <= 1024) {
            d_chunks = ws.pair_chunks.as<AccumChunk>(chunks);
            d_last = ws.pair_offsets.as<uint32_t>((size_t)NB + 1);
            size_t room_bytes = (size_t)caps.slots[0] * (8 + 64 + 32) + 16 * (PAIR_LEVELS_MAX + 4);
            if (levels > 1) room_bytes += 64 * (size_t)caps.slots[1];
            for (int k = 1; k < levels; ++k) room_bytes += 4 * (size_t)caps.slots[k];
            room = pair_room(ws, room_bytes, st);  // last: an allocation could give it back
        }
        if (room) {
            const size_t c1 = caps.slots[0], c2 = levels > 1 ? caps.slots[1] : 0;
            PairDescs descs{};
            size_t at = 0;
            const auto take = [&](size_t bytes) {
                uint8_t* p = room + at;
                at += (bytes + 15) & ~(size_t)15;
                return p;
            };
            uint4* prefix = reinterpret_cast<uint4*>(take(32 * c1));
            uint4* buf[2] = {reinterpret_cast<uint4*>(take(64 * c1)), reinterpret_cast<uint4*>(take(64 * c2))};
            descs.first = reinterpret_cast<uint2*>(take(8 * c1));
            for (int k = 1; k < levels; ++k) descs.next[k - 1] = reinterpret_cast<uint32_t*>(take(4 * (size_t)caps.slots[k]));
            k_pair_chunks<<<1, 1024, 0, st>>>(d_offsets, NB, (uint32_t)chunks, levels, caps, d_chunks);
            DV_LAUNCH();
            const uint32_t pgrid = (uint32_t)sm_count() * PAIR_BLOCKS;
            for (uint64_t c = 0; c < chunks; ++c) {
                const AccumChunk* ch = d_chunks + c;
                k_pair_descs<<<dim3(sm_count() * 8, levels + 1), 256, 0, st>>>(ch, d_offsets, d_sorted, levels, descs,
                                                                              d_last);
                DV_LAUNCH();
                const size_t stride[2] = {c1, c2};
                for (int k = 1; k <= levels; ++k) {
                    const uint4* in = k > 1 ? buf[k & 1] : nullptr;
                    uint4* out = buf[(k + 1) & 1];
                    const size_t is = stride[k & 1], os = stride[(k + 1) & 1];
                    if (k == 1 && levels == 1)
                        k_pair_level<true, true><<<pgrid, 128, 0, st>>>(ch, k, pts, descs, in, is, prefix, c1, out, os);
                    else if (k == 1)
                        k_pair_level<true, false><<<pgrid, 128, 0, st>>>(ch, k, pts, descs, in, is, prefix, c1, out, os);
                    else if (k == levels)
                        k_pair_level<false, true><<<pgrid, 128, 0, st>>>(ch, k, pts, descs, in, is, prefix, c1, out, os);
                    else
                        k_pair_level<false, false><<<pgrid, 128, 0, st>>>(ch, k, pts, descs, in, is, prefix, c1, out, os);
                    DV_LAUNCH();
                }
                sum_and_merge(ch, reinterpret_cast<const Affine<F>*>(buf[(levels + 1) & 1]), d_last);
            }
            if (ws.timeline.enabled) DV_CUDA(cudaEventRecord(ws.timeline.acc_ev[1], st));
            return;
        }
    }
    sum_and_merge(nullptr, nullptr, nullptr);
}

template <class F>
void msm_enqueue(MsmWorkspace& ws, const Affine<F>* d_points, const uint32_t* d_scalars, const SetMap& map,
                 uint32_t n, const MsmPlan& plan, const MsmPrecomp<F>* pre, uint32_t* d_err, cudaStream_t st,
                 const MsmHost<F>* host) {
    const uint32_t count = map.count;
    const int c = plan.c, W = plan.windows;
    const uint32_t B = plan.buckets;
    const uint32_t Wr = pre ? 1u : (uint32_t)W;  // bucket sets (reduction windows) per MSM
    if (pre && (uint64_t)n * plan.windows >= (1ull << 31)) throw InvalidArgument("precomputed MSM too large");
    if ((uint64_t)count * Wr * plan.buckets > (1ull << 31) || (uint64_t)n * plan.windows > 0xffffffffull)
        throw InvalidArgument("MSM batch too large for one launch sequence");
    const uint32_t NW = count * Wr;
    const uint32_t NB = NW * B;

    uint32_t* d_counts = ws.counts.as<uint32_t>(NB);
    uint32_t* d_offsets = ws.offsets.as<uint32_t>(NB + 1);
    uint32_t* d_cursor = ws.cursor.as<uint32_t>(NB);
    uint32_t* d_sorted = ws.sorted.as<uint32_t>((size_t)n * W);
    XYZZ<F>* d_buckets = ws.buckets.as<XYZZ<F>>(NB);
    DV_CUDA(cudaMemsetAsync(d_counts, 0, (size_t)NB * sizeof(uint32_t), st));

    MsmTimeline& tl = ws.timeline;
    auto mark = [&](int k) {
        if (tl.enabled) DV_CUDA(cudaEventRecord(tl.ev[k], st));
    };
    mark(0);
    // threads a scalar: one once the scalars alone fill the GPU
    const uint32_t share = (uint32_t)std::clamp<uint64_t>((uint64_t)sm_count() * 1024 / n, 1, (uint64_t)W);
    const dim3 digit_grid(blocks_for(n, 256), share);
    if (pre) k_hist<true><<<digit_grid, 256, 0, st>>>(d_scalars, n, map, c, W, d_counts, d_err);
    else k_hist<false><<<digit_grid, 256, 0, st>>>(d_scalars, n, map, c, W, d_counts, d_err);
    DV_LAUNCH();
    mark(1);
    if (NB <= SCAN_ONE) {
        k_scan_one<<<1, 1024, 0, st>>>(d_counts, NB, d_offsets, d_cursor);
        DV_LAUNCH();
    } else {
        const uint32_t ntiles = (NB + SCAN_TILE - 1) / SCAN_TILE;
        uint32_t* d_tiles = ws.scan_tiles.as<uint32_t>(ntiles);
        k_scan_tiles<<<ntiles, 1024, 0, st>>>(d_counts, NB, d_tiles);
        DV_LAUNCH();
        k_scan_top<<<1, 1024, 0, st>>>(d_tiles, ntiles, d_offsets + NB);
        DV_LAUNCH();
        k_scan_apply<<<ntiles, 1024, 0, st>>>(d_counts, NB, d_tiles, d_offsets, d_cursor);
        DV_LAUNCH();
    }
    mark(2);
    if (pre) k_scatter<true><<<digit_grid, 256, 0, st>>>(d_scalars, n, map, c, W, d_cursor, d_sorted);
    else k_scatter<false><<<digit_grid, 256, 0, st>>>(d_scalars, n, map, c, W, d_cursor, d_sorted);
    DV_LAUNCH();
    mark(3);

    const int seg_log = plan.seg_force > 0 ? std::min(plan.seg_force, c - 1)
                                           : msm_seg_log((uint64_t)NW * B, B, c, sizeof(F) == sizeof(Fq));
    const uint32_t S = B >> seg_log;
    XYZZ<F>* d_seg_u = ws.segs.as<XYZZ<F>>(4ull * NW * S);
    XYZZ<F>* d_seg_r = d_seg_u + (size_t)NW * S;
    XYZZ<F>* d_lvl_u = d_seg_r + (size_t)NW * S;  // ping-pong buffers of the upper levels
    XYZZ<F>* d_lvl_r = d_lvl_u + (size_t)NW * S;
    XYZZ<F>* d_win = host ? host->windows : ws.windows.as<XYZZ<F>>(NW);

    if (tl.enabled) DV_CUDA(cudaEventRecord(tl.acc_ev[0], st));
    accumulate<F>(ws, pre ? pre->table : d_points, d_sorted, d_offsets, NB, (uint64_t)n * W, d_buckets, st);
    mark(4);
    k_segments<F><<<blocks_for((uint64_t)NW * S, 128), 128, 0, st>>>(d_buckets, d_offsets, B, NW, seg_log, d_seg_u,
                                                                     d_seg_r);
    DV_LAUNCH();
    // upper levels: (U, V) pairs
    XYZZ<F>* u = d_seg_u;
    XYZZ<F>* r = d_seg_r;
    XYZZ<F>* u2 = d_lvl_u;
    XYZZ<F>* r2 = d_lvl_r;
    uint32_t len = S;
    for (;;) {
        const uint32_t nblk = len > (uint32_t)WTREE ? len / WTREE : 1u;
        XYZZ<F>* u_dst = nblk == 1 ? d_win : u2;
        k_wtree<F><<<NW * nblk, 256, 0, st>>>(u, r, len, u_dst, r2, d_err, host ? host->d_points_bad : nullptr,
                                              host && nblk == 1 ? host->bad : nullptr);
        DV_LAUNCH();
        if (nblk == 1) break;
        len = nblk;
        std::swap(u, u2);
        std::swap(r, r2);
    }
    mark(5);
}

template <class F>
void msm_run(MsmWorkspace& ws, const Affine<F>* d_points, const uint32_t* d_scalars, const uint32_t* set_offsets,
             uint32_t count, int force_c, cudaStream_t st, uint8_t* host_out, MsmStats* stats,
             const MsmPrecomp<F>* pre, const uint32_t* d_points_bad, uint32_t* points_bad) {
    typedef typename HostOf<F>::T HF;
    const size_t out_bytes = 2 * sizeof(F);
    const uint32_t n = set_offsets[count];
    uint32_t max_set = 0;
    for (uint32_t k = 0; k < count; ++k) max_set = std::max(max_set, set_offsets[k + 1] - set_offsets[k]);
    if (n == 0 || count == 0) {
        memset(host_out, 0, (size_t)count * out_bytes);
        return;
    }
    const MsmPlan plan = msm_plan_batch<F>(count, max_set, n, force_c, pre);
    const int c = plan.c, W = plan.windows;
    const uint32_t Wr = pre ? 1u : (uint32_t)W;
    const uint32_t NW = count * Wr;

    uint32_t* d_set = ws.set_off.as<uint32_t>(count + 1);
    uint32_t* d_err = ws.err.as<uint32_t>(1);
    uint32_t* h_err = ws.host_err.as<uint32_t>(2);
    DV_CUDA(cudaMemcpyAsync(d_set, set_offsets, (count + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    DV_CUDA(cudaMemsetAsync(d_err, 0xff, sizeof(uint32_t), st));
    XYZZ<F>* h_win = ws.host_windows.as<XYZZ<F>>(NW);
    const MsmHost<F> host{h_win, d_points_bad, h_err};
    msm_enqueue<F>(ws, d_points, d_scalars, SetMap{d_set, nullptr, count, 0}, n, plan, pre, d_err, st, &host);
    DV_CUDA(cudaStreamSynchronize(st));
    if (*h_err != NO_INDEX)
        throw InvalidArgument("non-canonical scalar at index " + std::to_string(*h_err));
    if (points_bad) *points_bad = h_err[1];
    static_assert(sizeof(XYZZ<F>) == sizeof(dvh::XYZZ<HF>), "host/device XYZZ layout");
    const auto* hw = reinterpret_cast<const dvh::XYZZ<HF>*>(h_win);
    for (uint32_t k = 0; k < count; ++k) horner(hw + (size_t)k * Wr, (int)Wr, c, host_out + (size_t)k * out_bytes);
    MsmTimeline& tl = ws.timeline;
    if (tl.enabled) {
        DV_CUDA(cudaEventRecord(tl.ev[6], st));
        DV_CUDA(cudaEventSynchronize(tl.ev[6]));
        auto span = [&](cudaEvent_t a, cudaEvent_t b) {
            float ms = 0;
            DV_CUDA(cudaEventElapsedTime(&ms, a, b));
            return (double)ms;
        };
        const double acc = span(tl.acc_ev[0], tl.acc_ev[1]);
        tl.ms[0] += span(tl.ev[0], tl.ev[1]);        // digit histogram
        tl.ms[1] += span(tl.ev[1], tl.ev[2]);        // offsets scan
        tl.ms[2] += span(tl.ev[2], tl.ev[3]);        // scatter
        tl.ms[3] += acc;                             // bucket accumulation
        tl.ms[4] += span(tl.ev[3], tl.ev[4]) - acc;  // split-bucket merges
        tl.ms[5] += span(tl.ev[4], tl.ev[5]);        // bucket reduction
        tl.ms[7] += span(tl.ev[5], tl.ev[6]);        // window D2H + host Horner
        tl.calls++;
        tl.accum_mixed_adds += (uint64_t)n * W;
    }
    if (stats) {
        stats->calls++;
        stats->sets += count;
        stats->points += n;
        stats->last_c = (uint64_t)c;
    }
}

// ---------------------------------------------------------------- direct small sparse MSMs
constexpr int SD_THREADS = 256, SD_TERMS = SD_THREADS / 4;
struct SdJob {
    uint32_t request, first, items, pad;  // terms first .. first + items - 1 (term = entry W + window)
};

// Coordinate read past L1: written by another block of this launch (made
// visible by its __threadfence before the counter increment below).
DV_INL Fq load_cg(const Fq* p) {
    Fq r;
    const uint4* src = reinterpret_cast<const uint4*>(p);
    uint4* dst = reinterpret_cast<uint4*>(&r);
    for (int i = 0; i < (int)(sizeof(Fq) / 16); ++i) dst[i] = __ldcg(src + i);
    return r;
}

// Sum over the block's quads; the first quad ends with it.
DV_INL Fq quads_sum_block(Fq acc, Fq (*sh)[4]) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = threadIdx.x & 3;
    acc = quads_sum_warp<Fq>(acc);
    if (lane < 4) sh[warp][r] = acc;
    __syncthreads();
    if (warp == 0) acc = quads_sum_warp<Fq>(sh[lane >> 2][r]);
    __syncthreads();
    return acc;
}

// Tree sum of sm[0 .. live) into sm[0] (entries up to the next power of two
// hold infinity): only the levels the live entries need.
DV_INL void block_sum(XYZZ<Fq>* sm, uint32_t live) {
    uint32_t span = 1;
    while (span < live) span <<= 1;
    for (uint32_t stride = span >> 1; stride > 0; stride >>= 1) {
        if (threadIdx.x < stride) sm[threadIdx.x] = XYZZ<Fq>::add_paired(sm[threadIdx.x], sm[threadIdx.x + stride]);
        __syncthreads();
    }
}

// Term `term` of a sparse MSM: its table entry with the digit's sign in
// `point`; returns the digit's magnitude, 0 where nothing is to be added (a
// non-canonical scalar and an index out of range are noted in err).
DV_INL uint32_t sparse_term(const G1A* __restrict__ table, uint64_t nbases, int c, int W,
                            const uint64_t* __restrict__ idx, const uint32_t* __restrict__ vals, uint32_t term,
                            uint32_t* __restrict__ err, G1A& point) {
    const uint32_t e = term / (uint32_t)W, w = term % (uint32_t)W;
    uint32_t s[8];
    load_scalar(vals, e, s);
    const uint64_t ix = idx[e];
    if (!Fr::is_canonical(s)) {
        if (w == 0) atomicMin(err, e);
        return 0;
    }
    if (ix >= nbases) {
        if (w == 0) atomicMin(err + 1, e);
        return 0;
    }
    // signed digit of window w (the recoding of k_hist)
    const uint32_t B = 1u << (c - 1), full = 1u << c;
    const uint32_t* words = vals + 8ull * e;
    const uint32_t d = window_raw(words, (int)w * c, c) + carry_into(words, (int)w, c);
    const bool neg = d > B;
    point = table[ix * (uint64_t)W + w];
    if (neg) point.y = Fq::neg(point.y);
    return point.is_inf() ? 0u : neg ? full - d : d;
}

// Sparse MSMs over a window table in one launch.  Each block takes up to
// SD_TERMS (entry, window) terms of one request: a lane quad forms d T (the
// signed c-bit digit d of the entry's window, T the table's multiple
// 2^(c w) P) by double-and-add, the block sums its quads.  The last block
// of a request to finish (a per-request counter) sums the request's block partials and writes the XYZZ sum
// and the error words to pinned memory.
// The launch is one chain: up to c doublings and c / 2 additions, a tree of
// six additions, the same over the partials, each three or four dependent
// products in a quad.  256 entries of 32 windows, a whole call from host
// memory: 210 us with a thread a term and one bit a step, 137 us so, 125
// without fills and copies beside the kernel.
// The host normalises all requests with one batch inversion, as the
// reference does (icicle_msm.cu:417-421): one thread's inversion on the
// device takes longer than that copy and a host batch inversion.
__global__ void __launch_bounds__(SD_THREADS) k_sparse_quads(const G1A* __restrict__ table, uint64_t nbases, int c,
                                                             int W, const uint64_t* __restrict__ idx,
                                                             const uint32_t* __restrict__ vals,
                                                             const SdJob* __restrict__ jobs,
                                                             const uint32_t* __restrict__ req_blocks,
                                                             XYZZ<Fq>* __restrict__ partial, uint32_t* __restrict__ done,
                                                             XYZZ<Fq>* __restrict__ out, uint32_t* __restrict__ err,
                                                             uint32_t* __restrict__ host_err) {
    __shared__ Fq sh[SD_THREADS / 32][4];
    __shared__ bool last;
    const SdJob job = jobs[blockIdx.x];
    const uint32_t quad = threadIdx.x >> 2, r = threadIdx.x & 3;
    uint32_t mag = 0;
    Fq t = Quad<Fq>::inf();
    if (quad < job.items) {
        G1A a;
        mag = sparse_term(table, nbases, c, W, idx, vals, job.first + quad, err, a);
        if (mag) t = r == 0 ? a.x : r == 1 ? a.y : Fq::one();
    }
    // d T by two bits a step over T, 2 T, 3 T, from each quad's top pair of
    // bits on, the warp in step with its longest digit
    const Fq t2 = Quad<Fq>::dbl(t), t3 = Quad<Fq>::add(t2, t);
    const auto multiple = [&](uint32_t m) { return m == 1 ? t : m == 2 ? t2 : t3; };
    const int top = mag ? (31 - __clz(mag)) >> 1 : -1;
    Fq p = mag ? multiple(mag >> (2 * top)) : Quad<Fq>::inf();
    for (int b = __reduce_max_sync(0xffffffffu, top) - 1; b >= 0; --b) {
        const Fq four = Quad<Fq>::dbl(Quad<Fq>::dbl(p));
        if (b < top) p = four;
        const uint32_t m = b < top ? (mag >> (2 * b)) & 3u : 0u;
        const Fq sum = Quad<Fq>::add(p, multiple(m));
        if (m) p = sum;
    }
    p = quads_sum_block(p, sh);
    const uint32_t req = job.request, b0 = req_blocks[req], b1 = req_blocks[req + 1];
    if (threadIdx.x < 4) {
        reinterpret_cast<Fq*>(partial + blockIdx.x)[r] = p;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();  // the block's error words
        last = atomicAdd(done + req, 1u) == b1 - b0 - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    p = Quad<Fq>::inf();
    for (uint32_t b = b0 + quad; __any_sync(0xffffffffu, b < b1); b += SD_TERMS)
        p = Quad<Fq>::add(p, b < b1 ? load_cg(reinterpret_cast<const Fq*>(partial + b) + r) : Quad<Fq>::inf());
    p = quads_sum_block(p, sh);
    if (threadIdx.x < 4) reinterpret_cast<Fq*>(out + req)[r] = p;
    // at least the errors of this request; the host takes the least of all
    if (threadIdx.x < 2) host_err[2 * req + threadIdx.x] = static_cast<volatile const uint32_t*>(err)[threadIdx.x];
}

// The same with a thread per term and blocks of four times the terms, for
// calls of many requests whose quads would take several waves: a quad is the
// shorter chain, but a quarter more multiply-adds.
__global__ void __launch_bounds__(SD_THREADS) k_sparse_threads(const G1A* __restrict__ table, uint64_t nbases, int c,
                                                               int W, const uint64_t* __restrict__ idx,
                                                               const uint32_t* __restrict__ vals,
                                                               const SdJob* __restrict__ jobs,
                                                               const uint32_t* __restrict__ req_blocks,
                                                               XYZZ<Fq>* __restrict__ partial,
                                                               uint32_t* __restrict__ done, XYZZ<Fq>* __restrict__ out,
                                                               uint32_t* __restrict__ err,
                                                               uint32_t* __restrict__ host_err) {
    __shared__ XYZZ<Fq> sm[SD_THREADS];
    __shared__ bool last;
    const SdJob job = jobs[blockIdx.x];
    const uint32_t t = threadIdx.x;
    XYZZ<Fq> p = XYZZ<Fq>::inf();
    if (t < job.items) {
        G1A a;
        const uint32_t mag = sparse_term(table, nbases, c, W, idx, vals, job.first + t, err, a);
        if (mag) {
            p = XYZZ<Fq>::from_affine(a);
            for (int b = 30 - __clz(mag); b >= 0; --b) {
                p = XYZZ<Fq>::dbl_paired(p);
                if ((mag >> b) & 1) p = XYZZ<Fq>::add_affine(p, a);
            }
        }
    }
    sm[t] = p;
    __syncthreads();
    block_sum(sm, job.items);
    const uint32_t req = job.request, b0 = req_blocks[req], b1 = req_blocks[req + 1];
    if (t == 0) {
        partial[blockIdx.x] = sm[0];
        __threadfence();  // and the block's error words
        last = atomicAdd(done + req, 1u) == b1 - b0 - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    p = XYZZ<Fq>::inf();
    for (uint32_t b = b0 + t; b < b1; b += SD_THREADS) {
        const Fq* q = reinterpret_cast<const Fq*>(partial + b);
        p = XYZZ<Fq>::add_paired(p, {load_cg(q), load_cg(q + 1), load_cg(q + 2), load_cg(q + 3)});
    }
    sm[t] = p;
    __syncthreads();
    block_sum(sm, min(b1 - b0, (uint32_t)SD_THREADS));
    if (t == 0) out[req] = sm[0];
    if (t < 2) host_err[2 * req + t] = static_cast<volatile const uint32_t*>(err)[t];
}

void msm_sparse_direct(MsmWorkspace& ws, const MsmPrecomp<Fq>& pre, uint64_t nbases, const uint64_t* d_idx,
                       const uint32_t* d_vals, const uint32_t* offs, uint32_t count, uint8_t* host_out,
                       cudaStream_t st) {
    const uint32_t W = (uint32_t)pre.windows;
    // Quads while they are one wave of blocks, or where requests are so short
    // that threads would leave blocks mostly empty (32768 terms over a c = 8
    // table: one request 327 us by quads and 227 by threads, 256 requests 383 and
    // 348, 1024 requests 726 and 1027).
    uint64_t quad_blocks = 0, thread_blocks = 0;
    for (uint32_t r = 0; r < count; ++r) {
        const uint64_t terms = (uint64_t)(offs[r + 1] - offs[r]) * W;
        quad_blocks += (terms + SD_TERMS - 1) / SD_TERMS;
        thread_blocks += (terms + SD_THREADS - 1) / SD_THREADS;
    }
    const bool quads = quad_blocks <= 2 * (uint64_t)sm_count() || quad_blocks < 2 * thread_blocks;
    const uint32_t block_terms = quads ? SD_TERMS : SD_THREADS;
    std::vector<SdJob> jobs;
    std::vector<uint32_t> req_blocks(count + 1, 0);
    bool empty = false;
    for (uint32_t r = 0; r < count; ++r) {
        const uint32_t first = offs[r] * W, terms = (offs[r + 1] - offs[r]) * W;
        for (uint32_t t = 0; t < terms; t += block_terms)
            jobs.push_back(SdJob{r, first + t, std::min<uint32_t>(block_terms, terms - t), 0});
        req_blocks[r + 1] = (uint32_t)jobs.size();
        empty |= terms == 0;
    }
    if (jobs.empty()) {
        memset(host_out, 0, (size_t)count * 64);
        return;
    }
    // one upload: the block list, the per-request block offsets, the
    // requests' counters and the error words; the kernel writes sums and
    // error words to pinned memory, so nothing is copied or set beside it
    // (two fills and a copy back before)
    const size_t jb = jobs.size() * sizeof(SdJob), rb = (count + 1) * sizeof(uint32_t), cb = count * sizeof(uint32_t);
    uint8_t* h_desc = ws.host_desc.as<uint8_t>(jb + rb + cb + 8);
    memcpy(h_desc, jobs.data(), jb);
    memcpy(h_desc + jb, req_blocks.data(), rb);
    memset(h_desc + jb + rb, 0, cb);
    memset(h_desc + jb + rb + cb, 0xff, 8);
    uint8_t* d_desc = ws.sd_jobs.as<uint8_t>(jb + rb + cb + 8);
    uint32_t* d_done = reinterpret_cast<uint32_t*>(d_desc + jb + rb);
    XYZZ<Fq>* d_partial = ws.sd_partial.as<XYZZ<Fq>>(jobs.size());
    constexpr size_t XB = sizeof(XYZZ<Fq>);
    uint8_t* h_out = ws.host_windows.as<uint8_t>((size_t)count * (XB + 8));
    if (empty) memset(h_out, 0, (size_t)count * XB);  // all-zero XYZZ: infinity
    uint32_t* h_words = reinterpret_cast<uint32_t*>(h_out + (size_t)count * XB);
    memset(h_words, 0xff, (size_t)count * 8);
    DV_CUDA(cudaMemcpyAsync(d_desc, h_desc, jb + rb + cb + 8, cudaMemcpyHostToDevice, st));
    (quads ? k_sparse_quads : k_sparse_threads)<<<(unsigned)jobs.size(), SD_THREADS, 0, st>>>(
        pre.table, nbases, pre.c, (int)W, d_idx, d_vals, reinterpret_cast<const SdJob*>(d_desc),
        reinterpret_cast<const uint32_t*>(d_desc + jb), d_partial, d_done, reinterpret_cast<XYZZ<Fq>*>(h_out),
        d_done + count, h_words);
    DV_LAUNCH();
    DV_CUDA(cudaStreamSynchronize(st));
    uint32_t h_err[2] = {NO_INDEX, NO_INDEX};
    for (uint32_t k = 0; k < 2 * count; ++k) h_err[k & 1] = std::min(h_err[k & 1], h_words[k]);
    if (h_err[0] != NO_INDEX) throw InvalidArgument("non-canonical scalar at index " + std::to_string(h_err[0]));
    if (h_err[1] != NO_INDEX) throw InvalidArgument("sparse MSM index out of range");
    static_assert(sizeof(XYZZ<Fq>) == sizeof(dvh::XYZZ<dvh::Fq>), "host/device XYZZ layout");
    dvh::xyzz_batch_to_affine_bytes(reinterpret_cast<const dvh::XYZZ<dvh::Fq>*>(h_out), count, host_out);
}

template void msm_run<Fq>(MsmWorkspace&, const Affine<Fq>*, const uint32_t*, const uint32_t*, uint32_t, int,
                          cudaStream_t, uint8_t*, MsmStats*, const MsmPrecomp<Fq>*, const uint32_t*, uint32_t*);
template void msm_run<Fq2>(MsmWorkspace&, const Affine<Fq2>*, const uint32_t*, const uint32_t*, uint32_t, int,
                           cudaStream_t, uint8_t*, MsmStats*, const MsmPrecomp<Fq2>*, const uint32_t*, uint32_t*);
template MsmPlan msm_plan_batch<Fq>(uint32_t, uint32_t, uint64_t, int, const MsmPrecomp<Fq>*);
template MsmPlan msm_plan_batch<Fq2>(uint32_t, uint32_t, uint64_t, int, const MsmPrecomp<Fq2>*);
template void msm_enqueue<Fq>(MsmWorkspace&, const Affine<Fq>*, const uint32_t*, const SetMap&, uint32_t,
                              const MsmPlan&, const MsmPrecomp<Fq>*, uint32_t*, cudaStream_t, const MsmHost<Fq>*);
template void msm_enqueue<Fq2>(MsmWorkspace&, const Affine<Fq2>*, const uint32_t*, const SetMap&, uint32_t,
                               const MsmPlan&, const MsmPrecomp<Fq2>*, uint32_t*, cudaStream_t, const MsmHost<Fq2>*);

template <class F>
void msm_finish_device(const XYZZ<F>* d_windows, uint32_t count, int windows_per_set, int c, const uint32_t* d_out_idx,
                       uint8_t* d_out, cudaStream_t st) {
    if (!count) return;
    k_msm_finish<F><<<blocks_for(count, 64), 64, 0, st>>>(d_windows, count, windows_per_set, c, d_out_idx, d_out);
    DV_LAUNCH();
}
template void msm_finish_device<Fq>(const XYZZ<Fq>*, uint32_t, int, int, const uint32_t*, uint8_t*, cudaStream_t);
template void msm_finish_device<Fq2>(const XYZZ<Fq2>*, uint32_t, int, int, const uint32_t*, uint8_t*, cudaStream_t);

template <class F>
void msm_precompute(const Affine<F>* d_bases, uint64_t n, int c, int windows, Affine<F>* d_table, cudaStream_t st) {
    if (!n) return;
    k_precompute<F><<<blocks_for(n, 128), 128, 0, st>>>(d_bases, n, windows, c, d_table);
    DV_LAUNCH();
}
template void msm_precompute<Fq>(const Affine<Fq>*, uint64_t, int, int, Affine<Fq>*, cudaStream_t);
template void msm_precompute<Fq2>(const Affine<Fq2>*, uint64_t, int, int, Affine<Fq2>*, cudaStream_t);

MsmPlan msm_plan_precomputed(uint64_t n) {
    // one shared bucket set: windows * 10 n additions + 28 * 2^(c-1) for the reduction
    MsmPlan p{};
    double best = 1e300;
    for (int c = 8; c <= 22; ++c) {
        const double W = (255 + c - 1) / c;
        const double cost = W * 10.0 * (double)n + 28.0 * (double)(1u << (c - 1));
        if (cost < best) { best = cost; p.c = c; }
    }
    p.windows = (255 + p.c - 1) / p.c;
    p.buckets = 1u << (p.c - 1);
    p.seg_log = std::min(DV_SEG_LOG, p.c - 1);
    return p;
}
template void convert_points<Fq>(const uint8_t*, Affine<Fq>*, uint64_t, uint32_t*, cudaStream_t);
template void convert_points<Fq2>(const uint8_t*, Affine<Fq2>*, uint64_t, uint32_t*, cudaStream_t);
template void gather_points<Fq>(const Affine<Fq>*, uint64_t, const uint64_t*, uint64_t, Affine<Fq>*, uint32_t*,
                                cudaStream_t);
template void gather_points<Fq2>(const Affine<Fq2>*, uint64_t, const uint64_t*, uint64_t, Affine<Fq2>*, uint32_t*,
                                 cudaStream_t);

}  // namespace dv
