// ssort_kernels.cu -- sm_100a kernels of the MSD radix string sort.
//
// One refinement round works on the live segments at one depth (a multiple of
// 16 bytes).  For every live string it gathers the 16 bytes at arena[off+depth]
// as a big-endian key with every byte after the first NUL zeroed (the
// multi-byte form of the reference's get_char, src/util/get_char.h:42-89, built
// with unsigned shifts; the reference's int-promoted 64-bit form sign-extends
// bytes >= 0x80, :82, and is not reproduced).  Each segment is then sorted by
// (key, index): segments of <= 32 strings by one warp in registers (four
// segments of <= 8 per warp), those of up to SMALL_CAP (in large sorts LEAF_CAP)
// by a group of 32 to 512 threads of a CTA (by size), larger ones are first split
// by sample partitioning into range buckets and equality buckets with a stable
// scatter.  Equal runs whose key holds no NUL (the reference's is_end test,
// src/util/get_char.h:162-175, and its bucket-skip rule, src/msd_ce.cpp:402)
// become the next round's segments at depth+16; every other adjacent pair gets
// its LCP here.
#include <algorithm>
#include <atomic>

#include "ssort_internal.cuh"

namespace ssort {

namespace {

constexpr uint64_t W_MAX = ~0ull;
constexpr uint32_t IDX_MAX = ~0u;

// ---- kernels launched before their predecessor has ended -----------------------
// The kernels of a round follow each other on one stream, each needing all of
// what the last one wrote, and in small sorts most of them are short.  They are
// launched with programmatic stream serialization and wait here, before their
// first access to what a sort writes, until the predecessor has ended.  No kernel
// signals early, so a successor's CTAs start once every CTA of the predecessor
// has exited; what overlaps their start is the predecessor's final flush and
// the stream's hand-over: 1 M uniform strings 267 -> 254 us, 20 k URLs 277 ->
// 259 us, 3 M URLs 920 -> 885 us.
// Such a kernel's lifetime begins before its inputs are complete.  Everything
// that a sort writes is therefore read by ordinary loads: no __ldg and no
// const __restrict__ pointer, whose read-only loads the compiler may also move
// above the wait.  The arena and the offsets are inputs and may use them.
__device__ __forceinline__ void after_predecessor() { cudaGridDependencySynchronize(); }

// ---- 16-byte keys -----------------------------------------------------------
struct Key {
    uint64_t hi, lo;
};

__device__ __forceinline__ Key key_max() { return Key{W_MAX, W_MAX}; }
__device__ __forceinline__ Key to_key(ulonglong2 v) { return Key{v.x, v.y}; }
__device__ __forceinline__ ulonglong2 from_key(Key k) { return make_ulonglong2(k.hi, k.lo); }
__device__ __forceinline__ bool key_lt(const Key &a, const Key &b) {
    return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo);
}
__device__ __forceinline__ bool key_eq(const Key &a, const Key &b) {
    return a.hi == b.hi && a.lo == b.lo;
}
__device__ __forceinline__ bool pair_lt(const Key &a, uint32_t ia, const Key &b, uint32_t ib) {
    return a.hi < b.hi || (a.hi == b.hi && (a.lo < b.lo || (a.lo == b.lo && ia < ib)));
}

__device__ __forceinline__ uint64_t bswap64(uint64_t x) {
    const uint32_t lo = (uint32_t)x, hi = (uint32_t)(x >> 32);
    return ((uint64_t)__byte_perm(lo, 0, 0x0123) << 32) | __byte_perm(hi, 0, 0x0123);
}

// Classic zero-byte test on a little-endian word: the lowest flagged byte is
// the first NUL (no false positives below it).  Returns the word with that
// byte and everything after it cleared, and whether a NUL was found.
__device__ __forceinline__ uint64_t cut_at_nul(uint64_t w, bool &found) {
    const uint64_t z = (w - 0x0101010101010101ull) & ~w & 0x8080808080808080ull;
    found = z != 0;
    if (!found) return w;
    const uint32_t jb = (uint32_t)(__ffsll((long long)z) - 1) >> 3;
    return jb ? (w & ((1ull << (8 * jb)) - 1)) : 0ull;
}

// The key whose 16 bytes start at byte `off` of the two adjacent words v0, v1
// (v1 is not looked at when off is 0).
__device__ __forceinline__ Key key_of_words(const ulonglong2 &v0, const ulonglong2 &v1,
                                            uint32_t off) {
    const uint64_t q0 = off < 8 ? v0.x : v0.y, q1 = off < 8 ? v0.y : v1.x,
                   q2 = off < 8 ? v1.x : v1.y;
    const uint32_t sh = (off & 7) * 8;
    // little-endian: byte 0 of w0 is the string's first (two shifts, as a
    // shift by 64 is undefined)
    uint64_t w0 = (q0 >> sh) | (q1 << 1 << (63 - sh));
    uint64_t w1 = (q1 >> sh) | (q2 << 1 << (63 - sh));
    bool nul;
    w0 = cut_at_nul(w0, nul);
    if (nul)
        w1 = 0;
    else
        w1 = cut_at_nul(w1, nul);
    return Key{bswap64(w0), bswap64(w1)};
}

// Whether the two 16-byte words at `a` (16-byte aligned) lie inside the arena
// (no a + 32 here: an offset near 2^64 must not wrap into the fast path).
__device__ __forceinline__ bool key_words_inside(uint64_t arena_bytes, uint64_t a) {
    return arena_bytes >= 32 && a <= arena_bytes - 32;
}

// Byte-wise form for the last bytes of the arena and for offsets past it.
__device__ __noinline__ Key load_key_tail(const uint8_t *__restrict__ arena,
                                          uint64_t arena_bytes, uint64_t pos) {
    uint64_t hi = 0, lo = 0;
    for (int i = 0; i < 16; ++i) {
        const uint64_t q = pos + i;
        const uint64_t c = q >= pos && q < arena_bytes ? arena[q] : 0;
        if (!c) break;
        if (i < 8)
            hi |= c << (56 - 8 * i);
        else
            lo |= c << (120 - 8 * i);
    }
    return Key{hi, lo};
}

// The 16 bytes of the string at arena[pos..], big-endian, zero after the
// first NUL.  The arena base is 16-byte aligned; bytes at or beyond
// arena_bytes read as NUL.
__device__ __forceinline__ Key load_key(const uint8_t *__restrict__ arena, uint64_t arena_bytes,
                                        uint64_t pos) {
    const uint64_t a = pos & ~15ull;
    if (!key_words_inside(arena_bytes, a)) return load_key_tail(arena, arena_bytes, pos);
    const ulonglong2 *w = reinterpret_cast<const ulonglong2 *>(arena + a);
    const ulonglong2 v0 = __ldg(w);
    return key_of_words(v0, pos & 15 ? __ldg(w + 1) : v0, (uint32_t)pos & 15u);
}

// The key holds the end of its string (last byte NUL).
__device__ __forceinline__ bool key_is_end(const Key &k) { return (k.lo & 0xFF) == 0; }

__device__ __forceinline__ uint32_t len8(uint64_t w) {
    return w ? 8u - ((uint32_t)(__ffsll((long long)w) - 1) >> 3) : 0u;
}

// Number of string bytes in a key that contains the NUL.
__device__ __forceinline__ uint32_t key_len(const Key &k) {
    return (k.hi & 0xFF) ? 8u + len8(k.lo) : len8(k.hi);
}

// LCP contribution of two keys at the same depth (reference lcp(),
// src/mergesort_lcp.cpp:88-100: stop at the first difference or the NUL).
__device__ __forceinline__ uint32_t key_lcp(const Key &a, const Key &b) {
    if (a.hi != b.hi) return (uint32_t)__clzll((long long)(a.hi ^ b.hi)) >> 3;
    if ((a.hi & 0xFF) == 0) return len8(a.hi);
    if (a.lo != b.lo) return 8u + ((uint32_t)__clzll((long long)(a.lo ^ b.lo)) >> 3);
    return 8u + len8(a.lo);
}

__device__ __forceinline__ uint64_t string_offset(const void *offs, int off_width, uint32_t i) {
    return off_width == 8 ? __ldg(reinterpret_cast<const unsigned long long *>(offs) + i)
                          : (uint64_t)__ldg(reinterpret_cast<const uint32_t *>(offs) + i);
}

__device__ __forceinline__ uint32_t lanemask_lt() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ uint32_t next_pow2(uint32_t x) {
    return x <= 1 ? 1u : 1u << (32 - __clz(x - 1));
}

// Largest i in [0, n) with base[i] <= t (base ascending, base[0] = 0), found by
// a whole warp together: 32 probes a step, so two dependent reads for up to
// 1024 segments where a binary search takes ten.
__device__ __forceinline__ uint32_t find_seg(const uint32_t *base, uint32_t n, uint32_t t) {
    uint32_t lo = 0;
    while (n > 1) {
        const uint32_t step = (n + 31) / 32, i = (threadIdx.x & 31) * step;
        const uint32_t below =
            __ballot_sync(0xffffffffu, i < n && base[lo + i] <= t);  // a prefix, lane 0 set
        const uint32_t at = (31 - __clz(below)) * step;
        lo += at;
        n = min(step, n - at);
    }
    return lo;
}

// Warp-aggregated append to a list counter: all 32 lanes call it together;
// each lane with `want` gets its own slot, at the cost of one atomic per warp
// (appends from millions of small segments would otherwise serialise on one
// address).
// In two steps: warp_reserve issues the warp's atomic without waiting for
// it, so that the reservations a kernel makes on several counters overlap
// their round trips; warp_slot then hands each wanting lane its slot.
struct WarpRes {
    uint32_t mask, base;
};
__device__ __forceinline__ WarpRes warp_reserve(uint32_t *ctr, bool want) {
    const uint32_t mask = __ballot_sync(0xffffffffu, want);
    uint32_t base = 0;
    if (mask && (threadIdx.x & 31) == (uint32_t)(__ffs(mask) - 1))
        base = atomicAdd(ctr, (uint32_t)__popc(mask));
    return WarpRes{mask, base};
}
__device__ __forceinline__ uint32_t warp_slot(const WarpRes &r) {
    if (!r.mask) return 0;  // warp-uniform
    return __shfl_sync(0xffffffffu, r.base, __ffs(r.mask) - 1) + __popc(r.mask & lanemask_lt());
}
__device__ __forceinline__ uint32_t warp_append(uint32_t *ctr, bool want) {
    return warp_slot(warp_reserve(ctr, want));
}

// Append a next-round segment; warp-collective like warp_append.
__device__ __forceinline__ void emit_next_warp(Seg *N, Counters *c, bool want, uint32_t start,
                                               uint32_t len, uint32_t depth) {
    const uint32_t slot = warp_append(&c->n_next, want);
    if (want) N[slot] = Seg{start, len, depth, 0u};
}

// Single-thread append (rare paths only).
__device__ __forceinline__ void emit_next(Seg *N, Counters *c, uint32_t start, uint32_t len,
                                          uint32_t depth) {
    const uint32_t slot = atomicAdd(&c->n_next, 1u);
    N[slot] = Seg{start, len, depth, 0u};
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

__device__ __forceinline__ uint64_t window64(const Key &k, uint32_t f);

__device__ __forceinline__ uint32_t window_bits(const Key &k, uint32_t f) {
    return (uint32_t)(window64(k, f) >> (64 - TBL_BITS));
}

// Asks the memory system to stream the bytes of [p, p + bytes) into L2 (a
// TMA bulk prefetch: no registers, nothing to wait for).  The start is
// rounded up and the end down to 16-byte boundaries, so nothing outside the
// range is touched; ranges are issued in pieces of at most 1 MB.  Called by
// the CTA's first warp; its first thread asks.
__device__ __forceinline__ void prefetch_l2(const void *p, uint64_t bytes) {
    if (threadIdx.x != 0) return;
    uint64_t a = ((uint64_t)(uintptr_t)p + 15) & ~15ull;
    const uint64_t e = ((uint64_t)(uintptr_t)p + bytes) & ~15ull;
    while (a < e) {
        const uint32_t sz = (uint32_t)min(e - a, (uint64_t)(1u << 20));
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"(sz) : "memory");
        a += sz;
    }
}

// ---- packed 64-bit sort keys -------------------------------------------------
// In a segment of at most 32 strings every key shares its first f bits (f =
// leading zeros of the OR of key ^ key0).  The 53 bits after them, with the
// string's lane in the low bits, form a unique 64-bit sort key whose order
// agrees with (key, index) order except between keys whose windows are equal;
// those are checked afterwards and, on any disagreement, the segment is
// re-sorted with the full comparator.
constexpr uint32_t POS_BITS = 11;
constexpr uint64_t POS_MASK = (1ull << POS_BITS) - 1;

__device__ __forceinline__ uint32_t clz128(uint64_t hi, uint64_t lo) {
    return hi ? (uint32_t)__clzll((long long)hi)
              : 64u + (lo ? (uint32_t)__clzll((long long)lo) : 64u);
}

// Top 64 bits of the 128-bit key shifted left by f (0 <= f < 128).
__device__ __forceinline__ uint64_t window64(const Key &k, uint32_t f) {
    if (f == 0) return k.hi;
    if (f < 64) return (k.hi << f) | (k.lo >> (64 - f));
    return k.lo << (f - 64);
}

__device__ __forceinline__ uint64_t sort_key(const Key &k, uint32_t f, uint32_t pos) {
    return (window64(k, f) & ~POS_MASK) | pos;
}

// ---------------------------------------------------------------------------
__global__ void k_iota(uint32_t *idx, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        idx[i] = i;
}

// Appends segment o (when v) to the list its length selects: one-warp sorts
// of <= 32 or <= warp8_cap strings, the CTA sorts' four size classes (up to
// cap strings), or the large list L (counter nl).  Warp-collective; the
// reservations are all issued before any is waited for.
__device__ __forceinline__ void append_by_length(const Seg &o, bool v, uint32_t warp8_cap,
                                                 uint32_t cap, Seg *W1, Seg *W8,
                                                 const SmallLists &S, Seg *L, uint32_t *nl,
                                                 Counters *c) {
    const bool w1 = v && o.len <= (uint32_t)WARP1_CAP;
    const bool w8 = v && !w1 && o.len <= warp8_cap;
    const bool sm = v && !w1 && !w8 && o.len <= cap;
    const bool c0 = sm && o.len <= (uint32_t)BLOCK_CAP1;
    const bool c1 = sm && !c0 && o.len <= (uint32_t)BLOCK_CAP2;
    const bool c2 = sm && !c0 && !c1 && o.len <= (uint32_t)SMALL_CAP;
    const bool c3 = sm && !c0 && !c1 && !c2;
    const bool lg = v && !w1 && !w8 && !sm;
    const WarpRes r1 = warp_reserve(&c->n_w1, w1), r8 = warp_reserve(&c->n_w8, w8),
                  rs0 = warp_reserve(&c->n_small, c0), rs1 = warp_reserve(&c->n_small2, c1),
                  rs2 = warp_reserve(&c->n_small3, c2), rs3 = warp_reserve(&c->n_small4, c3),
                  rl = warp_reserve(nl, lg);
    const uint32_t t1 = warp_slot(r1), t8 = warp_slot(r8), ts0 = warp_slot(rs0),
                   ts1 = warp_slot(rs1), ts2 = warp_slot(rs2), ts3 = warp_slot(rs3), tl = warp_slot(rl);
    if (w1) W1[t1] = o;
    if (w8) W8[t8] = o;
    if (c0) S.s[0][ts0] = o;
    if (c1) S.s[1][ts1] = o;
    if (c2) S.s[2][ts2] = o;
    if (c3) S.s[3][ts3] = o;
    if (lg) L[tl] = o;
}

__device__ __forceinline__ void classify_list(const Seg *R, uint32_t nR,
                                              uint32_t warp8_cap, Seg *W1, Seg *W8,
                                              const SmallLists &S, Seg *L, Counters *c) {
    // Block-uniform trip count: every warp reaches the collective appends.
    for (uint32_t b0 = blockIdx.x * blockDim.x; b0 < nR; b0 += gridDim.x * blockDim.x) {
        const uint32_t i = b0 + threadIdx.x;
        const bool v = i < nR;
        const Seg s = v ? R[i] : Seg{0, 0, 0, 0};
        append_by_length(s, v, warp8_cap, SMALL_CAP, W1, W8, S, L, &c->n_large, c);
        const bool lg = v && s.len > (uint32_t)SMALL_CAP && s.len > warp8_cap;
        const unsigned long long live = warp_sum(v ? s.len : 0);
        const unsigned long long big = warp_sum(lg ? s.len : 0);
        if ((threadIdx.x & 31) == 0) {
            if (live) atomicAdd(&c->live_next, live);
            if (big) atomicAdd(&c->gather_elems, big);
        }
    }
}

// End of a kernel whose counts the host waits for: the last CTA to get here
// copies the counters to pinned host memory and sets the host's flag.  The
// host polls the flag, which saves the copy engine's launch and the stream
// synchronisation (a round trip of about 4 us instead of 12).  True in the
// last CTA.
__device__ __forceinline__ bool publish(const Publish &p, RoundCounters *rc) {
    if (!p.host) return false;
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&rc->ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return false;
    __threadfence();
    const uint32_t *w = reinterpret_cast<const uint32_t *>(rc);
    volatile uint32_t *h = p.host;
    constexpr uint32_t WORDS = sizeof(RoundCounters) / 4;
    for (uint32_t i = threadIdx.x; i < WORDS; i += blockDim.x) h[i] = __ldcg(w + i);
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
        rc->ticket = 0;
        h[WORDS] = p.seq;
    }
    return true;
}

__global__ void k_begin(uint32_t *idx, uint32_t n_idx, uint32_t *lcp, RoundCounters *rc,
                        Seg first, Seg *list, uint32_t *count) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_idx;
         i += gridDim.x * blockDim.x)
        idx[i] = i;
    if (blockIdx.x != 0) return;
    uint32_t *w = reinterpret_cast<uint32_t *>(rc);
    for (uint32_t i = threadIdx.x; i < sizeof(RoundCounters) / 4; i += blockDim.x) w[i] = 0;
    __syncthreads();
    if (threadIdx.x != 0) return;
    if (n_idx || first.len) lcp[0] = 0;
    if (first.len) {
        *list = first;
        *count = 1;
        rc->c[0].live_next = first.len;
        if (first.len > (uint32_t)SMALL_CAP) rc->c[0].gather_elems = first.len;
    }
}

__global__ void k_classify(const Seg *__restrict__ R, Count cnt, uint32_t warp8_cap, Seg *W1,
                           Seg *W8, SmallLists S, Seg *L, Counters *c, RoundCounters *rc,
                           Publish pub) {
    classify_list(R, count_of(cnt), warp8_cap, W1, W8, S, L, c);
    publish(pub, rc);
}

// ---- batches of independent instances ---------------------------------------
// Instance i owns positions inst_start[i] .. inst_start[i+1]-1: it enters
// round 0 as its own segment, and its first LCP entry is 0.
__global__ void k_init_batch(const uint32_t *__restrict__ inst_start, uint32_t ninst, Seg *R,
                             uint32_t *lcp, Counters *c) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool v = i < ninst;
    const uint32_t s = v ? inst_start[i] : 0, e = v ? inst_start[i + 1] : 0;
    if (v && e > s) lcp[s] = 0;
    const bool seg = v && e - s >= 2;
    const uint32_t slot = warp_append(&c->n_next, seg);
    if (seg) R[slot] = Seg{s, e - s, 0, SEG_IOTA};
}

// The three kernels below give every position the instance or request it lies
// in.  A warp takes SPAN_ITEMS * 32 consecutive positions: one search for the
// first, then every lane only passes on to a later range (a search per
// position took 0.37 ms over 69 M positions in 353 instances; reading and
// writing them takes 0.09).
constexpr uint32_t SPAN_ITEMS = 8;

// Largest j in [i, n) with first[j] <= p (first ascending, first[i] <= p): in
// doubling steps, then back in halving ones.  As many reads as one step at a
// time takes to pass a few ranges, and few where many empty ones follow each
// other, of which a batch may hold any number (100,000 in a row: one step at a
// time the batch took 5.9 ms, now 0.27, as without them).
__device__ __forceinline__ uint32_t pass_on(const uint32_t *first, uint32_t n, uint32_t i,
                                            uint32_t p) {
    uint64_t d = 1;
    while (d < n - i && first[i + d] <= p) {
        i += (uint32_t)d;
        d *= 2;
    }
    while (d /= 2)
        if (d < n - i && first[i + d] <= p) i += (uint32_t)d;
    return i;
}

// Global positions -> indices within each position's instance.
__global__ void k_localize(uint32_t *perm, uint32_t n, const uint32_t *__restrict__ inst_start,
                           uint32_t ninst) {
    const uint32_t lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint64_t p0 = (uint64_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32 * SPAN_ITEMS;
         p0 < n; p0 += (uint64_t)warps * 32 * SPAN_ITEMS) {
        // The span's indices are on their way during the search (read where
        // they are used, 69 M positions took 168 us, now 108; 5.1 TB/s).
        uint32_t v[SPAN_ITEMS];
#pragma unroll
        for (uint32_t k = 0; k < SPAN_ITEMS; ++k) {
            const uint64_t p = p0 + k * 32 + lane;
            v[k] = p < n ? perm[p] : 0;
        }
        uint32_t i = find_seg(inst_start, ninst, (uint32_t)p0);
        uint32_t end = __ldg(inst_start + i + 1), start = __ldg(inst_start + i);
#pragma unroll
        for (uint32_t k = 0; k < SPAN_ITEMS; ++k) {
            const uint64_t p = p0 + k * 32 + lane;
            if (p < n) {
                if (p >= end) {
                    i = pass_on(inst_start, ninst, i, (uint32_t)p);
                    start = __ldg(inst_start + i);
                    end = __ldg(inst_start + i + 1);
                }
                perm[p] = v[k] - start;
            }
        }
    }
}

// ---- request server: joining and retiring requests between rounds ----------
// The requests of one step are described by ReqJob records; a flat index q
// over all their positions (jobs[j].first = positions of the jobs before j)
// finds its job by binary search.
__device__ __forceinline__ uint32_t find_job(const ReqJob *__restrict__ jobs, uint32_t njobs,
                                             uint32_t q) {
    uint32_t lo = 0, hi = njobs;  // largest j with jobs[j].first <= q
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (jobs[mid].first <= q)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// The copies of many requests in one launch, between buffers of this device.
// A copy per buffer kept the copy streams busy with launches instead: 24
// requests took 72 copies and fills in, 48 out, at 3 to 4 us each.  A CTA moves
// one chunk, in the widest words that both ends' alignment allows.
template <typename W>
__device__ __forceinline__ void copy_words(uint8_t *dst, const uint8_t *src, uint64_t bytes) {
    const uint64_t n = bytes / sizeof(W);
    for (uint64_t i = threadIdx.x; i < n; i += blockDim.x)
        reinterpret_cast<W *>(dst)[i] = reinterpret_cast<const W *>(src)[i];
    for (uint64_t i = n * sizeof(W) + threadIdx.x; i < bytes; i += blockDim.x) dst[i] = src[i];
}

__global__ void __launch_bounds__(512) k_copies(const CopyJob *__restrict__ jobs, uint32_t njobs) {
    uint32_t lo = 0, hi = njobs;  // largest j with jobs[j].first <= chunk
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (jobs[mid].first <= blockIdx.x)
            lo = mid;
        else
            hi = mid;
    }
    const CopyJob jb = jobs[lo];
    const uint64_t at = (uint64_t)(blockIdx.x - jb.first) * COPY_CHUNK;
    const uint64_t end = min(at + COPY_CHUNK, jb.bytes + jb.fill);
    const uint64_t stop = min(end, jb.bytes);
    if (at < stop) {
        const uint8_t *s = jb.src + at;
        uint8_t *d = jb.dst + at;
        const uint32_t both = (uint32_t)((uintptr_t)s | (uintptr_t)d);
        if ((both & 15) == 0)
            copy_words<uint4>(d, s, stop - at);
        else if ((both & 3) == 0)
            copy_words<uint32_t>(d, s, stop - at);
        else
            copy_words<uint8_t>(d, s, stop - at);
    }
    for (uint64_t i = max(at, jb.bytes) + threadIdx.x; i < end; i += blockDim.x) jb.dst[i] = 0;
}

// Joins admitted requests: request j occupies positions [pos, pos + n) and its
// bytes sit at region_base in the pool arena.  Its offsets arrive either as
// uint64 in place in goffs or as uint32 staged in lcp at its positions; each
// becomes a pool offset.  An offset at or past the request's own arena_bytes
// is clamped to arena_bytes, where the server stores a NUL byte: the same
// empty string the single-request sort reads past the end of its arena.
// Positions get their identity index, lcp of the first position becomes 0,
// and a request of two or more strings becomes one depth-0 segment at
// R[slot].
__global__ void k_join(uint64_t *goffs, uint32_t *lcp, uint32_t *perm,
                       const ReqJob *__restrict__ jobs, uint32_t njobs, uint32_t total, Seg *R) {
    const uint32_t lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint64_t q0 = (uint64_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32 * SPAN_ITEMS;
         q0 < total; q0 += (uint64_t)warps * 32 * SPAN_ITEMS) {
        uint32_t j = find_job(jobs, njobs, (uint32_t)q0);
#pragma unroll
        for (uint32_t k = 0; k < SPAN_ITEMS; ++k) {
            const uint64_t q = q0 + k * 32 + lane;
            if (q >= total) break;
            while (j + 1 < njobs && jobs[j + 1].first <= q) ++j;
            const ReqJob jb = jobs[j];
            const uint32_t i = (uint32_t)q - jb.first;
            const uint32_t p = jb.pos + i;
            uint64_t o = jb.off_width == 4 ? (uint64_t)lcp[p] : goffs[p];
            if (o > jb.arena_bytes) o = jb.arena_bytes;
            goffs[p] = jb.region_base + o;
            perm[p] = p;
            if (i == 0) {
                lcp[p] = 0;
                if (jb.n >= 2) R[jb.slot] = Seg{jb.pos, jb.n, 0, 0};
            }
        }
    }
}

// flag[j] = 1 for every active request j that still owns a segment of R;
// base[] holds the active requests' first positions in ascending order.
__global__ void k_mark(const Seg *__restrict__ R, uint32_t nR, const uint32_t *__restrict__ base,
                       uint32_t nact, uint32_t *flag) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nR;
         i += gridDim.x * blockDim.x) {
        const uint32_t s = R[i].start;
        uint32_t lo = 0, hi = nact;  // largest j with base[j] <= s
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(base + mid) <= s)
                lo = mid;
            else
                hi = mid;
        }
        flag[lo] = 1;
    }
}

// Global positions of finished requests -> indices within each request.
__global__ void k_unbase(uint32_t *perm, const ReqJob *__restrict__ jobs, uint32_t njobs,
                         uint32_t total) {
    const uint32_t lane = threadIdx.x & 31, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint64_t q0 = (uint64_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32 * SPAN_ITEMS;
         q0 < total; q0 += (uint64_t)warps * 32 * SPAN_ITEMS) {
        uint32_t j = find_job(jobs, njobs, (uint32_t)q0);
        uint32_t pos[SPAN_ITEMS], at[SPAN_ITEMS], v[SPAN_ITEMS];
#pragma unroll
        for (uint32_t k = 0; k < SPAN_ITEMS; ++k) {
            const uint64_t q = q0 + k * 32 + lane;
            if (q < total) {
                while (j + 1 < njobs && jobs[j + 1].first <= q) ++j;
                pos[k] = jobs[j].pos;
                at[k] = pos[k] + ((uint32_t)q - jobs[j].first);
                v[k] = perm[at[k]];
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < SPAN_ITEMS; ++k)
            if (q0 + k * 32 + lane < total) perm[at[k]] = v[k] - pos[k];
    }
}

// ---- text inputs: string starts in a delimited text ---------------------------
// The reference's sortstring turns a file into strings by create_strings_delim
// (src/sortstring.c:310-335): every delimiter byte ('\n', or NUL with --raw)
// ends one string, the next string starts right after it, text after the last
// delimiter is not a string, and '\n' delimiters are overwritten with NUL.
// Each CTA covers TEXT_TILE bytes: every thread TEXT_VEC consecutive 16-byte
// chunks, loaded together before any is examined.
constexpr int TEXT_THREADS = 256;
constexpr int TEXT_VEC = 4;
constexpr uint64_t TEXT_TILE = TEXT_THREADS * 16 * TEXT_VEC;

// Bit b of a 4-byte word's result is set when byte b equals the delimiter.
__device__ __forceinline__ uint32_t delim_bits4(uint32_t w, uint32_t d4) {
    const uint32_t t = __vcmpeq4(w, d4) & 0x01010101u;
    return (t | (t >> 7) | (t >> 14) | (t >> 21)) & 0xFu;
}

// m[c], bit b: text[base + 16 c + b] == delim (positions at or past len never
// match); the thread's chunks start at base (a multiple of 16).
__device__ __forceinline__ void delim_masks(const uint8_t *__restrict__ text, uint64_t len,
                                            uint64_t base, uint8_t delim,
                                            uint32_t (&m)[TEXT_VEC]) {
    if (base + 16 * TEXT_VEC <= len) {
        const uint32_t d4 = 0x01010101u * delim;
        uint4 v[TEXT_VEC];
#pragma unroll
        for (int c = 0; c < TEXT_VEC; ++c) v[c] = reinterpret_cast<const uint4 *>(text + base)[c];
#pragma unroll
        for (int c = 0; c < TEXT_VEC; ++c)
            m[c] = delim_bits4(v[c].x, d4) | delim_bits4(v[c].y, d4) << 4 |
                   delim_bits4(v[c].z, d4) << 8 | delim_bits4(v[c].w, d4) << 12;
    } else {
#pragma unroll
        for (int c = 0; c < TEXT_VEC; ++c) {
            m[c] = 0;
            for (uint64_t b = 0; b < 16 && base + 16 * c + b < len; ++b)
                if (text[base + 16 * c + b] == delim) m[c] |= 1u << b;
        }
    }
}

__global__ void __launch_bounds__(TEXT_THREADS)
    k_text_count(const uint8_t *__restrict__ text, uint64_t len, uint8_t delim,
                 uint32_t *tile_cnt, unsigned long long *total) {
    __shared__ uint32_t warp_sums[TEXT_THREADS / 32];
    const uint64_t base = blockIdx.x * TEXT_TILE + threadIdx.x * (16ull * TEXT_VEC);
    uint32_t m[TEXT_VEC];
    delim_masks(text, len, base, delim, m);
    uint32_t c = 0;
#pragma unroll
    for (int q = 0; q < TEXT_VEC; ++q) c += __popc(m[q]);
#pragma unroll
    for (int d = 16; d; d >>= 1) c += __shfl_xor_sync(0xffffffffu, c, d);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int w = 0; w < TEXT_THREADS / 32; ++w) t += warp_sums[w];
        tile_cnt[blockIdx.x] = t;
        if (t) atomicAdd(total, (unsigned long long)t);
    }
}

// tile_base: exclusive prefix of the tile counts; n: total delimiters.  String
// r + 1 starts right after delimiter r; string 0 starts at 0.
__global__ void __launch_bounds__(TEXT_THREADS)
    k_text_starts(uint8_t *text, uint64_t len, uint8_t delim, const uint32_t *__restrict__ tile_base,
                  uint64_t n, void *offs, int off_width) {
    __shared__ uint32_t warp_sums[TEXT_THREADS / 32];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t base = blockIdx.x * TEXT_TILE + threadIdx.x * (16ull * TEXT_VEC);
    uint32_t m[TEXT_VEC];
    delim_masks(text, len, base, delim, m);
    uint32_t c = 0;
#pragma unroll
    for (int q = 0; q < TEXT_VEC; ++q) c += __popc(m[q]);
    uint32_t v = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= (uint32_t)d) v += y;
    }
    if (lane == 31) warp_sums[w] = v;
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t q = 0; q < w; ++q) before += warp_sums[q];
    uint64_t r = (uint64_t)tile_base[blockIdx.x] + before + v - c;
#pragma unroll
    for (int q = 0; q < TEXT_VEC; ++q) {
        uint32_t mq = m[q];
        while (mq) {
            const int b = __ffs(mq) - 1;
            mq &= mq - 1;
            const uint64_t i = base + 16 * q + b;
            if (r + 1 < n) {
                if (off_width == 8)
                    static_cast<uint64_t *>(offs)[r + 1] = i + 1;
                else
                    static_cast<uint32_t *>(offs)[r + 1] = (uint32_t)(i + 1);
            }
            if (delim) text[i] = 0;
            ++r;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && n) {
        if (off_width == 8)
            static_cast<uint64_t *>(offs)[0] = 0;
        else
            static_cast<uint32_t *>(offs)[0] = 0;
    }
}

// offs[i] = i: every suffix of the text (sortstring --suffix-sorting,
// create_suffixes, src/sortstring.c:349-358).
__global__ void k_iota_offs(void *offs, int off_width, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        if (off_width == 8)
            static_cast<uint64_t *>(offs)[i] = i;
        else
            static_cast<uint32_t *>(offs)[i] = (uint32_t)i;
    }
}

// out[k] = offs[perm[k]]: the sorted string starts.
// out[k] = offs[perm[k]], as out_width-byte values (4 only when every
// offset fits, which the caller knows).
__global__ void k_sorted_offs(const uint32_t *__restrict__ perm, const void *offs, int off_width,
                              uint64_t n, void *out, int out_width) {
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < n;
         k += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t i = perm[k];
        const uint64_t o = off_width == 8 ? static_cast<const uint64_t *>(offs)[i]
                                          : static_cast<const uint32_t *>(offs)[i];
        if (out_width == 8)
            static_cast<uint64_t *>(out)[k] = o;
        else
            static_cast<uint32_t *>(out)[k] = (uint32_t)o;
    }
}

// ---- tuning: byte histogram of a sample of keys -----------------------------
// hist[b] += occurrences of byte value b among the first 8 key bytes of
// `samples` strings spread evenly over the n input strings (one CTA).
__global__ void k_byte_hist(const uint8_t *__restrict__ arena, uint64_t arena_bytes,
                            const void *offs, int off_width, uint32_t n, uint32_t samples,
                            uint32_t *hist) {
    __shared__ uint32_t h[256];
    for (uint32_t b = threadIdx.x; b < 256; b += blockDim.x) h[b] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < samples; i += blockDim.x) {
        const uint32_t id = (uint32_t)((uint64_t)i * n / samples);
        const Key k = load_key(arena, arena_bytes, string_offset(offs, off_width, id));
#pragma unroll
        for (int b = 0; b < 8; ++b) atomicAdd(&h[(k.hi >> (56 - 8 * b)) & 0xFF], 1u);
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < 256; b += blockDim.x) hist[b] = h[b];
}

// ---- single-CTA exclusive scans of short per-segment arrays -----------------
constexpr int SMALL_SCAN_THREADS = 1024;

// Inclusive scan of v across the CTA; returns the CTA total in `total`.
template <int THREADS>
__device__ __forceinline__ uint32_t cta_inclusive_scan(uint32_t v, uint32_t &total,
                                                       uint32_t *warp_sums) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= (uint32_t)d) v += y;
    }
    if (lane == 31) warp_sums[w] = v;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
    for (uint32_t q = 0; q < THREADS / 32; ++q) {
        const uint32_t x = warp_sums[q];
        if (q < w) before += x;
        total += x;
    }
    __syncthreads();
    return v + before;
}

// out = exclusive scan of ceil(len / tile) over the segments; out[n] = total.
__global__ void __launch_bounds__(SMALL_SCAN_THREADS) k_seg_tiles(const Seg *segs,
                                                                   Count cnt, uint32_t tile,
                                                                   uint32_t *out) {
    after_predecessor();
    __shared__ uint32_t warp_sums[SMALL_SCAN_THREADS / 32];
    const uint32_t n = count_of(cnt);
    uint32_t c = 0;
    for (uint32_t b = 0; b < n; b += SMALL_SCAN_THREADS) {
        const uint32_t i = b + threadIdx.x;
        const uint32_t v = i < n ? (segs[i].len + tile - 1) / tile : 0;
        uint32_t t;
        const uint32_t s = cta_inclusive_scan<SMALL_SCAN_THREADS>(v, t, warp_sums);
        if (i < n) out[i] = c + s - v;
        c += t;
    }
    if (threadIdx.x == 0) out[n] = c;
}

// ---- exclusive scan (u32), three phases ----------------------------------
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 16;
constexpr int SCAN_CHUNK = SCAN_THREADS * SCAN_ITEMS;

// Block-wide exclusive scan of one value per thread; returns the block total.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t &excl) {
    __shared__ uint32_t warp_tot[SCAN_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    uint32_t wbase = 0, total = 0;
    for (int i = 0; i < SCAN_THREADS / 32; ++i) {
        const uint32_t t = warp_tot[i];
        if (i < w) wbase += t;
        total += t;
    }
    excl = wbase + x - v;
    __syncthreads();
    return total;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_reduce(const uint32_t *__restrict__ in,
                                                              Count cnt, uint32_t *partials) {
    const uint32_t n = count_of(cnt);
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_CHUNK;
    uint32_t s = 0;
    if (base < n) {
        for (int k = 0; k < SCAN_ITEMS; ++k) {
            const uint64_t i = base + (uint64_t)k * SCAN_THREADS + threadIdx.x;
            if (i < n) s += in[i];
        }
    }
    uint32_t excl;
    const uint32_t tot = block_exclusive_scan(s, excl);
    if (threadIdx.x == 0) partials[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_partials(uint32_t *partials,
                                                                uint32_t nparts) {
    uint32_t carry = 0;
    for (uint32_t b = 0; b < nparts; b += SCAN_THREADS) {
        const uint32_t i = b + threadIdx.x;
        const uint32_t v = i < nparts ? partials[i] : 0;
        uint32_t excl;
        const uint32_t tot = block_exclusive_scan(v, excl);
        if (i < nparts) partials[i] = carry + excl;
        carry += tot;
    }
    if (threadIdx.x == 0) partials[nparts] = carry;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_down(const uint32_t *in, uint32_t *out,
                                                            Count cnt,
                                                            const uint32_t *__restrict__ partials,
                                                            uint32_t nparts) {
    __shared__ uint32_t buf[SCAN_CHUNK];
    const uint32_t n = count_of(cnt);
    const uint64_t base = (uint64_t)blockIdx.x * SCAN_CHUNK;
    if (blockIdx.x == 0 && threadIdx.x == 0) out[n] = partials[nparts];
    if (base >= n) return;
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const int j = k * SCAN_THREADS + threadIdx.x;
        const uint64_t i = base + j;
        buf[j] = i < n ? in[i] : 0;
    }
    __syncthreads();
    uint32_t s = 0;
    for (int k = 0; k < SCAN_ITEMS; ++k) s += buf[threadIdx.x * SCAN_ITEMS + k];
    uint32_t excl;
    block_exclusive_scan(s, excl);
    uint32_t run = partials[blockIdx.x] + excl;
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const int j = threadIdx.x * SCAN_ITEMS + k;
        const uint32_t v = buf[j];
        buf[j] = run;
        run += v;
    }
    __syncthreads();
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const int j = k * SCAN_THREADS + threadIdx.x;
        const uint64_t i = base + j;
        if (i < n) out[i] = buf[j];
    }
}

// ---- key gather for large segments ----------------------------------------
// KEEP (a.key2 given): depth 0 also keeps key bytes 16..31 for round 1 (their
// sectors are read here anyway), depth 16 reads those copies.
// Bound by memory: index, offset, the strings' sectors and the 16 (KEEP: 32)
// bytes written.  Without copies, 4 strings a thread and 8 CTAs per SM keep
// more reads in flight than 8 strings in 4 CTAs: 100 M words 0.92 -> 0.73 ms
// (5.2 TB/s), a 16 MB text's suffixes 127 -> 97 us.  With copies the longer
// batches stay the faster form: 50 M URLs 0.86 ms, with 4 strings a thread 0.94.
// Reading both key words of a batch before the first use took 1.0 and 1.4 ms
// (80 registers, 3 CTAs).
template <bool KEEP>
__global__ void __launch_bounds__(GATHER_THREADS, KEEP ? 4 : 8)
    k_gather(SortArgs a, const Seg *L, Count cnt,
             const uint32_t *tile_base, Counters *ctr) {
    after_predecessor();
    const uint32_t nL = count_of(cnt);
    constexpr int U = KEEP ? 8 : 4;
    static_assert(GATHER_TILE % (GATHER_THREADS * U) == 0, "tile shape");
    constexpr uint32_t SUBT = GATHER_TILE / (GATHER_THREADS * U);
    const uint32_t total_tiles = tile_base[nL] * SUBT;
    unsigned long long n_save = 0, n_used = 0;
    for (uint32_t t2 = blockIdx.x; t2 < total_tiles; t2 += gridDim.x) {
        const uint32_t t = t2 / SUBT;
        const uint32_t si = find_seg(tile_base, nL, t);
        const Seg s = L[si];
        const uint32_t lo = (t - tile_base[si]) * GATHER_TILE + (t2 % SUBT) * GATHER_THREADS * U;
        if (lo >= s.len) continue;
        const uint32_t *I = a.idx[0];
        const bool save = KEEP && s.depth == 0, saved = KEEP && s.depth == KEY_BYTES;
        const bool iota = s.flags & SEG_IOTA;
        uint32_t id[U];
        uint64_t off[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t i = lo + u * GATHER_THREADS + threadIdx.x;
            id[u] = i >= s.len ? IDX_MAX : iota ? s.start + i : I[s.start + i];
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            off[u] = id[u] != IDX_MAX && !saved ? string_offset(a.offs, a.off_width, id[u]) : 0;
        uint32_t kept = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t i = lo + u * GATHER_THREADS + threadIdx.x;
            if (id[u] != IDX_MAX) {
                a.key[0][s.start + i] =
                    saved ? a.key2[id[u]]
                          : from_key(load_key(a.arena, a.arena_bytes, off[u] + s.depth));
                if (save)
                    a.key2[id[u]] =
                        from_key(load_key(a.arena, a.arena_bytes, off[u] + KEY_BYTES));
                ++kept;
            }
        }
        if (save) n_save += kept;
        if (saved) n_used += kept;
    }
    if (KEEP) {
        n_save = warp_sum(n_save);
        n_used = warp_sum(n_used);
        if ((threadIdx.x & 31) == 0 && n_save) atomicAdd(&ctr->window_saved, n_save);
        if ((threadIdx.x & 31) == 0 && n_used) atomicAdd(&ctr->window_used, n_used);
    }
}

// Keys at `depth` of up to G strings per thread: elements e0 + q * stride
// below len, whose indices stand at I[at[q]].  Every step's loads are issued for all G strings
// before any is used (index, then offset, then the two 16-byte words that
// hold the key), so that G chains of dependent reads overlap.
template <int G>
__device__ __forceinline__ void gather_keys_at(const SortArgs &a, const uint32_t *I,
                                               uint32_t depth, const uint32_t (&at)[G],
                                               uint32_t e0, uint32_t stride, uint32_t len,
                                               Key (&kk)[G], uint32_t (&ii)[G]) {
    uint64_t pos[G];
    ulonglong2 v0[G], v1[G];
#pragma unroll
    for (int q = 0; q < G; ++q) ii[q] = e0 + q * stride < len ? I[at[q]] : IDX_MAX;
#pragma unroll
    for (int q = 0; q < G; ++q)
        pos[q] = ii[q] != IDX_MAX ? string_offset(a.offs, a.off_width, ii[q]) + depth : 0ull;
#pragma unroll
    for (int q = 0; q < G; ++q) {
        const uint64_t base = pos[q] & ~15ull;
        const bool in = ii[q] != IDX_MAX && key_words_inside(a.arena_bytes, base);
        const ulonglong2 *w = reinterpret_cast<const ulonglong2 *>(a.arena + base);
        v0[q] = in ? __ldg(w) : make_ulonglong2(0, 0);
        v1[q] = in && (pos[q] & 15) ? __ldg(w + 1) : make_ulonglong2(0, 0);
    }
#pragma unroll
    for (int q = 0; q < G; ++q) {
        if (key_words_inside(a.arena_bytes, pos[q] & ~15ull))
            kk[q] = key_of_words(v0[q], v1[q], (uint32_t)pos[q] & 15u);
        else if (ii[q] != IDX_MAX)
            kk[q] = load_key_tail(a.arena, a.arena_bytes, pos[q]);
    }
}

// The same for the elements' own places in I.
template <int G>
__device__ __forceinline__ void gather_keys(const SortArgs &a, const uint32_t *I,
                                            uint32_t depth, uint32_t e0, uint32_t stride,
                                            uint32_t len, Key (&kk)[G], uint32_t (&ii)[G]) {
    uint32_t at[G];
#pragma unroll
    for (int q = 0; q < G; ++q) at[q] = e0 + q * stride;
    gather_keys_at<G>(a, I, depth, at, e0, stride, len, kk, ii);
}

// ---- register sorts of 32-bit values (samples and on-chip segments) ---------
// The threads that sort one set of values together: one warp, or 2 to 16 of a
// CTA's warps with a named barrier of their own (0 is __syncthreads).  The
// CTA form holds its size at run time (LOG2 = 0) or as a constant.
struct WarpGroup {
    static constexpr bool warp = true;
    uint32_t t;
    __device__ __forceinline__ constexpr uint32_t threads() const { return 32; }
    __device__ __forceinline__ constexpr uint32_t log2() const { return 5; }
    __device__ __forceinline__ void sync() const { __syncwarp(); }
    // whether any thread of the group has `want`; a barrier of the group
    __device__ __forceinline__ bool any(bool want) const {
        return __any_sync(0xffffffffu, want);
    }
};

template <int LOG2 = 0>
struct CtaGroup {
    static constexpr bool warp = false;
    uint32_t t, log2_threads, barrier;
    __device__ __forceinline__ constexpr uint32_t log2() const {
        return LOG2 ? LOG2 : log2_threads;
    }
    __device__ __forceinline__ constexpr uint32_t threads() const { return 1u << log2(); }
    __device__ __forceinline__ void sync() const {
        asm volatile("bar.sync %0, %1;" ::"r"(barrier), "r"(threads()) : "memory");
    }
    __device__ __forceinline__ bool any(bool want) const {
        uint32_t r;
        asm volatile(
            "{ .reg .pred p, q; setp.ne.u32 p, %1, 0; bar.red.or.pred q, %2, %3, p; "
            "selp.u32 %0, 1, 0, q; }"
            : "=r"(r)
            : "r"((uint32_t)want), "r"(barrier), "r"(threads())
            : "memory");
        return r != 0;
    }
};

template <typename V>
__device__ __forceinline__ void cmp_swap(V &a, V &b) {
    const V lo = min(a, b), hi = max(a, b);
    a = lo;
    b = hi;
}

// One exchange between threads: the lower one keeps the smaller value, the
// upper one (up) the larger.
template <typename V>
__device__ __forceinline__ V keep_side(V v, V o, bool up) {
    return (o < v) != up ? o : v;
}

// Batcher's odd-even merge sort of v[LO .. LO + N), as templates so that every
// index is a constant and the values stay in registers.
template <int LO, int N, int R, int ITEMS, typename V>
__device__ __forceinline__ void net_merge(V (&v)[ITEMS]) {
    if constexpr (2 * R < N) {
        net_merge<LO, N, 2 * R>(v);
        net_merge<LO + R, N, 2 * R>(v);
#pragma unroll
        for (int i = LO + R; i + R < LO + N; i += 2 * R) cmp_swap(v[i], v[i + R]);
    } else {
        cmp_swap(v[LO], v[LO + R]);
    }
}

template <int LO, int N, int ITEMS, typename V>
__device__ __forceinline__ void net_sort(V (&v)[ITEMS]) {
    if constexpr (N > 1) {
        net_sort<LO, N / 2>(v);
        net_sort<LO + N / 2, N / 2>(v);
        net_merge<LO, N, 1>(v);
    }
}

// Bitonic half-cleaners of strides M, M / 2, .. 1 inside a thread.
template <int M, int ITEMS, typename V>
__device__ __forceinline__ void net_clean(V (&v)[ITEMS]) {
    if constexpr (M >= 1) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            if ((i & M) == 0) cmp_swap(v[i], v[i + M]);
        net_clean<M / 2>(v);
    }
}

// Half-cleaners of lane strides m, m / 2, .. 1, then inside the lanes.  The
// loop over strides stays a loop: unrolled, the sorts outgrow the
// instruction cache.
template <int ITEMS, typename V>
__device__ __forceinline__ void warp_clean(V (&v)[ITEMS], uint32_t m, uint32_t lane) {
#pragma unroll 1
    for (; m >= 1; m /= 2) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i)
            v[i] = keep_side(v[i], __shfl_xor_sync(0xffffffffu, v[i], m), up);
    }
    net_clean<ITEMS / 2>(v);
}

// Every thread stores its values to x (16-byte words, consecutive threads
// next to each other) and loads those of thread `from`.  Two barriers.
template <class G, int ITEMS, typename V>
__device__ __forceinline__ void swap_values(const G &g, const V (&v)[ITEMS], V (&o)[ITEMS],
                                            void *x, uint32_t from) {
    constexpr int PER = 16 / sizeof(V);  // values per 16-byte word
    V w[PER];
#pragma unroll
    for (int j = 0; j < ITEMS / PER; ++j) {
#pragma unroll
        for (int q = 0; q < PER; ++q) w[q] = v[j * PER + q];
        static_cast<uint4 *>(x)[j * g.threads() + g.t] = *reinterpret_cast<const uint4 *>(w);
    }
    g.sync();
#pragma unroll
    for (int j = 0; j < ITEMS / PER; ++j) {
        *reinterpret_cast<uint4 *>(w) = static_cast<const uint4 *>(x)[j * g.threads() + from];
#pragma unroll
        for (int q = 0; q < PER; ++q) o[j * PER + q] = w[q];
    }
    g.sync();
}

// Sorts the ITEMS values of each of a group's threads; thread t ends with
// ranks t * ITEMS .. t * ITEMS + ITEMS - 1.  Odd-even merge sort inside a
// thread, then bitonic merges of 2, 4, .. threads whose first stage compares
// mirrored positions, so that every stage sorts ascending; strides of 32
// threads and more go through shared memory (x: a value per thread and item).
// Aligned blocks of `threads` (a power of two, at least 32) sort on their own.
template <class G, int ITEMS, typename V>
__device__ __forceinline__ void group_net_sort(const G &g, V (&v)[ITEMS], void *x,
                                               uint32_t threads) {
    const uint32_t t = g.t, lane = t & 31;
    net_sort<0, ITEMS>(v);
#pragma unroll 1
    for (uint32_t half = 1; half < 32; half *= 2) {
        const bool up = (lane & half) != 0;
        const uint32_t mirror = 2 * half - 1;
#pragma unroll
        for (int i = 0; i < ITEMS / 2; ++i) {
            const V p = __shfl_xor_sync(0xffffffffu, v[ITEMS - 1 - i], mirror);
            const V q = __shfl_xor_sync(0xffffffffu, v[i], mirror);
            v[i] = keep_side(v[i], p, up);
            v[ITEMS - 1 - i] = keep_side(v[ITEMS - 1 - i], q, up);
        }
        warp_clean<ITEMS>(v, half / 2, lane);
    }
    if constexpr (!G::warp) {
#pragma unroll 1
        for (uint32_t half = 32; half < threads; half *= 2) {
            V o[ITEMS];
            swap_values<G, ITEMS>(g, v, o, x, t ^ (2 * half - 1));
            const bool up = (t & half) != 0;
#pragma unroll
            for (int i = 0; i < ITEMS; ++i) v[i] = keep_side(v[i], o[ITEMS - 1 - i], up);
#pragma unroll 1
            for (uint32_t m = half / 2; m >= 32; m /= 2) {
                swap_values<G, ITEMS>(g, v, o, x, t ^ m);
                const bool um = (t & m) != 0;
#pragma unroll
                for (int i = 0; i < ITEMS; ++i) v[i] = keep_side(v[i], o[i], um);
            }
            warp_clean<ITEMS>(v, 16, lane);
        }
    }
}

// The first differing bits of a set of keys, as the high bits of 32-bit
// values: bits that all keys share carry no order and are squeezed out.
template <int ITEMS>
struct Squeezed {
    uint32_t v[ITEMS];  // squeezed bits << pos_bits | position, all ones past the end
    uint32_t f;         // first differing key bit
    uint32_t used;      // squeezed bits taken
    uint32_t byte_of;   // in lane j < used: the key byte of squeezed bit j; else `none`
    uint32_t m0, m1;    // differing bits of the 64 from bit f on that were not taken
};

// Squeezes the keys at positions e = q * stride + t < len (q < ITEMS) whose
// differing bits are mh, ml (not both 0): the first 32 - pos_bits differing
// ones of the 64 bits from the first on, run by run of adjacent bits.
template <int ITEMS>
__device__ __forceinline__ void squeeze_keys(Squeezed<ITEMS> &o, const ulonglong2 *key,
                                             uint32_t len, uint32_t stride, uint32_t t,
                                             uint64_t mh, uint64_t ml, uint32_t pos_bits,
                                             uint32_t none) {
    const uint32_t lane = t & 31, want = 32 - pos_bits;
    const uint32_t f = clz128(mh, ml);
    const uint64_t wm = window64(Key{mh, ml}, f);
    uint32_t wh[ITEMS], wl[ITEMS];
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        const uint32_t e = q * stride + t;
        const Key k = e < len ? to_key(key[e]) : Key{0, 0};
        // the 96 bits from the 32-bit word that holds bit f on
        const uint64_t top = f < 64 ? k.hi : k.lo, next = f < 64 ? k.lo : 0;
        const uint32_t w0 = (uint32_t)(top >> 32), w1 = (uint32_t)top,
                       w2 = (uint32_t)(next >> 32), w3 = (uint32_t)next;
        wh[q] = f & 32 ? __funnelshift_l(w2, w1, f) : __funnelshift_l(w1, w0, f);
        wl[q] = f & 32 ? __funnelshift_l(w3, w2, f) : __funnelshift_l(w2, w1, f);
        o.v[q] = 0;
    }
    uint32_t used = 0, byte_of = none;
    auto squeeze = [&](uint32_t &m, const uint32_t(&w)[ITEMS], uint32_t base) {
#pragma unroll 1
        while (m && used < want) {
            const uint32_t lead = __clz(m);
            const uint32_t width = min((uint32_t)__clz(~(m << lead)), want - used);
            const uint32_t mul = 1u << width, low = mul - 1, sh = 32 - lead - width;
#pragma unroll
            for (int q = 0; q < ITEMS; ++q) o.v[q] = o.v[q] * mul + ((w[q] >> sh) & low);
            if (lane - used < width) byte_of = (f + base + lead + lane - used) >> 3;
            used += width;
            m &= ~(low << sh);
        }
    };
    o.m0 = (uint32_t)(wm >> 32);
    o.m1 = (uint32_t)wm;
    squeeze(o.m0, wh, 0);
    squeeze(o.m1, wl, 32);
    o.f = f;
    o.used = used;
    o.byte_of = byte_of;
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        const uint32_t e = q * stride + t;
        o.v[q] = e < len ? o.v[q] << pos_bits | e : ~0u;
    }
}

__device__ __forceinline__ uint64_t warp_or64(uint64_t x) {
    return (uint64_t)__reduce_or_sync(0xffffffffu, (uint32_t)(x >> 32)) << 32 |
           __reduce_or_sync(0xffffffffu, (uint32_t)x);
}

// ---- asynchronous copies into shared memory -----------------------------------
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
// Waits until at most N of this thread's committed copy groups are pending.
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ---- splitter selection: one CTA per large segment ------------------------
constexpr int SAMPLE_THREADS = 512;
static_assert(SAMPLE_THREADS == 1 << 9 && SAMPLES_MAX == SAMPLE_THREADS * 8,
              "8 samples per thread");

// The samples' keys, their sorted values (later the splitters' window bits),
// the candidates: 89 KB, two CTAs per SM.
struct SampleSmem {
    ulonglong2 key[SAMPLES_MAX];
    ulonglong2 cands[SAMPLE_THREADS];
    uint32_t val[SAMPLES_MAX];
    uint64_t red[SAMPLE_THREADS / 32][2];
    uint32_t warp_cnt[SAMPLE_THREADS / 32 + 1];
    uint32_t last;
};

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}

// Splitters of segment si.  The samples are ordered as 32-bit values (their
// first differing bits and the sample number) by the register network of the
// on-chip sorts: with 4096 samples and 64-bit keys merged in shared memory
// this CTA took most of the first level's latency (one segment of 10 M URLs
// 35 us).  The order only picks quantiles: samples that tie on 20 to 24
// differing bits may stand in any order, and the chosen candidates are put in
// full-key order below.
__device__ __forceinline__ void sample_segment(const SortArgs &a, const Seg *L,
                                               uint32_t si, SampleSmem &sm, ulonglong2 *spl,
                                               uint32_t *nspl, uint16_t *tbl, uint32_t *ntiles,
                                               uint32_t *cm_size, bool from_arena) {
    const Seg s = L[si];
    const ulonglong2 *K = a.keyb(s.flags & SEG_BUF1) + s.start;
    const uint32_t t = threadIdx.x, lane = t & 31, w = t >> 5;
    const uint32_t tcls = a.target_by_class[31 - __clz(s.len)];
    const uint32_t tb = tcls ? tcls : a.target_bucket;
    uint32_t k = (s.len + tb - 1) / tb;
    if (k > a.max_splitters) k = a.max_splitters;
    if (k < 1) k = 1;
    // Eight samples per splitter keep a bucket's size within about a third of
    // its mean.  In a sort that one CTA's time counts in (below LEAF_MIN_N
    // strings), four do where the most splitters still leave buckets that are
    // mostly split again: the CTA's sort, the longest part of a level's first
    // kernel, halves (1 M uniform strings 252 -> 239 us; with four in every
    // sort 69 M batched strings 4.94 -> 4.97 ms).
    const uint32_t per = a.n < LEAF_MIN_N && s.len / (k + 1) > 2 * tb ? 4 : 8;
    uint32_t S = next_pow2(per * (k + 1));
    if (S < 256) S = 256;
    if (S > (uint32_t)SAMPLES_MAX) S = SAMPLES_MAX;
    // Sample i is the string at position pos_of(i) of the segment.  On the
    // first partition level of a round the segment's keys are not in the key
    // buffer yet (the count kernel gathers them): read them from the arena.
    auto pos_of = [&](uint32_t i) -> uint32_t {
        const uint32_t r = hash32(s.start * 0x9E3779B1u + i * 0x85EBCA77u + s.len);
        return (uint32_t)(((uint64_t)r * s.len) >> 32);
    };
    if (from_arena) {
        constexpr int G = 4;  // strings in flight per thread
#pragma unroll 1
        for (uint32_t e0 = t; e0 < S; e0 += G * SAMPLE_THREADS) {
            uint32_t at[G], id[G];
            Key kk[G];
#pragma unroll
            for (int q = 0; q < G; ++q) at[q] = s.start + pos_of(e0 + q * SAMPLE_THREADS);
            gather_keys_at<G>(a, a.idx[0], s.depth, at, e0, SAMPLE_THREADS, S, kk, id);
#pragma unroll
            for (int q = 0; q < G; ++q)
                if (e0 + q * SAMPLE_THREADS < S) sm.key[e0 + q * SAMPLE_THREADS] = from_key(kk[q]);
        }
    } else {
        // all of a thread's reads in flight at once, past the registers
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const uint32_t e = t + q * SAMPLE_THREADS;
            if (e < S) cp_async16(sm.key + e, K + pos_of(e));
        }
        cp_async_commit();
        cp_async_wait<0>();
    }
    __syncthreads();
    // The first S / 8 threads order the samples, 8 each.
    const uint32_t act = S / 8;
    uint64_t mh = 0, ml = 0;
    {
        const Key k0 = to_key(sm.key[0]);
        for (uint32_t e = t; e < S; e += SAMPLE_THREADS) {
            const Key x = to_key(sm.key[e]);
            mh |= x.hi ^ k0.hi;
            ml |= x.lo ^ k0.lo;
        }
        mh = warp_or64(mh);
        ml = warp_or64(ml);
        if (lane == 0) {
            sm.red[w][0] = mh;
            sm.red[w][1] = ml;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < SAMPLE_THREADS / 32; ++q) {
            mh |= sm.red[q][0];
            ml |= sm.red[q][1];
        }
    }
    if (mh | ml) {
        Squeezed<8> z;
        squeeze_keys<8>(z, sm.key, t < act ? S : 0u, act, t, mh, ml, 31 - __clz(S), 0u);
        group_net_sort<CtaGroup<9>, 8>(CtaGroup<9>{t, 9, 1}, z.v, sm.val, act);
        if (t < act) {
            uint4 *o = reinterpret_cast<uint4 *>(sm.val + 8 * t);
            o[0] = make_uint4(z.v[0], z.v[1], z.v[2], z.v[3]);
            o[1] = make_uint4(z.v[4], z.v[5], z.v[6], z.v[7]);
        }
    } else {  // all samples equal
        for (uint32_t e = t; e < S; e += SAMPLE_THREADS) sm.val[e] = e;
    }
    __syncthreads();
    // Candidates at ranks (j+1)*S/(k+1), padded with the all-ones key.  They
    // are in full-key order unless two values tie; only then a bitonic network
    // over the next power of two >= k slots sorts them by full key.
    ulonglong2 *cands = sm.cands;
    if (t < k)
        cands[t] = sm.key[sm.val[((t + 1) * S) / (k + 1)] & (S - 1)];
    else
        cands[t] = from_key(key_max());
    __syncthreads();
    const bool out_of_order = t + 1 < k && key_lt(to_key(cands[t + 1]), to_key(cands[t]));
    if (__syncthreads_or(out_of_order)) {
        const uint32_t kp = next_pow2(k);
        for (uint32_t kk = 2; kk <= kp; kk <<= 1) {
            for (uint32_t jj = kk >> 1; jj > 0; jj >>= 1) {
                const uint32_t i = t, l = i ^ jj;
                bool take = false;
                Key y{0, 0};
                if (i < kp) {
                    const Key x = to_key(cands[i]);
                    y = to_key(cands[l]);
                    const bool lower = l > i;
                    const bool asc = (i & kk) == 0;
                    // the lower slot keeps the min when ascending, the max otherwise
                    take = lower ? (asc ? key_lt(y, x) : key_lt(x, y))
                                 : (asc ? key_lt(x, y) : key_lt(y, x));
                }
                __syncthreads();
                if (take) cands[i] = from_key(y);
                __syncthreads();
            }
        }
    }
    // Survivors: the distinct candidates, compacted in order.
    Key cand{0, 0};
    bool keep = false;
    if (t < k) {
        cand = to_key(cands[t]);
        keep = t == 0 || !key_eq(to_key(cands[t - 1]), cand);
    }
    const uint32_t bal = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) sm.warp_cnt[w] = __popc(bal);
    __syncthreads();
    if (t == 0) {
        uint32_t run = 0;
        for (int q = 0; q < SAMPLE_THREADS / 32; ++q) {
            const uint32_t v = sm.warp_cnt[q];
            sm.warp_cnt[q] = run;
            run += v;
        }
        sm.warp_cnt[SAMPLE_THREADS / 32] = run;
    }
    __syncthreads();
    const uint32_t u = sm.warp_cnt[SAMPLE_THREADS / 32];
    ulonglong2 *out = spl + (uint64_t)si * SPL_STRIDE;
    if (keep) {
        const uint32_t pos = sm.warp_cnt[w] + __popc(bal & lanemask_lt());
        out[pos] = from_key(cand);
        cands[pos] = from_key(cand);  // candidates were read before the barriers
    }
    const uint32_t kp2 = next_pow2(u + 1);
    for (uint32_t q = u + t; q + 1 < kp2; q += SAMPLE_THREADS) out[q] = from_key(key_max());
    __syncthreads();
    // Lookup table over the TBL_BITS bits after the splitters' common prefix.
    const Key s0 = to_key(cands[0]), sl = to_key(cands[u - 1]);
    const uint32_t f = u >= 2 ? clz128(s0.hi ^ sl.hi, s0.lo ^ sl.lo) : 128u;
    if (f < 128) {
        // Entry w is the number of splitters whose window bits are below w: a
        // histogram of the splitters' window bits (in the values' area, which
        // is free by now) and its exclusive scan, 8 entries per thread.
        static_assert(TBL_N == SAMPLE_THREADS * 8 && TBL_N <= SAMPLES_MAX, "table entries");
        uint4 *h = reinterpret_cast<uint4 *>(sm.val + 8 * t);
        h[0] = h[1] = make_uint4(0, 0, 0, 0);
        __syncthreads();
        for (uint32_t j = t; j < u; j += SAMPLE_THREADS)
            atomicAdd(&sm.val[window_bits(to_key(cands[j]), f)], 1u);
        __syncthreads();
        uint32_t e[8], sum = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t x = sm.val[8 * t + i];
            e[i] = sum;
            sum += x;
        }
        uint32_t total;
        const uint32_t before =
            cta_inclusive_scan<SAMPLE_THREADS>(sum, total, sm.warp_cnt) - sum;
        uint16_t *T = tbl + (uint64_t)si * TBL_STRIDE;
        uint32_t tv[4];
#pragma unroll
        for (int i = 0; i < 8; i += 2)
            tv[i / 2] = (before + e[i]) | (before + e[i + 1]) << 16;
        *reinterpret_cast<uint4 *>(T + 8 * t) = make_uint4(tv[0], tv[1], tv[2], tv[3]);
        if (t == 0) T[TBL_N] = (uint16_t)u;
    }
    if (t == 0) {
        nspl[si] = u | (f << 16);
        const uint32_t nt = (s.len + a.tile - 1) / a.tile;
        ntiles[si] = nt;
        cm_size[si] = (2 * u + 1) * nt;
    }
}

// One CTA per large segment at a time (segments si = blockIdx.x, + gridDim.x,
// ...).  The last CTA to finish turns the segments' tile and count-matrix
// sizes into bases (exclusive scans, totals at [nL]) and clears the look-back
// scan's state for the level's total: two launches less per level.
__global__ void __launch_bounds__(SAMPLE_THREADS, 2)
    k_sample(SortArgs a, const Seg *L, Count cnt, ulonglong2 *spl, uint32_t *nspl,
             uint16_t *tbl, LevelBases lb, bool from_arena, Counters *c) {
    after_predecessor();
    extern __shared__ __align__(16) unsigned char sample_smem[];
    SampleSmem &sm = *reinterpret_cast<SampleSmem *>(sample_smem);
    const uint32_t nL = count_of(cnt), t = threadIdx.x;
    for (uint32_t si = blockIdx.x; si < nL; si += gridDim.x) {
        sample_segment(a, L, si, sm, spl, nspl, tbl, lb.ntiles, lb.cm_size, from_arena);
        __syncthreads();  // shared memory is reused by the next segment
    }
    __threadfence();
    __syncthreads();
    if (t == 0) sm.last = atomicAdd(&c->sample_ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!sm.last) return;
    __threadfence();
    // both scans at once: tiles in the upper half, matrix entries in the lower
    uint64_t carry = 0;
    for (uint32_t b = 0; b < nL; b += SAMPLE_THREADS) {
        const uint32_t i = b + t;
        const uint64_t v =
            i < nL ? (uint64_t)__ldcg(lb.ntiles + i) << 32 | __ldcg(lb.cm_size + i) : 0;
        uint64_t x = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, x, d);
            if ((t & 31) >= (uint32_t)d) x += y;
        }
        if ((t & 31) == 31) sm.red[t >> 5][0] = x;
        __syncthreads();
        uint64_t before = carry;
        for (uint32_t q = 0; q < SAMPLE_THREADS / 32; ++q) {
            if (q < t >> 5) before += sm.red[q][0];
            carry += sm.red[q][0];
        }
        __syncthreads();
        if (i < nL) {
            lb.tile_base[i] = (uint32_t)((before + x - v) >> 32);
            lb.cm_base[i] = (uint32_t)(before + x - v);
        }
    }
    const uint32_t c1 = (uint32_t)carry;
    if (t == 0) {
        lb.tile_base[nL] = (uint32_t)(carry >> 32);
        lb.cm_base[nL] = c1;
        c->sample_ticket = 0;
    }
    if (t == 0) c->count_ticket = c->scatter_ticket = 0;
    // ticket word and one status word per scan tile
    for (uint32_t q = t; q < 1 + (c1 + SCAN_CHUNK_ELEMS - 1) / SCAN_CHUNK_ELEMS;
         q += SAMPLE_THREADS)
        lb.lookback[q] = 0;
}

// ---- partition count: per-tile bucket histograms ---------------------------
// Each warp counts its own 256 consecutive keys into a private row, one
// shared-memory update per distinct bucket per 32 keys.  Bound by issued
// instructions (ALU pipe) and by the latency of its phases.  Measured, launches
// of one sort: 100 M words 1.78 -> 1.66 ms, 50 M URLs 0.79 -> 0.73 ms (1.33 ->
// 1.19 ms where it gathers), 69 M batched strings 0.95 -> 0.81 ms, against
// 16-byte compares with both end splitters, all ranks by the match unit and
// two CTAs per SM.
// Shared memory of the count kernel.
struct PartSmem {
    ulonglong2 spl[SPL_STRIDE];            // the segment's splitters
    uint64_t win[SPL_STRIDE];              // their 64 bits after the common prefix
    uint32_t tbl[TBL_N];                   // per window value: first and end splitter
    uint16_t cnt[PART_WARPS][NB_MAX + 1];  // per-warp bucket counters
};

// Keys of a lane (of PART_ITEMS) worked on at a time, and how many of these the
// match unit ranks.  Two at a time let three CTAs share an SM (40 registers);
// while gathering, four random reads in flight per lane and two CTAs are
// better.
template <bool GATHER>
constexpr int PART_HALF = GATHER ? 4 : 2;
template <bool GATHER>
constexpr int MATCH_ITEMS = GATHER ? 2 : 1;
template <bool GATHER>
constexpr int COUNT_CTAS = GATHER ? 2 : 3;

// What classification needs of a segment besides shared memory: its u
// splitters share their first f bits, the bits (ph, pl) under the mask
// (mh, ml).
struct Splitters {
    uint32_t u, f;
    uint64_t ph, pl, mh, ml;
};

// Splitters, their windows and (when f < 128) the lookup table of segment si.
__device__ __forceinline__ void load_splitters(PartSmem &sm, const ulonglong2 *spl,
                                               const uint16_t *tbl, uint32_t si,
                                               uint32_t u, uint32_t f) {
    for (uint32_t q = threadIdx.x; q < u; q += PART_THREADS) {
        const ulonglong2 x = spl[(uint64_t)si * SPL_STRIDE + q];
        sm.spl[q] = x;
        if (f < 128) sm.win[q] = window64(to_key(x), f);
    }
    if (f < 128) {
        const uint16_t *src = tbl + (uint64_t)si * TBL_STRIDE;
        for (uint32_t q = threadIdx.x * 8; q < TBL_N; q += PART_THREADS * 8) {
            const uint4 x = *reinterpret_cast<const uint4 *>(src + q);
            const uint32_t e = src[q + 8];
            uint4 *d = reinterpret_cast<uint4 *>(sm.tbl + q);
            // entry i: T[i] | T[i + 1] << 16
            d[0] = make_uint4(x.x, __funnelshift_r(x.x, x.y, 16), x.y,
                              __funnelshift_r(x.y, x.z, 16));
            d[1] = make_uint4(x.z, __funnelshift_r(x.z, x.w, 16), x.w,
                              __funnelshift_r(x.w, e, 16));
        }
    }
}

// Bucket of `key` among the u sorted distinct splitters s[0..u): range bucket
// 2j holds s[j-1] < key < s[j], equality bucket 2j+1 holds key == s[j].  A key
// without the splitters' common prefix lies before or after all of them.
// Any other is placed by the 64 bits after the prefix: the table bounds the
// splitters with its first TBL_BITS bits, and full keys are compared only
// with splitters whose 64 bits tie.
__device__ __forceinline__ uint32_t classify(const PartSmem &sm, const Splitters &p,
                                             const Key &key) {
    uint64_t off = (key.hi ^ p.ph) & p.mh;
    if (p.f > 64) off |= (key.lo ^ p.pl) & p.ml;  // the same branch for the whole CTA
    if (off) return key_lt(key, Key{p.ph, p.pl}) ? 0 : 2 * p.u;
    if (p.f >= 128) return 1;  // one splitter, all of whose bits are the prefix
    // the 64 bits from bit f on, as two shifts across 32-bit words
    const uint64_t top = p.f < 64 ? key.hi : key.lo, next = p.f < 64 ? key.lo : 0;
    const uint32_t w0 = (uint32_t)(top >> 32), w1 = (uint32_t)top, w2 = (uint32_t)(next >> 32),
                   w3 = (uint32_t)next;
    const uint32_t wh = p.f & 32 ? __funnelshift_l(w2, w1, p.f) : __funnelshift_l(w1, w0, p.f);
    const uint32_t wl = p.f & 32 ? __funnelshift_l(w3, w2, p.f) : __funnelshift_l(w2, w1, p.f);
    const uint64_t w = (uint64_t)wh << 32 | wl;
    const uint32_t r = sm.tbl[wh >> (32 - TBL_BITS)];
    uint32_t lo = r & 0xFFFF, hi = r >> 16;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (sm.win[mid] < w)
            lo = mid + 1;
        else
            hi = mid;
    }
    hi = r >> 16;
    if (lo < hi && sm.win[lo] == w) {
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (key_lt(to_key(sm.spl[mid]), key))
                lo = mid + 1;
            else
                hi = mid;
        }
        if (lo < p.u && key_eq(to_key(sm.spl[lo]), key)) return 2 * lo + 1;
    }
    return 2 * lo;
}

// Tiles for a CTA of the partition kernels, in ticket order: the first is its
// own index, later ones come from a counter, asked for while the current tile
// is worked on.  The kernels share the chip with the on-chip sorts, so a CTA
// may start late; with a fixed stride it would keep the whole kernel waiting.
// Called by all threads; a tile's work holds at least one __syncthreads.
struct TileQueue {
    uint32_t *ticket;
    uint32_t turn;
    __device__ __forceinline__ explicit TileQueue(uint32_t *t) : ticket(t), turn(0) {}
    __device__ __forceinline__ static uint32_t *slots() {
        __shared__ uint32_t s[2];
        return s;
    }
    __device__ __forceinline__ void ask() {
        if (threadIdx.x == 0) slots()[turn] = atomicAdd(ticket, 1u) + gridDim.x;
    }
    __device__ __forceinline__ uint32_t next() {
        const uint32_t t = slots()[turn];
        turn ^= 1;
        return t;
    }
};

// GATHER (first partition level of a round): the keys are loaded from the
// arena through idx and offsets and stored to the key buffer here, so the
// key gather's random arena reads overlap the classification work.
template <bool GATHER>
__global__ void __launch_bounds__(PART_THREADS, COUNT_CTAS<GATHER>) k_count(SortArgs a, const Seg *L,
                                                        Count cnt,
                                                        const uint32_t *tile_base,
                                                        const ulonglong2 *spl,
                                                        const uint32_t *nspl,
                                                        const uint16_t *tbl,
                                                        const uint32_t *cm_base,
                                                        uint32_t *cm, Counters *cnt_ctr) {
    after_predecessor();
    extern __shared__ __align__(16) unsigned char part_smem[];
    PartSmem &sm = *reinterpret_cast<PartSmem *>(part_smem);
    auto &hist = sm.cnt;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t SUB = a.tile / PART_WARPS;
    const uint32_t nL = count_of(cnt);
    const uint32_t total_tiles = tile_base[nL];
    const uint32_t lt = lanemask_lt();
    uint32_t loaded = ~0u;
    TileQueue tiles(&cnt_ctr->count_ticket);
    for (uint32_t t = blockIdx.x; t < total_tiles; t = tiles.next()) {
        tiles.ask();
        const uint32_t si = find_seg(tile_base, nL, t);
        const Seg s = L[si];
        const uint32_t u = nspl[si] & 0xFFFF, f = nspl[si] >> 16, nb = 2 * u + 1;
        const uint32_t bbits = 32 - __clz(nb);  // bucket ids are 0..nb
        if (a.l2_prefetch && threadIdx.x < 32 && t + gridDim.x < total_tiles) {
            // the keys (or, when gathering, the indices) of this CTA's next tile
            const uint32_t t2 = t + gridDim.x;
            const uint32_t s2i = find_seg(tile_base, nL, t2);
            const Seg s2 = L[s2i];
            const uint32_t lo2 = (t2 - tile_base[s2i]) * a.tile;
            const uint32_t len2 = min(a.tile, s2.len - lo2);
            if (GATHER)
                prefetch_l2(a.idx[0] + s2.start + lo2, (uint64_t)len2 * 4);
            else
                prefetch_l2(a.keyb(s2.flags & SEG_BUF1) + s2.start + lo2, (uint64_t)len2 * 16);
        }
        if (si != loaded) {
            load_splitters(sm, spl, tbl, si, u, f);
            loaded = si;
        }
        {
            uint4 *h = reinterpret_cast<uint4 *>(&hist[0][0]);
            for (uint32_t q = threadIdx.x; q < PART_WARPS * (NB_MAX + 1) / 8; q += PART_THREADS)
                h[q] = make_uint4(0, 0, 0, 0);
        }
        __syncthreads();
        Splitters sp{u, f, 0, 0, 0, 0};
        sp.mh = f >= 64 ? ~0ull : f ? ~0ull << (64 - f) : 0ull;
        sp.ml = f >= 128 ? ~0ull : f > 64 ? ~0ull << (128 - f) : 0ull;
        sp.ph = sm.spl[0].x & sp.mh;
        sp.pl = sm.spl[0].y & sp.ml;
        const uint32_t tl = t - tile_base[si];
        const uint32_t nt = tile_base[si + 1] - tile_base[si];
        const uint32_t lo = tl * a.tile + w * SUB, end = min(s.len, lo + SUB);
        // Keys and their buckets, HALF keys of a lane at a time.
        constexpr int HALF = PART_HALF<GATHER>, MATCH = MATCH_ITEMS<GATHER>;
        const bool kept = GATHER && a.key2 && s.depth == KEY_BYTES;
        const bool save = GATHER && a.key2 && s.depth == 0;
        uint32_t bk[PART_ITEMS];
#pragma unroll
        for (int h = 0; h < PART_ITEMS; h += HALF) {
            if (h * 32 >= SUB) break;  // a smaller tile
            const uint32_t e0 = lo + h * 32 + lane;
            Key kk[HALF];
            if (GATHER) {
                // round-start segments live in buffer 0
                const uint32_t *I = a.idx[0] + s.start;
                ulonglong2 *KW = a.key[0] + s.start;
                if (kept) {
                    // round 1: the keys round 0's gather kept, by string id
#pragma unroll
                    for (int q = 0; q < HALF; ++q)
                        if (e0 + q * 32 < end) kk[q] = to_key(a.key2[I[e0 + q * 32]]);
                } else {
                    uint32_t id[HALF];
                    gather_keys<HALF>(a, I, s.depth, e0, 32, end, kk, id);
                    // Depth 0 with a.key2 (a fresh round gathered here): also
                    // keep key bytes 16..31 for round 1, as k_gather does.
                    if (save) {
#pragma unroll
                        for (int q = 0; q < HALF; ++q)
                            if (e0 + q * 32 < end)
                                a.key2[id[q]] = from_key(
                                    load_key(a.arena, a.arena_bytes,
                                             string_offset(a.offs, a.off_width, id[q]) +
                                                 KEY_BYTES));
                    }
                }
#pragma unroll
                for (int q = 0; q < HALF; ++q)
                    if (e0 + q * 32 < end) KW[e0 + q * 32] = from_key(kk[q]);
            } else {
                const ulonglong2 *K = a.keyb(s.flags & SEG_BUF1) + s.start;
#pragma unroll
                for (int q = 0; q < HALF; ++q)
                    if (e0 + q * 32 < end) kk[q] = to_key(K[e0 + q * 32]);
            }
#pragma unroll
            for (int q = 0; q < HALF; ++q)
                bk[h + q] = e0 + q * 32 < end ? classify(sm, sp, kk[q]) : nb;
        }
        if ((kept || save) && lane == 0 && lo < end)
            atomicAdd(kept ? &cnt_ctr->window_used : &cnt_ctr->window_saved,
                      (unsigned long long)(end - lo));
        // The lanes of the warp that share each key's bucket: for some keys
        // from the match unit, for the others by a ballot per bucket-id bit.
        // The match unit alone (one result every 60 cycles per SM) took 60 % of
        // this kernel's time; the ballots load the ALU, which classification
        // keeps busy.  Then each key's rank among the warp's earlier keys of
        // the same bucket (keys are visited in position order: the scatter
        // stays stable).
#pragma unroll
        for (int h = 0; h < PART_ITEMS; h += HALF) {
            if (h * 32 >= SUB) break;
            uint32_t peers[HALF], sh[HALF];
#pragma unroll
            for (int q = 0; q < HALF; ++q) {
                if (q < MATCH) {
                    peers[q] = __match_any_sync(0xffffffffu, bk[h + q]);
                } else {
                    peers[q] = 0xffffffffu;
                    sh[q] = bk[h + q] << (32 - bbits);  // the highest id bit is the sign
                }
            }
#pragma unroll 1
            for (uint32_t k = 0; k < bbits; ++k) {
#pragma unroll
                for (int q = MATCH; q < HALF; ++q) {
                    const uint32_t m = __ballot_sync(0xffffffffu, (int32_t)sh[q] < 0);
                    peers[q] &= ~(m ^ (uint32_t)((int32_t)sh[q] >> 31));
                    sh[q] += sh[q];
                }
            }
#pragma unroll
            for (int q = 0; q < HALF; ++q) {
                const uint32_t b = bk[h + q], r = __popc(peers[q] & lt), base = hist[w][b];
                __syncwarp();
                if (r == 0) hist[w][b] = (uint16_t)(base + __popc(peers[q]));
                __syncwarp();
                bk[h + q] = (b << 16) | (base + r);
            }
        }
        __syncthreads();
        // Per bucket: the tile's count (to the count matrix) and each warp's
        // offset inside the tile's run of that bucket; two buckets at a time
        // (counts stay below 2^16).
        {
            uint32_t *h = reinterpret_cast<uint32_t *>(&hist[0][0]);
            for (uint32_t q = threadIdx.x; 2 * q < nb; q += PART_THREADS) {
                uint32_t run = 0;
#pragma unroll
                for (int ww = 0; ww < PART_WARPS; ++ww) {
                    const uint32_t x = h[ww * (NB_MAX + 1) / 2 + q];
                    h[ww * (NB_MAX + 1) / 2 + q] = run;
                    run += x;
                }
                uint32_t *d = cm + cm_base[si] + (uint64_t)(2 * q) * nt + tl;
                d[0] = run & 0xFFFF;
                if (2 * q + 1 < nb) d[nt] = run >> 16;
            }
        }
        __syncthreads();
        // Packed destination for the scatter: bucket << 12 | offset in the
        // tile's run of that bucket (< PART_TILE).
#pragma unroll
        for (int c = 0; c < PART_ITEMS; ++c) {
            const uint32_t e = lo + c * 32 + lane;
            if (e < end) {
                const uint32_t b = bk[c] >> 16;
                a.bkt[s.start + e] = (b << 12) | (hist[w][b] + (bk[c] & 0xFFFF));
            }
        }
        __syncthreads();
    }
}

// ---- partition scatter: a copy to precomputed destinations --------------------
// k_count left every key's bucket and its offset inside the tile's run of that
// bucket; the run's start comes from the scanned count matrix.  Tile order
// and within-tile order follow positions, so the scatter is stable.  A tile's
// indices and destinations are laid out in shared memory in output order (its
// bucket runs back to back), with each record's place in the tile; the
// write-out reads the keys from there (the tile's 64 KB, which the CTA is
// about to leave in L2) and stores consecutive records to consecutive
// addresses within every run.
// Bound by how the memory system takes the scattered stores, not by latency:
// more stores in flight are slower.  100 M words, scatter time of a sort with
// 256 threads and 1, 2, 3, 4 CTAs per SM: 2.36, 1.82, 1.84, 3.5 ms; with 512
// threads and 1 or 2: 2.11, 1.80; with the keys staged in shared memory too
// (98 KB, 1 or 2 CTAs): 2.03, 2.45; each record stored straight to its place:
// 4.1 to 4.7.
constexpr int SCATTER_THREADS = 512;
constexpr int SCATTER_ITEMS = PART_TILE / SCATTER_THREADS;  // 8
struct ScatterSmem {
    uint32_t idx[PART_TILE];    // indices in output order
    uint32_t dst[PART_TILE];    // destinations in output order
    uint16_t src[PART_TILE];    // tile position of the record at each output slot
    uint32_t gbase[NB_MAX + 1];
    uint32_t tstart[NB_MAX + 1];
    uint32_t wsum[SCATTER_THREADS / 32];
};
constexpr int SCATTER_BATCH = 4;  // keys in flight per thread in the write-out

__global__ void __launch_bounds__(SCATTER_THREADS, 2) k_scatter(
    SortArgs a, const Seg *L, Count cnt, const uint32_t *tile_base,
    const uint32_t *nspl, const uint32_t *cm_base,
    const uint32_t *cm_scan, Counters *ctr) {
    after_predecessor();
    extern __shared__ __align__(16) unsigned char scatter_smem[];
    ScatterSmem &sm = *reinterpret_cast<ScatterSmem *>(scatter_smem);
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr uint32_t QPT = (NB_MAX + 1) / SCATTER_THREADS;  // buckets per thread (2)
    const uint32_t nL = count_of(cnt);
    const uint32_t total_tiles = tile_base[nL];
    TileQueue tiles(&ctr->scatter_ticket);
    for (uint32_t t = blockIdx.x; t < total_tiles; t = tiles.next()) {
        tiles.ask();
        const uint32_t si = find_seg(tile_base, nL, t);
        const Seg s = L[si];
        const uint32_t u = nspl[si] & 0xFFFF, nb = 2 * u + 1;
        if (a.l2_prefetch && threadIdx.x < 32 && t + gridDim.x < total_tiles) {
            const uint32_t t2 = t + gridDim.x;
            const uint32_t s2i = find_seg(tile_base, nL, t2);
            const Seg s2 = L[s2i];
            const uint32_t lo2 = (t2 - tile_base[s2i]) * a.tile;
            const uint32_t len2 = min(a.tile, s2.len - lo2);
            const int b2 = s2.flags & SEG_BUF1;
            prefetch_l2(a.keyb(b2) + s2.start + lo2, (uint64_t)len2 * 16);
            if (!(s2.flags & SEG_IOTA))
                prefetch_l2(a.idxb(b2) + s2.start + lo2, (uint64_t)len2 * 4);
            prefetch_l2(a.bkt + s2.start + lo2, (uint64_t)len2 * 4);
        }
        const uint32_t tl = t - tile_base[si];
        const uint32_t nt = tile_base[si + 1] - tile_base[si];
        const uint32_t cmb = cm_base[si];
        const uint32_t seg0 = cm_scan[cmb];
        const uint32_t lo = tl * a.tile;
        const uint32_t tlen = min(a.tile, s.len - lo);
        const int ib = s.flags & SEG_BUF1;
        const ulonglong2 *Kin = a.keyb(ib) + s.start + lo;
        const uint32_t *Iin = a.idxb(ib) + s.start;
        const bool iota = s.flags & SEG_IOTA;
        const uint32_t *Din = a.bkt + s.start;
        uint32_t ii[SCATTER_ITEMS], dd[SCATTER_ITEMS];
#pragma unroll
        for (int c = 0; c < SCATTER_ITEMS; ++c) {
            const uint32_t e = c * SCATTER_THREADS + threadIdx.x;
            if (e < tlen) {
                ii[c] = iota ? s.start + lo + e : Iin[lo + e];
                dd[c] = Din[lo + e];
            }
        }
        uint32_t cnt4[QPT];
        uint32_t mysum = 0;
#pragma unroll
        for (uint32_t j = 0; j < QPT; ++j) {
            const uint32_t q = threadIdx.x * QPT + j;
            uint32_t c0 = 0;
            if (q < nb) {
                const uint64_t at = cmb + (uint64_t)q * nt + tl;
                const uint32_t g = cm_scan[at];
                c0 = cm_scan[at + 1] - g;
                sm.gbase[q] = g - seg0;
            }
            cnt4[j] = c0;
            mysum += c0;
        }
        uint32_t incl = mysum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += y;
        }
        if (lane == 31) sm.wsum[w] = incl;
        __syncthreads();
        uint32_t run = incl - mysum;
        for (uint32_t q = 0; q < w; ++q) run += sm.wsum[q];
#pragma unroll
        for (uint32_t j = 0; j < QPT; ++j) {
            sm.tstart[threadIdx.x * QPT + j] = run;
            run += cnt4[j];
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < SCATTER_ITEMS; ++c) {
            const uint32_t e = c * SCATTER_THREADS + threadIdx.x;
            if (e < tlen) {
                const uint32_t b = dd[c] >> 12, off = dd[c] & (PART_TILE - 1);
                const uint32_t slot = sm.tstart[b] + off;
                sm.src[slot] = (uint16_t)e;
                sm.idx[slot] = ii[c];
                sm.dst[slot] = sm.gbase[b] + off;
            }
        }
        __syncthreads();
        ulonglong2 *Kout = a.keyb(ib ^ 1) + s.start;
        uint32_t *Iout = a.idxb(ib ^ 1) + s.start;
        for (uint32_t i0 = 0; i0 < tlen; i0 += SCATTER_BATCH * SCATTER_THREADS) {
            ulonglong2 kv[SCATTER_BATCH];
#pragma unroll
            for (int q = 0; q < SCATTER_BATCH; ++q) {
                const uint32_t i = i0 + q * SCATTER_THREADS + threadIdx.x;
                if (i < tlen) kv[q] = Kin[sm.src[i]];
            }
#pragma unroll
            for (int q = 0; q < SCATTER_BATCH; ++q) {
                const uint32_t i = i0 + q * SCATTER_THREADS + threadIdx.x;
                if (i < tlen) {
                    const uint32_t o = sm.dst[i];
                    Kout[o] = kv[q];
                    Iout[o] = sm.idx[i];
                }
            }
        }
        __syncthreads();
    }
}

// ---- bucket emission: EMIT_CHUNKS CTAs per partitioned segment --------------
// A CTA takes 256 buckets of a segment: the reads, the key of an equality
// bucket and the list appends are one chain of dependent round trips, so that
// four CTAs side by side take a quarter of the time one takes over 1023
// buckets (26 -> 8 us for one segment).
constexpr int EMIT_THREADS = 256;
constexpr int EMIT_CHUNKS = (NB_MAX + EMIT_THREADS) / EMIT_THREADS;
__global__ void k_emit(SortArgs a, const Seg *L, Count cnt,
                       const uint32_t *tile_base,
                       const uint32_t *nspl, const uint32_t *cm_base,
                       const uint32_t *cm_scan, Seg *W1, Seg *W8, SmallLists S,
                       Seg *L2, Seg *E, uint2 *B, Seg *N, Counters *c, RoundCounters *rc,
                       Publish pub) {
    after_predecessor();
    const uint32_t nL = count_of(cnt);
    for (uint32_t q = blockIdx.x; q < nL * EMIT_CHUNKS; q += gridDim.x) {
    const uint32_t si = q / EMIT_CHUNKS, b0 = q % EMIT_CHUNKS * EMIT_THREADS;
    const uint32_t u = nspl[si] & 0xFFFF, nb = 2 * u + 1;
    if (b0 < nb) {  // the whole CTA reaches the collective appends
        const Seg s = L[si];
        const uint32_t nt = tile_base[si + 1] - tile_base[si];
        const uint32_t cmb = cm_base[si];
        const uint32_t seg0 = cm_scan[cmb];
        const uint32_t ob = (s.flags & SEG_BUF1) ^ 1u;
        const uint32_t flags = ob | SEG_KEYS;
        const uint32_t b = b0 + threadIdx.x;
        uint32_t off = 0, len = 0;
        if (b < nb) {
            off = cm_scan[cmb + (uint64_t)b * nt] - seg0;
            const uint32_t end =
                b + 1 < nb ? cm_scan[cmb + (uint64_t)(b + 1) * nt] - seg0 : s.len;
            len = end - off;
        }
        const uint32_t p = s.start + off;
        const bool bnd = len > 0 && off > 0;
        if (len == 1 && ob) {
            a.idx[0][p] = a.idx[1][p];
            a.key[0][p] = a.key[1][p];
        }
        const bool multi = len > 1;
        const bool eq = multi && (b & 1);
        bool direct = false;
        uint32_t nch = 0;
        if (eq) {
            const Key k = to_key(a.keyb(ob)[p]);
            // In buffer 0 with its keys and not final: straight to the next round.
            direct = !ob && !key_is_end(k);
            if (!direct) nch = (len + EQ_TILE - 1) / EQ_TILE;
        }
        // Every list reservation of the bucket is issued before any result
        // is used (boundary, next round, equality work items here; the
        // length-selected lists in append_by_length).
        const WarpRes rb = warp_reserve(&c->n_bound, bnd), rn = warp_reserve(&c->n_next, direct);
        // nch equality work items per bucket: warp-level exclusive sum.
        uint32_t incl = nch;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
            if ((threadIdx.x & 31) >= (uint32_t)d) incl += y;
        }
        const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
        uint32_t ebase = 0;
        if ((threadIdx.x & 31) == 31 && tot) ebase = atomicAdd(&c->n_equal, tot);
        const bool rng = multi && !(b & 1);
        append_by_length(Seg{p, len, s.depth, flags}, rng, a.warp8_cap, a.leaf_cap, W1, W8, S,
                         L2, &c->n_large_next, c);
        const uint32_t tb = warp_slot(rb), tn = warp_slot(rn);
        if (bnd) B[tb] = make_uint2(p, s.depth);
        if (direct) N[tn] = Seg{p, len, s.depth + KEY_BYTES, 0u};
        ebase = __shfl_sync(0xffffffffu, ebase, 31) + incl - nch;
        for (uint32_t ch = 0; ch < nch; ++ch)
            E[ebase + ch] = Seg{p, len, s.depth, ob | (ch << SEG_CHUNK_SHIFT)};
        if (b == 0) atomicAdd(&c->partitioned, (unsigned long long)s.len);
    }
    }
    // (the count of the level just emitted starts the next one at 0)
    if (publish(pub, rc) && threadIdx.x == 0) c->n_large_next = 0;
}

// ---- segments of <= 32 strings: one warp, one string per lane -------------
constexpr int WARP_THREADS = 256;

__device__ __forceinline__ void load_elem(const SortArgs &a, const Seg &s, uint32_t e, Key &k,
                                          uint32_t &id) {
    const int b = s.flags & SEG_BUF1;
    id = a.idxb(b)[s.start + e];
    k = (s.flags & SEG_KEYS)
            ? to_key(a.keyb(b)[s.start + e])
            : load_key(a.arena, a.arena_bytes, string_offset(a.offs, a.off_width, id) + s.depth);
}

// Order of records in the in-warp refinement: run head first, then (key,
// index).  Records outside runs carry their own lane as head.
__device__ __forceinline__ bool run_lt(uint32_t h1, const Key &k1, uint32_t i1, uint32_t h2,
                                       const Key &k2, uint32_t i2) {
    return h1 != h2 ? h1 < h2 : pair_lt(k1, i1, k2, i2);
}

// Runs of exactly two strings, resolved by the whole warp: lane j compares the
// two strings' 16-byte windows at depth + 16 j, so one step covers 512 bytes;
// the first lane whose windows differ or end decides order and LCP (what a
// lane past the end of a string reads is never used).  A pair still equal
// after PAIR_CHUNKS steps stays a run, 512 * PAIR_CHUNKS bytes deeper.
// `start` is the lane's group's segment start; a pair's members keep
// ascending indices (their order when equal).  Warp-collective.
constexpr uint32_t PAIR_CHUNKS = 16;

template <int W>
__device__ __forceinline__ void warp1_pairs(const uint8_t *__restrict__ arena,
                                            uint64_t arena_bytes, const void *__restrict__ offs,
                                            int off_width, uint32_t *__restrict__ idx0,
                                            uint32_t *__restrict__ lcp, uint32_t start,
                                            uint32_t lane, uint32_t id, bool &run, uint32_t &h,
                                            uint32_t &depth, uint32_t &moved) {
    const uint32_t li = lane & (W - 1);
    const uint32_t nh1 = __shfl_down_sync(0xffffffffu, h, 1);
    const uint32_t nh2 = __shfl_down_sync(0xffffffffu, h, 2);
    const bool nr1 = __shfl_down_sync(0xffffffffu, (int)run, 1) != 0;
    const bool nr2 = __shfl_down_sync(0xffffffffu, (int)run, 2) != 0;
    const bool pair_head = run && h == lane && li + 1 < (uint32_t)W && nr1 && nh1 == h &&
                           !(li + 2 < (uint32_t)W && nr2 && nh2 == h);
    uint32_t pairs = __ballot_sync(0xffffffffu, pair_head);
    while (pairs) {
        const uint32_t p = __ffs(pairs) - 1;
        pairs &= pairs - 1;
        const uint32_t ia = __shfl_sync(0xffffffffu, id, p);
        const uint32_t ib = __shfl_sync(0xffffffffu, id, p + 1);
        const uint32_t d0 = __shfl_sync(0xffffffffu, depth, p);
        const uint32_t pos = __shfl_sync(0xffffffffu, start, p) + (p & (W - 1));
        const uint64_t oa = string_offset(offs, off_width, ia);
        const uint64_t ob = string_offset(offs, off_width, ib);
        uint32_t chunk = 0, found = 0;
        for (; chunk < PAIR_CHUNKS; ++chunk) {
            const uint64_t at = (uint64_t)d0 + chunk * (32u * KEY_BYTES) + lane * KEY_BYTES;
            const Key ka = load_key(arena, arena_bytes, oa + at);
            const Key kb = load_key(arena, arena_bytes, ob + at);
            const bool same = key_eq(ka, kb);
            const uint32_t stop = __ballot_sync(0xffffffffu, !same || key_is_end(ka));
            if (stop) {
                const uint32_t f = __ffs(stop) - 1;
                if (lane == f) {
                    const uint32_t base_d = (uint32_t)at;
                    const bool swap = !same && key_lt(kb, ka);
                    idx0[pos] = swap ? ib : ia;
                    idx0[pos + 1] = swap ? ia : ib;
                    lcp[pos + 1] = base_d + (same ? key_len(ka) : key_lcp(ka, kb));
                }
                found = 1;
                break;
            }
        }
        if (lane == p || lane == p + 1) {
            if (found) {
                run = false;
                h = lane;
            } else {
                depth += PAIR_CHUNKS * 32u * KEY_BYTES;
            }
        }
        if (lane == p) moved += 2 * (chunk + found);
    }
}

// In-warp refinement of the runs a one-per-lane sort left (lanes with `run`,
// h = the run's first lane, keys equal up to `depth`, id = the lane's record).
// Each step first resolves the runs of two with the whole warp (warp1_pairs);
// then the members of the other runs load their next 16 bytes, each run is
// re-sorted inside its own lanes, the LCPs decided at this depth are written,
// and the runs of equal keys that remain become the next step's runs.  At
// most `steps` steps, then what is left goes to the next round.  This is the
// next round's one-warp sort of those runs done without a round trip: the
// same order and LCPs.  The keys of the segment's first and last position,
// which the round's boundary pass reads, stay as the first sort wrote them.
// Returns this lane's count of string steps (for the statistics).
// Warp-collective.
template <int W>
__device__ __forceinline__ uint32_t warp1_deepen(const uint8_t *__restrict__ arena,
                                              uint64_t arena_bytes, const void *__restrict__ offs,
                                              int off_width, uint32_t *__restrict__ idx0,
                                              uint32_t *__restrict__ lcp, uint32_t steps,
                                              uint32_t start, uint32_t depth, uint32_t lane,
                                              uint32_t id, bool run, uint32_t h, Seg *N,
                                              Counters *c) {
    const uint32_t li = lane & (W - 1), base = lane & ~(uint32_t)(W - 1);
    const uint32_t m = lane == 31 ? 0xffffffffu : ((2u << lane) - 1u);
    uint32_t moved = 0;
    Key k = key_max();  // records outside runs are never compared by key
    for (uint32_t it = 0; it < steps && __any_sync(0xffffffffu, run); ++it) {
        warp1_pairs<W>(arena, arena_bytes, offs, off_width, idx0, lcp, start, lane, id, run, h,
                       depth, moved);
        if (!__any_sync(0xffffffffu, run)) break;
        if (run) k = load_key(arena, arena_bytes, string_offset(offs, off_width, id) + depth);
        moved += run;
        // Sorting by (head, key, index) keeps every record outside a run in
        // its lane and every run inside its own lanes.
        uint32_t hh = run ? h : lane;
        bool r = run;
#pragma unroll
        for (int kk = 2; kk <= W; kk <<= 1) {
#pragma unroll
            for (int j = kk >> 1; j > 0; j >>= 1) {
                Key ok;
                ok.hi = __shfl_xor_sync(0xffffffffu, k.hi, j);
                ok.lo = __shfl_xor_sync(0xffffffffu, k.lo, j);
                const uint32_t oi = __shfl_xor_sync(0xffffffffu, id, j);
                const uint32_t oh = __shfl_xor_sync(0xffffffffu, hh, j);
                const bool orr = __shfl_xor_sync(0xffffffffu, (int)r, j) != 0;
                const bool up = kk == W || (lane & kk) == 0;
                const bool keep_min = ((lane & j) == 0) == up;
                const bool take = keep_min ? run_lt(oh, ok, oi, hh, k, id)
                                           : run_lt(hh, k, id, oh, ok, oi);
                if (take) {
                    k = ok;
                    id = oi;
                    hh = oh;
                    r = orr;
                }
            }
        }
        Key prev, next;
        prev.hi = __shfl_up_sync(0xffffffffu, k.hi, 1);
        prev.lo = __shfl_up_sync(0xffffffffu, k.lo, 1);
        next.hi = __shfl_down_sync(0xffffffffu, k.hi, 1);
        next.lo = __shfl_down_sync(0xffffffffu, k.lo, 1);
        const uint32_t ph = __shfl_up_sync(0xffffffffu, hh, 1);
        const uint32_t nh = __shfl_down_sync(0xffffffffu, hh, 1);
        // A run's head is one of its members' lanes, never another record's
        // own lane, so equal heads mean the same run.
        const bool same_prev = r && li > 0 && ph == hh;
        const bool same_next = r && li + 1 < (uint32_t)W && nh == hh;
        const bool eqp = same_prev && key_eq(prev, k);
        const bool eqn = same_next && key_eq(next, k);
        if (r) {
            const uint32_t p = start + li;
            idx0[p] = id;
            if (same_prev) {
                if (!eqp)
                    lcp[p] = depth + key_lcp(prev, k);
                else if (key_is_end(k))
                    lcp[p] = depth + key_len(k);
            }
        }
        run = r && !key_is_end(k) && (eqp || eqn);
        const uint32_t heads = __ballot_sync(0xffffffffu, run && !eqp);
        h = run ? 31 - __clz(heads & m) : lane;
        depth += KEY_BYTES;
    }
    // What is still unresolved goes to the next round at the depth reached.
    const uint32_t nh = __shfl_down_sync(0xffffffffu, h, 1);
    const bool nrun = __shfl_down_sync(0xffffffffu, (int)run, 1) != 0;
    const bool tail = run && !(li + 1 < (uint32_t)W && nrun && nh == h);
    emit_next_warp(N, c, tail, start + (h - base), lane - h + 1, depth);
    return moved;
}

// Sorts one segment of at most W strings held by the W lanes of one aligned
// lane group (W = 8 or 32; lane li of the group holds string li).  Every
// lane of the warp calls this with its group's segment (len 0 for idle
// groups): the shuffles, ballots and the next-round append are
// warp-collective.
template <int W>
__device__ __forceinline__ uint32_t warp1_group(const SortArgs &a, const Seg &s, uint32_t lane,
                                                uint32_t steps, Seg *N, Counters *c) {
    const uint32_t li = lane & (W - 1), base = lane & ~(uint32_t)(W - 1);
    const bool v = li < s.len;
    uint32_t id = IDX_MAX;
    Key k = key_max();
    if (v) load_elem(a, s, li, k, id);
    // Bits in which the group's keys differ.
    Key k0;
    k0.hi = __shfl_sync(0xffffffffu, k.hi, base);
    k0.lo = __shfl_sync(0xffffffffu, k.lo, base);
    uint64_t dh = v ? (k.hi ^ k0.hi) : 0, dl = v ? (k.lo ^ k0.lo) : 0;
#pragma unroll
    for (int d = W / 2; d > 0; d >>= 1) {
        dh |= __shfl_xor_sync(0xffffffffu, dh, d);
        dl |= __shfl_xor_sync(0xffffffffu, dl, d);
    }
    // Packed 64-bit keys (window after the common prefix, source lane), a
    // bitonic sort inside the group (the last stage ascending for every
    // group), then each record moves to its rank.  Groups whose keys are all
    // equal sort by lane alone, which keeps them in place.
    const bool diff = (dh | dl) != 0;
    const uint32_t f = diff ? clz128(dh, dl) : 0u;
    bool bad = false;
    if (__any_sync(0xffffffffu, diff)) {  // else every group's keys are all equal
        uint64_t x = !v ? ~0ull : (diff ? sort_key(k, f, lane) : (uint64_t)lane);
#pragma unroll
        for (int kk = 2; kk <= W; kk <<= 1) {
#pragma unroll
            for (int j = kk >> 1; j > 0; j >>= 1) {
                const uint64_t y = __shfl_xor_sync(0xffffffffu, x, j);
                const bool up = kk == W || (lane & kk) == 0;
                const bool keep_min = ((lane & j) == 0) == up;
                x = keep_min ? (y < x ? y : x) : (y < x ? x : y);
            }
        }
        const uint32_t src = v ? (uint32_t)(x & 31) : lane;
        Key kn;
        kn.hi = __shfl_sync(0xffffffffu, k.hi, src);
        kn.lo = __shfl_sync(0xffffffffu, k.lo, src);
        const uint32_t idn = __shfl_sync(0xffffffffu, id, src);
        k = kn;
        id = idn;
        // Pairs with equal windows must also be in full-key order.
        Key kp;
        kp.hi = __shfl_up_sync(0xffffffffu, k.hi, 1);
        kp.lo = __shfl_up_sync(0xffffffffu, k.lo, 1);
        bad = v && diff && li > 0 &&
              (window64(kp, f) >> POS_BITS) == (window64(k, f) >> POS_BITS) && key_lt(k, kp);
    }
    if (__any_sync(0xffffffffu, bad)) {
        // Full (key, index) comparator over every group (rare).
#pragma unroll
        for (int kk = 2; kk <= W; kk <<= 1) {
#pragma unroll
            for (int j = kk >> 1; j > 0; j >>= 1) {
                Key ok;
                ok.hi = __shfl_xor_sync(0xffffffffu, k.hi, j);
                ok.lo = __shfl_xor_sync(0xffffffffu, k.lo, j);
                const uint32_t oi = __shfl_xor_sync(0xffffffffu, id, j);
                const bool up = kk == W || (lane & kk) == 0;
                const bool keep_min = ((lane & j) == 0) == up;
                const bool take = keep_min ? pair_lt(ok, oi, k, id) : pair_lt(k, id, ok, oi);
                if (take) {
                    k = ok;
                    id = oi;
                }
            }
        }
    }
    Key prev, next;
    prev.hi = __shfl_up_sync(0xffffffffu, k.hi, 1);
    prev.lo = __shfl_up_sync(0xffffffffu, k.lo, 1);
    next.hi = __shfl_down_sync(0xffffffffu, k.hi, 1);
    next.lo = __shfl_down_sync(0xffffffffu, k.lo, 1);
    const bool head = v && (li == 0 || !key_eq(prev, k));
    const uint32_t heads = __ballot_sync(0xffffffffu, head);
    if (v) {
        const uint32_t p = s.start + li;
        a.idx[0][p] = id;
        if (li == 0 || li == s.len - 1) a.key[0][p] = from_key(k);
        if (li > 0) {
            if (!key_eq(prev, k))
                a.lcp[p] = s.depth + key_lcp(prev, k);
            else if (key_is_end(k))
                a.lcp[p] = s.depth + key_len(k);
        }
    }
    // Runs: maximal groups of at least two equal keys that do not end; h is
    // the run's first lane (at or after the group's lane 0).
    const bool eq_next = v && li + 1 < s.len && key_eq(next, k);
    bool run = v && !key_is_end(k) && (!head || eq_next);
    const uint32_t m = lane == 31 ? 0xffffffffu : ((2u << lane) - 1u);
    uint32_t h = run ? 31 - __clz(heads & m) : lane;
    if (steps && __any_sync(0xffffffffu, run))
        return warp1_deepen<W>(a.arena, a.arena_bytes, a.offs, a.off_width, a.idx[0], a.lcp,
                               steps, s.start, s.depth + KEY_BYTES, lane, id, run, h, N,
                               c);
    const bool tail = run && !eq_next;  // a run's last lane
    emit_next_warp(N, c, tail, s.start + (h - base), lane - h + 1, s.depth + KEY_BYTES);
    return 0;
}

// Segments of <= WARP1_CAP strings.  First pass: a warp takes W1_PACK
// consecutive list entries and sorts those of at most 8 strings together, one
// per 8-lane group, so that their loads overlap.  Second pass: one warp per
// remaining segment.
constexpr uint32_t W1_PACK = 4, W1_SMALL = 8;

__global__ void __launch_bounds__(WARP_THREADS) k_warp1(SortArgs a, const Seg *T0,
                                                        Span sp, Seg *N, Counters *c) {
    after_predecessor();
    const uint32_t lo = count_of(sp.lo);
    const Seg *T = T0 + lo;
    const uint32_t nT = count_of(sp.hi) - lo;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warp0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
    unsigned long long fresh = 0, keyed = 0, deep = 0;
    for (uint32_t g0 = warp0 * W1_PACK; g0 < nT; g0 += nwarps * W1_PACK) {
        const uint32_t j = lane >> 3;
        const Seg sj = g0 + j < nT ? T[g0 + j] : Seg{0, 0, 0, 0};
        const bool small = sj.len <= W1_SMALL;
        if ((lane & 7) == 0) {
            if (sj.flags & SEG_KEYS)
                keyed += sj.len;
            else
                fresh += sj.len;
        }
        if (__any_sync(0xffffffffu, small && sj.len > 0))
            deep += warp1_group<8>(a, small ? sj : Seg{0, 0, 0, 0}, lane, a.warp1_deep, N, c);
    }
    for (uint32_t g = warp0; g < nT; g += nwarps) {
        const Seg s = T[g];
        if (s.len > W1_SMALL) deep += warp1_group<32>(a, s, lane, a.warp1_deep, N, c);
    }
    if ((lane & 7) == 0 && (fresh | keyed)) {  // each 8-lane group's leader
        atomicAdd(&c->warp1_fresh, fresh);
        atomicAdd(&c->warp1_keyed, keyed);
    }
    deep = warp_sum(deep);
    if (lane == 0 && deep) atomicAdd(&c->warp1_deep, deep);
}

// ---- segments of 33..4096 strings: a group of threads each ------------------
// A group of GT = 32, 64, 128, 256 or 512 threads sorts one segment of up to
// ITEMS * GT strings (8 per thread; 2 or 4 for the smallest).  Records (16-byte
// key, index) sit in shared memory at their positions; what moves is one
// 32-bit value per record in registers: the first bits in which the segment's
// keys differ at all, with the position in the low bits.  Bits that every key
// of the segment shares carry no order, so they are squeezed out (letters
// leave 5 bits of each byte): the 20 to 26 squeezed bits order most segments
// completely.  Values whose squeezed bits tie are checked against the full
// keys; a tied run out of order is put right in place when it is short, else
// the segment is refined on further bits.
//
// The sort is bound by issued instructions and shared-memory latency, not by
// HBM: 32-bit values make a compare-exchange one min and one max, and an
// exchange between lanes one shuffle and one select; a neighbour's LCP follows
// from the first differing bit of two values, so full keys are read for ties
// only.  24 bytes of shared memory per string let 1024 threads share an SM.
// Measured on B200 against 64-bit packed keys merged in shared memory (80
// registers, 768 threads per SM): 10,000 partitioned segments of 400 strings
// at 55 G strings/s; the CTA-sort launches of 69 M batched strings 2.79 -> 1.53
// ms, of 16 M suffixes 4.23 -> 2.59 ms, of 50 M URLs 2.27 -> 1.62 ms.  In a sort
// of 10 M URLs a warp of 256 strings issues 2400 instructions, the ALU pipe is
// active 66 % of the time and DRAM 11 %.
// The other side: strings that begin with one of a few prefixes use the bits up
// on these, tie in long runs and are sorted twice.  Lists of 250 to 2000 strings
// whose first 6 letters come from 5 to 100 groups take 0.78 to 0.9 of the 64-bit
// sorts' speed (prefixes of 3, 9, 12 letters 1.1 to 6 times).  Sorting on 64-bit
// values at once where a sample of records ties mends most of these and costs
// 1.5 % of the 69 M batched strings' time.

// Shared memory of one group, for 8 strings per thread: keys, values (in
// passing between threads, and the final order), indices, and what its warps
// tell each other.  Values and indices together also hold 64-bit values while
// a segment is refined.
struct SegMem {
    ulonglong2 *key;
    uint32_t *val, *idx;
    uint64_t *red;          // two per warp
    uint32_t *last, *first; // values at the edges of each warp
};
constexpr __host__ __device__ size_t seg_bytes(uint32_t threads) {
    return threads * 8 * 24 + (threads + 31) / 32 * 32;
}
__device__ __forceinline__ SegMem seg_mem(unsigned char *base, uint32_t threads) {
    SegMem m;
    m.key = reinterpret_cast<ulonglong2 *>(base);
    m.val = reinterpret_cast<uint32_t *>(base + threads * 128);
    m.idx = m.val + threads * 8;
    m.red = reinterpret_cast<uint64_t *>(base + threads * 192);
    m.last = reinterpret_cast<uint32_t *>(base + threads * 192 + threads / 32 * 16);
    m.first = m.last + threads / 32;
    return m;
}

// Final order: per rank the record's position and, above it, the key bytes
// it shares with the record before, up to 14 (SEG_TIE: 15 or not known from
// the values).
constexpr uint32_t SEG_ORD_BITS = 12, SEG_TIE = 15;

// Bits of a position among threads * ITEMS.
template <int ITEMS, class G>
__device__ __forceinline__ constexpr uint32_t pos_bits(const G &g) {
    return g.log2() + (ITEMS == 2 ? 1 : ITEMS == 4 ? 2 : 3);
}

// Takes the next bits of `mask` (most significant first, at most `need`) off
// it as one run of adjacent bits: `width` bits that start `lead` bits from the
// top.  False when the mask is empty.
__device__ __forceinline__ bool next_run(uint64_t &mask, uint32_t need, uint32_t &lead,
                                         uint32_t &width) {
    if (!mask || !need) return false;
    lead = (uint32_t)__clzll((long long)mask);
    const uint64_t inv = ~(mask << lead);
    const uint32_t run = inv ? (uint32_t)__clzll((long long)inv) : 64u;
    width = min(run, need);
    mask &= ~((width == 64 ? ~0ull : ((1ull << width) - 1)) << (64 - lead - width));
    return true;
}

// Orders the records by further differing bits after a first sort whose tied
// runs were out of order: every pass sorts (first rank of the record's tied
// run, its next differing bits, position) as 64-bit values; 40 or more bits
// a pass, so at most four passes for the 128 key bits.  mh, ml: the differing
// bits not used yet.  On return sm.val holds positions only, in (key,
// position) order; sm.idx is read again from I.
template <class G, int ITEMS>
__device__ __noinline__ void group_refine(G g, SegMem sm, const uint32_t *I, uint32_t len,
                                          uint64_t mh, uint64_t ml) {
    const uint32_t PB = pos_bits<ITEMS>(g), PM = (1u << PB) - 1, MORE = 64 - 2 * PB;
    constexpr int GRP = ITEMS < 4 ? ITEMS : 4;
    const uint32_t t = g.t, lane = t & 31, gw = t >> 5;
    uint64_t v[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t r = t * ITEMS + i;
        v[i] = r < len ? (uint64_t)sm.val[r] : ~0ull;
    }
#pragma unroll 1
    for (int pass = 0; pass < 5; ++pass) {
        // First rank of each record's tied run (a running maximum of the ranks
        // at which a run starts), in place of the bits used so far.
        if (lane == 31) sm.red[2 * gw] = v[ITEMS - 1];
        g.sync();
        uint64_t pv = __shfl_up_sync(0xffffffffu, v[ITEMS - 1], 1);
        if (lane == 0 && gw) pv = sm.red[2 * gw - 2];
        uint32_t h = 0;
        bool tie = false;
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            const uint32_t r = t * ITEMS + i;
            const uint64_t cur = v[i];
            const bool start = r == 0 || (cur >> PB) != (pv >> PB);
            tie |= !start && r < len;
            if (start) h = r;
            v[i] = (uint64_t)h << (64 - PB) | ((uint32_t)cur & PM);
            pv = cur;
        }
        uint32_t hm = h;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, hm, d);
            if (lane >= (uint32_t)d) hm = max(hm, y);
        }
        if (lane == 31) sm.red[2 * gw + 1] = hm;
        hm = __shfl_up_sync(0xffffffffu, hm, 1);
        if (lane == 0) hm = 0;
        if (!g.any(tie) || !(mh | ml)) break;
        for (uint32_t q = 0; q < gw; ++q) hm = max(hm, (uint32_t)sm.red[2 * q + 1]);
        uint64_t nh = mh, nl = ml;
#pragma unroll
        for (int g = 0; g < ITEMS; g += GRP) {
            Key k[GRP];
            uint64_t acc[GRP];
#pragma unroll
            for (int q = 0; q < GRP; ++q) {
                k[q] = t * ITEMS + g + q < len ? to_key(sm.key[(uint32_t)v[g + q] & PM]) : key_max();
                acc[q] = 0;
            }
            uint32_t need = MORE, lead, width;
            nh = mh;
            nl = ml;
            while (next_run(nh, need, lead, width)) {
#pragma unroll
                for (int q = 0; q < GRP; ++q)
                    acc[q] = (acc[q] << width) | (k[q].hi << lead >> (64 - width));
                need -= width;
            }
            while (next_run(nl, need, lead, width)) {
#pragma unroll
                for (int q = 0; q < GRP; ++q)
                    acc[q] = (acc[q] << width) | (k[q].lo << lead >> (64 - width));
                need -= width;
            }
#pragma unroll
            for (int q = 0; q < GRP; ++q) {
                const uint64_t head = max((uint32_t)(v[g + q] >> (64 - PB)), hm);
                v[g + q] = t * ITEMS + g + q < len
                               ? head << (64 - PB) | acc[q] << PB | ((uint32_t)v[g + q] & PM)
                               : ~0ull;
            }
        }
        mh = nh;
        ml = nl;
        group_net_sort<G, ITEMS>(g, v, sm.val, g.threads());
        g.sync();
    }
    g.sync();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) sm.val[t * ITEMS + i] = (uint32_t)v[i] & PM;
    for (uint32_t e = t; e < len; e += g.threads()) sm.idx[e] = I[e];
    g.sync();
}

// Puts the tied runs that are out of full-key order right, each by the thread
// that finds its first inversion (insertion sort; equal keys keep position
// order).  With a run of more than SEG_FIX records among them nothing is
// moved: returns 1, or 2 when one is longer than SEG_FULL; else 0.
constexpr uint32_t SEG_FIX = 12, SEG_FULL = 64;

template <class G, int ITEMS>
__device__ __noinline__ uint32_t group_fix_runs(G g, SegMem sm, uint32_t len) {
    const uint32_t PB = pos_bits<ITEMS>(g), PM = (1u << PB) - 1, t = g.t;
    auto val = [&](uint32_t r) -> uint32_t & { return sm.val[r]; };
    auto key = [&](uint32_t r) -> Key { return to_key(sm.key[val(r) & PM]); };
    auto tied = [&](uint32_t r) -> bool { return ((val(r) ^ val(r - 1)) >> PB) == 0; };
    // The run around rank e, as far as SEG_FULL + 1 records.  Sorting a run
    // moves values of equal squeezed bits only, so what this reads of other
    // threads' runs (one value past either end) does not change under it.
    auto extent = [&](uint32_t e, uint32_t &lo, uint32_t &hi) {
        lo = e - 1;
        while (lo > 0 && e - lo <= SEG_FULL && tied(lo)) --lo;
        hi = e + 1;
        while (hi < len && hi - lo <= SEG_FULL && tied(hi)) ++hi;
    };
    uint32_t own = 0, longest = 0;
#pragma unroll 1
    for (int q = 0; q < ITEMS; ++q) {
        const uint32_t e = q * g.threads() + t;
        if (e == 0 || e >= len || !tied(e) || !key_lt(key(e), key(e - 1))) continue;
        uint32_t lo, hi;
        extent(e, lo, hi);
        longest = max(longest, hi - lo);
        if (hi - lo > SEG_FIX) continue;
        bool first = true;  // no earlier inversion in the run
        for (uint32_t r = lo + 1; first && r < e; ++r) first = !key_lt(key(r), key(r - 1));
        if (first) own |= 1u << q;
    }
    if (g.any(longest > SEG_FIX)) return g.any(longest > SEG_FULL) ? 2 : 1;
    for (; own; own &= own - 1) {
        uint32_t lo, hi;
        extent((__ffs(own) - 1) * g.threads() + t, lo, hi);
        for (uint32_t i = lo + 1; i < hi; ++i) {
            const uint32_t x = val(i);
            const Key kx = to_key(sm.key[x & PM]);
            uint32_t j = i;
            while (j > lo && key_lt(kx, key(j - 1))) {
                val(j) = val(j - 1);
                --j;
            }
            val(j) = x;
        }
    }
    g.sync();
    return 0;
}

// Orders a segment of `len` records (at most GT * ITEMS, in sm.key at their
// positions) whose keys differ in the bits mh, ml (not both 0): writes the
// final order to sm.val.  Returns whether a run of more than SEG_FULL tied
// records was out of order.
template <class G, int ITEMS>
__device__ __forceinline__ bool order_segment(const G &g, const SegMem &sm, const uint32_t *I,
                                              uint32_t len, uint64_t mh, uint64_t ml) {
    const uint32_t PB = pos_bits<ITEMS>(g), PM = (1u << PB) - 1;
    const uint32_t t = g.t, lane = t & 31, gw = t >> 5;
    Squeezed<ITEMS> z;
    squeeze_keys<ITEMS>(z, sm.key, len, g.threads(), t, mh, ml, PB, SEG_TIE);
    uint32_t(&v)[ITEMS] = z.v;
    group_net_sort<G, ITEMS>(g, v, sm.val, g.threads());
    // Ties on the squeezed bits must be in full-key order.  A pair out of
    // order that both lie in one thread and tie with nothing else is swapped
    // on the spot; other runs out of order go through shared memory.
    uint32_t pv = __shfl_up_sync(0xffffffffu, v[ITEMS - 1], 1);
    uint32_t nv = __shfl_down_sync(0xffffffffu, v[0], 1);
    if constexpr (!G::warp) {
        if (lane == 31) sm.last[gw] = v[ITEMS - 1];
        if (lane == 0) sm.first[gw] = v[0];
        g.sync();
        if (lane == 0 && gw) pv = sm.last[gw - 1];
        if (lane == 31 && gw + 1 < g.threads() / 32) nv = sm.first[gw + 1];
    }
    if (t == 0) pv = ~v[0];
    if (t == g.threads() - 1) nv = ~v[ITEMS - 1];
    bool full = false, bad = false;
    uint32_t tie = 0;  // bit i: rank t * ITEMS + i ties with the one before
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
        if ((v[i] ^ (i ? v[i ? i - 1 : 0] : pv)) <= PM) tie |= 1u << i;
    if ((nv ^ v[ITEMS - 1]) <= PM) tie |= 1u << ITEMS;
    if (tie && t * ITEMS < len) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if ((tie >> i & 1u) && t * ITEMS + i < len) {
                const uint32_t y = i ? v[i ? i - 1 : 0] : pv;
                if (key_lt(to_key(sm.key[v[i] & PM]), to_key(sm.key[y & PM]))) {
                    if (i > 0 && (tie >> (i ? i - 1 : 0) & 7u) == 2u) {
                        v[i ? i - 1 : 0] = v[i];
                        v[i] = y;
                    } else {
                        bad = true;
                    }
                }
            }
        }
    }
    // (a swap changes no value that another thread compares by more than its
    // position, and those it does belong to a longer run)
    if (g.any(bad)) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) sm.val[t * ITEMS + i] = v[i];
        g.sync();
        const uint32_t run = group_fix_runs<G, ITEMS>(g, sm, len);
        if (run) {
            full = run == 2;
            z.byte_of = SEG_TIE;  // the values are positions only
            // The differing bits not used: m0, m1 of the window, and what
            // lies past the window's 64 bits.
            const uint32_t f = z.f;
            const uint64_t m = (uint64_t)z.m0 << 32 | z.m1;
            const uint64_t rh = f < 64 ? m >> f : 0ull;
            const uint64_t rl = f == 0   ? ml
                                : f < 64 ? (m << (64 - f)) | ((ml << f) >> f)
                                         : m >> (f - 64);
            group_refine<G, ITEMS>(g, sm, I, len, rh, rl);
        }
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) v[i] = sm.val[t * ITEMS + i];
        if (t) pv = sm.val[t * ITEMS - 1];
        g.sync();
    }
    // The order, with the bytes shared with the neighbour where the first
    // differing squeezed bit tells (no NUL can precede it in either key).
    uint32_t o[ITEMS / 2];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t x = (v[i] ^ (i ? v[i ? i - 1 : 0] : pv)) >> PB;
        const uint32_t l = __shfl_sync(0xffffffffu, z.byte_of, __clz(x) + z.used - 32);
        const uint32_t h = l * (1u << SEG_ORD_BITS) + (v[i] & PM);
        if (i & 1)
            o[i / 2] += h * 65536u;
        else
            o[i / 2] = h;
    }
    if constexpr (ITEMS == 8)
        reinterpret_cast<uint4 *>(sm.val)[t] = make_uint4(o[0], o[1], o[2], o[3]);
    else if constexpr (ITEMS == 4)
        reinterpret_cast<uint2 *>(sm.val)[t] = make_uint2(o[0], o[1]);
    else
        sm.val[t] = o[0];
    return full;
}

// Sorts segment s (at most 8 strings per thread) with a group of threads.
// Returns whether a run of more than SEG_FULL tied records was out of order.
// One warp orders up to 64 or 128 strings with 2 or 4 per thread.
template <class G>
__device__ __forceinline__ bool sort_segment(const G &g, const SortArgs &a, const Seg &s,
                                             const SegMem &sm, Seg *N, Counters *c) {
    const uint32_t t = g.t, GT = g.threads();
    constexpr int GRP = 4;  // strings at a time
    const uint32_t lane = t & 31, gw = t >> 5;
    const int b = s.flags & SEG_BUF1;
    const uint32_t *I = a.idxb(b) + s.start;
    // Records into shared memory: asynchronous copies of the partition's keys
    // (no registers, all in flight at once), or the strings' own bytes through
    // index and offset.
    if (s.flags & SEG_KEYS) {
        const ulonglong2 *K = a.keyb(b) + s.start;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const uint32_t e = q * g.threads() + t;
            if (e < s.len) {
                cp_async16(sm.key + e, K + e);
                cp_async4(sm.idx + e, I + e);
            }
        }
        cp_async_commit();
        cp_async_wait<0>();
    } else {
#pragma unroll 1
        for (uint32_t e0 = t; e0 < s.len; e0 += GRP * GT) {
            Key k[GRP];
            uint32_t id[GRP];
            gather_keys<GRP>(a, I, s.depth, e0, GT, s.len, k, id);
#pragma unroll
            for (int q = 0; q < GRP; ++q)
                if (e0 + q * GT < s.len) {
                    sm.key[e0 + q * GT] = from_key(k[q]);
                    sm.idx[e0 + q * GT] = id[q];
                }
        }
    }
    g.sync();
    // The bits in which the keys differ.
    uint64_t mh = 0, ml = 0;
    {
        const Key k0 = to_key(sm.key[0]);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const uint32_t e = q * g.threads() + t;
            if (e < s.len) {
                const Key k = to_key(sm.key[e]);
                mh |= k.hi ^ k0.hi;
                ml |= k.lo ^ k0.lo;
            }
        }
        mh = warp_or64(mh);
        ml = warp_or64(ml);
        if constexpr (!G::warp) {
            if (lane == 0) {
                sm.red[2 * gw] = mh;
                sm.red[2 * gw + 1] = ml;
            }
            g.sync();
            for (uint32_t q = 0; q < GT / 32; ++q) {
                mh |= sm.red[2 * q];
                ml |= sm.red[2 * q + 1];
            }
        }
    }
    bool full = false;
    if (mh | ml) {
        if (G::warp && s.len <= 64)
            full = order_segment<G, G::warp ? 2 : 8>(g, sm, I, s.len, mh, ml);
        else if (G::warp && s.len <= 128)
            full = order_segment<G, G::warp ? 4 : 8>(g, sm, I, s.len, mh, ml);
        else
            full = order_segment<G, 8>(g, sm, I, s.len, mh, ml);
    } else {  // all keys equal: position order
        for (uint32_t e = t; e < s.len; e += GT)
            reinterpret_cast<uint16_t *>(sm.val)[e] = (uint16_t)(SEG_TIE << SEG_ORD_BITS | e);
    }
    g.sync();
    // Results in rank order: indices, LCPs, first and last key, next-round
    // runs.  Ties read both keys.
    const uint16_t *ord = reinterpret_cast<const uint16_t *>(sm.val);
    constexpr uint32_t OM = (1u << SEG_ORD_BITS) - 1;
    auto key_at = [&](uint32_t r) -> Key { return to_key(sm.key[ord[r] & OM]); };
    uint32_t *oi = a.idx[0] + s.start + t, *ol = a.lcp + s.start + t;
    if (t < 2) {
        const uint32_t r = t ? s.len - 1 : 0;
        a.key[0][s.start + r] = from_key(key_at(r));
    }
#pragma unroll 4
    for (uint32_t e0 = 0; e0 < s.len; e0 += GT) {
        const uint32_t e = e0 + t;
        const bool on = e < s.len;
        const uint32_t w = on ? ord[e] : 0u;
        if (on) oi[e0] = sm.idx[w & OM];
        bool cont = false;  // goes on a run of equal keys that do not end
        if (on && e) {
            uint32_t l = w >> SEG_ORD_BITS;
            if (l == SEG_TIE) {
                const Key k = to_key(sm.key[w & OM]), kp = key_at(e - 1);
                const bool same = key_eq(kp, k);
                cont = same && !key_is_end(k);
                l = same ? key_len(k) : key_lcp(kp, k);
            }
            if (!cont) ol[e0] = s.depth + l;
        }
        const uint32_t cm = __ballot_sync(0xffffffffu, cont);
        if (cm) {  // warp-uniform
            bool tail = cont && !((cm >> 1) >> lane & 1u);
            if (tail && lane == 31 && e + 1 < s.len) tail = !key_eq(key_at(e + 1), key_at(e));
            uint32_t lo = 0;
            if (tail) {
                const uint32_t heads = ~cm & lanemask_lt();
                if (heads) {
                    lo = e - lane + 31 - __clz(heads);
                } else {  // the run starts before this warp's ranks
                    const Key k = key_at(e);
                    uint32_t hi = e;
                    while (lo < hi) {
                        const uint32_t mid = (lo + hi) >> 1;
                        if (key_lt(key_at(mid), k))
                            lo = mid + 1;
                        else
                            hi = mid;
                    }
                }
            }
            emit_next_warp(N, c, tail, s.start + lo, e - lo + 1, s.depth + KEY_BYTES);
        }
    }
    g.sync();
    return full;
}

// Sorts segments lo + g, g = first, first + step, .. < nT of list T with the
// thread group grp.
template <class G>
__device__ __forceinline__ void sort_list(const G &grp, const SortArgs &a,
                                          const Seg *T, uint32_t nT, uint32_t first,
                                          uint32_t step, const SegMem &sm, Seg *N, Counters *c) {
    unsigned long long fresh = 0, keyed = 0, full = 0;
    for (uint32_t g = first; g < nT; g += step) {
        const Seg s = T[g];
        if (s.flags & SEG_KEYS)
            keyed += s.len;
        else
            fresh += s.len;
        if (sort_segment(grp, a, s, sm, N, c)) full += s.len;
    }
    if (grp.t == 0 && (fresh | keyed)) {
        atomicAdd(G::warp ? &c->warp8_fresh : &c->block_fresh, fresh);
        atomicAdd(G::warp ? &c->warp8_keyed : &c->block_keyed, keyed);
        if (full) atomicAdd(&c->full_sorted, full);
    }
}

// Segments of 33..256 strings: one warp each.
constexpr size_t WARPSORT_SMEM = SMALL_THREADS / 32 * seg_bytes(32);

__global__ void __launch_bounds__(SMALL_THREADS, 4)
    k_warpsort(SortArgs a, const Seg *T0, Span sp, Seg *N, Counters *c) {
    after_predecessor();
    extern __shared__ __align__(16) unsigned char seg_smem[];
    const uint32_t lo = count_of(sp.lo), w = threadIdx.x / 32, per = SMALL_THREADS / 32;
    sort_list(WarpGroup{threadIdx.x & 31}, a, T0 + lo, count_of(sp.hi) - lo, blockIdx.x * per + w,
              gridDim.x * per, seg_mem(seg_smem + w * seg_bytes(32), 32), N, c);
}

// Classes with few segments, in one launch: class k's segments (up to 512 << k
// strings, 64 << k threads each) are taken by CTAs cta[k] .. cta[k + 1] - 1 of
// SEG_CTA threads, 8 >> k segments side by side.  Such a launch spends most of
// its time fetching instructions, which the classes share here, and a level's
// classes run side by side: 3 M URLs 1.08 -> 0.94 ms, 200 small instances 201
// -> 171 us.
constexpr int SEG_CTA = 512;
constexpr size_t SEG_SMEM = SEG_CTA / 64 * seg_bytes(64);
static_assert(SEG_SMEM >= seg_bytes(512) && SEG_SMEM >= 2 * seg_bytes(256), "group slots");

__global__ void __launch_bounds__(SEG_CTA, 2)
    k_segsort(SortArgs a, SmallWork wk, Seg *N, Counters *c) {
    after_predecessor();
    extern __shared__ __align__(16) unsigned char seg_smem[];
    uint32_t k = 0;
    while (k + 1 < SMALL_CLASSES && blockIdx.x >= wk.cta[k + 1]) ++k;
    const uint32_t log2_threads = 6 + k, per = SEG_CTA >> log2_threads;
    const uint32_t lo = count_of(wk.span[k].lo), nT = count_of(wk.span[k].hi) - lo;
    const Seg *T = wk.list.s[k] + lo;
    const uint32_t gi = threadIdx.x >> log2_threads;
    const CtaGroup<> grp{threadIdx.x & ((1u << log2_threads) - 1), log2_threads, 1 + gi};
    const SegMem sm = seg_mem(seg_smem + gi * seg_bytes(grp.threads()), grp.threads());
    sort_list(grp, a, T, nT, (blockIdx.x - wk.cta[k]) * per + gi,
              (wk.cta[k + 1] - wk.cta[k]) * per, sm, N, c);
}

// A class with many segments: its group size is a constant (fewer
// instructions: 69 M batched strings 5.80 -> 5.53 ms against the shared
// launch).  CTAs of 512 threads, although four of 256 per SM sort alone
// faster (5.40 ms): these sorts run beside the partition, whose CTAs have 512
// threads and whose next kernel waits for room on every SM; small CTAs keep
// filling each half that comes free (50 M URLs 7.33 ms with 512, 7.86 with
// 256).
template <int K>
constexpr size_t CLASS_SMEM = SEG_CTA / (64 << K) * seg_bytes(64 << K);

template <int K>
__global__ void __launch_bounds__(SEG_CTA, 2)
    k_segsort_class(SortArgs a, const Seg *T0, Span sp, Seg *N, Counters *c) {
    after_predecessor();
    extern __shared__ __align__(16) unsigned char seg_smem[];
    constexpr uint32_t GT = 64u << K, per = SEG_CTA / GT;
    const uint32_t lo = count_of(sp.lo), gi = threadIdx.x / GT;
    const CtaGroup<6 + K> grp{threadIdx.x % GT, 6 + K, 1 + gi};
    sort_list(grp, a, T0 + lo, count_of(sp.hi) - lo, blockIdx.x * per + gi, gridDim.x * per,
              seg_mem(seg_smem + gi * seg_bytes(GT), GT), N, c);
}

// ---- equality buckets: work items of up to EQ_TILE strings ------------------
// Bound by memory (12 bytes per string).  A thread's four reads go out before
// its stores, which the compiler may not pass: 3 M URLs 61 -> 40 us, 100 M
// words 237 -> 231 us (4.4 TB/s); eight in flight 262.
__global__ void k_equal(SortArgs a, const Seg *E0, Span sp, Seg *N, Counters *c) {
    after_predecessor();
    const uint32_t lo = count_of(sp.lo);
    const Seg *E = E0 + lo;
    const uint32_t nE = count_of(sp.hi) - lo;
    unsigned long long moved = 0, fin = 0;
    for (uint32_t g = blockIdx.x; g < nE; g += gridDim.x) {
        const Seg s = E[g];
        const int b = s.flags & SEG_BUF1;
        const uint32_t ch = s.flags >> SEG_CHUNK_SHIFT;
        const Key k = to_key(a.keyb(b)[s.start]);
        const bool end = key_is_end(k);
        if (ch == 0 && threadIdx.x == 0) {
            a.key[0][s.start] = from_key(k);
            a.key[0][s.start + s.len - 1] = from_key(k);
            if (!end) emit_next(N, c, s.start, s.len, s.depth + KEY_BYTES);
        }
        const uint32_t lo = ch * EQ_TILE;
        const uint32_t hi = min(lo + (uint32_t)EQ_TILE, s.len);
        if (threadIdx.x == 0) {
            if (b) moved += hi - lo;
            if (end) fin += hi - lo;
        }
        const uint32_t l = s.depth + key_len(k);
        constexpr uint32_t U = 4;  // indices in flight per thread
        for (uint32_t i0 = lo + threadIdx.x; i0 < hi; i0 += U * blockDim.x) {
            uint32_t id[U];
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t i = i0 + u * blockDim.x;
                if (b && i < hi) id[u] = a.idx[1][s.start + i];
            }
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t i = i0 + u * blockDim.x;
                if (b && i < hi) a.idx[0][s.start + i] = id[u];
                if (end && i > 0 && i < hi) a.lcp[s.start + i] = l;
            }
        }
    }
    if (threadIdx.x == 0 && (moved | fin)) {
        atomicAdd(&c->equal_moved, moved);
        atomicAdd(&c->equal_final, fin);
    }
}

__device__ __forceinline__ void boundary_lcps(const SortArgs &a, const uint2 *B,
                                              uint32_t nB) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nB; i += gridDim.x * blockDim.x) {
        const uint2 e = B[i];
        a.lcp[e.x] = e.y + key_lcp(to_key(a.key[0][e.x - 1]), to_key(a.key[0][e.x]));
    }
}

__global__ void k_boundary(SortArgs a, const uint2 *__restrict__ B, Counters *c) {
    boundary_lcps(a, B, c->n_bound);
}

// End of a round whose next round follows at once: one launch and one host
// round trip for the boundary LCPs and the next round's classification.  The
// finished round's counters are cleared for the round after the next.
__global__ void k_round_end(SortArgs a, const uint2 *B, const Seg *N,
                            Seg *W1, Seg *W8, SmallLists S, Seg *L, RoundCounters *rc, int i,
                            Publish pub) {
    after_predecessor();
    const Counters *old = rc->c + i;
    boundary_lcps(a, B, old->n_bound);
    classify_list(N, old->n_next, a.warp8_cap, W1, W8, S, L, rc->c + (i ^ 1));
    if (publish(pub, rc)) {
        uint32_t *w = reinterpret_cast<uint32_t *>(rc->c + i);
        for (uint32_t q = threadIdx.x; q < sizeof(Counters) / 4; q += blockDim.x) w[q] = 0;
    }
}

// ---- a whole small sort in one CTA -----------------------------------------
// At most SMALL_CAP strings need no partition: one CTA sorts them, then keeps
// refining the runs of equal keys round by round, with the code of the
// on-chip sorts (the whole CTA on segments of more than 256 strings, a warp on
// each smaller one).  What the rounds of the general loop cost such a sort is
// launches and host round trips: 500 words took 134 us, now 39.  A round with
// more segments than TINY_SEGMENTS (which the general loop spreads over the
// chip), or the TINY_ROUNDS-th, is left to the general loop.
// So are many runs that stay equal for long: in-warp refinement takes about
// 4 us per 16 bytes and run, and this CTA's eight warps take the runs in turn.
// A round whose runs of at most 32 strings are more than the warps gets
// TINY_STEPS steps in all, and where the next one is as crowded that is left to
// the general loop: by then this CTA has spent about what a round of that loop
// costs.  16 strings in each of 128 groups, sharing 1000, 100, 40 bytes: 1047,
// 189, 127 us; the general loop from the start 1074, 223, 164; without a limit
// 3784, 378, 139.  With TINY_STEPS 128: 1105, 236, 138; leaving every crowded
// round at once: 1030, 170, 110, but 500 URLs 89 us instead of 57.
constexpr uint32_t TINY_SEGMENTS = 128;
constexpr uint32_t TINY_STEPS = 64;
constexpr size_t TINY_SMEM =
    seg_bytes(SMALL_THREADS) > WARPSORT_SMEM ? seg_bytes(SMALL_THREADS) : WARPSORT_SMEM;

__global__ void __launch_bounds__(SMALL_THREADS, 1)
    k_tiny(SortArgs a, Seg *A, Seg *B, RoundCounters *rc, Publish pub) {
    extern __shared__ __align__(16) unsigned char seg_smem[];
    __shared__ unsigned long long sums;
    const uint32_t t = threadIdx.x, lane = t & 31, w = t >> 5;
    Counters *c = rc->c;
    {
        uint32_t *z = reinterpret_cast<uint32_t *>(rc);
        for (uint32_t i = t; i < sizeof(RoundCounters) / 4; i += SMALL_THREADS) z[i] = 0;
    }
    for (uint32_t i = t; i < a.n; i += SMALL_THREADS) a.idx[0][i] = i;
    if (t == 0) {
        a.lcp[0] = 0;
        A[0] = Seg{0, a.n, 0, 0};
    }
    __syncthreads();
    uint32_t n_cur = 1, round = 0, segments = 0;
    bool crowded = false;
    for (; round < TINY_ROUNDS && n_cur && n_cur <= TINY_SEGMENTS; ++round) {
        if (t == 0) {
            sums = 0;
            c->n_next = 0;
        }
        __syncthreads();
        const Seg own = t < n_cur ? A[t] : Seg{0, 0, 0, 0};
        // live strings, segments of 9..32 strings, segments of up to 8
        const bool few = own.len && own.len <= W1_SMALL;
        const bool one = own.len > W1_SMALL && own.len <= (uint32_t)WARP1_CAP;
        const unsigned long long sum =
            warp_sum(own.len | (unsigned long long)one << 32 | (unsigned long long)few << 48);
        if (lane == 0 && sum) atomicAdd(&sums, sum);
        const bool any_large = __syncthreads_or(own.len > (uint32_t)WARP8_CAP);
        const uint32_t live = (uint32_t)sums, n_few = (uint32_t)(sums >> 48);
        const uint32_t tasks =
            ((uint32_t)(sums >> 32) & 0xFFFFu) + (n_few + W1_PACK - 1) / W1_PACK;
        const bool again = crowded;
        crowded = tasks > SMALL_THREADS / 32;
        if (crowded && again) break;
        const uint32_t steps = crowded ? min(a.warp1_deep, TINY_STEPS / tasks) : a.warp1_deep;
        if (any_large) {
            for (uint32_t g = 0; g < n_cur; ++g) {
                const Seg s = A[g];
                if (s.len <= (uint32_t)WARP8_CAP) continue;
                const bool full = sort_segment(CtaGroup<8>{t, 8, 1}, a, s,
                                               seg_mem(seg_smem, SMALL_THREADS), B, c);
                if (t == 0) {
                    c->block_fresh += s.len;
                    if (full) c->full_sorted += s.len;
                }
            }
            __syncthreads();
        }
        unsigned long long deep = 0, fresh = 0;
        // As in k_warp1: up to W1_PACK segments of at most 8 strings together.
        for (uint32_t g0 = w * W1_PACK; n_few && g0 < n_cur;
             g0 += SMALL_THREADS / 32 * W1_PACK) {
            const uint32_t j = lane >> 3;
            Seg s = g0 + j < n_cur ? A[g0 + j] : Seg{0, 0, 0, 0};
            if (s.len > W1_SMALL) s.len = 0;
            if ((lane & 7) == 0) fresh += s.len;
            if (__any_sync(0xffffffffu, s.len > 0)) deep += warp1_group<8>(a, s, lane, steps, B, c);
        }
        for (uint32_t g = w; g < n_cur; g += SMALL_THREADS / 32) {
            const Seg s = A[g];
            if (s.len <= W1_SMALL || s.len > (uint32_t)WARP8_CAP) continue;
            if (s.len <= (uint32_t)WARP1_CAP) {
                deep += warp1_group<32>(a, s, lane, steps, B, c);
                if (lane == 0) fresh += s.len;
            } else {
                const bool full = sort_segment(WarpGroup{lane}, a, s,
                                               seg_mem(seg_smem + w * seg_bytes(32), 32), B, c);
                if (lane == 0) {
                    atomicAdd(&c->warp8_fresh, (unsigned long long)s.len);
                    if (full) atomicAdd(&c->full_sorted, (unsigned long long)s.len);
                }
            }
        }
        if (fresh) atomicAdd(&c->warp1_fresh, fresh);
        deep = warp_sum(deep);
        if (lane == 0 && deep) atomicAdd(&c->warp1_deep, deep);
        __syncthreads();
        if (t == 0) rc->tiny_live[round] = live;
        segments += n_cur;
        n_cur = atomicAdd(&c->n_next, 0u);
        Seg *x = A;
        A = B;
        B = x;
        __syncthreads();
    }
    if (t == 0) {
        rc->tiny_rounds = round;
        rc->tiny_segments = segments;
        rc->tiny_left = n_cur;
    }
    publish(pub, rc);
}

// ---- control kernels of the device-driven round loop --------------------------
// The graph's loops (rounds, partition levels) and branches (separate gather,
// gathering count) are CUDA graph conditional nodes; these kernels read the
// device counters and set their conditions, so no host round trip is needed
// between launches.  None of them waits on another block: the multi-CTA ones
// copy a list and let the last CTA to finish (atomic ticket) do the update.

// Each loop body first clears its own condition, and only the kernel that
// ends the body sets it again when another iteration is due: a body whose
// last kernel did not run cannot repeat.
__global__ void k_g_round_begin(GraphState *g, Counters *c, cudaGraphConditionalHandle h_round) {
    uint32_t *w = reinterpret_cast<uint32_t *>(c);
    for (uint32_t i = threadIdx.x; i < sizeof(Counters) / 4; i += blockDim.x) w[i] = 0;
    if (threadIdx.x == 0) {
        cudaGraphSetConditional(h_round, 0u);
        g->cur_w1 = g->cur_w8 = g->cur_e = 0;
        for (uint32_t &s : g->cur_s) s = 0;
        g->levels = 0;
    }
}

__global__ void k_g_after_classify(GraphState *g, const Counters *c,
                                   cudaGraphConditionalHandle h_level,
                                   cudaGraphConditionalHandle h_gather) {
    if (threadIdx.x != 0) return;
    const uint32_t nl = c->n_large;
    g->n_large = nl;
    g->levels = 0;
    if (g->round < 64) g->live[g->round] = c->live_next;
    const bool fused = gather_fused(g->fused, g->round == 0, c->gather_elems);
    g->fused_round = fused ? 1u : 0u;
    g->first = fused ? 1u : 0u;
    cudaGraphSetConditional(h_gather, (nl > 0 && !fused) ? 1u : 0u);
    cudaGraphSetConditional(h_level, nl > 0 ? 1u : 0u);
}

__global__ void k_g_level_begin(const GraphState *g, cudaGraphConditionalHandle h_level,
                                cudaGraphConditionalHandle h_first) {
    if (threadIdx.x != 0) return;
    cudaGraphSetConditional(h_level, 0u);
    cudaGraphSetConditional(h_first, g->first ? 1u : 0u);
}

// True in thread 0 of the last CTA of the grid to get here (after its own
// writes are visible); that CTA resets the ticket for the next launch.
__device__ __forceinline__ bool last_cta(uint32_t *ticket) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last || threadIdx.x != 0) return false;
    __threadfence();
    *ticket = 0;
    return true;
}

__global__ void k_g_level_end(GraphState *g, Counters *c, Seg *L, const Seg *__restrict__ L2,
                              cudaGraphConditionalHandle h_level) {
    const uint32_t n = c->n_large_next;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        L[i] = L2[i];
    if (!last_cta(&g->ticket)) return;
    g->n_large = n;
    c->n_large_next = 0;
    g->first = 0;
    g->levels += 1;
    g->partition_levels += 1;
    g->cur_w1 = c->n_w1;
    g->cur_w8 = c->n_w8;
    g->cur_s[0] = c->n_small;
    g->cur_s[1] = c->n_small2;
    g->cur_s[2] = c->n_small3;
    g->cur_s[3] = c->n_small4;
    g->cur_e = c->n_equal;
    bool more = n > 0;
    if (more && g->levels >= g->max_levels) {
        g->error = 1;  // reported by the host as an internal error, not a hang
        more = false;
    }
    cudaGraphSetConditional(h_level, more ? 1u : 0u);
}

__global__ void k_g_round_end(GraphState *g, const Counters *c, Seg *R, const Seg *__restrict__ N,
                              cudaGraphConditionalHandle h_round) {
    const uint32_t n = c->n_next;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        R[i] = N[i];
    if (!last_cta(&g->ticket)) return;
    const bool fused = g->fused_round != 0;
    g->small_segments += (unsigned long long)c->n_w1 + c->n_w8 + c->n_small + c->n_small2 +
                         c->n_small3 + c->n_small4;
    g->partitioned += c->partitioned;
    g->gather_elems += c->gather_elems;
    if (fused) g->gather_fused += c->gather_elems;
    g->warp1_fresh += c->warp1_fresh;
    g->warp1_keyed += c->warp1_keyed;
    g->warp8_fresh += c->warp8_fresh;
    g->warp8_keyed += c->warp8_keyed;
    g->block_fresh += c->block_fresh;
    g->block_keyed += c->block_keyed;
    g->equal_moved += c->equal_moved;
    g->equal_final += c->equal_final;
    g->boundaries += c->n_bound;
    g->warp1_deep += c->warp1_deep;
    g->full_sorted += c->full_sorted;
    g->window_saved += c->window_saved;
    g->window_used += c->window_used;
    if (c->error) g->error = 2;  // a scan's look-back waited past its bound
    g->n_cur = n;
    g->round += 1;
    g->round_in_launch += 1;
    g->done = n == 0 ? 1u : 0u;
    const bool more = n > 0 && !g->error && g->round_in_launch < GRAPH_ROUNDS_PER_LAUNCH;
    cudaGraphSetConditional(h_round, more ? 1u : 0u);
}

// ---- exclusive scan (u32), one pass with decoupled look-back ---------------
// A CTA takes tiles from a ticket until none is left (a tile is published
// before its CTA takes another, so every tile it waits for has started and
// waits for nothing newer; the host knows only a bound of n, and one CTA per
// tile of that bound took 10 us to find nothing), scans its 4096 values, publishes its sum, and warp 0 walks back
// over its predecessors' status words 32 at a time, adding sums until it
// meets an inclusive prefix; then it publishes its own inclusive prefix.
// Status word: flag (1 = tile sum, 2 = inclusive prefix) << 32 | value.  The
// wait for a predecessor is bounded; past the bound the CTA records an
// error and goes on (the host reports it; the result is then not used).
constexpr uint64_t LB_SUM = 1ull << 32, LB_INCL = 2ull << 32;
constexpr uint32_t LB_SPIN_MAX = 1u << 22;

__device__ __forceinline__ uint32_t warp_sum32(uint32_t v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

__global__ void __launch_bounds__(SCAN_THREADS) k_scan_lookback(const uint32_t *in, uint32_t *out,
                                                                Count cnt,
                                                                unsigned long long *status,
                                                                uint32_t *ticket, uint32_t *err) {
    after_predecessor();
    __shared__ uint32_t buf[SCAN_CHUNK];
    __shared__ uint32_t s_tile, s_prefix;
    const uint32_t n = count_of(cnt);
    const uint32_t lane = threadIdx.x & 31;
    if (n == 0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) out[0] = 0;
        return;
    }
    while (true) {
    if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t t = s_tile;
    const uint64_t base = (uint64_t)t * SCAN_CHUNK;
    if (base >= n) return;
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const int j = k * SCAN_THREADS + threadIdx.x;
        const uint64_t i = base + j;
        buf[j] = i < n ? in[i] : 0;
    }
    __syncthreads();
    uint32_t s = 0;
    for (int k = 0; k < SCAN_ITEMS; ++k) s += buf[threadIdx.x * SCAN_ITEMS + k];
    uint32_t excl;
    const uint32_t total = block_exclusive_scan(s, excl);
    if (threadIdx.x < 32) {
        uint32_t prefix = 0;
        if (t == 0) {
            if (lane == 0) atomicExch(&status[0], LB_INCL | total);
        } else {
            if (lane == 0) atomicExch(&status[t], LB_SUM | total);
            int64_t j = (int64_t)t - 1;  // nearest predecessor not yet added
            uint32_t spins = 0;
            bool failed = false;
            while (true) {
                const int64_t idx = j - (int64_t)lane;
                const volatile unsigned long long *sp = status + (idx >= 0 ? idx : 0);
                unsigned long long w = idx >= 0 ? *sp : LB_INCL;
                while (__any_sync(0xffffffffu, (w >> 32) == 0)) {
                    if (++spins > LB_SPIN_MAX) {
                        failed = true;
                        break;
                    }
                    __nanosleep(32);
                    if ((w >> 32) == 0) w = *sp;
                }
                if (failed) break;
                const uint32_t incl = __ballot_sync(0xffffffffu, (w >> 32) == 2);
                if (incl) {
                    const uint32_t k = __ffs(incl) - 1;  // the nearest inclusive prefix
                    prefix += warp_sum32(lane <= k ? (uint32_t)w : 0u);
                    break;
                }
                prefix += warp_sum32((uint32_t)w);
                j -= 32;
            }
            if (lane == 0) {
                if (failed) atomicExch(err, 1u);
                atomicExch(&status[t], LB_INCL | (prefix + total));
            }
        }
        if (lane == 0) s_prefix = prefix;
    }
    __syncthreads();
    uint32_t run = s_prefix + excl;
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const int j = threadIdx.x * SCAN_ITEMS + k;
        const uint32_t v = buf[j];
        buf[j] = run;
        run += v;
    }
    __syncthreads();
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        const int j = k * SCAN_THREADS + threadIdx.x;
        const uint64_t i = base + j;
        if (i < n) out[i] = buf[j];
    }
    if (threadIdx.x == 0 && base + SCAN_CHUNK >= n) out[n] = s_prefix + total;
    __syncthreads();  // shared memory is reused by the CTA's next tile
    }
}

}  // namespace

// ---- launchers --------------------------------------------------------------
static inline uint32_t cdiv(uint64_t a, uint64_t b) { return (uint32_t)((a + b - 1) / b); }

// Launch of a kernel that starts with after_predecessor().
template <class... P, class... Q>
static void launch_next(void (*kernel)(P...), uint32_t grid, uint32_t threads, size_t smem,
                        cudaStream_t st, const Q &...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    // (a failure stays the thread's last error, which every caller checks)
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Opt-in to more than 48 KB of dynamic shared memory for the kernels that use
// it.  The attribute belongs to the function in the current device's context,
// so it is set once per device (bit d of the mask), for all kernels at once;
// two threads that race here both set the same values, which is harmless.
static void set_smem_attrs() {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return;  // the launch reports it
    const uint64_t bit = dev < 64 ? 1ull << dev : 0ull;
    if (bit && (done.load(std::memory_order_acquire) & bit)) return;
    cudaFuncSetAttribute(k_sample, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(SampleSmem));
    cudaFuncSetAttribute(k_count<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(PartSmem));
    cudaFuncSetAttribute(k_count<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(PartSmem));
    cudaFuncSetAttribute(k_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(ScatterSmem));
    cudaFuncSetAttribute(k_tiny, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TINY_SMEM);
    cudaFuncSetAttribute(k_warpsort, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)WARPSORT_SMEM);
    cudaFuncSetAttribute(k_segsort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SEG_SMEM);
    cudaFuncSetAttribute(k_segsort_class<0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)CLASS_SMEM<0>);
    cudaFuncSetAttribute(k_segsort_class<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)CLASS_SMEM<1>);
    cudaFuncSetAttribute(k_segsort_class<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)CLASS_SMEM<2>);
    cudaFuncSetAttribute(k_segsort_class<3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)CLASS_SMEM<3>);
    done.fetch_or(bit, std::memory_order_release);
}

void launch_iota(uint32_t *idx, uint32_t n, cudaStream_t st) {
    const uint32_t g = cdiv(n, 256) < 148 * 16 ? cdiv(n, 256) : 148 * 16;
    k_iota<<<g ? g : 1, 256, 0, st>>>(idx, n);
}

// Grid for a launcher given `grid` (> 0: as given) or a host count of work
// units of `per` each (capped at cap CTAs; 0 when there is no work).
static int grid_of(int grid, const Count &n, uint32_t per, uint32_t cap) {
    if (grid > 0) return grid;
    if (n.dev) return (int)cap;
    const uint32_t g = cdiv(n.host, per);
    return (int)(g < cap ? g : cap);
}

void launch_begin(uint32_t *idx, uint32_t n_idx, uint32_t *lcp, RoundCounters *rc, Seg first,
                  Seg *list, uint32_t *count, cudaStream_t st) {
    const uint32_t g = cdiv(n_idx, 256) < 148 * 16 ? cdiv(n_idx, 256) : 148 * 16;
    k_begin<<<g ? g : 1, 256, 0, st>>>(idx, n_idx, lcp, rc, first, list, count);
}

void launch_tiny(const SortArgs &a, Seg *A, Seg *B, RoundCounters *rc, Publish pub,
                 cudaStream_t st) {
    set_smem_attrs();
    k_tiny<<<1, SMALL_THREADS, TINY_SMEM, st>>>(a, A, B, rc, pub);
}

void launch_classify(const Seg *R, Count nR, uint32_t warp8_cap, Seg *W1, Seg *W8,
                     SmallLists S, Seg *L, Counters *c, int grid, cudaStream_t st,
                     RoundCounters *rc, Publish pub) {
    const int g = grid_of(grid, nR, 256, 1u << 30);
    if (!g) return;
    k_classify<<<g, 256, 0, st>>>(R, nR, warp8_cap, W1, W8, S, L, c, rc, pub);
}

void launch_round_end(const SortArgs &a, const uint2 *B, const Seg *N, Seg *W1, Seg *W8,
                      SmallLists S, Seg *L, RoundCounters *rc, int i, Publish pub, int grid,
                      cudaStream_t st) {
    launch_next(k_round_end, grid, 256, 0, st, a, B, N, W1, W8, S, L, rc, i, pub);
}

void launch_init_batch(const uint32_t *inst_start, uint32_t ninst, Seg *R, uint32_t *lcp,
                       Counters *c, cudaStream_t st) {
    if (!ninst) return;
    k_init_batch<<<cdiv(ninst, 256), 256, 0, st>>>(inst_start, ninst, R, lcp, c);
}

void launch_localize(uint32_t *perm, uint32_t n, const uint32_t *inst_start, uint32_t ninst,
                     cudaStream_t st) {
    const uint32_t g = cdiv(n, 256) < 148 * 8 ? cdiv(n, 256) : 148 * 8;
    k_localize<<<g ? g : 1, 256, 0, st>>>(perm, n, inst_start, ninst);
}

void launch_copies(const CopyJob *jobs, uint32_t njobs, uint32_t chunks, cudaStream_t st) {
    if (njobs && chunks) k_copies<<<chunks, 512, 0, st>>>(jobs, njobs);
}

void launch_join(uint64_t *goffs, uint32_t *lcp, uint32_t *perm, const ReqJob *jobs,
                 uint32_t njobs, uint32_t total, Seg *R, cudaStream_t st) {
    if (!njobs || !total) return;
    const uint32_t g = cdiv(total, 256) < 148 * 8 ? cdiv(total, 256) : 148 * 8;
    k_join<<<g, 256, 0, st>>>(goffs, lcp, perm, jobs, njobs, total, R);
}

void launch_mark(const Seg *R, uint32_t nR, const uint32_t *base, uint32_t nact, uint32_t *flag,
                 cudaStream_t st) {
    if (!nR || !nact) return;
    const uint32_t g = cdiv(nR, 256) < 148 * 8 ? cdiv(nR, 256) : 148 * 8;
    k_mark<<<g, 256, 0, st>>>(R, nR, base, nact, flag);
}

void launch_unbase(uint32_t *perm, const ReqJob *jobs, uint32_t njobs, uint32_t total,
                   cudaStream_t st) {
    if (!njobs || !total) return;
    const uint32_t g = cdiv(total, 256) < 148 * 8 ? cdiv(total, 256) : 148 * 8;
    k_unbase<<<g, 256, 0, st>>>(perm, jobs, njobs, total);
}

uint64_t text_tiles(uint64_t len) { return (len + TEXT_TILE - 1) / TEXT_TILE; }

void launch_text_count(const uint8_t *text, uint64_t len, uint8_t delim, uint32_t *tile_cnt,
                       unsigned long long *total, cudaStream_t st) {
    const uint64_t t = text_tiles(len);
    if (t) k_text_count<<<(unsigned)t, TEXT_THREADS, 0, st>>>(text, len, delim, tile_cnt, total);
}

void launch_text_starts(uint8_t *text, uint64_t len, uint8_t delim, const uint32_t *tile_base,
                        uint64_t n, void *offs, int off_width, cudaStream_t st) {
    const uint64_t t = text_tiles(len);
    if (t)
        k_text_starts<<<(unsigned)t, TEXT_THREADS, 0, st>>>(text, len, delim, tile_base, n, offs,
                                                            off_width);
}

void launch_iota_offs(void *offs, int off_width, uint64_t n, cudaStream_t st) {
    const uint64_t g = (n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16;
    k_iota_offs<<<(unsigned)(g ? g : 1), 256, 0, st>>>(offs, off_width, n);
}

void launch_sorted_offs(const uint32_t *perm, const void *offs, int off_width, uint64_t n,
                        void *out, int out_width, cudaStream_t st) {
    const uint64_t g = (n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16;
    k_sorted_offs<<<(unsigned)(g ? g : 1), 256, 0, st>>>(perm, offs, off_width, n, out,
                                                         out_width);
}

void launch_byte_hist(const uint8_t *arena, uint64_t arena_bytes, const void *offs, int off_width,
                      uint32_t n, uint32_t samples, uint32_t *hist, cudaStream_t st) {
    k_byte_hist<<<1, 256, 0, st>>>(arena, arena_bytes, offs, off_width, n, samples, hist);
}

void launch_seg_tiles(const Seg *segs, Count n, uint32_t tile, uint32_t *out, cudaStream_t st) {
    launch_next(k_seg_tiles, 1, SMALL_SCAN_THREADS, 0, st, segs, n, tile, out);
}

uint32_t scan_partials_needed(uint32_t n) { return cdiv(n ? n : 1, SCAN_CHUNK) + 1; }

void launch_scan_lookback(const uint32_t *in, uint32_t *out, uint32_t cap, Count n,
                          unsigned char *state, uint32_t *err, cudaStream_t st) {
    const uint32_t nb = std::min<uint32_t>(cdiv(cap ? cap : 1, SCAN_CHUNK), 148 * 8);
    launch_next(k_scan_lookback, nb, SCAN_THREADS, 0, st, in, out, n, reinterpret_cast<unsigned
                long long *>(state + 8), reinterpret_cast<uint32_t *>(state), err);
}

void launch_scan(const uint32_t *in, uint32_t *out, uint32_t cap, Count n, uint32_t *partials,
                 cudaStream_t st) {
    const uint32_t nb = cdiv(cap ? cap : 1, SCAN_CHUNK);
    k_scan_reduce<<<nb, SCAN_THREADS, 0, st>>>(in, n, partials);
    k_scan_partials<<<1, SCAN_THREADS, 0, st>>>(partials, nb);
    k_scan_down<<<nb, SCAN_THREADS, 0, st>>>(in, out, n, partials, nb);
}

void launch_gather(const SortArgs &a, const Seg *L, Count nL, const uint32_t *tile_base,
                   Counters *c, int grid, cudaStream_t st) {
    if (!nL.dev && !nL.host) return;
    launch_next(a.key2 ? k_gather<true> : k_gather<false>, grid, GATHER_THREADS, 0, st, a, L, nL,
                tile_base, c);
}

void launch_sample(const SortArgs &a, const Seg *L, Count nL, ulonglong2 *spl, uint32_t *nspl,
                   uint16_t *tbl, const LevelBases &lb, bool from_arena, Counters *c, int grid,
                   cudaStream_t st) {
    const int g = grid_of(grid, nL, 1, 1u << 30);
    if (!g) return;
    set_smem_attrs();
    launch_next(k_sample, g, SAMPLE_THREADS, sizeof(SampleSmem), st, a, L, nL, spl, nspl, tbl,
                lb, from_arena, c);
}

void launch_count(const SortArgs &a, const Seg *L, Count nL, const uint32_t *tile_base,
                  const ulonglong2 *spl, const uint32_t *nspl, const uint16_t *tbl,
                  const uint32_t *cm_base, uint32_t *cm, Counters *c, bool gather, int grid,
                  cudaStream_t st) {
    if (!nL.dev && !nL.host) return;
    set_smem_attrs();
    if (gather)
        launch_next(k_count<true>, grid, PART_THREADS, sizeof(PartSmem), st, a, L, nL, tile_base,
                    spl, nspl, tbl, cm_base, cm, c);
    else
        launch_next(k_count<false>, grid / 2 * COUNT_CTAS<false>, PART_THREADS, sizeof(PartSmem),
                    st, a, L, nL, tile_base, spl, nspl, tbl, cm_base, cm, c);
}

void launch_scatter(const SortArgs &a, const Seg *L, Count nL, const uint32_t *tile_base,
                    const uint32_t *nspl, const uint32_t *cm_base, const uint32_t *cm_scan,
                    Counters *c, int grid, cudaStream_t st) {
    if (!nL.dev && !nL.host) return;
    set_smem_attrs();
    launch_next(k_scatter, grid, SCATTER_THREADS, sizeof(ScatterSmem), st, a, L, nL, tile_base,
                nspl, cm_base, cm_scan, c);
}

void launch_emit(const SortArgs &a, const Seg *L, Count nL, const uint32_t *tile_base,
                 const uint32_t *nspl, const uint32_t *cm_base, const uint32_t *cm_scan,
                 Seg *W1, Seg *W8, SmallLists S, Seg *L2, Seg *E, uint2 *B, Seg *N,
                 Counters *c, int grid, cudaStream_t st, RoundCounters *rc, Publish pub) {
    const int g = grid > 0 ? grid : grid_of(grid, nL, 1, 1u << 28) * EMIT_CHUNKS;
    if (!g) return;
    launch_next(k_emit, g, EMIT_THREADS, 0, st, a, L, nL, tile_base, nspl, cm_base, cm_scan, W1,
                W8, S, L2, E, B, N, c, rc, pub);
}

// A span with host bounds and nothing in it launches nothing.
static bool span_empty(const Span &sp) {
    return !sp.lo.dev && !sp.hi.dev && sp.hi.host <= sp.lo.host;
}

void launch_warp1(const SortArgs &a, const Seg *W1, Span sp, Seg *N, Counters *c, int grid,
                  cudaStream_t st) {
    if (span_empty(sp) || grid <= 0) return;
    launch_next(k_warp1, grid, WARP_THREADS, 0, st, a, W1, sp, N, c);
}

void launch_warp8(const SortArgs &a, const Seg *W8, Span sp, Seg *N, Counters *c, int grid,
                  cudaStream_t st) {
    if (span_empty(sp) || grid <= 0) return;
    set_smem_attrs();
    launch_next(k_warpsort, grid, SMALL_THREADS, WARPSORT_SMEM, st, a, W8, sp, N, c);
}

void launch_block(const SortArgs &a, const SmallWork &wk, Seg *N, Counters *c, cudaStream_t st) {
    const uint32_t grid = wk.cta[SMALL_CLASSES];
    if (!grid) return;
    set_smem_attrs();
    launch_next(k_segsort, grid, SEG_CTA, SEG_SMEM, st, a, wk, N, c);
}

template <int K>
static void class_launch(const SortArgs &a, const Seg *S, Span sp, Seg *N, Counters *c,
                         cudaStream_t st) {
    constexpr uint32_t per = SEG_CTA / (64 << K);
    launch_next(k_segsort_class<K>, cdiv(sp.hi.host - sp.lo.host, per), SEG_CTA, CLASS_SMEM<K>,
                st, a, S, sp, N, c);
}

void launch_block_class(const SortArgs &a, const Seg *S, Span sp, int cls, Seg *N, Counters *c,
                        cudaStream_t st) {
    if (span_empty(sp)) return;
    set_smem_attrs();
    if (cls == 0)
        class_launch<0>(a, S, sp, N, c, st);
    else if (cls == 1)
        class_launch<1>(a, S, sp, N, c, st);
    else if (cls == 2)
        class_launch<2>(a, S, sp, N, c, st);
    else
        class_launch<3>(a, S, sp, N, c, st);
}

void launch_equal(const SortArgs &a, const Seg *E, Span sp, Seg *N, Counters *c, int grid,
                  cudaStream_t st) {
    if (span_empty(sp) || grid <= 0) return;
    launch_next(k_equal, grid, 256, 0, st, a, E, sp, N, c);
}

void launch_boundary(const SortArgs &a, const uint2 *B, Counters *c, int grid, cudaStream_t st) {
    k_boundary<<<grid, 256, 0, st>>>(a, B, c);
}

void launch_g_round_begin(GraphState *g, Counters *c, unsigned long long h_round,
                          cudaStream_t st) {
    k_g_round_begin<<<1, 128, 0, st>>>(g, c, (cudaGraphConditionalHandle)h_round);
}

void launch_g_after_classify(GraphState *g, Counters *c, unsigned long long h_level,
                             unsigned long long h_gather, cudaStream_t st) {
    k_g_after_classify<<<1, 32, 0, st>>>(g, c, (cudaGraphConditionalHandle)h_level,
                                         (cudaGraphConditionalHandle)h_gather);
}

void launch_g_level_begin(GraphState *g, unsigned long long h_level, unsigned long long h_first,
                          cudaStream_t st) {
    k_g_level_begin<<<1, 32, 0, st>>>(g, (cudaGraphConditionalHandle)h_level,
                                      (cudaGraphConditionalHandle)h_first);
}

void launch_g_level_end(GraphState *g, Counters *c, Seg *L, const Seg *L2,
                        unsigned long long h_level, int grid, cudaStream_t st) {
    k_g_level_end<<<grid, 256, 0, st>>>(g, c, L, L2, (cudaGraphConditionalHandle)h_level);
}

void launch_g_round_end(GraphState *g, Counters *c, Seg *R, const Seg *N,
                        unsigned long long h_round, int grid, cudaStream_t st) {
    k_g_round_end<<<grid, 256, 0, st>>>(g, c, R, N, (cudaGraphConditionalHandle)h_round);
}

}  // namespace ssort
