// rsbd8g_prefix.cuh - the prefix sort of 8- and 16-byte keys.
//
// An LSD sort of n keys runs one scatter pass per digit, but where the keys are spread out the top
// few digits already tell nearly all of them apart: 2^28 uniform 64-bit keys share their top 32 bits
// with one other key in 16.  So a large sort of wide keys first runs stable passes over a prefix --
// the top digits that are not all in one bucket -- and then settles the short groups of keys whose
// prefixes are equal, in one read of the keys:
//   * prefix_sample   each CTA of the histogram launch sorts a small random sample of the keys and
//                     counts, by highest differing digit, the neighbours that differ
//   * prefix_choose   (in the plan) the shortest prefix whose sample pairs leave groups of few keys on
//                     average; none when the sample says that more than kPrefixSlots digits, or nearly
//                     all of them, are needed: then the plain LSD passes run
//   * k_settle        puts every group of equal prefixes into the order of the whole keys, ties in
//                     the order they came (the passes were stable), so the result is the LSD sort's
//                     bit for bit.  One that is out of order and longer than the samples let pass
//                     (settle_limit) sets settle_fail, and the plain passes over every digit then sort the
//                     array as it stands: still a stable arrangement of the input, with the same histograms.
// Everything is decided on the device, so a sort still never synchronises with the host.
#pragma once
#include "rsbd8g_device.cuh"

namespace rsbd8g {

struct PlanArgs {
    uint64_t spin_limit_ns;
    uint32_t inplace;      // radixsort / radixsortnoalloc: sort `in` using `buf`
    uint32_t to_buffer;    // movetobuffer
    uint32_t rev;          // effective isrevorder
    uint32_t indirect;
    uint32_t stall_tile;
    uint32_t passes;       // digits of the key
    uint32_t prefetch;     // every array is device memory (Control::prefetch)
    uint32_t hot_ok;       // crowded digits may be ranked with ballots (PassPlan::hot)
    uint32_t prefix_ok;    // the launches of a prefix sort follow (slots before and after k_settle)
};

// The settle step compares a key with its whole group, so its work grows with the group size: up to
// this many equal-prefix keys on average are left to it.
constexpr uint64_t kSettleGroup = 2;
// the copies of one key that count when the sample's pairs are weighted (a window of positions fits a word)
constexpr uint32_t kSampleRun = 32;

// Every CTA of the histogram launch sorts up to a key per thread, drawn at random places (independent
// draws, so an input that is already in order is judged as any other), and counts the pairs of
// neighbours that differ, weighted with the copies each of the two has, by the highest digit in which
// they differ.  Many small samples tell as much about equal prefixes as one large one of as many
// pairs, and sort side by side: a bitonic network, by shuffles within a warp and through shared memory
// beyond.
// The pairs that the samples can form should outnumber the keys, for one pair too many to show: the smallest
// size of sample that forms half as many again (152 samples of 256 keys form 5 M pairs, of 1024 keys 80 M; with no more
// than the keys, 2^24 uniform ones lay so near the line that a fourth pass was taken, 473 us for 440), or several rounds
// of the largest.  A sample of 1024 keys adds 9 us to the histogram, of 256 keys 4 to 5 (2^21 int64 keys 28.4 -> 24.4 us, 19.1
// without samples).
constexpr int kSampleLeast = 256, kSampleDirect = 1024;    // k_histogram: up to one key per thread
constexpr int kSampleGather = 512;                         // k_gather_histogram: one key per thread (smaller samples took as long)
__host__ __device__ __forceinline__ uint64_t prefix_pairs(uint32_t samples, uint32_t size) { return uint64_t(samples) * (size * (size - 1u) / 2u); }
template <int LEAST, int MOST>
__host__ __device__ __forceinline__ uint32_t prefix_size(uint64_t n, uint32_t samples) {
    uint32_t size = LEAST;
    while (size < MOST && prefix_pairs(samples, size) < n + n / 2) size *= 2;
    return size;
}
__host__ __device__ __forceinline__ uint32_t prefix_rounds(uint64_t n, uint32_t samples, uint32_t size) {
    const uint64_t r = n / prefix_pairs(samples, size) + 1u;
    return r > 16 ? 16u : uint32_t(r);
}
template <typename U>
__device__ __forceinline__ U shfl_key(U k, int mask) { return __shfl_xor_sync(0xFFFFFFFFu, k, mask); }
template <int HB>
__device__ __forceinline__ KeyWide<HB> shfl_key(KeyWide<HB> k, int mask) {
    return KeyWide<HB>{__shfl_xor_sync(0xFFFFFFFFu, k.lo, mask), __shfl_xor_sync(0xFFFFFFFFu, k.hi, mask)};
}
template <typename U>
__device__ __forceinline__ U shfl_up_key(U k) { return __shfl_up_sync(0xFFFFFFFFu, k, 1); }
template <int HB>
__device__ __forceinline__ KeyWide<HB> shfl_up_key(KeyWide<HB> k) {
    return KeyWide<HB>{__shfl_up_sync(0xFFFFFFFFu, k.lo, 1), __shfl_up_sync(0xFFFFFFFFu, k.hi, 1)};
}
template <typename U>
__device__ __forceinline__ U shfl_down_key(U k) { return __shfl_down_sync(0xFFFFFFFFu, k, 1); }
template <int HB>
__device__ __forceinline__ KeyWide<HB> shfl_down_key(KeyWide<HB> k) {
    return KeyWide<HB>{__shfl_down_sync(0xFFFFFFFFu, k.lo, 1), __shfl_down_sync(0xFFFFFFFFu, k.hi, 1)};
}
// the threads of a sample
template <int SIZE, int THREADS>
__device__ __forceinline__ void sample_sync() {
    if constexpr (SIZE == THREADS) __syncthreads();
    else asm volatile("bar.sync 2, %0;" ::"n"(SIZE) : "memory");
}

// where draw `index` lies among n keys (splitmix64 of its index)
__device__ __forceinline__ uint64_t sample_place(uint64_t index, uint64_t n) {
    uint64_t z = (index + 1u) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return __umul64hi(z ^ (z >> 31), n);
}

// `rounds` samples of SIZE keys, by the first SIZE threads of a CTA of THREADS; the round that enough() ends is
// the last.  s: SIZE keys; heads: SIZE / 32 + 1 words; DRAWN: a0 is this thread's key of the first round
template <int SIZE, int THREADS, bool DRAWN, typename U, typename F, typename E>
__device__ __forceinline__ void prefix_sample(U *s, uint32_t *heads, uint64_t n, uint32_t rounds, uint64_t first, uint32_t *pairs, U a0,
                                              F key, E enough) {
    static_assert((SIZE & (SIZE - 1)) == 0, "a bitonic network of one key per thread");
    constexpr uint32_t size = SIZE;
    const uint32_t i = threadIdx.x;
    if (i < uint32_t(kMaxPasses)) pairs[i] = 0;
    if (i == 0) heads[size / 32] = 0xFFFFFFFFu;
    for (uint32_t round = 0; round < rounds; ++round) {
        U a = DRAWN && round == 0 ? a0 : key(sample_place((first + round) * size + i, n));
        for (uint32_t k = 2; k <= size; k <<= 1) {
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                U b;
                if (j >= 32) {
                    sample_sync<SIZE, THREADS>();
                    s[i] = a;
                    sample_sync<SIZE, THREADS>();
                    b = s[i ^ j];
                } else {
                    b = shfl_key(a, int(j));
                }
                const bool low = ((i & j) == 0) == ((i & k) == 0);      // this thread keeps the smaller key
                if (low ? key_less(b, a) : key_less(a, b)) a = b;
            }
        }
        sample_sync<SIZE, THREADS>();
        s[i] = a;
        sample_sync<SIZE, THREADS>();
        const U prev = s[i ? i - 1 : 0];
        const bool head = i == 0 || !key_same(prev, a);
        const uint32_t hm = __ballot_sync(0xFFFFFFFFu, head);
        if ((i & 31u) == 0) heads[i / 32] = hm;
        sample_sync<SIZE, THREADS>();
        if (head && i > 0) {
            // the copies of the key before (the head at or before i - 1) and of this one (the next head), from the
            // heads of the 32 positions on either side
            const uint32_t w = i / 32, l = i & 31u;
            const uint32_t below = uint32_t(((uint64_t(heads[w]) << 32) | (w ? heads[w - 1] : 0u)) >> l);
            const uint32_t above = uint32_t(((uint64_t(heads[w + 1]) << 32) | heads[w]) >> (l + 1));
            const uint32_t before = below ? uint32_t(__clz(below)) + 1u : kSampleRun, after = above ? uint32_t(__ffs(above)) : kSampleRun;
            atomicAdd(pairs + top_diff(prev, a), before * after);
        }
        sample_sync<SIZE, THREADS>();                                             // s and heads are free again
        if (round + 1 < rounds && enough()) break;
    }
}
// a thread's first key of the samples of its CTA (below)
template <typename U, int LEAST, int MOST, typename F>
__device__ __forceinline__ U prefix_draw(uint64_t n, F key) {
    const uint32_t size = prefix_size<LEAST, MOST>(n, gridDim.x), rounds = prefix_rounds(n, gridDim.x, size);
    return threadIdx.x < size ? key(sample_place(uint64_t(blockIdx.x) * rounds * size + threadIdx.x, n)) : U{};
}
// the samples of one histogram CTA, of LEAST to MOST keys, added to the sort's; a0: the thread's first key (if the size
// is not a fixed one)
template <typename U, int THREADS, int LEAST, int MOST, typename F>
__device__ __forceinline__ void prefix_sample_cta(U *s, uint64_t n, Control *__restrict__ ctrl, U a0, F key) {
    __shared__ uint32_t pairs[kMaxPasses], heads[MOST / 32 + 1];
    const uint32_t size = prefix_size<LEAST, MOST>(n, gridDim.x), rounds = prefix_rounds(n, gridDim.x, size);
    const uint64_t first = uint64_t(blockIdx.x) * rounds;
    auto all = [] { return false; };
    if (threadIdx.x < size) {
        if (LEAST == MOST || size == MOST) prefix_sample<MOST, THREADS, LEAST != MOST>(s, heads, n, rounds, first, pairs, a0, key, all);
        else if (size == LEAST) prefix_sample<LEAST, THREADS, true>(s, heads, n, rounds, first, pairs, a0, key, all);
        else prefix_sample<2 * LEAST, THREADS, true>(s, heads, n, rounds, first, pairs, a0, key, all);
    }
    static_assert(LEAST == MOST || MOST == 4 * LEAST, "the sizes between");
    __syncthreads();
    if (threadIdx.x < kMaxPasses && pairs[threadIdx.x]) atomicAdd(&ctrl->sample_pairs[threadIdx.x], pairs[threadIdx.x]);
}

// The passes of the shortest prefix that leaves groups of about kSettleGroup keys or fewer, *low its
// lowest digit; 0 for a plain sort.  W pairs of a sample that can form `all` pairs stand for n W / all
// other keys with the same prefix per key.  One thread calls it.
__device__ __forceinline__ uint32_t prefix_choose(const uint32_t *sample_pairs, uint32_t survive, uint64_t n, uint64_t all,
                                                  uint32_t *low) {
    const int digits = __popc(survive);
    uint64_t pairs = 0;
    uint32_t k = 0;
    for (int q = 0; q < kMaxPasses && pairs < (1u << 20); ++q) {   // pairs: their highest differing digit is below q
        if ((survive >> q) & 1u) {
            const int passes = __popc(survive >> q);
            // at least two passes must be saved: the settle step reads every key once
            if (passes <= kPrefixSlots && passes <= digits - 2 && (pairs + 1u) * n <= kSettleGroup * all) {
                k = uint32_t(passes);
                *low = uint32_t(q);
            }
        }
        pairs += sample_pairs[q];
    }
    return k;
}
// will prefix_choose find none, whatever pairs are still to come?
__device__ __forceinline__ bool prefix_hopeless(const uint32_t *sample_pairs, uint32_t survive, uint64_t n, uint64_t all) {
    const int most = min(__popc(survive) - 2, kPrefixSlots);
    uint64_t pairs = 0;
    int q = 0;
    for (; q < kMaxPasses && !(((survive >> q) & 1u) && __popc(survive >> q) <= most); ++q) pairs += sample_pairs[q];
    return (pairs + 1u) * n > kSettleGroup * all;
}

// Plan the passes over the digits of `mask`, lowest first, from array `cur` on; returns where they
// end.  Launch slots: keys of up to 4 bytes take the slot of the digit's number, wider keys consecutive
// slots from slot0.  A copy form must end in its output; `even` makes the number of passes even (by
// sorting by the lowest digit twice) for a chain that starts there.  keep_keys: the last pass of an
// indirect sort writes its keys too; hot: the crowded digit of each position.  One thread calls it.
__host__ __device__ __forceinline__ uint32_t plan_chain(Control *__restrict__ ctrl, const PlanArgs &a, const uint32_t *hot, uint32_t mask, bool even,
                                               int slot0, uint32_t cur, uint32_t &curk, bool rev, bool keep_keys) {
    int digits = 0;
    for (uint32_t m = mask; m; m &= m - 1) ++digits;
    const int again = even ? digits & 1 : 0;
    const int k = digits + again;
    int p = -1;
    for (int i = 1; i <= k; ++i) {
        if (!(again && i == 2)) {
            do ++p;
            while (!((mask >> p) & 1u));
        }
        const int slot = a.passes >= 8 ? slot0 + i - 1 : p;
        PassPlan &pp = ctrl->plan[slot];
        pp.active = 1u;
        pp.hot = hot[p];
        pp.digit = uint16_t(p);
        pp.status = uint16_t(a.passes >= 8 ? i - 1 : p);
        uint32_t dst;
        if (a.inplace) dst = (cur == kArrIn) ? kArrBuf : kArrIn;
        else dst = ((k - i) % 2 == 0) ? kArrOut : kArrBuf;
        pp.reverse = (i == 1) && rev;
        if (a.indirect) {
            pp.src_vals = cur;
            pp.dst_vals = dst;
            pp.src_keys = curk;
            const uint32_t dk = (curk == kArrKeysA) ? kArrKeysB : kArrKeysA;
            pp.dst_keys = (i == k && !keep_keys) ? kArrNone : dk;
            curk = dk;
        } else {
            pp.src_keys = cur;
            pp.dst_keys = dst;
            pp.src_vals = kArrNone;
            pp.dst_vals = kArrNone;
        }
        cur = dst;
    }
    return cur;
}

// The copy step after passes that end in array `cur` (no_pass: none of them runs, so a reversal of
// the order is still to be done).  One thread calls it.
__device__ __forceinline__ void plan_copy(Control *__restrict__ ctrl, const PlanArgs &a, uint32_t cur, bool no_pass) {
    ctrl->copy_mode = kCopyNone;
    if (!a.inplace) {
        if (no_pass) {
            ctrl->copy_mode = a.rev ? kCopyReversed : kCopyPlain;
            ctrl->copy_src = kArrIn;
            ctrl->copy_dst = kArrOut;
        }
    } else {
        const uint32_t target = a.to_buffer ? kArrBuf : kArrIn;
        if (no_pass && a.rev) {
            ctrl->copy_mode = a.to_buffer ? kCopyReversed : kReverseInPlace;
            ctrl->copy_src = kArrIn;
            ctrl->copy_dst = target;
        } else if (cur != target) {
            ctrl->copy_mode = kCopyPlain;
            ctrl->copy_src = cur;
            ctrl->copy_dst = target;
        }
    }
}

// ---- the settle step ---------------------------------------------------------------------------
// Warps take chunks in turn, each on its own (no barrier, so many warps' loads are in flight).  A lane
// holds kItems neighbouring keys in registers; the last lane's keys are the halo, the first keys of
// the next chunk.  A key is a head if its prefix differs from the one before it, else an inversion if
// it is below the key before it.  A group belongs to the chunk it starts in, and is put in order by rounds
// of exchanges between neighbours of one group (only a key below the one before it passes it, so equal
// keys keep their order): a round per key that another has to pass, a few for groups of a few keys.
//   A group that is still open at the end of the halo, or takes more than kRounds rounds, is settled by
// the warp in shared memory, with kView keys in view, every key moving to the place found by comparing
// it with its group (settle_wide).  One of more than kMost keys, or that runs past the view, is settled by the first
// warp that meets an inversion in it, whichever chunk that is in, after its chunks: by digit passes of its own over
// the digits below the prefix, through the array that the scatter passes left free (settle_long).
//   A group from an earlier chunk is otherwise left alone, as that chunk's warp settles it.  No inversion is passed
// over: each lies in some warp's chunk, and its group either ends within the view of the chunk it starts in
// or is taken by settle_long, which raises settle_fail where the group is too long.  Neighbouring chunks read keys
// that a chunk moves only for their prefixes, which a move within a group leaves as they are (settle_ld).
template <typename U>
struct SettleShape {
    static constexpr int kThreads = sizeof(U) == 8 ? 256 : 128;     // (static shared memory stays below 48 KB)
    static constexpr int kWarps = kThreads / 32;
    static constexpr int kItems = 8;
    static constexpr int kChunk = 31 * kItems;
    static constexpr int kCtaKeys = kWarps * kChunk;
    static constexpr int kView = kChunk + 224;
    static constexpr int kWords = (kView + 31) / 32;
    static constexpr int kRounds = 12;
    static constexpr int kMost = 96;        // keys of the longest group that settle_wide settles (its work grows with the square)
};

// The longest group of n keys that a warp settles: 2 sqrt(n) keys, rounded up.  A crowd of g keys among
// spread ones shows as (g / n)^2 of the samples' pairs, which prefix_choose takes for too many from g =
// sqrt(2 n) on, give or take the few pairs that make the difference; so a longer group that no sample saw is
// rare, and one as long as this costs far less than the plain passes would (2^28 int64 keys, 10,000 of them one
// group: 6.2 ms, 14.9 with the plain passes and 5.9 without such a group; 2^21 keys, 500: 152, 274 and 131 us).
__host__ __device__ __forceinline__ uint64_t settle_limit(uint64_t n) {
    int bits = 0;
    while (bits < 40 && (uint64_t(1) << bits) < n) ++bits;
    const uint64_t m = uint64_t(1) << ((bits + 1) / 2 + 1);
    return m < 1024 ? 1024 : m;
}

// inversions in long groups that a warp keeps (more fail the step: crowds are for the samples to see)
constexpr uint32_t kSettleLater = 12;
// a warp's shared memory in the settle step
template <typename U>
struct alignas(16) SettleWarp {
    U key[SettleShape<U>::kView];
    uint32_t head[SettleShape<U>::kWords], inv[SettleShape<U>::kWords];
    // inversions found in long groups (tag + place), for settle_long after the warp's chunks
    uint32_t found;
    uint64_t later[kSettleLater], tag;
};
// what settle_long needs beside the keys: the arrays that are free, the long groups that were taken up (a hash table
// of start + tag + 1, 0 for none), settle_limit, and the surviving digits below the prefix
template <typename U>
struct SettleLong {
    U *free_keys;
    uint64_t *free_vals;
    unsigned long long *taken;
    uint64_t tag, limit;
    uint32_t room, digits;
};
constexpr uint32_t kTakenRoom = 4096;      // entries of the table, at most

// the last set bit of w[] at or below position i, -1 if there is none
__device__ __forceinline__ int bit_at_or_below(const uint32_t *w, int i) {
    int x = i >> 5;
    uint32_t m = w[x] & (0xFFFFFFFFu >> (31 - (i & 31)));
    while (!m && --x >= 0) m = w[x];
    return m ? x * 32 + 31 - __clz(m) : -1;
}
// the first set bit of w[0, words) at or above position i, words * 32 if there is none
__device__ __forceinline__ int bit_at_or_above(const uint32_t *w, int i, int words) {
    int x = i >> 5;
    if (x >= words) return words * 32;
    uint32_t m = w[x] & (0xFFFFFFFFu << (i & 31));
    while (!m && ++x < words) m = w[x];
    return m ? x * 32 + __ffs(m) - 1 : words * 32;
}

// the key as the sort orders it
template <int MODE, typename U>
__device__ __forceinline__ U settle_order(U b, bool desc) {
    const U q = filter_key<MODE>(b);
    return desc ? key_not(q) : q;
}

// Keys that another warp may be moving are read, and written, in one piece.  An 8-byte key is one access; of a 16-byte
// key PTX promises that only for the 128-bit type.  Two words of different keys of a group do no harm where the order
// is taken word by word: the group's prefix is in each.  Where a word's bits depend on the other's (a negation, a
// shift: the float, absolute signed and tiered orders) they could show a prefix that no key has.
template <int MODE, typename U>
constexpr bool kWholeKeys = sizeof(U) == 16 && (MODE == 1 || MODE == 3 || MODE == 5 || MODE == 6);
template <int MODE, typename U>
__device__ __forceinline__ U settle_ld(const U *p) {
    if constexpr (kWholeKeys<MODE, U>) {
        U k;
        asm volatile("{ .reg .b128 v; ld.relaxed.gpu.global.b128 v, [%2]; mov.b128 {%0, %1}, v; }" : "=l"(k.lo), "=l"(k.hi) : "l"(p) : "memory");
        return k;
    } else {
        return *p;
    }
}
template <int MODE, typename U>
__device__ __forceinline__ void settle_st(U *p, U k) {
    if constexpr (kWholeKeys<MODE, U>)
        asm volatile("{ .reg .b128 v; mov.b128 v, {%1, %2}; st.relaxed.gpu.global.b128 [%0], v; }" ::"l"(p), "l"(k.lo), "l"(k.hi) : "memory");
    else
        *p = k;
}

// ITEMS keys from p on: 16-byte loads where the address allows; whole: settle_ld
template <int MODE, int ITEMS, typename U>
__device__ __forceinline__ void load_run(U (&v)[ITEMS], const U *p, bool whole) {
    if (kWholeKeys<MODE, U> && whole) {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) v[i] = settle_ld<MODE>(p + i);
    } else if (sizeof(U) == 8 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) {
        constexpr int V = 16 / int(sizeof(U));
#pragma unroll
        for (int i = 0; i < ITEMS; i += V) {
            const uint4 q = *reinterpret_cast<const uint4 *>(p + i);
            memcpy(&v[i], &q, 16);
        }
    } else {
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) v[i] = p[i];
    }
}

// take up the long group `id`: 1, or 0 if another warp has, -1 if the table is full
template <typename U>
__device__ __forceinline__ int settle_take(const SettleLong<U> &w, unsigned long long id) {
    if (w.room == 0) return -1;
    uint32_t h = uint32_t((id * 0x9E3779B97F4A7C15ull) >> 32) % w.room;
    for (int i = 0; i < 64; ++i) {
        const unsigned long long old = atomicCAS(w.taken + h, 0ull, id);
        if (old == 0ull) return 1;
        if (old == id) return 0;
        h = h + 1 == w.room ? 0 : h + 1;
    }
    return -1;
}

// keep an inversion in a long group for settle_long (any lanes may call it)
template <typename U>
__device__ __noinline__ void settle_later(SettleWarp<U> *warp, uint64_t at, uint32_t *fail, uint32_t fail_bit) {
    const uint32_t i = atomicAdd(&warp->found, 1u);
    if (i < kSettleLater) warp->later[i] = warp->tag + at;
    else atomicOr(fail, fail_bit);
}
template <typename U>
__device__ __forceinline__ uint32_t settle_found(const SettleWarp<U> &warp) { return min(warp.found, kSettleLater); }

// the largest d <= most with ok(d), by a warp: 32 probes a round; ok(lo) holds, and ok is true up to that d
template <typename F>
__device__ __forceinline__ uint32_t warp_last(uint32_t lo, uint32_t most, F ok) {
    uint32_t hi = most + 1;                               // the first that may not be
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32, d = lo + ((threadIdx.x & 31u) + 1) * step;
        const uint32_t c = uint32_t(__popc(__ballot_sync(0xFFFFFFFFu, d < hi && ok(d))));
        hi = min(hi, lo + (c + 1) * step);
        lo += c * step;
    }
    return lo;
}

__device__ __forceinline__ void or_diff(uint64_t &acc, uint64_t a, uint64_t b) { acc |= a ^ b; }
template <int HB>
__device__ __forceinline__ void or_diff(KeyWide<HB> &acc, KeyWide<HB> a, KeyWide<HB> b) {
    acc.lo |= a.lo ^ b.lo;
    acc.hi |= a.hi ^ b.hi;
}
// the digits in which any lane's bits are set
__device__ __forceinline__ uint32_t diff_digits(uint64_t d) {
    const uint32_t w[2] = {__reduce_or_sync(0xFFFFFFFFu, uint32_t(d)), __reduce_or_sync(0xFFFFFFFFu, uint32_t(d >> 32))};
    uint32_t m = 0;
#pragma unroll
    for (int p = 0; p < 8; ++p) m |= ((w[p / 4] >> (p % 4 * 8)) & 0xFFu) ? 1u << p : 0u;
    return m;
}
template <int HB>
__device__ __forceinline__ uint32_t diff_digits(KeyWide<HB> d) { return diff_digits(d.lo) | (diff_digits(d.hi) << 8); }

// One warp sorts the group that has an inversion at key `at`, unless it is settle_wide's or another warp has taken it
// up: a stable pass per digit below the prefix that is not the same in all, ranked by matching
// digits, between the group's place and the same place in the free arrays (a key's place always holds a key of
// the group, as the neighbours' reads want it).  A pass counts the next one's digits as it goes.
template <int MODE, bool HAS_VAL, typename U>
__device__ __noinline__ void settle_long(U *keys, uint64_t *vals, uint64_t at, uint64_t n, U mask, bool desc, SettleWarp<U> *warp,
                                         const SettleLong<U> &w, uint32_t *fail, uint32_t fail_bit) {
    using S = SettleShape<U>;
    constexpr int B = sizeof(U) == 8 && !HAS_VAL ? 8 : 4;     // loads of a lane in flight
    static_assert(sizeof(warp->key) >= 2 * kBuckets * 4, "the offsets and the next counts fit the view's memory");
    const int lane = int(threadIdx.x & 31u);
    const uint32_t limit = uint32_t(w.limit);
    const U ref = settle_order<MODE>(settle_ld<MODE>(keys + at), desc);
    auto same = [&](uint64_t i) { return same_masked(settle_order<MODE>(settle_ld<MODE>(keys + i), desc), ref, mask); };
    const uint32_t back = warp_last(1, uint32_t(at < limit ? at : limit), [&](uint32_t d) { return same(at - d); });
    const uint32_t on = warp_last(0, uint32_t(n - 1 - at < limit ? n - 1 - at : limit), [&](uint32_t d) { return same(at + d); });
    const uint32_t len = back + on + 1;
    const uint64_t s = at - back, c0 = s / S::kChunk * S::kChunk;
    if (len <= uint32_t(S::kMost) && (s + len < c0 + S::kView || c0 + S::kView >= n)) return;      // settle_wide's
    int mine = -1;
    if (lane == 0 && len <= limit) mine = settle_take(w, s + w.tag + 1u);
    mine = __shfl_sync(0xFFFFFFFFu, mine, 0);
    if (mine < 0 && lane == 0) atomicOr(fail, fail_bit);
    if (mine <= 0) return;
    uint32_t *off = reinterpret_cast<uint32_t *>(warp->key), *cnt = off + kBuckets;
    U *src = keys + s, *dst = w.free_keys + s;
    uint64_t *src_v = vals, *dst_v = vals;
    if constexpr (HAS_VAL) {
        src_v = vals + s;
        dst_v = w.free_vals + s;
    }
    U diff{};
    for (uint32_t x0 = 0; x0 < len; x0 += 32 * B) {
        U k[B];
#pragma unroll
        for (int q = 0; q < B; ++q) k[q] = src[min(x0 + uint32_t(q * 32 + lane), len - 1)];
#pragma unroll
        for (int q = 0; q < B; ++q) or_diff(diff, settle_order<MODE>(k[q], desc), ref);
    }
    const uint32_t digits = diff_digits(diff) & w.digits;
    for (int i = lane; i < kBuckets; i += 32) cnt[i] = 0;
    __syncwarp();
    if (digits) {
        const int p = __ffs(digits) - 1;
        for (uint32_t x0 = 0; x0 < len; x0 += 32 * B) {
            U k[B];
#pragma unroll
            for (int q = 0; q < B; ++q) k[q] = src[min(x0 + uint32_t(q * 32 + lane), len - 1)];
#pragma unroll
            for (int q = 0; q < B; ++q)
                if (x0 + uint32_t(q * 32 + lane) < len) atomicAdd(cnt + digit_of(settle_order<MODE>(k[q], desc), p), 1u);
        }
    }
    for (uint32_t m = digits; m; m &= m - 1) {
        const int p = __ffs(m) - 1, next = (m & (m - 1)) ? __ffs(m & (m - 1)) - 1 : -1;
        __syncwarp();
        uint32_t sum = 0;
#pragma unroll
        for (int i = 0; i < kBuckets / 32; ++i) sum += cnt[lane * (kBuckets / 32) + i];
        uint32_t to0 = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, to0, o);
            if (lane >= o) to0 += y;
        }
        to0 -= sum;
#pragma unroll
        for (int i = 0; i < kBuckets / 32; ++i) {
            off[lane * (kBuckets / 32) + i] = to0;
            to0 += cnt[lane * (kBuckets / 32) + i];
            cnt[lane * (kBuckets / 32) + i] = 0;
        }
        __syncwarp();
        for (uint32_t x0 = 0; x0 < len; x0 += 32 * B) {
            U k[B];
            uint64_t v[HAS_VAL ? B : 1];
#pragma unroll
            for (int q = 0; q < B; ++q) {
                const uint32_t x = min(x0 + uint32_t(q * 32 + lane), len - 1);
                k[q] = src[x];
                if constexpr (HAS_VAL) v[q] = src_v[x];
            }
#pragma unroll
            for (int q = 0; q < B; ++q) {
                const bool in = x0 + uint32_t(q * 32 + lane) < len;
                const U b = settle_order<MODE>(k[q], desc);
                const uint32_t d = in ? digit_of(b, p) : uint32_t(kBuckets);
                const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d), before = uint32_t(__popc(peers & ((1u << lane) - 1u)));
                const uint32_t to = in ? off[d] + before : len;
                __syncwarp();
                if (in && before == 0) off[d] += uint32_t(__popc(peers));
                __syncwarp();
                if (to < len) {
                    settle_st<MODE>(dst + to, k[q]);
                    if constexpr (HAS_VAL) dst_v[to] = v[q];
                }
                if (in && next >= 0) atomicAdd(cnt + digit_of(b, next), 1u);
            }
        }
        U *t = src;
        src = dst;
        dst = t;
        uint64_t *tv = src_v;
        src_v = dst_v;
        dst_v = tv;
    }
    __syncwarp();
    if (src != keys + s) {
#pragma unroll 4
        for (uint32_t x = uint32_t(lane); x < len; x += 32) {
            settle_st<MODE>(dst + x, src[x]);
            if constexpr (HAS_VAL) dst_v[x] = src_v[x];
        }
    }
    __syncwarp();                                         // the warp's shared memory is free again
}

// One warp settles the groups that start in the chunk at c0, in shared memory: every key of a group that is out of
// order finds its place by comparing itself with its group, all groups side by side (one group after another took 13 us
// a chunk of groups of six).  Long ones, and one that runs on past the view, are kept for settle_long (2^23 keys of 64 k
// values, some of whose groups have 256 keys: 248 us with all of them settled here, 59 so).
template <int MODE, bool HAS_VAL, typename S, typename U>
__device__ __noinline__ void settle_wide(U *keys, uint64_t *vals, uint64_t c0, uint64_t n, U mask, bool desc, SettleWarp<U> *warp,
                                         uint32_t *fail, uint32_t fail_bit) {
    constexpr int WORDS = S::kWords;
    U *key = warp->key;
    uint32_t *hw = warp->head, *vw = warp->inv;
    const int lane = int(threadIdx.x & 31u);
    const int view = int(n - c0 < uint64_t(S::kView) ? n - c0 : uint64_t(S::kView));
    for (int x = lane; x < view; x += 32) key[x] = settle_ld<MODE>(keys + c0 + x);
    __syncwarp();
    for (int w = 0; w < WORDS; ++w) {
        const int x = w * 32 + lane;
        bool h = x == 0 ? c0 == 0 : x >= view, v = false;
        if (!h) {
            const U a = settle_order<MODE>(x ? key[x ? x - 1 : 0] : settle_ld<MODE>(keys + c0 - 1), desc), b = settle_order<MODE>(key[x], desc);
            h = !same_masked(a, b, mask);
            v = !h && key_less(b, a);
        }
        const uint32_t hm = __ballot_sync(0xFFFFFFFFu, h), vm = __ballot_sync(0xFFFFFFFFu, v);
        if (lane == 0) {
            hw[w] = hm;
            vw[w] = vm;
        }
    }
    __syncwarp();
    int to[WORDS];                                        // where this lane's keys go (-1: they stay)
    uint64_t p[HAS_VAL ? WORDS : 1];
    for (int r = 0; r < WORDS; ++r) {
        const int i = r * 32 + lane;
        to[r] = -1;
        if (i >= view) continue;
        const int s = bit_at_or_below(hw, i);
        if (s < 0 || s >= S::kChunk) continue;            // from an earlier chunk, or of the next
        const int x = bit_at_or_above(vw, s, WORDS), e = bit_at_or_above(hw, i + 1, WORDS);
        if (x >= e) continue;                             // in order
        if (e - s > S::kMost || (e == view && c0 + uint64_t(view) < n)) {
            if (i == x) settle_later(warp, c0 + uint64_t(x), fail, fail_bit);
            continue;
        }
        const U b = settle_order<MODE>(key[i], desc);
        int at = s;
#pragma unroll 4
        for (int j = s; j < e; ++j) {
            const U a = settle_order<MODE>(key[j], desc);
            at += key_less(a, b) || (j < i && key_same(a, b)) ? 1 : 0;
        }
        if (at == i) continue;
        to[r] = at;
        if constexpr (HAS_VAL) p[r] = vals[c0 + i];
    }
    __syncwarp();                                         // every pointer that moves has been read
    for (int r = 0; r < WORDS; ++r) {
        if (to[r] < 0) continue;
        settle_st<MODE>(keys + c0 + to[r], key[r * 32 + lane]);
        if constexpr (HAS_VAL) vals[c0 + to[r]] = p[r];
    }
    __syncwarp();                                         // the warp's shared memory is free again
}

// Does the group of the key at c0 + 255 have an inversion between there and the end of the view?  (Most groups that are
// open at the halo's end and in order so far stay so, many copies of one key above all: 2^26 keys of 64 k values 186 us
// with settle_wide for each such chunk, 141 so.)
template <int MODE, typename S, typename U>
__device__ __noinline__ bool settle_peek(const U *keys, uint64_t c0, uint64_t n, U mask, bool desc) {
    constexpr int SEEN = 32 * S::kItems;
    const int lane = int(threadIdx.x & 31u), view = int(n - c0 < uint64_t(S::kView) ? n - c0 : uint64_t(S::kView));
    const U last = settle_order<MODE>(settle_ld<MODE>(keys + c0 + SEEN - 1), desc);
    bool inv = false;
#pragma unroll
    for (int j = 0; j < (S::kView - SEEN + 31) / 32; ++j) {
        const int x = min(SEEN + j * 32 + lane, view - 1);
        const U a = settle_order<MODE>(settle_ld<MODE>(keys + c0 + x - 1), desc), b = settle_order<MODE>(settle_ld<MODE>(keys + c0 + x), desc);
        inv |= same_masked(last, b, mask) && key_less(b, a);
    }
    return __any_sync(0xFFFFFFFFu, inv) != 0;
}

// one warp settles the groups that start in the chunk at c0, and keeps what it meets of long groups for later (a
// call of settle_long from here would cost the loop around it registers)
template <int MODE, bool HAS_VAL, typename S, typename U>
__device__ __forceinline__ void settle_chunk(U *keys, uint64_t *vals, uint64_t c0, uint64_t n, U mask, bool desc, SettleWarp<U> *warp,
                                             uint32_t *fail, uint32_t fail_bit) {
    constexpr int ITEMS = S::kItems, C = S::kChunk;
    // v holds the keys as they are where ordering them takes an exclusive-or, else as the sort orders them:
    // a key that moves is then fetched again from where it came (as a pointer is)
    constexpr bool RAW = MODE == 0 || MODE == 2, INDEX = HAS_VAL || !RAW;
    auto ordered = [&](const U &k) { return RAW ? settle_order<MODE>(k, desc) : k; };
    const int lane = int(threadIdx.x & 31u);
    const bool full = n - c0 >= uint64_t(32 * ITEMS);
    const int own = full ? ITEMS : int(n - c0) - lane * ITEMS;      // this lane's keys (may be < 0 or > ITEMS)
    U v[ITEMS], before{};
    uint32_t hb, vb, heads;
    for (bool whole = false;; whole = true) {
        if (full) {
            load_run<MODE, ITEMS>(v, keys + c0 + lane * ITEMS, whole || lane == 0 || lane == 31);
        } else {
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                v[j] = U{};
                if (j < own) v[j] = settle_ld<MODE>(keys + c0 + lane * ITEMS + j);
            }
        }
        before = lane == 0 && c0 ? settle_ld<MODE>(keys + c0 - 1) : U{};
        if constexpr (!RAW) {
            before = settle_order<MODE>(before, desc);
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) v[j] = settle_order<MODE>(v[j], desc);
        }
        // heads and inversions among this lane's keys (bit j: key j)
        hb = vb = 0;
        {
            const U up = shfl_up_key(v[ITEMS - 1]);
            U a = ordered(lane ? up : before);
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                const U b = ordered(v[j]);
                const bool h = !same_masked(a, b, mask);
                if (h) hb |= 1u << j;
                else if (key_less(b, a)) vb |= 1u << j;
                a = b;
            }
        }
        if (c0 == 0 && lane == 0) hb |= 1u;
        if (!full) hb |= own >= ITEMS ? 0u : own <= 0 ? 0xFFu : 0xFFu << own;     // past the end: each alone
        vb &= ~hb;
        heads = __ballot_sync(0xFFFFFFFFu, hb != 0);
        // Another warp moves keys here only of a group that came in or of one that runs far past the halo.  The first and
        // the last lane's keys, which are read whole, tell: a head in the first, and one after the last's first key.
        if (!kWholeKeys<MODE, U> || !full || whole) break;
        if ((heads & 1u) && __any_sync(0xFFFFFFFFu, lane == 31 && (hb & 0xFEu))) break;
    }
    const bool open = !(heads >> 31) && (heads & 0x7FFFFFFFu) && n - c0 > uint64_t(32 * ITEMS);
    if (!__any_sync(0xFFFFFFFFu, vb != 0) && !open) return;
    // this lane's keys of the group that came in, and of the groups that the next chunk settles
    const uint32_t below = hb ? (hb & (0u - hb)) - 1u : 0xFFu;      // keys before the lane's first head
    const uint32_t in = (heads & ((1u << lane) - 1u)) == 0 ? below : 0u;
    const uint32_t out = lane == 31 ? ~below & 0xFFu : 0u;
    const uint32_t bad_in = vb & in;
    if (__any_sync(0xFFFFFFFFu, bad_in != 0)) {
        // met by the chunk before too, if it holds the start and has the inversion in its view
        bool left = bad_in && lane * ITEMS + 31 - __clz(bad_in) >= S::kView - C;
        if (bad_in && c0 > uint64_t(C)) {
            const U a = settle_order<MODE>(settle_ld<MODE>(keys + c0 - C - 1), desc), b = settle_order<MODE>(settle_ld<MODE>(keys + c0 - 1), desc);
            left |= same_masked(a, b, mask);
        }
        const uint32_t any = __ballot_sync(0xFFFFFFFFu, left);
        if (left && lane == __ffs(any) - 1) settle_later(warp, c0 + uint64_t(lane * ITEMS + 31 - __clz(bad_in)), fail, fail_bit);
    }
    const uint32_t pass = ~hb & ~in & ~out & 0xFFu;          // keys that may pass the one before them
    // (open: with no inversion in the group so far, it is looked at on to the view's end)
    bool wide = open;
    if (open && !__any_sync(0xFFFFFFFFu, (vb & ~in) != 0)) wide = settle_peek<MODE, S>(keys, c0, n, mask, desc);
    if (!open) {
        uint32_t moved = 0, from[INDEX ? ITEMS : 1];
        if constexpr (INDEX) {
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) from[j] = uint32_t(lane * ITEMS + j);
        }
        const uint32_t next = __shfl_down_sync(0xFFFFFFFFu, pass, 1);
        const bool pass0 = (pass & 1u) && lane, pass8 = lane < 31 && (next & 1u);
        // one round settles a chunk whose groups have two keys at most
        const bool several = __any_sync(0xFFFFFFFFu, (pass & (pass << 1)) != 0 || (pass8 && (pass >> (ITEMS - 1))));
        for (int r = 0;; ++r) {
            bool swapped = false;
            // across the lanes: both sides see the same two keys and come to the same answer
            const U up = shfl_up_key(v[ITEMS - 1]), down = shfl_down_key(v[0]);
            uint32_t fup = 0, fdown = 0;
            if constexpr (INDEX) {
                fup = __shfl_up_sync(0xFFFFFFFFu, from[ITEMS - 1], 1);
                fdown = __shfl_down_sync(0xFFFFFFFFu, from[0], 1);
            }
            if (pass0 && key_less(ordered(v[0]), ordered(up))) {
                v[0] = up;
                if constexpr (INDEX) from[0] = fup;
                moved |= 1u;
                swapped = true;
            }
            if (pass8 && key_less(ordered(down), ordered(v[ITEMS - 1]))) {
                v[ITEMS - 1] = down;
                if constexpr (INDEX) from[INDEX ? ITEMS - 1 : 0] = fdown;
                moved |= 1u << (ITEMS - 1);
                swapped = true;
            }
#pragma unroll
            for (int j = 1; j < ITEMS; ++j) {
                if (((pass >> j) & 1u) && key_less(ordered(v[j]), ordered(v[j - 1]))) {
                    const U t = v[j];
                    v[j] = v[j - 1];
                    v[j - 1] = t;
                    if constexpr (INDEX) {
                        const uint32_t f = from[INDEX ? j : 0];
                        from[INDEX ? j : 0] = from[INDEX ? j - 1 : 0];
                        from[INDEX ? j - 1 : 0] = f;
                    }
                    moved |= 3u << (j - 1);
                    swapped = true;
                }
            }
            if (!several || !__any_sync(0xFFFFFFFFu, swapped)) break;
            if (r == S::kRounds) {
                wide = true;
                break;
            }
        }
        if (!wide) {
            // every pointer (and key) that moves is read before one is written
            U *dst = keys + c0 + lane * ITEMS;
            if constexpr (HAS_VAL) {
                uint64_t p[ITEMS];
#pragma unroll
                for (int j = 0; j < ITEMS; ++j)
                    if ((moved >> j) & 1u) p[j] = vals[c0 + from[j]];
                __syncwarp();
#pragma unroll
                for (int j = 0; j < ITEMS; ++j)
                    if ((moved >> j) & 1u) vals[c0 + lane * ITEMS + j] = p[j];
            }
            if constexpr (!RAW) {
#pragma unroll
                for (int j = 0; j < ITEMS; ++j)
                    if ((moved >> j) & 1u) v[j] = keys[c0 + from[j]];
                __syncwarp();
            }
#pragma unroll
            for (int j = 0; j < ITEMS; ++j)
                if ((moved >> j) & 1u) settle_st<MODE>(dst + j, v[j]);
        }
    }
    if (wide) settle_wide<MODE, HAS_VAL, S>(keys, vals, c0, n, mask, desc, warp, fail, fail_bit);
}

template <typename U, int MODE, bool HAS_VAL>
__global__ void __launch_bounds__(SettleShape<U>::kThreads, sizeof(U) == 8 ? (HAS_VAL || (MODE != 0 && MODE != 2) ? 4 : 5) : 6)
    k_settle(Control *__restrict__ ctrl, const SortArrays arrs, uint64_t n, uint32_t desc, unsigned char *status,
             size_t status_bytes, PlanArgs pa) {
    using S = SettleShape<U>;
    constexpr int THREADS = S::kThreads, C = S::kChunk;
    next_may_start();
    after_previous();
    const uint32_t k = ctrl->prefix_passes, low = ctrl->prefix_low, survive = ctrl->survive;
    if (k == 0 || ctrl->abort) return;
    __shared__ SettleWarp<U> warps[S::kWarps];
    __shared__ uint32_t last;
    const int tid = threadIdx.x, warp = tid >> 5;
    bool bad = !prefix_in_range<KeyTraits<U>::kDigits>(k, low, survive);
    const PassPlan &end = ctrl->plan[bad ? 0u : k - 1];
    U *keys = static_cast<U *>(sort_array(arrs, end.dst_keys, HAS_VAL ? kArrKeysA : kArrBuf, &bad));
    uint64_t *vals = static_cast<uint64_t *>(sort_array(arrs, end.dst_vals, kArrBuf, &bad));
    if (bad || !keys || (HAS_VAL && !vals)) {       // a damaged control block
        if (tid == 0) atomicOr(&ctrl->error, kDevFault);
        return;
    }
    if ((tid & 31) == 0) {
        warps[warp].found = 0;
        warps[warp].tag = 0;
    }
    __syncwarp();
    // the prefix passes' look-back words, cleared for the plain passes that a failure calls for
    for (uint64_t i = uint64_t(blockIdx.x) * THREADS + tid; i < uint64_t(k) * status_bytes / 16; i += uint64_t(gridDim.x) * THREADS)
        reinterpret_cast<uint4 *>(status)[i] = make_uint4(0, 0, 0, 0);
    const U mask = prefix_mask<U>(low);
    const uint64_t stride = uint64_t(gridDim.x) * S::kCtaKeys;
    for (uint64_t c0 = uint64_t(blockIdx.x) * S::kCtaKeys + uint32_t(warp * C); c0 < n; c0 += stride)
        settle_chunk<MODE, HAS_VAL, S>(keys, vals, c0, n, mask, desc != 0, &warps[warp], &ctrl->settle_fail, 1u);
    __syncwarp();
    const uint32_t found = settle_found(warps[warp]);
    if (found && !__any_sync(0xFFFFFFFFu, ld_relaxed(&ctrl->settle_fail) != 0)) {
        // the array that is free: what the last pass read from or could have, the copy forms' buffer or the in-place
        // forms' other array; the table of long groups lies where the last digit's look-back words do, which are
        // clear (a prefix leaves two digits out)
        const uint32_t free = (HAS_VAL ? end.dst_vals : end.dst_keys) == kArrBuf ? (pa.inplace ? kArrIn : kArrOut) : kArrBuf;
        void *arr = sort_array(arrs, free, kArrBuf, &bad);
        SettleLong<U> w;
        w.free_keys = HAS_VAL ? static_cast<U *>(sort_array(arrs, end.dst_keys == kArrKeysA ? kArrKeysB : kArrKeysA, kArrKeysA, &bad))
                              : static_cast<U *>(arr);
        w.free_vals = static_cast<uint64_t *>(arr);
        w.taken = reinterpret_cast<unsigned long long *>(status + (KeyTraits<U>::kDigits - 1) * status_bytes);
        w.tag = 0;
        w.limit = settle_limit(n);
        w.room = uint32_t(status_bytes / 8 < kTakenRoom ? status_bytes / 8 : kTakenRoom);
        w.digits = survive & ((1u << low) - 1u);
        bad = __any_sync(0xFFFFFFFFu, bad);
        for (uint32_t i = 0; i < found && !bad; ++i)
            settle_long<MODE, HAS_VAL>(keys, vals, warps[warp].later[i], n, mask, desc != 0, &warps[warp], w, &ctrl->settle_fail, 1u);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) last = atomicAdd(&ctrl->settle_done, 1u) == gridDim.x - 1 ? 1u : 0u;
    __syncthreads();
    if (!last || !ld_relaxed(&ctrl->settle_fail)) return;
    // a group was too long to settle: the plain passes, over every digit, from where the data stand
    // (the table of long groups is cleared for them)
    for (uint64_t i = tid; i < status_bytes / 8 && i < kTakenRoom; i += THREADS)
        reinterpret_cast<unsigned long long *>(status + (KeyTraits<U>::kDigits - 1) * status_bytes)[i] = 0;
    if (tid != 0) return;
    const uint32_t digits = ctrl->survive & ((1u << KeyTraits<U>::kDigits) - 1u);
    uint32_t curk = end.dst_keys;
    const uint32_t done = plan_chain(ctrl, pa, ctrl->hot, digits, !pa.inplace, kPrefixSlots, HAS_VAL ? end.dst_vals : end.dst_keys,
                                     curk, false, false);
    plan_copy(ctrl, pa, done, false);
}

}  // namespace rsbd8g
