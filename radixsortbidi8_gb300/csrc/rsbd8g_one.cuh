// rsbd8g_one.cuh - sorts that fit the chip at once: one kernel runs the whole sort.
//
// Up to one tile per SM, a sort is bound by what surrounds its passes: a launch per digit with its
// plan to fetch, its tables to clear and its code to bring in took 10.5 us for a pass over a single
// tile.  Here every CTA keeps one tile for the whole sort.  It loads its keys once, adds its digit
// counts to the histograms, and runs the surviving passes in a loop: rank (TileRank), look back over
// the CTAs before it, stage, write out; a grid barrier lies between two passes.  A sort of one tile
// has no barrier and no look-back, and its keys stay in shared memory between the passes.
//   CTAs wait for one another, so more than one of them is a cooperative launch; every wait is bounded.
#pragma once
#include "rsbd8g_kernels.cuh"

namespace rsbd8g {

struct OneArgs {
    uint64_t n;
    uint64_t spin_limit_ns;
    uint32_t inplace, to_buffer, rev, dmask;   // as PlanArgs
    int32_t level;                             // indirect: where the key lies (k_gather_histogram)
    int64_t off1, off2;
    const void *keys_in;
};

template <typename U, bool HAS_VAL, int THREADS, int ITEMS>
struct OneSmem {
    static constexpr int kTile = THREADS * ITEMS;
    static constexpr int kUnits = THREADS / 16;          // ranking units (half-warps)
    static constexpr int kShare = THREADS / kBuckets;    // threads per digit
    static constexpr int kDigits = KeyTraits<U>::kDigits;
    static constexpr size_t kOffV = size_t(kTile) * sizeof(U);
    static constexpr size_t kOffTab = kOffV + (HAS_VAL ? size_t(kTile) * 8 : 0);          // u32: the TileRank table
    static constexpr size_t kOffPart = kOffTab + size_t(kUnits) * kBuckets * 4;            // u32 [kShare][256]
    static constexpr size_t kOffBst = kOffPart + size_t(kShare) * kBuckets * 4;                         // u32 [digits][256]
    static constexpr size_t kOffGofs = kOffBst + size_t(kDigits) * kBuckets * 4;           // i32 [256]
    static constexpr size_t kOffTs = kOffGofs + kBuckets * 4;                              // u32 [256]
    static constexpr size_t kOffMisc = kOffTs + kBuckets * 4;                              // u32 [64]
    static constexpr size_t kBytes = kOffMisc + 256;
    // counters per bin while the digits are counted (a lane class each, as in k_histogram)
    static constexpr int kFit = kUnits / kDigits;
    static constexpr int kCopies = kFit >= 32 ? 32 : kFit >= 16 ? 16 : kFit >= 8 ? 8 : kFit >= 4 ? 4 : 2;
    static_assert(kCopies * kDigits <= kUnits, "the counters fit the ranking table");
};

// every CTA of the grid arrives, and none leaves before all have (a bounded wait: false on a timeout)
__device__ __forceinline__ bool one_barrier(Control *ctrl, uint32_t target, uint64_t limit, uint32_t *flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&ctrl->hist_done, 1u);
        uint64_t t0 = 0;
        uint32_t ok = 1;
        for (uint32_t spins = 1; ld_relaxed(&ctrl->hist_done) < target; ++spins) {
            if (spins % 64u) continue;
            const uint64_t now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > limit) {
                atomicOr(&ctrl->error, kDevTimeout);
                ok = 0;
                break;
            }
        }
        __threadfence();
        *flag = ok;
    }
    __syncthreads();
    return *flag != 0;
}

constexpr int kOneGroup = 16;      // CTAs whose counts are summed one by one

// the sum of digit d's words of rows [j, e) of `rows`, this thread's share of them (one in SHARE); words
// of another epoch are not published yet and are waited for (a bounded wait)
template <int SHARE, int MOST>
__device__ __forceinline__ uint32_t one_sum(const uint32_t *rows, int j, int e, int share, int d, uint32_t epoch, uint64_t limit,
                                            Control *ctrl, uint32_t *bad) {
    constexpr int W = MOST / SHARE;
    uint64_t t0 = 0;
    for (uint32_t spins = 1;; ++spins) {
        uint32_t w[W], sum = 0;
        bool all = true;
#pragma unroll
        for (int q = 0; q < W; ++q) {
            const int r = j + share + q * SHARE;
            w[q] = r < e ? ld_relaxed(rows + r * kBuckets + d) : epoch << 24;
        }
#pragma unroll
        for (int q = 0; q < W; ++q) {
            all = all && (w[q] >> 24) == epoch;
            sum += w[q] & ((1u << 24) - 1u);
        }
        if (all) return sum;
        if (spins % 16u == 0) {
            const uint64_t now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > limit) {
                atomicOr(&ctrl->error, kDevTimeout);
                *bad = 1u;
                return 0;
            }
        }
    }
}

// the sum of the shares of digit d, in the threads of share 0
template <int SHARE>
__device__ __forceinline__ uint32_t one_fold(uint32_t *part, uint32_t v, int tid, int d) {
    __syncthreads();                     // (part has been read)
    part[tid] = v;
    __syncthreads();
#pragma unroll
    for (int q = 1; q < SHARE; ++q) v += tid < kBuckets ? part[q * kBuckets + d] : 0u;
    return v;
}

template <typename U, int MODE, bool HAS_VAL, int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS, 1)
    k_sort_one(Control *ctrl, const SortArrays arrs, uint32_t *hist, uint32_t *status, const OneArgs a) {
    using L = OneSmem<U, HAS_VAL, THREADS, ITEMS>;
    using R = TileRank<THREADS, ITEMS, 16>;
    constexpr int P = L::kDigits, TILE = L::kTile, SHARE = L::kShare;
    constexpr int PM = HAS_VAL ? 0 : MODE;             // gathered keys are filtered (and complemented) already
    extern __shared__ __align__(16) unsigned char smem[];
    U *stage = reinterpret_cast<U *>(smem);
    uint64_t *stage_v = reinterpret_cast<uint64_t *>(smem + L::kOffV);
    uint32_t *tab = reinterpret_cast<uint32_t *>(smem + L::kOffTab);
    uint32_t *part = reinterpret_cast<uint32_t *>(smem + L::kOffPart);
    uint32_t *bst = reinterpret_cast<uint32_t *>(smem + L::kOffBst);
    int32_t *gofs = reinterpret_cast<int32_t *>(smem + L::kOffGofs);
    uint32_t *tsx = reinterpret_cast<uint32_t *>(smem + L::kOffTs);
    uint32_t *misc = reinterpret_cast<uint32_t *>(smem + L::kOffMisc);   // [0..31] scan [32] barrier [33] bad [40..55] skip
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int share = tid >> 8, d = tid & (kBuckets - 1);                // SHARE threads per digit
    const uint32_t G = gridDim.x, cta = blockIdx.x;
    const uint32_t n = uint32_t(a.n);
    const uint32_t base = cta * uint32_t(TILE);
    const uint32_t tvalid = n - base < uint32_t(TILE) ? n - base : uint32_t(TILE);
    const uint32_t dm = HAS_VAL ? 0u : a.dmask;
    const uint32_t slot0 = R::slot0();
    if (G == 1 && tid == 0 && ctrl) ctrl->error = 0;
    uint32_t bar = 0;

    // ---- load the tile, count every digit
    U keys[ITEMS];
    uint64_t vals[HAS_VAL ? ITEMS : 1];
    for (int i = tid; i < P * kBuckets * L::kCopies; i += THREADS) tab[i] = 0u;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const uint32_t slot = slot0 + uint32_t(i) * 16u, x = a.rev ? n - 1u - (base + slot) : base + slot;
        keys[i] = KeyTraits<U>::fill();
        if constexpr (HAS_VAL) vals[i] = 0;
        if (slot < tvalid) {
            if constexpr (HAS_VAL) {
                vals[i] = static_cast<const uint64_t *>(arrs.p[kArrIn])[x];
                U raw;
                if (a.level == 3) {
                    raw = static_cast<const U *>(a.keys_in)[x];
                } else {
                    const unsigned char *obj = reinterpret_cast<const unsigned char *>(vals[i]) + a.off1;
                    if (a.level == 2) obj = load_ptr(obj) + a.off2;
                    raw = load_member<U>(obj);
                }
                keys[i] = a.dmask ? key_not(filter_key<MODE>(raw)) : filter_key<MODE>(raw);
            } else {
                keys[i] = static_cast<const U *>(arrs.p[kArrIn])[x];
            }
        }
    }
    __syncthreads();
    {
        uint32_t *c = tab + (lane & (L::kCopies - 1));
#pragma unroll
        for (int i = 0; i < ITEMS; ++i) {
            if (slot0 + uint32_t(i) * 16u >= tvalid) continue;
            const U k = filter_key<PM>(keys[i]);
#pragma unroll
            for (int p = 0; p < P; ++p) atomicAdd(c + (p * kBuckets + (digit_of(k, p) ^ dm)) * L::kCopies, 1u);
        }
    }
    __syncthreads();
    for (int i = tid; i < P * kBuckets; i += THREADS) {
        uint32_t t = 0;
#pragma unroll
        for (int c = 0; c < L::kCopies; ++c) t += tab[i * L::kCopies + ((c + i) & (L::kCopies - 1))];
        if (G == 1) bst[i] = t;
        else if (t) atomicAdd(hist + i, t);
    }
    if (G > 1) {
        if (!one_barrier(ctrl, bar += G, a.spin_limit_ns, misc + 32)) return;
        for (int i = tid; i < P * kBuckets; i += THREADS) bst[i] = __ldcg(hist + i);
    }
    __syncthreads();
    // bucket starts of every digit (256 threads a digit), and the pass-skip test
    if (tid < kMaxPasses) misc[40 + tid] = 0u;
    for (int i = tid; i < L::kUnits * kBuckets; i += THREADS) tab[i] = 0u;
    for (int p0 = 0; p0 < P; p0 += SHARE) {
        const int p = p0 + share;
        uint32_t c = 0, x = 0;
        __syncthreads();
        if (p < P) {
            c = x = bst[p * kBuckets + d];
            if (c == n) misc[40 + p] = 1u;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) misc[warp] = x;
        }
        __syncthreads();
        if (p < P) {
            uint32_t before = 0;
            for (int w = share * 8; w < warp; ++w) before += misc[w];
            bst[p * kBuckets + d] = before + x - c;
        }
    }
    __syncthreads();
    uint32_t survive = 0;
    for (int p = 0; p < P; ++p) survive |= misc[40 + p] ? 0u : 1u << p;
    const int k = __popc(survive);
    if (tid == 0) misc[33] = 0u;

    // ---- the passes
    const uint32_t target = a.inplace ? (a.to_buffer ? kArrBuf : kArrIn) : kArrOut;   // where the result goes
    uint32_t cur = kArrIn, curk = kArrKeysA;
    bool bad_arr = false;
    int i = 0;
    for (uint32_t m = survive; m; m &= m - 1) {
        const int p = __ffs(m) - 1;
        ++i;
        const bool last = i == k;
        const uint32_t dst = last ? target : a.inplace ? (cur == kArrIn ? kArrBuf : kArrIn) : ((k - i) % 2 == 0 ? kArrOut : kArrBuf);
        if (i > 1) {           // (the first pass sorts the keys as they were loaded)
            if (G == 1) {
#pragma unroll
                for (int q = 0; q < ITEMS; ++q) {
                    keys[q] = stage[slot0 + uint32_t(q) * 16u];
                    if constexpr (HAS_VAL) vals[q] = stage_v[slot0 + uint32_t(q) * 16u];
                }
            } else {
                const U *sk = static_cast<const U *>(sort_array(arrs, HAS_VAL ? curk : cur, kArrBuf, &bad_arr));
                const uint64_t *sv = static_cast<const uint64_t *>(sort_array(arrs, cur, kArrBuf, &bad_arr));
#pragma unroll
                for (int q = 0; q < ITEMS; ++q) {
                    const uint32_t slot = slot0 + uint32_t(q) * 16u;
                    keys[q] = KeyTraits<U>::fill();
                    if (slot < tvalid) {
                        keys[q] = ld_l2(sk + base + slot);
                        if constexpr (HAS_VAL) vals[q] = __ldcg(reinterpret_cast<const unsigned long long *>(sv + base + slot));
                    }
                }
            }
        }
        uint32_t rk[R::kRankRegs];
        R::template rank<PM, 0, false>(keys, rk, tab, slot0, tvalid, p, dm);
        __syncthreads();
        // the digit's count: 16 units per thread
        uint32_t *mine = tab + share * 16 * kBuckets;
        part[tid] = R::template total_of<0, 16>(mine, d);
        __syncthreads();
        uint32_t part_total = 0;
        if (share == 0) {
            uint32_t run = 0;
#pragma unroll
            for (int q = 0; q < SHARE; ++q) run += part[q * kBuckets + d];
            part_total = run;
            if (G > 1) st_relaxed(status + cta * kBuckets + d, (uint32_t(i) << 24) | run);
            uint32_t x = run;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) misc[warp] = x;
            tsx[d] = x - run;
        }
        __syncthreads();
        uint32_t ts = tsx[d];
        for (int w = 0; w < (d >> 5); ++w) ts += misc[w];
        {
            uint32_t at = ts;
            for (int q = 0; q < share; ++q) at += part[q * kBuckets + d];
            R::template offsets_of<0, 16>(mine, d, at);
        }
        if (G > 1) {
            // The digit's keys in the CTAs before this one: the counts of those in its group of 16, and the
            // totals of the groups before, which the last CTA of a group publishes.  All publish at about
            // the same time, so these are two rounds of loads in flight together; a walk along a chain of
            // inclusive counts waits for itself, and the sum over every CTA is bound by L2 (7,500 and
            // 6,400 cycles a pass for 128 CTAs).
            const int g0 = int(cta) & ~(kOneGroup - 1);
            uint32_t excl = one_sum<SHARE, kOneGroup>(status, g0, int(cta), share, d, uint32_t(i), a.spin_limit_ns, ctrl, misc + 33);
            excl = one_fold<SHARE>(part, excl, tid, d);
            uint32_t *totals = status + G * kBuckets;
            if (share == 0 && (cta & (kOneGroup - 1)) == kOneGroup - 1)
                st_relaxed(totals + cta / kOneGroup * kBuckets + d, (uint32_t(i) << 24) | (excl + part_total));
            if (g0 > 0) {
                const uint32_t more = one_sum<SHARE, kOneGroup>(totals, 0, g0 / kOneGroup, share, d, uint32_t(i), a.spin_limit_ns, ctrl, misc + 33);
                excl += one_fold<SHARE>(part, more, tid, d);
            }
            if (share == 0) gofs[d] = int32_t(bst[p * kBuckets + d] + excl) - int32_t(ts);
        } else if (share == 0) {
            gofs[d] = int32_t(bst[p * kBuckets + d]) - int32_t(ts);
        }
        __syncthreads();
        if (misc[33]) return;
        const uint32_t *urow = R::row(tab);
#pragma unroll
        for (int q = 0; q < ITEMS; ++q) {
            if (slot0 + uint32_t(q) * 16u >= tvalid) continue;
            const uint32_t dg = R::template digit_of_item<PM>(rk, q, keys[q], slot0 + uint32_t(q) * 16u, tvalid, p, dm);
            const uint32_t pos = *R::word(urow, dg) + R::rank_of(rk, q);
            stage[pos] = keys[q];
            if constexpr (HAS_VAL) stage_v[pos] = vals[q];
        }
        R::clear_own(tab);
        __syncthreads();
        // a result that goes where the last pass read from is written once every tile has been read
        if (G > 1 && last && dst == cur && !one_barrier(ctrl, bar += G, a.spin_limit_ns, misc + 32)) return;
        if (G > 1 || last) {
            const uint32_t dk = curk == kArrKeysA ? kArrKeysB : kArrKeysA;
            U *out_k = HAS_VAL && last ? nullptr : static_cast<U *>(sort_array(arrs, HAS_VAL ? dk : dst, kArrBuf, &bad_arr));
            uint64_t *out_v = static_cast<uint64_t *>(sort_array(arrs, dst, kArrBuf, &bad_arr));
#pragma unroll
            for (int q = 0; q < ITEMS; ++q) {
                const uint32_t s = uint32_t(tid) + uint32_t(q) * THREADS;
                if (s < tvalid) {
                    const U kk = stage[s];
                    const uint32_t g = uint32_t(*tile_offset<PM>(gofs, kk, p, dm) + int32_t(s));
                    if (g < n) {
                        if (!HAS_VAL || !last) out_k[g] = kk;
                        if constexpr (HAS_VAL) out_v[g] = stage_v[s];
                    } else if (ctrl) {
                        atomicOr(&ctrl->error, kDevFault);
                    }
                }
            }
            cur = dst;
            curk = dk;
        }
        if (G > 1 && !last && !one_barrier(ctrl, bar += G, a.spin_limit_ns, misc + 32)) return;
    }
    if (k == 0 && (target != kArrIn || a.rev)) {       // every digit skipped: the keys in the order they were loaded
        if (G > 1 && target == kArrIn && !one_barrier(ctrl, bar += G, a.spin_limit_ns, misc + 32)) return;
        __syncthreads();
        void *out = sort_array(arrs, target, kArrBuf, &bad_arr);
#pragma unroll
        for (int q = 0; q < ITEMS; ++q) {
            const uint32_t slot = slot0 + uint32_t(q) * 16u;
            if (slot < tvalid) {
                if constexpr (HAS_VAL) static_cast<uint64_t *>(out)[base + slot] = vals[q];
                else static_cast<U *>(out)[base + slot] = keys[q];
            }
        }
    }
}

}  // namespace rsbd8g
