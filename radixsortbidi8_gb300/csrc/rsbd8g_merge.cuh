// rsbd8g_merge.cuh - stable merge of sorted runs on the device (the reference's mergehalves* /
// mergethirds*, Radixsortbidi8.hpp:54437-56418).
//
// Two runs A and B, each sorted by the same descriptor, merge into one stably sorted array: an
// element of A goes before an element of B when its filtered key orders first, and on equal keys
// when A has precedence -- the earlier run in forward order, the later run under isrevorder (the
// reference walks its halves from the top and swaps their roles for isrevorder,
// Radixsortbidi8.hpp:54453-54456).  Three runs are merged as (A merge B) merge C through a buffer,
// which gives the same order as the reference's three-way walk (:55381-55386).
//
// k_merge2: persistent CTAs, each writing one contiguous range of the output (see the kernel).
// No scratch memory.
#pragma once
#include "rsbd8g_device.cuh"

namespace rsbd8g {

// the filtered key of raw bits in the order of the sort: complemented for descending sorts
template <int MODE, typename U>
__host__ __device__ __forceinline__ U order_key(U b, bool desc) {
    const U k = filter_key<MODE>(b);
    return desc ? key_not(k) : k;
}

// does a (from run A) go before b (from run B)?  a_first: A has precedence on equal keys
template <int MODE, typename U>
__host__ __device__ __forceinline__ bool a_before_b(U a, U b, bool desc, bool a_first) {
    const U ka = order_key<MODE>(a, desc), kb = order_key<MODE>(b, desc);
    return a_first ? !key_less(kb, ka) : key_less(ka, kb);
}

// elements of A among the first d elements of the merge of A[0, na) and B[0, nb), found by one
// warp (all 32 lanes call it with the same arguments): each round probes 32 points of the interval
// holding the answer and keeps the gap between the last true and the first false probe, so a
// search over n elements takes about log32(n) dependent loads instead of log2(n)
template <int MODE, typename U>
__device__ __forceinline__ uint64_t merge_path_warp(const U *A, uint64_t na, const U *B, uint64_t nb, uint64_t d,
                                                    bool desc, bool a_first) {
    uint64_t lo = d > nb ? d - nb : 0, hi = d < na ? d : na;      // the answer lies in [lo, hi]
    const uint32_t lane = threadIdx.x & 31u;
    while (hi - lo > 32) {
        const uint64_t p = lo + (hi - lo) * (lane + 1) / 33;      // 32 increasing points of (lo, hi)
        const bool t = a_before_b<MODE>(A[p], B[d - 1 - p], desc, a_first);
        const int k = __popc(__ballot_sync(0xFFFFFFFFu, t));     // the true probes are a prefix
        const uint64_t below = __shfl_sync(0xFFFFFFFFu, p, k > 0 ? k - 1 : 0);
        const uint64_t above = __shfl_sync(0xFFFFFFFFu, p, k < 32 ? k : 31);
        if (k > 0) lo = below + 1;
        if (k < 32) hi = above;
    }
    const uint64_t p = lo + lane;
    const bool t = p < hi && a_before_b<MODE>(A[p], B[d - 1 - p], desc, a_first);
    return lo + uint64_t(__popc(__ballot_sync(0xFFFFFFFFu, t)));
}

// Tiles of kTile outputs, THREADS x kItems: an odd number of outputs per thread, so that the threads'
// runs of outputs lie in different banks, and one item fewer than the window holds per thread, so that a
// window cut at a 16-byte boundary still holds every element a tile can take.
template <typename U, int THREADS>
struct MergeShape {
    static constexpr int kItems = sizeof(U) >= 16 ? 3 : (sizeof(U) == 8 ? 7 : 15);
    static constexpr int kTile = THREADS * kItems;
    static constexpr uint32_t kWin = uint32_t(THREADS * (kItems + 1));    // elements of one run's window
    static constexpr uint32_t kVec = 16 / sizeof(U);                      // elements of a 16-byte load
    static_assert((kWin & (kWin - 1)) == 0, "the windows are circular buffers of a power of two");
    static constexpr size_t kOffOut = 2 * size_t(kWin) * sizeof(U);
    static constexpr size_t kOffMisc = kOffOut + size_t(kTile) * sizeof(U);
    static constexpr size_t kBytes = kOffMisc + 64;
};

// elements of A among the first d of the merge of the windows: element x of the A window is
// w[(a0 + x) % kWin], of the B window w[kWin + (b0 + x) % kWin]; they hold na and nb elements
template <int MODE, uint32_t WIN, typename U>
__device__ __forceinline__ uint32_t merge_path_window(const U *w, uint32_t a0, uint32_t na, uint32_t b0, uint32_t nb,
                                                      uint32_t d, bool desc) {
    uint32_t lo = d > nb ? d - nb : 0, hi = d < na ? d : na;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a_before_b<MODE>(w[(a0 + mid) & (WIN - 1)], w[WIN | ((b0 + d - 1 - mid) & (WIN - 1))], desc, true)) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Persistent merge, A first on equal keys: CTA c writes the outputs [c * per, (c + 1) * per) tile by
// tile.  One warp finds where the range starts on the merge path; from there the CTA keeps a window of the
// next kWin elements of A and of B in circular shared-memory buffers.  Per tile every thread finds where
// its outputs start (a search in the windows) and merges them one by one; the elements that slide into
// the windows are loaded, the tile is stored, and the loaded elements replace the consumed ones.  Every
// element is read from global memory once.
//   What bounds it is instructions: an output costs the comparison, the choice of key and place, and one
// load from the side that advanced (the two windows are one array, so the side is a bit of the index);
// while both windows hold more than a tile there are no ends to check, and global loads, window
// stores and output stores move 16 bytes.  2^28 uint32 keys in halves: 0.82 -> 0.58 ms, int64 1.34 -> 1.12 ms; with the
// sides as two branches, ends checked at every output and elements moved one by one, 105 instructions an
// output instead of 52.
template <typename U, int MODE, int THREADS>
__global__ void __launch_bounds__(THREADS) k_merge2(const U *__restrict__ A, uint64_t na, const U *__restrict__ B,
                                                    uint64_t nb, U *__restrict__ out, uint32_t desc, uint64_t per) {
    using L = MergeShape<U, THREADS>;
    constexpr int TILE = L::kTile, ITEMS = L::kItems;
    constexpr uint32_t WIN = L::kWin, M = WIN - 1, V = L::kVec;
    extern __shared__ __align__(16) unsigned char smem[];
    U *w = reinterpret_cast<U *>(smem);                       // the A window, then the B window
    U *sout = reinterpret_cast<U *>(smem + L::kOffOut);
    uint64_t *misc = reinterpret_cast<uint64_t *>(smem + L::kOffMisc);   // [0] range start split [1] tile split
    const uint64_t total = na + nb;
    uint64_t o = uint64_t(blockIdx.x) * per;
    if (o >= total) return;
    const uint64_t oend = o + per < total ? o + per : total;
    const bool dsc = desc != 0;
    const int tid = threadIdx.x;
    // element i of a run lies at slot (i + its run's misalignment) % WIN, so 16-byte blocks stay whole
    const uint32_t ma = uint32_t(reinterpret_cast<uintptr_t>(A) / sizeof(U)) % V, mb = uint32_t(reinterpret_cast<uintptr_t>(B) / sizeof(U)) % V;
    const bool out16 = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
    // where the window of a run of n elements that starts at i ends: the run's end or a 16-byte boundary
    auto window_end = [](uint64_t i, uint64_t n, uint32_t mis) {
        const uint64_t e = i + WIN;
        return e < n ? e - (e + mis) % V : n;
    };
    if (tid < 32) {
        const uint64_t sp = merge_path_warp<MODE>(A, na, B, nb, o, dsc, true);
        if (tid == 0) misc[0] = sp;
    }
    __syncthreads();
    uint64_t ia = misc[0], ib = o - ia;
    uint64_t aend = window_end(ia, na, ma), bend = window_end(ib, nb, mb);
    for (uint64_t x = ia + tid; x < aend; x += THREADS) w[uint32_t(x + ma) & M] = A[x];
    for (uint64_t x = ib + tid; x < bend; x += THREADS) w[WIN | (uint32_t(x + mb) & M)] = B[x];
    __syncthreads();
    while (o < oend) {
        const uint32_t r = uint32_t(oend - o < uint64_t(TILE) ? oend - o : uint64_t(TILE));
        const uint32_t ca = uint32_t(aend - ia), cb = uint32_t(bend - ib);       // elements in the windows
        const uint32_t a0 = uint32_t(ia + ma) & M, b0 = uint32_t(ib + mb) & M;
        const uint32_t d0 = uint32_t(tid) * ITEMS;
        if (d0 < r) {
            uint32_t xa = merge_path_window<MODE, WIN>(w, a0, ca, b0, cb, d0, dsc);
            uint32_t pa = (a0 + xa) & M, pb = WIN | ((b0 + d0 - xa) & M);
            U ua = w[pa], ub = w[pb];
            U ka = order_key<MODE>(ua, dsc), kb = order_key<MODE>(ub, dsc);
            if (r == uint32_t(TILE) && ca > uint32_t(TILE) && cb > uint32_t(TILE)) {
#pragma unroll
                for (int q = 0; q < ITEMS; ++q) {
                    const bool a = !key_less(kb, ka);
                    sout[d0 + q] = a ? ua : ub;
                    xa += a ? 1u : 0u;
                    uint32_t t = a ? pa : pb;
                    t = ((t + 1u) & M) | (t & WIN);
                    const U u = w[t], k = order_key<MODE>(u, dsc);
                    pa = a ? t : pa;
                    pb = a ? pb : t;
                    ua = a ? u : ua;
                    ub = a ? ub : u;
                    ka = a ? k : ka;
                    kb = a ? kb : k;
                }
                if (tid == THREADS - 1) misc[1] = xa;
            } else {                 // a window ends in this tile, or the range does
                const uint32_t cnt = r - d0 < uint32_t(ITEMS) ? r - d0 : uint32_t(ITEMS);
                uint32_t xb = d0 - xa;
                for (uint32_t q = 0; q < cnt; ++q) {
                    const bool a = xa < ca && (xb >= cb || !key_less(kb, ka));
                    sout[d0 + q] = a ? ua : ub;
                    if (a) {
                        ++xa;
                        ua = w[(a0 + xa) & M];
                        ka = order_key<MODE>(ua, dsc);
                    } else {
                        ++xb;
                        ub = w[WIN | ((b0 + xb) & M)];
                        kb = order_key<MODE>(ub, dsc);
                    }
                }
                if (d0 + cnt == r) misc[1] = xa;
            }
        }
        __syncthreads();
        const uint32_t sa = uint32_t(misc[1]);
        const uint64_t ia2 = ia + sa, ib2 = ib + (r - sa);
        // the elements that slide into the windows: whole 16-byte blocks (of both runs, shared out over the
        // threads), and at a run's end the elements after the last block
        const uint64_t aend2 = aend < na ? window_end(ia2, na, ma) : na, bend2 = bend < nb ? window_end(ib2, nb, mb) : nb;
        const uint32_t va = uint32_t(aend2 - aend) / V, vb = uint32_t(bend2 - bend) / V;
        const uint32_t ta = uint32_t(aend2 - aend) % V, tb = uint32_t(bend2 - bend) % V;
        constexpr int NV = (TILE / int(V) + 2 + THREADS - 1) / THREADS;
        uint4 blk[NV];
        U rest{};
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const uint32_t x = uint32_t(tid) + uint32_t(j) * THREADS;
            if (x < va + vb) blk[j] = *reinterpret_cast<const uint4 *>(x < va ? A + aend + x * V : B + bend + (x - va) * V);
        }
        if (uint32_t(tid) < ta) rest = A[aend + va * V + tid];
        else if (uint32_t(tid) >= V && uint32_t(tid) - V < tb) rest = B[bend + vb * V + (tid - V)];
        if (r == uint32_t(TILE) && out16) {
            const uint4 *so = reinterpret_cast<const uint4 *>(sout);
            uint4 *dst = reinterpret_cast<uint4 *>(out + o);
#pragma unroll
            for (int x = tid; x < TILE / int(V); x += THREADS) dst[x] = so[x];
        } else {
            for (uint32_t x = uint32_t(tid); x < r; x += THREADS) out[o + x] = sout[x];
        }
#pragma unroll
        for (int j = 0; j < NV; ++j) {
            const uint32_t x = uint32_t(tid) + uint32_t(j) * THREADS;
            if (x < va + vb)
                *reinterpret_cast<uint4 *>(x < va ? w + (uint32_t(aend + ma + x * V) & M)
                                                  : w + (WIN | (uint32_t(bend + mb + (x - va) * V) & M))) = blk[j];
        }
        if (uint32_t(tid) < ta) w[uint32_t(aend + ma + va * V + tid) & M] = rest;
        else if (uint32_t(tid) >= V && uint32_t(tid) - V < tb) w[WIN | (uint32_t(bend + mb + vb * V + (tid - V)) & M)] = rest;
        __syncthreads();
        o += r;
        ia = ia2;
        ib = ib2;
        aend = aend2;
        bend = bend2;
    }
}

}  // namespace rsbd8g
