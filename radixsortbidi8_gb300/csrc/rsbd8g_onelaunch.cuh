// rsbd8g_onelaunch.cuh - host side of the one-kernel sorts (rsbd8g_one.cuh), templated on the key type;
// each rsbd8g_one_k*.cu instantiates it for one key size.
//
// A sort of one tile is one launch; more tiles take a memset of the control block, the histograms and
// the look-back words, and a cooperative launch (the CTAs wait for one another).
#pragma once
#include <algorithm>
#include <mutex>

#include "rsbd8g_internal.h"
#include "rsbd8g_one.cuh"

namespace rsbd8g {

constexpr uint64_t kOneMaxKeys = uint64_t(1) << 22;     // 24-bit counts in the look-back words

// The tile sizes of a key type, smallest first: threads x keys (0 keys: no such size), as shared memory
// and the 64 registers of a thread allow.  The smallest has half the ranking units, whose table is what
// a pass over few keys spends its time on.
struct OneShape {
    int threads, items;
};
constexpr uint64_t kOneFew = 64;     // tiles of the smallest size
constexpr OneShape one_shape(int key_bytes, bool indirect, int i) {
    return i == 0   ? OneShape{512, 4}
           : i == 1 ? OneShape{1024, 4}
           : i == 2 ? OneShape{1024, key_bytes == 16 ? 0 : 8}
                    : OneShape{1024, !indirect && key_bytes <= 4 ? 16 : 0};
}

static_assert(kOneTileKeys == 1024 * 4, "the larger of the two sizes that sort in one tile");

// set the kernel up on device `dev` (which also loads it); returns the CTAs that fit the device at once
template <typename U, int MODE, bool HAS_VAL, int SHAPE>
uint64_t one_setup(int dev) {
    static std::once_flag once[64];
    static uint64_t fit[64];
    std::call_once(once[dev & 63], [&] {
        constexpr OneShape sh = one_shape(int(sizeof(U)), HAS_VAL, SHAPE);
        using L = OneSmem<U, HAS_VAL, sh.threads, sh.items>;
        auto kern = k_sort_one<U, MODE, HAS_VAL, sh.threads, sh.items>;
        int b = 0;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(L::kBytes)) == cudaSuccess &&
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, sh.threads, L::kBytes) == cudaSuccess && b > 0)
            fit[dev & 63] = uint64_t(device_sms(dev));      // one CTA per SM
        else
            (void)cudaGetLastError();
    });
    return fit[dev & 63];
}

struct OneCall {
    uint64_t n;
    unsigned char *scratch;
    size_t scratch_bytes;
    SortArrays arrs;
    OneArgs args;
    cudaStream_t s;
};

// launch with at most `most` tiles of shape SHAPE; false when they do not fit (nothing launched)
template <typename U, int MODE, bool HAS_VAL, int SHAPE>
bool launch_one_shape(const OneCall &c, uint64_t most, cudaError_t *e) {
    constexpr OneShape sh = one_shape(int(sizeof(U)), HAS_VAL, SHAPE);
    if constexpr (sh.items == 0) {
        return false;
    } else {
        using L = OneSmem<U, HAS_VAL, sh.threads, sh.items>;
        const uint64_t tiles = (c.n + L::kTile - 1) / L::kTile;
        const size_t hist = 1024, status = hist + size_t(L::kDigits) * kBuckets * 4;
        const size_t used = status + size_t(tiles + tiles / kOneGroup) * kBuckets * 4;
        int dev = 0;
        cudaGetDevice(&dev);
        if ((tiles > 1 && used > c.scratch_bytes) || tiles > most || tiles > one_setup<U, MODE, HAS_VAL, SHAPE>(dev)) return false;
        if (tiles > 1) {
            LaunchTimer t(c.s, RSBD8G_KERNEL_MEMSET, uint32_t(sizeof(U)), 0, c.n);
            if ((*e = cudaMemsetAsync(c.scratch, 0, used, c.s)) != cudaSuccess) return true;
        }
        LaunchTimer t(c.s, RSBD8G_KERNEL_ONE, uint32_t(sizeof(U)), 0, c.n);
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(uint32_t(tiles));
        cfg.blockDim = dim3(sh.threads);
        cfg.dynamicSmemBytes = L::kBytes;
        cfg.stream = c.s;
        cfg.attrs = &at;
        cfg.numAttrs = tiles > 1 ? 1 : 0;
        *e = cudaLaunchKernelEx(&cfg, k_sort_one<U, MODE, HAS_VAL, sh.threads, sh.items>, reinterpret_cast<Control *>(c.scratch), c.arrs,
                                tiles > 1 ? reinterpret_cast<uint32_t *>(c.scratch + hist) : nullptr,
                                tiles > 1 ? reinterpret_cast<uint32_t *>(c.scratch + status) : nullptr, c.args);
        if (*e == cudaErrorCooperativeLaunchTooLarge || *e == cudaErrorNotSupported) {
            // a context that may not use every SM: the launches per digit need no CTAs side by side
            (void)cudaGetLastError();
            *e = cudaSuccess;
            return false;
        }
        return true;
    }
}

template <typename U, int MODE, bool HAS_VAL>
bool launch_one_mode(const OneCall &c, cudaError_t *e) {
    // One tile of up to 4096 keys: its passes need no barrier (4096 uint32 keys 18 us, int64 33 us; one tile
    // of 8192 keys took 25 and 49 us where two to four of 2048 take 24 and 44).  Then the smallest tiles
    // that fit the SMs, those of 2048 keys while there are few: a pass spends more time on a tile's keys
    // than on looking back over more CTAs (2^19 int64 keys as 128 tiles of 4096: 70 us, 64 of 8192: 94 us).
    // Past the largest the launch per digit takes over: those sorts fill the SMs several times.
    // Whole sorts, a launch per digit against one kernel: uint32 2^10 55 -> 12 us (the caller's Python
    // included), 2^18 61 -> 37, 2^20 66 -> 45, 2^21 87 -> 60; int64 2^14 106 -> 49, 2^20 137 -> 91.
    return launch_one_shape<U, MODE, HAS_VAL, 0>(c, 1, e) || launch_one_shape<U, MODE, HAS_VAL, 1>(c, 1, e) ||
           launch_one_shape<U, MODE, HAS_VAL, 0>(c, kOneFew, e) ||
           launch_one_shape<U, MODE, HAS_VAL, 1>(c, ~uint64_t(0), e) ||
           launch_one_shape<U, MODE, HAS_VAL, 2>(c, ~uint64_t(0), e) ||
           launch_one_shape<U, MODE, HAS_VAL, 3>(c, ~uint64_t(0), e);
}

// Run the sort as one kernel if it fits; false (nothing launched) if it does not.  A sort of one tile may
// come without scratch and buffer.
template <typename U>
bool launch_one_t(const Resolved &r, uint64_t n, unsigned char *scratch, size_t scratch_bytes, const void *in, void *out,
                  void *buf, const Layout &L, bool inplace, bool to_buffer, cudaStream_t s, cudaError_t *e) {
    if (n >= kOneMaxKeys || (r.flags & (RSBD8G_FLAG_DIAG_STALL | RSBD8G_FLAG_DIAG_LAUNCHES))) return false;
    OneCall c{};
    c.n = n;
    c.scratch = scratch;
    c.scratch_bytes = r.indirect ? L.keys_a : scratch_bytes;
    c.s = s;
    c.arrs.p[kArrIn] = in;
    c.arrs.p[kArrOut] = out;
    c.arrs.p[kArrBuf] = buf;
    if (scratch && r.indirect) {
        c.arrs.p[kArrKeysA] = scratch + L.keys_a;
        c.arrs.p[kArrKeysB] = scratch + L.keys_b;
    }
    c.args.n = n;
    c.args.spin_limit_ns = 1000000000ull;
    c.args.inplace = inplace;
    c.args.to_buffer = to_buffer;
    c.args.rev = r.rev;
    c.args.dmask = r.f.desc ? 0xFFu : 0u;
    c.args.level = int(r.indirect);
    c.args.off1 = r.off1;
    c.args.off2 = r.off2;
    c.args.keys_in = r.keys;
    const int mode = int(r.f.absv | (r.f.sign << 1) | (r.f.fltp << 2));
    bool done = false;
#define RSBD8G_ONE(M) done = r.indirect ? launch_one_mode<U, M, true>(c, e) : launch_one_mode<U, M, false>(c, e)
    RSBD8G_MODE_SWITCH(mode, RSBD8G_ONE)
#undef RSBD8G_ONE
    return done;
}

// load and set up the kernels that launch_one_t can launch for r
template <typename U, int MODE, bool HAS_VAL>
void prepare_one_mode(int dev) {
    one_setup<U, MODE, HAS_VAL, 0>(dev);
    one_setup<U, MODE, HAS_VAL, 1>(dev);
    if constexpr (one_shape(int(sizeof(U)), HAS_VAL, 2).items != 0) one_setup<U, MODE, HAS_VAL, 2>(dev);
    if constexpr (one_shape(int(sizeof(U)), HAS_VAL, 3).items != 0) one_setup<U, MODE, HAS_VAL, 3>(dev);
}
template <typename U>
cudaError_t prepare_one_t(const Resolved &r) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const int mode = int(r.f.absv | (r.f.sign << 1) | (r.f.fltp << 2));
#define RSBD8G_PREP(M) r.indirect ? prepare_one_mode<U, M, true>(dev) : prepare_one_mode<U, M, false>(dev)
    RSBD8G_MODE_SWITCH(mode, RSBD8G_PREP)
#undef RSBD8G_PREP
    return cudaGetLastError();
}

}  // namespace rsbd8g

#define RSBD8G_DEFINE_ONE(name, U)                                                                             \
    namespace rsbd8g {                                                                                         \
    bool name(const Resolved &r, uint64_t n, unsigned char *scratch, size_t scratch_bytes, const void *in,     \
              void *out, void *buf, const Layout &L, bool inplace, bool to_buffer, cudaStream_t s,             \
              cudaError_t *e) {                                                                                \
        return launch_one_t<U>(r, n, scratch, scratch_bytes, in, out, buf, L, inplace, to_buffer, s, e);       \
    }                                                                                                          \
    cudaError_t name##_prepare(const Resolved &r) { return prepare_one_t<U>(r); }                              \
    }
