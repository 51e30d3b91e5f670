// rsbd8g_internal.h - shared host-side declarations of the GB300 radix sort library.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <type_traits>

#include "rsbd8g.h"
#include "rsbd8g_device.cuh"

namespace rsbd8g {

// a descriptor after the reference's compile-time mode resolution
struct Resolved {
    Filter f;
    uint32_t rev;         // effective isrevorder
    uint32_t key_bytes;   // 1, 2, 4, 8, 16
    uint32_t x87;         // 16-byte x87 extended precision keys (10 digits)
    uint32_t digits;      // 8-bit digit passes of the key
    uint32_t elem_bytes;  // bytes per array element (key bytes, or 8 for object pointers)
    uint32_t indirect;    // RSBD8G_DIRECT / RSBD8G_MEMBER / RSBD8G_MEMBER2
    uint32_t flags;       // RSBD8G_FLAG_* of the descriptor (other bits of it mean nothing)
    uint32_t shared_gpu;  // a served batch: its kernels share the GPU with other streams'
    uint32_t prefetch;    // every array of the call is device memory (tiles may be prefetched into L2)
    int64_t off1, off2;
    const void *keys;     // RSBD8G_KEYED: the caller's key array
};

// A batch whose kernels share the GPU with other streams' (Resolved::shared_gpu) is not sorted by a prefix, as the
// launches that leaves idle would each wait for their CTAs' turn behind another stream's passes (29 mixed
// requests of up to 2^22 keys: 1.22-1.29 ms with them, 1.11 without; one large request alone still gains
// more than it waits: 48 requests of up to 2^24 keys 2.85 ms, 3.07 without).  The server's batches come in here:
rsbd8g_status segmented_shared_gpu(const rsbd8g_desc *desc, size_t total, size_t nsegs, const uint64_t *offsets,
                                   const uint64_t *input_ptrs, const uint64_t *output_ptrs, const uint64_t *buffer_ptrs,
                                   const uint8_t *directions, void *scratch, size_t scratch_bytes,
                                   const rsbd8g_segtuning *tuning, rsbd8g_stream stream);

// byte offsets of the parts of a scratch area
struct Layout {
    size_t ctrl, ghist, bstart, status, status_pass_bytes, zero_bytes, keys_a, keys_b, total;
    uint32_t num_tiles;
    bool wide_status;
    bool large_tiles;     // sweep_geometry_large applies
    bool small_tiles;     // sweep_geometry_small applies
};

// brackets one kernel launch with CUDA events on its stream while launch profiling is on
class LaunchTimer {
public:
    LaunchTimer(cudaStream_t s, uint32_t kernel, uint32_t key_bytes, uint32_t pass, uint64_t n);
    ~LaunchTimer();
    LaunchTimer(const LaunchTimer &) = delete;
    LaunchTimer &operator=(const LaunchTimer &) = delete;

private:
    cudaStream_t s_;
    cudaEvent_t a_, b_;
    rsbd8g_launch_record rec_{};
};

int device_sms(int dev);

// launch a kernel that calls after_previous(): it may start while the stream's previous kernel drains
template <typename... A>
cudaError_t launch_after(void (*kern)(A...), uint32_t grid, int threads, size_t smem, cudaStream_t s,
                         std::common_type_t<A>... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(unsigned(threads));
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kern, args...);
}

// the launch sequence of one sort, per key size (rsbd8g_sort_k{1,2,4,8}.cu)
#define RSBD8G_DECLARE_LAUNCH(name)                                                                          \
    cudaError_t name(const Resolved &r, uint64_t n, const Layout &L, unsigned char *scratch, const void *in, \
                     void *out, void *buf, bool inplace, bool to_buffer, cudaStream_t s);                   \
    cudaError_t name##_prepare(const Resolved &r);   /* load every kernel this sort can launch */
RSBD8G_DECLARE_LAUNCH(launch_sort_k1)
RSBD8G_DECLARE_LAUNCH(launch_sort_k2)
RSBD8G_DECLARE_LAUNCH(launch_sort_k4)
RSBD8G_DECLARE_LAUNCH(launch_sort_k8)
RSBD8G_DECLARE_LAUNCH(launch_sort_k16)
RSBD8G_DECLARE_LAUNCH(launch_sort_x87)

// the one-kernel sorts of small arrays, per key size (rsbd8g_one_k*.cu): false (nothing launched) when
// the sort does not fit one
#define RSBD8G_DECLARE_ONE(name)                                                                             \
    bool name(const Resolved &r, uint64_t n, unsigned char *scratch, size_t scratch_bytes, const void *in,   \
              void *out, void *buf, const Layout &L, bool inplace, bool to_buffer, cudaStream_t s,           \
              cudaError_t *e);                                                                               \
    cudaError_t name##_prepare(const Resolved &r);
RSBD8G_DECLARE_ONE(launch_one_k1)
RSBD8G_DECLARE_ONE(launch_one_k2)
RSBD8G_DECLARE_ONE(launch_one_k4)
RSBD8G_DECLARE_ONE(launch_one_k8)
RSBD8G_DECLARE_ONE(launch_one_k16)
RSBD8G_DECLARE_ONE(launch_one_x87)

// the largest sort that one tile holds (rsbd8g_onelaunch.cuh); such a sort uses neither scratch nor buffer
constexpr uint64_t kOneTileKeys = 4096;

// tile geometry of the onesweep passes, per key size (keys per tile = threads * items)
struct SweepGeometry {
    int threads, items;
};
constexpr SweepGeometry sweep_geometry(int key_bytes, bool indirect) {
    if (indirect) return SweepGeometry{512, key_bytes == 16 ? 6 : 8};
    return SweepGeometry{512, key_bytes == 16 ? 6 : (key_bytes == 8 ? 16 : 24)};
}
// Direct keys of up to 4 bytes take three tile sizes by the count of the sort (narrow look-back
// words only, under 2^30 keys): 512 x 32 from kLargeTileMinKeys keys on -- fewer tiles mean fewer
// per-tile phases and shorter look-back chains (uint32 2^28: -5 % against 512 x 24) -- 512 x 24 in
// between, and 512 x 16 below kSmallTileMaxKeys, where more tiles keep every SM busy and fill the
// pipelined pass sooner (uint32 2^20 / 2^21 / 2^22: -10 / -10 / -5 %).  The choice depends on the
// count alone, so a scratch size computed once fits every call of that count.
constexpr uint64_t kLargeTileMinKeys = uint64_t(1) << 25;
constexpr uint64_t kSmallTileMaxKeys = uint64_t(1) << 23;
// Sorts of 8- and 16-byte keys from this many keys on may run as prefix sorts (rsbd8g_prefix.cuh): below,
// the launches that a prefix sort leaves idle cost what the passes it saves do (8-byte keys 2^20: 137 us
// plain, 130-142 us by a prefix, and 91 us as one kernel; 2^21: 182 and 111-132 us; 128-bit 2^20: 320 and
// 137 us).
constexpr uint64_t prefix_min_keys(int key_bytes) { return uint64_t(1) << (key_bytes == 16 ? 20 : 21); }
constexpr SweepGeometry sweep_geometry_large(int key_bytes) {
    return key_bytes <= 4 ? SweepGeometry{512, 32} : sweep_geometry(key_bytes, false);
}
constexpr SweepGeometry sweep_geometry_small(int key_bytes) {
    return key_bytes <= 4 ? SweepGeometry{512, 16} : sweep_geometry(key_bytes, false);
}
// the segmented sort's large segments, two tile sizes per key size, picked per batch shape by the
// autotuner (rsbd8g_segtuning::large_variant).  Variant 0: 512 x 28 for keys up to 4 bytes (measured
// against 24 and 32 on the 2^28-key batch of uint32 arrays) and 512 x 12 for 8-byte keys, smaller
// than the plain sort's tiles because a segment's last tile is partly empty.  Variant 1: 512 x 20
// and 512 x 16, for batches of shorter or longer large segments.  16-byte keys: 512 x 6 in both.
constexpr int kSegLargeVariants = 2;
constexpr SweepGeometry seg_sweep_geometry(int key_bytes, int variant) {
    return SweepGeometry{512, key_bytes == 16 ? 6
                              : key_bytes == 8 ? (variant == 1 ? 16 : 12)
                                               : (variant == 1 ? 20 : 28)};
}

#define RSBD8G_MODE_SWITCH(mode, CALL) \
    switch (mode) {                    \
        case 0: CALL(0); break;        \
        case 1: CALL(1); break;        \
        case 2: CALL(2); break;        \
        case 3: CALL(3); break;        \
        case 4: CALL(4); break;        \
        case 5: CALL(5); break;        \
        case 6: CALL(6); break;        \
        default: CALL(7); break;       \
    }

// shapes of the small-segment block sort (threads x items = the largest small segment)
struct SegSmallShape {
    int threads, items;
};
constexpr SegSmallShape seg_small_shape(int key_bytes, int variant) {
    return key_bytes == 16 ? (variant == 0 ? SegSmallShape{256, 4} : variant == 1 ? SegSmallShape{256, 6} : SegSmallShape{512, 4})
         : key_bytes == 8 ? (variant == 0 ? SegSmallShape{256, 8} : variant == 1 ? SegSmallShape{256, 12} : SegSmallShape{512, 12})
                          : (variant == 0 ? SegSmallShape{256, 8} : variant == 1 ? SegSmallShape{256, 16} : SegSmallShape{512, 16});
}
constexpr int kSegSmallVariants = 3;

// byte offsets of the parts of a segmented-sort scratch area
struct SegLayout {
    size_t ctrl, large_seg, large_tbase, small_seg, seg_hist, seg_mask, tile_seg, status, status_bytes, zero_bytes, total;
    uint64_t nlarge_max, tiles_max;
    uint32_t cutoff, small_variant, tile, large_variant;
};

struct SegArgs;
#define RSBD8G_DECLARE_SEG_LAUNCH(name)                                                                \
    cudaError_t name(const Resolved &r, const SegArgs &a, const SegLayout &L, unsigned char *scratch, \
                     const void *in, void *out, void *buf, cudaStream_t s);                           \
    cudaError_t name##_prepare(const Resolved &r);   /* load every kernel this sort can launch */
RSBD8G_DECLARE_SEG_LAUNCH(launch_segmented_k1)
RSBD8G_DECLARE_SEG_LAUNCH(launch_segmented_k2)
RSBD8G_DECLARE_SEG_LAUNCH(launch_segmented_k4)
RSBD8G_DECLARE_SEG_LAUNCH(launch_segmented_k8)
RSBD8G_DECLARE_SEG_LAUNCH(launch_segmented_k16)

rsbd8g_status resolve(const rsbd8g_desc *d, Resolved *r);
cudaError_t prepare_segmented(const Resolved &r);   // rsbd8g_segmented_api.cu: rsbd8g_prepare's segmented part
// p is device memory (cudaMalloc, a memory pool, a __device__ array); null counts as such
bool device_memory(const void *p);
// the resolved filter of a descriptor (isabsvalue | issignmode << 1 | isfltpmode << 2 | x87 << 3),
// -1 for a bad descriptor: descriptors of one key size and filter sort alike but for direction
int filter_class(const rsbd8g_desc *d);
Layout layout_for(const Resolved &r, uint64_t n);
rsbd8g_status enqueue_sort(const Resolved &r, uint64_t n, void *scratch, size_t scratch_bytes, const void *in,
                           void *out, void *buf, bool inplace, bool to_buffer, cudaStream_t s);
rsbd8g_status read_device_status(void *scratch, cudaStream_t s, bool clear);

}  // namespace rsbd8g
