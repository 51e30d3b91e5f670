"""Sorts that run as one kernel: one tile, several tiles with a grid barrier between the passes, and the
edges between them (tiles of 2048, 4096, 8192 and 16384 keys, 16 CTAs to a group, the SMs' count of tiles
and the sorts just past it), copy and in-place forms with even, odd and no surviving digits, reversed
ties, and pointers.  Every order is compared with the oracle's, bit for bit."""
import numpy as np
import pytest

from conftest import empty_dev, from_dev, same_bits, to_dev
from oracle import oracle as O
from radixsortbidi8_gb300 import synth as S

pytestmark = pytest.mark.gpu

SIZES = [2, 31, 2047, 2048, 2049, 4096, 4097, 16 * 2048, 16 * 2048 + 1, 33 * 2048 - 5, 64 * 2048, 64 * 2048 + 1,
         152 * 4096, 152 * 4096 + 1, 152 * 8192, 152 * 8192 + 1, 152 * 16384, 152 * 16384 + 1]


def keys(dtype, n, seed):
    dt = np.dtype(dtype)
    return S.float_specials(seed, n, dt) if dt.kind == "f" else S.uniform_bits(seed, n, dt)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("dtype,mode,direction", [(np.uint8, "native", "ascfwdorder"), (np.int16, "nativetieredabs", "dscfwdorder"),
                                                  (np.uint32, "native", "dscfwdorder"), (np.float32, "nativeabs", "dscrevorder"),
                                                  (np.int64, "native", "ascfwdorder"), (np.float64, "native", "ascrevorder")],
                         ids=lambda x: str(getattr(x, "__name__", x)))
def test_every_tile_size(dtype, mode, direction, n):
    import torch
    import radixsortbidi8_gb300 as rs
    a = keys(dtype, n, n)
    want = O.sortcopy(a, mode, direction)
    x, y = to_dev(a), empty_dev(n, dtype)
    assert rs.radixsortcopy(x, y, direction, mode, key_dtype=dtype)
    assert same_bits(from_dev(y, dtype), want)
    assert rs.radixsort(x, direction, mode, key_dtype=dtype)
    assert same_bits(from_dev(x, dtype), want)
    x, buf = to_dev(a), empty_dev(n, dtype)
    scratch = torch.empty(rs.scratch_bytes(dtype, n, direction, mode), dtype=torch.uint8, device="cuda")
    scratch.fill_(0xA5)                       # any content: the call clears what it needs
    rs.radixsortnoalloc(x, buf, scratch, True, direction, mode, key_dtype=dtype)
    assert rs.scratch_status(scratch) == 0
    assert same_bits(from_dev(buf, dtype), want)


@pytest.mark.parametrize("n", [5, 2049, 70001, 700001])
@pytest.mark.parametrize("digits", [0, 1, 2, 3])
def test_surviving_digits(digits, n):
    """0 to 3 digits that differ: a copy or reversal alone, and every parity of the passes"""
    import radixsortbidi8_gb300 as rs
    m = (1 << (8 * digits)) - 1
    a = ((S.uniform_bits(2, n, np.uint32) & np.uint32(m)) | np.uint32(0x40000000)).view(np.float32)
    for direction in ("ascfwdorder", "dscrevorder"):
        for mode in ("native", "nativeabs"):
            sign = a.copy()
            if mode == "nativeabs":           # ties of opposite sign: the reversal shows
                sign[::3] = -sign[::3]
            want = O.sortcopy(sign, mode, direction)
            x, y = to_dev(sign), empty_dev(n, np.float32)
            assert rs.radixsortcopy(x, y, direction, mode, key_dtype=np.float32)
            assert same_bits(from_dev(y, np.float32), want)
            assert rs.radixsort(x, direction, mode, key_dtype=np.float32)
            assert same_bits(from_dev(x, np.float32), want)


@pytest.mark.parametrize("n", [3, 2048, 2049, 50001, 152 * 4096 + 1, 152 * 8192 + 1])
@pytest.mark.parametrize("dtype", [np.uint16, np.uint32, np.uint64], ids=lambda x: x.__name__)
@pytest.mark.parametrize("direction", ["ascfwdorder", "dscrevorder"])
def test_pointers(dtype, direction, n):
    import torch
    import radixsortbidi8_gb300 as rs
    key = S.uniform_bits(7, n, dtype)
    key[::2] = key[n // 3]                    # ties
    rec = np.zeros((n, 3), dtype=np.uint64)
    rec[:, 1] = key
    dev = torch.from_numpy(rec.view(np.int64)).cuda()
    ptr = dev.data_ptr() + 24 * torch.arange(n, dtype=torch.int64, device="cuda")
    k = key if direction == "ascfwdorder" else ~key
    order = np.argsort(k, kind="stable") if direction == "ascfwdorder" else n - 1 - np.argsort(k[::-1], kind="stable")
    want = dev.data_ptr() + 24 * order
    out = torch.empty_like(ptr)
    assert rs.radixsortcopy_member(ptr, out, dtype, 8, direction, "native")
    assert np.array_equal(out.cpu().numpy(), want)
    assert rs.radixsort_member(ptr, dtype, 8, direction, "native")
    assert np.array_equal(ptr.cpu().numpy(), want)


@pytest.mark.parametrize("n", [2048, 100003, (1 << 22) + 3])      # one tile, several, a launch per digit
def test_captured_in_a_graph(n):
    import torch
    import radixsortbidi8_gb300 as rs
    a = S.uniform_bits(11, n, np.uint32)
    x, y, buf = to_dev(a), empty_dev(n, np.uint32), empty_dev(n, np.uint32)
    scratch = torch.empty(rs.scratch_bytes(np.uint32, n), dtype=torch.uint8, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        rs.radixsortcopynoalloc(x, y, buf, scratch, key_dtype=np.uint32)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            rs.radixsortcopynoalloc(x, y, buf, scratch, key_dtype=np.uint32)
        y.zero_()
        g.replay()
        g.replay()
    s.synchronize()
    assert same_bits(from_dev(y, np.uint32), O.sortcopy(a))


@pytest.mark.parametrize("n", [2, 31, 2047, 4096, 4097, 8192, 8193, 100003, 300007])
@pytest.mark.parametrize("dtype,mode,direction", [(np.uint8, "native", "ascfwdorder"), (np.int16, "nativetieredabs", "dscfwdorder"),
                                                  (np.uint32, "native", "dscfwdorder"), (np.float32, "nativeabs", "dscrevorder"),
                                                  (np.int64, "native", "ascfwdorder"), (np.float64, "native", "ascrevorder")],
                         ids=lambda x: str(getattr(x, "__name__", x)))
def test_small_sorts_by_a_launch_per_digit(dtype, mode, direction, n):
    """the route of small sorts where no cooperative launch fits, and that it is the one taken"""
    import torch
    import radixsortbidi8_gb300 as rs
    from radixsortbidi8_gb300 import api
    a = keys(dtype, n, n)
    want = O.sortcopy(a, mode, direction)
    x, y = to_dev(a), empty_dev(n, dtype)
    api.profile_enable(True)
    assert rs.radixsortcopy(x, y, direction, mode, key_dtype=dtype, flags=api.FLAG_DIAG_LAUNCHES)
    api.profile_enable(False)
    ran = [r["kernel"] for r in api.profile_collect()]
    assert "histogram" in ran and ran.count("onesweep") == np.dtype(dtype).itemsize and "one" not in ran, ran
    assert same_bits(from_dev(y, dtype), want)
    assert rs.radixsort(x, direction, mode, key_dtype=dtype, flags=api.FLAG_DIAG_LAUNCHES)
    assert same_bits(from_dev(x, dtype), want)
    key = keys(dtype, n, n + 1)
    rec = np.zeros((n, 24 // key.itemsize), dtype=dtype)
    rec[:, 8 // key.itemsize] = key
    dev = torch.from_numpy(rec.view(np.int64)).cuda()
    ptr = dev.data_ptr() + 24 * torch.arange(n, dtype=torch.int64, device="cuda")
    out = torch.empty_like(ptr)
    assert rs.radixsortcopy_member(ptr, out, dtype, 8, direction, mode, flags=api.FLAG_DIAG_LAUNCHES)
    assert np.array_equal((out.cpu().numpy() - dev.data_ptr()) // 24, O.numpy_sort_indices(key, mode, direction))


def test_one_kernel_sorts_on_several_streams():
    """sorts that each want most of the SMs at once, queued on eight streams beside larger and smaller ones"""
    import torch
    import radixsortbidi8_gb300 as rs
    sizes = [1 << 20, 152 * 4096, 152 * 8192, 100003, 1000, (1 << 22) + 3, 1 << 20, 600011]
    arrs = [S.uniform_bits(i, n, np.uint32) for i, n in enumerate(sizes)]
    st = []
    for a in arrs:
        x = to_dev(a)
        st.append((x, [torch.empty_like(x) for _ in range(3)], torch.empty_like(x),
                   torch.empty(rs.scratch_bytes(np.uint32, a.size), dtype=torch.uint8, device="cuda"), torch.cuda.Stream()))
    torch.cuda.synchronize()
    for k in range(3):
        for x, outs, buf, scratch, s in st:
            rs.radixsortcopynoalloc(x, outs[k], buf, scratch, key_dtype=np.uint32, stream=s)
    torch.cuda.synchronize()
    for a, (x, outs, buf, scratch, s) in zip(arrs, st):
        assert rs.scratch_status(scratch) == 0
        want = np.sort(a)
        for y in outs:
            assert same_bits(from_dev(y, np.uint32), want)
