"""Prefix sorts whose samples miss a crowd of equal prefixes, and the routes that the plan takes.

The sampled positions are a function of the count alone, so a crowd that the samples cannot see is laid out
beside them, and what the sort then did is read from the control block in its scratch."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import oracle as O
from radixsortbidi8_gb300 import synth as S

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1


def sampled(n, draws):
    """the positions of the first `draws` samples of n keys (splitmix64 of the sample's index, scaled)"""
    out = np.empty(draws, dtype=np.int64)
    for i in range(draws):
        z = (i + 1) * 0x9E3779B97F4A7C15 & M64
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9 & M64
        z = (z ^ (z >> 27)) * 0x94D049BB133111EB & M64
        out[i] = (z ^ (z >> 31)) * n >> 64
    return out


def unseen(n, size, draws, seed=1):
    """`size` positions of n, in rising order, that no sample reads"""
    free = np.ones(n, dtype=bool)
    free[sampled(n, draws)] = False
    at = np.flatnonzero(free)
    return at[np.sort(np.argsort(S.uniform_bits(seed, at.size, np.uint64))[:size])]


def with_crowd(n, size, draws, seed=1):
    """uniform keys, `size` of which (seen by no sample) share their top 5 bytes"""
    k = S.uniform_bits(seed, n, np.uint64)
    at = unseen(n, size, draws, seed + 1)
    k[at] = np.uint64(0x0077777777000000) | (k[at] & np.uint64(0xFFFFFF))
    return k


def segment(n, size, first, seed):
    """a crowd that the samples of a batch's large segment number `first` do not see (17 rounds of 256 at most)"""
    return with_crowd(n, size, (first + 1) * 17 * 256, seed)


def sorter(segs, kt, direction, mode):
    import torch
    from radixsortbidi8_gb300 import batched
    a = np.concatenate(segs)
    offs = np.zeros(len(segs) + 1, dtype=np.int64)
    np.cumsum([s.size for s in segs], out=offs[1:])
    return a, offs, batched.SegmentedSorter(torch.from_numpy(a.view(np.int64)).cuda(), torch.from_numpy(offs).cuda(),
                                            direction, mode, key_dtype=kt)


def seg_passes(s):
    """digits that some large segment sorted by: before the settle step, after it (SegControl::pass_mask)"""
    import torch
    torch.cuda.synchronize()
    return [int(x) for x in s.scratch[152:160].cpu().numpy().view(np.uint32)]


def test_a_failed_segment_is_copied_back_by_the_whole_gpu():
    """Seven digits: the passes of a segment that cannot be settled end in the buffer.  One warp copies 256
    bytes per round trip to memory, 0.3 us at the very least: 9.4 ms for 10^6 keys of 8 bytes; all SMs copy
    them in well under 0.1 ms.  The bound lies between."""
    from radixsortbidi8_gb300 import api
    low7 = np.uint64((1 << 56) - 1)
    segs = [segment(1000003, 200000, 0, 3) & low7] + [S.uniform_bits(7 + i, 300007, np.uint64) & low7 for i in range(4)]
    a, offs, s = sorter(segs, np.int64, "dscfwdorder", "native")
    s.run()
    ms = []
    for _ in range(3):
        api.profile_enable(True)
        out = s.run()
        api.profile_enable(False)
        ms.append([r["ms"] for r in api.profile_collect() if r["kernel"] == "copy"])
    assert seg_passes(s)[1] == 0x7F                    # it failed, with an odd number of digits
    got = out.cpu().numpy()
    for b, e in zip(offs[:-1], offs[1:]):
        assert same_bits(got[b:e], O.sortcopy(a[b:e].view(np.int64), "native", "dscfwdorder"))
    assert min(m for [m] in ms) < 1.0, ms


@pytest.mark.parametrize("direction", ["ascfwdorder", "ascrevorder"])
@pytest.mark.parametrize("kt", [np.uint32, np.float64], ids=lambda t: t.__name__)
def test_segments_of_one_value_are_copied(kt, direction):
    """large segments of which every digit is skipped (ties of both signs reversed), between others"""
    import torch
    from radixsortbidi8_gb300 import batched
    lens = [20000, 8193, 300001, 50, 8192 * 5, 100003]
    a = np.concatenate([np.full(n, 3.5, dtype=kt) if i % 2 == 0 else S.uniform_bits(i, n, np.uint64).astype(kt) for i, n in enumerate(lens)])
    if kt == np.float64:
        a[::3] = -a[::3]
    offs = np.concatenate([[0], np.cumsum(lens)])
    s = batched.SegmentedSorter(torch.from_numpy(a.view(np.int64 if kt == np.float64 else np.int32)).cuda(), torch.from_numpy(offs).cuda(),
                                direction, "nativeabs", key_dtype=kt)
    got = s.run().cpu().numpy().view(kt)
    for b, e in zip(offs[:-1], offs[1:]):
        assert same_bits(got[b:e], O.sortcopy(a[b:e], "nativeabs", direction))


def plan_of(scratch):
    """what the plain sort did, from its control block (Control of rsbd8g_device.cuh, at the scratch's start)"""
    import torch
    torch.cuda.synchronize()
    w = scratch[:160].cpu().numpy().view(np.uint32)
    return dict(error=int(w[0]), low=int(w[31]), passes=int(w[32]), failed=int(w[33]))


DRAWS = 160 * 1024                  # of one round, up to 160 histogram CTAs
CROWDS = [(3000, 0), (4000, 0), (30000, 1)]          # the last is too long to settle


@pytest.mark.parametrize("size,failed", CROWDS)
@pytest.mark.parametrize("form", ["copy", "inplace", "tobuffer"])
def test_a_crowd_that_no_sample_saw(size, failed, form):
    """out-of-order groups longer than a warp's view: up to settle_limit (4096 of 2^21 keys) they are settled, in
    the array that the passes left free; beyond it the plain passes run"""
    import torch
    import radixsortbidi8_gb300 as rs
    n = (1 << 21) + 77
    a = with_crowd(n, size, DRAWS).view(np.int64)
    x = torch.from_numpy(a.copy()).cuda()
    y, buf = torch.empty_like(x), torch.empty_like(x)
    for direction in ("ascfwdorder", "dscfwdorder"):
        x.copy_(torch.from_numpy(a))
        scratch = torch.empty(rs.scratch_bytes(np.int64, n, direction, "native"), dtype=torch.uint8, device="cuda")
        if form == "copy":
            rs.radixsortcopynoalloc(x, y, buf, scratch, direction, "native", key_dtype=np.int64)
        else:
            rs.radixsortnoalloc(x, buf, scratch, form == "tobuffer", direction, "native", key_dtype=np.int64)
        p = plan_of(scratch)
        assert p["passes"] > 0 and p["failed"] == failed and p["error"] == 0, p
        got = (y if form == "copy" else x if form == "inplace" else buf).cpu().numpy()
        assert same_bits(got, O.sortcopy(a, "native", direction))
        if form == "copy":
            assert same_bits(x.cpu().numpy(), a)          # the copy form leaves its input alone


CHUNK, VIEW = 248, 472              # SettleShape::kChunk, kView


def crowds_of_every_length(n, lengths):
    """a crowd of each length, spread over the key range; and where each starts and ends in the sorted array"""
    a = S.uniform_bits(21, n, np.uint64)
    at, o = unseen(n, int(np.sum(lengths)), DRAWS, 22), 0
    tops = np.sort(S.uniform_bits(23, len(lengths), np.uint64)) & np.uint64(0xFFFFFFFFFF000000)
    for top, m in zip(tops, lengths):
        p = at[o:o + m]
        a[p] = top | (a[p] & np.uint64(0xFFFFFF))
        o += m
    srt = np.sort(a) >> np.uint64(24)
    return a, np.searchsorted(srt, tops >> np.uint64(24)), np.searchsorted(srt, tops >> np.uint64(24), side="right")


def test_crowds_about_the_view():
    """crowds that end before, at and after the end of the view of the chunk they start in, and of the next"""
    import torch
    import radixsortbidi8_gb300 as rs
    n = 1 << 22
    a, b, e = crowds_of_every_length(n, np.tile(np.arange(200, 760), 2))
    past = e - (b // CHUNK * CHUNK + VIEW)
    assert {-1, 0, 1} <= set(past.tolist())
    x = torch.from_numpy(a.view(np.int64)).cuda()
    y, buf = torch.empty_like(x), torch.empty_like(x)
    scratch = torch.empty(rs.scratch_bytes(np.uint64, n), dtype=torch.uint8, device="cuda")
    rs.radixsortcopynoalloc(x, y, buf, scratch, key_dtype=np.uint64)
    p = plan_of(scratch)
    assert p["passes"] > 0 and p["failed"] == 0 and p["error"] == 0, p
    assert same_bits(y.cpu().numpy().view(np.uint64), np.sort(a))


@pytest.mark.parametrize("size,failed", CROWDS)
@pytest.mark.parametrize("mode,direction", [("nativeabs", "ascrevorder"), ("nativeabs", "dscrevorder"), ("native", "ascrevorder")])
def test_a_crowd_of_floats_with_ties(size, failed, mode, direction):
    """float orders: the crowd's values come eight times each, and under nativeabs with both signs (reversed ties)"""
    import torch
    import radixsortbidi8_gb300 as rs
    n = (1 << 21) + 77
    a = with_crowd(n, size, DRAWS) & np.uint64((1 << 63) - 1)
    at = np.flatnonzero(a >> np.uint64(24) == 0x77777777)
    a[at] = a[at[np.arange(at.size) // 8 * 8]] ^ ((S.uniform_bits(6, at.size, np.uint64) & np.uint64(1)) << np.uint64(63) if mode == "nativeabs"
                                                  else np.uint64(0))
    x = torch.from_numpy(a.view(np.int64)).cuda()
    y, buf = torch.empty_like(x), torch.empty_like(x)
    scratch = torch.empty(rs.scratch_bytes(np.float64, n, direction, mode), dtype=torch.uint8, device="cuda")
    rs.radixsortcopynoalloc(x, y, buf, scratch, direction, mode, key_dtype=np.float64)
    p = plan_of(scratch)
    assert p["passes"] > 0 and p["failed"] == failed and p["error"] == 0, p
    assert same_bits(y.cpu().numpy().view(np.float64), O.sortcopy(a.view(np.float64), mode, direction))


@pytest.mark.parametrize("size,failed", CROWDS)
@pytest.mark.parametrize("direction", ["ascfwdorder", "dscrevorder"])
def test_a_crowd_of_pointers(size, failed, direction):
    import torch
    import radixsortbidi8_gb300 as rs
    from radixsortbidi8_gb300 import api
    n = (1 << 21) + 77
    key = with_crowd(n, size, 640 * 512)                  # up to 640 CTAs of 512 gather
    at = np.flatnonzero(key >> np.uint64(24) == 0x77777777)
    key[at] = key[at[np.arange(at.size) // 4 * 4]]        # ties
    rec = torch.zeros((n, 2), dtype=torch.int64, device="cuda")
    rec[:, 1] = torch.from_numpy(key.view(np.int64)).cuda()
    ptr = rec.data_ptr() + 16 * torch.arange(n, dtype=torch.int64, device="cuda")
    out, buf = torch.empty_like(ptr), torch.empty_like(ptr)
    scratch = torch.empty(rs.scratch_bytes(np.uint64, n, direction, "native", indirection=api.MEMBER, offset1=8), dtype=torch.uint8, device="cuda")
    rs.radixsortcopynoalloc_member(ptr, out, buf, scratch, np.uint64, 8, direction, "native")
    p = plan_of(scratch)
    assert p["passes"] > 0 and p["failed"] == failed and p["error"] == 0, p
    k = key if direction == "ascfwdorder" else ~key
    order = np.argsort(k, kind="stable") if direction == "ascfwdorder" else n - 1 - np.argsort(k[::-1], kind="stable")
    assert np.array_equal(out.cpu().numpy(), rec.data_ptr() + 16 * order)


@pytest.mark.parametrize("size,failed", [(1500, 0), (2000, 0), (30000, 1)])
@pytest.mark.parametrize("kind,mode,direction", [("u128", "native", "dscfwdorder"), ("f128", "native", "ascrevorder"), ("x87", "nativeabs", "ascrevorder"),
                                                 ("u128", 3, "dscrevorder"), ("u128", 1, "ascfwdorder"), ("f128", 5, "dscfwdorder"),
                                                 ("x87", "native", "dscrevorder")])
def test_a_crowd_of_16_byte_keys(size, failed, kind, mode, direction):
    """(settle_limit is 2048 of 2^20 keys; modes 3, 1, 5 and the float order carry from word to word: half of the keys
    of the absolute signed mode are negated, some with a low word of zero)"""
    import torch
    import radixsortbidi8_gb300 as rs
    n = 1 << 20
    hi = with_crowd(n, size, DRAWS) & np.uint64((1 << 63) - 1)
    lo = S.uniform_bits(8, n, np.uint64)
    at = np.flatnonzero(hi >> np.uint64(24) == 0x77777777)
    if kind == "x87":                 # 64-bit significands of one exponent: the crowd in the low word, signs mixed
        w = np.stack([hi, np.uint64(0x3FFF) | ((lo & np.uint64(1)) << np.uint64(15))], axis=1)
    else:
        w = np.stack([lo, hi], axis=1)
    w[at] = w[at[np.arange(at.size) // 2 * 2]]            # ties
    if mode == 3:
        w[at[::8], 0] = 0
        w[1::2, 1] = ~w[1::2, 1] + (w[1::2, 0] == 0)
        w[1::2, 0] = ~w[1::2, 0] + np.uint64(1)
    x = torch.from_numpy(w.view(np.int64).reshape(-1)).cuda()
    y, buf = torch.empty_like(x), torch.empty_like(x)
    scratch = torch.empty(rs.scratch_bytes(kind, n, direction, mode), dtype=torch.uint8, device="cuda")
    rs.radixsortcopynoalloc(x, y, buf, scratch, direction, mode, key_dtype=kind)
    p = plan_of(scratch)
    assert p["passes"] > 0 and p["failed"] == failed and p["error"] == 0, p
    want = O.sortcopy_wide(w, kind, mode, direction)
    assert np.array_equal(y.cpu().numpy().view(np.uint64).reshape(n, 2), np.asarray(want).reshape(n, 2))


@pytest.mark.parametrize("kt,mode,direction", [(np.int64, "native", "ascfwdorder"), (np.float64, "nativeabs", "dscrevorder"),
                                               (np.float64, "native", "ascrevorder")], ids=str)
@pytest.mark.parametrize("size,failed", [(1500, 0), (30000, 1)])
def test_a_crowd_in_a_batch(kt, mode, direction, size, failed):
    """(settle_limit is 2048 of 600,000 keys); the ties of a failed segment turn once, not twice"""
    segs = [segment(600011, size, i, 3 + i) & np.uint64((1 << 63) - 1) for i in range(4)]
    for sg in segs:
        at = np.flatnonzero(sg >> np.uint64(24) == 0x77777777)
        sg[at] = sg[at[np.arange(at.size) // 4 * 4]]
        if mode == "nativeabs":
            sg[1::2] |= np.uint64(1 << 63)
    a, offs, s = sorter(segs, kt, direction, mode)
    got = s.run().cpu().numpy().view(kt)
    for b, e in zip(offs[:-1], offs[1:]):
        assert same_bits(got[b:e], O.sortcopy(a[b:e].view(kt), mode, direction))
    first, second = seg_passes(s)
    assert first and not first & 1 and (second != 0) == bool(failed), (first, second)


def test_unnamed_flag_bits_change_no_route():
    """bits of the descriptor's flags that the header does not name are without meaning"""
    import torch
    from radixsortbidi8_gb300 import batched
    n = 1 << 21
    x = torch.from_numpy(S.uniform_bits(3, n, np.int64)).cuda()
    offs = torch.tensor([0, n // 2, n], dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    seen = []
    for flags in [0] + [1 << b for b in (4, 17, 30, 31)]:
        s = batched.SegmentedSorter(x, offs, "ascfwdorder", "native", key_dtype=np.int64)
        batched.segmented_sortcopy(x, s.output, s.buffer, offs, s.scratch, "ascfwdorder", "native", np.int64, s.tuning, s.stream, flags)
        seen.append(seg_passes(s))
    assert seen[0][0] and not seen[0][0] & 1 and all(p == seen[0] for p in seen), seen     # (a prefix, without the lowest digit)


@pytest.mark.parametrize("kt,mode", [(np.int64, "native"), (np.float64, "nativeabs")], ids=str)
def test_pointer_tables_and_directions_with_a_prefix(kt, mode):
    """batches of separate arrays, each with its direction: settled segments, a crowd in the view's length and one
    too long, reversed ties, small segments beside them"""
    import torch
    from radixsortbidi8_gb300 import batched
    arrs = [segment(600011, 1500, 0, 3), S.uniform_bits(5, 700001, np.uint64), segment(600011, 30000, 2, 7), S.uniform_bits(6, 5000, np.uint64),
            S.uniform_bits(8, 250007, np.uint64), segment(300011, 700, 5, 9)]
    arrs = [(a & np.uint64((1 << 63) - 1)).view(np.int64) for a in arrs]
    for a in arrs:
        at = np.flatnonzero(a >> 24 == 0x77777777)
        a[at] = a[at[np.arange(at.size) // 4 * 4]]
        if mode == "nativeabs":
            a[1::2] |= np.int64(-1 << 63)
    dirs = ["ascfwdorder", "dscrevorder", "dscfwdorder", "ascrevorder", "ascrevorder", "dscrevorder"]
    ins = [torch.from_numpy(a).cuda() for a in arrs]
    outs, bufs = [torch.empty_like(x) for x in ins], [torch.empty_like(x) for x in ins]
    total = sum(a.size for a in arrs)
    assert total >= 1 << 21                                # (a prefix is possible)
    scratch = torch.empty(batched.segmented_scratch_bytes(kt, total, len(arrs), "ascfwdorder", mode), dtype=torch.uint8, device="cuda")
    keep = batched.segmented_sortcopy_ptrs(ins, outs, bufs, scratch, mode=mode, key_dtype=kt, directions=dirs)
    torch.cuda.synchronize()
    first, second = [int(v) for v in scratch[152:160].cpu().numpy().view(np.uint32)]
    assert first and not first & 1 and second, (first, second)
    for a, d, y in zip(arrs, dirs, outs):
        assert same_bits(y.cpu().numpy().view(kt), O.sortcopy(a.view(kt), mode, d))
    del keep


def places(n, draws):
    """sampled() of many draws of fewer than 2^32 keys"""
    z = (np.arange(1, draws + 1, dtype=np.uint64)) * np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    z ^= z >> np.uint64(31)
    low = np.uint64(0xFFFFFFFF)
    return (((z >> np.uint64(32)) * np.uint64(n) + ((z & low) * np.uint64(n) >> np.uint64(32))) >> np.uint64(32)).astype(np.int64)


@pytest.mark.parametrize("size,failed", [(60000, 0), (300000, 1)])
def test_a_crowd_with_wide_look_back_words(size, failed):
    """2^30 keys and more: 8-byte look-back words, settle_limit 131,072; the order is torch.sort's"""
    import torch
    import radixsortbidi8_gb300 as rs
    n = (1 << 30) + 5
    assert np.array_equal(places(1000003, 500), sampled(1000003, 500))
    at = np.arange(size, dtype=np.int64) * 3001 + 11
    at = at[~np.isin(at, places(n, 160 * 1024 * 16))]     # 16 rounds at most
    assert at.size > size * 0.9
    x = S.uniform_bits_torch(3, n, 8)
    p = torch.from_numpy(at).cuda()
    x[p] = (x[p] & 0xFFFFFF) | 0x0077777777000000
    y, buf = torch.empty_like(x), torch.empty_like(x)
    scratch = torch.empty(rs.scratch_bytes(np.int64, n), dtype=torch.uint8, device="cuda")
    rs.radixsortcopynoalloc(x, y, buf, scratch, key_dtype=np.int64)
    q = plan_of(scratch)
    assert q["passes"] > 0 and q["failed"] == failed and q["error"] == 0, q
    del buf, scratch
    assert torch.equal(y, torch.sort(x)[0])
