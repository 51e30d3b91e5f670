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
