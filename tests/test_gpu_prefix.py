"""Large sorts of 8- and 16-byte keys: passes over a prefix of the digits, then the settle step.

Groups of equal prefixes of every kind go through: pairs and short groups (exchanges in registers),
groups across the edges of a warp's chunk of 248 keys, groups of up to a few hundred keys (the warp's
view in shared memory), long groups that are in order already, and groups too long to settle (the plain
passes then sort the array).  Every order is compared with the oracle's, bit for bit."""
import numpy as np
import pytest

from conftest import empty_dev, from_dev, same_bits, to_dev
from oracle import oracle as O
from radixsortbidi8_gb300 import synth as S

pytestmark = pytest.mark.gpu

N8, N16 = 1 << 21, 1 << 20          # the smallest prefix sorts (8- and 16-byte keys)


def spread(n, group, seed=1):
    """n keys of about n / group prefixes (the top 3 bytes and more random), low bytes random"""
    r = S.uniform_bits(seed, n, np.uint64)
    top = S.uniform_bits(seed + 1, max(1, n // group), np.uint64) & np.uint64(0xFFFFFFFFFF000000)
    return top[(r >> np.uint64(20)).astype(np.int64) % top.size] | (r & np.uint64(0xFFFFFF))


def with_cluster(n, size, at, seed=1):
    """uniform keys, `size` of which share their top 5 bytes"""
    k = S.uniform_bits(seed, n, np.uint64)
    k[at:at + size] = np.uint64(0x7777777700000000) | (k[at:at + size] & np.uint64(0xFFFFFF))
    return k


CASES = {
    "uniform": lambda n: S.uniform_bits(3, n, np.uint64),
    "pairs": lambda n: spread(n, 2),
    "groups_of_5": lambda n: spread(n, 5),
    "groups_of_40": lambda n: spread(n, 40),
    "cluster_11": lambda n: with_cluster(n, 11, 100),
    "cluster_60": lambda n: with_cluster(n, 60, 5),
    "cluster_224": lambda n: with_cluster(n, 224, 7),
    "cluster_460": lambda n: with_cluster(n, 460, 9),
    "cluster_480": lambda n: with_cluster(n, 480, 9),
    "cluster_5000": lambda n: with_cluster(n, 5000, 50),
    "sorted": lambda n: np.sort(S.uniform_bits(3, n, np.uint64)),
    "few_values": lambda n: S.uniform_bits(9, 1000, np.uint64)[(S.uniform_bits(4, n, np.uint64) % np.uint64(1000)).astype(np.int64)],
    "low_40_bits": lambda n: S.uniform_bits(3, n, np.uint64) & np.uint64((1 << 40) - 1),
}


@pytest.mark.parametrize("n", [N8 - 1, N8, N8 + 247, 3000017])
@pytest.mark.parametrize("case", list(CASES))
def test_prefix_sort_of_8_byte_keys(case, n):
    import radixsortbidi8_gb300 as rs
    a = CASES[case](n).view(np.int64)
    x, y = to_dev(a), empty_dev(n, np.int64)
    assert rs.radixsortcopy(x, y, "ascfwdorder", "native", key_dtype=np.int64)
    assert same_bits(from_dev(y, np.int64), O.sortcopy(a, "native", "ascfwdorder"))
    assert rs.radixsort(x, "dscfwdorder", "native", key_dtype=np.int64)
    assert same_bits(from_dev(x, np.int64), O.sortcopy(a, "native", "dscfwdorder"))


@pytest.mark.parametrize("mode,direction", [("native", "ascrevorder"), ("nativeabs", "dscrevorder"), ("nativeabs", "ascfwdorder"),
                                            ("nativetieredabs", "dscfwdorder"), ("specialfloatingp", "ascfwdorder")])
@pytest.mark.parametrize("dup", [False, True])
def test_prefix_sort_keeps_ties(mode, direction, dup):
    import radixsortbidi8_gb300 as rs
    n = 2500003
    a = S.float_specials(5, n, np.float64)
    if dup:                       # signed copies of fewer values: ties of the absolute modes in every group
        a = np.where(np.arange(n) % 2 == 0, -a[np.arange(n) // 8 * 8], a[np.arange(n) // 8 * 8])
    x, y = to_dev(a), empty_dev(n, np.float64)
    assert rs.radixsortcopy(x, y, direction, mode, key_dtype=np.float64)
    assert same_bits(from_dev(y, np.float64), O.sortcopy(a, mode, direction))


@pytest.mark.parametrize("case", ["uniform", "groups_of_5", "cluster_460", "cluster_5000", "few_values"])
@pytest.mark.parametrize("direction", ["ascfwdorder", "dscrevorder"])
def test_prefix_sort_of_pointers(case, direction):
    import torch
    import radixsortbidi8_gb300 as rs
    n = N8 + 1001
    key = CASES[case](n)
    rec = torch.zeros((n, 2), dtype=torch.int64, device="cuda")
    rec[:, 1] = torch.from_numpy(key.view(np.int64)).cuda()
    ptr = rec.data_ptr() + 16 * torch.arange(n, dtype=torch.int64, device="cuda")
    out = torch.empty_like(ptr)
    assert rs.radixsortcopy_member(ptr, out, np.uint64, 8, direction, "native")
    k = key if direction == "ascfwdorder" else ~key
    order = np.argsort(k, kind="stable") if direction == "ascfwdorder" else n - 1 - np.argsort(k[::-1], kind="stable")
    want = rec.data_ptr() + 16 * order
    assert np.array_equal(out.cpu().numpy(), want)
    inp = ptr.clone()
    assert rs.radixsort_member(inp, np.uint64, 8, direction, "native")
    assert np.array_equal(inp.cpu().numpy(), want)


@pytest.mark.parametrize("kind", ["u128", "f128", "x87"])
@pytest.mark.parametrize("case", ["uniform", "groups_of_5", "cluster_460", "cluster_5000"])
def test_prefix_sort_of_16_byte_keys(kind, case):
    import torch
    import radixsortbidi8_gb300 as rs
    n = N16 + 333
    w = np.empty((n, 2), dtype=np.uint64)
    hi = CASES[case](n)
    w[:, 0] = S.uniform_bits(8, n, np.uint64) if kind != "x87" else hi
    w[:, 1] = hi if kind != "x87" else S.uniform_bits(8, n, np.uint64)
    x = torch.from_numpy(w.view(np.int64).reshape(-1)).cuda()
    y = torch.empty_like(x)
    assert rs.radixsortcopy(x, y, "dscfwdorder", "native", key_dtype=kind)
    want = O.sortcopy_wide(w, kind, "native", "dscfwdorder")
    assert np.array_equal(y.cpu().numpy().view(np.uint64).reshape(n, 2), np.asarray(want).reshape(n, 2))


@pytest.mark.parametrize("kind", ["i64", "f64", "u128"])
def test_prefix_in_batches(kind):
    """the segmented sort decides per segment: uniform segments, clusters that are settled or bring the
    plain passes back (an even and an odd number of digits), long runs of equal keys, few digits"""
    import torch
    from radixsortbidi8_gb300 import api, batched
    segs = []
    for i, n in enumerate([6145, 262144, 7001, 50, 100003, 248 * 40, 8192 * 3 + 1, 200000, 1 << 19, 150000, 99999]):
        for j, case in enumerate(["uniform", "pairs", "groups_of_5", "cluster_480", "few_values"]):
            if (i + j) % 2:
                segs.append(CASES[case](max(n, 600) if case.startswith("cluster") else n))
        segs.append(with_cluster(max(n, 6000), 500, 3) & np.uint64((1 << 56) - 1))      # seven digits
        segs.append(with_cluster(max(n, 6000), 520, 5000))
    a = np.concatenate(segs)
    offs = np.zeros(len(segs) + 1, dtype=np.int64)
    np.cumsum([s.size for s in segs], out=offs[1:])
    if kind == "u128":
        w = np.stack([S.uniform_bits(4, a.size, np.uint64), a], axis=1)
        x, kt = torch.from_numpy(w.view(np.int64).reshape(-1)).cuda(), "u128"
    else:
        kt = np.int64 if kind == "i64" else np.float64
        x = torch.from_numpy(a.view(np.int64)).cuda()
    s = batched.SegmentedSorter(x, torch.from_numpy(offs).cuda(), "dscfwdorder", "native", key_dtype=kt)
    for out in (s.run(), s.capture().replay()):
        torch.cuda.synchronize()
        assert s.status() == api.OK
        got = out.cpu().numpy()
        for b, e in zip(offs[:-1], offs[1:]):
            if kind == "u128":
                want = O.sortcopy_wide(w[b:e], "u128", "native", "dscfwdorder")
                assert np.array_equal(got[2 * b:2 * e].view(np.uint64).reshape(-1, 2), np.asarray(want).reshape(-1, 2))
            else:
                assert same_bits(got[b:e].view(kt), O.sortcopy(a[b:e].view(kt), "native", "dscfwdorder"))
