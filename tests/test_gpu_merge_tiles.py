"""Merges at the edges of the merge kernel's tiles and windows (1920 outputs and 2048 elements for keys of
up to 4 bytes, 896 and 1024 for 8-byte keys, 384 and 512 for 16-byte keys): run lengths around
them, one-sided merges that empty a window, runs and outputs that do not start on 16 bytes, ties in both
tie orders.  Compared with the oracle's stable sort of the whole array."""
import numpy as np
import pytest

from conftest import same_bits, to_dev
from oracle import oracle as O
from radixsortbidi8_gb300 import synth as S

pytestmark = pytest.mark.gpu


def runs_of(a, lens, mode, direction, side):
    """the unsorted array and its runs, sorted; side: "mixed" keys, or all of run 1 before / after run 2"""
    o, parts = 0, []
    if side != "mixed":
        s = O.sortcopy(a, mode, direction)
        a = s if side == "before" else np.concatenate([s[lens[1]:], s[:lens[1]]])
    for m in lens:
        parts.append(O.sortcopy(a[o:o + m], mode, direction))
        o += m
    return a, np.concatenate(parts)


@pytest.mark.parametrize("dtype,mode,direction", [(np.uint8, "native", "ascfwdorder"), (np.int16, "nativeabs", "dscrevorder"),
                                                  (np.uint32, "native", "dscfwdorder"), (np.float32, "nativeabs", "ascrevorder"),
                                                  (np.float64, "native", "ascfwdorder"), (np.int64, "nativetieredabs", "dscfwdorder")],
                         ids=lambda x: str(getattr(x, "__name__", x)))
@pytest.mark.parametrize("lens", [(1, 1), (1919, 1), (960, 960), (961, 960), (2047, 2049), (2048, 0), (1, 8191), (895, 897), (896, 3),
                                  (70001, 50003), (3, 300001)], ids=str)
def test_tile_edges(dtype, mode, direction, lens):
    import torch
    from radixsortbidi8_gb300 import api
    n = sum(lens)
    a = S.float_specials(n, n, dtype) if np.dtype(dtype).kind == "f" else S.uniform_bits(n, n, dtype)
    for side in ("mixed", "before", "after"):
        whole, r = runs_of(a, lens, mode, direction, side)
        want = O.sortcopy(whole, mode, direction)
        for shift in (0, 1, 3):            # arrays that start past a 16-byte boundary
            x = torch.zeros(n + 8, dtype=to_dev(r).dtype, device="cuda")
            y = torch.zeros_like(x)
            x[shift:shift + n] = to_dev(r)
            api.merge_runs(x[shift:shift + n], y[(shift * 5) % 7:(shift * 5) % 7 + n], lens, None, direction, mode, key_dtype=dtype)
            got = y.cpu().numpy()
            o = (shift * 5) % 7
            assert same_bits(got[o:o + n].view(dtype), want), (side, shift)
            assert not got[:o].any() and not got[o + n:].any()


@pytest.mark.parametrize("lens", [(383, 1), (192, 193), (512, 511), (5, 3000), (20001, 9999)], ids=str)
@pytest.mark.parametrize("direction", ["ascfwdorder", "dscrevorder"])
def test_tile_edges_of_16_byte_keys(lens, direction):
    import torch
    from radixsortbidi8_gb300 import api
    n = sum(lens)
    w = S.uniform_bits(n, 2 * n, np.uint64).reshape(n, 2)
    w[::3, 1] = 5                           # ties of the high word
    r = np.concatenate([np.asarray(O.sortcopy_wide(np.ascontiguousarray(w[:lens[0]]), "u128", "native", direction)).reshape(-1, 2),
                        np.asarray(O.sortcopy_wide(np.ascontiguousarray(w[lens[0]:]), "u128", "native", direction)).reshape(-1, 2)])
    x = torch.from_numpy(np.ascontiguousarray(r).view(np.int64).reshape(-1)).cuda()
    y = torch.empty_like(x)
    api.merge_runs(x, y, lens, None, direction, "native", key_dtype="u128")
    want = np.asarray(O.sortcopy_wide(np.ascontiguousarray(w), "u128", "native", direction)).reshape(-1, 2)
    assert np.array_equal(y.cpu().numpy().view(np.uint64).reshape(n, 2), want)
