"""The work this framework is measured on: sorts, batches, merges and served requests as programs ask for them.

Each case is a dict of plain values.  ``prepare`` makes what a program holds before the call (keys on the device, and the
buffers, sorter or server that it keeps), ``run`` is one call through the public entry points, ``work`` the bytes that no
implementation can do without (every key read once and written once).  Outputs are key bits (or object addresses), so they
are compared as whole numbers.
"""
import numpy as np
import torch

import radixsortbidi8_gb300 as rs
from radixsortbidi8_gb300 import api, batched, serving, synth

KEY_BYTES = {"u8": 1, "u16": 2, "u32": 4, "i32": 4, "f32": 4, "i64": 8, "u64": 8, "f64": 8, "u128": 16}
KEY_TYPES = {"u8": np.uint8, "u16": np.uint16, "u32": np.uint32, "i32": np.int32, "f32": np.float32,
             "i64": np.int64, "u64": np.uint64, "f64": np.float64, "u128": "u128"}


def listed():
    return [
        # the smallest call a program makes: one short array through the allocating form, which waits for its result
        dict(name="u32_copy_1k", kind="sort", key="u32", n=1000, form="copy", direction="ascfwdorder", mode="native", bits=32),
        # a short odd-sized array sorted in place, floats by absolute value (each pass on a fresh copy of the input)
        dict(name="f32_inplace_50k", kind="sort", key="f32", n=50021, form="inplace", direction="dscfwdorder", mode="nativeabs", bits=32),
        # the plain mid-size sort of the benchmark, with the caller's own buffer and scratch: stream-ordered
        dict(name="u32_2p20", kind="sort", key="u32", n=1 << 20, form="noalloc", direction="ascfwdorder", mode="native", bits=32),
        # an ordinary ragged array of 64-bit keys
        dict(name="i64_3m", kind="sort", key="i64", n=3000017, form="noalloc", direction="dscfwdorder", mode="native", bits=64),
        # the three large sorts: uniform 32-bit keys, floats by absolute value with signed zeros, infinities and NaNs, 64-bit keys
        dict(name="u32_2p28", kind="sort", key="u32", n=1 << 28, form="noalloc", direction="ascfwdorder", mode="native", bits=32),
        dict(name="f32_abs_2p28", kind="sort", key="f32", n=1 << 28, form="noalloc", direction="dscfwdorder", mode="nativeabs", bits=32),
        dict(name="i64_2p28", kind="sort", key="i64", n=1 << 28, form="noalloc", direction="ascfwdorder", mode="native", bits=64),
        # pointers to 24-byte records sorted by a double member (10 % duplicated keys)
        dict(name="records_2p26", kind="records", n=1 << 26, direction="ascfwdorder", mode="native"),
        # batches of independent arrays of uneven lengths, replayed as one graph
        dict(name="batch_u32", kind="batch", key="u32", arrays=2889, lo=16, hi=1 << 20, direction="ascfwdorder", mode="native", bits=32),
        dict(name="batch_f64", kind="batch", key="f64", arrays=5000, lo=64, hi=1 << 18, direction="ascfwdorder", mode="native", bits=64),
        # a stable merge of two sorted halves
        dict(name="merge_u32", kind="merge", key="u32", n=1 << 28, runs=2, direction="ascfwdorder", mode="native", bits=32),
        # a queue of mixed requests served together: four key types, both directions, with and without the absolute filter
        dict(name="serve_48", kind="serve", requests=48, lo=1 << 10, hi=1 << 24),
    ]


def _log_uniform(rng, lo, hi):
    return int(lo * (hi / lo) ** rng.random())


def draw(rng):
    kind = rng.choice(["sort"] * 6 + ["records", "batch", "merge", "serve"])
    direction = rng.choice(["ascfwdorder", "dscfwdorder", "ascrevorder", "dscrevorder"])
    mode = rng.choice(["native", "native", "nativeabs", "nativetieredabs"])
    if kind == "records":
        return dict(kind=kind, n=_log_uniform(rng, 1000, 1 << 26), direction=direction, mode=mode)
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(4, 60), lo=1 << 10, hi=1 << rng.randint(16, 24))
    # whole key ranges mostly; sometimes integers of which only the low bits vary (counters, ids, small values)
    key = rng.choice(["u8", "u16", "u32", "i32", "f32", "i64", "u64", "f64", "u128"])
    if kind == "sort":
        bits = 8 * KEY_BYTES[key]
        if key in ("u32", "i64", "u64") and rng.random() < 0.3:
            bits = rng.randint(8, bits - 4)
        return dict(kind=kind, key=key, n=_log_uniform(rng, 1000, (1 << 30) // KEY_BYTES[key] if KEY_BYTES[key] > 2 else 1 << 28),
                    form=rng.choice(["copy", "noalloc", "inplace"]), direction=direction, mode=mode, bits=bits)
    key = rng.choice(["u16", "u32", "f32", "i64", "f64"])
    bits = 8 * KEY_BYTES[key]
    if kind == "batch":
        return dict(kind=kind, key=key, arrays=_log_uniform(rng, 100, 3000), lo=rng.choice([16, 64]), hi=1 << rng.randint(16, 19),
                    direction=direction, mode=mode, bits=bits)
    return dict(kind=kind, key=key, n=_log_uniform(rng, 100000, (1 << 30) // KEY_BYTES[key] if KEY_BYTES[key] > 2 else 1 << 28),
                runs=rng.choice([2, 2, 3]), direction=direction, mode=mode, bits=bits)


def _keys(key, n, bits, seed):
    """n keys as a signed integer tensor of the key's width: uniform bits, floats around zero with signed zeros,
    infinities and NaNs, or integers of which only the low `bits` vary."""
    kb = KEY_BYTES[key]
    if key == "u128":
        return synth.uniform_bits_torch(seed, 2 * n, 8)
    out = torch.empty(n, dtype={1: torch.int8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[kb], device="cuda")
    chunk = 1 << 26
    for o in range(0, n, chunk):         # in parts: the generators' temporaries are several times their output
        m = min(chunk, n - o)
        if key in ("f32", "f64"):
            out[o:o + m] = synth.float_specials_torch(seed + 7919 * (o // chunk), m, kb)
        elif bits < 8 * kb:
            out[o:o + m] = (synth.splitmix64_torch(seed + 7919 * (o // chunk), m) & ((1 << bits) - 1)).to(out.dtype)
        else:
            out[o:o + m] = synth.uniform_bits_torch(seed + 7919 * (o // chunk), m, kb)
    return out


def _serve_requests(case, seed):
    lens = synth.log_uniform_lengths(seed, case["requests"], case["lo"], case["hi"])
    pick = synth.splitmix64(seed, 3 * case["requests"], stream=41).reshape(3, -1)
    names = ("u16", "i32", "f32", "f64")
    return [(names[int(k % np.uint64(4))], int(n), "dscfwdorder" if int(d) & 1 else "ascfwdorder",
             "nativeabs" if int(a) & 1 else "native") for n, k, d, a in zip(lens, *pick)]


# the lengths of a batch are part of the case (a program's batch shape), not of the seed
def _batch_lengths(case):
    return synth.log_uniform_lengths(synth.BATCH_A_SEED, case["arrays"], case["lo"], case["hi"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        reqs = _serve_requests(case, case["requests"])
        ins = [_keys(k, n, 8 * KEY_BYTES[k], seed * 1009 + i) for i, (k, n, _, _) in enumerate(reqs)]
        outs = [torch.empty_like(x) for x in ins]
        return dict(case=case, reqs=reqs, ins=ins, outs=outs, server=serving.Server(4 << 30, 4))
    direction, mode = case["direction"], case["mode"]
    if kind == "records":
        n = case["n"]
        rec = synth.records24_torch(seed, n)
        ptrs = rec.data_ptr() + 24 * torch.arange(n, dtype=torch.int64, device="cuda")
        nb = rs.scratch_bytes(np.float64, n, direction, mode, indirection=api.MEMBER, offset1=8)
        return dict(case=case, rec=rec, inp=ptrs, out=torch.empty_like(ptrs), buf=torch.empty_like(ptrs),
                    scratch=torch.empty(nb, dtype=torch.uint8, device="cuda"))
    key, kt = case["key"], KEY_TYPES[case["key"]]
    if kind == "batch":
        lens = _batch_lengths(case)
        offs = np.zeros(lens.size + 1, dtype=np.int64)
        np.cumsum(lens, out=offs[1:])
        inp = _keys(key, int(offs[-1]), case["bits"], seed)
        sorter = batched.SegmentedSorter(inp, torch.from_numpy(offs).cuda(), direction, mode, key_dtype=kt)
        return dict(case=case, sorter=sorter.capture())
    n = case["n"]
    inp = _keys(key, n, case["bits"], seed)
    st = dict(case=case, inp=inp, out=torch.empty_like(inp))
    if kind == "merge":
        st["runs"] = api.halves(n) if case["runs"] == 2 else api.thirds(n)
        o, parts = 0, torch.empty_like(inp)
        for m in st["runs"]:
            if not rs.radixsortcopy(inp[o:o + m], parts[o:o + m], direction, mode, key_dtype=kt):
                raise MemoryError("sorting the runs")
            o += m
        st["inp"] = parts
        st["buf"] = torch.empty_like(inp) if case["runs"] > 2 else None
    elif case["form"] == "noalloc":
        nb = rs.scratch_bytes(kt, n, direction, mode)
        st["buf"] = torch.empty_like(inp)
        st["scratch"] = torch.empty(nb, dtype=torch.uint8, device="cuda")
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "serve":
        server = st["server"]
        ids = [server.submit(x, y, d, m, key_dtype=KEY_TYPES[k]) for (k, _, d, m), x, y in zip(st["reqs"], st["ins"], st["outs"])]
        for r in ids:
            server.wait(r)
        return st["outs"]
    if kind == "batch":
        return st["sorter"].replay()
    direction, mode = case["direction"], case["mode"]
    if kind == "records":
        rs.radixsortcopynoalloc_member(st["inp"], st["out"], st["buf"], st["scratch"], np.float64, 8, direction, mode)
        return st["out"] - st["rec"].data_ptr()      # as offsets into the records: the addresses differ from run to run
    kt = KEY_TYPES[case["key"]]
    if kind == "merge":
        api.merge_runs(st["inp"], st["out"], st["runs"], st["buf"], direction, mode, key_dtype=kt)
    elif case["form"] == "copy":
        if not rs.radixsortcopy(st["inp"], st["out"], direction, mode, key_dtype=kt):
            raise MemoryError("radixsortcopy")
    elif case["form"] == "inplace":
        st["out"].copy_(st["inp"])
        if not rs.radixsort(st["out"], direction, mode, key_dtype=kt):
            raise MemoryError("radixsort")
    else:
        rs.radixsortcopynoalloc(st["inp"], st["out"], st["buf"], st["scratch"], direction, mode, key_dtype=kt)
    return st["out"]


def work(case):
    kind = case["kind"]
    if kind == "serve":
        return {"bytes": sum(2 * n * KEY_BYTES[k] for k, n, _, _ in _serve_requests(case, case["requests"])), "flops": 0}
    if kind == "records":
        return {"bytes": case["n"] * (8 + 8 + 8), "flops": 0}       # a pointer and a key read, a pointer written
    if kind == "batch":
        return {"bytes": 2 * int(_batch_lengths(case).sum()) * KEY_BYTES[case["key"]], "flops": 0}
    return {"bytes": 2 * case["n"] * KEY_BYTES[case["key"]], "flops": 0}
