"""bench.py host logic on CPU: the reference arm's JSON line, rank > 0 staying silent, and the
max-over-ranks aggregation of the replica path over a real 2-process gloo group."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(args, env_extra=None):
    env = dict(os.environ, **(env_extra or {}))
    return subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), *args], capture_output=True, text=True,
                          env=env, timeout=600, cwd=ROOT)


def test_reference_arm_line():
    r = _run(["--impl", "reference", "--steps", "1", "--warmup", "1", "--log2n", "16"])
    assert r.returncode == 0, r.stderr
    line = json.loads(r.stdout.strip().splitlines()[-1])
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
              "config", "impl", "cpu_baseline", "e2e"):
        assert k in line, k
    assert line["impl"] == "reference" and line["value"] > 0
    assert line["e2e"]["h2d_bytes_per_step"] == 0 and line["cpu_baseline"]["kind"] == "port"


def test_reference_arm_other_ranks_silent():
    r = _run(["--impl", "reference", "--steps", "1", "--warmup", "1", "--log2n", "12"],
             {"RANK": "1", "WORLD_SIZE": "2"})
    assert r.returncode == 0 and r.stdout.strip() == ""


def test_passes_that_ran_are_the_plans():
    """the launches that moved keys are named by the control block, whatever their times: one that took eight times as
    long as the others changes nothing, and a record too many or too few is an error"""
    import torch
    sys.path.insert(0, ROOT)
    import bench
    w = torch.zeros(256, dtype=torch.int32)
    for slot in (0, 1, 2, 9):
        w[bench.CTRL_PLAN + bench.PLAN_WORDS * slot + bench.PLAN_ACTIVE] = 1
    slots = bench.planned_slots(w.view(torch.uint8))
    assert slots == {0, 1, 2, 9}
    times = [(p, 100.0 if (step, p) == (1, 1) else 1.0 if p in slots else 0.01) for step in range(3) for p in range(14)]
    assert sorted(bench.passes_that_ran(times, slots, 3)) == [1.0] * 11 + [100.0]
    with pytest.raises(AssertionError):
        bench.passes_that_ran(times[1:], slots, 3)
    assert bench.passes_that_ran([], set(), 3) == []


def test_control_block_words_of_the_bench(tmp_path):
    """the words that bench.py reads are where the library's Control has them"""
    import shutil
    sys.path.insert(0, ROOT)
    import bench
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src = tmp_path / "ctrl.cu"
    src.write_text('#include <cstddef>\n#include <cstdio>\n#include "rsbd8g_device.cuh"\nint main() { using namespace rsbd8g; '
                   'std::printf("%zu %zu %zu %d", offsetof(Control, plan), sizeof(PassPlan), offsetof(PassPlan, active), kMaxSlots); }')
    exe = str(tmp_path / "ctrl")
    r = subprocess.run([nvcc, "-std=c++17", "-I", os.path.join(ROOT, "radixsortbidi8_gb300", "csrc"), str(src), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    got = [int(x) for x in subprocess.run([exe], capture_output=True, text=True).stdout.split()]
    assert got == [4 * bench.CTRL_PLAN, 4 * bench.PLAN_WORDS, 4 * bench.PLAN_ACTIVE, bench.CTRL_SLOTS]


def _worker(rank, world, port, q):
    import torch.distributed as dist
    sys.path.insert(0, ROOT)
    import bench
    dist.init_process_group("gloo", init_method=f"tcp://127.0.0.1:{port}", rank=rank, world_size=world)
    ms = bench.max_over_ranks(10.0 + rank * 5.0, world, "cpu")
    q.put((rank, ms, bench.whole_job_gkeys(3 << 28, world, ms)))
    dist.barrier()
    dist.destroy_process_group()


def test_replicas_take_the_slowest_rank_gloo():
    import socket
    import torch.multiprocessing as mp
    s = socket.socket()
    s.bind(("127.0.0.1", 0))
    port = s.getsockname()[1]
    s.close()
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    ps = [ctx.Process(target=_worker, args=(r, 2, port, q)) for r in range(2)]
    for p in ps:
        p.start()
    res = sorted(q.get(timeout=120) for _ in ps)
    for p in ps:
        p.join(timeout=60)
        assert p.exitcode == 0
    assert [r[1] for r in res] == [15.0, 15.0]
    assert res[0][2] == pytest.approx(2 * (3 << 28) / 15e-3 / 1e9)
