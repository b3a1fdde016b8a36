"""The multi-GPU bookkeeping of the benchmark on CPU: world-size-2 gloo ranks
(127.0.0.1 rendezvous) agree on the job's time as the largest rank's, and the
whole-job rate counts every rank's instance; the reference arm runs on rank 0
alone (the others exit 0 without work)."""
import os
import socket
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _free_port():
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        return s.getsockname()[1]


def _rank(rank, world, port, times, out):
    import datetime

    import torch.distributed as dist
    sys.path.insert(0, ROOT)
    import bench
    dist.init_process_group("gloo", init_method=f"tcp://127.0.0.1:{port}", rank=rank, world_size=world,
                            timeout=datetime.timedelta(seconds=60))
    try:
        dist.barrier()
        t = bench.max_over_ranks(dist, times[rank], "cpu")
        rate = bench.whole_job_rate(1000, world, 10, t)
        out.put((rank, t, rate))
        dist.barrier()
    finally:
        dist.destroy_process_group()


def test_two_gloo_ranks_take_the_slowest_time():
    import torch.multiprocessing as mp
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    port = _free_port()
    times = [12.5, 20.0]
    procs = [ctx.Process(target=_rank, args=(r, 2, port, times, q)) for r in range(2)]
    for p in procs:
        p.start()
    for p in procs:
        p.join(120)
        assert p.exitcode == 0
    got = sorted(q.get(timeout=10) for _ in range(2))
    for rank, t, rate in got:
        assert t == 20.0
        assert rate == pytest.approx(1000 * 2 * 10 / 0.020)


def test_reference_arm_runs_on_rank_zero_only():
    env = dict(os.environ, RANK="1", WORLD_SIZE="2", LOCAL_RANK="1", MASTER_ADDR="127.0.0.1", MASTER_PORT="29555")
    r = subprocess.run([sys.executable, os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "2",
                        "--steps", "1", "--warmup", "0"], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0
    assert r.stdout.strip() == ""


def test_single_rank_needs_no_process_group():
    sys.path.insert(0, ROOT)
    import bench
    assert bench.max_over_ranks(None, 7.0, "cpu") == 7.0
    assert bench.whole_job_rate(100, 1, 4, 2.0) == pytest.approx(100 * 4 / 0.002)


def test_vcycle_words_are_those_of_its_launches():
    """Two levels, 4 x 4 and 2 x 2 columns of 3 cells. Fine: a relaxation from
    zero (7), the residual with its restriction (7.25), the prolongation
    (2.25), a relaxation (8). Coarse: one relaxation from zero and seven more."""
    from types import SimpleNamespace

    import bench
    opts = SimpleNamespace(max_levels=12, min_coarse=2, nu1=1, nu2=1, nu_coarse=8)
    assert bench.vcycle_words(4, 4, 3, opts) == (48 * 24.5 + 12 * 63, 2)
    opts.nu1 = 0  # the fine correction is zero until the prolongation
    assert bench.vcycle_words(4, 4, 3, opts) == (48 * 17.5 + 12 * 63, 2)
