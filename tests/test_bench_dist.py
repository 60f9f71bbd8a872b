"""The benchmark's multi-process plumbing on the CPU: two gloo ranks.

``bench.py`` runs one process per GPU; the ranks share nothing on the data
path (independent lattices / requests) and meet only in a barrier and a max
over ranks.  Here that plumbing runs as two gloo ranks, and the reference arm
runs under the real launcher with world size 2 (rank 0 alone prints).
"""
import json
import multiprocessing
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


def _rank_main(rank, port, out):
    os.environ.update({"WORLD_SIZE": "2", "RANK": str(rank), "LOCAL_RANK": str(rank),
                       "MASTER_ADDR": "127.0.0.1", "MASTER_PORT": str(port),
                       "XK_BENCH_BACKEND": "gloo"})
    sys.path.insert(0, ROOT)
    import bench
    from xentica_gb300.batch import ensemble_workload
    dist = bench.Dist()
    try:
        dist.barrier()
        top = dist.max(1.5 + rank)
        # each rank seeds its own lattices, as run_ours does
        widths, heights, rules, _, cells = ensemble_workload(3, 2041 + 7919 * rank)
        out.put((rank, dist.world, top, int(cells.sum()), list(rules)))
    finally:
        dist.close()


def test_barrier_and_max_over_two_gloo_ranks():
    ctx = multiprocessing.get_context("spawn")
    out = ctx.Queue()
    port = _free_port()
    procs = [ctx.Process(target=_rank_main, args=(r, port, out)) for r in range(2)]
    for p in procs:
        p.start()
    res = sorted(out.get(timeout=180) for _ in procs)
    for p in procs:
        p.join(timeout=60)
        assert p.exitcode == 0
    assert [r[1] for r in res] == [2, 2]
    assert [r[2] for r in res] == [2.5, 2.5]          # the max reaches every rank
    assert res[0][3:] != res[1][3:]                    # ranks hold different lattices


def test_reference_arm_under_the_launcher():
    env = dict(os.environ, XK_BENCH_BACKEND="gloo")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node", "2",
           "--master-addr", "127.0.0.1", "--master-port", str(_free_port()),
           os.path.join(ROOT, "bench.py"), "--impl", "reference", "--gpus", "2", "--steps", "1",
           "--warmup", "0", "--cpu-seconds", "1", "--instances", "4"]
    proc = subprocess.run(cmd, cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert proc.returncode == 0, proc.stderr[-2000:]
    lines = [l for l in proc.stdout.splitlines() if l.startswith("{")]
    assert len(lines) == 1                             # rank 0 alone prints
    line = json.loads(lines[0])
    assert line["impl"] == "reference" and line["n_gpus"] == 2
    assert line["value"] > 0 and line["cpu_baseline"]["cores"] >= 1
    assert line["e2e"]["h2d_bytes_per_step"] == 0


def test_default_line_is_short_and_last(capsys):
    """The default run's JSON line holds what a reader of the output's end
    needs, in at most 2400 characters; the parts go before it, none of them a
    line that starts as JSON."""
    import bench
    long = "x" * 300
    part = {"value": 1.0 / 3, "note": long, "parity": {"bit_exact": True, "note": long}}
    line = {"metric": bench.METRIC, "value": 2.1468494262370832e13, "unit": "cell-updates/s", "n_gpus": 1,
            "steps": 20, "warmup": 5, "ms_per_step": 7.62847363948822, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "u8",
            "data": "synthetic (seeded Bernoulli lattices, random rules)",
            "config": {"workload": "ensemble of 4096 LifelikeCA lattices x 256 generations per step",
                       "instances": 4096, "generations_per_step": 256, "cells": 639733760,
                       "sides": [64, 128, 256, 512, 1024],
                       "l2": "inputs (640 MB) larger than L2, no flush", "rows_per_band": 16,
                       "parallelism": "replicas x1"},
            "e2e": {"value": 1.882642715356418e13, "unit": "cell-updates/s", "h2d_bytes_per_step": 639733760,
                    "d2h_bytes_per_step": 639733760, "ms_per_step": 8.69903998374939},
            "plain": part, "reference_gpu": part, "seeding": part,
            "parity": {"lattices": 25, "size_classes": 25, "generations": 256, "band": 16, "bit_exact": True,
                       "note": long},
            "gpu_launches": 140, "wall_s": 0.1531725760000029,
            "roofline": {"bound": "hbm", "achieved": 42936.98852474166, "peak": 6785.9, "unit": "GB/s",
                         "frac": 6.327383033163127, "peak_kind": "measured", "traffic": 947253778.4319999,
                         "kernel": "xk_k_life_resident<true> (all instance classes of one graph)",
                         "algorithmic_bytes_per_launch": 327543685120.0, "note": long,
                         "bit_packed": {"bytes_per_cell_update": 0.25, "achieved": 5367.123565592708,
                                        "frac": 0.7909228791453908}},
            "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": [], "samples": 4},
            "cpu_baseline": {"value": 384767722.12694144, "unit": "cell-updates/s", "cores": 16,
                             "kind": "reference",
                             "sample": "25 lattices (one per size class, 3936256 cells) x 1174 generations, "
                                       "12.0 s, reference LifelikeCA kernels compiled for the CPU (OpenMP)"},
            "extras": {name: part for name in ("life512", "evolife", "mass")}}
    bench.report(line)
    out = capsys.readouterr().out.splitlines()
    assert [o.split()[1] for o in out[:-1]] == ["plain", "reference_gpu", "seeding", "life512", "evolife",
                                               "mass", "roofline", "parity", "cpu_baseline"]
    assert all(o.startswith("# ") and json.loads(o.split(" ", 2)[2]) for o in out[:-1])
    assert len(out[-1]) <= 2400
    last = json.loads(out[-1])
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
                "scaling", "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "roofline",
                "parity", "cpu_baseline"):
        assert key in last, key
    assert last["value"] == line["value"] and last["e2e"] == line["e2e"] and last["parity"]["bit_exact"]
