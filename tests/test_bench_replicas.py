"""The multi-GPU form of the benchmark is independent replicas (the operator
does not shard without a halo exchange): each rank times its own sweep, the
job's time is the max over ranks, the rate counts every rank's work.  The
aggregation runs here on CPU with two gloo ranks; the reference arm does its
work on rank 0 only."""

from __future__ import annotations

import os
import socket

import pytest
import torch.multiprocessing as mp


def _free_port() -> int:
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        return s.getsockname()[1]


def _rank_main(rank, world, port, out):
    import torch.distributed as dist

    import bench
    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port))
    dist.init_process_group("gloo", rank=rank, world_size=world)
    try:
        local_s = 1.0 + rank                      # rank 1 finishes last
        job_s = bench.max_over_ranks(local_s, "cpu")
        out[rank] = (job_s, bench.replica_rate(100.0, job_s, world))
    finally:
        dist.destroy_process_group()


def test_two_gloo_replicas_aggregate_by_the_slowest_rank():
    world, port = 2, _free_port()
    with mp.Manager() as mgr:
        out = mgr.dict()
        mp.spawn(_rank_main, args=(world, port, out), nprocs=world, join=True)
        res = dict(out)
    assert res[0] == res[1] == (2.0, 100.0)       # 2 x 100 units in 2 s


def test_single_process_is_unchanged():
    import bench
    assert bench.max_over_ranks(3.5, "cpu") == 3.5
    assert bench.replica_rate(10.0, 2.0, 1) == 5.0


def test_reference_arm_does_no_work_off_rank_zero(monkeypatch, capsys):
    import bench
    monkeypatch.setenv("RANK", "1")
    monkeypatch.setenv("WORLD_SIZE", "2")
    calls = []
    monkeypatch.setattr(bench, "run_oracle_sweep", lambda *a, **k: calls.append(a))

    class Args:
        cpu_scale, warmup, steps = 4, 1, 1
    bench.reference_arm(Args())
    assert not calls and capsys.readouterr().out == ""


def test_printed_line_is_short_and_keeps_the_results():
    """The record of a full run is tens of kilobytes (every variant of every case); the
    printed line has every result in a few."""
    import json

    import bench
    variants = {f"{eq}{p}": {f"variant {k}, its grid and products": 1.0 / (7 + k)
                             for k in range(11)} for eq, p, _ in bench.CASES}
    extra = {"value": 1.0 / 3.0, "unit": bench.UNIT, "ms_per_step": 19.9, "ok": True,
             "workload": "w" * 100, "variant_ms": variants, "variant_rel_l2": variants}
    record = {
        "metric": bench.METRIC, "value": 1e10 / 3.0, "unit": bench.UNIT, "n_gpus": 1,
        "steps": 20, "warmup": 5, "ms_per_step": 100.0 / 3.0, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": bench.WORKLOAD, "precision": "fp64"}, "gflops_suite": 1.0 / 3.0,
        "e2e": {"value": 1e9 / 7.0, "unit": bench.UNIT, "h2d_bytes_per_step": 10**10,
                "d2h_bytes_per_step": 10**10, "host_matches_device": True,
                "step_ms": [123.4] * 5, "split_ms": dict.fromkeys("abcdefgh", 12.34),
                "logged_steps": [dict.fromkeys("abcdefgh", 1.0 / 3.0)] * 5, "overlap": "o" * 300},
        "roofline": {"bound": "hbm", "achieved": 1.0 / 3.0, "kernel": "k" * 80,
                     "fp64_pipe": {"frac": 1.0 / 3.0}},
        "cpu_baseline": {"value": 5e7 / 3.0, "sample": "s" * 80},
        "parity": {"bound": 1e-12, "max_rel_l2": 9.9e-14, "ok": True, "cases": variants},
        "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []},
        "gpu_launches": 560, "autotuned_variant": dict.fromkeys(variants, 2), "setup_s": 9.0 / 7.0,
        "cases": [{"case": f"{eq} P{p} n={n}", "nel": 6 * n**3, "ms": 10.0 / 3.0,
                   "gdof_s": 1.0 / 3.0, "fp64_frac": None} for eq, p, n in bench.CASES],
        "extras": {f"extra_{k}": dict(extra) for k in range(6)} | {"bad": {"error": "e" * 1000}},
    }
    line = bench.result_line(record)
    assert len(json.dumps(record)) > 20000 and len(json.dumps(line)) < 6000
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
                "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config",
                "roofline", "cpu_baseline", "clocks", "gpu_launches"):
        assert line[key] == record[key]
    for key in ("value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"):
        assert line["e2e"][key] == record["e2e"][key]
    assert line["case_ms"]["maxwell P4"] == 3.3333 and len(line["case_ms"]) == 12
    assert line["extras"]["extra_0"] == {"value": 0.33333, "ms_per_step": 19.9, "ok": True}
    assert line["extras"]["bad"] == {"error": "e" * 100}
    assert len(record["cases"]) == 12 and "extras" in record      # left as it was
