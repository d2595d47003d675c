"""Host-side helpers of bench.py on CPU: the whole-job throughput and the histogram quantiles
that the 4096^2 precision ablation reports."""
from __future__ import annotations

import numpy as np
import torch

import bench


def test_job_throughput_counts_every_rank():
    # 2 ranks x 1000 rays in 2 ms (the slowest rank) = 1 Mrays/s
    assert abs(bench.job_mrays_s(1000, 2, 2.0) - 1.0) < 1e-12


def test_histogram_quantiles_are_within_one_bin():
    rng = np.random.default_rng(0)
    x = torch.tensor(10.0 ** rng.uniform(-9.0, -2.0, size=200_000))
    hist = torch.zeros(1300, dtype=torch.float64)
    bench._log_hist(x, hist)
    assert float(hist.sum()) == x.numel()
    for q in (0.5, 0.99, 0.999):
        exact = float(np.quantile(x.numpy(), q))
        got = bench._hist_quantile(hist, q)
        assert exact <= got <= exact * 10 ** 0.02 * 1.0001, (q, exact, got)
    # zeros land in the first bin
    hz = torch.zeros(1300, dtype=torch.float64)
    bench._log_hist(torch.zeros(10, dtype=torch.float64), hz)
    assert float(hz[0]) == 10
    assert bench._hist_quantile(torch.zeros(1300, dtype=torch.float64), 0.5) is None


def test_both_arms_describe_the_same_workload(kt, orc):
    """bench.py's own arm builds its scene through the library's host entry points, the
    reference arm through the oracle's restatement (so that it loads no product library); both
    must print the same config.workload and see the same scene and camera bits."""
    from kerrtrace_b200 import workloads
    for size in (None, "480x270"):
        c_lib, cam_lib = bench.rank_camera(workloads, "c2", 0, 1, size)
        c_ref, cam_ref = bench.rank_camera(workloads, "c2", 0, 1, size, host=orc.Host())
        assert bench.workload_label("c2", c_lib) == bench.workload_label("c2", c_ref)
        assert bytes(c_lib) == bytes(c_ref) and bytes(cam_lib) == bytes(cam_ref)


def test_headline_line_keeps_its_keys_and_stays_short():
    """The stdout line: headline keys whole, of each leg the plain values only, and a few KB however many
    rows the tables of a leg hold."""
    import json
    rows = [{"ms": 1.0 + i, "tuning": {"schedule": 0}} for i in range(500)]
    line = {"metric": "m", "value": 1.5, "config": {"tuning": {"block_x": 8}, "l2": "flushed"},
            "e2e": {"value": 1.0, "h2d_bytes_per_step": 52}, "roofline": {"frac": 0.5, "work": {"rays": 1}},
            "clocks": {"sm_mhz": 1965.0, "reasons": []}, "gpu_launches": 30,
            "autotune": {"best": {"block_x": 8}, "best_ms": 2.0, "top": rows, "candidates": 500},
            "precision": {"fp64": {"mrays_s": 3.0, "tuning": {"a": 1}, "err": {"p99": 1.0}}, "clocks": {"sm_mhz": 1.0}},
            "pareto": {"scenes": {"c2": {"size": "1x1", "points": rows}}, "tolerances": [1e-5] * 500},
            "c3": {"size": 4096, "runs": rows}, "batch": {"tuner": rows, "batched_launch": {"mrays_s": 1.0}}}
    out = bench.headline(line)
    for k in ("metric", "value", "config", "e2e", "roofline", "clocks", "gpu_launches"):
        assert out[k] == line[k]
    assert out["autotune"] == {"best_ms": 2.0, "candidates": 500, "best": {"block_x": 8}}
    assert out["precision"] == {"fp64": {"mrays_s": 3.0}} and out["c3"] == {"size": 4096}
    assert out["batch"] == {"batched_launch": {"mrays_s": 1.0}} and out["pareto"] == {}
    assert len(json.dumps(out)) < 2000
