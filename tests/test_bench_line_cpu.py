"""bench.py's printed line: every key of the metric, and short enough for a
reader that keeps a few kilobytes, however long the record is."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def record():
    solve = {k: {"solve_ms": 83.024834678, "iterations": 657, "true_relres": 9.69e-9, "error_vs_oracle": 3.4e-15}
             for k in ("fp64", "mixed")}
    work = {"value": 11527588893.7, "ms_per_step": 2.7588160276412963, "nnz": 31802497, "element_ms": 2.2035,
            "gather_ms": 0.5553, "config": {"workload": "w" * 80, "step": "s" * 80}, "gpu_launches": 10,
            "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []},
            "roofline": {"bound": "fp64", "achieved": 437.8, "peak": 526.6, "unit": "G", "frac": 0.83, "kernel": "k",
                         "note": "n" * 400},
            "cpu_baseline": {"value": 2.1e8, "unit": "nnz/s", "cores": 16, "kind": "port", "sample": "x" * 60,
                             "bit_exact_vs_gpu": True, "plan_baselines": {"B": "y" * 500}},
            "minimal_formulation": {"ms_per_step": 2.25, "note": "n" * 600},
            "structure": {"node_cell_ms": 0.73, "sparsity_ms": 0.89, "note": "n" * 60},
            "e2e": {"value": 9.6e9, "unit": "nnz/s", "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 2,
                    "ms_per_step": 3.3, "includes": "z" * 500}, "solve": dict(solve, bc={"steps": "t" * 300})}
    learned = {k: {"solve_ms": 2.1, "iterations": 12, "status": 0} for k in
               ("plain_fp64_cg_jacobi", "fcg_vcycle_untrained", "fcg_learned")}
    return {"metric": "assembled nnz/s", "unit": "nnz/s", "n_gpus": 1, "steps": 20, "warmup": 5,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            **work, "workloads": {k: work for k in ("elasticity3d", "poisson2d", "poisson3d_hex")},
            "learned": dict(learned, network="n" * 300),
            "batched": {"instances": 64, "rhs_per_instance": 4, "batch_ms": 413.8, "max_relres": 9.5e-9,
                        "config": {"c": "d" * 300}}}


def test_the_line_has_the_metric_and_is_short():
    import bench
    full = record()
    line = json.dumps(bench.headline(full))
    assert len(line) < 4096 and "\n" not in line
    out = json.loads(line)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "gpu_launches", "clocks"):
        assert out[k] == full[k], k
    assert {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"} <= set(out["e2e"])
    assert out["sections"]["elasticity3d"]["solve"]["mixed"]["iterations"] == 657


def test_sections_that_were_skipped_are_left_out():
    import bench
    full = record()
    for k in ("e2e", "solve", "cpu_baseline"):
        del full[k]
    full.update(workloads={}, learned=None, batched=None)
    out = json.loads(json.dumps(bench.headline(full)))
    assert "e2e" not in out and out["sections"]["main"]["solve"] == {} and out["sections"]["learned"] is None
