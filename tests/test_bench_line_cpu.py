"""The GPU arm's line is short enough for a log's tail and keeps the contract's keys; the studies
that it summarises are whole in the details."""
import json
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
import bench  # noqa: E402


def test_line_of_a_full_run_fits_a_tail():
    x = 123456.78901234567
    run = {"tol": 1e-8, "seconds": x, "iterations": 123456, "rel_err": x, "rel_residual": x,
           "status": 0, "outer": 1, "fallback": 0}
    solver = dict(run, met=True, runs=[run] * 11, label="a solver " * 9, total_seconds=x,
                  total_includes="FP64 assembly + FP32 copy + solver layout + two-level set-up + solve")
    names = list(bench.SOLVER_TABLE)
    solve = dict({n: dict(solver) for n in names}, target_rel_error=1e-8, layout_seconds=x,
                 coarse_unknowns=3072, reference_solution={"how": "so " * 60, "rel_residual_history": [x] * 9},
                 cpu_reference={"label": "extrapolated " * 20},
                 speedup_total_vs_pcg_fp64={n: x for n in names})
    roof = {"bound": "hbm", "achieved": x, "peak": x, "unit": "GB/s", "frac": x, "us_per_launch": x,
            "traffic": {"bytes": 123456789, "source": "profiles/ncu_traffic.json"}, "algorithmic_bytes": 10**9}
    cube = {"edge": 44, "dofs": 273375, **{n: dict(run) for n in ("pcg_fp64", "twolevel_pcg", "learned_fcg")}}
    ratios = {f"median_{k}_ratio_{a}_over_{b}": x for k in ("iterations", "seconds")
              for a, b in (("learned_fcg", "pcg_fp64"), ("twolevel_pcg", "pcg_fp64"), ("learned_fcg", "twolevel_pcg"))}
    line = {"metric": bench.METRIC, "value": x, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": x, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic", "config": {"model": "m" * 60, "elements": 262144, "l2": "flushed " * 20},
            "matrix": {"dofs": 1577986, "nnz": 10**8, "ell_width": 42}, "timing": "device time " * 10,
            "value_with_pattern": {"value": x, "unit": bench.UNIT, "ms_per_step": x, "includes": "i" * 60},
            "roofline": roof, "roofline_assembly": dict(roof), "roofline_spmv": dict(roof), "scatter": "auto",
            "scatter_variants": {n: {"value": x, "unit": bench.UNIT, "ms": x} for n in
                                 ("owner", "colour", "atomic", "atomic_tcgen05", "owner_tcgen05")},
            "e2e": {"value": x, "unit": bench.UNIT, "h2d_bytes_per_step": 10**8, "d2h_bytes_per_step": 10**9,
                    "includes": "mesh upload, pattern, assembly, ELL download"},
            "gpu_launches": 40, "clocks": {"sm_mhz": 1965, "sm_max_mhz": 1965, "reasons": ["sw_power_cap"]},
            "solve": solve, "brick20_64": {"workload": "brick20_64", "assembly": {}, "solve": dict(solve)},
            "learned": {"summary": dict(ratios, application_brick8_48={"us": x}), "held_out": [cube] * 16},
            "cpu_baseline": {"value": x, "unit": bench.UNIT, "cores": 1, "kind": "port", "sample": "Q8 " * 20}}
    assert len(json.dumps(line)) > 20000
    short, details = bench.short_line(dict(line))
    assert len(json.dumps(short)) <= 3000, len(json.dumps(short))
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
                "scaling", "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks",
                "roofline", "cpu_baseline"):
        assert short[key] == line[key]
    assert all(details[k] == line[k] for k in details) and set(line) == set(short)
    assert short["solve"] == {"target_rel_error": 1e-8, "total_seconds": {n: 123500.0 for n in names}}


def test_line_without_studies():
    line = {"value": 1.0, "solve": None, "brick20_64": None, "learned": None, "scatter_variants": {},
            "roofline_assembly": {"achieved": 1.0, "frac": 0.5, "unit": "GB/s"}}
    short, details = bench.short_line(line)
    assert short == {"value": 1.0, "roofline_assembly": {"achieved": 1.0, "frac": 0.5}}
    assert details == {"roofline_assembly": line["roofline_assembly"]}
