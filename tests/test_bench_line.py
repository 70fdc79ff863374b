"""The line that bench.py prints (no GPU)."""
import json
import os
import sys

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), ".."))
import bench  # noqa: E402


def test_stdout_is_one_short_line_and_the_records_go_to_stderr(capsys):
    contract = {"metric": "mul_mat TFLOPS", "value": 1.5, "unit": "TFLOP/s", "config": {"workload": "w" * 300}, "e2e": {"value": 1.0},
                "clocks": {"sm_mhz": 1965}, "gpu_launches": 10}
    records = {"per_shape": [{"M": i, "us": 1.0, "note": "x" * 100} for i in range(36)], "kernels": [{"kernel": "k" * 200}] * 30,
               "dev_forward_calls": {"calls": ["x" * 100] * 98, "calls_checked": 98, "worst_err": 5e-4, "checked": True},
               "sharded_block": {"ms_per_block": 1.9, "workload": "x" * 600}, "sharded_extra_block": {"ms_per_block": 2.0, "workload": "x" * 600},
               "reference_cpu_kernels": []}
    bench.print_line({**contract, **records})
    out, err = capsys.readouterr()
    assert out.endswith("\n") and out.count("\n") == 1 and len(out) < 3000
    line = json.loads(out)
    assert {k: line[k] for k in contract} == contract and not set(records) & set(line)
    assert line["detail_on_stderr"]["sharded_block"] == {"ms_per_block": 1.9} and line["detail_on_stderr"]["per_shape"] == 36
    details = [json.loads(x) for x in err.splitlines()]
    assert {d["detail"]: d["record"] for d in details} == records
