"""The benchmark's result line stays short whatever the details hold: one line is JSON,
it is the last one, fits the end of a captured output and carries the headline.  CPU
only."""
import json
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))


def test_one_short_json_line_at_the_end(capsys):
    import bench
    headline = {"metric": bench.METRIC, "value": 1.75e9, "unit": bench.UNIT, "n_gpus": 1,
                "steps": 20, "warmup": 5, "ms_per_step": 15.0,
                "config": {"workload": "orszag_tang_512x512_mlw_m3"},
                "e2e": {"value": 1.7e9, "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 1},
                "gpu_launches": 8000, "clocks": {"sm_mhz": 2070}}
    long = {k: {f"case_{i}": {"ms": 1.0 / (i + 3)} for i in range(900)}
            for k in ("df64_policy", "parity_vs_oracle", "workloads")}
    bench.emit({**headline, **long, "cpu_baseline": {"value": 9e7}})
    lines = capsys.readouterr().out.splitlines()
    assert [ln.startswith("{") for ln in lines] == [False, True]
    assert len(lines[-1]) < 4000
    assert json.loads(lines[-1]) == {**headline, "cpu_baseline": {"value": 9e7}}
    name, _, details = lines[0].partition(" ")
    assert name == "details" and json.loads(details) == long
