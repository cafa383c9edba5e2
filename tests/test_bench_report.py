"""The bench's output: one line of JSON on stdout that a reader who keeps the last
4 KB has whole, whatever the other workloads report."""
import importlib.util
import json
import os


def _bench():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    spec = importlib.util.spec_from_file_location("bench_report_mod",
                                                  os.path.join(root, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m, open(os.path.join(root, "bench.py")).read()


def test_stdout_is_the_headline_line(capsys):
    bench, _ = _bench()
    line = {"metric": "m", "value": 1.5, "unit": "GFLOP/s", "e2e": {"value": 1.0}}
    details = {"reference_size_sweep": [{"size": i, "ms": 0.1 * i} for i in range(5000)],
               "serving": None}
    bench.report(line, details)
    out, err = capsys.readouterr()
    assert out.count("\n") == 1 and json.loads(out) == line
    assert err.startswith("bench details: ") and err.count("\n") == 1
    assert json.loads(err[len("bench details: "):]) == details


def test_other_workloads_stay_out_of_the_line():
    _, src = _bench()
    keys = src[src.index("        line = {\n            \"metric\": \"batched FFT"):]
    keys = keys[:keys.index("        report(line, {")]
    for k in ("extra", "serving", "config4_precision", "real_transforms", "reference_size_sweep"):
        assert f'"{k}"' not in keys
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
              "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config", "e2e",
              "gpu_launches", "clocks"):
        assert f'"{k}"' in keys
