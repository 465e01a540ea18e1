"""The line that bench.py prints fits the end of an output that a reader keeps
(8 KB), with every key of the benchmark's contract; the whole record goes to a
file."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

MODES = ("plain", "plain_direct_uvort", "plain_perturbed", "mixed", "mixed_f64uvort", "learned")
CONTRACT = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
            "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "config", "clocks",
            "e2e", "gpu_launches", "roofline", "cpu_baseline")


def record():
    """A record of the default workload's shape and more than its length."""
    import bench
    f = 1.0 / 3.0
    steps = [f * 1e-8] * 20
    line = {k: f for k in CONTRACT + bench.LINE_KEYS}
    kernel = dict(kernel="k" * 70, bound="fp32", limited_by="x" * 40, achieved=f, peak=f,
                  unit="TFLOP/s", frac=f, traffic=10 ** 9, peak_source="p" * 60, flop_per_pair=31,
                  fma_pipe_active_ncu=f, pairs=10 ** 10, ms=f)
    clocks = dict(sm_mhz=1965.0, sm_max_mhz=1965.0, reasons=["sw_power_cap"])
    line.update(
        mode="mixed", headline_rule="h" * 500, clocks=clocks, load_error_note="n" * 500,
        config=dict(model="m" * 60, workload="w" * 400, l2="l" * 80, parallelism="p" * 60),
        e2e=dict(value=f, unit="ms", h2d_bytes_per_step=10 ** 9, d2h_bytes_per_step=10 ** 9,
                 note="n" * 300),
        cpu_baseline=dict(value=f, unit="ms", cores=16, kind="port", sample="s" * 500),
        load_error_max_over_steps={k: f for k in MODES}, loads_by_step={k: [steps] * 20 for k in MODES},
        load_error_by_step={k: steps for k in MODES},
        modes={k: dict(ms=f, load_error_vs_fp64=f, load_error_max_over_steps=f,
                       particle_error_vs_fp64=dict(vel=f), solve=dict(residual=f)) for k in MODES},
        phases_ms={k: {"phase_%d" % i: f for i in range(20)} for k in MODES},
        roofline=dict(kernel, others=[dict(kernel, flops=dict(kernel)) for _ in range(4)]),
        workloads=dict(
            fmm=dict(results={"p%d_%s" % (p, m): dict(ms=f, roofline=kernel) for p in (4, 6, 8)
                              for m in ("fp64", "fp32c")}),
            dense=dict(results={m: dict(ms=f, backward_error=f, report=kernel)
                                for m in ("lu64", "mixed")}),
            learned=dict(results={m: dict(ms_mean=f, iterations_mean=f, fallbacks=0)
                                  for m in ("lu64", "gmres_untrained", "gmres_nn")}),
            wing=dict(ms_per_step_mean=f, ms_per_step_last20=f, phases_ms_last20=dict(live=f),
                      solution_rel_error_vs_oracle_max_over_steps=f)))
    return line


def test_line_is_short_and_whole(tmp_path):
    import bench
    line = record()
    path = str(tmp_path / "details.json")
    bench.write_details(line, path)
    text = json.dumps(bench.short_line(line, path))
    assert len(text) < 8000 < len(json.dumps(line))
    got = json.loads(text)
    for k in CONTRACT:
        assert got[k] == line[k] or k == "roofline"
    for k in ("kernel", "bound", "achieved", "peak", "unit", "frac", "traffic"):
        assert got["roofline"][k] == line["roofline"][k]
    assert got["phases_ms"] == line["phases_ms"]["mixed"]
    assert got["workloads"]["fmm"]["p4_fp32c"] == {"ms": 1.0 / 3.0}
    assert json.load(open(path)) == line


def test_details_that_cannot_be_written(tmp_path):
    import bench
    assert bench.write_details({}, str(tmp_path / "no" / "such" / "folder.json")) is None
