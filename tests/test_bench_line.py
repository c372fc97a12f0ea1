"""bench.py's result line: short enough to survive where only the end of a
run's output is kept, and complete in what identifies and values the result,
however many images, sizes and rates the run measured."""
import json
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)


def full_result():
    images = [[1.23e-07, 4.56e-08]] * 800
    parity = {"images": 512, "pixels_checked": 131072, "max_rel_err": 1.5e-6, "rms_rel_err": 1.1e-7,
              "images_within_tolerance": 512, "tolerance": 1e-5, "per_image": images, "what": "x" * 80,
              "full_images": [{"size": "576x336", "max_rel_err": 1e-7}] * 8}
    roof = {"bound": "l2", "achieved": 16517.604136473645, "peak": 19468.774360537194, "unit": "GB/s",
            "frac": 0.8484152022406962, "units": "x" * 90, "peak_source": "y" * 200}
    return {
        "metric": "images/s & p99 latency: batched/served vs plain GPU render at ≤1e-5 rel err",
        "value": 10053.050625958678, "unit": "images/s", "n_gpus": 1, "steps": 20, "warmup": 5,
        "ms_per_step": 50.929814147949216, "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic", "config": {"workload": "w" * 160, "cube": "c" * 50, "requests": 512, "fov_deg": [27.0, 16.0],
                                        "ray_length_re": 44.0, "l2": "l" * 70, "parallelism": "1 GPU"},
        "e2e": {"value": 9959.2889167307, "unit": "images/s", "h2d_bytes_per_step": 163984, "d2h_bytes_per_step": 449360640},
        "plain": {"value": 6920.60979223019, "unit": "images/s"}, "batched_vs_plain": 1.452624974932888,
        "by_size": {f"{k}x{k}": {"batched": 1.0 / 3, "plain": 2.0 / 3} for k in range(12)}, "e2e_vs_plain": 1.4390767888,
        "e2e_breakdown": {"kernel_ms": 51.09508171081543, "d2h_ms": 0.00212, "host_ms": 0.31208973603482093},
        "serving": {"offered_rate": 7037.1, "requests": 21122, "achieved_images_s": 6991.753403954441, "p50_ms": 0.717232,
                    "p99_ms": 2.852404800000001, "runs_p50_p99_ms": [[0.7, 2.8]] * 3},
        "ray_samples_per_s": 1794965072195.9502, "roofline": roof, "roofline_issue": roof, "roofline_per_sample": roof,
        "roofline_hbm": roof, "cpu_baseline": {"value": 1.0898001383113973, "unit": "images/s", "cores": 16, "kind": "port",
                                               "sample": "s" * 190, "single_core": {"value": 0.07}},
        "gpu_launches": 120, "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": ["gpu_idle"], "samples": 30},
        "exact_fp64_rays_per_step": 1.0 / 3, "samples_per_cell": 4.346792809333324,
        "c3": {"requests": 776, "images_s": 11345.288912821643, "batched_vs_plain": 1.5025359107857015, "parity": parity},
        "c4": {"saturation_images_s": 3776.6, "sweep": [{"offered_req_s": 1.0 / 3}] * 40, "parity": parity,
               "at_70pct_of_saturation": {"served_images_s": 2654.4, "p50_ms": 2.1, "p99_ms": 11.1}}, "parity": parity}


def test_result_line():
    import bench
    full = full_result()
    text = bench.result_line(full)
    assert "\n" not in text and len(text) <= 2400
    line = json.loads(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "e2e", "plain", "gpu_launches", "clocks"):
        assert line[k] == full[k], k
    assert line["parity"]["max_rel_err"] == full["parity"]["max_rel_err"]
    assert line["c3"]["images_s"] == 11345.3 and line["c4"]["at_70pct_of_saturation"]["p99_ms"] == 11.1


def test_details_file(tmp_path, capsys):
    import bench
    path = tmp_path / "details.json"
    bench.print_result(full_result(), str(path))
    out = capsys.readouterr().out
    assert json.loads(out)["value"] == 10053.050625958678 and out.count("\n") == 1
    assert len(json.loads(path.read_text())["parity"]["per_image"]) == 800
