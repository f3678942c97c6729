"""The result line of bench.py: whole for a reader that keeps the last 3000 characters of the output,
with the measured entries untouched, whatever else ran."""
import json
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def _bench():
    if str(ROOT) not in sys.path:
        sys.path.insert(0, str(ROOT))
    import bench

    return bench


def _result(filler):
    head = {"plain_ms": 293.26490020751953, "plain": "measured", "plain_spp": 128, "denoised_ms": 4.150976002216339,
            "denoised_input_spp": 1, "speedup": 70.6496255461212}
    return {
        "metric": "Mrays/s", "value": 2765.432109876543, "unit": "Mrays/s", "n_gpus": 1, "steps": 20, "warmup": 5,
        "ms_per_step": 18.123456789012345, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "f32", "data": "synthetic",
        "config": {"workload": "icospheres-256 1920x1080 8spp depth8", "width": 1920, "height": 1080, "spp": 8,
                   "depth": 8, "count": 256, "level": 4, "seed": 0, "triangles": 1310720,
                   "rays_per_frame": 50123456.0, "l2": "flushed (512 MiB write) before every timed step",
                   "parallelism": "replicas x1"},
        "roofline": {"bound": "l2", "kernel": "k_trace_dyn<closest-hit>", "achieved": 12345.678901234567,
                     "peak": 23456.78901234567, "unit": "GB/s", "frac": 0.5263157894736842, "traffic": 2061000000,
                     "peak_source": filler, "achieved_basis": filler},
        "blas": {"shared": {"note": filler}}, "bvh_build_ms": {"default": 50.1, "gpu_lbvh": 40.2, "note": filler},
        "cpu_baseline": {"value": 3.3765428920679215, "unit": "Mrays/s", "cores": 16, "kind": "port",
                         "sample": "512x512 centre crop", "cornell_256_64spp": {"sample": filler}},
        "e2e": {"value": 2600.0, "unit": "Mrays/s", "h2d_bytes_per_step": 5000, "d2h_bytes_per_step": 8294400},
        "clocks": {"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "reasons": []}, "gpu_launches": 1280,
        "time_to_relmse": {"scene": filler, "headline_tau": 1e-3, "headline": head, "thresholds": [filler] * 9,
                           "shipped_network": {"headline": head, "denoised": [filler]},
                           "mixed_network": {"headline": head, "training": filler},
                           "icosphere_headline": {"mixed": head, "in_run": head},
                           "denoiser_roofline": {"bound": "tensor", "achieved": 712.7, "peak": 1954.3, "frac": 0.36}},
        "batched": {"workload": filler, "default": {"ms_per_batch": 373.9, "mrays_s": 4007.7},
                    "autotuned": {"ms_per_batch": 356.0, "mrays_s": 4209.9}},
        "active_light": {"workload": filler, "ms_per_batch": 7.28, "mrays_s": 4980.4, "rgb_denoise_ms": 0.41},
    }


def test_line_fits_and_keeps_what_was_measured(capsys):
    bench = _bench()
    full = _result("x" * 900)
    bench.print_result(full)
    cap = capsys.readouterr()
    (line,) = cap.out.splitlines()
    assert len(line) <= bench.LINE_LIMIT <= 2800
    got = json.loads(line)
    for k in bench.CONTRACT:
        assert got[k] == full[k], k
    assert got["time_to_relmse"]["mixed"]["speedup"] == 70.6496
    assert got["batched"]["default"]["mrays_s"] == 4007.7 and got["roofline"]["frac"] == 0.526316
    details = dict(l.removeprefix("detail ").split(": ", 1) for l in cap.err.splitlines())
    assert {k: json.loads(v) for k, v in details.items()} == {k: v for k, v in full.items() if isinstance(v, dict)}


def test_line_without_the_further_parts_and_with_failed_ones():
    bench = _bench()
    full = {k: v for k, v in _result("x").items() if k in bench.CONTRACT}
    assert json.loads(bench.result_line(full)) == full
    full.update(time_to_relmse={"error": "OSError: " + "y" * 5000}, batched={"error": "KfError: no memory"})
    got = json.loads(bench.result_line(full))
    assert got["batched"] == {"error": "KfError: no memory"} and len(json.dumps(got)) <= bench.LINE_LIMIT
    assert got["value"] == full["value"]
