"""The benchmark's printed line: one JSON object that a log's tail holds whole, with the
keys that its readers need, however much the run recorded."""
import json
import math

import bench

KEYS = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
        "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "roofline")


def _errors():
    return {k: {f: math.pi * 1e-5 for f in bench.FIELDS} for k in ("rel_l2", "rel_linf", "mom_l2", "mom_linf")}


def _record(steps):
    """A run's full record with every form, as main() fills it in."""
    ms = {"fill_prim": 0.6906, "face_y": 19.5411, "face_z": 18.2445, "xface_update": 27.0714, "viscous": 5.9034}
    fma = {"fp64": 36.09, "fp32": 68.08}
    hbm, comp = bench.rooflines("fp64_char", ms, 512, 75.02977905273437, {"hbm_gbs": 6550.7}, fma, 1)
    hist = {k: [math.pi] * steps for k in ("step", "time", "kinetic", "enstrophy")}
    forms = {}
    for f in bench.FORMS:
        forms[f] = {"value": 5366578298.424641, "ms_per_step": 75.02977905273437, "gpu_launches": 150,
                    "vs_fp64_char": 0.9335860842737383, "kernel_ms_per_step": ms, "roofline": hbm,
                    "compute_roofline": comp, "history": hist, "sensor_fraction": 0.10043443785662853,
                    "errors_vs_fp64_char": dict(_errors(), steps=steps)}
    train = {"faces": 45066240, "epoch_loss": [0.17900866270065308] * 5, "seconds": 0.9023167529999796,
             "held_out": {"faces": 5007360, "precision": 0.5635645920077867, "recall": 0.9822472025635314}}
    sod = {"workload": "sod " * 80, "t_end": 0.2, "steps": 1210, "fp64_char_nonfinite": False,
           "forms": {f: dict(_errors(), time=0.2011307, sensor_fraction=None, cell_updates_per_s=6340321947.223903)
                     for f in ("fp64_comp", "fp32_char", "fp32_comp", "fp32_sensor", "fp32_sensor_p4")}}
    sample = bench._ref_sample_text("tgv", 256, 512, 16, 2)
    return {
        "metric": bench.METRIC, "value": 5366578298.424641, "unit": bench.UNIT, "n_gpus": 1, "steps": steps,
        "warmup": 5, "ms_per_step": 75.02977905273437, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": bench.workload_name("tgv", 512, "fp64_char"), "grid": [512] * 3, "form": "fp64_char",
                   "l2": "no flush: device state 22.2 GB > 126 MB L2",
                   "parallelism": "1 independent replica(s), no data-path collective"},
        "roofline": hbm, "compute_roofline": comp, "kernel_ms_per_step": ms,
        "cpu_baseline": {"value": 6756897.0, "unit": bench.UNIT, "cores": 16, "kind": "reference", "sample": sample,
                         "seconds": 14.89785},
        "e2e": {"value": 1649673261.2862763, "unit": bench.UNIT, "h2d_bytes_per_step": 5559673280,
                "d2h_bytes_per_step": 5559673280, "steps": 3, "api": "ns_time_step"},
        "gpu_launches": 150,
        "clocks": {"sm_mhz": 1792.0, "sm_max_mhz": 1965.0, "reasons": ["sw_power_cap"], "samples": 11},
        "forms": forms, "sensor_training": {"physical": train, "reference": train}, "sod_512x128x128": sod,
    }


def test_line_is_short_and_whole():
    rec = _record(steps=50)
    assert len(json.dumps(rec)) > 4 * bench.MAX_LINE  # what a run of all forms records
    text = bench.result_line(rec)
    assert "\n" not in text and len(text) <= bench.MAX_LINE
    line = json.loads(text)
    for k in KEYS:
        assert k in line, k
    for k in ("value", "ms_per_step", "steps", "gpu_launches", "clocks"):
        assert line[k] == rec[k], k
    assert line["config"]["form"] == "fp64_char" and line["e2e"] == rec["e2e"]
    # the metric's other half: the FP32 and sensor forms' rates at their stated errors
    f = line["forms"]["fp32_sensor"]
    assert f["value"] == float("%.5g" % rec["value"]) and len(f["rel_l2"]) == len(line["fields"]) == 5
    assert set(line["sod_512x128x128"]["forms"]) == set(rec["sod_512x128x128"]["forms"])


def test_line_of_failed_parts_and_of_a_run_without_extras(tmp_path, capsys):
    rec = _record(steps=3)
    rec["forms"]["fp32_char"] = {"error": "x" * 5000}
    rec["sod_512x128x128"] = {"error": "y" * 5000}
    rec["cpu_baseline"] = {"error": "z" * 5000}
    text = bench.result_line(rec)
    assert len(text) <= bench.MAX_LINE and json.loads(text)["value"] == rec["value"]
    bare = {k: rec[k] for k in KEYS}
    bench.report(bare, str(tmp_path / "full.json"))
    assert json.loads(capsys.readouterr().out)["value"] == rec["value"]
    assert json.load(open(tmp_path / "full.json")) == bare
