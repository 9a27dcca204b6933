"""The benchmark's stdout line: one JSON object that fits the tail of a log, details on stderr."""
import importlib.util
import json
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _bench():
    spec = importlib.util.spec_from_file_location("cfft_bench_line", os.path.join(ROOT, "bench.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_line_is_short_and_whole(capsys):
    b = _bench()
    third = 10000000 / 3
    contract = {"metric": b.METRIC, "value": third, "unit": "products/s", "n_gpus": 1, "steps": 20, "warmup": 5,
                "ms_per_step": third / 1e7, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
                "dtype": "f64", "data": "synthetic (seeded numpy PCG64)"}
    line = dict(contract, config={"workload": "w" * 120, "l2": "inputs 384 MiB > L2 (no flush needed)"},
                roofline={"frac": third, "fp64": b.fp64_roof(3.0, 2.0, third, third)},
                plain_path={"note": "x" * 400, "value": third}, cpu_baseline={"sample": "y" * 400, "value": third},
                accuracy={"bound": "z" * 1600, "worst_bits": third, "ok": True},
                e2e={"value": third, "h2d_bytes_per_step": 1, "d2h_bytes_per_step": 1},
                clocks={"sm_mhz": 2070, "sm_max_mhz": 2070, "reasons": []}, gpu_launches=20)
    configs = {"config_%d" % i: {"value": third, "rows": ["r" * 50] * 100} for i in range(6)}
    configs["failed"] = {"error": "e" * 500}
    b.print_headline(line, dict(line, configs=configs))
    out, err = capsys.readouterr()
    assert out.count("\n") == 1 and len(out) <= b.LINE_MAX
    got = json.loads(out)
    assert set(got) == set(line) | {"configs"}
    assert abs(got["value"] / third - 1) < 1e-6 and got["accuracy"]["ok"] and "bound" not in got["accuracy"]
    assert got["configs"]["config_0"] == 3333300.0 and got["configs"]["failed"] == "error"
    assert json.loads(err)["configs"] == configs and json.loads(err)["value"] == third


def test_issued_fp64_instructions():
    """8192 products of N = 2048 on Dif4 executed 12.66 M FP64 warp instructions: the counted ones and
    the conversions of fold and round."""
    b = _bench()
    issued = b.fp64_ops_per_product(2048, 1024, 2, b.CORE_ISSUED) * 8192 / 32
    assert 0.9 * 12.66e6 < issued < 12.66e6
    for algo in range(8):
        assert b.fp64_ops_per_transform(2048, 512, algo, b.CORE_ISSUED) < b.fp64_ops_per_transform(2048, 512, algo)
