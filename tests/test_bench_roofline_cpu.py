"""The benchmark's roofline names the kernel that ran: three iterations per pass over memory at the benchmark's size, two
or three below, none where the grid stays on the chip."""
import importlib.util
import pathlib

spec = importlib.util.spec_from_file_location("bench_under_test", pathlib.Path(__file__).parents[1] / "bench.py")
bench = importlib.util.module_from_spec(spec)
spec.loader.exec_module(bench)


def test_roofline_by_what_ran():
    r = bench.roofline(2048, 30000, 10050, 1000.0, 6500.0, "measured")
    assert r["kernel"] == "k_pt_march (3 PT iterations per launch)" and r["bound"] == "hbm"
    want = 128 * 2047 ** 2 * 10000 / 1.0 / 1e9
    assert abs(r["achieved"] - want) < 0.1 and abs(r["frac"] - want / 6500.0) < 1e-4
    assert r["traffic"] == round(bench.TRAFFIC_PER_LAUNCH_2048)
    r = bench.roofline(700, 30000, 10050, 200.0, 6500.0, "measured")
    assert r["kernel"].startswith("k_pt_march (3") and r["traffic"] is None     # (its fields stay in the L2)
    assert bench.roofline(300, 30000, 15010, 100.0, 6500.0, "m")["kernel"] == "k_pt_march (2 PT iterations per launch)"
    assert bench.roofline(2048, 3000, 3000, 100.0, 6500.0, "m")["algorithmic_bytes_per_launch"] == 104 * 2047 ** 2
    r = bench.roofline(512, 30000, 70, 100.0, 6500.0, "measured")
    assert "k_pt_resident" in r["kernel"] and r["achieved"] is None and r["frac"] is None and r["bound"] == "latency"
