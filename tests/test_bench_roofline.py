"""bench.py's roofline entry names a kernel that the timed solves launched."""
from test_bench_host import load_bench


def stats(counts, launches=5000, iterations=900):
    return {"kernel_ms": [0.01 * c for c in counts], "kernel_count": counts, "kernel_launches": launches,
            "iterations": iterations}


def test_roofline_of_the_timed_region():
    bench = load_bench()
    pcg = {"solves_per_s": 300.0, "iterations": 900, "ms_krylov": 3.0, "stats": [], "on_chip": True}
    amg = {"solves_per_s": 200.0, "iterations": 30, "ms_krylov": 4.0, "stats": [stats([0, 0, 0, 0, 90, 30])]}
    off = {"solves_per_s": 300.0, "iterations": 900, "ms_krylov": 9.0, "stats": [stats([900, 900, 0, 0, 0, 0])],
           "on_chip": False}
    assert bench.on_chip(stats([0] * 6, launches=7)) and not bench.on_chip(stats([0] * 6, launches=2000))
    roof = bench.timed_region_roofline({"pcg64": pcg, "amg": amg}, "pcg64", 50000, 350000, None)
    assert roof["bound"] == "latency" and "k_cg_resident" in roof["kernel"]
    assert abs(roof["us_per_iteration"] - 1e3 * 3.0 / 900) < 1e-3 and "frac" not in roof
    roof = bench.timed_region_roofline({"pcg64": off, "amg": amg}, "pcg64", 50000, 350000, None)
    assert roof["kernel"].startswith("k_cg_") and "<double>" in roof["kernel"]
    assert bench.timed_region_roofline({"amg": amg}, "amg", 50000, 350000, None)["kernel"].startswith("k_fine")
    none = dict(amg, stats=[])
    assert bench.timed_region_roofline({"amg": none}, "amg", 50000, 350000, None) is None
