"""bench.py's roofline record of the sketch says which units ran, and compares with their peak (no GPU)."""
import bench


def test_sketch_roofline_follows_the_path():
    m, n, L = 100000, 20000, 4096
    d = bench.sketch_roofline(m, n, L, 0.49, False, 35.5, None)
    assert d["kernel"].startswith("dgemm_kernel") and "as_fp64" not in d
    assert d["unit"] == "TFLOP/s" and abs(d["frac"] - 2.0 * m * n * L / 0.49 / 1e12 / 35.5) < 1e-4
    i = bench.sketch_roofline(m, n, L, 0.12, True, 35.5, 4000.0)
    assert i["kernel"].startswith("rns_gemm_kernel") and i["unit"].startswith("TOP/s")
    assert abs(i["achieved"] - 15 * 2.0 * m * n * L / 0.12 / 1e12) < 0.1 and 0 < i["frac"] < 1
    assert i["as_fp64"]["frac"] > 1                      # a speed-up over the FP64 units, not a fraction of a pipe
    assert bench.sketch_roofline(m, n, L, 0.12, True, 35.5, None)["frac"] is None
