"""bench.py's JSON line against the benchmark contract: the reference arm
on the CPU, the GPU arm on R-MAT 16 (marked gpu)."""
import json
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_reference_arm_prints_one_contract_line():
    """The default (partitioned) workload at a small scale: the same code path
    as R-MAT 23, which takes minutes of CPU here."""
    out = subprocess.run([sys.executable, "bench.py", "--impl", "reference", "--steps", "1", "--warmup", "0",
                          "--scale", "14"],
                         cwd=ROOT, capture_output=True, text=True, timeout=600, check=True).stdout
    lines = [line for line in out.splitlines() if line.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert d["impl"] == "reference" and d["metric"] == "oriented edges/s" and d["unit"] == "edges/s"
    assert d["value"] > 0 and d["ms_per_step"] > 0 and d["higher_is_better"] is True
    assert (d["n_gpus"], d["steps"], d["warmup"]) == (1, 1, 0)
    assert d["scaling"] == "strong" and d["vs_baseline"] is None and d["dtype"] == "int32"
    assert d["config"]["workload"] == "rmat14_ef16_halo_parts" and d["config"]["oriented_edges"] == 213184
    assert d["config"]["parts_k"] == [2, 4, 8]
    cb = d["cpu_baseline"]
    assert cb["value"] == d["value"] and cb["unit"] == d["unit"] and cb["cores"] >= 1
    assert cb["kind"] in ("port", "reference") and cb["sample"]
    e2e = d["e2e"]
    assert e2e["value"] == d["value"] and e2e["unit"] == d["unit"]
    assert e2e["h2d_bytes_per_step"] == 0 and e2e["d2h_bytes_per_step"] == 0


@pytest.mark.gpu
def test_gpu_arm_line_carries_roofline_baseline_e2e_and_clocks():
    """The GPU arm on R-MAT 16: roofline of the dominant kernel, the CPU
    baseline, the end-to-end number with its host copies, clocks and the
    launch count, with the count checked against the oracle inside."""
    out = subprocess.run([sys.executable, "bench.py", "--workload", "rmat16", "--steps", "3", "--warmup", "3"],
                         cwd=ROOT, capture_output=True, text=True, timeout=900, check=True).stdout
    lines = [line for line in out.splitlines() if line.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert d["metric"] == "oriented edges/s" and d["value"] > 0 and d["n_gpus"] == 1 and d["steps"] == 3
    r = d["roofline"]
    assert r["bound"] == "hbm" and r["unit"] == "GB/s" and r["achieved"] > 0 and r["peak"] > 0
    assert abs(r["frac"] - r["achieved"] / r["peak"]) < 1e-9
    assert d["cpu_baseline"]["value"] > 0 and d["cpu_baseline"]["cores"] >= 1
    e2e = d["e2e"]
    assert e2e["value"] > 0 and e2e["h2d_bytes_per_step"] > 0 and e2e["d2h_bytes_per_step"] > 0
    assert d["gpu_launches"] > 0 and "sm_mhz" in d["clocks"] and "reasons" in d["clocks"]
    assert d["config"]["workload"] == "rmat16_ef16_plain"


def test_reference_arm_loads_no_library_code():
    """The reference arm builds its input with the oracle's generators: the
    process never maps libtc.so."""
    code = ("import sys, runpy; sys.argv = ['bench.py', '--impl', 'reference', '--steps', '1', '--warmup', '0', "
            "'--scale', '12']; runpy.run_path('bench.py', run_name='__main__'); "
            "maps = open('/proc/self/maps').read(); print('LIBTC' if 'libtc.so' in maps else 'CLEAN')")
    out = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=600,
                         check=True).stdout
    assert out.strip().splitlines()[-1] == "CLEAN"


@pytest.mark.gpu
def test_gpu_arm_partitioned_line_is_complete():
    """The default workload at scale 16: per-k timings in both halo modes,
    the roofline with its three figures, the end-to-end parts path, clocks."""
    out = subprocess.run([sys.executable, "bench.py", "--steps", "2", "--warmup", "3", "--scale", "16"],
                         cwd=ROOT, capture_output=True, text=True, timeout=900, check=True).stdout
    lines = [line for line in out.splitlines() if line.startswith("{")]
    assert len(lines) == 1
    d = json.loads(lines[0])
    assert d["config"]["workload"] == "rmat16_ef16_halo_parts" and d["value"] > 0 and d["scaling"] == "strong"
    r = d["roofline"]
    assert r["achieved"] > 0 and abs(r["frac"] - r["achieved"] / r["peak"]) < 1e-9
    assert r["wedge_model_bytes"] >= r["algorithmic_bytes_per_launch"] > 0
    for k in ("2", "4", "8"):
        row = d["detail"]["parts"][k]
        assert row["count"]["parts_nnz_total"] <= row["reference"]["parts_nnz_total"]
        assert sum(row["count"]["per_part_counts"]) == d["detail"]["triangles"]
    e2e = d["e2e"]
    assert e2e["value"] > 0 and e2e["h2d_bytes_per_step"] > 0 and e2e["d2h_bytes_per_step"] > 0
    assert d["gpu_launches"] > 0 and "sm_mhz" in d["clocks"]
    assert d["cpu_baseline"]["count_matches"] is True


def test_counting_kernel_is_named_by_what_ran():
    sys.path.insert(0, ROOT)
    import bench
    assert [bench.counting_kernel(1, d) for d in (0, 4, 5, 8, 9, 64)] == \
        ["flat4_kernel"] * 2 + ["flat_kernel"] * 2 + ["single_kernel"] * 2
    assert bench.counting_kernel(5, 100) == "packed_kernel"
    assert [bench.counting_kernel(n, 100) for n in (6, 7, 9, 11)] == ["count_kernel"] * 4


def test_packed_bytes_of_small_graphs():
    """By hand, every id of a low block.  K_4 of ids 0..3 (rows of 3, 2, 1 and 0):
    the roots of two or more members have five out-neighbours, three of them with
    members, each a row of one octet."""
    import numpy as np
    import torch
    sys.path.insert(0, ROOT)
    import bench
    rp, col = np.array([0, 3, 5, 6, 6], np.int32), np.array([1, 2, 3, 2, 3, 3], np.int32)
    assert bench.packed_bytes(rp, col, 4, torch.device("cpu")) == 5 * 20 + 3 * 32
    assert bench.packed_bytes(rp, col, 1, torch.device("cpu")) == 3 * 20 + 2 * 32
    assert bench.packed_bytes(rp, col, 0, torch.device("cpu")) == 0
    # every id popular once: 40,000 members in rows of one, the first 30,720 ids low
    n = 40_001
    rp = np.concatenate(([0, 40_000], np.full(n - 1, 40_000))).astype(np.int32)
    got = bench.packed_bytes(rp, np.arange(1, n, dtype=np.int32), n, torch.device("cpu"))
    assert got == 40_000 * 20


@pytest.mark.gpu
def test_roofline_names_the_kernel_that_counted():
    """R-MAT 16 counts packed, a road network flat, an unskewed batch's or the probing tables' count by count_kernel."""
    for extra, kernel in ((["--workload", "rmat16", "--no-tune"], "packed_kernel"),
                          (["--workload", "rmat16", "--tuning", '{"probe_kicks": 0}'], "count_kernel")):
        out = subprocess.run([sys.executable, "bench.py", "--steps", "2", "--warmup", "3", "--no-cpu"] + extra,
                             cwd=ROOT, capture_output=True, text=True, timeout=900, check=True).stdout
        d = json.loads([line for line in out.splitlines() if line.startswith("{")][0])
        assert d["roofline"]["kernel"] == kernel
        assert (d["roofline"]["probes_done"] == d["config"]["W_plus"]) == (kernel == "packed_kernel")
