"""The committed DRAM counts that bench.py divides by a kernel's time belong to the
launches that the library makes now."""
import json
import os

import bench

ROOT = os.path.join(os.path.dirname(__file__), "..")


def test_counts_belong_to_the_launches_of_the_library(pa):
    with open(os.path.join(ROOT, "profiles", "kernel_traffic.json")) as f:
        entries = json.load(f)
    for name, t in entries.items():
        w = bench.WORKLOADS[name]
        prm = pa.make_params(w["n"], w["d"], w["p"], id_bits=w["id_bits"], seed_mode=w["seed_mode"],
                             model=w.get("model", 0))
        assert t["launches"] == pa.generate_launches(prm) - 1, name   # all but the set-up kernel
        assert bench.load_traffic(name, t["launches"]) == (t["dram_bytes"], t["source"])
        if "dram_read" in t:
            assert t["dram_bytes"] == t["dram_read"] + t["dram_write"]
        else:
            assert t["source"].startswith("estimated")
        assert bench.load_traffic(name, t["launches"] + 1) == (None, None)
    assert bench.load_traffic("no such workload", 1) == (None, None)
