"""The bench names the slices that the engine took, not the ones a workload asked for, and
scales a recorded DRAM traffic only to the kernel it was captured of."""
import json
import os
import types

import bench


def test_slices_and_kernels_are_the_engines():
    eng = types.SimpleNamespace(nx=[16384, 2048, 2048, 4096], slices=[1024, 512, 512, 512])
    assert bench.slices_used(eng) == {"2048": 512, "4096": 512, "16384": 1024}
    assert bench.evolve_kernels(eng) == "k_evolve<1024>, k_evolve<512>"
    eng = types.SimpleNamespace(nx=[4096, 4096], slices=[512, 2048])
    assert bench.slices_used(eng) == {"4096": [512, 2048]}


def test_traffic_is_of_the_kernel_that_ran(tmp_path, monkeypatch):
    os.makedirs(tmp_path / "profiles")
    rec = {"ensemble": {"dram_bytes_per_rhs_pt": 400, "kernel": "k_evolve<2048>", "capture": "c", "build": "b"}}
    (tmp_path / "profiles" / "traffic.json").write_text(json.dumps(rec))
    monkeypatch.setattr(bench, "ROOT", str(tmp_path))
    assert bench.profile_traffic("ensemble", "k_evolve<2048>")[0] == 400.0
    assert bench.profile_traffic("ensemble", "k_evolve<1024>, k_evolve<512>")[0] is None
    assert bench.profile_traffic("2d")[0] is None
