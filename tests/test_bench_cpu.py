"""bench.py's reference arm on the CPU: the JSON line carries the contract's keys (the
metric and config of the GPU arm, impl, cpu_baseline, e2e with zero copies), says which
samples of the workload it ran, honours --warmup, and uses every host core it asks for."""
import json
import subprocess
import sys
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_reference_arm_json_line():
    out = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--impl", "reference", "--steps", "2",
                          "--warmup", "1", "--cpu-n", "48", "--n", "512"],
                         cwd=ROOT, capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]
    d = json.loads(out.stdout.strip().splitlines()[-1])
    for key in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better",
                "dtype", "data", "config", "impl", "cpu_baseline", "e2e"):
        assert key in d, key
    assert d["impl"] == "reference" and d["value"] > 0 and d["higher_is_better"] is True
    # the line names the GPU arm's workload and what the CPU ran of it (one sample per core)
    assert "rain-on-terrain dense 512x512" in d["config"]["workload"]
    assert f"x 48x48 samples" in d["config"]["workload"]
    assert d["warmup"] == 1
    assert d["cpu_baseline"]["kind"] == "port" and d["cpu_baseline"]["cores"] >= 1
    assert d["e2e"] == {"value": d["value"], "unit": d["unit"], "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}


def _bench():
    import importlib.util
    spec = importlib.util.spec_from_file_location("bench_under_test", ROOT / "bench.py")
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def test_no_figure_from_another_builds_counters(monkeypatch):
    """Counts per cell of other sources give no traffic and no issue roofline."""
    b = _bench()
    entry = {"dram_bytes_per_cell": 36.0, "warp_inst_per_cell": 30.0, "workload": "w", "sources": "0"}
    monkeypatch.setattr(b, "counters", lambda: {"dense": dict(entry, current_build=False)})
    assert b._traffic("dense", 100) == (None, None)
    assert b.issue_roofline("dense", 1 << 26, 1.6, {"sm_mhz": 1965.0}) is None
    monkeypatch.setattr(b, "counters", lambda: {"dense": dict(entry, current_build=True)})
    assert b._traffic("dense", 1000)[0] == 36.0 * 1000 / 1e9


def test_counters_name_every_source_of_their_kernel():
    """An entry's `files` are a kernel's source and all the headers that it includes, so that an
    edit of any of them shows."""
    import re
    csrc = ROOT / "geoswe_b200" / "csrc"

    def headers(name, seen):
        for inc in re.findall(r'#include "(gsw_\w+\.cuh)"', (csrc / name).read_text()):
            if inc not in seen:
                seen.add(inc)
                headers(inc, seen)
        return seen

    of = {"dense": ("gsw_dense.cu", "gsw_dense_march.cuh"), "dense_fast": ("gsw_fast.cu", "gsw_dense_march.cuh"),
          "flat_tidal": ("gsw_flat.cu", "gsw_flat_march.cuh"), "flat_compressed": ("gsw_flat.cu", "gsw_flat_march.cuh")}
    c = _bench().counters()
    assert set(c) == set(of)
    for kind, (source, march) in of.items():
        need = headers(march, {source, march})
        assert need <= set(c[kind]["files"]), (kind, need - set(c[kind]["files"]))
        assert (ROOT / c[kind]["summary"]).exists()
