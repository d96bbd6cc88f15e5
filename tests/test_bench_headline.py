"""The default workload's line on standard output: the contract's keys, valid
JSON, and short enough to be kept whole by whoever keeps the last few KB of the
output."""
import importlib.util
import json
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def bench():
    spec = importlib.util.spec_from_file_location("bench_mod", os.path.join(ROOT, "bench.py"))
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def full_line(m):
    """A record with everything run_serving collects, at its usual sizes."""
    roof = {"bound": "host-link", "kernel": "k" * 90, "achieved": 202.01489631552374, "peak": 211.6171026709776,
            "unit": "GB/s", "frac": 0.9546246204382479, "traffic": 11515450782.18, "traffic_note": "n" * 300,
            "link_probes": {"a": 211.3312144230467, "b": 211.6171026709776}}
    leg = {"metric": "queries/s", "value": 13.133782776339311, "unit": "queries/s", "ms_per_step": 4872.9296875,
           "config": {"workload": "w" * 400}, "roofline": roof, "e2e": {"value": 11.352565621626415, "unit": "queries/s"},
           "wall_s": 179.93689489364624, "notes": "x" * 1500}
    graphs = {str(s): {"V": 1 << s, "E": 32 << s, "budget_bytes": 1 << 33, "sssp_sources_per_pass": 16}
              for s in (22, 24, 26, 27)}
    line = {k: 1234.567890123456 for k in m.HEADLINE_KEYS}
    line.update(metric="served queries/s", unit="queries/s", n_gpus=1, steps=20, warmup=5, higher_is_better=True,
                scaling="weak", vs_baseline=None, dtype="u32/f32", data="synthetic",
                config={"workload": "serving-rmat22-24-26-27-24GiB", "graphs": graphs, "rest": "c" * 420},
                clocks={"sm_mhz": 2070.0, "sm_max_mhz": 2070.0, "samples": 34, "reasons": []}, gpu_launches=1780,
                results_identical_to_plain=True,
                e2e={"value": 156.53007861746153, "unit": "queries/s", "h2d_bytes_per_step": 1600,
                     "d2h_bytes_per_step": 50600083456, "passes": 3, "note": "n" * 170},
                roofline=roof, rooflines=[roof, roof], breakdown={"rmat%d/bfs" % i: {"x": 1.2345678901} for i in range(40)},
                cpu_baseline={"value": 0.5472329260629598, "unit": "queries/s", "cores": 16, "kind": "port",
                              "sample": "s" * 300},
                configs={key: dict(leg) for key, _ in m.CONFIG_LEGS})
    line["configs"]["cc-oom"] = {"error": "exit 1: " + "e" * 400, "wall_s": 1.0}
    return line


def test_headline_is_short_and_whole():
    m = bench()
    text = json.dumps(m.headline(full_line(m)))
    assert len(text) < 3500 and "\n" not in text
    d = json.loads(text)
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "e2e", "clocks", "gpu_launches", "cpu_baseline", "roofline"):
        assert k in d, k
    assert set(d["e2e"]) == {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"}
    assert set(d["configs"]) == {k for k, _ in m.CONFIG_LEGS}
    assert d["configs"]["cc-oom"]["error"].startswith("exit 1")
    assert d["configs"]["sssp-oom"]["frac"] == 0.954625


def test_headline_of_a_bare_line():
    """Without configurations, CPU baseline (more than one rank) or roofline."""
    m = bench()
    line = {k: v for k, v in full_line(m).items() if k not in ("configs", "roofline")}
    line["cpu_baseline"] = None
    d = m.headline(line)
    assert d["cpu_baseline"] is None and d["roofline"] is None and "configs" not in d
    assert d["value"] == 1234.57
