"""The line bench.py prints: short enough for its reader whatever was measured, with
the contract's keys as they are, and no rate of work that the timed kernel does not do."""
import json
import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))
import bench


def test_line_is_short_and_keeps_its_keys():
    core = {"metric": "probes/s", "value": 5496798.30545664, "unit": "probes/s", "n_gpus": 1, "steps": 20, "warmup": 5,
            "ms_per_step": 47.690307235717775, "config": bench.config_dict(262144, 49162), "gpu_launches": 130,
            "e2e": {"value": 5483464.963490376, "unit": "probes/s"}, "clocks": {"sm_mhz": 2070.0, "reasons": []}}
    trials = [{"ctas_per_sm": k, "node_steps": 6, "ms": 69.79424285888672 + k} for k in range(40)]
    sections = {f"section_{n}": {"workload": "w" * 200, "fused": {"ms": 1.23456789, "trials": trials},
                                 "runs": [{"p50_ms": 0.123456789, "p99_ms": 2.0}] * n} for n in (1, 5, 20, 60, 400)}
    line = bench.printed_line({**core, **sections})
    assert len(json.dumps(line)) <= bench.LINE_LIMIT
    assert {k: line[k] for k in core} == core
    assert line["section_1"] == {"fused": {"ms": 1.2346}, "runs": [{"p50_ms": 0.12346, "p99_ms": 2.0}]}
    assert line["left_out"] == ["section_400"] and "section_60" in line
    assert bench.printed_line(core) == core


def test_roofline_gives_no_rate_of_walks_from_the_root():
    stats = {"bytes": 1.5e12, "node_tests_per_ray": 58.0, "node_fetches_per_ray": 58.0}
    for kname, bound in (("trace_tile", "issue"), ("a kernel without a capture", "hbm")):
        r = bench.trace_roofline(kname, 47.0, stats, {"sm_max_mhz": 2070.0}, 152, 6788.6, True, 262144, 49162, 9, 4, True)
        assert r["bound"] == bound and 0 < r["frac"] < 1.2
        assert not {"achieved", "frac", "peak"} & set(r["l1"])
