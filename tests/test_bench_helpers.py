"""bench.py host-side helpers that run on the GPU box unattended: clock-sample parsing / windowing and
the ncu-capture reader behind `roofline.traffic` (no GPU needed)."""
import datetime
import json
import sys
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
sys.path.insert(0, str(ROOT))

import bench  # noqa: E402


def _line(ts, sm, reasons=("Not Active",) * 4):
    stamp = datetime.datetime.fromtimestamp(ts).strftime("%Y/%m/%d %H:%M:%S.%f")[:-3]
    return f"{stamp}, {sm}, 1965, 700.0, 0x0000000000000000, " + ", ".join(reasons) + "\n"


def _sampler(tmp_path, lines):
    s = bench.ClockSampler.__new__(bench.ClockSampler)
    p = tmp_path / "clk.csv"
    p.write_text("".join(lines))

    class Done:
        def terminate(self): pass
        def wait(self, timeout=None): return 0
        def kill(self): pass
    s.proc, s.path, s.dev = Done(), str(p), 0
    return s


def test_clock_samples_are_windowed_to_the_timed_region(tmp_path):
    t = time.time()
    lines = [_line(t - 1.0, 1200), _line(t + 0.1, 1965), _line(t + 0.2, 1950),
             _line(t + 0.3, 1965, ("Not Active", "Not Active", "Not Active", "Active")), _line(t + 2.0, 300),
             "garbage line\n"]
    out = _sampler(tmp_path, lines).stop(t, t + 0.5)
    assert out["samples"] == 3 and out["sm_mhz"] == 1965.0 and out["sm_max_mhz"] == 1965.0
    assert out["reasons"] == ["sw_power_cap"] and out["window"] == "timed regions"


def test_clock_samples_fall_back_when_the_window_is_empty(tmp_path):
    t = time.time()
    out = _sampler(tmp_path, [_line(t - 1.0, 1900), _line(t - 0.9, 1910)]).stop(t, t + 0.01)
    assert out["samples"] == 2 and "no sample fell inside" in out["window"]
    assert _sampler(tmp_path, []).stop(t, t + 1)["reasons"] == ["no samples"]


def test_ncu_traffic_reads_the_committed_capture():
    t = bench.ncu_traffic("decode_paged_kernel")
    assert t is not None and t["file"].startswith("profiles/")
    # K and V of 32 x 4096 tokens x 8 heads x 128 x 2 B once, plus q, o, block table: ~537.4 MB algorithmic
    assert 537e6 < t["bytes"] < 1.05 * 537.5e6
    assert bench.ncu_traffic("no_such_kernel") is None


def test_committed_bench_lines_follow_the_contract():
    for name in ("r01_bench_ours.json", "r01_bench_reference.json", "r02_bench_ours.json", "r02_bench_reference.json"):
        d = json.loads((ROOT / "profiles" / name).read_text())
        for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
                  "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "roofline", "cpu_baseline"):
            assert k in d, (name, k)
        assert "workload" in d["config"] and "model" not in d["config"]
        assert {"value", "unit", "h2d_bytes_per_step", "d2h_bytes_per_step"} <= set(d["e2e"])
        assert {"bound", "achieved", "peak", "unit", "frac", "traffic"} <= set(d["roofline"])
        assert {"value", "unit", "cores", "kind", "sample"} <= set(d["cpu_baseline"])
    for name in ("r01_bench_reference.json", "r02_bench_reference.json"):
        ref = json.loads((ROOT / "profiles" / name).read_text())
        assert ref["impl"] == "reference" and ref["e2e"]["h2d_bytes_per_step"] == 0
    # the metric is the headline one, without a scope qualifier, and the step holds no library kernel
    ours = json.loads((ROOT / "profiles" / "r02_bench_ours.json").read_text())
    assert ours["metric"] == json.loads((ROOT / "BASELINE.json").read_text()).get("metric", ours["metric"]) or "(" not in ours["metric"]
    assert ours["gpu_launches"] == ours["launches_per_step"] * ours["steps"] and "cuBLAS" not in ours["config"]["gemm"]


def test_tp_roofline_is_the_slower_of_hbm_and_nvlink():
    """north_star: TP scaling as a fraction of the NVLink-bound roofline (bench.tp_roofline, added to every N > 1 line)."""
    payload, ars = 32 * 4096 * 2, 64                      # [B, hidden] bf16, two all-reduces per layer
    r = bench.tp_roofline(3.0, 4_024_180_736, 6542.4, 8, payload, ars, fused_push=True)
    assert r["bound"] == "hbm" and abs(r["hbm_ms"] - 0.6151) < 1e-3
    assert r["nvlink_bytes_per_rank_per_step"] == int(ars * 2 * 7 / 8 * payload)          # reduce-scatter + all-gather
    assert r["nvlink_bytes_per_rank_per_step_as_sent"] == ars * 2 * 7 * payload           # one-shot push, 8-byte flagged units
    assert abs(r["frac"] - r["target_ms"] / 3.0) < 1e-12 and r["frac"] < r["frac_serial"] < 1.0
    # a step that streams almost nothing per rank is bound by the link
    r = bench.tp_roofline(1.0, 1_000_000, 6542.4, 8, payload, ars, fused_push=False)
    assert r["bound"] == "nvlink" and r["target_ms"] == r["nvlink_ms"] == r["nvlink_ms_as_sent"]
    # derived from the committed lines (measured step times): the strong-scaling curve against this roofline
    for n in (2, 4, 8):
        d = json.loads((ROOT / "profiles" / f"r02_bench_tp{n}_ours.json").read_text())
        c = d["config"]
        r = bench.tp_roofline(d["ms_per_step"], c["hbm_bytes_per_step_per_rank"], d["roofline"]["peak"], n,
                              c["batch"] * c["hidden"] * 2, 2 * c["layers"], fused_push=True)
        assert r["bound"] == "hbm" and abs(r["frac"] - c["step_hbm_roofline_frac"]) < 1e-6
