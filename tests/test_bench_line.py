"""bench.py's line on standard output: short enough that a reader of a log's end has
all of it, with every key of the contract, whatever the workload's own line holds;
the whole line goes to standard error."""
import io
import json
import sys
from contextlib import redirect_stderr, redirect_stdout
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parent.parent


@pytest.fixture()
def bench():
    sys.path[:0] = [str(REPO), str(REPO / "stochastic-parker_gb300")]
    import bench
    return bench


def _line():
    """A line of the size the headline workload makes, with its three extra
    configurations (the batch's errors of 64 runs among them)."""
    roofline = dict(bound="l1", achieved=7233.123456789, peak=10068.48, unit="GB/s", frac=0.7183912345,
                    peak_source="x" * 200, traffic=1.2e9, kernel_steps_per_s=5.3e10, note="y" * 300,
                    kernel="mover_mixed_kernel<2>", hbm=dict(frac=0.88, peak_source="measured"))
    base = dict(metric="particle-steps/s on 1 GB300 (mixed/learned vs plain FP64) at f(p) tail err <=2%",
                value=50175289496.06126, unit="particle-steps/s", n_gpus=1, steps=20, warmup=5,
                ms_per_step=208.7602783203125, higher_is_better=True, scaling="weak",
                vs_baseline=None, dtype="f32", data="synthetic",
                config={k: "z" * 60 for k in ("workload", "precision", "step", "l2", "parallelism")},
                clocks=dict(sm_mhz=2070.0, sm_max_mhz=2070.0, power_w_max=592.47, samples=6,
                            reasons=[]),
                gpu_launches=260, e2e=dict(value=4.7e10, unit="particle-steps/s",
                                           h2d_bytes_per_step=1112236692,
                                           d2h_bytes_per_step=1135877271))
    runs = [dict(run=f"run{k}", tail_err=1e-3 * (-1) ** k * k, per_bin=[0.123456789] * 30)
            for k in range(64)]
    arms = {a: {k: 1.0 / 3 for k in map(str, range(40))} for a in ("plain", "fixed", "learned")}
    return dict(base, roofline=roofline,
                accuracy=dict(tail_err=5.5e-6, tail_err_sigma=1.3e-3, per_bin_rel_err_top=[0.1] * 30,
                              workload="w" * 100, device_hist_matches=True),
                fp64_gpu=dict(value=1.6e9, unit="particle-steps/s", sample="s" * 80),
                cpu_baseline=dict(value=9e7, unit="particle-steps/s", cores=16, kind="port",
                                  sample="s" * 200),
                configs={"turbulence_3d_256": dict(base, roofline=roofline),
                         "batched_shock_2d_64": dict(base, roofline=roofline, per_run_fp_error=runs),
                         "learned_3d_scale_0.1": dict(base, learned_splitting=dict(
                             arms=arms, ess_per_s_learned_over_fixed=dict(above_100p0=289.0,
                                                                          above_p_label=3.7),
                             ess_per_s_learned_over_plain=dict(above_100p0=5000.0,
                                                               above_p_label=11.3)))})


def test_one_short_line_with_the_contracts_keys(bench):
    line = _line()
    out, err = io.StringIO(), io.StringIO()
    with redirect_stdout(out), redirect_stderr(err):
        bench.emit(line)
    text = out.getvalue()
    assert text.count("\n") == 1 and len(text) <= bench.LINE_BYTES + 1 < 4000
    got = json.loads(text)
    for key in bench.CONTRACT_KEYS:
        assert got.get(key) == line.get(key), key
    assert got["roofline"]["frac"] == 0.718391 and got["roofline"]["hbm_frac"] == 0.88
    assert got["accuracy"]["tail_err"] == 5.5e-6 and "per_bin_rel_err_top" not in got["accuracy"]
    configs = got["configs"]
    assert configs["turbulence_3d_256"]["value"] == float(f"{line['value']:.6g}")
    assert configs["batched_shock_2d_64"]["max_abs_tail_err"] == 0.063
    assert configs["learned_3d_scale_0.1"]["ess_per_s_learned_over_plain"]["above_100p0"] == 5000.0
    whole = [ln for ln in err.getvalue().splitlines() if ln.startswith("bench: details ")]
    assert json.loads(whole[0][len("bench: details "):]) == json.loads(json.dumps(line))


def test_details_give_way_to_the_contracts_keys(bench):
    line = _line()
    line["configs"] = {f"config{k}": dict(value=1.0, unit="u", ms_per_step=2.0, error="e" * 90)
                       for k in range(60)}
    short = bench.short_line(line)
    assert len(json.dumps(short)) <= bench.LINE_BYTES and "configs" not in short
    assert short["value"] == line["value"] and short["e2e"] == line["e2e"]


def test_other_workloads_lines(bench):
    batch = dict(_line()["configs"]["batched_shock_2d_64"])
    short = bench.short_line(batch)
    assert len(json.dumps(short)) <= bench.LINE_BYTES
    assert short["runs_compared"] == 64 and short["value"] == batch["value"]
    failed = bench.short_line(dict(metric="m", value=None, configs={"a": {"error": "out of memory"}}))
    assert failed["configs"] == {"a": {"error": "out of memory"}}


def test_traffic_only_where_it_was_counted(bench):
    """DRAM bytes per push depend on the particles per cell: given for the workload and
    the count of the capture, not for others, not for the brick mover."""
    peaks = {"hbm_gbs": 6800.0, "source": "fallback"}
    for ndim, ncu in bench.NCU_MOVER.items():
        args = ("global", ndim, 25.0, 1.25e9, 1e7, 152, 2070.0, peaks)
        own = bench.roofline_of(*args, ncu["workload"], ncu["particles"])
        assert own["traffic"] == ncu["dram_bytes_per_push"] * 1.25e9
        assert own["traffic_source"] == ncu["profile"] and (REPO / ncu["profile"]).exists()
        assert own["achieved"] == pytest.approx(ncu["wavefronts_per_push"] * 128 * 1.25e9 / 25e-3 / 1e9)
        for other in ((ncu["workload"], ncu["particles"] // 10), ("other", ncu["particles"]), ()):
            assert bench.roofline_of(*args, *other)["traffic"] is None
        assert str(ncu["particles"]) in own["l1_measured_at"]
    tile = bench.roofline_of("tile", 3, 25.0, 1.25e9, 1e7, 152, 2070.0, peaks, "turbulence_3d_256^3",
                             100_000_000)
    assert tile["traffic"] is None and tile["l1_measured_at"] == "nominal"
