"""bench.py's line for a workload of a small grid, whose steps run in the whole-step kernel: the launches and the roofline
are that kernel's, not those of the stage kernels, which the timed region does not launch. Checked on the CPU with the
stand-in solver of tests/test_bench_cpu.py."""
import json
import sys

import pytest

import bench
from test_bench_cpu import STEP_MS, fake_nsfsi


@pytest.mark.parametrize("steps,launches", [(1, 1), (32, 1), (33, 2), (200, 7)])
def test_small_grid_line_describes_the_kernel_that_ran(steps, launches, monkeypatch, capsys):
    m = fake_nsfsi()

    class Cfg:
        NI = NJ = NK = 48

    def no_profile(self, n):
        raise AssertionError("the launch sequence is not what the timed region ran")

    m.config_load = lambda path: Cfg()
    m.Solver.launches_per_step = lambda self: 1
    m.Solver.profile_steps = no_profile
    monkeypatch.setitem(sys.modules, "nsfsi", m)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--workload", "sphere48", "--steps", str(steps), "--warmup", "3",
                                      "--no-e2e", "--ensemble-steps", "0", "--no-adjoint", "--no-cpu-baseline",
                                      "--no-snapshots"])
    bench.main()
    line = json.loads(capsys.readouterr().out.strip().splitlines()[-1])
    assert line["gpu_launches"] == launches
    r = line["roofline"]
    assert r["kernel"].startswith("k_step") and "stage_share" not in r
    assert r["achieved"] == pytest.approx(680 * 48 ** 3 / (STEP_MS / 1e3) / 1e9)
    assert r["frac"] == pytest.approx(r["achieved"] / r["peak"]) and r["traffic"] is None
