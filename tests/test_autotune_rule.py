"""What the autotuner times and which records it applies, on the CPU: only variants that run different kernels on the
problem's mesh are candidates, and a choice made where the tile kernel did not run does not stand on a mesh where it does."""
import json
from types import SimpleNamespace

KEY = "q4_n16_fp64_nointerior"


def problem(points, runs_tile, q=4, N=16, precision="fp64"):
    return SimpleNamespace(q=q, precision=precision, forest=SimpleNamespace(N=N), case=SimpleNamespace(interior=None),
                           computed_points=lambda: points,
                           pi_kernel=lambda form, pi: "tile" if pi == "tile" and runs_tile else "l1")


def record(tmp_path, choice, sweep, points, key=KEY):
    f = tmp_path / "record.json"
    f.write_text(json.dumps({key: {"choice": {"pi": choice, "threads": 64, "pi_mb": 4}, "points_per_rhs": points,
                                   "sweep": [{"pi": s, "threads": 64, "pi_mb": 4, "ms_per_rhs": 1.0} for s in sweep]}}))
    return f


def test_candidates_run_different_kernels(tgh):
    at = tgh.autotune
    small, large = problem(32768, False), problem(262144, True)
    assert [c for c in at.candidates(small) if c["pi"] == "tile"] == []
    assert len([c for c in at.candidates(large) if c["pi"] == "tile"]) == 2
    # the number of resident CTAs is a choice of the N = 32 kernels in FP64 only
    for p in (small, large, problem(1, False, N=32, precision="mixed")):
        assert {c["pi_mb"] for c in at.candidates(p)} == {4}
    assert {c["pi_mb"] for c in at.candidates(problem(1, False, q=6, N=32)) if c["pi"] == "l1"} == {3, 4, 5}


def test_a_choice_from_a_small_mesh_leaves_large_ones_the_default(tgh, tmp_path):
    at = tgh.autotune
    f = record(tmp_path, "l1", ["l1"], 32768)
    assert at.recorded_choice(problem(32768, False), path=f) == {"pi": "l1", "threads": 64, "pi_mb": 4}
    assert at.recorded_choice(problem(262144, True), path=f) == {"pi": "tile", "threads": 64, "pi_mb": 4}
    # timed with the tile kernel on a mesh of this size it stands, on one of under half the points it does not
    f = record(tmp_path, "l1", ["l1", "tile"], 131072)
    assert at.recorded_choice(problem(262144, True), path=f)["pi"] == "l1"
    assert at.recorded_choice(problem(262145, True), path=f)["pi"] == "tile"
    # a tile choice holds on every mesh: the launch falls back below the line
    f = record(tmp_path, "tile", ["l1", "tile"], 262144)
    assert at.recorded_choice(problem(32768, False), path=f)["pi"] == "tile"
