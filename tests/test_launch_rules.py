"""The choice of sweep build (csu_b200/csrc/cuda/launch_rules.h), compiled for the host: WIDE only where it saves enough
waves, the same choice for the same cells per multiprocessor, PLAIN for every mesh of one wave."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("rules") / "launch_rules_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-o", exe,
                    os.path.join(ROOT, "tests", "native", "launch_rules_check.cpp")], check=True)

    def ask(rows):
        r = subprocess.run([exe], input="\n".join("%d %d %d %d" % q for q in rows), capture_output=True, text=True,
                           check=True)
        return [tuple(int(v) for v in line.split()) for line in r.stdout.splitlines()]
    return ask


# (cells per multiprocessor, FP64 WIDE, FP32 WIDE): either side of each line between wave counts
LINES = [(640, 0, 0), (641, 1, 1), (1152, 1, 1), (1153, 0, 0), (1280, 0, 0), (1281, 0, 1), (1920, 0, 1), (1921, 1, 1),
         (2304, 1, 1), (2305, 0, 0), (2560, 0, 0), (2561, 0, 1), (3200, 0, 1), (3201, 1, 1), (3456, 1, 1),
         (3457, 0, 1)]


@pytest.mark.parametrize("sms", [148, 132, 20])
def test_wide_where_it_saves_waves(rules, sms):
    for per_sm, f64, f32 in LINES:
        got = rules([(0, 0, per_sm * sms, sms), (0, 1, per_sm * sms, sms), (1, 1, per_sm * sms, sms),
                     (2, 0, per_sm * sms, sms)])
        assert [g[0] for g in got] == [f64, f32, 0, 0], per_sm


def test_tune_class_separates_builds(rules):
    """Meshes of one class have one sweep build, at every size from the smallest tuned mesh up."""
    for fp32 in (0, 1):
        seen = {}
        sizes = range(16384, 700000, 97)
        for cells, (wide, cls, early, _) in zip(sizes, rules([(0, fp32, c, 148) for c in sizes])):
            assert seen.setdefault(cls, (wide, early)) == (wide, early), cells
        assert set(seen.values()) == {(0, 0), (0, 1), (1, 0)}


@pytest.mark.parametrize("sms", [148, 132, 20])
def test_early_by_cells_per_multiprocessor(rules, sms):
    """The line of EARLY scales with the device, as WIDE's does."""
    for model, fp32, per_sm in ((0, 0, 256), (0, 1, 320), (1, 0, 192), (1, 1, 192), (2, 0, 0), (2, 1, 0)):
        at, above = rules([(model, fp32, per_sm * sms, sms), (model, fp32, per_sm * sms + 1, sms)])
        assert (at[2], above[2]) == (int(per_sm > 0), 0)
        assert not (at[0] or above[0])


@pytest.mark.parametrize("sms", [148, 20])
def test_small_gradient_budget_by_blocks_per_multiprocessor(rules, sms):
    """Three blocks of 32 cells a multiprocessor for Euler and laminar, two for the wider blocks of SA and SST."""
    for model, blocks in ((0, 3), (1, 2), (2, 2)):
        at, above = rules([(model, 0, 32 * blocks * sms, sms), (model, 0, 32 * blocks * sms + 1, sms)])
        assert (at[3], above[3]) == (1, 0)
