"""The schedule of the fp32 kernel's split teams, walked on the host: rings of every number of stages that the planner can
choose, over many rounds."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "portdnn_b200", "csrc")

PROGRAM = r"""
#include "split_ring.cuh"
#include <cstdio>
int main() {
  std::printf("%d\n", pdnn::kSplitTeams);
  for (int stage = 0; stage < 8; ++stage) std::printf("%d\n", pdnn::split_team_of_stage(stage));
}
"""


def waits_that_may_return_early(stages, team_of, steps=200):
    """Steps whose wait, by a parity, can find its stage's barrier a whole phase behind: those of a team that did not
    itself wait for the stage's use before, at step - stages."""
    return [g for g in range(stages, steps) if team_of(g, g % stages) != team_of(g - stages, g % stages)]


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("split_ring")
    src, exe = str(d / "ring.cc"), str(d / "ring")
    with open(src, "w") as f:
        f.write(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I" + CSRC, src, "-o", exe], check=True)
    out = [int(v) for v in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()]
    return out[0], out[1:]


@pytest.mark.parametrize("stages", range(1, 9))
def test_every_wait_follows_the_wait_for_the_use_before(rule, stages):
    teams, of_stage = rule
    assert waits_that_may_return_early(stages, lambda step, stage: of_stage[stage]) == []
    load = [of_stage[:stages].count(t) for t in range(teams)]
    assert sum(load) == stages and max(load) - min(load) <= 1  # every stage is somebody's, in fair shares


@pytest.mark.parametrize("stages", range(1, 9))
def test_the_walk_finds_teams_that_take_turns_by_the_step(stages):
    assert (waits_that_may_return_early(stages, lambda step, stage: step % 2) != []) == (stages % 2 == 1)


def test_the_kernel_goes_by_the_rule():
    text = open(os.path.join(CSRC, "tc_gemm.cu")).read()
    assert text.count("if (split_team_of_stage(s) == team) {") == 1 and text.count("== team)") == 1
