// Which team of split warps takes which stage of an fp32 pipeline's ring (tc_gemm.cu).  Plain C++, so that the
// schedule can be walked on the host.
#pragma once

namespace pdnn {

constexpr int kSplitTeams = 2;

// A team belongs to stages, not to steps.  Waits on a stage's barrier name a phase by its parity only: while use u - 1 of a
// stage is still being filled, the wait for use u finds the parity of use u - 2 and returns at once.  So whoever waits
// for one use of a stage must have waited for the use before it - and must have a part in each of those uses, or the
// barrier could run two phases ahead.  Teams that took every second step would meet, in a ring of an odd number of
// stages, stages whose use before was the other team's.  Tiles of 16 and 32 columns have seven stages: four to one team
// and three to the other.  32 images, 56x56 128 -> 32 3x3 input gradient 63.3 us, 64 images, 28x28 512 -> 16 1x1 20.9;
// six stages 62.5 and 22.2; turns by the step, each behind a wait for the stage's release, 74.4 and 21.7.
constexpr int split_team_of_stage(int stage) { return stage & (kSplitTeams - 1); }

}  // namespace pdnn
