// Who expands which block of gemm_q_kernel, and into which stage of the ring (gemm.cu; plain C++, also built by host_selftest.cpp).
// A warp knows a stage's uses by the parity of its barrier, so it has to see every one of them: a stage belongs to ONE group of warps.
// (Groups that took turns at a stage could meet its barrier two uses on, which reads as none.)
#pragma once

namespace b2 {

constexpr int GM_GROUPS = 2;                                              // group g expands blocks g, g + 2, ..
constexpr int gm_group(int block) { return block % GM_GROUPS; }
constexpr int gm_stage(int block, int stages) { return block % stages; }
// stages of a plan: weights in shared memory (32 KB a stage) or in tensor memory (64 columns a stage beside two halves of 128 sums);
// wanted: fewer, for experiments
constexpr int gm_stages(bool in_smem, int wanted) {
    const int most = in_smem ? 2 : 4, s = wanted >= GM_GROUPS && wanted < most ? wanted : most;
    return s - s % GM_GROUPS;
}

}  // namespace b2
