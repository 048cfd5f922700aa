/*
 * rigid_plan.h -- how a rigid scoring batch is launched.  Plain C++: the rule
 * is the same wherever it is asked (scoring, the autotuner, the tests).
 */
#ifndef GBA_RIGID_PLAN_H_
#define GBA_RIGID_PLAN_H_

#include <algorithm>
#include <cstddef>

namespace gba {

/* split: a warp per 64-bead round of a pose (rigid_rounds_kernel), else a
 * warp per pose. */
struct RigidPlan {
	bool split;
	int threads, blocks;
};

/* A scoring launch is split into 64-bead rounds while it brings at most this
 * many poses per resident warp: there the slowest warp's whole poses set the
 * time, beyond it the rounds' extra records and totals cost more than the
 * shorter tail saves.  Measured, whole poses against rounds (4,864 warps):
 * 2000/700 beads 100 poses 201 -> 41 us, 2,000 296 -> 127, 10,000 (2.1 a warp)
 * 566 -> 469, 30,000 (6.2) 1,282 both; 500/200 beads 10,000 190 -> 189, 30,000
 * 416 -> 451. */
constexpr size_t kSplitPosesPerWarp = 4;
/* and its totals stay below this (ligands of thousands of beads) */
constexpr size_t kSplitBytes = (size_t)64 << 20;

/* Whether n poses of a ligand of `rounds` rounds are split; resident: blocks
 * of 256 threads per SM of the split form. */
inline bool rigid_splits(size_t n, size_t rounds, int num_sms, int resident) {
	return rounds > 1 && n <= kSplitPosesPerWarp * num_sms * 8 * resident && n * rounds * 16 * sizeof(float) <= kSplitBytes;
}

/* The launch in the shape asked for, capped by the blocks per SM that are
 * resident in the chosen form at that block size. */
inline RigidPlan rigid_plan(bool split, size_t n, size_t rounds, int num_sms, int threads, int blocks_per_sm, int resident) {
	const size_t warps = threads / 32, units = split ? n * rounds : n;
	const size_t most = (size_t)num_sms * std::min(blocks_per_sm, resident);
	return RigidPlan{split, threads, (int)std::max<size_t>(1, std::min<size_t>((units + warps - 1) / warps, most))};
}

}  // namespace gba

#endif /* GBA_RIGID_PLAN_H_ */
