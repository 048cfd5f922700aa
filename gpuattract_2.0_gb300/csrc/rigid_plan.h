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

/* A scoring launch is split into 64-bead rounds while it brings few poses per
 * resident warp: there the slowest warp's whole poses set the time, beyond it
 * the rounds' extra records and totals cost more than the shorter tail saves.
 * The more rounds a pose has, the longer its tail, so the line rises with the
 * ligand's beads: (beads - 72) / 64 poses a warp, 4 at most.  Measured with
 * 4,864 warps, whole poses against rounds in us (octets; native grids lie
 * higher by up to one pose a warp):
 *    beads   2,000 poses     4,000      6,000     10,000      19,400     line
 *       70         37 42     49 55      79 91    103 121     156 190     none
 *      100         44 41     59 61     96 102    121 134     183 212    2,128
 *      200         79 58    101 94    149 135    189 188     296 312    9,728
 *      300        134 83   156 132    217 183    278 266     433 456   17,328
 *      700       292 127   322 214    442 310    578 474     916 858   19,456
 *     1000       394 157   434 280    588 399    778 622   1244 1153   19,456
 * Above the line whole poses, 30,000 (6.2 a warp): 2000/700 beads 1,282 both,
 * 500/200 416 against 451. */
constexpr size_t kSplitPosesPerWarp = 4, kSplitFreeBeads = 72;
/* and its totals stay below this (ligands of thousands of beads) */
constexpr size_t kSplitBytes = (size_t)64 << 20;

/* Whether n poses of a ligand of `beads` beads are split; resident: blocks of
 * 256 threads per SM of the split form. */
inline bool rigid_splits(size_t n, size_t beads, int num_sms, int resident) {
	const size_t warps = (size_t)num_sms * 8 * resident, rounds = (beads + 63) / 64;
	return beads > kSplitFreeBeads && 64 * n <= std::min(64 * kSplitPosesPerWarp, beads - kSplitFreeBeads) * warps &&
			n * rounds * 16 * sizeof(float) <= kSplitBytes;
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
