/* The launch rule of rigid scoring batches behind a C face. */
#include "../../gpuattract_2.0_gb300/csrc/rigid_plan.h"

extern "C" void plan(size_t n, size_t beads, int sms, int threads, int bps, int resident, int* out) {
	const bool split = gba::rigid_splits(n, beads, sms, 4);
	const gba::RigidPlan p = gba::rigid_plan(split, n, (beads + 63) / 64, sms, threads, bps, resident);
	out[0] = p.split;
	out[1] = p.threads;
	out[2] = p.blocks;
}
