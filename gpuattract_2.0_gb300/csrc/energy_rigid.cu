/*
 * energy_rigid.cu -- fused rigid-body docking energy + DOF gradient, one
 * launch per batch of poses.
 *
 * Replaces the reference GPU pipeline of five launches with global
 * intermediates per 100-pose item (src/service/GPUEnergyService6D.tpp:163-430):
 *   d_DOF2Pos        src/model/transform.cu:18-52        x' = R x + t
 *   d_potForce       src/model/interpolation.cu:18-140   inner/outer trilinear
 *   d_NLPotForce     src/model/neighborlist.cu:21-171    NL pair term
 *   blockReduce      src/model/reduction.cu:50-391       13 sums per pose
 *   h_finalReduce    src/model/reduction.h:160-205       ForceLim + TorqueMat
 * by one kernel in which a warp owns a pose and nothing per bead leaves the
 * SM; lanes 0..6 store the 28-byte Result_6D.  Batches too small to keep every
 * warp slot busy for several poses split each pose into its 64-bead rounds
 * (rigid_rounds_kernel).
 */
#include <atomic>

#include "rigid_pose.cuh"

namespace gba {

/* BOUND4: registers capped for four resident 256-thread blocks per SM
 * (GBA_KOPT_FOUR_BLOCKS), else for three: a few registers more than 80 would
 * leave two (30,000 poses, 1500/600 beads, every option off: 1,962 against
 * 1,795 us; without FOUR_BLOCKS alone 1,547 against 1,214). */
template <bool CENSUS, bool BOUND4>
__global__ void __launch_bounds__(256, BOUND4 ? 4 : 3) rigid_energy_kernel(const RigidLaunch L) {
	__shared__ WarpStage stage[8];   /* one per warp of a <=256-thread block */
	const int lane = threadIdx.x & 31;
	for (size_t k = next_pose(L.next, lane); k < L.n; k = next_pose(L.next, lane)) {
		const size_t p = L.order ? (size_t)__ldg(&L.order[k]) : k;
		const float* dofp = reinterpret_cast<const float*>(L.dofs + p);
		const float dv = lane < 6 ? __ldg(dofp + lane) : 0.f;
		const float tx = __shfl_sync(GBA_FULL_MASK, dv, 0);
		const float ty = __shfl_sync(GBA_FULL_MASK, dv, 1);
		const float tz = __shfl_sync(GBA_FULL_MASK, dv, 2);
		const float a0 = __shfl_sync(GBA_FULL_MASK, dv, 3);
		const float a1 = __shfl_sync(GBA_FULL_MASK, dv, 4);
		const float a2 = __shfl_sync(GBA_FULL_MASK, dv, 5);
		float res[7];
		WarpStage& W = stage[threadIdx.x >> 5];
		if (lane == 0) W.slot = p;
		eval_pose_rigid<CENSUS>(L.m, tx, ty, tz, a0, a1, a2, lane, W, res, CENSUS ? L.census + p : nullptr);
		store_result7(reinterpret_cast<float*>(L.out + *(volatile unsigned long long*)&W.slot), res, lane);
		__syncwarp();
	}
}

/* Before rigid_rounds_kernel: each pose's rotation and translation as the
 * staging area holds them (a warp per round would repeat the double sincos,
 * whose pipe issues one warp instruction per 16 cycles and SM, once a round),
 * and its count of finished rounds and the launch's counter cleared.  Four
 * lanes per pose, one Euler angle each. */
__global__ void __launch_bounds__(128) rigid_setup_kernel(const RigidLaunch L) {
	const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	const size_t p = t >> 2;
	const bool in = p < L.n;
	if (t == 0) *L.next = 0;
	if (in && (t & 3) == 0) L.split.done[p] = 0;
	write_pose_record(reinterpret_cast<const float*>(L.dofs + (in ? p : 0)), L.m.trig, in, threadIdx.x & 31,
			L.split.pose + kPoseRecord * p);
}

/* A warp takes one 64-bead round of a pose at a time; the warp that finishes
 * a pose's last round adds the totals of all of them in round order, so the
 * result is eval_pose_rigid's bit for bit.  Bound by the latency of one
 * round, where a warp walking whole poses is bound by the sum of them. */
__global__ void __launch_bounds__(256, 4) rigid_rounds_kernel(const RigidLaunch L) {
	__shared__ WarpStage stage[8];
	const int lane = threadIdx.x & 31;
	WarpStage& W = stage[threadIdx.x >> 5];
	const uint32_t rounds = L.split.rounds;
	const size_t units = L.n * rounds;
	for (size_t u = next_pose(L.next, lane); u < units; u = next_pose(L.next, lane)) {
		const size_t k = u / rounds;
		const uint32_t r = (uint32_t)(u - k * rounds);
		const size_t p = L.order ? (size_t)__ldg(&L.order[k]) : k;
		if (lane < 18) W.pose[lane] = __ldg(L.split.pose + kPoseRecord * p + lane);
		__syncwarp();
		RoundCensus cen;
		PoseSums S = held_sums();
		eval_round<false>(L.m, r * kBeadsPerRound, lane, W, cen, S);
		const float v = round_total(S, W, lane);
		float* tot = L.split.totals + (size_t)p * rounds * 16 + (lane >> 1);
		if ((lane & 1) == 0) __stcg(tot + 16 * r, v);
		/* the pose's last round: release this total, then acquire the others */
		__threadfence();
		__syncwarp();
		uint32_t before = 0;
		if (lane == 0) before = atomicAdd(&L.split.done[p], 1u);
		before = __shfl_sync(GBA_FULL_MASK, before, 0);
		if (before + 1 != rounds) continue;
		__threadfence();
		clear_totals(W, lane);
		for (uint32_t q = 0; q < rounds; ++q) add_round(W, __ldcg(tot + 16 * q), lane);
		float res[7];
		finish_pose(W, res);
		store_result7(reinterpret_cast<float*>(L.out + p), res, lane);
		__syncwarp();
	}
}

/* GBA_KOPT_REFERENCE_ORDER: each pose summed in the reference CPU path's
 * order (eval_pose_rigid_ref).  Compiled for four resident 256-thread blocks
 * per SM (64 registers, 16 bytes spilled): the latency of its
 * double-precision chains wants the warps (100,000 poses of 2000/700 beads,
 * when this was chosen: 15.4 ms at four blocks, 16.7 at three, 20.7 at two). */
__global__ void __launch_bounds__(256, 4) rigid_energy_ref_kernel(const RigidLaunch L) {
	__shared__ WarpStage stage[8];
	const int lane = threadIdx.x & 31;
	for (size_t k = next_pose(L.next, lane); k < L.n; k = next_pose(L.next, lane)) {
		const size_t p = L.order ? (size_t)__ldg(&L.order[k]) : k;
		const float* dofp = reinterpret_cast<const float*>(L.dofs + p);
		const float dv = lane < 6 ? __ldg(dofp + lane) : 0.f;
		float c[6];
#pragma unroll
		for (int j = 0; j < 6; ++j) c[j] = __shfl_sync(GBA_FULL_MASK, dv, j);
		float res[7];
		eval_pose_rigid_ref(L.m, c[0], c[1], c[2], c[3], c[4], c[5], lane, stage[threadIdx.x >> 5], res);
		store_result7(reinterpret_cast<float*>(L.out + p), res, lane);
	}
}

/* Poses of many pairs in one launch: pose p belongs to pair pair_of[p]. */
template <bool REF>
__global__ void __launch_bounds__(256) batch_energy_kernel(const BatchEnergyLaunch L) {
	__shared__ WarpStage stage[8];   /* one per warp of a <=256-thread block */
	const int lane = threadIdx.x & 31;
	for (size_t p = next_pose(L.next, lane); p < L.n; p = next_pose(L.next, lane)) {
		const RigidModel& M = L.models[__ldg(&L.pair_of[p])];
		const float* dofp = reinterpret_cast<const float*>(L.dofs + p);
		const float dv = lane < 6 ? __ldg(dofp + lane) : 0.f;
		float c[6];
#pragma unroll
		for (int k = 0; k < 6; ++k) c[k] = __shfl_sync(GBA_FULL_MASK, dv, k);
		float res[7];
		if (REF)
			eval_pose_rigid_ref(M, c[0], c[1], c[2], c[3], c[4], c[5], lane, stage[threadIdx.x >> 5], res);
		else
			eval_pose_rigid<false>(M, c[0], c[1], c[2], c[3], c[4], c[5], lane, stage[threadIdx.x >> 5], res,
					nullptr);
		store_result7(reinterpret_cast<float*>(L.out + p), res, lane);
	}
}

cudaError_t launch_batch_energy(const BatchEnergyLaunch& L, int blocks, int threads, cudaStream_t s) {
	if (L.ref_order)
		batch_energy_kernel<true><<<blocks, threads, 0, s>>>(L);
	else
		batch_energy_kernel<false><<<blocks, threads, 0, s>>>(L);
	return cudaGetLastError();
}

cudaError_t launch_rigid_energy(const RigidLaunch& L, int blocks, int threads, cudaStream_t s) {
	if (L.census)
		rigid_energy_kernel<true, false><<<blocks, threads, 0, s>>>(L);
	else if (L.ref_order)
		rigid_energy_ref_kernel<<<blocks, threads, 0, s>>>(L);
	else if (L.bound4)
		rigid_energy_kernel<false, true><<<blocks, threads, 0, s>>>(L);
	else
		rigid_energy_kernel<false, false><<<blocks, threads, 0, s>>>(L);
	return cudaGetLastError();
}

cudaError_t launch_rigid_rounds(const RigidLaunch& L, int blocks, int threads, cudaStream_t s) {
	rigid_setup_kernel<<<(unsigned)((4 * L.n + 127) / 128), 128, 0, s>>>(L);
	rigid_rounds_kernel<<<blocks, threads, 0, s>>>(L);
	return cudaGetLastError();
}

/* resident blocks per SM, queried once per device, instantiation and block
 * size (the query costs host time on every launch otherwise) */
int rigid_blocks_per_sm(int threads, bool census, bool bound4, bool ref_order, bool rounds) {
	static std::atomic<int> cache[64][5][33];
	int dev = 0;
	cudaGetDevice(&dev);
	const int v = rounds ? 4 : census ? 0 : ref_order ? 1 : bound4 ? 2 : 3, t = threads / 32;
	const bool cacheable = dev >= 0 && dev < 64 && threads % 32 == 0 && t >= 1 && t <= 32;
	if (cacheable) {
		const int c = cache[dev][v][t].load(std::memory_order_relaxed);
		if (c > 0) return c;
	}
	int nb = 0;
	if (rounds)
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, rigid_rounds_kernel, threads, 0);
	else if (census)
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, rigid_energy_kernel<true, false>, threads, 0);
	else if (ref_order)
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, rigid_energy_ref_kernel, threads, 0);
	else if (bound4)
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, rigid_energy_kernel<false, true>, threads, 0);
	else
		cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, rigid_energy_kernel<false, false>, threads, 0);
	nb = nb > 0 ? nb : 1;
	if (cacheable) cache[dev][v][t].store(nb, std::memory_order_relaxed);
	return nb;
}

}  // namespace gba
