/*
 * energy_modes.cu -- fused normal-mode (flexible) docking energy + gradients.
 *
 * CPU semantics followed: CPUEnergyService6DModes::createItemProcessor
 * (src/service/CPUEnergyService6DModes.tpp:121-327).  One warp owns one pose
 * and works in rounds of 64 beads staged in shared memory, like the rigid
 * kernel (rigid_pose.cuh), in two passes:
 *   receptor pass  deform by the receptor amplitudes (rotate_translate_deform,
 *                  src/model/transform_modes.h:54-93), move into the ligand
 *                  frame with the "inverted" DOF (invertDOF, :27-41: angles
 *                  negated, t' = R^T (-t)), interpolate in the LIGAND grid,
 *                  rotate the force back by R (rotate_forces, :146-166) and
 *                  project it on the receptor modes (reduceModeForce without
 *                  rotation, src/model/reduction_modes.h:68-90);
 *   ligand pass    deform + transform the ligand, interpolate in the receptor
 *                  grid, add the NL pair term against the DEFORMED receptor
 *                  (neighborlist_modes.h:21-206) whose reaction forces are
 *                  projected on the receptor modes pair by pair; energy, force,
 *                  torque (undeformed ligand coordinates, reduceTorque) and the
 *                  ligand mode projection of R^T f (reduceModeForce with
 *                  rotation, reduction_modes.h:29-57) are summed per lookup
 *                  and per pair (all linear in the bead forces);
 *   epilogue       warp sums, correctModeForce (delta += 4 k delta^4,
 *                  reduction_modes.h:101-115), ForceLim, TorqueMat.
 * The energy holds only the ligand-side terms, as in the reference.
 * Neighbour receptor positions are re-deformed per pair with the same unfused
 * operation sequence as the receptor pass, so no per-pose scratch is needed.
 *
 * Every mode projection is linear in the force: f . (R^T v) replaces
 * (R f) . v and f . (R v) replaces (R^T f) . v, so each staged bead's mode
 * vectors are rotated once per round into shared memory (ModeStage) and a
 * projection costs no global load and no rotation.  On octet grids the grid
 * lookups of both passes take the rigid kernel's cooperative form
 * (CoopStep): the lane holding force component c adds f_c times component
 * c of the staged vector.  Kernels are compiled for mode capacities 5 and 10
 * (arrays sized to the capacity, not to GBA_MODES_MAX).
 * The reference's own GPU modes kernels are not followed: they mis-index the
 * deformed receptor and mode buffers (src/model/neighborlist_modes.cu:81-83,
 * src/model/transform_modes.cu:154, src/model/reduction_modes.cu:68-69).
 */
#include <algorithm>
#include <array>
#include <map>
#include <mutex>

#include "rigid_pose.cuh"
#include "va13.cuh"

namespace gba {

namespace {

/* The grid layout a pass is compiled for. */
constexpr int kNative = 0, kOctets = 1, kAnyLayout = 2;

/* Floats of a bead's mode record held in registers (mode_stride(MM)). */
template <int MM>
constexpr int kModeWords = (3 * MM + 7) / 8 * 2;

/* The bead's M mode vectors from its 32-byte aligned record v (padded to
 * eights of floats): one 32-byte load per eight floats -- the records of a
 * warp's beads lie apart, so every load is an L1 wavefront per lane (16-byte
 * loads: 20,000 poses at 5 modes 1,837 against 1,803 us, 5,000 at 10 modes 598
 * against 533). */
template <int MM>
__device__ __forceinline__ void load_modes(const float* __restrict__ v, uint32_t M, float (&w)[4 * kModeWords<MM>]) {
#pragma unroll
	for (int k = 0; k < kModeWords<MM>; k += 2) {
		float t[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
		if (4 * k < 3 * (int)M) ldg_32(v + 4 * k, t);
#pragma unroll
		for (int j = 0; j < 8; ++j) w[4 * k + j] = t[j];
	}
}

/* The same in 16-byte loads, for the reference order, whose kernels the wide
 * ones cost registers (500 poses, 700/300 beads, 5 modes: 363 against 433 us)
 * but for ten modes and many poses (kRefWide). */
template <int MM>
__device__ __forceinline__ void load_modes16(const float* __restrict__ v, uint32_t M, float (&w)[4 * kModeWords<MM>]) {
	const float4* q = reinterpret_cast<const float4*>(v);
#pragma unroll
	for (int k = 0; k < kModeWords<MM>; ++k) {
		const float4 t = 4 * k < 3 * (int)M ? __ldg(q + k) : make_float4(0.f, 0.f, 0.f, 0.f);
		w[4 * k] = t.x; w[4 * k + 1] = t.y; w[4 * k + 2] = t.z; w[4 * k + 3] = t.w;
	}
}

/* x + sum_m a_m v_m, unfused in mode order (rotate_translate_deform), with
 * the bead's vectors w already loaded. */
template <int MM>
__device__ __forceinline__ void deform_w(const float (&w)[4 * kModeWords<MM>], uint32_t M, const float* amp,
		float& x, float& y, float& z) {
#pragma unroll
	for (int m = 0; m < MM; ++m)
		if (m < (int)M) {
			x = fadd(x, fmul(amp[m], w[3 * m]));
			y = fadd(y, fmul(amp[m], w[3 * m + 1]));
			z = fadd(z, fmul(amp[m], w[3 * m + 2]));
		}
}

template <int MM, bool WIDE>
__device__ __forceinline__ void deform(const float* __restrict__ v, uint32_t M, const float* amp,
		float& x, float& y, float& z) {
	float w[4 * kModeWords<MM>];
	if (WIDE) load_modes<MM>(v, M, w);
	else load_modes16<MM>(v, M, w);
	deform_w<MM>(w, M, amp, x, y, z);
}

/* acc[m] += sign * (f . v_m) */
template <int MM>
__device__ __forceinline__ void project(const float* __restrict__ v, uint32_t M, float fx, float fy,
		float fz, float sign, float* acc) {
	float w[4 * kModeWords<MM>];
	load_modes<MM>(v, M, w);
#pragma unroll
	for (int m = 0; m < MM; ++m)
		if (m < (int)M)
			acc[m] = ffma(sign, ffma(fz, w[3 * m + 2], ffma(fy, w[3 * m + 1], fmul(fx, w[3 * m]))), acc[m]);
}

/* Per warp and round: each staged bead's mode vectors, rotated into the frame
 * of the forces they are projected on, component-major. */
template <int MM>
struct ModeStage {
	float w[kBeadsPerRound][3][MM];
	/* the pose: R [0, 9), its sin/cos [9, 15), R(-ang) [15, 24), t' [24, 27),
	 * t [27, 30), then the receptor's and the ligand's amplitudes.  Kept here
	 * rather than in registers (31 to 50 of them), read back where a round or
	 * its pairs need some. */
	float pose[(30 + 2 * MM + 3) & ~3];
};

/* What the receptor pass stages of a round: charges, lookups, weights and (for
 * the native layout) bead indices, in the fields the lookups expect of a
 * WarpStage, without its pairs and torque. */
struct RecStage {
	float cw[kBeadsPerRound * kCornerStride];
	uint2 look[2 * kBeadsPerRound];
	float q[kBeadsPerRound];
	uint32_t j[kBeadsPerRound];
	__device__ __forceinline__ float charge(uint32_t s) const { return q[s]; }
	__device__ __forceinline__ void put_rec(int s, float charge, uint32_t bead) {
		q[s] = charge;
		j[s] = bead;
	}
	__device__ __forceinline__ uint32_t bead(uint32_t s) const { return j[s]; }
};
/* The same of a whole WarpStage. */
struct FullStage : WarpStage {
	__device__ __forceinline__ void put_rec(int s, float charge, uint32_t bead) {
		put_bead(*this, s, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, charge, bead);
	}
	__device__ __forceinline__ uint32_t bead(uint32_t s) const { return __float_as_uint(ut[s].w); }
};

/* Rotated mode vectors of slot s: w_m = R v_m (transpose = false) or R^T v_m,
 * from the bead's loaded vectors w. */
template <int MM>
__device__ __forceinline__ void stage_modes(ModeStage<MM>& S, int s, const float (&w)[4 * kModeWords<MM>],
		uint32_t M, const float m9[9], bool transpose) {
#pragma unroll
	for (int m = 0; m < MM; ++m)
		if (m < (int)M) {
			const float vx = w[3 * m], vy = w[3 * m + 1], vz = w[3 * m + 2];
			float a, b, c;
			if (transpose) rot_apply_t(m9, vx, vy, vz, a, b, c);
			else rot_apply(m9, vx, vy, vz, a, b, c);
			S.w[s][0][m] = a;
			S.w[s][1][m] = b;
			S.w[s][2][m] = c;
		}
}

/* acc[m] += sign * (f . w_m) with the staged vectors of slot s */
template <int MM>
__device__ __forceinline__ void project_staged(const ModeStage<MM>& S, uint32_t s, uint32_t M, float fx,
		float fy, float fz, float sign, float* acc) {
#pragma unroll
	for (int m = 0; m < MM; ++m)
		if (m < (int)M)
			acc[m] = ffma(sign, ffma(fz, S.w[s][2][m], ffma(fy, S.w[s][1][m], fmul(fx, S.w[s][0][m]))), acc[m]);
}

/* acc[m] -= f_c * w_m[c]: the cooperative lane holding force component c */
template <int MM>
__device__ __forceinline__ void project_component(const ModeStage<MM>& S, uint32_t s, int c, uint32_t M,
		float f, float* acc) {
#pragma unroll
	for (int m = 0; m < MM; ++m)
		if (m < (int)M) acc[m] = ffma(-f, S.w[s][c][m], acc[m]);
}

}  // namespace

/* The pose frame of both passes: the rotation, its "inverted" counterpart
 * R(-ang) and t' = R^T (-t) (invertDOF, src/model/transform_modes.h:27-41),
 * and the translation. */
struct ModesFrame {
	PoseRot R;
	float Ri[9];
	float ip[3];
	float t[3];
};

/* Lane k (k < 26) brings the k-th float of the DOF_6D_Modes record; every
 * lane gets the frame and the amplitudes. */
template <int MM>
__device__ __forceinline__ ModesFrame modes_frame(const float dv, const int lane, float ampR[MM], float ampL[MM],
		const DevTrig& T) {
	ModesFrame F;
	F.t[0] = __shfl_sync(GBA_FULL_MASK, dv, 0);
	F.t[1] = __shfl_sync(GBA_FULL_MASK, dv, 1);
	F.t[2] = __shfl_sync(GBA_FULL_MASK, dv, 2);
	const float a0 = __shfl_sync(GBA_FULL_MASK, dv, 3);
	const float a1 = __shfl_sync(GBA_FULL_MASK, dv, 4);
	const float a2 = __shfl_sync(GBA_FULL_MASK, dv, 5);
#pragma unroll
	for (int m = 0; m < MM; ++m) {
		ampR[m] = __shfl_sync(GBA_FULL_MASK, dv, 6 + m);
		ampL[m] = __shfl_sync(GBA_FULL_MASK, dv, 16 + m);
	}
	F.R = pose_rotation(a0, a1, a2, lane, T);
	const PoseRot& R = F.R;
	/* R(-ang): same sin/cos with the sines negated (exact sign flips) */
	{
		const float cphi = R.cphi, sphi = -R.sphi, cssi = R.cssi, sssi = -R.sssi;
		const float crot = R.crot, srot = -R.srot;
		const float cSSI_cPHI = fmul(cssi, cphi), cSSI_sPHI = fmul(cssi, sphi);
		const float sSSI_cPHI = fmul(sssi, cphi), sSSI_sPHI = fmul(sssi, sphi);
		F.Ri[0] = fadd(fmul(crot, cSSI_cPHI), fmul(srot, sphi));
		F.Ri[1] = fsub(fmul(srot, cSSI_cPHI), fmul(crot, sphi));
		F.Ri[2] = sSSI_cPHI;
		F.Ri[3] = fsub(fmul(crot, cSSI_sPHI), fmul(srot, cphi));
		F.Ri[4] = fadd(fmul(srot, cSSI_sPHI), fmul(crot, cphi));
		F.Ri[5] = sSSI_sPHI;
		F.Ri[6] = fmul(-crot, sssi);
		F.Ri[7] = fmul(-srot, sssi);
		F.Ri[8] = cssi;
	}
	/* t' = R^T * (-t), RotMat * Vec3 on the transposed matrix */
	const float tx = F.t[0], ty = F.t[1], tz = F.t[2];
	F.ip[0] = fadd(fadd(fmul(R.m[0], -tx), fmul(R.m[3], -ty)), fmul(R.m[6], -tz));
	F.ip[1] = fadd(fadd(fmul(R.m[1], -tx), fmul(R.m[4], -ty)), fmul(R.m[7], -tz));
	F.ip[2] = fadd(fadd(fmul(R.m[2], -tx), fmul(R.m[5], -ty)), fmul(R.m[8], -tz));
	return F;
}

/* The pose frame and amplitudes of record dv, parked in the warp's staging. */
template <int MM>
__device__ __forceinline__ void put_frame(const ModesLaunch& L, const float dv, const int lane, ModeStage<MM>& MS) {
	float ampR[MM], ampL[MM];
	const ModesFrame F = modes_frame<MM>(dv, lane, ampR, ampL, L.trig);
	if (lane == 0) {
		float* v = MS.pose;
#pragma unroll
		for (int k = 0; k < 9; ++k) {
			v[k] = F.R.m[k];
			v[15 + k] = F.Ri[k];
		}
		v[9] = F.R.cphi; v[10] = F.R.sphi; v[11] = F.R.cssi; v[12] = F.R.sssi; v[13] = F.R.crot; v[14] = F.R.srot;
#pragma unroll
		for (int k = 0; k < 3; ++k) {
			v[24 + k] = F.ip[k];
			v[27 + k] = F.t[k];
		}
#pragma unroll
		for (int m = 0; m < MM; ++m) {
			v[30 + m] = ampR[m];
			v[30 + MM + m] = ampL[m];
		}
	}
	__syncwarp();
}

/* N parked floats from `at`; volatile, so that the compiler does not keep
 * them in registers from one use to the next. */
template <int N, int MM>
__device__ __forceinline__ void get_frame(const ModeStage<MM>& MS, int at, float (&out)[N]) {
	const volatile float* v = MS.pose + at;
#pragma unroll
	for (int k = 0; k < N; ++k) out[k] = v[k];
}

/* What staging a round takes of the parked frame.  Five modes on native grids
 * read it once per pass: reading it each round left the compiler few
 * registers' worth of lookups in flight (6,000 poses, 700/300 beads, 3 modes:
 * 482 against 392 us).  On octets, and at ten modes, the registers are better
 * spent on warps. */
template <int MM, int LAYOUT>
constexpr bool kHoldFrame = LAYOUT == kNative && MM <= 5;
template <int MM>
struct RecFrame {
	float Rm[9], Ri[9], ip[3], ampR[MM];
	__device__ __forceinline__ void read(const ModeStage<MM>& MS) {
		get_frame(MS, 0, Rm);
		get_frame(MS, 15, Ri);
		get_frame(MS, 24, ip);
		get_frame(MS, 30, ampR);
	}
};
template <int MM>
struct LigFrame {
	float Rm[9], tr[3], ampL[MM];
	__device__ __forceinline__ void read(const ModeStage<MM>& MS) {
		get_frame(MS, 0, Rm);
		get_frame(MS, 27, tr);
		get_frame(MS, 30 + MM, ampL);
	}
};

/* Stages 64 receptor beads from j0: deformed, moved into the ligand frame,
 * their lookups in the LIGAND grid queued, their mode vectors rotated for the
 * cooperative lookups.  Returns the number of lookups. */
template <int MM, class Stage>
__device__ __forceinline__ uint32_t modes_rec_stage(const ModesLaunch& L, const RecFrame<MM>& F, const uint32_t j0,
		const int lane, Stage& W, ModeStage<MM>& MS) {
	const uint32_t Mr = L.rec.n_modes;
	const float (&Rm)[9] = F.Rm, (&Ri)[9] = F.Ri, (&ip)[3] = F.ip, (&ampR)[MM] = F.ampR;
	uint32_t nlk[2];
	BeadGrid bg[2];
#pragma unroll
	for (int h = 0; h < 2; ++h) {
		const int s = lane + 32 * h;
		const uint32_t j = j0 + s;
		nlk[h] = 0;
		bg[h] = BeadGrid{0u, 0u};
		if (j < L.rec.n) {
			const float4 r = __ldg(&L.rec.xyzq[j]);
			const uint32_t mapped = __ldg(&L.rec.tm[j]) >> 16;
			float vw[4 * kModeWords<MM>];
			load_modes<MM>(L.rec_modes + (size_t)j * L.rec_ms, Mr, vw);
			float x = r.x, y = r.y, z = r.z;
			deform_w<MM>(vw, Mr, ampR, x, y, z);
			float px, py, pz;
			rot_apply(Ri, x, y, z, px, py, pz);
			px = fadd(px, ip[0]); py = fadd(py, ip[1]); pz = fadd(pz, ip[2]);
			W.put_rec(s, r.w, j);
			nlk[h] = stage_grid(L.grid_lig, px, py, pz, mapped, r.w, s, W, bg[h]);
			/* the ligand-frame force f is rotated back by R before the
			 * projection: (R f) . v = f . (R^T v); staged for the
			 * cooperative lookups only (one lookup per bead or two: the
			 * per-lane form rotates f instead) */
			if (nlk[h] && L.grid_lig.coop_lookup) stage_modes<MM>(MS, s, vw, Mr, Rm, true);
		}
	}
	const uint32_t n_look = queue_lookups(W, nlk, bg, lane);
	__syncwarp();
	return n_look;
}

/* Receptor pass: the receptor beads, deformed and moved into the ligand
 * frame, in the LIGAND grid; each force rotated back by R and projected on
 * the receptor modes into the lane sums gR.  BLOCKS: lookup blocks in flight
 * per cooperative step; the scoring kernel has the registers for four (20,000
 * poses, 1500/600 beads: 1,837 -> 1,765 us), the minimizer's code has not
 * (15.0 -> 16.0 ms for 6,000 poses). */
template <int MM, int LAYOUT = kAnyLayout, int BLOCKS = 2, class Stage>
__device__ __forceinline__ void modes_rec_pass(const ModesLaunch& L, const int lane, Stage& W, ModeStage<MM>& MS,
		float gR[MM]) {
	const uint32_t Mr = L.rec.n_modes;
	const int comp = coop_component(lane);
	RecFrame<MM> F;
	if (kHoldFrame<MM, LAYOUT>) F.read(MS);
	for (uint32_t j0 = 0; j0 < L.rec.n; j0 += kBeadsPerRound) {
		if (!kHoldFrame<MM, LAYOUT>) F.read(MS);
		const uint32_t n_look = modes_rec_stage<MM>(L, F, j0, lane, W, MS);
		if (LAYOUT == kAnyLayout ? L.grid_lig.coop_lookup != 0 : LAYOUT == kOctets) {
			for (uint32_t k0 = 0; k0 < n_look; k0 += 8 * BLOCKS) {
				CoopStep<BLOCKS> st;
				st.load(L.grid_lig, W, k0, n_look, lane);
#pragma unroll
				for (int b = 0; b < BLOCKS; ++b) {
					const float v = st.component(b, lane);
					if (st.ok[b] && comp < 3) project_component<MM>(MS, st.sl[b], comp, Mr, fmul(v, st.sc[b]), gR);
				}
			}
		} else {
			float (&Rm)[9] = F.Rm;
			for (uint32_t q = lane; q < n_look; q += 32) {
				const uint32_t s = lookup_slot(W, q);
				const float4 v = grid_lookup(L.grid_lig, W, q);
				/* back into the receptor frame, then -(force . mode) */
				float fx, fy, fz;
				rot_apply(Rm, v.x, v.y, v.z, fx, fy, fz);
				project<MM>(L.rec_modes + (size_t)W.bead(s) * L.rec_ms, Mr, fx, fy, fz, -1.f, gR);
			}
		}
		__syncwarp();
	}

}

/* Stages 64 ligand beads from i0: deformed, moved into the receptor frame,
 * lookups and neighbour lists queued, mode vectors rotated.  Returns the
 * number of lookups; n_pair, nln, start as queue_pairs has them. */
template <int MM>
__device__ __forceinline__ uint32_t modes_lig_stage(const ModesLaunch& L, const LigFrame<MM>& F, const uint32_t i0,
		const int lane, WarpStage& W, ModeStage<MM>& MS, uint32_t nln[2], uint32_t start[2], uint32_t& n_pair) {
	const uint32_t Ml = L.lig.n_modes;
	const float (&Rm)[9] = F.Rm, (&tr)[3] = F.tr, (&ampL)[MM] = F.ampL;
	uint32_t nlk[2];
	BeadGrid bg[2];
#pragma unroll
	for (int h = 0; h < 2; ++h) {
		const int s = lane + 32 * h;
		const uint32_t i = i0 + s;
		nlk[h] = 0;
		nln[h] = 0;
		bg[h] = BeadGrid{0u, 0u};
		if (i < L.lig.n) {
			const float4 b = __ldg(&L.lig.xyzq[i]);
			const uint32_t tm = __ldg(&L.lig.tm[i]);
			const uint32_t type = tm & 0xffffu, mapped = tm >> 16;
			float vw[4 * kModeWords<MM>];
			load_modes<MM>(L.lig_modes + (size_t)i * L.lig_ms, Ml, vw);
			float x = b.x, y = b.y, z = b.z;
			deform_w<MM>(vw, Ml, ampL, x, y, z);
			float px, py, pz;
			rot_apply(Rm, x, y, z, px, py, pz);
			px = fadd(px, tr[0]); py = fadd(py, tr[1]); pz = fadd(pz, tr[2]);
			put_bead(W, s, b.x, b.y, b.z, px, py, pz, b.w, type);
			nlk[h] = stage_grid(L.grid_rec, px, py, pz, mapped, b.w, s, W, bg[h]);
			bool in_nl;
			if (type != 0) nln[h] = stage_nl(L.grid_rec.nl, px, py, pz, s, W, in_nl);
			/* the global-frame force f is projected in the ligand frame:
			 * (R^T f) . v = f . (R v) */
			if (nlk[h] | nln[h]) stage_modes<MM>(MS, s, vw, Ml, Rm, false);
		}
	}
	const uint32_t n_look = queue_lookups(W, nlk, bg, lane);
	n_pair = queue_pairs(W, nln, lane, start);
	__syncwarp();
	return n_look;
}

/* One flattened pair -- ligand bead staged in slot s, list entry at `at` --
 * against the deformed receptor: receptor bead j, its mode vectors vw, force
 * and energy; false outside the plateau. */
template <int MM>
__device__ __forceinline__ bool modes_pair(const ModesLaunch& L, const float ampR[MM], const WarpStage& W, uint32_t s,
		uint32_t at, uint32_t& j, float (&vw)[4 * kModeWords<MM>], float& fx, float& fy, float& fz, float& e) {
	const uint32_t Mr = L.rec.n_modes;
	j = __ldg(&L.grid_rec.nl.list[at]);
	const float4 r = __ldg(&L.rec.xyzq[j]);
	float rx = r.x, ry = r.y, rz = r.z;
	load_modes<MM>(L.rec_modes + (size_t)j * L.rec_ms, Mr, vw);
	deform_w<MM>(vw, Mr, ampR, rx, ry, rz);
	const uint32_t trec = __ldg(&L.rec.tm[j]) & 0xffffu;
	const float4 b = W.pq[s];
	return nl_pair(L.grid_rec.nl, L.par, __float_as_uint(W.ut[s].w), b.w, b.x, b.y, b.z, rx, ry, rz, r.w, trec, fx, fy,
			fz, e);
}

/* gR[m] += f . v_m: the reaction on a receptor bead is -f, and its mode
 * gradient gets -(-f . v). */
template <int MM>
__device__ __forceinline__ void project_reaction(const float (&vw)[4 * kModeWords<MM>], uint32_t Mr, float fx, float fy,
		float fz, float gR[MM]) {
#pragma unroll
	for (int m = 0; m < MM; ++m)
		if (m < (int)Mr)
			gR[m] = ffma(1.f, ffma(fz, vw[3 * m + 2], ffma(fy, vw[3 * m + 1], fmul(fx, vw[3 * m]))), gR[m]);
}

/* A finished component f of a lookup in slot s, on the lane holding component
 * comp: the cooperative sums without the ligand modes. */
__device__ __forceinline__ void coop_add(const WarpStage& W, uint32_t s, int comp, float f, CoopSums& C) {
	C.f = fadd(C.f, f);
	if (comp != 3) {
		const float4 u = W.ut[s];
		C.t0 = ffma(u.x, f, C.t0);
		C.t1 = ffma(u.y, f, C.t1);
		C.t2 = ffma(u.z, f, C.t2);
	}
}

/* Ligand pass: the ligand beads, deformed and moved into the receptor frame,
 * in the receptor grid, plus the NL pairs against the deformed receptor:
 * energy, force and torque into S and C, ligand mode projections into gL,
 * the pairs' reaction forces projected on the receptor modes into gR. */
template <int MM, int LAYOUT = kAnyLayout>
__device__ __forceinline__ void modes_lig_pass(const ModesLaunch& L, const int lane, WarpStage& W, ModeStage<MM>& MS,
		PoseSums& S, CoopSums& C, float gL[MM], float gR[MM]) {
	const uint32_t Mr = L.rec.n_modes, Ml = L.lig.n_modes;
	const int comp = coop_component(lane);
	LigFrame<MM> F;
	float ampR[MM];
	if (kHoldFrame<MM, LAYOUT>) {
		F.read(MS);
		get_frame(MS, 30, ampR);
	}
	for (uint32_t i0 = 0; i0 < L.lig.n; i0 += kBeadsPerRound) {
		uint32_t nln[2], start[2], n_pair;
		if (!kHoldFrame<MM, LAYOUT>) F.read(MS);
		const uint32_t n_look = modes_lig_stage<MM>(L, F, i0, lane, W, MS, nln, start, n_pair);
		if (LAYOUT == kAnyLayout ? L.grid_rec.coop_lookup != 0 : LAYOUT == kOctets) {
			for (uint32_t k0 = 0; k0 < n_look; k0 += 16) {
				CoopStep<2> st;
				st.load(L.grid_rec, W, k0, n_look, lane);
#pragma unroll
				for (int b = 0; b < 2; ++b) {
					const float v = st.component(b, lane);
					if (st.ok[b]) {
						const float f = fmul(v, st.sc[b]);
						coop_add(W, st.sl[b], comp, f, C);
						if (comp != 3) project_component<MM>(MS, st.sl[b], comp, Ml, f, gL);
					}
				}
			}
		} else {
			for (uint32_t q = lane; q < n_look; q += 32) {
				const uint32_t s = lookup_slot(W, q);
				const float4 v = grid_lookup(L.grid_rec, W, q);
				const float4 u = W.ut[s];
				S.add(v.w, v.x, v.y, v.z, u.x, u.y, u.z);
				project_staged<MM>(MS, s, Ml, v.x, v.y, v.z, -1.f, gL);
			}
		}
		/* neighbour pairs after the lookups: measured faster here (the rigid
		 * kernel measured the opposite) */
		if (!kHoldFrame<MM, LAYOUT>) get_frame(MS, 30, ampR);
		PairWindow win;
		for (uint32_t w = 0; w < n_pair; w += 64) {
			uint32_t so[2];
			win.owners(W, w, start, nln, lane, so[0], so[1]);
#pragma unroll
			for (int h = 0; h < 2; ++h) {
				const uint32_t q = w + 32 * h + lane;
				if (q >= n_pair) continue;
				const uint32_t s = so[h];
				uint32_t j;
				float vw[4 * kModeWords<MM>], fx, fy, fz, e;
				if (!modes_pair<MM>(L, ampR, W, s, W.lbase[s] + q, j, vw, fx, fy, fz, e)) continue;
				const float4 u = W.ut[s];
				S.add(e, fx, fy, fz, u.x, u.y, u.z);
				project_reaction<MM>(vw, Mr, fx, fy, fz, gR);
				project_staged<MM>(MS, s, Ml, fx, fy, fz, -1.f, gL);
			}
		}
		__syncwarp();
	}
}

/* The Result_6D_Modes record from the pose's sums (energy, force, torque
 * matrix; gR and gL the modes' gradients): correctModeForce (delta += 4 k
 * delta^4, src/model/reduction_modes.h:101-115), ForceLim, TorqueMat.  Lane k
 * (k < 27) returns float k of the record. */
template <int MM>
__device__ __forceinline__ float modes_record(const ModesLaunch& L, const PoseRot& R, float sE, float sFx, float sFy,
		float sFz, const float T[9], float gL[MM], float gR[MM], const int lane) {
	const uint32_t Mr = L.rec.n_modes, Ml = L.lig.n_modes;
	force_lim(sFx, sFy, sFz);
	float ang[3];
	torque_reduce(R, T, ang);
	/* correctModeForce: delta += (float)(4 k * delta^4) */
#pragma unroll
	for (int m = 0; m < MM; ++m) {
		if (m < (int)Mr) {
			const double dl = gR[m];
			gR[m] = fadd(gR[m], (float)__dmul_rn(__dmul_rn((double)fmul(4.0f, L.rec.mode_force[m]),
					__dmul_rn(dl, dl)), __dmul_rn(dl, dl)));
		}
		if (m < (int)Ml) {
			const double dl = gL[m];
			gL[m] = fadd(gL[m], (float)__dmul_rn(__dmul_rn((double)fmul(4.0f, L.lig.mode_force[m]),
					__dmul_rn(dl, dl)), __dmul_rn(dl, dl)));
		}
	}
	/* Result_6D_Modes: E, pos xyz, ang xyz, modesRec[10], modesLig[10] */
	float v = 0.f;
	if (lane == 0) v = sE;
	else if (lane == 1) v = sFx;
	else if (lane == 2) v = sFy;
	else if (lane == 3) v = sFz;
	else if (lane == 4) v = ang[0];
	else if (lane == 5) v = ang[1];
	else if (lane == 6) v = ang[2];
#pragma unroll
	for (int m = 0; m < MM; ++m) {
		if (lane == 7 + m) v = m < (int)Mr ? gR[m] : 0.f;
		if (lane == 17 + m) v = m < (int)Ml ? gL[m] : 0.f;
	}
	return v;
}

template <int MM>
__device__ __forceinline__ PoseRot frame_rotation(const ModeStage<MM>& MS) {
	PoseRot R;
	float c[6];
	get_frame(MS, 0, R.m);
	get_frame(MS, 9, c);
	R.cphi = c[0]; R.sphi = c[1]; R.cssi = c[2]; R.sssi = c[3]; R.crot = c[4]; R.srot = c[5];
	return R;
}

/* modes_record from the ligand pass's lane sums and the two passes'
 * receptor-mode gradients (the receptor pass's warp-summed, added first). */
template <int MM>
__device__ __forceinline__ float modes_epilogue(const ModesLaunch& L, const ModeStage<MM>& MS, PoseSums& S,
		const CoopSums& C, float gL[MM], const float gR_rec[MM], float gR_nl[MM], const int lane) {
	const uint32_t Mr = L.rec.n_modes, Ml = L.lig.n_modes;
	fold_coop(C, S, lane);
	const float sE = warp_sum(S.E), sFx = warp_sum(S.Fx), sFy = warp_sum(S.Fy), sFz = warp_sum(S.Fz);
	float T[9];
#pragma unroll
	for (int k = 0; k < 9; ++k) T[k] = warp_sum(S.T[k]);
	float gR[MM];
#pragma unroll
	for (int m = 0; m < MM; ++m) {
		gR[m] = 0.f;
		if (m < (int)Mr) gR[m] = fadd(gR_rec[m], warp_sum(gR_nl[m]));
		if (m < (int)Ml) gL[m] = warp_sum(gL[m]);
	}
	return modes_record<MM>(L, frame_rotation(MS), sE, sFx, sFy, sFz, T, gL, gR, lane);
}

/* Warp sums of the receptor pass's mode gradients (every lane). */
template <int MM>
__device__ __forceinline__ void sum_rec_modes(uint32_t Mr, float gR[MM]) {
#pragma unroll
	for (int m = 0; m < MM; ++m)
		if (m < (int)Mr) gR[m] = warp_sum(gR[m]);
}

/* One pose of the modes energy, both passes in one warp (the minimizer's
 * form).  Lane k (k < 26) brings the k-th float of the DOF_6D_Modes record;
 * returns on lane k (k < 27) the k-th float of the Result_6D_Modes record.
 * Only the model fields of L are read.  MM >= the receptor's and the
 * ligand's mode counts.  Bit for bit the result of the split scoring
 * kernels (modes_rec_kernel then modes_lig_kernel). */
template <int MM, int LAYOUT>
__device__ __forceinline__ float eval_pose_modes(const ModesLaunch& L, const float dv, const int lane,
		FullStage& W, ModeStage<MM>& MS) {
	put_frame<MM>(L, dv, lane, MS);
	float gRr[MM], gRn[MM], gL[MM];
#pragma unroll
	for (int m = 0; m < MM; ++m) { gRr[m] = 0.f; gRn[m] = 0.f; gL[m] = 0.f; }
	modes_rec_pass<MM, LAYOUT>(L, lane, W, MS, gRr);
	sum_rec_modes<MM>(L.rec.n_modes, gRr);
	PoseSums S;
	CoopSums C;
	modes_lig_pass<MM, LAYOUT>(L, lane, W, MS, S, C, gL, gRn);
	return modes_epilogue<MM>(L, MS, S, C, gL, gRr, gRn, lane);
}

/* ---- a pose split over the warps of a block ---------------------------------
 *
 * One warp's evaluation is a chain of rounds (777/333 beads, 7 modes each: 13
 * receptor and 6 ligand rounds, 112 + 135 us for a warp by itself), and every
 * sum is a chain too: each lane adds its terms in round order, which the
 * results' bits rest on.  The terms are independent, though, and most of the
 * work.  A team takes as many rounds at a time as it has warps: warp t stages
 * round t, drains its lookups and computes its pairs, leaving each lane's
 * term (a lookup's finished component; a pair's force, energy, slot and
 * receptor bead) in shared memory; then the sums are continued over the
 * rounds in order, each by one warp -- the receptor modes dealt over all
 * warps, and of the ligand pass energy, force and torque, the reactions on
 * the receptor modes, and the ligand modes by up to three.  Where a round has
 * more pairs than a warp's buffer holds (a clash), all warps compute pairs of
 * one round at a time.  Bit for bit eval_pose_modes on octet grids. */
constexpr int kModesMaxTeam = 8;
constexpr int kTeamHalves = 4;      /* half-windows (32 pairs) of a round held at once */

template <int MM>
struct ModesTeamWarp {
	FullStage W;
	ModeStage<MM> MS;
	float f[2 * kBeadsPerRound / 8][32];     /* component of the lane's lookup in block b */
	float4 pv[kTeamHalves][32];              /* force and energy of the lane's pair */
	uint32_t pj[kTeamHalves][32];            /* receptor bead | slot << 24 | 1 << 31; 0: no pair */
	uint32_t start[kBeadsPerRound], len[kBeadsPerRound];   /* the round's flattened pairs by slot */
};

template <int MM>
struct ModesTeamShared {
	float gRr[MM], gRn[MM], gL[MM];          /* warp sums of the modes' gradients */
	uint32_t n_look[kModesMaxTeam];
	uint32_t halves[kModesMaxTeam];
	float dof[26];
	int stop;
	unsigned long long pose;
};

/* The lane's lookup of block b (eight lookups), if there is one. */
__device__ __forceinline__ uint32_t coop_lookup_index(uint32_t b, int lane) {
	return 8 * b + 4 * (lane & 1) + (lane >> 3);
}

/* Drains the round's lookups into f. */
template <int MM>
__device__ __forceinline__ void team_lookups(const DevGrid& G, ModesTeamWarp<MM>& T, uint32_t n_look, int lane) {
	for (uint32_t k0 = 0; k0 < n_look; k0 += 16) {
		CoopStep<2> st;
		st.load(G, T.W, k0, n_look, lane);
#pragma unroll
		for (int b = 0; b < 2; ++b) T.f[k0 / 8 + b][lane] = fmul(st.component(b, lane), st.sc[b]);
	}
}

/* The pairs of half-windows [h0, h0 + kTeamHalves) of the round staged in R
 * into the buffer of T (this warp's). */
template <int MM>
__device__ __forceinline__ void team_pairs(const ModesLaunch& L, const ModesTeamWarp<MM>& R,
		ModesTeamWarp<MM>& T, uint32_t h0, int lane) {
	float ampR[MM];
	get_frame(T.MS, 30, ampR);
	const uint32_t start[2] = {R.start[lane], R.start[lane + 32]}, len[2] = {R.len[lane], R.len[lane + 32]};
	const uint32_t n_pair = __reduce_max_sync(GBA_FULL_MASK, max(len[0] ? start[0] + len[0] : 0u, len[1] ? start[1] + len[1] : 0u));
	if (32 * h0 >= n_pair) return;
	PairWindow win;
	if (h0 > 0) {
		/* the bead that covers the pair before the first window */
		const uint32_t q = 32 * h0 - 1;
		uint32_t slot = 0;
#pragma unroll
		for (int h = 0; h < 2; ++h)
			if (q >= start[h] && q - start[h] < len[h]) slot = 1u + lane + 32 * h;
		win.carry = __reduce_max_sync(GBA_FULL_MASK, slot) - 1u;
	}
	for (uint32_t hw = 0; hw < kTeamHalves && 32 * (h0 + hw) < n_pair; hw += 2) {
		const uint32_t w = 32 * (h0 + hw);
		uint32_t so[2];
		win.owners(T.W, w, start, len, lane, so[0], so[1]);
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			const uint32_t q = w + 32 * h + lane;
			uint32_t pj = 0;
			if (q < n_pair) {
				uint32_t j;
				float vw[4 * kModeWords<MM>], fx, fy, fz, e;
				if (modes_pair<MM>(L, ampR, R.W, so[h], R.W.lbase[so[h]] + q, j, vw, fx, fy, fz, e)) {
					T.pv[hw + h][lane] = make_float4(fx, fy, fz, e);
					pj = j | so[h] << 24 | 0x80000000u;
				}
			}
			T.pj[hw + h][lane] = pj;
		}
	}
}

/* One pose by a block of G warps; every warp calls it with the pose's record
 * in dv (lane k: float k).  Warp 0's lane k (k < 27) returns float k of the
 * result. */
template <int MM>
__device__ __forceinline__ float eval_pose_modes_team(const ModesLaunch& L, const float dv, const int lane, const int t,
		const int G, ModesTeamWarp<MM>* team, ModesTeamShared<MM>& sh) {
	const uint32_t Mr = L.rec.n_modes, Ml = L.lig.n_modes;
	const int comp = coop_component(lane);
	ModesTeamWarp<MM>& me = team[t];
	put_frame<MM>(L, dv, lane, me.MS);
	uint32_t mine = 0;      /* the receptor modes this warp sums over the receptor pass */
	for (int m = t; m < (int)Mr; m += G) mine |= 1u << m;

	/* receptor pass */
	{
		const uint32_t rounds = (L.rec.n + kBeadsPerRound - 1) / kBeadsPerRound;
		float gR[MM];
#pragma unroll
		for (int m = 0; m < MM; ++m) gR[m] = 0.f;
		for (uint32_t r0 = 0; r0 < rounds; r0 += G) {
			uint32_t n_look = 0;
			if (r0 + t < rounds) {
				RecFrame<MM> F;
				F.read(me.MS);
				n_look = modes_rec_stage<MM>(L, F, (r0 + t) * kBeadsPerRound, lane, me.W, me.MS);
				team_lookups<MM>(L.grid_lig, me, n_look, lane);
			}
			if (lane == 0) sh.n_look[t] = n_look;
			__syncthreads();
			for (int u = 0; u < G; ++u) {
				const uint32_t nl = sh.n_look[u];
				for (uint32_t b = 0; 8 * b < nl; ++b) {
					const uint32_t k = coop_lookup_index(b, lane);
					if (k < nl && comp < 3) {
						const uint32_t s = lookup_slot(team[u].W, k);
						const float f = team[u].f[b][lane];
#pragma unroll
						for (int m = 0; m < MM; ++m)
							if (mine >> m & 1u) gR[m] = ffma(-f, team[u].MS.w[s][comp][m], gR[m]);
					}
				}
			}
			__syncthreads();
		}
#pragma unroll
		for (int m = 0; m < MM; ++m)
			if (mine >> m & 1u) {
				const float v = warp_sum(gR[m]);
				if (lane == 0) sh.gRr[m] = v;
			}
	}

	/* ligand pass: energy, force, torque on warp 0; reactions; ligand modes */
	const bool do_nl = t == 1 % G, do_lig = t == 2 % G;
	const uint32_t rounds = (L.lig.n + kBeadsPerRound - 1) / kBeadsPerRound;
	PoseSums S;
	CoopSums C;
	float gRn[MM], gL[MM];
#pragma unroll
	for (int m = 0; m < MM; ++m) {
		gRn[m] = 0.f;
		gL[m] = 0.f;
	}
	for (uint32_t r0 = 0; r0 < rounds; r0 += G) {
		uint32_t n_look = 0, n_pair = 0, nln[2] = {0, 0}, start[2] = {0, 0};
		if (r0 + t < rounds) {
			LigFrame<MM> F;
			F.read(me.MS);
			n_look = modes_lig_stage<MM>(L, F, (r0 + t) * kBeadsPerRound, lane, me.W, me.MS, nln, start, n_pair);
			team_lookups<MM>(L.grid_rec, me, n_look, lane);
		}
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			me.start[lane + 32 * h] = start[h];
			me.len[lane + 32 * h] = nln[h];
		}
		if (lane == 0) {
			sh.n_look[t] = n_look;
			sh.halves[t] = (n_pair + 31) / 32;
		}
		__syncthreads();
		uint32_t most = 0;
		for (int u = 0; u < G; ++u) most = max(most, sh.halves[u]);
		const bool apart = most <= kTeamHalves;      /* every warp holds its own round's pairs */
		if (apart) {
			team_pairs<MM>(L, me, me, 0, lane);
			__syncthreads();
		}
		for (int u = 0; u < G; ++u) {
			const ModesTeamWarp<MM>& you = team[u];
			const uint32_t nl = sh.n_look[u], nh = sh.halves[u];
			if (t == 0 || do_lig)
				for (uint32_t b = 0; 8 * b < nl; ++b) {
					const uint32_t k = coop_lookup_index(b, lane);
					if (k < nl) {
						const uint32_t s = lookup_slot(you.W, k);
						const float f = you.f[b][lane];
						if (t == 0) coop_add(you.W, s, comp, f, C);
						if (do_lig && comp != 3) project_component<MM>(you.MS, s, comp, Ml, f, gL);
					}
				}
			for (uint32_t h0 = 0; h0 < nh; h0 += kTeamHalves) {
				const uint32_t part = h0 / kTeamHalves % G;
				if (!apart && part == 0) {
					__syncthreads();      /* the buffers have been read */
					team_pairs<MM>(L, you, me, h0 + t * kTeamHalves, lane);
					__syncthreads();
				}
				if (!(t == 0 || do_nl || do_lig)) continue;
				const ModesTeamWarp<MM>& held = apart ? you : team[part];
				const uint32_t n = min(nh - h0, (uint32_t)kTeamHalves);
				for (uint32_t h = 0; h < n; ++h) {
					const uint32_t pj = held.pj[h][lane];
					if (!pj) continue;
					const float4 v = held.pv[h][lane];
					const uint32_t s = pj >> 24 & 0x7fu;
					if (t == 0) {
						const float4 x = you.W.ut[s];
						S.add(v.w, v.x, v.y, v.z, x.x, x.y, x.z);
					}
					if (do_nl) {
						float vw[4 * kModeWords<MM>];
						load_modes<MM>(L.rec_modes + (size_t)(pj & 0xffffffu) * L.rec_ms, Mr, vw);
						project_reaction<MM>(vw, Mr, v.x, v.y, v.z, gRn);
					}
					if (do_lig) project_staged<MM>(you.MS, s, Ml, v.x, v.y, v.z, -1.f, gL);
				}
			}
		}
		__syncthreads();
	}
#pragma unroll
	for (int m = 0; m < MM; ++m) {
		if (do_nl && m < (int)Mr) {
			const float v = warp_sum(gRn[m]);
			if (lane == 0) sh.gRn[m] = v;
		}
		if (do_lig && m < (int)Ml) {
			const float v = warp_sum(gL[m]);
			if (lane == 0) sh.gL[m] = v;
		}
	}
	__syncthreads();
	if (t != 0) return 0.f;
	fold_coop(C, S, lane);
	const float sE = warp_sum(S.E), sFx = warp_sum(S.Fx), sFy = warp_sum(S.Fy), sFz = warp_sum(S.Fz);
	float T[9];
#pragma unroll
	for (int k = 0; k < 9; ++k) T[k] = warp_sum(S.T[k]);
	float gRt[MM], gLt[MM];
#pragma unroll
	for (int m = 0; m < MM; ++m) {
		gRt[m] = m < (int)Mr ? fadd(sh.gRr[m], sh.gRn[m]) : 0.f;
		gLt[m] = m < (int)Ml ? sh.gL[m] : 0.f;
	}
	return modes_record<MM>(L, frame_rotation(me.MS), sE, sFx, sFy, sFz, T, gLt, gRt, lane);
}

/* ---- the reference CPU path's order (GBA_KOPT_REFERENCE_ORDER) ----------
 *
 * CPUEnergyService6DModes evaluates a pose array by array
 * (src/service/CPUEnergyService6DModes.tpp:121-327): the receptor deformed
 * and moved into the ligand frame, its grid forces (ligand grid) rotated back
 * per bead; the ligand deformed and moved, its grid forces (receptor grid);
 * the NL term bead by bead in list order, adding each pair's four sub-terms
 * to the ligand bead and their reaction to the receptor bead; then sums in
 * bead order: energy and force, the ligand mode projections of R^T f, the
 * receptor mode projections, correctModeForce, the torque.  The rigid
 * reference order's pieces (ref_grid_term, ref_pair_terms, ref_fold,
 * ref_accumulate) follow it operation for operation; the receptor bead
 * forces need a per-pose array (scratch in global memory, one per warp,
 * float4 per receptor bead), and each receptor reaction is added to it in
 * the reference's pair order by three lanes, one per component. */

/* Receptor bead index of each window position (the reactions' scatter). */
struct RefModesExtra {
	uint32_t j[32];
};

/* x^4 correctly rounded, standing in for std::pow(x, 4) of
 * correctModeForce: x^2 = p + e and p^2 = hi + lo exactly (Dekker's
 * products through fma), x^4 = hi + (lo + 2 p e + e^2). */
__device__ __forceinline__ double pow4_rn(double x) {
	const double p = __dmul_rn(x, x);
	const double e = __fma_rn(x, x, -p);
	const double hi = __dmul_rn(p, p);
	const double lo = __fma_rn(p, p, -hi);
	return __dadd_rn(hi, __fma_rn(__dmul_rn(2.0, p), e, __fma_rn(e, e, lo)));
}

/* One pose in the reference's order; rf: this warp's receptor array.  Lane
 * k (k < 26) brings the k-th float of the DOF_6D_Modes record; returns on
 * lane k (k < 27) the k-th float of the Result_6D_Modes record. */
template <int MM, bool WIDE>
__device__ __forceinline__ float eval_pose_modes_ref(const ModesLaunch& L, const float dv, const int lane,
		WarpStage& W, RefModesExtra& X, float4* __restrict__ rf) {
	const uint32_t Mr = L.rec.n_modes, Ml = L.lig.n_modes;
	const float tx = __shfl_sync(GBA_FULL_MASK, dv, 0);
	const float ty = __shfl_sync(GBA_FULL_MASK, dv, 1);
	const float tz = __shfl_sync(GBA_FULL_MASK, dv, 2);
	const float a0 = __shfl_sync(GBA_FULL_MASK, dv, 3);
	const float a1 = __shfl_sync(GBA_FULL_MASK, dv, 4);
	const float a2 = __shfl_sync(GBA_FULL_MASK, dv, 5);
	float ampR[MM], ampL[MM];
#pragma unroll
	for (int m = 0; m < MM; ++m) {
		ampR[m] = __shfl_sync(GBA_FULL_MASK, dv, 6 + m);
		ampL[m] = __shfl_sync(GBA_FULL_MASK, dv, 16 + m);
	}
	const PoseRot R0 = pose_rotation(a0, a1, a2, lane, L.trig);

	/* receptor: invertDOF (src/model/transform_modes.h:27-41) -- R(-ang)
	 * from the sin/cos of the negated angles, t' = R^T (-t) -- then per bead
	 * the ligand-grid force rotated back by R */
	{
		const PoseRot Rn = pose_rotation(-a0, -a1, -a2, lane, L.trig);
		const float ipx = fadd(fadd(fmul(R0.m[0], -tx), fmul(R0.m[3], -ty)), fmul(R0.m[6], -tz));
		const float ipy = fadd(fadd(fmul(R0.m[1], -tx), fmul(R0.m[4], -ty)), fmul(R0.m[7], -tz));
		const float ipz = fadd(fadd(fmul(R0.m[2], -tx), fmul(R0.m[5], -ty)), fmul(R0.m[8], -tz));
		for (uint32_t j0 = 0; j0 < L.rec.n; j0 += kBeadsPerRound) {
#pragma unroll
			for (int h = 0; h < 2; ++h) {
				const int s = lane + 32 * h;
				const uint32_t j = j0 + s;
				if (j >= L.rec.n) continue;
				const float4 r = __ldg(&L.rec.xyzq[j]);
				const uint32_t mapped = __ldg(&L.rec.tm[j]) >> 16;
				float x = r.x, y = r.y, z = r.z;
				deform<MM, WIDE>(L.rec_modes + (size_t)j * L.rec_ms, Mr, ampR, x, y, z);
				float px, py, pz;
				rot_apply(Rn.m, x, y, z, px, py, pz);
				px = fadd(px, ipx); py = fadd(py, ipy); pz = fadd(pz, ipz);
				const float4 pot = ref_grid_term(L.grid_lig, px, py, pz, mapped, r.w, s, W);
				float fx, fy, fz;
				rot_apply(R0.m, pot.x, pot.y, pot.z, fx, fy, fz);
				rf[j] = make_float4(fx, fy, fz, 0.f);
			}
		}
	}
	__syncwarp();

	/* ligand: grid term, NL term with the receptor reactions, sums in bead
	 * order -- lanes 0..12 energy, force, torque; lanes 16 + m the ligand
	 * mode projections */
	const uint32_t* lst = L.grid_rec.nl.typed_list ? L.grid_rec.nl.typed_list : L.grid_rec.nl.list;
	const bool typed = L.grid_rec.nl.typed_list != nullptr;
	float acc = 0.f;
	for (uint32_t i0 = 0; i0 < L.lig.n; i0 += kBeadsPerRound) {
		float4 pot[2];
		uint32_t nln[2];
		bool in_nl[2];
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			const int s = lane + 32 * h;
			const uint32_t i = i0 + s;
			pot[h] = make_float4(0.f, 0.f, 0.f, 0.f);
			nln[h] = 0;
			in_nl[h] = false;
			if (i >= L.lig.n) continue;
			const float4 b = __ldg(&L.lig.xyzq[i]);
			const uint32_t tm = __ldg(&L.lig.tm[i]);
			const uint32_t type = tm & 0xffffu, mapped = tm >> 16;
			float x = b.x, y = b.y, z = b.z;
			deform<MM, WIDE>(L.lig_modes + (size_t)i * L.lig_ms, Ml, ampL, x, y, z);
			float px, py, pz;
			rot_apply(R0.m, x, y, z, px, py, pz);
			px = fadd(px, tx); py = fadd(py, ty); pz = fadd(pz, tz);
			put_bead(W, s, b.x, b.y, b.z, px, py, pz, b.w, type);
			pot[h] = ref_grid_term(L.grid_rec, px, py, pz, mapped, b.w, s, W);
			if (type != 0) nln[h] = stage_nl(L.grid_rec.nl, px, py, pz, s, W, in_nl[h]);
		}
		uint32_t start[2];
		const uint32_t n_pair = queue_pairs(W, nln, lane, start);
		__syncwarp();   /* weights read, list bases final: the overlay may be written */
		RefTerms& T = ref_terms(W);
		if (n_pair > 0) {
#pragma unroll
			for (int k = 0; k < 8; ++k) (&T.acc[0][0])[lane + 32 * k] = 0.f;
		}
		PairWindow win;
		for (uint32_t w = 0; w < n_pair; w += 64) {
			uint32_t sa, sb, ea = 0, eb = 0;
			win.owners(W, w, start, nln, lane, sa, sb);
			if (w + lane < n_pair) ea = __ldg(&lst[W.lbase[sa] + w + lane]);
			if (w + 32 + lane < n_pair) eb = __ldg(&lst[W.lbase[sb] + w + 32 + lane]);
#pragma unroll
			for (int half = 0; half < 2; ++half) {
				const uint32_t wb = w + 32 * half;
				if (wb >= n_pair) break;
				if (wb + lane < n_pair) {
					const uint32_t ent = half ? eb : ea;
					const uint32_t j = typed ? ent & 0xffffffu : ent;
					const uint32_t trec = typed ? ent >> 24 : __ldg(&L.rec.tm[j]) & 0xffffu;
					const float4 r = __ldg(&L.rec.xyzq[j]);
					float rx = r.x, ry = r.y, rz = r.z;
					deform<MM, WIDE>(L.rec_modes + (size_t)j * L.rec_ms, Mr, ampR, rx, ry, rz);
					ref_pair_terms(L.grid_rec.nl, L.par, W, half ? sb : sa, make_float4(rx, ry, rz, r.w), trec,
							lane);
					X.j[lane] = j;
				}
				__syncwarp();
				const uint32_t n = min(n_pair - wb, 32u);
				ref_fold(T, n, half ? sb : sa, lane);
				/* each pair's reaction on its receptor bead (0 - LJ(r) + LJ(plateau)
				 * [- Coulomb(r) + Coulomb(plateau)]), added pair by pair */
				if (lane < 3) {
					for (uint32_t k = 0; k < n; ++k) {
						const uint32_t f = T.flags[k];
						if (!(f & 1u)) continue;
						const float* t = reinterpret_cast<const float*>(T.t[k]);
						float v = fsub(0.f, t[lane]);
						v = fadd(v, t[4 + lane]);
						if (f & 2u) {
							v = fsub(v, t[8 + lane]);
							v = fadd(v, t[12 + lane]);
						}
						float* d = reinterpret_cast<float*>(rf + X.j[k]) + lane;
						*d = fadd(*d, v);
					}
				}
				__syncwarp();
			}
		}
		float4 a[2];
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			const int s = lane + 32 * h;
			a[h] = n_pair > 0 ? make_float4(T.acc[s][0], T.acc[s][1], T.acc[s][2], T.acc[s][3])
			                  : make_float4(0.f, 0.f, 0.f, 0.f);
		}
		__syncwarp();   /* accumulators read: the totals may overwrite them */
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			const int s = lane + 32 * h;
			if (i0 + s >= L.lig.n) continue;
			float4 v = pot[h];
			if (in_nl[h]) {
				v.x = fadd(v.x, a[h].x); v.y = fadd(v.y, a[h].y); v.z = fadd(v.z, a[h].z); v.w = fadd(v.w, a[h].w);
			}
			float* cw = W.cw + kCornerStride * s;
			cw[0] = v.x; cw[1] = v.y; cw[2] = v.z; cw[3] = v.w;
		}
		__syncwarp();
		const uint32_t nb = min((uint32_t)kBeadsPerRound, L.lig.n - i0);
		acc = ref_accumulate(W, nb, lane, acc);
		if (lane >= 16 && (uint32_t)(lane - 16) < Ml) {
			/* reduceModeForce with rotation (src/model/reduction_modes.h:29-57):
			 * -= (R^T f) . v */
			const int m = lane - 16;
			for (uint32_t s = 0; s < nb; ++s) {
				const float* f = W.cw + kCornerStride * s;
				float ox, oy, oz;
				rot_apply_t(R0.m, f[0], f[1], f[2], ox, oy, oz);
				const float* v = L.lig_modes + (size_t)(i0 + s) * L.lig_ms + 3 * m;
				acc = fsub(acc, fadd(fadd(fmul(ox, __ldg(v)), fmul(oy, __ldg(v + 1))), fmul(oz, __ldg(v + 2))));
			}
		}
		__syncwarp();
	}
	float c[13];
#pragma unroll
	for (int k = 0; k < 13; ++k) c[k] = __shfl_sync(GBA_FULL_MASK, acc, k);
	float gL[MM], gR[MM];
#pragma unroll
	for (int m = 0; m < MM; ++m) gL[m] = __shfl_sync(GBA_FULL_MASK, acc, 16 + m);
	/* reduceModeForce without rotation over the receptor forces, bead order */
	float g = 0.f;
	if ((uint32_t)lane < Mr) {
		for (uint32_t j = 0; j < L.rec.n; ++j) {
			const float4 f = rf[j];
			const float* v = L.rec_modes + (size_t)j * L.rec_ms + 3 * lane;
			g = fsub(g, fadd(fadd(fmul(f.x, __ldg(v)), fmul(f.y, __ldg(v + 1))), fmul(f.z, __ldg(v + 2))));
		}
	}
#pragma unroll
	for (int m = 0; m < MM; ++m) gR[m] = __shfl_sync(GBA_FULL_MASK, g, m);
	__syncwarp();   /* rf read: the next pose may overwrite it */
	float sFx = c[1], sFy = c[2], sFz = c[3];
	force_lim(sFx, sFy, sFz);
	float ang[3];
	torque_reduce(R0, c + 4, ang);
	/* correctModeForce (src/model/reduction_modes.h:101-115):
	 * delta + (float)((double)(4 k) * pow(delta, 4)) */
#pragma unroll
	for (int m = 0; m < MM; ++m) {
		if (m < (int)Mr)
			gR[m] = fadd(gR[m], (float)__dmul_rn((double)fmul(4.0f, L.rec.mode_force[m]), pow4_rn((double)gR[m])));
		if (m < (int)Ml)
			gL[m] = fadd(gL[m], (float)__dmul_rn((double)fmul(4.0f, L.lig.mode_force[m]), pow4_rn((double)gL[m])));
	}
	float v = 0.f;
	if (lane == 0) v = c[0];
	else if (lane == 1) v = sFx;
	else if (lane == 2) v = sFy;
	else if (lane == 3) v = sFz;
	else if (lane == 4) v = ang[0];
	else if (lane == 5) v = ang[1];
	else if (lane == 6) v = ang[2];
#pragma unroll
	for (int m = 0; m < MM; ++m) {
		if (lane == 7 + m) v = m < (int)Mr ? gR[m] : 0.f;
		if (lane == 17 + m) v = m < (int)Ml ? gL[m] : 0.f;
	}
	return v;
}

namespace {

/* Scoring kernels' blocks and how many of them the registers are bounded for:
 * latency bounds both passes, so warps count for more than registers until
 * the compiler spills, which it does at five modes and octets above six
 * receptor and five ligand blocks (20,000 poses, 1500/600 beads: 2,285 us at
 * 5 and 4, 2,107 at 6 and 5, 2,159 at 6 and 6; ten modes 644 at 5 and 4, 697 at
 * 6 and 5; native grids 187 against 268). */
constexpr int kModesThreads = 128;
template <int MM, int LAYOUT>
constexpr int kModesRecBlocks = MM <= 5 && LAYOUT == kOctets ? 6 : 5;
template <int MM, int LAYOUT>
constexpr int kModesLigBlocks = MM <= 5 && LAYOUT == kOctets ? 5 : 4;
constexpr int kModesMinThreads = 128;    /* minimizer kernel block */
constexpr int kModesRefThreads = 128;    /* reference-order scoring kernel block */

/* mode capacity compiled for a launch: 5 or GBA_MODES_MAX */
int mode_capacity(const ModesLaunch& L) {
	return (L.rec.n_modes <= 5 && L.lig.n_modes <= 5) ? 5 : GBA_MODES_MAX;
}

}  // namespace

extern __shared__ float4 modes_dyn_smem[];

/* Scoring in two kernels, so that each runs at the occupancy its own
 * registers allow: the receptor pass (most of the grid lookups) parks its
 * warp-summed receptor-mode gradients in the result record's modesRec slots;
 * the ligand pass reads them back, adds its own and writes the record. */
template <int MM, int LAYOUT>
__global__ void __launch_bounds__(kModesThreads, kModesRecBlocks<MM, LAYOUT>) modes_rec_kernel(const ModesLaunch L) {
	__shared__ RecStage stage[kModesThreads / 32];
	ModeStage<MM>* ms = reinterpret_cast<ModeStage<MM>*>(modes_dyn_smem);
	const int lane = threadIdx.x & 31;
	const int wib = threadIdx.x >> 5;
	const uint32_t Mr = L.rec.n_modes;
	for (size_t p = next_pose(L.next, lane); p < L.n; p = next_pose(L.next, lane)) {
		const float* d = reinterpret_cast<const float*>(L.dofs + p);
		const float dv = lane < 26 ? __ldg(d + lane) : 0.f;
		put_frame<MM>(L, dv, lane, ms[wib]);
		float gR[MM];
#pragma unroll
		for (int m = 0; m < MM; ++m) gR[m] = 0.f;
		modes_rec_pass<MM, LAYOUT, 4>(L, lane, stage[wib], ms[wib], gR);
		sum_rec_modes<MM>(Mr, gR);
		__syncwarp();
		float v = 0.f;
#pragma unroll
		for (int m = 0; m < MM; ++m) v = lane == m ? gR[m] : v;
		if ((uint32_t)lane < Mr) reinterpret_cast<float*>(L.out + p)[7 + lane] = v;
	}
}

template <int MM, int LAYOUT>
__global__ void __launch_bounds__(kModesThreads, kModesLigBlocks<MM, LAYOUT>) modes_lig_kernel(const ModesLaunch L) {
	__shared__ WarpStage stage[kModesThreads / 32];
	ModeStage<MM>* ms = reinterpret_cast<ModeStage<MM>*>(modes_dyn_smem);
	const int lane = threadIdx.x & 31;
	const int wib = threadIdx.x >> 5;
	const uint32_t Mr = L.rec.n_modes;
	for (size_t p = next_pose(L.next2, lane); p < L.n; p = next_pose(L.next2, lane)) {
		const float* d = reinterpret_cast<const float*>(L.dofs + p);
		const float dv = lane < 26 ? __ldg(d + lane) : 0.f;
		put_frame<MM>(L, dv, lane, ms[wib]);
		float gRr[MM], gRn[MM], gL[MM];
		const float* o = reinterpret_cast<const float*>(L.out + p);
#pragma unroll
		for (int m = 0; m < MM; ++m) {
			gRr[m] = m < (int)Mr ? o[7 + m] : 0.f;
			gRn[m] = 0.f;
			gL[m] = 0.f;
		}
		__syncwarp();
		PoseSums S;
		CoopSums C;
		modes_lig_pass<MM, LAYOUT>(L, lane, stage[wib], ms[wib], S, C, gL, gRn);
		const float v = modes_epilogue<MM>(L, ms[wib], S, C, gL, gRr, gRn, lane);
		__syncwarp();
		if (lane < 27) reinterpret_cast<float*>(L.out + p)[lane] = v;
	}
}

/* Few poses: a block of warps each (eval_pose_modes_team). */
template <int MM>
__global__ void __launch_bounds__(32 * kModesMaxTeam, 2) modes_team_kernel(const ModesLaunch L) {
	ModesTeamWarp<MM>* team = reinterpret_cast<ModesTeamWarp<MM>*>(modes_dyn_smem);
	const int lane = threadIdx.x & 31, t = threadIdx.x >> 5, G = blockDim.x >> 5;
	ModesTeamShared<MM>& sh = *reinterpret_cast<ModesTeamShared<MM>*>(team + G);
	for (size_t p = blockIdx.x; p < L.n; p += gridDim.x) {
		const float dv = lane < 26 ? __ldg(reinterpret_cast<const float*>(L.dofs + p) + lane) : 0.f;
		const float v = eval_pose_modes_team<MM>(L, dv, lane, t, G, team, sh);
		if (t == 0 && lane < 27) reinterpret_cast<float*>(L.out + p)[lane] = v;
	}
}

/* GBA_KOPT_REFERENCE_ORDER scoring: a warp takes whole poses
 * (eval_pose_modes_ref) with its own receptor array in L.ref_rf.  FEW, for
 * launches whose poses are all resident: latency bounds them, and the kernel
 * asks for the registers of five blocks per SM (ten modes: four); beyond, the
 * compiler's own 80 or 72 hold more warps.  Measured, few against many in us,
 * 700/300 beads, native grids: 5 modes 500 poses 296 372, 3,000 427 490, 20,000
 * poses on octets 2,798 2,683; 10 modes 500 poses 320 434, 50,000 on octets
 * 8,500 (with five blocks) 7,186. */
template <int MM, bool FEW>
constexpr int kRefBlocks = FEW ? (MM <= 5 ? 5 : 4) : 0;
template <int MM, bool FEW>
constexpr bool kRefWide = MM > 5 && !FEW;
template <int MM, bool FEW>
__global__ void __launch_bounds__(kModesRefThreads, kRefBlocks<MM, FEW>) modes_ref_kernel(const ModesLaunch L) {
	__shared__ WarpStage stage[kModesRefThreads / 32];
	__shared__ RefModesExtra extra[kModesRefThreads / 32];
	const int lane = threadIdx.x & 31;
	const int wib = threadIdx.x >> 5;
	float4* rf = L.ref_rf + (((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * L.rec.n;
	for (size_t p = next_pose(L.next, lane); p < L.n; p = next_pose(L.next, lane)) {
		const float* d = reinterpret_cast<const float*>(L.dofs + p);
		const float dv = lane < 26 ? __ldg(d + lane) : 0.f;
		const float v = eval_pose_modes_ref<MM, kRefWide<MM, FEW>>(L, dv, lane, stage[wib], extra[wib], rf);
		if (lane < 27) reinterpret_cast<float*>(L.out + p)[lane] = v;
	}
}

/* Persistent VA13 over (ang xyz, pos xyz, modesRec[0..Mr), modesLig[0..Ml)):
 * the minimizer of minimize.cu generalised to 6 + Mr + Ml DOF (minfor.f is
 * fixed at 6, src/apps/em/minfor.f:16,33). */
__device__ __forceinline__ unsigned long long modes_global_ns() {
	unsigned long long t;
	asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
	return t;
}

/* The record's float that element j of the machine's point belongs to is
 * found from either side: the element behind float k (or -1), and the result
 * entry behind gradient element j (1-based; neg: its sign turns). */
__device__ __forceinline__ int modes_point_element(int k, int Mr, int Ml) {
	if (k < 3) return 3 + k;
	if (k < 6) return k - 3;
	if (k < 6 + Mr) return k;
	if (k >= 16 && k < 16 + Ml) return k - 10 + Mr;
	return -1;
}
/* -(ang), -(pos), then the mode entries, which are gradients already
 * (reduceModeForce) */
__device__ __forceinline__ int modes_gradient_entry(int j, int Mr, int jn, bool& neg) {
	neg = false;
	const int k = j - 1;
	if (j < 1 || j > jn) return 0;
	if (k < 6) {
		neg = true;
		return k < 3 ? 4 + k : k - 2;
	}
	return k < 6 + Mr ? 7 + (k - 6) : 17 + (k - 6 - Mr);
}

/* LAYOUT: compiled for octets where both grids have them, which leaves the
 * native lookups' code out (6,000 poses, 700/300 beads, 20 evaluations: 17.6 ->
 * 16.9 ms).  Elsewhere three blocks per SM are asked for: with no
 * number named the compiler schedules the native lookups and the reference
 * order worse in as many registers (3,000 poses, 700/300 beads, 3 modes, 15
 * evaluations: 9.6 against 6.2 ms on native grids, 20.3 against 16.8 in the
 * * reference order; one block 6.9 and 18.7); on octets three lose (6,000 poses:
 * 11.3 against 12.8), and so they do in the reference order at ten modes. */
template <int MM, bool REF, int LAYOUT>
__global__ void __launch_bounds__(kModesMinThreads, LAYOUT == kOctets || (REF && MM > 5) ? 0 : 3)
		minimize_modes_kernel(const ModesMinLaunch M) {
	__shared__ FullStage stage[kModesMinThreads / 32];
	ModeStage<MM>* ms = reinterpret_cast<ModeStage<MM>*>(modes_dyn_smem);
	/* per warp, after the mode staging areas: its pose's VA13 state, which
	 * every lane of the warp steps (the warp form) */
	static_assert(sizeof(ModeStage<MM>) % 16 == 0, "VA13 states follow the staging areas");
	VA13<6 + 2 * MM>* vas = reinterpret_cast<VA13<6 + 2 * MM>*>(ms + kModesMinThreads / 32);
	const int lane = threadIdx.x & 31;
	const int wib = threadIdx.x >> 5;
	const ModesLaunch& L = M.m;
	const uint32_t Mr = L.rec.n_modes, Ml = L.lig.n_modes;
	const int jn = 6 + (int)Mr + (int)Ml;
	unsigned long long t_start = 0;
	if (lane == 0) t_start = modes_global_ns();
	t_start = __shfl_sync(GBA_FULL_MASK, t_start, 0);
	/* lane 0 reads the clock, the warp decides together */
	auto over_cap = [&]() {
		int over = 0;
		if (lane == 0) over = modes_global_ns() - t_start > kMinimizeHardCapNs;
		return __shfl_sync(GBA_FULL_MASK, over, 0) != 0;
	};
	for (;;) {
		unsigned long long slot = 0;
		if (lane == 0) slot = atomicAdd(M.counter, 1ull);
		slot = __shfl_sync(GBA_FULL_MASK, slot, 0);
		if (slot >= M.n) break;
		if (over_cap()) {
			if (lane == 0) atomicExch(M.status, GBA_ERR_TIMEOUT);
			break;
		}
		const size_t p = (size_t)slot;
		VA13<6 + 2 * MM>& va = vas[wib];
		/* lane k holds DOF float k (pos, ang, modesRec[10], modesLig[10]) */
		float dv = 0.f;
		if (lane == 0) {
			double x0[6 + 2 * MM];
			const float* s = reinterpret_cast<const float*>(M.start + p);
			for (int k = 0; k < 3; ++k) { x0[k] = s[3 + k]; x0[3 + k] = s[k]; }
			for (uint32_t m = 0; m < Mr; ++m) x0[6 + m] = s[6 + m];
			for (uint32_t m = 0; m < Ml; ++m) x0[6 + Mr + m] = s[16 + m];
			va.start(x0, jn, M.max_evals);
		}
		__syncwarp();
		float v = 0.f;
		int nev = 0;
		for (;;) {
			/* lane j converts element j of the point (one FP64 instruction for
			 * all); lane k takes float k of the record from its lane */
			const float pf = lane < jn ? (float)va.point()[lane] : 0.f;
			const int from = modes_point_element(lane, (int)Mr, (int)Ml);
			const float xf = __shfl_sync(GBA_FULL_MASK, pf, max(from, 0));
			dv = from >= 0 ? xf : 0.f;
			if (REF)
				v = eval_pose_modes_ref<MM, (MM > 5)>(L, dv, lane, stage[wib], *reinterpret_cast<RefModesExtra*>(&ms[wib]),
						L.ref_rf + (((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * L.rec.n);
			else
				v = eval_pose_modes<MM, LAYOUT>(L, dv, lane, stage[wib], ms[wib]);
			++nev;
			/* lane j takes gradient element j from the lane holding its entry
			 * of the result record */
			bool neg;
			const int src = modes_gradient_entry(lane, (int)Mr, jn, neg);
			const float gv = __shfl_sync(GBA_FULL_MASK, v, src);
			const double gl = (double)(neg ? -gv : gv);
			const float e = __shfl_sync(GBA_FULL_MASK, v, 0);
			va.provide_w((double)e, [&](int) { return gl; }, VaWarp{lane});
			/* lane 0's reading for all: no lane may see a state that lane 0,
			 * gone on to the next pose, has already restarted */
			if (__shfl_sync(GBA_FULL_MASK, (int)va.done(), 0)) break;
			if (nev > M.max_evals + 1) {
				if (lane == 0) atomicExch(M.status, GBA_ERR_DEVICE_CHECK);
				break;
			}
			if ((nev & 15) == 0 && over_cap()) {
				if (lane == 0) atomicExch(M.status, GBA_ERR_TIMEOUT);
				break;
			}
		}
		if (lane < 27) reinterpret_cast<float*>(M.out_result + p)[lane] = v;
		if (lane < 26) reinterpret_cast<float*>(M.out_state + p)[lane] = dv;
		if (lane == 0 && M.out_nevals) M.out_nevals[p] = nev;
	}
}

/* The same with a block of warps per pose (eval_pose_modes_team), warp 0
 * stepping its VA13: for jobs whose poses all get a block of their own. */
template <int MM>
__global__ void __launch_bounds__(32 * kModesMaxTeam, 2) minimize_modes_team_kernel(const ModesMinLaunch M) {
	ModesTeamWarp<MM>* team = reinterpret_cast<ModesTeamWarp<MM>*>(modes_dyn_smem);
	const int lane = threadIdx.x & 31, t = threadIdx.x >> 5, G = blockDim.x >> 5;
	ModesTeamShared<MM>& sh = *reinterpret_cast<ModesTeamShared<MM>*>(team + G);
	VA13<6 + 2 * MM>& va = *reinterpret_cast<VA13<6 + 2 * MM>*>(&sh + 1);
	const ModesLaunch& L = M.m;
	const int Mr = (int)L.rec.n_modes, Ml = (int)L.lig.n_modes, jn = 6 + Mr + Ml;
	const unsigned long long t_start = modes_global_ns();
	for (;;) {
		if (threadIdx.x == 0) {
			unsigned long long slot = atomicAdd(M.counter, 1ull);
			if (slot < M.n && modes_global_ns() - t_start > kMinimizeHardCapNs) {
				atomicExch(M.status, GBA_ERR_TIMEOUT);
				slot = ~0ull;
			}
			sh.pose = slot;
			if (slot < M.n) {
				double x0[6 + 2 * MM];
				const float* s = reinterpret_cast<const float*>(M.start + slot);
				for (int k = 0; k < 3; ++k) { x0[k] = s[3 + k]; x0[3 + k] = s[k]; }
				for (int m = 0; m < Mr; ++m) x0[6 + m] = s[6 + m];
				for (int m = 0; m < Ml; ++m) x0[6 + Mr + m] = s[16 + m];
				va.start(x0, jn, M.max_evals);
			}
		}
		__syncthreads();
		const size_t p = (size_t)sh.pose;
		if (p >= M.n) break;
		int nev = 0;
		for (;;) {
			if (t == 0) {
				const float pf = lane < jn ? (float)va.point()[lane] : 0.f;
				const int from = modes_point_element(lane, Mr, Ml);
				const float xf = __shfl_sync(GBA_FULL_MASK, pf, max(from, 0));
				if (lane < 26) sh.dof[lane] = from >= 0 ? xf : 0.f;
			}
			__syncthreads();
			const float dv = lane < 26 ? sh.dof[lane] : 0.f;
			const float v = eval_pose_modes_team<MM>(L, dv, lane, t, G, team, sh);
			++nev;
			if (t == 0) {
				bool neg;
				const int src = modes_gradient_entry(lane, Mr, jn, neg);
				const float gv = __shfl_sync(GBA_FULL_MASK, v, src);
				const double gl = (double)(neg ? -gv : gv);
				const float e = __shfl_sync(GBA_FULL_MASK, v, 0);
				va.provide_w((double)e, [&](int) { return gl; }, VaWarp{lane});
				if (lane == 0) {
					int stop = va.done();
					if (!stop && nev > M.max_evals + 1) {
						atomicExch(M.status, GBA_ERR_DEVICE_CHECK);
						stop = 1;
					}
					if (!stop && (nev & 15) == 0 && modes_global_ns() - t_start > kMinimizeHardCapNs) {
						atomicExch(M.status, GBA_ERR_TIMEOUT);
						stop = 1;
					}
					sh.stop = stop;
				}
				__syncwarp();
				if (sh.stop) {
					if (lane < 27) reinterpret_cast<float*>(M.out_result + p)[lane] = v;
					if (lane < 26) reinterpret_cast<float*>(M.out_state + p)[lane] = dv;
					if (lane == 0 && M.out_nevals) M.out_nevals[p] = nev;
				}
			}
			__syncthreads();
			if (sh.stop) break;
		}
	}
}

namespace {

template <int MM>
size_t mode_stage_bytes(int threads) {
	return (size_t)(threads / 32) * sizeof(ModeStage<MM>);
}

/* Resident blocks per SM (0: the kernel does not fit), with the opt-in to
 * dynamic shared memory beyond the 48 KB default; queried once per device,
 * kernel, block size and shared memory (the queries cost a small call more
 * host time than its launches).  The opt-in only grows: launches of other
 * sizes may be in flight. */
template <class K>
int blocks_that_fit(K kernel, int threads, size_t dyn) {
	static std::mutex mu;
	static std::map<std::array<size_t, 4>, int> known;
	static std::map<std::pair<size_t, size_t>, size_t> opted;
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess) return 0;
	std::lock_guard<std::mutex> g(mu);
	const std::array<size_t, 4> key{(size_t)dev, (size_t)kernel, (size_t)threads, dyn};
	const auto it = known.find(key);
	if (it != known.end()) return it->second;
	size_t& most = opted[{(size_t)dev, (size_t)kernel}];
	int nb = 0;
	if (dyn <= most || cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn) == cudaSuccess) {
		most = std::max(most, dyn);
		if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, dyn) != cudaSuccess) nb = 0;
	}
	cudaGetLastError();      /* a size that does not fit is an answer */
	if (known.size() >= 256) known.clear();
	return known[key] = nb;
}

template <class K>
int resident_blocks(K kernel, int threads, size_t dyn) {
	return std::max(1, blocks_that_fit(kernel, threads, dyn));
}

/* shared memory of a team of G warps; the minimizer's VA13 state follows */
template <int MM>
size_t team_bytes(int G, bool minimize) {
	static_assert(sizeof(ModesTeamWarp<MM>) % 16 == 0 && sizeof(ModesTeamShared<MM>) % 8 == 0, "laid out in a row");
	return (size_t)G * sizeof(ModesTeamWarp<MM>) + sizeof(ModesTeamShared<MM>) +
			(minimize ? sizeof(VA13<6 + 2 * MM>) : 0);
}

/* Warps per pose for n poses: the largest team with which every pose has a
 * resident block of its own, or 0 (a pose then takes a warp by itself).  The
 * terms' records hold 24 bits of a receptor bead's index and come from
 * cooperative lookups.  Measured, a warp per pose against teams: scoring
 * 777/333 beads, 7 modes, 100 poses 210 -> 73 us; 1500/600, 5 modes, 500 poses
 * 317 -> 157, 1,000 poses 307 -> 205, and 1,200 poses, not all resident in
 * teams of two, 308 against 370; minimizing 700/300, 5 modes, 50 evaluations
 * 100 poses 16.6 -> 6.4 ms, 500 12.7 -> 7.0, 800 13.4 -> 10.2. */
template <int MM, class K>
int team_size(K kernel, bool minimize, const ModesLaunch& L, size_t n, int num_sms) {
	if (!L.grid_rec.coop_lookup || !L.grid_lig.coop_lookup || L.rec.n > (1u << 24)) return 0;
	const uint32_t rounds = std::max((L.rec.n + 63) / 64, (L.lig.n + 63) / 64);
	if (n > (size_t)num_sms * 8) return 0;       /* 16 warps of 128 registers, two at least to a team */
	for (int G = (int)std::min<uint32_t>(kModesMaxTeam, rounds); G >= 2; --G)
		if (n <= (size_t)num_sms * blocks_that_fit(kernel, 32 * G, team_bytes<MM>(G, minimize))) return G;
	return 0;
}

template <int MM>
cudaError_t launch_modes_mm(const ModesLaunch& L, int num_sms, cudaStream_t s) {
	const int team = team_size<MM>(modes_team_kernel<MM>, false, L, L.n, num_sms);
	if (team > 0) {
		modes_team_kernel<MM><<<(unsigned)L.n, 32 * team, team_bytes<MM>(team, false), s>>>(L);
		return cudaGetLastError();
	}
	/* each pass by its own grid's layout */
	const size_t dyn = mode_stage_bytes<MM>(kModesThreads), warps = kModesThreads / 32;
	auto blocks = [&](auto kernel) {
		return (unsigned)std::max<size_t>(1, std::min<size_t>((L.n + warps - 1) / warps,
				(size_t)num_sms * resident_blocks(kernel, kModesThreads, dyn)));
	};
	if (L.grid_lig.coop_lookup)
		modes_rec_kernel<MM, kOctets><<<blocks(modes_rec_kernel<MM, kOctets>), kModesThreads, dyn, s>>>(L);
	else
		modes_rec_kernel<MM, kNative><<<blocks(modes_rec_kernel<MM, kNative>), kModesThreads, dyn, s>>>(L);
	cudaError_t e = cudaGetLastError();
	if (e != cudaSuccess) return e;
	if (L.grid_rec.coop_lookup)
		modes_lig_kernel<MM, kOctets><<<blocks(modes_lig_kernel<MM, kOctets>), kModesThreads, dyn, s>>>(L);
	else
		modes_lig_kernel<MM, kNative><<<blocks(modes_lig_kernel<MM, kNative>), kModesThreads, dyn, s>>>(L);
	return cudaGetLastError();
}

/* The reference-order scoring kernel for L's poses, and its blocks. */
struct RefLaunch {
	void (*kernel)(ModesLaunch);
	size_t blocks;
};
template <int MM>
RefLaunch ref_launch_mm(const ModesLaunch& L, int num_sms) {
	constexpr size_t warps = kModesRefThreads / 32;
	const size_t want = std::max<size_t>(1, (L.n + warps - 1) / warps);
	const size_t few = (size_t)num_sms * resident_blocks(modes_ref_kernel<MM, true>, kModesRefThreads, 0);
	if (want <= few) return {modes_ref_kernel<MM, true>, want};
	return {modes_ref_kernel<MM, false>, std::min<size_t>(want,
			(size_t)num_sms * resident_blocks(modes_ref_kernel<MM, false>, kModesRefThreads, 0))};
}

template <int MM>
cudaError_t launch_ref_mm(const ModesLaunch& L, int num_sms, cudaStream_t s) {
	const RefLaunch r = ref_launch_mm<MM>(L, num_sms);
	r.kernel<<<(unsigned)r.blocks, kModesRefThreads, 0, s>>>(L);
	return cudaGetLastError();
}

/* the minimizer's: staging areas and VA13 states, one each per warp */
template <int MM>
size_t min_modes_bytes(int threads) {
	return (size_t)(threads / 32) * (sizeof(ModeStage<MM>) + sizeof(VA13<6 + 2 * MM>));
}

template <int MM, bool REF>
cudaError_t launch_min_mm(const ModesMinLaunch& M, int blocks, int threads, cudaStream_t s) {
	if (!REF) {
		const int team = team_size<MM>(minimize_modes_team_kernel<MM>, true, M.m, M.n, M.num_sms);
		if (team > 0) {
			const size_t dyn = team_bytes<MM>(team, true);
			minimize_modes_team_kernel<MM><<<(unsigned)M.n, 32 * team, dyn, s>>>(M);
			return cudaGetLastError();
		}
	}
	const size_t dyn = min_modes_bytes<MM>(threads);
	/* resident_blocks: the opt-in to the shared memory */
	if (!REF && M.m.grid_rec.coop_lookup && M.m.grid_lig.coop_lookup) {
		resident_blocks(minimize_modes_kernel<MM, false, kOctets>, threads, dyn);
		minimize_modes_kernel<MM, false, kOctets><<<blocks, threads, dyn, s>>>(M);
	} else {
		resident_blocks(minimize_modes_kernel<MM, REF, kAnyLayout>, threads, dyn);
		minimize_modes_kernel<MM, REF, kAnyLayout><<<blocks, threads, dyn, s>>>(M);
	}
	return cudaGetLastError();
}

template <int MM, bool REF>
int min_bps_mm(int threads, const ModesLaunch& L) {
	const size_t dyn = min_modes_bytes<MM>(threads);
	return !REF && L.grid_rec.coop_lookup && L.grid_lig.coop_lookup
			? resident_blocks(minimize_modes_kernel<MM, false, kOctets>, threads, dyn)
			: resident_blocks(minimize_modes_kernel<MM, REF, kAnyLayout>, threads, dyn);
}

}  // namespace

cudaError_t launch_modes_energy(const ModesLaunch& L, int num_sms, cudaStream_t s) {
	if (L.ref_order) {
		if (!L.ref_rf) return cudaErrorInvalidValue;
		return mode_capacity(L) == 5 ? launch_ref_mm<5>(L, num_sms, s) : launch_ref_mm<GBA_MODES_MAX>(L, num_sms, s);
	}
	return mode_capacity(L) == 5 ? launch_modes_mm<5>(L, num_sms, s)
	                             : launch_modes_mm<GBA_MODES_MAX>(L, num_sms, s);
}

size_t modes_ref_warps(const ModesLaunch& L, int num_sms) {
	const size_t blocks = mode_capacity(L) == 5 ? ref_launch_mm<5>(L, num_sms).blocks
	                                            : ref_launch_mm<GBA_MODES_MAX>(L, num_sms).blocks;
	return blocks * (kModesRefThreads / 32);
}

cudaError_t launch_minimize_modes(const ModesMinLaunch& M, int blocks, int threads, cudaStream_t s) {
	if (threads != kModesMinThreads || (M.m.ref_order && !M.m.ref_rf)) return cudaErrorInvalidValue;
	if (M.m.ref_order)
		return mode_capacity(M.m) == 5 ? launch_min_mm<5, true>(M, blocks, threads, s)
		                               : launch_min_mm<GBA_MODES_MAX, true>(M, blocks, threads, s);
	return mode_capacity(M.m) == 5 ? launch_min_mm<5, false>(M, blocks, threads, s)
	                               : launch_min_mm<GBA_MODES_MAX, false>(M, blocks, threads, s);
}

int minimize_modes_blocks_per_sm(int threads, const ModesLaunch& L) {
	if (L.ref_order)
		return mode_capacity(L) == 5 ? min_bps_mm<5, true>(threads, L) : min_bps_mm<GBA_MODES_MAX, true>(threads, L);
	return mode_capacity(L) == 5 ? min_bps_mm<5, false>(threads, L) : min_bps_mm<GBA_MODES_MAX, false>(threads, L);
}

}  // namespace gba
