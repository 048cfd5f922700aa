/*
 * adjoint.cu -- pairwise (grid-free) docking energy and its adjoint.
 *
 * The pairwise path scores a pose with the exact ATTRACT pair terms over
 * every receptor-ligand pair closer than `cutoff`:
 *   8-6 Lennard-Jones of LJPotForce (src/model/forcefield.h:30-83) with
 *   rc = eps r0^8, ac = eps r0^6, emin = -27 ac^4 / (256 rc^3),
 *   rmin2 = 4 rc / (3 ac) as readParamTableFromFile derives them
 *   (src/fileIO/readFile.cpp:484-497), and the distance-dependent Coulomb
 *   term of ChargePotForce (src/model/forcefield.h:87-146),
 * with per-bead charges and per-type-pair (r0, eps) as free parameters.
 * Candidate receptor beads come from the receptor's neighbour-list grid
 * (voxel lists cover every bead within cutoff of a ligand bead).  Like the
 * rigid kernel, a warp takes one pose and walks the flattened
 * (bead, neighbour) pairs of 64 staged ligand beads at a time.
 *
 * The backward kernel recomputes the transformed coordinates and pair terms
 * (nothing is stored by the forward) and produces, scaled by the upstream
 * gradient of each pose's energy:
 *   dE/dDOF   (pos xyz, ang xyz): -(force sum), -(TorqueMat . torque), the
 *             reference's gradient convention (src/apps/em/meta.h:114-121)
 *   dE/dq     per ligand and per receptor bead
 *   dE/dr0, dE/deps per type pair [rec type - 1][lig type - 1]
 * Parameter gradients accumulate in the block's shared memory as unevaluated
 * sums of two floats (TwoFloat: 48 bits; a block adds some hundred FP32 terms
 * to a cell), are written out per block in double and added up by a last
 * kernel.
 */
#include <cub/cub.cuh>

#include "gba_context.h"
#include "pairwise_limits.h"
#include "rigid_pose.cuh"

namespace gba {

struct PairwiseLaunch {
	DevProtein rec, lig;
	DevNL nl;
	uint32_t T;
	const float* r0;       /* T*T */
	const float* eps;      /* T*T */
	const int32_t* ipon;   /* T*T */
	const float* q_lig;
	const float* q_rec;
	int dielec;
	float ffelec;
	float cut2;
	const gba_dof6d* dofs;
	size_t n;
	float* E;              /* forward output (n) */
	const float* gE;       /* backward input (n) */
	float* g_dofs;         /* n*6 (pos, ang) */
	double* g_qlig;        /* lig.n */
	double* g_qrec;        /* rec.n */
	double* g_r0;          /* T*T */
	double* g_eps;         /* T*T */
	float4* tab;           /* 2*T*T: per type pair the constants of the 8-6 term (pairwise_setup_kernel) */
	float4* rq;            /* rec.n: receptor x, y, z and this call's charge */
	const uint32_t* tlist; /* the neighbour list with receptor types in bits 24..31, or nullptr */
	unsigned long long* next;   /* pose (or round) counter, zero at launch (next_pose) */
	uint32_t* order;            /* visiting order (nearest ligands first), or nullptr */
	RoundSplit split;           /* pose records; totals and done only when split */
	int by_round;               /* units are 64-bead rounds, else poses */
	uint32_t copies;            /* backward: of the type pairs' cells in a block, 1 or 2 */
	double* part;               /* backward: per block, then once for what no TwoFloat holds, the sums of
	                               every cell (PairCells) */
};

/* The cells of the parameter gradients: per type pair the sums of
 * w d(energy)/d(rc) and w d(energy)/d(ac), side by side, then the ligand and receptor charges'.
 * Type pairs are stored ligand type major: neighbouring lanes hold pairs of
 * one ligand bead, whose cells then lie in one row, in banks of their own.
 * Receptor type major, as the caller's arrays are, put the 32 types of a row
 * into one bank, and the adds to these cells took 730 us of a 1,190 us
 * backward pass (10,000 poses, 2000/700 beads). */
struct PairCells {
	uint32_t T2, lig, rec;
	__host__ __device__ uint32_t qlig() const { return 2 * T2; }
	__host__ __device__ uint32_t qrec() const { return 2 * T2 + lig; }
	__host__ __device__ uint32_t count() const { return 2 * T2 + lig + rec; }
};

namespace {

/* An unevaluated sum hi + lo, |lo| <= ulp(hi)/2: about 48 bits.  The additions
 * are Knuth's two-sum (no ordering of the operands needed) and a
 * renormalisation, ten FP32 operations, where a double costs a conversion and
 * an addition on the FP64 pipe, 16 cycles each for a warp and SM. */
struct TwoFloat {
	float hi, lo;
};
__device__ __forceinline__ TwoFloat two_add(TwoFloat a, float v) {
	const float s = __fadd_rn(a.hi, v);
	const float b = __fsub_rn(s, a.hi);
	const float err = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, b)), __fsub_rn(v, b));
	const float l = __fadd_rn(a.lo, err);
	const float hi = __fadd_rn(s, l);
	return TwoFloat{hi, __fsub_rn(l, __fsub_rn(hi, s))};
}

/* Terms enter the cells times 2^40 (exactly): a term is a pair's derivative
 * times the pose's weight, derivatives go down to 1e-8, and with weights of
 * 1e-30 the terms themselves would leave FP32's normal range. */
constexpr float kCellScale = 0x1p40f;
constexpr double kCellUnscale = 0x1p-40;

/* Adds w x to a shared cell; what would overflow a TwoFloat (or is no number)
 * goes, unscaled, to the launch's double cell instead.  There is no shared
 * FP64 reduction: atomicAdd loops over a compare-and-swap too.  26 M adds to
 * each of two random cells of 1,024: 0.28 ms as doubles, 0.14 ms as
 * TwoFloats; global FP64 reductions 0.34-1.3 ms.  In the kernel lanes meet in
 * cells (a ligand bead's 32 type pairs), and the loops repeat: cell_add2
 * halves them. */
__device__ __forceinline__ void cell_add(unsigned long long* cell, float w, float x, double* beyond) {
	constexpr float kBig = 1e37f;
	const float v = w * kCellScale * x;
	if (v == 0.f) return;
	if (!(fabsf(v) < kBig)) {
		atomicAdd(beyond, (double)(w * x));
		return;
	}
	unsigned long long old = *(volatile unsigned long long*)cell, was;
	do {
		was = old;
		const TwoFloat a{__uint_as_float((uint32_t)was), __uint_as_float((uint32_t)(was >> 32))};
		if (!(fabsf(a.hi) < kBig)) {
			atomicAdd(beyond, (double)(w * x));
			return;
		}
		const TwoFloat t = two_add(a, v);
		old = atomicCAS(cell, was, (unsigned long long)__float_as_uint(t.lo) << 32 | __float_as_uint(t.hi));
	} while (old != was);
}

/* The same for a type pair's two sums, neighbours in shared memory, in one
 * 128-bit compare-and-swap. */
struct __align__(16) TwoFloat2 {
	TwoFloat a, b;
};
__device__ __forceinline__ void cell_add2(TwoFloat2* cell, float w, float xa, float xb, double* beyond_a, double* beyond_b) {
	constexpr float kBig = 1e37f;
	const float va = w * kCellScale * xa, vb = w * kCellScale * xb;
	if (va == 0.f && vb == 0.f) return;
	if (!(fabsf(va) < kBig && fabsf(vb) < kBig)) {
		atomicAdd(beyond_a, (double)(w * xa));
		atomicAdd(beyond_b, (double)(w * xb));
		return;
	}
	TwoFloat2 old = *cell, was;
	bool again;
	do {
		was = old;
		if (!(fabsf(was.a.hi) < kBig && fabsf(was.b.hi) < kBig)) {
			atomicAdd(beyond_a, (double)(w * xa));
			atomicAdd(beyond_b, (double)(w * xb));
			return;
		}
		old = atomicCAS(cell, was, TwoFloat2{two_add(was.a, va), two_add(was.b, vb)});
		again = __float_as_uint(old.a.hi) != __float_as_uint(was.a.hi) || __float_as_uint(old.a.lo) != __float_as_uint(was.a.lo) ||
				__float_as_uint(old.b.hi) != __float_as_uint(was.b.hi) || __float_as_uint(old.b.lo) != __float_as_uint(was.b.lo);
	} while (again);
}

/* ---- before the pair kernel ------------------------------------------------- */

/* Poses nearest the receptor's centre first: their ligands meet the most
 * pairs, so the launch ends with cheap poses.  A counting sort on the top bits
 * of |t|^2 (non-negative floats order like their bit patterns, NaN last; 3 %
 * bins), one block. */
constexpr int kSetupThreads = 512;
constexpr int kNearBins = 8192, kNearShift = 18;
constexpr size_t kNearFirstMinPoses = 2048;
/* Beyond these the radix sort (near_first_order).  Forward, the last size of
 * one and the first of the other: 300/60 beads 227 against 242 us, 500/200 387
 * against 403, 2000/700 1,073 against 1,086; the one block's time grows with
 * the poses, the sort's 30 us hardly. */
constexpr size_t kNearOneBlock = 65536;

__device__ __forceinline__ uint32_t near_key(const gba_dof6d* __restrict__ dofs, size_t p) {
	const float* d = reinterpret_cast<const float*>(dofs + p);
	const float x = __ldg(d), y = __ldg(d + 1), z = __ldg(d + 2);
	return __float_as_uint(x * x + y * y + z * z) & 0x7fffffffu;
}

__device__ void near_first_block(const PairwiseLaunch& L, uint32_t* bin) {
	__shared__ uint32_t warp_tot[kSetupThreads / 32];
	constexpr int per = kNearBins / kSetupThreads;
	const int t = threadIdx.x, lane = t & 31, w = t >> 5;
	for (int k = t; k < kNearBins; k += kSetupThreads) bin[k] = 0;
	__syncthreads();
	for (size_t p = t; p < L.n; p += kSetupThreads) atomicAdd(&bin[near_key(L.dofs, p) >> kNearShift], 1u);
	__syncthreads();
	uint32_t v[per], sum = 0;
#pragma unroll
	for (int k = 0; k < per; ++k) {
		v[k] = bin[t * per + k];
		sum += v[k];
	}
	const uint32_t incl = warp_incl_scan(sum, lane);
	if (lane == 31) warp_tot[w] = incl;
	__syncthreads();
	uint32_t run = incl - sum;
	for (int k = 0; k < w; ++k) run += warp_tot[k];
#pragma unroll
	for (int k = 0; k < per; ++k) {
		bin[t * per + k] = run;
		run += v[k];
	}
	__syncthreads();
	for (size_t p = t; p < L.n; p += kSetupThreads)
		L.order[atomicAdd(&bin[near_key(L.dofs, p) >> kNearShift], 1u)] = (uint32_t)p;
}

/* One launch for everything the pair kernel reads, by block: block 0 the
 * visiting order and the counter; then the pose records (and the counts of
 * finished rounds); then per type pair the constants of the 8-6 term,
 *   {rc, ac, ipon, 0}, {emin, rmin2, -3 emin / rc, 4 emin / ac}
 * with rc = eps r0^8, ac = eps r0^6, emin = -27 ac^4 / (256 rc^3),
 * rmin2 = 4 rc / (3 ac) as readParamTableFromFile derives them
 * (src/fileIO/readFile.cpp:484-497), ligand type major, the receptor's positions with this
 * call's charges, and zeros for the double cells.  Six launches before (two of
 * them a 30 us radix sort). */
__global__ void __launch_bounds__(kSetupThreads) pairwise_setup_kernel(const PairwiseLaunch L, const uint32_t pose_blocks,
		const int sort, const uint32_t cells) {
	__shared__ uint32_t bin[kNearBins];
	cudaTriggerProgrammaticLaunchCompletion();      /* the pair kernel's blocks may come and wait */
	if (blockIdx.x == 0) {
		if (threadIdx.x == 0) *L.next = 0;
		if (sort) near_first_block(L, bin);
		return;
	}
	if (blockIdx.x <= pose_blocks) {
		const size_t t = (size_t)(blockIdx.x - 1) * kSetupThreads + threadIdx.x;
		const size_t p = t >> 2;
		const bool in = p < L.n;
		if (L.by_round && in && (t & 3) == 0) L.split.done[p] = 0;
		write_pose_record(reinterpret_cast<const float*>(L.dofs + (in ? p : 0)), DevTrig{nullptr, 0u, 0u}, in,
				threadIdx.x & 31, L.split.pose + kPoseRecord * p);
		return;
	}
	const uint32_t stride = (gridDim.x - 1 - pose_blocks) * kSetupThreads;
	const uint32_t first = (blockIdx.x - 1 - pose_blocks) * kSetupThreads + threadIdx.x;
	const size_t T2 = (size_t)L.T * L.T;
	for (size_t k = first; k < T2; k += stride) {
		const uint32_t from = L.T * ((uint32_t)k % L.T) + (uint32_t)k / L.T;      /* the caller's: receptor type major */
		const float r0 = L.r0[from], eps = L.eps[from];
		const float r0_2 = r0 * r0, r0_6 = r0_2 * r0_2 * r0_2, r0_8 = r0_6 * r0_2;
		const float rc = eps * r0_8, ac = eps * r0_6;
		const bool ok = ac > 0.f && rc > 0.f;
		const float emin = ok ? -27.f * (ac * ac) * (ac * ac) / (256.f * rc * rc * rc) : 0.f;
		L.tab[k] = make_float4(rc, ac, (float)L.ipon[from], 0.f);
		L.tab[T2 + k] = make_float4(emin, ok ? 4.f * rc / (3.f * ac) : 0.f, ok ? -3.f * emin / rc : 0.f,
				ok ? 4.f * emin / ac : 0.f);
	}
	for (size_t j = first; j < L.rec.n; j += stride) {
		const float4 r = L.rec.xyzq[j];
		L.rq[j] = make_float4(r.x, r.y, r.z, L.q_rec[j]);
	}
	for (uint32_t k = first; k < cells; k += stride) L.part[k] = 0.0;
}

/* The same for more poses than one block sorts quickly: a radix sort of the
 * bits of |t|^2. */
__global__ void near_first_keys_kernel(const gba_dof6d* __restrict__ dofs, uint32_t n, uint32_t* __restrict__ keys,
		uint32_t* __restrict__ idx) {
	const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= n) return;
	const float* d = reinterpret_cast<const float*>(dofs + p);
	const float x = __ldg(d), y = __ldg(d + 1), z = __ldg(d + 2);
	keys[p] = __float_as_uint(x * x + y * y + z * z);
	idx[p] = p;
}

/* Poses ordered nearest first (sorted on the top 16 bits of the key: the
 * exponent and 7 mantissa bits of |t|^2, about 0.4 % bins), scratch from S. */
uint32_t* near_first_order(const gba_dof6d* dofs, size_t n, StreamScratch& S, cudaStream_t s) {
	cub::DoubleBuffer<uint32_t> kb(nullptr, nullptr), ib(nullptr, nullptr);
	size_t tmp = 0;
	check_cuda(cub::DeviceRadixSort::SortPairs(nullptr, tmp, kb, ib, (int)n, 16, 32, s), "pairwise order: size");
	const size_t a = (n * sizeof(uint32_t) + 255) & ~(size_t)255;
	char* base = (char*)S.get(4 * a + tmp, s);
	uint32_t* k0 = (uint32_t*)base;
	uint32_t* k1 = (uint32_t*)(base + a);
	uint32_t* i0 = (uint32_t*)(base + 2 * a);
	uint32_t* i1 = (uint32_t*)(base + 3 * a);
	near_first_keys_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(dofs, (uint32_t)n, k0, i0);
	check_cuda(cudaGetLastError(), "pairwise order: keys");
	kb = cub::DoubleBuffer<uint32_t>(k0, k1);
	ib = cub::DoubleBuffer<uint32_t>(i0, i1);
	check_cuda(cub::DeviceRadixSort::SortPairs(base + 4 * a, tmp, kb, ib, (int)n, 16, 32, s),
			"pairwise order: sort");
	return ib.Current();
}

/* Per-warp staging of the pairwise kernels: one round of 64 ligand beads. */
struct PairStage {
	float4 pq[kBeadsPerRound];       /* transformed x, y, z; charge */
	float4 ut[kBeadsPerRound];       /* unrotated x, y, z (torque lever); type (bits) */
	uint32_t lbase[kBeadsPerRound];  /* list start - first flattened pair of the slot */
	float gq[kBeadsPerRound];        /* backward: dE/dq of the slot's bead over this round */
	uint8_t own[64];                 /* PairWindow: slot of the bead starting at window position b */
	float pose[kPoseRecord];         /* as WarpStage::pose */
	float tot[16];                   /* the sum of the round totals so far */
	unsigned long long slot;         /* the pose's index */
	unsigned long long pad;
};
static_assert(13 * kTotalRow * sizeof(float) <= 2 * kBeadsPerRound * sizeof(float4), "sums_total overlays the bead records");
static_assert(sizeof(PairStage) % 16 == 0 && offsetof(PairStage, pose) % 16 == 0, "records are read as words");

/* Sum of v over the run of lanes with the same owner, on the run's first
 * lane; last: the run's last lane.  Every lane of the warp calls it. */
__device__ __forceinline__ float run_sum(float v, int lane, int last) {
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const float t = __shfl_down_sync(GBA_FULL_MASK, v, o);
		if (lane + o <= last) v += t;
	}
	return v;
}

/* A round of a pose: 64 ligand beads from i0, the flattened (bead, neighbour)
 * pairs two per lane.  Forward: energies into S.E.  Backward: forces and
 * torques into S, the parameters' sums into the cells. */
template <bool BACKWARD>
__device__ __forceinline__ void pairwise_round(const PairwiseLaunch& L, const PairCells& cells, uint32_t i0, int lane,
		float w, PairStage& W, unsigned long long* cell, PoseSums& S) {
	const bool cdiel = L.dielec == GBA_DIELEC_CONSTANT;
	/* odd lanes add to the second copy of the type pairs' cells, where there is one */
	const uint32_t pair_cells = BACKWARD && L.copies > 1 && (lane & 1) ? (cells.count() + 1) & ~1u : 0;
	uint32_t nln[2];
	{
		float tx, ty, tz;
		const PoseRot R = get_pose(W, tx, ty, tz);
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			const int s = lane + 32 * h;
			const uint32_t i = i0 + s;
			nln[h] = 0;
			if (i < L.lig.n) {
				const float4 b = __ldg(&L.lig.xyzq[i]);
				const uint32_t tl = __ldg(&L.lig.tm[i]) & 0xffffu;
				if (tl != 0) {
					float px, py, pz;
					rot_apply(R.m, b.x, b.y, b.z, px, py, pz);
					px = fadd(px, tx); py = fadd(py, ty); pz = fadd(pz, tz);
					W.pq[s] = make_float4(px, py, pz, __ldg(&L.q_lig[i]));
					W.ut[s] = make_float4(b.x, b.y, b.z, __uint_as_float(tl));
					if (BACKWARD) W.gq[s] = 0.f;
					bool in_nl;
					nln[h] = stage_nl(L.nl, px, py, pz, s, W, in_nl);
				}
			}
		}
	}
	uint32_t start[2];
	const uint32_t n_pair = queue_pairs(W, nln, lane, start);
	__syncwarp();
	/* the next window's list entries are on their way while this one is computed */
	const uint32_t* lst = L.tlist ? L.tlist : L.nl.list;
	PairWindow win;
	uint32_t so[2] = {0, 0}, en[2] = {0, 0};
	if (n_pair > 0) {
		win.owners(W, 0, start, nln, lane, so[0], so[1]);
#pragma unroll
		for (int h = 0; h < 2; ++h)
			if ((uint32_t)lane + 32 * h < n_pair) en[h] = __ldg(&lst[W.lbase[so[h]] + lane + 32 * h]);
	}
	for (uint32_t w0 = 0; w0 < n_pair; w0 += 64) {
		const uint32_t sc[2] = {so[0], so[1]}, ec[2] = {en[0], en[1]};
		if (w0 + 64 < n_pair) {
			win.owners(W, w0 + 64, start, nln, lane, so[0], so[1]);
#pragma unroll
			for (int h = 0; h < 2; ++h)
				if (w0 + 64 + 32 * h + lane < n_pair) en[h] = __ldg(&lst[W.lbase[so[h]] + w0 + 64 + 32 * h + lane]);
		}
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			const uint32_t q0 = w0 + 32 * h;
			if (q0 >= n_pair) break;
			const uint32_t s = sc[h];
			float gqv = 0.f;      /* this pair's part of dE/dq of the ligand bead */
			bool in = q0 + lane < n_pair;
			uint32_t j = 0, tr = 0;
			if (in) {
				j = L.tlist ? ec[h] & 0xffffffu : ec[h];
				tr = L.tlist ? ec[h] >> 24 : __ldg(&L.rec.tm[j]) & 0xffffu;
				in = tr != 0;
			}
			if (in) {
				const float4 r = __ldg(&L.rq[j]);
				const float4 b = W.pq[s];
				const float4 u = W.ut[s];
				const float dx = b.x - r.x, dy = b.y - r.y, dz = b.z - r.z;
				const float r2 = dx * dx + dy * dy + dz * dz;
				if (r2 < L.cut2) {
					const uint32_t tp = L.T * (__float_as_uint(u.w) - 1) + (tr - 1);
					const float4 c = __ldg(&L.tab[tp]);           /* rc, ac, ipon */
					const float ir2 = __frcp_rn(r2);              /* = 1.0f / r2, correctly rounded */
					const float ir6 = ir2 * ir2 * ir2, ir8 = ir6 * ir2;
					const float vlj = c.x * ir8 - c.y * ir6;
					float e = vlj, fb = 6.f * vlj + 2.f * c.x * ir8;      /* force factor: f = fb d / r^2 */
					float drc = ir8, dac = -ir6;
					if (c.z != 1.f) {
						const float4 m = __ldg(&L.tab[(size_t)L.T * L.T + tp]);   /* emin, rmin2, -3 emin / rc, 4 emin / ac */
						if (r2 < m.y) {
							e = vlj + (c.z - 1.f) * m.x;
							drc = ir8 + (c.z - 1.f) * m.z;
							dac = -ir6 + (c.z - 1.f) * m.w;
						} else {
							e = c.z * vlj;
							fb *= c.z;
							drc *= c.z;
							dac *= c.z;
						}
					}
					/* Coulomb, no |q q| switch: smooth in the charges */
					const float qi = b.w, qj = r.w;
					float dd, fcf;
					if (cdiel) {
						const float ir = sqrtf(ir2);
						dd = ir - 0.02f;
						fcf = dd > 0.f ? ir : 0.f;      /* f = ffelec qq (1/r) d / r^2 */
					} else {
						dd = ir2 - 4.0e-4f;
						fcf = dd > 0.f ? 2.f * ir2 : 0.f;  /* f = ffelec qq 2/r^2 d / r^2 */
					}
					dd = fmaxf(dd, 0.f);
					const float qq = L.ffelec * qi * qj;
					if (!BACKWARD) {
						S.E += e + qq * dd;
					} else {
						const float ff = (fb + qq * fcf) * ir2;
						const float fx = ff * dx, fy = ff * dy, fz = ff * dz;
						S.Fx += fx; S.Fy += fy; S.Fz += fz;
						S.T[0] += u.x * fx; S.T[1] += u.y * fx; S.T[2] += u.z * fx;
						S.T[3] += u.x * fy; S.T[4] += u.y * fy; S.T[5] += u.z * fy;
						S.T[6] += u.x * fz; S.T[7] += u.y * fz; S.T[8] += u.z * fz;
						gqv = L.ffelec * qj * dd;
						cell_add(cell + cells.qrec() + j, w, L.ffelec * qi * dd, L.part + cells.qrec() + j);
						cell_add2(reinterpret_cast<TwoFloat2*>(cell + pair_cells) + tp, w, drc, dac, L.part + 2 * tp, L.part + 2 * tp + 1);
					}
				}
			}
			if (BACKWARD) {
				/* the pairs of a bead are neighbouring lanes: their sum goes to the
				 * slot at once (an atomic per pair had up to 32 lanes retrying on
				 * one address).  Lanes past the end are their own runs. */
				const uint32_t key = q0 + lane < n_pair ? s : 64u + lane;
				const uint32_t prev = __shfl_up_sync(GBA_FULL_MASK, key, 1);
				const uint32_t heads = __ballot_sync(GBA_FULL_MASK, lane == 0 || key != prev);
				const uint32_t after = lane == 31 ? 0u : heads >> (lane + 1);
				const int last = after ? lane + __ffs(after) - 1 : 31;
				const float g = run_sum(gqv, lane, last);
				if ((heads >> lane & 1u) && key < 64u) W.gq[s] += g;
				__syncwarp();
			}
		}
	}
	if (BACKWARD) {
		__syncwarp();
#pragma unroll
		for (int h = 0; h < 2; ++h)
			if (nln[h]) {
				const uint32_t i = i0 + lane + 32 * h;
				cell_add(cell + cells.qlig() + i, w, W.gq[lane + 32 * h], L.part + cells.qlig() + i);
			}
	}
	__syncwarp();
}

/* The pose's outputs from the sum of its round totals in W.tot. */
template <bool BACKWARD>
__device__ __forceinline__ void pairwise_finish(const PairwiseLaunch& L, size_t p, float w, int lane, PairStage& W) {
	__syncwarp();
	const volatile float* t = W.tot;
	if (!BACKWARD) {
		if (lane == 0) L.E[p] = t[0];
		return;
	}
	float T[9], ang[3], tx, ty, tz;
#pragma unroll
	for (int k = 0; k < 9; ++k) T[k] = t[4 + k];
	torque_reduce(get_pose(W, tx, ty, tz), T, ang);
	/* dE/dDOF = -(force, Euler torque), DOF_6D order (pos, ang) */
	const float g[6] = {-w * t[1], -w * t[2], -w * t[3], -w * ang[0], -w * ang[1], -w * ang[2]};
	float v = 0.f;
#pragma unroll
	for (int k = 0; k < 6; ++k) v = lane == k ? g[k] : v;
	if (lane < 6) L.g_dofs[6 * p + lane] = v;
}

/* Adds a type pair's (k: ligand type major) or a charge's (q: ligand, then
 * receptor beads) sums to the caller's gradients: with rc = eps r0^8 and
 * ac = eps r0^6, d/dr0 = eps (8 r0^7 d/drc + 6 r0^5 d/dac) and
 * d/deps = r0^8 d/drc + r0^6 d/dac.  Atomics for callers that add several
 * calls' gradients at once. */
__device__ __forceinline__ bool is_zero(double v) { return (__double_as_longlong(v) & 0x7fffffffffffffffll) == 0; }
__device__ __forceinline__ void add_type_pair(const PairwiseLaunch& L, uint32_t k, double drc, double dac) {
	if (is_zero(drc) && is_zero(dac)) return;
	const uint32_t to = L.T * (k % L.T) + k / L.T;
	const double r0 = L.r0[to], eps = L.eps[to];
	const double p2 = r0 * r0, p5 = p2 * p2 * r0, p6 = p5 * r0, p7 = p6 * r0;
	atomicAdd(&L.g_r0[to], eps * (8.0 * p7 * drc + 6.0 * p5 * dac));
	atomicAdd(&L.g_eps[to], p7 * r0 * drc + p6 * dac);
}
__device__ __forceinline__ void add_charge(const PairwiseLaunch& L, uint32_t q, double g) {
	if (!is_zero(g)) atomicAdd(q < L.lig.n ? &L.g_qlig[q] : &L.g_qrec[q - L.lig.n], g);
}

/* Backward: large blocks, so that few copies of the cells take shared memory
 * (256 threads where they leave no room for more); forward: small ones. */
constexpr int kPairwiseThreads = 512, kForwardThreads = 256;

extern __shared__ __align__(16) unsigned char pairwise_smem[];

/* A warp takes a pose -- or, by_round, one 64-bead round of a pose, the warp
 * that finishes the last of them adding the totals -- from the counter.  Each
 * round is reduced on its own and the totals are added in round order, so a
 * pose's result does not depend on the launch (as in rigid_rounds_kernel). */
template <bool BACKWARD>
__global__ void __launch_bounds__(BACKWARD ? kPairwiseThreads : kForwardThreads, BACKWARD ? 2 : 5)
		pairwise_kernel(const PairwiseLaunch L) {
	PairStage* stage = reinterpret_cast<PairStage*>(pairwise_smem);
	unsigned long long* cell = reinterpret_cast<unsigned long long*>(stage + (blockDim.x >> 5));
	const PairCells cells{L.T * L.T, L.lig.n, L.rec.n};
	/* a second copy of the type pairs' cells lies behind the rest, an even
	 * number of cells from the first */
	const uint32_t second = (cells.count() + 1) & ~1u, spare = L.copies > 1 ? 2 * cells.T2 : 0;
	if (BACKWARD) {
		for (uint32_t k = threadIdx.x; k < second + spare; k += blockDim.x) cell[k] = 0;
		__syncthreads();
	}
	cudaGridDependencySynchronize();      /* the setup kernel's records and tables */
	const int lane = threadIdx.x & 31;
	PairStage& W = stage[threadIdx.x >> 5];
	const uint32_t rounds = L.split.rounds;
	const size_t units = L.by_round ? L.n * rounds : L.n;
	for (size_t k = next_pose(L.next, lane); k < units; k = next_pose(L.next, lane)) {
		const size_t at = L.by_round ? k / rounds : k;
		const size_t p = L.order ? (size_t)L.order[at] : at;
		if (lane < kPoseRecord / 4)
			reinterpret_cast<float4*>(W.pose)[lane] = reinterpret_cast<const float4*>(L.split.pose + kPoseRecord * p)[lane];
		if (lane == 0) W.slot = p;
		__syncwarp();
		const float w = BACKWARD ? __ldg(&L.gE[p]) : 0.f;
		const uint32_t r0 = L.by_round ? (uint32_t)(k - at * rounds) : 0, r1 = L.by_round ? r0 + 1 : rounds;
		clear_totals(W, lane);
		for (uint32_t r = r0; r < r1; ++r) {
			PoseSums S = held_sums();
			pairwise_round<BACKWARD>(L, cells, r * kBeadsPerRound, lane, w, W, cell, S);
			const float v = BACKWARD ? sums_total(S, reinterpret_cast<float*>(W.pq), lane) : warp_sum(S.E);
			add_round(W, v, lane);
		}
		const size_t pose = *(volatile unsigned long long*)&W.slot;
		if (L.by_round) {
			/* the round's totals out; the pose's last round reads the others' back */
			float* tot = L.split.totals + pose * rounds * 16 + (lane >> 1);
			if ((lane & 1) == 0) __stcg(tot + 16 * r0, *(volatile float*)&W.tot[lane >> 1]);
			__threadfence();
			__syncwarp();
			uint32_t before = 0;
			if (lane == 0) before = atomicAdd(&L.split.done[pose], 1u);
			before = __shfl_sync(GBA_FULL_MASK, before, 0);
			if (before + 1 != rounds) continue;
			__threadfence();
			clear_totals(W, lane);
			for (uint32_t q = 0; q < rounds; ++q) add_round(W, __ldcg(tot + 16 * q), lane);
		}
		pairwise_finish<BACKWARD>(L, pose, w, lane, W);
		__syncwarp();
	}
	if (BACKWARD) {
		cudaTriggerProgrammaticLaunchCompletion();
		__syncthreads();
		double* out = L.part + (size_t)(1 + blockIdx.x) * cells.count();
		for (uint32_t k = threadIdx.x; k < cells.count(); k += blockDim.x) {
			const unsigned long long c = cell[k], d = k < spare ? cell[second + k] : 0ull;
			double v = 0.0;
			/* most cells of few poses, or of a large table, are empty: the
			 * FP64 pipe's conversions are for the others (200 poses, 500/60
			 * beads, 98 types: 130 -> 99 us; 10,000: 242 -> 211) */
			if ((c | d) != 0ull) {
				v = (double)__uint_as_float((uint32_t)c) + (double)__uint_as_float((uint32_t)(c >> 32));
				if (d != 0ull) v += (double)__uint_as_float((uint32_t)d) + (double)__uint_as_float((uint32_t)(d >> 32));
			}
			out[k] = v;
		}
	}
}

/* Adds the blocks' sums up, scaled as they are (taking the scale off in the
 * blocks cost each of them 2 us of its FP64 pipe), and what no TwoFloat held.
 * 32 cells per block, eight warps a share of the blocks' sums each (one thread
 * per cell waited 34 us for 456 loads in a row). */
__device__ __forceinline__ double cell_sum(const PairwiseLaunch& L, const PairCells& cells, uint32_t k, uint32_t blocks,
		double (*share)[32]) {
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	double v = 0.0;
	const bool in = k < cells.count();
	const double beyond = in && w == 0 ? L.part[k] : 0.0;
	if (in)
#pragma unroll 8
		for (uint32_t b = w + 1; b <= blocks; b += 8) v += L.part[(size_t)b * cells.count() + k];
	share[w][lane] = v;
	__syncthreads();
	if (w == 0) {
		v = 0.0;
#pragma unroll
		for (int q = 0; q < 8; ++q) v += share[q][lane];
		v = v * kCellUnscale + beyond;
	}
	__syncthreads();
	return v;      /* warp 0's */
}

__global__ void __launch_bounds__(256) pairwise_gather_kernel(const PairwiseLaunch L, const uint32_t blocks) {
	__shared__ double share[8][32];
	cudaGridDependencySynchronize();      /* the blocks' sums */
	const PairCells cells{L.T * L.T, L.lig.n, L.rec.n};
	const uint32_t type_blocks = (cells.T2 + 31) / 32;
	const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
	if (blockIdx.x < type_blocks) {
		const uint32_t k = blockIdx.x * 32 + lane;
		const bool in = k < cells.T2;
		const double drc = cell_sum(L, cells, in ? 2 * k : cells.count(), blocks, share);
		const double dac = cell_sum(L, cells, in ? 2 * k + 1 : cells.count(), blocks, share);
		if (w == 0 && in) add_type_pair(L, k, drc, dac);
		return;
	}
	const uint32_t q = (blockIdx.x - type_blocks) * 32 + lane;
	const bool in = q < cells.lig + cells.rec;
	const double g = cell_sum(L, cells, in ? cells.qlig() + q : cells.count(), blocks, share);
	if (w == 0 && in) add_charge(L, q, g);
}

/* The shared memory a block may use. */
constexpr size_t kPairwiseSmem = 227 * 1024;
static_assert(kPairwiseCellBytes + 8 * sizeof(PairStage) <= kPairwiseSmem, "a block of 256 threads always fits");

/* Launches of few poses per resident warp take rounds (their totals within
 * kPairwiseSplitBytes), others whole poses: at most 2.5 a warp backward;
 * forward, where poses are ordered nearest first, so that the tail is short
 * and rounds cost more sooner, (beads - 72) / 256 and at most one.  Measured,
 * whole poses against rounds in us:
 *              poses   2,000     4,000     6,000    10,000      19,000
 *   forward   300/100  35 41     38 45     43 57     54 86      90 153
 *             500/200  54 52     58 58     65 83    76 132     127 241
 *            2000/700 166 90   180 128   193 184   216 296     334 550
 *   backward  300/100 103 97   119 109   139 126   158 174     248 285
 *             500/200 158 114  181 129   208 166   224 241     366 408
 *            2000/700 477 195  516 274   598 379   606 586    981 1060
 * (6,080 and 4,864 resident warps). */
constexpr size_t kPairwiseSplitBytes = (size_t)64 << 20;
inline bool pairwise_splits(bool backward, size_t n, size_t beads, size_t warps) {
	const size_t rounds = (beads + kBeadsPerRound - 1) / kBeadsPerRound;
	if (rounds < 2 || n * rounds * 16 * sizeof(float) > kPairwiseSplitBytes) return false;
	return backward ? 2 * n <= 5 * warps : beads > 72 && 256 * n <= std::min<size_t>(256, beads - 72) * warps;
}

/* Resident blocks per SM: the opt-in to the shared memory and the query once
 * per device, kernel, block size and shared memory. */
int pairwise_blocks_per_sm(const void* kernel, bool backward, int threads, size_t smem) {
	static std::mutex mu;
	static std::map<std::array<size_t, 4>, int> known;
	int dev = 0;
	check_cuda(cudaGetDevice(&dev), "pairwise: device");
	std::lock_guard<std::mutex> g(mu);
	const std::array<size_t, 4> key{(size_t)dev, (size_t)backward, (size_t)threads, smem};
	auto it = known.find(key);
	if (it != known.end()) return it->second;
	/* the largest any launch may ask for: launches of other sizes may be in flight */
	check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPairwiseSmem),
			"pairwise: shared memory");
	int nb = 0;
	check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, smem), "pairwise: occupancy");
	if (known.size() >= 256) known.clear();
	return known[key] = std::max(nb, 1);
}

/* A launch's poses at most: what it takes of scratch per pose (a record of 80
 * bytes, 16 and the sort's own for the order) stays within 128 MB however many
 * poses a call brings. */
constexpr size_t kPairwiseChunk = (size_t)1 << 20;

/* A launch that, if `early`, may begin while the kernel before it runs; the
 * kernel itself waits for that one's results (cudaGridDependencySynchronize). */
template <class... P, class... A>
void launch_after(bool early, void (*kernel)(P...), size_t blocks, int threads, size_t smem, cudaStream_t s,
		const A&... args) {
	cudaLaunchAttribute attr{};
	attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr.val.programmaticStreamSerializationAllowed = early ? 1 : 0;
	cudaLaunchConfig_t cfg{};
	cfg.gridDim = dim3((unsigned)blocks);
	cfg.blockDim = dim3(threads);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cfg.attrs = &attr;
	cfg.numAttrs = 1;
	check_cuda(cudaLaunchKernelEx(&cfg, kernel, P(args)...), "pairwise launch");
}

/* The launches for the poses of L, at most kPairwiseChunk. */
void launch_pairwise(Context& ctx, PairwiseLaunch L, bool backward, cudaStream_t s) {
	const size_t n = L.n;
	const PairCells cells{L.T * L.T, L.lig.n, L.rec.n};
	const size_t cell_bytes = backward ? pairwise_cell_bytes(L.T, L.lig.n, L.rec.n) : 0;
	const size_t rounds = (L.lig.n + kBeadsPerRound - 1) / kBeadsPerRound;
	const int threads = !backward ? kForwardThreads
			: cell_bytes + kPairwiseThreads / 32 * sizeof(PairStage) <= kPairwiseSmem ? kPairwiseThreads : 256;
	const size_t warps = threads / 32;
	/* a second copy of the type pairs' cells where two blocks still fit an
	 * SM: half as many lanes meet in a cell.  2000/700 beads, 32 types, forward
	 * and backward, one copy against two: 10,000 poses 901 -> 876 us, 30,000
	 * 2,312 -> 2,218; 500/200, 30,000 poses: 887 -> 825. */
	const size_t two_copies = (cell_bytes + 15) / 16 * 16 + (size_t)2 * L.T * L.T * sizeof(unsigned long long);
	L.copies = backward && threads == kPairwiseThreads &&
			2 * (two_copies + warps * sizeof(PairStage) + 1024) <= kPairwiseSmem ? 2 : 1;
	const size_t smem = (L.copies > 1 ? two_copies : (cell_bytes + 15) / 16 * 16) + warps * sizeof(PairStage);
	const void* kernel = backward ? (const void*)pairwise_kernel<true> : (const void*)pairwise_kernel<false>;
	const size_t resident = (size_t)ctx.num_sms * pairwise_blocks_per_sm(kernel, backward, threads, smem);
	L.by_round = pairwise_splits(backward, n, L.lig.n, resident * warps);
	const size_t units = L.by_round ? n * rounds : n;
	const size_t blocks = std::max<size_t>(1, std::min<size_t>((units + warps - 1) / warps, resident));
	/* one block of scratch, every part 16-byte aligned */
	StreamScratch scratch(ctx.scratch_pool);
	const bool sorted = n >= kNearFirstMinPoses && n <= kNearOneBlock;
	const size_t T2 = cells.T2;
	size_t at = 0;
	auto place = [&](size_t bytes) {
		const size_t o = at;
		at += (bytes + 15) & ~(size_t)15;
		return o;
	};
	const size_t o_next = place(sizeof(unsigned long long)), o_tab = place(2 * T2 * sizeof(float4)),
			o_rq = place(L.rec.n * sizeof(float4)), o_pose = place(n * kPoseRecord * sizeof(float)),
			o_done = place(L.by_round ? n * sizeof(uint32_t) : 0),
			o_tot = place(L.by_round ? n * rounds * 16 * sizeof(float) : 0),
			o_order = place(sorted ? n * sizeof(uint32_t) : 0),
			o_part = place(backward ? (blocks + 1) * cells.count() * sizeof(double) : 0);
	char* base = (char*)scratch.get(at, s);
	L.next = (unsigned long long*)(base + o_next);
	L.tab = (float4*)(base + o_tab);
	L.rq = (float4*)(base + o_rq);
	L.split.pose = (float*)(base + o_pose);
	L.split.done = (uint32_t*)(base + o_done);
	L.split.totals = (float*)(base + o_tot);
	L.split.rounds = (uint32_t)rounds;
	L.part = (double*)(base + o_part);
	L.order = sorted ? (uint32_t*)(base + o_order) : n > kNearOneBlock ? near_first_order(L.dofs, n, scratch, s) : nullptr;
	const uint32_t pose_blocks = (uint32_t)((4 * n + kSetupThreads - 1) / kSetupThreads);
	const uint32_t table_blocks = (uint32_t)std::min<size_t>(
			(std::max<size_t>(T2, backward ? cells.count() : L.rec.n) + kSetupThreads - 1) / kSetupThreads, 256);
	pairwise_setup_kernel<<<1 + pose_blocks + std::max(1u, table_blocks), kSetupThreads, 0, s>>>(L, pose_blocks, sorted,
			backward ? cells.count() : 0);
	check_cuda(cudaGetLastError(), "pairwise: setup");
	/* few blocks: the launches overlap (one pose, 300/60 beads, backward 34 ->
	 * 29 us; 64 poses, 56/17: 37.5 -> 32.5).  A launch that fills the chip would
	 * have its blocks placed around the setup's (30,000 poses, 2000/700 beads,
	 * forward 509 -> 524). */
	const bool early = 2 * blocks <= resident;
	if (backward) {
		launch_after(early, pairwise_kernel<true>, blocks, threads, smem, s, L);
		launch_after(early, pairwise_gather_kernel, (T2 + 31) / 32 + (L.lig.n + L.rec.n + 31) / 32, 256, 0, s, L,
				(uint32_t)blocks);
	} else {
		launch_after(early, pairwise_kernel<false>, blocks, threads, smem, s, L);
	}
	check_cuda(cudaGetLastError(), "pairwise launch");
}

}  // namespace

}  // namespace gba

using namespace gba;

extern "C" int gba_pairwise_6d(gba_ctx* ctx, gba_id rec, gba_id lig, gba_id grid,
		const gba_pairwise_params* pp, const gba_dof6d* dofs, size_t n, float* E_out,
		const float* gE, float* g_dofs, double* g_qlig, double* g_qrec, double* g_r0,
		double* g_eps, void* stream) {
	if (!ctx) return GBA_ERR_INVALID_ARGUMENT;
	try {
		if (!pp || !pp->r0 || !pp->eps || !pp->ipon || !pp->q_lig || !pp->q_rec)
			throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_pairwise_6d: null parameter array");
		if (n == 0) return GBA_OK;
		const bool backward = gE != nullptr;
		if (!dofs || (!backward && !E_out) ||
				(backward && (!g_dofs || !g_qlig || !g_qrec || !g_r0 || !g_eps)))
			throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_pairwise_6d: null pose/output pointer");
		for (const void* ptr : {(const void*)dofs, (const void*)pp->r0, (const void*)pp->eps,
					(const void*)pp->ipon, (const void*)pp->q_lig, (const void*)pp->q_rec})
			if (!is_device_pointer(ptr))
				throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_pairwise_6d: device pointers required");
		if (pp->potshape != GBA_POTSHAPE_8_6)
			throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_pairwise_6d: only the 8-6 shape is differentiable here");
		ctx->bind();
		PairwiseLaunch L{};
		{
			Lock g(ctx->mu);
			auto* R = static_cast<ProteinItem*>(ctx->find(rec, ItemKind::Protein));
			auto* Lg = static_cast<ProteinItem*>(ctx->find(lig, ItemKind::Protein));
			auto* G = static_cast<GridItem*>(ctx->find(grid, ItemKind::Grid));
			if (R->max_type > pp->num_types || Lg->max_type > pp->num_types)
				throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_pairwise_6d: bead type exceeds num_types");
			if (G->nl_has_entries && G->nl_max_index >= R->dev.n)
				throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_pairwise_6d: neighbour list indexes beyond the receptor");
			/* the voxel lists must cover every pair within the cutoff */
			const double reach = (double)pp->cutoff + 0.5 * std::sqrt(3.0) * G->nl_desc.gridSpacing;
			if (!(pp->cutoff > 0) || reach > G->nl_list_radius + 1e-6)
				throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_pairwise_6d: cutoff exceeds what the neighbour grid covers");
			L.rec = R->dev;
			L.lig = Lg->dev;
			L.nl = G->dev.nl;
			L.tlist = ctx->typed_list(*G, rec, *R, true);
		}
		L.T = pp->num_types;
		L.r0 = pp->r0;
		L.eps = pp->eps;
		L.ipon = pp->ipon;
		L.q_lig = pp->q_lig;
		L.q_rec = pp->q_rec;
		L.dielec = pp->dielec;
		L.ffelec = pp->ffelec;
		L.cut2 = pp->cutoff * pp->cutoff;
		L.dofs = dofs;
		L.n = n;
		L.E = E_out;
		L.gE = gE;
		L.g_dofs = g_dofs;
		L.g_qlig = g_qlig;
		L.g_qrec = g_qrec;
		L.g_r0 = g_r0;
		L.g_eps = g_eps;
		cudaStream_t s = (cudaStream_t)stream;
		if (const char* why = pairwise_refused(backward, L.T, L.lig.n, L.rec.n))
			throw ApiError(GBA_ERR_INVALID_ARGUMENT, why);
		/* per-pose results do not depend on the launch, and the sums are added */
		for (size_t at = 0; at < n; at += kPairwiseChunk) {
			PairwiseLaunch C = L;
			C.n = std::min(kPairwiseChunk, n - at);
			C.dofs = dofs + at;
			if (backward) {
				C.gE = gE + at;
				C.g_dofs = g_dofs + 6 * at;
			} else {
				C.E = E_out + at;
			}
			launch_pairwise(*ctx, C, backward, s);
		}
	} catch (const ApiError& e) {
		ctx->set_error(e.what());
		return e.code;
	} catch (const std::exception& e) {
		ctx->set_error(e.what());
		return GBA_ERR_INVALID_ARGUMENT;
	}
	return GBA_OK;
}
