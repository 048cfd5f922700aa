/*
 * gridbuild.cu -- builds a receptor's inner/outer potential grids and its
 * neighbour-list grid on the device.
 *
 * The reference only reads ATTRACT grid files (src/fileIO/readFile.cpp:261-422;
 * the builder attract::Grid::calculate_std is declared at
 * src/fileIO/grid_orig.h:143 and defined nowhere).  This builder produces the
 * same in-memory layout with these semantics:
 *   channel c >= 1 (ligand type alphabet[c-1]) and the charge channel 0 hold,
 *   at each voxel centre p, the sum over receptor beads j (type != 0) of the
 *   ATTRACT pair force/energy evaluated at max(|p - x_j|, plateau) along the
 *   direction p - x_j (LJPotForce / ChargePotForce, src/model/forcefield.h),
 *   so that grid + NL(r) - NL(plateau) is the exact pair term inside the
 *   plateau (src/model/neighborlist.h:104-157);
 *   voxel v's neighbour list holds, in increasing index, every receptor bead
 *   (type != 0) with |p_v - x_j|^2 <= nl_cutoff^2, tested in double with
 *   unfused operations so the lists are bit-identical to the CPU builder.
 * Arithmetic of the potentials (the CPU builder performs the same operations
 * in the same order, so both produce the same bits): the voxel centre in
 * double, unfused, rounded to float; per bead the separation, its square,
 * the plateau rescaling (plateau / sqrt(r^2)) and 1/r^2 in IEEE-rounded FP32
 * (no approximate reciprocal or square root, nothing contracted); the pair
 * terms of energy_dev.cuh; FP32 partial sums over each block of 256
 * consecutive receptor beads, in bead order; those partials added in double,
 * block after block; the total rounded to float.
 * Layout: inner box = bead bounding box + margin, spacing d; outer grid
 * spacing 2d, extended by outer_ext inner voxels per side; NL grid = inner.
 */
#include <algorithm>
#include <cmath>
#include <vector>

#include "energy_dev.cuh"
#include "gba_context.h"

namespace gba {

namespace {

constexpr int kTile = 256;   /* receptor beads per FP32 partial sum; voxels per block of the list kernels */

struct BuildArgs {
	const float4* xyzq;      /* receptor beads */
	const uint32_t* tm;      /* type | mapped << 16 */
	uint32_t n;
	DevParams par;
	uint32_t n_alphabet;
	float plateau, plat2;
	double cut2;
	/* per receptor type (row 0: dummy beads, all zero) and type channel
	 * (n_lj of them, the alphabet padded to whole warps): the pair parameters
	 * as grid_potential_kernel reads them (pair_rows_kernel) */
	const float4* rows;
	uint32_t n_lj;
	float one;               /* 1 */
	uint32_t blank[4];       /* channels of ligand type 0 (a bit each): all zero */
};

/* ---- potentials -------------------------------------------------------------
 *
 * Per voxel, channel and bead 12 FP32 operations, each rounded on its own (the
 * CPU builder's bits): 6.6e11 for 1,500 beads, 1.15 M voxels and 32 channels,
 * 17.5 ms at the 37.8e12 a second of the FP32 pipe.  A block holds a brick of
 * 4 x 4 x 4 voxels and up to 32 channels: two warps compute the geometry of 16
 * beads at a time into shared memory (one also sums the charge channel; with
 * one such warp the others waited, 36.8 ms against 27.5, with three 29.0),
 * warps of four or eight channels each read it back, two voxels per lane in
 * packed FP32 instructions, which halve the issue slots.  Double-buffered, one
 * barrier per 16 beads (8: 6 % slower).
 *   What the channel warps read bounds it next (L1 data pipe 81 % busy): four
 * 8-byte words per bead and lane (1/d^6 is two products away) and a 16-byte row
 * per two channels.  The double sums, touched every 256 beads, lie in local
 * memory, where they leave the partial sums their registers.  Eight channels a
 * warp share a word among more of them but leave fewer warps: with the lists
 * 25.1 against 26.6 ms; 600 beads and 8, 20, 28, 32 and 33 channels 2.90, 5.89,
 * 6.22, 6.25 and 11.75 ms against 2.58, 5.24, 6.05, 6.35 and 11.98 with four. */

constexpr int kBlockChan = 32;                /* most type channels per block */
constexpr int kCube = 4;                      /* voxels per axis of a block */
constexpr int kChunk = 16;                    /* beads per barrier */
static_assert(kTile % kChunk == 0, "a partial sum ends with a chunk");

/* Two voxels of a lane (z and z + 2 of its column): packed FP32, each half
 * rounded as the scalar operation. */
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) {
	f2 r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
	return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
	f2 r;
	asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
	f2 r;
	asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
	return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
	f2 r;
	asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
	return r;
}

/* One bead's geometry for a lane's two voxels: 1/d^2 and the direction over d^2
 * at d = max(r, plateau); for the general form 1/d^6 and d^2 too. */
struct VoxelGeo {
	f2 rr2[32], ux[32], uy[32], uz[32], rr23[32], d2[32];
};
struct Chunk {
	VoxelGeo geo[kChunk];
	uint32_t row[kChunk];      /* receptor type, 0: no contribution */
	float qf[kChunk];          /* charge times ffelec, 0: no contribution */
};

/* For k = receptor type * n_lj + channel: plain, the k-th pair of floats is
 * {rc, -ac}; else out[2 k] = {rc, rc, -ac, -ac} and out[2 k + 1] = {ipon, ipon,
 * rmin2, emin}. */
__global__ void pair_rows_kernel(DevParams par, const uint32_t* __restrict__ alphabet, uint32_t n_alphabet,
		uint32_t n_lj, int plain, float4* __restrict__ out) {
	const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (k >= (size_t)(par.num_types + 1) * n_lj) return;
	const uint32_t tr = (uint32_t)(k / n_lj), c = (uint32_t)(k % n_lj);
	const uint32_t tl = c < n_alphabet ? alphabet[c] : 0u;
	float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
	float iv = 0.f;
	if (tr != 0 && tl != 0 && tl <= par.num_types) {
		const size_t t = (size_t)par.num_types * (tr - 1) + (tl - 1);
		p = par.lj[t];
		iv = par.ivor[t];
	}
	if (plain) {
		reinterpret_cast<float2*>(out)[k] = make_float2(p.x, -p.y);
		return;
	}
	out[2 * k] = make_float4(p.x, p.x, -p.y, -p.y);
	out[2 * k + 1] = make_float4(iv, iv, p.z, p.w);
}

/* A geometry warp's share of the beads of a chunk, in pairs: the warp that
 * also sums the charge channel takes fewer. */
constexpr int kPairs = kChunk / 2, kChargePairs = 3;

/* Bead j of the receptor as one lane holds it for its chunk.  A dummy bead
 * (type 0) or one past the end adds zeros to every sum, and lies so far away
 * that its powers of 1/d are finite: within a plateau of 1e-7 A of a voxel
 * 1/d^6 is infinite, and zero times that no number. */
constexpr float kNowhere = 1e18f;
struct Bead {
	float4 r;
	uint32_t type;
};
__device__ __forceinline__ Bead load_bead(const BuildArgs& a, uint32_t j) {
	Bead b{make_float4(kNowhere, kNowhere, kNowhere, 0.f), 0u};
	if (j < a.n) {
		b.type = __ldg(&a.tm[j]) & 0xffffu;
		if (b.type != 0) b.r = __ldg(&a.xyzq[j]);
	}
	return b;
}

/* The geometry of the bead pairs [i0, i1) of a chunk for the brick, by one
 * warp: lane = column (x, y) of the brick and half = bead of the pair; lane b
 * (< kChunk) brings bead b of the chunk. */
template <bool PLAIN>
__device__ __forceinline__ void fill_chunk(const BuildArgs& a, const Bead& mine, int i0, int i1, float px, float py,
		const float pz[kCube], int lane, Chunk& C) {
	const int col = lane & 15, half = lane >> 4;
	for (int i = i0; i < i1; ++i) {
		const int b = 2 * i + half;
		const uint32_t tr = __shfl_sync(0xffffffffu, mine.type, b);
		const float rx = __shfl_sync(0xffffffffu, mine.r.x, b), ry = __shfl_sync(0xffffffffu, mine.r.y, b),
				rz = __shfl_sync(0xffffffffu, mine.r.z, b), rq = __shfl_sync(0xffffffffu, mine.r.w, b);
		if (col == 0) {
			const float qf = fmul(rq, a.par.ffelec);
			C.row[b] = tr;
			C.qf[b] = fabsf(qf) > 0.001f ? qf : 0.f;
		}
		const float ex0 = fsub(px, rx), ey0 = fsub(py, ry);
		const float exy = fadd(fmul(ex0, ex0), fmul(ey0, ey0));
		float ex[kCube], ey[kCube], ez[kCube], e2[kCube];
		bool near = false;
#pragma unroll
		for (int z = 0; z < kCube; ++z) {
			ex[z] = ex0;
			ey[z] = ey0;
			ez[z] = fsub(pz[z], rz);
			e2[z] = fadd(exy, fmul(ez[z], ez[z]));
			near |= e2[z] < a.plat2;
		}
		if (near) {
#pragma unroll
			for (int z = 0; z < kCube; ++z)
				if (e2[z] < a.plat2) {
					/* a bead at the voxel's centre has no direction */
					const float sc = e2[z] > 0.f ? __fdiv_rn(a.plateau, __fsqrt_rn(e2[z])) : 0.f;
					ex[z] = fmul(ex[z], sc); ey[z] = fmul(ey[z], sc); ez[z] = fmul(ez[z], sc);
					e2[z] = a.plat2;
				}
		}
		float rr2[kCube];
#pragma unroll
		for (int z = 0; z < kCube; ++z) rr2[z] = __frcp_rn(e2[z]);
		VoxelGeo& g = C.geo[b];
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			const int l = col + 16 * h;
			const f2 i2 = pack2(rr2[h], rr2[h + 2]);
			g.rr2[l] = i2;
			g.ux[l] = mul2(pack2(ex[h], ex[h + 2]), i2);
			g.uy[l] = mul2(pack2(ey[h], ey[h + 2]), i2);
			g.uz[l] = mul2(pack2(ez[h], ez[h + 2]), i2);
			if (!PLAIN) {
				g.rr23[l] = mul2(mul2(i2, i2), i2);
				g.d2[l] = pack2(e2[h], e2[h + 2]);
			}
		}
	}
}

/* Adds a partial sum's packed pair to the two voxels' double sums. */
template <class Acc>
__device__ __forceinline__ void fold2(f2& part, Acc* acc) {
	float lo, hi;
	unpack2(part, lo, hi);
	acc[0] = __dadd_rn(acc[0], (double)lo);
	acc[1] = __dadd_rn(acc[1], (double)hi);
	part = 0;
}

/* PLAIN: every pair's ipon is 1, its minimum lies inside the plateau (no
 * branch on d^2 < rmin2) and 2 (rep rr23) = rep (2 rr23) without underflow;
 * the host checks all three (plain_pairs).  8-6 shape only.  CH: type channels
 * per warp. */
template <bool PLAIN, int CH>
__global__ void __launch_bounds__(32 * (kBlockChan / CH + 2), 2) grid_potential_kernel(const BuildArgs a,
		const gba_intrpl_desc d, float4* __restrict__ out) {
	__shared__ Chunk buf[2];
	const uint32_t Nx = d.dimN[0], Ny = d.dimN[1], Nz = d.dimN[2];
	const size_t N = (size_t)Nx * Ny * Nz;
	const int lane = threadIdx.x & 31;
	const int warp = threadIdx.x >> 5, lj_warps = (blockDim.x >> 5) - 2;
	const uint32_t bx = (Nx + kCube - 1) / kCube, by = (Ny + kCube - 1) / kCube;
	const uint32_t x0 = blockIdx.x % bx * kCube, y0 = blockIdx.x / bx % by * kCube,
			z0 = blockIdx.x / (bx * by) * kCube;
	const uint32_t chunks = (a.n + kChunk - 1) / kChunk;
	/* the lane's voxels when it holds sums: (x, y, z) and (x, y, z + 2) */
	const uint32_t vx = x0 + (lane & 3), vy = y0 + ((lane >> 2) & 3), vz = z0 + (lane >> 4);
	const size_t v0 = (size_t)Nx * ((size_t)vz * Ny + vy) + vx, v1 = v0 + 2 * (size_t)Nx * Ny;
	const bool in0 = vx < Nx && vy < Ny && vz < Nz, in1 = vx < Nx && vy < Ny && vz + 2 < Nz;
	if (warp >= lj_warps) {
		/* the geometry warps, one chunk ahead (the beads' records two), the
		 * first of them with the charge channel */
		const double sp = (double)d.gridSpacing;
		const float px = (float)__dadd_rn((double)d.posMin[0], __dmul_rn((double)vx, sp));
		const float py = (float)__dadd_rn((double)d.posMin[1], __dmul_rn((double)vy, sp));
		float pz[kCube];
#pragma unroll
		for (int z = 0; z < kCube; ++z)
			pz[z] = (float)__dadd_rn((double)d.posMin[2], __dmul_rn((double)(z0 + z), sp));
		const bool charge = warp == lj_warps && blockIdx.y == 0, cdiel = a.par.dielec == GBA_DIELEC_CONSTANT;
		const int i0 = warp == lj_warps ? 0 : kChargePairs, i1 = warp == lj_warps ? kChargePairs : kPairs;
		double acc[4][2] = {};
		f2 part[4] = {0, 0, 0, 0};
		/* lanes past the chunk load its beads again: inside the receptor or nothing */
		Bead mine = load_bead(a, lane & (kChunk - 1));
		fill_chunk<PLAIN>(a, mine, i0, i1, px, py, pz, lane, buf[0]);
		mine = load_bead(a, kChunk + (lane & (kChunk - 1)));
		__syncthreads();
		for (uint32_t k = 0; k < chunks; ++k) {
			if (k + 1 < chunks) {
				const Bead now = mine;
				mine = load_bead(a, (k + 2) * kChunk + (lane & (kChunk - 1)));
				fill_chunk<PLAIN>(a, now, i0, i1, px, py, pz, lane, buf[(k + 1) & 1]);
			}
			if (charge) {
				const Chunk& C = buf[k & 1];
				for (int b = 0; b < kChunk; ++b) {
					const float qf = C.qf[b];
					if (qf == 0.f) continue;
					const VoxelGeo& g = C.geo[b];
					float i[2], ux[2], uy[2], uz[2], fx[2], fy[2], fz[2], e[2];
					unpack2(g.rr2[lane], i[0], i[1]);
					unpack2(g.ux[lane], ux[0], ux[1]);
					unpack2(g.uy[lane], uy[0], uy[1]);
					unpack2(g.uz[lane], uz[0], uz[1]);
#pragma unroll
					for (int h = 0; h < 2; ++h)
						charge_pot_force(i[h], ux[h], uy[h], uz[h], qf, cdiel, fx[h], fy[h], fz[h], e[h]);
					part[0] = add2(part[0], pack2(fx[0], fx[1]));
					part[1] = add2(part[1], pack2(fy[0], fy[1]));
					part[2] = add2(part[2], pack2(fz[0], fz[1]));
					part[3] = add2(part[3], pack2(e[0], e[1]));
				}
				if ((k + 1) % (kTile / kChunk) == 0 || k + 1 == chunks)
#pragma unroll
					for (int c = 0; c < 4; ++c) fold2(part[c], acc[c]);
			}
			__syncthreads();
		}
		if (charge) {
			if (in0) out[v0] = make_float4((float)acc[0][0], (float)acc[1][0], (float)acc[2][0], (float)acc[3][0]);
			if (in1) out[v1] = make_float4((float)acc[0][1], (float)acc[1][1], (float)acc[2][1], (float)acc[3][1]);
		}
		return;
	}
	constexpr int kAhead = PLAIN ? 2 : 4;      /* beads whose rows a warp loads together */
	const bool shape86 = PLAIN || a.par.potshape == GBA_POTSHAPE_8_6;
	const uint32_t c0 = blockIdx.y * kBlockChan + warp * CH;   /* first type channel */
	const float4* rows = PLAIN ? a.rows + c0 / 2 : a.rows + 2 * (size_t)c0;
	/* The assembler fuses a packed product into a packed sum that follows it,
	 * although both round; a factor of one that it cannot see keeps them apart,
	 * in every such sum below (a product's second use may keep it whole too,
	 * but nothing says so). */
	const f2 six = pack2(6.f, 6.f), two = pack2(2.f, 2.f), one = pack2(a.one, a.one);
	/* in local memory, read and written every 256 beads: the registers are the
	 * partial sums' */
	volatile double acc[CH][4][2];
#pragma unroll
	for (int i = 0; i < CH; ++i)
#pragma unroll
		for (int c = 0; c < 4; ++c) acc[i][c][0] = acc[i][c][1] = 0.0;
	f2 part[CH][4] = {};
	__syncthreads();
	for (uint32_t k = 0; k < chunks; ++k) {
		const Chunk& C = buf[k & 1];
		if (PLAIN) {
#pragma unroll kAhead
			for (int b = 0; b < kChunk; ++b) {
				const VoxelGeo& g = C.geo[b];
				const f2 rr2 = g.rr2[lane], ux = g.ux[lane], uy = g.uy[lane], uz = g.uz[lane];
				const f2 rr23 = mul2(mul2(rr2, rr2), rr2), dbl = mul2(rr23, two);
				const float4* row = rows + (size_t)(C.row[b] * (a.n_lj / 2));
				float4 q[CH / 2];
#pragma unroll
				for (int i = 0; i < CH / 2; ++i) q[i] = __ldg(row + i);
#pragma unroll
				for (int i = 0; i < CH; ++i) {
					const float rc = i & 1 ? q[i / 2].z : q[i / 2].x, ac = i & 1 ? q[i / 2].w : q[i / 2].y;
					const f2 rep = mul2(pack2(rc, rc), rr2);
					const f2 vlj = mul2(fma2(rep, one, pack2(ac, ac)), rr23);
					const f2 fb = fma2(six, vlj, mul2(rep, dbl));
					part[i][0] = fma2(mul2(fb, ux), one, part[i][0]);
					part[i][1] = fma2(mul2(fb, uy), one, part[i][1]);
					part[i][2] = fma2(mul2(fb, uz), one, part[i][2]);
					part[i][3] = fma2(vlj, one, part[i][3]);
				}
			}
		} else {
#pragma unroll kAhead
			for (int b = 0; b < kChunk; ++b) {
				const float4* row = rows + 2 * (size_t)(C.row[b] * a.n_lj);
				const VoxelGeo& g = C.geo[b];
				const f2 rr2 = g.rr2[lane], ux = g.ux[lane], uy = g.uy[lane], uz = g.uz[lane], rr23 = g.rr23[lane];
				const f2 sd = shape86 ? pack2(2.f, 2.f) : six;
				const f2 rrd = shape86 ? rr2 : rr23;
				float da, db;
				unpack2(g.d2[lane], da, db);
#pragma unroll
				for (int i = 0; i < CH; ++i) {
					const float4 p = __ldg(row + 2 * i), m = __ldg(row + 2 * i + 1);   /* m: ipon, ipon, rmin2, emin */
					const f2 rep = mul2(pack2(p.x, p.y), rrd);
					const f2 vlj = mul2(fma2(rep, one, pack2(p.z, p.w)), rr23);
					const f2 fb = fma2(six, vlj, mul2(sd, mul2(rep, rr23)));
					const f2 iv = pack2(m.x, m.y), off = pack2(fsub(m.x, 1.0f), fsub(m.x, 1.0f));
					float e_in[2], e_out[2], f_in[2], f_out[2];
					unpack2(fma2(off, pack2(m.w, m.w), vlj), e_in[0], e_in[1]);
					unpack2(mul2(iv, vlj), e_out[0], e_out[1]);
					unpack2(fb, f_in[0], f_in[1]);
					unpack2(mul2(iv, fb), f_out[0], f_out[1]);
					const f2 e = pack2(da < m.z ? e_in[0] : e_out[0], db < m.z ? e_in[1] : e_out[1]);
					const f2 f = pack2(da < m.z ? f_in[0] : f_out[0], db < m.z ? f_in[1] : f_out[1]);
					part[i][0] = fma2(mul2(f, ux), one, part[i][0]);
					part[i][1] = fma2(mul2(f, uy), one, part[i][1]);
					part[i][2] = fma2(mul2(f, uz), one, part[i][2]);
					part[i][3] = fma2(e, one, part[i][3]);
				}
			}
		}
		if ((k + 1) % (kTile / kChunk) == 0 || k + 1 == chunks)
#pragma unroll
			for (int i = 0; i < CH; ++i)
#pragma unroll
				for (int c = 0; c < 4; ++c) fold2(part[i][c], acc[i][c]);
		__syncthreads();
	}
#pragma unroll
	for (int i = 0; i < CH; ++i)
		if (c0 + i < a.n_alphabet) {
			float4* o = out + (size_t)(1 + c0 + i) * N;
			if (!PLAIN && (a.blank[(c0 + i) >> 5] >> ((c0 + i) & 31) & 1u)) {
				if (in0) o[v0] = make_float4(0.f, 0.f, 0.f, 0.f);
				if (in1) o[v1] = make_float4(0.f, 0.f, 0.f, 0.f);
				continue;
			}
			if (in0) o[v0] = make_float4((float)acc[i][0][0], (float)acc[i][1][0], (float)acc[i][2][0], (float)acc[i][3][0]);
			if (in1) o[v1] = make_float4((float)acc[i][0][1], (float)acc[i][1][1], (float)acc[i][2][1], (float)acc[i][3][1]);
		}
}

/* The three conditions of grid_potential_kernel's plain form, over the whole
 * table; reach2: a bound of the squared distance between a voxel and a bead. */
bool plain_pairs(const std::vector<gba_ffparam>& table, int potshape, float plat2, double reach2) {
	if (potshape != GBA_POTSHAPE_8_6 || !(plat2 >= 1e-6f)) return false;
	for (const gba_ffparam& p : table) {
		if (p.ipon != 1 || p.rmin2 > plat2 || !std::isfinite(p.rc)) return false;
		/* rep rr23 >= rc / reach2^4 has to stay a normal number */
		if (p.rc != 0.f && std::fabs((double)p.rc) / (reach2 * reach2 * reach2 * reach2) < 1e-36) return false;
	}
	return true;
}

void launch_potentials(const BuildArgs& a, bool plain, const gba_intrpl_desc& d, float4* out, cudaStream_t s) {
	uint64_t bricks = 1;
	for (int k = 0; k < 3; ++k) bricks *= (d.dimN[k] + kCube - 1) / kCube;
	const unsigned groups = std::max<uint32_t>(1, (a.n_alphabet + kBlockChan - 1) / kBlockChan);
	const uint32_t chan = std::min<uint32_t>(a.n_alphabet, kBlockChan);
	/* eight channels a warp where they fill the block's warps (grid_potential_kernel) */
	auto launch = [&](auto kernel, uint32_t per) {
		kernel<<<dim3((unsigned)bricks, groups), 32 * ((chan + per - 1) / per + 2), 0, s>>>(a, d, out);
	};
	if (!plain)
		launch(grid_potential_kernel<false, 4>, 4);
	else if (a.n_alphabet > 28)
		launch(grid_potential_kernel<true, 8>, 8);
	else
		launch(grid_potential_kernel<true, 4>, 4);
	check_cuda(cudaGetLastError(), "grid build: potentials");
}

/* Neighbour membership, unfused double arithmetic (bit-identical to the CPU builder). */
__device__ __forceinline__ bool nl_member(double px, double py, double pz, float4 r, double cut2) {
	const double dx = __dsub_rn(px, (double)r.x);
	const double dy = __dsub_rn(py, (double)r.y);
	const double dz = __dsub_rn(pz, (double)r.z);
	const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
	return d2 <= cut2;
}

/* Bounds of the FP32 test that decides most memberships without FP64: with
 * every coordinate of the grid and the beads within `extent` of zero, the
 * FP32 squared distance is off the double one by less than `band` around the
 * cutoff, so below `sure` a bead is a member, above `never` it is not, and
 * only in between (or for a NaN) does nl_member decide. */
struct NlBounds {
	float sure, never;
	float brick;         /* as `never`, for the distance to a brick's box */
};

NlBounds nl_bounds(double cut2, double extent) {
	const double cut = std::sqrt(cut2);
	/* per coordinate: the voxel centre's rounding to FP32, the difference's
	 * rounding and (brick) the box's own, each below extent 2^-23 */
	const double e = extent * 4.76837158203125e-7;      /* 2^-21 */
	const double band = 8.0 * cut * e + 16.0 * e * e + cut2 * 9.5367431640625e-7;
	auto up = [](double v) { return std::nextafter((float)v, INFINITY); };
	NlBounds b;
	b.sure = std::nextafter((float)(cut2 - band), -INFINITY);
	b.never = up(cut2 + band);
	b.brick = up(cut2 + 2.0 * band);
	return b;
}

/* A block's voxels: a brick of 8 x 8 x 4, one per thread. */
constexpr int kBrick[3] = {8, 8, 4};
static_assert(kBrick[0] * kBrick[1] * kBrick[2] == kTile, "one voxel per thread");

/* Neighbour lists.  Bounded by instruction issue: brute force tested every
 * bead against every voxel in FP64, whose pipe issues one warp instruction
 * per 16 cycles and SM (1,500 beads, 0.69 M voxels: 23.6 ms a pass).  A block
 * takes a compact brick of voxels instead: each thread tests one bead of the
 * tile against the brick's box and the block keeps those within the cutoff,
 * in bead order (a tenth of a large receptor); every voxel then tests only
 * those, in FP32, with nl_member deciding where FP32 cannot (NlBounds). */
template <bool FILL>
__global__ void __launch_bounds__(kTile) nl_kernel(BuildArgs a, gba_nl_desc d, NlBounds bd,
		uint32_t* __restrict__ count, const uint2* __restrict__ desc, uint32_t* __restrict__ list) {
	__shared__ float4 cand[kTile];         /* x, y, z, bead index (bits) */
	__shared__ uint32_t warp_n[kTile / 32];
	const uint32_t Nx = d.dimN[0], Ny = d.dimN[1], Nz = d.dimN[2];
	const uint32_t tx = threadIdx.x % kBrick[0], ty = (threadIdx.x / kBrick[0]) % kBrick[1],
			tz = threadIdx.x / (kBrick[0] * kBrick[1]);
	const uint32_t bx = (Nx + kBrick[0] - 1) / kBrick[0], by = (Ny + kBrick[1] - 1) / kBrick[1];
	const uint32_t x0 = blockIdx.x % bx * kBrick[0], y0 = blockIdx.x / bx % by * kBrick[1],
			z0 = blockIdx.x / (bx * by) * kBrick[2];
	const uint32_t x = x0 + tx, y = y0 + ty, z = z0 + tz;
	const bool valid = x < Nx && y < Ny && z < Nz;
	const size_t v = (size_t)Nx * ((size_t)z * Ny + y) + x;
	const double sp = (double)d.gridSpacing;
	const double px = __dadd_rn((double)d.posMin[0], __dmul_rn((double)x, sp));
	const double py = __dadd_rn((double)d.posMin[1], __dmul_rn((double)y, sp));
	const double pz = __dadd_rn((double)d.posMin[2], __dmul_rn((double)z, sp));
	const float fx = (float)px, fy = (float)py, fz = (float)pz;
	const float lx = (float)(d.posMin[0] + x0 * sp), hx = (float)(d.posMin[0] + (x0 + kBrick[0] - 1) * sp);
	const float ly = (float)(d.posMin[1] + y0 * sp), hy = (float)(d.posMin[1] + (y0 + kBrick[1] - 1) * sp);
	const float lz = (float)(d.posMin[2] + z0 * sp), hz = (float)(d.posMin[2] + (z0 + kBrick[2] - 1) * sp);
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	uint32_t cnt = 0;
	uint32_t* dst = FILL && valid ? list + desc[v].y : nullptr;
	for (uint32_t t0 = 0; t0 < a.n; t0 += kTile) {
		const uint32_t j = t0 + threadIdx.x;
		float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
		bool in = false;
		if (j < a.n) {
			r = __ldg(&a.xyzq[j]);
			const float gx = fmaxf(fmaxf(lx - r.x, r.x - hx), 0.f), gy = fmaxf(fmaxf(ly - r.y, r.y - hy), 0.f),
					gz = fmaxf(fmaxf(lz - r.z, r.z - hz), 0.f);
			in = (__ldg(&a.tm[j]) & 0xffffu) != 0 && !(gx * gx + gy * gy + gz * gz > bd.brick);
		}
		const uint32_t m = __ballot_sync(0xffffffffu, in);
		if (lane == 0) warp_n[warp] = __popc(m);
		__syncthreads();
		uint32_t at = 0, n = 0;
#pragma unroll
		for (int w = 0; w < kTile / 32; ++w) {
			if (w < warp) at += warp_n[w];
			n += warp_n[w];
		}
		if (in) cand[at + __popc(m & ((1u << lane) - 1u))] = make_float4(r.x, r.y, r.z, __uint_as_float(j));
		__syncthreads();
		if (valid)
			for (uint32_t b = 0; b < n; ++b) {
				const float4 c = cand[b];
				const float dx = fx - c.x, dy = fy - c.y, dz = fz - c.z;
				const float d2 = dx * dx + dy * dy + dz * dz;
				if (d2 > bd.never) continue;
				if (!(d2 < bd.sure) && !nl_member(px, py, pz, c, a.cut2)) continue;
				if (FILL) dst[cnt] = __float_as_uint(c.w);
				++cnt;
			}
	}
	if (valid && !FILL) count[v] = cnt;
}

/* Exclusive prefix sums of the list lengths, three launches: sums of
 * kScanBlock voxels, their prefix (one block, 64-bit), and the voxels'
 * descriptors {numEl, idx} (src/model/NLGrid.h:151-165). */
constexpr int kScanThreads = 256;
constexpr int kScanPer = 16;
constexpr int kScanBlock = kScanThreads * kScanPer;

__device__ __forceinline__ unsigned long long block_sum(unsigned long long v) {
	__shared__ unsigned long long part[32];
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
	__syncthreads();
	v = 0;
	for (uint32_t w = 0; w < blockDim.x / 32; ++w) v += part[w];
	__syncthreads();
	return v;
}

__global__ void __launch_bounds__(kScanThreads) nl_block_sums_kernel(const uint32_t* __restrict__ count, size_t n,
		unsigned long long* __restrict__ sums) {
	unsigned long long v = 0;
	const size_t base = (size_t)blockIdx.x * kScanBlock;
#pragma unroll
	for (int k = 0; k < kScanPer; ++k) {
		const size_t i = base + (size_t)k * kScanThreads + threadIdx.x;
		if (i < n) v += count[i];
	}
	v = block_sum(v);
	if (threadIdx.x == 0) sums[blockIdx.x] = v;
}

/* sums[0 .. n) -> exclusive prefix, the total in sums[n] */
__global__ void __launch_bounds__(1024) nl_scan_sums_kernel(unsigned long long* __restrict__ sums, uint32_t n) {
	__shared__ unsigned long long part[1024];
	unsigned long long run = 0;
	for (uint32_t b = 0; b < n; b += 1024) {
		const uint32_t i = b + threadIdx.x;
		const unsigned long long v = i < n ? sums[i] : 0;
		part[threadIdx.x] = v;
		__syncthreads();
		for (int o = 1; o < 1024; o <<= 1) {
			const unsigned long long t = (int)threadIdx.x >= o ? part[threadIdx.x - o] : 0;
			__syncthreads();
			part[threadIdx.x] += t;
			__syncthreads();
		}
		if (i < n) sums[i] = run + part[threadIdx.x] - v;
		run += part[1023];
		__syncthreads();
	}
	if (threadIdx.x == 0) sums[n] = run;
}

__global__ void __launch_bounds__(kScanThreads) nl_desc_kernel(const uint32_t* __restrict__ count, size_t n,
		const unsigned long long* __restrict__ sums, uint2* __restrict__ desc) {
	__shared__ uint32_t warp_tot[kScanThreads / 32];
	uint32_t run = (uint32_t)sums[blockIdx.x];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (int k = 0; k < kScanPer; ++k) {
		const size_t i = (size_t)blockIdx.x * kScanBlock + (size_t)k * kScanThreads + threadIdx.x;
		const uint32_t c = i < n ? count[i] : 0;
		uint32_t incl = c;
#pragma unroll
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
			if (lane >= o) incl += t;
		}
		if (lane == 31) warp_tot[warp] = incl;
		__syncthreads();
		uint32_t before = 0, all = 0;
#pragma unroll
		for (int w = 0; w < kScanThreads / 32; ++w) {
			if (w < warp) before += warp_tot[w];
			all += warp_tot[w];
		}
		if (i < n) desc[i] = make_uint2(c, run + before + incl - c);
		run += all;
		__syncthreads();
	}
}

/* Layout as the CPU builder (double arithmetic, same formulas). */
void grid_layout(const std::vector<float>& xyz, uint32_t n, const gba_grid_build_opts& o,
		gba_intrpl_desc& inner, gba_intrpl_desc& outer, gba_nl_desc& nl) {
	const double s = o.spacing;
	inner.numGrids = outer.numGrids = o.n_alphabet + 1;
	for (int a = 0; a < 3; ++a) {
		const float* P = xyz.data() + (size_t)a * n;
		double lo = P[0], hi = P[0];
		for (uint32_t i = 1; i < n; ++i) { lo = std::min(lo, (double)P[i]); hi = std::max(hi, (double)P[i]); }
		lo -= o.margin;
		hi += o.margin;
		unsigned N = (unsigned)std::ceil((hi - lo) / s) + 1;
		inner.dimN[a] = N;
		inner.posMin[a] = (float)lo;
		/* ATTRACT stores the float inner origin and derives the outer one from
		 * it (readGridFromGridFile, src/fileIO/readFile.cpp:322-324) */
		outer.posMin[a] = (float)((double)inner.posMin[a] - o.outer_ext * s);
		outer.dimN[a] = (unsigned)std::ceil(((N - 1) * s + 2.0 * o.outer_ext * s) / (2 * s)) + 1;
		nl.dimN[a] = N;
		nl.posMin[a] = inner.posMin[a];
	}
	inner.gridSpacing = o.spacing;
	outer.gridSpacing = 2 * o.spacing;
	nl.gridSpacing = o.spacing;
	nl.dPlateau = o.plateau;
	nl.numEl = 0;
}

}  // namespace

}  // namespace gba

using namespace gba;

extern "C" int gba_build_grid(gba_ctx* ctx, gba_id rec, gba_id params,
		const gba_grid_build_opts* opt, gba_id* out) {
	if (!ctx) return GBA_ERR_INVALID_ARGUMENT;
	try {
		if (!opt || !out) throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_build_grid: null argument");
		if (!(opt->spacing > 0) || !(opt->plateau > 0) || !(opt->nl_cutoff > 0) || opt->n_alphabet > 98 ||
				opt->margin < 0)
			throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_build_grid: bad options");
		ctx->bind();
		ProteinItem* R;
		ParamsItem* P;
		{
			Lock g(ctx->mu);
			R = static_cast<ProteinItem*>(ctx->find(rec, ItemKind::Protein));
			P = static_cast<ParamsItem*>(ctx->find(params, ItemKind::Params));
		}
		if (R->max_type > P->dev.num_types)
			throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_build_grid: receptor type exceeds the table");
		for (uint32_t c = 0; c < opt->n_alphabet; ++c)
			if (opt->alphabet[c] > P->dev.num_types)
				throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_build_grid: alphabet type exceeds the table");
		auto item = std::make_unique<GridItem>();
		grid_layout(R->host_xyz, R->dev.n, *opt, item->inner_desc, item->outer_desc, item->nl_desc);
		const size_t Ni = (size_t)item->inner_desc.dimN[0] * item->inner_desc.dimN[1] * item->inner_desc.dimN[2];
		const size_t No = (size_t)item->outer_desc.dimN[0] * item->outer_desc.dimN[1] * item->outer_desc.dimN[2];
		const uint32_t C = opt->n_alphabet + 1;
		if ((double)C * std::max(Ni, No) > 4.0e9)
			throw ApiError(GBA_ERR_INVALID_ARGUMENT, "gba_build_grid: grid exceeds 2^32 float4");
		item->inner.alloc(Ni * C * sizeof(float4));
		item->outer.alloc(No * C * sizeof(float4));
		DevBuffer alpha;
		alpha.upload(opt->alphabet, std::max<size_t>(1, opt->n_alphabet) * sizeof(uint32_t));
		BuildArgs a{};
		a.xyzq = R->dev.xyzq;
		a.tm = R->dev.tm;
		a.n = R->dev.n;
		a.one = 1.0f;
		for (uint32_t c = 0; c < opt->n_alphabet; ++c)
			if (opt->alphabet[c] == 0) a.blank[c >> 5] |= 1u << (c & 31);
		a.par = P->dev;
		a.n_alphabet = opt->n_alphabet;
		a.plateau = opt->plateau;
		a.plat2 = opt->plateau * opt->plateau;
		a.cut2 = (double)opt->nl_cutoff * opt->nl_cutoff;
		cudaStream_t s = 0;
		/* whole blocks of channel warps, so that every warp's row loads stay inside */
		a.n_lj = (opt->n_alphabet + kBlockChan - 1) / kBlockChan * kBlockChan;
		const size_t nrow = (size_t)(a.par.num_types + 1) * a.n_lj;
		DevBuffer rows;
		rows.alloc(std::max<size_t>(1, nrow) * 2 * sizeof(float4));
		a.rows = (const float4*)rows.ptr;
		double reach2 = 0.0;      /* beads lie inside the outer grid's box */
		for (int k = 0; k < 3; ++k) {
			const double e = (item->outer_desc.dimN[k] + kCube) * (double)item->outer_desc.gridSpacing;
			reach2 += e * e;
		}
		const bool plain = plain_pairs(P->host_table, a.par.potshape, a.plat2, reach2);
		if (nrow > 0) {
			pair_rows_kernel<<<(unsigned)((nrow + 255) / 256), 256, 0, s>>>(a.par, (const uint32_t*)alpha.ptr, a.n_alphabet,
					a.n_lj, plain, (float4*)rows.ptr);
			check_cuda(cudaGetLastError(), "grid build: pair rows");
		}
		launch_potentials(a, plain, item->inner_desc, (float4*)item->inner.ptr, s);
		launch_potentials(a, plain, item->outer_desc, (float4*)item->outer.ptr, s);
		DevBuffer counts, sums;
		counts.alloc(Ni * sizeof(uint32_t));
		const gba_nl_desc& nd = item->nl_desc;
		uint64_t bricks = 1;
		double extent = 0.0;
		for (int k = 0; k < 3; ++k) {
			bricks *= (nd.dimN[k] + kBrick[k] - 1) / kBrick[k];
			const double lo = nd.posMin[k], hi = lo + (double)(nd.dimN[k] + kBrick[k]) * nd.gridSpacing;
			extent = std::max(extent, std::max(std::fabs(lo), std::fabs(hi)));
		}
		const NlBounds bd = nl_bounds(a.cut2, extent);
		nl_kernel<false><<<(unsigned)bricks, kTile, 0, s>>>(a, nd, bd, (uint32_t*)counts.ptr, nullptr, nullptr);
		check_cuda(cudaGetLastError(), "grid build: NL count launch");
		const uint32_t nsum = (uint32_t)((Ni + kScanBlock - 1) / kScanBlock);
		sums.alloc((nsum + 1) * sizeof(unsigned long long));
		item->nlgrid.alloc(Ni * sizeof(uint2));
		nl_block_sums_kernel<<<nsum, kScanThreads, 0, s>>>((const uint32_t*)counts.ptr, Ni, (unsigned long long*)sums.ptr);
		nl_scan_sums_kernel<<<1, 1024, 0, s>>>((unsigned long long*)sums.ptr, nsum);
		nl_desc_kernel<<<nsum, kScanThreads, 0, s>>>((const uint32_t*)counts.ptr, Ni, (const unsigned long long*)sums.ptr,
				(uint2*)item->nlgrid.ptr);
		check_cuda(cudaGetLastError(), "grid build: NL scan launch");
		uint64_t total = 0;
		check_cuda(cudaMemcpy(&total, (const unsigned long long*)sums.ptr + nsum, sizeof(total), cudaMemcpyDeviceToHost),
				"grid build: NL total");
		if (total > 0xffffffffull) throw ApiError(GBA_ERR_INVALID_ARGUMENT, "neighbour list exceeds 2^32 entries");
		item->nllist.alloc(std::max<uint64_t>(1, total) * sizeof(uint32_t));
		nl_kernel<true><<<(unsigned)bricks, kTile, 0, s>>>(a, nd, bd, nullptr, (const uint2*)item->nlgrid.ptr,
				(uint32_t*)item->nllist.ptr);
		check_cuda(cudaGetLastError(), "grid build: NL fill launch");
		item->nl_desc.numEl = (uint32_t)total;
		item->dev.inner = intrpl_from_desc(item->inner_desc);
		item->dev.inner.data = (const float4*)item->inner.ptr;
		item->dev.outer = intrpl_from_desc(item->outer_desc);
		item->dev.outer.data = (const float4*)item->outer.ptr;
		item->dev.nl = nl_from_desc(item->nl_desc);
		nl_ratio_table(item->dev.nl.dPlateau2, item->ratio);
		item->dev.nl.grid = (const uint2*)item->nlgrid.ptr;
		item->dev.nl.list = (const uint32_t*)item->nllist.ptr;
		item->dev.nl.ratio = (const float*)item->ratio.ptr;
		item->nl_max_index = R->dev.n - 1;
		item->nl_has_entries = total > 0;
		item->nl_list_radius = opt->nl_cutoff;
		check_cuda(cudaDeviceSynchronize(), "grid build");
		*out = ctx->add(std::move(item));
	} catch (const ApiError& e) {
		ctx->set_error(e.what());
		return e.code;
	} catch (const std::exception& e) {
		ctx->set_error(e.what());
		return GBA_ERR_INVALID_ARGUMENT;
	}
	return GBA_OK;
}

extern "C" int gba_grid_info(gba_ctx* ctx, gba_id grid, gba_intrpl_desc* inner,
		gba_intrpl_desc* outer, gba_nl_desc* nl) {
	if (!ctx) return GBA_ERR_INVALID_ARGUMENT;
	try {
		Lock g(ctx->mu);
		auto* G = static_cast<GridItem*>(ctx->find(grid, ItemKind::Grid));
		if (inner) *inner = G->inner_desc;
		if (outer) *outer = G->outer_desc;
		if (nl) *nl = G->nl_desc;
	} catch (const ApiError& e) {
		ctx->set_error(e.what());
		return e.code;
	}
	return GBA_OK;
}

extern "C" int gba_download_grid(gba_ctx* ctx, gba_id grid, float* inner, float* outer,
		gba_neighbour_desc* nl_grid, uint32_t* nl_list) {
	if (!ctx) return GBA_ERR_INVALID_ARGUMENT;
	try {
		ctx->bind();
		GridItem* G;
		{
			Lock g(ctx->mu);
			G = static_cast<GridItem*>(ctx->find(grid, ItemKind::Grid));
		}
		if (inner) check_cuda(cudaMemcpy(inner, G->inner.ptr, G->inner.bytes, cudaMemcpyDeviceToHost), "D2H");
		if (outer) check_cuda(cudaMemcpy(outer, G->outer.ptr, G->outer.bytes, cudaMemcpyDeviceToHost), "D2H");
		if (nl_grid) check_cuda(cudaMemcpy(nl_grid, G->nlgrid.ptr, G->nlgrid.bytes, cudaMemcpyDeviceToHost), "D2H");
		if (nl_list && G->nl_desc.numEl)
			check_cuda(cudaMemcpy(nl_list, G->nllist.ptr, (size_t)G->nl_desc.numEl * 4, cudaMemcpyDeviceToHost), "D2H");
	} catch (const ApiError& e) {
		ctx->set_error(e.what());
		return e.code;
	}
	return GBA_OK;
}

/* ---- duplicated-octet layout ---------------------------------------------- */

namespace gba {
namespace {

__global__ void build_octets_kernel(const float4* __restrict__ src, uint32_t Nx, uint32_t Ny,
		uint32_t Nz, uint32_t C, float4* __restrict__ dst) {
	const size_t nocts = (size_t)(Nx - 1) * (Ny - 1) * (Nz - 1);
	const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= nocts * C) return;
	const size_t c = t / nocts, o = t % nocts;
	const uint32_t x = (uint32_t)(o % (Nx - 1));
	const uint32_t y = (uint32_t)((o / (Nx - 1)) % (Ny - 1));
	const uint32_t z = (uint32_t)(o / ((size_t)(Nx - 1) * (Ny - 1)));
	const size_t sxy = (size_t)Nx * Ny;
	const float4* b = src + c * sxy * Nz + (size_t)Nx * ((size_t)z * Ny + y) + x;
	float4* d = dst + 8 * t;
	d[0] = b[0];
	d[1] = b[1];
	d[2] = b[Nx];
	d[3] = b[Nx + 1];
	d[4] = b[sxy];
	d[5] = b[sxy + 1];
	d[6] = b[sxy + Nx];
	d[7] = b[sxy + Nx + 1];
}

void make_octets(const gba_intrpl_desc& d, const DevBuffer& src, DevBuffer& dst) {
	const size_t nocts = (size_t)(d.dimN[0] - 1) * (d.dimN[1] - 1) * (d.dimN[2] - 1);
	const size_t total = nocts * d.numGrids;
	dst.alloc(total * 8 * sizeof(float4));
	build_octets_kernel<<<(unsigned)((total + 255) / 256), 256>>>((const float4*)src.ptr, d.dimN[0],
			d.dimN[1], d.dimN[2], d.numGrids, (float4*)dst.ptr);
	check_cuda(cudaGetLastError(), "octet layout");
}

}  // namespace
}  // namespace gba

extern "C" int gba_grid_octets(gba_ctx* ctx, gba_id grid, int enable) {
	if (!ctx) return GBA_ERR_INVALID_ARGUMENT;
	try {
		ctx->bind();
		Lock lk(ctx->stage_mu);
		Lock g(ctx->mu);
		auto* G = static_cast<GridItem*>(ctx->find(grid, ItemKind::Grid));
		if (enable) {
			if (!G->inner_oct.ptr) make_octets(G->inner_desc, G->inner, G->inner_oct);
			if (!G->outer_oct.ptr) make_octets(G->outer_desc, G->outer, G->outer_oct);
			check_cuda(cudaDeviceSynchronize(), "octet layout");
		} else {
			G->inner_oct.release();
			G->outer_oct.release();
		}
		G->dev.inner.oct = (const float4*)G->inner_oct.ptr;
		G->dev.outer.oct = (const float4*)G->outer_oct.ptr;
		/* cached device copies of the pair descriptors hold the old pointers */
		ctx->model_cache.clear();
		ctx->clear_graphs();
	} catch (const ApiError& e) {
		ctx->set_error(e.what());
		return e.code;
	} catch (const std::exception& e) {
		ctx->set_error(e.what());
		return GBA_ERR_INVALID_ARGUMENT;
	}
	return GBA_OK;
}
