/*
 * va13.cuh -- the VA13 variable-metric minimizer as a resumable state machine.
 *
 * Follows the Harwell routine the reference runs for every pose
 * (src/apps/em/minfor.f:1-182 with mc11a/mc11e, src/apps/em/mc11a.f:1-143),
 * in FP64 like the Fortran's real*8, generalised from its fixed 6 DOF to n DOF.
 * Instead of calling the energy function, the machine stops whenever minfor
 * would call it: `point()` is the DOF vector to evaluate, `provide(f, g)` hands
 * back the objective and gradient and runs to the next evaluation (or to the
 * end).  The host (plain per-step driver) runs `provide`; the device kernels
 * run `provide_w`, the same arithmetic spread over a warp's lanes (the warp
 * form, below), which takes the same trajectory bit for bit.  Arrays are
 * 1-based, mirroring the Fortran.
 */
#ifndef GBA_VA13_CUH_
#define GBA_VA13_CUH_

#include <cmath>

#ifdef __CUDACC__
#define GBA_HD __host__ __device__ __forceinline__
#else
#define GBA_HD inline
#endif

/* Device code of the machine stays small: its loops rolled, its divisions in
 * one function (va_div), mc11a there once.  It runs between two evaluations,
 * the warps of an SM are spread over both, and what the instruction cache
 * does not hold every one of them waits for (8,000 poses of a 120-bead ligand,
 * 40 evaluations: 159 KB of code 13.4 ms, 15 of 27 cycles per instruction
 * waiting for it; 97 KB 10.2 ms, 9 of 21). */
#ifdef __CUDA_ARCH__
#define GBA_VA_LOOP _Pragma("unroll 1")
#else
#define GBA_VA_LOOP
#endif

namespace gba {

/* max, min and abs with the C++ library's semantics (std::max(a, b) =
 * a < b ? b : a, std::min(a, b) = b < a ? b : a, fabs clears the sign bit),
 * which decide what a NaN or a signed zero does: a pose whose energy
 * overflows hands the machine NaN gradients, and every form of the
 * minimizer must take the same branch on them. */
GBA_HD double va_max(double a, double b) { return a < b ? b : a; }
GBA_HD double va_min(double a, double b) { return b < a ? b : a; }
GBA_HD double va_abs(double a) { return fabs(a); }

/* Division of the warp form: out of line on the device (sixteen places of a
 * step divide). */
#ifdef __CUDACC__
static __device__ __noinline__ double va_div_device(double x, double y) { return x / y; }
#endif
GBA_HD double va_div(double x, double y) {
#ifdef __CUDA_ARCH__
	return va_div_device(x, y);
#else
	return x / y;
#endif
}

/* Products are never contracted with a following add: the host build runs
 * with -ffp-contract=off and the device uses round-to-nearest multiplies, so
 * both sides take bit-identical steps (nvcc would otherwise form FMAs). */
GBA_HD double vm(double a, double b) {
#ifdef __CUDA_ARCH__
	return __dmul_rn(a, b);
#else
	return a * b;
#endif
}

/* mc11a: rank-one update of the packed LDL^T factors (mc11a.f:1-112). */
GBA_HD void mc11a(double* a, int n, double* z, double sig, double* w, int& ir, int mk, double eps) {
	double ti = 0, v, tim, b, r, y, gm, al;
	int np, ij = 1, ip, mm, j;
	if (n > 1) goto L1;
	a[1] = a[1] + vm(vm(sig, z[1]), z[1]);
	ir = 1;
	if (a[1] > 0.0) return;
	a[1] = 0.0;
	ir = 0;
	return;
L1:
	np = n + 1;
	if (sig > 0.0) goto L40;
	if (sig == 0.0 || ir == 0) return;
	ti = 1.0 / sig;
	ij = 1;
	if (mk == 0) goto L10;
	GBA_VA_LOOP
	for (int i = 1; i <= n; ++i) {
		if (a[ij] != 0.0) ti = ti + vm(w[i], w[i]) / a[ij];
		ij = ij + np - i;
	}
	goto L20;
L10:
	GBA_VA_LOOP
	for (int i = 1; i <= n; ++i) w[i] = z[i];
	GBA_VA_LOOP
	for (int i = 1; i <= n; ++i) {
		ip = i + 1;
		v = w[i];
		if (a[ij] > 0.0) {
			ti = ti + vm(v, v) / a[ij];
			if (i != n)
				for (j = ip; j <= n; ++j) {
					ij = ij + 1;
					w[j] = w[j] - vm(v, a[ij]);
				}
			ij = ij + 1;
		} else {
			w[i] = 0.0;
			ij = ij + np - i;
		}
	}
L20:
	if (ir <= 0) {
		ti = 0.;
		ir = -ir - 1;
		goto L23;
	}
	if (ti > 0.0) {
		ti = eps / sig;
		if (eps == 0.0) ir = ir - 1;
		goto L23;
	}
	if (mk - 1 <= 0) goto L40;
L23:
	mm = 1;
	tim = ti;
	GBA_VA_LOOP
	for (int i = 1; i <= n; ++i) {
		j = np - i;
		ij = ij - i;
		if (a[ij] != 0.0) tim = ti - vm(w[j], w[j]) / a[ij];
		w[j] = ti;
		ti = tim;
	}
	goto L41;
L40:
	mm = 0;
	tim = 1.0 / sig;
L41:
	ij = 1;
	GBA_VA_LOOP
	for (int i = 1; i <= n; ++i) {
		ip = i + 1;
		v = z[i];
		if (!(a[ij] > 0.0)) {
			if (ir > 0 || sig < 0.0 || v == 0.0) {
				ti = tim;
				ij = ij + np - i;
				continue;
			}
			ir = 1 - ir;
			a[ij] = vm(v, v) / tim;
			if (i == n) return;
			GBA_VA_LOOP
			for (j = ip; j <= n; ++j) {
				ij = ij + 1;
				a[ij] = z[j] / v;
			}
			return;
		}
		al = v / a[ij];
		if (mm <= 0) ti = tim + vm(v, al);
		else ti = w[i];
		r = ti / tim;
		a[ij] = vm(a[ij], r);
		if (r == 0.0) break;
		if (i == n) break;
		b = al / ti;
		if (r > 4.0) {
			gm = tim / ti;
			GBA_VA_LOOP
			for (j = ip; j <= n; ++j) {
				ij = ij + 1;
				y = a[ij];
				a[ij] = vm(b, z[j]) + vm(y, gm);
				z[j] = z[j] - vm(v, y);
			}
		} else {
			GBA_VA_LOOP
			for (j = ip; j <= n; ++j) {
				ij = ij + 1;
				z[j] = z[j] - vm(v, a[ij]);
				a[ij] = a[ij] + vm(b, z[j]);
			}
		}
		tim = ti;
		ij = ij + 1;
	}
	if (ir < 0) ir = -ir;
}

/* mc11e: solves with the packed factors (entry mc11e, mc11a.f:114-142). */
GBA_HD void mc11e(const double* a, int n, double* z, double* w, int ir) {
	if (ir < n) return;
	w[1] = z[1];
	if (n <= 1) {
		z[1] = z[1] / a[1];
		return;
	}
	int ij = 0;
	GBA_VA_LOOP
	for (int i = 2; i <= n; ++i) {
		ij = i;
		double v = z[i];
		GBA_VA_LOOP
		for (int j = 1; j <= i - 1; ++j) {
			v = v - vm(a[ij], z[j]);
			ij = ij + n - j;
		}
		w[i] = v;
		z[i] = v;
	}
	z[n] = z[n] / a[ij];
	const int np = n + 1;
	GBA_VA_LOOP
	for (int nip = 2; nip <= n; ++nip) {
		const int i = np - nip;
		int ii = ij - nip;
		double v = z[i] / a[ii];
		ij = ii;
		GBA_VA_LOOP
		for (int j = i + 1; j <= n; ++j) {
			ii = ii + 1;
			v = v - vm(a[ii], z[j]);
		}
		z[i] = v;
	}
}

/* ---- the warp form ----------------------------------------------------
 * On GB300 every FP64 instruction a warp issues occupies the narrow FP64
 * pipe for the whole warp, whether one lane or 32 take part, so the machine
 * run by one lane costs what its ~650 FP64 instructions per step cost.  The
 * warp form runs the same arithmetic with every lane of the warp:
 * - scalar work is done redundantly by all lanes (same operands, same
 *   results), so it costs no more than on one lane;
 * - element-wise updates (element j on lane j) take one instruction for all
 *   elements instead of one per element;
 * - divisions that do not depend on each other are issued together on
 *   separate lanes.
 * Each element sees the same operations in the same order as in mc11a,
 * mc11e and minfor, so the trajectory is the same bit for bit.
 *
 * Executors.  `each(lo, hi, f)` runs f(j) for the elements j in [lo, hi]:
 * on the device on lanes lo..hi between two __syncwarp()s; on the host (the
 * tests) in DESCENDING order, so that an element that depended on another
 * element of the same section would change the trajectory.  `halves(f)` runs
 * f(h, k) on lane k of each half warp h, `per_half(f)` f(h) on every lane of
 * it; what a half keeps between sections is its lanes' own (state(h): the
 * host keeps both), and second() is half 1's value for all.  Shared state is
 * written only inside `each` (so no lane can read a location in scalar code
 * while another lane writes it); scalar code between sections only reads. */
struct VaSerial {
	GBA_HD void sync() const {}
	template <class F>
	GBA_HD void each(int lo, int hi, F f) const {
		for (int j = hi; j >= lo; --j) f(j);
	}
	template <class F>
	GBA_HD void halves(F f) const {
		for (int h = 1; h >= 0; --h)
			for (int k = 15; k >= 0; --k) f(h, k);
	}
	template <class F>
	GBA_HD void per_half(F f) const {
		f(1);
		f(0);
	}
	GBA_HD int state(int h) const { return h; }
	GBA_HD int second(int, int of1) const { return of1; }
};

struct VaWarp {
	int lane;
	/* lane k of half h; on the host as VaSerial */
	template <class F>
	GBA_HD void halves(F f) const {
#ifdef __CUDA_ARCH__
		__syncwarp();
		f(lane >> 4, lane & 15);
		__syncwarp();
#else
		VaSerial{}.halves(f);
#endif
	}
	template <class F>
	GBA_HD void per_half(F f) const {
#ifdef __CUDA_ARCH__
		f(lane >> 4);
#else
		VaSerial{}.per_half(f);
#endif
	}
	GBA_HD int state(int h) const {
#ifdef __CUDA_ARCH__
		return 0;
#else
		return h;
#endif
	}
	GBA_HD int second(int own, int of1) const {
#ifdef __CUDA_ARCH__
		return __shfl_sync(0xffffffffu, own, 16);
#else
		return of1;
#endif
	}
	GBA_HD void sync() const {
#ifdef __CUDA_ARCH__
		__syncwarp();
#endif
	}
	template <class F>
	GBA_HD void each(int lo, int hi, F f) const {
#ifdef __CUDA_ARCH__
		__syncwarp();
		if (lane >= lo && lane <= hi) f(lane);
		__syncwarp();
#else
		for (int j = hi; j >= lo; --j) f(j);
#endif
	}
};

/* index of diagonal entry i in the packed upper triangle (row-major, rows of
 * n, n-1, ... entries; 1-based) */
GBA_HD int va_diag(int i, int n) { return (i - 1) * (2 * n - i + 2) / 2 + 1; }

/* mc11a in the warp form (every lane calls it; ir in and out on every lane;
 * q, t: scratch of n + 1 doubles).  Beyond the element-wise updates:
 * - the first loop (mk != 0) only feeds ti, which ir <= 0 discards at L20
 *   (minfor's first call always has ir = -n): it runs only for ir > 0, its
 *   divisions together;
 * - the divisions of the L23 recurrence, w_j^2 / a_jj, depend only on the
 *   entry values: all at once;
 * - in the L41 loop, r = ti/tim, b = al/ti, gm = tim/ti and the next row's
 *   al = (z_{i+1} - v a_{i,i+1}) / a_{i+1,i+1} -- z_{i+1} after this row's
 *   update, which both branches compute as z - v * (old a) -- in one
 *   division on four lanes. */
template <class X>
GBA_HD void mc11a_w(double* a, int n, double* z, double sig, double* w, int& ir, int mk, double eps, double* q,
		double* t, const X& ex) {
	if (n <= 1) {
		const double a1 = a[1] + vm(vm(sig, z[1]), z[1]);
		ex.each(1, 1, [&](int) { a[1] = a1 > 0.0 ? a1 : 0.0; });
		ir = a1 > 0.0 ? 1 : 0;
		return;
	}
	const int np = n + 1;
	double ti = 0.0, tim = 0.0;
	int mm = 0;
	if (sig > 0.0) goto L40;
	if (sig == 0.0 || ir == 0) return;
	ti = va_div(1.0, sig);
	if (mk == 0) goto L10;
	if (ir > 0) {
		ex.each(1, n, [&](int j) {
			const double dj = a[va_diag(j, n)];
			q[j] = dj != 0.0 ? va_div(vm(w[j], w[j]), dj) : 0.0;
		});
		GBA_VA_LOOP
		for (int i = 1; i <= n; ++i)
			if (a[va_diag(i, n)] != 0.0) ti = ti + q[i];
	}
	goto L20;
L10:
	ex.each(1, n, [&](int j) { w[j] = z[j]; });
	GBA_VA_LOOP
	for (int i = 1; i <= n; ++i) {
		const int ij = va_diag(i, n);
		const double v = w[i];
		if (a[ij] > 0.0) {
			ti = ti + va_div(vm(v, v), a[ij]);
			if (i != n) ex.each(i + 1, n, [&](int j) { w[j] = w[j] - vm(v, a[ij + j - i]); });
		} else {
			ex.each(i, i, [&](int) { w[i] = 0.0; });
		}
	}
L20:
	if (ir <= 0) {
		ti = 0.;
		ir = -ir - 1;
		goto L23;
	}
	if (ti > 0.0) {
		ti = va_div(eps, sig);
		if (eps == 0.0) ir = ir - 1;
		goto L23;
	}
	if (mk - 1 <= 0) goto L40;
L23:
	mm = 1;
	ex.each(1, n, [&](int j) {
		const double dj = a[va_diag(j, n)];
		q[j] = dj != 0.0 ? va_div(vm(w[j], w[j]), dj) : 0.0;
	});
	tim = ti;
	GBA_VA_LOOP
	for (int i = 1; i <= n; ++i) {
		const int j = np - i;
		if (a[va_diag(j, n)] != 0.0) tim = ti - q[j];
		ex.each(0, 0, [&](int) { t[j] = ti; });
		ti = tim;
	}
	ex.each(1, n, [&](int j) { w[j] = t[j]; });
	goto L41;
L40:
	mm = 0;
	tim = va_div(1.0, sig);
L41: {
	bool have_al = false;
	double al = 0.0;
	GBA_VA_LOOP
	for (int i = 1; i <= n; ++i) {
		const int ij = va_diag(i, n);
		const double v = z[i];
		const double aii = a[ij];
		if (!(aii > 0.0)) {
			if (ir > 0 || sig < 0.0 || v == 0.0) {
				ti = tim;
				have_al = false;
				continue;
			}
			ir = 1 - ir;
			ex.each(i, n, [&](int j) {
				if (j == i) a[ij] = va_div(vm(v, v), tim);
				else a[ij + j - i] = va_div(z[j], v);
			});
			return;
		}
		if (!have_al) al = va_div(v, aii);
		if (mm <= 0) ti = tim + vm(v, al);
		else ti = w[i];
		ex.each(0, 3, [&](int k) {
			double nu = ti, de = tim;                     /* r */
			if (k == 1) { nu = al; de = ti; }             /* b */
			else if (k == 2) { nu = tim; de = ti; }       /* gm */
			else if (k == 3) {                            /* the next row's al */
				nu = 0.0;
				de = 1.0;
				if (i < n) {
					nu = z[i + 1] - vm(v, a[ij + 1]);
					de = a[va_diag(i + 1, n)];
				}
			}
			q[k] = va_div(nu, de);
		});
		const double r = q[0], b = q[1], gm = q[2];
		al = q[3];
		have_al = true;
		if (r == 0.0 || i == n) {
			ex.each(i, i, [&](int) { a[ij] = vm(aii, r); });
			break;
		}
		if (r > 4.0) {
			ex.each(i, n, [&](int j) {
				if (j == i) {
					a[ij] = vm(aii, r);
					return;
				}
				const int k = ij + j - i;
				const double y = a[k];
				a[k] = vm(b, z[j]) + vm(y, gm);
				z[j] = z[j] - vm(v, y);
			});
		} else {
			ex.each(i, n, [&](int j) {
				if (j == i) {
					a[ij] = vm(aii, r);
					return;
				}
				const int k = ij + j - i;
				z[j] = z[j] - vm(v, a[k]);
				a[k] = a[k] + vm(b, z[j]);
			});
		}
		tim = ti;
	}
}
	if (ir < 0) ir = -ir;
}

/* minfor's two updates of one step, mc11a(a, n, z0, 1 / dga, w, ir = -n, 1, 0)
 * and, with its ir negated, mc11a(a, n, z1, 1 / den, z1, ir, 0, 0), side by side: the
 * first on half warp 0, the second two rows behind it on half 1, so that a
 * row's division and its elements' updates are one instruction for both.
 * Returns the second's ir.  For n >= 2 and 0 > dga, den > 0, both finite, when
 * - the first starts with ir = -n: ti is 0 at L23 (its 1 / sig is not needed),
 *   ir is n - 1 > 0 from there on, and a row whose diagonal entry is not
 *   positive is passed over;
 * - the second starts at L40 with ir = 1 - n: such a row ends it (with ir = n)
 *   unless z_i is 0.
 * Every element sees the operations of mc11a in their order.  A row's
 * al = z_i / a_ii comes with the row before it (row 0: z_1 / a_11); half 1
 * reads rows that half 0 has left.  w and q, t: its results are not used after.
 * About 21 FP64 instructions a row, nine of them the division: 8 rows and one
 * division before them a step for n = 6, where one update after the other took
 * 12 rows and seven.  1,000 poses, 500/200 beads, 100 evaluations 4.84 ->
 * 4.61 ms; 8,000, 400/120, 40: 9.80 -> 9.19; 12,000 of four pairs, 1,500/600,
 * 40: 23.7 -> 22.8. */
template <class X>
GBA_HD int mc11a_pair_w(double* a, int n, double* z0, double* z1, double den, double* w, double* q, double* t,
		const X& ex) {
	enum Mode { kIdle, kStart, kSkip, kRow, kFill };
	struct Half {
		double tim, al, v, aii, ti;
		Mode mode;
		int ij, ir;
		bool active;
	} st[2];
	/* L23's quotients; z_1 / a_11; sig of the second */
	ex.each(0, n + 1, [&](int j) {
		const double dj = a[va_diag(j < 1 || j > n ? 1 : j, n)];
		double nu = j > n ? 1.0 : z0[1], de = j > n ? den : dj;
		if (j >= 1 && j <= n) nu = vm(w[j], w[j]);
		const double x = va_div(nu, de);
		if (j > n) t[0] = x;
		else q[j] = j == 0 || dj != 0.0 ? x : 0.0;
	});
	const double sig = t[0], al0 = q[0];
	/* L23: t_j = the ti of row j, t_0 the tim that the rows begin with */
	ex.each(0, n, [&](int j) {
		double ti = 0.0;
		GBA_VA_LOOP
		for (int m = n; m > j; --m) ti = ti - q[m];
		t[j] = ti;
	});
	ex.per_half([&](int h) {
		Half& S = st[ex.state(h)];
		S.tim = h == 0 ? t[0] : sig;
		S.al = al0;
		S.v = S.aii = S.ti = 0.0;
		S.mode = kIdle;
		S.ij = 0;
		S.ir = 1 - n;
		S.active = true;
	});
	GBA_VA_LOOP
	for (int s = 1; s <= n + 2; ++s) {
		ex.per_half([&](int h) {
			Half& S = st[ex.state(h)];
			const int i = s - 2 * h;
			S.mode = !S.active || i > n ? kIdle : i < 0 ? kStart : kSkip;
			if (S.mode != kSkip || i < 1) return;
			const double* z = h == 0 ? z0 : z1;
			S.ij = va_diag(i, n);
			S.v = z[i];
			S.aii = a[S.ij];
			if (S.aii > 0.0) {
				S.mode = kRow;
				S.ti = h == 0 ? t[i] : S.tim + vm(S.v, S.al);
			} else if (h == 1 && S.v != 0.0) {
				S.mode = kFill;
			}
		});
		ex.halves([&](int h, int k) {
			const Half& S = st[ex.state(h)];
			const int i = s - 2 * h, j = k + 1;
			const bool fill = S.mode == kFill;
			if (S.mode == kIdle || (fill ? j < i || j > n : k > 3)) return;
			const double* z = h == 0 ? z0 : z1;
			double nu = S.ti, de = S.tim;                          /* r; kStart: tim */
			if (fill) {
				nu = j == i ? vm(S.v, S.v) : z[j];
				if (j != i) de = S.v;
			} else if (S.mode == kStart) {
				nu = 1.0;
			} else if (k == 1) {                                   /* b */
				nu = S.al;
				de = S.ti;
			} else if (k == 2) {                                   /* gm */
				nu = S.tim;
				de = S.ti;
			} else if (k == 3) {                                   /* the next row's al */
				nu = 0.0;
				de = 1.0;
				if (i < n) {
					nu = z[i + 1];
					if (S.mode == kRow) nu = nu - vm(S.v, a[S.ij + 1]);
					de = a[va_diag(i + 1, n)];
				}
			}
			(fill ? a + S.ij + j - i : (h == 0 ? q : w) + k)[0] = va_div(nu, de);
		});
		ex.halves([&](int h, int k) {
			const Half& S = st[ex.state(h)];
			const int i = s - 2 * h, j = k + 1;
			if (S.mode != kRow || j < i || j > n) return;
			const double* out = h == 0 ? q : w;
			double* z = h == 0 ? z0 : z1;
			const double r = out[0], b = out[1], gm = out[2];
			double* aj = a + S.ij + j - i;
			if (j == i) {
				*aj = vm(S.aii, r);
				return;
			}
			if (r == 0.0) return;
			const double y = *aj, zj = z[j] - vm(S.v, y);
			*aj = r > 4.0 ? vm(b, z[j]) + vm(y, gm) : y + vm(b, zj);
			z[j] = zj;
		});
		ex.per_half([&](int h) {
			Half& S = st[ex.state(h)];
			const double* out = h == 0 ? q : w;
			if (S.mode == kStart) S.tim = out[0];
			if (S.mode == kFill) {
				S.active = false;
				S.ir = n;
			}
			if (S.mode == kRow || S.mode == kSkip) S.al = out[3];
			if (S.mode == kRow) {
				if (out[0] == 0.0) S.active = false;
				S.tim = S.ti;
			}
		});
	}
	const int ir = ex.second(st[ex.state(0)].ir, st[ex.state(1)].ir);
	return ir < 0 ? -ir : ir;
}

/* mc11e in the warp form (q, t: scratch of n + 1 doubles).  The forward
 * substitution by columns: after z_j is final, lanes i > j subtract
 * a(j,i) z_j, so each z_i meets a(1,i) z_1, a(2,i) z_2, ... in the row
 * form's order.  The back substitution's divisions z_i / a_ii use the
 * forward values and go together; each row's products go together, its
 * differences stay a chain in the row form's order. */
template <class X>
GBA_HD void mc11e_w(const double* a, int n, double* z, double* w, int ir, double* q, double* t, const X& ex) {
	if (ir < n) return;
	if (n <= 1) {
		ex.each(1, 1, [&](int) {
			w[1] = z[1];
			z[1] = va_div(z[1], a[1]);
		});
		return;
	}
	GBA_VA_LOOP
	for (int j = 1; j < n; ++j) {
		const double zj = z[j];
		const int dj = va_diag(j, n);
		ex.each(j + 1, n, [&](int i) {
			z[i] = z[i] - vm(a[dj + i - j], zj);
			if (i == j + 1) w[i] = z[i];
		});
	}
	/* the divisions; z_n's is its result; the products of row n - 1 */
	const int dm = va_diag(n - 1, n);
	ex.each(1, n, [&](int i) {
		if (i == 1) w[1] = z[1];
		q[i] = va_div(z[i], a[va_diag(i, n)]);
		if (i == n) {
			z[n] = q[n];
			t[n] = vm(a[dm + 1], q[n]);
		}
	});
	GBA_VA_LOOP
	for (int i = n - 1; i >= 1; --i) {
		double v = q[i];
		GBA_VA_LOOP
		for (int j = i + 1; j <= n; ++j) v = v - t[j];
		/* z_i final; the products of row i - 1 (z_i's from v) */
		const int dp = i > 1 ? va_diag(i - 1, n) : 0;
		ex.each(i, n, [&](int j) {
			if (j == i) z[i] = v;
			if (i > 1) t[j] = vm(a[dp + j - (i - 1)], j == i ? v : z[j]);
		});
	}
}

/* minfor (minfor.f:1-182) as a machine stopped at each energy call. */
template <int NMAX>
struct VA13 {
	enum Phase { kInit = 0, kAfterFirst = 1, kAfterLine = 2, kDone = 3 };
	int phase, jn, ivmax, nfun, itr, isfv, ir;
	double gesa, c, acc, dff, dgb, fa, fb, fmin, gmin, dga;
	double step, stepbd, steplb, stmin;
	double h[NMAX * (NMAX + 1) / 2 + 1];
	double x[NMAX + 1], g[NMAX + 1], ga[NMAX + 1], gb[NMAX + 1], w[NMAX + 1];
	double xaa[NMAX + 1], xbb[NMAX + 1], d[NMAX + 1];
	double q[NMAX + 1], t[NMAX + 1];   /* scratch of the warp form */

	/* minfor.f:31-61 up to the first energy call */
	GBA_HD void start(const double* x0, int n, int max_eval) {
		jn = n;
		ivmax = max_eval;
		const double xnull = 0.0;
		dga = xnull;
		GBA_VA_LOOP
		for (int i = 1; i <= jn; ++i) {
			x[i] = x0[i - 1];
			ga[i] = xnull;
			d[i] = xnull;
			xaa[i] = x[i];
		}
		nfun = 0;
		itr = 0;
		const int np = jn + 1;
		acc = 0.000000001;
		c = 1.0;
		int k = (jn * np) / 2;
		GBA_VA_LOOP
		for (int i = 1; i <= k; ++i) h[i] = xnull;
		k = 1;
		GBA_VA_LOOP
		for (int i = 1; i <= jn; ++i) {
			h[k] = vm(0.01, c);
			k = k + np - i;
		}
		dff = xnull;
		phase = kAfterFirst;
	}

	GBA_HD bool done() const { return phase == kDone; }

	/* The DOF vector (0-based view) minfor evaluates next. */
	GBA_HD const double* point() const { return phase == kAfterFirst ? xaa + 1 : xbb + 1; }

	/* Hands back f and grad (0-based) at point(); runs to the next call. */
	GBA_HD void provide(double f, const double* grad) {
		const double xnull = 0.0;
		int i;
		if (phase == kAfterFirst) {
			gesa = f;
			GBA_VA_LOOP
			for (i = 1; i <= jn; ++i) g[i] = grad[i - 1];
			goto L110;
		}
		if (phase != kAfterLine) return;
		fb = f;
		GBA_VA_LOOP
		for (i = 1; i <= jn; ++i) gb[i] = grad[i - 1];
		/* minfor.f:114-144 */
		isfv = isfv < 2 ? isfv : 2;
		if (fb > gesa) goto L220;
		if (fb < gesa) goto L200;
		{
			double gl1 = xnull, gl2 = xnull;
			GBA_VA_LOOP
			for (i = 1; i <= jn; ++i) {
				gl1 = gl1 + vm(g[i], g[i]);
				gl2 = gl2 + vm(gb[i], gb[i]);
			}
			if (gl2 >= gl1) goto L220;
		}
	L200:
		isfv = 3;
		gesa = fb;
		GBA_VA_LOOP
		for (i = 1; i <= jn; ++i) {
			x[i] = xbb[i];
			g[i] = gb[i];
		}
	L220:
		dgb = xnull;
		GBA_VA_LOOP
		for (i = 1; i <= jn; ++i) dgb = dgb + vm(gb[i], d[i]);
		if (fb - fa <= vm(vm(0.1, c), dga)) goto L280;
		if (step > steplb) goto L270;
	L240:
		if (isfv >= 2) goto L110;
		phase = kDone;
		return;
	L270:
		stepbd = step;
		c = gmin + dgb - vm(3.0, fb - fmin) / step;
		c = gmin / (c + gmin - sqrt(vm(c, c) - vm(gmin, dgb)));
		step = vm(step, va_max(0.1, c));
		goto L170;
	L280:
		stepbd = stepbd - step;
		stmin = c;
		fmin = fb;
		gmin = dgb;
		step = vm(9.0, stmin);
		if (stepbd > xnull) step = vm(0.5, stepbd);
		c = dga + vm(3.0, dgb) - vm(4.0, fb - fa) / stmin;
		if (c > xnull) step = va_min(step, vm(stmin, va_max(1.0, -dgb / c)));
		if (dgb < vm(0.7, dga)) goto L170;
		isfv = 4 - isfv;
		if (stmin + step <= steplb) goto L240;
		ir = -jn;
		GBA_VA_LOOP
		for (i = 1; i <= jn; ++i) {
			xaa[i] = xbb[i];
			xbb[i] = ga[i];
			d[i] = gb[i] - ga[i];
			ga[i] = gb[i];
		}
		mc11a(h, jn, xbb, 1.0 / dga, w, ir, 1, xnull);
		ir = -ir;
		mc11a(h, jn, d, 1.0 / vm(stmin, dgb - dga), d, ir, 0, xnull);
		if (ir < jn) {
			phase = kDone;
			return;
		}
		dff = fa - fb;
		fa = fb;
		goto L135;
	L110:
		fa = gesa;
		isfv = 1;
		GBA_VA_LOOP
		for (i = 1; i <= jn; ++i) ga[i] = g[i];
	L135:
		itr = itr + 1;
		GBA_VA_LOOP
		for (i = 1; i <= jn; ++i) d[i] = -ga[i];
		mc11e(h, jn, d, w, jn);
		c = xnull;
		dga = xnull;
		GBA_VA_LOOP
		for (i = 1; i <= jn; ++i) {
			c = va_max(c, va_abs(d[i]));
			dga = dga + vm(ga[i], d[i]);
		}
		if (dga >= xnull) goto L240;
		stmin = xnull;
		stepbd = xnull;
		steplb = acc / c;
		fmin = fa;
		gmin = dga;
		step = 1.0;
		if (dff <= xnull) step = va_min(step, 1.0 / c);
		if (dff > xnull) step = va_min(step, (dff + dff) / (-dga));
	L170:
		c = stmin + step;
		if (nfun >= ivmax) {
			phase = kDone;
			return;
		}
		nfun = nfun + 1;
		GBA_VA_LOOP
		for (i = 1; i <= jn; ++i) xbb[i] = xaa[i] + vm(c, d[i]);
		phase = kAfterLine;
	}

	/* provide() in the warp form (see VaWarp): every lane of the warp calls
	 * it, the state in memory all lanes read (shared memory).  grad(j) is
	 * gradient element j (1-based), called on the lane that owns element j.
	 * The scalars live in registers, identical on every lane, and go back to
	 * the state at the end. */
	template <class X, class Grad>
	GBA_HD void provide_w(double f, Grad grad, const X& ex) {
		static_assert(NMAX >= 3 && NMAX <= 31, "one lane per element; four division lanes");
		ex.sync();   /* start() or the last step wrote the state */
		int phase = this->phase;
		if (phase != kAfterFirst && phase != kAfterLine) return;
		const int jn = this->jn, ivmax = this->ivmax;
		const double acc = this->acc;
		int nfun = this->nfun, itr = this->itr, isfv = this->isfv, ir = this->ir;
		double gesa = this->gesa, c = this->c, dff = this->dff, dgb = this->dgb, fa = this->fa, fb = this->fb;
		double fmin = this->fmin, gmin = this->gmin, dga = this->dga;
		double step = this->step, stepbd = this->stepbd, steplb = this->steplb, stmin = this->stmin;
		const double xnull = 0.0;
		int i;
		if (phase == kAfterFirst) {
			gesa = f;
			ex.each(1, jn, [&](int j) { g[j] = grad(j); });
			goto L110;
		}
		fb = f;
		ex.each(1, jn, [&](int j) { gb[j] = grad(j); });
		isfv = isfv < 2 ? isfv : 2;
		if (fb > gesa) goto L220;
		if (fb < gesa) goto L200;
		{
			double gl1 = xnull, gl2 = xnull;
			GBA_VA_LOOP
			for (i = 1; i <= jn; ++i) {
				gl1 = gl1 + vm(g[i], g[i]);
				gl2 = gl2 + vm(gb[i], gb[i]);
			}
			if (gl2 >= gl1) goto L220;
		}
	L200:
		isfv = 3;
		gesa = fb;
		ex.each(1, jn, [&](int j) {
			x[j] = xbb[j];
			g[j] = gb[j];
		});
	L220:
		dgb = xnull;
		ex.each(1, jn, [&](int j) { t[j] = vm(gb[j], d[j]); });
		GBA_VA_LOOP
		for (i = 1; i <= jn; ++i) dgb = dgb + t[i];
		if (fb - fa <= vm(vm(0.1, c), dga)) goto L280;
		if (step > steplb) goto L270;
	L240:
		if (isfv >= 2) goto L110;
		phase = kDone;
		goto Lsave;
	L270:
		stepbd = step;
		c = gmin + dgb - va_div(vm(3.0, fb - fmin), step);
		c = va_div(gmin, c + gmin - sqrt(vm(c, c) - vm(gmin, dgb)));
		step = vm(step, va_max(0.1, c));
		goto L170;
	L280:
		stepbd = stepbd - step;
		stmin = c;
		fmin = fb;
		gmin = dgb;
		step = vm(9.0, stmin);
		if (stepbd > xnull) step = vm(0.5, stepbd);
		c = dga + vm(3.0, dgb) - va_div(vm(4.0, fb - fa), stmin);
		if (c > xnull) step = va_min(step, vm(stmin, va_max(1.0, va_div(-dgb, c))));
		if (dgb < vm(0.7, dga)) goto L170;
		isfv = 4 - isfv;
		if (stmin + step <= steplb) goto L240;
		ir = -jn;
		ex.each(1, jn, [&](int j) {
			xaa[j] = xbb[j];
			xbb[j] = ga[j];
			d[j] = gb[j] - ga[j];
			ga[j] = gb[j];
		});
		{
			const double den = vm(stmin, dgb - dga), most = 1.7976931348623157e308;
			if (jn >= 2 && jn <= 16 && dga < 0.0 && dga >= -most && den > 0.0 && den <= most) {
				ir = mc11a_pair_w(h, jn, xbb, d, den, w, q, t, ex);
			} else {
				/* one after the other, in a loop so that mc11a's code is there once */
				GBA_VA_LOOP
				for (int u = 0; u < 2; ++u) {
					if (u == 1) ir = -ir;
					mc11a_w(h, jn, u == 0 ? xbb : d, va_div(1.0, u == 0 ? dga : den), u == 0 ? w : d, ir, 1 - u, xnull, q, t, ex);
				}
			}
		}
		if (ir < jn) {
			phase = kDone;
			goto Lsave;
		}
		dff = fa - fb;
		fa = fb;
		goto L135;
	L110:
		fa = gesa;
		isfv = 1;
		ex.each(1, jn, [&](int j) { ga[j] = g[j]; });
	L135:
		itr = itr + 1;
		ex.each(1, jn, [&](int j) { d[j] = -ga[j]; });
		mc11e_w(h, jn, d, w, jn, q, t, ex);
		c = xnull;
		dga = xnull;
		ex.each(1, jn, [&](int j) { t[j] = vm(ga[j], d[j]); });
		GBA_VA_LOOP
		for (i = 1; i <= jn; ++i) {
			c = va_max(c, va_abs(d[i]));
			dga = dga + t[i];
		}
		if (dga >= xnull) goto L240;
		stmin = xnull;
		stepbd = xnull;
		steplb = va_div(acc, c);
		fmin = fa;
		gmin = dga;
		step = 1.0;
		if (dff <= xnull) step = va_min(step, va_div(1.0, c));
		if (dff > xnull) step = va_min(step, va_div(dff + dff, -dga));
	L170:
		c = stmin + step;
		if (nfun >= ivmax) {
			phase = kDone;
			goto Lsave;
		}
		nfun = nfun + 1;
		ex.each(1, jn, [&](int j) { xbb[j] = xaa[j] + vm(c, d[j]); });
		phase = kAfterLine;
	Lsave:
		ex.each(0, 0, [&](int) {
			this->phase = phase;
			this->nfun = nfun;
			this->itr = itr;
			this->isfv = isfv;
			this->ir = ir;
			this->gesa = gesa;
			this->c = c;
			this->dff = dff;
			this->dgb = dgb;
			this->fa = fa;
			this->fb = fb;
			this->fmin = fmin;
			this->gmin = gmin;
			this->dga = dga;
			this->step = step;
			this->stepbd = stepbd;
			this->steplb = steplb;
			this->stmin = stmin;
		});
	}
};

}  // namespace gba

#endif
