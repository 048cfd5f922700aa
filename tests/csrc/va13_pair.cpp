/* minfor's two rank-one updates of a step: mc11a called twice against
 * mc11a_pair_w, from the same factors, vectors and scalars.  out_*: the packed
 * factors (n (n + 1) / 2 entries), the second update's z (n) and ir; the first
 * update's z is not used after either. */
#include "../../gpuattract_2.0_gb300/csrc/va13.cuh"

extern "C" int va13_update_pair(int n, const double* a0, const double* z0, const double* z1, const double* w0,
		double dga, double den, double* out_seq, double* out_pair) {
	if (n < 2 || n > 16) return -1;
	const int na = n * (n + 1) / 2;
	for (int form = 0; form < 2; ++form) {
		double a[16 * 17 / 2 + 1], y[17], z[17], w[17], q[17], t[17];
		for (int k = 0; k < na; ++k) a[k + 1] = a0[k];
		for (int k = 0; k < n; ++k) {
			y[k + 1] = z0[k];
			z[k + 1] = z1[k];
			w[k + 1] = w0[k];
		}
		int ir = -n;
		if (form == 0) {
			gba::mc11a(a, n, y, 1.0 / dga, w, ir, 1, 0.0);
			ir = -ir;
			gba::mc11a(a, n, z, 1.0 / den, z, ir, 0, 0.0);
		} else {
			ir = gba::mc11a_pair_w(a, n, y, z, den, w, q, t, gba::VaSerial{});
		}
		double* out = form == 0 ? out_seq : out_pair;
		for (int k = 0; k < na; ++k) out[k] = a[k + 1];
		for (int k = 0; k < n; ++k) out[na + k] = z[k + 1];
		out[na + n] = ir;
	}
	return 0;
}
