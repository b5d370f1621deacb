// A cell's part of the radiation sweep with its divisions (Recip,
// trg_device.cuh) and exponentials overlapped: what the sweeps walked by one CTA (sweep_chain.cuh) and the plain
// per-shell kernel run.  Included by kernels_fp64.cu inside its build's
// namespace.  Results are those of rad_shell's general loop: bit for bit in the
// exact build.

// tau_interp of two sets of optical depths at once.
__device__ __forceinline__ void tau_interp2(const Params& P, const double* ta, const double* tb, const double* w0,
                                            double& out_a, double& out_b) {
#ifdef TRG_FAST_MATH
	double m[8];
#pragma unroll
	for (int i = 0; i < 4; ++i) {
		m[i] = smax(P.tau0, ta[i]);
		m[4 + i] = smax(P.tau0, tb[i]);
	}
	double num[2], den[2], big = 0;
#pragma unroll
	for (int s = 0; s < 2; ++s) {
		const double *t = s ? tb : ta, *n = m + 4 * s;
		const double m01 = n[0] * n[1], m23 = n[2] * n[3];
		const double p0 = n[1] * m23, p1 = n[0] * m23, p2 = n[3] * m01, p3 = n[2] * m01;
		num[s] = w0[0] * p0 * t[0] + w0[1] * p1 * t[1] + w0[2] * p2 * t[2] + w0[3] * p3 * t[3];
		den[s] = w0[0] * p0 + w0[1] * p1 + w0[2] * p2 + w0[3] * p3;
		big = smax(big, m01 * m23);
	}
	if (big < 1.0e120) {  // the weights sum to 1: both denominators lie between tau0^3 and 1e90
		Recip ra, rb;
		ra.set(den[0]);
		rb.set(den[1]);
		out_a = ra.div(num[0]);
		out_b = rb.div(num[1]);
		return;
	}
	out_a = tau_interp(P, ta, w0);
	out_b = tau_interp(P, tb, w0);
#else
	// w0 / m rounded, then each over their sum, as in tau_interp; a zero weight
	// stays zero through both
	Recip r[8];
	bool ok = true;
	double w[8];
#pragma unroll
	for (int i = 0; i < 8; ++i) {
		r[i].set(smax(P.tau0, i < 4 ? ta[i] : tb[i - 4]));
		ok &= r[i].takes(w0[i & 3]);
		w[i] = r[i].quotient(w0[i & 3]);
	}
	Recip ra, rb;
	ra.set(w[0] + w[1] + w[2] + w[3]);
	rb.set(w[4] + w[5] + w[6] + w[7]);
	double a = 0.0, b = 0.0;
#pragma unroll
	for (int i = 0; i < 4; ++i) {
		ok &= ra.takes(w[i]) && rb.takes(w[4 + i]);
		a += ra.quotient(w[i]) * ta[i];
		b += rb.quotient(w[4 + i]) * tb[i];
	}
	out_a = ok ? a : tau_interp(P, ta, w0);
	out_b = ok ? b : tau_interp(P, tb, w0);
#endif
}
// Picard solve of a cell: the plain path of rad_shell in its arithmetic.
// What the neighbours' optical depths do not decide - the first iteration's
// exp(-dtau) and the reciprocal of its neutral column - is formed by
// solve_pre.
struct SolveCell {
	double n_H, alphaB, A_ci, x, ds, shellVol;  // x: x_HII at the start of the sweep
	double em0;
	Recip r0;
};
__device__ __forceinline__ void solve_pre(const Params& P, SolveCell& c) {
	c.em0 = d_exp(-((1.0 - c.x) * c.n_H * P.photoIonXsec * c.ds));
	c.r0.set((1.0 - c.x) * c.n_H * c.shellVol);
}
// |now - before| / |now| < 1e-3 as rounded, without the division where a
// product settles it
__device__ __forceinline__ bool small_change(double now, double before) {
	const double d = fabs(now - before), m = fabs(now);
#ifdef TRG_FAST_MATH
	return d < 1.0e-3 * m;
#else
	if (d < 0.9999999e-3 * m) return true;
	if (d > 1.0000001e-3 * m) return false;
	return fabs((now - before) / now) < 1.0e-3;
#endif
}
__device__ __forceinline__ void solve_cell(const Params& P, const State& S, const SolveCell& c, double dt,
                                            double tau_avg, double& x_new, double& HII_avg) {
	const double epsilon = 1.0e-8;
	const double em_tau = d_exp(-tau_avg);
	const double scale = P.photonRate * em_tau;
	HII_avg = c.x;
	int niter = 0, miter = 0;
	bool first = true;
	for (;;) {
		niter++;
		const double old = HII_avg;
		// photoionisation_rate_e
		const double nHI = (1.0 - HII_avg) * c.n_H;
		const double dtau = nHI * P.photoIonXsec * c.ds;
		double A_pi = 0.0;
		if (!(nHI == 0 || c.shellVol == 0 || (em_tau == 0 && dtau == dtau))) {
			if (first) {
				A_pi = c.r0.div(scale * (1.0 - c.em0));
			} else {
				Recip r;
				r.set(nHI * c.shellVol);
				A_pi = r.div(scale * (1.0 - d_exp(-dtau)));
			}
		}
		first = false;
		// doric
		const double nHII_aB = HII_avg * c.n_H * c.alphaB, nHII_Aci = HII_avg * c.n_H * c.A_ci;
		const double ion = A_pi + nHII_Aci, inv_ti = ion + nHII_aB, t = dt * inv_ti;
		if (t < 1.0e-8) {
			x_new = smax(smin(c.x, 1.0), 0.0);
			if (1.0 - x_new < epsilon) x_new = 1.0 - epsilon;
			HII_avg = x_new;
		} else {
			Recip rt;
			rt.set(t);
#ifdef TRG_FAST_MATH
			const double ti_dt = rt.div(1.0);
			const double xeq = nHII_aB == 0.0 ? 1.0 : ion * (ti_dt * dt);
			const double e = d_exp(-t);
			HII_avg = xeq + (c.x - xeq) * (1.0 - e) * ti_dt;
#else
			Recip ri;
			ri.set(inv_ti);
			const double xeq = nHII_aB == 0.0 ? 1.0 : ri.div(ion);
			const double e = d_exp(-t);
			HII_avg = xeq + rt.div((c.x - xeq) * (1.0 - e));
#endif
			x_new = xeq + (c.x - xeq) * e;
			x_new = smax(smin(x_new, 1.0), 0.0);
			if (1.0 - x_new < epsilon) x_new = 1.0 - epsilon;
			HII_avg = smax(smin(HII_avg, 1.0), 0.0);
			if (1.0 - HII_avg < epsilon) HII_avg = 1.0 - epsilon;
		}
		const bool converged = small_change(HII_avg, old) || HII_avg < 1.0e-5 || A_pi == 0;
		if (niter > 10005) {
			miter++;
			niter = 0;
			HII_avg = 0.5 * (HII_avg + old);
		}
		if (miter > 5 || x_new != x_new) {
			atomicOr(S.err, ERRB_PICARD);
			return;
		}
		if (converged) return;
	}
}

