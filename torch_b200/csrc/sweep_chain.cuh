// Causal sweeps of small grids as one launch: a CTA per grid walks the grid's
// shells, the shells' results passing through shared memory.  Included by
// kernels_fp64.cu inside its build's namespace.
//
// What bounds it: the chain of shells.  A 2-D grid of 150 x 200 cells has 260
// shells of about 115 cells, so a launch per shell is launch latency
// (2.4-2.7 us each, whatever the cells' work), and with the launches gone the
// latency of one cell's arithmetic per shell is what is left.  So:
//  * two groups of warps take the shells in turn.  Between a group's two
//    shells lie the loads of its next cells (inputs, interpolation weights and
//    the places of their neighbours' values, fixed by the geometry and worked
//    out once per run), everything that does not depend on the neighbours
//    (the first iteration's exponential, reciprocals) and the stores of its
//    last ones, while the other group computes: only the wait for a named
//    barrier, the neighbours' values and what follows from them are in the
//    chain;
//  * divisions are formed without the branch of the built-in one, so that
//    independent ones overlap (Recip), and those by a divisor known before
//    the neighbours are cost five operations.
// Measured (B200, radiation / column-density sweep, per-shell launches ->
// this): 150 x 200 grid, exact build 1203 -> 451 / 668 -> 127 us, fast build
// 590 -> 329 / 595 -> 94 us; 1-D grid of 200 cells, exact build 926 -> 294 us;
// 64 grids of 64-256 x 64-320 cells together, fast build 3017 -> 978 / 2008 ->
// 334 us.  (One group of warps, with clusters of 1 to 8 CTAs that pass their
// shells on by st.async: 1150-1200 / 580-640 us for the 150 x 200 grid in the
// exact build whatever the number of CTAs, since every cell's loads, reciprocals
// and stores were then part of the chain.)
// Results are bit for bit those of the per-shell kernels in the exact build.

// Division by one divisor: a reciprocal by Newton's iteration, then a / b by
// two corrections with exact remainders (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. R&D 34,
// 1990): with y the correctly rounded reciprocal, which its last iteration
// gives unless b's significand is all ones, and a quotient within one ulp,
// fma(remainder, y, quotient) is a / b rounded to nearest.  Operands outside
// 2^-500 .. 2^500 (where a remainder or a quotient could leave the normal
// range) and such divisors take the built-in division.
struct Recip {
	double b, y;
	bool ok;
	__device__ __forceinline__ static bool mid(double v) {  // 2^-500 <= |v| < 2^500
		return (unsigned)(__double2hiint(v) & 0x7fffffff) - 0x20b00000u < 0x3e800000u;
	}
	__device__ __forceinline__ void set(double divisor) {
		b = divisor;
		ok = mid(b) && __double2loint(b) != -1;
		asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
		y = fma(y, fma(-b, y, 1.0), y);
		y = fma(y, fma(-b, y, 1.0), y);
		y = fma(y, fma(-b, y, 1.0), y);
	}
	__device__ __forceinline__ double quotient(double a) const {
		double q = a * y;
		q = fma(fma(-b, q, a), y, q);
		return fma(fma(-b, q, a), y, q);
	}
	__device__ __forceinline__ bool takes(double a) const { return ok && (mid(a) || a == 0.0); }
	__device__ __forceinline__ double div(double a) const { return takes(a) ? quotient(a) : a / b; }
};

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
// colden_interp with the same divisions.
__device__ __forceinline__ double colden_interp_chain(const double* c, const double* w0) {
#ifdef TRG_FAST_MATH
	return colden_interp(c, w0);
#else
	double w[4], sum = 0.0, out = 0.0;
	bool ok = true;
#pragma unroll
	for (int i = 0; i < 4; ++i) {
		Recip r;
		r.set(c[i] == 0 ? 1.0 : c[i]);
		const double n = c[i] == 0 ? 0.0 : w0[i];
		ok &= r.takes(n);
		w[i] = r.quotient(n);
	}
	sum = w[0] + w[1] + w[2] + w[3];
	Recip rs;
	rs.set(sum);
#pragma unroll
	for (int i = 0; i < 4; ++i) {
		ok &= rs.takes(w[i]);
		out += rs.quotient(w[i]) * c[i];
	}
	return ok ? out : colden_interp(c, w0);  // (a zero sum is not taken)
#endif
}

// Picard solve of a cell: the plain path of rad_shell in its arithmetic.
// What the neighbours' optical depths do not decide - the first iteration's
// exp(-dtau) and the reciprocal of its neutral column - is formed by
// chain_pre.
struct ChainCell {
	double n_H, alphaB, A_ci, x, ds, shellVol;  // x: x_HII at the start of the sweep
	double em0;
	Recip r0;
};
__device__ __forceinline__ void chain_pre(const Params& P, ChainCell& c) {
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
__device__ __forceinline__ void chain_solve(const Params& P, const State& S, const ChainCell& c, double dt,
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

// A thread's cell of a shell: its position p in the sweep list, cell id,
// weights, ring places of its neighbours (-1: not read, or a wind cell, whose
// optical depths are 0) and inputs.
template <bool RAD>
struct ChainItem {
	int p, id;
	int4 slot;
	double w[4];
	double own;  // column density
	ChainCell c;  // radiation
	__device__ __forceinline__ void load(const SweepChain& ch, const State& S, int pos) {
		p = pos;
		id = __ldg(&ch.cells[p]);
		slot = __ldg(reinterpret_cast<const int4*>(ch.slot) + p);
#pragma unroll
		for (int k = 0; k < 4; ++k) w[k] = __ldg(&ch.w[(long long)k * ch.n + p]);
		if (RAD) {
			const double* in = S.sw_rad + p;
			c.n_H = in[0];
			c.alphaB = in[S.sw_rad_n];
			c.A_ci = in[2 * S.sw_rad_n];
			c.x = in[3 * S.sw_rad_n];
			c.ds = in[4 * S.sw_rad_n];
			c.shellVol = in[5 * S.sw_rad_n];
		} else {
			own = S.sw_col[p];
		}
	}
};
struct ChainResult {
	double tau, tau_a, dtau, dtau_a, x, x_avg;
};
template <bool RAD>
__device__ __forceinline__ double2 chain_cell(const Params& P, const State& S, const ChainItem<RAD>& it,
                                              const double2* ring, double dt, ChainResult& r) {
	const int slot[4] = {it.slot.x, it.slot.y, it.slot.z, it.slot.w};
	double a[4], b[4];
#pragma unroll
	for (int k = 0; k < 4; ++k) {
		const double2 v = slot[k] >= 0 ? ring[slot[k]] : make_double2(0.0, 0.0);
		a[k] = v.x;
		b[k] = v.y;
	}
	if (RAD) {
		const ChainCell& c = it.c;
		tau_interp2(P, a, b, it.w, r.tau, r.tau_a);
		chain_solve(P, S, c, dt, r.tau_a, r.x, r.x_avg);
		r.dtau = (1.0 - r.x) * c.n_H * P.photoIonXsec * c.ds;
		r.dtau_a = (1.0 - r.x_avg) * c.n_H * P.photoIonXsec * c.ds;
		return make_double2(r.tau + r.dtau, r.tau_a + r.dtau_a);
	}
	r.tau = colden_interp_chain(a, it.w);
	return make_double2(r.tau + it.own, 0.0);
}
template <bool RAD>
__device__ __forceinline__ void chain_store(const Params& P, const State& S, const ChainItem<RAD>& it,
                                            const ChainResult& r) {
	if (RAD) {
		S.sw_rad[SW_TAU_A * S.sw_rad_n + it.p] = r.tau_a;
		RFLD(S.R, R_HII_A, it.id) = r.x_avg;
		FLD(S.Q, HII, it.id) = r.x;
		if (r.x > 0.001) FLD(S.Q, ADV, it.id) = 1;
		store_taus(S, it.id, r.tau, r.dtau, r.tau_a, r.dtau_a);
	} else {
		reinterpret_cast<double2*>(S.T + (long long)it.id * 2)[0] = make_double2(r.tau, it.own);
	}
}

// The ring holds three shells: a cell reads the two before its own (an upwind
// neighbour's key is at most 2 smaller).  Barrier 1 + (s & 1) passes from the
// group of shell s, which arrives, to the group of shell s + 1, which waits;
// a slot is overwritten three shells later, when the group that read it last
// has arrived.
template <bool RAD>
__device__ __forceinline__ void chain_sweep(const Params& P, const State& S, double h) {
	extern __shared__ __align__(16) unsigned char sm_chain[];
	const SweepChain ch = RAD ? *S.chain_rad : *S.chain_col;
	double2* ring = reinterpret_cast<double2*>(sm_chain);
	int* off = reinterpret_cast<int*>(sm_chain + 48 * (size_t)ch.maxshell);
	for (int i = threadIdx.x; i <= ch.nshell; i += blockDim.x) off[i] = ch.off[i];
	__syncthreads();
	const int T = (int)blockDim.x / 2, group = (int)threadIdx.x >= T ? 1 : 0, tid = (int)threadIdx.x - group * T;
	const double dt = RAD ? h * S.scal[0] : 0.0;
	ChainItem<RAD> it;
	it.id = -1;
	if (group < ch.nshell && off[group] + tid < off[group + 1]) it.load(ch, S, off[group] + tid);
	for (int s = group; s < ch.nshell; s += 2) {
		const int o0 = off[s], n = off[s + 1] - o0;
		double2* out = ring + (s % 3) * ch.maxshell;
		ChainItem<RAD> cur = it;
		it.id = -1;
		if (s + 2 < ch.nshell && off[s + 2] + tid < off[s + 3]) it.load(ch, S, off[s + 2] + tid);
		if (RAD && cur.id >= 0) chain_pre(P, cur.c);
		if (s > 0) asm volatile("bar.sync %0, %1;" ::"r"(1 + ((s - 1) & 1)), "r"(2 * T) : "memory");
		ChainResult r;
		if (cur.id >= 0) out[tid] = chain_cell<RAD>(P, S, cur, ring, dt, r);
		for (int t = tid + T; t < n; t += T) {  // shells of more than T cells
			ChainItem<RAD> more;
			ChainResult rm;
			more.load(ch, S, o0 + t);
			if (RAD) chain_pre(P, more.c);
			out[t] = chain_cell<RAD>(P, S, more, ring, dt, rm);
			chain_store<RAD>(P, S, more, rm);
		}
		if (s + 1 < ch.nshell) asm volatile("bar.arrive %0, %1;" ::"r"(1 + (s & 1)), "r"(2 * T) : "memory");
		if (cur.id >= 0) chain_store<RAD>(P, S, cur, r);
	}
}
template <bool RAD>
__device__ __forceinline__ void chain_kernel(const Params& P, const State& S, double h) {
	if (TRG_BATCHED && P.batch) chain_sweep<RAD>(P.batch->P[blockIdx.x], P.batch->S[blockIdx.x], h);
	else chain_sweep<RAD>(P, S, h);
}
__global__ void __launch_bounds__(2 * CHAIN_GROUP, 1) k_rad_chain(Params P, State S, double h) {
	chain_kernel<true>(P, S, h);
}
__global__ void __launch_bounds__(2 * CHAIN_GROUP, 1) k_colden_chain(Params P, State S) {
	chain_kernel<false>(P, S, 0.0);
}

// The chain's tables of one grid: each cell's weights and the ring places of
// its neighbours, by its position in the sweep list.  pos[cell]: the position,
// or -1 for a cell the list leaves out.  *bad is set where a neighbour does not
// lie in one of the two shells before the cell's.
__global__ void __launch_bounds__(256) k_chain_positions(const int* __restrict__ cells, int n, int* __restrict__ pos) {
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	if (t < n) pos[cells[t]] = t;
}
__device__ __forceinline__ int shell_at(const SweepChain& ch, int p) {
	int lo = 0, hi = ch.nshell - 1;
	while (lo < hi) {
		const int mid = (lo + hi + 1) >> 1;
		if (ch.off[mid] <= p) lo = mid;
		else hi = mid - 1;
	}
	return lo;
}
__global__ void __launch_bounds__(256) k_chain_tables(Params P, SweepChain ch, const int* __restrict__ pos,
                                                      int rad, ChainSlots* __restrict__ slot,
                                                      double* __restrict__ w, int* __restrict__ bad) {
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= ch.n) return;
	const int s = shell_at(ch, t);
	int code[4] = {-1, -1, -1, -1};
	double w0[4] = {1.0, 0.0, 0.0, 0.0};
	const SweepCell cell(P, ch.cells[t]);
	if (cell.inner()) {
		long long nb[4];
		neighbours(P, cell, ch.cells[t], nb, w0);
#pragma unroll
		for (int k = 0; k < 4; ++k) {
			if (w0[k] == 0 || nb[k] < 0 || pos[nb[k]] < 0) continue;
			const int p = pos[nb[k]], sn = shell_at(ch, p);
			if (sn >= s || sn < s - 2) *bad = 1;
			code[k] = (sn % 3) * ch.maxshell + (p - ch.off[sn]);
		}
	}
	if (rad && cell.star(P)) *bad = 1;  // a swept star cell (Radiation::isStar) is not solved: left to the per-shell kernels
	slot[t] = ChainSlots{code[0], code[1], code[2], code[3]};
#pragma unroll
	for (int k = 0; k < 4; ++k) w[(long long)k * ch.n + t] = w0[k];
}
