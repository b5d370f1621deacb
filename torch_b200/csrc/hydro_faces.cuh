// Face fluxes of the FP64 hydrodynamics: reconstruction (Hydro.cpp:44-67),
// Riemann solvers (Riemann.cpp) and the kernels that run them over a grid's
// faces.  Included by kernels_fp64.cu inside its build's namespace.
//
// What bounds it: FP64 arithmetic.  A face of the rotated solver takes about
// 50 divisions and square roots in the reference's operation order, which
// the exact build has to round one by one, against 112 bytes of memory
// traffic.  So the work here is to do no operation twice and to keep a
// face's state in registers:
//  * the dimension of the face (DIM) and the grid's (ND) are compile-time
//    constants, so no array is indexed at run time (the one-kernel form with
//    a run-time dimension kept 776 bytes of states per thread in local memory);
//  * the rotations of the rotated solver use their structure (below), and
//    HLL and HLLC share what does not depend on the direction;
//  * a cell's limited slope is computed once per dimension: along x by the
//    lane that holds the cell, its neighbours' values and slopes passed
//    through shuffles; along y and z by the thread that marches down the
//    column, which also loads each cell once instead of four times.
// Measured (B200, rotated solver, exact build, all directions together, before
// -> after): Sedov blast 97^3 554 -> 238 us, HII region 100^3 1283 -> 395 us,
// 257^2 blast 55 -> 19 us.  128 registers (16 warps per SM) with 1.1 KB of
// spills beat 168 registers by 7% on the HII region and equal them on the
// blasts; unbounded (230 registers, 8 warps) is 20-30% slower.
// Every value is formed by the reference's own operations in its own order;
// what is left out are products with the exact zeros and ones of the axis
// vector (which can change the sign of a zero, nothing else).

// ------------------------------------------------------------------ limiters
__device__ __forceinline__ double minmod(double a, double b) { return (a * b > 0) ? (fabs(a) < fabs(b) ? a : b) : 0; }
__device__ __forceinline__ double maxmod(double a, double b) { return (a * b > 0) ? (fabs(a) > fabs(b) ? a : b) : 0; }

// SlopeLimiter::calculate variants, SlopeLimiter.cpp:5-54.  Albada, the
// configured and default one, is inlined where it is used; the others are
// called, which keeps seven copies of this switch out of the face loops.
__device__ __forceinline__ double albada(double a, double b) {
	return a * b <= 1.0e-30 ? 0 : a * b * (a + b) / (a * a + b * b);
}
__device__ __noinline__ double limiter_other(int kind, double a, double b) {
	switch (kind) {
	case 0: return minmod((a + b) / 2.0, minmod(2.0 * a, 2.0 * b));
	case 1: return maxmod(minmod(b, 2.0 * a), minmod(2.0 * b, a));
	case 2: return minmod(a, b);
	case 3: return maxmod(a, b);
	case 4: {
		if (b == 0) return 0;
		double r = fabs(a / b);
		return (a + b * r) / (1.0 + r);
	}
	case 5: return (a * b <= 1.0e-30) ? 0 : 1.5 * b * (a * a + a * b) / (a * a + a * b + b * b);
	default: return albada(a, b);
	}
}
// Limited slopes of a cell from its differences to the cells before and after
// it; velocity components beyond the grid's dimensions are 0.
template <int ND>
__device__ __forceinline__ void cell_slopes(int kind, const double* before, const double* cell, const double* after,
                                            double* slope) {
	if (kind == 6) {
#pragma unroll
		for (int f = 0; f < VEL + ND; ++f) slope[f] = albada(cell[f] - before[f], after[f] - cell[f]);
	} else {
#pragma unroll
		for (int f = 0; f < VEL + ND; ++f) slope[f] = limiter_other(kind, cell[f] - before[f], after[f] - cell[f]);
	}
#pragma unroll
	for (int f = VEL + ND; f < NU; ++f) slope[f] = 0;
}

// ----------------------------------------------------------- Riemann solvers
// Axes of a face with normal d = e_DIM: D = DIM and the next two, A and B, in
// cyclic order, in which a cross product has the same form for every DIM.
// Sums over the three components keep the index order of the reference's
// vendored Eigen 3.2.1: x + (y + z) for a dot product or norm, (x + y) + z
// for a matrix row.
template <int DIM>
__device__ __forceinline__ double dot_order(double tD, double tA, double tB) {
	return DIM == 0 ? tD + (tA + tB) : (DIM == 1 ? tB + (tD + tA) : tA + (tB + tD));
}
template <int DIM>
__device__ __forceinline__ double row_order(double tD, double tA, double tB) {
	return DIM == 0 ? (tD + tA) + tB : (DIM == 1 ? (tB + tD) + tA : (tA + tB) + tD);
}

// getRotationFromA2B, Riemann.cpp:161-171 (Rodrigues: I + [v]x + (1-c)/s^2
// [v]x^2, v = a x b, s = |v|, c = a . b) between a unit vector n and the axis
// d: v = (0, vA, vB) in the (D, A, B) frame, so [v]x^2 has five non-zero
// entries.  The rotation from d to n is the one from n to d with v negated:
// the squared terms are the same, so one set of entries serves both.
struct Rotation {
	double dd, aa, ab, ba, bb;  // I + (1-c)/s^2 [v]x^2
	double vA, vB;
	// n = (nD, ., .), v = n x d, s = |v|
	__device__ __forceinline__ void set(double nD, double va, double vb, double s) {
		vA = va;
		vB = vb;
		const double k = (1.0 - nD) / (s * s);
		const double ka = k * va, kb = k * vb;
		dd = 1.0 + (-(kb * vb) - ka * va);
		aa = 1.0 - kb * vb;
		ab = kb * va;
		ba = ka * vb;
		bb = 1.0 - ka * va;
	}
	// rotate, Riemann.cpp:154-159: n to d (sgn = 1) or d to n (sgn = -1)
	template <int DIM>
	__device__ __forceinline__ void apply(double sgn, double* v) const {
		constexpr int A = (DIM + 1) % 3, B = (DIM + 2) % 3;
		const double a = sgn * vA, b = sgn * vB;
		const double x = v[DIM], y = v[A], z = v[B];
		v[DIM] = row_order<DIM>(dd * x, -b * y, a * z);
		v[A] = row_order<DIM>(b * x, aa * y, ab * z);
		v[B] = row_order<DIM>(-a * x, ba * y, bb * z);
	}
};

// One side of a face: the state, and what its fluxes share whatever the
// direction of the velocities.
struct Side {
	double d, p, x, a, v[3];
	double pg;  // p / (gamma - 1)
};
// UfromQ's total energy (GridCell.cpp:163-175)
template <int ND>
__device__ __forceinline__ double side_energy(const Side& s) {
	double ke = 0;
#pragma unroll
	for (int k = 0; k < ND; ++k) ke += 0.5 * s.d * s.v[k] * s.v[k];
	return s.pg + ke;
}
// FfromQ, GridCell.cpp:193-213
template <int DIM, int ND>
__device__ __forceinline__ void side_flux(const Side& s, double g2, double* F) {
	const double u = s.v[DIM];
	double ke = 0;
#pragma unroll
	for (int k = 0; k < 3; ++k) F[VEL + k] = 0;
#pragma unroll
	for (int k = 0; k < ND; ++k) {
		ke += s.v[k] * s.v[k];
		F[VEL + k] = s.d * s.v[k] * u;
	}
	ke *= 0.5 * s.d;
	F[DEN] = s.d * u;
	F[VEL + DIM] += s.p;
	F[PRE] = u * (g2 * s.p + ke);
	F[HII] = s.d * u * s.x;
	F[ADV] = s.d * u * s.a;
}
// The direction-independent part of characteristicWaveSpeeds (Einfeldt),
// Riemann.cpp:27-42.
struct SpeedBase {
	double sl, sr, sum, nu2, c2;
	__device__ __forceinline__ void set(const Side& L, const Side& R, double a_l2, double a_r2) {
		sl = sqrt(L.d);
		sr = sqrt(R.d);
		sum = sl + sr;
		nu2 = 0.5 * sr * sl / (sum * sum);
		c2 = (sl * a_l2 + sr * a_r2) / sum;
	}
	__device__ __forceinline__ void speeds(double ul, double ur, double& Sl, double& Sr) const {
		const double u_tilde = (sl * ul + sr * ur) / sum;
		const double d = sqrt(c2 + nu2 * (ur - ul) * (ur - ul));
		Sl = u_tilde - d;
		Sr = u_tilde + d;
	}
};

// HartenLaxLeerSolver::solve, Riemann.cpp:108-140.
template <int DIM, int ND>
__device__ __forceinline__ void hll(const Side& L, const Side& R, const SpeedBase& sp, double g2, double* F) {
	double S_l, S_r;
	sp.speeds(L.v[DIM], R.v[DIM], S_l, S_r);
	if (S_r <= 0) {
		side_flux<DIM, ND>(R, g2, F);
	} else if (S_l >= 0) {
		side_flux<DIM, ND>(L, g2, F);
	} else {
		double FR[7];
		side_flux<DIM, ND>(L, g2, F);
		side_flux<DIM, ND>(R, g2, FR);
		const double w = S_r - S_l, ss = S_l * S_r;
		auto mean = [&](int i, double ul, double ur) { F[i] = (S_r * F[i] - S_l * FR[i] + ss * (ur - ul)) / w; };
		mean(DEN, L.d, R.d);
		mean(PRE, side_energy<ND>(L), side_energy<ND>(R));
		mean(HII, L.x * L.d, R.x * R.d);
		mean(ADV, L.a * L.d, R.a * R.d);
#pragma unroll
		for (int k = 0; k < ND; ++k) mean(VEL + k, L.v[k] * L.d, R.v[k] * R.d);
	}
}

// HartenLaxLeerContactSolver::solve, Riemann.cpp:52-104.
template <int DIM, int ND>
__device__ __forceinline__ void hllc(const Side& L, const Side& R, const SpeedBase& sp, double g2, double* F) {
	double S_l, S_r;
	const double ul = L.v[DIM], ur = R.v[DIM];
	sp.speeds(ul, ur, S_l, S_r);
	// the side the flux is taken from, and whether it is the plain flux of that side
	bool left = S_l >= 0, plain = true;
	double S_c = 0;
	if (!left && !(S_r <= 0)) {
		plain = false;
		S_c = R.p - L.p;
		S_c += L.d * ul * (S_l - ul);
		S_c -= R.d * ur * (S_r - ur);
		S_c /= (L.d * (S_l - ul) - R.d * (S_r - ur));
		left = S_c >= 0;
	}
	Side K;
	K.d = left ? L.d : R.d;
	K.p = left ? L.p : R.p;
	K.x = left ? L.x : R.x;
	K.a = left ? L.a : R.a;
	K.pg = left ? L.pg : R.pg;
#pragma unroll
	for (int k = 0; k < 3; ++k) K.v[k] = left ? L.v[k] : R.v[k];
	side_flux<DIM, ND>(K, g2, F);
	if (plain) return;
	const double S = left ? S_l : S_r, u = K.v[DIM];
	const double m = K.d * (S - u);
	const double A = m / (S - S_c);
	const double E = side_energy<ND>(K);
	F[DEN] = F[DEN] + S * (A - K.d);
	F[PRE] = F[PRE] + S * (A * ((E / K.d) + (S_c - u) * (S_c + K.p / m)) - E);
	F[HII] = F[HII] + S * (A * K.x - K.x * K.d);
	F[ADV] = F[ADV] + S * (A * K.a - K.a * K.d);
#pragma unroll
	for (int k = 0; k < ND; ++k) F[VEL + k] = F[VEL + k] + S * (A * (k == DIM ? S_c : K.v[k]) - K.v[k] * K.d);
}

// Flux through a face with normal e_DIM between the reconstructed states L and
// R: HLL, HLLC or the rotated HLLC-HLL solver (Nishikawa & Kitamura 2008),
// RotatedHartenLaxLeerSolver::solve, Riemann.cpp:181-244, which takes HLL
// along the velocity jump (n1) and HLLC across it (n2), or one of the two
// alone where the jump or its part across the face vanishes.  Each solver is
// inlined once.
template <int DIM, int ND>
__device__ __forceinline__ void face_solve(const Params& P, const double* Lq, const double* Rq, double* F) {
	constexpr int A = (DIM + 1) % 3, B = (DIM + 2) % 3;
	const double g2 = P.gamma / (P.gamma - 1.0);
	Side L, R;
	L.d = Lq[DEN]; L.p = Lq[PRE]; L.x = Lq[HII]; L.a = Lq[ADV];
	R.d = Rq[DEN]; R.p = Rq[PRE]; R.x = Rq[HII]; R.a = Rq[ADV];
#pragma unroll
	for (int k = 0; k < 3; ++k) {
		L.v[k] = Lq[VEL + k];
		R.v[k] = Rq[VEL + k];
	}
	L.pg = L.p / (P.gamma - 1.0);
	R.pg = R.p / (P.gamma - 1.0);
	SpeedBase sp;
	sp.set(L, R, P.gamma * L.p / L.d, P.gamma * R.p / R.d);
	bool with_hll = P.riemann == RS_HLL, with_hllc = P.riemann == RS_HLLC, rotated = false;
	Rotation r1, r2;
	double w1 = 0, w2 = 0;
	if (!with_hll && !with_hllc) {
		double nD = R.v[DIM] - L.v[DIM], nA = R.v[A] - L.v[A], nB = R.v[B] - L.v[B];
		if (nD < 0) {
			nD = -nD;
			nA = -nA;
			nB = -nB;
		}
		const double len = sqrt(dot_order<DIM>(nD * nD, nA * nA, nB * nB));
		if (len < 1.0e-6) {
			with_hllc = true;
		} else {
			const double r = 1.0 / len;
			nD *= r;
			nA *= r;
			nB *= r;
			// t = n1 x d = (0, nB, -nA); n2 = t x n1 = (|t|^2, -nA nD, -nB nD)
			const double t2 = nB * nB + nA * nA, s1 = sqrt(t2);
			double mA = -(nA * nD), mB = -(nB * nD);
			const double mlen = sqrt(dot_order<DIM>(t2 * t2, mA * mA, mB * mB));
			if (s1 == 0 || mlen == 0) {
				with_hll = true;
			} else {
				const double rm = 1.0 / mlen, mD = t2 * rm;
				mA *= rm;
				mB *= rm;
				const double s2 = sqrt(mB * mB + mA * mA);
				if (s2 == 0) {
					with_hllc = true;
				} else {
					with_hll = with_hllc = rotated = true;
					w1 = fabs(nD);
					w2 = fabs(mD);
					r1.set(nD, nB, -nA, s1);
					r2.set(mD, mB, -mA, s2);
				}
			}
		}
	}
	double F1[7];
	if (with_hll) {
		if (ND > 1 && rotated) {
			r1.apply<DIM>(1.0, L.v);
			r1.apply<DIM>(1.0, R.v);
		}
		hll<DIM, ND>(L, R, sp, g2, F1);
		if (ND > 1 && rotated) {
			r1.apply<DIM>(-1.0, L.v);
			r1.apply<DIM>(-1.0, R.v);
			r1.apply<DIM>(-1.0, F1 + VEL);
		}
	}
	if (with_hllc) {
		if (ND > 1 && rotated) {
			r2.apply<DIM>(1.0, L.v);
			r2.apply<DIM>(1.0, R.v);
		}
		hllc<DIM, ND>(L, R, sp, g2, F);
		if (ND > 1 && rotated) {
			r2.apply<DIM>(-1.0, F + VEL);
#pragma unroll
			for (int i = 0; i < NU; ++i) F[i] = w1 * F1[i] + w2 * F[i];
		}
	} else {
#pragma unroll
		for (int i = 0; i < NU; ++i) F[i] = F1[i];
	}
}

// ------------------------------------------------------------- hydro faces
// Ghost position p (< 0 or >= n) along DIM -> interior source index and the
// velocity rule of Grid::applyBCs (Grid.cpp:649-836).  Layer k = 1 is adjacent.
// A PARTITION face (x-slab decomposition) takes ghost layer k from the
// neighbour's halo, S.halo_recv [side][k - 1][field][ny * nz], as the
// reference's ghost cells take the neighbour's Q (Grid.cpp:804-833).
// Velocity components beyond the grid's dimensions are 0 in Q and not read.
template <int DIM, int ND>
__device__ __forceinline__ void load_line(const Params& P, const State& S, long long base, int pos, double* q) {
	const int n = ncell(P, DIM);
	const long long stride = DIM == 0 ? 1 : (DIM == 1 ? P.nx : (long long)P.nx * P.ny);
	int src = pos, cond = -1, side = 0;
	if (pos < 0) {
		int k = -pos;
		cond = P.lbc[DIM];
		src = cond == BC_PERIODIC ? n - k : (cond == BC_REFLECTING ? k : 0);
	} else if (pos >= n) {
		int k = pos - n + 1;
		cond = P.rbc[DIM];
		side = 1;
		src = cond == BC_PERIODIC ? k - 1 : (cond == BC_REFLECTING ? n - 1 - k : n - 1);
	}
#pragma unroll
	for (int f = VEL + ND; f < NU; ++f) q[f] = 0;
	if (DIM == 0 && cond == BC_PARTITION) {  // base = (j + ny k) nx
		const long long nyz = (long long)P.ny * P.nz, trans = base / P.nx;
		const int layer = (side ? pos - n + 1 : -pos) - 1;
		const double* h = static_cast<const double*>(S.halo_recv) + (long long)(side * 2 + layer) * NU * nyz + trans;
#pragma unroll
		for (int f = 0; f < VEL + ND; ++f) q[f] = h[(long long)f * nyz];
		return;
	}
	const double* Q = S.Q + base + (long long)src * stride;
#pragma unroll
	for (int f = 0; f < VEL + ND; ++f) q[f] = __ldg(&Q[(long long)f * P.N]);
	if (cond >= 0) {
		double v = q[VEL + DIM];
		if (cond == BC_INFLOW) {
			if (side == 0 ? v < 0 : v > 0) q[VEL + DIM] = -1.0 * v;
		} else if (cond == BC_OUTFLOW) {
			if (side == 0 ? v > 0 : v < 0) q[VEL + DIM] = -1.0 * v;
		} else if (cond == BC_REFLECTING) {
			q[VEL + DIM] = -v;
		}
	}
}
template <int DIM>
__device__ __forceinline__ void store_flux(const State& S, long long t, const double* F) {
	if (F[HII] != F[HII]) atomicOr(S.err, ERRB_FLUX);
	double* Fd = S.F[DIM] + t;
	const long long nf = S.nfaces[DIM];
#pragma unroll
	for (int i = 0; i < NU; ++i) Fd[(long long)i * nf] = F[i];
}

// Hydrodynamics::calcFluxes (Hydro.cpp:91-115) along x for one row: a warp
// holds 32 consecutive cells of the row, two of them ghosts or cells of the
// neighbouring segments at its low end and one at its high end, and computes
// the 29 faces between the others.
constexpr int XSEG = 29;
template <int ND>
__device__ __forceinline__ void faces_x(const Params& P, const State& S, long long warp) {
	const int lane = threadIdx.x & 31, segs = (P.nx + XSEG) / XSEG;  // ceil((nx + 1) / XSEG)
	const long long row = warp / segs;
	if (row >= (long long)P.ny * P.nz) return;  // the whole warp
	const int pos = (int)(warp - row * segs) * XSEG - 2 + lane;  // this lane's cell, and the face below it
	double c[7], before[7], L[7];
	load_line<0, ND>(P, S, row * P.nx, min(max(pos, -P.ng), P.nx - 1 + P.ng), c);
#pragma unroll
	for (int f = 0; f < VEL + ND; ++f) before[f] = __shfl_up_sync(0xffffffffu, c[f], 1);
	if (P.order == 1) {
		double after[7], s[7];
#pragma unroll
		for (int f = 0; f < VEL + ND; ++f) after[f] = __shfl_down_sync(0xffffffffu, c[f], 1);
		cell_slopes<ND>(P.limiter, before, c, after, s);
#pragma unroll
		for (int f = 0; f < NU; ++f) {
			const double hs = 0.5 * s[f];
			L[f] = f < VEL + ND ? before[f] + __shfl_up_sync(0xffffffffu, hs, 1) : 0.0;
			c[f] = f < VEL + ND ? c[f] - hs : 0.0;
		}
	} else {
#pragma unroll
		for (int f = 0; f < NU; ++f) L[f] = f < VEL + ND ? before[f] : 0.0;
	}
	if (lane < 2 || lane > 30 || pos > P.nx) return;
	double F[7];
	face_solve<0, ND>(P, L, c, F);
	store_flux<0>(S, row * (P.nx + 1) + pos, F);
}

// The same along y or z for `chunk` consecutive faces of one column, from face
// f0 on: the thread keeps the cell below the face, its slope, and the face's
// own cell from one face to the next.
template <int DIM, int ND>
__device__ __forceinline__ void faces_column(const Params& P, const State& S, long long col, int f0, int chunk) {
	const int n = ncell(P, DIM);
	long long base, t0, stride;  // first cell of the column, its first face, and the step between its faces
	if (DIM == 1) {
		const long long k = col / P.nx;
		const int i = (int)(col - k * P.nx);
		base = i + (long long)P.nx * P.ny * k;
		t0 = i + (long long)P.nx * (P.ny + 1) * k;
		stride = P.nx;
	} else {
		base = t0 = col;
		stride = (long long)P.nx * P.ny;
	}
	const int f1 = min(f0 + chunk, n + 1);
	double c[7], L[7], R[7], F[7];
	if (P.order != 1) {
		load_line<DIM, ND>(P, S, base, f0 - 1, L);
		for (int f = f0; f < f1; ++f) {
			load_line<DIM, ND>(P, S, base, f, c);
			face_solve<DIM, ND>(P, L, c, F);
			store_flux<DIM>(S, t0 + f * stride, F);
#pragma unroll
			for (int q = 0; q < NU; ++q) L[q] = c[q];
		}
		return;
	}
	{
		double a[7], b[7], s[7];
		load_line<DIM, ND>(P, S, base, f0 - 2, a);
		load_line<DIM, ND>(P, S, base, f0 - 1, b);
		load_line<DIM, ND>(P, S, base, f0, c);
		cell_slopes<ND>(P.limiter, a, b, c, s);
#pragma unroll
		for (int q = 0; q < NU; ++q) {
			L[q] = b[q] + 0.5 * s[q];
			R[q] = b[q];  // the cell before c, until the loop forms the face's right state
		}
	}
	for (int f = f0; f < f1; ++f) {
		double e[7], s[7];
		load_line<DIM, ND>(P, S, base, f + 1, e);
		cell_slopes<ND>(P.limiter, R, c, e, s);
#pragma unroll
		for (int q = 0; q < NU; ++q) {
			s[q] = 0.5 * s[q];
			R[q] = c[q] - s[q];
		}
		face_solve<DIM, ND>(P, L, R, F);
		store_flux<DIM>(S, t0 + f * stride, F);
#pragma unroll
		for (int q = 0; q < NU; ++q) {
			L[q] = c[q] + s[q];
			R[q] = c[q];
			c[q] = e[q];
		}
	}
}

// One face anywhere (t: its index in S.F[DIM]): the batches, whose grids are
// laid end to end face by face, and the FP32 form's list of FP64 faces.
template <int DIM, int ND>
__device__ __forceinline__ void one_face(const Params& P, const State& S, long long t) {
	if (DIM == 0) {
		const long long row = t / (P.nx + 1);
		const int f = (int)(t - row * (P.nx + 1));
		double a[7], b[7], c[7], e[7], s[7], F[7];
		load_line<0, ND>(P, S, row * P.nx, f - 1, b);
		load_line<0, ND>(P, S, row * P.nx, f, c);
		if (P.order == 1) {
			load_line<0, ND>(P, S, row * P.nx, f - 2, a);
			load_line<0, ND>(P, S, row * P.nx, f + 1, e);
			cell_slopes<ND>(P.limiter, a, b, c, s);
#pragma unroll
			for (int q = 0; q < NU; ++q) a[q] = b[q] + 0.5 * s[q];
			cell_slopes<ND>(P.limiter, b, c, e, s);
#pragma unroll
			for (int q = 0; q < NU; ++q) {
				b[q] = a[q];
				c[q] = c[q] - 0.5 * s[q];
			}
		}
		face_solve<0, ND>(P, b, c, F);
		store_flux<0>(S, t, F);
		return;
	}
	const long long plane = DIM == 1 ? P.nx : (long long)P.nx * P.ny;
	const long long rest = t / plane;
	if (DIM == 1) {
		const long long k = rest / (P.ny + 1);
		faces_column<1, ND>(P, S, (t - rest * plane) + P.nx * k, (int)(rest - k * (P.ny + 1)), 1);
	} else {
		faces_column<2, ND>(P, S, t - rest * plane, (int)rest, 1);
	}
}
__device__ __forceinline__ void one_face_of(const Params& P, const State& S, long long t, int dim) {
	if (P.nd == 3) {
		if (dim == 0) one_face<0, 3>(P, S, t);
		else if (dim == 1) one_face<1, 3>(P, S, t);
		else one_face<2, 3>(P, S, t);
	} else if (P.nd == 2) {
		if (dim == 0) one_face<0, 2>(P, S, t);
		else one_face<1, 2>(P, S, t);
	} else {
		one_face<0, 1>(P, S, t);
	}
}
// Every face of a batch along dim.
__global__ void __launch_bounds__(128) k_faces_batch_fp64(Params P, State S, int dim) {
	grid_begin();
#if TRG_BATCHED
	const BatchTable& B = *P.batch;
	const long long* off = B.face_off[dim];
	const int g = batch_slot(off, B.G, blockIdx.x * (long long)blockDim.x);
	const long long lt = blockIdx.x * (long long)blockDim.x + threadIdx.x - off[g];
	if (lt < B.S[g].nfaces[dim]) one_face_of(B.P[g], B.S[g], lt, dim);
#endif
}
// Every face of one grid in one launch: blocks [0, G.bx) take the x faces,
// [G.bx, G.bx + G.by) the y faces and the rest the z faces (FaceGrid,
// trg_types.h), so that a small grid's three directions run side by side.
template <int ND>
__device__ __forceinline__ void all_faces(const Params& P, const State& S, const FaceGrid& G) {
	const unsigned b = blockIdx.x;
	if (b < G.bx) {
		faces_x<ND>(P, S, b * 4LL + (threadIdx.x >> 5));
		return;
	}
	const bool y = b < G.bx + G.by;
	const long long cols = y ? (long long)P.nx * P.nz : (long long)P.nx * P.ny;
	const long long t = (b - G.bx - (y ? 0 : G.by)) * 128LL + threadIdx.x;
	const long long c = t / cols;  // which chunk of the columns
	if (y) {
		if (ND > 1 && c * G.chunk <= P.ny) faces_column<1, ND>(P, S, t - c * cols, (int)c * G.chunk, G.chunk);
	} else {
		if (ND > 2 && c * G.chunk <= P.nz) faces_column<2, ND>(P, S, t - c * cols, (int)c * G.chunk, G.chunk);
	}
}
__global__ void __launch_bounds__(128) k_faces1_fp64(Params P, State S, FaceGrid G) {
	grid_begin();
	all_faces<1>(P, S, G);
}
__global__ void __launch_bounds__(128, 4) k_faces2_fp64(Params P, State S, FaceGrid G) {
	grid_begin();
	all_faces<2>(P, S, G);
}
__global__ void __launch_bounds__(128, 4) k_faces3_fp64(Params P, State S, FaceGrid G) {
	grid_begin();
	all_faces<3>(P, S, G);
}
