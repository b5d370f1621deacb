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
//    independent ones overlap (Recip, trg_device.cuh), and those by a divisor known before
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

// A thread's cell of a shell: its position p in the sweep list, cell id,
// weights, ring places of its neighbours (-1: not read, or a wind cell, whose
// optical depths are 0) and inputs.
template <bool RAD>
struct ChainItem {
	int p, id;
	int4 slot;
	double w[4];
	double own;  // column density
	SolveCell c;  // radiation
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
		const SolveCell& c = it.c;
		tau_interp2(P, a, b, it.w, r.tau, r.tau_a);
		solve_cell(P, S, c, dt, r.tau_a, r.x, r.x_avg);
		r.dtau = (1.0 - r.x) * c.n_H * P.photoIonXsec * c.ds;
		r.dtau_a = (1.0 - r.x_avg) * c.n_H * P.photoIonXsec * c.ds;
		return make_double2(r.tau + r.dtau, r.tau_a + r.dtau_a);
	}
	r.tau = colden_interp_recip(a, it.w);
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
		if (RAD && cur.id >= 0) solve_pre(P, cur.c);
		if (s > 0) asm volatile("bar.sync %0, %1;" ::"r"(1 + ((s - 1) & 1)), "r"(2 * T) : "memory");
		ChainResult r;
		if (cur.id >= 0) out[tid] = chain_cell<RAD>(P, S, cur, ring, dt, r);
		for (int t = tid + T; t < n; t += T) {  // shells of more than T cells
			ChainItem<RAD> more;
			ChainResult rm;
			more.load(ch, S, o0 + t);
			if (RAD) solve_pre(P, more.c);
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
	grid_begin();
	chain_kernel<true>(P, S, h);
}
__global__ void __launch_bounds__(2 * CHAIN_GROUP, 1) k_colden_chain(Params P, State S) {
	grid_begin();
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
