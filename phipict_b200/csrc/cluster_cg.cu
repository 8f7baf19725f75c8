// CG of small instances, one thread-block cluster per instance (one right-hand side): the solve of
// kCgPersistent (persistent.cu) for instances of at most CCG_MAX_TILES tiles.
//
// What bounds it: latency. An iteration of the grid-wide kernel on such an instance is two grid
// barriers and some ten dependent L2 round trips, 8 us at 2 tiles and 12 us at 16, whatever the
// arithmetic. Here r, p and q of a tile stay in the shared memory of the CTA that owns it, the
// stencil rows, x and the neighbours' addresses in registers, p is read at the neighbours through
// distributed shared memory, and the phases meet at cluster barriers; partial sums are written to
// every CTA of the cluster and reduced by each of them. Nothing but the result goes to memory.
// Instances of a batch run and stop independently. A cluster has 16 CTAs at most and a CTA two
// tiles (512 threads of 128 registers), which sets the size up to which it applies.
//
// Same arithmetic and summation order as the tile bodies of phb_krylov.cuh (same bits): the inner
// products are summed over four consecutive cells per thread, the stencil work is done on cells
// 256 apart, which keeps shared memory free of bank conflicts for every row length.
// Measured (B200, per iteration): 2 tiles float32 7.9 -> 2.7 us, 16 tiles float64 11.9 -> 3.4 us.
#include <atomic>
#include "phb_krylov.cuh"

namespace phb {

constexpr int CCG_MAX_CTAS = 16;
constexpr int CCG_SLOTS = 2;
constexpr int CCG_MAX_TILES = CCG_MAX_CTAS * CCG_SLOTS; // a warp reduces the partials, a lane per tile
static_assert(CCG_MAX_TILES <= 32, "one lane per tile");

template <typename T, int D>
struct CcgArgs {
	Dom<double, D> dom;
	const T *A, *b;
	T *x;
	SysState *st;
	Control *ctrl;
	phb_tolerance tol;
	int returnBest, maxit, stopStart, fromInner, slots;
};

__device__ __forceinline__ unsigned int clusterRank() {
	unsigned int r;
	asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
	return r;
}
__device__ __forceinline__ unsigned int clusterSize() {
	unsigned int r;
	asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
	return r;
}
// every thread of every CTA of the cluster takes it
__device__ __forceinline__ void clusterBarrier() {
	asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// address of this CTA's shared variable in CTA `rank` of the cluster
__device__ __forceinline__ unsigned int clusterAddr(const void *p, unsigned int rank) {
	const unsigned int a = (unsigned int)__cvta_generic_to_shared(p);
	unsigned int r;
	asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
	return r;
}
__device__ __forceinline__ float ldCluster(unsigned int a, float) {
	float v;
	asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
	return v;
}
__device__ __forceinline__ double ldCluster(unsigned int a, double) {
	double v;
	asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
	return v;
}
__device__ __forceinline__ void stCluster(unsigned int a, double v) {
	asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

template <typename T, int D>
__global__ void __launch_bounds__(PHB_TILE *CCG_SLOTS, 1) kCgCluster(const __grid_constant__ CcgArgs<T, D> a) {
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ SysState ss;
	__shared__ double part[2][2][CCG_MAX_TILES]; // [parity][quantity][tile]
	__shared__ double wsum[CCG_SLOTS][2][NWARPS];
	const int slots = a.slots;
	const int slot = int(threadIdx.x) / PHB_TILE, lt = int(threadIdx.x) & (PHB_TILE - 1);
	const int lane = threadIdx.x & 31, warp = lt >> 5;
	const unsigned int rank = clusterRank(), csize = clusterSize();
	const int inst = int(blockIdx.x / csize);
	const int32_t *in = a.dom.insts + inst * PHB_IREC;
	const int t0 = __ldg(in + I_TILESTART), tc = __ldg(in + I_TILECOUNT);
	T *rS = reinterpret_cast<T *>(smem), *pS = rS + slots * PHB_TILE_CELLS, *qS = pS + slots * PHB_TILE_CELLS;
	T *rT = rS + slot * PHB_TILE_CELLS, *pT = pS + slot * PHB_TILE_CELLS, *qT = qS + slot * PHB_TILE_CELLS;
	const int tile = int(rank) * slots + slot; // of the instance
	const bool own = tile < tc;
	const int64_t N = a.dom.ncells;
	if (threadIdx.x == 0) {
		ss = initialState(a.tol, inst, a.fromInner ? a.st[inst].innerTol : 0.0, a.fromInner, a.maxit);
		if (blockIdx.x == 0) a.ctrl->barErr = 0; // phb_solve_results reads it
	}
	// this thread's cells lt, lt + 256, ... of its tile: stencil rows, the neighbours' addresses in
	// the cluster's p arrays (a face without neighbour: the cell itself with coefficient 0), x, b
	T c0[CPT], cf[CPT][2 * D], xv[CPT], xb[CPT];
	unsigned int na[CPT][2 * D];
	int nc = 0;        // cells of the tile
	int64_t g0 = 0;    // its first cell
#pragma unroll
	for (int j = 0; j < CPT; ++j) {
		c0[j] = 0;
		xv[j] = xb[j] = 0;
#pragma unroll
		for (int f = 0; f < 2 * D; ++f) { cf[j][f] = 0; na[j][f] = 0; }
	}
	if (own) {
		const int b = __ldg(a.dom.tiles + 2 * (t0 + tile)), l0 = __ldg(a.dom.tiles + 2 * (t0 + tile) + 1);
		const int32_t *B = a.dom.blk(b);
		const int nx = B[B_NX], ny = B[B_NY], n = nx * ny * (D > 2 ? B[B_NZ] : 1);
		nc = min(PHB_TILE_CELLS, n - l0);
		g0 = (int64_t)B[B_CELLOFF] + l0;
#pragma unroll
		for (int j = 0; j < CPT; ++j) {
			const int l = lt + j * PHB_TILE;
			if (l >= nc) {
				rT[l] = pT[l] = qT[l] = 0;
				continue;
			}
			Cell c;
			c.B = B;
			c.b = b;
			const int row = (l0 + l) / nx;
			c.p[0] = l0 + l - row * nx;
			c.p[1] = D > 2 ? row % ny : row;
			c.p[2] = D > 2 ? row / ny : 0;
			c.g = (int)(g0 + l);
			c.mi = 0;
			c0[j] = a.A[c.g];
			xv[j] = a.x[c.g];
#pragma unroll
			for (int f = 0; f < 2 * D; ++f) {
				int64_t nb = c.g;
				const int32_t *NB = B;
				const bool end = atBound(B, f, c.p);
				if (!end || fType(B, f) != FT_FIXED) {
					const Nbr k = neighbor<double, D>(a.dom, c, f);
					nb = k.g;
					NB = k.B;
					cf[j][f] = a.A[(f + 1) * N + c.g];
				}
				const int nl = (int)(nb - NB[B_CELLOFF]);
				const int nt = NB[B_TILESTART] + nl / PHB_TILE_CELLS - t0;
				const int nr = nt / slots;
				na[j][f] = clusterAddr(pS + (nt - nr * slots) * PHB_TILE_CELLS + nl % PHB_TILE_CELLS, (unsigned int)nr);
			}
		}
	}
	// y = A p at this thread's cells
	auto apply = [&](T(&y)[CPT]) {
		constexpr int J = sizeof(T) == 8 && D == 3 ? 2 : CPT; // cells whose loads are in flight together
#pragma unroll
		for (int j0 = 0; j0 < CPT; j0 += J) {
			T v[J][2 * D];
#pragma unroll
			for (int j = 0; j < J; ++j)
#pragma unroll
				for (int f = 0; f < 2 * D; ++f) v[j][f] = lt + (j0 + j) * PHB_TILE < nc ? ldCluster(na[j0 + j][f], T(0)) : T(0);
#pragma unroll
			for (int j = 0; j < J; ++j) {
				const int l = lt + (j0 + j) * PHB_TILE;
				y[j0 + j] = l < nc ? c0[j0 + j] * pT[l] : T(0);
#pragma unroll
				for (int f = 0; f < 2 * D; ++f) y[j0 + j] = fma(cf[j0 + j][f], v[j][f], y[j0 + j]);
			}
		}
	};
	auto tileSync = [&] { asm volatile("barrier.sync %0, %1;" ::"r"(slot + 1), "n"(PHB_TILE) : "memory"); };
	// sums over the tile of u v (and of w w) in the order of the tile bodies, sent to every CTA; the
	// cluster barrier that follows makes them visible
	int par = 0;
	auto sendSums = [&](const T *u, const T *v, const T *w) {
		double acc[2] = {0, 0};
		tileSync(); // the tile's values are in shared memory
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			acc[0] = fma(double(u[4 * lt + i]), double(v[4 * lt + i]), acc[0]);
			if (w) acc[1] = fma(double(w[4 * lt + i]), double(w[4 * lt + i]), acc[1]);
		}
		acc[0] = warpSum(acc[0]);
		if (w) acc[1] = warpSum(acc[1]);
		if (lane == 0) { wsum[slot][0][warp] = acc[0]; wsum[slot][1][warp] = acc[1]; }
		tileSync();
		if (own && lt < 2 * CCG_MAX_CTAS) {
			const int q = lt / CCG_MAX_CTAS;
			const unsigned int to = lt % CCG_MAX_CTAS;
			if (to < csize && (q == 0 || w)) {
				double s = 0;
#pragma unroll
				for (int k = 0; k < NWARPS; ++k) s += wsum[slot][q][k];
				stCluster(clusterAddr(&part[par][q][tile], to), s);
			}
		}
		clusterBarrier();
		par ^= 1;
	};
	// the first warp reduces quantity q of the last sums and calls fn(sum 0, sum 1) in one lane
	auto decide = [&](auto fn) {
		if (threadIdx.x < 32) {
			const double s0 = warpSum(lane < tc ? part[par ^ 1][0][lane] : 0.0);
			const double s1 = warpSum(lane < tc ? part[par ^ 1][1][lane] : 0.0);
			if (lane == 0) fn(s0, s1);
		}
		__syncthreads();
	};
	// r = b - A x through the p array
#pragma unroll
	for (int j = 0; j < CPT; ++j) {
		const int l = lt + j * PHB_TILE;
		if (l < nc) { pT[l] = xv[j]; qT[l] = a.b[g0 + l]; }
		else if (!own) rT[l] = pT[l] = qT[l] = 0;
	}
	if (threadIdx.x < 4 * CCG_MAX_TILES) (&part[0][0][0])[threadIdx.x] = 0.0;
	clusterBarrier();
	{
		T y[CPT];
		apply(y);
#pragma unroll
		for (int j = 0; j < CPT; ++j) {
			const int l = lt + j * PHB_TILE;
			if (l < nc) rT[l] = qT[l] - y[j];
		}
	}
	sendSums(rT, rT, qT);
	const double ns = normScale(a.dom.insts, inst);
	decide([&](double rr, double bb) {
		if (ss.done != RUNNING) return;
		const double red[1] = {rr};
		if (a.stopStart) residualDecision<1, false, true>(nullptr, ss, ns, red, bb, a.tol);
		else residualDecision<1, false, false>(nullptr, ss, ns, red, bb, a.tol);
	});
	for (int iter = 0; ss.done == RUNNING && iter <= a.maxit + 1; ++iter) {
		// p' = r + beta p
		{
			const T beta = T(ss.beta);
			const bool rs = ss.restart;
#pragma unroll
			for (int j = 0; j < CPT; ++j) {
				const int l = lt + j * PHB_TILE;
				if (l < nc) pT[l] = rs ? rT[l] : fma(beta, pT[l], rT[l]);
			}
		}
		clusterBarrier();
		// q = A p', (p', q)
		T y[CPT];
		apply(y);
#pragma unroll
		for (int j = 0; j < CPT; ++j) {
			const int l = lt + j * PHB_TILE;
			if (l < nc) qT[l] = y[j];
		}
		sendSums(pT, qT, nullptr);
		decide([&](double pq, double) {
			const double alpha = ss.rho / pq;
			ss.restart = 0;
			if (!fin(alpha)) { ss.done = NONFINITE; ss.usedIt = ss.it; }
			else ss.alpha = alpha;
		});
		if (ss.done != RUNNING) break;
		// x += alpha p', r -= alpha q, (r, r)
		{
			const T alpha = T(ss.alpha);
			const bool save = ss.saveBest;
#pragma unroll
			for (int j = 0; j < CPT; ++j) {
				const int l = lt + j * PHB_TILE;
				if (l >= nc) continue;
				if (save) xb[j] = xv[j];
				xv[j] = fma(alpha, pT[l], xv[j]);
				rT[l] = fma(-alpha, y[j], rT[l]);
			}
		}
		sendSums(rT, rT, nullptr);
		decide([&](double rr, double) {
			SysState &s = ss;
			const double crit = sqrt(rr) * ns;
			++s.it;
			s.crit = crit;
			s.saveBest = 0;
			s.usedIt = s.it - 1;
			if (!fin(crit)) { s.done = NONFINITE; return; }
			if (a.returnBest) {
				if (crit < s.best) { s.best = crit; s.bestIt = s.it - 1; s.saveBest = 1; }
				if (s.it > 1 && crit >= s.last) ++s.rising; else s.rising = 0;
				s.last = crit;
			}
			if (crit < s.tol) s.done = CONVERGED;
			else if (s.it >= s.maxit) s.done = MAXIT;
			else if (a.returnBest && s.rising >= RISING_CUTOFF) s.done = RISING;
			else {
				s.beta = rr / s.rho;
				s.rho = rr;
				if (!fin(s.beta)) s.done = NONFINITE;
			}
		});
	}
	// the result; a system that stopped without converging returns its best iterate
	const bool best = a.returnBest && (ss.done == MAXIT || ss.done == RISING) && ss.bestIt >= 0 && ss.best < ss.crit;
#pragma unroll
	for (int j = 0; j < CPT; ++j) {
		const int l = lt + j * PHB_TILE;
		if (l < nc) a.x[g0 + l] = best ? xb[j] : xv[j];
	}
	if (rank == 0 && threadIdx.x == 0) a.st[inst] = ss;
	clusterBarrier(); // no CTA leaves while another may still read its shared memory
}

// Whether `ninst` clusters, `resident` of them at a time, beat the grid-wide kernel: its iteration takes
// about 8 us and 0.24 us more per instance (every SM sums every system; flat from some 128 instances
// on), a cluster's 3.7 us. Every cluster has the size that the largest instance may have, so a batch of many
// small instances and one large one holds few at a time. Measured (microseconds per iteration of all, cluster
// and grid): 22 instances of 2 tiles in clusters of 32 tiles, 7 at a time, 13.3 and 11.5, 16 of them
// 10.2 and 10.3; 64 in clusters of 16 tiles, 14 at a time, 15.7 and 22.7; 301 66 and 38; 301 in clusters of 8 29 and 38.
inline bool clustersWin(int ninst, int resident) {
	const int64_t waves = (ninst + resident - 1) / resident;
	return 31 * waves <= 66 + 2 * std::min(ninst, 128);
}

// Launch the cluster solve when every instance fits a cluster (the largest has at most all tiles but
// one per other instance), the device can hold such a cluster and holds enough of them at a time;
// *taken says whether it did.
template <typename T, int D>
int launchClusterCg(const phb_domain *dom, const phb_solve *sv, cudaStream_t s, bool stopStart, int fromInner, bool *taken) {
	*taken = false;
	const int tiles = dom->ntiles - (dom->ninst - 1);
	if (sv->ctas_per_sm > 0 || tiles < 1 || tiles > CCG_MAX_TILES) return PHB_OK;
	const int slots = tiles > CCG_MAX_CTAS ? 2 : 1;
	int csize = 1, lg = 0;
	while (csize * slots < tiles) { csize *= 2; ++lg; }
	auto kern = kCgCluster<T, D>;
	const size_t smem = (size_t)slots * 3 * PHB_TILE_CELLS * sizeof(T);
	cudaLaunchConfig_t cfg = {};
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeClusterDimension;
	attr[0].val.clusterDim.x = csize;
	attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
	cfg.gridDim = dim3(dom->ninst * csize);
	cfg.blockDim = dim3(PHB_TILE * slots);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	// such clusters that this device holds at a time, -1: none (asked once per device and shape)
	static std::atomic<int> fits[64][CCG_SLOTS][5];
	int dev = 0;
	PHB_CUDA(cudaGetDevice(&dev));
	if (dev < 0 || dev >= 64) return PHB_OK;
	int resident = fits[dev][slots - 1][lg].load();
	if (resident == 0) {
		PHB_CUDA(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CCG_SLOTS * 3 * PHB_TILE_CELLS * (int)sizeof(T)));
		PHB_CUDA(cudaFuncSetAttribute((const void *)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
		int n = 0;
		cudaLaunchConfig_t full = cfg; // the device's capacity, whatever this launch's grid
		full.gridDim = dim3(csize * numSMs());
		resident = cudaOccupancyMaxActiveClusters(&n, (const void *)kern, &full) == cudaSuccess && n >= 1 ? n : -1;
		if (resident < 0) (void)cudaGetLastError();
		fits[dev][slots - 1][lg].store(resident);
	}
	if (resident < 0 || !clustersWin(dom->ninst, resident)) return PHB_OK;
	const StateLayout SL = stateLayout(dom, 1);
	CcgArgs<T, D> a = {};
	a.dom = Dom<double, D>(*dom);
	a.A = (const T *)sv->A;
	a.b = (const T *)sv->b;
	a.x = (T *)sv->x;
	a.st = (SysState *)((char *)sv->state + SL.st);
	a.ctrl = (Control *)((char *)sv->state + SL.ctrl);
	a.tol = sv->tol;
	a.returnBest = sv->return_best;
	a.maxit = std::max(1, sv->maxit);
	a.stopStart = stopStart;
	a.fromInner = fromInner;
	a.slots = slots;
	PHB_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
	*taken = true;
	return PHB_OK;
}
#define PHB_CLUSTER(T, D) template int launchClusterCg<T, D>(const phb_domain *, const phb_solve *, cudaStream_t, bool, int, bool *);
PHB_CLUSTER(float, 2)
PHB_CLUSTER(float, 3)
PHB_CLUSTER(double, 2)
PHB_CLUSTER(double, 3)

} // namespace phb
