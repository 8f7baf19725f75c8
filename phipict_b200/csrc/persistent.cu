// The persistent Krylov solvers: one cooperative launch runs a whole CG or BiCGStab solve, with
// grid barriers between its phases (phb_krylov.cuh). The multigrid-preconditioned CG is in pcg.cu.
#include "phb_krylov.cuh"

namespace phb {

template <typename T, int D, int K, bool STOPSTART>
__device__ __forceinline__ void cgPersistentBody(const Dom<double, D> &dom, const T *__restrict__ A, const T *__restrict__ b,
		T *__restrict__ x, T *__restrict__ r, T *__restrict__ p0, T *__restrict__ p1, T *__restrict__ q, T *__restrict__ xbest,
		SysState *st, double *partial, Control *ctrl, const phb_tolerance &tol, int returnBest, int maxit) {
	extern __shared__ SysState sst[];
	__shared__ int32_t sB[PHB_BREC];
	const int nsys = dom.ninst * K;
	for (int s = threadIdx.x; s < nsys; s += blockDim.x) sst[s] = st[s];
	__syncthreads();
	const int64_t N = dom.ncells;
	// consecutive phases write alternate halves of the partials, so that a CTA that has left
	// a barrier cannot overwrite partials another CTA is still reducing
	const size_t half = (size_t)dom.ntiles * K * 3;
	int ph = 0;
	double *pp = partial;
	// r = b - A x, (r, r), (b, b)
	pp = partial + (size_t)(ph++ & 1) * half;
	forMyTiles<D>(dom, sB, [&](int tile, int l0, int nc) {
		const int inst = sB[B_INST];
		bool act[K];
#pragma unroll
		for (int k = 0; k < K; ++k) act[k] = sst[inst * K + k].done == RUNNING;
		double acc[2 * K];
#pragma unroll
		for (int k = 0; k < 2 * K; ++k) acc[k] = 0;
		tileResidual<T, D, K>(dom, sB, l0, nc, A, b, x, act, acc,
				[&](int, int64_t o, const Quad &q, const T (&rv)[4]) { st4(r + o, q.n, q.al, rv); });
		blockSumTo<2 * K>(acc, pp + (size_t)tile * 2 * K);
	});
	if (!gridBarrier(ctrl)) return;
	int running = reduceStates<K, 2, 1>(dom.insts, dom.ninst, pp, sst, [&](SysState &s, int in, const double *red, double bb) {
		residualDecision<K, false, STOPSTART>(nullptr, s, normScale(dom.insts, in), red, bb, tol);
	});
	T *pIn = p0, *pOut = p1;
	for (int iter = 0; running > 0 && iter <= maxit + 1; ++iter) {
		// p' = r + beta p, q = A p', (p', q)
		pp = partial + (size_t)(ph++ & 1) * half;
		forMyTiles<D>(dom, sB, [&](int tile, int l0, int nc) {
			const int inst = sB[B_INST];
			bool act[K], rs[K];
			T beta[K];
#pragma unroll
			for (int k = 0; k < K; ++k) {
				const SysState &s = sst[inst * K + k];
				act[k] = s.done == RUNNING;
				rs[k] = s.restart;
				beta[k] = T(s.beta);
			}
			double acc[K];
#pragma unroll
			for (int k = 0; k < K; ++k) acc[k] = 0;
			tileCgDirection<T, D, K>(dom, sB, l0, nc, A, r, pIn, pOut, q, act, rs, beta, acc);
			blockSumTo<K>(acc, pp + (size_t)tile * K);
		});
		if (!gridBarrier(ctrl)) return;
		reduceStates<K, 1>(dom.insts, dom.ninst, pp, sst, [&](SysState &s, int, const double *red, double) {
			const double alpha = s.rho / red[0];
			s.restart = 0;
			if (!fin(alpha)) { s.done = NONFINITE; s.usedIt = s.it; }
			else s.alpha = alpha;
		});
		// x += alpha p', r -= alpha q, (r, r)
		pp = partial + (size_t)(ph++ & 1) * half;
		forMyTiles<D>(dom, sB, [&](int tile, int l0, int nc) {
			double acc[K];
#pragma unroll
			for (int k = 0; k < K; ++k) acc[k] = 0;
			tileCgUpdate<T, D, K>(dom, sB, l0, nc, r, pOut, q, x, xbest, sst, acc);
			blockSumTo<K>(acc, pp + (size_t)tile * K);
		});
		if (!gridBarrier(ctrl)) return;
		running = reduceStates<K, 1>(dom.insts, dom.ninst, pp, sst, [&](SysState &s, int in, const double *red, double) {
			const double crit = sqrt(red[0]) * normScale(dom.insts, in);
			++s.it;
			s.crit = crit;
			s.saveBest = 0;
			s.usedIt = s.it - 1;
			if (!fin(crit)) { s.done = NONFINITE; return; }
			if (returnBest) {
				if (crit < s.best) { s.best = crit; s.bestIt = s.it - 1; s.saveBest = 1; }
				if (s.it > 1 && crit >= s.last) ++s.rising; else s.rising = 0;
				s.last = crit;
			}
			if (crit < s.tol) s.done = CONVERGED;
			else if (s.it >= s.maxit) s.done = MAXIT;
			else if (returnBest && s.rising >= RISING_CUTOFF) s.done = RISING;
			else {
				s.beta = red[0] / s.rho;
				s.rho = red[0];
				if (!fin(s.beta)) s.done = NONFINITE;
			}
		});
		T *tmp = pIn; pIn = pOut; pOut = tmp;
	}
	// systems that stopped without converging return their best iterate (kRestoreBest)
	if (xbest) {
		forMyTiles<D>(dom, sB, [&](int, int l0, int nc) {
			const int inst = sB[B_INST];
			for (int j = 0; j < CPT; ++j) {
				Cell c;
				if (!cellAt<D>(sB, l0, nc, j, c)) break;
#pragma unroll
				for (int k = 0; k < K; ++k) {
					const SysState &s = sst[inst * K + k];
					if ((s.done == MAXIT || s.done == RISING) && s.bestIt >= 0 && s.best < s.crit) {
						const int64_t o = vk<K>(c.B, c.g, k);
						x[o] = xbest[o];
					}
				}
			}
		});
	}
	if (blockIdx.x == 0) {
		__syncthreads();
		for (int s = threadIdx.x; s < nsys; s += blockDim.x) st[s] = sst[s];
	}
}

// Resident CTAs per SM that the register budget must allow. The plain float32 CG is bound
// by HBM on large grids and is faster with more warps in flight: four CTAs in 3D (64
// registers), five in 2D (48), which it fits without spilling. Several right-hand sides and
// float64 need more registers per thread.
template <typename T, int D, int K>
constexpr int cgMinBlocks() {
	return (std::is_same<T, float>::value && K == 1) ? (D == 2 ? 5 : 4) : (K == 1 ? 3 : 2);
}

template <typename T, int D, int K, bool STOPSTART>
__global__ void __launch_bounds__(PHB_TILE, (cgMinBlocks<T, D, K>())) kCgPersistent(Dom<double, D> dom, const T *__restrict__ A, const T *__restrict__ b,
		T *__restrict__ x, T *__restrict__ r, T *__restrict__ p0, T *__restrict__ p1, T *__restrict__ q, T *__restrict__ xbest,
		SysState *st, double *partial, Control *ctrl, phb_tolerance tol, int returnBest, int maxit) {
	cgPersistentBody<T, D, K, STOPSTART>(dom, A, b, x, r, p0, p1, q, xbest, st, partial, ctrl, tol, returnBest, maxit);
}

template <typename T, int D, int K>
__global__ void __launch_bounds__(PHB_TILE) kBicgPersistent(Dom<double, D> dom, const T *__restrict__ A, const T *__restrict__ b,
		T *__restrict__ x, T *__restrict__ r, T *__restrict__ r0, T *__restrict__ p0, T *__restrict__ p1, T *__restrict__ v0,
		T *__restrict__ v1, T *__restrict__ t, SysState *st, double *partial, Control *ctrl, phb_tolerance tol, int maxit) {
	extern __shared__ SysState sst[];
	__shared__ int32_t sB[PHB_BREC];
	const int nsys = dom.ninst * K;
	for (int s = threadIdx.x; s < nsys; s += blockDim.x) sst[s] = st[s];
	__syncthreads();
	const int64_t N = dom.ncells;
	// consecutive phases write alternate halves of the partials, so that a CTA that has left
	// a barrier cannot overwrite partials another CTA is still reducing
	const size_t half = (size_t)dom.ntiles * K * 3;
	int ph = 0;
	double *pp = partial;
	pp = partial + (size_t)(ph++ & 1) * half;
	forMyTiles<D>(dom, sB, [&](int tile, int l0, int nc) {
		const int inst = sB[B_INST];
		bool act[K];
#pragma unroll
		for (int k = 0; k < K; ++k) act[k] = sst[inst * K + k].done == RUNNING;
		double acc[2 * K];
#pragma unroll
		for (int k = 0; k < 2 * K; ++k) acc[k] = 0;
		tileResidual<T, D, K>(dom, sB, l0, nc, A, b, x, act, acc, [&](int, int64_t o, const Quad &q, const T (&rv)[4]) {
			st4(r + o, q.n, q.al, rv);
			st4(r0 + o, q.n, q.al, rv);
		});
		blockSumTo<2 * K>(acc, pp + (size_t)tile * 2 * K);
	});
	if (!gridBarrier(ctrl)) return;
	int running = reduceStates<K, 2, 1>(dom.insts, dom.ninst, pp, sst, [&](SysState &s, int in, const double *red, double bb) {
		residualDecision<K, true, true>(nullptr, s, normScale(dom.insts, in), red, bb, tol);
	});
	T *pIn = p0, *pOut = p1, *vIn = v0, *vOut = v1;
	for (int iter = 0; running > 0 && iter <= maxit + 1; ++iter) {
		// p = r + beta (p - omega v), v = A p, (r0, v)
		pp = partial + (size_t)(ph++ & 1) * half;
		forMyTiles<D>(dom, sB, [&](int tile, int l0, int nc) {
			const int inst = sB[B_INST];
			bool act[K], rs[K];
			T beta[K], omega[K];
#pragma unroll
			for (int k = 0; k < K; ++k) {
				const SysState &s = sst[inst * K + k];
				act[k] = s.done == RUNNING;
				rs[k] = s.restart;
				beta[k] = T(s.beta);
				omega[k] = T(s.omega);
			}
			double acc[K];
#pragma unroll
			for (int k = 0; k < K; ++k) acc[k] = 0;
			tileBicgV<T, D, K>(dom, sB, l0, nc, A, r, pIn, vIn, pOut, vOut, r0, act, rs, beta, omega, acc);
			blockSumTo<K>(acc, pp + (size_t)tile * K);
		});
		if (!gridBarrier(ctrl)) return;
		reduceStates<K, 1>(dom.insts, dom.ninst, pp, sst, [&](SysState &s, int, const double *red, double) {
			const double alpha = s.rho / red[0];
			s.restart = 0;
			if (!fin(alpha)) { s.done = NONFINITE; s.usedIt = s.it; }
			else s.alpha = alpha;
		});
		// s = r - alpha v, t = A s, (t,s), (t,t), (s,s)
		pp = partial + (size_t)(ph++ & 1) * half;
		forMyTiles<D>(dom, sB, [&](int tile, int l0, int nc) {
			const int inst = sB[B_INST];
			bool act[K];
			T alpha[K];
#pragma unroll
			for (int k = 0; k < K; ++k) {
				const SysState &s = sst[inst * K + k];
				act[k] = s.done == RUNNING;
				alpha[k] = T(s.alpha);
			}
			double acc[3 * K];
#pragma unroll
			for (int k = 0; k < 3 * K; ++k) acc[k] = 0;
			tileBicgT<T, D, K>(dom, sB, l0, nc, A, r, vOut, t, act, alpha, acc);
			blockSumTo<3 * K>(acc, pp + (size_t)tile * 3 * K);
		});
		if (!gridBarrier(ctrl)) return;
		reduceStates<K, 3>(dom.insts, dom.ninst, pp, sst, [&](SysState &s, int in, const double *red, double) {
			const double critS = sqrt(red[2]) * normScale(dom.insts, in);
			s.halfCrit = critS;
			if (!fin(critS)) { s.done = NONFINITE; s.crit = critS; s.usedIt = s.it; }
			else if (critS < s.tol) { s.halfDone = 1; s.omega = 0.0; }
			else {
				const double omega = red[0] / red[1];
				if (!fin(omega)) { s.done = NONFINITE; s.crit = critS; s.usedIt = s.it; }
				else s.omega = omega;
			}
		});
		// x += alpha p + omega s, r = s - omega t, (r0, r), (r, r)
		pp = partial + (size_t)(ph++ & 1) * half;
		forMyTiles<D>(dom, sB, [&](int tile, int l0, int nc) {
			double acc[2 * K];
#pragma unroll
			for (int k = 0; k < 2 * K; ++k) acc[k] = 0;
			tileBicgUpdate<T, D, K>(dom, sB, l0, nc, r, r0, pOut, vOut, t, x, sst, acc);
			blockSumTo<2 * K>(acc, pp + (size_t)tile * 2 * K);
		});
		if (!gridBarrier(ctrl)) return;
		running = reduceStates<K, 2>(dom.insts, dom.ninst, pp, sst, [&](SysState &s, int in, const double *red, double) {
			if (s.halfDone) { s.done = CONVERGED; s.crit = s.halfCrit; s.usedIt = s.it; return; }
			const double crit = sqrt(red[1]) * normScale(dom.insts, in);
			s.crit = crit;
			if (!fin(crit)) { s.done = NONFINITE; s.usedIt = s.it; }
			else if (crit < s.tol) { s.done = CONVERGED; s.usedIt = s.it + 1; }
			else {
				++s.it;
				s.usedIt = s.it - 1;
				const double beta = (red[0] / s.rho) * (s.alpha / s.omega);
				s.rho = red[0];
				s.beta = beta;
				if (!fin(beta)) s.done = NONFINITE;
				else if (s.it >= s.maxit) s.done = MAXIT;
			}
		});
		T *tmp = pIn; pIn = pOut; pOut = tmp;
		tmp = vIn; vIn = vOut; vOut = tmp;
	}
	if (blockIdx.x == 0) {
		__syncthreads();
		for (int s = threadIdx.x; s < nsys; s += blockDim.x) st[s] = sst[s];
	}
}

// A persistent solve: kInit, then one cooperative launch of the whole iteration (the grid is
// sized so that every CTA is resident; the launch fails rather than deadlocks otherwise).
template <typename T, int D, int K>
int launchPersistent(const phb_domain *dom, const phb_solve *sv, cudaStream_t s, bool stopStart, int fromInner) {
	if constexpr (std::is_same<T, float>::value && K == 1) {
		if (sv->amg && sv->kind == 0) return launchPcg<D>(dom, sv, s, stopStart, fromInner);
	}
	Dom<double, D> dm(*dom);
	const Layout L = solveLayout(dom, sv->kind, sizeof(T), K);
	const StateLayout SL = stateLayout(dom, K);
	char *w = (char *)sv->work;
	char *sb = (char *)sv->state;
	Control *ctrl = (Control *)(sb + SL.ctrl);
	SysState *st = (SysState *)(sb + SL.st);
	double *partial = (double *)(w + L.off[10]);
	const T *A = (const T *)sv->A;
	const T *b = (const T *)sv->b;
	T *x = (T *)sv->x;
	dm.vec4 = vec4Ok(dom, {A, b, x, w});
	const int nsys = dom->ninst * K;
	const size_t smem = (size_t)nsys * sizeof(SysState);
	if (smem > 160 * 1024) return setError(PHB_ERR_RANGE, "persistent solve: too many systems for the per-CTA state copy");
	const int maxit = std::max(1, sv->maxit);
	const int rc = launchInit(st, nsys, sv->tol, fromInner, maxit, ctrl, s);
	if (rc) return rc;
	cudaLaunchConfig_t cfg = {};
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeCooperative;
	attr[0].val.cooperative = 1;
	cfg.blockDim = dim3(PHB_TILE);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	auto grid = [&](const void *kern) -> int {
		if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
		int perSM = 0;
		if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, kern, PHB_TILE, smem) != cudaSuccess || perSM < 1) perSM = 1;
		if (sv->ctas_per_sm > 0) perSM = std::min(perSM, sv->ctas_per_sm); // a tuned, smaller grid
		return std::max(1, std::min(dom->ntiles, perSM * numSMs()));
	};
	if (sv->kind == 0) {
		T *r = (T *)(w + L.off[0]), *q = (T *)(w + L.off[1]), *p0 = (T *)(w + L.off[2]), *p1 = (T *)(w + L.off[3]);
		T *xbest = sv->return_best ? (T *)(w + L.off[4]) : nullptr;
		auto launch = [&](auto kern) -> int {
			cfg.gridDim = dim3(grid((const void *)kern));
			PHB_CUDA(cudaLaunchKernelEx(&cfg, kern, dm, A, b, x, r, p0, p1, q, xbest, st, partial, ctrl, sv->tol, sv->return_best, maxit));
			return PHB_OK;
		};
		return stopStart ? launch(kCgPersistent<T, D, K, true>) : launch(kCgPersistent<T, D, K, false>);
	}
	T *r = (T *)(w + L.off[0]), *r0 = (T *)(w + L.off[1]), *p0 = (T *)(w + L.off[2]), *p1 = (T *)(w + L.off[3]);
	T *v0 = (T *)(w + L.off[4]), *v1 = (T *)(w + L.off[5]), *t = (T *)(w + L.off[6]);
	auto kern = kBicgPersistent<T, D, K>;
	cfg.gridDim = dim3(grid((const void *)kern));
	PHB_CUDA(cudaLaunchKernelEx(&cfg, kern, dm, A, b, x, r, r0, p0, p1, v0, v1, t, st, partial, ctrl, sv->tol, maxit));
	return PHB_OK;
}

#define PHB_PERSISTENT(T, D, K) template int launchPersistent<T, D, K>(const phb_domain *, const phb_solve *, cudaStream_t, bool, int);
PHB_PERSISTENT(double, 2, 1)
PHB_PERSISTENT(double, 2, 2)
PHB_PERSISTENT(double, 3, 1)
PHB_PERSISTENT(double, 3, 3)
PHB_PERSISTENT(float, 2, 1)
PHB_PERSISTENT(float, 2, 2)
PHB_PERSISTENT(float, 3, 1)
PHB_PERSISTENT(float, 3, 3)

} // namespace phb
