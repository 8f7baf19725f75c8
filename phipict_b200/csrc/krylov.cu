// Fused, batched Krylov solvers on stencil matrices: CG and BiCGStab for many systems at
// once (instances x right-hand sides), plus FP64 iterative refinement around FP32 inner
// solves.
//
// Algorithm and stop rule follow phiPICT's fused solvers (solvers/krylov/krylov.cu):
// classic CG in two fused phases per iteration (:428-568), van der Vorst BiCGStab with a
// half-step convergence check (:599-824), the criterion ||r||_2/sqrt(n) < tol per system,
// FP64 accumulation of every inner product and a deterministic fixed-order reduction in
// the last CTA to finish (:157-202). The B200 design differs where the hardware rewards it:
//   - the SpMV reads a stencil (2d+1 values per row, no column indices, neighbours by
//     index arithmetic), one CTA per 256-cell tile of one block, so every CTA belongs to
//     one instance and per-instance reductions are contiguous CTA ranges;
//   - the search direction update is folded into the SpMV of the next phase (p is evaluated
//     on the fly at the stencil points), which also removes BiCGStab's separate p kernel;
//   - the iteration loop is a conditional WHILE node of a CUDA graph whose condition the
//     last CTA sets, so a solve is one graph launch with no host round trip, and when the
//     caller is capturing a stream (a whole PISO step as one graph) the loop is spliced
//     into that capture instead.
#include <map>
#include <vector>
#include <mutex>
#include <string>
#include <functional>
#include <cuda_pipeline.h>
#include "phb_krylov.cuh"
#include "phb_faces.cuh"

int phbCheckAmg(const phb_amg *amg); // amg.cu

namespace phb {

// Block-reduce NV values, write this CTA's partials, and return whether this CTA is the
// last of the grid to finish (the ticket pattern of krylov.cu:157-182).
template <int NV>
__device__ __forceinline__ bool storePartials(double (&v)[NV], double *partial, unsigned int *counter) {
	__shared__ double sm[NV][NWARPS];
	__shared__ bool isLast;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
	for (int q = 0; q < NV; ++q) {
		const double s = warpSum(v[q]);
		if (lane == 0) sm[q][warp] = s;
	}
	__syncthreads();
	if (threadIdx.x < NV) {
		double s = 0;
#pragma unroll
		for (int w = 0; w < NWARPS; ++w) s += sm[threadIdx.x][w];
		partial[(size_t)blockIdx.x * NV + threadIdx.x] = s;
	}
	__syncthreads();
	if (threadIdx.x == 0) {
		__threadfence();
		const unsigned int ticket = atomicAdd(counter, 1u);
		isLast = ticket == gridDim.x - 1;
	}
	__syncthreads();
	return isLast;
}

// In the last CTA: the warps are split into groups of G (a power of two, as many as fit
// NWARPS/nsys); each group sums the CTA partials of one system's instance in a fixed order
// (lanes strided over the tiles, two accumulators in flight, then warp and group sums) and
// its leader calls fn(state, inst, sums, instSum). allDone is updated and the ticket
// counter reset for the next kernel. With INSTQ >= 0 the group also sums quantity INSTQ over
// all K systems of the instance (instSum), e.g. the whole right-hand side norm.
template <int K, int NQ, int INSTQ = -1, typename Fn>
__device__ __forceinline__ void finalizeSystems(const int32_t *insts, int ninst, const double *partial, SysState *st, Control *ctrl, Fn fn) {
	constexpr int NV = NQ + 1;
	__shared__ int running;
	__shared__ double gsm[NWARPS][NV];
	if (threadIdx.x == 0) running = 0;
	__threadfence();
	__syncthreads();
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	const int nsys = ninst * K;
	int G = NWARPS;
	while (G > 1 && G * nsys > NWARPS) G >>= 1;
	const int NG = NWARPS / G;
	const int group = warp / G, wg = warp - group * G;
	for (int base = 0; base < nsys; base += NG) {
		const int s = base + group;
		const bool act = s < nsys && st[s].done == RUNNING;
		double a0[NV], a1[NV];
#pragma unroll
		for (int q = 0; q < NV; ++q) { a0[q] = 0; a1[q] = 0; }
		if (act) {
			const int inst = s / K, k = s - inst * K;
			const int t0 = insts[inst * PHB_IREC + I_TILESTART], tc = insts[inst * PHB_IREC + I_TILECOUNT];
			const int stride = G * 32;
			auto load = [&](int t, double *a) {
				const double *pp = partial + (size_t)(t0 + t) * K * NQ;
#pragma unroll
				for (int q = 0; q < NQ; ++q) a[q] += __ldcg(pp + k * NQ + q);
				if (INSTQ >= 0) {
#pragma unroll
					for (int kk = 0; kk < K; ++kk) a[NQ] += __ldcg(pp + kk * NQ + (INSTQ < 0 ? 0 : INSTQ));
				}
			};
			int t = wg * 32 + lane;
			for (; t + stride < tc; t += 2 * stride) { load(t, a0); load(t + stride, a1); }
			if (t < tc) load(t, a0);
		}
#pragma unroll
		for (int q = 0; q < NV; ++q) {
			const double v = warpSum(a0[q] + a1[q]);
			if (lane == 0) gsm[warp][q] = v;
		}
		__syncthreads();
		if (act && wg == 0 && lane == 0) {
			double red[NV];
#pragma unroll
			for (int q = 0; q < NV; ++q) {
				double v = 0;
				for (int w = 0; w < G; ++w) v += gsm[group * G + w][q];
				red[q] = v;
			}
			fn(st[s], s / K, red, red[NQ]);
		}
		if (wg == 0 && lane == 0 && s < nsys && st[s].done == RUNNING) atomicAdd(&running, 1);
		__syncthreads();
	}
	if (threadIdx.x == 0) {
		ctrl->allDone = running == 0;
		ctrl->counter = 0;
	}
}

struct LoopCond {
	cudaGraphConditionalHandle handle;
	int active; // this kernel sets the loop condition
};
__device__ __forceinline__ void setLoop(const LoopCond lc, Control *ctrl) {
	if (!lc.active) return;
	const int loops = ++ctrl->loops; // one count per pass of the loop body
	const bool cont = !ctrl->allDone && loops < ctrl->maxLoops;
	cudaGraphSetConditional(lc.handle, cont ? 1u : 0u);
}

// kernels ------------------------------------------------------------------------------
// Initial state of every system and a fresh control block.
__global__ void kInit(SysState *st, int nsys, phb_tolerance tol, int fromInner, int maxit, Control *ctrl, int maxLoops) {
	for (int s = threadIdx.x; s < nsys; s += blockDim.x) {
		st[s] = initialState(tol, s, fromInner ? st[s].innerTol : 0.0, fromInner, maxit);
	}
	if (threadIdx.x == 0) {
		ctrl->counter = 0; ctrl->allDone = 0; ctrl->loops = 0; ctrl->maxLoops = maxLoops;
		ctrl->barCount = 0; ctrl->barErr = 0;
	}
}

// r = b - A x (and r0 = r for BiCGStab); rho = (r, r); the relative tolerance from (b, b);
// initial convergence check (krylov.cu:292-366). The reference CG stops on an exactly zero
// residual only, BiCGStab (and, here, every inner solve of the refinement: STOPSTART) on
// crit < tol.
template <typename T, int D, int K, bool BICG, bool STOPSTART>
__global__ void __launch_bounds__(PHB_TILE) kResidual(Dom<double, D> dom, const T *__restrict__ A, const T *__restrict__ b,
		const T *__restrict__ x, T *__restrict__ r, T *__restrict__ r0, SysState *st, double *partial, Control *ctrl, phb_tolerance tol,
		LoopCond arm) {
	__shared__ int32_t sB[PHB_BREC];
	int l0_, nc_;
	loadTile<double, D>(dom, sB, l0_, nc_);
	const int inst = sB[B_INST];
	bool act[K];
#pragma unroll
	for (int k = 0; k < K; ++k) act[k] = st[inst * K + k].done == RUNNING;
	double acc[2 * K];
#pragma unroll
	for (int k = 0; k < 2 * K; ++k) acc[k] = 0;
	tileResidual<T, D, K>(dom, sB, l0_, nc_, A, b, x, act, acc, [&](int, int64_t o, const Quad &q, const T (&rv)[4]) {
		st4(r + o, q.n, q.al, rv);
		if (BICG) st4(r0 + o, q.n, q.al, rv);
	});
	if (storePartials<2 * K>(acc, partial, &ctrl->counter)) {
		const bool relative = tol.mode == 1;
		finalizeSystems<K, 2, 1>(dom.insts, dom.ninst, partial, st, ctrl, [&](SysState &s, int in, const double *red, double bb) {
			const double ns = normScale(dom.insts, in);
			// the rhs scale of the whole instance: all K right-hand sides together
			if (relative) s.tol = resolveTol(tol, sqrt(bb / double(K)) * ns);
			const double crit = sqrt(red[0]) * ns;
			s.rho = red[0];
			s.restart = 1;
			s.crit = crit;
			if (!fin(crit)) { s.done = NONFINITE; s.usedIt = 0; }
			else if ((BICG || STOPSTART) ? crit < s.tol : crit == 0.0) { s.done = CONVERGED; s.usedIt = BICG ? -1 : 0; }
		});
		// arm the WHILE loop that follows: run its body only if a system is still running
		if (threadIdx.x == 0 && arm.active) cudaGraphSetConditional(arm.handle, ctrl->allDone ? 0u : 1u);
	}
}

// CG phase 1 (kCgDirection, krylov.cu:428-498): p' = r + beta p (p' = r on restart,
// evaluated at the stencil points), q = A p', (p', q); last CTA: alpha = rho / (p', q)
template <typename T, int D, int K>
__global__ void __launch_bounds__(PHB_TILE) kCgDirection(Dom<double, D> dom, const T *__restrict__ A, const T *__restrict__ r,
		const T *__restrict__ pIn, T *__restrict__ pOut, T *__restrict__ q, SysState *st, double *partial, Control *ctrl) {
	__shared__ int32_t sB[PHB_BREC];
	int l0_, nc_;
	loadTile<double, D>(dom, sB, l0_, nc_);
	const int inst = sB[B_INST];
	bool act[K], rs[K];
	T beta[K];
#pragma unroll
	for (int k = 0; k < K; ++k) {
		const SysState &s = st[inst * K + k];
		act[k] = s.done == RUNNING;
		rs[k] = s.restart;
		beta[k] = T(s.beta);
	}
	double acc[K];
#pragma unroll
	for (int k = 0; k < K; ++k) acc[k] = 0;
	tileCgDirection<T, D, K>(dom, sB, l0_, nc_, A, r, pIn, pOut, q, act, rs, beta, acc);
	if (storePartials<K>(acc, partial, &ctrl->counter)) {
		finalizeSystems<K, 1>(dom.insts, dom.ninst, partial, st, ctrl, [&](SysState &s, int, const double *red, double) {
			const double alpha = s.rho / red[0];
			s.restart = 0;
			if (!fin(alpha)) { s.done = NONFINITE; s.usedIt = s.it; }
			else s.alpha = alpha;
		});
	}
}

// CG phase 2 (kCgUpdate, krylov.cu:502-568): x += alpha p, r -= alpha q, (r, r); last CTA:
// convergence, beta = (r, r)_new / (r, r)_old, optional best-iterate tracking. Preconditioned
// (PC): beta comes from (r, z) after the next V-cycle instead (kPcgPrecond).
template <typename T, int D, int K, bool PC = false>
__global__ void __launch_bounds__(PHB_TILE) kCgUpdate(Dom<double, D> dom, T *__restrict__ r, const T *__restrict__ p,
		const T *__restrict__ q, T *__restrict__ x, T *__restrict__ xbest, SysState *st, double *partial, Control *ctrl,
		int returnBest, LoopCond lc) {
	__shared__ int32_t sB[PHB_BREC];
	int l0_, nc_;
	loadTile<double, D>(dom, sB, l0_, nc_);
	double acc[K];
#pragma unroll
	for (int k = 0; k < K; ++k) acc[k] = 0;
	tileCgUpdate<T, D, K>(dom, sB, l0_, nc_, r, p, q, x, xbest, st, acc);
	if (storePartials<K>(acc, partial, &ctrl->counter)) {
		finalizeSystems<K, 1>(dom.insts, dom.ninst, partial, st, ctrl, [&](SysState &s, int in, const double *red, double) {
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
			else if (!PC) {
				s.beta = red[0] / s.rho;
				s.rho = red[0];
				if (!fin(s.beta)) s.done = NONFINITE;
			}
		});
		if (threadIdx.x == 0) setLoop(lc, ctrl);
	}
}

// Last step of the V-cycle on level 0 (prolongation and post-smoothing, z written to the
// hierarchy's level-0 x) fused with (r, z); last CTA: rho and beta (pcgRho).
template <int D>
__global__ void __launch_bounds__(PHB_TILE) kPcgPrecond(Dom<double, D> dom, AmgView<D> mg, SysState *st, double *partial, Control *ctrl) {
	__shared__ int32_t sB[PHB_BREC];
	double acc[1] = {amgProlongQuad<D>(mg, 0, blockIdx.x, sB, mg.x[0])};
	if (storePartials<1>(acc, partial, &ctrl->counter)) {
		finalizeSystems<1, 1>(dom.insts, dom.ninst, partial, st, ctrl, [&](SysState &s, int, const double *red, double) { pcgRho(s, red[0]); });
	}
}

// BiCGStab phase 1 (kBicgP + kBicgV, krylov.cu:599-676): p = r + beta (p - omega v) (p = r
// on restart) evaluated at the stencil points, v = A p, (r0, v); last CTA: alpha
template <typename T, int D, int K>
__global__ void __launch_bounds__(PHB_TILE) kBicgV(Dom<double, D> dom, const T *__restrict__ A, const T *__restrict__ r,
		const T *__restrict__ pIn, const T *__restrict__ vIn, T *__restrict__ pOut, T *__restrict__ vOut, const T *__restrict__ r0,
		SysState *st, double *partial, Control *ctrl) {
	__shared__ int32_t sB[PHB_BREC];
	int l0_, nc_;
	loadTile<double, D>(dom, sB, l0_, nc_);
	const int inst = sB[B_INST];
	bool act[K], rs[K];
	T beta[K], omega[K];
#pragma unroll
	for (int k = 0; k < K; ++k) {
		const SysState &s = st[inst * K + k];
		act[k] = s.done == RUNNING;
		rs[k] = s.restart;
		beta[k] = T(s.beta);
		omega[k] = T(s.omega);
	}
	double acc[K];
#pragma unroll
	for (int k = 0; k < K; ++k) acc[k] = 0;
	tileBicgV<T, D, K>(dom, sB, l0_, nc_, A, r, pIn, vIn, pOut, vOut, r0, act, rs, beta, omega, acc);
	if (storePartials<K>(acc, partial, &ctrl->counter)) {
		finalizeSystems<K, 1>(dom.insts, dom.ninst, partial, st, ctrl, [&](SysState &s, int, const double *red, double) {
			const double alpha = s.rho / red[0];
			s.restart = 0;
			if (!fin(alpha)) { s.done = NONFINITE; s.usedIt = s.it; }
			else s.alpha = alpha;
		});
	}
}

// BiCGStab phase 2 (kBicgT, krylov.cu:680-750): s = r - alpha v on the fly, t = A s,
// (t,s), (t,t), (s,s); last CTA: omega, or convergence after the half step.
template <typename T, int D, int K>
__global__ void __launch_bounds__(PHB_TILE) kBicgT(Dom<double, D> dom, const T *__restrict__ A, const T *__restrict__ r,
		const T *__restrict__ v, T *__restrict__ t, SysState *st, double *partial, Control *ctrl) {
	__shared__ int32_t sB[PHB_BREC];
	int l0_, nc_;
	loadTile<double, D>(dom, sB, l0_, nc_);
	const int inst = sB[B_INST];
	bool act[K];
	T alpha[K];
#pragma unroll
	for (int k = 0; k < K; ++k) {
		const SysState &s = st[inst * K + k];
		act[k] = s.done == RUNNING;
		alpha[k] = T(s.alpha);
	}
	double acc[3 * K];
#pragma unroll
	for (int k = 0; k < 3 * K; ++k) acc[k] = 0;
	tileBicgT<T, D, K>(dom, sB, l0_, nc_, A, r, v, t, act, alpha, acc);
	if (storePartials<3 * K>(acc, partial, &ctrl->counter)) {
		finalizeSystems<K, 3>(dom.insts, dom.ninst, partial, st, ctrl, [&](SysState &s, int in, const double *red, double) {
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
	}
}

// BiCGStab phase 3 (kBicgUpdate, krylov.cu:754-824): x += alpha p + omega s, r = s - omega t,
// (r0, r), (r, r); last CTA: convergence and beta.
template <typename T, int D, int K>
__global__ void __launch_bounds__(PHB_TILE) kBicgUpdate(Dom<double, D> dom, T *__restrict__ r, const T *__restrict__ r0,
		const T *__restrict__ p, const T *__restrict__ v, const T *__restrict__ t, T *__restrict__ x, SysState *st,
		double *partial, Control *ctrl, LoopCond lc) {
	__shared__ int32_t sB[PHB_BREC];
	int l0_, nc_;
	loadTile<double, D>(dom, sB, l0_, nc_);
	double acc[2 * K];
#pragma unroll
	for (int k = 0; k < 2 * K; ++k) acc[k] = 0;
	tileBicgUpdate<T, D, K>(dom, sB, l0_, nc_, r, r0, p, v, t, x, st, acc);
	if (storePartials<2 * K>(acc, partial, &ctrl->counter)) {
		finalizeSystems<K, 2>(dom.insts, dom.ninst, partial, st, ctrl, [&](SysState &s, int in, const double *red, double) {
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
		if (threadIdx.x == 0) setLoop(lc, ctrl);
	}
}

// kRestoreBest (krylov.cu:370-375): systems that stopped without converging return their
// best iterate
template <typename T, int K>
__global__ void kRestoreBest(const int32_t *__restrict__ insts, int ninst, int64_t ncells, T *x, const T *xbest, const SysState *st) {
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < ncells * K; i += (int64_t)gridDim.x * blockDim.x) {
		// instance of vector entry i in the [inst][K][cells] layout
		int lo = 0, hi = ninst - 1;
		while (lo < hi) {
			const int mid = (lo + hi + 1) >> 1;
			if ((int64_t)K * insts[mid * PHB_IREC + I_CELLOFF] <= i) lo = mid; else hi = mid - 1;
		}
		const int64_t base = (int64_t)K * insts[lo * PHB_IREC + I_CELLOFF];
		const int k = int((i - base) / insts[lo * PHB_IREC + I_NCELLS]);
		const SysState &s = st[lo * K + k];
		if ((s.done == MAXIT || s.done == RISING) && s.bestIt >= 0 && s.best < s.crit) x[i] = xbest[i];
	}
}

// FP64 refinement residual: r64 = b - A64 x; r32 = float(r64), e32 = 0; last CTA: the
// outer tolerance (resolved from b on the first sweep), outer convergence per system, the
// inner tolerance innerRtol * ||r||/sqrt(n) (infinite for systems that are done) and the
// outer loop condition.
template <int D, int K>
__global__ void __launch_bounds__(PHB_TILE) kRefineResidual(Dom<double, D> dom, const double *__restrict__ A, const double *__restrict__ b,
		const double *__restrict__ x, float *__restrict__ r32, float *__restrict__ e32, SysState *st, double *partial, Control *ctrl,
		double innerRtol, int maxOuter, phb_tolerance tol, SysState *inner, LoopCond lc) {
	__shared__ int32_t sB[PHB_BREC];
	int l0_, nc_;
	loadTile<double, D>(dom, sB, l0_, nc_);
	double acc[2 * K];
#pragma unroll
	for (int k = 0; k < 2 * K; ++k) acc[k] = 0;
	bool act[K];
#pragma unroll
	for (int k = 0; k < K; ++k) act[k] = true;
	tileResidual<double, D, K>(dom, sB, l0_, nc_, A, b, x, act, acc, [&](int, int64_t o, const Quad &q, const double (&rv)[4]) {
		float r4[4], z4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
		for (int i = 0; i < 4; ++i) r4[i] = float(rv[i]);
		st4(r32 + o, q.n, q.al, r4);
		st4(e32 + o, q.n, q.al, z4);
	});
	if (storePartials<2 * K>(acc, partial, &ctrl->counter)) {
		const int nsys = dom.ninst * K;
		// every system is visited, also once done, so that the inner solve of a finished
		// system sees an infinite tolerance and stops at once
		__shared__ int running;
		__shared__ double gsm[NWARPS][2];
		if (threadIdx.x == 0) running = 0;
		__threadfence();
		__syncthreads();
		const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
		int G = NWARPS;
		while (G > 1 && G * nsys > NWARPS) G >>= 1;
		const int NG = NWARPS / G;
		const int group = warp / G, wg = warp - group * G;
		for (int base = 0; base < nsys; base += NG) {
			const int s = base + group;
			double a = 0, bb = 0;
			if (s < nsys) {
				const int inst = s / K, k = s - inst * K;
				const int t0 = dom.insts[inst * PHB_IREC + I_TILESTART], tc = dom.insts[inst * PHB_IREC + I_TILECOUNT];
				for (int t = wg * 32 + lane; t < tc; t += G * 32) {
					const double *pp = partial + (size_t)(t0 + t) * K * 2;
					a += __ldcg(pp + k * 2);
#pragma unroll
					for (int kk = 0; kk < K; ++kk) bb += __ldcg(pp + kk * 2 + 1);
				}
			}
			a = warpSum(a);
			bb = warpSum(bb);
			if (lane == 0) { gsm[warp][0] = a; gsm[warp][1] = bb; }
			__syncthreads();
			if (s < nsys && wg == 0 && lane == 0) {
				a = 0;
				bb = 0;
				for (int w = 0; w < G; ++w) { a += gsm[group * G + w][0]; bb += gsm[group * G + w][1]; }
				const int inst = s / K;
				SysState &o = st[s];
				const double ns = normScale(dom.insts, inst);
				if (o.it == 0 && o.done == RUNNING && tol.mode == 1) o.tol = resolveTol(tol, sqrt(bb / double(K)) * ns);
				const double crit = sqrt(a) * ns;
				o.crit = crit;
				if (o.launched) { o.innerIts += max(inner[s].usedIt, 0); o.launched = 0; }
				if (o.done == RUNNING) {
					if (!fin(crit)) o.done = NONFINITE;
					else if (crit < o.tol) o.done = CONVERGED;
					else if (o.it >= maxOuter) o.done = MAXIT;
					else { ++o.it; o.launched = 1; }
				}
				o.usedIt = o.it;
				inner[s].innerTol = o.done == RUNNING ? fmax(innerRtol * crit, 0.25 * o.tol) : INFINITY;
				if (o.done == RUNNING) atomicAdd(&running, 1);
			}
			__syncthreads();
		}
		if (threadIdx.x == 0) {
			ctrl->allDone = running == 0;
			ctrl->counter = 0;
			setLoop(lc, ctrl);
		}
	}
}

template <int K>
__global__ void kRefineUpdate(int64_t n, double *__restrict__ x, const float *__restrict__ e) {
	for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) x[i] += double(e[i]);
}

__global__ void kInitOuter(SysState *st, int nsys, phb_tolerance tol, Control *ctrl, int maxLoops) {
	for (int s = threadIdx.x; s < nsys; s += blockDim.x) {
		SysState z;
		memset(&z, 0, sizeof(z));
		z.tol = tol.mode == 0 ? tol.atol : tol.mode == 2 ? tol.values[s] : NAN;
		st[s] = z;
	}
	if (threadIdx.x == 0) {
		ctrl->counter = 0; ctrl->allDone = 0; ctrl->loops = 0; ctrl->maxLoops = maxLoops;
	}
}

int launchInit(SysState *st, int nsys, const phb_tolerance &tol, int fromInner, int maxit, Control *ctrl, cudaStream_t s) {
	kInit<<<1, 256, 0, s>>>(st, nsys, tol, fromInner, maxit, ctrl, maxit / 2 + 2);
	return checkLaunch("kInit");
}

// The bounded wait under test: every CTA but `absent` takes `rounds` grid barriers with spin
// limit `spinLimit`; the absent CTA leaves at once, so the others' waits run out, set barErr
// and end the kernel. rounds_done[0] counts the barriers CTA 0 passed.
__global__ void kBarrierProbe(Control *ctrl, int rounds, int absent, unsigned int spinLimit, int *roundsDone) {
	if ((int)blockIdx.x == absent) return;
	int done = 0;
	for (int i = 0; i < rounds; ++i) {
		if (!gridBarrier(ctrl, spinLimit)) break;
		++done;
	}
	if (blockIdx.x == 0 && threadIdx.x == 0) *roundsDone = done;
}

// host side --------------------------------------------------------------------------------
// capture helpers ----------------------------------------------------------------------------
struct Streams { cudaStream_t s[3] = {nullptr, nullptr, nullptr}; int device = -1; };
static thread_local Streams tlStreams;
static int getStreams(Streams *&out) {
	int dev;
	PHB_CUDA(cudaGetDevice(&dev));
	if (tlStreams.device != dev) {
		for (auto &s : tlStreams.s) {
			if (s) cudaStreamDestroy(s);
			s = nullptr;
		}
		for (auto &s : tlStreams.s) PHB_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
		tlStreams.device = dev;
	}
	out = &tlStreams;
	return PHB_OK;
}

// Create the condition handle of a WHILE loop on the graph `cap` is capturing. The kernel
// launched just before the loop sets it (armCondition), so that a loop nested in another
// conditional body is re-armed on every pass of the outer body: a handle's default value is
// only applied when the graph that owns it is launched.
static int createCondition(cudaStream_t cap, cudaGraphConditionalHandle *handle) {
	cudaStreamCaptureStatus status;
	cudaGraph_t graph;
	PHB_CUDA(cudaStreamGetCaptureInfo(cap, &status, nullptr, &graph, nullptr, nullptr));
	if (status != cudaStreamCaptureStatusActive) return setError(PHB_ERR_STATE, "createCondition: stream is not capturing");
	PHB_CUDA(cudaGraphConditionalHandleCreate(handle, graph, 1, cudaGraphCondAssignDefault));
	return PHB_OK;
}

// Add a conditional WHILE node on `handle` to the graph `cap` is capturing and capture
// `body` into it on `bodyStream`; the body's last kernel sets the condition.
static int addWhile(cudaStream_t cap, cudaStream_t bodyStream, cudaGraphConditionalHandle handle,
		const std::function<int(cudaStream_t, LoopCond)> &body) {
	cudaStreamCaptureStatus status;
	cudaGraph_t graph;
	const cudaGraphNode_t *deps = nullptr;
	size_t ndeps = 0;
	PHB_CUDA(cudaStreamGetCaptureInfo(cap, &status, nullptr, &graph, &deps, &ndeps));
	if (status != cudaStreamCaptureStatusActive) return setError(PHB_ERR_STATE, "addWhile: stream is not capturing");
	cudaGraphNodeParams params = {};
	params.type = cudaGraphNodeTypeConditional;
	params.conditional.handle = handle;
	params.conditional.type = cudaGraphCondTypeWhile;
	params.conditional.size = 1;
	cudaGraphNode_t node;
	PHB_CUDA(cudaGraphAddNode(&node, graph, deps, ndeps, &params));
	PHB_CUDA(cudaStreamUpdateCaptureDependencies(cap, &node, 1, cudaStreamSetCaptureDependencies));
	cudaGraph_t bodyGraph = params.conditional.phGraph_out[0];
	PHB_CUDA(cudaStreamBeginCaptureToGraph(bodyStream, bodyGraph, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
	const int st = body(bodyStream, LoopCond{handle, 1});
	cudaGraph_t ended;
	const cudaError_t e = cudaStreamEndCapture(bodyStream, &ended);
	if (st != PHB_OK) return st;
	PHB_CUDA(e);
	return PHB_OK;
}

struct CachedGraph { cudaGraphExec_t exec; };
static std::mutex gMutex;
static std::map<std::string, CachedGraph> gGraphs;

static int releaseGraphsLocked() {
	for (auto &kv : gGraphs) cudaGraphExecDestroy(kv.second.exec);
	gGraphs.clear();
	return PHB_OK;
}

// Run `emit` (which records work on a capturing stream) either spliced into the caller's
// ongoing capture, or as a cached graph launched on `stream`.
static int runGraph(cudaStream_t stream, const std::string &key, const std::function<int(cudaStream_t, Streams &)> &emit) {
	Streams *ss;
	int rc = getStreams(ss);
	if (rc) return rc;
	cudaStreamCaptureStatus status;
	PHB_CUDA(cudaStreamIsCapturing(stream, &status));
	if (status == cudaStreamCaptureStatusActive) return emit(stream, *ss);
	std::lock_guard<std::mutex> lock(gMutex);
	auto it = gGraphs.find(key);
	if (it == gGraphs.end()) {
		if (gGraphs.size() >= 64) releaseGraphsLocked();
		PHB_CUDA(cudaStreamBeginCapture(ss->s[0], cudaStreamCaptureModeThreadLocal));
		rc = emit(ss->s[0], *ss);
		cudaGraph_t graph = nullptr;
		const cudaError_t e = cudaStreamEndCapture(ss->s[0], &graph);
		if (rc) { if (graph) cudaGraphDestroy(graph); return rc; }
		PHB_CUDA(e);
		CachedGraph cg;
		const cudaError_t ei = cudaGraphInstantiate(&cg.exec, graph, 0);
		cudaGraphDestroy(graph);
		PHB_CUDA(ei);
		it = gGraphs.emplace(key, cg).first;
	}
	PHB_CUDA(cudaGraphLaunch(it->second.exec, stream));
	return PHB_OK;
}

template <typename A, typename B>
static std::string makeKey(const char *tag, const A &a, const B &b) {
	std::string k(tag);
	k.append(reinterpret_cast<const char *>(&a), sizeof(A));
	k.append(reinterpret_cast<const char *>(&b), sizeof(B));
	return k;
}

static int gridFor(int64_t n) { return (int)std::min<int64_t>((n + 255) / 256, 148 * 16); }

// the Krylov loop for one solve, recorded on `s`
template <typename T, int D, int K>
static int emitSolve(const phb_domain *dom, const phb_solve *sv, cudaStream_t s, Streams &ss, int useGraph, bool stopStart, int fromInner = 0) {
	if (sv->use_graph >= 2) return launchPersistent<T, D, K>(dom, sv, s, stopStart, fromInner);
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
	const int tiles = dom->ntiles;
	const int maxit = std::max(1, sv->maxit);
	if (sv->kind == 0) {
		T *r = (T *)(w + L.off[0]), *q = (T *)(w + L.off[1]), *p0 = (T *)(w + L.off[2]), *p1 = (T *)(w + L.off[3]);
		T *xbest = sv->return_best ? (T *)(w + L.off[4]) : nullptr;
		const int maxLoops = maxit / 2 + 2;
		LoopCond arm{0, 0};
		if (useGraph) {
			const int rc0 = createCondition(s, &arm.handle);
			if (rc0) return rc0;
			arm.active = 1;
		}
		kInit<<<1, 256, 0, s>>>(st, nsys, sv->tol, fromInner, maxit, ctrl, maxLoops);
		if (stopStart) kResidual<T, D, K, false, true><<<tiles, PHB_TILE, 0, s>>>(dm, A, b, x, r, nullptr, st, partial, ctrl, sv->tol, arm);
		else kResidual<T, D, K, false, false><<<tiles, PHB_TILE, 0, s>>>(dm, A, b, x, r, nullptr, st, partial, ctrl, sv->tol, arm);
		int rc = checkLaunch("kResidual");
		if (rc) return rc;
		// preconditioned (float, one right-hand side): V-cycle on r down to level 1, then level
		// 0's prolongation with (r, z) and beta, and the direction taken from z
		bool pc = false;
		AmgView<D> mg = {};
		const T *dsrc = r;
		if constexpr (std::is_same<T, float>::value && K == 1) {
			if (sv->amg) {
				pc = true;
				mg = makeAmgView<D>(*sv->amg, (const float *)r, sv->amg->levels[0].x);
				dsrc = (const T *)mg.x[0];
			}
		}
		auto body = [&](cudaStream_t bs, LoopCond lc) -> int {
			for (int half = 0; half < 2; ++half) {
				T *pIn = half == 0 ? p0 : p1, *pOut = half == 0 ? p1 : p0;
				LoopCond l2 = lc;
				l2.active = half == 1 ? lc.active : 0;
				if (pc) {
					PHB_CUDA(launchAmgCycle<D>(mg, bs, 1));
					kPcgPrecond<D><<<tiles, PHB_TILE, 0, bs>>>(dm, mg, st, partial, ctrl);
					kCgDirection<T, D, K><<<tiles, PHB_TILE, 0, bs>>>(dm, A, dsrc, pIn, pOut, q, st, partial, ctrl);
					kCgUpdate<T, D, K, true><<<tiles, PHB_TILE, 0, bs>>>(dm, r, pOut, q, x, xbest, st, partial, ctrl, sv->return_best, l2);
				} else {
					kCgDirection<T, D, K><<<tiles, PHB_TILE, 0, bs>>>(dm, A, r, pIn, pOut, q, st, partial, ctrl);
					kCgUpdate<T, D, K><<<tiles, PHB_TILE, 0, bs>>>(dm, r, pOut, q, x, xbest, st, partial, ctrl, sv->return_best, l2);
				}
			}
			return checkLaunch("CG body");
		};
		if (useGraph) { rc = addWhile(s, ss.s[useGraph == 2 ? 2 : 1], arm.handle, body); if (rc) return rc; }
		else {
			// host loop (no graph): poll allDone every check_every iterations
			int *hflag = nullptr;
			PHB_CUDA(cudaMallocHost(&hflag, sizeof(int)));
			const int chk = std::max(1, sv->check_every);
			for (int loops = 0; loops < maxLoops; loops += chk) {
				for (int i = 0; i < chk; ++i) { rc = body(s, LoopCond{0, 0}); if (rc) break; }
				if (rc) break;
				cudaMemcpyAsync(hflag, &ctrl->allDone, sizeof(int), cudaMemcpyDeviceToHost, s);
				cudaStreamSynchronize(s);
				if (*hflag) break;
			}
			cudaFreeHost(hflag);
			if (rc) return rc;
		}
		if (xbest) kRestoreBest<T, K><<<gridFor(dom->ncells * K), 256, 0, s>>>(dom->insts, dom->ninst, dom->ncells, x, xbest, st);
		return checkLaunch("CG epilogue");
	}
	T *r = (T *)(w + L.off[0]), *r0 = (T *)(w + L.off[1]), *p0 = (T *)(w + L.off[2]), *p1 = (T *)(w + L.off[3]);
	T *v0 = (T *)(w + L.off[4]), *v1 = (T *)(w + L.off[5]), *t = (T *)(w + L.off[6]);
	const int maxLoops = maxit / 2 + 2;
	LoopCond arm{0, 0};
	if (useGraph) {
		const int rc0 = createCondition(s, &arm.handle);
		if (rc0) return rc0;
		arm.active = 1;
	}
	kInit<<<1, 256, 0, s>>>(st, nsys, sv->tol, fromInner, maxit, ctrl, maxLoops);
	kResidual<T, D, K, true, true><<<tiles, PHB_TILE, 0, s>>>(dm, A, b, x, r, r0, st, partial, ctrl, sv->tol, arm);
	int rc = checkLaunch("kResidual");
	if (rc) return rc;
	auto body = [&](cudaStream_t bs, LoopCond lc) -> int {
		for (int half = 0; half < 2; ++half) {
			T *pIn = half == 0 ? p0 : p1, *pOut = half == 0 ? p1 : p0;
			T *vIn = half == 0 ? v0 : v1, *vOut = half == 0 ? v1 : v0;
			kBicgV<T, D, K><<<tiles, PHB_TILE, 0, bs>>>(dm, A, r, pIn, vIn, pOut, vOut, r0, st, partial, ctrl);
			kBicgT<T, D, K><<<tiles, PHB_TILE, 0, bs>>>(dm, A, r, vOut, t, st, partial, ctrl);
			LoopCond l2 = lc;
			l2.active = half == 1 ? lc.active : 0;
			kBicgUpdate<T, D, K><<<tiles, PHB_TILE, 0, bs>>>(dm, r, r0, pOut, vOut, t, x, st, partial, ctrl, l2);
		}
		return checkLaunch("BiCGStab body");
	};
	if (useGraph) return addWhile(s, ss.s[useGraph == 2 ? 2 : 1], arm.handle, body);
	int *hflag = nullptr;
	PHB_CUDA(cudaMallocHost(&hflag, sizeof(int)));
	const int chk = std::max(1, sv->check_every);
	for (int loops = 0; loops < maxLoops; loops += chk) {
		for (int i = 0; i < chk; ++i) { rc = body(s, LoopCond{0, 0}); if (rc) break; }
		if (rc) break;
		cudaMemcpyAsync(hflag, &ctrl->allDone, sizeof(int), cudaMemcpyDeviceToHost, s);
		cudaStreamSynchronize(s);
		if (*hflag) break;
	}
	cudaFreeHost(hflag);
	return rc;
}

// Y[v] = A X[v], v < nvec, for float64 vectors of one component (stride values apart): the
// products of the basis of a projected initial guess with the system matrix. The stencil row and
// neighbours of a cell stay in registers while the vectors go by, so the matrix is read once (per
// CTA that shares in the vectors) and not once per vector. What bounds it: a chain of one round trip to
// memory per vector and cell of a thread. Two cells of a thread at a time spilled; one cell, quarter tiles
// and the vectors of small domains shared out over CTAs: 12 rows of 442,368 cells 70 -> 51 us, of 2048 cells
// 43 -> 8, of 2.1 M cells 289 -> 221. The centre and face terms are summed in the order of the solvers' own products.
template <int D, int PARTS>
__global__ void __launch_bounds__(PHB_TILE, 4) kStencilApply(Dom<double, D> dom, int run, const double *__restrict__ A,
		const double *__restrict__ X, double *__restrict__ Y, int nvec, int64_t stride) {
	__shared__ int32_t sB[PHB_BREC];
	__shared__ FaceMap sF[6];
	const int64_t N = dom.ncells;
	const int v0 = int((int64_t)blockIdx.y * nvec / gridDim.y), v1 = int(((int64_t)blockIdx.y + 1) * nvec / gridDim.y);
	forTiles<PARTS, double, D>(dom, run, sB, sF, [&](int l0, int nc, int j0, auto) {
		for (int j = j0; j < j0 + CPT / PARTS; ++j) {
			Cell c;
			if (!cellAt<D>(sB, l0, nc, j, c)) return;
			const Faces<D> n = cellFaces<D>(sB, sF, c);
			double a[2 * D + 1];
#pragma unroll
			for (int k = 0; k < 2 * D + 1; ++k) a[k] = A[k * N + c.g];
#pragma unroll 1
			for (int v = v0; v < v1; ++v) {
				const double *x = X + v * stride;
				double xn[2 * D];
				const double xc = x[c.g];
#pragma unroll
				for (int f = 0; f < 2 * D; ++f) xn[f] = x[n.o[f]];
				double y = a[0] * xc;
#pragma unroll
				for (int f = 0; f < 2 * D; ++f) y = fma(a[f + 1], (n.fixed >> f) & 1 ? 0.0 : xn[f], y);
				Y[v * stride + c.g] = y;
			}
		}
	});
}

// The coefficients of a Galerkin projection, one CTA: G (m x m, row-major, the Gram matrix
// D A D^T of the basis rows) alpha = c. Jacobi-scaled (s_i = |G_ii|^-1/2), the diagonal
// raised by reg relative to the scaled unit diagonal, Gaussian elimination with partial
// pivoting; a basis row whose pivot falls below 1e-14 of the largest gets coefficient 0, and
// so does every row when a value is not finite (the guess is then the zero vector's
// projection: alpha = 0).
constexpr int PROJ_MAX = 16;
__global__ void kProjectionSolve(const double *__restrict__ G, const double *__restrict__ c, int m, double reg,
		double *__restrict__ alpha) {
	__shared__ double M[PROJ_MAX][PROJ_MAX + 1];
	__shared__ double sc[PROJ_MAX];
	const int t = threadIdx.x;
	if (t < m) {
		const double d = fabs(G[t * m + t]);
		sc[t] = d > 0 && isfinite(d) ? rsqrt(d) : 0.0;
	}
	__syncthreads();
	for (int e = t; e < m * (m + 1); e += blockDim.x) {
		const int i = e / (m + 1), j = e - i * (m + 1);
		double v = j < m ? G[i * m + j] * sc[i] * sc[j] : c[i] * sc[i];
		if (j == i) v += (G[i * m + i] < 0 ? -reg : reg);
		M[i][j] = v;
	}
	__syncthreads();
	// one warp, lane i on row i (one division per pivot; lane j on column j needed all multipliers in every
	// lane: 24 us at 12 rows, now 12), the pivot search the same in every lane
	if (t >= 32) return;
	bool ok = true;
	double big = 0;
	for (int i = 0; i < m; ++i) big = fmax(big, fabs(M[i][i]));
	unsigned int skip = 0;
	for (int k = 0; k < m; ++k) {
		int p = k;
		double best = fabs(M[k][k]);
		for (int i = k + 1; i < m; ++i) {
			const double v = fabs(M[i][k]);
			if (v > best) { best = v; p = i; }
		}
		__syncwarp();
		if (p != k && t <= m) { const double tmp = M[k][t]; M[k][t] = M[p][t]; M[p][t] = tmp; }
		__syncwarp();
		const double pivot = M[k][k];
		if (!(fabs(pivot) > 1e-14 * big)) { skip |= 1u << k; continue; }
		if (t > k && t < m) {
			const double f = M[t][k] / pivot;
			for (int j = k; j <= m; ++j) M[t][j] -= f * M[k][j];
		}
		__syncwarp();
	}
	// back substitution, lane i on row i: its right-hand side loses the solved unknowns
	double v = t < m ? M[t][m] : 0.0, x = 0;
	for (int k = m - 1; k >= 0; --k) {
		double xk = (skip >> k) & 1 ? 0.0 : __shfl_sync(0xffffffffu, v, k) / M[k][k];
		if (!isfinite(xk)) ok = false;
		if (t == k) x = xk;
		if (t < k) v -= M[t][k] * xk;
	}
	if (t < m) alpha[t] = ok ? x * sc[t] : 0.0;
}

// G[i][j] = sum_c V[i][c] Y[j][c] and g[i] = sum_c V[i][c] b[c] (i, j < m): each CTA stages
// chunks of GRAM_CHUNK cells of the m rows of V, the m rows of Y and b (as row m of Y) in shared
// memory (rows padded by one value against bank conflicts). A thread takes GRAM_R x GRAM_R pairs of
// rows over every slices-th cell, so a value read from shared memory serves GRAM_R products; one
// thread per pair was bound by its two shared loads per product, with half the threads idle (12 rows
// of 442,368 values: 76 us, now 45 us). The CTA's sums are added atomically into G and g, which the
// caller zeroes.
constexpr int GRAM_CHUNK = 128, GRAM_R = 3;
constexpr int GRAM_ROWS = (PROJ_MAX + 1 + GRAM_R - 1) / GRAM_R * GRAM_R;
__global__ void __launch_bounds__(256) kProjectionGram(const double *__restrict__ V, const double *__restrict__ Y,
		const double *__restrict__ b, int m, int64_t n, int64_t stride, double *__restrict__ G, double *__restrict__ g) {
	__shared__ double sv[GRAM_ROWS][GRAM_CHUNK + 1];
	__shared__ double sy[GRAM_ROWS][GRAM_CHUNK + 1];
	static_assert(256 * GRAM_R * GRAM_R <= GRAM_ROWS * (GRAM_CHUNK + 1), "the sums fit where V was");
	const int ti = (m + GRAM_R - 1) / GRAM_R, tj = (m + GRAM_R) / GRAM_R;
	const int tasks = ti * tj, slices = 256 / tasks;
	const int slice = int(threadIdx.x) / tasks, task = int(threadIdx.x) - slice * tasks;
	const int i0 = task / tj * GRAM_R, j0 = (task % tj) * GRAM_R;
	const int rows = ti * GRAM_R, cols = tj * GRAM_R; // rows of zeros past m and m + 1
	double acc[GRAM_R][GRAM_R];
#pragma unroll
	for (int i = 0; i < GRAM_R; ++i)
#pragma unroll
		for (int j = 0; j < GRAM_R; ++j) acc[i][j] = 0;
	for (int64_t base = (int64_t)blockIdx.x * GRAM_CHUNK; base < n; base += (int64_t)gridDim.x * GRAM_CHUNK) {
		const int64_t rest = n - base;
		const int len = rest < GRAM_CHUNK ? (int)rest : GRAM_CHUNK;
		// row by row, half a CTA each; zeros past the rows and the last cell
		for (int r = int(threadIdx.x) / GRAM_CHUNK; r < rows + cols; r += 256 / GRAM_CHUNK) {
			const int kk = int(threadIdx.x) & (GRAM_CHUNK - 1), c = r - rows;
			const bool inV = c < 0, in = kk < len && (inV ? r < m : c <= m);
			const double *src = inV ? V + (r < m ? r : 0) * stride : (c < m ? Y + c * stride : b);
			__pipeline_memcpy_async((inV ? sv[r] : sy[c]) + kk, src + (in ? base + kk : base), 8, in ? 0 : 8);
		}
		__pipeline_commit();
		__pipeline_wait_prior(0);
		__syncthreads();
		if (slice < slices)
			for (int k = slice; k < GRAM_CHUNK; k += slices) {
				double vi[GRAM_R], yj[GRAM_R];
#pragma unroll
				for (int i = 0; i < GRAM_R; ++i) {
					vi[i] = sv[i0 + i][k];
					yj[i] = sy[j0 + i][k];
				}
#pragma unroll
				for (int i = 0; i < GRAM_R; ++i)
#pragma unroll
					for (int j = 0; j < GRAM_R; ++j) acc[i][j] = fma(vi[i], yj[j], acc[i][j]);
			}
		__syncthreads();
	}
	double *red = &sv[0][0]; // [thread][GRAM_R * GRAM_R]
#pragma unroll
	for (int i = 0; i < GRAM_R; ++i)
#pragma unroll
		for (int j = 0; j < GRAM_R; ++j) red[int(threadIdx.x) * GRAM_R * GRAM_R + i * GRAM_R + j] = acc[i][j];
	__syncthreads();
	for (int p = threadIdx.x; p < m * m + m; p += 256) {
		const int i = p < m * m ? p / m : p - m * m, j = p < m * m ? p - i * m : m;
		const int t = i / GRAM_R * tj + j / GRAM_R, q = i % GRAM_R * GRAM_R + j % GRAM_R;
		double a = 0;
		for (int s = 0; s < slices; ++s) a += red[(t + s * tasks) * GRAM_R * GRAM_R + q];
		atomicAdd(j < m ? G + p : g + i, a);
	}
}

#define PHB_SOLVE_DISPATCH(DIMS, VEC, K, ...)                                                   \
	do {                                                                                        \
		if ((DIMS) == 2 && (VEC) == PHB_F64 && (K) == 1) { using T = double; constexpr int D = 2, KK = 1; __VA_ARGS__; } \
		else if ((DIMS) == 2 && (VEC) == PHB_F64 && (K) == 2) { using T = double; constexpr int D = 2, KK = 2; __VA_ARGS__; } \
		else if ((DIMS) == 3 && (VEC) == PHB_F64 && (K) == 1) { using T = double; constexpr int D = 3, KK = 1; __VA_ARGS__; } \
		else if ((DIMS) == 3 && (VEC) == PHB_F64 && (K) == 3) { using T = double; constexpr int D = 3, KK = 3; __VA_ARGS__; } \
		else if ((DIMS) == 2 && (VEC) == PHB_F32 && (K) == 1) { using T = float; constexpr int D = 2, KK = 1; __VA_ARGS__; } \
		else if ((DIMS) == 2 && (VEC) == PHB_F32 && (K) == 2) { using T = float; constexpr int D = 2, KK = 2; __VA_ARGS__; } \
		else if ((DIMS) == 3 && (VEC) == PHB_F32 && (K) == 1) { using T = float; constexpr int D = 3, KK = 1; __VA_ARGS__; } \
		else if ((DIMS) == 3 && (VEC) == PHB_F32 && (K) == 3) { using T = float; constexpr int D = 3, KK = 3; __VA_ARGS__; } \
		else return setError(PHB_ERR_ARG, "unsupported dims/dtype/nrhs combination");            \
	} while (0)

} // namespace phb

using namespace phb;

extern "C" int64_t phb_solve_work_bytes(const phb_domain *dom, int kind, int vec_dtype, int nrhs) {
	if (!dom) return -1;
	return (int64_t)solveLayout(dom, kind, vec_dtype == PHB_F64 ? 8 : 4, nrhs).total;
}
extern "C" int64_t phb_solve_state_bytes(const phb_domain *dom, int nrhs) {
	if (!dom) return -1;
	return (int64_t)stateLayout(dom, nrhs).total;
}

// BiCGStab of one float32 or of two right-hand sides on instances of at least 2^23 cells runs as per-phase
// kernels in a CUDA graph even in the persistent mode. On rows of four cells the persistent kernel is the faster one
// at every size (4096^2 float32, two right-hand sides 666 against 808 us an iteration, one 399 against 492), but on
// odd rows, which it takes a cell at a time, it loses there (4001 x 4003: 1299 against 979 and 717 against
// 571; 254 x 253 x 250, one: 964 against 730), and the row length is not known to the host. With three
// right-hand sides and with one in float64 it is as fast or faster on all of them (256^3 float32 three 1095 against
// 1312, 251 x 253 x 249 1861 against 2073, 4001 x 4003 float64 one 886 against 893).
static bool bicgPrefersGraph(const phb_domain *dom, int kind, bool f32, int nrhs) {
	return kind == 1 && (nrhs == 2 || (nrhs == 1 && f32)) && dom->ninst > 0 && dom->ncells / dom->ninst >= (int64_t(1) << 23);
}

extern "C" int phb_solve_run(const phb_domain *dom, const phb_solve *s_in, phb_stream stream) {
	phb_solve sAdj;
	const phb_solve *s = s_in;
	if (s_in && dom && s_in->use_graph == 2 && bicgPrefersGraph(dom, s_in->kind, s_in->vec_dtype == PHB_F32, s_in->nrhs)) {
		sAdj = *s_in;
		sAdj.use_graph = 1;
		s = &sAdj;
	}
	if (!dom || !s || !s->A || !s->b || !s->x || !s->work || !s->state || (s->tol.mode == 2 && !s->tol.values)) return setError(PHB_ERR_ARG, "phb_solve_run: null argument");
	if (s->vec_dtype != s->mat_dtype) return setError(PHB_ERR_ARG, "phb_solve_run: matrix and vector dtype must match");
	if (s->kind != 0 && s->kind != 1) return setError(PHB_ERR_ARG, "phb_solve_run: kind must be 0 (CG) or 1 (BiCGStab)");
	if (s->amg) {
		if (s->kind != 0 || s->vec_dtype != PHB_F32 || s->nrhs != 1) return setError(PHB_ERR_ARG, "phb_solve_run: the AMG preconditioner takes float32 CG with one right-hand side");
		const int rc = phbCheckAmg(s->amg);
		if (rc) return rc;
		if (s->amg->levels[0].dom.ncells != dom->ncells || !s->amg->levels[0].x) return setError(PHB_ERR_ARG, "phb_solve_run: hierarchy does not match the domain");
	}
	if (dom->ntiles == 0) return PHB_OK;
	cudaStream_t st = (cudaStream_t)stream;
	std::string key = makeKey("solve", *dom, *s);
	if (s->amg) key.append(reinterpret_cast<const char *>(s->amg), sizeof(phb_amg));
	PHB_SOLVE_DISPATCH(dom->dims, s->vec_dtype, s->nrhs, {
		if (s->use_graph != 1) {
			Streams *ss; int rc = getStreams(ss); if (rc) return rc;
			return emitSolve<T, D, KK>(dom, s, st, *ss, 0, false);
		}
		return runGraph(st, key, [&](cudaStream_t cs, Streams &ss) { return emitSolve<T, D, KK>(dom, s, cs, ss, 1, false); });
	});
	return PHB_OK;
}

extern "C" int phb_solve_results(const phb_domain *dom, const phb_solve *s, phb_solve_result *out, phb_stream stream) {
	if (!dom || !s || !out || !s->state) return setError(PHB_ERR_ARG, "phb_solve_results: null argument");
	const int nsys = dom->ninst * s->nrhs;
	std::vector<SysState> h(nsys);
	const StateLayout SL = stateLayout(dom, s->nrhs);
	Control c{};
	PHB_CUDA(cudaMemcpyAsync(h.data(), (char *)s->state + SL.st, nsys * sizeof(SysState), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
	PHB_CUDA(cudaMemcpyAsync(&c, (char *)s->state + SL.ctrl, sizeof(Control), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
	PHB_CUDA(cudaStreamSynchronize((cudaStream_t)stream));
	for (int i = 0; i < nsys; ++i) {
		const SysState &x = h[i];
		phb_solve_result &o = out[i];
		o.final_residual = x.crit;
		o.used_iterations = x.usedIt;
		o.converged = x.done == CONVERGED;
		o.finite = std::isfinite(x.crit);
		o.status = x.done;
		o.inner_iterations = 0;
		o.pad = 0;
		if (c.barErr) { // a persistent solve left early at a grid-barrier wait that ran out
			o.converged = 0;
			o.finite = 0;
			o.status = NONFINITE;
			o.final_residual = NAN;
			continue;
		}
		if (s->return_best && (x.done == MAXIT || x.done == RISING) && x.bestIt >= 0 && x.best < x.crit) {
			o.used_iterations = x.bestIt;
			o.final_residual = x.best;
		}
	}
	return PHB_OK;
}

extern "C" int phb_stencil_apply(const phb_domain *dom, const double *A, const double *X, double *Y, int32_t nvec,
		int64_t stride, phb_stream stream) {
	if (!dom || !A || !X || !Y) return setError(PHB_ERR_ARG, "phb_stencil_apply: null argument");
	// the layout that the header asks of callers, wide enough for vector loads of rows of four (the kernel takes
	// a cell at a time)
	if (nvec < 1 || stride < dom->ncells || (stride & 3) != 0)
		return setError(PHB_ERR_ARG, "phb_stencil_apply: nvec < 1, stride < ncells or stride not a multiple of 4");
	if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Y)) & 31)
		return setError(PHB_ERR_ARG, "phb_stencil_apply: A, X and Y must be 32-byte aligned");
	if (dom->dims != 2 && dom->dims != 3) return setError(PHB_ERR_ARG, "phb_stencil_apply: dims");
	if (dom->ntiles == 0) return PHB_OK;
	cudaStream_t s = (cudaStream_t)stream;
	auto launch = [&](auto dims) {
		constexpr int D = decltype(dims)::value;
		// longer runs of quarter tiles with more vectors (442,368 cells, whole tiles and runs of three: one vector
		// 10.4 and 12.4 us, 12 vectors 61 and 51); never strided (the least use is 1 percent)
		const TileShare ts = tileShare<kStencilApply<D, 1>, kStencilApply<D, CPT>>(dom, nvec >= 4 ? 1 : 0);
		// the vectors are shared out over CTAs too where the tiles leave room for it
		const dim3 grid(ts.ctas, std::max(1, std::min(nvec, residentCtas<kStencilApply<D, CPT>>() / ts.ctas)));
		auto kern = ts.quarters ? kStencilApply<D, CPT> : kStencilApply<D, 1>;
		kern<<<grid, PHB_TILE, 0, s>>>(Dom<double, D>(*dom), ts.run, A, X, Y, nvec, stride);
	};
	if (dom->dims == 2) launch(std::integral_constant<int, 2>{});
	else launch(std::integral_constant<int, 3>{});
	return checkLaunch("kStencilApply");
}

extern "C" int phb_projection_gram(const double *V, const double *Y, const double *b, int32_t m, int64_t n, int64_t stride,
		double *G, double *c, phb_stream stream) {
	if (!V || !Y || !b || !G || !c) return setError(PHB_ERR_ARG, "phb_projection_gram: null argument");
	if (m < 1 || m > PROJ_MAX) return setError(PHB_ERR_RANGE, "phb_projection_gram: m outside 1..16");
	if (n < 0 || stride < n) return setError(PHB_ERR_ARG, "phb_projection_gram: n < 0 or stride < n");
	cudaStream_t s = (cudaStream_t)stream;
	PHB_CUDA(cudaMemsetAsync(G, 0, sizeof(double) * m * m, s));
	PHB_CUDA(cudaMemsetAsync(c, 0, sizeof(double) * m, s));
	if (n == 0) return PHB_OK;
	int dev = 0, sms = 0;
	PHB_CUDA(cudaGetDevice(&dev));
	PHB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
	const int64_t chunks = (n + GRAM_CHUNK - 1) / GRAM_CHUNK;
	const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(chunks, (int64_t)sms * 5));
	kProjectionGram<<<grid, 256, 0, s>>>(V, Y, b, m, n, stride, G, c);
	return checkLaunch("kProjectionGram");
}

extern "C" int phb_projection_solve(const double *G, const double *c, int32_t m, double reg, double *alpha,
		phb_stream stream) {
	if (!G || !c || !alpha) return setError(PHB_ERR_ARG, "phb_projection_solve: null argument");
	if (m < 1 || m > PROJ_MAX) return setError(PHB_ERR_RANGE, "phb_projection_solve: m outside 1..16");
	kProjectionSolve<<<1, 256, 0, (cudaStream_t)stream>>>(G, c, m, reg, alpha);
	return checkLaunch("kProjectionSolve");
}

extern "C" int phb_release_graphs(void) {
	std::lock_guard<std::mutex> lock(gMutex);
	return releaseGraphsLocked();
}

// refinement ------------------------------------------------------------------------------
extern "C" int64_t phb_refine_work_bytes(const phb_domain *dom, int kind, int nrhs) {
	if (!dom) return -1;
	const size_t inner = solveLayout(dom, kind, 4, nrhs).total;
	const size_t v = align256((size_t)dom->ncells * nrhs * 4);
	return (int64_t)(inner + 2 * v + align256((size_t)dom->ntiles * nrhs * 2 * sizeof(double)));
}

template <int D, int K>
static int emitRefine(const phb_domain *dom, const phb_refine *rf, cudaStream_t s, Streams &ss) {
	Dom<double, D> dm(*dom);
	const size_t inner = solveLayout(dom, rf->kind, 4, K).total;
	const size_t vb = align256((size_t)dom->ncells * K * 4);
	char *w = (char *)rf->work;
	float *r32 = (float *)(w + inner);
	float *e32 = (float *)(w + inner + vb);
	double *partial = (double *)(w + inner + 2 * vb);
	dm.vec4 = vec4Ok(dom, {rf->A64, rf->b, rf->x, w});
	const StateLayout SL = stateLayout(dom, K);
	char *sb = (char *)rf->state;
	Control *ctrlO = (Control *)(sb + SL.ctrl2);
	SysState *stO = (SysState *)(sb + SL.st2);
	SysState *stI = (SysState *)(sb + SL.st);
	const int nsys = dom->ninst * K;
	phb_solve in = {};
	in.kind = rf->kind;
	in.vec_dtype = PHB_F32;
	in.mat_dtype = PHB_F32;
	in.nrhs = K;
	in.maxit = rf->inner_maxit;
	in.return_best = 0;
	in.use_graph = 1;
	in.A = rf->A32;
	in.b = r32;
	in.x = e32;
	in.tol = phb_tolerance{}; // unused: the inner tolerance is SysState::innerTol
	in.work = rf->work;
	in.state = rf->state;
	in.amg = rf->amg;
	in.ctas_per_sm = rf->ctas_per_sm;
	// 1: nested graph loops; 2: graph outer loop, persistent inner solves; 3: host outer loop,
	// persistent inner solves (every launch visible to a kernel profiler); 0: host loops
	const bool graph = rf->use_graph == 1 || rf->use_graph == 2;
	in.use_graph = rf->use_graph >= 2 ? 2 : (graph ? 1 : 0);
	if (rf->use_graph == 2 && bicgPrefersGraph(dom, rf->kind, true, K)) in.use_graph = 1; // nested graph loop
	in.check_every = 8;
	cudaGraphConditionalHandle outerHandle{};
	if (graph) {
		const int rc0 = createCondition(s, &outerHandle);
		if (rc0) return rc0;
	}
	kInitOuter<<<1, 256, 0, s>>>(stO, nsys, rf->tol, ctrlO, rf->max_outer + 2);
	PHB_CUDA(cudaGetLastError());
	// The residual comes before the loop and at the end of its body, so that a system that needs no
	// (further) correction starts no inner solve: the pass of the loop that would only have found
	// that out cost 20 to 40 us a solve.
	auto residual = [&](cudaStream_t os, LoopCond lc) -> int {
		kRefineResidual<D, K><<<dom->ntiles, PHB_TILE, 0, os>>>(dm, rf->A64, rf->b, rf->x, r32, e32, stO, partial, ctrlO,
			rf->inner_rtol, rf->max_outer, rf->tol, stI, lc);
		return checkLaunch("kRefineResidual");
	};
	auto sweep = [&](cudaStream_t os, LoopCond lc) -> int {
		int rc = emitSolve<float, D, K>(dom, &in, os, ss, graph ? 2 : 0, true, 1);
		if (rc) return rc;
		kRefineUpdate<K><<<gridFor(dom->ncells * K), 256, 0, os>>>(dom->ncells * K, rf->x, e32);
		rc = checkLaunch("kRefineUpdate");
		if (rc) return rc;
		return residual(os, lc);
	};
	int rc = residual(s, LoopCond{outerHandle, graph ? 1 : 0});
	if (rc) return rc;
	if (graph) return addWhile(s, ss.s[1], outerHandle, sweep);
	// host loop: every kernel launched on its own (profilers see each launch)
	int *hflag = nullptr;
	PHB_CUDA(cudaMallocHost(&hflag, sizeof(int)));
	for (int k = 0; k < rf->max_outer + 2; ++k) {
		cudaMemcpyAsync(hflag, &ctrlO->allDone, sizeof(int), cudaMemcpyDeviceToHost, s);
		cudaStreamSynchronize(s);
		if (*hflag) break;
		rc = sweep(s, LoopCond{0, 0});
		if (rc) break;
	}
	cudaFreeHost(hflag);
	return rc;
}

extern "C" int phb_refine_results(const phb_domain *dom, const phb_refine *r, phb_solve_result *out, int *outer_used, phb_stream stream);

extern "C" int phb_refine_run(const phb_domain *dom, const phb_refine *r, phb_solve_result *out, int *outer_used, phb_stream stream) {
	if (!dom || !r || !r->A64 || !r->A32 || !r->b || !r->x || !r->work || !r->state || (r->tol.mode == 2 && !r->tol.values))
		return setError(PHB_ERR_ARG, "phb_refine_run: null argument");
	if (r->amg) {
		if (r->kind != 0 || r->nrhs != 1) return setError(PHB_ERR_ARG, "phb_refine_run: the AMG preconditioner takes CG with one right-hand side");
		const int rc = phbCheckAmg(r->amg);
		if (rc) return rc;
		if (r->amg->levels[0].dom.ncells != dom->ncells || !r->amg->levels[0].x) return setError(PHB_ERR_ARG, "phb_refine_run: hierarchy does not match the domain");
	}
	if (dom->ntiles == 0) return PHB_OK;
	cudaStream_t st = (cudaStream_t)stream;
	std::string key = makeKey("refine", *dom, *r);
	if (r->amg) key.append(reinterpret_cast<const char *>(r->amg), sizeof(phb_amg));
	int rc = PHB_OK;
	const int K = r->nrhs;
	if (r->use_graph == 0 || r->use_graph == 3) {
		Streams *ss;
		rc = getStreams(ss);
		if (rc) return rc;
		if (dom->dims == 2 && K == 1) rc = emitRefine<2, 1>(dom, r, st, *ss);
		else if (dom->dims == 2 && K == 2) rc = emitRefine<2, 2>(dom, r, st, *ss);
		else if (dom->dims == 3 && K == 1) rc = emitRefine<3, 1>(dom, r, st, *ss);
		else if (dom->dims == 3 && K == 3) rc = emitRefine<3, 3>(dom, r, st, *ss);
		else return setError(PHB_ERR_ARG, "phb_refine_run: unsupported dims/nrhs");
		if (rc) return rc;
		if (out) return phb_refine_results(dom, r, out, outer_used, stream);
		return PHB_OK;
	}
	if (dom->dims == 2 && K == 1) rc = runGraph(st, key, [&](cudaStream_t cs, Streams &ss) { return emitRefine<2, 1>(dom, r, cs, ss); });
	else if (dom->dims == 2 && K == 2) rc = runGraph(st, key, [&](cudaStream_t cs, Streams &ss) { return emitRefine<2, 2>(dom, r, cs, ss); });
	else if (dom->dims == 3 && K == 1) rc = runGraph(st, key, [&](cudaStream_t cs, Streams &ss) { return emitRefine<3, 1>(dom, r, cs, ss); });
	else if (dom->dims == 3 && K == 3) rc = runGraph(st, key, [&](cudaStream_t cs, Streams &ss) { return emitRefine<3, 3>(dom, r, cs, ss); });
	else return setError(PHB_ERR_ARG, "phb_refine_run: unsupported dims/nrhs");
	if (rc) return rc;
	if (out) return phb_refine_results(dom, r, out, outer_used, stream);
	return PHB_OK;
}

extern "C" int phb_refine_results(const phb_domain *dom, const phb_refine *r, phb_solve_result *out, int *outer_used, phb_stream stream) {
	if (!dom || !r || !out || !r->state) return setError(PHB_ERR_ARG, "phb_refine_results: null argument");
	const int K = r->nrhs;
	const int nsys = dom->ninst * K;
	std::vector<SysState> h(nsys);
	const StateLayout SL = stateLayout(dom, K);
	cudaStream_t st = (cudaStream_t)stream;
	PHB_CUDA(cudaMemcpyAsync(h.data(), (char *)r->state + SL.st2, nsys * sizeof(SysState), cudaMemcpyDeviceToHost, st));
	PHB_CUDA(cudaStreamSynchronize(st));
	int mo = 0;
	for (int i = 0; i < nsys; ++i) {
		out[i].final_residual = h[i].crit;
		out[i].used_iterations = h[i].it;
		out[i].converged = h[i].done == CONVERGED;
		out[i].finite = std::isfinite(h[i].crit);
		out[i].status = h[i].done;
		out[i].inner_iterations = h[i].innerIts;
		mo = std::max(mo, h[i].it);
	}
	if (outer_used) *outer_used = mo;
	return PHB_OK;
}

// no-allocation CG -------------------------------------------------------------------------
// Some hosts cannot hand this library device memory for solver workspace: a program that
// carves the GPU into fixed per-environment slices at start-up and forbids any later
// allocation, or a plugin host whose device allocator is not reachable through a C ABI.
// For them the CG solve below keeps its workspace (residual, search directions, partial
// sums, per-system state) in this file-scope array instead of the caller-provided `work`
// and `state` buffers of phb_solve_run. Every GPU that loads the library holds the array
// until the process exits.
static __device__ __align__(256) unsigned char gNoAllocScratch[PHB_NOALLOC_SCRATCH_BYTES];

// Device address of the array on each device. In host code `gNoAllocScratch` names a
// host-side stand-in, not device memory, so the address is looked up with the device
// current: by the first call on a device, and again by every call whose stream is not
// capturing (a cheap host call), so that a context that was reset and re-created, which
// reloads the module and may move the array, is followed. A call made while its stream is
// capturing uses the address of the last call that was not, so the first call on a device
// must come before any capture.
static std::mutex gNoAllocMutex;
static void *gNoAllocPtr[64] = {nullptr};

static int noAllocScratch(cudaStream_t s, void **out) {
	int dev;
	PHB_CUDA(cudaGetDevice(&dev));
	if (dev < 0 || dev >= 64) return setError(PHB_ERR_RANGE, "phb_cg_solve_noalloc: device index out of range");
	cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
	PHB_CUDA(cudaStreamIsCapturing(s, &cap));
	std::lock_guard<std::mutex> lock(gNoAllocMutex);
	if (cap == cudaStreamCaptureStatusNone) {
		void *p = nullptr;
		PHB_CUDA(cudaGetSymbolAddress(&p, gNoAllocScratch));
		gNoAllocPtr[dev] = p;
	} else if (!gNoAllocPtr[dev]) {
		return setError(PHB_ERR_ARG, "phb_cg_solve_noalloc: the first call on a device must not be made while its stream is capturing");
	}
	*out = gNoAllocPtr[dev];
	return PHB_OK;
}

template <typename T, int D, int K>
static int runCgNoAlloc(const phb_domain *dom, const phb_solve *sv, phb_solve_result *out, cudaStream_t s) {
	Dom<double, D> dm(*dom);
	const Layout L = solveLayout(dom, 0, sizeof(T), K, true);
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
	T *r = (T *)(w + L.off[0]), *q = (T *)(w + L.off[1]), *p0 = (T *)(w + L.off[2]), *p1 = (T *)(w + L.off[3]);
	T *xbest = sv->return_best ? (T *)(w + L.off[4]) : nullptr;
	const int nsys = dom->ninst * K;
	const int tiles = dom->ntiles;
	const int maxit = std::max(1, sv->maxit);
	const int maxLoops = maxit / 2 + 2;
	// kInit resets the state and the ticket counter the reductions count with, so nothing
	// left in the array by an earlier call is read before it is written
	kInit<<<1, 256, 0, s>>>(st, nsys, sv->tol, 0, maxit, ctrl, maxLoops);
	kResidual<T, D, K, false, false><<<tiles, PHB_TILE, 0, s>>>(dm, A, b, x, r, nullptr, st, partial, ctrl, sv->tol, LoopCond{0, 0});
	PHB_CUDA(cudaGetLastError());
	const int chk = std::max(1, sv->check_every);
	for (int loops = 0; loops < maxLoops; loops += chk) {
		for (int i = 0; i < chk; ++i) {
			for (int half = 0; half < 2; ++half) {
				T *pIn = half == 0 ? p0 : p1, *pOut = half == 0 ? p1 : p0;
				kCgDirection<T, D, K><<<tiles, PHB_TILE, 0, s>>>(dm, A, r, pIn, pOut, q, st, partial, ctrl);
				kCgUpdate<T, D, K><<<tiles, PHB_TILE, 0, s>>>(dm, r, pOut, q, x, xbest, st, partial, ctrl, sv->return_best, LoopCond{0, 0});
			}
		}
		PHB_CUDA(cudaGetLastError());
		int done = 0; // pageable stack copy: synchronous, no staging buffer of ours
		PHB_CUDA(cudaMemcpyAsync(&done, &ctrl->allDone, sizeof(int), cudaMemcpyDeviceToHost, s));
		PHB_CUDA(cudaStreamSynchronize(s));
		if (done) break;
	}
	if (xbest) kRestoreBest<T, K><<<gridFor(dom->ncells * K), 256, 0, s>>>(dom->insts, dom->ninst, dom->ncells, x, xbest, st);
	PHB_CUDA(cudaGetLastError());
	if (out) {
		for (int i = 0; i < nsys; ++i) {
			SysState h;
			PHB_CUDA(cudaMemcpyAsync(&h, st + i, sizeof(SysState), cudaMemcpyDeviceToHost, s));
			PHB_CUDA(cudaStreamSynchronize(s));
			phb_solve_result &o = out[i];
			o.final_residual = h.crit;
			o.used_iterations = h.usedIt;
			o.converged = h.done == CONVERGED;
			o.finite = std::isfinite(h.crit);
			o.status = h.done;
			o.inner_iterations = 0;
			o.pad = 0;
			if (sv->return_best && (h.done == MAXIT || h.done == RISING) && h.bestIt >= 0 && h.best < h.crit) {
				o.used_iterations = h.bestIt;
				o.final_residual = h.best;
			}
		}
	}
	return PHB_OK;
}

extern "C" int64_t phb_cg_noalloc_bytes(const phb_domain *dom, int dtype, int nrhs) {
	if (!dom) return -1;
	const int vb = dtype == PHB_F64 ? 8 : 4;
	return (int64_t)(solveLayout(dom, 0, vb, nrhs, true).total + stateLayout(dom, nrhs).total);
}

extern "C" int phb_cg_solve_noalloc(const phb_domain *dom, int dtype, int nrhs, const void *A, const void *b, void *x,
		const phb_tolerance *tol, int maxit, int return_best, phb_solve_result *out, phb_stream stream) {
	if (!dom || !A || !b || !x || !tol || (tol->mode == 2 && !tol->values))
		return setError(PHB_ERR_ARG, "phb_cg_solve_noalloc: null argument");
	if (dtype != PHB_F32 && dtype != PHB_F64) return setError(PHB_ERR_ARG, "phb_cg_solve_noalloc: dtype");
	const int64_t need = phb_cg_noalloc_bytes(dom, dtype, nrhs);
	if (need > (int64_t)PHB_NOALLOC_SCRATCH_BYTES) {
		char msg[256];
		snprintf(msg, sizeof(msg), "phb_cg_solve_noalloc: the solve needs %lld bytes of scratch, more than the %lld of the "
			"static array (PHB_NOALLOC_SCRATCH_BYTES)", (long long)need, (long long)PHB_NOALLOC_SCRATCH_BYTES);
		return setError(PHB_ERR_RANGE, msg);
	}
	if (dom->ntiles == 0) { // nothing to solve: every system reports a converged empty solve
		if (out) {
			for (int i = 0; i < dom->ninst * nrhs; ++i) {
				phb_solve_result &o = out[i];
				o.final_residual = 0.0;
				o.used_iterations = 0;
				o.converged = 1;
				o.finite = 1;
				o.status = CONVERGED;
				o.inner_iterations = 0;
				o.pad = 0;
			}
		}
		return PHB_OK;
	}
	void *scratch = nullptr;
	int rc = noAllocScratch((cudaStream_t)stream, &scratch);
	if (rc) return rc;
	phb_solve sv = {};
	sv.kind = 0;
	sv.vec_dtype = sv.mat_dtype = dtype;
	sv.nrhs = nrhs;
	sv.maxit = maxit;
	sv.return_best = return_best ? 1 : 0;
	sv.use_graph = 0;
	sv.check_every = 16;
	sv.tol = *tol;
	sv.A = A;
	sv.b = b;
	sv.x = x;
	sv.work = scratch;
	sv.state = (char *)scratch + solveLayout(dom, 0, dtype == PHB_F64 ? 8 : 4, nrhs, true).total;
	cudaStream_t st = (cudaStream_t)stream;
	PHB_SOLVE_DISPATCH(dom->dims, dtype, nrhs, return runCgNoAlloc<T, D, KK>(dom, &sv, out, st));
	return PHB_OK;
}

extern "C" int phb_barrier_selftest(int ctas, int rounds, int absent_cta, unsigned int spin_limit, void *scratch, int *bar_err,
		int *rounds_done, phb_stream stream) {
	if (ctas < 1 || rounds < 0 || !scratch || !bar_err || !rounds_done || spin_limit < 1024)
		return setError(PHB_ERR_ARG, "phb_barrier_selftest: bad argument");
	if (((uintptr_t)scratch & 15) != 0) return setError(PHB_ERR_ARG, "phb_barrier_selftest: scratch must be 16-byte aligned");
	int perSM = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, kBarrierProbe, PHB_TILE, 0) != cudaSuccess || perSM < 1) perSM = 1;
	if (ctas > perSM * numSMs()) return setError(PHB_ERR_RANGE, "phb_barrier_selftest: more CTAs than can be co-resident");
	cudaStream_t s = (cudaStream_t)stream;
	Control *ctrl = (Control *)scratch;
	int *done = (int *)((char *)scratch + 256);
	PHB_CUDA(cudaMemsetAsync(scratch, 0, 256 + sizeof(int), s));
	cudaLaunchConfig_t cfg = {};
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeCooperative;
	attr[0].val.cooperative = 1;
	cfg.gridDim = dim3(ctas);
	cfg.blockDim = dim3(PHB_TILE);
	cfg.stream = s;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	PHB_CUDA(cudaLaunchKernelEx(&cfg, kBarrierProbe, ctrl, rounds, absent_cta, spin_limit, done));
	PHB_CUDA(cudaMemcpyAsync(bar_err, &ctrl->barErr, sizeof(int), cudaMemcpyDeviceToHost, s));
	PHB_CUDA(cudaMemcpyAsync(rounds_done, done, sizeof(int), cudaMemcpyDeviceToHost, s));
	PHB_CUDA(cudaStreamSynchronize(s));
	return PHB_OK;
}
