// The persistent Krylov solvers: one cooperative launch runs a whole CG or BiCGStab solve, with
// grid barriers between its phases (phb_krylov.cuh). The multigrid-preconditioned CG is in pcg.cu,
// the CG of small instances in cluster_cg.cu.
//
// What bounds a phase on grids that fit L2: the barrier (1.2 to 1.6 us) and the chain of dependent
// L2 round trips after it; on larger grids, bytes in flight. Block tables and the CTA's tile list
// stay in shared memory for the whole solve, all neighbour indices are formed before the loads,
// and the loads are issued without a branch between them. Rows of four cells are loaded as vectors
// where every row allows it; elsewhere a thread takes cells 256 apart, whose loads stay contiguous
// over a warp for every row length, and the inner products are formed through shared memory in
// the order of four consecutive cells per thread: the same bits as the per-phase kernels.
// Measured (B200, microseconds per iteration, before -> after): CG float64 on 442,368 cells 16.6 ->
// 14.3 and on 3.3 M cells 99 -> 81; BiCGStab float32 with three right-hand sides inside a
// refinement on 442,368 cells 77 -> 60, on 136,530 cells (odd rows) 86 -> 67, on 2.1 M 286 -> 192,
// with two on 64 2D instances (1.2 M) 180 -> 100.
#include "phb_krylov.cuh"

namespace phb {

constexpr int TILE_ITEMS = 16; // tiles whose (block, first cell) a CTA keeps in shared memory

// A CTA's view of the domain in a persistent kernel: block tables and its tiles.
template <typename T, int D, int K>
struct TileCtx {
	const Dom<double, D> &dom;
	const BlockTab *blk;
	Worker wk;
	const int2 *items; // of the group
	T *stage; // of the group: a tile of values for the inner products of unaligned rows
	bool vec; // operands on 16-byte boundaries
	int n;    // the group's tiles
	// Every phase visits them in the opposite order of the phase before: what that one touched last
	// (up to the 126 MB of L2) is read from L2, where in the same order it would just have been
	// evicted (CG on 3.3 M float64 cells 88 -> 81 us, with the reduction's wider loads).
	bool back;

	// f(block, first cell) for every tile of this group
	template <typename F>
	__device__ __forceinline__ void tiles(F f) const {
		for (int i = 0; i < n; ++i) {
			const int k = back ? n - 1 - i : i, t = wk.first + k * wk.step;
			const int2 w = k < TILE_ITEMS ? items[k] : make_int2(__ldg(dom.tiles + 2 * t), __ldg(dom.tiles + 2 * t + 1));
			f(blk[w.x], w.y);
		}
	}
	// the same with sums over every tile into dst: f(block, first cell, values)
	template <int NV, typename F>
	__device__ __forceinline__ void tileSums(double *dst, double *ws, F f) {
		TileSums<NV> sums{wk, reinterpret_cast<double (*)[NV][NWARPS]>(ws), dst, 0, back ? n - 1 : -1};
		tiles([&](const BlockTab &B, int l0) {
			double acc[NV];
#pragma unroll
			for (int q = 0; q < NV; ++q) acc[q] = 0;
			f(B, l0, acc);
			sums.add(acc);
			sums.next();
		});
		sums.finish();
		back = !back;
	}
	__device__ __forceinline__ bool rows4(const BlockTab &B) const {
		return vec && B.rows4() && (K == 1 || ((B.instOff | B.instN) & 3) == 0);
	}
	__device__ __forceinline__ static int64_t base(const BlockTab &B, int k) { return (int64_t)(K - 1) * B.instOff + (int64_t)k * B.instN; }
};

// y = A f and f at the quad g (x, y, z) of an aligned row, every active right-hand side
template <typename T, int D, int K, typename F>
__device__ __forceinline__ void rowApply(const BlockTab &B, int g, int x, int y, int z, int64_t N, const T *__restrict__ A,
		const bool (&act)[K], const F (&fld)[K], T (&yv)[K][4], T (&fv)[K][4]) {
	int o[2 * D];
	const unsigned int has = tabNeighbors<D, 4>(B, g, x, y, z, o);
	const bool hw = has & 1, he = has & 2;
	T a[2 * D + 1][4];
#pragma unroll
	for (int s = 0; s < 2 * D + 1; ++s) ld4(A + s * N + g, 4, true, a[s]);
#pragma unroll
	for (int k = 0; k < K; ++k) {
		if (!act[k]) {
#pragma unroll
			for (int i = 0; i < 4; ++i) yv[k][i] = fv[k][i] = 0;
			continue;
		}
		const int64_t d = TileCtx<T, D, K>::base(B, k);
		T v[2 * D - 2][4];
		fld[k].at4(g + d, 4, true, fv[k]);
		T w = fld[k].at(o[0] + d), e = fld[k].at(o[1] + d);
#pragma unroll
		for (int s = 0; s < 2 * D - 2; ++s) fld[k].at4(o[s + 2] + d, 4, true, v[s]);
		if (!hw) w = 0;
		if (!he) e = 0;
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			T s = a[0][i] * fv[k][i];
			s = fma(a[1][i], i ? fv[k][i ? i - 1 : 0] : w, s);
			s = fma(a[2][i], i < 3 ? fv[k][i < 3 ? i + 1 : 3] : e, s);
#pragma unroll
			for (int f = 2; f < 2 * D; ++f) s = fma(a[f + 1][i], (has >> f) & 1 ? v[f - 2][i] : T(0), s);
			yv[k][i] = s;
		}
	}
}
// the same at one cell
template <typename T, int D, int K, typename F>
__device__ __forceinline__ void cellApply(const BlockTab &B, int g, int x, int y, int z, int64_t N, const T *__restrict__ A,
		const bool (&act)[K], const F (&fld)[K], T (&yv)[K], T (&fv)[K]) {
	int o[2 * D];
	const unsigned int has = tabNeighbors<D, 1>(B, g, x, y, z, o);
	T a[2 * D + 1];
#pragma unroll
	for (int s = 0; s < 2 * D + 1; ++s) a[s] = A[s * N + g];
#pragma unroll
	for (int k = 0; k < K; ++k) {
		yv[k] = fv[k] = 0;
		if (!act[k]) continue;
		const int64_t d = TileCtx<T, D, K>::base(B, k);
		T v[2 * D];
		fv[k] = fld[k].at(g + d);
#pragma unroll
		for (int f = 0; f < 2 * D; ++f) v[f] = fld[k].at(o[f] + d);
		T s = a[0] * fv[k];
#pragma unroll
		for (int f = 0; f < 2 * D; ++f) s = fma(a[f + 1], (has >> f) & 1 ? v[f] : T(0), s);
		yv[k] = s;
	}
}

// One tile of a phase with a stencil product: y = A f and f per cell, emit(k, index, count, y, f)
// stores them (count 4: an aligned row of four, 1: one cell), dots(k, y, f, i0, acc) adds the
// thread's share of the inner products from four consecutive cells.
template <typename T, int D, int K, int NV, typename F, typename Emit, typename Dots>
__device__ __forceinline__ void tilePhase(const TileCtx<T, D, K> &cx, const BlockTab &B, int l0, int64_t N, const T *__restrict__ A,
		const bool (&act)[K], const F (&fld)[K], double (&acc)[NV], Emit emit, Dots dots) {
	const int nc = B.cells();
	auto where = [&](int l, int &x, int &y, int &z) {
		const int row = l / B.nx;
		z = D > 2 ? row / B.ny : 0;
		x = l - row * B.nx;
		y = row - z * B.ny;
	};
	if (cx.rows4(B)) {
		const int l = l0 + 4 * cx.wk.lt;
		if (l >= nc) return;
		int x, y, z;
		where(l, x, y, z);
		const int g = B.off + l;
		T yv[K][4], fv[K][4];
		rowApply<T, D, K>(B, g, x, y, z, N, A, act, fld, yv, fv);
#pragma unroll
		for (int k = 0; k < K; ++k) {
			if (!act[k]) continue;
			const int64_t o = g + TileCtx<T, D, K>::base(B, k);
			emit(k, o, 4, yv[k], fv[k]);
			dots(k, o, 4, yv[k], fv[k], acc);
		}
		return;
	}
	T yv[CPT][K], fv[CPT][K];
#pragma unroll
	for (int j = 0; j < CPT; ++j) {
		const int l = l0 + cx.wk.lt + j * PHB_TILE;
		const int lc = l < nc ? l : l0; // past the end: the tile's first cell, not used
		int x, y, z;
		where(lc, x, y, z);
		cellApply<T, D, K>(B, B.off + lc, x, y, z, N, A, act, fld, yv[j], fv[j]);
	}
	const int q0 = 4 * cx.wk.lt;
	const int n = max(0, min(4, nc - l0 - q0));
#pragma unroll
	for (int k = 0; k < K; ++k) {
		if (!act[k]) continue;
		const int64_t d = TileCtx<T, D, K>::base(B, k) + B.off;
		T y4[4], f4[4];
		// y, then f, from the thread that has the cell to the thread that sums it
		auto pass = [&](auto value, T(&v4)[4]) {
			cx.wk.sync();
#pragma unroll
			for (int j = 0; j < CPT; ++j) cx.stage[cx.wk.lt + j * PHB_TILE] = value(j);
			cx.wk.sync();
#pragma unroll
			for (int i = 0; i < 4; ++i) v4[i] = i < n ? cx.stage[q0 + i] : T(0);
		};
#pragma unroll
		for (int j = 0; j < CPT; ++j) {
			const int c = cx.wk.lt + j * PHB_TILE;
			if (l0 + c < nc) {
				const T y1[4] = {yv[j][k], 0, 0, 0}, f1[4] = {fv[j][k], 0, 0, 0};
				emit(k, d + l0 + c, 1, y1, f1);
			}
		}
		pass([&](int j) { return yv[j][k]; }, y4);
		pass([&](int j) { return fv[j][k]; }, f4);
		dots(k, d + l0 + q0, n, y4, f4, acc);
	}
	cx.wk.sync();
}

// values of a row of four (n = 4 with vec) or of the first n of four cells
template <typename T>
__device__ __forceinline__ void put(T *p, int n, const T (&v)[4]) {
	if (n == 4) st4(p, 4, true, v);
	else p[0] = v[0];
}

// The first phase: r = b - A x, (r, r) and (b, b) into acc[2k], acc[2k + 1]; emit(index, n, r)
template <typename T, int D, int K, typename F, typename Emit>
__device__ __forceinline__ void residualTile(const TileCtx<T, D, K> &cx, const BlockTab &B, int l0, int64_t N, const T *__restrict__ A,
		const T *__restrict__ b, const bool (&act)[K], const F (&fx)[K], double (&acc)[2 * K], Emit emit) {
	auto residual = [&](int64_t o, int n, const T (&y)[4], T (&bv)[4], T (&rv)[4]) {
		ld4(b + o, n, cx.rows4(B) && n == 4, bv);
#pragma unroll
		for (int i = 0; i < 4; ++i) rv[i] = bv[i] - y[i];
	};
	tilePhase<T, D, K>(cx, B, l0, N, A, act, fx, acc,
		[&](int, int64_t o, int n, const T (&y)[4], const T (&)[4]) {
			T bv[4], rv[4];
			residual(o, n, y, bv, rv);
			emit(o, n, rv);
		},
		[&](int k, int64_t o, int n, const T (&y)[4], const T (&)[4], double (&ac)[2 * K]) {
			T bv[4], rv[4];
			residual(o, n, y, bv, rv);
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				ac[2 * k] = fma(double(rv[i]), double(rv[i]), ac[2 * k]);
				ac[2 * k + 1] = fma(double(bv[i]), double(bv[i]), ac[2 * k + 1]);
			}
		});
}

// Shared prologue of the persistent kernels: states, block tables, tile list.
template <typename T, int D, int K>
__device__ __forceinline__ TileCtx<T, D, K> tileContext(const Dom<double, D> &dom, const BlockTab *blocks, SysState *sst, const SysState *st,
		int2 (*items)[TILE_ITEMS], T (*stage)[PHB_TILE_CELLS]) {
	const Worker wk;
	const int nsys = dom.ninst * K;
	BlockTab *sBlk = reinterpret_cast<BlockTab *>(sst + nsys);
	for (int s = threadIdx.x; s < nsys; s += blockDim.x) sst[s] = st[s];
	if (!blocks)
		for (int b = threadIdx.x; b < dom.nblocks; b += blockDim.x) buildBlockTab<D>(dom.blocks, b, sBlk[b]);
	if (wk.lt < TILE_ITEMS) {
		const int t = wk.first + wk.lt * wk.step;
		items[wk.id][wk.lt] = t < dom.ntiles ? make_int2(__ldg(dom.tiles + 2 * t), __ldg(dom.tiles + 2 * t + 1)) : make_int2(0, 0);
	}
	__syncthreads();
	return TileCtx<T, D, K>{dom, blocks ? blocks : sBlk, wk, items[wk.id], stage[wk.id], dom.vec4 != 0, wk.count(dom.ntiles), false};
}

// Worker groups per CTA: float32 with one right-hand side is bound by HBM on large grids and is
// faster with more warps in flight (four groups of 64 registers a thread); several right-hand sides
// and float64 need more registers.
template <typename T, int D, int K>
constexpr int cgGroups() {
	return (std::is_same<T, float>::value && K == 1) ? 4 : (K == 1 ? 3 : 2);
}
constexpr int BICG_GROUPS = 2;

template <typename T, int D, int K, bool STOPSTART>
__device__ __forceinline__ void cgPersistentBody(const Dom<double, D> &dom, const BlockTab *blocks, const T *__restrict__ A, const T *__restrict__ b,
		T *__restrict__ x, T *__restrict__ r, T *__restrict__ p0, T *__restrict__ p1, T *__restrict__ q, T *__restrict__ xbest,
		SysState *st, double *partial, Control *ctrl, const phb_tolerance &tol, int returnBest, int maxit) {
	extern __shared__ __align__(16) SysState sst[];
	constexpr int G = cgGroups<T, D, K>();
	__shared__ int2 items[G][TILE_ITEMS];
	__shared__ __align__(16) T stage[G][PHB_TILE_CELLS];
	__shared__ double sums[G][TILE_SUMS * 2 * K * NWARPS];
	TileCtx<T, D, K> cx = tileContext<T, D, K>(dom, blocks, sst, st, items, stage);
	double *ws = sums[cx.wk.id];
	const int64_t N = dom.ncells;
	auto range = [&](int inst) {
		const int32_t *in = dom.insts + inst * PHB_IREC;
		return make_int2(__ldg(in + I_TILESTART), __ldg(in + I_TILECOUNT));
	};
	// consecutive phases write alternate halves of the partials, so that a CTA that has left
	// a barrier cannot overwrite partials another CTA is still reducing
	const size_t half = (size_t)dom.ntiles * K * 3;
	int ph = 0;
	double *pp = partial;
	// r = b - A x, (r, r), (b, b)
	pp = partial + (size_t)(ph++ & 1) * half;
	cx.template tileSums<2 * K>(pp, ws, [&](const BlockTab &B, int l0, double (&acc)[2 * K]) {
		bool act[K];
		FX<T> fx[K];
#pragma unroll
		for (int k = 0; k < K; ++k) { act[k] = sst[B.inst * K + k].done == RUNNING; fx[k].x = x; }
		residualTile<T, D, K>(cx, B, l0, N, A, b, act, fx, acc, [&](int64_t o, int n, const T (&rv)[4]) { put(r + o, n, rv); });
	});
	if (!gridBarrier(ctrl)) return;
	int running = reduceSystems<K, 2, 1>(dom.ninst, pp, sst, range, [&](SysState &s, int in, const double *red, double bb) {
		residualDecision<K, false, STOPSTART>(nullptr, s, normScale(dom.insts, in), red, bb, tol);
	});
	T *pIn = p0, *pOut = p1;
	for (int iter = 0; running > 0 && iter <= maxit + 1; ++iter) {
		// p' = r + beta p, q = A p', (p', q)
		pp = partial + (size_t)(ph++ & 1) * half;
		cx.template tileSums<K>(pp, ws, [&](const BlockTab &B, int l0, double (&acc)[K]) {
			bool act[K];
			FDir<T> fd[K];
#pragma unroll
			for (int k = 0; k < K; ++k) {
				const SysState &s = sst[B.inst * K + k];
				act[k] = s.done == RUNNING;
				// a restart (p not yet written) takes p' = r: r + 0 r
				fd[k] = FDir<T>{r, s.restart ? r : pIn, s.restart ? T(0) : T(s.beta), false};
			}
			tilePhase<T, D, K>(cx, B, l0, N, A, act, fd, acc,
				[&](int, int64_t o, int n, const T (&y)[4], const T (&f)[4]) { put(pOut + o, n, f); put(q + o, n, y); },
				[&](int k, int64_t, int, const T (&y)[4], const T (&f)[4], double (&ac)[K]) {
#pragma unroll
					for (int i = 0; i < 4; ++i) ac[k] = fma(double(f[i]), double(y[i]), ac[k]);
				});
		});
		if (!gridBarrier(ctrl)) return;
		reduceSystems<K, 1, -1>(dom.ninst, pp, sst, range, [&](SysState &s, int, const double *red, double) {
			const double alpha = s.rho / red[0];
			s.restart = 0;
			if (!fin(alpha)) { s.done = NONFINITE; s.usedIt = s.it; }
			else s.alpha = alpha;
		});
		// x += alpha p', r -= alpha q, (r, r)
		pp = partial + (size_t)(ph++ & 1) * half;
		cx.template tileSums<K>(pp, ws, [&](const BlockTab &B, int l0, double (&acc)[K]) {
			const int l = l0 + 4 * cx.wk.lt;
			const int n = max(0, min(4, B.cells() - l));
			const bool al = cx.rows4(B) && n == 4;
#pragma unroll
			for (int k = 0; k < K; ++k) {
				const SysState &s = sst[B.inst * K + k];
				if (s.done != RUNNING) continue;
				const T alpha = T(s.alpha);
				const int64_t o = B.off + l + cx.base(B, k);
				T xv[4], pv[4], rv[4], qq[4];
				ld4(x + o, n, al, xv);
				ld4(pOut + o, n, al, pv);
				ld4(r + o, n, al, rv);
				ld4(q + o, n, al, qq);
				if (s.saveBest && xbest) st4(xbest + o, n, al, xv);
#pragma unroll
				for (int i = 0; i < 4; ++i) {
					xv[i] = fma(alpha, pv[i], xv[i]);
					rv[i] = fma(-alpha, qq[i], rv[i]);
					acc[k] = fma(double(rv[i]), double(rv[i]), acc[k]);
				}
				st4(x + o, n, al, xv);
				st4(r + o, n, al, rv);
			}
		});
		if (!gridBarrier(ctrl)) return;
		running = reduceSystems<K, 1, -1>(dom.ninst, pp, sst, range, [&](SysState &s, int in, const double *red, double) {
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
		cx.tiles([&](const BlockTab &B, int l0) {
			const int end = min(B.cells(), l0 + PHB_TILE_CELLS);
#pragma unroll
			for (int k = 0; k < K; ++k) {
				const SysState &s = sst[B.inst * K + k];
				if (!((s.done == MAXIT || s.done == RISING) && s.bestIt >= 0 && s.best < s.crit)) continue;
				const int64_t d = B.off + cx.base(B, k);
				for (int l = l0 + cx.wk.lt; l < end; l += PHB_TILE) x[d + l] = xbest[d + l];
			}
		});
	}
	if (blockIdx.x == 0) {
		__syncthreads();
		for (int s = threadIdx.x; s < dom.ninst * K; s += blockDim.x) st[s] = sst[s];
	}
}

template <typename T, int D, int K, bool STOPSTART>
__global__ void __launch_bounds__(PHB_TILE * cgGroups<T, D, K>(), 1) kCgPersistent(Dom<double, D> dom, const BlockTab *blocks, const T *__restrict__ A,
		const T *__restrict__ b, T *__restrict__ x, T *__restrict__ r, T *__restrict__ p0, T *__restrict__ p1, T *__restrict__ q,
		T *__restrict__ xbest, SysState *st, double *partial, Control *ctrl, phb_tolerance tol, int returnBest, int maxit) {
	cgPersistentBody<T, D, K, STOPSTART>(dom, blocks, A, b, x, r, p0, p1, q, xbest, st, partial, ctrl, tol, returnBest, maxit);
}

template <typename T, int D, int K, int G = BICG_GROUPS>
__global__ void __launch_bounds__(PHB_TILE *G, 1) kBicgPersistent(Dom<double, D> dom, const BlockTab *blocks, const T *__restrict__ A, const T *__restrict__ b,
		T *__restrict__ x, T *__restrict__ r, T *__restrict__ r0, T *__restrict__ p0, T *__restrict__ p1, T *__restrict__ v0,
		T *__restrict__ v1, T *__restrict__ t, SysState *st, double *partial, Control *ctrl, phb_tolerance tol, int maxit) {
	extern __shared__ __align__(16) SysState sst[];
	__shared__ int2 items[G][TILE_ITEMS];
	__shared__ __align__(16) T stage[G][PHB_TILE_CELLS];
	__shared__ double sums[G][TILE_SUMS * 3 * K * NWARPS];
	TileCtx<T, D, K> cx = tileContext<T, D, K>(dom, blocks, sst, st, items, stage);
	double *ws = sums[cx.wk.id];
	const int64_t N = dom.ncells;
	auto range = [&](int inst) {
		const int32_t *in = dom.insts + inst * PHB_IREC;
		return make_int2(__ldg(in + I_TILESTART), __ldg(in + I_TILECOUNT));
	};
	// consecutive phases write alternate halves of the partials, so that a CTA that has left
	// a barrier cannot overwrite partials another CTA is still reducing
	const size_t half = (size_t)dom.ntiles * K * 3;
	int ph = 0;
	double *pp = partial;
	pp = partial + (size_t)(ph++ & 1) * half;
	cx.template tileSums<2 * K>(pp, ws, [&](const BlockTab &B, int l0, double (&acc)[2 * K]) {
		bool act[K];
		FX<T> fx[K];
#pragma unroll
		for (int k = 0; k < K; ++k) { act[k] = sst[B.inst * K + k].done == RUNNING; fx[k].x = x; }
		residualTile<T, D, K>(cx, B, l0, N, A, b, act, fx, acc, [&](int64_t o, int n, const T (&rv)[4]) {
			put(r + o, n, rv);
			put(r0 + o, n, rv);
		});
	});
	if (!gridBarrier(ctrl)) return;
	int running = reduceSystems<K, 2, 1>(dom.ninst, pp, sst, range, [&](SysState &s, int in, const double *red, double bb) {
		residualDecision<K, true, true>(nullptr, s, normScale(dom.insts, in), red, bb, tol);
	});
	T *pIn = p0, *pOut = p1, *vIn = v0, *vOut = v1;
	for (int iter = 0; running > 0 && iter <= maxit + 1; ++iter) {
		// p = r + beta (p - omega v), v = A p, (r0, v)
		pp = partial + (size_t)(ph++ & 1) * half;
		cx.template tileSums<K>(pp, ws, [&](const BlockTab &B, int l0, double (&acc)[K]) {
			bool act[K];
			FBicgP<T> fp[K];
#pragma unroll
			for (int k = 0; k < K; ++k) {
				const SysState &s = sst[B.inst * K + k];
				act[k] = s.done == RUNNING;
				// a restart (p and v not yet written) takes p = r: r + 0 (r - 0 r)
				const bool rs = s.restart;
				fp[k] = FBicgP<T>{r, rs ? r : pIn, rs ? r : vIn, rs ? T(0) : T(s.beta), rs ? T(0) : T(s.omega), false};
			}
			tilePhase<T, D, K>(cx, B, l0, N, A, act, fp, acc,
				[&](int, int64_t o, int n, const T (&y)[4], const T (&f)[4]) { put(pOut + o, n, f); put(vOut + o, n, y); },
				[&](int k, int64_t o, int n, const T (&y)[4], const T (&)[4], double (&ac)[K]) {
					T w[4];
					ld4(r0 + o, n, cx.rows4(B) && n == 4, w);
#pragma unroll
					for (int i = 0; i < 4; ++i) ac[k] = fma(double(w[i]), double(y[i]), ac[k]);
				});
		});
		if (!gridBarrier(ctrl)) return;
		reduceSystems<K, 1, -1>(dom.ninst, pp, sst, range, [&](SysState &s, int, const double *red, double) {
			const double alpha = s.rho / red[0];
			s.restart = 0;
			if (!fin(alpha)) { s.done = NONFINITE; s.usedIt = s.it; }
			else s.alpha = alpha;
		});
		// s = r - alpha v, t = A s, (t,s), (t,t), (s,s)
		pp = partial + (size_t)(ph++ & 1) * half;
		cx.template tileSums<3 * K>(pp, ws, [&](const BlockTab &B, int l0, double (&acc)[3 * K]) {
			bool act[K];
			FBicgS<T> fs[K];
#pragma unroll
			for (int k = 0; k < K; ++k) {
				const SysState &s = sst[B.inst * K + k];
				act[k] = s.done == RUNNING;
				fs[k] = FBicgS<T>{r, vOut, T(s.alpha)};
			}
			tilePhase<T, D, K>(cx, B, l0, N, A, act, fs, acc,
				[&](int, int64_t o, int n, const T (&y)[4], const T (&)[4]) { put(t + o, n, y); },
				[&](int k, int64_t, int, const T (&y)[4], const T (&f)[4], double (&ac)[3 * K]) {
#pragma unroll
					for (int i = 0; i < 4; ++i) {
						ac[3 * k + 0] = fma(double(y[i]), double(f[i]), ac[3 * k + 0]);
						ac[3 * k + 1] = fma(double(y[i]), double(y[i]), ac[3 * k + 1]);
						ac[3 * k + 2] = fma(double(f[i]), double(f[i]), ac[3 * k + 2]);
					}
				});
		});
		if (!gridBarrier(ctrl)) return;
		reduceSystems<K, 3, -1>(dom.ninst, pp, sst, range, [&](SysState &s, int in, const double *red, double) {
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
		cx.template tileSums<2 * K>(pp, ws, [&](const BlockTab &B, int l0, double (&acc)[2 * K]) {
			const int l = l0 + 4 * cx.wk.lt;
			const int n = max(0, min(4, B.cells() - l));
			const bool al = cx.rows4(B) && n == 4;
#pragma unroll
			for (int k = 0; k < K; ++k) {
				const SysState &s = sst[B.inst * K + k];
				if (s.done != RUNNING) continue;
				const T alpha = T(s.alpha), omega = T(s.omega);
				const int64_t o = B.off + l + cx.base(B, k);
				T rv[4], vv[4], pv[4], xv[4];
				ld4(r + o, n, al, rv);
				ld4(vOut + o, n, al, vv);
				ld4(pOut + o, n, al, pv);
				ld4(x + o, n, al, xv);
				if (s.halfDone) {
#pragma unroll
					for (int i = 0; i < 4; ++i) {
						xv[i] = fma(alpha, pv[i], xv[i]);
						rv[i] = fma(-alpha, vv[i], rv[i]);
					}
				} else {
					T tv[4], r0v[4];
					ld4(t + o, n, al, tv);
					ld4(r0 + o, n, al, r0v);
#pragma unroll
					for (int i = 0; i < 4; ++i) {
						const T si = fma(-alpha, vv[i], rv[i]);
						xv[i] = fma(omega, si, fma(alpha, pv[i], xv[i]));
						rv[i] = fma(-omega, tv[i], si);
						acc[2 * k + 0] = fma(double(r0v[i]), double(rv[i]), acc[2 * k + 0]);
						acc[2 * k + 1] = fma(double(rv[i]), double(rv[i]), acc[2 * k + 1]);
					}
				}
				st4(x + o, n, al, xv);
				st4(r + o, n, al, rv);
			}
		});
		if (!gridBarrier(ctrl)) return;
		running = reduceSystems<K, 2, -1>(dom.ninst, pp, sst, range, [&](SysState &s, int in, const double *red, double) {
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
		for (int s = threadIdx.x; s < dom.ninst * K; s += blockDim.x) st[s] = sst[s];
	}
}

template <int D>
__global__ void kBlockTabs(const int32_t *blocks, int n, BlockTab *out) {
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) buildBlockTab<D>(blocks, i, out[i]);
}

// A persistent solve: kInit, then one cooperative launch of the whole iteration (the grid is
// sized so that every CTA is resident; the launch fails rather than deadlocks otherwise).
template <typename T, int D, int K>
int launchPersistent(const phb_domain *dom, const phb_solve *sv, cudaStream_t s, bool stopStart, int fromInner) {
	if constexpr (std::is_same<T, float>::value && K == 1) {
		if (sv->amg && sv->kind == 0) return launchPcg<D>(dom, sv, s, stopStart, fromInner);
	}
	const int nsys = dom->ninst * K;
	const size_t stBytes = (size_t)nsys * sizeof(SysState);
	// the limit of the grid kernels' state copies, and of the mode: the same for every kernel it may pick
	if (stBytes > 160 * 1024) return setError(PHB_ERR_RANGE, "persistent solve: too many systems for the per-CTA state copy");
	if constexpr (K == 1) {
		if (sv->kind == 0) {
			bool taken = false;
			const int rc = launchClusterCg<T, D>(dom, sv, s, stopStart, fromInner, &taken);
			if (rc || taken) return rc;
		}
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
	const int maxit = std::max(1, sv->maxit);
	const int rc = launchInit(st, nsys, sv->tol, fromInner, maxit, ctrl, s);
	if (rc) return rc;
	const size_t tabBytes = (size_t)dom->nblocks * sizeof(BlockTab);
	size_t smem = stBytes + tabBytes;
	const BlockTab *tabs = nullptr;
	if (tabBytes > TAB_SMEM_MAX || smem > 160 * 1024) {
		smem = stBytes;
		BlockTab *t = (BlockTab *)(w + L.off[9]);
		kBlockTabs<D><<<std::max(1, std::min(1024, (dom->nblocks + 127) / 128)), 128, 0, s>>>(dom->blocks, dom->nblocks, t);
		PHB_CUDA(cudaGetLastError());
		tabs = t;
	}
	cudaLaunchConfig_t cfg = {};
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeCooperative;
	attr[0].val.cooperative = 1;
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	auto configure = [&](const void *kern, int most) -> int {
		if (smem > 8 * 1024) PHB_CUDA(allowSmem(kern));
		int groups = 1, ctas = 1;
		persistentGrid(dom->ntiles, most, sv->ctas_per_sm, groups, ctas);
		cfg.gridDim = dim3(ctas);
		cfg.blockDim = dim3(PHB_TILE * groups);
		return PHB_OK;
	};
	if (sv->kind == 0) {
		T *r = (T *)(w + L.off[0]), *q = (T *)(w + L.off[1]), *p0 = (T *)(w + L.off[2]), *p1 = (T *)(w + L.off[3]);
		T *xbest = sv->return_best ? (T *)(w + L.off[4]) : nullptr;
		auto launch = [&](auto kern) -> int {
			const int rc2 = configure((const void *)kern, cgGroups<T, D, K>());
			if (rc2) return rc2;
			PHB_CUDA(cudaLaunchKernelEx(&cfg, kern, dm, tabs, A, b, x, r, p0, p1, q, xbest, st, partial, ctrl, sv->tol, sv->return_best, maxit));
			return PHB_OK;
		};
		return stopStart ? launch(kCgPersistent<T, D, K, true>) : launch(kCgPersistent<T, D, K, false>);
	}
	T *r = (T *)(w + L.off[0]), *r0 = (T *)(w + L.off[1]), *p0 = (T *)(w + L.off[2]), *p1 = (T *)(w + L.off[3]);
	T *v0 = (T *)(w + L.off[4]), *v1 = (T *)(w + L.off[5]), *t = (T *)(w + L.off[6]);
	auto launch = [&](auto kern) -> int {
		const int rc2 = configure((const void *)kern, BICG_GROUPS);
		if (rc2) return rc2;
		PHB_CUDA(cudaLaunchKernelEx(&cfg, kern, dm, tabs, A, b, x, r, r0, p0, p1, v0, v1, t, st, partial, ctrl, sv->tol, maxit));
		return PHB_OK;
	};
	// float64 with three right-hand sides needs more than the 128 registers of two groups (it spills 456 bytes):
	// a grid of one group per SM (one tile per SM or less) takes the kernel that may have twice as many: 32^3
	// cells 32 -> 26 us per iteration, 48^3 35 -> 28
	if constexpr (std::is_same<T, double>::value && K == 3) {
		int groups = 1, ctas = 1;
		persistentGrid(dom->ntiles, BICG_GROUPS, sv->ctas_per_sm, groups, ctas);
		if (groups == 1) return launch(kBicgPersistent<T, D, K, 1>);
	}
	return launch(kBicgPersistent<T, D, K>);
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
