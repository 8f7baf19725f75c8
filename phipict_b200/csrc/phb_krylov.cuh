// Device code shared by the Krylov translation units: per-system state, the stencil products on
// quads, the tile bodies of CG and BiCGStab, the grid barrier and the reductions of the
// persistent kernels, and the workspace layouts.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>
#include <initializer_list>
#include <type_traits>
#include "phb_device.cuh"
#include "phb_amg.cuh"
#include "phb_launch.cuh"

namespace phb {

constexpr int NWARPS = PHB_TILE / 32;
enum Done : int { RUNNING = 0, CONVERGED = 1, NONFINITE = 2, MAXIT = 3, RISING = 4 };
constexpr int RISING_CUTOFF = 100;

struct SysState {
	double tol, rho, alpha, beta, omega, crit, best, last, halfCrit, innerTol;
	int it, maxit, bestIt, rising, done, restart, saveBest, halfDone, usedIt, innerIts;
	int launched, pad2;
};
static_assert(sizeof(SysState) == 128, "SysState layout");

struct Control {
	unsigned int counter;
	int allDone;
	int loops;
	int maxLoops;
	unsigned int barCount; // grid barrier of the persistent solvers: arrival counter
	int barErr;            // set when a barrier wait ran out (the kernel then returns)
	int pad[2];
};
static_assert(sizeof(Control) == 32, "Control layout");

// device helpers -----------------------------------------------------------------------
__device__ __forceinline__ double warpSum(double v) {
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	return v;
}

__device__ __forceinline__ bool fin(double v) { return isfinite(v); }
__device__ __forceinline__ double normScale(const int32_t *insts, int inst) { return 1.0 / sqrt(double(insts[inst * PHB_IREC + I_NCELLS])); }

template <int K>
__device__ __forceinline__ int64_t vk(const int32_t *B, int64_t g, int k) {
	return g + (int64_t)(K - 1) * B[B_INSTOFF] + (int64_t)k * B[B_INSTN];
}

template <int D>
__device__ __forceinline__ void stencilNeighbors(const Dom<double, D> &dom, const Cell &c, int64_t *nb) {
#pragma unroll
	for (int f = 0; f < 2 * D; ++f) nb[f] = neighborIndex<double, D>(dom, c, f);
}

// Krylov tile bodies on quads ------------------------------------------------------------
// Fields evaluated at the stencil points: at(o) one value, at4(o) four consecutive values.
// Every multiply-add is an explicit fma, so that the persistent kernel and the per-phase
// kernels round identically whatever contraction the compiler would choose in each.
template <typename T>
struct FX { // a stored vector
	const T *x;
	__device__ __forceinline__ T at(int64_t o) const { return x[o]; }
	__device__ __forceinline__ void at4(int64_t o, int n, bool al, T (&v)[4]) const { ld4(x + o, n, al, v); }
};
template <typename T>
struct FDir { // CG direction p' = z + beta p (z after a restart)
	const T *z, *p;
	T beta;
	bool rs;
	__device__ __forceinline__ T at(int64_t o) const { return rs ? z[o] : fma(beta, p[o], z[o]); }
	__device__ __forceinline__ void at4(int64_t o, int n, bool al, T (&v)[4]) const {
		ld4(z + o, n, al, v);
		if (rs) return;
		T b[4];
		ld4(p + o, n, al, b);
#pragma unroll
		for (int i = 0; i < 4; ++i) v[i] = fma(beta, b[i], v[i]);
	}
};
template <typename T>
struct FBicgP { // BiCGStab direction p = r + beta (p - omega v) (r after a restart)
	const T *r, *p, *v;
	T beta, omega;
	bool rs;
	__device__ __forceinline__ T at(int64_t o) const { return rs ? r[o] : fma(beta, fma(-omega, v[o], p[o]), r[o]); }
	__device__ __forceinline__ void at4(int64_t o, int n, bool al, T (&w)[4]) const {
		ld4(r + o, n, al, w);
		if (rs) return;
		T a[4], b[4];
		ld4(p + o, n, al, a);
		ld4(v + o, n, al, b);
#pragma unroll
		for (int i = 0; i < 4; ++i) w[i] = fma(beta, fma(-omega, b[i], a[i]), w[i]);
	}
};
template <typename T>
struct FBicgS { // BiCGStab half step s = r - alpha v
	const T *r, *v;
	T alpha;
	__device__ __forceinline__ T at(int64_t o) const { return fma(-alpha, v[o], r[o]); }
	__device__ __forceinline__ void at4(int64_t o, int n, bool al, T (&w)[4]) const {
		T b[4];
		ld4(r + o, n, al, w);
		ld4(v + o, n, al, b);
#pragma unroll
		for (int i = 0; i < 4; ++i) w[i] = fma(-alpha, b[i], w[i]);
	}
};

// y = A f and f itself at the quad's cells for every active right-hand side (zeros for the
// others and past q.n). On the fast path (a quad inside one row whose y and z neighbours are
// in the block or absent behind a prescribed face) the four cells' stencil rows and neighbour
// groups are loaded at once, slot by slot; elsewhere every cell resolves its neighbours
// across faces. The products are summed in the same order on both paths (centre, then faces
// -x +x -y +y -z +z, a face without neighbour skipped).
template <typename T, int D, int K, typename F>
__device__ __forceinline__ void quadApply(const Dom<double, D> &dom, const T *__restrict__ A, const Quad &q, const bool (&act)[K],
		const F (&fld)[K], T (&y)[K][4], T (&f)[K][4]) {
	const int64_t N = dom.ncells;
	if (q.fastW) {
		// x neighbours of the row ends: across the block's x face when the quad touches it
		int64_t gW = q.g - 1, gE = q.g + 4;
		if (q.p[0] == 0 || q.p[0] + 3 == q.B[B_NX] - 1) {
			Cell c;
			c.B = q.B;
			c.p[1] = q.p[1];
			c.p[2] = q.p[2];
			if (q.p[0] == 0) {
				c.p[0] = 0;
				c.g = (int)q.g;
				gW = neighborIndex<double, D>(dom, c, 0);
			}
			if (q.p[0] + 3 == q.B[B_NX] - 1) {
				c.p[0] = q.p[0] + 3;
				c.g = (int)(q.g + 3);
				gE = neighborIndex<double, D>(dom, c, 1);
			}
		}
		int64_t o[K];
#pragma unroll
		for (int k = 0; k < K; ++k) o[k] = vk<K>(q.B, q.g, k);
		T a[4];
		ld4(A + q.g, 4, q.al, a);
#pragma unroll
		for (int k = 0; k < K; ++k) {
			if (!act[k]) {
#pragma unroll
				for (int i = 0; i < 4; ++i) f[k][i] = 0;
			} else {
				fld[k].at4(o[k], 4, q.al, f[k]);
			}
#pragma unroll
			for (int i = 0; i < 4; ++i) y[k][i] = a[i] * f[k][i];
		}
		ld4(A + N + q.g, 4, q.al, a);
#pragma unroll
		for (int k = 0; k < K; ++k) {
			if (!act[k]) continue;
			if (gW >= 0) y[k][0] = fma(a[0], fld[k].at(vk<K>(q.B, gW, k)), y[k][0]);
#pragma unroll
			for (int i = 1; i < 4; ++i) y[k][i] = fma(a[i], f[k][i - 1], y[k][i]);
		}
		ld4(A + 2 * N + q.g, 4, q.al, a);
#pragma unroll
		for (int k = 0; k < K; ++k) {
			if (!act[k]) continue;
#pragma unroll
			for (int i = 0; i < 3; ++i) y[k][i] = fma(a[i], f[k][i + 1], y[k][i]);
			if (gE >= 0) y[k][3] = fma(a[3], fld[k].at(vk<K>(q.B, gE, k)), y[k][3]);
		}
#pragma unroll
		for (int sl = 3; sl < 2 * D + 1; ++sl) {
			if ((q.miss >> (sl - 3)) & 1) continue; // behind a prescribed face: no neighbour
			const int64_t off = sl == 3 ? -(int64_t)q.sy : sl == 4 ? (int64_t)q.sy : sl == 5 ? -(int64_t)q.sz : (int64_t)q.sz;
			const bool al = sl < 5 ? q.alY : q.alZ;
			ld4(A + sl * N + q.g, 4, q.al, a);
#pragma unroll
			for (int k = 0; k < K; ++k) {
				if (!act[k]) continue;
				T v[4];
				fld[k].at4(o[k] + off, 4, al, v);
#pragma unroll
				for (int i = 0; i < 4; ++i) y[k][i] = fma(a[i], v[i], y[k][i]);
			}
		}
		return;
	}
#pragma unroll
	for (int i = 0; i < 4; ++i) {
#pragma unroll
		for (int k = 0; k < K; ++k) { y[k][i] = 0; f[k][i] = 0; }
		if (i >= q.n) continue;
		Cell c;
		quadCell<D>(q, i, c);
		int64_t nb[2 * D];
		stencilNeighbors<D>(dom, c, nb);
		const T a0 = A[c.g];
		T af[2 * D];
#pragma unroll
		for (int fc = 0; fc < 2 * D; ++fc) af[fc] = A[(fc + 1) * N + c.g];
#pragma unroll
		for (int k = 0; k < K; ++k) {
			if (!act[k]) continue;
			const T ci = fld[k].at(vk<K>(c.B, c.g, k));
			T s = a0 * ci;
#pragma unroll
			for (int fc = 0; fc < 2 * D; ++fc)
				if (nb[fc] >= 0) s = fma(af[fc], fld[k].at(vk<K>(c.B, nb[fc], k)), s);
			y[k][i] = s;
			f[k][i] = ci;
		}
	}
}

// r = b - A x per right-hand side, (r, r) and (b, b) into acc[2k], acc[2k+1]; emit(k, o, q,
// r[4]) stores r.
template <typename T, int D, int K, typename Emit>
__device__ __forceinline__ void tileResidual(const Dom<double, D> &dom, const int32_t *sB, int l0, int nc, const T *__restrict__ A,
		const T *__restrict__ b, const T *__restrict__ x, const bool (&act)[K], double (&acc)[2 * K], Emit emit) {
	Quad q;
	quadAt<D, K>(dom.vec4, sB, l0, nc, q);
	FX<T> fx[K];
#pragma unroll
	for (int k = 0; k < K; ++k) fx[k].x = x;
	T y[K][4], f[K][4];
	quadApply<T, D, K>(dom, A, q, act, fx, y, f);
#pragma unroll
	for (int k = 0; k < K; ++k) {
		if (!act[k]) continue;
		const int64_t o = vk<K>(q.B, q.g, k);
		T bv[4], rv[4];
		ld4(b + o, q.n, q.al, bv);
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			rv[i] = bv[i] - y[k][i];
			acc[2 * k] = fma(double(rv[i]), double(rv[i]), acc[2 * k]);
			acc[2 * k + 1] = fma(double(bv[i]), double(bv[i]), acc[2 * k + 1]);
		}
		emit(k, o, q, rv);
	}
}

// CG phase 1 on a tile: p' = z + beta p, q = A p', (p', q)
template <typename T, int D, int K>
__device__ __forceinline__ void tileCgDirection(const Dom<double, D> &dom, const int32_t *sB, int l0, int nc, const T *__restrict__ A,
		const T *z, const T *pIn, T *pOut, T *qv, const bool (&act)[K], const bool (&rs)[K], const T (&beta)[K], double (&acc)[K]) {
	Quad q;
	quadAt<D, K>(dom.vec4, sB, l0, nc, q);
	FDir<T> fd[K];
#pragma unroll
	for (int k = 0; k < K; ++k) fd[k] = FDir<T>{z, pIn, beta[k], rs[k]};
	T y[K][4], f[K][4];
	quadApply<T, D, K>(dom, A, q, act, fd, y, f);
#pragma unroll
	for (int k = 0; k < K; ++k) {
		if (!act[k]) continue;
		const int64_t o = vk<K>(q.B, q.g, k);
		st4(pOut + o, q.n, q.al, f[k]);
		st4(qv + o, q.n, q.al, y[k]);
#pragma unroll
		for (int i = 0; i < 4; ++i) acc[k] = fma(double(f[k][i]), double(y[k][i]), acc[k]);
	}
}

// CG phase 2 on a tile: x += alpha p, r -= alpha q, (r, r) (xbest = x before, when asked)
template <typename T, int D, int K>
__device__ __forceinline__ void tileCgUpdate(const Dom<double, D> &dom, const int32_t *sB, int l0, int nc, T *r, const T *p,
		const T *qv, T *x, T *xbest, const SysState *sst, double (&acc)[K]) {
	Quad q;
	quadAt<D, K>(dom.vec4, sB, l0, nc, q);
	const int inst = sB[B_INST];
#pragma unroll
	for (int k = 0; k < K; ++k) {
		const SysState &s = sst[inst * K + k];
		if (s.done != RUNNING) continue;
		const T alpha = T(s.alpha);
		const int64_t o = vk<K>(q.B, q.g, k);
		T xv[4], pv[4], rv[4], qq[4];
		ld4(x + o, q.n, q.al, xv);
		ld4(p + o, q.n, q.al, pv);
		ld4(r + o, q.n, q.al, rv);
		ld4(qv + o, q.n, q.al, qq);
		if (s.saveBest && xbest) st4(xbest + o, q.n, q.al, xv);
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			xv[i] = fma(alpha, pv[i], xv[i]);
			rv[i] = fma(-alpha, qq[i], rv[i]);
			acc[k] = fma(double(rv[i]), double(rv[i]), acc[k]);
		}
		st4(x + o, q.n, q.al, xv);
		st4(r + o, q.n, q.al, rv);
	}
}

// BiCGStab phase 1 on a tile: p = r + beta (p - omega v), v = A p, (r0, v)
template <typename T, int D, int K>
__device__ __forceinline__ void tileBicgV(const Dom<double, D> &dom, const int32_t *sB, int l0, int nc, const T *__restrict__ A,
		const T *r, const T *pIn, const T *vIn, T *pOut, T *vOut, const T *r0, const bool (&act)[K], const bool (&rs)[K],
		const T (&beta)[K], const T (&omega)[K], double (&acc)[K]) {
	Quad q;
	quadAt<D, K>(dom.vec4, sB, l0, nc, q);
	FBicgP<T> fp[K];
#pragma unroll
	for (int k = 0; k < K; ++k) fp[k] = FBicgP<T>{r, pIn, vIn, beta[k], omega[k], rs[k]};
	T y[K][4], f[K][4];
	quadApply<T, D, K>(dom, A, q, act, fp, y, f);
#pragma unroll
	for (int k = 0; k < K; ++k) {
		if (!act[k]) continue;
		const int64_t o = vk<K>(q.B, q.g, k);
		st4(pOut + o, q.n, q.al, f[k]);
		st4(vOut + o, q.n, q.al, y[k]);
		T r0v[4];
		ld4(r0 + o, q.n, q.al, r0v);
#pragma unroll
		for (int i = 0; i < 4; ++i) acc[k] = fma(double(r0v[i]), double(y[k][i]), acc[k]);
	}
}

// BiCGStab phase 2 on a tile: s = r - alpha v, t = A s, (t, s), (t, t), (s, s)
template <typename T, int D, int K>
__device__ __forceinline__ void tileBicgT(const Dom<double, D> &dom, const int32_t *sB, int l0, int nc, const T *__restrict__ A,
		const T *r, const T *v, T *t, const bool (&act)[K], const T (&alpha)[K], double (&acc)[3 * K]) {
	Quad q;
	quadAt<D, K>(dom.vec4, sB, l0, nc, q);
	FBicgS<T> fs[K];
#pragma unroll
	for (int k = 0; k < K; ++k) fs[k] = FBicgS<T>{r, v, alpha[k]};
	T y[K][4], f[K][4];
	quadApply<T, D, K>(dom, A, q, act, fs, y, f);
#pragma unroll
	for (int k = 0; k < K; ++k) {
		if (!act[k]) continue;
		const int64_t o = vk<K>(q.B, q.g, k);
		st4(t + o, q.n, q.al, y[k]);
#pragma unroll
		for (int i = 0; i < 4; ++i) {
			acc[3 * k + 0] = fma(double(y[k][i]), double(f[k][i]), acc[3 * k + 0]);
			acc[3 * k + 1] = fma(double(y[k][i]), double(y[k][i]), acc[3 * k + 1]);
			acc[3 * k + 2] = fma(double(f[k][i]), double(f[k][i]), acc[3 * k + 2]);
		}
	}
}

// BiCGStab phase 3 on a tile: x += alpha p + omega s, r = s - omega t, (r0, r), (r, r); after
// a converged half step x += alpha p, r = s
template <typename T, int D, int K>
__device__ __forceinline__ void tileBicgUpdate(const Dom<double, D> &dom, const int32_t *sB, int l0, int nc, T *r, const T *r0,
		const T *p, const T *v, const T *t, T *x, const SysState *sst, double (&acc)[2 * K]) {
	Quad q;
	quadAt<D, K>(dom.vec4, sB, l0, nc, q);
	const int inst = sB[B_INST];
#pragma unroll
	for (int k = 0; k < K; ++k) {
		const SysState &s = sst[inst * K + k];
		if (s.done != RUNNING) continue;
		const T alpha = T(s.alpha), omega = T(s.omega);
		const int64_t o = vk<K>(q.B, q.g, k);
		T rv[4], vv[4], pv[4], xv[4];
		ld4(r + o, q.n, q.al, rv);
		ld4(v + o, q.n, q.al, vv);
		ld4(p + o, q.n, q.al, pv);
		ld4(x + o, q.n, q.al, xv);
		if (s.halfDone) {
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				xv[i] = fma(alpha, pv[i], xv[i]);
				rv[i] = fma(-alpha, vv[i], rv[i]);
			}
		} else {
			T tv[4], r0v[4];
			ld4(t + o, q.n, q.al, tv);
			ld4(r0 + o, q.n, q.al, r0v);
#pragma unroll
			for (int i = 0; i < 4; ++i) {
				const T si = fma(-alpha, vv[i], rv[i]);
				xv[i] = fma(omega, si, fma(alpha, pv[i], xv[i]));
				rv[i] = fma(-omega, tv[i], si);
				acc[2 * k + 0] = fma(double(r0v[i]), double(rv[i]), acc[2 * k + 0]);
				acc[2 * k + 1] = fma(double(rv[i]), double(rv[i]), acc[2 * k + 1]);
			}
		}
		st4(x + o, q.n, q.al, xv);
		st4(r + o, q.n, q.al, rv);
	}
}

// SolverTolerance._resolve_scale (solvers/tolerance.py:241-257)
__device__ __forceinline__ double resolveTol(const phb_tolerance &t, double scale) {
	double tol = 0.0;
	if (t.rtol > 0) tol = t.rtol * scale;
	if (t.atol > 0) tol = fmax(tol, t.atol);
	tol = fmax(tol, t.floor_eps * scale);
	if (!(tol > 0.0)) tol = t.fallback;
	return tol;
}

// rho/beta of a running system from the new (r, z) (the preconditioned CG of
// amg_pcg_solve, solvers/amg.py:1544): the first iteration after a restart takes rho only.
__device__ __forceinline__ void pcgRho(SysState &s, double rz) {
	if (s.restart) s.rho = rz;
	else {
		s.beta = rz / s.rho;
		s.rho = rz;
		if (!fin(s.beta)) s.done = NONFINITE;
	}
	if (!fin(rz)) s.done = NONFINITE;
}

// persistent solvers ---------------------------------------------------------------------
// One cooperative launch runs a whole solve. The CTAs are co-resident (cooperative launch)
// and meet at grid barriers instead of kernel boundaries, so an iteration costs a few
// barrier round trips instead of kernel launches and the vectors stay in L2. Every barrier
// wait is bounded: when it runs out it sets Control::barErr and every CTA leaves the kernel
// (phb_solve_results then reports every system non-finite; inside a refinement the unfinished
// inner solve leaves the outer loop unconverged). Each CTA keeps its own copy of the per-system
// scalars in shared memory and reduces the per-tile partials itself, in the same fixed order
// as every other CTA, so all CTAs take the same decisions without broadcasting them.
constexpr unsigned int BARRIER_SPIN_LIMIT = 1u << 24;
constexpr unsigned int BARRIER_ERR_POLL = 1023; // spins between reads of Control::barErr

// Sense-reversing arrival counter: CTA 0 adds 2^31 - (gridDim.x - 1), every other CTA adds 1,
// so the counter's top bit flips exactly when the last CTA of a generation arrives and the
// low bits return to where they were (no reset, no second atomic). The arrival is a release
// and the poll an acquire at GPU scope; with the CTA barriers on both sides that orders every
// thread's writes before the barrier against every thread's reads after it. A CTA that has
// seen the flip does not read barErr: a CTA that gave up at this barrier had arrived at it
// (arrival comes before the wait), so the flip proves the phase complete, and the next
// barrier, where that CTA never arrives, ends everyone else's wait through barErr.
__device__ __forceinline__ unsigned int barrierArrive(unsigned int *count, unsigned int add) {
	unsigned int old;
	asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(count), "r"(add) : "memory");
	return old;
}

__device__ __forceinline__ unsigned int barrierPoll(const unsigned int *count) {
	unsigned int v;
	asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
	return v;
}

__device__ __forceinline__ bool gridBarrier(Control *ctrl, unsigned int spinLimit = BARRIER_SPIN_LIMIT) {
	__shared__ int sOk;
	__syncthreads();
	if (threadIdx.x == 0) {
		const unsigned int add = blockIdx.x == 0 ? 0x80000000u - (gridDim.x - 1) : 1u;
		const unsigned int old = barrierArrive(&ctrl->barCount, add);
		int ok = 1;
		for (unsigned int spins = 1; ((barrierPoll(&ctrl->barCount) ^ old) & 0x80000000u) == 0; ++spins) {
			if ((spins & BARRIER_ERR_POLL) == 0 && (spins > spinLimit || *(volatile int *)&ctrl->barErr)) {
				atomicExch(&ctrl->barErr, 1);
				ok = 0;
				break;
			}
			__nanosleep(32);
		}
		sOk = ok;
	}
	__syncthreads();
	return sOk;
}

// A persistent kernel runs one CTA per SM made of worker groups of PHB_TILE threads, each with its own
// tiles (a grid of CTAs of PHB_TILE threads, several to an SM, would do the same work but its
// barrier would wait for three times as many arrivals: 2.0 against 1.4 us at 432 and 148 CTAs, and
// 2.6 against 1.8 with a reduction behind it). Microseconds per iteration, before and after: CG on 432
// float64 tiles 15.4 -> 14.9, on 3240 tiles 91 -> 88.5; preconditioned CG on 3 x 64 x 48 x 48 cells 44
// -> 42, on 64 channels of 2D 91 -> 77; BiCGStab on 2 x 37 x 45 x 41 to 128^3 cells 65 -> 60, 223 -> 211.
struct Worker {
	int lt;    // thread of the group
	int id;    // group of the CTA
	int first; // the group's first item; the others are `step` apart
	int step;
	__device__ __forceinline__ Worker()
		: lt(int(threadIdx.x) & (PHB_TILE - 1)), id(int(threadIdx.x) / PHB_TILE), first(int(blockIdx.x) + id * int(gridDim.x)),
		  step(int(gridDim.x) * (int(blockDim.x) / PHB_TILE)) {}
	// number of the group's items of n
	__device__ __forceinline__ int count(int n) const { return n > first ? (n - 1 - first) / step + 1 : 0; }
	// barrier of the group's threads
	__device__ __forceinline__ void sync() const { asm volatile("barrier.sync %0, %1;" ::"r"(id + 1), "n"(PHB_TILE) : "memory"); }
};

// Sums of NV values over each tile (item) that a group visits in a phase, without a barrier per
// tile: the warps leave their sums in shared memory and stream on, and one barrier for TILE_SUMS
// tiles lets a thread per value add the warps up, in warp order (the order of storePartials). A barrier
// per tile made the warps of a CTA wait for the slowest load of every tile: on grids of several
// tiles per CTA a quarter of the stall cycles.
constexpr int TILE_SUMS = 8;
template <int NV>
struct TileSums {
	const Worker &wk;
	double (*ws)[NV][NWARPS]; // [TILE_SUMS], shared memory of the group
	double *dst;              // the phase's partials, [item][NV]
	int k;                    // items visited so far
	int last;                 // index of the group's last item where they are visited backwards, else -1
	__device__ __forceinline__ void add(double (&v)[NV]) {
		const int lane = wk.lt & 31, warp = wk.lt >> 5;
#pragma unroll
		for (int q = 0; q < NV; ++q) {
			const double s = warpSum(v[q]);
			if (lane == 0) ws[k % TILE_SUMS][q][warp] = s;
		}
	}
	// after every item, whether it added its sums or was left out (all threads)
	__device__ __forceinline__ void next() {
		if (++k % TILE_SUMS == 0) flush(TILE_SUMS);
	}
	// after the last item
	__device__ __forceinline__ void finish() {
		if (k % TILE_SUMS) flush(k % TILE_SUMS);
	}
	__device__ __forceinline__ void flush(int n) {
		wk.sync();
		for (int i = wk.lt; i < n * NV; i += PHB_TILE) {
			const int slot = i / NV, q = i - slot * NV;
			double s = 0;
#pragma unroll
			for (int w = 0; w < NWARPS; ++w) s += ws[slot][q][w];
			const int item = k - n + slot;
			dst[(size_t)(wk.first + (last < 0 ? item : last - item) * wk.step) * NV + q] = s;
		}
		wk.sync();
	}
};

// block tables -----------------------------------------------------------------------------
// What the phases of a persistent kernel need of one block of one level, kept in shared memory for
// the whole solve. The cell across a face that is not fixed is an affine function of the position
// (periodic: the other end of the row; connected: phiPICT's axis mapping):
// map[f] = c0 + cx x + cy y + cz z.
struct __align__(16) BlockTab {
	int nx, ny, nz, off;
	int inst, instOff, instN;
	unsigned int bits; // bit f: face f is not fixed; bit 8: rows of four may be loaded as vectors here and across every open face
	int4 map[6];
	__device__ __forceinline__ int cells() const { return nx * ny * nz; }
	__device__ __forceinline__ bool open(int f) const { return (bits >> f) & 1; }
	__device__ __forceinline__ bool rows4() const { return (bits >> 8) & 1; }
};
static_assert(sizeof(BlockTab) == 128, "BlockTab layout");
constexpr size_t TAB_SMEM_MAX = 48 * 1024; // tables kept in shared memory up to this size, else in global memory

template <int D>
__device__ __forceinline__ void buildBlockTab(const int32_t *blocks, int b, BlockTab &o) {
	const int32_t *B = blocks + b * PHB_BREC;
	const int n[3] = {B[B_NX], B[B_NY], D > 2 ? B[B_NZ] : 1};
	o.nx = n[0]; o.ny = n[1]; o.nz = n[2];
	o.off = B[B_CELLOFF];
	o.inst = B[B_INST];
	o.instOff = B[B_INSTOFF];
	o.instN = B[B_INSTN];
	unsigned int open = 0;
	bool al = ((n[0] | o.off) & 3) == 0;
	for (int f = 0; f < 6; ++f) {
		int4 m = make_int4(0, 0, 0, 0);
		if (f < 2 * D && fType(B, f) != FT_FIXED) {
			open |= 1u << f;
			Dom<float, D> d;
			d.blocks = blocks;
			// the map from its values at the corner (0, 0, 0) of the face and one step along each
			// tangential axis (the position along the face's own axis does not matter)
			int v[4];
			for (int k = 0; k < 4; ++k) {
				Cell c;
				c.B = B;
				c.p[0] = c.p[1] = c.p[2] = 0;
				c.p[f >> 1] = (f & 1) ? n[f >> 1] - 1 : 0;
				if (k && k - 1 != (f >> 1) && n[k - 1] > 1) c.p[k - 1] = 1;
				c.g = 0; c.mi = 0;
				v[k] = (int)neighbor<float, D>(d, c, f).g;
			}
			m = make_int4(v[0], v[1] - v[0], v[2] - v[0], v[3] - v[0]);
			if (f >= 2) al = al && m.y == 1 && ((m.x | m.z | m.w) & 3) == 0;
		}
		o.map[f] = m;
	}
	o.bits = open | (al ? 256u : 0u);
}
__device__ __forceinline__ int tabMap(const int4 &m, int x, int y, int z) { return m.x + m.y * x + m.z * y + m.w * z; }

// Indices of the neighbours of cell g (x, y, z), or of four cells of an aligned row from g on
// (W = 4: the +x neighbour is that of the last one, the y and z neighbours start rows of four).
// A face without neighbour gets g itself and no bit in `has`: every load is issued without a
// branch, and what it brings is left out of the sum.
template <int D, int W>
__device__ __forceinline__ unsigned int tabNeighbors(const BlockTab &B, int g, int x, int y, int z, int (&o)[2 * D]) {
	unsigned int has = (1u << (2 * D)) - 1;
	const int sy = B.nx, sz = B.nx * B.ny;
	o[0] = g - 1; o[1] = g + W; o[2] = g - sy; o[3] = g + sy;
	if constexpr (D > 2) { o[4] = g - sz; o[5] = g + sz; }
	bool end[2 * D];
	end[0] = x == 0; end[1] = x + W == B.nx; end[2] = y == 0; end[3] = y + 1 == B.ny;
	if constexpr (D > 2) { end[4] = z == 0; end[5] = z + 1 == B.nz; }
#pragma unroll
	for (int f = 0; f < 2 * D; ++f)
		if (end[f]) {
			if (B.open(f)) {
				o[f] = tabMap(B.map[f], x, y, z);
			} else {
				o[f] = g;
				has &= ~(1u << f);
			}
		}
	return has;
}

// Every CTA reduces the partials of every running system (K right-hand sides per instance, NQ
// values each, [item][K][NQ]; items range(inst) = first, count) and updates its own copy of the
// states: all the warps on few systems, a warp per system (four in flight) on many, each in the
// order of finalizeSystems. With INSTQ >= 0 the last argument of fn is quantity INSTQ summed over
// the instance's right-hand sides. Returns the systems still running.
template <int K, int NQ, int INSTQ, typename Range, typename Fn>
__device__ __forceinline__ int reduceSystems(int ninst, const double *pp, SysState *sst, Range range, Fn fn) {
	constexpr int NV = NQ + (INSTQ >= 0 ? 1 : 0);
	__shared__ int running;
	__shared__ double gsm[NWARPS][NV];
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
	const int nsys = ninst * K;
	if (threadIdx.x == 0) running = 0;
	auto load = [&](int item, int k, double (&a)[NV]) {
		const double *p = pp + (size_t)item * K * NQ;
#pragma unroll
		for (int q = 0; q < NQ; ++q) a[q] += __ldcg(p + k * NQ + q);
		if constexpr (INSTQ >= 0) {
#pragma unroll
			for (int kk = 0; kk < K; ++kk) a[NQ] += __ldcg(p + kk * NQ + INSTQ);
		}
	};
	if (nsys >= NWARPS) {
		constexpr int U = K == 1 ? 4 : 2;
		__syncthreads();
		int mine = 0;
		for (int s0 = warp; s0 < nsys; s0 += U * warps) {
			double a0[U][NV];
			bool act[U];
#pragma unroll
			for (int u = 0; u < U; ++u) {
				const int s = s0 + u * warps;
				act[u] = s < nsys && sst[s].done == RUNNING;
				double a1[NV];
#pragma unroll
				for (int q = 0; q < NV; ++q) a0[u][q] = a1[q] = 0;
				if (act[u]) {
					const int2 rg = range(s / K);
					int t = lane;
					for (; t + 32 < rg.y; t += 64) { load(rg.x + t, s % K, a0[u]); load(rg.x + t + 32, s % K, a1); }
					if (t < rg.y) load(rg.x + t, s % K, a0[u]);
				}
#pragma unroll
				for (int q = 0; q < NV; ++q) a0[u][q] += a1[q];
			}
#pragma unroll
			for (int u = 0; u < U; ++u) {
#pragma unroll
				for (int q = 0; q < NV; ++q) a0[u][q] = warpSum(a0[u][q]);
				if (act[u] && lane == u) fn(sst[s0 + u * warps], (s0 + u * warps) / K, a0[u], a0[u][NV - 1]);
			}
			if (lane < U) {
				const int s = s0 + lane * warps;
				if (s < nsys && sst[s].done == RUNNING) ++mine;
			}
		}
		if (mine) atomicAdd(&running, mine);
		__syncthreads();
		return running;
	}
	int G = NWARPS;
	while (G > 1 && G * nsys > NWARPS) G >>= 1;
	const int s = warp / G, wg = warp - s * G; // the first NWARPS warps
	const bool act = warp < NWARPS && s < nsys && sst[s].done == RUNNING;
	double a0[NV], a1[NV];
#pragma unroll
	for (int q = 0; q < NV; ++q) a0[q] = a1[q] = 0;
	if (act) {
		const int2 rg = range(s / K);
		const int stride = G * 32;
		int t = wg * 32 + lane;
		if constexpr (INSTQ >= 0) {
			for (; t + stride < rg.y; t += 2 * stride) { load(rg.x + t, s % K, a0); load(rg.x + t + stride, s % K, a1); }
			if (t < rg.y) load(rg.x + t, s % K, a0);
		} else {
			// 2 P items in flight (predicated, not clamped: a clamped load past the end makes every warp
			// of the grid wait its turn at one address). Two in flight made this
			// 3.2 us of every phase on 3240 tiles, 4.8 us on 3567 tiles of six systems.
			constexpr int P = 4;
			for (; t < rg.y; t += 2 * P * stride) {
				double v[2 * P][NQ];
#pragma unroll
				for (int i = 0; i < 2 * P; ++i) {
					const double *p = pp + ((size_t)(rg.x + t + i * stride) * K + s % K) * NQ;
#pragma unroll
					for (int q = 0; q < NQ; ++q) v[i][q] = t + i * stride < rg.y ? __ldcg(p + q) : 0.0;
				}
#pragma unroll
				for (int i = 0; i < 2 * P; ++i) {
					double(&a)[NV] = i & 1 ? a1 : a0;
#pragma unroll
					for (int q = 0; q < NQ; ++q)
						if (t + i * stride < rg.y) a[q] += v[i][q];
				}
			}
		}
	}
#pragma unroll
	for (int q = 0; q < NV; ++q) {
		const double v = warpSum(a0[q] + a1[q]);
		if (lane == 0 && warp < NWARPS) gsm[warp][q] = v;
	}
	__syncthreads();
	if (warp < NWARPS && s < nsys && wg == 0 && lane == 0) {
		if (act) {
			double red[NV];
#pragma unroll
			for (int q = 0; q < NV; ++q) {
				double v = 0;
				for (int w = 0; w < G; ++w) v += gsm[warp + w][q];
				red[q] = v;
			}
			fn(sst[s], s / K, red, red[NV - 1]);
		}
		if (sst[s].done == RUNNING) atomicAdd(&running, 1);
	}
	__syncthreads();
	return running;
}

// The reference stop rule of the first residual (kResidual) applied to a CTA state copy.
template <int K, bool BICG, bool STOPSTART>
__device__ __forceinline__ void residualDecision(const Dom<double, 3> *, SysState &s, double ns, const double *red, double bb,
		const phb_tolerance &tol) {
	if (tol.mode == 1) s.tol = resolveTol(tol, sqrt(bb / double(K)) * ns);
	const double crit = sqrt(red[0]) * ns;
	s.rho = red[0];
	s.restart = 1;
	s.crit = crit;
	if (!fin(crit)) { s.done = NONFINITE; s.usedIt = 0; }
	else if ((BICG || STOPSTART) ? crit < s.tol : crit == 0.0) { s.done = CONVERGED; s.usedIt = BICG ? -1 : 0; }
}

// host side --------------------------------------------------------------------------------
inline size_t align256(size_t v) { return (v + 255) & ~size_t(255); }

// Dom::vec4 of a launch: every operand on a 16-byte boundary and a cell count that keeps the
// stencil's slot rows aligned
inline int vec4Ok(const phb_domain *dom, std::initializer_list<const void *> ptrs) {
	if (dom->ncells % 4) return 0;
	for (const void *p : ptrs)
		if (p && ((uintptr_t)p & 15)) return 0;
	return 1;
}

struct Layout {
	size_t off[12];
	size_t total;
};

// CG: r q p0 p1 xbest, and the second residual of the preconditioned CG (float, one right-hand
// side); BiCG: r r0 p0 p1 v0 v1 t
inline int vecCount(int kind, bool pcg) { return kind == 0 ? (pcg ? 6 : 5) : 7; }

// partials per tile of the preconditioned CG: its finest restriction has at most 16 items per
// coarse tile, and no level has more tiles than the finest
constexpr int PCG_PARTIALS = 16;

// plain: the layout of a solve that is never preconditioned
inline Layout solveLayout(const phb_domain *dom, int kind, int vecBytes, int nrhs, bool plain = false) {
	Layout L;
	size_t o = 0;
	const bool pcg = !plain && kind == 0 && vecBytes == 4 && nrhs == 1;
	const size_t vb = align256((size_t)dom->ncells * nrhs * vecBytes);
	for (int i = 0; i < vecCount(kind, pcg); ++i) { L.off[i] = o; o += vb; }
	L.off[9] = o; // block tables (BlockTab), of every multigrid level for a preconditioned solve
	if (!plain) o += align256((size_t)dom->nblocks * (pcg ? PHB_AMG_MAX_LEVELS : 1) * sizeof(BlockTab));
	L.off[10] = o; // partials: two halves of up to 3 values per tile and right-hand side
	o += align256((size_t)dom->ntiles * (pcg ? PCG_PARTIALS : nrhs * 3) * 2 * sizeof(double));
	L.total = o;
	return L;
}

struct StateLayout { size_t ctrl, st, ctrl2, st2, total; };
inline StateLayout stateLayout(const phb_domain *dom, int nrhs) {
	StateLayout L;
	const size_t nsys = (size_t)dom->ninst * nrhs;
	L.ctrl = 0;
	L.st = 256;
	L.ctrl2 = align256(L.st + nsys * sizeof(SysState));
	L.st2 = L.ctrl2 + 256;
	L.total = align256(L.st2 + nsys * sizeof(SysState));
	return L;
}

inline int numSMs() {
	static int cache[64] = {0};
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
	if (!cache[dev]) {
		int v = 0;
		if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 148;
		cache[dev] = v;
	}
	return cache[dev];
}

// Initial state of system s: its tolerance from the options, or (fromInner) the one that the
// refinement residual left in SysState::innerTol.
__device__ __forceinline__ SysState initialState(const phb_tolerance &tol, int s, double innerTol, int fromInner, int maxit) {
	SysState z;
	memset(&z, 0, sizeof(z));
	z.tol = fromInner ? innerTol : tol.mode == 0 ? tol.atol : tol.mode == 2 ? tol.values[s] : NAN; // NAN: resolved from the right-hand side
	z.innerTol = z.tol;
	z.maxit = maxit;
	z.best = INFINITY;
	z.restart = 1;
	z.bestIt = -1;
	return z;
}

// Lets launches of `kern` ask for as much dynamic shared memory as the device has (always the same
// limit, so that threads launching with different sizes do not undo each other's).
inline cudaError_t allowSmem(const void *kern) {
	cudaFuncAttributes at;
	int dev = 0, optin = 0;
	cudaError_t e = cudaFuncGetAttributes(&at, kern);
	if (e == cudaSuccess) e = cudaGetDevice(&dev);
	if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
	if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)at.sharedSizeBytes);
	return e;
}

// The launch of a persistent kernel: worker groups per CTA (at most `most`, or the caller's ctas_per_sm;
// fewer where the items would not give every group of every SM one) and CTAs.
inline void persistentGrid(int items, int most, int ctasPerSm, int &groups, int &ctas) {
	const int sms = numSMs();
	groups = std::min(most, ctasPerSm > 0 ? ctasPerSm : most);
	groups = std::max(1, std::min(groups, (items + sms - 1) / sms));
	ctas = std::max(1, std::min(sms, (items + groups - 1) / groups));
}

// kInit launched on `s`: the initial state of the nsys systems of a solve (krylov.cu)
int launchInit(SysState *st, int nsys, const phb_tolerance &tol, int fromInner, int maxit, Control *ctrl, cudaStream_t s);

// The CG of small instances as one cluster per instance (cluster_cg.cu); *taken: whether it applies.
template <typename T, int D>
int launchClusterCg(const phb_domain *dom, const phb_solve *sv, cudaStream_t s, bool stopStart, int fromInner, bool *taken);

// A persistent preconditioned CG recorded on `s` (pcg.cu).
template <int D>
int launchPcg(const phb_domain *dom, const phb_solve *sv, cudaStream_t s, bool stopStart, int fromInner);

// A persistent solve recorded on `s` (persistent.cu).
template <typename T, int D, int K>
int launchPersistent(const phb_domain *dom, const phb_solve *sv, cudaStream_t s, bool stopStart, int fromInner);

} // namespace phb
