// Multigrid-preconditioned CG of the pressure and potential systems as one cooperative kernel
// (float32, one right-hand side per instance): the CG of amg_pcg_solve (phiPICT
// solvers/amg.py:1544) with the V-cycle of phb_amg.cuh, whose phases meet at grid barriers.
//
// What bounds it: on grids that fit L2 every phase costs a barrier (1.2 to 1.6 us) plus its
// chain of dependent L2 round trips (0.3 to 0.5 us each); on larger grids the bytes of the four
// finest-level passes. So the phases are as few as the algorithm allows and their chains short:
//   A   x += alpha p, r' = r - alpha q evaluated at the stencil points, t = r' - A omega D^-1 r'
//       and its restriction (the update and the finest restriction share one pass: r and q are
//       read at the neighbours instead of being met at one more barrier; r is double-buffered)
//   R_l t_l = b_l - A_l omega D^-1 b_l and its restriction, coarser levels
//   T   the dense operator of the last level
//   P_l z = omega D^-1 b + P e + omega D^-1 (t - A P e): with t kept from the way down, the way up
//       reads the stencil and a few coarse values instead of b, omega/D and e at every neighbour
//   D   p' = z + beta p, q = A p', (p', q)
// Block records of all levels and the CTA's work items stay in shared memory for the whole
// solve (a phase otherwise starts with three dependent reads: tile, block record, data).
// Finished instances of a batch are skipped by every phase. All neighbour indices of a cell group
// are formed before its loads, and the loads are issued without a branch between them: a face
// resolved by a branch of its own costs its own round trip to L2, which made most of an iteration
// of the form before this one. Microseconds per iteration, before and after (B200):
//   3 blocks 64x48x48 (442,368 cells, rows of four)          67 -> 40
//   2 blocks 37x45x41 (136,530 cells, odd rows)               72 -> 37
//   128^3 (2.1 M cells)                                      213 -> 98
//   64 2D instances of 32^2 to 256^2 (1.2 M cells)           170 -> 77
//   6 3D instances of 32^3 to 112^3 (3.6 M cells, odd rows)  430 -> 226
#include "phb_krylov.cuh"

namespace phb {

constexpr int PCG_ITEMS = 8; // work items per phase that a group keeps in shared memory
constexpr int PCG_GROUPS = 3; // 768 threads of 80 registers
// Four fine cells per lane in the restriction from this many fine cells on (below, two: the
// coarse levels have too few rows to fill the chip)
constexpr int64_t PCG_WIDE_MIN = 1 << 17;

// Below this many tiles (two per SM) the finest prolongation and direction take quarter tiles
constexpr int PCG_QUARTER_TILES = 296;

// the same tables in global memory, for domains with too many blocks for shared memory
template <int D>
__global__ void kPcgTabs(AmgView<D> mg, BlockTab *out) {
	const int nblk = mg.lv[0].nblocks;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nblk * mg.nlevels; i += gridDim.x * blockDim.x)
		buildBlockTab<D>(mg.lv[i / nblk].blocks, i % nblk, out[i]);
}
template <int D>
struct PcgArgs {
	Dom<double, D> dom;
	AmgView<D> mg;
	const float *A, *b;
	float *x, *r0, *r1, *p0, *p1, *q, *xbest;
	SysState *st;
	double *partial;
	int64_t half; // doubles per half of the partials
	Control *ctrl;
	phb_tolerance tol;
	const BlockTab *blocks; // tables in global memory, or null: built in shared memory
	int returnBest, maxit, stopStart, quarter;
	unsigned int vec; // bit l: the operands of level l start on 16-byte boundaries
};

// lanes per aggregate in the restriction: one per fine row
template <int D> struct PcgRows { static constexpr int R = D > 2 ? 4 : 2; };
// coarse cells of one restriction item, items per coarse tile
template <int D, int V> struct PcgItem {
	static constexpr int CELLS = PHB_TILE / PcgRows<D>::R * (V / 2);
	static constexpr int PER = PHB_TILE_CELLS / CELLS;
};

__device__ __forceinline__ void ld4f(const float *p, float (&v)[4]) {
	const float4 f = *reinterpret_cast<const float4 *>(p);
	v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
}
__device__ __forceinline__ void st4f(float *p, const float (&v)[4]) { *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]); }

// the finest field of the restriction: r' = r - alpha q (UPD) or r, and s = omega/D r'
template <bool UPD>
struct PcgFine {
	const float *r, *q, *wd;
	float alpha;
	__device__ __forceinline__ void at(int o, float &rv, float &s) const {
		rv = UPD ? fmaf(-alpha, q[o], r[o]) : r[o];
		s = rv * __ldg(wd + o);
	}
	__device__ __forceinline__ void at4(int o, float (&rv)[4], float (&s)[4]) const {
		float w[4];
		ld4f(r + o, rv);
		if constexpr (UPD) {
			float qq[4];
			ld4f(q + o, qq);
#pragma unroll
			for (int i = 0; i < 4; ++i) rv[i] = fmaf(-alpha, qq[i], rv[i]);
		}
		ld4f(wd + o, w);
#pragma unroll
		for (int i = 0; i < 4; ++i) s[i] = rv[i] * w[i];
	}
	// V cells o, o + st, ... (index o again past cnt), as vectors on aligned rows (V = 4)
	template <int V>
	__device__ __forceinline__ void row(int o, int st, int cnt, float (&rv)[V], float (&s)[V]) const {
		if constexpr (V == 4) {
			at4(o, rv, s);
		} else {
#pragma unroll
			for (int i = 0; i < V; ++i) at(i < cnt ? o + i * st : o, rv[i], s[i]);
		}
	}
};
template <int V>
__device__ __forceinline__ void ldRow(const float *p, int cnt, float (&v)[V]) {
	if constexpr (V == 4) {
		ld4f(p, v);
	} else {
#pragma unroll
		for (int i = 0; i < V; ++i) v[i] = p[i < cnt ? i : 0];
	}
}
template <int V>
__device__ __forceinline__ void stRow(float *p, int cnt, const float (&v)[V]) {
	if constexpr (V == 4) {
		st4f(p, v);
	} else {
#pragma unroll
		for (int i = 0; i < V; ++i)
			if (i < cnt) p[i] = v[i];
	}
}

// One restriction item: PcgItem::CELLS coarse cells from `first` of block B -> CB. A lane takes V
// consecutive fine cells of one fine row of its V/2 aggregates, the R lanes of an aggregate its
// rows; rows of the same aggregate come by shuffle, only the rows outside it are loaded again.
// t = r' - A omega D^-1 r' is stored for the way up, the aggregate sums (x pairs, then y, then z:
// a fixed order) go to bc. UPD: also x += alpha p, r' stored, (r', r') returned. All loads are
// issued before the first product (a face that is resolved by a branch of its own costs its own
// round trip to L2). V = 4: rows of four as vectors (BlockTab::rows4); V = 2: any rows.
template <int D, int V, bool UPD>
__device__ __forceinline__ double pcgRestrictItem(const BlockTab &B, const BlockTab &CB, int first, int64_t N,
		const float *__restrict__ A, const PcgFine<UPD> f, float *__restrict__ t, float *__restrict__ bc,
		float *__restrict__ rOut, float *__restrict__ x, const float *__restrict__ p, float *xbest) {
	constexpr int R = PcgRows<D>::R, H = V / 2;
	const int lt = int(threadIdx.x) & (PHB_TILE - 1);
	const int grp = lt / R, rr = lt & (R - 1);
	const int fnx = B.nx, fny = B.ny, fnz = B.nz;
	const int cnx = CB.nx, cny = CB.ny;
	const bool kx = cnx < fnx, ky = cny < fny, kz = D > 2 && CB.nz < fnz;
	const int lc = first + grp * H;
	const bool valid = lc < CB.cells();
	const int crow = lc / cnx;
	const int cx = lc - crow * cnx;
	const int cz = D > 2 ? crow / cny : 0;
	const int cy = crow - cz * cny;
	const int oy = rr & 1, oz = rr >> 1;
	const int y = ky ? 2 * cy + oy : cy, z = kz ? 2 * cz + oz : cz;
	const bool rowOk = valid && (ky ? y < fny : oy == 0) && (D < 3 || (kz ? z < fnz : oz == 0));
	const int x0 = kx ? 2 * cx : cx;
	const int cnt = !rowOk ? 0 : V == 4 ? 4 : kx ? min(V, fnx - x0) : 1;
	float s[V], rv[V], yo[V], zo[V], tv[V];
#pragma unroll
	for (int i = 0; i < V; ++i) s[i] = rv[i] = tv[i] = 0.f;
	const int sy = fnx, sz = fnx * fny;
	const int g = B.off + x0 + sy * y + sz * z;
	if (cnt > 0) {
		f.row(g, 1, cnt, rv, s);
		if (V == 2 && cnt == 1) rv[1] = s[1] = 0.f;
	}
#pragma unroll
	for (int i = 0; i < V; ++i) {
		yo[i] = __shfl_xor_sync(0xffffffffu, s[i], 1);
		zo[i] = D > 2 ? __shfl_xor_sync(0xffffffffu, s[i], 2) : 0.f;
	}
	double acc = 0;
	if (cnt > 0) {
		// x neighbours beside the lane's cells; of the y and z neighbours one is outside the
		// aggregate (the lower for the aggregate's lower row), the other by shuffle unless the
		// aggregate is one row thin there
		int ow = g - 1, oe = g + cnt;
		bool hw = true, he = true;
		if (x0 == 0) { hw = B.open(0); ow = hw ? tabMap(B.map[0], x0, y, z) : g; }
		if (x0 + cnt == fnx) { he = B.open(1); oe = he ? tabMap(B.map[1], x0 + cnt - 1, y, z) : g; }
		auto outside = [&](int fc, bool atEnd, int off, int &o, int &st, bool &has) {
			o = g + off;
			st = 1;
			has = true;
			if (atEnd) {
				has = B.open(fc);
				o = has ? tabMap(B.map[fc], x0, y, z) : g;
				st = has ? B.map[fc].y : 1;
			}
		};
		int o1, st1, o2 = g, st2 = 1;
		bool h1, h2 = false;
		if (ky && oy) outside(3, y + 1 == fny, sy, o1, st1, h1);
		else outside(2, y == 0, -sy, o1, st1, h1);
		if constexpr (D > 2) {
			if (kz && oz) outside(5, z + 1 == fnz, sz, o2, st2, h2);
			else outside(4, z == 0, -sz, o2, st2, h2);
		}
		float r1[V], s1[V], r2[V], s2[V], w, e, dump;
		f.row(o1, st1, cnt, r1, s1);
		f.at(ow, dump, w);
		f.at(oe, dump, e);
		if constexpr (D > 2) f.row(o2, st2, cnt, r2, s2);
		float a[2 * D + 1][V];
#pragma unroll
		for (int k = 0; k < 2 * D + 1; ++k) ldRow<V>(A + k * N + g, cnt, a[k]);
		float xv[V], pv[V];
		if constexpr (UPD) {
			ldRow<V>(x + g, cnt, xv);
			ldRow<V>(p + g, cnt, pv);
		}
		// the inner y and z neighbours
		const bool inY = ky && (oy || y + 1 < fny), inZ = D > 2 && kz && (oz || z + 1 < fnz);
		bool h1b = inY, h2b = inZ;
		if (!inY) {
			// one row thin: the upper neighbour is across the block's end
			int o, st;
			outside(3, true, 0, o, st, h1b);
			f.row(o, st, cnt, r1, yo);
		}
		if constexpr (D > 2) {
			if (!inZ) {
				int o, st;
				outside(5, true, 0, o, st, h2b);
				f.row(o, st, cnt, r2, zo);
			}
		}
		if (!h1) for (int i = 0; i < V; ++i) s1[i] = 0.f;
		if (!h1b) for (int i = 0; i < V; ++i) yo[i] = 0.f;
		if (!hw) w = 0.f;
		if (!he) e = 0.f;
		const bool up = ky && oy; // the outside row is the upper one
#pragma unroll
		for (int i = 0; i < V; ++i) {
			float yv = a[0][i] * s[i];
			yv = fmaf(a[1][i], i ? s[i ? i - 1 : 0] : w, yv);
			yv = fmaf(a[2][i], i + 1 < cnt && i + 1 < V ? s[i + 1 < V ? i + 1 : i] : e, yv);
			yv = fmaf(a[3][i], up ? yo[i] : s1[i], yv);
			yv = fmaf(a[4][i], up ? s1[i] : yo[i], yv);
			if constexpr (D > 2) {
				const bool upz = kz && oz;
				const float so = h2 ? s2[i] : 0.f, si = h2b ? zo[i] : 0.f;
				yv = fmaf(a[5][i], upz ? si : so, yv);
				yv = fmaf(a[6][i], upz ? so : si, yv);
			}
			tv[i] = i < cnt ? rv[i] - yv : 0.f;
		}
		stRow<V>(t + g, cnt, tv);
		if constexpr (UPD) {
			if (xbest) stRow<V>(xbest + g, cnt, xv);
#pragma unroll
			for (int i = 0; i < V; ++i) {
				xv[i] = fmaf(f.alpha, pv[i], xv[i]);
				acc = fma(double(rv[i]), double(rv[i]), acc); // rv is 0 past cnt
			}
			stRow<V>(x + g, cnt, xv);
			stRow<V>(rOut + g, cnt, rv);
		}
	}
#pragma unroll
	for (int h = 0; h < H; ++h) {
		float v = kx ? tv[2 * h] + tv[2 * h + 1] : tv[h];
		v += __shfl_xor_sync(0xffffffffu, v, 1);
		if (D > 2) v += __shfl_xor_sync(0xffffffffu, v, 2);
		if (valid && rr == 0) bc[CB.off + lc + h] = v;
	}
	return acc;
}

// z at one cell of a level: s + e + omega/D (t - A P e) with s = omega/D b, e the coarse correction
// of its aggregate
template <int D>
__device__ __forceinline__ float pcgProlongCell(const BlockTab &B, const BlockTab &CB, int g, int x, int y, int z, int64_t N,
		const float *__restrict__ A, const float *__restrict__ wd, float bv, float tv, const float *__restrict__ e) {
	const int kx = CB.nx < B.nx, ky = CB.ny < B.ny, kz = D > 2 ? CB.nz < B.nz : 0;
	const int cx = x >> kx, cy = y >> ky, cz = z >> kz;
	const int ce = CB.off + cx + CB.nx * (cy + CB.ny * cz);
	// neighbours of the same aggregate share its coarse cell
	int o[2 * D];
	unsigned int has = (1u << (2 * D)) - 1;
	const int sy = CB.nx, sz = CB.nx * CB.ny;
	o[0] = kx && (x & 1) ? ce : ce - 1;
	o[1] = kx && !(x & 1) ? ce : ce + 1;
	o[2] = ky && (y & 1) ? ce : ce - sy;
	o[3] = ky && !(y & 1) ? ce : ce + sy;
	if constexpr (D > 2) {
		o[4] = kz && (z & 1) ? ce : ce - sz;
		o[5] = kz && !(z & 1) ? ce : ce + sz;
	}
	bool end[2 * D];
	end[0] = x == 0; end[1] = x + 1 == B.nx; end[2] = y == 0; end[3] = y + 1 == B.ny;
	if constexpr (D > 2) { end[4] = z == 0; end[5] = z + 1 == B.nz; }
#pragma unroll
	for (int f = 0; f < 2 * D; ++f)
		if (end[f]) {
			if (B.open(f)) {
				o[f] = tabMap(CB.map[f], cx, cy, cz);
			} else {
				o[f] = ce;
				has &= ~(1u << f);
			}
		}
	float a[2 * D + 1], ev[2 * D];
#pragma unroll
	for (int f = 0; f < 2 * D; ++f) ev[f] = e[o[f]];
	const float e0 = e[ce];
#pragma unroll
	for (int k = 0; k < 2 * D + 1; ++k) a[k] = __ldg(A + k * N + g);
	const float w = __ldg(wd + g);
	float yv = a[0] * e0;
#pragma unroll
	for (int f = 0; f < 2 * D; ++f) yv = fmaf(a[f + 1], (has >> f) & 1 ? ev[f] : 0.f, yv);
	return fmaf(w, tv - yv, fmaf(bv, w, e0));
}

// The same for four cells of an aligned row (its x size is a multiple of four, so it is halved)
template <int D>
__device__ __forceinline__ void pcgProlongQuad(const BlockTab &B, const BlockTab &CB, int g, int x, int y, int z, int64_t N,
		const float *__restrict__ A, const float *__restrict__ wd, const float (&bv)[4], const float (&tv)[4],
		const float *__restrict__ e, float (&out)[4]) {
	const int ky = CB.ny < B.ny, kz = D > 2 ? CB.nz < B.nz : 0;
	const int cx = x >> 1, cy = y >> ky, cz = z >> kz;
	const int ce = CB.off + cx + CB.nx * (cy + CB.ny * cz);
	const int sy = CB.nx, sz = CB.nx * CB.ny;
	// first and second coarse cell of the row across each y and z face, first and last of x
	int o[2 * D], st[2 * D];
	unsigned int has = (1u << (2 * D)) - 1;
	o[0] = ce - 1; o[1] = ce + 2;
	o[2] = ky && (y & 1) ? ce : ce - sy;
	o[3] = ky && !(y & 1) ? ce : ce + sy;
	if constexpr (D > 2) {
		o[4] = kz && (z & 1) ? ce : ce - sz;
		o[5] = kz && !(z & 1) ? ce : ce + sz;
	}
	bool end[2 * D];
	end[0] = x == 0; end[1] = x + 4 == B.nx; end[2] = y == 0; end[3] = y + 1 == B.ny;
	if constexpr (D > 2) { end[4] = z == 0; end[5] = z + 1 == B.nz; }
#pragma unroll
	for (int f = 0; f < 2 * D; ++f) {
		st[f] = 1;
		if (end[f]) {
			if (B.open(f)) {
				o[f] = tabMap(CB.map[f], f == 1 ? cx + 1 : cx, cy, cz);
				st[f] = CB.map[f].y;
			} else {
				o[f] = ce;
				has &= ~(1u << f);
			}
		}
	}
	float lo[2 * D], hi[2 * D], a[2 * D + 1][4], w[4];
	const float e0 = e[ce], e1 = e[ce + 1];
#pragma unroll
	for (int f = 0; f < 2 * D; ++f) {
		lo[f] = e[o[f]];
		hi[f] = f < 2 ? 0.f : e[o[f] + st[f]];
	}
#pragma unroll
	for (int k = 0; k < 2 * D + 1; ++k) ld4f(A + k * N + g, a[k]);
	ld4f(wd + g, w);
#pragma unroll
	for (int f = 0; f < 2 * D; ++f)
		if (!((has >> f) & 1)) lo[f] = hi[f] = 0.f;
#pragma unroll
	for (int i = 0; i < 4; ++i) {
		const float ec = i < 2 ? e0 : e1;
		float yv = a[0][i] * ec;
		yv = fmaf(a[1][i], i == 0 ? lo[0] : i < 3 ? e0 : e1, yv);
		yv = fmaf(a[2][i], i == 0 ? e0 : i < 3 ? e1 : lo[1], yv);
#pragma unroll
		for (int f = 2; f < 2 * D; ++f) yv = fmaf(a[f + 1][i], i < 2 ? lo[f] : hi[f], yv);
		out[i] = fmaf(w[i], tv[i] - yv, fmaf(bv[i], w[i], ec));
	}
}

// y = A f at one cell and f there (fields of phb_krylov.cuh) ...
template <int D, typename F>
__device__ __forceinline__ float pcgCellApply(const BlockTab &B, int g, int x, int y, int z, int64_t N, const float *__restrict__ A,
		const F &f, float &fc) {
	int o[2 * D];
	const unsigned int has = tabNeighbors<D, 1>(B, g, x, y, z, o);
	float a[2 * D + 1], v[2 * D];
	fc = f.at(g);
#pragma unroll
	for (int s = 0; s < 2 * D; ++s) v[s] = f.at(o[s]);
#pragma unroll
	for (int k = 0; k < 2 * D + 1; ++k) a[k] = __ldg(A + k * N + g);
	float yv = a[0] * fc;
#pragma unroll
	for (int s = 0; s < 2 * D; ++s) yv = fmaf(a[s + 1], (has >> s) & 1 ? v[s] : 0.f, yv);
	return yv;
}
// ... and at four cells of an aligned row
template <int D, typename F>
__device__ __forceinline__ void pcgQuadApply(const BlockTab &B, int g, int x, int y, int z, int64_t N, const float *__restrict__ A,
		const F &f, float (&yv)[4], float (&fc)[4]) {
	int o[2 * D];
	const unsigned int has = tabNeighbors<D, 4>(B, g, x, y, z, o);
	float a[4], v[2 * D - 2][4];
	f.at4(g, 4, true, fc);
	float w = f.at(o[0]), e = f.at(o[1]);
#pragma unroll
	for (int s = 0; s < 2 * D - 2; ++s) f.at4(o[s + 2], 4, true, v[s]);
	if (!(has & 1)) w = 0.f;
	if (!(has & 2)) e = 0.f;
	ld4f(A + g, a);
#pragma unroll
	for (int i = 0; i < 4; ++i) yv[i] = a[i] * fc[i];
	ld4f(A + N + g, a);
#pragma unroll
	for (int i = 0; i < 4; ++i) yv[i] = fmaf(a[i], i ? fc[i ? i - 1 : 0] : w, yv[i]);
	ld4f(A + 2 * N + g, a);
#pragma unroll
	for (int i = 0; i < 4; ++i) yv[i] = fmaf(a[i], i < 3 ? fc[i < 3 ? i + 1 : 3] : e, yv[i]);
#pragma unroll
	for (int s = 2; s < 2 * D; ++s) {
		ld4f(A + (s + 1) * N + g, a);
		const bool h = (has >> s) & 1;
#pragma unroll
		for (int i = 0; i < 4; ++i) yv[i] = fmaf(a[i], h ? v[s - 2][i] : 0.f, yv[i]);
	}
}

// a restriction without update, of either width
template <int D>
__device__ __forceinline__ void pcgRestrictItemAny(bool w4, const BlockTab &B, const BlockTab &CB, int first, int64_t N,
		const float *__restrict__ A, const PcgFine<false> f, float *__restrict__ t, float *__restrict__ bc) {
	if (w4) pcgRestrictItem<D, 4, false>(B, CB, first, N, A, f, t, bc, nullptr, nullptr, nullptr, nullptr);
	else pcgRestrictItem<D, 2, false>(B, CB, first, N, A, f, t, bc, nullptr, nullptr, nullptr, nullptr);
}

// The dense operator of the last level, a warp per row, finished instances left out
template <int D>
__device__ __forceinline__ void pcgDense(const AmgView<D> &mg, const SysState *sst) {
	const int L = mg.nlevels - 1;
	const Dom<float, D> &cd = mg.lv[L];
	const int lane = threadIdx.x & 31;
	const int cn = mg.cn;
	const float *b = mg.b[L];
	float *x = mg.x[L];
	const int rows = cd.ninst * cn;
	// rows dealt out over the CTAs first
	const int nwarps = int(gridDim.x) * int(blockDim.x >> 5);
	for (int row = int(blockIdx.x) + int(gridDim.x) * int(threadIdx.x >> 5); row < rows; row += nwarps) {
		const int inst = row / cn, r = row - inst * cn;
		if (sst[inst].done != RUNNING) continue;
		const int off = __ldg(cd.insts + inst * PHB_IREC + I_CELLOFF);
		const int n = min(cn, __ldg(cd.insts + inst * PHB_IREC + I_NCELLS));
		if (r >= n) continue;
		const double *M = mg.inv + ((size_t)inst * cn + r) * cn;
		double s = 0;
#pragma unroll 8
		for (int c = lane; c < n; c += 32) s += __ldg(M + c) * double(b[off + c]);
		s = warpSum(s);
		if (lane == 0) x[off + r] = float(s);
	}
}

template <int N>
using Count = std::integral_constant<int, N>;

template <int D>
__global__ void __launch_bounds__(PHB_TILE *PCG_GROUPS, 1) kPcg(const __grid_constant__ PcgArgs<D> a) {
	extern __shared__ __align__(16) SysState sst[];
	__shared__ int2 sItems[PCG_GROUPS][(2 * AMG_MAX_LEVELS) * PCG_ITEMS]; // slot 2l: restriction of level l, 2l+1: its prolongation
	__shared__ int sCount[PCG_GROUPS][2]; // the group's items of slots 0 and 1
	__shared__ unsigned int sAl;
	__shared__ double sums_[PCG_GROUPS][TILE_SUMS * 2 * NWARPS];
	const Worker wk;
	int2 *sItem = sItems[wk.id];
	double *ws = sums_[wk.id];
	const int ninst = a.dom.ninst;
	const int nblk = a.dom.nblocks;
	const int T = a.mg.nlevels - 1;
	BlockTab *sBlk = reinterpret_cast<BlockTab *>(sst + ninst);
	if (threadIdx.x == 0) sAl = a.vec;
	for (int s = threadIdx.x; s < ninst; s += blockDim.x) sst[s] = a.st[s];
	if (!a.blocks)
		for (int i = threadIdx.x; i < (T + 1) * nblk; i += blockDim.x) buildBlockTab<D>(a.mg.lv[i / nblk].blocks, i % nblk, sBlk[i]);
	__syncthreads();
	const BlockTab *blks = a.blocks ? a.blocks : sBlk;
	// rows of four only where every block of the level allows them
	for (int i = threadIdx.x; i < (T + 1) * nblk; i += blockDim.x)
		if (!blks[i].rows4()) atomicAnd(&sAl, ~(1u << (i / nblk)));
	__syncthreads();
	const unsigned int alMask = sAl;
	auto blocksOf = [&](int l) -> const BlockTab * { return blks + l * nblk; };
	auto wide = [&](int l) -> bool { return ((alMask >> l) & 1) && a.mg.lv[l].ncells >= PCG_WIDE_MIN; };
	auto perR = [&](int l) -> int { return wide(l) ? PcgItem<D, 4>::PER : PcgItem<D, 2>::PER; };
	// Finest level outside the restriction: whole tiles (rows of four, or four cells per thread
	// 256 apart) or, where that would leave most warp slots empty, quarter tiles of a cell per thread
	const bool quarter = a.quarter;
	const int per0 = quarter ? CPT : 1, cells0 = quarter ? PHB_TILE : PHB_TILE_CELLS;
	// item `it` of a list of tiles in parts of `cells` cells: (block, first cell)
	auto decode = [&](const int32_t *tiles, int it, int per, int cells) -> int2 {
		const int tile = it / per;
		return make_int2(__ldg(tiles + 2 * tile), __ldg(tiles + 2 * tile + 1) + (it - tile * per) * cells);
	};
	for (int i = wk.lt; i < 2 * T * PCG_ITEMS; i += PHB_TILE) {
		const int slot = i / PCG_ITEMS, l = slot >> 1;
		const int it = wk.first + (i % PCG_ITEMS) * wk.step;
		int2 w = make_int2(0, 0);
		if (slot & 1) {
			const int per = l ? CPT : per0;
			if (it < a.mg.lv[l].ntiles * per) w = decode(a.mg.lv[l].tiles, it, per, l ? PHB_TILE : cells0);
		} else if (it < a.mg.lv[l + 1].ntiles * perR(l)) {
			w = decode(a.mg.lv[l + 1].tiles, it, perR(l), PHB_TILE_CELLS / perR(l));
		}
		sItem[i] = w;
	}
	if (wk.lt < 2) sCount[wk.id][wk.lt] = wk.count(wk.lt ? a.dom.ntiles * per0 : a.mg.lv[1].ntiles * perR(0));
	__syncthreads();
	int ph = 0;
	double *pp = a.partial;
	// Visit the group's items of a slot: f(item, block, first cell). The passes over the finest level
	// alternate in direction: what the one before touched last is still in L2 (six odd ducts of 3.6 M cells 250 -> 226 us per
	// iteration, with the reduction's wider loads).
	bool back = false;
	auto visit = [&](int slot, const int32_t *tiles, int n, int per, int cells, auto f) {
		int k = 0, it = wk.first, dk = 1;
		if (slot < 2) {
			if (back) { k = sCount[wk.id][slot] - 1; it += k * wk.step; dk = -1; }
			back = !back;
		}
		for (; dk < 0 ? k >= 0 : it < n; k += dk, it += dk * wk.step) {
			const int2 w = k < PCG_ITEMS ? sItem[slot * PCG_ITEMS + k] : decode(tiles, it, per, cells);
			f(it, w.x, w.y);
		}
	};
	// the same with sums over every item into the phase's partials: f(block, first cell, values)
	auto visitSums = [&](auto count, int slot, const int32_t *tiles, int n, int per, int cells, auto f) {
		constexpr int NV = decltype(count)::value;
		TileSums<NV> sums{wk, reinterpret_cast<double (*)[NV][NWARPS]>(ws), pp, 0, back ? sCount[wk.id][slot] - 1 : -1};
		visit(slot, tiles, n, per, cells, [&](int, int b, int first) {
			double acc[NV];
#pragma unroll
			for (int q = 0; q < NV; ++q) acc[q] = 0;
			f(b, first, acc);
			sums.add(acc);
			sums.next();
		});
		sums.finish();
	};
	const int64_t N = a.dom.ncells;
	const BlockTab *blk0 = blocksOf(0);
	const bool al0 = (alMask & 1) && !quarter;
	const int perA = perR(0);
	const int n0 = a.dom.ntiles * per0;
	auto nextPartials = [&] { pp = a.partial + (size_t)(ph++ & 1) * a.half; };
	auto tileRange = [&](int inst) {
		const int32_t *in = a.dom.insts + inst * PHB_IREC;
		return make_int2(__ldg(in + I_TILESTART) * per0, __ldg(in + I_TILECOUNT) * per0);
	};
	auto itemRange = [&](int inst) {
		const int32_t *in = a.mg.lv[1].insts + inst * PHB_IREC;
		return make_int2(__ldg(in + I_TILESTART) * perA, __ldg(in + I_TILECOUNT) * perA);
	};
	auto quad = [&](const BlockTab &B, int l0, auto f) {
		const int l = l0 + 4 * wk.lt;
		if (l >= B.cells()) return;
		const int row = l / B.nx, z = D > 2 ? row / B.ny : 0;
		f(B.off + l, l - row * B.nx, row - z * B.ny, z);
	};
	// cells 256 apart (loads of a warp stay contiguous whatever the row length), two at a time; the one cell
	// per thread of a quarter tile by itself
	auto cellsOf = [&](auto width, const BlockTab &B, int l0, auto f) {
		constexpr int W = decltype(width)::value;
		const int end = min(B.cells(), l0 + cells0);
		for (int l = l0 + wk.lt; l < end; l += W * PHB_TILE) {
			int g[W], x[W], y[W], z[W];
			const int n = W > 1 && l + PHB_TILE < end ? 2 : 1;
#pragma unroll
			for (int j = 0; j < W; ++j) {
				const int lj = j < n ? l + j * PHB_TILE : l;
				const int row = lj / B.nx;
				z[j] = D > 2 ? row / B.ny : 0;
				x[j] = lj - row * B.nx;
				y[j] = row - z[j] * B.ny;
				g[j] = B.off + lj;
			}
			f(width, n, g, x, y, z);
		}
	};
	auto cells = [&](const BlockTab &B, int l0, auto f) {
		if (quarter) cellsOf(Count<1>{}, B, l0, f);
		else cellsOf(Count<2>{}, B, l0, f);
	};
	float *rIn = a.r0, *rOut = a.r1, *pIn = a.p0, *pOut = a.p1;
	// r = b - A x, (r, r), (b, b)
	nextPartials();
	visitSums(Count<2>{}, 1, a.dom.tiles, n0, per0, cells0, [&](int b, int l0, double (&acc)[2]) {
		const BlockTab &B = blk0[b];
		if (sst[B.inst].done != RUNNING) return;
		const FX<float> fx{a.x};
		if (al0) {
			quad(B, l0, [&](int g, int x, int y, int z) {
				float yv[4], fc[4], bv[4];
				ld4f(a.b + g, bv);
				pcgQuadApply<D>(B, g, x, y, z, N, a.A, fx, yv, fc);
#pragma unroll
				for (int i = 0; i < 4; ++i) {
					yv[i] = bv[i] - yv[i];
					acc[0] = fma(double(yv[i]), double(yv[i]), acc[0]);
					acc[1] = fma(double(bv[i]), double(bv[i]), acc[1]);
				}
				st4f(rIn + g, yv);
			});
		} else {
			cells(B, l0, [&](auto width, int n, const auto &g, const auto &x, const auto &y, const auto &z) {
				constexpr int W = decltype(width)::value;
				float fc, rv[W], bv[W];
#pragma unroll
				for (int j = 0; j < W; ++j) {
					bv[j] = a.b[g[j]];
					rv[j] = bv[j] - pcgCellApply<D>(B, g[j], x[j], y[j], z[j], N, a.A, fx, fc);
				}
#pragma unroll
				for (int j = 0; j < W; ++j)
					if (j < n) {
						acc[0] = fma(double(rv[j]), double(rv[j]), acc[0]);
						acc[1] = fma(double(bv[j]), double(bv[j]), acc[1]);
						rIn[g[j]] = rv[j];
					}
			});
		}
	});
	if (!gridBarrier(a.ctrl)) return;
	int running = reduceSystems<1, 2, -1>(ninst, pp, sst, tileRange, [&](SysState &s, int in, const double *red, double) {
		if (a.stopStart) residualDecision<1, false, true>(nullptr, s, normScale(a.dom.insts, in), red, red[1], a.tol);
		else residualDecision<1, false, false>(nullptr, s, normScale(a.dom.insts, in), red, red[1], a.tol);
	});
	const float *z0 = a.mg.x[0];
	bool update = false;
	for (int iter = 0; running > 0 && iter <= a.maxit + 2; ++iter) {
		// A: the update of the last direction (from the second pass on) and the finest restriction
		nextPartials();
		{
			const BlockTab *cblk = blocksOf(1);
			const bool w4 = wide(0);
			visitSums(Count<1>{}, 0, a.mg.lv[1].tiles, a.mg.lv[1].ntiles * perA, perA, PHB_TILE_CELLS / perA, [&](int b, int first, double (&acc)[1]) {
				const BlockTab &B = blk0[b];
				const SysState &s = sst[B.inst];
				if (s.done != RUNNING) return;
				float *xb = s.saveBest ? a.xbest : nullptr;
				if (update) {
					const PcgFine<true> f{rIn, a.q, a.mg.wd[0], float(s.alpha)};
					if (w4) acc[0] = pcgRestrictItem<D, 4, true>(B, cblk[b], first, N, a.A, f, a.mg.x[0], a.mg.b[1], rOut, a.x, pIn, xb);
					else acc[0] = pcgRestrictItem<D, 2, true>(B, cblk[b], first, N, a.A, f, a.mg.x[0], a.mg.b[1], rOut, a.x, pIn, xb);
				} else {
					const PcgFine<false> f{rIn, nullptr, a.mg.wd[0], 0.f};
					pcgRestrictItemAny<D>(w4, B, cblk[b], first, N, a.A, f, a.mg.x[0], a.mg.b[1]);
				}
			});
		}
		if (!gridBarrier(a.ctrl)) return;
		if (update) {
			float *tmp = rIn; rIn = rOut; rOut = tmp;
			running = reduceSystems<1, 1, -1>(ninst, pp, sst, itemRange, [&](SysState &s, int in, const double *red, double) {
				const double crit = sqrt(red[0]) * normScale(a.dom.insts, in);
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
			});
			if (running == 0) break;
		}
		update = true;
		for (int l = 1; l < T; ++l) {
			const BlockTab *blk = blocksOf(l), *cblk = blocksOf(l + 1);
			const int per = perR(l);
			const bool w4 = wide(l);
			const PcgFine<false> f{a.mg.b[l], nullptr, a.mg.wd[l], 0.f};
			visit(2 * l, a.mg.lv[l + 1].tiles, a.mg.lv[l + 1].ntiles * per, per, PHB_TILE_CELLS / per, [&](int, int b, int first) {
				if (sst[blk[b].inst].done != RUNNING) return;
				pcgRestrictItemAny<D>(w4, blk[b], cblk[b], first, a.mg.lv[l].ncells, a.mg.A[l], f, a.mg.x[l], a.mg.b[l + 1]);
			});
			if (!gridBarrier(a.ctrl)) return;
		}
		pcgDense<D>(a.mg, sst);
		if (!gridBarrier(a.ctrl)) return;
		for (int l = T - 1; l >= 1; --l) {
			const BlockTab *blk = blocksOf(l), *cblk = blocksOf(l + 1);
			const float *bl = a.mg.b[l], *e = a.mg.x[l + 1];
			float *xl = a.mg.x[l];
			visit(2 * l + 1, a.mg.lv[l].tiles, a.mg.lv[l].ntiles * CPT, CPT, PHB_TILE, [&](int, int b, int first) {
				const BlockTab &B = blk[b];
				if (sst[B.inst].done != RUNNING) return;
				const int c = first + wk.lt;
				if (c >= B.cells()) return;
				const int row = c / B.nx, z = D > 2 ? row / B.ny : 0;
				const int g = B.off + c;
				xl[g] = pcgProlongCell<D>(B, cblk[b], g, c - row * B.nx, row - z * B.ny, z, a.mg.lv[l].ncells, a.mg.A[l], a.mg.wd[l], bl[g], xl[g], e);
			});
			if (!gridBarrier(a.ctrl)) return;
		}
		// finest level: z over t in place, (r, z)
		nextPartials();
		{
			const BlockTab *cblk = blocksOf(1);
			const float *e = a.mg.x[1];
			float *zz = a.mg.x[0];
			visitSums(Count<1>{}, 1, a.dom.tiles, n0, per0, cells0, [&](int b, int l0, double (&acc)[1]) {
				const BlockTab &B = blk0[b];
				if (sst[B.inst].done != RUNNING) return;
				if (al0) {
					quad(B, l0, [&](int g, int x, int y, int z) {
						float rv[4], tv[4], out[4];
						ld4f(rIn + g, rv);
						ld4f(zz + g, tv);
						pcgProlongQuad<D>(B, cblk[b], g, x, y, z, N, a.A, a.mg.wd[0], rv, tv, e, out);
#pragma unroll
						for (int i = 0; i < 4; ++i) acc[0] = fma(double(rv[i]), double(out[i]), acc[0]);
						st4f(zz + g, out);
					});
				} else {
					cells(B, l0, [&](auto width, int n, const auto &g, const auto &x, const auto &y, const auto &z) {
						constexpr int W = decltype(width)::value;
						float out[W], rv[W];
#pragma unroll
						for (int j = 0; j < W; ++j) {
							rv[j] = rIn[g[j]];
							out[j] = pcgProlongCell<D>(B, cblk[b], g[j], x[j], y[j], z[j], N, a.A, a.mg.wd[0], rv[j], zz[g[j]], e);
						}
#pragma unroll
						for (int j = 0; j < W; ++j)
							if (j < n) {
								acc[0] = fma(double(rv[j]), double(out[j]), acc[0]);
								zz[g[j]] = out[j];
							}
					});
				}
			});
		}
		if (!gridBarrier(a.ctrl)) return;
		reduceSystems<1, 1, -1>(ninst, pp, sst, tileRange, [&](SysState &s, int, const double *red, double) { pcgRho(s, red[0]); });
		// D: p' = z + beta p, q = A p', (p', q)
		nextPartials();
		visitSums(Count<1>{}, 1, a.dom.tiles, n0, per0, cells0, [&](int b, int l0, double (&acc)[1]) {
			const BlockTab &B = blk0[b];
			const SysState &s = sst[B.inst];
			if (s.done != RUNNING) return;
			// a restart (p not yet written) takes p' = z: z + 0 * z
			const FDir<float> fd{z0, s.restart ? z0 : pIn, s.restart ? 0.f : float(s.beta), false};
			if (al0) {
				quad(B, l0, [&](int g, int x, int y, int z) {
					float yv[4], fc[4];
					pcgQuadApply<D>(B, g, x, y, z, N, a.A, fd, yv, fc);
#pragma unroll
					for (int i = 0; i < 4; ++i) acc[0] = fma(double(fc[i]), double(yv[i]), acc[0]);
					st4f(pOut + g, fc);
					st4f(a.q + g, yv);
				});
			} else {
				cells(B, l0, [&](auto width, int n, const auto &g, const auto &x, const auto &y, const auto &z) {
					constexpr int W = decltype(width)::value;
					float yv[W], fc[W];
#pragma unroll
					for (int j = 0; j < W; ++j) yv[j] = pcgCellApply<D>(B, g[j], x[j], y[j], z[j], N, a.A, fd, fc[j]);
#pragma unroll
					for (int j = 0; j < W; ++j)
						if (j < n) {
							acc[0] = fma(double(fc[j]), double(yv[j]), acc[0]);
							pOut[g[j]] = fc[j];
							a.q[g[j]] = yv[j];
						}
				});
			}
		});
		if (!gridBarrier(a.ctrl)) return;
		running = reduceSystems<1, 1, -1>(ninst, pp, sst, tileRange, [&](SysState &s, int, const double *red, double) {
			const double alpha = s.rho / red[0];
			s.restart = 0;
			if (!fin(alpha)) { s.done = NONFINITE; s.usedIt = s.it; }
			else s.alpha = alpha;
		});
		float *tmp = pIn; pIn = pOut; pOut = tmp;
	}
	// systems that stopped without converging return their best iterate (kRestoreBest)
	if (a.xbest) {
		visit(1, a.dom.tiles, n0, per0, cells0, [&](int, int b, int l0) {
			const BlockTab &B = blk0[b];
			const SysState &s = sst[B.inst];
			if (!((s.done == MAXIT || s.done == RISING) && s.bestIt >= 0 && s.best < s.crit)) return;
			const int end = min(B.cells(), l0 + cells0);
			for (int l = l0 + wk.lt; l < end; l += PHB_TILE) a.x[B.off + l] = a.xbest[B.off + l];
		});
	}
	if (blockIdx.x == 0) {
		__syncthreads();
		for (int s = threadIdx.x; s < ninst; s += blockDim.x) a.st[s] = sst[s];
	}
}

template <int D>
int launchPcg(const phb_domain *dom, const phb_solve *sv, cudaStream_t s, bool stopStart, int fromInner) {
	const Layout L = solveLayout(dom, 0, sizeof(float), 1);
	const StateLayout SL = stateLayout(dom, 1);
	char *w = (char *)sv->work;
	char *sb = (char *)sv->state;
	PcgArgs<D> a = {};
	a.dom = Dom<double, D>(*dom);
	a.A = (const float *)sv->A;
	a.b = (const float *)sv->b;
	a.x = (float *)sv->x;
	a.r0 = (float *)(w + L.off[0]);
	a.q = (float *)(w + L.off[1]);
	a.p0 = (float *)(w + L.off[2]);
	a.p1 = (float *)(w + L.off[3]);
	a.xbest = sv->return_best ? (float *)(w + L.off[4]) : nullptr;
	a.r1 = (float *)(w + L.off[5]);
	a.partial = (double *)(w + L.off[10]);
	a.half = (int64_t)dom->ntiles * PCG_PARTIALS;
	a.ctrl = (Control *)(sb + SL.ctrl);
	a.st = (SysState *)(sb + SL.st);
	a.tol = sv->tol;
	a.returnBest = sv->return_best;
	a.maxit = std::max(1, sv->maxit);
	a.stopStart = stopStart;
	a.mg = makeAmgView<D>(*sv->amg, a.r0, sv->amg->levels[0].x);
	for (int l = 0; l < a.mg.nlevels; ++l) {
		const void *ps[4] = {a.mg.A[l], a.mg.wd[l], a.mg.b[l], a.mg.x[l]};
		bool ok = a.mg.lv[l].ncells % 4 == 0;
		for (const void *p : ps) ok = ok && ((uintptr_t)p & 15) == 0;
		if (l == 0) ok = ok && vec4Ok(dom, {a.A, a.b, a.x, w});
		if (ok) a.vec |= 1u << l;
	}
	const int rc = launchInit(a.st, dom->ninst, sv->tol, fromInner, a.maxit, a.ctrl, s);
	if (rc) return rc;
	const size_t stBytes = (size_t)dom->ninst * sizeof(SysState);
	const size_t recBytes = (size_t)a.mg.nlevels * dom->nblocks * sizeof(BlockTab);
	if (stBytes > 160 * 1024) return setError(PHB_ERR_RANGE, "persistent solve: too many systems for the per-CTA state copy");
	size_t smem = stBytes + recBytes;
	if (recBytes > TAB_SMEM_MAX || smem > 160 * 1024) {
		smem = stBytes;
		a.blocks = (BlockTab *)(w + L.off[9]);
		kPcgTabs<D><<<std::max(1, std::min(1024, (dom->nblocks * a.mg.nlevels + 127) / 128)), 128, 0, s>>>(a.mg, (BlockTab *)(w + L.off[9]));
		PHB_CUDA(cudaGetLastError());
	}
	a.quarter = dom->ntiles < PCG_QUARTER_TILES;
	auto kern = kPcg<D>;
	if (smem > 32 * 1024) PHB_CUDA(allowSmem((const void *)kern));
	int groups = 1, ctas = 1;
	persistentGrid(dom->ntiles * (a.quarter ? CPT : 1), PCG_GROUPS, sv->ctas_per_sm, groups, ctas);
	cudaLaunchConfig_t cfg = {};
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeCooperative;
	attr[0].val.cooperative = 1;
	cfg.gridDim = dim3(ctas);
	cfg.blockDim = dim3(PHB_TILE * groups);
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	PHB_CUDA(cudaLaunchKernelEx(&cfg, kern, a));
	return PHB_OK;
}
template int launchPcg<2>(const phb_domain *, const phb_solve *, cudaStream_t, bool, int);
template int launchPcg<3>(const phb_domain *, const phb_solve *, cudaStream_t, bool, int);

} // namespace phb
