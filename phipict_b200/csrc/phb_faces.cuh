// Neighbours of a cell without branches between the loads: what the assembly kernels of the
// orthogonal, central step use.
//
// The cell across a face of a block that is not fixed is an affine function of the position
// (periodic: the other end of the row; connected: phiPICT's axis mapping, topology.cuh:168-246), so
// one map per face, staged once per CTA, gives every neighbour by arithmetic. A kernel first forms
// all indices (a fixed face gets the cell itself), then issues all loads, then corrects the few
// cells on fixed faces: resolving each face in a branch of its own makes a cell's loads wait for
// one another.
#pragma once

#include <algorithm>
#include <type_traits>
#include "phb_device.cuh"

namespace phb {

struct FaceMap {
	int c0, cx, cy, cz; // state index of the cell across: c0 + cx x + cy y + cz z
	int met;            // its metric index minus its state index
	int comp;           // component of its block that the face's axis maps to
	int flip;           // the face flux changes sign
	int open;           // not a fixed face
};

// Map of face f of the block staged in sB.
template <typename S, int D>
__device__ __forceinline__ void buildFaceMap(const Dom<S, D> &dom, const int32_t *sB, int f, FaceMap &m) {
	const int ax = f >> 1;
	const int32_t *fr = fRec(sB, f);
	m = FaceMap{0, 0, 0, 0, 0, ax, 0, fr[0] != FT_FIXED};
	if (fr[0] == FT_FIXED) return;
	int cf[3] = {0, 0, 0}; // coefficients of x, y, z
	if (fr[0] == FT_CONNECTED) {
		const int32_t *OB = dom.blk(fr[1]);
		const int stride[3] = {1, OB[B_NX], OB[B_NX] * OB[B_NY]};
		m.c0 = OB[B_CELLOFF];
		// the axis across the face is at its end, the tangential ones follow, mirrored where flagged
		const int c0 = fr[2] >> 1;
		if (fr[2] & 1) m.c0 += (OB[B_NX + c0] - 1) * stride[c0];
#pragma unroll
		for (int k = 1; k < D; ++k) {
			const int axis = (ax + k) % D, ca = fr[2 + k] >> 1;
			if (fr[2 + k] & 1) {
				m.c0 += (OB[B_NX + ca] - 1) * stride[ca];
				cf[axis] = -stride[ca];
			} else {
				cf[axis] = stride[ca];
			}
		}
		m.met = OB[B_METOFF] - OB[B_CELLOFF];
		m.comp = c0;
		m.flip = connectedSameSide(sB, f);
	} else {
		const int stride[3] = {1, sB[B_NX], sB[B_NX] * sB[B_NY]};
		m.c0 = sB[B_CELLOFF] + ((f & 1) ? 0 : (sB[B_NX + ax] - 1) * stride[ax]);
#pragma unroll
		for (int k = 1; k < D; ++k) cf[(ax + k) % D] = stride[(ax + k) % D];
		m.met = sB[B_METOFF] - sB[B_CELLOFF];
	}
	m.cx = cf[0]; m.cy = cf[1]; m.cz = cf[2];
}

// Visit the CTA's share of the tiles: f(first cell of the tile, cells of the block, first of its cells per
// thread, aligned) with the block record and its face maps staged; aligned: no face of the block maps its axis to
// another component (compile-time components make half the index arithmetic). A CTA takes several (the grid is
// the CTAs that fit the chip): a CTA per tile spends more than half its life on the reads that lead to its first
// cell (tile, block record, instance parameters); here they are made once per block. PARTS = 1: whole tiles;
// PARTS = CPT: quarter tiles of a cell per thread, `run` consecutive ones per CTA or (run 0) gridDim.x apart
// (tileShare chooses).
template <int PARTS, typename S, int D, typename F>
__device__ __forceinline__ void forTiles(const Dom<S, D> &dom, int run, int32_t *sB, FaceMap *sF, F f) {
	static_assert(PARTS == 1 || PARTS == CPT, "whole or quarter tiles");
	int staged = -1; // the block in sB (uniform over the CTA)
	bool aligned = false;
	const int items = dom.ntiles * PARTS;
	const bool row = PARTS != 1 && run > 0;
	const int step = row ? 1 : int(gridDim.x);
	const int first = row ? int(blockIdx.x) * run : int(blockIdx.x);
	const int end = row ? min(items, first + run) : items;
	int b = 0, l0 = 0;
	if (first < end) {
		b = __ldg(dom.tiles + 2 * (first / PARTS));
		l0 = __ldg(dom.tiles + 2 * (first / PARTS) + 1);
	}
	for (int t = first; t < end; t += step) {
		const int n = (t + step < end ? t + step : t) / PARTS;
		const int bn = __ldg(dom.tiles + 2 * n), ln = __ldg(dom.tiles + 2 * n + 1); // the next tile
		if (b != staged) {
			__syncthreads();
			if (threadIdx.x < PHB_BREC) sB[threadIdx.x] = __ldg(dom.blocks + b * PHB_BREC + threadIdx.x);
			__syncthreads();
			bool same = true;
			if (threadIdx.x < 2 * D) {
				buildFaceMap<S, D>(dom, sB, int(threadIdx.x), sF[threadIdx.x]);
				same = sF[threadIdx.x].comp == int(threadIdx.x >> 1);
			}
			aligned = __syncthreads_and(same);
			staged = b;
		}
		const int nc = sB[B_NX] * sB[B_NY] * (D > 2 ? sB[B_NZ] : 1);
		const int j0 = PARTS == 1 ? 0 : t % PARTS;
		if (aligned) f(l0, nc, j0, std::true_type{});
		else f(l0, nc, j0, std::false_type{});
		b = bn;
		l0 = ln;
	}
}

// How a launch shares out its tiles: a kernel has a form for whole and one for quarter tiles.
// - Quarter tiles in runs, where whole tiles would give most CTAs one or none (a thread then walks its four
//   cells one after the other while most of the chip idles) or leave the last of a few rounds nearly empty: where the
//   longest run is at most three quarters (kernels of few loads, `least` 0, and 2D: five eighths) of the cells that a
//   thread of the whole form takes, up to MAX_RUN. 64 x 32 cells float32: matrix 14.3 -> 9.2 us, HbyA 17.4 -> 9.3;
//   32^3 float64: HbyA 38 -> 17; 432 tiles float64 on 296 CTAs: potential right-hand side 35.8 -> 29.7. Three
//   quarters where five eighths are the rule: 2D divergence, 256 tiles, 8.4 -> 10.2; 96^3 float32 advection
//   right-hand side 26.8 -> 29.7.
// - Quarter tiles gridDim.x apart, in 3D on blocks of eight tiles and more (runs meet fewer blocks), where whole
//   tiles would use less than `least` percent of their rounds: 99 x 101 x 97 float64, 948 tiles in 4 rounds of
//   296: matrix 74.7 -> 64.5 us, HbyA 85 -> 67.
// - Whole tiles otherwise: fewer reads of tile records, four cells' index arithmetic unrolled.
struct TileShare {
	bool quarters;
	int ctas, run;
};
template <auto KERN>
inline int residentCtas() { // CTAs of a kernel that the device holds at a time
	static const int resident = [] {
		int dev = 0, sms = 0, per = 0;
		if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
				cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, KERN, PHB_TILE, 0) != cudaSuccess || per < 1 || sms < 1) {
			(void)cudaGetLastError();
			return 148;
		}
		return per * sms;
	}();
	return resident;
}
template <auto WHOLE, auto QUARTER>
inline TileShare tileShare(const phb_domain *dom, int least) {
	constexpr int MAX_RUN = 6;
	const int64_t tiles = dom->ntiles, quarter = residentCtas<QUARTER>(), whole = residentCtas<WHOLE>();
	const int64_t rounds = (tiles + whole - 1) / whole, run = (tiles * CPT + quarter - 1) / quarter;
	const int64_t fill = std::max<int64_t>(1, std::min<int64_t>(CPT, (dom->ncells + tiles * PHB_TILE - 1) / (tiles * PHB_TILE))); // cells of a thread
	if (run <= MAX_RUN && 8 * run <= (least ? 6 : 5) * rounds * fill) return {true, int((tiles * CPT + run - 1) / run), int(run)};
	if (tiles >= 8 * (int64_t)dom->nblocks && 100 * tiles < least * rounds * whole) return {true, int(std::min(quarter, tiles * CPT)), 0};
	return {false, int(std::min(tiles, whole)), 0};
}

// The neighbours of one cell: state and metric indices, the neighbour's component across the face.
template <int D>
struct Faces {
	int o[2 * D], om[2 * D], comp[2 * D];
	unsigned int fixed, flip; // bit f
};
template <int D>
__device__ __forceinline__ Faces<D> cellFaces(const int32_t *sB, const FaceMap *sF, const Cell &c) {
	Faces<D> r;
	r.fixed = r.flip = 0;
	const int stride[3] = {1, sB[B_NX], sB[B_NX] * sB[B_NY]};
#pragma unroll
	for (int f = 0; f < 2 * D; ++f) {
		const int ax = f >> 1;
		const int step = (f & 1) ? stride[ax] : -stride[ax];
		r.o[f] = c.g + step;
		r.om[f] = c.mi + step;
		r.comp[f] = ax;
		if (atBound(sB, f, c.p)) {
			const FaceMap &m = sF[f];
			if (m.open) {
				r.o[f] = m.c0 + m.cx * c.p[0] + m.cy * c.p[1] + m.cz * c.p[2];
				r.om[f] = r.o[f] + m.met;
				r.comp[f] = m.comp;
				r.flip |= (unsigned int)m.flip << f;
			} else {
				r.o[f] = c.g;
				r.om[f] = c.mi;
				r.fixed |= 1u << f;
			}
		}
	}
	return r;
}

// A vector field [inst][D][cells] of the staged block's instance: component k of cell g is c[k][g].
template <typename S, int D>
struct Comps {
	const S *c[D];
	__device__ __forceinline__ Comps(const int32_t *sB, const S *field) {
#pragma unroll
		for (int k = 0; k < D; ++k) c[k] = field + vidx<D>(sB, 0, k);
	}
};
// contraAt with the component pointers formed before
template <typename S, int D>
__device__ __forceinline__ S contraComps(const Dom<S, D> &dom, const Comps<S, D> &v, int g, int mi, int c) {
	S s = 0;
#pragma unroll
	for (int j = 0; j < D; ++j) s += dom.m(Tr<D>::MINV + c * D + j, mi) * v.c[j][g];
	return dom.m(Tr<D>::DET, mi) * s;
}

// Face fluxes of a vector field (faceFluxes of phb_upwind.cuh): the mean of the two cells'
// contravariant components, the boundary velocity's on fixed faces.
template <typename S, int D, bool SAME>
__device__ __forceinline__ void cellFluxes(const Dom<S, D> &dom, const Cell &c, const Faces<D> &n, const Comps<S, D> &v, S (&fl)[2 * D]) {
	S vN[2 * D], vC[D];
#pragma unroll
	for (int f = 0; f < 2 * D; ++f) vN[f] = contraComps<S, D>(dom, v, n.o[f], n.om[f], SAME ? f >> 1 : n.comp[f]);
#pragma unroll
	for (int d = 0; d < D; ++d) vC[d] = contraComps<S, D>(dom, v, c.g, c.mi, d);
#pragma unroll
	for (int f = 0; f < 2 * D; ++f) fl[f] = (((n.flip >> f) & 1 ? -vN[f] : vN[f]) + vC[f >> 1]) * S(0.5);
	if (n.fixed) {
#pragma unroll
		for (int f = 0; f < 2 * D; ++f)
			if ((n.fixed >> f) & 1) fl[f] = contraFixed<S, D>(dom, dom.fix(fRec(c.B, f)[5]), faceCell(c.B, f, c.p), f >> 1);
	}
}

} // namespace phb
