// Operator implementations and the (delta, dims, precision) dispatch table.
#include <algorithm>
#include <cstdio>
#include <cstdint>
#include <cuda.h>
#include "ibk_internal.h"
#include "ibk_direct.cuh"
#include "ibk_tiled.cuh"

namespace ibk {

namespace {

constexpr int kThreads = 128;

// Threads of an FP32C spread CTA on grids of at most two tiles per SM, whose
// time is the candidates per thread (128 x 64 x 128 cells, 124,700 points, 256
// tiles: 91 -> 82 us; 64^3, 64 tiles: 72 -> 64; at 6 x 12 x 12 tiles and more no
// difference, and with 1024 threads 94 and 62).
constexpr int kFewThreads = 512;

// The FP64 spread of the cubic B-spline, by the candidates of an average tile
// (about 2.5 per point), in us, binning included, n points on cells^3:
//   owners, the candidates split over several CTAs, where the tiles are few
//   and full (132,600 points on 26^3: 257, unsplit atomics 678; on 32^3: 248, 379);
//   atomics where the tiles are fewer than the SMs and have many candidates all
//   the same, since then the time is that of the longest chain (22,100 on 26^3:
//   160, owners 199; 132,600 on 40^3: 266, 297, and on 72^3: 243, 286), and where
//   tiles of more than kS64SmallTile cells have few, often in clumps (11,050
//   points on 96^3: 84, 99; 2,210 on 160^3: 82, 93; but 8,832 of one finely
//   sampled cell on 96^3: 187, 166);
//   owners else (1.36 M points on 256 x 128 x 256: 1009, atomics 1036; 124,700
//   on 128 x 64 x 128: 166, 173; 8,832 on 64^3 in small tiles: 91, 101).
constexpr int kS64SplitCandidates = 4096, kS64ManyCandidates = 800, kS64FewCandidates = 160, kS64SmallTile = 2048;

inline int blocks_for(long long n, int threads) { return (int) ((n + threads - 1) / threads); }

// Per-point kernels for degenerate grids (an axis with fewer cells than the
// stencil is wide, where one stencil would reach the same face twice).
template <typename D, int DIMS>
ibk_status spread_direct(Plan& plan, const OpArgs& a, const double* fl, CompPtrs fe)
{
	const GridGeom& g = *a.g;
	for (int c = 0; c < DIMS; ++c) {
		cudaError_t e = cudaMemsetAsync(fe.p[c], 0, sizeof(double) * (size_t) g.comp[c].size, a.stream);
		if (e != cudaSuccess) return set_error(IBK_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
	}
	return launch(plan, "spread_direct_kernel", a.stream, [&] {
		spread_direct_kernel<D, DIMS><<<blocks_for(a.n, kThreads), kThreads, 0, a.stream>>>(g, a.n, a.x, fl, fe);
	});
}

template <typename D, int DIMS>
ibk_status interp_direct(Plan& plan, const OpArgs& a, ConstCompPtrs ue, double* ul)
{
	return launch(plan, "interp_direct_kernel", a.stream, [&] {
		interp_direct_kernel<D, DIMS><<<blocks_for(a.n, kThreads), kThreads, 0, a.stream>>>(*a.g, a.n, a.x, ue, ul);
	});
}

// What the binning leaves: records in bin order, the bin offsets and, for an
// FP32C spread, the points' forces beside the records and the deferral list
// with its count zeroed.
struct Binned {
	const PointRec* recs = nullptr;
	const int* off = nullptr;
	const float4* forces = nullptr;
	Deferral defer{nullptr, nullptr};
};

// Counting sort of the points by (tile, reach class); f: the forces an FP32C
// spread of these points takes, or null.
template <int M, int DIMS>
ibk_status bin_points(Plan& plan, const OpArgs& a, const TileGeom& tg, Binned& out, const double* f = nullptr)
{
	ibk_status s;
	const int need = a.n > plan.reserved_points ? a.n : plan.reserved_points;
	if ((s = ensure_scratch(plan, kSlotCount, sizeof(int) * (size_t) tg.num_bins, a.stream, true)) != IBK_OK) return s;
	if ((s = ensure_scratch(plan, kSlotOffset, sizeof(int) * ((size_t) tg.num_bins + 1), a.stream)) != IBK_OK) return s;
	if ((s = ensure_scratch(plan, kSlotRank, sizeof(int) * (size_t) need, a.stream)) != IBK_OK) return s;
	if ((s = ensure_scratch(plan, kSlotRecs, sizeof(PointRec) * (size_t) need, a.stream)) != IBK_OK) return s;
	const int nchunks = (tg.num_bins + kScanChunk - 1) / kScanChunk;
	// the count kernel's ticket, then the chunk sums
	if ((s = ensure_scratch(plan, kSlotChunk, sizeof(int) * ((size_t) nchunks + 2), a.stream, true)) != IBK_OK) return s;
	int* count = static_cast<int*>(plan.scratch[kSlotCount].ptr);
	int* off = static_cast<int*>(plan.scratch[kSlotOffset].ptr);
	int* rank = static_cast<int*>(plan.scratch[kSlotRank].ptr);
	PointRec* recs = static_cast<PointRec*>(plan.scratch[kSlotRecs].ptr);
	unsigned* ticket = static_cast<unsigned*>(plan.scratch[kSlotChunk].ptr);
	int* chunk = static_cast<int*>(plan.scratch[kSlotChunk].ptr) + 1;
	const GridGeom& g = *a.g;
	const int nb = blocks_for(a.n, 256);
	BinForces bf{f, g.res, nullptr};
	int* clear = nullptr;
	// Room for as many forces as records, from the first spread on: a spread
	// under capture then finds it whenever the records' own room suffices.  An
	// interpolation does without.
	if (f || plan.scratch[kSlotForces].ptr) {
		const size_t held = plan.scratch[kSlotRecs].bytes / sizeof(PointRec);
		if ((s = ensure_scratch(plan, kSlotForces, sizeof(float4) * held, a.stream)) != IBK_OK && f) return s;
	}
	if (f) {
		if ((s = ensure_scratch(plan, kSlotDefer, sizeof(int) * ((size_t) tg.num_tiles * DIMS + 4), a.stream)) != IBK_OK)
			return s;
		bf.out = static_cast<float4*>(plan.scratch[kSlotForces].ptr);
		clear = static_cast<int*>(plan.scratch[kSlotDefer].ptr);
		out.forces = bf.out;
		out.defer = Deferral{clear + 4, clear};
	}
	out.recs = recs;
	out.off = off;
	const bool tail = tg.num_bins <= kTailBins;
	if (a.n <= (tail ? kSmallThreads : kSmallPoints) && tg.num_bins <= kSmallBins) {
		const size_t smem = sizeof(int) * (size_t) tg.num_bins;
		auto kern = bin_small_kernel<M, DIMS>;
		if ((s = allow_smem(kern)) != IBK_OK) return s;
		return launch(plan, "bin_small_kernel", a.stream, [&] {
			kern<<<1, kSmallThreads, smem, a.stream>>>(g, tg, a.n, a.x, off, recs, bf, clear);
		});
	}
	const ScanTail scan{off, ticket, tg.num_bins};
	if ((s = launch(plan, "bin_count_kernel", a.stream, [&] {
		if (tail) bin_count_kernel<M, DIMS, true><<<nb, 256, 0, a.stream>>>(g, tg, a.n, a.x, count, rank, scan);
		else bin_count_kernel<M, DIMS, false><<<nb, 256, 0, a.stream>>>(g, tg, a.n, a.x, count, rank, scan);
	})) != IBK_OK) return s;
	if (!tail) {
		if ((s = launch(plan, "bin_chunk_sum_kernel", a.stream, [&] {
			bin_chunk_sum_kernel<<<nchunks, kScanThreads, 0, a.stream>>>(count, chunk, tg.num_bins);
		})) != IBK_OK) return s;
		if ((s = launch(plan, "bin_scan_kernel", a.stream, [&] {
			bin_scan_kernel<<<nchunks, kScanThreads, 0, a.stream>>>(count, chunk, off, tg.num_bins, nchunks);
		})) != IBK_OK) return s;
	}
	if ((s = launch(plan, "bin_scatter_kernel", a.stream, [&] {
		bin_scatter_kernel<M, DIMS><<<nb, 256, 0, a.stream>>>(g, tg, a.n, a.x, rank, off, recs, bf, clear);
	})) != IBK_OK) return s;
	return IBK_OK;
}

// An FP64 spread; parts > 1: as many CTAs share a tile's candidates (owners
// only) and add their sums to zeroed faces.
template <typename D, int DIMS, bool OWNERS>
ibk_status launch_spread64(Plan& plan, const OpArgs& a, const TileGeom& tg, const Binned& b, const double* fl, CompPtrs fe,
                           int parts = 1)
{
	const size_t smem = spread_smem_bytes(*a.g, tg, D::M, IBK_PRECISION_FP64, OWNERS);
	auto kern = spread_tile64_kernel<D, DIMS, OWNERS>;
	ibk_status s = allow_smem(kern);
	if (s != IBK_OK) return s;
	for (int c = 0; c < DIMS && parts > 1; ++c) {
		cudaError_t e = cudaMemsetAsync(fe.p[c], 0, sizeof(double) * (size_t) a.g->comp[c].size, a.stream);
		if (e != cudaSuccess) return set_error(IBK_ERR_CUDA, std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
	}
	return launch(plan, "spread_tile_kernel", a.stream, [&] {
		kern<<<dim3(tg.num_tiles, DIMS, parts), s64_threads<OWNERS>(), smem, a.stream>>>(*a.g, tg, a.n, a.x, fl, b.recs,
		                                                                                b.off, fe);
	});
}

template <typename D, int DIMS, int PREC>
ibk_status launch_spread(Plan& plan, const OpArgs& a, const TileGeom& tg, const Binned& b, const double* fl, CompPtrs fe)
{
	ibk_status s;
	if constexpr (PREC == IBK_PRECISION_FP64) {
		if constexpr (s64_owners<D, DIMS>()) {
			const long long items = (long long) tg.num_tiles * DIMS, cand = 5LL * a.n / (2 * tg.num_tiles);
			if (items < 2LL * plan.num_sms && cand >= kS64SplitCandidates)
				return launch_spread64<D, DIMS, true>(plan, a, tg, b, fl, fe, (int) std::min(
					(4LL * plan.num_sms + items - 1) / items, cand / (kS64SplitCandidates / 4)));
			const bool few = tg.num_tiles < plan.num_sms, small = tg.T[0] * tg.T[1] * tg.T[2] <= kS64SmallTile;
			if (few ? cand < kS64ManyCandidates : small || cand >= kS64FewCandidates)
				return launch_spread64<D, DIMS, true>(plan, a, tg, b, fl, fe);
		}
		return launch_spread64<D, DIMS, false>(plan, a, tg, b, fl, fe);
	} else {
		// one CTA per tile for every component, dense tiles deferred to the
		// folded kernel
		const size_t smem = spread_smem_bytes(*a.g, tg, D::M, PREC, false);
		const bool few = tg.num_tiles <= 2 * plan.num_sms;
		auto kern = few ? spread_tile_kernel<D, DIMS, kFewThreads> : spread_tile_kernel<D, DIMS>;
		const int nt = few ? kFewThreads : kTileThreads;
		auto dense = spread_dense_kernel<D, DIMS>;
		const size_t dsmem = folded_layout(tg, DIMS).bytes;
		if ((s = allow_smem(kern)) != IBK_OK || (s = allow_smem(dense)) != IBK_OK) return s;
		if ((s = launch(plan, "spread_tile_kernel", a.stream, [&] {
			kern<<<tg.num_tiles, nt, smem, a.stream>>>(*a.g, tg, b.recs, b.forces, b.off, fe, b.defer);
		})) != IBK_OK) return s;
		// no face can receive more terms than there are points
		if (a.n <= 2 * kFoldChunk) return IBK_OK;
		const int gd = std::max(1, std::min(tg.num_tiles * DIMS, 2 * plan.num_sms));
		return launch(plan, "spread_dense_kernel", a.stream, [&] {
			dense<<<gd, kDenseThreads, dsmem, a.stream>>>(*a.g, tg, b.recs, b.forces, b.off, fe, b.defer.list, b.defer.count);
		});
	}
}

template <int KIND, int ORDER, int DIMS, int PREC>
ibk_status spread_impl(Plan& plan, const OpArgs& a, const double* fl, CompPtrs fe)
{
	using D = Delta<KIND, ORDER>;
	if (!plan.tiled) return spread_direct<D, DIMS>(plan, a, fl, fe);
	Binned b;
	constexpr bool fix = PREC == IBK_PRECISION_FP32C;
	ibk_status s = bin_points<D::M, DIMS>(plan, a, plan.spread_tiles, b, fix ? fl : nullptr);
	if (s != IBK_OK) return s;
	return launch_spread<D, DIMS, PREC>(plan, a, plan.spread_tiles, b, fl, fe);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// dependency on libcuda).
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
	static EncodeTiledFn fn = [] {
		void* p = nullptr;
		cudaDriverEntryPointQueryResult q{};
		if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
		    q != cudaDriverEntryPointSuccess) {
			cudaGetLastError();
			return (EncodeTiledFn) nullptr;
		}
		return reinterpret_cast<EncodeTiledFn>(p);
	}();
	return fn;
}

} // namespace

// Tensor map of one FP64 component grid with box `box` (elements per axis).
// False when the grid or box violates a TMA rule (16-byte base and strides,
// box rows a multiple of 16 bytes, at most 256 elements per box axis).
bool grid_tensor_map(CUtensorMap* map, const double* base, const CompGeom& cg, int dims, const int* box)
{
	EncodeTiledFn fn = encode_fn();
	if (!fn || (reinterpret_cast<uintptr_t>(base) & 15) != 0) return false;
	if ((cg.points[0] * sizeof(double)) % 16 != 0 || (box[0] * sizeof(double)) % 16 != 0) return false;
	cuuint64_t gdim[3], gstride[2];
	cuuint32_t bdim[3], estride[3] = {1, 1, 1};
	cuuint64_t stride = sizeof(double);
	for (int d = 0; d < dims; ++d) {
		if (box[d] > 256 || box[d] > cg.points[d]) return false;
		gdim[d] = (cuuint64_t) cg.points[d];
		bdim[d] = (cuuint32_t) box[d];
		if (d > 0) gstride[d - 1] = stride;
		stride *= (cuuint64_t) cg.points[d];
	}
	CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, (cuuint32_t) dims, const_cast<double*>(base),
	                gdim, gstride, bdim, estride, CU_TENSOR_MAP_INTERLEAVE_NONE,
	                CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
	                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	return r == CUDA_SUCCESS;
}

namespace {

template <typename D, int DIMS, int PREC>
ibk_status launch_interp(Plan& plan, const OpArgs& a, const TileGeom& tg, const Binned& b, ConstCompPtrs ue, double* ul)
{
	const GridGeom& g = *a.g;
	const size_t smem = interp_smem_bytes<D::M>(g, tg);
	// TMA needs every region's x origin on a 16-byte boundary: even tile
	// extents along x (the region's lower x offset is even by construction)
	TmaMaps maps{};
	int use_tma = tg.T[0] % 2 == 0;
	for (int c = 0; c < DIMS && use_tma; ++c) {
		int lower[3], box[3];
		region_of<D::M>(g, tg, c, lower, box);
		use_tma = grid_tensor_map(&maps.map[c], ue.p[c], g.comp[c], DIMS, box);
	}
	auto kern = interp_tile_kernel<D, DIMS, PREC>;
	ibk_status s = allow_smem(kern);
	if (s != IBK_OK) return s;
	return launch(plan, "interp_tile_kernel", a.stream, [&] {
		kern<<<dim3(tg.num_tiles, DIMS), kTileThreads, smem, a.stream>>>(g, tg, a.n, a.x, b.recs, b.off, ue, ul,
		                                                                   maps, use_tma, plan.d_status);
	});
}

template <int KIND, int ORDER, int DIMS, int PREC>
ibk_status interp_impl(Plan& plan, const OpArgs& a, ConstCompPtrs ue, double* ul)
{
	using D = Delta<KIND, ORDER>;
	if (!plan.tiled) return interp_direct<D, DIMS>(plan, a, ue, ul);
	Binned b;
	ibk_status s = bin_points<D::M, DIMS>(plan, a, plan.tiles, b);
	if (s != IBK_OK) return s;
	return launch_interp<D, DIMS, PREC>(plan, a, plan.tiles, b, ue, ul);
}

bool same_tiles(const TileGeom& a, const TileGeom& b)
{
	return a.T[0] == b.T[0] && a.T[1] == b.T[1] && a.T[2] == b.T[2];
}

// Spread and interpolation at the same positions: one binning serves both
// when the plan's spread and interpolation tiles agree.
template <int KIND, int ORDER, int DIMS, int PREC>
ibk_status both_impl(Plan& plan, const OpArgs& a, const double* fl, CompPtrs fe, ConstCompPtrs ue, double* ul)
{
	using D = Delta<KIND, ORDER>;
	if (!plan.tiled) {
		ibk_status s = spread_direct<D, DIMS>(plan, a, fl, fe);
		return s != IBK_OK ? s : interp_direct<D, DIMS>(plan, a, ue, ul);
	}
	Binned b;
	constexpr bool fix = PREC == IBK_PRECISION_FP32C;
	ibk_status s = bin_points<D::M, DIMS>(plan, a, plan.spread_tiles, b, fix ? fl : nullptr);
	if (s != IBK_OK) return s;
	if ((s = launch_spread<D, DIMS, PREC>(plan, a, plan.spread_tiles, b, fl, fe)) != IBK_OK) return s;
	if (!same_tiles(plan.spread_tiles, plan.tiles)) {
		if ((s = bin_points<D::M, DIMS>(plan, a, plan.tiles, b)) != IBK_OK) return s;
	}
	return launch_interp<D, DIMS, PREC>(plan, a, plan.tiles, b, ue, ul);
}

template <int KIND, int ORDER, int DIMS>
ibk_status keys_impl(Plan& plan, const OpArgs& a, int comp, int* keys)
{
	using D = Delta<KIND, ORDER>;
	return launch(plan, "keys_kernel", a.stream, [&] {
		keys_kernel<D, DIMS><<<blocks_for(a.n, kThreads), kThreads, 0, a.stream>>>(*a.g, comp, a.n, a.x, keys);
	});
}

template <int KIND, int ORDER, int DIMS, int PREC>
constexpr OpTable make_table()
{
	return OpTable{&spread_impl<KIND, ORDER, DIMS, PREC>, &interp_impl<KIND, ORDER, DIMS, PREC>,
	               &keys_impl<KIND, ORDER, DIMS>, &both_impl<KIND, ORDER, DIMS, PREC>};
}

struct Entry { int kind, order, dims, prec; OpTable ops; };

#define IBK_ENTRY(K, O, DIM, PR) Entry{K, O, DIM, PR, make_table<K, O, DIM, PR>()}
#define IBK_DELTA_ENTRIES(DIM, PR)                                          \
	IBK_ENTRY(kBspline, 1, DIM, PR), IBK_ENTRY(kBspline, 2, DIM, PR),     \
	IBK_ENTRY(kBspline, 3, DIM, PR), IBK_ENTRY(kBspline, 4, DIM, PR),     \
	IBK_ENTRY(kBspline, 5, DIM, PR), IBK_ENTRY(kPeskin, 0, DIM, PR),      \
	IBK_ENTRY(kRoma, 0, DIM, PR), IBK_ENTRY(kCosine, 0, DIM, PR),         \
	IBK_ENTRY(kHat, 0, DIM, PR)

const Entry kTable[] = {
	IBK_DELTA_ENTRIES(2, IBK_PRECISION_FP64),
	IBK_DELTA_ENTRIES(3, IBK_PRECISION_FP64),
	IBK_DELTA_ENTRIES(2, IBK_PRECISION_FP32C),
	IBK_DELTA_ENTRIES(3, IBK_PRECISION_FP32C),
};

} // namespace

// Tile extent per axis: the preferred extent (by default 16 cells, or a
// quarter of a small axis, at least 8) where the last tile keeps at least M
// cells (a stencil can then reach at most one
// neighbour per side), otherwise the nearest size that does; an axis no
// longer than the preferred extent is one tile.
TileGeom make_tiles(const GridGeom& g, int tag, int M, const int* pref_extent)
{
	TileGeom tg{};
	tg.tag_mac = tag == IBK_TAG_MAC;
	tg.num_tiles = 1;
	const int minlast = M > 2 ? M : 2;
	for (int d = 0; d < kMaxDims; ++d) {
		if (d >= g.dims) { tg.T[d] = 1; tg.ntiles[d] = 1; tg.cells[d] = 1; continue; }
		const int cells = g.comp[0].cells[d];
		tg.cells[d] = cells;
		// default: 16 cells, but at least four tiles per axis on small grids
		// (extents of at least 8), so their work spreads over more CTAs
		const int want = pref_extent ? pref_extent[d] : std::min(16, std::max(8, cells / 4));
		int T = cells;
		if (cells > want) {
			static const int prefs[] = {16, 14, 18, 12, 20, 10, 8, 9, 11, 13, 15, 17, 19};
			T = 0;
			if (want != 16) {
				// the preferred extent, then its nearest neighbours (larger
				// first), then the regular ladder
				for (int dist = 0; dist <= 6 && T == 0; ++dist)
					for (int sgn = 1; sgn >= -1 && T == 0; sgn -= 2) {
						const int t = want + sgn * dist;
						if (t < minlast || t < 4 || t >= cells) continue;
						const int r = cells % t;
						if (r == 0 || r >= minlast) T = t;
					}
			}
			for (int i = 0; i < (int) (sizeof(prefs) / sizeof(prefs[0])) && T == 0; ++i) {
				const int r = cells % prefs[i];
				if (r == 0 || r >= minlast) T = prefs[i];
			}
			if (T == 0) T = 8;   // unreachable for M <= 6: some t in [8, 20] leaves r == 0 or r >= M
		}
		tg.T[d] = T;
		tg.ntiles[d] = (cells + T - 1) / T;
		tg.num_tiles *= tg.ntiles[d];
	}
	tg.nclass = ipow3(g.dims);
	tg.num_bins = tg.num_tiles * tg.nclass;
	return tg;
}

size_t spread_tile_bytes(const GridGeom& g, const TileGeom& tg, int kind, int order, int M, int precision)
{
	return spread_smem_bytes(g, tg, M, precision, spread64_owners(kind, order, g.dims));
}

size_t dense_tile_bytes(const TileGeom& tg, int dims) { return folded_layout(tg, dims).bytes; }

size_t spread_limit_bytes(const GridGeom& g, const TileGeom& tg, int M, int precision)
{
	return spread_tile_limit_bytes(g, tg, M, precision);
}

void interp_region(const GridGeom& g, const TileGeom& tg, int M, int c, int* lower, int* extent)
{
	switch (M) {
	case 2: region_of<2>(g, tg, c, lower, extent); return;
	case 3: region_of<3>(g, tg, c, lower, extent); return;
	case 4: region_of<4>(g, tg, c, lower, extent); return;
	case 5: region_of<5>(g, tg, c, lower, extent); return;
	case 6: region_of<6>(g, tg, c, lower, extent); return;
	}
}

size_t interp_region_bytes(const GridGeom& g, const TileGeom& tg, int M)
{
	switch (M) {
	case 2: return interp_smem_bytes<2>(g, tg);
	case 3: return interp_smem_bytes<3>(g, tg);
	case 4: return interp_smem_bytes<4>(g, tg);
	case 5: return interp_smem_bytes<5>(g, tg);
	case 6: return interp_smem_bytes<6>(g, tg);
	}
	return 0;
}

const OpTable* find_ops(int kind, int order, int dims, int precision)
{
	if (kind != kBspline) order = 0;
	for (const Entry& e : kTable)
		if (e.kind == kind && e.order == order && e.dims == dims && e.prec == precision)
			return &e.ops;
	return nullptr;
}

} // namespace ibk
