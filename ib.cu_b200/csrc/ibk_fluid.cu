// The fluid step that consumes the spread's force density: one implicit
// diffusion step of a component grid (ins::diffusion,
// include/ins/diffusion.h:12-78),
//     out = u + (I~ - lambda L)^-1 (k I~ f + k mu (L u + rhs)),
// with L the second-order finite-difference Laplacian and I~ the
// boundary-corrected identity (fd::laplacian, fd::identity with
// correction::second_order).  Both are Kronecker sums / products of 1-D
// operators (include/fd/combine.h:24-30): along an axis L_d is the 3-point
// Laplacian res^2 (1, -2, 1) with a wrap entry per corner on a periodic axis,
// or on a solid axis the ghost-point weight of each wall added to its corner
// diagonal, and I~_d is the identity plus each wall's second-order error
// coefficient on its corner (include/fd/laplacian.h:18-46,
// include/fd/identity.h:22-47, include/fd/discretization.h:47-80).  So
//     (L u)_ijk = Iz Iy (Lx u) + Iz (Ly u) Ix + (Lz u) Iy Ix,   I~ = Iz Iy Ix,
// a 7-point stencil whose coefficients differ from the interior only at the
// walls: applied matrix-free here.  The solve is the reference's
// preconditioned CG loop (include/solvers/pcg.h:12-45: stop when |d|_2 <=
// tolerance for the search direction d, bail out when <d, H d> is below
// tolerance^2) with the reference's preconditioner, a degree-4 Chebyshev
// polynomial in H = I~ - lambda L on its Gershgorin interval
// (include/solvers/chebpcg.h, include/solvers/preconditioners/chebyshev.h,
// include/algo/chebyshev.h, include/algo/gershgorin.h), or, selectable, a
// Jacobi preconditioner.  FP64, compiled without contraction; the kernels of
// the Chebyshev loop use fused multiply-adds, each written out.
#include <algorithm>
#include <cmath>
#include <string>
#include <type_traits>
#include <vector>
#include "ibk_internal.h"

namespace ibk {
namespace {

constexpr int kFluidThreads = 256;
constexpr int kFluidBlocks = 1184;          // 8 CTAs per SM on 148 SMs: fixed, so sums have one order

// 1-D operators of one axis: L (lo, diag, hi; lo[0] / hi[P-1] wrap on a
// periodic axis, else 0) and the corrected identity id.
struct AxisOps {
	const double* lo;
	const double* diag;
	const double* hi;
	const double* id;
	int P;
	int periodic;
};

struct FluidOps {
	AxisOps ax[3];
	int dims;
	long long size;
	double lambda;
};

// Axis coordinates of face idx (x fastest); 32-bit arithmetic below 2^31 faces.
__device__ __forceinline__ void face_coords(long long idx, int P0, int P1, int& i, int& j, int& k)
{
	if (idx < 0x7fffffffLL) {
		const unsigned u = (unsigned) idx, r = u / (unsigned) P0;
		i = (int) (u - r * (unsigned) P0);
		j = (int) (r % (unsigned) P1);
		k = (int) (r / (unsigned) P1);
	} else {
		i = (int) (idx % P0);
		const long long r = idx / P0;
		j = (int) (r % P1);
		k = (int) (r / P1);
	}
}

// op 0: L u, 1: I~ u, 2: H u with H = I~ - lambda L, 3: the right-hand side
// of the solve, k I~ f + kmu (L u + rhs0) (diffusion.h:51-53: gemv(1, L, u,
// 1, rhs), then gemv(k, I~, f, k mu, rhs)), per face
//     (L u) = Iz Iy (Lx u) + Iz (Ly u) Ix + (Lz u) Iy Ix
// with (L_d u) = lo u[-1] + diag u + hi u[+1] along axis d (wrapping on a
// periodic axis).  Each thread marches along z through zrun planes of one
// (x, y) column: its x and y coefficients and neighbour offsets are taken
// once, the z neighbours move through registers (one new load per face), and
// no face needs a division for its coordinates.  A block is 32 columns along
// x (one warp, coalesced) by 8 along y.  With dot != nullptr the per-block
// partial sums of u . out go to dot[block] (fixed order).  zrun is 16 where
// that gives four blocks per SM, else shorter (march_run): a 64^3 grid has
// only 64 blocks of 16 planes.
constexpr int kMarchX = 32, kMarchY = 8, kMarchZ = 16;

template <int OP, int DIMS>
__global__ void __launch_bounds__(kMarchX * kMarchY, 5)
march_apply_kernel(FluidOps o, const double* __restrict__ u, double* __restrict__ out, double* __restrict__ dot,
                   int zrun, const double* __restrict__ f, const double* __restrict__ rhs0, double kf, double kmu)
{
	constexpr int op = OP;
	__shared__ double red[kMarchY];
	const int P0 = o.ax[0].P;
	const int P1 = DIMS > 1 ? o.ax[1].P : 1;
	const int P2 = DIMS > 2 ? o.ax[2].P : 1;
	const int i = blockIdx.x * kMarchX + threadIdx.x;
	const int j = blockIdx.y * kMarchY + threadIdx.y;
	// two dimensions: one plane, and the compiler told so (1000 x 1000 faces: a
	// product took 11.4 us as a loop of up to 16 planes, 14.9 as one of any length, now
	// 10.6)
	const int k0 = DIMS > 2 ? blockIdx.z * zrun : 0;
	const int k1 = DIMS > 2 ? min(k0 + zrun, P2) : 1;
	double acc = 0.0;
	if (i < P0 && j < P1) {
		// 32-bit offsets: the plan's grids hold fewer than 2^31 faces
		const int sy = P0, sz = P0 * P1;
		const AxisOps& X = o.ax[0];
		const double ix = X.id[i], xl = X.lo[i], xd = X.diag[i], xh = X.hi[i];
		const bool has_xm = i > 0 || X.periodic, has_xp = i + 1 < P0 || X.periodic;
		const int dxm = i > 0 ? -1 : P0 - 1, dxp = i + 1 < P0 ? 1 : 1 - P0;
		double iy = 1.0, yl = 0.0, yd = 0.0, yh = 0.0;
		bool has_ym = false, has_yp = false;
		int dym = 0, dyp = 0;
		if (DIMS > 1) {
			const AxisOps& Y = o.ax[1];
			iy = Y.id[j]; yl = Y.lo[j]; yd = Y.diag[j]; yh = Y.hi[j];
			has_ym = j > 0 || Y.periodic;
			has_yp = j + 1 < P1 || Y.periodic;
			dym = j > 0 ? -sy : (P1 - 1) * sy;
			dyp = j + 1 < P1 ? sy : (1 - P1) * sy;
		}
		// z coefficients from one base: lo, diag, hi and id lie P2 apart
		const double* __restrict__ zc = o.ax[2].lo;
		const bool zper = o.ax[2].periodic;
		const int base = i + j * sy + k0 * sz;
		const double* __restrict__ pu = u + base;      // this column at plane k
		const double* __restrict__ pf = OP == 3 ? f + base : nullptr;
		const double* __restrict__ pr = OP == 3 ? rhs0 + base : nullptr;
		double* __restrict__ po = out + base;
		// register window along z: uzm, uc, uzp = planes k - 1, k, k + 1 (wrapped
		// on a periodic axis, 0 past a wall), and the plane after next loaded
		// one iteration ahead
		double uc = *pu;
		double uzm = 0.0, uzp = 0.0;
		if (DIMS > 2) {
			uzm = k0 > 0 ? pu[-sz] : (zper ? pu[(P2 - 1) * sz] : 0.0);
			uzp = k0 + 1 < P2 ? pu[sz] : (zper ? pu[(1 - P2) * sz] : 0.0);
		}
		for (int k = k0; k < k1; ++k) {
			double unx = 0.0;
			if (DIMS > 2 && k + 1 < k1)      // k + 2 <= P2: plane k + 2, or plane 0 past a periodic end
				unx = k + 2 < P2 ? pu[2 * sz] : (zper ? pu[(2 - P2) * sz] : 0.0);
			const double iz = DIMS > 2 ? zc[3 * P2 + k] : 1.0;
			double v = 0.0;
			if (op != 1) {
				const double um = has_xm ? pu[dxm] : 0.0, up = has_xp ? pu[dxp] : 0.0;
				double l = iz * iy * (xl * um + xd * uc + xh * up);
				if (DIMS > 1) {
					const double vm = has_ym ? pu[dym] : 0.0, vp = has_yp ? pu[dyp] : 0.0;
					l += iz * (yl * vm + yd * uc + yh * vp) * ix;
				}
				if (DIMS > 2) l += (zc[k] * uzm + zc[P2 + k] * uc + zc[2 * P2 + k] * uzp) * iy * ix;
				v = l;
			}
			if (op == 1) v = iz * iy * ix * uc;
			if (op == 2) v = iz * iy * ix * uc - o.lambda * v;
			if constexpr (OP == 3) {
				const double idf = iz * iy * ix * *pf;
				v = kf * idf + kmu * (v + *pr);
				pf += sz;
				pr += sz;
			}
			if (dot) acc += uc * v;
			*po = v;
			uzm = uc;
			uc = uzp;
			uzp = unx;
			pu += sz;
			po += sz;
		}
	}
	if (!dot) return;
	for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
	if (threadIdx.x == 0) red[threadIdx.y] = acc;
	__syncthreads();
	if (threadIdx.x == 0 && threadIdx.y == 0) {
		double t = 0.0;
		for (int w = 0; w < kMarchY; ++w) t += red[w];
		dot[blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z)] = t;
	}
}

// Planes per thread and grid of the marching operator.
struct March {
	dim3 grid;
	int zrun = kMarchZ;
	int blocks() const { return (int) (grid.x * grid.y * grid.z); }
};

template <int OP>
void launch_march_dims(const FluidOps& o, const March& m, const double* u, double* out, double* dot, const double* f,
                       const double* rhs0, double kf, double kmu, cudaStream_t s)
{
	const dim3 block(kMarchX, kMarchY);
	if (o.dims == 3) march_apply_kernel<OP, 3><<<m.grid, block, 0, s>>>(o, u, out, dot, m.zrun, f, rhs0, kf, kmu);
	else march_apply_kernel<OP, 2><<<m.grid, block, 0, s>>>(o, u, out, dot, m.zrun, f, rhs0, kf, kmu);
}

void launch_march(const FluidOps& o, int op, const March& m, const double* u, double* out, double* dot, cudaStream_t s,
                  const double* f = nullptr, const double* rhs0 = nullptr, double kf = 0.0, double kmu = 0.0)
{
	switch (op) {
	case 0: launch_march_dims<0>(o, m, u, out, dot, f, rhs0, kf, kmu, s); break;
	case 1: launch_march_dims<1>(o, m, u, out, dot, f, rhs0, kf, kmu, s); break;
	case 2: launch_march_dims<2>(o, m, u, out, dot, f, rhs0, kf, kmu, s); break;
	default: launch_march_dims<3>(o, m, u, out, dot, f, rhs0, kf, kmu, s); break;
	}
}

// Gershgorin interval of H = I~ - lambda L (algo/gershgorin.h:14-49): per
// block the smallest diagonal - sum |off-diagonal| and the largest diagonal
// + sum |off-diagonal| of its rows (minimum and maximum are exact in any
// order).  part: 2 per block.
__global__ void __launch_bounds__(kFluidThreads)
gershgorin_kernel(FluidOps o, double* __restrict__ part)
{
	__shared__ double smin[kFluidThreads], smax[kFluidThreads];
	double mn = INFINITY, mx = -INFINITY;
	const int P0 = o.ax[0].P, P1 = o.ax[1].P;
	for (long long idx = (long long) blockIdx.x * blockDim.x + threadIdx.x; idx < o.size;
	     idx += (long long) gridDim.x * blockDim.x) {
		int i, j, k;
		face_coords(idx, P0, P1, i, j, k);
		const double ix = o.ax[0].id[i], iy = o.dims > 1 ? o.ax[1].id[j] : 1.0;
		const double iz = o.dims > 2 ? o.ax[2].id[k] : 1.0;
		double l = iz * iy * o.ax[0].diag[i];
		if (o.dims > 1) l += iz * o.ax[1].diag[j] * ix;
		if (o.dims > 2) l += o.ax[2].diag[k] * iy * ix;
		const double diag = iz * iy * ix - o.lambda * l;
		double off = fabs(o.lambda * (iz * iy * o.ax[0].lo[i])) + fabs(o.lambda * (iz * iy * o.ax[0].hi[i]));
		if (o.dims > 1)
			off += fabs(o.lambda * (iz * o.ax[1].lo[j] * ix)) + fabs(o.lambda * (iz * o.ax[1].hi[j] * ix));
		if (o.dims > 2)
			off += fabs(o.lambda * (o.ax[2].lo[k] * iy * ix)) + fabs(o.lambda * (o.ax[2].hi[k] * iy * ix));
		mn = fmin(mn, diag - off);
		mx = fmax(mx, diag + off);
	}
	smin[threadIdx.x] = mn;
	smax[threadIdx.x] = mx;
	__syncthreads();
	for (int w = kFluidThreads / 2; w > 0; w >>= 1) {
		if (threadIdx.x < w) {
			smin[threadIdx.x] = fmin(smin[threadIdx.x], smin[threadIdx.x + w]);
			smax[threadIdx.x] = fmax(smax[threadIdx.x], smax[threadIdx.x + w]);
		}
		__syncthreads();
	}
	if (threadIdx.x == 0) {
		part[2 * blockIdx.x] = smin[0];
		part[2 * blockIdx.x + 1] = smax[0];
	}
}

// Reciprocal of the diagonal of I~ - lambda L (the Jacobi preconditioner).
__global__ void __launch_bounds__(kFluidThreads)
diagonal_kernel(FluidOps o, double* __restrict__ diag)
{
	const int P0 = o.ax[0].P, P1 = o.ax[1].P;
	for (long long idx = (long long) blockIdx.x * blockDim.x + threadIdx.x; idx < o.size;
	     idx += (long long) gridDim.x * blockDim.x) {
		int i, j, k;
		face_coords(idx, P0, P1, i, j, k);
		const double ix = o.ax[0].id[i], iy = o.dims > 1 ? o.ax[1].id[j] : 1.0;
		const double iz = o.dims > 2 ? o.ax[2].id[k] : 1.0;
		double l = iz * iy * o.ax[0].diag[i];
		if (o.dims > 1) l += iz * o.ax[1].diag[j] * ix;
		if (o.dims > 2) l += o.ax[2].diag[k] * iy * ix;
		diag[idx] = 1.0 / (iz * iy * ix - o.lambda * l);   // the preconditioner's reciprocal
	}
}

__device__ __forceinline__ void block_partial(double acc, double* __restrict__ out)
{
	__shared__ double red[kFluidThreads / 32];
	for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
	__syncthreads();
	if (threadIdx.x == 0) {
		double t = 0.0;
		for (int w = 0; w < kFluidThreads / 32; ++w) t += red[w];
		out[blockIdx.x] = t;
	}
}

// Sum of n per-block partials by one block of kSumThreads threads in a
// fixed order (strided per-thread sums, then a fixed tree); every thread
// returns the total.
constexpr int kSumThreads = 256;

__device__ __forceinline__ double sum_partials(const double* __restrict__ partial, int n)
{
	__shared__ double s[kSumThreads];
	double t = 0.0;
	for (int b = threadIdx.x; b < n; b += kSumThreads) t += partial[b];
	s[threadIdx.x] = t;
	__syncthreads();
	for (int w = kSumThreads / 2; w > 0; w >>= 1) {
		if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
		__syncthreads();
	}
	return s[0];
}

__global__ void __launch_bounds__(kSumThreads) sum_kernel(const double* __restrict__ partial, int n,
                                                          double* __restrict__ out)
{
	const double t = sum_partials(partial, n);
	if (threadIdx.x == 0) *out = t;
}

// Start of the loop: x = 0, d = M^-1 r (dinv: the reciprocal diagonal),
// partials of r . d and d . d.
__global__ void __launch_bounds__(kFluidThreads)
start_kernel(long long n, const double* __restrict__ r, const double* __restrict__ diag, double* __restrict__ x,
             double* __restrict__ d, double* __restrict__ rd, double* __restrict__ dd)
{
	double a = 0.0, b = 0.0;
	for (long long i = (long long) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x) {
		const double z = r[i] * diag[i];
		x[i] = 0.0;
		d[i] = z;
		a += r[i] * z;
		b += z * z;
	}
	block_partial(a, rd);
	__syncthreads();
	block_partial(b, dd);
}

// Device scalars of the loop (sc): [0] delta = r . M^-1 r, [1] nu = d . H d,
// [2] |d|^2, [3] alpha, [4] beta, [5] stop (0 running, else a Stop), [6]
// finished iterations (Chebyshev loop).
constexpr int kScalars = 8;
enum Stop { kBailOut = 1, kConverged = 2, kLimit = 3 };    // nu below tol^2; |d| <= tol; max_iterations

// nu from its partials; alpha = delta / nu, or stop (pcg.h:23-31).
__global__ void __launch_bounds__(kSumThreads) alpha_kernel(const double* __restrict__ partial, int n, double tol2,
                                                            double* __restrict__ sc)
{
	const double t = sum_partials(partial, n);
	if (threadIdx.x != 0) return;
	sc[1] = t;
	if (fabs(t) < tol2) { sc[5] = 1.0; sc[3] = 0.0; return; }
	sc[3] = sc[0] / t;
}

// delta_new from its partials; beta = delta_new / delta (pcg.h:36-39).
__global__ void __launch_bounds__(kSumThreads) beta_kernel(const double* __restrict__ partial, int n,
                                                           double* __restrict__ sc)
{
	if (sc[5] != 0.0) return;
	const double t = sum_partials(partial, n);
	if (threadIdx.x != 0) return;
	sc[4] = t / sc[0];
	sc[0] = t;
}

// x += alpha d, r -= alpha q, q = M^-1 r; partial sums of r . q.  Does
// nothing once the loop has stopped.
__global__ void __launch_bounds__(kFluidThreads, 8)
update_kernel(long long n, const double* __restrict__ sc, const double* __restrict__ d, double* __restrict__ q,
              double* __restrict__ x, double* __restrict__ r, const double* __restrict__ dinv, double* __restrict__ rq)
{
	if (sc[5] != 0.0) return;
	const double alpha = sc[3];
	double a = 0.0;
	for (long long i = (long long) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x) {
		x[i] += alpha * d[i];
		const double ri = r[i] - alpha * q[i];
		r[i] = ri;
		const double z = ri * dinv[i];
		q[i] = z;
		a += ri * z;
	}
	block_partial(a, rq);
}

// d = q + beta d; partial sums of d . d.
__global__ void __launch_bounds__(kFluidThreads)
direction_kernel(long long n, const double* __restrict__ sc, const double* __restrict__ q, double* __restrict__ d,
                 double* __restrict__ dd)
{
	if (sc[5] != 0.0) return;
	const double beta = sc[4];
	double a = 0.0;
	for (long long i = (long long) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x) {
		const double v = q[i] + beta * d[i];
		d[i] = v;
		a += v * v;
	}
	block_partial(a, dd);
}

// ------------------------------------------ Chebyshev-preconditioned loop
// One iteration is two kernels, each a tile of (x, y) columns marched along
// z, with the plane that the x and y neighbours come from in shared memory
// (two buffers, one barrier per plane) and the z neighbours in registers:
//   direction_apply_kernel  d' = z + beta d, x += alpha d, q = H d' and the
//                           sums of d' . q and d' . d'; the stopping tests'
//                           outcome also goes to the host's memory
//   polynomial_kernel       r' = r - alpha q, z = p(H) r' (the three steps
//                           s <- w_i r' - H s of the degree-4 polynomial in
//                           one pass, on a halo of 3) and the sum of r' . z
// Both write r and d to the other of two buffers: neighbouring blocks still
// read the old values on their halos.  The last block to finish adds up the
// blocks' partial sums in block order (so every run has the same bits) and
// forms alpha or beta and the stopping tests there.  HBM traffic per face and
// iteration: 48 + 32 bytes (one kernel per operator product, update and
// direction moved 152).  The products use fused multiply-adds with lambda
// folded into the coefficients; the operators themselves
// (march_apply_kernel) keep the reference's operation order.  Grids of two
// dimensions have kernels of their own (direction_plane_kernel,
// polynomial_plane_kernel): one plane, nothing to march.

// Index of an extended coordinate on an axis: wrapped on a periodic axis, -1
// outside a wall.
__device__ __forceinline__ int fold_index(const AxisOps& a, int v)
{
	if (a.periodic) {
		v %= a.P;
		return v < 0 ? v + a.P : v;
	}
	return v >= 0 && v < a.P ? v : -1;
}

// One axis' coefficients at index v of -lambda L and I~; all 0 for v < 0
// (nothing of the grid there: such a face stays 0 through every step) and for
// an axis the run does not have, but for id = 1 at v = 0.
struct AxisCoef { double lo, diag, hi, id; };

__device__ __forceinline__ AxisCoef axis_coef(const AxisOps& a, bool present, double lambda, int v)
{
	if (v < 0) return {0.0, 0.0, 0.0, 0.0};
	if (!present) return {0.0, 0.0, 0.0, 1.0};
	return {-lambda * __ldg(a.lo + v), -lambda * __ldg(a.diag + v), -lambda * __ldg(a.hi + v), __ldg(a.id + v)};
}

// Sums over the block, in a fixed order: valid in thread 0.
template <int NT, int N>
__device__ __forceinline__ void block_sums(double* v)
{
	__shared__ double red[N][NT / 32];
#pragma unroll
	for (int q = 0; q < N; ++q) {
		for (int s = 16; s > 0; s >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], s);
		if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = v[q];
	}
	__syncthreads();
	if (threadIdx.x == 0) {
#pragma unroll
		for (int q = 0; q < N; ++q) {
			double t = 0.0;
			for (int w = 0; w < NT / 32; ++w) t += red[q][w];
			v[q] = t;
		}
	}
	__syncthreads();
}

// Leaves the block's N sums in part and returns true in every thread of the
// last block to do so, with the totals over all blocks in v of thread 0.
// done: zero before the launch and after it.
template <int NT, int N>
__device__ __forceinline__ bool grid_sums(double* v, double* part, unsigned* done)
{
	__shared__ bool last;
	const int nblocks = gridDim.x * gridDim.y * gridDim.z;
	block_sums<NT, N>(v);
	if (threadIdx.x == 0) {
		const int b = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
#pragma unroll
		for (int q = 0; q < N; ++q) __stcg(part + (size_t) q * nblocks + b, v[q]);
		__threadfence();
		last = atomicAdd(done, 1u) == (unsigned) nblocks - 1u;
	}
	__syncthreads();
	if (!last) return false;
	__threadfence();
#pragma unroll
	for (int q = 0; q < N; ++q) {
		v[q] = 0.0;
		for (int b = threadIdx.x; b < nblocks; b += NT) v[q] += __ldcg(part + (size_t) q * nblocks + b);
	}
	block_sums<NT, N>(v);
	if (threadIdx.x == 0) *done = 0u;
	return true;
}

// Points an axis has at least: the tiles' halos then reach no further than one
// period past an end.
constexpr int kMinPoints = 3;

// Plane p on the z axis, at most kMinPoints planes past its ends: wrapped on a
// periodic axis, -1 outside a wall.
__device__ __forceinline__ int fold_plane(const AxisOps& a, int p)
{
	if (p < 0) return a.periodic ? p + a.P : -1;
	if (p >= a.P) return a.periodic ? p - a.P : -1;
	return p;
}

// Whether the faces lo .. hi of an axis all carry the interior's coefficients
// and exist: no wall in reach.
__device__ __forceinline__ bool alike(const AxisOps& a, int lo, int hi)
{
	return a.periodic || (lo >= 1 && hi <= a.P - 2);
}

// H at a face in two parts: partial() without the plane above (c the face's
// value, then its neighbours left, right, in the rows before and after and in
// the plane below), and the weight top() of the plane above.  Row and plane
// index the block's tables.  Three forms, by what walls a block can reach:
// none (one weight for the face and one for its six neighbours, and no
// coefficient to load),
struct UniformH {
	static constexpr bool uniform = true;       // every column and plane in reach is on the grid
	double centre, side;
	__device__ __forceinline__ UniformH(const FluidOps& o, const AxisCoef& cx, const AxisCoef*, const AxisCoef*)
		: centre(1.0 + o.dims * cx.diag), side(cx.lo) {}
	__device__ __forceinline__ double partial(int, int, double c, double xm, double xp, double ym, double yp, double zm) const
	{
		return __fma_rn(centre, c, side * (((xm + xp) + (ym + yp)) + zm));
	}
	__device__ __forceinline__ double top(int, int) const { return side; }
	__device__ __forceinline__ double plane(int, double c, double xm, double xp, double ym, double yp) const
	{
		return __fma_rn(centre, c, side * ((xm + xp) + (ym + yp)));
	}
};

// walls along y only (a channel),
struct WallYH {
	static constexpr bool uniform = false;
	double centre, side;
	const AxisCoef* yt;
	__device__ __forceinline__ WallYH(const FluidOps&, const AxisCoef& cx, const AxisCoef* y, const AxisCoef*)
		: centre(1.0 + 2.0 * cx.diag), side(cx.lo), yt(y) {}
	__device__ __forceinline__ double partial(int row, int, double c, double xm, double xp, double ym, double yp,
	                                          double zm) const
	{
		const AxisCoef y = yt[row];
		const double xz = __fma_rn(centre, c, side * ((xm + xp) + zm));
		return __fma_rn(y.id, xz, __fma_rn(y.hi, yp, __fma_rn(y.lo, ym, y.diag * c)));
	}
	__device__ __forceinline__ double top(int row, int) const { return side * yt[row].id; }
};

// and any.
struct GeneralH {
	static constexpr bool uniform = false;
	AxisCoef x;
	const AxisCoef *yt, *zt;
	__device__ __forceinline__ GeneralH(const FluidOps&, const AxisCoef& cx, const AxisCoef* y, const AxisCoef* z)
		: x(cx), yt(y), zt(z) {}
	__device__ __forceinline__ double partial(int row, int plane, double c, double xm, double xp, double ym, double yp,
	                                          double zm) const
	{
		const AxisCoef y = yt[row], z = zt[plane];
		const double ax = __fma_rn(x.hi, xp, __fma_rn(x.lo, xm, (x.id + x.diag) * c));
		const double ay = __fma_rn(y.hi, yp, __fma_rn(y.lo, ym, y.diag * c));
		const double az = __fma_rn(z.lo, zm, z.diag * c);
		return __fma_rn(x.id * y.id, az, z.id * __fma_rn(x.id, ay, y.id * ax));
	}
	__device__ __forceinline__ double top(int row, int plane) const { return x.id * yt[row].id * zt[plane].hi; }
};

// In two dimensions H at a face is one expression, plane(): UniformH's, or this
// one where the block reaches a wall.
struct PlaneH {
	AxisCoef x;
	const AxisCoef* yt;
	__device__ __forceinline__ PlaneH(const AxisCoef& cx, const AxisCoef* y) : x(cx), yt(y) {}
	__device__ __forceinline__ double plane(int row, double c, double xm, double xp, double ym, double yp) const
	{
		const AxisCoef y = yt[row];
		const double ax = __fma_rn(x.hi, xp, __fma_rn(x.lo, xm, (x.id + x.diag) * c));
		const double ay = __fma_rn(y.hi, yp, __fma_rn(y.lo, ym, y.diag * c));
		return __fma_rn(x.id, ay, y.id * ax);
	}
};

// The coefficients of `count` faces from `first` on along an axis.
__device__ __forceinline__ void fill_table(const FluidOps& o, int axis, int first, int count, AxisCoef* t)
{
	for (int i = threadIdx.x; i < count; i += blockDim.x)
		t[i] = axis_coef(o.ax[axis], axis < o.dims, o.lambda, fold_index(o.ax[axis], first + i));
}

// After a direction: the loop test of pcg.h:21, then alpha or the bail-out of
// pcg.h:23-31; sums: d . H d and d . d.
__device__ __forceinline__ void judge(const double* sums, double* sc, double tol, int max_iterations, double* host)
{
	sc[1] = sums[0];
	sc[2] = sums[1];
	if (!(sqrt(sums[1]) > tol)) sc[5] = kConverged;
	else if (sc[6] >= (double) max_iterations) sc[5] = kLimit;
	else if (fabs(sums[0]) < tol * tol) sc[5] = kBailOut;
	else sc[3] = sc[0] / sums[0];
	host[0] = sc[5];
	host[1] = sc[6];
}

// After a polynomial: delta = r . z, and beta but for the first.
__device__ __forceinline__ void advance(double delta, double* sc, int first)
{
	if (first) {
		sc[0] = delta;              // pcg.h:14-18: delta = r . d
	} else {
		sc[4] = delta / sc[0];      // pcg.h:36-39: beta = delta' / delta
		sc[0] = delta;
		sc[6] += 1.0;
	}
}

// Time of one step of polynomial_kernel's wide tile over the others' (see
// PolyWide).
constexpr double kWideStep = 1.75;

// Longest run of planes per block (bounds the tables along z).
constexpr int kMaxRun = 64;

// direction_apply_kernel's tile: 64 x 16 columns, 256 threads with four
// neighbouring rows each; the first 160 threads also hold one column each of
// the halo.  Bound by HBM: 48 bytes per face, the next plane's z, d and x
// loaded a plane ahead.  512 x 256 x 512 faces: 511 us, 6.3 TB/s (operator,
// half the update and the direction as passes of their own: 336 + 237 + 241
// us; 64 x 8 columns with two rows a thread, three CTAs per SM: 551 us, and 2
// to 5 % more with four CTAs, which spill).
constexpr int kDirX = 64, kDirY = 16, kDirRows = 4, kDirThreads = 256, kDirBlocks = 2;
constexpr int kDirStride = kDirX + 2;

__global__ void __launch_bounds__(kDirThreads, kDirBlocks)
direction_apply_kernel(FluidOps o, double* __restrict__ sc, const double* __restrict__ z,
                       const double* __restrict__ dold, double* __restrict__ dnew, double* __restrict__ x,
                       double* __restrict__ q, double* __restrict__ part, unsigned* __restrict__ done, int zrun,
                       int first, double tol, int max_iterations, double* __restrict__ host)
{
	if (sc[5] != 0.0) return;
	__shared__ double plane[2][(kDirY + 2) * kDirStride];
	__shared__ AxisCoef zt[kMaxRun];
	__shared__ AxisCoef yt[kDirY];
	const double alpha = sc[3], beta = sc[4];
	const int P0 = o.ax[0].P, P1 = o.ax[1].P;
	const int tx = threadIdx.x % kDirX, ty = threadIdx.x / kDirX;
	const int x0 = blockIdx.x * kDirX, y0 = blockIdx.y * kDirY;
	const int k0 = blockIdx.z * zrun, k1 = min(k0 + zrun, o.ax[2].P);
	const int sz = P0 * P1;

	const int gi = fold_index(o.ax[0], x0 + tx);
	int off[kDirRows];          // the column's offset in a plane, -1 outside
	bool own[kDirRows];         // this block writes it
#pragma unroll
	for (int c = 0; c < kDirRows; ++c) {
		const int y = y0 + ty * kDirRows + c;
		const int gj = fold_index(o.ax[1], y);
		off[c] = gi >= 0 && gj >= 0 ? gi + gj * P0 : -1;
		own[c] = x0 + tx < P0 && y < P1;
	}
	// halo columns: the rows above and below, then the columns left and right
	int hoff = -1, hslot = -1;
	if (threadIdx.x < 2 * kDirX + 2 * kDirY) {
		const int t = threadIdx.x, h = t - 2 * kDirX;
		const int ex = h < 0 ? t % kDirX : (h < kDirY ? -1 : kDirX);
		const int ey = h < 0 ? (t < kDirX ? -1 : kDirY) : h % kDirY;
		hslot = (ey + 1) * kDirStride + ex + 1;
		const int hi = fold_index(o.ax[0], x0 + ex), hj = fold_index(o.ax[1], y0 + ey);
		if (hi >= 0 && hj >= 0) hoff = hi + hj * P0;
	}
	const int slot = (ty * kDirRows + 1) * kDirStride + tx + 1;
	double sums[2] = {0.0, 0.0};

	auto march = [&](const auto& H) {
		constexpr bool uniform = std::decay_t<decltype(H)>::uniform;
		// loads of one plane, a plane ahead of their use
		double zv[kDirRows], dv[kDirRows], xv[kDirRows], hz = 0.0, hd = 0.0;
		auto fetch = [&](int p, bool inner) {
			const int g = fold_plane(o.ax[2], p);
			const double *zp = z + (long long) g * sz, *dp = dold + (long long) g * sz;
#pragma unroll
			for (int c = 0; c < kDirRows; ++c) {
				const bool on = uniform || (g >= 0 && off[c] >= 0);
				zv[c] = on ? __ldg(zp + off[c]) : 0.0;
				dv[c] = on && !first ? __ldg(dp + off[c]) : 0.0;
				xv[c] = inner && own[c] && !first ? x[g * sz + off[c]] : 0.0;
			}
			if (hslot >= 0) {
				const bool hon = uniform || (g >= 0 && hoff >= 0);
				hz = hon ? __ldg(zp + hoff) : 0.0;
				hd = hon && !first ? __ldg(dp + hoff) : 0.0;
			}
		};
		// plane k of d': registers and shared buffer k & 1; d' and x written
		auto take = [&](int k, bool inner, double* v) {
			double* buf = plane[k & 1];
#pragma unroll
			for (int c = 0; c < kDirRows; ++c) {
				v[c] = __fma_rn(beta, dv[c], zv[c]);
				buf[slot + c * kDirStride] = v[c];
				if (inner && own[c]) {
					dnew[k * sz + off[c]] = v[c];
					x[k * sz + off[c]] = __fma_rn(alpha, dv[c], xv[c]);
				}
			}
			if (hslot >= 0) buf[hslot] = __fma_rn(beta, hd, hz);
		};
		double vm[kDirRows], vc[kDirRows], vn[kDirRows];
		fetch(k0 - 1, false);
#pragma unroll
		for (int c = 0; c < kDirRows; ++c) vm[c] = __fma_rn(beta, dv[c], zv[c]);
		fetch(k0, true);
		take(k0, true, vc);
		fetch(k0 + 1, k0 + 1 < k1);
		for (int k = k0; k < k1; ++k) {
			__syncthreads();            // plane k is complete; every read of plane k - 1 is done
			take(k + 1, k + 1 < k1, vn);
			if (k + 1 < k1) fetch(k + 2, k + 2 < k1);
			const double* buf = plane[k & 1];
#pragma unroll
			for (int c = 0; c < kDirRows; ++c) {
				const int at = slot + c * kDirStride;
				const double ym = c > 0 ? vc[c - 1] : buf[at - kDirStride];
				const double yp = c + 1 < kDirRows ? vc[c + 1] : buf[at + kDirStride];
				const int row = ty * kDirRows + c;
				const double h = __fma_rn(H.top(row, k - k0), vn[c],
				                          H.partial(row, k - k0, vc[c], buf[at - 1], buf[at + 1], ym, yp, vm[c]));
				if (own[c]) {
					q[k * sz + off[c]] = h;
					sums[0] = __fma_rn(vc[c], h, sums[0]);
					sums[1] = __fma_rn(vc[c], vc[c], sums[1]);
				}
			}
#pragma unroll
			for (int c = 0; c < kDirRows; ++c) { vm[c] = vc[c]; vc[c] = vn[c]; }
		}
	};
	const AxisCoef cx = axis_coef(o.ax[0], true, o.lambda, gi);
	if (alike(o.ax[0], x0 - 1, x0 + kDirX) && alike(o.ax[1], y0 - 1, y0 + kDirY) && alike(o.ax[2], k0 - 1, k1)) {
		march(UniformH(o, cx, yt, zt));
	} else {
		fill_table(o, 1, y0, kDirY, yt);
		fill_table(o, 2, k0, k1 - k0, zt);
		if (alike(o.ax[0], x0 - 1, x0 + kDirX) && alike(o.ax[2], k0 - 1, k1))
			march(WallYH(o, cx, yt, zt));
		else
			march(GeneralH(o, cx, yt, zt));     // the first barrier comes before the tables are read
	}
	if (grid_sums<kDirThreads, 2>(sums, part, done) && threadIdx.x == 0) judge(sums, sc, tol, max_iterations, host);
}

// The same in two dimensions: one plane, no march, the arrays mostly in L2.
__global__ void __launch_bounds__(kDirThreads, 4)
direction_plane_kernel(FluidOps o, double* __restrict__ sc, const double* __restrict__ z,
                       const double* __restrict__ dold, double* __restrict__ dnew, double* __restrict__ x,
                       double* __restrict__ q, double* __restrict__ part, unsigned* __restrict__ done, int first,
                       double tol, int max_iterations, double* __restrict__ host)
{
	if (sc[5] != 0.0) return;
	__shared__ double plane[(kDirY + 2) * kDirStride];
	__shared__ AxisCoef yt[kDirY];
	const double alpha = sc[3], beta = sc[4];
	const int P0 = o.ax[0].P, P1 = o.ax[1].P;
	const int tx = threadIdx.x % kDirX, ty = threadIdx.x / kDirX;
	const int x0 = blockIdx.x * kDirX, y0 = blockIdx.y * kDirY;
	const int gi = fold_index(o.ax[0], x0 + tx);
	const int slot = (ty * kDirRows + 1) * kDirStride + tx + 1;
	int off[kDirRows];
	bool own[kDirRows];
	double v[kDirRows], sums[2] = {0.0, 0.0};
#pragma unroll
	for (int c = 0; c < kDirRows; ++c) {
		const int y = y0 + ty * kDirRows + c, gj = fold_index(o.ax[1], y);
		const bool on = gi >= 0 && gj >= 0;
		own[c] = x0 + tx < P0 && y < P1;
		off[c] = on ? gi + gj * P0 : 0;
		const double d = on && !first ? __ldg(dold + off[c]) : 0.0;
		v[c] = __fma_rn(beta, d, on ? __ldg(z + off[c]) : 0.0);
		plane[slot + c * kDirStride] = v[c];
		if (own[c]) {
			dnew[off[c]] = v[c];
			x[off[c]] = __fma_rn(alpha, d, first ? 0.0 : x[off[c]]);
		}
	}
	if (threadIdx.x < 2 * kDirX + 2 * kDirY) {      // the rows above and below, the columns left and right
		const int t = threadIdx.x, h = t - 2 * kDirX;
		const int ex = h < 0 ? t % kDirX : (h < kDirY ? -1 : kDirX);
		const int ey = h < 0 ? (t < kDirX ? -1 : kDirY) : h % kDirY;
		const int hi = fold_index(o.ax[0], x0 + ex), hj = fold_index(o.ax[1], y0 + ey);
		const bool on = hi >= 0 && hj >= 0;
		const int at = on ? hi + hj * P0 : 0;
		const double d = on && !first ? __ldg(dold + at) : 0.0;
		plane[(ey + 1) * kDirStride + ex + 1] = __fma_rn(beta, d, on ? __ldg(z + at) : 0.0);
	}
	auto apply = [&](const auto& H) {
#pragma unroll
		for (int c = 0; c < kDirRows; ++c) {
			const int at = slot + c * kDirStride;
			const double h = H.plane(ty * kDirRows + c, v[c], plane[at - 1], plane[at + 1],
			                         c > 0 ? v[c - 1] : plane[at - kDirStride],
			                         c + 1 < kDirRows ? v[c + 1] : plane[at + kDirStride]);
			if (own[c]) {
				q[off[c]] = h;
				sums[0] = __fma_rn(v[c], h, sums[0]);
				sums[1] = __fma_rn(v[c], v[c], sums[1]);
			}
		}
	};
	const AxisCoef cx = axis_coef(o.ax[0], true, o.lambda, gi);
	if (alike(o.ax[0], x0 - 1, x0 + kDirX) && alike(o.ax[1], y0 - 1, y0 + kDirY)) {
		__syncthreads();
		apply(UniformH(o, cx, yt, yt));
	} else {
		fill_table(o, 1, y0, kDirY, yt);
		__syncthreads();
		apply(PlaneH(cx, yt));
	}
	if (grid_sums<kDirThreads, 2>(sums, part, done) && threadIdx.x == 0) judge(sums, sc, tol, max_iterations, host);
}

// polynomial_kernel's tile: EX x TY * ROWS columns, of which the inner ones (a
// halo of 3) are the block's own, EX x TY threads with ROWS neighbouring rows
// each.  At step p the block takes plane p of r' and finishes the first
// step's plane p - 1, the second's p - 2 and the third's p - 3, each from the
// part that was formed as soon as the planes below were there: what follows
// the barrier is three independent parts.  Columns and planes at the rim of
// the halo hold values that nothing inside uses.  512 x 256 x 512 faces: 687 us
// (the three steps and half the update as passes of their own: 450 + 2 x 473 +
// 237 us), against 330 us for its 32 bytes per face: what bounds it is the
// shared-memory pipe (about 60 % of its peak: 11 64-bit accesses per column
// and plane) and FP64 issue (26 %) taking turns between barriers, at one CTA of
// 128 registers per thread.
template <int EX_, int TY_, int ROWS_, int BLOCKS_>
struct PolyTile {
	static constexpr int EX = EX_, TY = TY_, ROWS = ROWS_, BLOCKS = BLOCKS_, HALO = 3;
	static constexpr int EY = TY * ROWS, X = EX - 2 * HALO, Y = EY - 2 * HALO, THREADS = EX * TY;
	static constexpr int PLANE = EX * EY;
	static_assert(THREADS % 32 == 0, "whole warps");
	static_assert(HALO <= kMinPoints, "fold_plane adds or subtracts one period");
};
// Of the wide tile's columns 74 % are the block's own, of the small and the
// tall tile's half; these have four times the blocks.  Milliseconds a solve,
// wide / small: 512 x 256 x 512 faces 18.3 / 22.7, 256 x 128 x 256 2.86 / 3.26, 160^3
// 1.60 / 1.92, 128^3 1.06 / 1.04, 112^3 0.77 / 0.87, 104^3 0.69 / 0.72, 96^3 0.66 / 0.63,
// 64^3 0.47 / 0.41, 8 x 512 x 512 3.05 / 2.49.  The cost that pick_run gives is
// 1.53 times the wide tile's for the small one at 96^3, 1.71 at 128^3, 1.80 at
// 104^3: the line lies between the last two.  The tall tile is for grids of a
// few faces along x, most of which the small one spends on columns past the
// end.
using PolyWide = PolyTile<64, 8, 4, 1>;
using PolySmall = PolyTile<32, 16, 1, 2>;
using PolyTall = PolyTile<16, 32, 1, 2>;
enum PolyKind { kPolyWide, kPolySmall, kPolyTall };
template <typename T> constexpr int poly_bytes() { return 6 * T::PLANE * (int) sizeof(double); }

struct ChebWeights { double w[4]; };

template <typename T>
__global__ void __launch_bounds__(T::THREADS, T::BLOCKS)
polynomial_kernel(FluidOps o, double* __restrict__ sc, const double* __restrict__ r, const double* __restrict__ q,
                  double* __restrict__ rnew, double* __restrict__ z, double* __restrict__ part,
                  unsigned* __restrict__ done, int zrun, int first, ChebWeights cw)
{
	if (sc[5] != 0.0) return;
	extern __shared__ double poly_planes[];     // r', first and second step: two buffers each
	__shared__ AxisCoef zt[kMaxRun + 2 * T::HALO];
	__shared__ AxisCoef yt[T::EY];
	const double alpha = sc[3];
	const int P0 = o.ax[0].P, P1 = o.ax[1].P;
	const int tx = threadIdx.x % T::EX, ty = threadIdx.x / T::EX;
	const int ex0 = (int) blockIdx.x * T::X - T::HALO, ey0 = (int) blockIdx.y * T::Y - T::HALO;
	const int k0 = blockIdx.z * zrun, k1 = min(k0 + zrun, o.ax[2].P);
	const int sz = P0 * P1;

	const int gi = fold_index(o.ax[0], ex0 + tx);
	int off[T::ROWS];
	bool own[T::ROWS];
#pragma unroll
	for (int c = 0; c < T::ROWS; ++c) {
		const int ey = ty * T::ROWS + c, y = ey0 + ey;
		const int gj = fold_index(o.ax[1], y);
		off[c] = gi >= 0 && gj >= 0 ? gi + gj * P0 : -1;
		own[c] = tx >= T::HALO && tx < T::HALO + T::X && ex0 + tx < P0 && ey >= T::HALO &&
		         ey < T::HALO + T::Y && y < P1;
	}
	const int slot = ty * T::ROWS * T::EX + tx;
	const int left = tx > 0 ? -1 : 0, right = tx + 1 < T::EX ? 1 : 0;
	const int above = ty > 0 ? -T::EX : 0, below = ty + 1 < T::TY ? T::EX : 0;
	double sums[1] = {0.0};

	auto march = [&](const auto& H) {
		constexpr bool uniform = std::decay_t<decltype(H)>::uniform;
		double rv[T::ROWS], qv[T::ROWS];
		auto fetch = [&](int p) {
			const int g = fold_plane(o.ax[2], p);
			const double *rp = r + (long long) g * sz, *qp = q + (long long) g * sz;
#pragma unroll
			for (int c = 0; c < T::ROWS; ++c) {
				const bool on = uniform || (g >= 0 && off[c] >= 0);
				rv[c] = on ? __ldg(rp + off[c]) : 0.0;
				qv[c] = on && !first ? __ldg(qp + off[c]) : 0.0;
			}
		};
		// the part of w v - ws H s at plane k that does not need plane k + 1, for
		// this thread's columns: s and sm its values at planes k and k - 1, buf the
		// shared copy of plane k; above() adds the rest
		auto below_part = [&](const double* buf, int k, double w, double ws, const double* v, const double* s,
		                      const double* sm, double* out) {
#pragma unroll
			for (int c = 0; c < T::ROWS; ++c) {
				const int at = slot + c * T::EX;
				const double ym = c > 0 ? s[c - 1] : buf[at + above];
				const double yp = c + 1 < T::ROWS ? s[c + 1] : buf[at + below];
				const double h = H.partial(ty * T::ROWS + c, k - k0 + T::HALO, s[c], buf[at + left], buf[at + right], ym,
				                           yp, sm[c]);
				out[c] = __fma_rn(w, v[c], -ws * h);
			}
		};
		auto add_above = [&](int k, double ws, const double* part_, const double* sp, double* out) {
#pragma unroll
			for (int c = 0; c < T::ROWS; ++c)
				out[c] = __fma_rn(-ws * H.top(ty * T::ROWS + c, k - k0 + T::HALO), sp[c], part_[c]);
		};
		// r' at planes p - 1 .. p - 3, the first step at p - 2, the second at p -
		// 3, and the three steps' parts at p - 1, p - 2, p - 3
		double v1[T::ROWS] = {}, v2[T::ROWS] = {}, v3[T::ROWS] = {}, am[T::ROWS] = {}, bm[T::ROWS] = {};
		double pa[T::ROWS] = {}, pb[T::ROWS] = {}, pz[T::ROWS] = {};
		fetch(k0 - T::HALO);
		for (int p = k0 - T::HALO; p < k1 + T::HALO; ++p) {
			double v0[T::ROWS], a1[T::ROWS], b2[T::ROWS], out[T::ROWS];
			double* buf = poly_planes + (p & 1) * (3 * T::PLANE);
#pragma unroll
			for (int c = 0; c < T::ROWS; ++c) v0[c] = __fma_rn(-alpha, qv[c], rv[c]);
			if (p + 1 < k1 + T::HALO) fetch(p + 1);
			add_above(max(p - 1, k0 - T::HALO), cw.w[0], pa, v0, a1);
			add_above(max(p - 2, k0 - T::HALO), 1.0, pb, a1, b2);
			add_above(max(p - 3, k0 - T::HALO), 1.0, pz, b2, out);
#pragma unroll
			for (int c = 0; c < T::ROWS; ++c) {
				const int at = slot + c * T::EX;
				buf[at] = v0[c];
				buf[T::PLANE + at] = a1[c];
				buf[2 * T::PLANE + at] = b2[c];
			}
			if (p - 3 >= k0) {
#pragma unroll
				for (int c = 0; c < T::ROWS; ++c)
					if (own[c]) {
						const int at = (p - 3) * sz + off[c];
						rnew[at] = v3[c];
						z[at] = out[c];
						sums[0] = __fma_rn(v3[c], out[c], sums[0]);
					}
			}
			__syncthreads();        // this step's planes are complete; the other buffer's reads are done
			below_part(buf, p, cw.w[1], cw.w[0], v0, v0, v1, pa);
			below_part(buf + T::PLANE, max(p - 1, k0 - T::HALO), cw.w[2], 1.0, v1, a1, am, pb);
			below_part(buf + 2 * T::PLANE, max(p - 2, k0 - T::HALO), cw.w[3], 1.0, v2, b2, bm, pz);
#pragma unroll
			for (int c = 0; c < T::ROWS; ++c) {
				v3[c] = v2[c]; v2[c] = v1[c]; v1[c] = v0[c];
				am[c] = a1[c];
				bm[c] = b2[c];
			}
		}
	};
	const AxisCoef cx = axis_coef(o.ax[0], true, o.lambda, gi);
	if (alike(o.ax[0], ex0, ex0 + T::EX - 1) && alike(o.ax[1], ey0, ey0 + T::EY - 1) &&
	    alike(o.ax[2], k0 - T::HALO, k1 + T::HALO - 1)) {
		march(UniformH(o, cx, yt, zt));
	} else {
		fill_table(o, 1, ey0, T::EY, yt);
		fill_table(o, 2, k0 - T::HALO, k1 - k0 + 2 * T::HALO, zt);
		__syncthreads();
		if (alike(o.ax[0], ex0, ex0 + T::EX - 1) && alike(o.ax[2], k0 - T::HALO, k1 + T::HALO - 1))
			march(WallYH(o, cx, yt, zt));
		else
			march(GeneralH(o, cx, yt, zt));
	}
	if (grid_sums<T::THREADS, 1>(sums, part, done) && threadIdx.x == 0) advance(sums[0], sc, first);
}

// The same in two dimensions: the three steps one after the other on the block's
// columns, a barrier each.  A march of one plane through the kernel above
// takes seven plane steps, every block of them in GeneralH: a solve of 11
// iterations on 2400 x 600 faces took 2079 us (one kernel per product, before
// the fused loop: 1172), now 694; 1000 x 1000 1548 (998), now 534; 240 x 120 304
// (618), now 252.  Wide against small tiles: 96 x 96 faces 236 / 213 us, 256 x 256
// 265 / 256 (260 small blocks), 400 x 400 279 / 290 (640), 600 x 600 307 / 380,
// 2400 x 600 694 / 888.
using PlaneWide = PolyTile<64, 8, 4, 2>;
using PlaneSmall = PolyTile<32, 16, 1, 4>;

template <typename T>
__global__ void __launch_bounds__(T::THREADS, T::BLOCKS)
polynomial_plane_kernel(FluidOps o, double* __restrict__ sc, const double* __restrict__ r, const double* __restrict__ q,
                        double* __restrict__ rnew, double* __restrict__ z, double* __restrict__ part,
                        unsigned* __restrict__ done, int first, ChebWeights cw)
{
	if (sc[5] != 0.0) return;
	__shared__ double planes[2][T::PLANE];      // r' and the second step, the first step
	__shared__ AxisCoef yt[T::EY];
	const double alpha = sc[3];
	const int P0 = o.ax[0].P, P1 = o.ax[1].P;
	const int tx = threadIdx.x % T::EX, ty = threadIdx.x / T::EX;
	const int ex0 = (int) blockIdx.x * T::X - T::HALO, ey0 = (int) blockIdx.y * T::Y - T::HALO;
	const int gi = fold_index(o.ax[0], ex0 + tx);
	const int slot = ty * T::ROWS * T::EX + tx;
	const int left = tx > 0 ? -1 : 0, right = tx + 1 < T::EX ? 1 : 0;
	const int above = ty > 0 ? -T::EX : 0, below = ty + 1 < T::TY ? T::EX : 0;
	int off[T::ROWS];
	double v[T::ROWS], sums[1] = {0.0};
#pragma unroll
	for (int c = 0; c < T::ROWS; ++c) {
		const int gj = fold_index(o.ax[1], ey0 + ty * T::ROWS + c);
		const bool on = gi >= 0 && gj >= 0;
		off[c] = on ? gi + gj * P0 : 0;
		v[c] = __fma_rn(-alpha, on && !first ? __ldg(q + off[c]) : 0.0, on ? __ldg(r + off[c]) : 0.0);
		planes[0][slot + c * T::EX] = v[c];
	}
	auto run = [&](const auto& H) {
		// out = w r' - ws H s, s this thread's columns and their shared copy buf
		auto step = [&](const double* buf, double w, double ws, const double* s, double* out) {
#pragma unroll
			for (int c = 0; c < T::ROWS; ++c) {
				const int at = slot + c * T::EX;
				const double h = H.plane(ty * T::ROWS + c, s[c], buf[at + left], buf[at + right],
				                         c > 0 ? s[c - 1] : buf[at + above],
				                         c + 1 < T::ROWS ? s[c + 1] : buf[at + below]);
				out[c] = __fma_rn(w, v[c], -ws * h);
			}
		};
		double a[T::ROWS], b[T::ROWS];
		__syncthreads();
		step(planes[0], cw.w[1], cw.w[0], v, a);
#pragma unroll
		for (int c = 0; c < T::ROWS; ++c) planes[1][slot + c * T::EX] = a[c];
		__syncthreads();        // the first step is complete, every read of r' done
		step(planes[1], cw.w[2], 1.0, a, b);
#pragma unroll
		for (int c = 0; c < T::ROWS; ++c) planes[0][slot + c * T::EX] = b[c];
		__syncthreads();
		step(planes[0], cw.w[3], 1.0, b, a);
#pragma unroll
		for (int c = 0; c < T::ROWS; ++c) {
			const int ey = ty * T::ROWS + c;
			if (tx >= T::HALO && tx < T::HALO + T::X && ex0 + tx < P0 && ey >= T::HALO && ey < T::HALO + T::Y &&
			    ey0 + ey < P1) {
				rnew[off[c]] = v[c];
				z[off[c]] = a[c];
				sums[0] = __fma_rn(v[c], a[c], sums[0]);
			}
		}
	};
	const AxisCoef cx = axis_coef(o.ax[0], true, o.lambda, gi);
	if (alike(o.ax[0], ex0, ex0 + T::EX - 1) && alike(o.ax[1], ey0, ey0 + T::EY - 1)) {
		run(UniformH(o, cx, yt, yt));
	} else {
		fill_table(o, 1, ey0, T::EY, yt);       // read after the first barrier
		run(PlaneH(cx, yt));
	}
	if (grid_sums<T::THREADS, 1>(sums, part, done) && threadIdx.x == 0) advance(sums[0], sc, first);
}

// Planes per block of a tile kernel and the cost that comes with them: rounds
// of work over the resident blocks, a round being the block's planes, the
// halo planes that it recomputes and about three planes' time to start and
// finish.
struct Run { int planes; long long cost; };

Run pick_run(long long tiles, int planes, int halo, long long resident)
{
	Run best{1, -1};
	for (int run = 1; run <= std::min(planes, kMaxRun); ++run) {
		const long long blocks = tiles * ((planes + run - 1) / run);
		const long long cost = ((blocks + resident - 1) / resident) * (run + 2 * halo + 3);
		if (best.cost < 0 || cost <= best.cost) best = {run, cost};
	}
	return best;
}

// out = u + x
__global__ void __launch_bounds__(kFluidThreads)
finish_kernel(long long n, const double* __restrict__ u, const double* __restrict__ x, double* __restrict__ out)
{
	for (long long i = (long long) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long) gridDim.x * blockDim.x)
		out[i] = x[i] + u[i];
}

// util::math::modulo for the non-negative arguments met here
double modulo1(double x) { return x - std::floor(x); }

// Ghost-point weights of one wall (fd::__1::coefficients,
// include/fd/discretization.h:47-80): Robin condition a u + b du/dn, signed
// mesh width h, alignment s of the grid against the wall.
struct WallWeights { double interior, laplacian; };

WallWeights wall_weights(const double* p, double h, double s_in)
{
	const double s = 1 - modulo1(1 - s_in);
	const double denom = p[1] - p[0] * s * h;
	return {(p[1] + p[0] * h * (1 - s)) / denom, (-(p[1] * (1 - 2 * s) - p[0] * s * h * (1 - s))) / (2 * denom)};
}

// impl::polynomial and impl::chebw<4> (algo/chebyshev.h:48-65, 124-145):
// p(a, b) = sum_i c_i a^i b^(n-1-i), evaluated as the reference does.
double cheb_poly(const double* c, int n, double a, double b)
{
	double v = 0.0;
	for (int i = 0; i < n; ++i) v += c[i] * std::pow(a, i) * std::pow(b, n - 1 - i);
	return v;
}

void chebyshev_weights(double a, double b, double* w)
{
	static const double p1[] = {128}, p2[] = {256, 256}, p3[] = {160, 448, 160}, p4[] = {32, 224, 224, 32};
	static const double q[] = {1, 28, 70, 28, 1};
	const double qv = cheb_poly(q, 5, a, b);
	w[0] = cheb_poly(p1, 1, a, b) / qv;
	w[1] = cheb_poly(p2, 2, a, b) / qv;
	w[2] = cheb_poly(p3, 3, a, b) / qv;
	w[3] = cheb_poly(p4, 4, a, b) / qv;
}

ibk_status cuda_fail(cudaError_t e, const char* what)
{
	return set_error(IBK_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

} // namespace
} // namespace ibk

using namespace ibk;

// Iterations queued beyond the one whose stopping test the host waits for.
// The test runs on the device and the kernels of a stopped loop return at
// once, so a few iterations too many cost a few microseconds, while waiting
// for every test before queueing more would leave the GPU idle for the round
// trip (about 20 us of each iteration; a 64^3 grid's takes about that long).
constexpr int kLookAhead = 2;

struct ibk_diffusion_s {
	int device = 0;
	FluidOps ops{};
	double mu = 0.0, timestep = 0.0, tolerance = 0.0;
	int max_iterations = 0;
	double* coef = nullptr;        // per axis: lo, diag, hi, id (4 P_d doubles)
	double* work = nullptr;        // 8 arrays of size doubles (see Work)
	int precond = IBK_PRECOND_CHEBYSHEV;
	double cheb_w[4] = {};         // chebw<4> on the Gershgorin interval
	double bounds[2] = {};         // that interval (lower, upper)
	double* partial = nullptr;     // the blocks' partial sums
	int first_partials = 0;        // room for the first of two sets
	March march;                   // march_apply_kernel's grid
	dim3 dir_grid, poly_grid;      // grids and planes per block of the Chebyshev loop's kernels
	int dir_run = 1, poly_run = 1;
	PolyKind poly_kind = kPolyWide;
	double* scalars = nullptr;     // device scalars of the loop, then the kernels' counter of finished blocks
	double* host_tests = nullptr;                   // pinned: stop and iterations of each look-ahead slot
	cudaEvent_t tested[kLookAhead + 1] = {};        // the kernel that writes each slot
};

namespace {

// The right-hand side of the solve: k I~ f + k mu (L u + rhs).
void launch_rhs(const ibk_diffusion_s& d, double gamma, const double* u, const double* rhs, const double* f, double* b,
                cudaStream_t s)
{
	const double k = gamma * d.timestep;
	launch_march(d.ops, 3, d.march, u, b, nullptr, s, f, rhs, k, k * d.mu);
}

const char* const kNoConvergence = "diffusion solve did not converge within max_iterations";

// The loop with the Chebyshev preconditioner (two kernels an iteration).
ibk_status step_chebyshev(ibk_diffusion_s& d, double gamma, const double* u, const double* rhs, const double* f,
                          double* out, int* iterations, cudaStream_t s)
{
	const long long n = d.ops.size;
	double* r[2] = {d.work, d.work + n};
	double* dv[2] = {d.work + 2 * n, d.work + 3 * n};
	double *q = d.work + 4 * n, *x = d.work + 6 * n, *z = d.work + 7 * n;
	double* sc = d.scalars;
	unsigned* done = reinterpret_cast<unsigned*>(sc + kScalars);
	ChebWeights cw;
	std::copy(d.cheb_w, d.cheb_w + 4, cw.w);
	cudaError_t e = cudaMemsetAsync(sc, 0, sizeof(double) * (kScalars + 1), s);
	if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync");
	launch_rhs(d, gamma, u, rhs, f, r[0], s);
	const bool flat = d.ops.dims == 2;
	const auto march = [&](auto tile, const double* rin, double* rout, int first) {
		using T = decltype(tile);
		polynomial_kernel<T><<<d.poly_grid, T::THREADS, poly_bytes<T>(), s>>>(d.ops, sc, rin, q, rout, z, d.partial, done,
		                                                                     d.poly_run, first, cw);
	};
	const auto plane = [&](auto tile, const double* rin, double* rout, int first) {
		using T = decltype(tile);
		polynomial_plane_kernel<T><<<d.poly_grid, T::THREADS, 0, s>>>(d.ops, sc, rin, q, rout, z, d.partial, done, first, cw);
	};
	const auto polynomial = [&](const double* rin, double* rout, int first) {
		switch (d.poly_kind) {
		case kPolyWide: return flat ? plane(PlaneWide(), rin, rout, first) : march(PolyWide(), rin, rout, first);
		case kPolySmall: return flat ? plane(PlaneSmall(), rin, rout, first) : march(PolySmall(), rin, rout, first);
		case kPolyTall: return march(PolyTall(), rin, rout, first);
		}
	};
	polynomial(r[0], r[1], 1);
	ibk_status st = check_launch("diffusion set-up kernels");
	if (st != IBK_OK) return st;
	const double* seen = nullptr;          // the test that stopped the loop
	for (long long it = 0; !seen; ++it) {
		const int a = (int) (it & 1), slot = (int) (it % (kLookAhead + 1));
		if (flat)
			direction_plane_kernel<<<d.dir_grid, kDirThreads, 0, s>>>(d.ops, sc, z, dv[a], dv[a ^ 1], x, q, d.partial, done,
			                                                          it == 0, d.tolerance, d.max_iterations,
			                                                          d.host_tests + 2 * slot);
		else
			direction_apply_kernel<<<d.dir_grid, kDirThreads, 0, s>>>(d.ops, sc, z, dv[a], dv[a ^ 1], x, q, d.partial, done,
			                                                          d.dir_run, it == 0, d.tolerance, d.max_iterations,
			                                                          d.host_tests + 2 * slot);
		if ((e = cudaEventRecord(d.tested[slot], s)) != cudaSuccess) return cuda_fail(e, "diffusion residual read");
		polynomial(r[a ^ 1], r[a], 0);
		if ((st = check_launch("diffusion iteration kernels")) != IBK_OK) return st;
		if (it < kLookAhead) continue;
		const int back = (int) ((it - kLookAhead) % (kLookAhead + 1));
		if ((e = cudaEventSynchronize(d.tested[back])) != cudaSuccess) return cuda_fail(e, "diffusion residual read");
		if (d.host_tests[2 * back] != 0.0) seen = d.host_tests + 2 * back;
	}
	// the queued iterations find the loop stopped; they are over before the
	// next call may start another on this handle's scalars
	if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_fail(e, "diffusion residual read");
	if (iterations) *iterations = (int) seen[1];
	if (seen[0] == kLimit) return set_error(IBK_ERR_DEVICE_CHECK, kNoConvergence);
	finish_kernel<<<kFluidBlocks, kFluidThreads, 0, s>>>(n, u, x, out);
	return check_launch("finish_kernel");
}

// The loop with the Jacobi preconditioner.
ibk_status step_jacobi(ibk_diffusion_s& d, double gamma, const double* u, const double* rhs, const double* f,
                       double* out, int* iterations, cudaStream_t s)
{
	const long long n = d.ops.size;
	double *r = d.work, *dv = d.work + 2 * n, *q = d.work + 4 * n, *diag = d.work + 5 * n, *x = d.work + 6 * n;
	double* pa = d.partial;
	double* pb = d.partial + d.first_partials;
	double* sc = d.scalars;
	cudaError_t e = cudaMemsetAsync(sc, 0, sizeof(double) * kScalars, s);
	if (e != cudaSuccess) return cuda_fail(e, "cudaMemsetAsync");
	launch_rhs(d, gamma, u, rhs, f, r, s);
	start_kernel<<<kFluidBlocks, kFluidThreads, 0, s>>>(n, r, diag, x, dv, pa, pb);
	sum_kernel<<<1, kSumThreads, 0, s>>>(pa, kFluidBlocks, sc + 0);
	sum_kernel<<<1, kSumThreads, 0, s>>>(pb, kFluidBlocks, sc + 2);
	ibk_status st = check_launch("diffusion set-up kernels");
	if (st != IBK_OK) return st;
	const double tol = d.tolerance;
	int it = 0;
	double hs[6];
	for (;;) {
		// the loop test of pcg.h:21 (|d| > tol) and its bail-out, read back once
		// per iteration; alpha and beta stay on the device
		e = cudaMemcpyAsync(hs, sc, sizeof(double) * 6, cudaMemcpyDeviceToHost, s);
		if (e == cudaSuccess) e = cudaStreamSynchronize(s);
		if (e != cudaSuccess) return cuda_fail(e, "diffusion residual read");
		if (hs[5] != 0.0 || !(std::sqrt(hs[2]) > tol)) break;
		if (it >= d.max_iterations) {
			if (iterations) *iterations = it;
			return set_error(IBK_ERR_DEVICE_CHECK, kNoConvergence);
		}
		launch_march(d.ops, 2, d.march, dv, q, pa, s);
		alpha_kernel<<<1, kSumThreads, 0, s>>>(pa, d.march.blocks(), tol * tol, sc);
		update_kernel<<<kFluidBlocks, kFluidThreads, 0, s>>>(n, sc, dv, q, x, r, diag, pa);
		beta_kernel<<<1, kSumThreads, 0, s>>>(pa, kFluidBlocks, sc);
		direction_kernel<<<kFluidBlocks, kFluidThreads, 0, s>>>(n, sc, q, dv, pb);
		sum_kernel<<<1, kSumThreads, 0, s>>>(pb, kFluidBlocks, sc + 2);
		if ((st = check_launch("diffusion iteration kernels")) != IBK_OK) return st;
		++it;
	}
	// a bail-out leaves the last iteration's update undone, as pcg.h does
	if (hs[5] != 0.0 && it > 0) --it;
	finish_kernel<<<kFluidBlocks, kFluidThreads, 0, s>>>(n, u, x, out);
	if (iterations) *iterations = it;
	return check_launch("finish_kernel");
}

} // namespace

extern "C" {

ibk_status ibk_diffusion_create(ibk_plan plan, int component, const double robin[3][2][2], double timestep,
                                double mu, double tolerance, int max_iterations, ibk_diffusion* out)
{
	if (!out) return set_error(IBK_ERR_INVALID_ARGUMENT, "null output handle");
	*out = nullptr;
	Plan* p = reinterpret_cast<Plan*>(plan);
	if (!p || !robin) return set_error(IBK_ERR_INVALID_ARGUMENT, "null plan or boundary conditions");
	const GridGeom& g = p->g;
	if (component < 0 || component >= g.dims) return set_error(IBK_ERR_INVALID_ARGUMENT, "component out of range");
	if (!(timestep > 0.0) || !(mu >= 0.0) || !(tolerance > 0.0) || max_iterations < 1)
		return set_error(IBK_ERR_INVALID_ARGUMENT, "timestep and tolerance must be positive, mu non-negative");
	for (int a = 0; a < g.dims; ++a)
		for (int side = 0; side < 2 && g.solid[a]; ++side)
			if (robin[a][side][0] == 0.0 && robin[a][side][1] == 0.0)
				return set_error(IBK_ERR_INVALID_ARGUMENT, "a wall's Robin condition needs a or b nonzero");
	const CompGeom& cg = g.comp[component];
	auto* d = new ibk_diffusion_s;
	cudaGetDevice(&d->device);
	d->mu = mu;
	d->timestep = timestep;
	d->tolerance = tolerance;
	d->max_iterations = max_iterations;
	d->ops.dims = g.dims;
	d->ops.lambda = timestep * mu / 2;       // diffusion.h:21-25
	long long size = 1;
	int total = 0;
	for (int a = 0; a < 3; ++a) {
		d->ops.ax[a].P = a < g.dims ? cg.points[a] : 1;
		size *= d->ops.ax[a].P;
		total += 4 * d->ops.ax[a].P;
	}
	d->ops.size = size;
	std::vector<double> host((size_t) total, 0.0);
	int off = 0;
	for (int a = 0; a < g.dims; ++a) {
		const int P = cg.points[a];
		if (P < kMinPoints) {
			delete d;
			return set_error(IBK_ERR_INVALID_ARGUMENT, "each axis needs at least 3 points");
		}
		double* lo = host.data() + off;
		double* dg = lo + P;
		double* hi = dg + P;
		double* id = hi + P;
		const double scale = g.r * g.r;          // laplacian.h:25-26
		for (int i = 0; i < P; ++i) {
			lo[i] = i > 0 ? scale : 0.0;
			dg[i] = -2 * scale;
			hi[i] = i + 1 < P ? scale : 0.0;
			id[i] = 1.0;
		}
		const int periodic = !g.solid[a];
		if (periodic) {
			// wrap entries (discretization.h:94-100: {!lower, lower, 1})
			lo[0] = scale * 1.0;
			hi[P - 1] = scale * 1.0;
		} else {
			// ghost-point weights of each wall on the corner diagonals, and the
			// second-order error coefficients on the identity's corners
			const double h = 1 / g.r;
			const double al = modulo1(cg.shift[a]);
			const WallWeights wl = wall_weights(robin[a][0], h, al);
			const WallWeights wu = wall_weights(robin[a][1], -h, 1 - al);
			dg[0] += scale * wl.interior;
			dg[P - 1] += scale * wu.interior;
			id[0] += wl.laplacian;
			id[P - 1] += wu.laplacian;
		}
		d->ops.ax[a].periodic = periodic;
		off += 4 * P;
	}
	const int P0 = d->ops.ax[0].P, P1 = d->ops.ax[1].P, P2 = d->ops.ax[2].P;
	const auto tiles = [](int p, int t) { return (unsigned) ((p + t - 1) / t); };
	d->march.grid = dim3(tiles(P0, kMarchX), tiles(P1, kMarchY), 1);
	while (d->march.zrun > 2 && (long long) d->march.grid.x * d->march.grid.y * tiles(P2, d->march.zrun) < 4LL * p->num_sms)
		d->march.zrun /= 2;
	d->march.grid.z = tiles(P2, d->march.zrun);
	d->dir_grid = dim3(tiles(P0, kDirX), tiles(P1, kDirY), 1);
	d->dir_run = pick_run((long long) d->dir_grid.x * d->dir_grid.y, P2, 1, (long long) kDirBlocks * p->num_sms).planes;
	d->dir_grid.z = tiles(P2, d->dir_run);
	// The tile of the cheapest run; the wide one's step takes kWideStep times as
	// long as the others'.  In two dimensions a step is short and the small
	// tile's extra halo counts once its blocks no longer run all at once (see
	// PlaneSmall).
	const bool flat = g.dims == 2;
	double best = -1.0;
	const auto consider = [&](auto tile, PolyKind kind, double step) {
		using T = decltype(tile);
		const dim3 grid(tiles(P0, T::X), tiles(P1, T::Y), 1);
		const Run run = pick_run((long long) grid.x * grid.y, P2, T::HALO, (long long) T::BLOCKS * p->num_sms);
		if (best >= 0.0 && step * (double) run.cost >= best) return;
		best = step * (double) run.cost;
		d->poly_kind = kind;
		d->poly_grid = grid;
		d->poly_run = run.planes;
	};
	const bool rounds = (long long) tiles(P0, PolySmall::X) * tiles(P1, PolySmall::Y) > 2LL * p->num_sms;
	if (!flat || rounds) consider(PolyWide(), kPolyWide, kWideStep);
	if (!flat || !rounds) consider(PolySmall(), kPolySmall, 1.0);
	if (!flat) consider(PolyTall(), kPolyTall, 1.0);
	d->poly_grid.z = tiles(P2, d->poly_run);
	for (const dim3& g : {d->march.grid, d->dir_grid, d->poly_grid})
		if (g.y > 65535u || g.z > 65535u || size >= (1LL << 31)) {
			delete d;
			return set_error(IBK_ERR_UNSUPPORTED, "grid too large for the operator kernel (2^31 faces)");
		}
	const auto count = [](const dim3& g) { return (int) (g.x * g.y * g.z); };
	d->first_partials = std::max({count(d->march.grid), 2 * count(d->dir_grid), count(d->poly_grid), kFluidBlocks});
	cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&d->coef), sizeof(double) * (size_t) total);
	if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&d->work), sizeof(double) * 8 * (size_t) size);
	if (e == cudaSuccess)
		e = cudaMalloc(reinterpret_cast<void**>(&d->partial), sizeof(double) * (size_t) (d->first_partials + kFluidBlocks));
	if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&d->scalars), sizeof(double) * (kScalars + 1));
	if (e == cudaSuccess)
		e = cudaHostAlloc(reinterpret_cast<void**>(&d->host_tests), sizeof(double) * 2 * (kLookAhead + 1),
		                  cudaHostAllocMapped);
	for (cudaEvent_t& ev : d->tested)
		if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(polynomial_kernel<PolyWide>, cudaFuncAttributeMaxDynamicSharedMemorySize, poly_bytes<PolyWide>());
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(polynomial_kernel<PolySmall>, cudaFuncAttributeMaxDynamicSharedMemorySize, poly_bytes<PolySmall>());
	if (e == cudaSuccess)
		e = cudaFuncSetAttribute(polynomial_kernel<PolyTall>, cudaFuncAttributeMaxDynamicSharedMemorySize, poly_bytes<PolyTall>());
	if (e == cudaSuccess) e = cudaMemcpy(d->coef, host.data(), sizeof(double) * (size_t) total, cudaMemcpyHostToDevice);
	if (e != cudaSuccess) {
		cudaGetLastError();
		ibk_diffusion_destroy(d);
		return set_error(IBK_ERR_OUT_OF_MEMORY, std::string("diffusion set-up: ") + cudaGetErrorString(e));
	}
	off = 0;
	for (int a = 0; a < 3; ++a) {
		AxisOps& ax = d->ops.ax[a];
		if (a < g.dims) {
			ax.lo = d->coef + off;
			ax.diag = ax.lo + ax.P;
			ax.hi = ax.diag + ax.P;
			ax.id = ax.hi + ax.P;
			off += 4 * ax.P;
		} else {
			ax.lo = ax.diag = ax.hi = ax.id = d->coef;    // never read (dims < 3)
			ax.periodic = 0;
		}
	}
	// the Jacobi preconditioner's reciprocal diagonal, kept in work slot 5, and
	// the Gershgorin interval of the Chebyshev preconditioner (through the
	// partial-sum buffer, 2 per block)
	diagonal_kernel<<<kFluidBlocks, kFluidThreads>>>(d->ops, d->work + 5 * size);
	gershgorin_kernel<<<kFluidBlocks, kFluidThreads>>>(d->ops, d->partial);
	ibk_status st = check_launch("diffusion set-up kernels");
	std::vector<double> part(2 * kFluidBlocks);
	if (st == IBK_OK && (e = cudaMemcpy(part.data(), d->partial, sizeof(double) * part.size(),
	                                    cudaMemcpyDeviceToHost)) != cudaSuccess)
		st = cuda_fail(e, "diffusion set-up");
	if (st != IBK_OK) {
		ibk_diffusion_destroy(d);
		return st;
	}
	double lower = INFINITY, upper = -INFINITY;
	for (int b = 0; b < kFluidBlocks; ++b) {
		lower = std::min(lower, part[2 * b]);
		upper = std::max(upper, part[2 * b + 1]);
	}
	d->bounds[0] = lower;
	d->bounds[1] = upper;
	chebyshev_weights(upper, lower, d->cheb_w);     // chebyshev(upper, lower, H): preconditioners/chebyshev.h:14-25
	*out = d;
	return IBK_OK;
}

ibk_status ibk_diffusion_set_preconditioner(ibk_diffusion d, int kind)
{
	if (!d) return set_error(IBK_ERR_INVALID_ARGUMENT, "null diffusion handle");
	if (kind != IBK_PRECOND_CHEBYSHEV && kind != IBK_PRECOND_JACOBI)
		return set_error(IBK_ERR_INVALID_ARGUMENT, "unknown preconditioner");
	d->precond = kind;
	return IBK_OK;
}

ibk_status ibk_diffusion_info(ibk_diffusion d, double* bounds, double* weights)
{
	if (!d) return set_error(IBK_ERR_INVALID_ARGUMENT, "null diffusion handle");
	if (bounds) { bounds[0] = d->bounds[0]; bounds[1] = d->bounds[1]; }
	if (weights) for (int q = 0; q < 4; ++q) weights[q] = d->cheb_w[q];
	return IBK_OK;
}

ibk_status ibk_diffusion_destroy(ibk_diffusion d)
{
	if (!d) return IBK_OK;
	int dev = 0;
	cudaGetDevice(&dev);
	cudaSetDevice(d->device);
	cudaFree(d->coef);
	cudaFree(d->work);
	cudaFree(d->partial);
	cudaFree(d->scalars);
	for (cudaEvent_t ev : d->tested)
		if (ev) cudaEventDestroy(ev);
	if (d->host_tests) cudaFreeHost(d->host_tests);
	cudaSetDevice(dev);
	delete d;
	return IBK_OK;
}

ibk_status ibk_diffusion_apply(ibk_diffusion d, int op, const double* u, double* out, void* stream)
{
	if (!d || !u || !out || op < 0 || op > 2) return set_error(IBK_ERR_INVALID_ARGUMENT, "null arrays or unknown operator");
	cudaStream_t s = static_cast<cudaStream_t>(stream);
	launch_march(d->ops, op, d->march, u, out, nullptr, s);
	return check_launch("march_apply_kernel");
}

ibk_status ibk_diffusion_step(ibk_diffusion d, double gamma, const double* u, const double* rhs, const double* f,
                              double* out, int* iterations, void* stream)
{
	if (!d || !u || !rhs || !f || !out) return set_error(IBK_ERR_INVALID_ARGUMENT, "null arrays");
	return d->precond == IBK_PRECOND_CHEBYSHEV ? step_chebyshev(*d, gamma, u, rhs, f, out, iterations, static_cast<cudaStream_t>(stream))
	                                           : step_jacobi(*d, gamma, u, rhs, f, out, iterations, static_cast<cudaStream_t>(stream));
}

} // extern "C"
