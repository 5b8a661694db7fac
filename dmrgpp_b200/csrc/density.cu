// Density-matrix truncation after a sector solve (dmrgpp_density_truncate in
// dmrgpp_kron.h): the reference's per-patch SVD route
// (DensityMatrixSvd.h:285-410 ParallelPsiSplit / ParallelSvd, Truncation.h:
// 218-285 changeBasis, 373-519 updateKeptStates / computeKeptStates).
//
// The reference stacks, for every group g of the block being truncated, the
// sector-vector entries of all patches of g (one column block per patch and
// target, scaled by sqrt(weight)) into M_g and takes svd('A', M_g); the
// density-matrix eigenvalues are the squared singular values and the kept
// transformation is U.  Here rho_g = M_g M_g^T is formed directly as a sum of
// X_p^T X_p (system side) or X_p X_p^T (environment side) by one grouped DGEMM
// launch on the FP64 tensor pipe and reduced to tridiagonal form there, one
// cluster of CTAs per group, their eigenvalues found by bisection (groups above
// kTriMaxN states go to the host cores meanwhile: tridiag.cpp); the host
// ranks the states (computeKeptStates) and forms the kept eigenvectors of the
// tridiagonals by inverse iteration on all cores (tridiag.cpp), and the device
// applies the Householder reflectors to them.
#include "devmem.h"
#include "trace.h"
#include "dmrgpp_kron.h"
#include "handle.h"
#include "kron_gemm.cuh"
#include "tridiag.h"

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <climits>
#include <memory>
#include <cmath>
#include <numeric>
#include <string>
#include <vector>

namespace dmrgpp {
namespace {

// one 32 x 32 tile of a weighted transpose: XT (cols x rows, ld cols) =
// w * X (rows x cols, ld rows)
struct TransposeTile {
	long long src, dst;
	int       rows, cols, r0, c0;
	double    w;
};

__global__ void __launch_bounds__(256)
k_transpose_tiles(const double* __restrict__ x, double* __restrict__ xt, const TransposeTile* __restrict__ tiles,
                  int ntiles)
{
	__shared__ double s[32][33];
	const int         tx = threadIdx.x & 31, ty = threadIdx.x >> 5; // 32 x 8
	for (int q = blockIdx.x; q < ntiles; q += gridDim.x) {
		const TransposeTile t = tiles[q];
		__syncthreads();
		for (int j = ty; j < 32; j += 8) { // column c0 + j, row r0 + tx
			const int r = t.r0 + tx, c = t.c0 + j;
			s[j][tx]    = (r < t.rows && c < t.cols) ? x[t.src + r + (long long)c * t.rows] : 0.0;
		}
		__syncthreads();
		for (int j = ty; j < 32; j += 8) { // XT row c0 + tx, column r0 + j
			const int c = t.c0 + tx, r = t.r0 + j;
			if (r < t.rows && c < t.cols)
				xt[t.dst + c + (long long)r * t.cols] = t.w * s[tx][j];
		}
	}
}

namespace cg = cooperative_groups;

// One group of the tridiagonal reduction.
struct TridiagJob {
	long long m_off; // rho_g (n x n)
	long long w_off; // its working copy
	long long e_off; // its place in the per-state arrays
	int       n;
	int       group;
};

constexpr int kTriCluster = 8;
constexpr int kTriThreads = 512;
constexpr int kTriMaxN    = 2048; // largest group (its vectors are in shared memory)

// sum over the block, the same in every thread (fixed order)
__device__ __forceinline__ double block_sum_all(double v, double* red)
{
	for (int o = 16; o > 0; o >>= 1)
		v += __shfl_xor_sync(0xffffffffu, v, o);
	__syncthreads(); // red free
	if ((threadIdx.x & 31) == 0)
		red[threadIdx.x >> 5] = v;
	__syncthreads();
	double s = 0.0;
#pragma unroll
	for (int w = 0; w < kTriThreads / 32; ++w)
		s += red[w];
	return s;
}

// Householder reduction of rho_g to tridiagonal form, T = Q^T rho Q with
// householder_tridiag's conventions (tridiag.cpp): diagonal d, off-diagonal
// off, reflectors h_k into column k of rho_g's own storage, beta.  One cluster
// of 8 CTAs per group; CTA r owns columns r, r + 8, ... of the working copy
// `work` (both triangles).  A step makes one pass over the owned trailing
// columns that applies the previous step's rank-2 update and forms this step's
// product y = A h (one warp per column, so y needs no sum across CTAs), sends
// y to all CTAs' shared memory and meets them at one cluster barrier; the
// column that makes the next reflector, its norm, and the vectors h and q are
// formed by every CTA for itself.  All groups run side by side: the launch
// lasts as long as the largest group's n steps of a few memory latencies each
// (the host cores took 10.6 ms for 241 groups of up to 532 states with their
// eigenvalues, this kernel 3.9).
__global__ void __cluster_dims__(kTriCluster, 1, 1) __launch_bounds__(kTriThreads)
k_tridiag(double* __restrict__ rho, double* __restrict__ work, const TridiagJob* __restrict__ jobs, double* d,
          double* off, double* beta, int* shift, int vec)
{
	extern __shared__ __align__(16) double smem[];
	__shared__ double                      red[kTriThreads / 32];
	__shared__ double                      amax_of[kTriCluster];
	cg::cluster_group                      cluster = cg::this_cluster();
	cluster.barrier_arrive(); // this CTA runs: its shared memory may be written to (waited for below)
	const int                              rank    = int(cluster.block_rank());
	const int                              tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const TridiagJob                       jb = jobs[blockIdx.x / kTriCluster];
	const int                              n  = jb.n;
	double*                                R  = rho + jb.m_off;
	double*                                A  = work + jb.w_off;
	d += jb.e_off;
	off += jb.e_off;
	beta += jb.e_off;
	// vectors of the step, `vec` doubles each: column and new h, previous h
	// and q (index 0 = row k), and y of this and the previous step
	double* h  = smem;
	double* hp = smem + vec;
	double* qp = smem + 2 * vec;
	double* y2 = smem + 3 * vec;

	// working copy, symmetrised; the largest entry outside [2^-64, 2^64]:
	// 2^shift rho instead (group_eigenvalues has the reason)
	double amax = 0.0;
	for (int c = rank + kTriCluster * warp; c < n; c += kTriCluster * (kTriThreads / 32))
		for (int i = lane; i < n; i += 32) {
			const double v = 0.5 * (R[i + (long long)c * n] + R[c + (long long)i * n]);
			A[i + (long long)c * n] = v;
			amax                    = fmax(amax, fabs(v));
		}
	for (int o = 16; o > 0; o >>= 1)
		amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
	if (lane == 0)
		red[warp] = amax;
	__syncthreads();
	cluster.barrier_wait(); // every CTA of the cluster has started: the stores below go to their shared memory
	if (tid < kTriCluster) {
		double m = 0.0;
		for (int w = 0; w < kTriThreads / 32; ++w)
			m = fmax(m, red[w]);
		*cluster.map_shared_rank(&amax_of[rank], tid) = m;
	}
	cluster.sync(); // every copy of rho_g is read, every maximum is here
	amax = 0.0;
	for (int r = 0; r < kTriCluster; ++r)
		amax = fmax(amax, amax_of[r]);
	int sh = 0;
	if (amax > 0.0 && isfinite(amax) && (amax < 0x1p-64 || amax > 0x1p64)) {
		int e = 0;
		frexp(amax, &e);
		sh = -e;
		for (int c = rank + kTriCluster * warp; c < n; c += kTriCluster * (kTriThreads / 32))
			for (int i = lane; i < n; i += 32)
				A[i + (long long)c * n] = ldexp(A[i + (long long)c * n], sh);
		cluster.sync();
	}
	if (rank == 0 && tid == 0)
		shift[jb.group] = sh;

	bool pending = false; // A <- A - hp qp^T - qp hp^T on rows / columns >= k
	for (int k = 0; k + 2 < n; ++k) {
		const int len = n - k - 1;
		double*   y   = y2 + (k & 1) * vec;
		// column k, rows k .. n-1, brought up to date (its owner wrote it in an
		// earlier step: read from L2)
		const double hk = pending ? hp[0] : 0.0, qk = pending ? qp[0] : 0.0;
		double       sigma = 0.0, dk = 0.0;
		for (int i = tid; i <= len; i += kTriThreads) {
			double v = __ldcg(A + (k + i) + (long long)k * n);
			if (pending)
				v -= hp[i] * qk + qp[i] * hk;
			if (i == 0)
				dk = v;
			else
				h[i - 1] = v;
			if (i >= 2)
				sigma += v * v;
		}
		sigma           = block_sum_all(sigma, red); // and h is complete
		const double x0 = h[0];
		double       b = 0.0, h0 = 0.0, offk = x0;
		if (sigma != 0.0) {
			const double mu = sqrt(x0 * x0 + sigma);
			h0              = x0 <= 0.0 ? x0 - mu : -sigma / (x0 + mu);
			b               = 2.0 * h0 * h0 / (sigma + h0 * h0);
			offk            = mu;
		}
		__syncthreads(); // x0 read by all before h changes
		if (b != 0.0)
			for (int i = tid; i < len; i += kTriThreads)
				h[i] = i == 0 ? 1.0 : h[i] / h0;
		if (rank == 0) {
			if (tid == 0) {
				d[k]    = dk;
				off[k]  = offk;
				beta[k] = b;
			}
			if (b != 0.0) // rho_g itself is no longer needed
				for (int i = tid; i < len; i += kTriThreads)
					R[i + (long long)k * n] = h[i]; // each thread its own entries
		}
		__syncthreads();
		// the pass over the owned columns c > k
		const int first = k + 1 + ((rank - (k + 1)) & (kTriCluster - 1)); // first column with c % 8 == rank
		if (pending || b != 0.0)
			// two columns at a time, eight loads of a lane in flight: a column is
			// a few memory latencies long, and there are 8 x 16 of them at once
			for (int c = first + 2 * kTriCluster * warp; c < n; c += 2 * kTriCluster * (kTriThreads / 32)) {
				const int    c1  = c + kTriCluster;
				const bool   two = c1 < n;
				double*      a0  = A + (k + 1) + (long long)c * n;
				double*      a1  = two ? A + (k + 1) + (long long)c1 * n : a0;
				const double h0j = pending ? hp[c - k] : 0.0, q0j = pending ? qp[c - k] : 0.0;
				const double h1j = pending && two ? hp[c1 - k] : 0.0, q1j = pending && two ? qp[c1 - k] : 0.0;
				double       s0 = 0.0, s1 = 0.0;
				for (int i0 = lane; i0 < len; i0 += 128) {
					double v0[4], v1[4];
#pragma unroll
					for (int u = 0; u < 4; ++u) {
						const int i = i0 + 32 * u;
						v0[u]       = i < len ? a0[i] : 0.0;
						v1[u]       = i < len ? a1[i] : 0.0;
					}
#pragma unroll
					for (int u = 0; u < 4; ++u) {
						const int i = i0 + 32 * u;
						if (i < len) {
							if (pending) {
								const double hi = hp[i + 1], qi = qp[i + 1];
								v0[u] -= hi * q0j + qi * h0j;
								v1[u] -= hi * q1j + qi * h1j;
								a0[i] = v0[u];
								if (two)
									a1[i] = v1[u];
							}
							s0 += v0[u] * h[i];
							s1 += v1[u] * h[i];
						}
					}
				}
				for (int o = 16; o > 0; o >>= 1) {
					s0 += __shfl_xor_sync(0xffffffffu, s0, o);
					s1 += __shfl_xor_sync(0xffffffffu, s1, o);
				}
				if (lane < kTriCluster) {
					double* yr    = cluster.map_shared_rank(y, lane);
					yr[c - k - 1] = s0;
					if (two)
						yr[c1 - k - 1] = s1;
				}
			}
		cluster.sync();
		pending = b != 0.0;
		if (!pending)
			continue; // (uniform over the cluster)
		double ph = 0.0;
		for (int i = tid; i < len; i += kTriThreads) {
			const double p = b * y[i];
			y[i]           = p;
			ph += p * h[i];
		}
		ph = block_sum_all(ph, red);
		for (int i = tid; i < len; i += kTriThreads) {
			const double hi = h[i];
			qp[i]           = y[i] - 0.5 * b * ph * hi;
			hp[i]           = hi;
		}
		__syncthreads();
	}
	if (rank == 0 && tid == 0) {
		if (n == 1) {
			d[0]    = A[0];
			off[0]  = 0.0;
			beta[0] = 0.0;
		} else {
			const int k0 = n - 2;
			double    a00 = __ldcg(A + k0 + (long long)k0 * n), a10 = __ldcg(A + k0 + 1 + (long long)k0 * n),
			       a11 = __ldcg(A + k0 + 1 + (long long)(k0 + 1) * n);
			if (pending) {
				a00 -= 2.0 * hp[0] * qp[0];
				a10 -= hp[1] * qp[0] + qp[1] * hp[0];
				a11 -= 2.0 * hp[1] * qp[1];
			}
			d[n - 2]    = a00;
			d[n - 1]    = a11;
			off[n - 2]  = a10;
			off[n - 1]  = 0.0;
			beta[n - 2] = beta[n - 1] = 0.0;
		}
	}
	cluster.sync(); // no CTA leaves while another may still write to its shared memory
}

// Eigenvalues of the tridiagonals, ascending, by Sturm counts: 8 lanes count
// at 8 points of an eigenvalue's interval at once, until the interval is below
// 2^-55 of the norm or an ulp.  n dependent steps a count set the time, so
// fewer rounds beat fewer counts, and the counts are sign changes of the
// leading minors p_i+1 = (d_i - x) p_i - off_i-1^2 p_i-1 (two dependent
// multiply-adds a step; the pivots' quotients, sturm_count in tridiag.cpp, take
// a division: 0.66 against 1.02 ms for 16000 eigenvalues of groups up to 532).
// The matrix is scaled to a norm of about 1, so a step multiplies the minors by
// at most 3, and every 8 steps both are scaled back by a power of two.
struct BisectJob {
	long long e_off;
	int       n, k0; // eigenvalues k0 .. k0 + 31 of the group
};

constexpr int kBisThreads = 256;

__global__ void __launch_bounds__(kBisThreads)
k_bisect(const double* __restrict__ d, const double* __restrict__ off, double* __restrict__ w,
         const BisectJob* __restrict__ jobs)
{
	extern __shared__ __align__(16) double smem[];
	__shared__ double                      lo_s[kBisThreads / 32], hi_s[kBisThreads / 32], sc_s[kBisThreads / 32];
	const BisectJob jb = jobs[blockIdx.x];
	const int       n = jb.n, tid = threadIdx.x, lane = tid & 31;
	double*         ds = smem;
	double*         e2 = smem + n; // off[i]^2
	double          lo = 1.7e308, hi = -1.7e308, sc = 0.0;
	for (int i = tid; i < n; i += kBisThreads) {
		const double di = d[jb.e_off + i], oi = i + 1 < n ? off[jb.e_off + i] : 0.0;
		const double om = i > 0 ? off[jb.e_off + i - 1] : 0.0;
		const double r  = fabs(om) + fabs(oi);
		ds[i]           = di;
		e2[i]           = oi * oi;
		lo              = fmin(lo, di - r);
		hi              = fmax(hi, di + r);
		sc              = fmax(sc, fabs(di) + r);
	}
	for (int o = 16; o > 0; o >>= 1) {
		lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
		hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
		sc = fmax(sc, __shfl_xor_sync(0xffffffffu, sc, o));
	}
	if (lane == 0) {
		lo_s[tid >> 5] = lo;
		hi_s[tid >> 5] = hi;
		sc_s[tid >> 5] = sc;
	}
	__syncthreads();
	for (int q = 0; q < kBisThreads / 32; ++q) {
		lo = fmin(lo, lo_s[q]);
		hi = fmax(hi, hi_s[q]);
		sc = fmax(sc, sc_s[q]);
	}
	const int k = jb.k0 + (tid >> 3); // this lane group's eigenvalue
	if (jb.k0 >= n)
		return;
	const int    kk   = min(k, n - 1) + 1; // idle groups repeat the last
	if (!(sc > 0.0)) { // the zero matrix, or not a number: lo says which
		if ((lane & 7) == 0 && k < n)
			w[jb.e_off + k] = lo;
		return; // (the whole block)
	}
	// 2^-e T, exactly
	int e = 0;
	frexp(sc, &e);
	__syncthreads();
	for (int i = tid; i < n; i += kBisThreads) {
		ds[i] = ldexp(ds[i], -e);
		e2[i] = ldexp(e2[i], -2 * e);
	}
	__syncthreads();
	sc = ldexp(sc, -e);
	lo = ldexp(lo, -e) - 1e-14 * sc;
	hi = ldexp(hi, -e) + 1e-14 * sc;
	const int sub = lane & 7;
	for (int it = 0; it < 200; ++it) {
		const double gap = hi - lo;
		if (!__any_sync(0xffffffffu, gap > 0x1p-55 * sc && lo + 0.5 * gap > lo && lo + 0.5 * gap < hi))
			break;
		const double x = lo + gap * (double(sub + 1) / 9.0);
		int          c = 0;
		double       p0 = 0.0, p1 = 1.0, f = 0.0; // p_{i-1}, p_i, off_{i-1}^2
		for (int i0 = 0; i0 < n; i0 += 8) {
			const int i1 = min(i0 + 8, n);
			for (int i = i0; i < i1; ++i) {
				double p2 = (ds[i] - x) * p1 - f * p0;
				if (p2 == 0.0) // a zero minor has the sign opposite to its predecessor's
					p2 = p1 < 0.0 ? 1e-280 : -1e-280;
				c += (p2 < 0.0) != (p1 < 0.0);
				f  = e2[i];
				p0 = p1;
				p1 = p2;
			}
			// the larger one back to [1, 2)
			const int ex = ilogb(fmax(fabs(p0), fabs(p1)));
			p0           = ldexp(p0, -ex);
			p1           = ldexp(p1, -ex);
		}
		// the first point with kk or more eigenvalues below it bounds it above
		const unsigned m  = (__ballot_sync(0xffffffffu, c >= kk) >> (lane & 24)) & 0xffu;
		const int      at = m ? __ffs(m) - 1 : 8;
		const double   xl = __shfl_sync(0xffffffffu, x, (lane & 24) + max(at - 1, 0));
		const double   xh = __shfl_sync(0xffffffffu, x, (lane & 24) + min(at, 7));
		lo                = at > 0 ? xl : lo;
		hi                = at < 8 ? xh : hi;
	}
	if (sub == 0 && k < n)
		w[jb.e_off + k] = ldexp(0.5 * (lo + hi), e);
}

// Eigenvectors.  For the kept states only, the host computes the tridiagonal
// eigenvectors Z by inverse iteration; the device applies the reflectors to
// them (V = Q Z), the O(n^2) per vector part of the work.

// V[:, j] = Q Z[:, j] for every kept column j of every group: one warp per
// column, the reflectors h_k (k = n-3 .. 0) applied in turn to the column in
// global memory (it stays in L1)
struct ColumnJob {
	long long z_off, v_off, h_off, b_off; // Z and V (n x kept), reflectors (n x n), beta (n)
	int       n, src;                     // src: the Z column
	int       j;
	int       pad;
};

__global__ void __launch_bounds__(256)
k_back_transform(const double* __restrict__ z, double* __restrict__ v, const double* __restrict__ hv,
                 const double* __restrict__ beta, const ColumnJob* __restrict__ jobs, int njobs)
{
	const int lane = threadIdx.x & 31;
	for (int q = blockIdx.x * 8 + (threadIdx.x >> 5); q < njobs; q += gridDim.x * 8) {
		const ColumnJob jb = jobs[q];
		const int       n  = jb.n;
		double*         x  = v + jb.v_off + (long long)jb.j * n;
		const double*   zc = z + jb.z_off + (long long)jb.src * n;
		for (int i = lane; i < n; i += 32)
			x[i] = zc[i];
		__syncwarp();
		for (int k = n - 3; k >= 0; --k) {
			const double bk = beta[jb.b_off + k];
			if (bk == 0.0)
				continue;
			const double* h   = hv + jb.h_off + (long long)k * n; // h[0..len)
			const int     len = n - k - 1;
			double        s   = 0.0;
			for (int i = lane; i < len; i += 32)
				s += h[i] * x[k + 1 + i];
			for (int o = 16; o > 0; o >>= 1)
				s += __shfl_xor_sync(0xffffffffu, s, o);
			s *= bk;
			for (int i = lane; i < len; i += 32)
				x[k + 1 + i] -= s * h[i];
			__syncwarp();
		}
	}
}

// Largest group that k_tridiag takes on this device, 0 where no cluster of it
// fits (a restricted share of the SMs, say).
cudaError_t tridiag_limit(size_t* n)
{
	const size_t smem = 5 * size_t(kTriMaxN) * sizeof(double);
	cudaError_t  e = cudaFuncSetAttribute(k_tridiag, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
	if (e)
		return e;
	cudaLaunchConfig_t cfg {};
	cfg.gridDim          = dim3(kTriCluster, 1, 1);
	cfg.blockDim         = dim3(kTriThreads, 1, 1);
	cfg.dynamicSmemBytes = smem;
	int clusters         = 0;
	if (cudaOccupancyMaxActiveClusters(&clusters, k_tridiag, &cfg) != cudaSuccess) {
		cudaGetLastError();
		clusters = 0;
	}
	*n = clusters > 0 ? size_t(kTriMaxN) : 0;
	return cudaSuccess;
}

// Truncation.h:476-512 (eigs ascending; tolerance < 0 keeps keptStates)
size_t compute_kept(size_t kept_states, double tolerance, size_t m_min, const std::vector<double>& eigs)
{
	if (tolerance < 0)
		return kept_states;
	const long long n     = (long long)eigs.size();
	long long       start = n - (long long)kept_states;
	if (start < 0)
		start = 0;
	long long max_to_remove = n - (long long)m_min;
	if (max_to_remove < 0)
		max_to_remove = 0;
	size_t total = m_min;
	double disc  = 0.0;
	for (long long i = 0; i < start; ++i)
		disc += std::fabs(eigs[size_t(i)]);
	for (long long i = start; i < max_to_remove; ++i) {
		disc += std::fabs(eigs[size_t(i)]);
		if (disc > tolerance) {
			total = size_t(n - i);
			break;
		}
	}
	if (total >= kept_states)
		return kept_states;
	if (total < m_min)
		return m_min;
	return total;
}

int fail(int status, const std::string& msg) { return handle_fail(nullptr, status, msg); }

using Clock = std::chrono::steady_clock;
thread_local double g_trunc_times[DMRGPP_TRUNC_NPHASES] = {};

// Page-locked host buffers of the calling thread, kept between calls (the
// density matrices, reflectors and vectors cross PCIe every call; pageable
// copies and first-touch page faults would cost more than the transfers).
struct PinnedSlot {
	void*  p   = nullptr;
	size_t cap = 0;
	~PinnedSlot()
	{
		if (p)
			cudaFreeHost(p);
	}
};
thread_local PinnedSlot g_pinned[4];

template <class T> T* pinned(int slot, size_t n)
{
	PinnedSlot& s     = g_pinned[slot];
	const size_t bytes = std::max<size_t>(n, 1) * sizeof(T);
	if (s.cap < bytes) {
		if (s.p)
			cudaFreeHost(s.p);
		s.p   = nullptr;
		s.cap = 0;
		if (cudaHostAlloc(&s.p, bytes, cudaHostAllocDefault) != cudaSuccess)
			return nullptr;
		s.cap = bytes;
	}
	return static_cast<T*>(s.p);
}

double seconds_since(Clock::time_point t0) { return std::chrono::duration<double>(Clock::now() - t0).count(); }

int cuda_fail(cudaError_t e, const char* where)
{
	return fail(e == cudaErrorMemoryAllocation ? DMRGPP_OOM : DMRGPP_CUDA_ERROR,
	            std::string(where) + ": " + cudaGetErrorString(e));
}

} // namespace
} // namespace dmrgpp

extern "C" int dmrgpp_density_truncate(const dmrgpp_density_desc* d, size_t m, double tolerance,
                                       size_t m_min, double* eigenvalues, double* vectors, size_t* kept,
                                       size_t* kept_total, double* discarded)
{
	DMRGPP_TRACE("dmrgpp_density_truncate");
	using namespace dmrgpp;
	if (!d || !eigenvalues || !kept || !kept_total || !discarded)
		return fail(DMRGPP_INVALID_ARG, "null argument");
	if (d->npatches == 0 || d->ngroups == 0 || d->ntargets == 0)
		return fail(DMRGPP_INVALID_ARG, "npatches, ngroups and ntargets must be >= 1");
	if (!d->left_patch_size || !d->right_patch_size || !d->patch_group || !d->group_size || !d->psi)
		return fail(DMRGPP_INVALID_ARG, "null table");
	if (d->side != 0 && d->side != 1)
		return fail(DMRGPP_INVALID_ARG, "side must be 0 (system) or 1 (environment)");
	const size_t np = d->npatches, ng = d->ngroups, nt = d->ntargets;
	const auto   t_start = Clock::now();
	for (double& x : g_trunc_times)
		x = 0.0;
	// sector layout, group membership and sizes
	std::vector<long long> xy(np + 1, 0);
	for (size_t p = 0; p < np; ++p) {
		const size_t l = d->left_patch_size[p], r = d->right_patch_size[p];
		if (l < 1 || r < 1 || l > size_t(INT_MAX) || r > size_t(INT_MAX))
			return fail(DMRGPP_INVALID_ARG, "patch " + std::to_string(p) + " has an empty or oversized group");
		if (d->patch_group[p] >= ng)
			return fail(DMRGPP_INVALID_ARG, "patch " + std::to_string(p) + ": group out of range");
		const size_t n = d->side == 0 ? l : r;
		if (d->group_size[d->patch_group[p]] != n)
			return fail(DMRGPP_INVALID_ARG,
			            "patch " + std::to_string(p) + ": its group's size differs from the patch's "
			                + (d->side == 0 ? "left" : "right") + " size");
		xy[p + 1] = xy[p] + (long long)(l * r);
	}
	const long long D = xy[np];
	std::vector<long long> goff(ng + 1, 0);
	size_t                 nmax = 0, N = 0;
	for (size_t g = 0; g < ng; ++g) {
		const size_t n = d->group_size[g];
		if (n > 46340) // n^2 within INT_MAX for the GEMM tiles' leading dimensions
			return fail(DMRGPP_INVALID_ARG, "group " + std::to_string(g) + " is too large");
		goff[g + 1] = goff[g] + (long long)(n * n);
		nmax        = std::max(nmax, n);
		N += n;
	}
	if (m_min > m)
		return fail(DMRGPP_INVALID_ARG, "m_min must not exceed m");
	std::vector<double> w(nt, 1.0);
	if (d->weights)
		for (size_t t = 0; t < nt; ++t)
			w[t] = d->weights[t];

	int prev = -1;
	cudaGetDevice(&prev);
	const int dev = d->device >= 0 ? d->device : prev;
	if (dev != prev && cudaSetDevice(dev) != cudaSuccess)
		return fail(DMRGPP_INVALID_ARG, "cannot select device " + std::to_string(dev));
	struct Restore {
		int dev, prev;
		~Restore()
		{
			if (dev != prev && prev >= 0)
				cudaSetDevice(prev);
		}
	} restore { dev, prev };
	cudaStream_t st = static_cast<cudaStream_t>(d->stream);

	// weighted transposed copies of every patch block, and the GEMM lists:
	// side 0: rho_g += (w X_p^T)(X_p), A = XT (l x r), B = X (r x l), K = r
	// side 1: rho_g += (X_p)(w X_p^T), A = X (r x l), B = XT (l x r), K = l
	std::vector<TransposeTile> tt;
	std::vector<std::vector<GemmSeg>> gseg(ng);
	for (size_t t = 0; t < nt; ++t)
		for (size_t p = 0; p < np; ++p) {
			const int       l = int(d->left_patch_size[p]), r = int(d->right_patch_size[p]);
			const long long off = (long long)t * D + xy[p];
			for (int c0 = 0; c0 < l; c0 += 32)
				for (int r0 = 0; r0 < r; r0 += 32)
					tt.push_back({ off, off, r, l, r0, c0, w[t] });
			GemmSeg s {};
			s.a_off = off;
			s.b_off = off;
			if (d->side == 0) {
				s.lda = l;
				s.ldb = r;
				s.K   = r;
			} else {
				s.lda = r;
				s.ldb = l;
				s.K   = l;
			}
			s.dep = int(p);
			gseg[d->patch_group[p]].push_back(s);
		}
	const int            bm = nmax > 192 ? 64 : 32;
	std::vector<GemmSeg>  segs;
	std::vector<GemmTile> tiles;
	for (size_t g = 0; g < ng; ++g) {
		if (gseg[g].empty())
			continue;
		const int sb = int(segs.size());
		segs.insert(segs.end(), gseg[g].begin(), gseg[g].end());
		const int n = int(d->group_size[g]);
		for (int n0 = 0; n0 < n; n0 += bm)
			for (int m0 = 0; m0 < n; m0 += bm) {
				GemmTile tl {};
				tl.c_off     = goff[g];
				tl.ldc       = n;
				tl.M         = n;
				tl.N         = n;
				tl.m0        = m0;
				tl.n0        = n0;
				tl.seg_begin = sb;
				tl.seg_end   = int(segs.size());
				tiles.push_back(tl);
			}
	}

	double*        xt    = nullptr;
	double*        rho   = nullptr;
	TransposeTile* d_tt  = nullptr;
	GemmSeg*       d_seg = nullptr;
	GemmTile*      d_til = nullptr;
	struct Free {
		double**        a;
		double**        b;
		TransposeTile** c;
		GemmSeg**       s;
		GemmTile**      t;
		~Free()
		{
			dev_free(*a);
			dev_free(*b);
			dev_free(*c);
			dev_free(*s);
			dev_free(*t);
		}
	} release { &xt, &rho, &d_tt, &d_seg, &d_til };
	cudaError_t e;
	const size_t rho_elems = size_t(std::max<long long>(goff[ng], 1));
	if ((e = init_grouped_dgemm()) || (e = dev_malloc(&xt, size_t(nt) * size_t(std::max<long long>(D, 1)) * sizeof(double)))
	    || (e = dev_malloc(&rho, rho_elems * sizeof(double)))
	    || (e = dev_malloc(&d_tt, std::max<size_t>(tt.size(), 1) * sizeof(TransposeTile)))
	    || (e = dev_malloc(&d_seg, std::max<size_t>(segs.size(), 1) * sizeof(GemmSeg)))
	    || (e = dev_malloc(&d_til, std::max<size_t>(tiles.size(), 1) * sizeof(GemmTile))))
		return cuda_fail(e, "density-matrix allocation");
	if ((e = cudaMemcpyAsync(d_tt, tt.data(), tt.size() * sizeof(TransposeTile), cudaMemcpyHostToDevice, st))
	    || (e = cudaMemcpyAsync(d_seg, segs.data(), segs.size() * sizeof(GemmSeg), cudaMemcpyHostToDevice, st))
	    || (e = cudaMemcpyAsync(d_til, tiles.data(), tiles.size() * sizeof(GemmTile), cudaMemcpyHostToDevice, st))
	    || (e = cudaMemsetAsync(rho, 0, rho_elems * sizeof(double), st)))
		return cuda_fail(e, "density-matrix set-up");
	const int tgrid = int(std::min<size_t>(std::max<size_t>(tt.size(), 1), 148 * 16));
	k_transpose_tiles<<<tgrid, 256, 0, st>>>(d->psi, xt, d_tt, int(tt.size()));
	if (!tiles.empty()) {
		GemmArgs ga {};
		ga.A      = d->side == 0 ? xt : d->psi;
		ga.B      = d->side == 0 ? d->psi : xt;
		ga.C      = rho;
		ga.segs   = d_seg;
		ga.tiles  = d_til;
		ga.ntiles = int(tiles.size());
		if ((e = launch_grouped_dgemm(ga, bm, bm, st)))
			return cuda_fail(e, "density-matrix GEMM launch");
	}
	std::vector<long long> eoff(ng + 1, 0);
	for (size_t g = 0; g < ng; ++g)
		eoff[g + 1] = eoff[g] + (long long)d->group_size[g];
	// largest groups first
	std::vector<size_t> by_size(ng);
	std::iota(by_size.begin(), by_size.end(), size_t(0));
	std::stable_sort(by_size.begin(), by_size.end(),
	                 [&](size_t x, size_t y) { return d->group_size[x] > d->group_size[y]; });
	std::vector<GroupReduction> ge;
	const int                   hw = host_threads();
	auto                        not_converged = [&](size_t g) {
        return fail(DMRGPP_NOT_CONVERGED, "eigensolver of group " + std::to_string(g) + " did not converge");
	};
	// reduction and eigenvalues of every group on the device, except of those
	// whose vectors do not fit its shared memory: the host cores take these
	// meanwhile
	size_t limit = 0;
	if ((e = tridiag_limit(&limit)))
		return cuda_fail(e, "tridiagonal kernel attributes");
	std::vector<size_t>     hg; // groups of the host, and their places in its buffers
	std::vector<long long>  hoff(1, 0);
	std::vector<TridiagJob> tj;
	std::vector<BisectJob>  bj;
	long long               work_elems = 0;
	int                     vec        = 1; // largest group of the device
	for (size_t g : by_size) {
		const int n = int(d->group_size[g]);
		if (n == 0)
			continue;
		if (size_t(n) > limit) {
			hg.push_back(g);
			hoff.push_back(hoff.back() + (long long)n * n);
			continue;
		}
		tj.push_back({ goff[g], work_elems, eoff[g], n, int(g) });
		work_elems += (long long)n * n;
		vec = std::max(vec, n);
		for (int k0 = 0; k0 < n; k0 += kBisThreads / 8)
			bj.push_back({ eoff[g], n, k0 });
	}
	double *work = nullptr, *tri = nullptr; // tri: d, off, eigenvalues, beta (N each)
	void*   d_tj = nullptr;
	struct FreeT {
		double **a, **b;
		void**   c;
		~FreeT()
		{
			dev_free(*a);
			dev_free(*b);
			dev_free(*c);
		}
	} freet { &work, &tri, &d_tj };
	// the lists and the groups' shifts in one allocation
	const size_t tjb = tj.size() * sizeof(TridiagJob), bjb = bj.size() * sizeof(BisectJob);
	std::vector<unsigned char> lists(tjb + bjb);
	std::copy_n(reinterpret_cast<const unsigned char*>(tj.data()), tjb, lists.data());
	std::copy_n(reinterpret_cast<const unsigned char*>(bj.data()), bjb, lists.data() + tjb);
	const size_t N1    = std::max<size_t>(N, 1);
	double*      h_tri = pinned<double>(0, 3 * N1 + (ng + 1) / 2 + 1);
	double*      h_rho = pinned<double>(1, size_t(hoff.back()));
	if (!h_tri || !h_rho)
		return fail(DMRGPP_OOM, "page-locked host buffers for the density matrices");
	int*         h_shift  = reinterpret_cast<int*>(h_tri + 3 * N1);
	const size_t tri_smem = 5 * size_t(vec) * sizeof(double), bis_smem = 2 * size_t(vec) * sizeof(double);
	if ((e = cudaGetLastError()) || (e = dev_malloc(&work, size_t(std::max(work_elems, 1LL)) * sizeof(double)))
	    || (e = dev_malloc(&tri, 4 * N1 * sizeof(double)))
	    || (e = dev_malloc(&d_tj, lists.size() + ng * sizeof(int) + 16)))
		return cuda_fail(e, "tridiagonal allocation");
	unsigned char* lp      = static_cast<unsigned char*>(d_tj);
	int*           d_shift = reinterpret_cast<int*>(lp + lists.size());
	if (!lists.empty() && (e = cudaMemcpyAsync(lp, lists.data(), lists.size(), cudaMemcpyHostToDevice, st)))
		return cuda_fail(e, "tridiagonal set-up");
	struct Event {
		cudaEvent_t v = nullptr;
		~Event()
		{
			if (v)
				cudaEventDestroy(v);
		}
	} formed; // the density matrices are there, the host's also in its buffer
	for (size_t q = 0; q < hg.size(); ++q)
		if ((e = cudaMemcpyAsync(h_rho + hoff[q], rho + goff[hg[q]], size_t(hoff[q + 1] - hoff[q]) * sizeof(double),
		                         cudaMemcpyDeviceToHost, st)))
			return cuda_fail(e, "density matrices");
	if ((e = cudaEventCreateWithFlags(&formed.v, cudaEventDisableTiming)) || (e = cudaEventRecord(formed.v, st)))
		return cuda_fail(e, "density matrices");
	double *dd = tri, *doff = tri + N1, *dw = tri + 2 * N1, *dbeta = tri + 3 * N1;
	if (!tj.empty()) {
		k_tridiag<<<unsigned(tj.size() * kTriCluster), kTriThreads, tri_smem, st>>>(
		    rho, work, reinterpret_cast<const TridiagJob*>(lp), dd, doff, dbeta, d_shift, vec);
		k_bisect<<<unsigned(bj.size()), kBisThreads, bis_smem, st>>>(
		    dd, doff, dw, reinterpret_cast<const BisectJob*>(lp + tjb));
	}
	if ((e = cudaGetLastError())
	    || (e = cudaMemcpyAsync(h_tri, tri, 3 * N1 * sizeof(double), cudaMemcpyDeviceToHost, st))
	    || (e = cudaMemcpyAsync(h_shift, d_shift, ng * sizeof(int), cudaMemcpyDeviceToHost, st)))
		return cuda_fail(e, "tridiagonal reduction");
	if ((e = cudaEventSynchronize(formed.v)))
		return cuda_fail(e, "density matrices");
	g_trunc_times[DMRGPP_TRUNC_RHO] = seconds_since(t_start);
	auto tp                         = Clock::now();
	ge.assign(ng, GroupReduction {});
	if (!hg.empty()) {
		std::vector<GroupReduction> red;
		std::vector<size_t>         hn;
		std::vector<double*>        ga, gw;
		for (size_t q = 0; q < hg.size(); ++q) {
			hn.push_back(d->group_size[hg[q]]);
			ga.push_back(h_rho + hoff[q]);
			gw.push_back(eigenvalues + eoff[hg[q]]);
		}
		const bool ok = group_eigenvalues(hg.size(), hn.data(), ga.data(), gw.data(), red, hw);
		for (size_t q = 0; q < hg.size(); ++q) {
			if (!ok && !red[q].ok) {
				cudaStreamSynchronize(st); // the copies to this thread's buffers
				return not_converged(hg[q]);
			}
			ge[hg[q]] = std::move(red[q]);
		}
	}
	if ((e = cudaStreamSynchronize(st)))
		return cuda_fail(e, "tridiagonal reduction");
	for (const TridiagJob& j : tj) {
		GroupReduction& r  = ge[size_t(j.group)];
		const size_t    n  = size_t(j.n);
		const double *  gd = h_tri + j.e_off, *go = gd + N1, *gv = go + N1;
		r.d.assign(gd, gd + n);
		r.off.assign(go, go + std::max<size_t>(n - 1, 1));
		r.shift = h_shift[j.group];
		double top = -INFINITY; // bisection may leave equal values an ulp out of order
		for (size_t i = 0; i < n; ++i) {
			if (!std::isfinite(gd[i]) || !std::isfinite(go[i]) || !std::isfinite(gv[i]))
				return not_converged(size_t(j.group));
			top                                  = std::max(top, gv[i]);
			eigenvalues[j.e_off + (long long)i] = r.shift ? std::ldexp(top, -r.shift) : top;
			if (r.shift)
				r.scaled_values.push_back(top);
		}
	}

	g_trunc_times[DMRGPP_TRUNC_EIGENVALUES] = seconds_since(tp);
	tp                                      = Clock::now();
	// rank every state (ascending eigenvalue, then group, then index) and keep K
	std::vector<long long> order(N);
	std::iota(order.begin(), order.end(), 0LL);
	std::vector<size_t> group_of(N);
	for (size_t g = 0; g < ng; ++g)
		for (long long q = eoff[g]; q < eoff[g + 1]; ++q)
			group_of[size_t(q)] = g;
	std::stable_sort(order.begin(), order.end(),
	                 [&](long long a, long long b) { return eigenvalues[a] < eigenvalues[b]; });
	std::vector<double> sorted(N);
	for (size_t q = 0; q < N; ++q)
		sorted[q] = eigenvalues[order[q]];
	const size_t K      = std::min(compute_kept(m, tolerance, m_min, sorted), N);
	const size_t remove = N - K;
	double       disc   = 0.0;
	for (size_t g = 0; g < ng; ++g)
		kept[g] = d->group_size[g];
	for (size_t q = 0; q < remove; ++q) {
		disc += std::fabs(sorted[q]);
		--kept[group_of[size_t(order[q])]];
	}
	g_trunc_times[DMRGPP_TRUNC_SELECT] = seconds_since(tp);
	tp                                 = Clock::now();
	if (vectors) {
		// the kept eigenvectors: inverse iteration on each tridiagonal (host
		// cores), then V = Q Z on the device
		std::vector<long long> koff(ng + 1, 0);
		for (size_t g = 0; g < ng; ++g)
			koff[g + 1] = koff[g] + (long long)(d->group_size[g] * kept[g]);
		const size_t        kelems = size_t(std::max<long long>(koff[ng], 1));
		double* zk = pinned<double>(2, kelems);
		double* vo = pinned<double>(3, kelems);
		if (!zk || !vo)
			return fail(DMRGPP_OOM, "page-locked host buffers for the eigenvectors");
		std::vector<const double*> gwk(ng);
		std::vector<double*>       gz(ng);
		for (size_t g = 0; g < ng; ++g) {
			gwk[g] = eigenvalues + eoff[g] + (long long)(d->group_size[g] - kept[g]);
			gz[g]  = zk + koff[g];
		}
		group_eigenvectors(ng, d->group_size, kept, ge.data(), gwk.data(), gz.data(), hw);
		// the host's reflectors take the place of their density matrices, as the
		// device's have (h_rho's buffer is free again)
		parallel_for(hg.size(), [&](size_t q) {
			std::copy(ge[hg[q]].hv.begin(), ge[hg[q]].hv.end(), h_rho + hoff[q]);
		});
		g_trunc_times[DMRGPP_TRUNC_VECTORS_HOST] = seconds_since(tp);
		tp                                       = Clock::now();
		std::vector<ColumnJob> cj;
		for (size_t g = 0; g < ng; ++g)
			for (int j = 0; j < int(kept[g]); ++j)
				cj.push_back({ koff[g], koff[g], goff[g], eoff[g], int(d->group_size[g]), j, j, 0 });
		if (!cj.empty()) {
			double *   z = nullptr, *v = nullptr;
			ColumnJob* d_cj = nullptr;
			struct FreeV {
				double**    a[2];
				ColumnJob** j;
				~FreeV()
				{
					for (double** p : a)
						dev_free(*p);
					dev_free(*j);
				}
			} freev { { &z, &v }, &d_cj };
			if ((e = dev_malloc(&z, kelems * sizeof(double))) || (e = dev_malloc(&v, kelems * sizeof(double)))
			    || (e = dev_malloc(&d_cj, cj.size() * sizeof(ColumnJob))))
				return cuda_fail(e, "eigenvector allocation");
			for (size_t q = 0; q < hg.size(); ++q) {
				const GroupReduction& r = ge[hg[q]];
				if (kept[hg[q]] == 0 || r.beta.empty())
					continue;
				if ((e = cudaMemcpyAsync(rho + goff[hg[q]], h_rho + hoff[q], size_t(hoff[q + 1] - hoff[q]) * sizeof(double),
				                         cudaMemcpyHostToDevice, st))
				    || (e = cudaMemcpyAsync(dbeta + eoff[hg[q]], r.beta.data(), r.beta.size() * sizeof(double),
				                            cudaMemcpyHostToDevice, st)))
					return cuda_fail(e, "reflector upload");
			}
			if ((e = cudaMemcpyAsync(z, zk, kelems * sizeof(double), cudaMemcpyHostToDevice, st))
			    || (e = cudaMemcpyAsync(d_cj, cj.data(), cj.size() * sizeof(ColumnJob), cudaMemcpyHostToDevice, st)))
				return cuda_fail(e, "eigenvector set-up");
			const int cgrid = int(std::min<size_t>((cj.size() + 7) / 8, 148 * 8));
			k_back_transform<<<std::max(cgrid, 1), 256, 0, st>>>(z, v, rho, dbeta, d_cj, int(cj.size()));
			if ((e = cudaGetLastError())
			    || (e = cudaMemcpyAsync(vo, v, size_t(koff[ng]) * sizeof(double), cudaMemcpyDeviceToHost, st))
			    || (e = cudaStreamSynchronize(st)))
				return cuda_fail(e, "eigenvectors");
			parallel_for(ng, [&](size_t g) { // to the caller's (pageable) buffer, group by group
				std::copy(vo + koff[g], vo + koff[g + 1], vectors + koff[g]);
			});
		}
	}
	if (vectors)
		g_trunc_times[DMRGPP_TRUNC_VECTORS_DEVICE] = seconds_since(tp);
	g_trunc_times[DMRGPP_TRUNC_TOTAL] = seconds_since(t_start);
	*kept_total                       = K;
	*discarded                        = disc;
	return DMRGPP_OK;
}

extern "C" int dmrgpp_density_profile(double* t, int n)
{
	if (!t || n < 0 || n > DMRGPP_TRUNC_NPHASES)
		return dmrgpp::fail(DMRGPP_INVALID_ARG, "need 0 <= n <= DMRGPP_TRUNC_NPHASES and a buffer");
	for (int i = 0; i < n; ++i)
		t[i] = dmrgpp::g_trunc_times[i];
	return DMRGPP_OK;
}
