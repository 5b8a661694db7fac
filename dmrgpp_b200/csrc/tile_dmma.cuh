// Device building blocks shared by the FP64 grouped-GEMM kernels: one
// CTA-tile of C(BM x BN) = sum over K-segments of A(M x K) * B(K x N) on the
// FP64 tensor pipe (mma.sync m8n8k4 .f64), with operands staged global ->
// shared by cp.async in a STAGES-deep ring.
#pragma once

#include "kron_plan.h"

#include <cuda_runtime.h>

namespace dmrgpp {
namespace tile {

__device__ __forceinline__ unsigned smem_u32(const void* p)
{
	return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// 8-byte asynchronous global->shared copy; src_bytes = 0 zero-fills the
// destination without reading the source.
__device__ __forceinline__ void cp_async_8(unsigned dst, const double* src, bool pred)
{
	const int n = pred ? 8 : 0;
	asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(n)
	             : "memory");
}

// The same where `issue` holds; nothing at all otherwise (the predicate is
// inside: a branch around each copy costs more than the copy).
__device__ __forceinline__ void cp_async_8_if(bool issue, unsigned dst, const double* src, bool pred)
{
	const int n = pred ? 8 : 0;
	asm volatile("{\n\t.reg .pred p;\n\t"
	             "setp.ne.b32 p, %3, 0;\n\t"
	             "@p cp.async.ca.shared.global [%0], [%1], 8, %2;\n\t}\n" ::"r"(dst),
	             "l"(src), "r"(n), "r"(int(issue))
	             : "memory");
}

__device__ __forceinline__ void cp_async_commit()
{
	asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <int N> __device__ __forceinline__ void cp_async_wait()
{
	asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// D(8x8) += A(8x4) * B(4x8) on the FP64 tensor pipe.  Fragments: lane holds
// A[lane/4][lane%4], B[lane%4][lane/4], and C/D[lane/4][2*(lane%4) + {0,1}].
__device__ __forceinline__ void dmma_8x8x4(double& d0, double& d1, double a, double b)
{
	asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
	             : "+d"(d0), "+d"(d1)
	             : "d"(a), "d"(b));
}

// SKIP: rows and columns past the matrix are not copied at all.  Otherwise the
// copy engine zero-fills them, which takes fewer predicates: better where
// latency counts (ladder of 6000 states with 32 x 32 tiles 139 us against 148,
// transformation of 4000 states 35 against 37), worse for the persistent 64 x
// 64 tiles, whose registers are full (16000 states 1347 against 1309).
template <int BM_, int BN_, int BK_, int WM_, int WN_, int STAGES_, bool SKIP_ = false> struct Cfg {
	static constexpr int BM = BM_, BN = BN_, BK = BK_, WM = WM_, WN = WN_, STAGES = STAGES_;
	static constexpr bool SKIP = SKIP_;
	static constexpr int WARPS_M = BM / WM, WARPS_N = BN / WN;
	static constexpr int THREADS = WARPS_M * WARPS_N * 32;
	static constexpr int MI = WM / 8, NI = WN / 8;
	// shared layouts As[k][m] and Bs[n][k]; the +4 padding makes a warp's
	// fragment reads hit every bank pair exactly twice (the minimum for 256 B)
	static constexpr int LDA_S = BM + 4;
	static constexpr int LDB_S = BK + 4;
	static constexpr int A_STAGE = BK * LDA_S;
	static constexpr int B_STAGE = BN * LDB_S;
	static constexpr size_t SMEM = size_t(STAGES) * (A_STAGE + B_STAGE) * sizeof(double);
	static constexpr int A_LOADS = BM * BK / THREADS;
	static constexpr int B_LOADS = BK * BN / THREADS;
	// resident CTAs the register count has to allow: four of 64 x 64 tiles
	// (128 registers) beat three with room for a deeper ring (29.7 against
	// 28.2 TFLOP/s at K = 333); five of 32 x 32
	static constexpr int CTAS = BM == 64 && BK == 16 ? 4 : 1;
	static_assert(BM * BK % THREADS == 0 && BK * BN % THREADS == 0, "load split");
	static_assert(BK % 4 == 0 && WM % 8 == 0 && WN % 8 == 0, "mma shape");
};

template <class C> struct Acc {
	double v[C::MI][C::NI][2];
};

// The place of this thread's warp in the tile, turned by rot (any value).
template <class C> __device__ __forceinline__ int warp_slot(int rot)
{
	constexpr int W = C::THREADS / 32;
	static_assert((W & (W - 1)) == 0, "warps per CTA");
	return int((threadIdx.x >> 5) + unsigned(rot)) & (W - 1);
}

// acc = sum over segments [sb, se) of A_s[m0.., :] * B_s[:, n0..].
// smem must hold C::SMEM bytes; on return every cp.async of this CTA has
// completed and all threads have passed a barrier after the last shared read.
//
// Bound by the FP64 tensor pipe, which all resident CTAs share, so what does
// not feed it is kept off the issue slots and off the pipe itself:
// * a thread's operand addresses are formed once per segment and advanced by
//   additions (64-bit index products per copy cost 8% at 64 x 64 tiles, 11%
//   at 32 x 32: 26.0 -> 28.2 and 21.9 -> 24.2 TFLOP/s at K = 333);
// * the 8 x 8 blocks of a warp that lie outside the matrix and the k-steps
//   past the segment's end issue no MMA, so a ragged edge costs its size
//   rounded up to 8 (k: 4) and not to the tile;
// * `rot` turns the warps' places in the tile: a ragged tile leaves the same
//   places empty, and each scheduler's share of the pipe has to see all of
//   them in turn.
// Rows and columns past the matrix are zero-filled or (Cfg's SKIP) not loaded;
// what their shared words hold only reaches outputs that are not stored.  k
// past the segment's end is zero-filled.
// A segment's operands lie in Abase and Bbase, or (kSegXA, kSegXB) in X.
template <class C>
__device__ __forceinline__ void mma_tile(Acc<C>&        acc,
                                         double*        smem,
                                         const double*  Abase,
                                         const double*  Bbase,
                                         const double*  X,
                                         const GemmSeg* segs,
                                         int            sb,
                                         int            se,
                                         int            m0,
                                         int            n0,
                                         int            M,
                                         int            N,
                                         int            rot)
{
	double*   As   = smem;
	double*   Bs   = smem + C::STAGES * C::A_STAGE;
	const int tid  = threadIdx.x;
	const int lane = tid & 31;
	const int slot = warp_slot<C>(rot);
	const int wm   = slot % C::WARPS_M;
	const int wn   = slot / C::WARPS_M;

#pragma unroll
	for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
		for (int ni = 0; ni < C::NI; ++ni)
			acc.v[mi][ni][0] = acc.v[mi][ni][1] = 0.0;

	// 8 x 8 blocks of this warp with a row and a column inside the matrix
	const int  vm   = min(C::MI, max(0, (M - m0 - wm * C::WM + 7) >> 3));
	const int  vn   = min(C::NI, max(0, (N - n0 - wn * C::WN + 7) >> 3));
	const bool full = vm == C::MI && vn == C::NI;

	int total = 0;
	for (int s = sb; s < se; ++s)
		total += (segs[s].K + C::BK - 1) / C::BK;

	// this thread's copies of a stage: A rows am, k = ak + e * AK; B columns
	// bn + e * BNS, k = bk
	constexpr int AK  = C::THREADS / C::BM;
	constexpr int BNS = C::THREADS / C::BK;
	static_assert(C::THREADS % C::BM == 0 && C::THREADS % C::BK == 0, "load split");
	const int      am = tid % C::BM, ak = tid / C::BM;
	const int      bk = tid % C::BK, bn = tid / C::BK;
	const bool     arow = m0 + am < M;
	const int      ncol = N - n0 - bn; // B columns bn + e * BNS < bn + ncol exist
	const unsigned sa   = smem_u32(As + ak * C::LDA_S + am);
	const unsigned sbm  = smem_u32(Bs + bn * C::LDB_S + bk);

	int           ls    = sb; // segment being loaded
	int           kleft = 0;  // its k still to load
	const double* ap    = nullptr;
	const double* bp    = nullptr;
	long long     astep = 0, bstep = 0;
	auto          open = [&]() {
		const GemmSeg& g = segs[ls];
		kleft           = g.K;
		astep           = (long long)AK * g.lda;
		bstep           = (long long)BNS * g.ldb;
		// X in one operand's place; with X as B, A is the operators, which are
		// the pass's B
		const double* a = g.dep == kSegXA ? X : g.dep == kSegXB ? Bbase : Abase;
		const double* b = g.dep == kSegXB ? X : Bbase;
		ap              = a + g.a_off + (m0 + am) + (long long)ak * g.lda;
		bp              = b + g.b_off + (long long)(n0 + bn) * g.ldb + bk;
	};
	auto issue = [&](int stage) {
		while (kleft <= 0) { // an empty segment has no chunk
			open();
			++ls;
		}
		const unsigned da = sa + unsigned(stage * C::A_STAGE * 8);
		const unsigned db = sbm + unsigned(stage * C::B_STAGE * 8);
		const double*  p  = ap;
#pragma unroll
		for (int e = 0; e < C::A_LOADS; ++e) {
			const bool in = ak + e * AK < kleft;
			if (C::SKIP)
				cp_async_8_if(arow, da + unsigned(e * AK * C::LDA_S * 8), in ? p : Abase, in);
			else
				cp_async_8(da + unsigned(e * AK * C::LDA_S * 8), in && arow ? p : Abase, in && arow);
			p += astep;
		}
		ap                = p;
		const double* q   = bp;
		const bool    kin = bk < kleft;
#pragma unroll
		for (int e = 0; e < C::B_LOADS; ++e) {
			const bool cin = e * BNS < ncol;
			if (C::SKIP)
				cp_async_8_if(cin, db + unsigned(e * BNS * C::LDB_S * 8), kin ? q : Bbase, kin);
			else
				cp_async_8(db + unsigned(e * BNS * C::LDB_S * 8), kin && cin ? q : Bbase, kin && cin);
			q += bstep;
		}
		bp += C::BK;
		kleft -= C::BK;
	};
	static_assert(C::A_LOADS * AK == C::BK && C::B_LOADS * BNS == C::BN, "a stage's copies");

#pragma unroll
	for (int st = 0; st < C::STAGES - 1; ++st) {
		if (st < total)
			issue(st);
		cp_async_commit();
	}

	int cseg = sb, ck = 0; // segment being consumed and its k still to consume
	int cst = 0, lst = C::STAGES - 1;
	for (int it = 0; it < total; ++it) {
		cp_async_wait<C::STAGES - 2>();
		__syncthreads();
		if (it + C::STAGES - 1 < total)
			issue(lst);
		cp_async_commit();
		lst = lst + 1 == C::STAGES ? 0 : lst + 1;
		while (ck <= 0)
			ck = segs[cseg++].K;

		const double* as = As + cst * C::A_STAGE + wm * C::WM + (lane >> 2);
		const double* bs = Bs + cst * C::B_STAGE + (wn * C::WN + (lane >> 2)) * C::LDB_S;
		cst              = cst + 1 == C::STAGES ? 0 : cst + 1;
		if (full && ck >= C::BK) {
#pragma unroll
			for (int ks = 0; ks < C::BK; ks += 4) {
				double af[C::MI], bf[C::NI];
#pragma unroll
				for (int mi = 0; mi < C::MI; ++mi)
					af[mi] = as[(ks + (lane & 3)) * C::LDA_S + mi * 8];
#pragma unroll
				for (int ni = 0; ni < C::NI; ++ni)
					bf[ni] = bs[ni * 8 * C::LDB_S + ks + (lane & 3)];
#pragma unroll
				for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
					for (int ni = 0; ni < C::NI; ++ni)
						dmma_8x8x4(acc.v[mi][ni][0], acc.v[mi][ni][1], af[mi], bf[ni]);
			}
		} else if (vm > 0 && vn > 0) {
			// unrolled: the next step's fragment loads overlap this one's MMAs
			// (one at a time, a transformation of patches below a tile took 18
			// us instead of 14)
			const int kv = min(ck, C::BK);
#pragma unroll
			for (int ks = 0; ks < C::BK; ks += 4) {
				if (ks >= kv)
					break;
				double af[C::MI], bf[C::NI];
#pragma unroll
				for (int mi = 0; mi < C::MI; ++mi)
					af[mi] = mi < vm ? as[(ks + (lane & 3)) * C::LDA_S + mi * 8] : 0.0;
#pragma unroll
				for (int ni = 0; ni < C::NI; ++ni)
					bf[ni] = ni < vn ? bs[ni * 8 * C::LDB_S + ks + (lane & 3)] : 0.0;
#pragma unroll
				for (int mi = 0; mi < C::MI; ++mi)
					if (mi < vm) {
#pragma unroll
						for (int ni = 0; ni < C::NI; ++ni)
							if (ni < vn)
								dmma_8x8x4(acc.v[mi][ni][0], acc.v[mi][ni][1], af[mi], bf[ni]);
					}
			}
		}
		ck -= C::BK;
	}
	cp_async_wait<0>();
	__syncthreads(); // shared ring free for the next tile of this CTA
}

// Row and column, inside the tile, of accumulator element (mi, ni, h) of a
// warp at place `slot` (warp_slot).
template <class C> __device__ __forceinline__ int acc_row(int slot, int mi)
{
	return (slot % C::WARPS_M) * C::WM + mi * 8 + ((threadIdx.x & 31) >> 2);
}
template <class C> __device__ __forceinline__ int acc_col(int slot, int ni, int h)
{
	return (slot / C::WARPS_M) * C::WN + ni * 8 + (threadIdx.x & 3) * 2 + h;
}

} // namespace tile
} // namespace dmrgpp
