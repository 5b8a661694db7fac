// FP64 grouped GEMM for the two Kronecker passes (see kron_gemm.cuh).
#include "kron_gemm.cuh"
#include "tile_dmma.cuh"

namespace dmrgpp {
namespace {

using tile::Cfg;

template <class C>
__global__ void __launch_bounds__(C::THREADS) grouped_dgemm_kernel(GemmArgs args)
{
	extern __shared__ __align__(16) double smem[];
	const GemmTile t = args.tiles[blockIdx.x];
	tile::Acc<C>   acc;
	tile::mma_tile<C>(acc, smem, args.A, args.B, args.X, args.segs, t.seg_begin, t.seg_end, t.m0, t.n0, t.M, t.N,
	                  int(blockIdx.x));
	const int slot = tile::warp_slot<C>(int(blockIdx.x));
	double*   Cp   = args.C + t.c_off;
#pragma unroll
	for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
		for (int ni = 0; ni < C::NI; ++ni)
#pragma unroll
			for (int h = 0; h < 2; ++h) {
				const int row = t.m0 + tile::acc_row<C>(slot, mi);
				const int col = t.n0 + tile::acc_col<C>(slot, ni, h);
				if (row < t.M && col < t.N)
					Cp[(long long)col * t.ldc + row] = acc.v[mi][ni][h];
			}
}

template <class C> cudaError_t launch_cfg(const GemmArgs& args, cudaStream_t stream)
{
	if (args.ntiles <= 0)
		return cudaSuccess;
	grouped_dgemm_kernel<C><<<args.ntiles, C::THREADS, C::SMEM, stream>>>(args);
	return cudaGetLastError();
}

using Cfg64 = Cfg<64, 64, 16, 32, 32, 2>;
using Cfg32 = Cfg<32, 32, 16, 16, 16, 3>;

template <class C> cudaError_t init_cfg()
{
	return cudaFuncSetAttribute(
	    grouped_dgemm_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(C::SMEM));
}

} // namespace

cudaError_t init_grouped_dgemm()
{
	cudaError_t e = init_cfg<Cfg64>();
	if (e == cudaSuccess)
		e = init_cfg<Cfg32>();
	return e;
}

cudaError_t launch_grouped_dgemm(const GemmArgs& args, int bm, int bn, cudaStream_t stream)
{
	if (bm == 64 && bn == 64)
		return launch_cfg<Cfg64>(args, stream);
	if (bm == 32 && bn == 32)
		return launch_cfg<Cfg32>(args, stream);
	return cudaErrorInvalidValue;
}

} // namespace dmrgpp
