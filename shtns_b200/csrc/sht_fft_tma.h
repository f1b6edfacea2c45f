// Tensor copies of latitude tiles, shared by the FFT kernels (sht_fft.cu,
// sht_fft_gen.cu): bounded mbarrier waits, 3-d tiled copies without multicast,
// and the tensor maps of their sources.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace shtb_fft_tma {

constexpr uint64_t FT_WAIT_NS = 1000000000ull;   // time limit of every mbarrier wait

__device__ __forceinline__ uint32_t su32(const void* ptr) { return static_cast<uint32_t>(__cvta_generic_to_shared(ptr)); }

__device__ __forceinline__ uint64_t gtimer()
{
	uint64_t t;
	asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
	return t;
}

__device__ __forceinline__ bool fbar_wait(uint64_t* bar, uint32_t parity)
{
	const uint32_t a = su32(bar);
	const uint64_t t0 = gtimer();
	for (int it = 0;; it++) {
		if ((it & 1023) == 1023 && gtimer() - t0 > FT_WAIT_NS) return false;
		uint32_t done;
		asm volatile("{\n\t.reg .pred p;\n\t"
		             "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
		             "selp.u32 %0, 1, 0, p;\n\t}"
		             : "=r"(done) : "r"(a), "r"(parity) : "memory");
		if (done) return true;
	}
}

__device__ __forceinline__ void tma_tile3(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar)
{
	asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
	             :: "r"(su32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(su32(bar))
	             : "memory");
}

// the driver's tensor-map encoder, resolved once (thread-safe static initialisation)
inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
	static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
		void* f = nullptr;
		cudaDriverEntryPointQueryResult q;
		if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
		    q == cudaDriverEntryPointSuccess)
			return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
		cudaGetLastError();
		return (PFN_cuTensorMapEncodeTiled_v12000) nullptr;
	}();
	return fn;
}

// 3-d tensor map of FP64 (or, with f32, FP32) values, dims / byte strides of dims 1 and 2 / box, no swizzle,
// zero fill out of range
inline bool encode3(CUtensorMap* m, const void* base, uint64_t d0, uint64_t d1, uint64_t d2, uint64_t s1, uint64_t s2,
             uint32_t b0, uint32_t b1, bool f32 = false)
{
	PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
	if (!enc || ((uintptr_t) base & 15) || (s1 & 15) || (s2 & 15) || ((b0 * (f32 ? 4 : 8)) & 15)) return false;
	const cuuint64_t dims[3] = {d0, d1, d2};
	const cuuint64_t strides[2] = {s1, s2};
	const cuuint32_t box[3] = {b0, b1, 1};
	const cuuint32_t es[3] = {1, 1, 1};
	return enc(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<void*>(base), dims, strides, box, es,
	           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
	           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

} // namespace shtb_fft_tma
