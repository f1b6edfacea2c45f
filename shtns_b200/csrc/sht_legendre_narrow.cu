// Narrow Legendre tiles: 128 rows x 16 columns (four warps) for two to four
// field-components.  The SIMT kernels (sht_legendre_simt.cu) do no work for
// padding columns, but read Y through shared memory at a row or k per lane and
// coefficients by broadcasts, which fills the shared-memory path at half of
// the FP64 rate; these tiles pad to four components and run at the MMA's.
// Stage times, SIMT / these tiles: analysis lmax 511, 3 components 86 / 54 us,
// lmax 1023, 3: 424 / 283 us, lmax 2047, 4: 2.69 / 1.88 ms; synthesis lmax 511,
// 4 components 77 / 53 us (the whole list is at leg_simt_selected).
#include "sht_internal.h"
#include "sht_legendre_tiles.h"

namespace {

template <int SEG, bool RB>
__global__ void __launch_bounds__(leg_nt(5), leg_minb(5)) leg_synth_narrow_kernel(LegParams p)
{
	leg_synth_tile<SEG, 5, RB>(p, p.im0 + blockIdx.y, blockIdx.x, 0);
}

template <int SEG, bool RB>
__global__ void __launch_bounds__(leg_nt(5), leg_minb(5)) leg_analys_narrow_kernel(LegParams p)
{
	leg_analys_tile<SEG, 5, RB>(p, p.im0 + blockIdx.y, blockIdx.x, 0);
}

template <class F>
void by_seg(int ckseg, F f)
{
	switch (ckseg) {
		case 8: f(std::integral_constant<int, 8>{}); break;
		case 16: f(std::integral_constant<int, 16>{}); break;
		default: f(std::integral_constant<int, 32>{}); break;
	}
}

} // namespace

void launch_leg_synth_narrow(const LegParams& p, cudaStream_t st)
{
	const dim3 grid((p.nlat_2 + 127) / 128, p.mlim + 1 - p.im0);
	by_seg(p.ckseg, [&](auto SC) {
		constexpr int SEG = decltype(SC)::value;
		if (p.rb.n) leg_synth_narrow_kernel<SEG, true><<<grid, leg_nt(5), 0, st>>>(p);
		else leg_synth_narrow_kernel<SEG, false><<<grid, leg_nt(5), 0, st>>>(p);
	});
}

void launch_leg_analys_narrow(const LegParams& p, int kmax_all, cudaStream_t st)
{
	const dim3 grid((kmax_all + 127) / 128, p.mlim + 1 - p.im0);
	by_seg(p.ckseg, [&](auto SC) {
		constexpr int SEG = decltype(SC)::value;
		if (p.rb.n) leg_analys_narrow_kernel<SEG, true><<<grid, leg_nt(5), 0, st>>>(p);
		else leg_analys_narrow_kernel<SEG, false><<<grid, leg_nt(5), 0, st>>>(p);
	});
}
