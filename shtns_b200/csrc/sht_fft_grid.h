// Access to the spatial grids of the FFT kernels, in double or single precision.
#pragma once

#include "sht_internal.h"

namespace shtb_fft_grid {

// Grid element type G: double, or float for the single-precision transforms
// (converted where the grid is read or written; the passes stay in FP64).
template <class G> struct Pair;
template <> struct Pair<double> { using T = double2; };
template <> struct Pair<float> { using T = float2; };

template <class G>
__device__ __forceinline__ void store_pair(G* o, double2 z, bool v2)
{
	typename Pair<G>::T v;
	v.x = (G) z.x; v.y = (G) z.y;
	if (v2) *reinterpret_cast<typename Pair<G>::T*>(o) = v;
	else { o[0] = v.x; o[1] = v.y; }
}
// Loads hand over the pair as it is stored and the caller widens it once all its
// loads are issued: a conversion beside the load, on one of the paths that the
// layout and the alignment select at run time, waits for that load before the
// next one.  The first passes with the conversion inside took 465 us for 50
// single-precision grids of 768 x 1536 (phi-contiguous; double 200), now 196.
__device__ __forceinline__ double2 widen(double2 v) { return v; }
__device__ __forceinline__ double2 widen(float2 v) { return make_double2(v.x, v.y); }

template <class G>
__device__ __forceinline__ typename Pair<G>::T load_pair(const G* i, bool v2)
{
	if (v2) return __ldg(reinterpret_cast<const typename Pair<G>::T*>(i));
	typename Pair<G>::T v;
	v.x = __ldg(i); v.y = __ldg(i + 1);
	return v;
}
template <class G>
__device__ __forceinline__ G* grid_out(const FftParams& p, int c, int fc)
{
	return reinterpret_cast<G*>(c == 0 ? p.spat[0] : c == 1 ? p.spat[1] : p.spat[2]) + (long)(fc - c * p.nf) * p.spat_dist;
}
template <class G>
__device__ __forceinline__ const G* grid_in(const FftParams& p, int c, int fc)
{
	return reinterpret_cast<const G*>(c == 0 ? p.spat_in[0] : c == 1 ? p.spat_in[1] : p.spat_in[2]) + (long)(fc - c * p.nf) * p.spat_dist;
}

} // namespace shtb_fft_grid
