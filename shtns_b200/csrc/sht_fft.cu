// Longitude (phi) FFT stage on sm_100a.
//
// Replaces the reference's FFTW / cuFFT step (sht_init.c:353-518,
// sht_gpu.cu:372-446).  As in the reference, two real latitudes a, b are
// packed into one complex sequence z = v_a + i v_b, so one complex DFT of
// length nphi transforms a latitude pair; the spectra are separated with
// Hermitian symmetry.  A tile is one field-component and 2*S consecutive
// latitudes; its S complex sequences are transformed in shared memory by a
// self-sorting Stockham chain.  Three kernel families:
//   * generic kernels (sht_fft_gen.cu): one tile per CTA, radices 2 .. 16
//     chosen at run time (any supported nphi);
//   * fused kernels (fft3_*): nphi = 3 * 2^k with a compile-time radix chain
//     in one padded in-place buffer, one tile per CTA;
//   * prefetching kernels (fft4_*, the default up to nphi 3072): persistent
//     CTAs that fetch their next tile with tensor copies while the current one
//     is transformed (below).
//
// Synthesis input is F[fc][m][theta] (m <= mlim, exact Fourier coefficients of
// each latitude); output is v(phi_j) = sum_m (2 - delta_m0) Re(F_m e^{i m phi_j}).
// Analysis computes F_m = (1/nphi) sum_j v(phi_j) e^{-i m phi_j}.
// The spatial arrays are theta-contiguous (v[j*nlat + theta]) or
// phi-contiguous (v[theta*nphi + j]).
#include "sht_internal.h"
#include "sht_dft.h"
#include "sht_fft_tma.h"
#include "sht_fft_grid.h"

#include <algorithm>
#include <atomic>
#include <type_traits>
#include <cstdint>

namespace {

using namespace shtb_dft;
using namespace shtb_fft_tma;
using namespace shtb_fft_grid;

// ===========================================================================
// Fused kernels for nphi = 3 * 2^k (192 ... 6144), the sizes of Gauss grids
// with nphi = 2 nlat = 3 (lmax+1).  The radix sequence is fixed at compile
// time, so every index, stride and twiddle step is a constant.  The first
// pass reads its butterfly inputs straight from global memory (no staging
// copy) and, for synthesis, the last pass writes straight to global memory.
// Intermediate passes work in place in one padded shared buffer: each thread
// loads its butterflies into registers, the block synchronises, then writes.
// Thread g of the block handles sequence g % S and butterfly g / S, so the
// S sequences of a butterfly index are neighbours in a warp (contiguous
// 16-byte latitude pairs in global memory).
template <int... Rs> struct RadixList {};

// Pass chain of nphi = N and complex values per thread D (the CTA has S N / D
// threads).  Few long passes win where the tile arrives by tensor copies and
// the shared memory allows two CTAs per SM whatever their threads: each pass is
// a round trip through shared memory and two barriers.  Measured (FFT stages,
// synthesis / analysis, us; before: 8 8 8 3, 8 8 4 3, 8 8 4 4 3 and 8 4 4 3 with
// 8 values per thread): nphi 1536, 96 grids of 768 latitudes 430/399 -> 398/364;
// 768, 256 x 384 278/243 -> 254/225; 3072, 6 phi-contiguous x 1536 129/140 ->
// 106/115; 384, 64 phi-contiguous x 192 25.1/26.5 -> 22.5/23.6.  1536 as 12 16 8
// (12 values per thread) spills: 492/395.  192 as 16 12 or 8 4 6, and two passes
// for the 96 and 128 of the four-step kernels, were not faster.
template <int N> struct NphiPlan;
template <> struct NphiPlan<192>  { using L = RadixList<8, 8, 3>; static constexpr int D = 8; };
template <> struct NphiPlan<384>  { using L = RadixList<8, 8, 6>; static constexpr int D = 8; };
template <> struct NphiPlan<768>  { using L = RadixList<16, 8, 6>; static constexpr int D = 16; };
template <> struct NphiPlan<1536> { using L = RadixList<16, 16, 6>; static constexpr int D = 16; };
template <> struct NphiPlan<3072> { using L = RadixList<16, 16, 12>; static constexpr int D = 16; };
template <> struct NphiPlan<48>  { using L = RadixList<8, 6>; static constexpr int D = 8; };
template <> struct NphiPlan<64>  { using L = RadixList<8, 8>; static constexpr int D = 8; };
template <> struct NphiPlan<96>  { using L = RadixList<8, 4, 3>; static constexpr int D = 8; };
template <> struct NphiPlan<128> { using L = RadixList<8, 4, 4>; static constexpr int D = 8; };
template <> struct NphiPlan<6144> { using L = RadixList<8, 8, 8, 4, 3>; static constexpr int D = 8; };
template <> struct NphiPlan<12288> { using L = RadixList<8, 8, 8, 8, 3>; static constexpr int D = 8; };

// CTAs per SM of the prefetching kernels that the shared memory allows
constexpr int fft4_minb(int SN) { return 6144 / SN < 1 ? 1 : (6144 / SN > 16 ? 16 : 6144 / SN); }

template <int N, int S>
struct Geo {
	static constexpr int A = N + (N >> 3);
	// sequence stride 8/S mod 8 (16-byte units) for S <= 8, 1 mod 8 beyond, so
	// that the 8 lanes of a 16-byte access phase, on consecutive sequences,
	// hit distinct banks
	static constexpr int SEQ = A + (((S >= 8 ? 1 : 8 / S) - A) & 7);
	// D values per thread, at most 768 threads (more values per thread beyond)
	static constexpr int D = NphiPlan<N>::D;
	static constexpr int T = (S * N / D <= 768) ? S * N / D : 768;
	static __device__ __forceinline__ int at(int s, int i) { return s * SEQ + i + (i >> 3); }
};

// twiddle powers u[q] *= w^q, w = exp(sign 2 pi i k step / N)
template <int R>
__device__ __forceinline__ void twiddle(double2* u, const double2* __restrict__ tw, int idx, int sign)
{
	double2 w1 = __ldg(tw + idx);
	if (sign < 0) w1.y = -w1.y;
	if constexpr (R > 8) twiddles<R>(u, w1);
	else {
		double2 w = w1;
		#pragma unroll
		for (int q = 1; q < R; q++) {
			u[q] = cmul(u[q], w);
			if (q + 1 < R) w = cmul(w, w1);
		}
	}
}

// One middle pass (in place in X).  P = product of earlier radices.
// DENSE: the outputs go to X[j * S + s] (rows of S complex values, for a
// tensor store) instead of the padded sequence layout
template <int N, int S, int R, int P, bool DENSE = false>
__device__ __forceinline__ void mid_pass(double2* X, const double2* __restrict__ tw, int sign, int tid)
{
	using G = Geo<N, S>;
	constexpr int NBF = N / R, TOT = S * NBF, NB = (TOT + G::T - 1) / G::T, TSTEP = N / (P * R);
	double2 u[NB][R];
	int dst[NB], ss[NB];
	#pragma unroll
	for (int i = 0; i < NB; i++) {
		const int g = tid + i * G::T;
		dst[i] = -1;
		if (g < TOT) {
			const int s = g % S, b = g / S, k = b % P;
			#pragma unroll
			for (int q = 0; q < R; q++) u[i][q] = X[G::at(s, b + q * NBF)];
			if (P > 1 && k) twiddle<R>(u[i], tw, k * TSTEP, sign);
			Dft<R>::run(u[i], sign);
			dst[i] = (b - k) * R + k;
			ss[i] = s;
		}
	}
	__syncthreads();
	#pragma unroll
	for (int i = 0; i < NB; i++)
		if (dst[i] >= 0) {
			#pragma unroll
			for (int q = 0; q < R; q++) X[DENSE ? (dst[i] + q * P) * S + ss[i] : G::at(ss[i], dst[i] + q * P)] = u[i][q];
		}
	__syncthreads();
}

// Last pass of an analysis chain, radix R (P = N/R): thread item (s, b), b = 0
// .. P/2, runs the butterflies b and P - b of sequence s.  They hold both
// members of the pairs (z_k, z_{N-k}) for k = b + q P and k = P - b + q P (b =
// 0 and b = P/2 pair with themselves), and each pair with k < N/2 goes to
// st(s, k, z_k, z_{N-k}).  Every k < N/2 is handed over once; no shared-memory
// output.
template <int N, int S, int R, class Store>
__device__ __forceinline__ void last_pass_pairs(const double2* X, const double2* __restrict__ tw, int sign, Store& st, int tid)
{
	using G = Geo<N, S>;
	constexpr int P = N / R, H = P / 2, ITEMS = S * (H + 1), NB = (ITEMS + G::T - 1) / G::T;
	static_assert(P % 2 == 0, "the pairs of a last pass");
	#pragma unroll
	for (int i = 0; i < NB; i++) {
		const int g = tid + i * G::T;
		if (g < ITEMS) {
			const int s = g % S, b = g / S;
			double2 u[R];
			#pragma unroll
			for (int q = 0; q < R; q++) u[q] = X[G::at(s, b + q * P)];
			if (b) twiddle<R>(u, tw, b, sign);
			Dft<R>::run(u, sign);                       // z_{b + q P} = u[q]
			if (b == 0) {
				#pragma unroll
				for (int q = 0; 2 * q < R; q++) st(s, q * P, u[q], u[(R - q) % R]);
			} else if (b == H) {
				#pragma unroll
				for (int q = 0; 2 * q + 1 < R; q++) st(s, H + q * P, u[q], u[R - 1 - q]);
			} else {
				const int bp = P - b;
				double2 v[R];
				#pragma unroll
				for (int q = 0; q < R; q++) v[q] = X[G::at(s, bp + q * P)];
				twiddle<R>(v, tw, bp, sign);
				Dft<R>::run(v, sign);                   // z_{P - b + q P} = v[q]
				#pragma unroll
				for (int q = 0; 2 * q < R; q++) st(s, b + q * P, u[q], v[R - 1 - q]);
				#pragma unroll
				for (int q = 0; 2 * q + 1 < R; q++) st(s, bp + q * P, v[q], u[R - 1 - q]);
			}
		}
	}
}

// Pass chain: first pass from a loader, middle passes in shared memory, last
// pass to shared memory (MODE 0), to a storer (MODE 1), to shared memory in
// rows of S complex values (MODE 2), or as (z_k, z_{N-k}) pairs to a storer
// (MODE 3).
template <int N, int S, int P, int MODE, int R, int... Rest>
struct Chain {
	template <class Store>
	static __device__ __forceinline__ void run(double2* X, const double2* tw, int sign, Store& st, int tid)
	{
		if constexpr (sizeof...(Rest) == 0) {
			if constexpr (MODE == 3) {
				last_pass_pairs<N, S, R>(X, tw, sign, st, tid);
			} else if constexpr (MODE == 1) {
				// last pass: k = b (b < P = N/R), outputs b + q*P go to global memory
				using G = Geo<N, S>;
				constexpr int NBF = N / R, TOT = S * NBF, NB = (TOT + G::T - 1) / G::T, TSTEP = N / (P * R);
				#pragma unroll
				for (int i = 0; i < NB; i++) {
					const int g = tid + i * G::T;
					if (g < TOT) {
						const int s = g % S, b = g / S;
						double2 u[R];
						#pragma unroll
						for (int q = 0; q < R; q++) u[q] = X[G::at(s, b + q * NBF)];
						if (b) twiddle<R>(u, tw, b * TSTEP, sign);
						Dft<R>::run(u, sign);
						#pragma unroll
						for (int q = 0; q < R; q++) st(s, b + q * P, u[q]);
					}
				}
			} else {
				mid_pass<N, S, R, P, MODE == 2>(X, tw, sign, tid);
			}
		} else {
			mid_pass<N, S, R, P>(X, tw, sign, tid);
			Chain<N, S, P * R, MODE, Rest...>::run(X, tw, sign, st, tid);
		}
	}
};

struct NoHook { __device__ __forceinline__ void operator()() const {} };

// after_first() runs once the first pass has written X and the block has
// synchronised (the input is no longer read)
template <int N, int S, int MODE, class Load, class Store, class Hook, int R0, int... Rest>
__device__ __forceinline__ void fused_fft(double2* X, const double2* tw, int sign, Load& ld, Store& st, const Hook& after_first,
                                          int tid, RadixList<R0, Rest...>)
{
	// first pass: butterfly b reads elements b + q*N/R0 from global, no twiddles
	using G = Geo<N, S>;
	constexpr int NBF = N / R0, TOT = S * NBF, NB = (TOT + G::T - 1) / G::T;
	decltype(ld(0, 0)) in[NB][R0];
	#pragma unroll
	for (int i = 0; i < NB; i++) {
		const int g = tid + i * G::T;
		if (g < TOT) {
			const int s = g % S, b = g / S;
			#pragma unroll
			for (int q = 0; q < R0; q++) in[i][q] = ld(s, b + q * NBF);
		}
	}
	#pragma unroll
	for (int i = 0; i < NB; i++) {
		const int g = tid + i * G::T;
		if (g < TOT) {
			const int s = g % S, b = g / S;
			double2 u[R0];
			#pragma unroll
			for (int q = 0; q < R0; q++) u[q] = widen(in[i][q]);
			Dft<R0>::run(u, sign);
			#pragma unroll
			for (int q = 0; q < R0; q++) X[G::at(s, b * R0 + q)] = u[q];
		}
	}
	__syncthreads();
	after_first();
	Chain<N, S, R0, MODE, Rest...>::run(X, tw, sign, st, tid);
}

template <int N, int S, class G>
__global__ void __launch_bounds__(Geo<N, S>::T) fft3_synth_kernel(FftParams p)
{
	extern __shared__ double2 smem[];
	const int fc = blockIdx.y;
	const int lat0 = blockIdx.x * 2 * S;
	const double2* __restrict__ Ff = p.F + (long)fc * p.fstride;
	const int ml = p.mlim, nlat = p.nlat;
	auto ld = [&](int s, int j) -> double2 {
		const int ra = lat0 + 2 * s;
		const int k = (j <= ml) ? j : ((j >= N - ml) ? N - j : -1);
		if (k < 0 || ra >= nlat) return make_double2(0.0, 0.0);
		double2 a = __ldg(Ff + (long)k * nlat + ra), b = __ldg(Ff + (long)k * nlat + ra + 1);
		if (k == 0) { a.y = 0.0; b.y = 0.0; }
		return (j <= ml) ? make_double2(a.x - b.y, a.y + b.x) : make_double2(a.x + b.y, b.x - a.y);
	};
	const int c = fc / p.nf;
	G* out = grid_out<G>(p, c, fc);
	const bool phi = p.phi_contiguous, v2 = p.vec2;
	auto st = [&](int s, int j, double2 z) {
		const int row = lat0 + 2 * s;
		if (row >= nlat) return;
		if (!phi) {
			store_pair(out + (long)j * nlat + row, z, v2);
		} else {
			out[(long)row * N + j] = (G) z.x;
			out[(long)(row + 1) * N + j] = (G) z.y;
		}
	};
	fused_fft<N, S, true>(smem, p.tw, +1, ld, st, NoHook{}, threadIdx.x, typename NphiPlan<N>::L{});
}

template <int N, int S, class G>
__global__ void __launch_bounds__(Geo<N, S>::T) fft3_analys_kernel(FftParams p)
{
	extern __shared__ double2 smem[];
	const int fc = blockIdx.y;
	const int lat0 = blockIdx.x * 2 * S;
	const int nlat = p.nlat;
	const int c = fc / p.nf;
	const G* in = grid_in<G>(p, c, fc);
	const bool phi = p.phi_contiguous, v2 = p.vec2;
	auto ld = [&](int s, int j) {
		const int row = lat0 + 2 * s;
		typename Pair<G>::T v = {};
		if (row >= nlat) return v;
		if (!phi) return load_pair(in + (long)j * nlat + row, v2);
		v.x = __ldg(in + (long)row * N + j); v.y = __ldg(in + (long)(row + 1) * N + j);
		return v;
	};
	// Fourier rows straight from the last radix pass (pairs z_k, z_{N-k})
	double2* Ff = p.F + (long)fc * p.fstride;
	const double sc = 0.5 / N;
	const int ml = p.mlim;
	auto st = [&](int s, int k, double2 z, double2 w) {
		const int ra = lat0 + 2 * s;
		if (k > ml || ra >= nlat) return;
		const double2 fa = make_double2(sc * (z.x + w.x), sc * (z.y - w.y));
		const double2 fb = make_double2(sc * (z.y + w.y), -sc * (z.x - w.x));
		double2* o = Ff + (long)k * nlat + ra;
		if (((uintptr_t) o & 31) == 0)      // one 32-byte store for the latitude pair
			asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};"
			             :: "l"(o), "d"(fa.x), "d"(fa.y), "d"(fb.x), "d"(fb.y) : "memory");
		else { o[0] = fa; o[1] = fb; }
	};
	fused_fft<N, S, 3>(smem, p.tw, -1, ld, st, NoHook{}, threadIdx.x, typename NphiPlan<N>::L{});
}

// ---------------------------------------------------------------------------
// Four-step FFT for nphi = N1 N2 = 96 x 128 = 12288 and 64 x 96 = 6144
// (theta-contiguous grids).
// With j = j1 + N1 j2 and k = k2 + N2 k1,
//   exp(s 2 pi i j k / N) = w_N^(j1 k2) w_N1^(j1 k1) w_N2^(j2 k2),
// so a length-N transform is N2 transforms of length N1 (over k1), a twiddle
// w_N^(j1 k2), and N1 transforms of length N2 (over k2).  Each CTA runs the
// short transforms of FS_S latitude pairs (one 256-byte run of a grid row per
// element), so its loads and stores are coalesced rows and many CTAs share an
// SM, where the one-pass kernel of this length holds one latitude pair per SM.
// The intermediate lives in grid row j = N1 k2 + j1: the synthesis works in
// place in its output grid (the second step reads and rewrites exactly the
// rows j1 + N1 k2 of its j1), the analysis writes it to a scratch grid.
// The analysis' second step takes k2 and N2 - k2 in one CTA, so that each
// order's pair (z_m, z_{N-m}) is at hand to separate the two real spectra.
constexpr int FS_S = 16;      // latitude pairs per CTA

template <int N1, int N2>
__global__ void __launch_bounds__(Geo<N1, FS_S>::T) fft_fs_synth1_kernel(FftParams p)
{
	extern __shared__ double2 smem[];
	constexpr int N = N1 * N2;
	const int fc = blockIdx.z, k2 = blockIdx.y;
	const int lat0 = blockIdx.x * 2 * FS_S;
	const double2* __restrict__ Ff = p.F + (long)fc * p.fstride;
	const int ml = p.mlim, nlat = p.nlat;
	auto ld = [&](int s, int k1) -> double2 {
		const int ra = lat0 + 2 * s;
		const int j = k2 + N2 * k1;                 // frequency index
		const int k = (j <= ml) ? j : ((j >= N - ml) ? N - j : -1);
		if (k < 0 || ra >= nlat) return make_double2(0.0, 0.0);
		double2 a = __ldg(Ff + (long)k * nlat + ra), b = __ldg(Ff + (long)k * nlat + ra + 1);
		if (k == 0) { a.y = 0.0; b.y = 0.0; }
		return (j <= ml) ? make_double2(a.x - b.y, a.y + b.x) : make_double2(a.x + b.y, b.x - a.y);
	};
	const int c = fc / p.nf;
	double* out = (c == 0 ? p.spat[0] : c == 1 ? p.spat[1] : p.spat[2]) + (long)(fc - c * p.nf) * p.spat_dist;
	auto st = [&](int s, int j1, double2 z) {
		const int row = lat0 + 2 * s;
		if (row >= nlat) return;
		z = cmul(z, __ldg(p.tw + (j1 * k2) % N));
		*reinterpret_cast<double2*>(out + (long)(N1 * k2 + j1) * nlat + row) = z;
	};
	fused_fft<N1, FS_S, 1>(smem, p.tw1, +1, ld, st, NoHook{}, threadIdx.x, typename NphiPlan<N1>::L{});
}

template <int N1, int N2>
__global__ void __launch_bounds__(Geo<N2, FS_S>::T) fft_fs_synth2_kernel(FftParams p)
{
	extern __shared__ double2 smem[];
	const int fc = blockIdx.z, j1 = blockIdx.y;
	const int lat0 = blockIdx.x * 2 * FS_S;
	const int nlat = p.nlat;
	const int c = fc / p.nf;
	double* out = (c == 0 ? p.spat[0] : c == 1 ? p.spat[1] : p.spat[2]) + (long)(fc - c * p.nf) * p.spat_dist;
	auto ld = [&](int s, int k2) -> double2 {
		const int row = lat0 + 2 * s;
		if (row >= nlat) return make_double2(0.0, 0.0);
		return *reinterpret_cast<const double2*>(out + (long)(N1 * k2 + j1) * nlat + row);
	};
	auto st = [&](int s, int j2, double2 z) {
		const int row = lat0 + 2 * s;
		if (row >= nlat) return;
		*reinterpret_cast<double2*>(out + (long)(j1 + N1 * j2) * nlat + row) = z;
	};
	fused_fft<N2, FS_S, 1>(smem, p.tw2, +1, ld, st, NoHook{}, threadIdx.x, typename NphiPlan<N2>::L{});
}

template <int N1, int N2>
__global__ void __launch_bounds__(Geo<N2, FS_S>::T) fft_fs_analys1_kernel(FftParams p)
{
	extern __shared__ double2 smem[];
	constexpr int N = N1 * N2;
	const int fc = blockIdx.z, j1 = blockIdx.y;
	const int lat0 = blockIdx.x * 2 * FS_S;
	const int nlat = p.nlat;
	const int c = fc / p.nf;
	const double* in = (c == 0 ? p.spat_in[0] : c == 1 ? p.spat_in[1] : p.spat_in[2]) + (long)(fc - c * p.nf) * p.spat_dist;
	double* scr = p.scratch + (long)fc * N * nlat;
	auto ld = [&](int s, int j2) -> double2 {
		const int row = lat0 + 2 * s;
		if (row >= nlat) return make_double2(0.0, 0.0);
		return __ldg(reinterpret_cast<const double2*>(in + (long)(j1 + N1 * j2) * nlat + row));
	};
	auto st = [&](int s, int k2, double2 z) {
		const int row = lat0 + 2 * s;
		if (row >= nlat) return;
		double2 w = __ldg(p.tw + (j1 * k2) % N);
		w.y = -w.y;
		*reinterpret_cast<double2*>(scr + (long)(N1 * k2 + j1) * nlat + row) = cmul(z, w);
	};
	fused_fft<N2, FS_S, 1>(smem, p.tw2, -1, ld, st, NoHook{}, threadIdx.x, typename NphiPlan<N2>::L{});
}

template <int N1, int N2>
__global__ void __launch_bounds__(Geo<N1, 2 * FS_S>::T) fft_fs_analys2_kernel(FftParams p)
{
	extern __shared__ double2 smem[];
	using G = Geo<N1, 2 * FS_S>;
	constexpr int N = N1 * N2;
	const int fc = blockIdx.z, ka = blockIdx.y;          // ka = 0 .. N2/2
	const int kb = (N2 - ka) % N2;                        // partner k2 (ka for 0 and N2/2)
	const int lat0 = blockIdx.x * 2 * FS_S;
	const int nlat = p.nlat, ml = p.mlim;
	const double* scr = p.scratch + (long)fc * N * nlat;
	// sequences s < FS_S: k2 = ka, latitude pair s; s >= FS_S: k2 = kb, pair s - FS_S
	auto ld = [&](int s, int j1) -> double2 {
		const int pr = s % FS_S, k2 = (s < FS_S) ? ka : kb;
		const int row = lat0 + 2 * pr;
		if (row >= nlat) return make_double2(0.0, 0.0);
		return *reinterpret_cast<const double2*>(scr + (long)(N1 * k2 + j1) * nlat + row);
	};
	NoHook no;
	fused_fft<N1, 2 * FS_S, 0>(smem, p.tw1, -1, ld, no, NoHook{}, threadIdx.x, typename NphiPlan<N1>::L{});
	// X[at(s, k1)] = z_k, k = k2(s) + N2 k1.  Partner z_{N-k}: for k2 = 0 at
	// (same sequence, (N1 - k1) % N1), else at (other k2, N1 - 1 - k1).
	double2* Ff = p.F + (long)fc * p.fstride;
	const double sc = 0.5 / N;
	const bool self = (ka == kb);
	const int nseq = self ? FS_S : 2 * FS_S;
	for (int e = threadIdx.x; e < nseq * N1; e += G::T) {
		const int s = e / N1, k1 = e - s * N1;
		const int pr = s % FS_S, k2 = (s < FS_S) ? ka : kb;
		const int k = k2 + N2 * k1;
		const int ra = lat0 + 2 * pr;
		if (k > ml || ra >= nlat) continue;
		int sp, kp;
		if (k2 == 0) { sp = s; kp = (N1 - k1) % N1; }
		else { sp = self ? s : (s < FS_S ? s + FS_S : s - FS_S); kp = N1 - 1 - k1; }
		const double2 z = smem[G::at(s, k1)], w = smem[G::at(sp, kp)];
		const double2 fa = make_double2(sc * (z.x + w.x), sc * (z.y - w.y));
		const double2 fb = make_double2(sc * (z.y + w.y), -sc * (z.x - w.x));
		double2* o = Ff + (long)k * nlat + ra;
		asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};"
		             :: "l"(o), "d"(fa.x), "d"(fa.y), "d"(fb.x), "d"(fb.y) : "memory");
	}
}

// ---------------------------------------------------------------------------
// Prefetched fused kernels.  A persistent CTA walks over tiles (2 S latitudes
// of one field-component, tile t = fc * nlg + latitude group) and keeps the
// input of its next tile in flight while the current one is transformed: one
// thread issues tensor copies (TMA, no multicast) of the next tile into a
// shared staging buffer right after the first pass has moved the current
// tile from there into the FFT buffer, and the copies complete on an
// mbarrier that the CTA waits on (bounded) before the next first pass.
//   synthesis input   F[fc][k][theta]: box (2 S latitudes x 2 doubles, <= 256 k)
//   analysis input    theta-contiguous v[f][j][theta]: box (2 S latitudes, 256 or 192 j)
// Outputs are written as by the direct kernels above.
// j rows per box of the analysis input: 256, or nphi for 192, 192 for 384
__host__ __device__ constexpr int box_j(int N) { return (N % 256 == 0) ? 256 : (N <= 256 ? N : 192); }

struct TmaTiles {
	int nlg;          // latitude groups (tiles per field-component)
	int ntiles;
	int ncopy;        // box copies per tile
	int box;          // rows (k or j) per box
	unsigned bytes;   // bytes per tile (all boxes, out-of-range parts included)
	int stage_off;    // staging buffer offset in the dynamic shared memory (bytes)
	int v4;           // F rows 32-byte aligned at even latitudes: one 32-byte store per latitude pair
};

__device__ int g_fft_wait_err;                    // set when a bounded wait gave up

// One thread: announce the bytes of a tile, then issue its box copies
// (latitude coordinate c0, rows c * box, field c2).
__device__ __forceinline__ void fetch_tile(uint64_t* bar, const CUtensorMap* map, char* stage, const TmaTiles& tt,
                                           int c0, int c2, int box_bytes)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(su32(bar)), "r"(tt.bytes) : "memory");
	for (int c = 0; c < tt.ncopy; c++)
		tma_tile3(stage + (size_t) c * box_bytes, map, c0, c * tt.box, c2, bar);
}

// Wait for the staged tile; false (uniformly in the CTA) if the wait gave up,
// after recording it and waiting once more (bounded) for the copies in flight.
__device__ __forceinline__ bool stage_ready(uint64_t* bar, uint32_t parity)
{
	const bool ok = fbar_wait(bar, parity);
	if (__syncthreads_or(!ok)) {
		if (threadIdx.x == 0) {
			atomicExch(&g_fft_wait_err, 1);
			fbar_wait(bar, parity);
		}
		return false;
	}
	return true;
}

__device__ __forceinline__ void stage_init(uint64_t* bar)
{
	if (threadIdx.x == 0) {
		asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(su32(bar)) : "memory");
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	__syncthreads();
}

__device__ __forceinline__ void tma_store3(const CUtensorMap* map, const void* src, int c0, int c1, int c2)
{
	asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];"
	             :: "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(su32(src)) : "memory");
}

// tensor stores of this thread have finished reading shared memory
__device__ __forceinline__ void store_reads_done() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// Results written to X by every thread become visible to the tensor copies,
// then one thread stores nbox boxes of box_bytes each.
__device__ __forceinline__ void store_tile(const CUtensorMap* map, const char* X, int nbox, int box, int box_bytes, int c0,
                                           int c2)
{
	asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
	__syncthreads();
	if (threadIdx.x == 0) {
		for (int c = 0; c < nbox; c++) tma_store3(map, X + (size_t) c * box_bytes, c0, c * box, c2);
		asm volatile("cp.async.bulk.commit_group;" ::: "memory");
	}
}

// TOUT: theta-contiguous output written by tensor stores of whole tiles
// (rows of 2 S latitudes) from X, instead of 16-byte stores per latitude pair
template <int N, int S, bool TOUT, class G>
__global__ void __launch_bounds__(Geo<N, S>::T, fft4_minb(S * N)) fft4_synth_kernel(
	const __grid_constant__ CUtensorMap fmap, const __grid_constant__ CUtensorMap o0, const __grid_constant__ CUtensorMap o1,
	const __grid_constant__ CUtensorMap o2, FftParams p, TmaTiles tt)
{
	extern __shared__ __align__(128) char fsm[];
	__shared__ __align__(8) uint64_t bar;
	char* base = fsm + ((128u - (su32(fsm) & 127u)) & 127u);   // tensor copies land on 128-byte boundaries
	double2* X = reinterpret_cast<double2*>(base);
	char* stage = base + tt.stage_off;
	const double2* stg = reinterpret_cast<const double2*>(stage);
	const int ml = p.mlim, nlat = p.nlat;
	const int box_bytes = tt.box * 2 * S * 16;
	stage_init(&bar);
	int tile = blockIdx.x;
	if (threadIdx.x == 0) {
		const int fc = tile / tt.nlg;
		fetch_tile(&bar, &fmap, stage, tt, 4 * S * (tile - fc * tt.nlg), fc, box_bytes);
	}
	for (uint32_t parity = 0; tile < tt.ntiles; tile += gridDim.x, parity ^= 1) {
		if (TOUT && threadIdx.x == 0) store_reads_done();     // X is free again (previous tile's stores)
		if (!stage_ready(&bar, parity)) return;
		const int fc = tile / tt.nlg;
		const int lat0 = (tile - fc * tt.nlg) * 2 * S;
		// ml opaque per tile: the first pass's shared addresses and predicates
		// are recomputed per tile instead of held in registers across tiles
		int mlo = ml;
		asm volatile("" : "+r"(mlo));
		auto ld = [&](int s, int j) -> double2 {
			const int k = (j <= mlo) ? j : ((j >= N - mlo) ? N - j : -1);
			if (k < 0) return make_double2(0.0, 0.0);
			// the two latitudes of sequence s, read in an order that alternates
			// with the row so that the 8 lanes of a shared-memory phase (4 rows)
			// hit distinct banks; swapped back in registers
			const int f = (k >> (S == 1 ? 2 : (S == 2 ? 1 : 0))) & 1;
			const double2 u0 = stg[k * 2 * S + 2 * s + f], u1 = stg[k * 2 * S + 2 * s + 1 - f];
			double2 a = f ? u1 : u0, b = f ? u0 : u1;
			if (k == 0) { a.y = 0.0; b.y = 0.0; }
			return (j <= mlo) ? make_double2(a.x - b.y, a.y + b.x) : make_double2(a.x + b.y, b.x - a.y);
		};
		const int c = fc / p.nf;
		const int next = tile + gridDim.x;
		auto prefetch = [&]() {
			if (threadIdx.x == 0 && next < tt.ntiles) {
				asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
				const int nfc = next / tt.nlg;
				fetch_tile(&bar, &fmap, stage, tt, 4 * S * (next - nfc * tt.nlg), nfc, box_bytes);
			}
		};
		if constexpr (TOUT) {
			int dummy = 0;
			auto st = [&](int, int, double2) { dummy++; };
			fused_fft<N, S, 2>(X, p.tw, +1, ld, st, prefetch, threadIdx.x, typename NphiPlan<N>::L{});
			constexpr int BJ = box_j(N);
			const CUtensorMap* om = (c == 0) ? &o0 : (c == 1 ? &o1 : &o2);
			store_tile(om, base, N / BJ, BJ, BJ * S * 16, lat0, fc - c * p.nf);
		} else {
			G* out = grid_out<G>(p, c, fc);
			const bool phi = p.phi_contiguous, v2 = p.vec2;
			auto st = [&](int s, int j, double2 z) {
				const int row = lat0 + 2 * s;
				if (row >= nlat) return;
				if (!phi) {
					store_pair(out + (long)j * nlat + row, z, v2);
				} else {
					out[(long)row * N + j] = (G) z.x;
					out[(long)(row + 1) * N + j] = (G) z.y;
				}
			};
			fused_fft<N, S, 1>(X, p.tw, +1, ld, st, prefetch, threadIdx.x, typename NphiPlan<N>::L{});
		}
	}
	if (TOUT && threadIdx.x == 0) store_reads_done();
}

template <int N, int S, class G>
__global__ void __launch_bounds__(Geo<N, S>::T, fft4_minb(S * N)) fft4_analys_kernel(
	const __grid_constant__ CUtensorMap m0, const __grid_constant__ CUtensorMap m1, const __grid_constant__ CUtensorMap m2,
	FftParams p, TmaTiles tt)
{
	extern __shared__ __align__(128) char fsm[];
	__shared__ __align__(8) uint64_t bar;
	char* base = fsm + ((128u - (su32(fsm) & 127u)) & 127u);   // tensor copies land on 128-byte boundaries
	double2* X = reinterpret_cast<double2*>(base);
	char* stage = base + tt.stage_off;
	const G* stg = reinterpret_cast<const G*>(stage);
	const int nlat = p.nlat, nf = p.nf;
	const int box_bytes = box_j(N) * 2 * S * sizeof(G);
	auto issue = [&](int t) {
		const int fc = t / tt.nlg, c = fc / nf;
		const CUtensorMap* m = (c == 0) ? &m0 : (c == 1 ? &m1 : &m2);
		fetch_tile(&bar, m, stage, tt, 2 * S * (t - fc * tt.nlg), fc - c * nf, box_bytes);
	};
	stage_init(&bar);
	int tile = blockIdx.x;
	if (threadIdx.x == 0) issue(tile);
	for (uint32_t parity = 0; tile < tt.ntiles; tile += gridDim.x, parity ^= 1) {
		if (!stage_ready(&bar, parity)) return;
		const int fc = tile / tt.nlg;
		const int lat0 = (tile - fc * tt.nlg) * 2 * S;
		int rs = 2 * S;                         // opaque per tile, as mlim in the synthesis
		asm volatile("" : "+r"(rs));
		auto ld = [&](int s, int j) { return *reinterpret_cast<const typename Pair<G>::T*>(stg + j * rs + 2 * s); };
		const int next = tile + gridDim.x;
		auto prefetch = [&]() {
			if (threadIdx.x == 0 && next < tt.ntiles) {
				asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
				issue(next);
			}
		};
		// Fourier rows straight from the last radix pass: F_k of the two
		// latitudes of sequence s from (z_k, z_{N-k}), one 32-byte store
		double2* Ff = p.F + (long)fc * p.fstride;
		const double sc = 0.5 / N;
		const int ml = p.mlim;
		auto st = [&](int s, int k, double2 z, double2 w) {
			const int ra = lat0 + 2 * s;
			if (k > ml || ra >= nlat) return;
			const double2 fa = make_double2(sc * (z.x + w.x), sc * (z.y - w.y));
			const double2 fb = make_double2(sc * (z.y + w.y), -sc * (z.x - w.x));
			double2* o = Ff + (long)k * nlat + ra;
			if (tt.v4)
				asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};"
				             :: "l"(o), "d"(fa.x), "d"(fa.y), "d"(fb.x), "d"(fb.y) : "memory");
			else { o[0] = fa; o[1] = fb; }
		};
		fused_fft<N, S, 3>(X, p.tw, -1, ld, st, prefetch, threadIdx.x, typename NphiPlan<N>::L{});
	}
}

int sm_count()
{
	static const int n = [] {
		int dev = 0, c = 0;
		cudaGetDevice(&dev);
		if (cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || c <= 0) { cudaGetLastError(); c = 148; }
		return c;
	}();
	return n;
}

// F[fc][k][theta] as FP64 rows of 2 nlat doubles: box (2 S latitudes, box k)
bool f_map(CUtensorMap* m, const FftParams& p, int nfc, int S, int box)
{
	return encode3(m, p.F, 2 * (uint64_t) p.nlat, p.mlim + 1, nfc, 16 * (uint64_t) p.nlat, 16 * (uint64_t) p.fstride, 4 * S, box);
}

// theta-contiguous spatial component c: dims (nlat, nphi, fields)
bool grid_map(CUtensorMap* m, const double* base, const FftParams& p, int N, int S)
{
	const uint64_t e = p.f32 ? 4 : 8;
	return encode3(m, base, p.nlat, N, p.nf, e * p.nlat, e * p.spat_dist, 2 * S, box_j(N), p.f32);
}

template <int N, int S>
bool launch_fft4(const FftParams& p, int nfc, cudaStream_t st, bool synth)
{
	using G = Geo<N, S>;
	alignas(64) CUtensorMap maps[4];        // synthesis: F, output components; analysis: input components
	TmaTiles tt;
	tt.nlg = (p.nlat + 2 * S - 1) / (2 * S);
	tt.ntiles = tt.nlg * nfc;
	const int rows = p.mlim + 1;
	const int kbox = rows < 256 ? rows : 256;            // k rows per box of F
	const int ncomp = (nfc + p.nf - 1) / p.nf;
	// tensor maps over the theta-contiguous grid (16-byte aligned, even nlat)
	const bool grid_ok = p.vec2 && !p.phi_contiguous && !(p.nlat & 1) && N % box_j(N) == 0;
	const bool tstore = (p.generic != 3);               // option 3 = 3: prefetched loads, direct stores
	bool tout = false;
	size_t stage_bytes;
	if (synth) {
		tt.box = kbox;
		tt.ncopy = (rows + tt.box - 1) / tt.box;
		stage_bytes = (size_t) tt.ncopy * tt.box * 2 * S * 16;
		if (!f_map(&maps[0], p, nfc, S, tt.box)) return false;
		tout = grid_ok && tstore && !p.f32;
		for (int c = 0; c < 3 && tout; c++) tout = grid_map(&maps[1 + c], p.spat[c < ncomp ? c : 0], p, N, S);
	} else {
		// theta-contiguous grids only (phi-contiguous rows are read faster
		// straight from global memory by the direct kernel)
		if (!grid_ok || (S == 1 && p.f32)) return false;      // a pair of floats is half of a tensor copy's 16 bytes
		tt.box = box_j(N);
		tt.ncopy = N / tt.box;
		stage_bytes = (size_t) N * 2 * S * (p.f32 ? 4 : 8);
		for (int c = 0; c < 3; c++)
			if (!grid_map(&maps[c], p.spat_in[c < ncomp ? c : 0], p, N, S)) return false;
	}
	tt.bytes = (unsigned) (stage_bytes + p.extra_tx);
	tt.v4 = !((uintptr_t) p.F & 31) && !(p.nlat & 1) && !(p.fstride & 1);
	tt.stage_off = (int)(((size_t) S * G::SEQ * sizeof(double2) + 127) / 128 * 128);
	const size_t smem = tt.stage_off + stage_bytes + 128;
	if (smem > 226 * 1024) return false;
	auto go = [&](auto kern) {
		// the occupancy of the thread's last kernel and size is kept: the query costs about as much as a launch
		static thread_local const void* last_fn = nullptr;
		static thread_local size_t last_smem = 0;
		static thread_local int per_sm = 0;
		if (last_fn != (const void*) kern || last_smem != smem) {
			last_fn = nullptr;
			if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, G::T, smem) != cudaSuccess || per_sm <= 0) {
				cudaGetLastError();
				return false;
			}
			last_fn = (const void*) kern; last_smem = smem;
		}
		const int grid = std::min(tt.ntiles, per_sm * sm_count());
		if constexpr (std::is_same_v<decltype(kern), decltype(&fft4_analys_kernel<N, S, double>)>)
			kern<<<grid, G::T, smem, st>>>(maps[0], maps[1], maps[2], p, tt);
		else
			kern<<<grid, G::T, smem, st>>>(maps[0], maps[tout ? 1 : 0], maps[tout ? 2 : 0], maps[tout ? 3 : 0], p, tt);
		return true;
	};
	if (synth) return p.f32 ? go(fft4_synth_kernel<N, S, false, float>)
	                        : (tout ? go(fft4_synth_kernel<N, S, true, double>) : go(fft4_synth_kernel<N, S, false, double>));
	if constexpr (S > 1) if (p.f32) return go(fft4_analys_kernel<N, S, float>);
	return go(fft4_analys_kernel<N, S, double>);
}

template <int N, int S>
bool launch_fft3(const FftParams& p, int nfc, cudaStream_t st, bool synth)
{
	using G = Geo<N, S>;
	const size_t smem = sizeof(double2) * (size_t) S * G::SEQ;
	dim3 grid((p.nlat + 2 * S - 1) / (2 * S), nfc);
	auto go = [&](auto kern) { kern<<<grid, G::T, smem, st>>>(p); };
	if (p.f32) go(synth ? fft3_synth_kernel<N, S, float> : fft3_analys_kernel<N, S, float>);
	else go(synth ? fft3_synth_kernel<N, S, double> : fft3_analys_kernel<N, S, double>);
	return true;
}

template <int N>
bool launch_fft3_n(const FftParams& p, int nfc, cudaStream_t st, bool synth)
{
	// latitude pairs per CTA: 8 (full 128-byte lines of a theta-contiguous
	// grid, two butterflies per thread) where the buffer fits, else up to 4
	// while the block stays at <= 768 threads
	if constexpr (8 * (N + (N >> 3) + 1) * 16 <= 227 * 1024) if (p.S >= 8) return launch_fft3<N, 8>(p, nfc, st, synth);
	if constexpr (4 * N / 8 <= 768) if (p.S >= 4) return launch_fft3<N, 4>(p, nfc, st, synth);
	if constexpr (2 * N / 8 <= 768) if (p.S >= 2) return launch_fft3<N, 2>(p, nfc, st, synth);
	return launch_fft3<N, 1>(p, nfc, st, synth);
}

} // namespace

// kernel family of the last FFT launch in the process (a diagnostic, any
// thread), and whether the launch in progress on this thread took the
// prefetching kernels
static std::atomic<int> g_last_fft_path{-1};
static thread_local bool g_fft4_ran = false;

namespace {

// prefetched kernels for the automatic choice (p.generic == 0); false where
// they do not apply (layout, alignment, shared memory), for the direct ones
template <int N>
bool launch_fft4_n(const FftParams& p, int nfc, cudaStream_t st, bool synth)
{
	if constexpr (N + (N >> 3) + 8 > 6400) return false;     // FFT buffer above 100 KB
	else {
		if (p.S == 1) return launch_fft4<N, 1>(p, nfc, st, synth);
		if constexpr (2 * N / 8 <= 768) if (p.S == 2) return launch_fft4<N, 2>(p, nfc, st, synth);
		if constexpr (4 * N / 8 <= 768) if (p.S == 4) return launch_fft4<N, 4>(p, nfc, st, synth);
		return false;
	}
}

// Four-step kernels, for a call that fft_fourstep_used admits.
template <int N1, int N2, bool ANALYS = true>
void launch_fourstep(const FftParams& p, int nfc, cudaStream_t st, bool synth)
{
	using G1 = Geo<N1, FS_S>;
	using G2 = Geo<N2, FS_S>;
	using G3 = Geo<N1, 2 * FS_S>;
	const size_t s1 = sizeof(double2) * (size_t) FS_S * G1::SEQ, s2 = sizeof(double2) * (size_t) FS_S * G2::SEQ;
	const size_t s3 = sizeof(double2) * (size_t)(2 * FS_S) * G3::SEQ;
	const int nlb = (p.nlat + 2 * FS_S - 1) / (2 * FS_S);
	if (synth) {
		fft_fs_synth1_kernel<N1, N2><<<dim3(nlb, N2, nfc), G1::T, s1, st>>>(p);
		fft_fs_synth2_kernel<N1, N2><<<dim3(nlb, N1, nfc), G2::T, s2, st>>>(p);
	} else if constexpr (ANALYS) {
		fft_fs_analys1_kernel<N1, N2><<<dim3(nlb, N1, nfc), G2::T, s2, st>>>(p);
		fft_fs_analys2_kernel<N1, N2><<<dim3(nlb, N2 / 2 + 1, nfc), G3::T, s3, st>>>(p);
	}
	shtb_count_launch();         // the second of the two launches is counted by the caller
}

template <int N1, int N2>
void set_fourstep_limits()
{
	cudaFuncSetAttribute(fft_fs_analys2_kernel<N1, N2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                     (int)(sizeof(double2) * 2 * FS_S * Geo<N1, 2 * FS_S>::SEQ));
}

// Latitude pairs per CTA of the one-pass kernels where option 1 leaves the
// choice: what fits the shared memory twice (fft_params), and half of that where
// the chains of 16 values per thread leave few warps to a CTA and rows of
// fewer latitudes cost little: phi-contiguous grids, and the FP64 synthesis of
// nphi 768.  Kernel times, synthesis / analysis, chains before those / with the
// larger tile / with this one: 51 phi-contiguous grids of 766 x 1536 221/195,
// 199/203 and 185/169 us; 8 of 384 x 768 13.1/11.1, 14.1/10.1 and 12.2/9.5; 814 of
// 192 x 384 208/185, 174/159 and 149/145; theta-contiguous synthesis, 8 of 384 x
// 768 13.4, 14.2 and 13.4, 204 of them 218, 199 and 185.
int fused_pairs(const FftParams& p, bool synth)
{
	if (p.pairs) return p.S;
	int S = p.S;
	if (p.phi_contiguous) {
		if (p.N == 384 || p.N == 768) S = 2;
		else if (p.N == 1536) S = 1;
	} else if (synth && p.N == 768 && !p.f32) S = 2;
	return std::min(S, p.S);
}

bool launch_fused(const FftParams& p0, int nfc, cudaStream_t st, bool synth)
{
	FftParams p = p0;
	p.S = fused_pairs(p0, synth);
	if (fft_fourstep_used(p, nfc, synth) && (synth || p.scratch)) {
		switch (p.N) {
			case 12288: launch_fourstep<96, 128>(p, nfc, st, synth); break;
			case 6144: launch_fourstep<64, 96>(p, nfc, st, synth); break;
			default: launch_fourstep<48, 64, false>(p, nfc, st, synth); break;      // 3072: synthesis only
		}
		return true;
	}
	if (p.generic == 0 || p.generic == 3) {
		bool done = false;
		switch (p.N) {
			case 192: done = launch_fft4_n<192>(p, nfc, st, synth); break;
			case 384: done = launch_fft4_n<384>(p, nfc, st, synth); break;
			case 768: done = launch_fft4_n<768>(p, nfc, st, synth); break;
			case 1536: done = launch_fft4_n<1536>(p, nfc, st, synth); break;
			case 3072: done = launch_fft4_n<3072>(p, nfc, st, synth); break;
			case 6144: done = launch_fft4_n<6144>(p, nfc, st, synth); break;
			default: break;
		}
		if (done) { g_fft4_ran = true; return true; }
	}
	switch (p.N) {
		case 192: return launch_fft3_n<192>(p, nfc, st, synth);
		case 384: return launch_fft3_n<384>(p, nfc, st, synth);
		case 768: return launch_fft3_n<768>(p, nfc, st, synth);
		case 1536: return launch_fft3_n<1536>(p, nfc, st, synth);
		case 3072: return launch_fft3_n<3072>(p, nfc, st, synth);
		case 6144: return launch_fft3_n<6144>(p, nfc, st, synth);
		case 12288: return launch_fft3_n<12288>(p, nfc, st, synth);
		default: return false;
	}
}

template <int N, int S>
void set_fft4_limits(int lim)
{
	auto set = [&](auto kern) { cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, lim); };
	set(fft4_synth_kernel<N, S, true, double>);
	set(fft4_synth_kernel<N, S, false, double>);
	set(fft4_synth_kernel<N, S, false, float>);
	set(fft4_analys_kernel<N, S, double>);
	if constexpr (S > 1) set(fft4_analys_kernel<N, S, float>);
}

template <int N, int S>
void set_fft3_limits(int lim)
{
	auto set = [&](auto kern) { cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, lim); };
	set(fft3_synth_kernel<N, S, double>);
	set(fft3_synth_kernel<N, S, float>);
	set(fft3_analys_kernel<N, S, double>);
	set(fft3_analys_kernel<N, S, float>);
}

template <int N>
void set_fused_limits()
{
	const int lim = 227 * 1024;
	if constexpr (N + (N >> 3) + 8 <= 6400) {
		// the prefetching kernels also hold an mbarrier in static shared memory
		const int lim4 = 226 * 1024;
		set_fft4_limits<N, 1>(lim4);
		if constexpr (2 * N / 8 <= 768) set_fft4_limits<N, 2>(lim4);
		if constexpr (4 * N / 8 <= 768) set_fft4_limits<N, 4>(lim4);
	}
	set_fft3_limits<N, 1>(lim);
	if constexpr (2 * N / 8 <= 768) {
		set_fft3_limits<N, 2>(lim);
	}
	if constexpr (4 * N / 8 <= 768) {
		set_fft3_limits<N, 4>(lim);
	}
	if constexpr (8 * (N + (N >> 3) + 1) * 16 <= 227 * 1024) {
		set_fft3_limits<N, 8>(lim);
	}
}

} // namespace

static int seq_len_host(int N, int S)
{
	const int a = N + (N >> 3);
	return a + (((S >= 8 ? 1 : 8 / S) - a) & 7);
}

size_t fft_smem_bytes(int N, int S) { return 2 * sizeof(double2) * (size_t) S * seq_len_host(N, S); }

// sizes with a fused pass chain (these may exceed the generic kernels' limit)
bool fft_fused_available(int N)
{
	switch (N) {
		case 192: case 384: case 768: case 1536: case 3072: case 6144: case 12288: return true;
		default: return false;
	}
}

// kernel family of the last FFT launch (host side): 0 generic, 1 fused
// direct loads, 2 fused with prefetched tiles
int fft_last_path() { return g_last_fft_path.load(); }

void launch_fft_synth(const FftParams& p, int nfc, cudaStream_t st)
{
	g_fft4_ran = false;
	if (p.generic != 1 && launch_fused(p, nfc, st, true)) { g_last_fft_path = g_fft4_ran ? 2 : 1; shtb_count_launch(); return; }
	g_last_fft_path = 0;
	launch_fft_gen(p, nfc, st, true);
	shtb_count_launch();
}

void launch_fft_analys(const FftParams& p, int nfc, cudaStream_t st)
{
	g_fft4_ran = false;
	if (p.generic != 1 && launch_fused(p, nfc, st, false)) { g_last_fft_path = g_fft4_ran ? 2 : 1; shtb_count_launch(); return; }
	g_last_fft_path = 0;
	launch_fft_gen(p, nfc, st, false);
	shtb_count_launch();
}

// Whether a call takes the four-step kernels (the analysis then needs a grid
// per field-component in p.scratch): FP64, theta-contiguous grids with 16-byte
// aligned latitude pairs; nphi 6144 and 12288, and the synthesis of nphi 3072
// where the grids do not stay in the L2 cache, in which the half sectors that
// the one-pass kernel stores would be completed.  Against the one-pass kernels,
// synthesis / analysis: nphi 6144, 8 grids of 3072 latitudes 1552/1155 ->
// 866/803 us; the synthesis of nphi 3072, 32 grids of 1536 latitudes 1417 -> 783,
// 3 grids 100 -> 83 us.  The launcher, the allocation of the scratch and the
// single-precision entry points all ask here.
bool fft_fourstep_used(const FftParams& p, int nfc, bool synth)
{
	if (p.phi_contiguous || !p.vec2 || !p.tw1 || p.generic != 0 || p.f32 || p.nlat % 2 || ((uintptr_t) p.F & 31)) return false;
	if (p.N == 3072) return synth && (size_t) nfc * p.N * p.nlat * 8 > ((size_t) 96 << 20);
	return p.N == 6144 || p.N == 12288;
}

// nphi = n1 n2 of the four-step kernels
bool fft_fourstep_factors(int N, int& n1, int& n2)
{
	if (N == 12288) { n1 = 96; n2 = 128; return true; }
	if (N == 6144) { n1 = 64; n2 = 96; return true; }
	if (N == 3072) { n1 = 48; n2 = 64; return true; }
	return false;
}

void fft_set_smem_limits()
{
	set_fourstep_limits<96, 128>();
	set_fourstep_limits<64, 96>();
	tensor_map_encoder();    // resolved here, outside any stream capture
	sm_count();
	set_fused_limits<192>(); set_fused_limits<384>(); set_fused_limits<768>();
	set_fused_limits<1536>(); set_fused_limits<3072>(); set_fused_limits<6144>(); set_fused_limits<12288>();
	fft_gen_set_smem_limits();
}

// Returns (and clears) the flag that a bounded wait of the prefetched FFT
// kernels gave up; waits for the device.
int fft_take_wait_error()
{
	int e = 0;
	cudaDeviceSynchronize();
	if (cudaMemcpyFromSymbol(&e, g_fft_wait_err, sizeof(int)) != cudaSuccess) { cudaGetLastError(); return 0; }
	if (e) {
		const int z = 0;
		cudaMemcpyToSymbol(g_fft_wait_err, &z, sizeof(int));
	}
	return e | fft_gen_take_wait_error();
}
