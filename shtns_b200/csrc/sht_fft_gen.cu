// Longitude FFT for every nphi with prime factors 2, 3, 5 and 7 (the sizes
// without a compile-time chain in sht_fft.cu).
//
// A CTA transforms 2 S consecutive latitudes of one field-component, packed in
// pairs into S complex sequences as in sht_fft.cu.  nphi is split into as few
// passes as possible with radices 2 .. 16 (three up to 4096), each butterfly
// in registers: the first pass reads its inputs from global memory, the last
// pass of the synthesis writes the grid, and the passes between exchange
// through one shared-memory buffer in place (a thread holds all its
// butterflies, at most E complex values, while the CTA synchronises).
// Thread g handles sequence g mod S and butterfly g / S, so the sequences of
// one butterfly are neighbours in a warp and read or write contiguous latitude
// pairs.
//
// What bounds it: instruction issue (the indices are run-time values) and the
// latency of the passes at 20 to 25 warps per SM, not memory.  The form
// before this one ran radices <= 8 with two buffers, separate staging loops
// for the input and the output and run-time divisions in them: 314
// instructions per complex point at nphi 1440, 53 % of the issue slots, DRAM
// at 13 %.  Now 114 and 137 instructions per point
// (synthesis, analysis) and (stage times, before / now) nphi 1440, 13 grids of
// 720 latitudes, theta-contiguous 115/147 and 70/64 us; nphi 512, 64 grids of 256,
// phi-contiguous 50/55 and 41/40; nphi 1024, 40 of 512 147/179 and 95/92; nphi 2688,
// 8 of 1302 phi-contiguous 278/309 and 175/162.  The carve-out is left to the
// driver: at the maximum of shared memory the L1 cache holds too few lines of
// the loads in flight (nphi 2160: 152 -> 203 us with direct loads).
#include "sht_internal.h"
#include "sht_dft.h"
#include "sht_fft_tma.h"
#include "sht_fft_grid.h"

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <type_traits>

namespace {

using namespace shtb_dft;
using namespace shtb_fft_tma;
using namespace shtb_fft_grid;

// Register classes: E complex values per thread, the largest CTA, and the
// threads per SM that the registers are bounded for (56, 72 and 96 of them)
constexpr int gen_tmax(int E) { return E == 8 ? 384 : (E == 12 ? 896 : 640); }
constexpr int gen_minb(int E) { return E == 8 ? 3 : 1; }

// element i of a sequence: one slot of padding per 8 elements, so that the
// stride-R writes of the first pass spread over the banks
__device__ __forceinline__ int pos(int i) { return i + (i >> 3); }

// What a thread knows of its tile: its sequence (latitude pair row, row + 1)
// and its first butterfly b0; butterflies b0 + i bstep are its own.
template <class G>
struct GenTile {
	double2* Xs;             // the sequence in shared memory
	double2* Ff;             // Fourier rows of the field-component
	const G* in;             // grid (analysis)
	G* out;                  // grid (synthesis)
	const double2* tw;
	const void* stg;         // the staged tile (STG): rows of S latitude pairs, this sequence's column
	int N, nlat, ml, row, b0, bstep, S;
	bool live, phi, v2, v4;
};

__device__ int g_gen_wait_err;                   // set when a bounded wait gave up

// Every pass recomputes its indices from here: without this the compiler
// keeps those of all radices in registers across the passes.
__device__ __forceinline__ void opaque(int& v) { asm volatile("" : "+r"(v)); }

// input element j of the sequence, from the staged tile (STG) or global memory
// (of the analysis as it is stored: see load_pair)
template <bool SYNTH, class G> using GenIn = std::conditional_t<SYNTH, double2, typename Pair<G>::T>;

template <bool SYNTH, bool STG, bool PHI, class G>
__device__ __forceinline__ GenIn<SYNTH, G> gen_load(const GenTile<G>& t, int j)
{
	if constexpr (SYNTH) {
		// Z_j = A_j + i B_j (j <= ml), Z_{N-j} = conj(A_j) + i conj(B_j), zero between
		const bool lo = j <= t.ml;
		const int k = lo ? j : t.N - j;
		const bool in = k <= t.ml && (STG || t.live);
		double2 a, b;
		if constexpr (STG) {
			if (!in) return make_double2(0.0, 0.0);
			// the two latitudes in an order that alternates with the row, so that
			// the 8 lanes of a shared-memory phase hit distinct banks
			const int f = (k >> (t.S == 1 ? 2 : (t.S == 2 ? 1 : 0))) & 1;
			const double2* r = static_cast<const double2*>(t.stg) + k * 2 * t.S;
			const double2 u0 = r[f], u1 = r[1 - f];
			a = f ? u1 : u0;
			b = f ? u0 : u1;
		} else {
			// in the zero band the first element, thrown away: a load on a path
			// of its own is waited for there.  One 32-byte load for both latitudes
			// where the rows are aligned.  Kernel times, cold L2, two loads in a
			// branch / this form: nphi 128, 504 pairs, orders up to nphi / 2
			// 7.5 / 6.3 us, nphi / 3 6.7 / 6.1; nphi 4096, 64 pairs 19.8 / 16.9 and
			// 17.5 / 15.5 (with a zero band of nearly all orders the branch would be
			// 0.1 to 0.3 us faster; both forms in one kernel lose this gain)
			const double2* f = t.Ff + (in ? (long)k * t.nlat + t.row : 0);
			if (t.v4) asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y) : "l"(f));
			else { a = __ldg(f); b = __ldg(f + 1); }
			if (!in) return make_double2(0.0, 0.0);
		}
		if (k == 0) { a.y = 0.0; b.y = 0.0; }
		return lo ? make_double2(a.x - b.y, a.y + b.x) : make_double2(a.x + b.y, b.x - a.y);
	} else if constexpr (STG) {
		return static_cast<const typename Pair<G>::T*>(t.stg)[j * t.S];
	} else {
		typename Pair<G>::T v = {};
		if constexpr (PHI) {
			const G* i0 = t.in + (long)t.row * t.N + j;
			if (t.live) { v.x = __ldg(i0); v.y = __ldg(i0 + t.N); }
		} else if (t.live) v = load_pair(t.in + (long)j * t.nlat + t.row, t.v2);
		return v;
	}
}

// first pass: no twiddles, outputs b R + q; a staged tile lies in the same
// shared memory, so every thread reads its inputs before any writes
template <int R, int E, bool SYNTH, bool STG, bool PHI, class G>
__device__ __forceinline__ void gen_first(GenTile<G> t, int nbf)
{
	opaque(t.b0);
	constexpr int NB = E / R;
	GenIn<SYNTH, G> in[NB][R];
	#pragma unroll
	for (int i = 0; i < NB; i++) {
		const int b = t.b0 + i * t.bstep;
		if (b < nbf) {
			#pragma unroll
			for (int q = 0; q < R; q++) in[i][q] = gen_load<SYNTH, STG, PHI>(t, b + q * nbf);
		}
	}
	if constexpr (STG) __syncthreads();
	#pragma unroll
	for (int i = 0; i < NB; i++) {
		const int b = t.b0 + i * t.bstep;
		if (b < nbf) {
			double2 u[R];
			#pragma unroll
			for (int q = 0; q < R; q++) u[q] = widen(in[i][q]);
			Dft<R>::run(u, SYNTH ? 1 : -1);
			#pragma unroll
			for (int q = 0; q < R; q++) t.Xs[pos(b * R + q)] = u[q];
		}
	}
	__syncthreads();
}

// middle pass, in place
template <int R, int E, bool SYNTH, class G>
__device__ __forceinline__ void gen_mid(GenTile<G> t, const FftPass& ps)
{
	opaque(t.b0);
	constexpr int NB = E / R;
	double2 u[NB][R];
	int o[NB];
	#pragma unroll
	for (int i = 0; i < NB; i++) {
		const int b = t.b0 + i * t.bstep;
		if (b < ps.nbf) {
			#pragma unroll
			for (int q = 0; q < R; q++) u[i][q] = t.Xs[pos(b + q * ps.nbf)];
			// k = b mod P by a float reciprocal and one correction (b < 2^13)
			int k = b - __float2int_rz(__int2float_rn(b) * ps.inv_p) * ps.P;
			if (k < 0) k += ps.P;
			else if (k >= ps.P) k -= ps.P;
			double2 w = __ldg(t.tw + k * ps.ts);
			if (!SYNTH) w.y = -w.y;
			twiddles<R>(u[i], w);
			Dft<R>::run(u[i], SYNTH ? 1 : -1);
			o[i] = (b - k) * R + k;
		} else {
			// defined on every path: otherwise the registers of all radices
			// stay live around the loop over the passes
			o[i] = 0;
			#pragma unroll
			for (int q = 0; q < R; q++) u[i][q] = make_double2(0.0, 0.0);
		}
	}
	__syncthreads();
	#pragma unroll
	for (int i = 0; i < NB; i++)
		if (t.b0 + i * t.bstep < ps.nbf) {
			#pragma unroll
			for (int q = 0; q < R; q++) t.Xs[pos(o[i] + q * ps.P)] = u[i][q];
		}
	__syncthreads();
}

// last pass of the synthesis (P = N / R, k = b), to the grid
template <int R, class G>
__device__ __forceinline__ void gen_last(GenTile<G> t, int nbf)
{
	opaque(t.b0);
	for (int b = t.b0; b < nbf; b += t.bstep) {
		double2 u[R];
		#pragma unroll
		for (int q = 0; q < R; q++) u[q] = t.Xs[pos(b + q * nbf)];
		twiddles<R>(u, __ldg(t.tw + b));
		Dft<R>::run(u, 1);
		if (!t.live) continue;
		if (t.phi) {
			G* o = t.out + (long)t.row * t.N + b;
			#pragma unroll
			for (int q = 0; q < R; q++) {
				o[q * nbf] = (G) u[q].x;
				o[q * nbf + t.N] = (G) u[q].y;
			}
		} else {
			G* o = t.out + (long)b * t.nlat + t.row;
			const long step = (long) nbf * t.nlat;
			#pragma unroll
			for (int q = 0; q < R; q++) store_pair(o + q * step, u[q], t.v2);
		}
	}
}

// call(R) for the run-time radix
#define GEN_CASE(call, R) call(R); break;
#define GEN_RADIX(radix, call) \
	switch (radix) { \
		case 1: GEN_CASE(call, 1) \
		case 2: GEN_CASE(call, 2) \
		case 3: GEN_CASE(call, 3) \
		case 4: GEN_CASE(call, 4) \
		case 5: GEN_CASE(call, 5) \
		case 6: GEN_CASE(call, 6) \
		case 7: GEN_CASE(call, 7) \
		case 8: GEN_CASE(call, 8) \
		case 9: if constexpr (E >= 9) { GEN_CASE(call, 9) } break; \
		case 10: if constexpr (E >= 10) { GEN_CASE(call, 10) } break; \
		case 12: if constexpr (E >= 12) { GEN_CASE(call, 12) } break; \
		case 15: if constexpr (E >= 15) { GEN_CASE(call, 15) } break; \
		case 16: if constexpr (E >= 16) { GEN_CASE(call, 16) } break; \
		default: break; \
	}

// E: complex values a thread holds (8, 12 or 16); a pass of radix R runs E / R
// butterflies per thread
// STG: the input tile arrives by tensor copies in the shared buffer that the
// passes use (box_rows rows per copy, ncopy copies of box_bytes); PHI: direct
// reads of a phi-contiguous grid.
template <int E, bool SYNTH, bool STG, bool PHI, class G>
__global__ void __launch_bounds__(gen_tmax(E), gen_minb(E))
fft_gen_kernel(const __grid_constant__ CUtensorMap m0, const __grid_constant__ CUtensorMap m1, const __grid_constant__ CUtensorMap m2,
               FftParams p, FftGenPlan g, int lgS, int seq, int ncopy, int box_rows, int box_bytes)
{
	extern __shared__ __align__(128) double2 gsm[];
	double2* X = gsm;
	__shared__ __align__(8) uint64_t bar;
	if constexpr (STG) {
		X += ((128u - (su32(gsm) & 127u)) & 127u) / 16;          // tensor copies land on 128-byte boundaries
		if (threadIdx.x == 0) {
			asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(su32(&bar)) : "memory");
			asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
			const int fcb = blockIdx.y, cb = fcb / p.nf;
			const CUtensorMap* m = (SYNTH || cb == 0) ? &m0 : (cb == 1 ? &m1 : &m2);
			const int x = (blockIdx.x << lgS) * (SYNTH ? 4 : 2), z = SYNTH ? fcb : fcb - cb * p.nf;
			asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
			             :: "r"(su32(&bar)), "r"((unsigned)(ncopy * box_bytes + p.extra_tx)) : "memory");
			for (int c = 0; c < ncopy; c++)
				tma_tile3(reinterpret_cast<char*>(X) + c * box_bytes, m, x, c * box_rows, z, &bar);
		}
	}
	const int tid = threadIdx.x, S = 1 << lgS;
	const int fc = blockIdx.y, c = fc / p.nf;
	GenTile<G> t;
	t.N = p.N; t.nlat = p.nlat; t.ml = p.mlim;
	t.Ff = p.F + (long)fc * p.fstride;
	t.in = nullptr; t.out = nullptr;
	if constexpr (SYNTH) t.out = grid_out<G>(p, c, fc);
	else t.in = grid_in<G>(p, c, fc);
	t.tw = p.tw;
	t.phi = p.phi_contiguous; t.v2 = p.vec2;
	t.v4 = !((uintptr_t) t.Ff & 31) && !(t.nlat & 1);          // rows of F 32-byte aligned at even latitudes
	t.Xs = X + (tid & (S - 1)) * seq;                          // CTAs are multiples of S threads: one sequence per thread
	t.row = (blockIdx.x * S + (tid & (S - 1))) * 2;
	t.live = t.row < t.nlat;
	t.b0 = tid >> lgS;
	t.bstep = blockDim.x >> lgS;
	t.S = S;
	t.stg = SYNTH ? static_cast<const void*>(X + 2 * (tid & (S - 1)))
	              : static_cast<const void*>(reinterpret_cast<const typename Pair<G>::T*>(X) + (tid & (S - 1)));
	if constexpr (STG) {
		__syncthreads();                                       // the barrier is initialised
		const bool ok = fbar_wait(&bar, 0);
		if (__syncthreads_or(!ok)) {
			if (tid == 0) {
				atomicExch(&g_gen_wait_err, 1);
				fbar_wait(&bar, 0);                              // copies still in flight (bounded)
			}
			return;
		}
	}

	#define GEN_FIRST(R) gen_first<R, E, SYNTH, STG, PHI>(t, g.ps[0].nbf)
	GEN_RADIX(g.ps[0].R, GEN_FIRST)
	const int nmid = SYNTH ? g.np - 1 : g.np;
	for (int r = 1; r < nmid; r++) {
		#define GEN_MID(R) gen_mid<R, E, SYNTH>(t, g.ps[r])
		GEN_RADIX(g.ps[r].R, GEN_MID)
	}
	if constexpr (SYNTH) {
		#define GEN_LAST(R) gen_last<R>(t, g.ps[g.np - 1].nbf)
		GEN_RADIX(g.ps[g.np - 1].R, GEN_LAST)
	} else {
		// separate the two real spectra: A_k = (Z_k + conj Z_{N-k}) / 2, B_k = (Z_k - conj Z_{N-k}) / 2i
		const double sc = 0.5 / t.N;
		if (t.live)
			for (int k = t.b0; k <= t.ml; k += t.bstep) {
				const double2 z = t.Xs[pos(k)], w = t.Xs[pos(k ? t.N - k : 0)];
				const double2 fa = make_double2(sc * (z.x + w.x), sc * (z.y - w.y));
				const double2 fb = make_double2(sc * (z.y + w.y), -sc * (z.x - w.x));
				double2* o = t.Ff + (long)k * t.nlat + t.row;
				if (t.v4)
					asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};"
					             :: "l"(o), "d"(fa.x), "d"(fa.y), "d"(fb.x), "d"(fb.y) : "memory");
				else { o[0] = fa; o[1] = fb; }
			}
	}
}

// padded sequence length: the S sequences a warp reads side by side start in
// distinct banks (8 / S mod 8 in 16-byte units)
int seq_len(int N, int S)
{
	const int a = N + (N >> 3);
	return a + (((S >= 8 ? 1 : 8 / S) - a) & 7);
}

// threads of a CTA with S sequences: every pass of the first and middle kind
// fits E / R butterflies per thread
int gen_threads(const FftGenPlan& g, int S)
{
	int t = 1;
	for (int r = 0; r < g.np; r++) {
		const int nb = g.E / g.ps[r].R;
		t = std::max(t, (S * g.ps[r].nbf + nb - 1) / nb);
	}
	return (t + 31) / 32 * 32;
}

} // namespace

// Passes of nphi = N: the fewest with radices <= emax, then the smallest register
// class (8, 12 or 16 values per thread), then the fewest threads.  The first
// radix is one whose padded stride is odd where there is a choice (no bank
// conflicts in the first pass's writes).
bool fft_gen_plan(int N, FftGenPlan& out, int emax)
{
	static const int rad[] = {16, 15, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
	out = FftGenPlan();
	if (N == 1) {
		out.np = 2; out.E = 8;
		out.ps[0] = out.ps[1] = FftPass{1, 1, 1, 1, 1.0f};
		return true;
	}
	int best[FFT_MAX_PASSES], nbest = 0, ebest = 0, tbest = 0;
	int cur[FFT_MAX_PASSES];
	for (int E = 8; E <= emax; E += 4) {
		// depth-first over non-increasing radices
		auto search = [&](auto&& self, int n, int np, int from) -> void {
			if (n == 1) {
				int t = 0;
				for (int i = 0; i < np; i++) t = std::max(t, (N / cur[i] + E / cur[i] - 1) / (E / cur[i]));
				if (t > gen_tmax(E)) return;
				if (!nbest || np < nbest || (np == nbest && E == ebest && t < tbest)) {
					nbest = np; ebest = E; tbest = t;
					for (int i = 0; i < np; i++) best[i] = cur[i];
				}
				return;
			}
			if (np >= FFT_MAX_PASSES || (nbest && np + 1 > nbest)) return;
			for (int i = from; i < (int)(sizeof(rad) / sizeof(rad[0])); i++)
				if (rad[i] <= E && n % rad[i] == 0) { cur[np] = rad[i]; self(self, n / rad[i], np + 1, i); }
		};
		search(search, N, 0, 0);
	}
	if (!nbest) return false;
	for (int i = 0; i < nbest; i++)
		if ((best[i] + (best[i] >> 3)) & 1) { std::swap(best[0], best[i]); break; }
	out.np = nbest; out.E = ebest;
	int P = 1;
	for (int i = 0; i < nbest; i++) {
		const int R = best[i];
		out.ps[i] = FftPass{R, P, N / R, N / (P * R), 1.0f / P};
		P *= R;
	}
	if (nbest == 1) { out.ps[1] = FftPass{1, N, N, 1, 1.0f / N}; out.np = 2; }     // the last pass of a single-radix synthesis copies
	return true;
}

static std::atomic<int> g_gen_last{-1};

// The last launch of this file in this process: 100 E + 10 passes + staged.
int fft_gen_last() { return g_gen_last.load(); }

void launch_fft_gen(const FftParams& p, int nfc, cudaStream_t st, bool synth)
{
	// Up to about a wave of latitude pairs the latency of the passes counts, not
	// the rate: short butterflies (radices <= 8, more threads, less code to
	// fetch) and direct loads.  Kernel times with cold L2, orders up to nphi / 3,
	// direct / staged: synthesis of 512 pairs at nphi 720 8.2/9.0 us, 1024
	// 10.2/11.8; analysis 720 8.0/8.5, 1440 13.3/13.1, 2880 32.2/34.4.  The same
	// synthesis with the longest butterflies the length allows: nphi 256, 256
	// pairs 5.6 -> 7.6, 1024 9.2 -> 10.5 (with warm caches 4.9 and 6.5).
	// The synthesis of longer rows is staged all the same (512 pairs, direct /
	// staged: nphi 1440 17.4/15.4, 2048 23.1/20.1, 4096 59.9/50.1), except up to
	// 2^19 points, where the whole call is bound by its launches, and with orders
	// up to less than nphi / 4 (nphi 4096, 192 pairs, nphi / 32: 18.9/20.3 warm).
	// Plans that need 16 values per thread lose to one more pass in large calls
	// too (nphi 1024, 2560 pairs 41.3/40.9 and 33.2/36.9, 10240 phi-contiguous
	// 87.7/92.1 and 78.6/92.6), so they stay for the lengths without the other.
	const long pairs = (long)((p.nlat + 1) / 2) * nfc;
	const bool small = pairs <= 1000;
	const FftGenPlan& g = (p.gen_small->np && (small || p.gen->E == 16)) ? *p.gen_small : *p.gen;
	const int tmax = gen_tmax(g.E);
	auto smem = [&](int S) { return sizeof(double2) * (size_t) S * seq_len(p.N, S); };
	int S = 1;
	if (p.pairs) {
		while (2 * S <= p.pairs && gen_threads(g, 2 * S) <= tmax && smem(2 * S) <= 224 * 1024) S *= 2;
	} else {
		// sequences per CTA: rows of up to 8 latitude pairs (whole lines) while the
		// CTA stays small enough for several per SM; phi-contiguous rows need none
		// (nphi 512, 8192 pairs, 2 and 4 sequences: 36.4/37.2 and 41.4/39.3 us
		// phi-contiguous, 41.0/39.9 and 41.3/39.0 theta-contiguous)
		while (S < 8 && gen_threads(g, 2 * S) <= (p.phi_contiguous ? 192 : 384) && smem(2 * S) <= 72 * 1024 && (pairs >= 2 * S * 2 * 148 || (S == 1 && small))) S *= 2;
	}
	while (S > 1 && 2 * S > p.nlat) S /= 2;
	int lgS = 0;
	while ((1 << lgS) < S) lgS++;
	// a grid of fewer CTAs than two per SM gets twice the threads: fewer
	// butterflies in series per thread
	const long ctas = (long)((p.nlat + 2 * S - 1) / (2 * S)) * nfc;
	int T = gen_threads(g, S);
	if (ctas < 2 * 148 * 2) T = std::min(tmax, std::max(T, (S * p.N / 8 + 31) / 32 * 32));
	dim3 grid((p.nlat + 2 * S - 1) / (2 * S), nfc);
	const int seq = seq_len(p.N, S);
	// staged input: the Fourier rows, or a theta-contiguous grid that tensor
	// copies can address (phi-contiguous rows are read in whole lines as they are)
	alignas(64) CUtensorMap maps[3];
	const int e = p.f32 ? 4 : 8;
	const bool long_rows = synth && p.N > 1024 && pairs * p.N > (1 << 19) && 4 * (p.mlim + 1) >= p.N;
	bool stg = (!small || long_rows) && !(p.nlat & 1) && (synth || (p.vec2 && !p.phi_contiguous));
	const int rows = synth ? p.mlim + 1 : p.N, row_bytes = synth ? 32 * S : 2 * e * S;
	const int ncopy = (rows + 255) / 256;
	const int box = ((rows + ncopy - 1) / ncopy + 15) & ~15;        // a multiple of 16: copies of 128-byte multiples
	if (stg && synth) {
		stg = encode3(&maps[0], p.F, 2 * (uint64_t) p.nlat, rows, nfc, 16 * (uint64_t) p.nlat, 16 * (uint64_t) p.fstride, 4 * S, box);
		maps[1] = maps[2] = maps[0];
	} else if (stg) {
		const int ncomp = (nfc + p.nf - 1) / p.nf;
		for (int c = 0; c < 3 && stg; c++)
			stg = encode3(&maps[c], p.spat_in[c < ncomp ? c : 0], p.nlat, p.N, p.nf, (uint64_t) e * p.nlat, (uint64_t) e * p.spat_dist,
			              2 * S, box, p.f32);
	}
	const size_t sm = std::max(smem(S), (size_t) ncopy * box * row_bytes) + 128;
	if (sm > 226 * 1024) stg = false;
	g_gen_last = 100 * g.E + 10 * g.np + (stg ? 1 : 0);
	auto go = [&](auto kern) {
		kern<<<grid, T, stg ? sm : smem(S), st>>>(maps[0], maps[1], maps[2], p, g, lgS, seq, ncopy, box, box * row_bytes);
	};
	auto pick = [&](auto EC, auto GC) {
		constexpr int E = decltype(EC)::value;
		using G = decltype(GC);
		if (synth) go(stg ? fft_gen_kernel<E, true, true, false, G> : fft_gen_kernel<E, true, false, false, G>);
		else if (stg) go(fft_gen_kernel<E, false, true, false, G>);
		else go(p.phi_contiguous ? fft_gen_kernel<E, false, false, true, G> : fft_gen_kernel<E, false, false, false, G>);
	};
	auto pick_e = [&](auto GC) {
		switch (g.E) {
			case 8: pick(std::integral_constant<int, 8>{}, GC); break;
			case 12: pick(std::integral_constant<int, 12>{}, GC); break;
			default: pick(std::integral_constant<int, 16>{}, GC); break;
		}
	};
	if (p.f32) pick_e(float{});
	else pick_e(double{});
}

void fft_gen_set_smem_limits()
{
	auto all = [&](auto EC, auto GC) {
		constexpr int E = decltype(EC)::value;
		using G = decltype(GC);
		// 1 KB short of the limit: the staged kernels also hold an mbarrier in static shared memory
		for (auto k : {fft_gen_kernel<E, true, true, false, G>, fft_gen_kernel<E, true, false, false, G>, fft_gen_kernel<E, false, true, false, G>,
		               fft_gen_kernel<E, false, false, true, G>, fft_gen_kernel<E, false, false, false, G>})
			cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
	};
	auto both = [&](auto EC) { all(EC, double{}); all(EC, float{}); };
	both(std::integral_constant<int, 8>{});
	both(std::integral_constant<int, 12>{});
	both(std::integral_constant<int, 16>{});
}

// Returns and clears the flag of this file's kernels (after a device synchronisation).
int fft_gen_take_wait_error()
{
	int e = 0;
	if (cudaMemcpyFromSymbol(&e, g_gen_wait_err, sizeof(int)) != cudaSuccess) { cudaGetLastError(); return 0; }
	if (e) {
		const int z = 0;
		cudaMemcpyToSymbol(g_gen_wait_err, &z, sizeof(int));
	}
	return e;
}
