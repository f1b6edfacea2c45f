// Legendre contraction tiles on the FP64 tensor cores, shared by the kernels of
// sht_legendre.cu (64 x 64 and 128 x 32 tiles, plan groups) and
// sht_legendre_narrow.cu (128 x 16 tiles).  Two files, because the register
// allocation of one kernel changes with the others compiled beside it: with
// the narrow tiles in the same file the 128 x 32 synthesis at 32-step
// checkpoints spilled and took 4.27 instead of 3.81 ms at lmax 2047, 8 fields.
#pragma once

#include "sht_internal.h"

#include <type_traits>

namespace {

// FP64 tensor-core product of a 16 x 4 A tile and a 4 x 8 B tile
// (mma.sync m16n8k4): A rows g and g + 8 (a0, a1), C rows g (c0, c1) and
// g + 8 (c2, c3) for lane = 4 g + t; the registers of two row-adjacent
// 8 x 8 fragments.  Measured on B200 against m8n8k4 pairs: analysis 5 % faster
// at 64 fields, 14 % at 8; m16n8k8 (two k steps per instruction) was slower.
__device__ __forceinline__ void dmma16(double (&c0)[2], double (&c1)[2], double a0, double a1, double b)
{
	asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
	             : "+d"(c0[0]), "+d"(c0[1]), "+d"(c1[0]), "+d"(c1[1]) : "d"(a0), "d"(a1), "d"(b));
}

// Read-only load that does not allocate in L1: the streamed operands (F rows,
// coefficient rows, checkpoints) are read once per CTA, and keeping them out
// of L1 leaves it to the small per-row tables that every chunk's staging reads
// (recurrence coefficients, weights, cos and 1/sin of the latitudes).
__device__ __forceinline__ double2 ldg_stream(const double2* q)
{
	double2 v;
	asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(q));
	return v;
}

// ---------------------------------------------------------------------------
// Synthesis contraction.  CTA = (order im, 64 north theta rows, 64 columns).
// 8 warps as 2 (theta) x 4 (columns); a warp owns 32 rows x 16 columns = one
// group of 4 field-components, so each lane ends with (E_re, E_im, O_re, O_im)
// of one (row, field-component) and folds north/south itself.
#define SA_LD 68   // shared row stride in doubles: 4 mod 16 keeps fragment loads conflict-free

// CTA shape: WM x WN warps of 32 rows x 16 columns.  WM = 2: 64 rows x 64
// columns; 4: 128 x 32, for calls with at most 8 field-components; 5 stands for
// four warps of 128 x 16 (at most 4 field-components).
__host__ __device__ constexpr int leg_wm(int WM) { return WM == 5 ? 4 : WM; }
__host__ __device__ constexpr int leg_wn(int WM) { return WM == 5 ? 1 : 8 / WM; }
__host__ __device__ constexpr int leg_nt(int WM) { return 32 * leg_wm(WM) * leg_wn(WM); }
__host__ __device__ constexpr int leg_minb(int WM) { return WM == 1 ? 2 : (WM == 5 ? 5 : 3); }

// RB: Fourier rows in per-block buffers (p.rb) instead of the plain F
template <int SEG, int WM, bool RB = false>
__device__ __forceinline__ void leg_synth_tile(const LegParams& p, int im, int tb, int nb)
{
	constexpr int WN = leg_wn(WM), BM = 32 * leg_wm(WM), BN = 16 * WN, NT = leg_nt(WM);
	__shared__ __align__(16) double As[LG_BK][BM + 4];   // [k][theta]; strides 4 mod 16:
	__shared__ __align__(16) double Bs[LG_BK][BN + 4];   // [k][col]    conflict-free fragment loads
	const int m = im * p.mres;
	const int t0 = tb * BM, c0 = nb * BN;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int wm = warp / WN, wn = warp % WN;
	const int nk = (p.llim + p.vec_extra - m) / 2 + 1;
	const int tmm = p.mt.tm[im];

	double acc[4][2][2];
	#pragma unroll
	for (int i = 0; i < 4; i++)
		#pragma unroll
		for (int j = 0; j < 2; j++) { acc[i][j][0] = 0.0; acc[i][j][1] = 0.0; }

	// 8 x 8 fragments of this warp that carry results: rows in [tmm, nlat/2),
	// columns below ncol (the others are discarded by the epilogue)
	const int wr = t0 + wm * 32, wc = c0 + wn * 16;
	const int ri0 = min(4, max(0, (tmm - wr) / 8));
	const int ri1 = min(4, max(0, (p.nlat_2 - wr + 7) / 8));
	const int cj1 = min(2, max(0, (p.ncol - wc + 7) / 8));
	if (t0 + BM > tmm) {
		const double* cm = p.c + p.mt.coff[im];
		const double2* ckm = p.ck + (long)p.mt.ckoff[im] * p.nlat_2;
		const double* qrow = p.qq + (long)p.mt.koff[im] * p.ncol;
		// software pipeline: the B tile and checkpoint of chunk k0+32 are
		// loaded into registers while the tensor cores work on chunk k0
		constexpr int NBV = LG_BK * (BN / 2) / NT;   // double2 per thread
		double2 bn[NBV];
		// generators: thread (row gr, segment sg = gj + u GPR) produces Y_k for
		// SEG consecutive k of the chunk from the checkpoint at its segment start
		constexpr int NSEGC = LG_BK / SEG;                    // segments per chunk
		constexpr int GPR = NT / BM;                  // generator threads per row
		constexpr int SPT = (NSEGC + GPR - 1) / GPR;          // segments per generator thread
		double2 ckn[SPT];
		const int gr = tid % BM, gj = tid / BM;
		const int tg = t0 + gr;
		const bool gen = tg < p.nlat_2;
		const double x2 = gen ? p.x2[tg] : 0.0;
		auto load_b = [&](int k0) {
			#pragma unroll
			for (int u = 0; u < NBV; u++) {
				const int e = tid + u * NT;
				const int kk = e / (BN / 2), cc2 = (e - kk * (BN / 2)) * 2;
				const int k = k0 + kk, col = c0 + cc2;
				bn[u] = (k < nk && col < p.ncol) ? ldg_stream(reinterpret_cast<const double2*>(qrow + (long)k * p.ncol + col))
				                                 : make_double2(0.0, 0.0);
			}
			#pragma unroll
			for (int u = 0; u < SPT; u++) {
				const int sg = gj + u * GPR;
				const int ks = k0 + sg * SEG;
				ckn[u] = (sg < NSEGC && gen && ks < nk) ? ldg_stream(ckm + (long)(ks / SEG) * p.ckrow + tg)
				                                       : make_double2(0.0, 0.0);
			}
		};
		load_b(0);
		for (int k0 = 0; k0 < nk; k0 += LG_BK) {
			#pragma unroll
			for (int u = 0; u < SPT; u++) {
				const int sg = gj + u * GPR;
				if (sg < NSEGC) {
					double y0 = ckn[u].x, y1 = ckn[u].y;
					As[sg * SEG][gr] = y0;
					As[sg * SEG + 1][gr] = y1;
					const double* cc = cm + 2 * (k0 + sg * SEG);
					#pragma unroll
					for (int j = 2; j < SEG; j++) {
						const double a = fma(cc[2 * j - 1], x2, cc[2 * j - 2]);
						const double y2 = fma(a, y1, y0);
						As[sg * SEG + j][gr] = y2;
						y0 = y1; y1 = y2;
					}
				}
			}
			#pragma unroll
			for (int u = 0; u < NBV; u++) {
				const int e = tid + u * NT;
				const int kk = e / (BN / 2), cc2 = (e - kk * (BN / 2)) * 2;
				*reinterpret_cast<double2*>(&Bs[kk][cc2]) = bn[u];
			}
			__syncthreads();
			if (k0 + LG_BK < nk) load_b(k0 + LG_BK);
			const int kv = nk - k0;                      // steps of this chunk below nk
			// P0, P1: row-fragment pairs (0, 1) and (2, 3) computed; NJ column
			// fragments.  The choice is made once per warp with a branch: an MMA
			// switched off by a predicate still occupies the tensor pipe.
			auto mma_chunk = [&](auto P0, auto P1, auto NJ) {
				#pragma unroll
				for (int kk = 0; kk < LG_BK; kk += 4) {
					if (kk >= kv) break;                  // rows of Bs beyond nk are zero
					double a[4], b[2];
					#pragma unroll
					for (int i = 0; i < 4; i++)
						if ((i < 2 && P0.value) || (i >= 2 && P1.value)) a[i] = As[kk + (lane & 3)][wm * 32 + i * 8 + (lane >> 2)];
					#pragma unroll
					for (int j = 0; j < NJ.value; j++) b[j] = Bs[kk + (lane & 3)][wn * 16 + j * 8 + (lane >> 2)];
					#pragma unroll
					for (int j = 0; j < NJ.value; j++) {
						if constexpr (P0.value) dmma16(acc[0][j], acc[1][j], a[0], a[1], b[j]);
						if constexpr (P1.value) dmma16(acc[2][j], acc[3][j], a[2], a[3], b[j]);
					}
				}
			};
			// fragment pairs (i, i + 1) carry results when either row fragment does
			const bool p0 = ri0 <= 1 && ri1 > 0, p1 = ri0 <= 3 && ri1 > 2;
			using T = std::true_type;
			using F = std::false_type;
			using J1 = std::integral_constant<int, 1>;
			using J2 = std::integral_constant<int, 2>;
			if (cj1 == 2) {
				if (p0 && p1) mma_chunk(T{}, T{}, J2{});
				else if (p0) mma_chunk(T{}, F{}, J2{});
				else if (p1) mma_chunk(F{}, T{}, J2{});
			} else if (cj1 == 1) {
				if (p0 && p1) mma_chunk(T{}, T{}, J1{});
				else if (p0) mma_chunk(T{}, F{}, J1{});
				else if (p1) mma_chunk(F{}, T{}, J1{});
			}
			__syncthreads();
		}
	}
	// epilogue: fold hemispheres, apply 1/sin for vector components, store F
	const int fc = ((c0 + wn * 16) >> 4) * 4 + (lane & 3);
	if (fc >= p.nfc) return;
	const bool vec = (p.ctype[fc / p.nf] != 0) && !p.robert;
	double2* Ff = p.F + (long)fc * p.fstride + (long)im * p.nlat;     // plain layout (p.rb.n == 0)
	#pragma unroll
	for (int i = 0; i < 4; i++) {
		const int t = t0 + wm * 32 + i * 8 + (lane >> 2);
		if (t >= p.nlat_2) continue;
		const double cx = p.x[t];
		double nr = fma(cx, acc[i][1][0], acc[i][0][0]), ni = fma(cx, acc[i][1][1], acc[i][0][1]);
		double sr = fma(-cx, acc[i][1][0], acc[i][0][0]), si = fma(-cx, acc[i][1][1], acc[i][0][1]);
		if (t < tmm) { nr = ni = sr = si = 0.0; }
		if (vec) { const double s = p.sinv[t]; nr *= s; ni *= s; sr *= s; si *= s; }
		if (p.adjoint) {
			// adjoint of the analysis: row weight W_t(m) / (nphi (2 - delta_m0))
			const double s = p.w[t] * (m > 0 ? p.mpos_inv : 1.0) / (p.nphi * (m > 0 ? 2.0 : 1.0));
			nr *= s; ni *= s; sr *= s; si *= s;
		}
		const int rn = p.south_first ? p.nlat - 1 - t : t;
		const int rs = p.nlat - 1 - rn;
		if constexpr (!RB) {
			Ff[rn] = make_double2(nr, ni);
			Ff[rs] = make_double2(sr, si);
		} else {
			*fourier_row(p, fc, im, rn) = make_double2(nr, ni);
			*fourier_row(p, fc, im, rs) = make_double2(sr, si);
		}
	}
}

// ---------------------------------------------------------------------------
// Analysis contraction.  CTA = (order im, 64 k rows, 64 columns); the K loop
// runs over north theta rows in chunks of 32, starting at the polar threshold.
// The B operand is built while staging: G_even = w (F_N + F_S),
// G_odd = w cos(theta) (F_N - F_S) (kernel_spat_to_SH.gen.c:485-491), times
// 1/sin(theta) for vector components (1/sin^2 in Robert form).
#define AA_LD 36   // As row stride (k rows x 32 theta): 4 mod 16

// WM = warps along the k rows (2: 64 k x 64 columns per CTA; 4: 128 k x 32
// columns, for calls with at most 8 field-components).
template <int SEG, int WM, bool RB = false>
__device__ __forceinline__ void leg_analys_tile(const LegParams& p, int im, int kb, int nb)
{
	constexpr int WN = leg_wn(WM), BM = 32 * leg_wm(WM), BN = 16 * WN, NT = leg_nt(WM);
	__shared__ __align__(16) double As[BM][AA_LD];       // [k][theta]
	__shared__ __align__(16) double Bs[LG_BK][BN + 4];   // [theta][col]
	const int m = im * p.mres;
	const int k0 = kb * BM, c0 = nb * BN;
	const int nk = (p.llim + p.vec_extra - m) / 2 + 1;
	if (k0 >= nk) return;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int wm = warp / WN, wn = warp % WN;
	const int tmm = p.mt.tm[im];
	const double wfac = (m > 0) ? p.mpos_inv : 1.0;
	const double* cm = p.c + p.mt.coff[im];
	const double2* ckm = p.ck + (long)p.mt.ckoff[im] * p.nlat_2;
	const int fc0 = c0 / 4;
	// 8 x 8 fragments of this warp that carry results: k below nk, columns
	// below ncol (the others are not stored)
	const int ki1 = min(4, max(0, (nk - k0 - wm * 32 + 7) / 8));
	const int cj1 = min(2, max(0, (p.ncol - c0 - wn * 16 + 7) / 8));

	double acc[4][2][2];
	#pragma unroll
	for (int i = 0; i < 4; i++)
		#pragma unroll
		for (int j = 0; j < 2; j++) { acc[i][j][0] = 0.0; acc[i][j][1] = 0.0; }

	// software pipeline: F values and checkpoints of the next theta chunk are
	// loaded into registers while the tensor cores work on the current one
	constexpr int NBF = LG_BK * (BN / 4) / NT;   // (theta, field-component) items per thread
	double2 fnn[NBF], fsn[NBF];
	// generators: thread (theta gtt, segment sg = gsg + u GPT) produces Y_k
	// for SEG consecutive k of the CTA's k rows from the checkpoint at its
	// segment start
	constexpr int NSG = BM / SEG;                         // segments per tile
	constexpr int GPT = NT / LG_BK;               // generator threads per theta
	constexpr int SPT = (NSG + GPT - 1) / GPT;            // segments per generator thread
	double2 ckn[SPT];
	const int gtt = tid % LG_BK, gsg = tid / LG_BK;
	// vector flag of each staging item's field-component (fixed per thread)
	bool vecn[NBF];
	#pragma unroll
	for (int u = 0; u < NBF; u++) {
		const int fc = fc0 + (tid + u * NT) / LG_BK;
		vecn[u] = fc < p.nfc && p.ctype[fc / p.nf] != 0;
	}
	auto load_next = [&](int tt0) {
		#pragma unroll
		for (int u = 0; u < NBF; u++) {
			const int e = tid + u * NT;
			const int tt = e % LG_BK, fl = e / LG_BK;
			const int t = tt0 + tt, fc = fc0 + fl;
			fnn[u] = make_double2(0.0, 0.0); fsn[u] = make_double2(0.0, 0.0);
			if (t < p.nlat_2 && t >= tmm && fc < p.nfc) {
				const int rn = p.south_first ? p.nlat - 1 - t : t;
				const int rs = p.nlat - 1 - rn;
				if constexpr (!RB) {
					const double2* Ff = p.F + (long)fc * p.fstride + (long)im * p.nlat;
					fnn[u] = ldg_stream(Ff + rn);
					fsn[u] = ldg_stream(Ff + rs);
				} else {
					fnn[u] = ldg_stream(fourier_row(p, fc, im, rn));
					fsn[u] = ldg_stream(fourier_row(p, fc, im, rs));
				}
			}
		}
		const int t = tt0 + gtt;
		#pragma unroll
		for (int u = 0; u < SPT; u++) {
			const int sg = gsg + u * GPT, gks = k0 + sg * SEG;
			ckn[u] = (sg < NSG && t < p.nlat_2 && gks < nk) ? ldg_stream(ckm + (long)(gks / SEG) * p.ckrow + t)
			                                               : make_double2(0.0, 0.0);
		}
	};
	// recurrence coefficients of the CTA's k rows, staged once (rows at or
	// beyond nk get zeros: their results are not stored)
	__shared__ double cs[2 * BM];
	for (int e = tid; e < 2 * BM; e += NT) cs[e] = (k0 + e / 2 < nk) ? cm[2 * k0 + e] : 0.0;
	__syncthreads();
	const int tstart = (tmm / LG_BK) * LG_BK;
	if (tstart < p.nlat_2) load_next(tstart);
	for (int tt0 = tstart; tt0 < p.nlat_2; tt0 += LG_BK) {
		{
			const int t = tt0 + gtt;
			const double x2 = (t < p.nlat_2) ? p.x2[t] : 0.0;
			#pragma unroll
			for (int u = 0; u < SPT; u++) {
				const int sg = gsg + u * GPT, gks = k0 + sg * SEG;
				if (sg >= NSG) break;
				double y0 = ckn[u].x, y1 = ckn[u].y;
				double* a = &As[sg * SEG][gtt];
				a[0] = y0;
				a[AA_LD] = y1;
				if (gks < nk) {
					const double* cc = cs + 2 * sg * SEG;
					#pragma unroll
					for (int j = 2; j < SEG; j++) {
						const double aa = fma(cc[2 * j - 1], x2, cc[2 * j - 2]);
						const double y2 = fma(aa, y1, y0);
						a[j * AA_LD] = y2;
						y0 = y1; y1 = y2;
					}
				} else {
					for (int j = 2; j < SEG; j++) a[j * AA_LD] = 0.0;
				}
			}
		}
		#pragma unroll
		for (int u = 0; u < NBF; u++) {
			const int e = tid + u * NT;
			const int tt = e % LG_BK, fl = e / LG_BK;
			const int t = tt0 + tt, fc = fc0 + fl;
			double er = 0.0, ei = 0.0, orr = 0.0, oi = 0.0;
			if (t < p.nlat_2 && fc < p.nfc) {
				// adjoint of the synthesis: no quadrature weight, factor nphi (2 - delta_m0)
				double w = p.adjoint ? p.nphi * (m > 0 ? 2.0 : 1.0) : p.w[t] * wfac;
				if (vecn[u]) {
					double s = p.sinv[t];
					if (p.robert) s *= s;
					w *= s;
				}
				const double wo = w * p.x[t];
				const double2 fn = fnn[u], fs = fsn[u];
				er = w * (fn.x + fs.x);  ei = w * (fn.y + fs.y);
				orr = wo * (fn.x - fs.x); oi = wo * (fn.y - fs.y);
			}
			// columns swizzled by row: bits 1-2 of the column XOR (row / 4) % 4, so
			// that the 16 rows a half-warp stores hit distinct banks; the fragment
			// loads read 4 consecutive rows (one swizzle) and stay conflict-free
			const int cb = (16 * (fl >> 2) + 2 * (fl & 3)) ^ (2 * ((tt >> 2) & 3));
			*reinterpret_cast<double2*>(&Bs[tt][cb]) = make_double2(er, ei);
			*reinterpret_cast<double2*>(&Bs[tt][cb + 8]) = make_double2(orr, oi);
		}
		__syncthreads();
		if (tt0 + LG_BK < p.nlat_2) load_next(tt0 + LG_BK);
		// NP row-fragment pairs and NJ column fragments, chosen once per warp
		// with a branch (a predicated-off MMA still occupies the tensor pipe)
		auto mma_chunk = [&](auto NP, auto NJ) {
			#pragma unroll
			for (int kk = 0; kk < LG_BK; kk += 4) {
				double a[4], b[2];
				#pragma unroll
				for (int i = 0; i < 2 * NP.value; i++) a[i] = As[wm * 32 + i * 8 + (lane >> 2)][kk + (lane & 3)];
				#pragma unroll
				for (int j = 0; j < NJ.value; j++)
					b[j] = Bs[kk + (lane & 3)][(wn * 16 + j * 8 + (lane >> 2)) ^ (2 * ((kk >> 2) & 3))];
				#pragma unroll
				for (int j = 0; j < NJ.value; j++)
					#pragma unroll
					for (int i = 0; i < 2 * NP.value; i += 2) dmma16(acc[i][j], acc[i + 1][j], a[i], a[i + 1], b[j]);
			}
		};
		using N1 = std::integral_constant<int, 1>;
		using N2 = std::integral_constant<int, 2>;
		if (ki1 > 2) {
			if (cj1 == 2) mma_chunk(N2{}, N2{});
			else if (cj1 == 1) mma_chunk(N2{}, N1{});
		} else if (ki1 > 0) {
			if (cj1 == 2) mma_chunk(N1{}, N2{});
			else if (cj1 == 1) mma_chunk(N1{}, N1{});
		}
		__syncthreads();
	}
	double* qrow = p.qq + (long)p.mt.koff[im] * p.ncol;
	#pragma unroll
	for (int i = 0; i < 4; i++) {
		const int k = k0 + wm * 32 + i * 8 + (lane >> 2);
		if (k >= nk) continue;
		#pragma unroll
		for (int j = 0; j < 2; j++) {
			const int col = c0 + wn * 16 + j * 8 + (lane & 3) * 2;
			if (col < p.ncol)
				*reinterpret_cast<double2*>(qrow + (long)k * p.ncol + col) = make_double2(acc[i][j][0], acc[i][j][1]);
		}
	}
}

} // namespace
