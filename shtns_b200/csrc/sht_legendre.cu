// Legendre stage of the spherical-harmonic transforms on sm_100a.
//
// Per azimuthal order m the Legendre sum is a real matrix product with an
// on-the-fly left operand:
//   synthesis  E/O[theta, col] = sum_k Y_k(theta) * qq[k, col]
//   analysis   qq[k, col]      = sum_theta Y_k(theta) * G[theta, col]
// where Y_k(theta) = sin^m(theta) * p_k(cos^2 theta) follows Ishioka's two-term
// recurrence Y_{k+1} = (c_{2k+1} x^2 + c_{2k}) Y_k + Y_{k-1} (the reference's
// SHT/kernel_SH_to_spat.gen.c:388-409 and kernel_spat_to_SH.gen.c:541-598),
// `col` runs over field-components x {even, odd} x {re, im}, and the even
// and odd degrees share Y_k (the odd part is multiplied by cos(theta) when the
// hemispheres are folded, kernel_SH_to_spat.gen.c:429-441).
//
// The product runs on the FP64 tensor cores (mma.sync m16n8k4 f64: tcgen05 has
// no FP64 kind).  Each CTA regenerates its Y tile in shared memory from
// recurrence checkpoints (Y_k, Y_{k+1}) stored every 8, 16 or 32 steps k, so
// tiles can start at any k and a thread's part of the recurrence is as short
// as one segment (leg_spaced picks the segments of a launch).
#include "sht_internal.h"
#include "sht_legendre_tiles.h"

#include <algorithm>
#include <type_traits>

namespace {

// ---------------------------------------------------------------------------
// Checkpoints: thread (t, im) runs the recurrence of order m at north row t and
// stores (Y_{seg*s}, Y_{seg*s+1}) for every segment s (seg = 8, 16 or 32).
// Y_0 = sin^m(theta) (sint_pow_n_ext, sht_legendre.c:110-139) and
// Y_1 = (c_1 x^2 + c_0) Y_0 (kernel_SH_to_spat.gen.c:303-315).
// Extended exponent: above degree ~1800, sin^m(theta) falls below the double
// range at latitudes where Y_k later grows to O(1).  The seed is formed as a
// mantissa times 2^E by binary powering with frexp normalisation, and the
// recurrence runs on scaled values y * 2^E (it is linear and homogeneous, so
// scaling by a power of two is exact) until the values have grown enough for
// E to be folded back to 0.  Each checkpoint stores y * 2^E as a plain double:
// a checkpoint that underflows is below 2^-1022 and stays below ~1e-280 over
// the next 32 steps, far under any threshold.  The reference keeps the same
// kind of scaled seed (sint_pow_n_ext, sht_legendre.c:109-139) and rescales
// its recurrence when values become significant (sht_legendre.c:159-187,
// sht_func.c:200-233).
#define CK_FOLD 600          // fold E into the values when E >= -CK_FOLD
#define CK_BIG 0x1p500       // rescale scaled values above this magnitude
__global__ void ck_kernel(int nlat_2, int mres, int seg, const double* __restrict__ x2g, const double* __restrict__ sing,
                          const double* __restrict__ c, MTables mt, const int* __restrict__ nseg, double2* __restrict__ ck)
{
	const int t = blockIdx.x * blockDim.x + threadIdx.x;
	const int im = blockIdx.y;
	if (t >= nlat_2) return;
	const int m = im * mres;
	const double x2 = x2g[t];
	// sin^m = y0 * 2^E, y0 in [0.5, 1)
	double y0 = 1.0;
	int E = 0;
	{
		int be, te;
		double b = frexp(sing[t], &be);
		for (int n = m; n; n >>= 1) {
			if (n & 1) { y0 = frexp(y0 * b, &te); E += be + te; }
			b = frexp(b * b, &te); be = 2 * be + te;
		}
	}
	if (E >= -CK_FOLD) { y0 = ldexp(y0, E); E = 0; }
	const double* cc = c + mt.coff[im];
	double y1 = fma(cc[1], x2, cc[0]) * y0;
	const int ns = nseg[im];
	double2* out = ck + (long)mt.ckoff[im] * nlat_2 + t;
	for (int s = 0; s < ns; s++) {
		out[(long)s * nlat_2] = E ? make_double2(ldexp(y0, E), ldexp(y1, E)) : make_double2(y0, y1);
		const int kb = s * seg + 1;
		for (int j = 0; j < seg; j++) {
			const int k = kb + j;
			const double a = fma(cc[2 * k + 1], x2, cc[2 * k]);
			const double y2 = fma(a, y1, y0);
			y0 = y1;
			y1 = y2;
			if (E && fabs(y1) > CK_BIG) {
				if (E >= -CK_FOLD) { y0 = ldexp(y0, E); y1 = ldexp(y1, E); E = 0; }
				else { y0 *= 0x1p-500; y1 *= 0x1p-500; E += 500; }
			}
		}
	}
}

// ---------------------------------------------------------------------------
// Synthesis prologue: spectral coefficients -> Ishioka basis, k-major layout.
//   even: qe_k = X0_k Q_{m+2k} + X1_k Q_{m+2k+2};  odd: qo_k = X2_k Q_{m+2k+1}
// (SH_to_ishioka, sht_private.h:442-483).  Vector components first form
//   V_l =  (st d/dth S)_l + i m T_l,  W_l = -(st d/dth T)_l + i m S_l
// for l = m..llim+1 (SH_vect_to_2scal, sht_private.h:534-584).
// Column layout: field-component fc owns columns 16*(fc/4) + 2*(fc%4) + {0,1}
// (even re, im) and the same +8 (odd re, im).
//
// CTA = (order im, PT_K = pt_items / PF Ishioka rows k, PF fields, group): the
// first group is the scalar component, the other one the vector pair.  The
// degree window [2 k0 - 1, 2 k0 + 2 PT_K + 2] of Q, or of S and T, is staged in
// shared memory with coalesced loads; then each thread forms the rows of one
// (k, field), for the vector pair V and W together from the same five degrees
// of S and T.  PF is the power of two up to 16 that the call's fields fill best
// (launch_prep_synth): with 16 for every call, one qst field at lmax 1023 kept 3
// of 16 lanes and took 68 us instead of 35 (8 scalar fields at lmax 4095: 684
// instead of 452).  Bound: instruction issue and the shared-memory path.  With V
// and W as field-components of their own, S and T were staged twice and read
// 18 instead of 10 times per pair (64 qst fields
// at lmax 511: 241 us, here 195; 32 vector fields at lmax 255: 33, here 28).
__host__ __device__ constexpr int pt_items(int PF) { return PF <= 2 ? 256 : 512; }     // (row, field) items of a CTA

// C: coefficient type, double2, or float2 for the single-precision transforms.
// VECTOR: the call has a vector pair (and perhaps a scalar component).
template <int PF, class C, bool VECTOR>
__global__ void __launch_bounds__(256, VECTOR ? 4 : 6) prep_synth_kernel(PrepParams p)
{
	constexpr int PT_F = PF, PT_K = pt_items(PF) / PF;
	constexpr int PT_W = 2 * PT_K + 5;       // window length, odd stride in 16-byte units
	constexpr int NA = VECTOR ? 2 : 1;       // arrays staged
	__shared__ double2 win[NA][PT_F][PT_W];
	__shared__ double cfs[NA][PT_W];         // sin d/dtheta coupling (lo, hi) of the window's degrees
	__shared__ double xk[3 * PT_K];          // basis change X of the CTA's k rows
	const int im = p.im0 + blockIdx.z;
	if (im > p.mlim) return;
	const int m = im * p.mres;
	const int kmax = (p.llim + 1 - m) / 2 + 1;
	const int k0 = blockIdx.x * PT_K;
	if (k0 >= kmax) return;
	const bool has_q = p.comp_type[0] == 0;
	const int nft = (p.nf + PT_F - 1) / PT_F;
	const int grp = blockIdx.y / nft;
	const int f0 = (blockIdx.y - grp * nft) * PT_F;
	const bool vec = VECTOR && !(has_q && grp == 0);
	const bool m0 = (m == 0);
	const int lrel_max = p.llim - m;
	const long off = (long)im * (2 * p.lmax + 2 - (im + 1) * p.mres) / 2 + m;   // LM(m, m)
	const int d0 = 2 * k0 - 1;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int voff = p.mt.voff[im];
	if (vec)
		for (int i = tid; i < PT_W; i += 256) {
			const int d = d0 + i;
			cfs[0][i] = (d > 0 && d <= lrel_max + 1) ? p.stdt_lo[voff + d] : 0.0;
			cfs[NA - 1][i] = (d >= 0 && d <= lrel_max + 1) ? p.stdt_hi[voff + d] : 0.0;
		}
	for (int e = tid; e < 3 * PT_K; e += 256) xk[e] = (k0 + e / 3 <= kmax) ? p.xs[p.mt.xoff[im] + 3 * k0 + e] : 0.0;
	// window of the degrees of each (array, field) pair (array = pair / PF, the
	// second one for vectors only), lanes along the degrees: WP warps share a
	// pair or a warp takes PW of them, QB pairs and up to UB loads of each before
	// the first store
	constexpr int NP = NA * PF, WP = (NP >= 8) ? 1 : 8 / NP, PW = (NP >= 8) ? NP / 8 : 1;
	constexpr int NI = (PT_W + 32 * WP - 1) / (32 * WP);
	constexpr int QB = (PW >= 2 && NI <= 3) ? 2 : 1, UB = (NI <= 5) ? NI : (NI + 1) / 2;
	const int q0 = (WP == 1) ? warp : warp / WP, i0 = lane + 32 * (warp % WP);
	#pragma unroll
	for (int h = 0; h < PW; h += QB) {
		const C* base[QB];
		#pragma unroll
		for (int qi = 0; qi < QB; qi++) {
			const int q = q0 + 8 * (h + qi), a = q / PT_F, f = f0 + q % PT_F;
			const double2* x = vec ? (a == 0 ? p.S : p.T) : (a == 0 ? p.Q : nullptr);
			base[qi] = (x && f < p.nf) ? reinterpret_cast<const C*>(x) + off + (long)f * p.spec_dist + d0 : nullptr;
		}
		#pragma unroll
		for (int u0 = 0; u0 < NI; u0 += UB) {
			double2 v[QB][UB];
			#pragma unroll
			for (int qi = 0; qi < QB; qi++)
				#pragma unroll
				for (int u = 0; u < UB; u++) {
					const int i = i0 + 32 * WP * (u0 + u), d = d0 + i;
					v[qi][u] = make_double2(0.0, 0.0);
					if (u0 + u < NI && base[qi] && i < PT_W && d >= 0 && d <= lrel_max) {
						const C x = base[qi][i];
						v[qi][u] = make_double2(x.x, m0 ? 0.0 : x.y);
					}
				}
			#pragma unroll
			for (int qi = 0; qi < QB; qi++) {
				const int q = q0 + 8 * (h + qi), a = q / PT_F, fl = q % PT_F;
				if (VECTOR && a != 0 && !vec) continue;
				#pragma unroll
				for (int u = 0; u < UB; u++) {
					const int i = i0 + 32 * WP * (u0 + u);
					if (u0 + u < NI && i < PT_W) win[a][fl][i] = v[qi][u];
				}
			}
		}
	}
	__syncthreads();
	const double em = (p.msign < 0) ? -(double) m : (double) m;   // signed m (negative orders of the _ml transforms)
	const long row0 = p.mt.koff[im];
	// even and odd parts of field-component fc at row k from its degrees 2k .. 2k + 2
	auto put = [&](int k, int fc, const double* x, double2 a, double2 b, double2 c) {
		double* row = p.qq + (row0 + k) * p.ncol + 16 * (fc >> 2) + 2 * (fc & 3);
		*reinterpret_cast<double2*>(row) = make_double2(fma(x[0], a.x, x[1] * c.x), fma(x[0], a.y, x[1] * c.y));
		*reinterpret_cast<double2*>(row + 8) = make_double2(x[2] * b.x, x[2] * b.y);
	};
	for (int e = tid; e < PT_K * PT_F; e += 256) {
		const int kl = e / PT_F, fl = e - kl * PT_F;
		const int k = k0 + kl, f = f0 + fl;
		if (k >= kmax || f >= p.nf) continue;
		const int w0 = 2 * kl;                     // window index of degree 2k - 1
		const double* x = xk + 3 * kl;
		if (!vec) {
			put(k, f, x, win[0][fl][w0 + 1], win[0][fl][w0 + 2], win[0][fl][w0 + 3]);
			continue;
		}
		// V = stdt S + i m T, W = -stdt T + i m S: the coupled array at degrees
		// d -/+ 1, the other one at d (zero beyond lrel_max + 1, where the
		// coupling is zero and so are S and T).  Fields from neg_from on carry the
		// order -m (complex-field transforms)
		const double emf = (p.neg_from > 0 && f >= p.neg_from) ? -em : em;
		double2 s[5], t[5];
		#pragma unroll
		for (int r = 0; r < 5; r++) { s[r] = win[0][fl][w0 + r]; t[r] = win[NA - 1][fl][w0 + r]; }
		double2 v[3], w[3];
		#pragma unroll
		for (int r = 0; r < 3; r++) {
			const double lo = cfs[0][w0 + 1 + r], hi = cfs[NA - 1][w0 + 1 + r];
			v[r] = make_double2(lo * s[r].x + hi * s[r + 2].x - emf * t[r + 1].y, lo * s[r].y + hi * s[r + 2].y + emf * t[r + 1].x);
			w[r] = make_double2(-(lo * t[r].x + hi * t[r + 2].x) - emf * s[r + 1].y, -(lo * t[r].y + hi * t[r + 2].y) + emf * s[r + 1].x);
		}
		const int fv = (has_q ? p.nf : 0) + f;
		put(k, fv, x, v[0], v[1], v[2]);
		put(k, fv + p.nf, x, w[0], w[1], w[2]);
	}
}

// ---------------------------------------------------------------------------
// Analysis epilogue: Ishioka basis -> spectral coefficients
//   Q_{m+2k} = X0_k e_k + X1_{k-1} e_{k-1},  Q_{m+2k+1} = X2_k o_k
// (ishioka_to_SH, sht_private.h:345-374), and for vectors
//   S_l = -((MX V)_l + i m W_l) / (l(l+1)),  T_l = -(i m V_l - (MX W)_l) / (l(l+1))
// with MX = 2 cos + sin d/dtheta (SH_2scal_to_vect, sht_private.h:296-337).
// Degrees above llim and orders above mlim are written as zero (SHT_VAR_LTR).
//
// CTA = (order im, PE_J degrees, PF fields, output group): the k rows covering
// the degree tile plus one row of halo on each side are staged in shared
// memory for the (one or two) field-components of the group.  PF (1, 4, 8 or
// 16) is what the call's fields fill best; with 16 for every call, one qst
// field at lmax 1023 took 118 us instead of 35 (8 scalar fields at lmax 4095:
// 831 instead of 523).
template <int PF>
struct PostTile {
	static constexpr int J = (PF == 1) ? 512 : (PF == 4) ? 128 : 1024 / PF;   // degrees
	static constexpr int R = J / 2 + 4;                     // staged k rows: j0/2-2 .. j0/2+J/2+1
	static constexpr int S = 2 * PF + 1;                    // row stride in double2: odd, so the 8 rows read by 8 lanes use distinct banks
};

// Staged rows: [row][2 fl] = even pair (re, im) of field fl, [2 fl + 1] = odd
// pair, row = k - kb; Xs[3 row + c] = basis-change coefficients of k (both zero
// outside the order).  Degree 2k, and degree 2k + 1:
template <int PE_S>
__device__ __forceinline__ double2 ish_even(const double2 (*E)[PE_S], const double* Xs, int r, int fl)
{
	const double2 e = E[r][2 * fl], e1 = E[r - 1][2 * fl];
	const double x = Xs[3 * r], x1 = Xs[3 * (r - 1) + 1];
	return make_double2(fma(x1, e1.x, x * e.x), fma(x1, e1.y, x * e.y));
}
template <int PE_S>
__device__ __forceinline__ double2 ish_odd(const double2 (*E)[PE_S], const double* Xs, int r, int fl)
{
	const double2 o = E[r][2 * fl + 1];
	const double x = Xs[3 * r + 2];
	return make_double2(x * o.x, x * o.y);
}

template <int PF, class C>
__global__ void __launch_bounds__(256, 4) post_analys_kernel(PrepParams p)
{
	constexpr int PE_F = PF, PE_J = PostTile<PF>::J, PE_R = PostTile<PF>::R, PE_S = PostTile<PF>::S;
	constexpr int NE = PE_R * PE_F * 2, NU = (NE + 255) / 256;
	__shared__ double2 sv[PE_R][PE_S];     // first component of the group (Q, or V)
	__shared__ double2 sw[PE_R][PE_S];     // second component (W) for the vector group
	__shared__ double xs[3 * PE_R];
	const int im = p.im0 + blockIdx.z;
	const int m = im * p.mres;
	const int nl = p.lmax - m + 1;
	const int j0 = blockIdx.x * PE_J;
	if (j0 >= nl) return;
	const bool has_q = (p.comp_type[0] == 0);
	const int nft = (p.nf + PE_F - 1) / PE_F;
	const int g = blockIdx.y / nft;                       // 0: first group, 1: second group
	const int f0 = (blockIdx.y - g * nft) * PE_F;
	const bool scalar_group = has_q && g == 0;
	const bool zero_m = (im > p.mlim);
	const long off = (long)im * (2 * p.lmax + 2 - (im + 1) * p.mres) / 2 + m;
	const int kb = j0 / 2 - 2;
	const int nk = (p.llim + ((p.comp_type[0] | p.comp_type[1] | p.comp_type[2]) ? 1 : 0) - m) / 2 + 1;
	if (!zero_m) {
		const int cv = scalar_group ? 0 : (has_q ? 1 : 0);
		const long r0 = p.mt.koff[im];
		// all row loads of a thread are issued before the first is stored
		double2 v[NU], w[NU];
		#pragma unroll
		for (int u = 0; u < NU; u++) {
			const int e = threadIdx.x + 256 * u;
			const int r = e / (PE_F * 2), rem = e - r * PE_F * 2;
			const int fl = rem >> 1, eo = rem & 1;
			const int k = kb + r, f = f0 + fl;
			v[u] = make_double2(0.0, 0.0);
			w[u] = make_double2(0.0, 0.0);
			if (e < NE && k >= 0 && k < nk && f < p.nf) {
				const double* row = p.qq + (r0 + k) * p.ncol;
				const int fcv = cv * p.nf + f;
				v[u] = *reinterpret_cast<const double2*>(row + 16 * (fcv >> 2) + 2 * (fcv & 3) + 8 * eo);
				if (!scalar_group) {
					const int fcw = (cv + 1) * p.nf + f;
					w[u] = *reinterpret_cast<const double2*>(row + 16 * (fcw >> 2) + 2 * (fcw & 3) + 8 * eo);
				}
			}
		}
		// basis-change coefficients of the staged rows (3 (kmax + 1) entries per order)
		const int kx = (p.lmax + 1 - m) / 2 + 1;
		const double* X = p.xa + p.mt.xoff[im];
		for (int e = threadIdx.x; e < 3 * PE_R; e += blockDim.x) {
			const int k = kb + e / 3;
			xs[e] = (k >= 0 && k <= kx) ? X[3 * kb + e] : 0.0;
		}
		#pragma unroll
		for (int u = 0; u < NU; u++) {
			const int e = threadIdx.x + 256 * u;
			if (e < NE) {
				const int r = e / (PE_F * 2), c = e - r * PE_F * 2;
				sv[r][c] = v[u];
				sw[r][c] = w[u];
			}
		}
	}
	// vector coupling (lo, hi) of degrees j0 - 1 .. j0 + PE_J and 1 / (l (l + 1))
	// of the tile's degrees, shared by its fields
	__shared__ double vlo[PE_J + 2], vhi[PE_J + 2], vl2[PE_J];
	const int voff = p.mt.voff[im];
	if (!scalar_group) {
		for (int e = threadIdx.x; e < PE_J + 2; e += blockDim.x) {
			const int j = j0 - 1 + e;
			vlo[e] = (j > 0 && j < nl) ? p.van_lo[voff + j] : 0.0;
			vhi[e] = (j >= 0 && j < nl) ? p.van_hi[voff + j] : 0.0;
			if (e < PE_J) vl2[e] = (j0 + e < nl) ? p.l2[m + j0 + e] : 0.0;
		}
	}
	__syncthreads();
	const double em = (p.msign < 0) ? -(double) m : (double) m;   // signed m (negative orders of the _ml transforms)
	auto store = [&](double2* to, long at, double2 v) {
		C x;
		x.x = v.x; x.y = v.y;
		reinterpret_cast<C*>(to)[at] = x;
	};
	// an item is a pair of degrees (2k, 2k + 1) of one field, 32 consecutive k to
	// a warp: the four degrees 2k - 1 .. 2k + 2 that its vector formulas need come
	// from five staged values per array (one degree per item read twice as much of
	// the shared-memory path: 64 qst fields at lmax 511 206 us, here 183; 32 scalar
	// fields at lmax 1023 140, here 132; 32 vector fields at lmax 255 27, here 23)
	for (int e = threadIdx.x; e < PE_J / 2 * PE_F; e += blockDim.x) {
		const int fl = e / (PE_J / 2), i = e - fl * (PE_J / 2), r = i + 2;
		const int j = j0 + 2 * i, f = f0 + fl;
		if (j >= nl || f >= p.nf) continue;
		const bool two = j + 1 < nl;
		const bool z0 = zero_m || m + j > p.llim, z1 = zero_m || m + j + 1 > p.llim;
		const long o = off + (long)f * p.spec_dist + j;
		double2 s0 = make_double2(0.0, 0.0), s1 = s0, t0 = s0, t1 = s0;
		if (scalar_group) {
			if (!z0) {
				s0 = ish_even(sv, xs, r, fl);
				if (m == 0) s0.y = 0.0;
			}
			if (!z1) {
				s1 = ish_odd(sv, xs, r, fl);
				if (m == 0) s1.y = 0.0;
			}
			store(p.Qo, o, s0);
			if (two) store(p.Qo, o + 1, s1);
			continue;
		}
		if (!z0) {
			const double emf = (p.neg_from > 0 && f >= p.neg_from) ? -em : em;   // order -m fields
			const double2 v[4] = {ish_odd(sv, xs, r - 1, fl), ish_even(sv, xs, r, fl), ish_odd(sv, xs, r, fl), ish_even(sv, xs, r + 1, fl)};
			const double2 w[4] = {ish_odd(sw, xs, r - 1, fl), ish_even(sw, xs, r, fl), ish_odd(sw, xs, r, fl), ish_even(sw, xs, r + 1, fl)};
			#pragma unroll
			for (int h = 0; h < 2; h++) {
				const double lo = vlo[2 * i + h + 1], hi = vhi[2 * i + h + 1], l2 = vl2[2 * i + h];
				const double2 v0 = v[h + 1], w0 = w[h + 1];
				const double mxv_r = lo * v[h].x + hi * v[h + 2].x, mxv_i = lo * v[h].y + hi * v[h + 2].y;
				const double mxw_r = lo * w[h].x + hi * w[h + 2].x, mxw_i = lo * w[h].y + hi * w[h + 2].y;
				double2 a = make_double2(-(mxv_r - emf * w0.y) * l2, -(mxv_i + emf * w0.x) * l2);
				double2 b = make_double2(-(-emf * v0.y - mxw_r) * l2, -(emf * v0.x - mxw_i) * l2);
				if (m == 0) { a.y = 0.0; b.y = 0.0; }
				if (h == 0) { s0 = a; t0 = b; }
				else if (!z1) { s1 = a; t1 = b; }
			}
		}
		store(p.So, o, s0);
		store(p.To, o, t0);
		if (two) { store(p.So, o + 1, s1); store(p.To, o + 1, t1); }
	}
}

// Single-plan kernels: blockIdx.y = order - p.im0, blockIdx.x = (row tile, column tile).
template <int SEG, int WM, bool RB>
__global__ void __launch_bounds__(LG_THREADS, WM == 1 ? 2 : 3) leg_synth_kernel(LegParams p)
{
	const int ntb = (p.nlat_2 + 32 * WM - 1) / (32 * WM);
	leg_synth_tile<SEG, WM, RB>(p, p.im0 + blockIdx.y, blockIdx.x % ntb, blockIdx.x / ntb);
}

template <int SEG, int WM, bool RB>
__global__ void __launch_bounds__(LG_THREADS, WM == 1 ? 2 : 3) leg_analys_kernel(LegParams p, int nkb)
{
	leg_analys_tile<SEG, WM, RB>(p, p.im0 + blockIdx.y, blockIdx.x % nkb, blockIdx.x / nkb);
}

// Persistent multi-plan kernels: CTAs (one wave) take work items (plan,
// order, row or k tile, column tile) from a queue in decreasing cost order,
// so plans of different lmax share one launch and balance over the SMs.
template <int SEG, bool SYNTH>
__global__ void __launch_bounds__(LG_THREADS, 3)
leg_multi_kernel(const LegParams* __restrict__ plist, const int4* __restrict__ work, int nwork, int* __restrict__ counter)
{
	__shared__ int wi;
	for (;;) {
		if (threadIdx.x == 0) wi = atomicAdd(counter, 1);
		__syncthreads();
		const int w = wi;
		__syncthreads();
		if (w >= nwork) break;
		const int4 it = work[w];
		if (SYNTH) leg_synth_tile<SEG, 2>(plist[it.x], it.y, it.z, it.w);
		else leg_analys_tile<SEG, 2>(plist[it.x], it.y, it.z, it.w);
	}
}

} // namespace

// ---------------------------------------------------------------------------
void launch_checkpoints(shtns_cfg s, cudaStream_t st)
{
	std::vector<int> nseg(s->mmax + 1);
	for (int im = 0; im <= s->mmax; im++) nseg[im] = (s->kmax_h[im] + s->ckseg - 1) / s->ckseg;
	int* d_nseg = nullptr;
	if (!shtb_cuda_ok(cudaMalloc(&d_nseg, sizeof(int) * nseg.size()), "checkpoint table")) return;
	cudaMemcpyAsync(d_nseg, nseg.data(), sizeof(int) * nseg.size(), cudaMemcpyHostToDevice, st);
	dim3 grid((s->nlat_2 + 127) / 128, s->mmax + 1);
	ck_kernel<<<grid, 128, 0, st>>>(s->nlat_2, s->mres, s->ckseg, s->d_x2, s->d_s, s->d_c, s->mt, d_nseg, s->d_ck);
	shtb_count_launch();
	shtb_cuda_ok(cudaGetLastError(), "checkpoint kernel");
	cudaStreamSynchronize(st);
	cudaFree(d_nseg);
}

// Fields per CTA of the prologue and epilogue kernels: 1 or 2 for so many, else
// 16, 8 or 4 (fewer split the 64-byte groups of four field-components).  A call
// whose CTAs of 4 fields are at most two per SM takes those: the less a CTA has
// to do the sooner the call ends (12 vector fields at lmax 63: prologue 9.0
// and epilogue 8.7 us, with 16 fields a CTA 12.0 and 10.6).  Beyond, whichever
// leaves the fewest items idle: the fields round up to the tile, and the rows of an order by half a
// tile of rows(f) on average.  (By the fields alone 156 vector fields took 4 at
// a time and 128 rows, of which lmax 63 has 33: 22 / 20 us, here 17 / 15.)
template <class Rows>
static int tile_fields(const PrepParams& p, int lmax, int mmax, int groups, Rows rows)
{
	if (p.nf <= 2) return p.nf;
	const int rows2 = lmax + 3 - (p.im0 + mmax) * p.mres / 2;     // twice the mean rows of an order
	const long ctas4 = (long) ((p.nf + 3) / 4) * groups * (mmax + 1 - p.im0) * (((lmax - p.im0 * p.mres) / 2 + rows(4)) / rows(4));
	if (ctas4 <= 2 * 148) return 4;
	int best = 0;
	long least = 0;
	for (int f = 16; f >= 4; f /= 2) {
		const long items = (long) ((p.nf + f - 1) / f * f) * (rows2 + rows(f));
		if (!best || items < least) { best = f; least = items; }
	}
	return best;
}

void launch_prep_synth(const PrepParams& p, cudaStream_t st)
{
	const int ngroups = (p.comp_type[0] == 0) ? 1 + (p.ncomp > 1 ? 1 : 0) : 1;
	const int kmax0 = (p.llim + 1) / 2 + 1;
	auto go = [&](auto kern, int PF) {
		const int K = pt_items(PF) / PF;
		dim3 grid((kmax0 + K - 1) / K, (p.nf + PF - 1) / PF * ngroups, p.mlim + 1 - p.im0);
		kern<<<grid, 256, 0, st>>>(p);
	};
	const int pf = tile_fields(p, p.llim, p.mlim, ngroups, [](int f) { return pt_items(f) / f; });
	auto pick = [&](auto c, auto VC) {
		using C = decltype(c);
		constexpr bool V = decltype(VC)::value;
		switch (pf) {
			case 1: go(prep_synth_kernel<1, C, V>, 1); break;
			case 2: go(prep_synth_kernel<2, C, V>, 2); break;
			case 4: go(prep_synth_kernel<4, C, V>, 4); break;
			case 8: go(prep_synth_kernel<8, C, V>, 8); break;
			default: go(prep_synth_kernel<16, C, V>, 16); break;
		}
	};
	const bool vector = ngroups > 1 || p.comp_type[0] != 0;
	if (p.f32) pick(float2{}, std::false_type{});      // single-precision transforms are scalar
	else if (vector) pick(double2{}, std::true_type{});
	else pick(double2{}, std::false_type{});
	shtb_count_launch();
}

namespace {

template <int WM>
void launch_leg_synth_wm(const LegParams& p, cudaStream_t st)
{
	constexpr int BM = 32 * WM, BN = 16 * (8 / WM);
	const int ntb = (p.nlat_2 + BM - 1) / BM;
	const int nnb = (p.ncol + BN - 1) / BN;
	dim3 grid(ntb * nnb, p.mlim + 1 - p.im0);
	switch (p.ckseg) {
		case 8: if (p.rb.n) leg_synth_kernel<8, WM, true><<<grid, LG_THREADS, 0, st>>>(p);
		        else leg_synth_kernel<8, WM, false><<<grid, LG_THREADS, 0, st>>>(p); break;
		case 16: if (p.rb.n) leg_synth_kernel<16, WM, true><<<grid, LG_THREADS, 0, st>>>(p);
		         else leg_synth_kernel<16, WM, false><<<grid, LG_THREADS, 0, st>>>(p); break;
		default: if (p.rb.n) leg_synth_kernel<32, WM, true><<<grid, LG_THREADS, 0, st>>>(p);
		         else leg_synth_kernel<32, WM, false><<<grid, LG_THREADS, 0, st>>>(p); break;
	}
}

template <int WM>
void launch_leg_analys_wm(const LegParams& p, int kmax_all, cudaStream_t st)
{
	constexpr int BM = 32 * WM, BN = 16 * (8 / WM);
	const int nkb = (kmax_all + BM - 1) / BM;
	const int nnb = (p.ncol + BN - 1) / BN;
	dim3 grid(nkb * nnb, p.mlim + 1 - p.im0);
	switch (p.ckseg) {
		case 8: if (p.rb.n) leg_analys_kernel<8, WM, true><<<grid, LG_THREADS, 0, st>>>(p, nkb);
		        else leg_analys_kernel<8, WM, false><<<grid, LG_THREADS, 0, st>>>(p, nkb); break;
		case 16: if (p.rb.n) leg_analys_kernel<16, WM, true><<<grid, LG_THREADS, 0, st>>>(p, nkb);
		         else leg_analys_kernel<16, WM, false><<<grid, LG_THREADS, 0, st>>>(p, nkb); break;
		default: if (p.rb.n) leg_analys_kernel<32, WM, true><<<grid, LG_THREADS, 0, st>>>(p, nkb);
		         else leg_analys_kernel<32, WM, false><<<grid, LG_THREADS, 0, st>>>(p, nkb); break;
	}
}

} // namespace

// Tile shape (p.tile_wm, warps along the rows): 1 = 32 x 128, 2 = 64 x 64,
// 4 = 128 x 32, 5 = 128 x 16.  Automatic (0): wide calls 64 x 64; calls with at
// most 32 GEMM columns (8 field-components) 128 x 32, which leaves no column
// padding; with at most 16 columns 128 x 16, except for the analysis on small
// grids, where its four warps leave too few in flight (lmax 127, 3 components:
// 14.8 against 12.7 us; lmax 340, 4: 37 against 35; lmax 511, 4: 56 against 72).
static int tile_wm(const LegParams& p, bool synth)
{
	if (p.tile_wm == 1 || p.tile_wm == 2 || p.tile_wm == 4) return p.tile_wm;
	if (p.ncol > 32) return 2;
	if (p.ncol > 16) return 4;
	return (synth || p.nlat_2 > 256) ? 5 : 4;
}

// Segments of at least `want` steps from a table of denser checkpoints: the
// recurrence reaches the values of the checkpoints it passes over exactly.
LegParams leg_spaced(const LegParams& p, int want)
{
	LegParams q = p;
	while (q.ckseg < want) { q.ckseg *= 2; q.ckrow *= 2; }
	return q;
}

// 64 x 64 tiles: 8 steps per segment, so that every thread generates one of the
// shortest chains (lmax 1023, 32 fields, synthesis / analysis: 8: 1553/1655 us, 16:
// 1671/1707).  128 rows: 16 steps keep every thread busy too and read half of
// the checkpoints (lmax 511, 8 fields: 8: 83/91 us, 16: 78/84; lmax 1023, 8 fields:
// 8: 491/454, 16: 468/451, 32: 541/491; lmax 2047: 3.48/3.25 ms, 3.35/3.21,
// 3.81/3.42).
static int tile_spacing(int wm) { return wm == 2 ? 8 : 16; }

void launch_leg_synth(const LegParams& p0, cudaStream_t st)
{
	if (leg_simt_selected(p0, true)) { launch_leg_synth_simt(p0, st); shtb_count_launch(); return; }
	const LegParams p = leg_spaced(p0, tile_spacing(tile_wm(p0, true)));
	switch (tile_wm(p, true)) {
		case 1: launch_leg_synth_wm<1>(p, st); break;
		case 4: launch_leg_synth_wm<4>(p, st); break;
		case 5: launch_leg_synth_narrow(p, st); break;
		default: launch_leg_synth_wm<2>(p, st); break;
	}
	shtb_count_launch();
}

void launch_leg_analys(const LegParams& p0, int kmax_all, cudaStream_t st)
{
	if (leg_simt_selected(p0, false)) { launch_leg_analys_simt(p0, kmax_all, st); shtb_count_launch(); return; }
	const LegParams p = leg_spaced(p0, tile_spacing(tile_wm(p0, false)));
	switch (tile_wm(p, false)) {
		case 1: launch_leg_analys_wm<1>(p, kmax_all, st); break;
		case 4: launch_leg_analys_wm<4>(p, kmax_all, st); break;
		case 5: launch_leg_analys_narrow(p, kmax_all, st); break;
		default: launch_leg_analys_wm<2>(p, kmax_all, st); break;
	}
	shtb_count_launch();
}

void launch_post_analys_m(const PrepParams& p, int mmax, cudaStream_t st)
{
	const int ngroups = (p.comp_type[0] == 0) ? 1 + (p.ncomp > 1 ? 1 : 0) : 1;
	auto go = [&](auto kern, int PF, int J) {
		dim3 grid((p.lmax + J) / J, (p.nf + PF - 1) / PF * ngroups, mmax + 1 - p.im0);
		kern<<<grid, 256, 0, st>>>(p);
	};
	const int pf = tile_fields(p, p.lmax, mmax, ngroups, [](int f) { return f == 16 ? PostTile<16>::J / 2 : f == 8 ? PostTile<8>::J / 2 : PostTile<4>::J / 2; });
	auto pick = [&](auto c) {
		using C = decltype(c);
		switch (pf) {
			case 1: go(post_analys_kernel<1, C>, 1, PostTile<1>::J); break;
			case 2: case 4: go(post_analys_kernel<4, C>, 4, PostTile<4>::J); break;
			case 8: go(post_analys_kernel<8, C>, 8, PostTile<8>::J); break;
			default: go(post_analys_kernel<16, C>, 16, PostTile<16>::J); break;
		}
	};
	if (p.f32) pick(float2{});
	else pick(double2{});
	shtb_count_launch();
}

void launch_leg_multi(const LegParams* d_plist, const int4* d_work, int nwork, int* d_counter, int ckseg, bool synth,
                      int nctas, cudaStream_t st)
{
	const int grid = std::max(1, std::min(nwork, nctas));
	cudaMemsetAsync(d_counter, 0, sizeof(int), st);
	switch (ckseg) {
		case 8:
			if (synth) leg_multi_kernel<8, true><<<grid, LG_THREADS, 0, st>>>(d_plist, d_work, nwork, d_counter);
			else leg_multi_kernel<8, false><<<grid, LG_THREADS, 0, st>>>(d_plist, d_work, nwork, d_counter);
			break;
		case 16:
			if (synth) leg_multi_kernel<16, true><<<grid, LG_THREADS, 0, st>>>(d_plist, d_work, nwork, d_counter);
			else leg_multi_kernel<16, false><<<grid, LG_THREADS, 0, st>>>(d_plist, d_work, nwork, d_counter);
			break;
		default:
			if (synth) leg_multi_kernel<32, true><<<grid, LG_THREADS, 0, st>>>(d_plist, d_work, nwork, d_counter);
			else leg_multi_kernel<32, false><<<grid, LG_THREADS, 0, st>>>(d_plist, d_work, nwork, d_counter);
			break;
	}
	shtb_count_launch();
}
