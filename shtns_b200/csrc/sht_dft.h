// Short DFTs in registers, shared by the FFT kernels (sht_fft.cu, sht_fft_gen.cu).
// Dft<R>::run(u, s): u[k] <- sum_q u[q] exp(s 2 pi i q k / R), s = +1 or -1,
// outputs in natural order.
#pragma once

namespace shtb_dft {

__device__ __forceinline__ double2 cmul(double2 a, double2 b)
{
	return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// multiply by sign*i
__device__ __forceinline__ double2 mul_si(double2 a, int sign) { return sign > 0 ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x); }

template <int R> struct Dft;

template <> struct Dft<2> {
	static __device__ __forceinline__ void run(double2* u, int) {
		double2 a = u[0], b = u[1];
		u[0] = cadd(a, b); u[1] = csub(a, b);
	}
};
template <> struct Dft<4> {
	static __device__ __forceinline__ void run(double2* u, int s) {
		double2 t0 = cadd(u[0], u[2]), t1 = csub(u[0], u[2]);
		double2 t2 = cadd(u[1], u[3]), t3 = mul_si(csub(u[1], u[3]), s);
		u[0] = cadd(t0, t2); u[2] = csub(t0, t2);
		u[1] = cadd(t1, t3); u[3] = csub(t1, t3);
	}
};
template <> struct Dft<8> {
	static __device__ __forceinline__ void run(double2* u, int s) {
		const double h = 0.70710678118654752440084436210485;
		// radix-2 split into even / odd halves, each a 4-point DFT
		double2 e[4] = {u[0], u[2], u[4], u[6]};
		double2 o[4] = {u[1], u[3], u[5], u[7]};
		Dft<4>::run(e, s);
		Dft<4>::run(o, s);
		// twiddles w8^q = exp(s*i*pi*q/4)
		double2 o1 = make_double2(h * (o[1].x - s * o[1].y), h * (o[1].y + s * o[1].x));
		double2 o2 = mul_si(o[2], s);
		double2 o3 = make_double2(h * (-o[3].x - s * o[3].y), h * (-o[3].y + s * o[3].x));
		u[0] = cadd(e[0], o[0]); u[4] = csub(e[0], o[0]);
		u[1] = cadd(e[1], o1);   u[5] = csub(e[1], o1);
		u[2] = cadd(e[2], o2);   u[6] = csub(e[2], o2);
		u[3] = cadd(e[3], o3);   u[7] = csub(e[3], o3);
	}
};
template <> struct Dft<3> {
	static __device__ __forceinline__ void run(double2* u, int s) {
		const double c1 = -0.5, s1 = s * 0.86602540378443864676372317075294;
		double2 t = cadd(u[1], u[2]), d = csub(u[1], u[2]);
		double2 mm = make_double2(fma(c1, t.x, u[0].x), fma(c1, t.y, u[0].y));
		u[0] = cadd(u[0], t);
		u[1] = make_double2(mm.x - s1 * d.y, mm.y + s1 * d.x);
		u[2] = make_double2(mm.x + s1 * d.y, mm.y - s1 * d.x);
	}
};
template <> struct Dft<5> {
	static __device__ __forceinline__ void run(double2* u, int s) {
		const double c1 = 0.30901699437494742410229341718282;   // cos(2pi/5)
		const double c2 = -0.80901699437494742410229341718282;  // cos(4pi/5)
		const double s1 = s * 0.95105651629515357211643933337938;  // sin(2pi/5)
		const double s2 = s * 0.58778525229247312916870595463907;  // sin(4pi/5)
		double2 a1 = cadd(u[1], u[4]), b1 = csub(u[1], u[4]);
		double2 a2 = cadd(u[2], u[3]), b2 = csub(u[2], u[3]);
		double2 x0 = u[0];
		u[0] = cadd(x0, cadd(a1, a2));
		double2 r1 = make_double2(x0.x + c1 * a1.x + c2 * a2.x, x0.y + c1 * a1.y + c2 * a2.y);
		double2 r2 = make_double2(x0.x + c2 * a1.x + c1 * a2.x, x0.y + c2 * a1.y + c1 * a2.y);
		// i*(s1 b1 + s2 b2) and i*(s2 b1 - s1 b2)
		double2 i1 = make_double2(-(s1 * b1.y + s2 * b2.y), s1 * b1.x + s2 * b2.x);
		double2 i2 = make_double2(-(s2 * b1.y - s1 * b2.y), s2 * b1.x - s1 * b2.x);
		u[1] = cadd(r1, i1); u[4] = csub(r1, i1);
		u[2] = cadd(r2, i2); u[3] = csub(r2, i2);
	}
};
// 7-point DFT as a direct sum with the roots of unity as literals
// (cos, sin of 2 pi k / 7, symmetric pairs folded).
template <> struct Dft<7> {
	static __device__ __forceinline__ void run(double2* u, int s) {
		const double c[4] = {1.0, 0.62348980185873353053, -0.22252093395631440429, -0.90096886790241912624};
		const double sn[4] = {0.0, 0.78183148246802980871, 0.97492791218182360702, 0.43388373911755812048};
		double2 a[4], b[4];
		#pragma unroll
		for (int q = 1; q < 4; q++) { a[q] = cadd(u[q], u[7 - q]); b[q] = csub(u[q], u[7 - q]); }
		const double2 x0 = u[0];
		u[0] = cadd(x0, cadd(a[1], cadd(a[2], a[3])));
		#pragma unroll
		for (int k = 1; k < 4; k++) {
			double2 r = x0, im = make_double2(0.0, 0.0);
			#pragma unroll
			for (int q = 1; q < 4; q++) {
				const int j = (q * k) % 7;
				const double cq = (j < 4) ? c[j] : c[7 - j];
				const double sq = (j < 4) ? sn[j] : -sn[7 - j];
				r.x = fma(cq, a[q].x, r.x);  r.y = fma(cq, a[q].y, r.y);
				im.x = fma(sq, b[q].x, im.x); im.y = fma(sq, b[q].y, im.y);
			}
			// y_k = r + i s im,  y_{7-k} = r - i s im
			const double2 t = make_double2(-s * im.y, s * im.x);
			u[k] = cadd(r, t);
			u[7 - k] = csub(r, t);
		}
	}
};

// R = R1 R2 with coprime factors (Good-Thomas: no twiddles): with the input
// index n = R2 n1 + R1 n2 mod R, w_R^(n k) = w_R1^(n1 k) w_R2^(n2 k), so
// output k is entry (k mod R1, k mod R2) of the two-dimensional transform.
template <int R1, int R2>
struct DftCoprime {
	static __device__ __forceinline__ void run(double2* u, int s) {
		constexpr int R = R1 * R2;
		double2 t[R1][R2];
		#pragma unroll
		for (int a = 0; a < R1; a++) {
			#pragma unroll
			for (int b = 0; b < R2; b++) t[a][b] = u[(R2 * a + R1 * b) % R];
			Dft<R2>::run(t[a], s);
		}
		#pragma unroll
		for (int b = 0; b < R2; b++) {
			double2 c[R1];
			#pragma unroll
			for (int a = 0; a < R1; a++) c[a] = t[a][b];
			Dft<R1>::run(c, s);
			#pragma unroll
			for (int a = 0; a < R1; a++) t[a][b] = c[a];
		}
		#pragma unroll
		for (int k = 0; k < R; k++) u[k] = t[k % R1][k % R2];
	}
};
template <> struct Dft<1> { static __device__ __forceinline__ void run(double2*, int) {} };
template <> struct Dft<6> { static __device__ __forceinline__ void run(double2* u, int s) { DftCoprime<2, 3>::run(u, s); } };
template <> struct Dft<10> { static __device__ __forceinline__ void run(double2* u, int s) { DftCoprime<2, 5>::run(u, s); } };
template <> struct Dft<12> { static __device__ __forceinline__ void run(double2* u, int s) { DftCoprime<3, 4>::run(u, s); } };
template <> struct Dft<15> { static __device__ __forceinline__ void run(double2* u, int s) { DftCoprime<3, 5>::run(u, s); } };

// R = Q^2: n = Q n1 + n2, k = k1 + Q k2, w_R^(n k) = w_Q^(n1 k1) w_R^(n2 k1) w_Q^(n2 k2).
// cs, sn: cos and sin of 2 pi j / R for the products j = n2 k1 <= (Q - 1)^2
template <int Q>
struct DftSquare {
	static __device__ __forceinline__ void run(double2* u, int s, const double* cs, const double* sn) {
		double2 t[Q][Q];
		#pragma unroll
		for (int n2 = 0; n2 < Q; n2++) {
			double2 c[Q];
			#pragma unroll
			for (int n1 = 0; n1 < Q; n1++) c[n1] = u[Q * n1 + n2];
			Dft<Q>::run(c, s);
			#pragma unroll
			for (int k1 = 0; k1 < Q; k1++)
				t[k1][n2] = (n2 * k1) ? cmul(c[k1], make_double2(cs[n2 * k1], s * sn[n2 * k1])) : c[k1];
		}
		#pragma unroll
		for (int k1 = 0; k1 < Q; k1++) {
			Dft<Q>::run(t[k1], s);
			#pragma unroll
			for (int k2 = 0; k2 < Q; k2++) u[k1 + Q * k2] = t[k1][k2];
		}
	}
};
template <> struct Dft<9> {
	static __device__ __forceinline__ void run(double2* u, int s) {
		// 2 pi j / 9, j = 0 .. 4
		constexpr double cs[5] = {1.0, 0.76604444311897803520, 0.17364817766693034885, -0.5, -0.93969262078590838405};
		constexpr double sn[5] = {0.0, 0.64278760968653932632, 0.98480775301220805937, 0.86602540378443864676, 0.34202014332566873304};
		DftSquare<3>::run(u, s, cs, sn);
	}
};
template <> struct Dft<16> {
	static __device__ __forceinline__ void run(double2* u, int s) {
		// 2 pi j / 16, j = 0 .. 9
		constexpr double a = 0.92387953251128675613, b = 0.38268343236508977173, h = 0.70710678118654752440;
		constexpr double cs[10] = {1.0, a, h, b, 0.0, -b, -h, -a, -1.0, -a};
		constexpr double sn[10] = {0.0, b, h, a, 1.0, a, h, b, 0.0, -b};
		DftSquare<4>::run(u, s, cs, sn);
	}
};

// u[q] *= w^q, the powers by products of at most 4 factors
template <int R>
__device__ __forceinline__ void twiddles(double2* u, double2 w1)
{
	if constexpr (R > 1) {
		double2 w[4];                            // w^1 .. w^4
		w[0] = w1;
		u[1] = cmul(u[1], w1);
		if constexpr (R > 2) { w[1] = cmul(w1, w1); u[2] = cmul(u[2], w[1]); }
		if constexpr (R > 3) { w[2] = cmul(w[1], w1); u[3] = cmul(u[3], w[2]); }
		if constexpr (R > 4) {
			w[3] = cmul(w[1], w[1]);
			double2 h = w[3];                    // w^4, w^8, w^12
			#pragma unroll
			for (int q = 4; q < R; q += 4) {
				u[q] = cmul(u[q], h);
				#pragma unroll
				for (int r = 1; r < 4; r++) if (q + r < R) u[q + r] = cmul(u[q + r], cmul(h, w[r - 1]));
				if (q + 4 < R) h = cmul(h, w[3]);
			}
		}
	}
}

} // namespace shtb_dft
