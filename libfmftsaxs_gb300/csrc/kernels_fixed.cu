/*
 * The plain path's contractions (rotation, translation, per-pose sums; see
 * kernels_contract.cu for the formulas) in fixed point on the integer
 * multiply-add pipe.
 *
 * This GPU's FP64 pipe takes 2 multiply-adds per clock and SM (measured 0.50
 * T/s over the GPU); its 32 x 32 + 64-bit integer multiply-add (IMAD.WIDE)
 * takes 27 (8.5 T/s).  A real number v of a table
 * row is held as v / 2^e = (h 2^29 + l) 2^-57 with two 32-bit limbs, |l| <=
 * 2^28, and one exponent e per molecule, channel and q; a product is then
 * three IMAD.WIDE,
 *   h h' -> a 64-bit sum, h l' + l h' -> a second 64-bit sum
 * (l l', at most 2^-58 of the first sum's scale, is dropped), and the sums are
 * exact: nothing is rounded until a sum is complete.
 *
 * The exponents come from norms that the operations keep: a rotation leaves
 * the 2-norm of a channel's coefficients at each q alone, so bounds of
 * |A_c(q)|_2 hold for every row of the rotated tables, and the translation by
 * z is a compression of the multiplication by f(t) = exp(i q z t), so that its
 * norm is at most max |f|, taken from the Bessel values in use.  With
 * Cauchy-Schwarz no sum overflows, and an entry is off by 2^-58 of its row's
 * bound, where FP64 rounds every term and partial sum at 2^-53 of its size:
 * against long double, and relative to the norms of its own two channels, no
 * channel pair's cross term is further off than the FP64 kernels' (rms over
 * poses; tests/test_gpu_fixed_channels.py has channels weaker than the others
 * by up to 1e6).  The exponents are a molecule's own: its rotation table
 * serves any partner.  A coefficient that is not finite makes all six terms
 * of its q NaN.
 */
#include "kernels.h"
#include "chain.cuh"
#include "limbs.cuh"

#include <math.h>

namespace {

/* first pair of row m >= 0 */
__device__ __forceinline__ int psym(int m, int K) { return m * K - m * (m - 1) / 2; }

typedef long long i64;

/* a b + c: a product and a sum, which the assembler joins to one IMAD.WIDE; the
 * single instruction mad.wide.s32 comes out with a second one beside it (16
 * independent sums: 7.6 against 8.5 T/s, 2.1 instructions per product), and
 * as a C expression the sums are reordered and not joined */
__device__ __forceinline__ i64 madw(int a, int b, i64 c)
{
	i64 r;
	asm("{\n\t.reg .s64 t;\n\tmul.wide.s32 t, %1, %2;\n\tadd.s64 %0, t, %3;\n\t}" : "=l"(r) : "r"(a), "r"(b), "l"(c));
	return r;
}

/* a sum of products: hh the products of the high limbs (unit 2^-56), mid the
 * mixed ones (unit 2^-85) */
struct Acc {
	i64 hh, mid;
};
__device__ __forceinline__ Acc acc0() { return {0, 1 << 27}; }   /* mid starts at half of what value() drops */
__device__ __forceinline__ void mul_add(Acc &s, int ah, int al, int bh, int bl)
{
	s.hh = madw(ah, bh, s.hh);
	s.mid = madw(ah, bl, s.mid);
	s.mid = madw(al, bh, s.mid);
}
/* the sum as an integer of unit 2^-57, rounded to nearest */
__device__ __forceinline__ i64 value(const Acc &s) { return 2 * s.hh + (s.mid >> 28); }
/* the limbs of v (unit 2^-57) */
__device__ __forceinline__ int hi_limb(i64 v) { return (int)((v + (1ll << 28)) >> 29); }
__device__ __forceinline__ int lo_limb(i64 v, int h) { return (int)((unsigned)v - ((unsigned)h << 29)); }

__device__ __forceinline__ int4 entry(i64 x, i64 y)
{
	int xh = hi_limb(x), yh = hi_limb(y);
	return make_int4(xh, lo_limb(x, xh), yh, lo_limb(y, yh));
}

/* 2^e for a normal result */
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }

/* sc[ch][q] = 2^(28 - e) of a molecule's coefficients (host flat layout
 * [3][Q][K2][2]), with the channel's norm at most 2^(e + 1) / 1.15, which
 * leaves room for the translation to lengthen a row by up to 1.12; NaN at all
 * three where a coefficient is not finite.  The norm is formed of the
 * coefficients over their largest exponent: squares neither overflow nor
 * vanish.  e is at least FIX_EMIN (the scale is a double); a channel without
 * entries has that.  A block per q, padded with ones up to Qp. */
#define FIX_EMIN (-995)
__global__ void __launch_bounds__(128) k_fix_scale(const double *__restrict__ flat, int Q, int K2, int Qp,
                                                   double *__restrict__ sc)
{
	__shared__ double part[4];
	__shared__ int top[3];
	int q = blockIdx.x;
	if (q >= Q) {
		if (threadIdx.x < 3) sc[threadIdx.x * Qp + q] = 1.0;
		return;
	}
	if (threadIdx.x < 3) top[threadIdx.x] = 0;
	__syncthreads();
	double c28[3];
	bool bad = false;
	for (int ch = 0; ch < 3; ch++) {
		const double *a = flat + ((size_t)ch * Q + q) * K2 * 2;
		int h = 0;                                    /* largest high word: exponent and leading bits */
		for (int i = threadIdx.x; i < 2 * K2; i += blockDim.x) h = max(h, __double2hiint(a[i]) & 0x7fffffff);
		h = __reduce_max_sync(0xffffffffu, h);
		if (threadIdx.x % 32 == 0) atomicMax(&top[ch], h);
		__syncthreads();
		int k = (top[ch] >> 20) - 1022, e = FIX_EMIN;  /* |a| < 2^k */
		bad |= k > 1024;
		double f = pow2(-k / 2), g = pow2(-k - -k / 2), s = 0.0;
		for (int i = threadIdx.x; i < 2 * K2; i += blockDim.x) {
			double v = a[i] * f * g;
			s = fma(v, v, s);
		}
		for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
		if (threadIdx.x % 32 == 0) part[threadIdx.x / 32] = s;
		__syncthreads();
		s = 0.575 * sqrt(part[0] + part[1] + part[2] + part[3]);
		__syncthreads();
		if (s > 0.0) {
			frexp(s, &e);                             /* s < 2^e */
			e = max(e + k, FIX_EMIN);
		}
		c28[ch] = pow2(28 - e);
	}
	if (threadIdx.x == 0)
		for (int ch = 0; ch < 3; ch++) sc[ch * Qp + q] = bad ? nan("") : c28[ch];
}
/* e of a scale 2^(28 - e) */
__device__ __forceinline__ int fix_exp(double c28) { return 28 + 1023 - (__double2hiint(c28) >> 20); }

/* [3][Q][K2][2] -> [3][K2][Q] limbs {re h, re l, im h, im l}, conjugated
 * when conj != 0 */
__global__ void k_fix_spf(const double *__restrict__ flat, const double *__restrict__ sc, int Q, int K2, int Qp,
                          int conj, int4 *__restrict__ t)
{
	long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= 3L * Q * K2) return;
	int iq = (int)(i % Q);
	long r = i / Q;
	int lm = (int)(r % K2), ch = (int)(r / K2);
	const double *s = flat + (((size_t)ch * Q + iq) * K2 + lm) * 2;
	double c28 = sc[ch * Qp + iq];
	int2 a = sxs_limbs(s[0], c28), b = sxs_limbs(conj ? -s[1] : s[1], c28);
	t[i] = make_int4(a.x, a.y, b.x, b.y);
}

__global__ void k_fix_dtab(const double *__restrict__ d, int2 *__restrict__ x, long n)
{
	long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) x[i] = sxs_limbs(d[i], 268435456.0);
}

/* nu2[iz][q] = 2^nu with |T(z q)|_2 <= 1.12 2^nu.  T is the compression to l
 * <= L of the multiplication by f(t) = sum_p i^p (2p + 1) j_p(z q) P_p(t), p
 * <= 2L (other p do not reach l, l1 <= L), so |T|_2 <= max |f| over [-1, 1].
 * Re(e^{i phi} f(cos theta)) is a cosine polynomial of degree 2L, so that its
 * maximum is at most that over theta = k pi / 256 divided by cos(2L pi /
 * 512); |f(-t)| = |f(t)| leaves half of those points.  FP32 is enough for a
 * bound.  NaN where f is not finite; a block per (iz, q), padded with ones. */
__global__ void __launch_bounds__(160) k_fix_nu(const double *__restrict__ bes, int Q, int L, int Qp,
                                                double *__restrict__ nu2)
{
	__shared__ float jp[2 * SXSK_FIX_LMAX + 1], mx[5];
	int iz = blockIdx.x / Qp, q = blockIdx.x % Qp, N = 2 * L + 1, k = threadIdx.x;
	if (q >= Q) {
		if (k == 0) nu2[(size_t)iz * Qp + q] = 1.0;
		return;
	}
	for (int p = k; p < N; p += blockDim.x) {
		float v = (2 * p + 1) * (float)bes[((size_t)iz * N + p) * Q + q];
		jp[p] = (p & 2) ? -v : v;                     /* i^p: even p real, odd p imaginary */
	}
	__syncthreads();
	float t = cospif(k / 256.0f), p0 = 1.0f, p1 = t, re = jp[0], im = 0.0f;
	for (int p = 1; p < N; p++) {
		if (p & 1) im += jp[p] * p1;
		else re += jp[p] * p1;
		float p2 = ((2 * p + 1) * t * p1 - p * p0) / (p + 1);
		p0 = p1;
		p1 = p2;
	}
	float f = k <= 128 ? sqrtf(re * re + im * im) : 0.0f;
	if (!isfinite(f)) f = __int_as_float(0x7f800000);
	for (int o = 16; o; o >>= 1) f = fmaxf(f, __shfl_xor_sync(0xffffffffu, f, o));
	if (k % 32 == 0) mx[k / 32] = f;
	__syncthreads();
	if (k == 0) {
		for (int w = 1; w < 5; w++) f = fmaxf(f, mx[w]);
		f *= 1.001f / cospif(2 * L / 512.0f);
		double v = nan("");
		if (isfinite(f)) {
			int e = 0;
			if (f > 1.12f) frexpf(f / 1.12f, &e);   /* f / 1.12 < 2^e */
			v = ldexp(1.0, e);
		}
		nu2[(size_t)iz * Qp + q] = v;
	}
}

/* Twiddles of the paired rotation sum (kernels_contract.cu): h+ and h- as
 * limbs; of h+ = (tw[k] + tw[N-k]) / 2 the real part is the large one and of
 * h- = (tw[k] - tw[N-k]) / 2 the imaginary one.  The other parts vanish but
 * for the rounded pi of the reference's table (1e-11): one limb of unit
 * 2^-57 holds them, and its product with a high limb has the unit of mid. */
struct FixTw {
	int4 a;   /* Re h+ (h, l), Im h- (h, l) */
	int2 b;   /* Im h+, Re h- */
};

__device__ __forceinline__ FixTw fix_tw(const double2 *tw, int k, int N)
{
	int kk = k % N;
	double2 a = tw[kk], b = tw[(N - kk) % N];
	int2 c = sxs_limbs(0.5 * (a.x + b.x), 268435456.0), s = sxs_limbs(0.5 * (a.y - b.y), 268435456.0);
	FixTw r;
	r.a = make_int4(c.x, c.y, s.x, s.y);
	r.b = make_int2((int)rint(0.5 * (a.y + b.y) * 0x1p57), (int)rint(0.5 * (a.x - b.x) * 0x1p57));
	return r;
}

#define FROT_GROUPS 4
#define FROT_THREADS (FROT_GROUPS * 3 * SXS_QT)

/* Rotation table of k_rotate in limbs: out[t][b*N+g][pair(m,l)][ch][q].
 * Block = (m, beta b, q tile t); thread = (group of G gamma pairs, channel,
 * q), as in the FP64 form.  Per m1 a thread forms S = y(m1) + y(-m1) and D =
 * y(m1) - y(-m1) (12 IMAD.WIDE and ~40 adds and shifts) and per gamma pair
 * four sums of 16 IMAD.WIDE in all, ~75 clocks of its pipe, where the FP64
 * form's 8 operations take 512.  Bound by that pipe; table stage (both tables,
 * per-z tables beside) at L = 20, Q = 101: 17.0 -> 3.5 ms (six gamma pairs: four
 * blocks on an SM, 166 registers instead of 178 and 4.3 ms). */
template <int G>
__global__ void __launch_bounds__(FROT_THREADS, (G == 6 ? 4 : 0))
k_fix_rotate(const int4 *__restrict__ spf, const int2 *__restrict__ dtab, const double2 *__restrict__ tw, int Q, int L,
             int4 *__restrict__ out)
{
	extern __shared__ __align__(16) unsigned char fsm[];
	int K = L + 1, N = 2 * L + 1, K2 = K * K, NP = K * (K + 1) / 2, nrow = K * N, ne = N + (G - 1) * L;
	int4 *ha = reinterpret_cast<int4 *>(fsm);
	int2 *hb = reinterpret_cast<int2 *>(ha + ne);
	for (int k = threadIdx.x; k < ne; k += blockDim.x) {
		FixTw h = fix_tw(tw, k, N);
		ha[k] = h.a;
		hb[k] = h.b;
	}
	__syncthreads();
	int bid = blockIdx.x;
	int m = bid % K;
	bid /= K;
	int b = bid % K, t = bid / K;
	int qq = threadIdx.x % SXS_QT, ch = (threadIdx.x / SXS_QT) % 3, gg = threadIdx.x / (3 * SXS_QT);
	int q = t * SXS_QT + qq;
	bool qok = q < Q;
	int g0 = gg * G;
	if (g0 > L) return;
	const int4 *C = spf + (size_t)ch * K2 * Q + (qok ? q : 0);
	const int2 *db = dtab + ((size_t)b * K * N + m + L) * N + L;
	int4 *ob = out + (((size_t)t * nrow + (size_t)b * N) * NP + psym(m, K)) * 3 * SXS_QT + ch * SXS_QT + qq;
	size_t gstride = (size_t)NP * 3 * SXS_QT;
	const int4 zero = make_int4(0, 0, 0, 0);
	for (int l = m; l <= L; l++) {
		const int2 *dl = db + (size_t)l * N * N;
		const int4 *Cl = C + (size_t)l * (l + 1) * Q;
		int2 d0 = __ldg(dl);
		int4 c0 = qok ? __ldg(Cl) : zero;
		Acc a = acc0();
		mul_add(a, d0.x, d0.y, c0.x, c0.y);
		i64 y0x = value(a);
		a = acc0();
		mul_add(a, d0.x, d0.y, c0.z, c0.w);
		i64 y0y = value(a);
		Acc Ax[G], Ay[G], Bx[G], By[G];
#pragma unroll
		for (int j = 0; j < G; j++) Ax[j] = Ay[j] = Bx[j] = By[j] = acc0();
		int base = 0;
		for (int m1 = 1; m1 <= l; m1++) {
			base += g0;
			if (base >= N) base -= N;
			int2 dp = __ldg(dl + m1), dm = __ldg(dl - m1);
			int4 cp = qok ? __ldg(Cl + (size_t)m1 * Q) : zero, cm = qok ? __ldg(Cl - (ptrdiff_t)m1 * Q) : zero;
			Acc px = acc0(), py = acc0(), nx = acc0(), ny = acc0();
			mul_add(px, dp.x, dp.y, cp.x, cp.y);
			mul_add(py, dp.x, dp.y, cp.z, cp.w);
			mul_add(nx, dm.x, dm.y, cm.x, cm.y);
			mul_add(ny, dm.x, dm.y, cm.z, cm.w);
			i64 vpx = value(px), vpy = value(py), vnx = value(nx), vny = value(ny);
			i64 sx = vpx + vnx, sy = vpy + vny, dx = vpx - vnx, dy = vpy - vny;
			int sxh = hi_limb(sx), sxl = lo_limb(sx, sxh), syh = hi_limb(sy), syl = lo_limb(sy, syh);
			int dxh = hi_limb(dx), dxl = lo_limb(dx, dxh), dyh = hi_limb(dy), dyl = lo_limb(dy, dyh);
			int k = base;
#pragma unroll
			for (int j = 0; j < G; j++) {
				int4 h = ha[k];
				int2 e = hb[k];
				/* A += h+ S, B += h- D */
				mul_add(Ax[j], h.x, h.y, sxh, sxl);
				mul_add(Ay[j], h.x, h.y, syh, syl);
				mul_add(By[j], h.z, h.w, dxh, dxl);
				mul_add(Bx[j], -h.z, -h.w, dyh, dyl);
				Ax[j].mid = madw(-e.x, syh, Ax[j].mid);
				Ay[j].mid = madw(e.x, sxh, Ay[j].mid);
				Bx[j].mid = madw(e.y, dxh, Bx[j].mid);
				By[j].mid = madw(e.y, dyh, By[j].mid);
				k += m1;
			}
		}
		int4 *o = ob + (size_t)(l - m) * 3 * SXS_QT;
#pragma unroll
		for (int j = 0; j < G; j++) {
			int g = g0 + j;
			if (g > L) break;
			i64 ax = y0x + value(Ax[j]), ay = y0y + value(Ay[j]), bx = value(Bx[j]), by = value(By[j]);
			i64 x = ax + bx, y = ay + by;
			o[(size_t)g * gstride] = entry(x, y);
			if (g > 0) o[(size_t)(N - g) * gstride] = entry(ax - bx, ay - by);
		}
	}
}

#define FTR_COMBOS 8
#define FTR_THREADS (FTR_COMBOS * 3 * SXS_QT)

/* The translation in limbs (column form, as k_translate_col): thread = the
 * column (combo, channel, q) of one m, its n = L + 1 - m entries of U in
 * registers; block = (tile, half a slice of combos sharing z, m), tau^m(q z)
 * staged in shared memory.  Rows in even/odd pairs, so that the parity of i +
 * k, which says whether an entry adds tau U or tau (-i U), is known at compile
 * time.  Bound by IMAD.WIDE: 6 per (i, k); 15.0 ms at L = 20, Q = 101, 70,000
 * poses (FP64: 59); 8 combos per block instead of the FP64
 * form's 16 so that two to four blocks' staging overlaps. */
template <int PAR, int NB>
__device__ __forceinline__ int4 fix_row(const int2 *__restrict__ row, const int4 (&u)[NB])
{
	/* re, and im as even minus odd terms */
	Acc re = acc0(), ie = acc0(), io = {0, 0};
#pragma unroll
	for (int k = 0; k < NB; k += 2) {
		int4 t2 = *reinterpret_cast<const int4 *>(row + k);
#pragma unroll
		for (int kk = 0; kk < 2; kk++) {
			int th = kk ? t2.z : t2.x, tl = kk ? t2.w : t2.y;
			const int4 &v = u[k + kk];
			if (((k + kk) & 1) == PAR) {
				mul_add(re, th, tl, v.x, v.y);
				mul_add(ie, th, tl, v.z, v.w);
			} else {
				mul_add(re, th, tl, v.z, v.w);
				mul_add(io, th, tl, v.x, v.y);
			}
		}
	}
	ie.hh -= io.hh;
	ie.mid -= io.mid;
	return entry(value(re), value(ie));
}

template <int NB>
__global__ void __launch_bounds__(FTR_THREADS, (NB <= 12 ? 4 : (NB <= 20 ? 3 : 2)))
k_fix_translate(const int4 *__restrict__ U, const int2 *__restrict__ tau, const int32_t *__restrict__ combo_zbg,
                const int32_t *__restrict__ slices, int nslice, int cbase, int ncombo, int L, int nzt, int m_lo, int nm,
                int4 *__restrict__ R)
{
	extern __shared__ __align__(16) unsigned char ftsm[];
	chain_begin();
	int2 *ts = reinterpret_cast<int2 *>(ftsm);   /* [8 q][NB i][NB k] (+ pad per q) */
	const int qstride = NB * NB + 2;
	int K = L + 1, N = 2 * L + 1, NP = K * (K + 1) / 2, nrow = K * N;
	const int per = SXS_SLICE / FTR_COMBOS;
	int bid = blockIdx.x;
	int mi = bid % nm;
	bid /= nm;
	int part = bid % per;
	bid /= per;
	int si = bid % nslice, t = bid / nslice;
	int m = m_lo + mi, n = K - m;
	int cfirst = slices[2 * si] - cbase + part * FTR_COMBOS, nc = slices[2 * si + 1] - part * FTR_COMBOS;
	if (nc <= 0) {
		chain_end();
		return;
	}
	int zi = combo_zbg[3 * cfirst];
	const int2 *tz = tau + ((((size_t)t * nzt + zi) * K + m) * K) * K * SXS_QT;
	for (int k = threadIdx.x; k < SXS_QT * NB * NB; k += blockDim.x) {
		int q = k % SXS_QT, r = k / SXS_QT;
		int i = r / NB, kk = r % NB;
		int2 v = make_int2(0, 0);
		if (i < n && kk < n) v = __ldg(tz + ((size_t)(m + i) * K + m + kk) * SXS_QT + q);
		ts[q * qstride + i * NB + kk] = v;
	}
	int q = threadIdx.x % SXS_QT, ch = (threadIdx.x / SXS_QT) % 3, cl = threadIdx.x / (3 * SXS_QT);
	bool act = cl < nc;
	int c = cfirst + (act ? cl : 0);
	int b2 = combo_zbg[3 * c + 1], g2 = combo_zbg[3 * c + 2], po = psym(m, K);
	const int4 *Ub = U + (((size_t)t * nrow + b2 * N + g2) * NP + po) * 3 * SXS_QT + ch * SXS_QT + q;
	int4 u[NB];
#pragma unroll
	for (int k = 0; k < NB; k++) u[k] = k < n ? __ldg(Ub + (size_t)k * 3 * SXS_QT) : make_int4(0, 0, 0, 0);
	__syncthreads();
	if (act) {
		const int2 *tq = ts + q * qstride;
		int4 *Rb = R + (((size_t)t * ncombo + c) * NP + po) * 3 * SXS_QT + ch * SXS_QT + q;
		for (int i = 0; i < n; i += 2) {
			Rb[(size_t)i * 3 * SXS_QT] = fix_row<0, NB>(tq + i * NB, u);
			if (i + 1 < n) Rb[(size_t)(i + 1) * 3 * SXS_QT] = fix_row<1, NB>(tq + (i + 1) * NB, u);
		}
	}
	chain_end();
}

/* 16-byte loads with L2 policies: receptor rows are read by many poses
 * (evict_last), translated rows by the few poses of their combo
 * (evict_first) */
__device__ __forceinline__ uint64_t fix_policy(bool keep)
{
	uint64_t pol;
	if (keep) asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
	else asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
	return pol;
}
__device__ __forceinline__ int4 ld_pol(const int4 *p, uint64_t pol)
{
	int4 v;
	asm("ld.global.nc.L2::cache_hint.v4.s32 {%0, %1, %2, %3}, [%4], %5;"
	    : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
	    : "l"(p), "l"(pol));
	return v;
}

/* the real and the imaginary part of p r for complex limbs, n = -Im p */
__device__ __forceinline__ void re_add(Acc &s, int4 p, int2 n, int4 r)
{
	s.hh = madw(p.x, r.x, s.hh);
	s.mid = madw(p.x, r.y, s.mid);
	s.hh = madw(n.x, r.z, s.hh);
	s.mid = madw(p.y, r.x, s.mid);
	s.mid = madw(n.x, r.w, s.mid);
	s.mid = madw(n.y, r.z, s.mid);
}
__device__ __forceinline__ void im_add(Acc &s, int4 p, int4 r)
{
	s.hh = madw(p.x, r.z, s.hh);
	s.mid = madw(p.x, r.w, s.mid);
	s.hh = madw(p.z, r.x, s.hh);
	s.mid = madw(p.y, r.z, s.mid);
	s.mid = madw(p.z, r.y, s.mid);
	s.mid = madw(p.w, r.x, s.mid);
}

#define FPC_POSES 16
#define FPC_THREADS (FPC_POSES * SXS_QT)

/* x + y 2^-d for d >= 0 and x 2^d + y below, rounded: two sums of a channel
 * pair in the unit of the larger one */
__device__ __forceinline__ i64 join(i64 x, i64 y, int d)
{
	i64 big = d < 0 ? y : x, small = d < 0 ? x : y;
	int k = min(abs(d), 62);
	return big + ((small + ((1ll << k) >> 1)) >> k);
}

/* Per-pose cross terms from limbs.  Thread = (pose, q); block = 16
 * consecutive poses (sorted by combo) x the 8 q of a tile, tile-major.
 * Per m the nine channel products are summed over l as complex numbers, the
 * two of a pair (P_a R_b and P_b R_a, whose units differ) joined in the larger
 * unit, and the pose's phase w_m is applied to the six sums.  Bound by
 * the integer pipe: 108 IMAD.WIDE per pair of rows, 54 at m = 0.  At L = 20, Q =
 * 101, 70,000 poses: 21.5 ms (FP64 kernel: 87.5; all 108 at m = 0: 22.8).  With one unit for all channels
 * six products do, (P_a + P_b)(R_a + R_b) - P_a R_a - P_b R_b, but a channel ten
 * times weaker then has up to 7 times the FP64 kernels' error (a thousand times:
 * 500); the same six with one operand of each sum shifted to the other's unit
 * 28.7; a thread per channel of P 23.7; rows two pairs ahead 23.8; mad.wide.s32
 * 25.1. */
__global__ void __launch_bounds__(FPC_THREADS, 3)
k_fix_cross(const sxsk_pose *__restrict__ poses, int npose, int combo_base, int ncombo,
            const int32_t *__restrict__ combo_zbg, const int4 *__restrict__ P, const int4 *__restrict__ R,
            const double2 *__restrict__ tw, const double *__restrict__ scA, const double *__restrict__ scB,
            const double *__restrict__ nu2, int Qp, const double *__restrict__ cst, int Q, int L,
            double *__restrict__ cross)
{
	__shared__ int4 tws[2 * 32 - 1];                  /* w_m as limbs {re h, re l, -im h, -im l} */
	__shared__ i64 F[12][FPC_THREADS];                /* the phased sums: six hh, six mid */
	int K = L + 1, N = 2 * L + 1, NP = K * (K + 1) / 2, nrow = K * N;
	for (int k = threadIdx.x; k < N; k += blockDim.x) {
		int2 a = sxs_limbs(tw[k].x, 268435456.0), b = sxs_limbs(-tw[k].y, 268435456.0);
		tws[k] = make_int4(a.x, a.y, b.x, b.y);
	}
	__syncthreads();
	int bpt = (npose + FPC_POSES - 1) / FPC_POSES;
	int t = blockIdx.x / bpt, pi = (blockIdx.x % bpt) * FPC_POSES + threadIdx.x / SXS_QT;
	int qq = threadIdx.x % SXS_QT, q = t * SXS_QT + qq;
	if (pi >= npose || q >= Q) return;
	sxsk_pose ps = poses[pi];
	const int4 *Pr = P + (((size_t)t * nrow + ps.b1 * N + ps.g1) * NP) * 3 * SXS_QT + qq;
	const int4 *Rr = R + (((size_t)t * ncombo + ps.combo - combo_base) * NP) * 3 * SXS_QT + qq;
	uint64_t polP = fix_policy(true), polR = fix_policy(false);
	const int ca[6] = {0, 0, 0, 1, 1, 2}, cb[6] = {0, 1, 2, 1, 2, 2};
	double nu = nu2[(size_t)combo_zbg[3 * (ps.combo - combo_base)] * Qp + q], ok = nu;
	int eA[3], eB[3], d[3];
#pragma unroll
	for (int c = 0; c < 3; c++) {
		double a = scA[c * Qp + q], b = scB[c * Qp + q];
		eA[c] = fix_exp(a);
		eB[c] = fix_exp(b);
		ok += a + b;
	}
	d[0] = eA[0] + eB[1] - eA[1] - eB[0];
	d[1] = eA[0] + eB[2] - eA[2] - eB[0];
	d[2] = eA[1] + eB[2] - eA[2] - eB[1];
	int e = 0;
	int4 p0 = ld_pol(Pr, polP), p1 = ld_pol(Pr + SXS_QT, polP), p2 = ld_pol(Pr + 2 * SXS_QT, polP);
	int4 r0 = ld_pol(Rr, polR), r1 = ld_pol(Rr + SXS_QT, polR), r2 = ld_pol(Rr + 2 * SXS_QT, polR);
	int left = NP;
	for (int m = 0; m < K; m++) {
		Acc re[9], im[9];
#pragma unroll
		for (int c = 0; c < 9; c++) re[c] = im[c] = acc0();
		for (int i = K - m; i > 0; i--) {
			int4 a0 = p0, a1 = p1, a2 = p2, b0 = r0, b1 = r1, b2 = r2;
			/* the next pair's rows stream in behind this pair's products */
			int step = --left > 0 ? 3 * SXS_QT : 0;
			Pr += step;
			Rr += step;
			p0 = ld_pol(Pr, polP);
			p1 = ld_pol(Pr + SXS_QT, polP);
			p2 = ld_pol(Pr + 2 * SXS_QT, polP);
			r0 = ld_pol(Rr, polR);
			r1 = ld_pol(Rr + SXS_QT, polR);
			r2 = ld_pol(Rr + 2 * SXS_QT, polR);
			int2 n0 = make_int2(-a0.z, -a0.w), n1 = make_int2(-a1.z, -a1.w), n2 = make_int2(-a2.z, -a2.w);
			re_add(re[0], a0, n0, b0);
			re_add(re[1], a0, n0, b1);
			re_add(re[2], a0, n0, b2);
			re_add(re[3], a1, n1, b1);
			re_add(re[4], a1, n1, b2);
			re_add(re[5], a2, n2, b2);
			re_add(re[6], a1, n1, b0);
			re_add(re[7], a2, n2, b0);
			re_add(re[8], a2, n2, b1);
			if (m > 0) {   /* w_0 = 1: only real parts count */
				im_add(im[0], a0, b0);
				im_add(im[1], a0, b1);
				im_add(im[2], a0, b2);
				im_add(im[3], a1, b1);
				im_add(im[4], a1, b2);
				im_add(im[5], a2, b2);
				im_add(im[6], a1, b0);
				im_add(im[7], a2, b0);
				im_add(im[8], a2, b1);
			}
		}
		/* F += Re(w_m G): the sums start with m = 0, which counts once where
		 * the others count twice (their mirror images) */
		int4 w = tws[e];
#pragma unroll
		for (int c = 0; c < 6; c++) {
			const int o[6] = {0, 6, 7, 0, 8, 0};              /* the pair's other product */
			i64 x = value(re[c]), y = value(im[c]);
			if (o[c]) {
				int dd = d[c == 4 ? 2 : c - 1];
				x = join(x, value(re[o[c]]), dd);
				y = join(y, value(im[o[c]]), dd);
			}
			int xh = hi_limb(x), xl = lo_limb(x, xh), yh = hi_limb(y), yl = lo_limb(y, yh);
			Acc f = {0, 0};
			if (m > 0) f = {F[c][threadIdx.x], F[6 + c][threadIdx.x]};
			mul_add(f, w.x, w.y, xh, xl);
			mul_add(f, w.z, w.w, yh, yl);
			if (m > 0) {
				F[c][threadIdx.x] = f.hh;
				F[6 + c][threadIdx.x] = f.mid;
			} else {
				F[c][threadIdx.x] = f.hh >> 1;        /* half, exactly: the lost bit is 2^29 of mid / 2 */
				F[6 + c][threadIdx.x] = ((f.mid + ((f.hh & 1) << 29)) >> 1);
			}
		}
		e += ps.a2;
		if (e >= N) e -= N;
	}
	double *o = cross + (size_t)ps.src * 6 * Q + q;
#pragma unroll
	for (int c = 0; c < 6; c++) {
		i64 hh = F[c][threadIdx.x], mid = F[6 + c][threadIdx.x];
		/* the pair's unit, in two factors that cannot overflow */
		int ex = max(eA[ca[c]] + eB[cb[c]], eA[cb[c]] + eB[ca[c]]) + (__double2hiint(nu) >> 20) - 1023 - 55;
		int ea = ex / 2, eb = ex - ea;
		double v = (double)(2 * hh + ((mid + (1 << 27)) >> 28)) * pow2(ea);
		if (isnan(ok)) v = ok;
		o[(size_t)c * Q] = fma(v, pow2(eb), cst[(size_t)c * Q + q]);
	}
}

inline int nblk(long n, int b) { return (int)((n + b - 1) / b); }

template <int G>
int rotate_launch(const void *spf, const int2 *dtab, const double2 *tw, int Q, int L, void *out, cudaStream_t s)
{
	int K = L + 1, N = 2 * L + 1, NT = (Q + SXS_QT - 1) / SXS_QT;
	size_t smem = (sizeof(int4) + sizeof(int2)) * (size_t)(N + (G - 1) * L);
	k_fix_rotate<G><<<(unsigned)(K * K * NT), FROT_THREADS, smem, s>>>((const int4 *)spf, dtab, tw, Q, L, (int4 *)out);
	return cudaGetLastError();
}

template <int NB>
int translate_launch(const void *U, const void *tau, const int32_t *combo_zbg, const int32_t *slices, int nslice,
                     int cbase, int ncombo, int nzt, int NT, int L, void *R, bool *linked, cudaStream_t s)
{
	int K = L + 1;
	/* m with n = K - m in (NB - 4, NB] */
	int m_hi = K - (NB - 3), m_lo = K - NB;
	if (m_hi > L) m_hi = L;
	if (m_lo < 0) m_lo = 0;
	if (m_hi < m_lo) return cudaSuccess;
	int nm = m_hi - m_lo + 1;
	long nb = (long)NT * nslice * (SXS_SLICE / FTR_COMBOS) * nm;
	if (nb > 0x7fffffffL) return cudaErrorInvalidValue;
	size_t smem = sizeof(int2) * SXS_QT * (NB * NB + 2);
	auto kern = k_fix_translate<NB>;
	cudaError_t e = cudaSuccess;
	if (smem > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (!e)
		e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
		                         (int)cudaSharedmemCarveoutMaxShared);
	if (e) return e;
	e = chain_launch(kern, (unsigned)nb, FTR_THREADS, smem, s, *linked, (const int4 *)U, (const int2 *)tau, combo_zbg,
	                 slices, nslice, cbase, ncombo, L, nzt, m_lo, nm, (int4 *)R);
	*linked = true;
	return e;
}

} // namespace

extern "C" {

int sxsk_fix_molecule(const double *flat, int Q, int L, int conj, double *sc, void *spf, cudaStream_t s)
{
	int K2 = (L + 1) * (L + 1), Qp = (Q + SXS_QT - 1) / SXS_QT * SXS_QT;
	k_fix_scale<<<Qp, 128, 0, s>>>(flat, Q, K2, Qp, sc);
	k_fix_spf<<<nblk(3L * Q * K2, 256), 256, 0, s>>>(flat, sc, Q, K2, Qp, conj, (int4 *)spf);
	return cudaGetLastError();
}

int sxsk_fix_dtab(const double *d, int2 *x, long n, cudaStream_t s)
{
	k_fix_dtab<<<nblk(n, 256), 256, 0, s>>>(d, x, n);
	return cudaGetLastError();
}

int sxsk_fix_nu(const double *bes, int nz, int Q, int L, double *nu2, cudaStream_t s)
{
	int Qp = (Q + SXS_QT - 1) / SXS_QT * SXS_QT;
	if (nz <= 0) return 0;
	if (L > SXSK_FIX_LMAX || (long)nz * Qp > 0x7fffffffL) return cudaErrorInvalidValue;
	k_fix_nu<<<(unsigned)(nz * Qp), 160, 0, s>>>(bes, Q, L, Qp, nu2);
	return cudaGetLastError();
}

int sxsk_fix_rotate(const void *spf, const int2 *dtab, const double2 *tw, int Q, int L, void *out, cudaStream_t s)
{
	/* gamma pairs per thread: L + 1 pairs over four groups */
	int need = (L + 1 + FROT_GROUPS - 1) / FROT_GROUPS;
	if (L < 1 || L > SXSK_FIX_LMAX || Q <= 0) return cudaErrorInvalidValue;
	if (need <= 2) return rotate_launch<2>(spf, dtab, tw, Q, L, out, s);
	if (need <= 3) return rotate_launch<3>(spf, dtab, tw, Q, L, out, s);
	if (need <= 4) return rotate_launch<4>(spf, dtab, tw, Q, L, out, s);
	if (need <= 5) return rotate_launch<5>(spf, dtab, tw, Q, L, out, s);
	if (need <= 6) return rotate_launch<6>(spf, dtab, tw, Q, L, out, s);
	return rotate_launch<8>(spf, dtab, tw, Q, L, out, s);
}

int sxsk_fix_translate(const void *U, const void *tau, const int32_t *combo_zbg, const int32_t *slices, int nslice,
                       int cbase, int ncombo, int nzt, int Q, int L, void *R, cudaStream_t s)
{
	if (nslice <= 0) return 0;
	if (L > SXSK_FIX_LMAX) return cudaErrorInvalidValue;
	int NT = (Q + SXS_QT - 1) / SXS_QT, e = 0;
	bool linked = false;
#define FTL(NB) \
	if (!e) e = translate_launch<NB>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, &linked, s);
	FTL(4) FTL(8) FTL(12) FTL(16) FTL(20) FTL(24) FTL(28) FTL(32)
#undef FTL
	return e;
}

int sxsk_fix_cross(const sxsk_pose *poses, int npose, int combo_base, int ncombo, const int32_t *combo_zbg,
                   const void *P, const void *R, const double2 *tw, const double *scA, const double *scB,
                   const double *nu2, const double *cst, int Q, int L, double *cross, cudaStream_t s)
{
	if (npose <= 0) return 0;
	int NT = (Q + SXS_QT - 1) / SXS_QT;
	long nb = (long)NT * ((npose + FPC_POSES - 1) / FPC_POSES);
	if (nb > 0x7fffffffL || L > SXSK_FIX_LMAX) return cudaErrorInvalidValue;
	k_fix_cross<<<(unsigned)nb, FPC_THREADS, 0, s>>>(poses, npose, combo_base, ncombo, combo_zbg, (const int4 *)P,
	                                                 (const int4 *)R, tw, scA, scB, nu2, NT * SXS_QT, cst, Q, L, cross);
	return cudaGetLastError();
}

} // extern "C"
