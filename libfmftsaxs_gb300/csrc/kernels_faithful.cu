/*
 * FP64 kernels whose rounding must follow the reference operation by
 * operation: the spherical-Bessel power series (its cancellation at large
 * q*r amplifies any reordering), the associated-Legendre recurrence, the
 * translation-matrix p-sum, the A_lm accumulation and the self terms.
 *
 * This translation unit is compiled with -fmad=false so that no multiply-add
 * is contracted: every expression below is evaluated in the reference's
 * order with one rounding per operation, as gcc -std=c11 does on the host.
 */
#include "kernels.h"
#include "limbs.cuh"

#include <math.h>

#define SXS_PI 3.14159265358 /* the reference's pi (src/define.h:14-16 under -std=c11) */

namespace {

__device__ __forceinline__ int lm_index(int l, int m) { return l * (l + 1) + m; }

/* (2l+1)!! as the reference's doublefact (src/sfbessel.c:21-37). */
__device__ double odd_factorial(int n)
{
	double r = 1.0;
	for (int i = 1; i <= n; i += 2) r *= (double)i;
	return r;
}

/* |Y_lm| <= sqrt((2l + 1) / 4 pi) < 2^y_exp(l) */
__device__ __forceinline__ int y_exp(int l) { return l == 0 ? -1 : (l < 6 ? 0 : (l < 25 ? 1 : 2)); }

/* Y_lm as 16 bytes: two doubles, or (fixed-point accumulation) the limbs {re h,
 * re l, im h, im l} of Y / 2^y_exp = (h 2^27 + l) 2^-54: a sum with 1.5 2^52
 * leaves the rounded integer in the low word, and the remainder is exact */
__device__ __forceinline__ void y_store(double2 *o, double re, double im, int) { *o = make_double2(re, im); }
__device__ __forceinline__ void y_store(int4 *o, double re, double im, int l)
{
	const double M = 6755399441055744.0, c = ldexp(1.0, 27 - y_exp(l));
	double a = __fma_rn(re, c, M), b = __fma_rn(im, c, M);
	double ar = __fma_rn(re, c, -(a - M)), br = __fma_rn(im, c, -(b - M));
	*o = make_int4(__double2loint(a), __double2loint(__fma_rn(ar, 134217728.0, M)), __double2loint(b),
	               __double2loint(__fma_rn(br, 134217728.0, M)));
}

#define YLM_ATOMS 16
#define YLM_THREADS 128

/* Per atom and m >= 0: P_l^m(cos theta) by the recurrence of
 * src/borrowed.c:40-65 (N = L+1), times the Y norm, times e^{-i m phi}
 * (src/pdb2spf.c:76-84), written for +m and -m.  Block = YLM_ATOMS atoms:
 * one thread per atom takes its angles, then threads take (atom, m); the
 * recurrence's quotients, which depend on (l, m) alone, are divided once per
 * block.  Bound by the FP64 pipe (3,500 atoms at L = 20: 0.40 ms with angles,
 * quotients and phase factors formed per (atom, m) or per l).  The radius of
 * an atom whose angles are not finite is written as NaN in the limb form,
 * which cannot hold its Y_lm. */
template <typename Y, bool LIMBS>
__global__ void __launch_bounds__(YLM_THREADS)
k_ylm(const double *__restrict__ xyz, int natoms, int L, const double *__restrict__ ynorm, Y *__restrict__ ylm,
      double *__restrict__ rad)
{
	extern __shared__ double2 quo[];           /* [L (L + 1) / 2]: (2l - 1) / (l - m), (l + m - 1) / (l - m) */
	__shared__ double ang[YLM_ATOMS][3];       /* cos theta, sin theta, phi */
	int K = L + 1, K2 = K * K, N = K;
	int a0 = blockIdx.x * YLM_ATOMS, na = min(YLM_ATOMS, natoms - a0);
	for (int i = threadIdx.x; i < K * K; i += YLM_THREADS) {
		int m = i / K, l = i % K;
		if (l > m + 1) quo[l * (l - 1) / 2 + m] = make_double2((2. * l - 1.) / (l - m), (l + m - 1.) / (l - m));
	}
	if (threadIdx.x < na) {
		int a = a0 + threadIdx.x;
		double x = xyz[3 * a], y = xyz[3 * a + 1], z = xyz[3 * a + 2];
		double r = sqrt(x * x + y * y + z * z);
		double th = acos(z / r);
		double ph;
		if (y > 0.0) ph = acos(x / sqrt(x * x + y * y));
		else ph = -acos(x / sqrt(x * x + y * y)) + 2.0 * SXS_PI;
		rad[a] = LIMBS && !(isfinite(th) && isfinite(ph)) ? nan("") : r;
		double c = cos(th);
		ang[threadIdx.x][0] = c;
		ang[threadIdx.x][1] = sqrt(1. - c * c);
		ang[threadIdx.x][2] = ph;
	}
	__syncthreads();
	for (int i = threadIdx.x; i < na * K; i += YLM_THREADS) {
		int m = i / na, ai = i % na;
		double c = ang[ai][0], s = ang[ai][1], ph = ang[ai][2];
		/* P_m^m: the reference's diagonal chain (lines 54 and 63 agree on the
		 * formula), then P_{m+1}^m and the upward recurrence in l. */
		double pmm = 1;
		for (int j = 1; j <= m; j++) pmm = -1. * (2. * j - 1.) * s * pmm;
		double p_lm2 = 0.0, p_lm1 = pmm;
		/* the phase factors do not depend on l; those of -m are the conjugates */
		double cp = cos(ph * m), sp = sin(-ph * m);
		Y *out = ylm + (size_t)(a0 + ai) * K2;
		for (int l = m; l < N; l++) {
			double p;
			if (l == m) {
				p = pmm;
			} else if (l == m + 1) {
				if (m == 0) p = c;                          /* P_1^0 = x */
				else p = (2. * m + 1.) * c * pmm;           /* P_{m+1}^m */
			} else {
				double2 f = quo[l * (l - 1) / 2 + m];
				p = f.x * c * p_lm1 - f.y * p_lm2;
			}
			p_lm2 = p_lm1;
			p_lm1 = p;
			if (l == m) { p_lm2 = 0.0; p_lm1 = p; }
			double hp = ynorm[l * (2 * L + 1) + (m + L)] * p;
			y_store(out + lm_index(l, m), hp * cp, hp * sp, l);
			if (m > 0) {
				double hn = ynorm[l * (2 * L + 1) + (-m + L)] * p;
				y_store(out + lm_index(l, -m), hn * cp, hn * -sp, l);
			}
		}
	}
}

/* series terms whose divisor (2k)(2k + 2l + 1) a block of k_expand_ql keeps
 * in a table for its l */
#define EXP_KTAB 128

/* a series divisor D, 2^(bits - 1) < D < 2^bits: itself and 1 / D rounded to
 * nearest, and inv = floor(2^(63 + bits) / D) */
struct SeriesDiv {
	double den, rcp;
	unsigned long long inv;
	int bits, pad;
};

__device__ __forceinline__ SeriesDiv series_div(int k, int l)
{
	SeriesDiv d;
	unsigned long long D = 2ull * k * (2ull * k + 2ull * l + 1ull);   /* never a power of two: it has an odd factor */
	d.den = (double)D;
	d.rcp = 1.0 / d.den;
	d.bits = 64 - __clzll((long long)D);
	unsigned long long q = (1ull << 63) / D, r = (1ull << 63) - q * D;
	for (int i = 0; i < d.bits; i++) {
		r <<= 1;
		q = 2 * q + (r >= D);
		if (r >= D) r -= D;
	}
	d.inv = q;
	d.pad = 0;
	return d;
}

/* num / den, correctly rounded, for an integer den > 0 with y = 1/den
 * rounded to nearest and |num| a normal number: q0 = num y, the remainder
 * num - den q0 exactly by an FMA, and one correction q0 + r y (Markstein's
 * final division step, P. Markstein, "Computation of elementary functions
 * on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34 (1990)): three
 * FP64 operations instead of a full division.  Checked against IEEE
 * division on 3.1e8 (num, den) pairs of this series' range with no
 * difference. */
__device__ __forceinline__ double div_by_int(double num, double den, double y)
{
	double q0 = num * y;
	double r = fma(-q0, den, num);
	return fma(r, y, q0);
}

/* -|num| / D, correctly rounded, in integers: mant = the 53-bit significand
 * of num at the top of 64 bits, en its exponent field.  R = floor(mant inv /
 * 2^64) is less than 2 below the quotient (scaled to [2^62, 2^64)), whose 53
 * leading bits are rounded to nearest; there are no ties (a quotient of a
 * 53-bit number by D has at most 53 bits or infinitely many), so only the
 * remainder one below the half is not decided (open). */
__device__ __forceinline__ double series_ratio(unsigned long long mant, int en, unsigned long long inv, int bits, bool &open)
{
	unsigned long long R = __umul64hi(mant, inv);
	int big = (int)(R >> 63), sh = 10 + big;
	unsigned half = 512u << big, low = (unsigned)R & (2 * half - 1);
	open = low == half - 1;
	unsigned long long S = (R >> sh) + (low >= half);
	return __longlong_as_double((long long)((((unsigned long long)(unsigned)(en - bits + big + 2047) << 52) + S)));
}

/* the rare exact forms, kept out of line so that no part of their divisions
 * is issued ahead of need */
__device__ __noinline__ bool series_goes_on(double term, double sum) { return fabs(term / sum) > 0.00001; }
__device__ __noinline__ double series_sum(int l, double x, double term0)
{
	double tl1 = 2.0 * (double)l + 1.0, term = term0, sum = term0;
	for (int k = 1; fabs(term / sum) > 0.00001 && k < 100000; k++) {
		double ratio = ((-1.0) * x * x) / ((2.0 * (double)k) * (2.0 * (double)k + tl1));
		term = term * ratio;
		sum = sum + term;
	}
	return sum;
}

/* The series of sbessel, x > 0, and the same sum: the same terms in the same
 * order, the product and the sum of each term on the FP64 pipe (2
 * operations of 73 clocks per warp and scheduler) and the rest beside it: the
 * ratio of consecutive terms, -x^2 / ((2k)(2k + 2l + 1)), in integers as above
 * with the block's table for k < EXP_KTAB, and the stop test fabs(term /
 * sum) > 1e-5 on the leading 20 bits of both (as floats relative to term0's
 * exponent), with the quotient only where those do not decide.  term0 = 1 /
 * (2l+1)!! is the block's.  Two or four series per thread at once measured
 * slower (registers). */
__device__ __forceinline__ double series_fast(int l, double x, double term0, const SeriesDiv *dk)
{
	double num = (-1.0) * x * x, term = term0, sum = term0;
	unsigned long long nb = (unsigned long long)__double_as_longlong(num);
	int en = (int)(nb >> 52) & 0x7ff;
	unsigned long long mant = (nb << 11) | 0x8000000000000000ull;
	int off = (__double2hiint(term0) & 0x7ff00000) - (127 << 20);
	bool slow = en <= 123 || en >= 1923;   /* |num| outside 2^+-900: quotients may be subnormal */
	for (int k = 1; !slow; k++) {
		int ht = (__double2hiint(term) & 0x7fffffff) - off, hs = (__double2hiint(sum) & 0x7fffffff) - off;
		float tf = __int_as_float(ht << 3), sf = __int_as_float(hs << 3) * 1e-5f;
		bool in = (unsigned)(ht - (20 << 20)) < (unsigned)(234 << 20) && (unsigned)(hs - (20 << 20)) < (unsigned)(234 << 20);
		if (in && tf < sf * 0.99999f) break;
		if (!(in && tf > sf * 1.00001f) && !series_goes_on(term, sum)) break;
		if (k == EXP_KTAB) {
			slow = true;
			break;
		}
		bool open;
		double ratio = series_ratio(mant, en, dk[k].inv, dk[k].bits, open);
		if (open) ratio = div_by_int(num, dk[k].den, dk[k].rcp);
		term = term * ratio;
		sum = sum + term;
	}
	return slow ? series_sum(l, x, term0) : sum;
}

/* j_l(x): x^l is formed by squaring (SQ) or as a chain of products, a few
 * ulps, outside the cancelling sum */
template <bool SQ>
__device__ __forceinline__ double sbessel_fast(int l, double x, double term0, const SeriesDiv *dk)
{
	if (!(x > 0.0)) return l == 0 ? 1.0 : 0.0;
	double sum = series_fast(l, x, term0, dk), xl = 1.0;
	if (SQ) {
		double b = x;
		for (int e = l; e; e >>= 1) {
			if (e & 1) xl = xl * b;
			if (e > 1) b = b * b;
		}
	} else {
		for (int i = 0; i < l; i++) xl = xl * x;
	}
	return sum * xl;
}

#define EXP_THREADS 128
/* atoms staged at a time by the fixed-point form: 512 products of its limbs
 * fit in 63 bits */
#define EXP_CHUNK 512

/* (double)v in two FP64 operations: each word under an exponent of its own */
__device__ __forceinline__ double to_double(long long v)
{
	double hi = __hiloint2double(0x45300000, (int)((unsigned)(v >> 32) ^ 0x80000000u));
	double lo = __hiloint2double(0x43300000, (int)(unsigned)v);
	return (hi - (0x1p84 + 0x1p63 + 0x1p52)) + lo;
}
/* 2^e for a normal result */
__device__ __forceinline__ double exp2i(int e)
{
	return __longlong_as_double((long long)(unsigned)(e + 1023) << 52);
}

/* 4 pi i^l times the sums of the block's (q, l): thread t < 2l + 1 writes m =
 * t - l of the three channels */
__device__ __forceinline__ void expand_write(double *spf, const double *v, int iq, int l, int t, int Q, int K2)
{
	const double fp = 4.0 * SXS_PI;
	double cre[4] = {fp, 0.0, -fp, 0.0}, cim[4] = {0.0, fp, 0.0, -fp};
	double c_r = cre[l % 4], c_i = cim[l % 4];
	size_t chs = (size_t)Q * K2 * 2;
	double *o = spf + ((size_t)iq * K2 + l * l + t) * 2;
	o[0] = c_r * v[0] - c_i * v[1];           o[1] = c_r * v[1] + c_i * v[0];
	o[chs] = c_r * v[2] - c_i * v[3];         o[chs + 1] = c_r * v[3] + c_i * v[2];
	o[2 * chs] = c_r * v[4] - c_i * v[5];     o[2 * chs + 1] = c_r * v[5] + c_i * v[4];
}

/* A[ch][q][l m] for one (q, l) per block: atoms in tiles of EXP_THREADS,
 * staged through shared memory as w_ch = f_ch(a) j_l(q r_a) (one series
 * per thread), then accumulated against Y*_lm(a) by (m, slice) threads,
 * each slice a fixed residue class of the tile's atoms; the slices are
 * summed in order and the 4 pi i^l phase applied (src/pdb2spf.c:104-147).
 * Deterministic: the same partition and order on every run.  The exact
 * scoring's L-BFGS-B fit runs on this form, whose last bits it would
 * amplify if they moved. */
__global__ void __launch_bounds__(EXP_THREADS) k_expand_ql(const double2 *__restrict__ ylm,
                                                            const double *__restrict__ rad,
                                                            const double *__restrict__ vac,
                                                            const double *__restrict__ dum,
                                                            const double *__restrict__ wfac, int natoms,
                                                            const double *__restrict__ q, int Q, int L,
                                                            double *__restrict__ spf)
{
	__shared__ double w[3][EXP_THREADS];
	__shared__ double red[EXP_THREADS][6];
	__shared__ SeriesDiv dk[EXP_KTAB];
	int K = L + 1, K2 = K * K;
	int iq = blockIdx.x / K, l = blockIdx.x % K;
	int nm = 2 * l + 1, nslice = EXP_THREADS / nm;
	int t = threadIdx.x;
	int mi = t % nm, sl = t / nm;
	bool acc_thread = sl < nslice;
	double qv = q[iq];
	double term0 = 1.0 / odd_factorial(2 * l + 1);
	for (int k = t; k < EXP_KTAB; k += blockDim.x)
		if (k) dk[k] = series_div(k, l);
	__syncthreads();
	double a6[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
	const double2 *yl = ylm + l * l;   /* this l's first (l, m) of every atom row */
	for (int a0 = 0; a0 < natoms; a0 += EXP_THREADS) {
		int a = a0 + t;
		if (a < natoms) {
			double j = sbessel_fast<false>(l, qv * rad[a], term0, dk);
			w[0][t] = vac[a] * j;
			w[1][t] = dum[a] * j;
			w[2][t] = wfac[a] * j;
		}
		__syncthreads();
		if (acc_thread) {
			int na = min(EXP_THREADS, natoms - a0);
			for (int k = sl; k < na; k += nslice) {
				double2 y = yl[(size_t)(a0 + k) * K2 + mi];
				double wv = w[0][k], wd = w[1][k], ww = w[2][k];
				a6[0] = fma(wv, y.x, a6[0]); a6[1] = fma(wv, y.y, a6[1]);
				a6[2] = fma(wd, y.x, a6[2]); a6[3] = fma(wd, y.y, a6[3]);
				a6[4] = fma(ww, y.x, a6[4]); a6[5] = fma(ww, y.y, a6[5]);
			}
		}
		__syncthreads();
	}
	if (acc_thread)
		for (int c = 0; c < 6; c++) red[t][c] = a6[c];
	__syncthreads();
	if (t < nm) {
		double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
		for (int sidx = 0; sidx < nslice; sidx++)
			for (int c = 0; c < 6; c++) v[c] = v[c] + red[sidx * nm + t][c];
		expand_write(spf, v, iq, l, t, Q, K2);
	}
}

__device__ __forceinline__ long long mad_wide(int a, int b, long long c)
{
	long long r;
	asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
	return r;
}

/* The same sums with the accumulation in fixed point, off the FP64 pipe,
 * which the series then has to itself.  Atoms in chunks of EXP_CHUNK: the
 * weights w_ch, scaled by the largest exponent in the chunk to 53-bit
 * integers h 2^27 + l, times the limbs of Y (h 2^27 + l, 54 bits) as three
 * 32 x 32 + 64-bit multiply-adds (h h', and h l' + l h'), sums exact; a
 * chunk's sums are added to the thread's in double.  A coefficient is accurate
 * relative to sum |f j_l| times the bound of |Y_lm|, not to its own size where
 * all Y_lm are small (large m, atoms near the z axis).  Bound by the FP64 pipe:
 * 2 operations per series term (8.4 terms on average, the longest of each
 * warp) and ~16 more per (atom, q, l), beside 18 IMAD.WIDE (~83 clocks) per
 * (atom, l, m); the FP64 form had 9 per term and 6 per (atom, l, m).  The
 * whole call (with k_ylm and one work buffer) 3,500 atoms, L = 20, Q = 101: 4.9
 * -> 1.43 ms; 8,000, L = 30, Q = 201: 36.2 -> 9.93; 4,909, L = 16, Q = 124:
 * 1.94.  NB, blocks per SM: 9 (56 registers) or, from L = EXP_NB10 on, 10 (48, more
 * spilled): 1.43 / 9.93 / 1.94 ms for these three with 9, 1.44 / 9.86 / 2.03 with
 * 10, 1.45 / 10.4 for the first two with 8. */
#define EXP_NB10 24
template <int NB>
__global__ void __launch_bounds__(EXP_THREADS, NB) k_expand_fix(const int4 *__restrict__ ylm,
                                                             const double *__restrict__ rad,
                                                             const double *__restrict__ vac,
                                                             const double *__restrict__ dum,
                                                             const double *__restrict__ wfac, int natoms,
                                                             const double *__restrict__ q, int Q, int L,
                                                             double *__restrict__ spf)
{
	__shared__ long long w[3][EXP_CHUNK];   /* the weights' bits, then their limbs; the slices' sums at the end */
	__shared__ SeriesDiv dk[EXP_KTAB];
	__shared__ int emax[3];
	int K = L + 1, K2 = K * K;
	int iq = blockIdx.x / K, l = blockIdx.x % K;
	int nm = 2 * l + 1, nslice = EXP_THREADS / nm;
	int t = threadIdx.x;
	int mi = t % nm, sl = t / nm;
	bool acc_thread = sl < nslice;
	double qv = q[iq];
	double term0 = 1.0 / odd_factorial(2 * l + 1);
	for (int k = t; k < EXP_KTAB; k += blockDim.x)
		if (k) dk[k] = series_div(k, l);
	if (t < 3) emax[t] = 0;
	__syncthreads();
	double a6[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
	const int4 *yl = ylm + l * l + mi;   /* this thread's (l, m) of every atom row */
	for (int a0 = 0; a0 < natoms; a0 += EXP_CHUNK) {
		int na = min(EXP_CHUNK, natoms - a0);
		int em[3] = {0, 0, 0};
		for (int k = t; k < na; k += EXP_THREADS) {
			int a = a0 + k;
			double r = rad[a], j = sbessel_fast<true>(l, qv * r, term0, dk);
			if (isnan(r)) j = r;
			double v[3] = {vac[a] * j, dum[a] * j, wfac[a] * j};
#pragma unroll
			for (int c = 0; c < 3; c++) {
				w[c][k] = __double_as_longlong(v[c]);
				em[c] = max(em[c], (__double2hiint(v[c]) >> 20) & 0x7ff);
			}
		}
#pragma unroll
		for (int c = 0; c < 3; c++) {
			int v = __reduce_max_sync(0xffffffffu, em[c]);
			if (t % 32 == 0) atomicMax(&emax[c], v);
		}
		__syncthreads();
		for (int c = 0; c < 3; c++) em[c] = max(emax[c], 1);
		/* w = M 2^(E - 1075) -> M >> (emax - E), rounded: unit 2^(emax - 1075);
		 * subnormal numbers have the exponent 1 without the leading bit */
		for (int k = t; k < na; k += EXP_THREADS)
#pragma unroll
			for (int c = 0; c < 3; c++) {
				long long b = w[c][k];
				int E = (int)(b >> 52) & 0x7ff, s = em[c] - max(E, 1);
				long long M = (b & 0xfffffffffffffll) | (E ? 0x10000000000000ll : 0);
				M = s > 53 ? 0 : (s > 0 ? (M + (1ll << (s - 1))) >> s : M);
				if (b < 0) M = -M;
				int h = (int)((M + (1ll << 26)) >> 27), lo = (int)((unsigned)M - ((unsigned)h << 27));
				w[c][k] = (long long)(((unsigned long long)(unsigned)lo << 32) | (unsigned)h);
			}
		__syncthreads();
		if (t < 3) emax[t] = 0;
		if (acc_thread) {
			long long hh[6] = {0, 0, 0, 0, 0, 0}, mid[6] = {0, 0, 0, 0, 0, 0};
			for (int k = sl; k < na; k += nslice) {
				int4 y = __ldg(yl + (size_t)(a0 + k) * K2);
#pragma unroll
				for (int c = 0; c < 3; c++) {
					long long b = w[c][k];
					int wh = (int)b, wl = (int)(b >> 32);
					hh[2 * c] = mad_wide(wh, y.x, hh[2 * c]);
					hh[2 * c + 1] = mad_wide(wh, y.z, hh[2 * c + 1]);
					mid[2 * c] = mad_wide(wh, y.y, mid[2 * c]);
					mid[2 * c + 1] = mad_wide(wh, y.w, mid[2 * c + 1]);
					mid[2 * c] = mad_wide(wl, y.x, mid[2 * c]);
					mid[2 * c + 1] = mad_wide(wl, y.z, mid[2 * c + 1]);
				}
			}
#pragma unroll
			for (int c = 0; c < 6; c++) {
				/* hh 2^54 + mid 2^27 in units of 2^(emax - 1075) 2^(y_exp - 54) */
				int e = em[c / 2], s2 = e - 1075 + y_exp(l);
				double v = to_double(hh[c] + ((mid[c] + (1 << 26)) >> 27));
				if (s2 > -1022) a6[c] = fma(v, e == 0x7ff ? nan("") : exp2i(s2), a6[c]);
				else a6[c] = a6[c] + v * exp2i(s2 + 512) * 0x1p-512;
			}
		}
		__syncthreads();
	}
	double *red = reinterpret_cast<double *>(&w[0][0]);   /* [EXP_THREADS][6] */
	if (acc_thread)
		for (int c = 0; c < 6; c++) red[t * 6 + c] = a6[c];
	__syncthreads();
	double *tot = red + EXP_THREADS * 6;                   /* [2l + 1][6] */
	for (int i = t; i < 6 * nm; i += EXP_THREADS) {
		double v = 0.0;
		for (int sidx = 0; sidx < nslice; sidx++) v = v + red[sidx * nm * 6 + i];
		tot[i] = v;
	}
	__syncthreads();
	if (t < nm) expand_write(spf, tot + 6 * t, iq, l, t, Q, K2);
}

/* bes[iz][p][q] = j_p(z q) (src/fftsaxs.c:110-121), q fastest: the
 * reference's truncated power series (src/sfbessel.c:40-60) times pow(x, p).
 * Block = one p and 128 (z, q), so that the series divisors are shared (0.077
 * -> 0.037 ms at L = 20, Q = 101, 16 z). */
__global__ void __launch_bounds__(128) k_bessel_z(const double *__restrict__ z, int nz, const double *__restrict__ q,
                                                  int Q, int L, double *__restrict__ bes)
{
	__shared__ SeriesDiv dk[EXP_KTAB];
	int N = 2 * L + 1, nb = (nz * Q + 127) / 128;
	int p = blockIdx.x / nb, t = blockIdx.x % nb * 128 + threadIdx.x;
	for (int k = threadIdx.x; k < EXP_KTAB; k += 128)
		if (k) dk[k] = series_div(k, p);
	double term0 = 1.0 / odd_factorial(2 * p + 1);
	__syncthreads();
	if (t >= nz * Q) return;
	int iq = t % Q, iz = t / Q;
	double x = z[iz] * q[iq];
	bes[((size_t)iz * N + p) * Q + iq] = x > 0.0 ? series_fast(p, x, term0, dk) * pow(x, (double)p) : (p == 0 ? 1.0 : 0.0);
}

/* forms of tau: double, float, and the limbs of tau / 2^nu (kernels_fixed.cu) */
__device__ __forceinline__ void tau_store(double *o, double v, double) { *o = v; }
__device__ __forceinline__ void tau_store(float *o, double v, double) { *o = (float)v; }
__device__ __forceinline__ void tau_store(int2 *o, double v, double c28) { *o = sxs_limbs(v, c28); }

/* sum over p = p0, p0 + 2, ..., p1 of +- dp[p] bp[p Q], the sign alternating
 * from neg: products and sums rounded one by one */
__device__ __forceinline__ double tm_sum(const double *dp, const double *bp, int Q, int p0, int p1, bool neg)
{
	double v = 0.0;
	for (int p = p0; p <= p1; p += 2) {
		double w = dp[p] * bp[(size_t)p * Q];
		v = neg ? v - w : v + w;
		neg = !neg;
	}
	return v;
}

/* What is stored as a float or as limbs is summed with fused multiply-adds
 * (half the operations of the FP64 pipe, which bounds the kernel).  With
 * n terms and partial sums of at most M the two sums differ by less than 4 n
 * 2^-53 M, for a term is the difference of two partial sums; a float is
 * therefore taken from the fused sum only if both ends of that interval
 * round to it, and else from tm_sum: the stored floats are those of tm_sum.
 * L = 30, Q = 201, 16 z: 1.69 -> 0.78 ms. */
__device__ __forceinline__ double tm_fused(const double *dp, const double *bp, int Q, int p0, int p1, bool neg, int &top)
{
	double v = 0.0;
	for (int p = p0; p <= p1; p += 2) {
		double d = dp[p];
		d = __hiloint2double(__double2hiint(d) ^ (neg ? 0x80000000 : 0), __double2loint(d));
		v = __fma_rn(d, bp[(size_t)p * Q], v);
		top = max(top, __double2hiint(v) & 0x7fffffff);
		neg = !neg;
	}
	return v;
}
__device__ __forceinline__ double tm_value(double *, const double *dp, const double *bp, int Q, int p0, int p1, bool neg)
{
	return tm_sum(dp, bp, Q, p0, p1, neg);
}
__device__ __forceinline__ double tm_value(int2 *, const double *dp, const double *bp, int Q, int p0, int p1, bool neg)
{
	int top = 0;
	return tm_fused(dp, bp, Q, p0, p1, neg, top);
}
__device__ __forceinline__ double tm_value(float *, const double *dp, const double *bp, int Q, int p0, int p1, bool neg)
{
	int top = 0;
	double v = tm_fused(dp, bp, Q, p0, p1, neg, top);
	/* M < the double whose high word is top + 1 */
	double d = __hiloint2double(top + 1, 0) * ((2 * (p1 - p0) + 4) * 0x1p-53);
	return (float)(v - d) == (float)(v + d) ? v : tm_sum(dp, bp, Q, p0, p1, neg);
}

/* T^{|m|}_{l l1}(q z) = sum_p (-1)^m i^p j_p d_lm(l1,p) for l <= l1, mirrored
 * (src/fftsaxs.c:182-243).  Thread = (iz, m, (m <= l, l1 >= l), q), q fastest;
 * nbx blocks per (iz, m), those past its pairs return at once.
 * Output in the q-tiled layout of the contraction tables (tiles of SXS_QT q,
 * zeros past Q), entries with l, l1 >= m only (no others are read).
 * The 3j factor 3j(l p l1; 0 0 0) vanishes unless l + p + l1 is even, so T
 * is real for even l + l1 and imaginary for odd l + l1 (the other part is
 * the sum of exact zeros and binary128 round-off below 1e-30 relative); the
 * table keeps that one real number, tau = Re T (even) or Im T (odd), in the
 * form that the run's translation reads.
 * The reference sums Re and Im with i^p in {1, i, -1, -i}; for the component
 * kept here the terms with p of the other parity add +-0, so summing only p
 * = l + l1 (mod 2), in the same order, gives the same value bit for bit; the
 * signs of (-1)^m and i^p are exact and turn the sum into alternate sums and
 * differences of the products: two FP64 operations per term (four with the
 * signs multiplied in), one where the sum is not stored as a double (tm_value).
 * Bound by that pipe (89 % busy).  16 z of the mixed path, with the float form
 * written here and not by a pass over a double table: 0.29 -> 0.14 ms at L =
 * 20, Q = 101, 2.43 -> 0.78 at L = 30, Q = 201. */
template <typename T>
__global__ void __launch_bounds__(128) k_tmatrix(const double *__restrict__ bes, const double *__restrict__ ds, int nz,
                                                 int Q, int L, const int2 *__restrict__ ll1, int nll1, int nbx,
                                                 const double *__restrict__ nu2, T *__restrict__ tau)
{
	int K = L + 1, N = 2 * L + 1, Qp = (Q + SXS_QT - 1) / SXS_QT * SXS_QT;
	int bx = blockIdx.x % nbx, zm = blockIdx.x / nbx;
	int m = zm % K, iz = zm / K;
	int j0 = m * K - m * (m - 1) / 2;         /* the pairs are in the order of l */
	int t = bx * 128 + threadIdx.x;
	if (t >= (nll1 - j0) * Qp) return;
	int iq = t % Qp;
	int2 pr = ll1[j0 + t / Qp];
	int l = pr.x, l1 = pr.y;
	double v = 0.0;
	if (iq < Q) {
		const double *dp = ds + ((size_t)lm_index(l, m) * K + l1) * N;
		const double *bp = bes + (size_t)iz * N * Q + iq;
		int p0 = l1 - l;                      /* |l - l1| with l <= l1, same parity as l + l1 */
		/* i^p: +1 (p % 4 == 0), -1 (2) for even p; the imaginary unit of i^p
		 * for odd p: +1 (1), -1 (3); so the sign alternates with p */
		bool neg = ((p0 & 2) != 0) != ((m & 1) != 0);
		v = tm_value(tau, dp, bp, Q, p0, l + l1, neg);
	}
	/* q-tiled: [tile][iz][m][l][l1][SXS_QT], tile = q / SXS_QT */
	size_t base = (((size_t)(iq / SXS_QT) * nz + iz) * K + m) * K;
	double c28 = nu2 ? 268435456.0 / nu2[(size_t)iz * Qp + iq] : 0.0;
	tau_store(tau + ((base + l) * K + l1) * SXS_QT + iq % SXS_QT, v, c28);
	tau_store(tau + ((base + l1) * K + l) * SXS_QT + iq % SXS_QT, v, c28);
}
/* Cross terms of single molecules (src/min_saxs.c:450-494): for each
 * molecule and q, sum over lm of |V|^2, |D|^2, |W|^2, Re(V conj D),
 * Re(V conj W), Re(D conj W) in the reference's order, the three mixed sums
 * doubled; spf in the host flat layout [mol][3][Q][K2][2], cross
 * [mol][6][Q] (VV VD VW DD DW WW).  Thread = (molecule, q). */
__global__ void k_self_cross(const double *__restrict__ spf, int nmol, int Q, int K2, double *__restrict__ cross)
{
	long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (t >= (long)nmol * Q) return;
	int iq = (int)(t % Q);
	long mol = t / Q;
	const double *V = spf + (((size_t)mol * 3 + 0) * Q + iq) * K2 * 2;
	const double *D = spf + (((size_t)mol * 3 + 1) * Q + iq) * K2 * 2;
	const double *W = spf + (((size_t)mol * 3 + 2) * Q + iq) * K2 * 2;
	double vv = 0.0, vd = 0.0, vw = 0.0, dd = 0.0, dw = 0.0, ww = 0.0;
	for (int id = 0; id < K2; id++) {
		double vr = V[2 * id], vi = V[2 * id + 1], dr = D[2 * id], di = D[2 * id + 1];
		double wr = W[2 * id], wi = W[2 * id + 1];
		vv += vr * vr + vi * vi;
		dd += dr * dr + di * di;
		ww += wr * wr + wi * wi;
		vd += vr * dr + vi * di;
		vw += vr * wr + vi * wi;
		dw += dr * wr + di * wi;
	}
	double *o = cross + (size_t)mol * 6 * Q + iq;
	o[0] = vv;
	o[Q] = vd * 2.0;
	o[2 * Q] = vw * 2.0;
	o[3 * Q] = dd;
	o[4 * Q] = dw * 2.0;
	o[5 * Q] = ww;
}

/* Shrake-Rupley accessible fraction (the restatement the workloads use;
 * the reference takes it from libmol2's accs): block = one atom i; the
 * block scans the atoms SASA_CAP at a time for neighbours j != i with
 * |x_i - x_j| < rr_i + rr_j (rr = radius + probe), keeps them in shared
 * memory, and each thread tests its sphere points p = x_i + rr_i s_k
 * against them (buried when |p - x_j|^2 < rr_j^2).  fraction = free points
 * / npts; 0 for a zero radius.  Compiled without contraction: the same
 * arithmetic as the host restatement, point for point. */
#define SASA_CAP 512
#define SASA_PPT 8
__global__ void __launch_bounds__(128) k_sasa(const double *__restrict__ xyz, const double *__restrict__ rad, int n,
                                              double probe, const double *__restrict__ sph, int npts,
                                              double *__restrict__ frac)
{
	__shared__ double nb[SASA_CAP][4];
	__shared__ int cnt;
	__shared__ int nfree[128];
	int i = blockIdx.x;
	double ri = rad[i];
	if (ri <= 0.0) {
		if (threadIdx.x == 0) frac[i] = 0.0;
		return;
	}
	double xi = xyz[3 * i], yi = xyz[3 * i + 1], zi = xyz[3 * i + 2];
	double rri = ri + probe;
	/* points of this thread: k = threadIdx.x + j blockDim.x, j < SASA_PPT */
	unsigned freebits = 0;
	for (int j = 0; j < SASA_PPT; j++)
		if (threadIdx.x + j * (int)blockDim.x < npts) freebits |= 1u << j;
	for (int j0 = 0; j0 < n; j0 += SASA_CAP) {
		__syncthreads();
		if (threadIdx.x == 0) cnt = 0;
		__syncthreads();
		int j1 = min(n, j0 + SASA_CAP);
		for (int j = j0 + threadIdx.x; j < j1; j += blockDim.x) {
			if (j == i) continue;
			double rrj = rad[j] + probe;
			double dx = xyz[3 * j] - xi, dy = xyz[3 * j + 1] - yi, dz = xyz[3 * j + 2] - zi;
			double d = sqrt(dx * dx + dy * dy + dz * dz);
			if (d < rri + rrj) {
				int slot = atomicAdd(&cnt, 1);   /* < SASA_CAP: at most SASA_CAP candidates per pass */
				nb[slot][0] = xyz[3 * j];
				nb[slot][1] = xyz[3 * j + 1];
				nb[slot][2] = xyz[3 * j + 2];
				nb[slot][3] = rrj * rrj;
			}
		}
		__syncthreads();
		int m = cnt;
		for (int pj = 0; pj < SASA_PPT; pj++) {
			if (!(freebits >> pj & 1u)) continue;
			int k = threadIdx.x + pj * blockDim.x;
			double px = xi + rri * sph[3 * k], py = yi + rri * sph[3 * k + 1], pz = zi + rri * sph[3 * k + 2];
			for (int t = 0; t < m; t++) {
				double ex = px - nb[t][0], ey = py - nb[t][1], ez = pz - nb[t][2];
				if (!(ex * ex + ey * ey + ez * ez >= nb[t][3])) {
					freebits &= ~(1u << pj);
					break;
				}
			}
		}
	}
	nfree[threadIdx.x] = __popc(freebits);
	__syncthreads();
	if (threadIdx.x == 0) {
		int c = 0;
		for (int t = 0; t < (int)blockDim.x; t++) c += nfree[t];
		frac[i] = (double)c / (double)npts;
	}
}

#define CI_CHUNK 256

/* Self terms of fill_const (src/fftsaxs.c:27-50, 52-85): per channel pair
 * and q, sum over lm of Re(A1 conj A2) then Re(B1 conj B2), interleaved as in
 * comp_const_int, times {1,2,2,1,2,1}.  spf in the host flat layout.  Block =
 * (channel pair, q): all threads form the terms, one adds them in the
 * reference's order.  0.043 ms at L = 20, Q = 101 (0.31 with a thread per sum
 * that also read and multiplied, all of it latency), 0.16 at L = 30, Q = 201
 * (0.67). */
__global__ void __launch_bounds__(128) k_const_int(const double *__restrict__ A, const double *__restrict__ B, int Q,
                                                   int L, double *__restrict__ cst)
{
	__shared__ double2 term[CI_CHUNK];
	int K2 = (L + 1) * (L + 1);
	int c = blockIdx.x / Q, iq = blockIdx.x % Q;
	const int pa[6] = {0, 0, 0, 1, 1, 2}, pb[6] = {0, 1, 2, 1, 2, 2};
	const double mul[6] = {1.0, 2.0, 2.0, 1.0, 2.0, 1.0};
	size_t chs = (size_t)Q * K2, at = (size_t)iq * K2;
	const double2 *A2 = reinterpret_cast<const double2 *>(A), *B2 = reinterpret_cast<const double2 *>(B);
	const double2 *a1 = A2 + pa[c] * chs + at, *a2 = A2 + pb[c] * chs + at;
	const double2 *b1 = B2 + pa[c] * chs + at, *b2 = B2 + pb[c] * chs + at;
	double s = 0.0;
	for (int i0 = 0; i0 < K2; i0 += CI_CHUNK) {
		int n = min(CI_CHUNK, K2 - i0);
		for (int i = threadIdx.x; i < n; i += blockDim.x) {
			double2 x = a1[i0 + i], y = a2[i0 + i], u = b1[i0 + i], v = b2[i0 + i];
			term[i] = make_double2(x.x * y.x + x.y * y.y, u.x * v.x + u.y * v.y);
		}
		__syncthreads();
		if (threadIdx.x == 0) {
#pragma unroll 8
			for (int i = 0; i < n; i++) {
				s += term[i].x;
				s += term[i].y;
			}
		}
		__syncthreads();
	}
	if (threadIdx.x == 0) cst[c * Q + iq] = s * mul[c];
}

inline int nblk(long n, int b) { return (int)((n + b - 1) / b); }

} // namespace

extern "C" {

size_t sxsk_expand_ws_ylm(int natoms, int L) { return (size_t)natoms * (L + 1) * (L + 1) * sizeof(double2); }
size_t sxsk_expand_ws_rad(int natoms) { return (size_t)natoms * sizeof(double); }

int sxsk_expand(const double *xyz, const double *vac, const double *dum, const double *wfac, int natoms,
                 const double *q, int Q, int L, const double *ynorm, double2 *ylm_ws, double *rad_ws,
                 double *spf_out, int fixed, cudaStream_t s)
{
	int K = L + 1;
	if (natoms <= 0) {
		cudaMemsetAsync(spf_out, 0, (size_t)3 * Q * K * K * 2 * sizeof(double), s);
		return cudaGetLastError();
	}
	if ((long)Q * K > 0x7fffffffL) return cudaErrorInvalidValue;
	size_t qsm = sizeof(double2) * (size_t)K * L / 2;   /* at most 29 KB (L = 60) */
	if (fixed) {
		k_ylm<int4, true><<<nblk(natoms, YLM_ATOMS), YLM_THREADS, qsm, s>>>(xyz, natoms, L, ynorm, (int4 *)ylm_ws, rad_ws);
		auto kern = L < EXP_NB10 ? k_expand_fix<9> : k_expand_fix<10>;
		kern<<<Q * K, EXP_THREADS, 0, s>>>((const int4 *)ylm_ws, rad_ws, vac, dum, wfac, natoms, q, Q, L, spf_out);
	} else {
		k_ylm<double2, false><<<nblk(natoms, YLM_ATOMS), YLM_THREADS, qsm, s>>>(xyz, natoms, L, ynorm, ylm_ws, rad_ws);
		k_expand_ql<<<Q * K, EXP_THREADS, 0, s>>>(ylm_ws, rad_ws, vac, dum, wfac, natoms, q, Q, L, spf_out);
	}
	return cudaGetLastError();
}

/* kernel launches of one sxsk_expand call with atoms */
int sxsk_expand_launches(void) { return 2; }

int sxsk_bessel_z(const double *z, int nz, const double *q, int Q, int L, double *bes, cudaStream_t s)
{
	long n = (long)nz * Q, nb = (n + 127) / 128 * (2 * L + 1);
	if (n == 0) return 0;
	if (n > 0x7fffff00L || nb > 0x7fffffffL) return cudaErrorInvalidValue;
	k_bessel_z<<<(unsigned)nb, 128, 0, s>>>(z, nz, q, Q, L, bes);
	return cudaGetLastError();
}

int sxsk_self_cross(const double *spf, int nmol, int Q, int L, double *cross, cudaStream_t s)
{
	long n = (long)nmol * Q;
	if (n <= 0) return 0;
	k_self_cross<<<nblk(n, 128), 128, 0, s>>>(spf, nmol, Q, (L + 1) * (L + 1), cross);
	return cudaGetLastError();
}

int sxsk_sasa(const double *xyz, const double *rad, int n, double probe, const double *sph, int npts, double *frac,
              cudaStream_t s)
{
	if (n <= 0) return 0;
	if (npts <= 0 || npts > 128 * SASA_PPT) return cudaErrorInvalidValue;
	k_sasa<<<n, 128, 0, s>>>(xyz, rad, n, probe, sph, npts, frac);
	return cudaGetLastError();
}

int sxsk_tmatrix(const double *bes, const double *dsymb, int nz, int Q, int L, const int2 *ll1, int nll1,
                 const double *nu2, void *tau, int form, cudaStream_t s)
{
	int K = L + 1, Qp = (Q + SXS_QT - 1) / SXS_QT * SXS_QT;
	long nbx = ((long)nll1 * Qp + 127) / 128, nb = nbx * nz * K;
	if (nb == 0) return 0;
	if (nb > 0x7fffffffL) return cudaErrorInvalidValue;
	if (form == SXSK_TAU_FP32)
		k_tmatrix<<<(unsigned)nb, 128, 0, s>>>(bes, dsymb, nz, Q, L, ll1, nll1, (int)nbx, nullptr, (float *)tau);
	else if (form == SXSK_TAU_FIXED)
		k_tmatrix<<<(unsigned)nb, 128, 0, s>>>(bes, dsymb, nz, Q, L, ll1, nll1, (int)nbx, nu2, (int2 *)tau);
	else
		k_tmatrix<<<(unsigned)nb, 128, 0, s>>>(bes, dsymb, nz, Q, L, ll1, nll1, (int)nbx, nullptr, (double *)tau);
	return cudaGetLastError();
}

int sxsk_const_int(const double *A, const double *B, int Q, int L, double *cst, cudaStream_t s)
{
	k_const_int<<<6 * Q, 128, 0, s>>>(A, B, Q, L, cst);
	return cudaGetLastError();
}

} // extern "C"

/* ------------------------------------------------------------------------
 * Expansion with no allocation (sxsg_expand_noalloc).
 *
 * For callers that must not allocate device memory themselves or through
 * this library: code that receives all device memory from a host
 * application's own pool, or runs where a (synchronising) cudaMalloc is not
 * allowed.  The work buffers of the expansion (Y_lm norms, Y_lm per atom,
 * j_l(q r) per atom) live in one file-scope device array of fixed size that
 * every GPU which loads this library keeps until the process exits.
 * ---------------------------------------------------------------------- */
#include <mutex>

#define SXS_NOALLOC_DOUBLES (8u * 1024u * 1024u) /* 64 MiB of doubles */
#define SXS_NOALLOC_LMAX 40

static __device__ __align__(256) double g_noalloc_scratch[SXS_NOALLOC_DOUBLES];

extern "C" void sxs_count_launches(int n);

/* The Y_lm normalisation table y[l][m + L] = sqrt((2l+1)/(4 pi) (l-m)!/(l+m)!),
 * times (-1)^m for -m, zero for |m| > l: the arithmetic of sxs_ynorm_host
 * (src/borrowed.c:19-38) in the same order with IEEE division and square
 * root, so both give the same bits.  One thread per l. */
__global__ void k_ynorm(int L, double *__restrict__ y)
{
	int l = blockIdx.x * blockDim.x + threadIdx.x;
	if (l > L) return;
	int N = 2 * L + 1;
	double *row = y + (size_t)l * N;
	for (int m = l + 1; m <= L; m++) {
		row[m + L] = 0.0;
		row[-m + L] = 0.0;
	}
	double fact = 1.;
	double tmp0 = __ddiv_rn(2 * l + 1., 4. * SXS_PI);
	for (int m = 0; m <= l; m++) {
		if (m > 0) fact = __dmul_rn(fact, (double)((l - m + 1) * (l + m)));
		double tmp = __dsqrt_rn(__ddiv_rn(tmp0, fact));
		double sgn = (m % 2 == 0) ? 1 : -1;
		row[m + L] = tmp;
		row[-m + L] = __dmul_rn(sgn, tmp);
	}
}

namespace {
std::mutex g_noalloc_lock;
double *g_noalloc_ptr[64]; /* device address of the scratch array, per device */
} // namespace

extern "C" int sxsg_expand_noalloc(const double *xyz, const double *vac, const double *dum, const double *water_w,
                                   int natoms, const double *q, int Q, int L, double *spf_out, void *stream)
{
	if (natoms < 0 || Q < 1 || Q > 4096 || L < 1 || L > SXS_NOALLOC_LMAX || !q || !spf_out ||
	    (natoms > 0 && (!xyz || !vac || !dum)))
		return -2;
	int K = L + 1, N = 2 * L + 1, K2 = K * K;
	/* layout in doubles: ynorm | Y_lm (complex) | radii | zero water weights */
	size_t off_y = ((size_t)K * N + 31) / 32 * 32;
	size_t off_r = off_y + ((size_t)natoms * K2 * 2 + 31) / 32 * 32;
	size_t off_w = off_r + ((size_t)natoms + 31) / 32 * 32;
	size_t need = off_w + (water_w ? 0 : (size_t)natoms);
	if (need > SXS_NOALLOC_DOUBLES) return -3;
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -4;
	double *base;
	{
		std::lock_guard<std::mutex> lk(g_noalloc_lock);
		if (!g_noalloc_ptr[dev]) {
			void *p = NULL;
			cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
			if (e != cudaSuccess || !p) return (int)(e != cudaSuccess ? e : cudaErrorInvalidSymbol);
			g_noalloc_ptr[dev] = (double *)p;
		}
		base = g_noalloc_ptr[dev];
	}
	cudaStream_t s = (cudaStream_t)stream;
	/* every call rewrites the norm table: a call with another L may have
	 * left other values there */
	k_ynorm<<<1, 64, 0, s>>>(L, base);
	cudaError_t e = cudaGetLastError();
	if (e != cudaSuccess) return (int)e;
	sxs_count_launches(1);
	const double *w = water_w;
	if (!w && natoms > 0) {
		/* no hydration shell: the weights must start at zero on every call */
		e = cudaMemsetAsync(base + off_w, 0, sizeof(double) * natoms, s);
		if (e != cudaSuccess) return (int)e;
		w = base + off_w;
	}
	int rc = sxsk_expand(xyz, vac, dum, w, natoms, q, Q, L, base, (double2 *)(base + off_y), base + off_r, spf_out, 1, s);
	sxs_count_launches(natoms > 0 ? sxsk_expand_launches() : 0);
	return rc;
}
