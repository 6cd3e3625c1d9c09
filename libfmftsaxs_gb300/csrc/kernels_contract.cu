/*
 * Contraction kernels of the factorized correlation, in FP64 (plain path)
 * or FP32 (mixed path); multiply-add fusion allowed.
 *
 * The reference evaluates, per touched (z, beta1, beta2) triple, the 6-channel
 * sums X[m,m1,m2] (src/fftsaxs.c:416-524) and then an angular DFT at each
 * listed cell (529-606 or FFTW).  Writing the DFT phase as a product of the
 * per-angle phases and moving each sum next to the angle it depends on gives,
 * for one listed pose (z, b1, b2, a2, g1, g2) and one q,
 *
 *   P^a[m,l](b1,g1) = sum_{m1} w^{m1' g1} d^l_{m m1}(beta_b1) A^a_{l m1}
 *   U^b[m,l1](b2,g2)= sum_{m2} w^{m2' g2} d^l1_{m m2}(beta_b2) conj(B^b_{l1 m2})
 *   R^b[m,l]        = sum_{l1>=|m|} conj(T^{|m|}_{l l1}(q z)) U^b[m,l1]
 *   F^{ab}          = sum_m w^{m' a2} sum_{l>=|m|} P^a[m,l] R^b[m,l]
 *
 * (w = the twiddle table, x' = x mod N), the reference's F with the same terms
 * regrouped.  A and B expand real densities, so A_{l,-m} = (-1)^{l+m}
 * conj(A_{lm}); with d^l_{-m,-m1} = (-1)^{m-m1} d^l_{m m1} and T real or
 * imaginary by the parity of l + l1 this gives P[-m,l] = (-1)^{l+m} conj(P[m,l])
 * and the same for U and R, so the m-sum is Re F = Re(w_0 G_0) +
 * 2 sum_{m>0} Re(w_m G_m) with G_m = sum_l P[m,l] R[m,l].  Only m >= 0 is
 * tabulated: pairs (m, l), m = 0..L, l = m..L, (L+1)(L+2)/2 of them.
 */
#include "kernels.h"
#include "chain.cuh"
#include "smem.cuh"

namespace {

template <typename S> struct Cx;
template <> struct Cx<double> { typedef double2 T; };
template <> struct Cx<float> { typedef float2 T; };

/* first pair of row m >= 0 */
__device__ __forceinline__ int psym(int m, int K) { return m * K - m * (m - 1) / 2; }

__device__ __forceinline__ void cfma(double2 &acc, double2 a, double2 b)
{
	acc.x = fma(a.x, b.x, acc.x);
	acc.x = fma(-a.y, b.y, acc.x);
	acc.y = fma(a.x, b.y, acc.y);
	acc.y = fma(a.y, b.x, acc.y);
}
__device__ __forceinline__ float fma_s(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_s(double a, double b, double c) { return fma(a, b, c); }
/* Roundings written out: the rotation, translation and per-pose code leaves
 * no multiply-add to the compiler to fuse or not, so every kernel that
 * inlines it (the single-dimer and the batched launches) computes the same
 * bits. */
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
template <typename V> __device__ __forceinline__ V zero2() { V v; v.x = 0; v.y = 0; return v; }
template <typename V> __device__ __forceinline__ V from2(double2 a) { V v; v.x = a.x; v.y = a.y; return v; }

/* [3][Q][K2][2] -> [3][K2][Q] complex */
template <typename S>
__global__ void k_spf_transpose(const double *__restrict__ flat, typename Cx<S>::T *__restrict__ t, int Q, int K2)
{
	typedef typename Cx<S>::T V;
	long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= 3L * Q * K2) return;
	int iq = (int)(i % Q);
	long r = i / Q;
	int lm = (int)(r % K2), ch = (int)(r / K2);
	const double *s = flat + (((size_t)ch * Q + iq) * K2 + lm) * 2;
	V v;
	v.x = (S)s[0];
	v.y = (S)s[1];
	t[i] = v;
}

/* Contraction tables are q-tiled: a tile holds QT = 8 consecutive q, and a
 * table row is stored as [tile][row][pair][ch][8], so the slice of one tile
 * (an eighth of the table at Q ~ 100) stays in L2 while the blocks of that
 * tile run, and each thread moves 2 adjacent q (16 or 32 bytes) per load. */

/* pairs per block of the slice translation kernel, poses per block of the
 * per-pose kernel: 128 threads of SXS_QP q pairs */
#define TR_PB (128 / SXS_QP)
#define PC_PPB (128 / SXS_QP)

template <typename S> struct Pair2 { typename Cx<S>::T a, b; };
__device__ __forceinline__ Pair2<float> ld2(const float2 *p)
{
	float4 v = *reinterpret_cast<const float4 *>(p);
	Pair2<float> r;
	r.a = make_float2(v.x, v.y);
	r.b = make_float2(v.z, v.w);
	return r;
}
__device__ __forceinline__ Pair2<double> ld2(const double2 *p)
{
	Pair2<double> r;
	r.a = p[0];
	r.b = p[1];
	return r;
}
/* L2 eviction policies for streamed (evict_first) and reused (evict_last) rows */
__device__ __forceinline__ uint64_t l2_policy(bool keep)
{
	uint64_t pol;
	if (keep) asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
	else asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
	return pol;
}
/* 16-byte load at p + OFF bytes with an L2 policy; the offset is an
 * immediate of the instruction, so loads off one base need no address
 * arithmetic of their own */
template <int OFF>
__device__ __forceinline__ Pair2<float> ld2_pol(const float2 *p, uint64_t pol)
{
	float4 v;
	asm("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4+%6], %5;"
	    : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
	    : "l"(p), "l"(pol), "n"(OFF));
	Pair2<float> r;
	r.a = make_float2(v.x, v.y);
	r.b = make_float2(v.z, v.w);
	return r;
}
template <int OFF>
__device__ __forceinline__ Pair2<double> ld2_pol(const double2 *p, uint64_t)
{
	return ld2(reinterpret_cast<const double2 *>(reinterpret_cast<const char *>(p) + OFF));
}
__device__ __forceinline__ void st2(float2 *p, float2 a, float2 b)
{
	*reinterpret_cast<float4 *>(p) = make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void st2(double2 *p, double2 a, double2 b)
{
	p[0] = a;
	p[1] = b;
}

/* Twiddle factors of the paired rotation sum, extended so that index
 * k + j m1 needs no wrap: entry k holds h+ = (tw[k] + tw[N-k])/2 and
 * h- = (tw[k] - tw[N-k])/2 (indices mod N).  The FP32 path keeps
 * (Re tw[k], Im tw[k]): with a conjugate-symmetric table h+ = Re tw and
 * h- = i Im tw; the reference's twiddles are symmetric to ~1e-11, far below
 * FP32 rounding.  The FP64 path keeps both complex halves exactly. */
template <typename S> struct RotTw;
template <> struct RotTw<float> { float2 cs; };
template <> struct RotTw<double> { double2 hp, hm; };
template <typename S> __device__ __forceinline__ RotTw<S> rot_tw(const double2 *tw, int k, int N);
template <> __device__ __forceinline__ RotTw<float> rot_tw<float>(const double2 *tw, int k, int N)
{
	double2 a = tw[k % N];
	RotTw<float> r;
	r.cs = make_float2((float)a.x, (float)a.y);
	return r;
}
template <> __device__ __forceinline__ RotTw<double> rot_tw<double>(const double2 *tw, int k, int N)
{
	int kk = k % N;
	double2 a = tw[kk], b = tw[(N - kk) % N];
	RotTw<double> r;
	r.hp = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y + b.y));
	r.hm = make_double2(0.5 * (a.x - b.x), 0.5 * (a.y - b.y));
	return r;
}
/* A += h+ S, B += h- D */
__device__ __forceinline__ void rot_acc(float2 &A, float2 &B, const RotTw<float> &h, float2 S, float2 D)
{
	A.x = fmaf(h.cs.x, S.x, A.x);
	A.y = fmaf(h.cs.x, S.y, A.y);
	B.x = fmaf(h.cs.y, D.x, B.x);   /* B = sum sin D; h- D = i B */
	B.y = fmaf(h.cs.y, D.y, B.y);
}
__device__ __forceinline__ void rot_acc(double2 &A, double2 &B, const RotTw<double> &h, double2 S, double2 D)
{
	cfma(A, h.hp, S);
	cfma(B, h.hm, D);
}
/* X(gamma) = y0 + A + (h- part), X(N - gamma) = y0 + A - (h- part) */
__device__ __forceinline__ void rot_out(float2 y0, float2 A, float2 B, float2 &xp, float2 &xm)
{
	float ax = add_rn(y0.x, A.x), ay = add_rn(y0.y, A.y);
	xp = make_float2(sub_rn(ax, B.y), add_rn(ay, B.x));
	xm = make_float2(add_rn(ax, B.y), sub_rn(ay, B.x));
}
__device__ __forceinline__ void rot_out(double2 y0, double2 A, double2 B, double2 &xp, double2 &xm)
{
	double ax = add_rn(y0.x, A.x), ay = add_rn(y0.y, A.y);
	xp = make_double2(add_rn(ax, B.x), add_rn(ay, B.y));
	xm = make_double2(sub_rn(ax, B.x), sub_rn(ay, B.y));
}

#define ROT_GROUPS 4
/* threads of a rotation block: ROT_GROUPS gamma groups x 3/CH channel groups x q */
#define ROT_THREADS(CH) (ROT_GROUPS * (3 / (CH)) * SXS_QT)

/* Rotation tables in the q-tiled layout:
 *   out[t][b*N+g][pair(m,l)][ch][q] = sum_{m1=-l..l} tw[(m1' g) mod N] d^l_{m m1}(beta_b) C[ch][l,m1][q]
 * (C = spf_t, conjugated when conj != 0).  With y(m1) = d^l_{m m1} C[l,m1],
 * S = y(m1) + y(-m1), D = y(m1) - y(-m1) and k = m1 g mod N, the terms of
 * m1 and -m1 at gamma g and N - g combine to
 *   X(g) = y(0) + sum_{m1>0} h+(k) S + h-(k) D,  X(N-g) = y(0) + sum h+(k) S - h-(k) D,
 * so each (m1 > 0, gamma pair) costs one S and one D product.
 * Block = (m, beta b, q tile t), blocks ordered m fastest so that the blocks
 * of one tile read the same coefficients from L1/L2; thread = (group of G
 * gamma pairs, CH channels, q): the thread forms S and D once per m1 and
 * channel and accumulates its G gamma pairs in registers; with CH = 3 one
 * twiddle load and index step serve the three channels.  The padding
 * q >= Q is written as zeros. */
/* the extended twiddles hs[ROT_NTW] of a rotation block (all threads) */
#define ROT_NTW(L, G) (2 * (L) + 1 + ((G) - 1) * (L))
template <typename S, int G>
__device__ __forceinline__ void rotate_stage(const double2 *__restrict__ tw, int L, RotTw<S> *hs)
{
	int N = 2 * L + 1, ne = ROT_NTW(L, G);
	for (int k = threadIdx.x; k < ne; k += blockDim.x) hs[k] = rot_tw<S>(tw, k, N);
}

/* one block of k_rotate: (m, beta b, q tile t), twiddles staged in hs */
template <typename S, int G, int CH>
__device__ __forceinline__ void rotate_block(const typename Cx<S>::T *__restrict__ spf_t, const S *__restrict__ dtab,
                                             const RotTw<S> *hs, int Q, int L, int conj,
                                             typename Cx<S>::T *__restrict__ out, int t, int b, int m)
{
	typedef typename Cx<S>::T V;
	int K = L + 1, N = 2 * L + 1, K2 = K * K, NP = K * (K + 1) / 2, nrow = K * N;
	int qq = threadIdx.x % SXS_QT;
	int ch0 = CH == 3 ? 0 : (threadIdx.x / SXS_QT) % 3;
	int gg = threadIdx.x / ((3 / CH) * SXS_QT);
	int q = t * SXS_QT + qq;
	bool qok = q < Q;
	int g0 = gg * G;
	if (g0 > L) return;
	S sg = conj ? (S)-1 : (S)1;
	const V *C = spf_t + (size_t)ch0 * K2 * Q + (qok ? q : 0);
	const S *db = dtab + ((size_t)b * K * N + m + L) * N + L;   /* d^l_{m m1}(beta_b) at l = 0, m1 = 0 */
	V *ob = out + (((size_t)t * nrow + (size_t)b * N) * NP + psym(m, K)) * 3 * SXS_QT + ch0 * SXS_QT + qq;
	size_t gstride = (size_t)NP * 3 * SXS_QT;
	size_t cstride = (size_t)K2 * Q;                     /* between channels of C */
	for (int l = m; l <= L; l++) {
		const S *dl = db + (size_t)l * N * N;
		const V *Cl = C + (size_t)l * (l + 1) * Q;    /* lm of m1 = 0 */
		S d0 = __ldg(dl), d0s = mul_rn(d0, sg);   /* the sign flips are exact */
		V y0[CH];
#pragma unroll
		for (int c = 0; c < CH; c++) {
			V c0 = zero2<V>();
			if (qok) c0 = __ldg(Cl + c * cstride);
			y0[c].x = mul_rn(d0, c0.x);
			y0[c].y = mul_rn(d0s, c0.y);
		}
		V A[G][CH], B[G][CH];
#pragma unroll
		for (int j = 0; j < G; j++)
#pragma unroll
			for (int c = 0; c < CH; c++) A[j][c] = B[j][c] = zero2<V>();
		int base = 0;                                  /* m1 g0 mod N */
		for (int m1 = 1; m1 <= l; m1++) {
			base += g0;
			if (base >= N) base -= N;
			S dp = __ldg(dl + m1), dm = __ldg(dl - m1);
			S dps = mul_rn(dp, sg), dms = mul_rn(dm, sg);
			V Sv[CH], Dv[CH];
#pragma unroll
			for (int c = 0; c < CH; c++) {
				V cp = zero2<V>(), cm = zero2<V>();
				if (qok) {
					cp = __ldg(Cl + c * cstride + (size_t)m1 * Q);
					cm = __ldg(Cl + c * cstride - (ptrdiff_t)m1 * Q);
				}
				/* S = y(m1) + y(-m1), D = y(m1) - y(-m1): y(-m1) rounded, y(m1)
				 * fused */
				S mx = mul_rn(dm, cm.x), my = mul_rn(dms, cm.y);
				Sv[c].x = fma_s(dp, cp.x, mx); Sv[c].y = fma_s(dps, cp.y, my);
				Dv[c].x = fma_s(dp, cp.x, -mx); Dv[c].y = fma_s(dps, cp.y, -my);
			}
			int k = base;
#pragma unroll
			for (int j = 0; j < G; j++) {
				RotTw<S> h = hs[k];
#pragma unroll
				for (int c = 0; c < CH; c++) rot_acc(A[j][c], B[j][c], h, Sv[c], Dv[c]);
				k += m1;
			}
		}
		V *o = ob + (size_t)(l - m) * 3 * SXS_QT;
#pragma unroll
		for (int j = 0; j < G; j++) {
			int g = g0 + j;
			if (g > L) break;
#pragma unroll
			for (int c = 0; c < CH; c++) {
				V xp, xm;
				rot_out(y0[c], A[j][c], B[j][c], xp, xm);
				o[(size_t)g * gstride + c * SXS_QT] = xp;
				if (g > 0) o[(size_t)(N - g) * gstride + c * SXS_QT] = xm;
			}
		}
	}
}

/* The FP32 rotation from 8 gamma pairs per thread on (L >= 24).  Block = (m,
 * two beta b0 and b0 + 1, q tile t); thread = (beta, group of G gamma pairs,
 * channel, 2 adjacent q).  Per l the block forms S and D of every m1 once, in
 * shared memory, for its four gamma groups (each group formed its own
 * before, waiting for the coefficients: 2.8 of 6.7 stall cycles per
 * instruction), and a twiddle load serves 8 multiply-adds instead of 4: the
 * kernel is bound by shared-memory wavefronts, 24 per 64 multiply-adds of a
 * warp (22 per 32 before).  2.73 -> 2.32 ms at L = 30, Q = 201 (staging 0.6,
 * stores 0.1), 0.73 -> 0.61 at L = 25, Q = 101; six blocks per SM instead of
 * the registers' five 2.50, seven 5.2 (spills).  The sums are those of
 * rotate_block, bit for bit.  sd: the block's 2 L 24 staged entries. */
#define ROT2_G 8
#define ROT2_THREADS (2 * ROT_GROUPS * 3 * SXS_QP)
#define ROT2_SMEM(L) (sizeof(float4) * 2 * (size_t)(L) * 3 * SXS_QT)
template <int G>
__device__ __forceinline__ void rotate2_block(const float2 *__restrict__ spf_t, const float *__restrict__ dtab,
                                              const RotTw<float> *hs, float4 *sd, int Q, int L, int conj,
                                              float2 *__restrict__ out, int t, int b0, int m)
{
	int K = L + 1, N = 2 * L + 1, K2 = K * K, NP = K * (K + 1) / 2, nrow = K * N;
	float sg = conj ? -1.0f : 1.0f;
	int sq = threadIdx.x % SXS_QT, sc = threadIdx.x / SXS_QT % 3, sr = threadIdx.x / (3 * SXS_QT);   /* staging */
	int j2 = 2 * (threadIdx.x % SXS_QP), ch = threadIdx.x / SXS_QP % 3;
	int gg = threadIdx.x / (3 * SXS_QP) % ROT_GROUPS, bb = threadIdx.x / (3 * SXS_QP * ROT_GROUPS);
	int g0 = gg * G, b = b0 + bb;
	bool act = b < K && g0 <= L, sok = t * SXS_QT + sq < Q;
	const float *db = dtab + ((size_t)b0 * K * N + m + L) * N + L;   /* d^l_{m m1}(beta_b0) at l = 0, m1 = 0 */
	size_t bstride = (size_t)K * N * N;                              /* between beta */
	const float2 *Cs = spf_t + (size_t)sc * K2 * Q + (sok ? t * SXS_QT + sq : 0);
	const float2 *C0 = spf_t + (size_t)ch * K2 * Q + t * SXS_QT + j2;
	bool qa = t * SXS_QT + j2 < Q, qb = t * SXS_QT + j2 + 1 < Q;
	float2 *ob = out + (((size_t)t * nrow + (size_t)b * N) * NP + psym(m, K)) * 3 * SXS_QT + ch * SXS_QT + j2;
	size_t gstride = (size_t)NP * 3 * SXS_QT;
	for (int l = m; l <= L; l++) {
		const float *dl = db + (size_t)l * N * N;
		const float2 *Cl = Cs + (size_t)l * (l + 1) * Q;             /* lm of m1 = 0 */
		for (int r = sr; r < 2 * l; r += ROT2_THREADS / (3 * SXS_QT)) {
			int ib = r >= l, m1 = r - (ib ? l : 0) + 1;
			if (b0 + ib >= K) break;
			float dp = __ldg(dl + ib * bstride + m1), dm = __ldg(dl + ib * bstride - m1);
			float dps = mul_rn(dp, sg), dms = mul_rn(dm, sg);
			float2 cp = zero2<float2>(), cm = zero2<float2>();
			if (sok) {
				cp = __ldg(Cl + (size_t)m1 * Q);
				cm = __ldg(Cl - (ptrdiff_t)m1 * Q);
			}
			float mx = mul_rn(dm, cm.x), my = mul_rn(dms, cm.y);
			sd[(r * 3 + sc) * SXS_QT + sq] = make_float4(fmaf(dp, cp.x, mx), fmaf(dps, cp.y, my), fmaf(dp, cp.x, -mx),
			                                             fmaf(dps, cp.y, -my));
		}
		__syncthreads();
		if (act) {
			float d0 = __ldg(dl + bb * bstride), d0s = mul_rn(d0, sg);
			const float2 *c0 = C0 + (size_t)l * (l + 1) * Q;
			float2 ca = qa ? __ldg(c0) : zero2<float2>(), cb = qb ? __ldg(c0 + 1) : zero2<float2>();
			float2 ya = make_float2(mul_rn(d0, ca.x), mul_rn(d0s, ca.y)), yb = make_float2(mul_rn(d0, cb.x), mul_rn(d0s, cb.y));
			float2 Aa[G], Ba[G], Ab[G], Bb[G];
#pragma unroll
			for (int j = 0; j < G; j++) Aa[j] = Ba[j] = Ab[j] = Bb[j] = zero2<float2>();
			int base = 0;                                        /* m1 g0 mod N */
			const float4 *sp = sd + ((size_t)bb * l * 3 + ch) * SXS_QT + j2;
			for (int m1 = 1; m1 <= l; m1++, sp += 3 * SXS_QT) {
				base += g0;
				if (base >= N) base -= N;
				float4 va = sp[0], vb = sp[1];
				float2 Sa = make_float2(va.x, va.y), Da = make_float2(va.z, va.w);
				float2 Sb = make_float2(vb.x, vb.y), Db = make_float2(vb.z, vb.w);
				int k = base;
#pragma unroll
				for (int j = 0; j < G; j++) {
					RotTw<float> h = hs[k];
					rot_acc(Aa[j], Ba[j], h, Sa, Da);
					rot_acc(Ab[j], Bb[j], h, Sb, Db);
					k += m1;
				}
			}
			float2 *o = ob + (size_t)(l - m) * 3 * SXS_QT;
#pragma unroll
			for (int j = 0; j < G; j++) {
				int g = g0 + j;
				if (g > L) break;
				float2 pa, ma, pb, mb;
				rot_out(ya, Aa[j], Ba[j], pa, ma);
				rot_out(yb, Ab[j], Bb[j], pb, mb);
				st2(o + (size_t)g * gstride, pa, pb);
				if (g > 0) st2(o + (size_t)(N - g) * gstride, ma, mb);
			}
		}
		__syncthreads();
	}
}

template <int G>
__global__ void __launch_bounds__(ROT2_THREADS)
k_rotate2(const float2 *__restrict__ spf_t, const float *__restrict__ dtab, const double2 *__restrict__ tw, int Q, int L,
          int conj, float2 *__restrict__ out)
{
	extern __shared__ __align__(16) unsigned char rsm_raw[];
	float4 *sd = reinterpret_cast<float4 *>(rsm_raw);
	RotTw<float> *hs = reinterpret_cast<RotTw<float> *>(rsm_raw + ROT2_SMEM(L));   /* [N + (G-1) L] */
	int K = L + 1, nb2 = (K + 1) / 2;
	int bid = blockIdx.x;
	int m = bid % K;
	bid /= K;
	int b0 = 2 * (bid % nb2), t = bid / nb2;
	rotate_stage<float, G>(tw, L, hs);
	__syncthreads();
	rotate2_block<G>(spf_t, dtab, hs, sd, Q, L, conj, out, t, b0, m);
}

template <typename S, int G, int CH>
__global__ void __launch_bounds__(ROT_THREADS(CH))
k_rotate(const typename Cx<S>::T *__restrict__ spf_t, const S *__restrict__ dtab, const double2 *__restrict__ tw,
         int Q, int L, int conj, typename Cx<S>::T *__restrict__ out)
{
	extern __shared__ __align__(16) unsigned char rsm_raw[];
	RotTw<S> *hs = reinterpret_cast<RotTw<S> *>(rsm_raw);   /* [N + (G-1) L] */
	int K = L + 1;
	int bid = blockIdx.x;
	int m = bid % K;
	bid /= K;
	int b = bid % K;
	int t = bid / K;
	rotate_stage<S, G>(tw, L, hs);
	__syncthreads();
	rotate_block<S, G, CH>(spf_t, dtab, hs, Q, L, conj, out, t, b, m);
}

/* The work items of a block of a batched kernel:
 *   for (it = item_begin(..); it < nitems; it = item_advance(..)) {
 *           nxt = item_claim(ctr); ...work on item it... }
 * Persistent launch (ctr != NULL): unclaimed items in order; thread 0
 * claims the next one through the counter when the block starts on the
 * current one, so the atomic's round trip overlaps the work, and publishes
 * it after a barrier (every thread is done with the current item).  One
 * block per item (ctr == NULL): item blockIdx.x, then none. */
__device__ __forceinline__ int item_begin(int *ctr, int *s_it)
{
	if (!ctr) return (int)blockIdx.x;
	if (threadIdx.x == 0) *s_it = atomicAdd(ctr, 1);
	__syncthreads();
	return *s_it;
}
__device__ __forceinline__ int item_claim(int *ctr) { return ctr && threadIdx.x == 0 ? atomicAdd(ctr, 1) : 0; }
__device__ __forceinline__ int item_advance(int *ctr, int *s_it, int nxt, int nitems)
{
	if (!ctr) return nitems;
	__syncthreads();
	if (threadIdx.x == 0) *s_it = nxt;
	__syncthreads();
	return *s_it;
}

/* rotation blocks of many tables (mixed path); the twiddles are restaged
 * when an item's table has other ones than the previous item's */
template <int G>
__global__ void __launch_bounds__(G >= ROT2_G ? ROT2_THREADS : ROT_THREADS(3))
k_rotate_batch(const sxsk_rot_job *__restrict__ jobs, const int4 *__restrict__ items, int nitems, int tw_max, int *ctr)
{
	extern __shared__ __align__(16) unsigned char rsm_raw[];
	RotTw<float> *hs = reinterpret_cast<RotTw<float> *>(rsm_raw);
	float4 *sd = reinterpret_cast<float4 *>(rsm_raw + (sizeof(RotTw<float>) * tw_max + 15) / 16 * 16);
	const double2 *cur = nullptr;
	int curL = -1;
	__shared__ int s_it;
	int nxt = 0;
	for (int it = item_begin(ctr, &s_it); it < nitems; it = item_advance(ctr, &s_it, nxt, nitems)) {
		nxt = item_claim(ctr);
		int4 w = items[it];
		sxsk_rot_job j = jobs[w.x];
		if (j.tw != cur || j.L != curL) {
			rotate_stage<float, G>(j.tw, j.L, hs);
			__syncthreads();
			cur = j.tw;
			curL = j.L;
		}
		if constexpr (G >= ROT2_G)
			rotate2_block<G>((const float2 *)j.spf_t, (const float *)j.dtab, hs, sd, j.Q, j.L, j.conj, (float2 *)j.out, w.y,
			                 w.z, w.w);
		else
			rotate_block<float, G, 3>((const float2 *)j.spf_t, (const float *)j.dtab, hs, j.Q, j.L, j.conj,
			                          (float2 *)j.out, w.y, w.z, w.w);
	}
}

/* Translated ligand rows, q-tiled:
 * R[tile][c][pair(m,l)][ch][8] = sum_{l1>=m} conj(T^m_{l l1}) U[tile][(b2,g2)][pair(m,l1)][ch][8],
 * conj(T) U = tau U for even l + l1 and tau (-i U) for odd.
 * Block = (tile, slice of combos sharing one z, TR_PB consecutive pairs);
 * thread = (pair, 2 adjacent q).  The block stages the tau rows of its 32
 * pairs (the same for every combo of the slice) in shared memory once, then
 * streams the slice's U rows: each thread accumulates its pair for the 3
 * channels and 2 q.  Threads of a warp with the same m read the same U
 * entries (broadcast).  Blocks are ordered tile-major. */
template <typename S>
__global__ void __launch_bounds__(128)
k_translate(const typename Cx<S>::T *__restrict__ U, const S *__restrict__ tau, const int32_t *__restrict__ combo_zbg,
            const int32_t *__restrict__ slices, int nslice, int cbase, int ncombo, int L, int nzt, int tstride,
            typename Cx<S>::T *__restrict__ R)
{
	typedef typename Cx<S>::T V;
	extern __shared__ __align__(16) unsigned char tsm_raw[];
	S *ts = reinterpret_cast<S *>(tsm_raw);   /* [TR_PB pairs][tstride]: tau[l1][QT q] of each pair */
	int K = L + 1, N = 2 * L + 1, NP = K * (K + 1) / 2, nrow = K * N;
	int npb = (NP + TR_PB - 1) / TR_PB;
	int bid = blockIdx.x;
	int pb = bid % npb;
	bid /= npb;
	int si = bid % nslice, t = bid / nslice;
	int cfirst = slices[2 * si] - cbase, nc = slices[2 * si + 1];
	int zi = combo_zbg[3 * cfirst];
	for (int k = threadIdx.x; k < TR_PB * K * SXS_QT; k += blockDim.x) {
		int pl = k / (K * SXS_QT), r = k % (K * SXS_QT);
		int l1 = r / SXS_QT, qq = r % SXS_QT;
		int pr = pb * TR_PB + pl;
		S v = 0;
		if (pr < NP) {
			int m = 0;
			while (pr >= psym(m + 1, K)) m++;
			int l = m + pr - psym(m, K);
			if (l1 >= m) v = tau[(((((size_t)t * nzt + zi) * K + m) * K + l) * K + l1) * SXS_QT + qq];
		}
		ts[pl * tstride + r] = v;
	}
	__syncthreads();
	int pl = threadIdx.x / SXS_QP, j2 = 2 * (threadIdx.x % SXS_QP);
	int pr = pb * TR_PB + pl;
	if (pr >= NP) return;
	int m = 0;
	while (pr >= psym(m + 1, K)) m++;
	int l = m + pr - psym(m, K);
	const S *tp = ts + pl * tstride + j2;
	int po = psym(m, K);
	for (int c = cfirst; c < cfirst + nc; c++) {
		int b2 = combo_zbg[3 * c + 1], g2 = combo_zbg[3 * c + 2];
		const V *Ub = U + (((size_t)t * nrow + b2 * N + g2) * NP + po) * 3 * SXS_QT + j2;
		/* sums over l1 = m, m+2, ... (e) and m+1, m+3, ... (o): the terms of
		 * the class with l + l1 even add tau U, the other tau (-i U), so the
		 * loop needs no per-thread branch */
		V ae[3][2], ao[3][2];
#pragma unroll
		for (int ch = 0; ch < 3; ch++) ae[ch][0] = ae[ch][1] = ao[ch][0] = ao[ch][1] = zero2<V>();
		for (int l1 = m; l1 <= L; l1 += 2) {
			const V *u = Ub + (size_t)(l1 - m) * 3 * SXS_QT;
			S t0 = tp[l1 * SXS_QT], t1 = tp[l1 * SXS_QT + 1];
#pragma unroll
			for (int ch = 0; ch < 3; ch++) {
				Pair2<S> uv = ld2(u + ch * SXS_QT);
				ae[ch][0].x += t0 * uv.a.x; ae[ch][0].y += t0 * uv.a.y;
				ae[ch][1].x += t1 * uv.b.x; ae[ch][1].y += t1 * uv.b.y;
			}
			if (l1 + 1 <= L) {
				u += 3 * SXS_QT;
				t0 = tp[(l1 + 1) * SXS_QT];
				t1 = tp[(l1 + 1) * SXS_QT + 1];
#pragma unroll
				for (int ch = 0; ch < 3; ch++) {
					Pair2<S> uv = ld2(u + ch * SXS_QT);
					ao[ch][0].x += t0 * uv.a.x; ao[ch][0].y += t0 * uv.a.y;
					ao[ch][1].x += t1 * uv.b.x; ao[ch][1].y += t1 * uv.b.y;
				}
			}
		}
		bool even = ((l + m) & 1) == 0;   /* class e has l + l1 even */
		V *o = R + (((size_t)t * ncombo + c) * NP + pr) * 3 * SXS_QT + j2;
#pragma unroll
		for (int ch = 0; ch < 3; ch++) {
			V r[2];
#pragma unroll
			for (int k = 0; k < 2; k++) {
				V a = even ? ae[ch][k] : ao[ch][k], b = even ? ao[ch][k] : ae[ch][k];
				r[k].x = a.x + b.y;        /* a + (-i) b */
				r[k].y = a.y - b.x;
			}
			st2(o + ch * SXS_QT, r[0], r[1]);
		}
	}
}

__device__ __forceinline__ void ld4(const float *p, float *v)
{
	float4 x = *reinterpret_cast<const float4 *>(p);
	v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void ld4(const double *p, double *v)
{
	double2 x = *reinterpret_cast<const double2 *>(p), y = *reinterpret_cast<const double2 *>(p + 2);
	v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
}

/* one output row of the column form for CH channels: sum_k tau[k] x
 * (U[k] for even i + k, -i U[k] for odd), with the parity of the row i
 * given as PAR; one tau load serves the CH channels */
template <int PAR, int CH, typename S, typename V, int NB>
__device__ __forceinline__ void tcol_row(const S *row, const V (&u)[CH][NB], V (&acc)[CH])
{
#pragma unroll
	for (int j = 0; j < CH; j++) acc[j] = zero2<V>();
#pragma unroll
	for (int k4 = 0; k4 < NB; k4 += 4) {
		S tv[4];
		ld4(row + k4, tv);
#pragma unroll
		for (int kk = 0; kk < 4; kk++) {
			int k = k4 + kk;
#pragma unroll
			for (int j = 0; j < CH; j++) {
				if ((k & 1) == PAR) {
					acc[j].x = fma_s(tv[kk], u[j][k].x, acc[j].x);
					acc[j].y = fma_s(tv[kk], u[j][k].y, acc[j].y);
				} else {
					acc[j].x = fma_s(tv[kk], u[j][k].y, acc[j].x);
					acc[j].y = fma_s(-tv[kk], u[j][k].x, acc[j].y);
				}
			}
		}
	}
}

/* threads of the column kernel: SXS_SLICE combos x 3/CH channel groups x q */
#define TCOL_THREADS(CH) (SXS_SLICE * (3 / (CH)) * SXS_QT)

/* Column form of the translation, for L < 32: a thread owns the columns
 * (combo c, CH channels from ch0, q) of one m; it holds
 * U[c][pair(m, m+k)][ch][q], k < n = L + 1 - m, in registers (NB = n
 * rounded up to 4, unrolled) and applies the n x n matrix tau^m(q z) staged
 * in shared memory:
 *   R[c][pair(m, m+i)][ch][q] = sum_k tau[i][k] (U[k] or -i U[k] by the
 *   parity of i + k).
 * Block = (tile, slice of <= SXS_SLICE combos sharing z, m); tau rows are
 * padded so the 8 q start on distinct banks and read as float4/double2
 * chunks that lanes of the same q share.  One launch per NB covers the m
 * with n in (NB - 4, NB].  The FP64 path runs it with CH = 1 (bound by the
 * FP64 pipe); FP32 runs the pipelined three-channel form below, since a
 * 128-bit shared load costs four wavefronts even as a broadcast and one
 * channel per tau load leaves the L1 data pipe ahead of the FMA rate. */
template <typename S, int NB, int CH>
__global__ void __launch_bounds__(TCOL_THREADS(CH), 1)
k_translate_col(const typename Cx<S>::T *__restrict__ U, const S *__restrict__ tau,
                const int32_t *__restrict__ combo_zbg, const int32_t *__restrict__ slices, int nslice, int cbase,
                int ncombo, int L, int nzt, int m_lo, int nm, typename Cx<S>::T *__restrict__ R)
{
	typedef typename Cx<S>::T V;
	extern __shared__ __align__(16) unsigned char tcs_raw[];
	S *ts = reinterpret_cast<S *>(tcs_raw);   /* [8 q][NB i][NB k] (+ pad per q) */
	const int qstride = NB * NB + 4;
	int K = L + 1, N = 2 * L + 1, NP = K * (K + 1) / 2, nrow = K * N;
	int bid = blockIdx.x;
	int mi = bid % nm;
	bid /= nm;
	int si = bid % nslice, t = bid / nslice;
	int m = m_lo + mi, n = K - m;
	int cfirst = slices[2 * si] - cbase, nc = slices[2 * si + 1];
	int zi = combo_zbg[3 * cfirst];
	const S *tz = tau + ((((size_t)t * nzt + zi) * K + m) * K) * K * SXS_QT;
	for (int k = threadIdx.x; k < SXS_QT * NB * NB; k += blockDim.x) {
		int q = k % SXS_QT, r = k / SXS_QT;
		int i = r / NB, kk = r % NB;
		S v = 0;
		if (i < n && kk < n) v = tz[((size_t)(m + i) * K + m + kk) * SXS_QT + q];
		ts[q * qstride + i * NB + kk] = v;
	}
	__syncthreads();
	int q = threadIdx.x % SXS_QT;
	int ch0 = CH == 3 ? 0 : (threadIdx.x / SXS_QT) % 3;
	int cl = threadIdx.x / (SXS_QT * (3 / CH));
	if (cl >= nc) return;
	int c = cfirst + cl;
	int b2 = combo_zbg[3 * c + 1], g2 = combo_zbg[3 * c + 2];
	int po = psym(m, K);
	const V *Ub = U + (((size_t)t * nrow + b2 * N + g2) * NP + po) * 3 * SXS_QT + ch0 * SXS_QT + q;
	V u[CH][NB];
#pragma unroll
	for (int j = 0; j < CH; j++)
#pragma unroll
		for (int k = 0; k < NB; k++) u[j][k] = k < n ? Ub[(size_t)k * 3 * SXS_QT + j * SXS_QT] : zero2<V>();
	const S *tq = ts + q * qstride;
	V *Rb = R + (((size_t)t * ncombo + c) * NP + po) * 3 * SXS_QT + ch0 * SXS_QT + q;
	/* rows in even/odd pairs so that the parity of i + k is known at
	 * compile time: every (k, channel) is two FMAs */
	for (int i = 0; i < n; i += 2) {
		V a[CH];
		tcol_row<0, CH, S, V, NB>(tq + i * NB, u, a);
#pragma unroll
		for (int j = 0; j < CH; j++) Rb[(size_t)i * 3 * SXS_QT + j * SXS_QT] = a[j];
		if (i + 1 < n) {
			tcol_row<1, CH, S, V, NB>(tq + (i + 1) * NB, u, a);
#pragma unroll
			for (int j = 0; j < CH; j++) Rb[(size_t)(i + 1) * 3 * SXS_QT + j * SXS_QT] = a[j];
		}
	}
}

/* 16-byte asynchronous global-to-shared copies (completion by wait_group,
 * a hardware wait on the thread's own copies) */
__device__ __forceinline__ void cp_async16(void *sdst, const void *gsrc)
{
	unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
/* one float, zero when !in */
__device__ __forceinline__ void cp_async4(float *sdst, const float *gsrc, bool in)
{
	unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
	asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(sa), "l"(gsrc), "r"(in ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

/* float2 between the staged U columns of two combos: half a bank row more
 * than the columns, because a half-warp reads 64 bytes of each of two combos
 * (without it every such read took twice its wavefronts: 2.29 against 2.15
 * ms at L = 20, Q = 101, all 18,000 combos) */
#define TP_UROW(NB) ((NB) * 3 * SXS_QT + 8)

/* shared bytes of k_translate_pipe<NB>: tau^m [8 q][NB NB + 4] and the U
 * columns of one slice [SXS_SLICE combos][NB pairs][3 ch][8 q] */
#define TP_SMEM(NB) (sizeof(float) * SXS_QT * ((NB) * (NB) + 4) + sizeof(float2) * SXS_SLICE * TP_UROW(NB))

/* The FP32 column form with three channels per thread, pipelined over
 * slices: block = (tile, run of sb consecutive slices, m); while the
 * threads apply tau^m to one slice's U columns (held in registers: 6 NB
 * floats), the U columns of the next slice stream into shared memory with
 * cp.async, so the global-load latency of the low occupancy that these
 * registers allow (1-5 blocks of 4 warps per SM by NB) overlaps the
 * arithmetic.  tau^m(q z) is restaged only where z changes between slices
 * (slices are z-major), by 4-byte cp.async as well, so that its one round
 * trip to L2 overlaps the U columns'.  The sums are those of k_translate_col
 * with CH = 3: rows in even/odd pairs, one tau load for three channels.
 * A block's serial chain is what the low occupancy leaves visible: with the
 * window of indices and tau through registers the above case took 2.02, now
 * 1.96 ms (20,000 poses at L = 25: 3.22; 3.68 before the three changes). */
#define TP_MINB(NB) (NB <= 8 ? 5 : (NB <= 12 ? 4 : (NB <= 20 ? 3 : (NB <= 28 ? 2 : 1))))

/* The slices of a window of TP_W: first combo - cbase, combos, z; and per
 * combo its row of U.  Read once per window by the whole block, so that the
 * copies of a slice start without two dependent reads of global memory
 * (2.15 -> 2.02 ms in the above case). */
#define TP_W 8
struct TpWin {
	int4 sl[TP_W];
	int row[TP_W][SXS_SLICE];
};
__device__ __forceinline__ void tp_window(TpWin &w, const int32_t *__restrict__ combo_zbg,
                                          const int32_t *__restrict__ slices, int cbase, int s0, int s1, int N)
{
	__syncthreads();   /* no thread still reads the last window */
	for (int i = threadIdx.x; i < TP_W * SXS_SLICE; i += TCOL_THREADS(3)) {
		int s = s0 + i / SXS_SLICE, c = i % SXS_SLICE;
		if (s >= s1) break;
		int cf = slices[2 * s] - cbase, nc = slices[2 * s + 1];
		if (c >= nc) continue;
		const int32_t *z = combo_zbg + 3 * (cf + c);
		w.row[i / SXS_SLICE][c] = z[1] * N + z[2];
		if (c == 0) w.sl[i / SXS_SLICE] = make_int4(cf, nc, z[0], 0);
	}
	__syncthreads();
}

/* one block of k_translate_pipe: (tile t, slice group gi, m); raw = the
 * block's TP_SMEM(NB) bytes of shared memory */
template <int NB>
__device__ __forceinline__ void tpipe_block(const float2 *__restrict__ U, const float *__restrict__ tau,
                                            const int32_t *__restrict__ combo_zbg, const int32_t *__restrict__ slices,
                                            int nslice, int cbase, int ncombo, int L, int nzt, int t, int gi, int m,
                                            int sb, float2 *__restrict__ R, unsigned char *raw)
{
	const int qstride = NB * NB + 4, rowf = 3 * SXS_QT;   /* float2 per pair of one combo */
	float *ts = reinterpret_cast<float *>(raw);
	float2 *us = reinterpret_cast<float2 *>(raw + sizeof(float) * SXS_QT * qstride);
	int K = L + 1, N = 2 * L + 1, NP = K * (K + 1) / 2, nrow = K * N;
	int n = K - m, po = psym(m, K);
	int s0 = gi * sb, s1 = s0 + sb < nslice ? s0 + sb : nslice;
	int q = threadIdx.x % SXS_QT, cl = threadIdx.x / SXS_QT;
	/* 16-byte chunks of one combo's n pairs: n x 3 x 8 float2 = 12 n; the
	 * 8 threads of combo cl copy its chunks in 128-byte rows */
	const int per = n * rowf / 2;
	__shared__ TpWin win;
	auto issue = [&](int s) {
		if ((s - s0) % TP_W == 0) tp_window(win, combo_zbg, slices, cbase, s, s1, N);
		int k = (s - s0) % TP_W;
		if (cl < win.sl[k].y) {
			const float2 *src = U + (((size_t)t * nrow + win.row[k][cl]) * NP + po) * rowf;
			float2 *dst = us + (size_t)cl * TP_UROW(NB);
			for (int r = q; r < per; r += SXS_QT) cp_async16(dst + 2 * r, src + 2 * r);
		}
		cp_async_commit();
	};
	int zcur = -1;
	if (s0 < s1) issue(s0);
	for (int s = s0; s < s1; s++) {
		int4 w = win.sl[(s - s0) % TP_W];
		int cf = w.x, nc = w.y, zi = w.z;
		if (zi != zcur) {
			__syncthreads();   /* no thread still reads the previous tau */
			const float *tz = tau + ((((size_t)t * nzt + zi) * K + m) * K) * K * SXS_QT;
			for (int k = threadIdx.x; k < SXS_QT * NB * NB; k += TCOL_THREADS(3)) {
				int qq = k % SXS_QT, r = k / SXS_QT;
				int i = r / NB, kk = r % NB;
				bool in = i < n && kk < n;
				cp_async4(ts + qq * qstride + i * NB + kk,
				          in ? tz + ((size_t)(m + i) * K + m + kk) * SXS_QT + qq : tz, in);
			}
			cp_async_commit();
			zcur = zi;
		}
		cp_async_wait_all();
		__syncthreads();   /* this slice's U columns and tau visible to all */
		bool act = cl < nc;
		float2 u[3][NB];
		if (act) {
			const float2 *uc = us + (size_t)cl * TP_UROW(NB) + q;
#pragma unroll
			for (int j = 0; j < 3; j++)
#pragma unroll
				for (int k = 0; k < NB; k++) u[j][k] = k < n ? uc[k * rowf + j * SXS_QT] : zero2<float2>();
		}
		__syncthreads();   /* the buffer is free for the next slice */
		if (s + 1 < s1) issue(s + 1);
		if (act) {
			int c = cf + cl;
			const float *tq = ts + q * qstride;
			float2 *Rb = R + (((size_t)t * ncombo + c) * NP + po) * rowf + q;
			for (int i = 0; i < n; i += 2) {
				float2 a[3];
				tcol_row<0, 3, float, float2, NB>(tq + i * NB, u, a);
#pragma unroll
				for (int j = 0; j < 3; j++) Rb[(size_t)i * rowf + j * SXS_QT] = a[j];
				if (i + 1 < n) {
					tcol_row<1, 3, float, float2, NB>(tq + (i + 1) * NB, u, a);
#pragma unroll
					for (int j = 0; j < 3; j++) Rb[(size_t)(i + 1) * rowf + j * SXS_QT] = a[j];
				}
			}
		}
	}
}

/* The FP32 translation in tiles, for n = 29 to 32, whose 6 n registers of U
 * leave the form above one block (a warp per scheduler) on an SM.  Block =
 * (tile, run of sb consecutive slices, m), TT_CP combos at a time; thread =
 * (q, two combos, TT_RB of the n rows).  Per k a thread reads TT_RB values
 * tau[i][k] (kept transposed) and its combos' U[k] from shared memory for 96
 * multiply-adds into 96 sums, each in the order of tcol_row.  82 KB and 219
 * registers: two blocks.  L = 30, Q = 201, 40,000 poses, all classes: 18.5 ->
 * 17.4 ms; for n = 25 to 28, where two blocks of the other form fit, it is
 * the slower one (17.8), and so on down (19.3 with it everywhere). */
#define TT_FROM 29
#define TT_USE(NB) ((NB) >= TT_FROM)
#define TT_RG 4
#define TT_CP (32 / TT_RG)
#define TT_RB(NB) ((((NB) + TT_RG - 1) / TT_RG + 1) / 2 * 2)
#define TT_UROW(NB) ((NB) * 3 * SXS_QT + 4)   /* 4: see TP_UROW; a quarter-warp's combos are two rows apart */
#define TT_TS(NB) ((NB) * TT_RB(NB) * TT_RG + 4)
#define TT_SMEM(NB) (sizeof(float) * SXS_QT * TT_TS(NB) + sizeof(float2) * TT_CP * TT_UROW(NB))
/* of the FP32 translation's blocks */
#define TR_SMEM(NB) (TT_USE(NB) ? TT_SMEM(NB) : TP_SMEM(NB))
#define TR_MINB(NB) (TT_USE(NB) ? 2 : TP_MINB(NB))

template <int RB>
struct TtIn {
	float t[RB];
	float2 u[2][3];
};

template <int NB>
__device__ __forceinline__ void tt_load(TtIn<TT_RB(NB)> &x, const float *tq, const float2 *uq, int k)
{
	constexpr int RB = TT_RB(NB), RT = RB * TT_RG;
	const float *t = tq + k * RT;
	static_assert(RB % 4 == 0, "tau in 16-byte loads");
#pragma unroll
	for (int i = 0; i < RB / 4; i++) ld4(t + 4 * i, x.t + 4 * i);
#pragma unroll
	for (int c = 0; c < 2; c++)
#pragma unroll
		for (int j = 0; j < 3; j++) x.u[c][j] = uq[c * TT_UROW(NB) + (k * 3 + j) * SXS_QT];
}

template <int PK, int RB>
__device__ __forceinline__ void tt_step(const TtIn<RB> &x, float2 (&acc)[2][3][RB])
{
#pragma unroll
	for (int c = 0; c < 2; c++)
#pragma unroll
		for (int j = 0; j < 3; j++)
#pragma unroll
			for (int i = 0; i < RB; i++) {
				float2 &a = acc[c][j][i];
				float2 u = x.u[c][j];
				if ((i & 1) == PK) {
					a.x = fma_s(x.t[i], u.x, a.x);
					a.y = fma_s(x.t[i], u.y, a.y);
				} else {
					a.x = fma_s(x.t[i], u.y, a.x);
					a.y = fma_s(-x.t[i], u.x, a.y);
				}
			}
}

template <int NB>
__device__ __forceinline__ void ttile_block(const float2 *__restrict__ U, const float *__restrict__ tau,
                                            const int32_t *__restrict__ combo_zbg, const int32_t *__restrict__ slices,
                                            int nslice, int cbase, int ncombo, int L, int nzt, int t, int gi, int m,
                                            int sb, float2 *__restrict__ R, unsigned char *raw)
{
	constexpr int RB = TT_RB(NB), RT = RB * TT_RG, CP = TT_CP, rowf = 3 * SXS_QT;
	constexpr int NTH = TCOL_THREADS(3), TPC = NTH / CP;   /* threads that copy a combo's columns */
	float *ts = reinterpret_cast<float *>(raw);
	float2 *us = reinterpret_cast<float2 *>(raw + sizeof(float) * SXS_QT * TT_TS(NB));
	int K = L + 1, N = 2 * L + 1, NP = K * (K + 1) / 2, nrow = K * N;
	int n = K - m, po = psym(m, K);
	int s0 = gi * sb, s1 = s0 + sb < nslice ? s0 + sb : nslice;
	int tid = threadIdx.x, q = tid % SXS_QT, pr = tid / SXS_QT % (CP / 2), i0 = tid / (SXS_QT * (CP / 2)) * RB;
	__shared__ TpWin win;
	int zcur = -1;
	for (int s = s0; s < s1; s++) {
		if ((s - s0) % TP_W == 0) tp_window(win, combo_zbg, slices, cbase, s, s1, N);
		int4 w = win.sl[(s - s0) % TP_W];
		int cf = w.x, nc = w.y, zi = w.z;
		for (int h = 0; h < nc; h += CP) {
			int nh = min(CP, nc - h);
			__syncthreads();   /* no thread still reads tau or U */
			int cl = tid / TPC;
			if (cl < nh) {
				const float2 *src = U + (((size_t)t * nrow + win.row[(s - s0) % TP_W][h + cl]) * NP + po) * rowf;
				float2 *dst = us + (size_t)cl * TT_UROW(NB);
				for (int r = tid % TPC; r < n * rowf / 2; r += TPC) cp_async16(dst + 2 * r, src + 2 * r);
			}
			cp_async_commit();
			if (zi != zcur) {
				const float *tz = tau + ((((size_t)t * nzt + zi) * K + m) * K) * K * SXS_QT;
				for (int k = tid; k < SXS_QT * NB * RT; k += NTH) {
					int qq = k % SXS_QT, r = k / SXS_QT;
					int i = r % RT, kk = r / RT;
					bool in = i < n && kk < n;
					cp_async4(ts + qq * TT_TS(NB) + kk * RT + i,
					          in ? tz + ((size_t)(m + i) * K + m + kk) * SXS_QT + qq : tz, in);
				}
				cp_async_commit();
				zcur = zi;
			}
			cp_async_wait_all();
			__syncthreads();   /* these U columns and tau visible to all */
			if (2 * pr >= nh || i0 >= n) continue;
			const float *tq = ts + q * TT_TS(NB) + i0;
			const float2 *uq = us + (size_t)2 * pr * TT_UROW(NB) + q;
			float2 acc[2][3][RB];
#pragma unroll
			for (int c = 0; c < 2; c++)
#pragma unroll
				for (int j = 0; j < 3; j++)
#pragma unroll
					for (int i = 0; i < RB; i++) acc[c][j][i] = make_float2(0.0f, 0.0f);
			TtIn<RB> x, y;
			tt_load<NB>(x, tq, uq, 0);
			int k = 0;
			for (; k + 1 < n; k += 2) {
				tt_load<NB>(y, tq, uq, k + 1);
				tt_step<0>(x, acc);
				tt_load<NB>(x, tq, uq, min(k + 2, n - 1));
				tt_step<1>(y, acc);
			}
			if (k < n) tt_step<0>(x, acc);
#pragma unroll
			for (int c = 0; c < 2; c++) {
				if (2 * pr + c >= nh) break;
				float2 *Rb = R + (((size_t)t * ncombo + cf + h + 2 * pr + c) * NP + po + i0) * rowf + q;
#pragma unroll
				for (int i = 0; i < RB; i++)
					if (i0 + i < n)
#pragma unroll
						for (int j = 0; j < 3; j++) Rb[(size_t)i * rowf + j * SXS_QT] = acc[c][j][i];
			}
		}
	}
}

template <int NB>
__device__ __forceinline__ void translate_block(const float2 *__restrict__ U, const float *__restrict__ tau,
                                                const int32_t *__restrict__ combo_zbg,
                                                const int32_t *__restrict__ slices, int nslice, int cbase, int ncombo,
                                                int L, int nzt, int t, int gi, int m, int sb, float2 *__restrict__ R,
                                                unsigned char *raw)
{
	if constexpr (TT_USE(NB))
		ttile_block<NB>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, L, nzt, t, gi, m, sb, R, raw);
	else
		tpipe_block<NB>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, L, nzt, t, gi, m, sb, R, raw);
}

/* poses per pass of a thread of the fused kernel: the per-pose sums
 * (6 floats each) share the registers with the U columns (6 NB floats) */
#define TF_KMAX(NB) ((NB) <= 16 ? 4 : ((NB) <= 24 ? 2 : 1))
/* resident blocks per SM the fused kernel is compiled for (registers of
 * the per-pose sums beside the U columns, without spills) */
#define TF_MINB(NB) ((NB) <= 12 ? 3 : ((NB) <= 20 ? 2 : 1))

/* F += the six channel products of one pair: Re(P_a (w R_b)) summed over
 * (a, b) and (b, a) as in k_pose_cross */
__device__ __forceinline__ void fused_acc(float *F, const float2 *__restrict__ pp, float wx, float wy, const float2 *a)
{
	float2 p0 = pp[0], p1 = pp[SXS_QT], p2 = pp[2 * SXS_QT];
	float2 s0, s1, s2;
	s0.x = fmaf(wx, a[0].x, __fmul_rn(-wy, a[0].y)); s0.y = fmaf(wx, a[0].y, __fmul_rn(wy, a[0].x));
	s1.x = fmaf(wx, a[1].x, __fmul_rn(-wy, a[1].y)); s1.y = fmaf(wx, a[1].y, __fmul_rn(wy, a[1].x));
	s2.x = fmaf(wx, a[2].x, __fmul_rn(-wy, a[2].y)); s2.y = fmaf(wx, a[2].y, __fmul_rn(wy, a[2].x));
	F[0] = __fadd_rn(F[0], fmaf(p0.x, s0.x, __fmul_rn(-p0.y, s0.y)));
	F[1] = __fadd_rn(F[1], fmaf(-p1.y, s0.y, fmaf(p1.x, s0.x, fmaf(p0.x, s1.x, __fmul_rn(-p0.y, s1.y)))));
	F[2] = __fadd_rn(F[2], fmaf(-p2.y, s0.y, fmaf(p2.x, s0.x, fmaf(p0.x, s2.x, __fmul_rn(-p0.y, s2.y)))));
	F[3] = __fadd_rn(F[3], fmaf(p1.x, s1.x, __fmul_rn(-p1.y, s1.y)));
	F[4] = __fadd_rn(F[4], fmaf(-p2.y, s1.y, fmaf(p2.x, s1.x, fmaf(p1.x, s2.x, __fmul_rn(-p1.y, s2.y)))));
	F[5] = __fadd_rn(F[5], fmaf(p2.x, s2.x, __fmul_rn(-p2.y, s2.y)));
}

/* shared bytes of the fused kernel: those of k_translate_pipe<NB> plus the
 * twiddles */
#define TF_SMEM(NB) (TP_SMEM(NB) + sizeof(float2) * (2 * SXS_LMAX_K))

/* One block of the fused translation for sparse pose lists: the block of
 * k_translate_pipe (tile t, slice group gi, m), whose translated rows are
 * contracted at once with the receptor rows of their combos' poses instead
 * of being stored: thread (combo, q) computes the rows R[m, m + i], i < n,
 * from its U columns in registers, up to TF_KMAX(NB) poses of the combo per
 * pass (a combo with more poses recomputes its rows per pass), and writes
 * per pose and m the six sums
 *   part[pose - pose_base][m][ch][t 8 + q] = sum_i Re(P_a(b1, g1)[m, m + i] w_m R_b[m, m + i])
 * (a, b as in k_pose_cross; w_m = tw[(m a2) mod N], doubled for m > 0).
 * cstart[c] = the first sorted pose of global combo c (cstart[ncombo] = the
 * pose count); raw = the block's TF_SMEM(NB) bytes. */
template <int NB>
__device__ __forceinline__ void tfused_block(const float2 *__restrict__ U, const float *__restrict__ tau,
                                             const int32_t *__restrict__ combo_zbg,
                                             const int32_t *__restrict__ slices, int nslice, int cbase, int L,
                                             int nzt, int t, int gi, int m, int sb,
                                             const sxsk_pose *__restrict__ poses, const int32_t *__restrict__ cstart,
                                             int pose_base, const float2 *__restrict__ P,
                                             const double2 *__restrict__ tw, float *__restrict__ part, int QP,
                                             unsigned char *raw)
{
	constexpr int KMAX = TF_KMAX(NB);
	const int qstride = NB * NB + 4, rowf = 3 * SXS_QT;
	float *ts = reinterpret_cast<float *>(raw);
	float2 *us = reinterpret_cast<float2 *>(raw + sizeof(float) * SXS_QT * qstride);
	float2 *tws = reinterpret_cast<float2 *>(raw + TP_SMEM(NB));
	int K = L + 1, N = 2 * L + 1, NP = K * (K + 1) / 2, nrow = K * N;
	int n = K - m, po = psym(m, K);
	int s0 = gi * sb, s1 = s0 + sb < nslice ? s0 + sb : nslice;
	int q = threadIdx.x % SXS_QT, cl = threadIdx.x / SXS_QT;
	for (int k = threadIdx.x; k < N; k += blockDim.x) tws[k] = from2<float2>(tw[k]);
	const int per = n * rowf / 2;
	auto issue = [&](int s) {
		int cf = slices[2 * s] - cbase, nc = slices[2 * s + 1];
		if (cl < nc) {
			int cc = cf + cl;
			int b2 = combo_zbg[3 * cc + 1], g2 = combo_zbg[3 * cc + 2];
			const float2 *src = U + (((size_t)t * nrow + b2 * N + g2) * NP + po) * rowf;
			float2 *dst = us + (size_t)cl * TP_UROW(NB);
			for (int r = q; r < per; r += SXS_QT) cp_async16(dst + 2 * r, src + 2 * r);
		}
		cp_async_commit();
	};
	int zcur = -1;
	if (s0 < s1) issue(s0);
	for (int s = s0; s < s1; s++) {
		int cf = slices[2 * s] - cbase, nc = slices[2 * s + 1];
		int zi = combo_zbg[3 * cf];
		if (zi != zcur) {
			__syncthreads();   /* no thread still reads the previous tau */
			const float *tz = tau + ((((size_t)t * nzt + zi) * K + m) * K) * K * SXS_QT;
			for (int k = threadIdx.x; k < SXS_QT * NB * NB; k += blockDim.x) {
				int qq = k % SXS_QT, r = k / SXS_QT;
				int i = r / NB, kk = r % NB;
				float v = 0;
				if (i < n && kk < n) v = __ldg(tz + ((size_t)(m + i) * K + m + kk) * SXS_QT + qq);
				ts[qq * qstride + i * NB + kk] = v;
			}
			zcur = zi;
		}
		cp_async_wait_all();
		__syncthreads();   /* this slice's U columns, tau and the twiddles visible to all */
		bool act = cl < nc;
		float2 u[3][NB];
		if (act) {
			const float2 *uc = us + (size_t)cl * TP_UROW(NB) + q;
#pragma unroll
			for (int j = 0; j < 3; j++)
#pragma unroll
				for (int k = 0; k < NB; k++) u[j][k] = k < n ? uc[k * rowf + j * SXS_QT] : zero2<float2>();
		}
		__syncthreads();   /* the buffer is free for the next slice */
		if (s + 1 < s1) issue(s + 1);
		if (act) {
			int c = cbase + cf + cl;
			const float *tq = ts + q * qstride;
			int p1 = cstart[c + 1];
			for (int pb = cstart[c]; pb < p1; pb += KMAX) {
				const float2 *Pp[KMAX];
				float wx[KMAX], wy[KMAX], F[KMAX][6];
#pragma unroll
				for (int kb = 0; kb < KMAX; kb++) {
					int pi = pb + kb < p1 ? pb + kb : pb;   /* a spare slot repeats the first pose */
					sxsk_pose ps = poses[pi];
					Pp[kb] = P + (((size_t)t * nrow + ps.b1 * N + ps.g1) * NP + po) * rowf + q;
					int e = (m * ps.a2) % N;
					float2 w = tws[e];
					float f = m > 0 ? 2.0f : 1.0f;
					wx[kb] = f * w.x;
					wy[kb] = f * w.y;
#pragma unroll
					for (int ch = 0; ch < 6; ch++) F[kb][ch] = 0.0f;
				}
				for (int i = 0; i < n; i += 2) {
					float2 a[3];
					tcol_row<0, 3, float, float2, NB>(tq + i * NB, u, a);
#pragma unroll
					for (int kb = 0; kb < KMAX; kb++) fused_acc(F[kb], Pp[kb] + (size_t)i * rowf, wx[kb], wy[kb], a);
					if (i + 1 < n) {
						tcol_row<1, 3, float, float2, NB>(tq + (i + 1) * NB, u, a);
#pragma unroll
						for (int kb = 0; kb < KMAX; kb++)
							fused_acc(F[kb], Pp[kb] + (size_t)(i + 1) * rowf, wx[kb], wy[kb], a);
					}
				}
#pragma unroll
				for (int kb = 0; kb < KMAX; kb++) {
					if (pb + kb < p1) {
						float *o = part + (((size_t)(pb + kb - pose_base) * K + m) * 6) * QP + t * SXS_QT + q;
#pragma unroll
						for (int ch = 0; ch < 6; ch++) o[(size_t)ch * QP] = F[kb][ch];
					}
				}
			}
		}
	}
}

template <int NB>
__global__ void __launch_bounds__(TCOL_THREADS(3), TF_MINB(NB))
k_translate_fused(const float2 *__restrict__ U, const float *__restrict__ tau, const int32_t *__restrict__ combo_zbg,
                  const int32_t *__restrict__ slices, int nslice, int cbase, int L, int nzt, int m_lo, int nm, int sb,
                  const sxsk_pose *__restrict__ poses, const int32_t *__restrict__ cstart, int pose_base,
                  const float2 *__restrict__ P, const double2 *__restrict__ tw, float *__restrict__ part, int QP)
{
	extern __shared__ __align__(16) unsigned char tps_raw[];
	int ng = (nslice + sb - 1) / sb;
	int bid = blockIdx.x;
	int mi = bid % nm;
	bid /= nm;
	int gi = bid % ng, t = bid / ng;
	tfused_block<NB>(U, tau, combo_zbg, slices, nslice, cbase, L, nzt, t, gi, m_lo + mi, sb, poses, cstart, pose_base,
	                 P, tw, part, QP, tps_raw);
}

/* fused translation blocks of many chunks */
template <int NB>
__global__ void __launch_bounds__(TCOL_THREADS(3), TF_MINB(NB))
k_translate_fused_batch(const sxsk_tf_job *__restrict__ jobs, const int4 *__restrict__ items, int nitems, int *ctr)
{
	extern __shared__ __align__(16) unsigned char tps_raw[];
	__shared__ int s_it;
	int nxt = 0;
	for (int it = item_begin(ctr, &s_it); it < nitems; it = item_advance(ctr, &s_it, nxt, nitems)) {
		nxt = item_claim(ctr);
		int4 w = items[it];
		sxsk_tf_job j = jobs[w.x];
		tfused_block<NB>((const float2 *)j.U, (const float *)j.tau, j.combo_zbg, j.slices, j.nslice, j.cbase, j.L,
		                 j.nzt, w.y, w.z, w.w, j.sb, j.poses, j.cstart, j.pose_base, (const float2 *)j.P, j.tw, j.part,
		                 ((j.Q + SXS_QT - 1) / SXS_QT) * SXS_QT, tps_raw);
	}
}

template <int NB>
__global__ void __launch_bounds__(TCOL_THREADS(3), TR_MINB(NB))
k_translate_pipe(const float2 *__restrict__ U, const float *__restrict__ tau, const int32_t *__restrict__ combo_zbg,
                 const int32_t *__restrict__ slices, int nslice, int cbase, int ncombo, int L, int nzt, int m_lo,
                 int nm, int sb, float2 *__restrict__ R)
{
	extern __shared__ __align__(16) unsigned char tps_raw[];
	chain_begin();
	int ng = (nslice + sb - 1) / sb;
	int bid = blockIdx.x;
	int mi = bid % nm;
	bid /= nm;
	int gi = bid % ng, t = bid / ng;
	translate_block<NB>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, L, nzt, t, gi, m_lo + mi, sb, R, tps_raw);
	chain_end();
}

/* pipelined translation blocks of many chunks (mixed path) */
template <int NB>
__global__ void __launch_bounds__(TCOL_THREADS(3), TR_MINB(NB))
k_translate_batch(const sxsk_tr_job *__restrict__ jobs, const int4 *__restrict__ items, int nitems, int *ctr)
{
	extern __shared__ __align__(16) unsigned char tps_raw[];
	__shared__ int s_it;
	int nxt = 0;
	for (int it = item_begin(ctr, &s_it); it < nitems; it = item_advance(ctr, &s_it, nxt, nitems)) {
		nxt = item_claim(ctr);
		int4 w = items[it];
		sxsk_tr_job j = jobs[w.x];
		translate_block<NB>((const float2 *)j.U, (const float *)j.tau, j.combo_zbg, j.slices, j.nslice, j.cbase,
		                j.ncombo, j.L, j.nzt, w.y, w.z, w.w, j.sb, (float2 *)j.R, tps_raw);
	}
}

/* Storage of the per-pose cross terms: double on the FP64 path; on the FP32
 * path a double-float pair {hi, lo} = cst + 2 f formed with an error-free
 * sum (explicit round-to-nearest adds, never contracted), so that the fit
 * reads it without the FP64 pipe. */
template <typename S> struct CrossT;
template <> struct CrossT<double> { typedef double T; };
template <> struct CrossT<float> { typedef float2 T; };
__device__ __forceinline__ void cross_store(double *o, const double *cst, size_t i, double f)
{
	o[i] = cst[i] + 2.0 * f;
}
__device__ __forceinline__ void cross_store(float2 *o, const float2 *cst, size_t i, float f)
{
	float2 c = cst[i];
	float t = 2.0f * f;                       /* exact */
	float s = __fadd_rn(c.x, t);
	float bb = __fsub_rn(s, c.x);
	float e = __fadd_rn(__fsub_rn(c.x, __fsub_rn(s, bb)), __fsub_rn(t, bb));
	e = __fadd_rn(e, c.y);
	float h = __fadd_rn(s, e);
	o[i] = make_float2(h, __fsub_rn(e, __fsub_rn(h, s)));
}

/* cross[src][c][q] = cst[c][q] + 2 sum_m part[p][m][c][q] (m ascending, FP32)
 * as double-float pairs; thread = (pose, q) */
__device__ __forceinline__ void fused_reduce_at(const sxsk_pose *__restrict__ poses, int npose,
                                                const float *__restrict__ part, int K, int Q, int QP,
                                                const float2 *__restrict__ cst, float2 *__restrict__ cross, long i)
{
	if (i >= (long)npose * Q) return;
	int p = (int)(i / Q), q = (int)(i % Q);
	const float *src = part + (size_t)p * K * 6 * QP + q;
	float2 *o = cross + (size_t)poses[p].src * 6 * Q;
#pragma unroll
	for (int c = 0; c < 6; c++) {
		float f = 0.0f;
		for (int m = 0; m < K; m++) f = __fadd_rn(f, src[((size_t)m * 6 + c) * QP]);
		cross_store(o, cst, (size_t)c * Q + q, f);
	}
}

__global__ void __launch_bounds__(128)
k_fused_reduce(const sxsk_pose *__restrict__ poses, int npose, const float *__restrict__ part, int K, int Q, int QP,
               const float2 *__restrict__ cst, float2 *__restrict__ cross)
{
	fused_reduce_at(poses, npose, part, K, Q, QP, cst, cross, (long)blockIdx.x * blockDim.x + threadIdx.x);
}

/* the sums over m of many chunks: items {job, block of 128 (pose, q)} */
__global__ void __launch_bounds__(128)
k_fused_reduce_batch(const sxsk_fr_job *__restrict__ jobs, const int4 *__restrict__ items, int nitems, int *ctr)
{
	__shared__ int s_it;
	int nxt = 0;
	for (int it = item_begin(ctr, &s_it); it < nitems; it = item_advance(ctr, &s_it, nxt, nitems)) {
		nxt = item_claim(ctr);
		int4 w = items[it];
		sxsk_fr_job j = jobs[w.x];
		int QP = ((j.Q + SXS_QT - 1) / SXS_QT) * SXS_QT;
		fused_reduce_at(j.poses, j.npose, j.part, j.L + 1, j.Q, QP, (const float2 *)j.cst, (float2 *)j.cross,
		                (long)w.y * blockDim.x + threadIdx.x);
	}
}

/* Per-pose cross terms of one chunk, all q tiles.  Thread = (pose, 2
 * adjacent q); block = 32 consecutive poses (sorted by combo, so their R
 * rows repeat and hit in L1) x 4 q pairs of one tile; blocks ordered
 * tile-major.  HINT: P rows (reused by every pose of the same rotation) are
 * loaded with the L2 evict_last policy, R rows (streamed once per chunk)
 * with evict_first.  The pose's phase w_m = tw[(m a2) mod N] (doubled for m > 0)
 * is applied to R first, so each channel product needs only its real part:
 *   cross[src][c][q] = cst[c][q] + 2 sum_{m,l} Re(P_a[m,l] (w_m R_b[m,l])). */
/* one block of k_pose_cross: (tile t, pose block pb), twiddles staged in tws */
template <typename S, bool HINT>
__device__ __forceinline__ void pcross_block(const sxsk_pose *__restrict__ poses, int npose, int combo_base,
                                             int ncombo, const typename Cx<S>::T *__restrict__ P,
                                             const typename Cx<S>::T *__restrict__ R, const typename Cx<S>::T *tws,
                                             const typename CrossT<S>::T *__restrict__ cst, int Q, int L,
                                             typename CrossT<S>::T *__restrict__ cross, int t, int pb)
{
	typedef typename Cx<S>::T V;
	int K = L + 1, N = 2 * L + 1, NP = K * (K + 1) / 2, nrow = K * N;
	int pi = pb * PC_PPB + threadIdx.x / SXS_QP, j2 = 2 * (threadIdx.x % SXS_QP);
	if (pi >= npose) return;
	int q0 = t * SXS_QT + j2;
	if (q0 >= Q) return;
	sxsk_pose ps = poses[pi];
	const V *Pr = P + (((size_t)t * nrow + ps.b1 * N + ps.g1) * NP) * 3 * SXS_QT + j2;
	const V *Rr = R + (((size_t)t * ncombo + ps.combo - combo_base) * NP) * 3 * SXS_QT + j2;
	S f[2][6];
#pragma unroll
	for (int k = 0; k < 2; k++)
#pragma unroll
		for (int c = 0; c < 6; c++) f[k][c] = 0;
	/* pairs in m-major order; the phase tw[(m a2) mod N] (doubled for m > 0)
	 * changes where a row of m starts */
	int m = 0, mend = K, e = 0;
	S wx = tws[0].x, wy = tws[0].y;
	uint64_t polP = 0, polR = 0;
	if (HINT) {
		polP = l2_policy(true);
		polR = l2_policy(false);
	}
#pragma unroll 2
	for (int p = 0; p < NP; p++) {
		if (p == mend) {
			m++;
			mend += K - m;
			e += ps.a2;
			if (e >= N) e -= N;
			wx = (S)2 * tws[e].x;
			wy = (S)2 * tws[e].y;
		}
		const V *pp = Pr + (size_t)p * 3 * SXS_QT;
		const V *rr = Rr + (size_t)p * 3 * SXS_QT;
		Pair2<S> cp[3], cr[3];
		if (HINT) {
			constexpr int CB = SXS_QT * (int)sizeof(V);   /* bytes between channels */
			cp[0] = ld2_pol<0>(pp, polP);
			cp[1] = ld2_pol<CB>(pp, polP);
			cp[2] = ld2_pol<2 * CB>(pp, polP);
			cr[0] = ld2_pol<0>(rr, polR);
			cr[1] = ld2_pol<CB>(rr, polR);
			cr[2] = ld2_pol<2 * CB>(rr, polR);
		} else {
#pragma unroll
			for (int c = 0; c < 3; c++) {
				cp[c] = ld2(pp + c * SXS_QT);
				cr[c] = ld2(rr + c * SXS_QT);
			}
		}
#pragma unroll
		for (int k = 0; k < 2; k++) {
			V a0 = k ? cp[0].b : cp[0].a, a1 = k ? cp[1].b : cp[1].a, a2 = k ? cp[2].b : cp[2].a;
			V r0 = k ? cr[0].b : cr[0].a, r1 = k ? cr[1].b : cr[1].a, r2 = k ? cr[2].b : cr[2].a;
			/* R' = w R */
			V s0, s1, s2;
			s0.x = fma_s(wx, r0.x, mul_rn(-wy, r0.y)); s0.y = fma_s(wx, r0.y, mul_rn(wy, r0.x));
			s1.x = fma_s(wx, r1.x, mul_rn(-wy, r1.y)); s1.y = fma_s(wx, r1.y, mul_rn(wy, r1.x));
			s2.x = fma_s(wx, r2.x, mul_rn(-wy, r2.y)); s2.y = fma_s(wx, r2.y, mul_rn(wy, r2.x));
			S *F = f[k];
			if (sizeof(S) == 8) {
				/* FP64 (bound by the FP64 pipe): the Re(a s) terms as FMA
				 * chains straight into the accumulators, 18 operations per q
				 * instead of 24 for sums of products added to F */
				F[0] = fma_s(a0.x, s0.x, F[0]); F[0] = fma_s(-a0.y, s0.y, F[0]);
				F[1] = fma_s(a0.x, s1.x, F[1]); F[1] = fma_s(-a0.y, s1.y, F[1]);
				F[1] = fma_s(a1.x, s0.x, F[1]); F[1] = fma_s(-a1.y, s0.y, F[1]);
				F[2] = fma_s(a0.x, s2.x, F[2]); F[2] = fma_s(-a0.y, s2.y, F[2]);
				F[2] = fma_s(a2.x, s0.x, F[2]); F[2] = fma_s(-a2.y, s0.y, F[2]);
				F[3] = fma_s(a1.x, s1.x, F[3]); F[3] = fma_s(-a1.y, s1.y, F[3]);
				F[4] = fma_s(a1.x, s2.x, F[4]); F[4] = fma_s(-a1.y, s2.y, F[4]);
				F[4] = fma_s(a2.x, s1.x, F[4]); F[4] = fma_s(-a2.y, s1.y, F[4]);
				F[5] = fma_s(a2.x, s2.x, F[5]); F[5] = fma_s(-a2.y, s2.y, F[5]);
			} else {
				/* FP32 (bound by the L1 data path): sums of products, whose
				 * short dependence on F keeps more loads in flight */
				F[0] = add_rn(F[0], fma_s(a0.x, s0.x, mul_rn(-a0.y, s0.y)));
				F[1] = add_rn(F[1], fma_s(-a1.y, s0.y, fma_s(a1.x, s0.x, fma_s(a0.x, s1.x, mul_rn(-a0.y, s1.y)))));
				F[2] = add_rn(F[2], fma_s(-a2.y, s0.y, fma_s(a2.x, s0.x, fma_s(a0.x, s2.x, mul_rn(-a0.y, s2.y)))));
				F[3] = add_rn(F[3], fma_s(a1.x, s1.x, mul_rn(-a1.y, s1.y)));
				F[4] = add_rn(F[4], fma_s(-a2.y, s1.y, fma_s(a2.x, s1.x, fma_s(a1.x, s2.x, mul_rn(-a1.y, s2.y)))));
				F[5] = add_rn(F[5], fma_s(a2.x, s2.x, mul_rn(-a2.y, s2.y)));
			}
		}
	}
	typename CrossT<S>::T *o = cross + (size_t)ps.src * 6 * Q;
#pragma unroll
	for (int k = 0; k < 2; k++) {
		int q = q0 + k;
		if (q < Q) {
#pragma unroll
			for (int c = 0; c < 6; c++) cross_store(o, cst, (size_t)c * Q + q, f[k][c]);
		}
	}
}

template <typename S, bool HINT>
__device__ __forceinline__ void pcross_grid(const sxsk_pose *__restrict__ poses, int npose, int combo_base, int ncombo,
                                            const typename Cx<S>::T *__restrict__ P,
                                            const typename Cx<S>::T *__restrict__ R, const double2 *__restrict__ tw,
                                            const typename CrossT<S>::T *__restrict__ cst, int Q, int L,
                                            typename CrossT<S>::T *__restrict__ cross)
{
	typedef typename Cx<S>::T V;
	__shared__ V tws[2 * SXS_LMAX_K - 1];
	int N = 2 * L + 1;
	for (int k = threadIdx.x; k < N; k += blockDim.x) tws[k] = from2<V>(tw[k]);
	__syncthreads();
	int bpt = (npose + PC_PPB - 1) / PC_PPB;
	int t = blockIdx.x / bpt, pb = blockIdx.x % bpt;
	pcross_block<S, HINT>(poses, npose, combo_base, ncombo, P, R, tws, cst, Q, L, cross, t, pb);
}

template <typename S, bool HINT>
__global__ void __launch_bounds__(128)
k_pose_cross(const sxsk_pose *__restrict__ poses, int npose, int combo_base, int ncombo,
             const typename Cx<S>::T *__restrict__ P, const typename Cx<S>::T *__restrict__ R,
             const double2 *__restrict__ tw, const typename CrossT<S>::T *__restrict__ cst, int Q, int L,
             typename CrossT<S>::T *__restrict__ cross)
{
	pcross_grid<S, HINT>(poses, npose, combo_base, ncombo, P, R, tw, cst, Q, L, cross);
}

/* The same with the loads of two pairs in flight: 93 registers and POSE_DEEP
 * blocks on an SM instead of 56 and POSE_FLAT.  Faster where rows come from
 * DRAM (pose_deep below). */
#define POSE_FLAT 9
#define POSE_DEEP 5
__global__ void __launch_bounds__(128, POSE_DEEP)
k_pose_cross_deep(const sxsk_pose *__restrict__ poses, int npose, int combo_base, int ncombo,
                  const float2 *__restrict__ P, const float2 *__restrict__ R, const double2 *__restrict__ tw,
                  const float2 *__restrict__ cst, int Q, int L, float2 *__restrict__ cross)
{
	chain_begin();
	pcross_grid<float, true>(poses, npose, combo_base, ncombo, P, R, tw, cst, Q, L, cross);
	chain_end();
}

/* per-pose blocks of many chunks (mixed path); the twiddles are restaged
 * when an item's job has other ones than the previous item's */
__global__ void __launch_bounds__(128)
k_pose_cross_batch(const sxsk_pc_job *__restrict__ jobs, const int4 *__restrict__ items, int nitems, int *ctr)
{
	__shared__ float2 tws[2 * SXS_LMAX_K - 1];
	const double2 *cur = nullptr;
	int curL = -1;
	__shared__ int s_it;
	int nxt = 0;
	for (int it = item_begin(ctr, &s_it); it < nitems; it = item_advance(ctr, &s_it, nxt, nitems)) {
		nxt = item_claim(ctr);
		int4 w = items[it];
		sxsk_pc_job j = jobs[w.x];
		if (j.tw != cur || j.L != curL) {
			int N = 2 * j.L + 1;
			for (int k = threadIdx.x; k < N; k += blockDim.x) tws[k] = from2<float2>(j.tw[k]);
			__syncthreads();
			cur = j.tw;
			curL = j.L;
		}
		pcross_block<float, true>(j.poses, j.npose, j.combo_base, j.ncombo, (const float2 *)j.P,
		                          (const float2 *)j.R, tws, (const float2 *)j.cst, j.Q, j.L, (float2 *)j.cross, w.y,
		                          w.z);
	}
}

__global__ void k_pose_decode(const int64_t *__restrict__ index, int64_t n, int N, int nb, int nz,
                              sxsk_pose *__restrict__ tmp, int32_t *__restrict__ key, int32_t *__restrict__ cnt,
                              int32_t *__restrict__ zused, unsigned long long *__restrict__ err)
{
	int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	int64_t v = index[i];
	if (v < 0) {
		atomicMin(&err[0], (unsigned long long)i);
		return;
	}
	sxsk_pose ps;
	ps.g2 = (int32_t)(v % N); v /= N;
	ps.g1 = (int32_t)(v % N); v /= N;
	ps.a2 = (int32_t)(v % N); v /= N;
	ps.b2 = (int32_t)(v % nb); v /= nb;
	ps.b1 = (int32_t)(v % nb); v /= nb;
	if (v >= nz) {
		atomicMin(&err[1], (unsigned long long)i);
		return;
	}
	ps.zi = (int32_t)v;
	ps.src = (int32_t)i;
	ps.combo = 0;
	int32_t k = (ps.zi * nb + ps.b2) * N + ps.g2;
	tmp[i] = ps;
	key[i] = k;
	atomicAdd(&cnt[k], 1);
	zused[ps.zi] = 1;
}

__global__ void k_pose_scatter(const sxsk_pose *__restrict__ tmp, const int32_t *__restrict__ key, int64_t n,
                               int32_t *__restrict__ pos, const int32_t *__restrict__ cid,
                               sxsk_pose *__restrict__ out)
{
	int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	int32_t k = key[i];
	sxsk_pose ps = tmp[i];
	ps.combo = cid[k];
	out[atomicAdd(&pos[k], 1)] = ps;
}

/* Grid fit (src/min_saxs.c:170-188 peak rescale, 261-320 best scale,
 * 391-448 point_score).  For one pose and one (c1, c2) cell the model at q_i
 * is in_i = al_i + c2 be_i + c2^2 ga_i with G_i = c1^3 exp(-mult (c1^2-1) q_i^2),
 * al = VV - G VD + G^2 DD, be = VW - G DW, ga = WW; point_score's piecewise
 * line is tan_i = (in_i - in_{i-1}) h_i (tan_0 = 0), buf_i = in_i - tan_i q_i,
 * and with the best scale k = up/down the score is sum a0 + k(-2 up + k down),
 *   up   = sum_i a1 buf + a2 tan = sum_i a1 in + u_i D_i
 *   down = sum_i a3 buf^2 + 2 a4 buf tan + a5 tan^2
 *        = sum_i a3 in^2 + 2 e_i in D_i + f_i D_i^2
 * where D_i = in_i - in_{i-1} and the per-q constants are folded on the host:
 *   fc[i] = {a3, e = (a4 - q a3) h, f = (a5 - 2 q a4 + q^2 a3) h^2, a1,
 *            u = (a2 - q a1) h}.
 * up is quadratic and down quartic in c2, so per (pose, c1) one pass over q
 * yields their coefficients and every c2 cell costs a few multiply-adds.
 * One thread per (pose, c1): no reductions and no repeated q work.  Within
 * a thread cells are ranked by up^2/down (score = sum a0 - up^2/down); the
 * threads of a pose then compare their best scores, ties going to the lower
 * cell index as in a c1-major scan. */
#define FIT_THREADS 128
#define FIT_NFC 5
/* Persistent: block b handles pose groups b, b + gridDim.x, ...; a group is
 * ppb consecutive slots of the pose order (order[slot].src is the pose's
 * position in cross and in the outputs; slot itself when order is NULL). */
__global__ void __launch_bounds__(FIT_THREADS)
k_fit_grid(const double *__restrict__ cross, const sxsk_pose *__restrict__ order, int slot0, int nslot, int Q,
           const double *__restrict__ fc, double a0sum, double peak, const double *__restrict__ gtab,
           const double *__restrict__ c1g, int n1, const double *__restrict__ c2g, int n2, int tp, int ppb,
           double *__restrict__ chi, double *__restrict__ c1o, double *__restrict__ c2o, int32_t *__restrict__ cello,
           double *__restrict__ grid)
{
	extern __shared__ double sm[];
	double *cs = sm;                                   /* [ppb][8][Q]: VV VD VW DD DW WW P3 P4 */
	double *fs = cs + (size_t)ppb * 8 * Q;             /* [FIT_NFC][Q] */
	double *c2s = fs + (size_t)FIT_NFC * Q;            /* [n2] */
	double *red = c2s + n2;                            /* [ppb*tp][2] partials / best score */
	int *redc = (int *)(red + 2 * ppb * tp);           /* [ppb*tp] best cell */
	double *sf = (double *)(redc + ((ppb * tp + 1) & ~1)); /* [ppb][3]: scale, U2, D4 */
	int *srcs = (int *)(sf + 3 * ppb);                 /* [ppb] pose index of each slot */
	int tid = threadIdx.x;
	int nthr = ppb * tp;
	int lp = tid / tp, lt = tid % tp;
	const double *F3 = fs, *FE = fs + Q, *FF = fs + 2 * Q, *F1 = fs + 3 * Q, *FU = fs + 4 * Q;

	for (int k = tid; k < FIT_NFC * Q; k += blockDim.x) fs[k] = fc[(k % Q) * FIT_NFC + k / Q];
	for (int k = tid; k < n2; k += blockDim.x) c2s[k] = c2g[k];
	int ngroup = (nslot + ppb - 1) / ppb;
	for (int grp = blockIdx.x; grp < ngroup; grp += gridDim.x) {
		int s0 = grp * ppb;
		int nhere = min(ppb, nslot - s0);
		bool live = tid < nthr && lp < nhere;
		__syncthreads();   /* previous group done with the shared arrays */
		if (tid < nhere) srcs[tid] = order ? order[slot0 + s0 + tid].src : slot0 + s0 + tid;
		__syncthreads();
		for (int k = tid; k < nhere * 6 * Q; k += blockDim.x) {
			int p = k / (6 * Q), r = k % (6 * Q);
			cs[(size_t)p * 8 * Q + r] = cross[(size_t)srcs[p] * 6 * Q + r];
		}
		__syncthreads();
		if (live && lt == 0) {
			const double *c = cs + (size_t)lp * 8 * Q;
			double sc = c[0] + c[3 * Q] + c[5 * Q] + c[2 * Q] - c[Q] - c[4 * Q];
			sf[3 * lp] = peak / sc;
		}
		__syncthreads();
		for (int k = tid; k < nhere * 6 * Q; k += blockDim.x) {
			int p = k / (6 * Q), r = k % (6 * Q);
			cs[(size_t)p * 8 * Q + r] *= sf[3 * p];
		}
		__syncthreads();
		double *c = cs + (size_t)lp * 8 * Q;
		const double *VV = c, *VD = c + Q, *VW = c + 2 * Q, *DD = c + 3 * Q, *DW = c + 4 * Q, *WW = c + 5 * Q;
		double *P3 = c + 6 * Q, *P4 = c + 7 * Q;
		/* c1-independent part: M (ga, D_ga) per q, and the c2^2 coefficients */
		if (live) {
			double u2 = 0, d4 = 0;
			for (int i = lt; i < Q; i += tp) {
				double ga = WW[i], dg = i > 0 ? ga - WW[i - 1] : 0.0;
				double p3 = fma(F3[i], ga, FE[i] * dg);
				double p4 = fma(FE[i], ga, FF[i] * dg);
				P3[i] = p3;
				P4[i] = p4;
				u2 = fma(F1[i], ga, fma(FU[i], dg, u2));
				d4 = fma(ga, p3, fma(dg, p4, d4));
			}
			red[2 * tid] = u2;
			red[2 * tid + 1] = d4;
		}
		__syncthreads();
		if (live && lt == 0) {
			double u2 = 0, d4 = 0;
			for (int t = 0; t < tp; t++) {
				u2 += red[2 * (tid + t)];
				d4 += red[2 * (tid + t) + 1];
			}
			sf[3 * lp + 1] = u2;
			sf[3 * lp + 2] = d4;
		}
		__syncthreads();
		double bscore = __longlong_as_double(0x7ff0000000000000LL);
		int bcell = -1;
		int pid = live ? srcs[lp] : 0;
		if (live) {
			double U2 = sf[3 * lp + 1], D4 = sf[3 * lp + 2];
			for (int j = lt; j < n1; j += tp) {
				const double *G = gtab + (size_t)j * Q;
				double U0 = 0, U1 = 0, D0 = 0, D1 = 0, D2a = 0, D2b = 0, D3 = 0;
				double g = __ldg(G);
				double alp = fma(g, fma(g, DD[0], -VD[0]), VV[0]);
				double bep = fma(-g, DW[0], VW[0]);
				for (int i = 0; i < Q; i++) {
					g = __ldg(G + i);
					double al = fma(g, fma(g, DD[i], -VD[i]), VV[i]);
					double be = fma(-g, DW[i], VW[i]);
					double d0 = al - alp, d1 = be - bep;
					double f3 = F3[i], fe = FE[i], ff = FF[i];
					double m0a = fma(f3, al, fe * d0), m0b = fma(fe, al, ff * d0);
					double m1a = fma(f3, be, fe * d1), m1b = fma(fe, be, ff * d1);
					double p3 = P3[i], p4 = P4[i];
					D0 = fma(al, m0a, fma(d0, m0b, D0));
					D1 = fma(be, m0a, fma(d1, m0b, D1));
					D2a = fma(be, m1a, fma(d1, m1b, D2a));
					D2b = fma(al, p3, fma(d0, p4, D2b));
					D3 = fma(be, p3, fma(d1, p4, D3));
					double f1 = F1[i], fu = FU[i];
					U0 = fma(f1, al, fma(fu, d0, U0));
					U1 = fma(f1, be, fma(fu, d1, U1));
					alp = al;
					bep = be;
				}
				D1 *= 2.0;
				double D2 = fma(2.0, D2b, D2a);
				D3 *= 2.0;
				/* best c2 of this c1 by up^2/down, then its score */
				double bu = 0, bd = 0;
				int bi = -1;
				for (int i2 = 0; i2 < n2; i2++) {
					double c2 = c2s[i2];
					double up = fma(c2, fma(c2, U2, U1), U0);
					double down = fma(c2, fma(c2, fma(c2, fma(c2, D4, D3), D2), D1), D0);
					if (grid) {
						double k = up / down;
						grid[((size_t)pid * n1 + j) * n2 + i2] = a0sum + k * (-2.0 * up + k * down);
					}
					if (down > 0.0) {
						double num = up * up;
						if (bi < 0 || num * bd > bu * bu * down) { bu = up; bd = down; bi = i2; }
					}
				}
				if (bi >= 0) {
					double k = bu / bd;
					double score = a0sum + k * (-2.0 * bu + k * bd);
					int cell = j * n2 + bi;
					if (score < bscore || (score == bscore && cell < bcell)) { bscore = score; bcell = cell; }
				}
			}
			red[2 * tid] = bscore;
			redc[tid] = bcell;
		}
		__syncthreads();
		if (live && lt == 0) {
			for (int t = 1; t < tp; t++) {
				double os = red[2 * (tid + t)];
				int oc = redc[tid + t];
				if (oc >= 0 && (bcell < 0 || os < bscore || (os == bscore && oc < bcell))) { bscore = os; bcell = oc; }
			}
			if (bcell >= 0) {
				chi[pid] = sqrt(bscore);
				c1o[pid] = c1g[bcell / n2];
				c2o[pid] = c2g[bcell % n2];
			} else {
				chi[pid] = __longlong_as_double(0x7ff8000000000000LL);
				c1o[pid] = __longlong_as_double(0x7ff8000000000000LL);
				c2o[pid] = __longlong_as_double(0x7ff8000000000000LL);
			}
			if (cello) cello[pid] = bcell;
		}
	}
}

inline int nblk(long n, int b) { return (int)((n + b - 1) / b); }

} // namespace

template <typename S, int NB>
static cudaError_t translate_col_launch(const void *U, const void *tau, const int32_t *combo_zbg,
                                        const int32_t *slices, int nslice, int cbase, int ncombo, int nzt, int NT,
                                        int L, void *R, int sb, bool *linked, cudaStream_t s)
{
	typedef typename Cx<S>::T V;
	int K = L + 1;
	/* m with n = K - m in (NB - 4, NB] */
	int m_hi = K - (NB - 3), m_lo = K - NB;
	if (m_hi > L) m_hi = L;
	if (m_lo < 0) m_lo = 0;
	if (m_hi < m_lo) return cudaSuccess;
	int nm = m_hi - m_lo + 1;
	if constexpr (sizeof(S) == 4) {
		/* FP32: three channels per thread, pipelined over runs of slices */
		long nb = (long)NT * ((nslice + sb - 1) / sb) * nm;
		if (nb > 0x7fffffffL) return cudaErrorInvalidValue;
		size_t smem = TR_SMEM(NB);
		auto kern = k_translate_pipe<NB>;
		if (smem > 48 * 1024) {
			cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		/* blocks of 75-131 KB (NB 20-32) need the largest carveout */
		cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
		                                     (int)cudaSharedmemCarveoutMaxShared);
		if (e != cudaSuccess) return e;
		e = chain_launch(kern, (unsigned)nb, TCOL_THREADS(3), smem, s, *linked, (const float2 *)U, (const float *)tau,
		                 combo_zbg, slices, nslice, cbase, ncombo, L, nzt, m_lo, nm, sb, (float2 *)R);
		*linked = true;
		return e;
	} else {
		/* FP64 (bound by its pipe): one channel per thread */
		long nb = (long)NT * nslice * nm;
		if (nb > 0x7fffffffL) return cudaErrorInvalidValue;
		size_t smem = sizeof(S) * SXS_QT * (NB * NB + 4);
		auto kern = k_translate_col<S, NB, 1>;
		if (smem > 48 * 1024) {
			cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
			if (e != cudaSuccess) return e;
		}
		kern<<<(unsigned)nb, TCOL_THREADS(1), smem, s>>>((const V *)U, (const S *)tau, combo_zbg, slices, nslice,
		                                                 cbase, ncombo, L, nzt, m_lo, nm, (V *)R);
		return cudaGetLastError();
	}
}

template <typename S>
static cudaError_t translate_col_all(const void *U, const void *tau, const int32_t *combo_zbg, const int32_t *slices,
                                     int nslice, int cbase, int ncombo, int nzt, int NT, int L, void *R, int sb,
                                     cudaStream_t s)
{
	cudaError_t e = cudaSuccess;
	bool linked = false;
	if (!e) e = translate_col_launch<S, 4>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, sb, &linked, s);
	if (!e) e = translate_col_launch<S, 8>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, sb, &linked, s);
	if (!e) e = translate_col_launch<S, 12>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, sb, &linked, s);
	if (!e) e = translate_col_launch<S, 16>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, sb, &linked, s);
	if (!e) e = translate_col_launch<S, 20>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, sb, &linked, s);
	if (!e) e = translate_col_launch<S, 24>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, sb, &linked, s);
	if (!e) e = translate_col_launch<S, 28>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, sb, &linked, s);
	if (!e) e = translate_col_launch<S, 32>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, sb, &linked, s);
	return e;
}

static int translate_slices(const void *U, const void *tau, const int32_t *combo_zbg, const int32_t *slices, int nslice,
                   int cbase, int ncombo, int nzt, int Q, int L, void *R, int fp32, cudaStream_t s)
{
	int K = L + 1, NT = (Q + SXS_QT - 1) / SXS_QT, NP = K * (K + 1) / 2;
	long nb = (long)NT * nslice * ((NP + TR_PB - 1) / TR_PB);
	if (nb > 0x7fffffffL) return cudaErrorInvalidValue;
	/* row stride of the staged tau: the pairs of a half warp start on
	 * distinct banks */
	int ts = K * SXS_QT, tgt = SXS_QT >= 16 ? 16 : 8;
	while (ts % 32 != tgt) ts += SXS_QT;
	size_t elem = fp32 ? sizeof(float) : sizeof(double), smem = (size_t)TR_PB * ts * elem;
	size_t most = (size_t)TR_PB * (SXS_LMAX_K * SXS_QT + 32) * elem;
	if (fp32) {
		cudaError_t e = smem_bound(k_translate<float>, smem, most);
		if (e != cudaSuccess) return e;
		k_translate<float><<<(unsigned)nb, 128, smem, s>>>((const float2 *)U, (const float *)tau, combo_zbg, slices,
		                                                    nslice, cbase, ncombo, L, nzt, ts, (float2 *)R);
	} else {
		cudaError_t e = smem_bound(k_translate<double>, smem, most);
		if (e != cudaSuccess) return e;
		k_translate<double><<<(unsigned)nb, 128, smem, s>>>((const double2 *)U, (const double *)tau, combo_zbg,
		                                                     slices, nslice, cbase, ncombo, L, nzt, ts,
		                                                     (double2 *)R);
	}
	return cudaGetLastError();
}

template <typename S, int G>
static int rotate_launch(const void *spf_t, const void *dtab, const double2 *tw, int Q, int L, int conj, void *out,
                         cudaStream_t s)
{
	typedef typename Cx<S>::T V;
	int K = L + 1, NT = (Q + SXS_QT - 1) / SXS_QT;
	/* three channels per thread in FP32 (one twiddle load for three) while
	 * their 12 G accumulators leave room for warps (G <= 6, L <= 23: measured
	 * 1.10 -> 1.04 ms at L = 20); FP64 is bound by its arithmetic pipe and
	 * keeps one */
	constexpr int CH = sizeof(S) == 4 ? 3 : 1;
	size_t smem = sizeof(RotTw<S>) * (size_t)ROT_NTW(L, G);
	auto kern = k_rotate<S, G, CH>;
	cudaError_t e = smem_bound(kern, smem, sizeof(RotTw<S>) * (size_t)ROT_NTW(SXS_LMAX_K - 1, G));
	if (e != cudaSuccess) return e;
	long nb = (long)K * K * NT;
	if (nb > 0x7fffffffL) return cudaErrorInvalidValue;
	kern<<<(unsigned)nb, ROT_THREADS(CH), smem, s>>>((const V *)spf_t, (const S *)dtab, tw, Q, L, conj, (V *)out);
	return cudaGetLastError();
}

template <int G>
static int rotate2_launch(const void *spf_t, const void *dtab, const double2 *tw, int Q, int L, int conj, void *out,
                          cudaStream_t s)
{
	int K = L + 1, NT = (Q + SXS_QT - 1) / SXS_QT;
	size_t smem = ROT2_SMEM(L) + sizeof(RotTw<float>) * (size_t)ROT_NTW(L, G);
	auto kern = k_rotate2<G>;
	cudaError_t e = smem_bound(kern, smem, ROT2_SMEM(SXS_LMAX_K - 1) +
	                                           sizeof(RotTw<float>) * (size_t)ROT_NTW(SXS_LMAX_K - 1, G));
	if (e != cudaSuccess) return e;
	long nb = (long)K * ((K + 1) / 2) * NT;
	if (nb > 0x7fffffffL) return cudaErrorInvalidValue;
	kern<<<(unsigned)nb, ROT2_THREADS, smem, s>>>((const float2 *)spf_t, (const float *)dtab, tw, Q, L, conj,
	                                              (float2 *)out);
	return cudaGetLastError();
}

extern "C" int sxsk_rotate_betas(int G) { return G >= ROT2_G ? 2 : 1; }

extern "C" int sxsk_rotate_group(int L, int gsel)
{
	int need = (L + 1 + ROT_GROUPS - 1) / ROT_GROUPS;
	if (gsel > need) need = gsel;
	static const int gs[6] = {2, 4, 6, 8, 12, 16};
	for (int i = 0; i < 6; i++)
		if (need <= gs[i]) return gs[i];
	return 0;
}

template <typename S>
static int rotate_any(const void *spf_t, const void *dtab, const double2 *tw, int Q, int L, int conj, void *out,
                      int gsel, cudaStream_t s)
{
	/* gamma pairs per thread: at least the L + 1 pairs over ROT_GROUPS
	 * groups; a larger choice (gsel) leaves groups idle for fewer blocks'
	 * worth of twiddle setup */
	constexpr bool f32 = sizeof(S) == 4;
	switch (sxsk_rotate_group(L, gsel)) {
	case 2: return rotate_launch<S, 2>(spf_t, dtab, tw, Q, L, conj, out, s);
	case 4: return rotate_launch<S, 4>(spf_t, dtab, tw, Q, L, conj, out, s);
	case 6: return rotate_launch<S, 6>(spf_t, dtab, tw, Q, L, conj, out, s);
	case 8:
		if constexpr (f32) return rotate2_launch<8>(spf_t, dtab, tw, Q, L, conj, out, s);
		else return rotate_launch<S, 8>(spf_t, dtab, tw, Q, L, conj, out, s);
	case 12:
		if constexpr (f32) return rotate2_launch<12>(spf_t, dtab, tw, Q, L, conj, out, s);
		else return rotate_launch<S, 12>(spf_t, dtab, tw, Q, L, conj, out, s);
	case 16:
		if constexpr (f32) return rotate2_launch<16>(spf_t, dtab, tw, Q, L, conj, out, s);
		else return rotate_launch<S, 16>(spf_t, dtab, tw, Q, L, conj, out, s);
	default: return cudaErrorInvalidValue;
	}
}

/* grid of a batched launch: persistent (ctr != NULL), every resident block
 * of the kernel on every SM, at most one block per item; else one block
 * per item */
template <typename F>
static cudaError_t persistent_grid(F kern, int threads, size_t smem, int nitems, const int *ctr, int *grid)
{
	if (!ctr) {
		*grid = nitems;
		return cudaSuccess;
	}
	int dev = 0, nsm = 0, per = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (!e) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
	if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem);
	if (e) return e;
	if (per < 1) return cudaErrorInvalidConfiguration;
	long g = (long)nsm * per;
	*grid = (int)(g < nitems ? g : nitems);
	return cudaSuccess;
}

template <int G>
static int rotate_batch_launch(const sxsk_rot_job *jobs, const int4 *items, int nitems, int tw_max, int l_max, int *ctr,
                               cudaStream_t s)
{
	constexpr int threads = G >= ROT2_G ? ROT2_THREADS : ROT_THREADS(3);   /* the FP32 choice of rotate_launch */
	size_t smem = sizeof(RotTw<float>) * (size_t)tw_max;
	if (G >= ROT2_G) smem = (smem + 15) / 16 * 16 + ROT2_SMEM(l_max);
	auto kern = k_rotate_batch<G>;
	cudaError_t e = smem_bound(kern, smem, sizeof(RotTw<float>) * (size_t)ROT_NTW(SXS_LMAX_K - 1, G) + 16 +
	                                           (G >= ROT2_G ? ROT2_SMEM(SXS_LMAX_K - 1) : 0));
	int grid = 0;
	if (!e) e = persistent_grid(kern, threads, smem, nitems, ctr, &grid);
	if (e) return e;
	kern<<<grid, threads, smem, s>>>(jobs, items, nitems, tw_max, ctr);
	return cudaGetLastError();
}

template <int NB>
static int translate_batch_launch(const sxsk_tr_job *jobs, const int4 *items, int nitems, int *ctr, cudaStream_t s)
{
	size_t smem = TR_SMEM(NB);
	auto kern = k_translate_batch<NB>;
	cudaError_t e = cudaSuccess;
	if (smem > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (!e)
		e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
		                         (int)cudaSharedmemCarveoutMaxShared);
	int grid = 0;
	if (!e) e = persistent_grid(kern, TCOL_THREADS(3), smem, nitems, ctr, &grid);
	if (e) return e;
	kern<<<grid, TCOL_THREADS(3), smem, s>>>(jobs, items, nitems, ctr);
	return cudaGetLastError();
}

template <int NB>
static cudaError_t translate_fused_launch(const float2 *U, const float *tau, const int32_t *combo_zbg,
                                          const int32_t *slices, int nslice, int cbase, int nzt, int NT, int L, int sb,
                                          const sxsk_pose *poses, const int32_t *cstart, int pose_base,
                                          const float2 *P, const double2 *tw, float *part, cudaStream_t s)
{
	int K = L + 1;
	int m_hi = K - (NB - 3), m_lo = K - NB;
	if (m_hi > L) m_hi = L;
	if (m_lo < 0) m_lo = 0;
	if (m_hi < m_lo) return cudaSuccess;
	int nm = m_hi - m_lo + 1;
	long nb = (long)NT * ((nslice + sb - 1) / sb) * nm;
	if (nb > 0x7fffffffL) return cudaErrorInvalidValue;
	size_t smem = TF_SMEM(NB);
	auto kern = k_translate_fused<NB>;
	cudaError_t e = cudaSuccess;
	if (smem > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (!e)
		e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
		                         (int)cudaSharedmemCarveoutMaxShared);
	if (e) return e;
	kern<<<(unsigned)nb, TCOL_THREADS(3), smem, s>>>(U, tau, combo_zbg, slices, nslice, cbase, L, nzt, m_lo, nm, sb,
	                                                 poses, cstart, pose_base, P, tw, part, NT * SXS_QT);
	return cudaGetLastError();
}

template <int NB>
static int translate_fused_batch_launch(const sxsk_tf_job *jobs, const int4 *items, int nitems, int *ctr,
                                        cudaStream_t s)
{
	size_t smem = TF_SMEM(NB);
	auto kern = k_translate_fused_batch<NB>;
	cudaError_t e = cudaSuccess;
	if (smem > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
	if (!e)
		e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
		                         (int)cudaSharedmemCarveoutMaxShared);
	int grid = 0;
	if (!e) e = persistent_grid(kern, TCOL_THREADS(3), smem, nitems, ctr, &grid);
	if (e) return e;
	kern<<<grid, TCOL_THREADS(3), smem, s>>>(jobs, items, nitems, ctr);
	return cudaGetLastError();
}

extern "C" {

int sxsk_spf_transpose(const double *flat, void *spf_t, int Q, int L, int fp32, cudaStream_t s)
{
	int K2 = (L + 1) * (L + 1);
	if (fp32) k_spf_transpose<float><<<nblk(3L * Q * K2, 256), 256, 0, s>>>(flat, (float2 *)spf_t, Q, K2);
	else k_spf_transpose<double><<<nblk(3L * Q * K2, 256), 256, 0, s>>>(flat, (double2 *)spf_t, Q, K2);
	return cudaGetLastError();
}

int sxsk_rotate(const void *spf_t, const void *dtab, const double2 *tw, int Q, int L, int conj, void *out, int fp32,
                int gsel, cudaStream_t s)
{
	if (L < 0 || L + 1 > SXS_LMAX_K || Q <= 0) return cudaErrorInvalidValue;
	if (fp32) return rotate_any<float>(spf_t, dtab, tw, Q, L, conj, out, gsel, s);
	return rotate_any<double>(spf_t, dtab, tw, Q, L, conj, out, gsel, s);
}

int sxsk_pose_decode(const int64_t *index, int64_t n, int N, int nb, int nz, sxsk_pose *tmp, int32_t *key,
                     int32_t *cnt, int32_t *zused, unsigned long long *err, cudaStream_t s)
{
	if (n <= 0) return 0;
	long nbk = (n + 255) / 256;
	if (nbk > 0x7fffffffL) return cudaErrorInvalidValue;
	k_pose_decode<<<(unsigned)nbk, 256, 0, s>>>(index, n, N, nb, nz, tmp, key, cnt, zused, err);
	return cudaGetLastError();
}

int sxsk_pose_scatter(const sxsk_pose *tmp, const int32_t *key, int64_t n, int32_t *pos, const int32_t *cid,
                      sxsk_pose *out, cudaStream_t s)
{
	if (n <= 0) return 0;
	long nbk = (n + 255) / 256;
	if (nbk > 0x7fffffffL) return cudaErrorInvalidValue;
	k_pose_scatter<<<(unsigned)nbk, 256, 0, s>>>(tmp, key, n, pos, cid, out);
	return cudaGetLastError();
}

int sxsk_translate_class(const void *U, const void *tau, const int32_t *combo_zbg, const int32_t *slices, int nslice,
                         int cbase, int ncombo, int nzt, int Q, int L, void *R, int sb, int NB, int linked, cudaStream_t s)
{
	if (nslice <= 0) return 0;
	if (L + 1 > 32) return cudaErrorInvalidValue;
	int NT = (Q + SXS_QT - 1) / SXS_QT;
	if (sb < 1) sb = SXSK_TP_SB;
	bool lk = linked;
#define TCL(C)                                                                                                     \
	case C:                                                                                                        \
		return translate_col_launch<float, C>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, sb,  \
		                                      &lk, s);
	switch (NB) {
		TCL(4) TCL(8) TCL(12) TCL(16) TCL(20) TCL(24) TCL(28) TCL(32)
	default: return cudaErrorInvalidValue;
	}
#undef TCL
}

int sxsk_translate_launches(int L)
{
	int K = L + 1;
	if (K > 32) return 1;
	int n = 0;
	for (int nb = 4; nb <= 32; nb += 4) {
		/* the m range of translate_col_launch<S, nb> */
		int m_hi = K - (nb - 3), m_lo = K - nb;
		if (m_hi > L) m_hi = L;
		if (m_lo < 0) m_lo = 0;
		n += m_hi >= m_lo;
	}
	return n;
}

int sxsk_translate(const void *U, const void *tau, const int32_t *combo_zbg, const int32_t *slices, int nslice,
                   int cbase, int ncombo, int nzt, int Q, int L, void *R, int fp32, int sb, cudaStream_t s)
{
	if (nslice <= 0) return 0;
	int NT = (Q + SXS_QT - 1) / SXS_QT;
	if (sb < 1) sb = SXSK_TP_SB;
	if (L + 1 <= 32) {
		if (fp32)
			return translate_col_all<float>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, sb, s);
		return translate_col_all<double>(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, NT, L, R, sb, s);
	}
	return translate_slices(U, tau, combo_zbg, slices, nslice, cbase, ncombo, nzt, Q, L, R, fp32, s);
}

size_t sxsk_fused_part_floats(int L, int Q)
{
	return (size_t)(L + 1) * 6 * ((Q + SXS_QT - 1) / SXS_QT) * SXS_QT;
}

int sxsk_translate_fused(const void *U, const void *tau, const int32_t *combo_zbg, const int32_t *slices, int nslice,
                         int cbase, int nzt, int Q, int L, int sb, const sxsk_pose *poses, const int32_t *cstart,
                         int pose_base, const void *P, const double2 *tw, float *part, cudaStream_t s)
{
	if (nslice <= 0) return 0;
	if (L + 1 > 32) return cudaErrorInvalidValue;
	int NT = (Q + SXS_QT - 1) / SXS_QT;
	if (sb < 1) sb = SXSK_TP_SB;
	const float2 *u = (const float2 *)U, *p = (const float2 *)P;
	const float *ta = (const float *)tau;
	cudaError_t e = cudaSuccess;
#define TFL(NB)                                                                                                     \
	if (!e) e = translate_fused_launch<NB>(u, ta, combo_zbg, slices, nslice, cbase, nzt, NT, L, sb, poses, cstart, \
	                                       pose_base, p, tw, part, s);
	TFL(4) TFL(8) TFL(12) TFL(16) TFL(20) TFL(24) TFL(28) TFL(32)
#undef TFL
	return e;
}

int sxsk_translate_fused_class(const void *U, const void *tau, const int32_t *combo_zbg, const int32_t *slices,
                               int nslice, int cbase, int nzt, int Q, int L, int sb, const sxsk_pose *poses,
                               const int32_t *cstart, int pose_base, const void *P, const double2 *tw, float *part,
                               int NB, cudaStream_t s)
{
	if (nslice <= 0) return 0;
	if (L + 1 > 32) return cudaErrorInvalidValue;
	int NT = (Q + SXS_QT - 1) / SXS_QT;
	if (sb < 1) sb = SXSK_TP_SB;
	const float2 *u = (const float2 *)U, *p = (const float2 *)P;
	const float *ta = (const float *)tau;
#define TFC(C)                                                                                                     \
	case C:                                                                                                        \
		return translate_fused_launch<C>(u, ta, combo_zbg, slices, nslice, cbase, nzt, NT, L, sb, poses, cstart,   \
		                                 pose_base, p, tw, part, s);
	switch (NB) {
		TFC(4) TFC(8) TFC(12) TFC(16) TFC(20) TFC(24) TFC(28) TFC(32)
	default: return cudaErrorInvalidValue;
	}
#undef TFC
}

int sxsk_fused_reduce(const sxsk_pose *poses, int npose, const float *part, int Q, int L, const void *cst,
                      void *cross, cudaStream_t s)
{
	if (npose <= 0) return 0;
	int QP = ((Q + SXS_QT - 1) / SXS_QT) * SXS_QT;
	long n = (long)npose * Q;
	k_fused_reduce<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(poses, npose, part, L + 1, Q, QP, (const float2 *)cst,
	                                                            (float2 *)cross);
	return cudaGetLastError();
}

/* Which form of the FP32 per-pose kernel: per pose, one row of P and 1 / (poses
 * per combo) rows of R are read; all of R and the part of the tile's P rows
 * beyond ~100 of the 129 MB of L2 come from DRAM.  Above 0.6 rows of those per
 * pose the deep form is faster, below it the occupancy of the flat one is (it
 * is bound by L2 there).  Flat / deep, ms:
 *   L   Q    poses    DRAM rows   flat    deep
 *   20  101   6,000   0.81        0.739   0.623
 *   20  101  12,000   0.67        1.009   0.989
 *   20  101  20,000   0.53        1.380   1.438
 *   25  101  20,000   0.65        2.823   2.366
 *   25  101  40,000   0.45        3.977   4.086
 *   30  201  60,000   0.87       23.60   18.12
 *   30  101 100,000   0.73       14.97   13.31
 *   28  101 150,000   0.46       14.57   15.83
 * A launch that fits the SMs at once only in the flat form keeps it (L = 15,
 * Q = 51, 4,000 poses, 875 blocks: 0.143 and 0.160).  In a chain the deep form
 * alone lets the next launch into its last wave, worth more than its 5 % at up
 * to a few waves (eight dimers of 750 to 12,000 poses, L 10-25: phases of a
 * batch 4.70 ms with it throughout, 5.23 by the rows' rule). */
static bool pose_deep(int npose, int ncombo, int L, long blocks, bool chain)
{
	int K = L + 1, N = 2 * L + 1, NP = K * (K + 1) / 2, dev = 0, nsm = 0;
	double tile = (double)K * N * NP * 3 * SXS_QT * sizeof(float2), miss = 1.0 - 100e6 / tile;
	if (cudaGetDevice(&dev) || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) return false;
	if (chain && blocks <= 8L * POSE_FLAT * nsm) return true;
	if ((double)ncombo / npose + (miss > 0.0 ? miss : 0.0) <= 0.6) return false;
	return blocks <= (long)POSE_DEEP * nsm || blocks > (long)POSE_FLAT * nsm;
}

int sxsk_pose_cross(const sxsk_pose *poses, int npose, int combo_base, int ncombo, const void *P, const void *R,
                    const double2 *tw, const void *cst, int Q, int L, void *cross, int fp32, int linked,
                    cudaStream_t s)
{
	if (npose <= 0) return 0;
	int NT = (Q + SXS_QT - 1) / SXS_QT;
	long nb = (long)NT * ((npose + PC_PPB - 1) / PC_PPB);
	if (nb > 0x7fffffffL) return cudaErrorInvalidValue;
	if (!fp32)
		k_pose_cross<double, false><<<(unsigned)nb, 128, 0, s>>>(poses, npose, combo_base, ncombo, (const double2 *)P,
		                                                   (const double2 *)R, tw, (const double *)cst, Q, L,
		                                                   (double *)cross);
	else if (pose_deep(npose, ncombo, L, nb, linked >= 0))
		return chain_launch(k_pose_cross_deep, (unsigned)nb, 128, 0, s, linked > 0, poses, npose, combo_base, ncombo,
		                    (const float2 *)P, (const float2 *)R, tw, (const float2 *)cst, Q, L, (float2 *)cross);
	else
		k_pose_cross<float, true><<<(unsigned)nb, 128, 0, s>>>(poses, npose, combo_base, ncombo, (const float2 *)P,
		                                                  (const float2 *)R, tw, (const float2 *)cst, Q, L,
		                                                  (float2 *)cross);
	return cudaGetLastError();
}

int sxsk_rotate_batch(const sxsk_rot_job *jobs, const int4 *items, int nitems, int G, int tw_max, int l_max, int *ctr,
                      cudaStream_t s)
{
	if (nitems <= 0) return 0;
	switch (G) {
	case 2: return rotate_batch_launch<2>(jobs, items, nitems, tw_max, l_max, ctr, s);
	case 4: return rotate_batch_launch<4>(jobs, items, nitems, tw_max, l_max, ctr, s);
	case 6: return rotate_batch_launch<6>(jobs, items, nitems, tw_max, l_max, ctr, s);
	case 8: return rotate_batch_launch<8>(jobs, items, nitems, tw_max, l_max, ctr, s);
	case 12: return rotate_batch_launch<12>(jobs, items, nitems, tw_max, l_max, ctr, s);
	case 16: return rotate_batch_launch<16>(jobs, items, nitems, tw_max, l_max, ctr, s);
	default: return cudaErrorInvalidValue;
	}
}

int sxsk_translate_fused_batch(const sxsk_tf_job *jobs, const int4 *items, int nitems, int NB, int *ctr,
                               cudaStream_t s)
{
	if (nitems <= 0) return 0;
	switch (NB) {
	case 4: return translate_fused_batch_launch<4>(jobs, items, nitems, ctr, s);
	case 8: return translate_fused_batch_launch<8>(jobs, items, nitems, ctr, s);
	case 12: return translate_fused_batch_launch<12>(jobs, items, nitems, ctr, s);
	case 16: return translate_fused_batch_launch<16>(jobs, items, nitems, ctr, s);
	case 20: return translate_fused_batch_launch<20>(jobs, items, nitems, ctr, s);
	case 24: return translate_fused_batch_launch<24>(jobs, items, nitems, ctr, s);
	case 28: return translate_fused_batch_launch<28>(jobs, items, nitems, ctr, s);
	case 32: return translate_fused_batch_launch<32>(jobs, items, nitems, ctr, s);
	default: return cudaErrorInvalidValue;
	}
}

int sxsk_fused_reduce_batch(const sxsk_fr_job *jobs, const int4 *items, int nitems, int *ctr, cudaStream_t s)
{
	if (nitems <= 0) return 0;
	int grid = 0;
	cudaError_t e = persistent_grid(k_fused_reduce_batch, 128, 0, nitems, ctr, &grid);
	if (e) return e;
	k_fused_reduce_batch<<<grid, 128, 0, s>>>(jobs, items, nitems, ctr);
	return cudaGetLastError();
}

int sxsk_translate_batch(const sxsk_tr_job *jobs, const int4 *items, int nitems, int NB, int *ctr, cudaStream_t s)
{
	if (nitems <= 0) return 0;
	switch (NB) {
	case 4: return translate_batch_launch<4>(jobs, items, nitems, ctr, s);
	case 8: return translate_batch_launch<8>(jobs, items, nitems, ctr, s);
	case 12: return translate_batch_launch<12>(jobs, items, nitems, ctr, s);
	case 16: return translate_batch_launch<16>(jobs, items, nitems, ctr, s);
	case 20: return translate_batch_launch<20>(jobs, items, nitems, ctr, s);
	case 24: return translate_batch_launch<24>(jobs, items, nitems, ctr, s);
	case 28: return translate_batch_launch<28>(jobs, items, nitems, ctr, s);
	case 32: return translate_batch_launch<32>(jobs, items, nitems, ctr, s);
	default: return cudaErrorInvalidValue;
	}
}

int sxsk_pose_cross_batch(const sxsk_pc_job *jobs, const int4 *items, int nitems, int *ctr, cudaStream_t s)
{
	if (nitems <= 0) return 0;
	int grid = 0;
	cudaError_t e = persistent_grid(k_pose_cross_batch, 128, 0, nitems, ctr, &grid);
	if (e) return e;
	k_pose_cross_batch<<<grid, 128, 0, s>>>(jobs, items, nitems, ctr);
	return cudaGetLastError();
}

int sxsk_fit_grid(const double *cross, const sxsk_pose *order, int slot0, int nslot, int Q, const double *fc,
                  double a0sum, double peak, const double *gtab, const double *c1g, int n1, const double *c2g, int n2,
                  int max_blocks, double *chi, double *c1, double *c2, int32_t *cell, double *grid, cudaStream_t s)
{
	if (nslot <= 0) return 0;
	if (n1 <= 0 || n2 <= 0) return cudaErrorInvalidValue;
	int tp = n1 < FIT_THREADS ? n1 : FIT_THREADS;
	int ppb = FIT_THREADS / tp;
	size_t smem;
	for (;;) {
		size_t nthr = (size_t)ppb * tp;
		smem = sizeof(double) * ((size_t)ppb * 8 * Q + (size_t)FIT_NFC * Q + n2 + 2 * nthr + 3 * ppb) +
		       sizeof(int) * (((nthr + 1) & ~(size_t)1) + ppb);
		if (smem <= 227 * 1024 || ppb == 1) break;
		ppb = (ppb + 1) / 2;
	}
	if (smem > SXS_SMEM_MAX) return cudaErrorInvalidValue;
	cudaError_t e = smem_bound(k_fit_grid, smem, SXS_SMEM_MAX);
	if (e != cudaSuccess) return e;
	long ngroup = (nslot + ppb - 1) / ppb;
	int grid_n = (int)(ngroup < (long)max_blocks || max_blocks <= 0 ? ngroup : max_blocks);
	k_fit_grid<<<grid_n, FIT_THREADS, smem, s>>>(cross, order, slot0, nslot, Q, fc, a0sum, peak, gtab, c1g, n1, c2g,
	                                              n2, tp, ppb, chi, c1, c2, cell, grid);
	return cudaGetLastError();
}

} // extern "C"

namespace {
/* independent FMA chains per thread, register resident */
__global__ void k_fp64_probe(double *out, int iters)
{
	double a0 = threadIdx.x * 1e-9, a1 = a0 + 1e-9, a2 = a0 + 2e-9, a3 = a0 + 3e-9;
	double a4 = a0 + 4e-9, a5 = a0 + 5e-9, a6 = a0 + 6e-9, a7 = a0 + 7e-9;
	const double b = 0.999999999, c = 1e-12;
	for (int i = 0; i < iters; i++) {
		a0 = fma(a0, b, c); a1 = fma(a1, b, c); a2 = fma(a2, b, c); a3 = fma(a3, b, c);
		a4 = fma(a4, b, c); a5 = fma(a5, b, c); a6 = fma(a6, b, c); a7 = fma(a7, b, c);
	}
	double s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
	if (s == 12345.678) out[threadIdx.x] = s; /* keeps the chains live */
}
/* FP32 FMA chains: 8 independent per thread, enough threads to fill every
 * SM's FP32 pipes */
__global__ void k_fp32_probe(float *out, int iters)
{
	float a[8];
#pragma unroll
	for (int k = 0; k < 8; k++) a[k] = threadIdx.x * 1e-6f + k * 1e-6f;
	const float b = 0.9999999f, c = 1e-9f;
	for (int i = 0; i < iters; i++) {
#pragma unroll
		for (int k = 0; k < 8; k++) a[k] = fmaf(a[k], b, c);
	}
	float s = a[0] + a[1] + a[2] + a[3] + a[4] + a[5] + a[6] + a[7];
	if (s == 12345.678f) out[threadIdx.x] = s;
}
} // namespace

namespace {
/* every thread streams 16-byte L2-only loads over an L2-resident buffer */
__global__ void k_l2_probe(const float4 *__restrict__ buf, long n4, int passes, float *out)
{
	float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
	long stride = (long)gridDim.x * blockDim.x;
	for (int pass = 0; pass < passes; pass++)
		for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride) {
			float4 v = __ldcg(buf + i);
			acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
		}
	float s = acc.x + acc.y + acc.z + acc.w;
	if (s == 12345.678f) out[threadIdx.x] = s;
}
} // namespace

/* L2-to-SM read bandwidth (GB/s): a 32 MiB buffer, warm in L2, read 200
 * times by every SM with L2-only 16-byte loads */
extern "C" double sxsk_l2_probe(cudaStream_t s)
{
	int dev = 0, nsm = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
	const long n4 = (32L << 20) / 16;
	const int passes = 200;
	float4 *buf = NULL;
	float *out = NULL;
	if (cudaMalloc((void **)&buf, n4 * 16) != cudaSuccess) return -1.0;
	if (cudaMalloc((void **)&out, 1024 * sizeof(float)) != cudaSuccess) {
		cudaFree(buf);
		return -1.0;
	}
	cudaMemsetAsync(buf, 0, n4 * 16, s);
	int blocks = nsm * 8, threads = 256;
	k_l2_probe<<<blocks, threads, 0, s>>>(buf, n4, 2, out);
	cudaEvent_t e0, e1;
	cudaEventCreate(&e0);
	cudaEventCreate(&e1);
	cudaEventRecord(e0, s);
	k_l2_probe<<<blocks, threads, 0, s>>>(buf, n4, passes, out);
	cudaEventRecord(e1, s);
	cudaEventSynchronize(e1);
	float ms = 0;
	cudaEventElapsedTime(&ms, e0, e1);
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	cudaFree(buf);
	cudaFree(out);
	return ms > 0 ? (double)n4 * 16 * passes / (ms * 1e-3) / 1e9 : -1.0;
}

extern "C" double sxsk_fp32_probe(cudaStream_t s)
{
	int dev = 0, nsm = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
	float *out = NULL;
	if (cudaMalloc((void **)&out, 1024 * sizeof(float)) != cudaSuccess) return -1.0;
	int blocks = nsm * 8, threads = 256, iters = 65536;
	k_fp32_probe<<<blocks, threads, 0, s>>>(out, 64);
	cudaEvent_t e0, e1;
	cudaEventCreate(&e0);
	cudaEventCreate(&e1);
	cudaEventRecord(e0, s);
	k_fp32_probe<<<blocks, threads, 0, s>>>(out, iters);
	cudaEventRecord(e1, s);
	cudaEventSynchronize(e1);
	float ms = 0;
	cudaEventElapsedTime(&ms, e0, e1);
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	cudaFree(out);
	double flops = 2.0 * 8.0 * iters * (double)blocks * threads;
	return ms > 0 ? flops / (ms * 1e-3) / 1e12 : -1.0;
}

extern "C" double sxsk_fp64_probe(cudaStream_t s)
{
	int dev = 0, nsm = 0;
	cudaGetDevice(&dev);
	cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
	double *out = NULL;
	if (cudaMalloc((void **)&out, 1024 * sizeof(double)) != cudaSuccess) return -1.0;
	int blocks = nsm * 8, threads = 256, iters = 4096;
	k_fp64_probe<<<blocks, threads, 0, s>>>(out, 64);
	cudaEvent_t e0, e1;
	cudaEventCreate(&e0);
	cudaEventCreate(&e1);
	cudaEventRecord(e0, s);
	k_fp64_probe<<<blocks, threads, 0, s>>>(out, iters);
	cudaEventRecord(e1, s);
	cudaEventSynchronize(e1);
	float ms = 0;
	cudaEventElapsedTime(&ms, e0, e1);
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	cudaFree(out);
	double flops = 2.0 * 8.0 * iters * (double)blocks * threads;
	return ms > 0 ? flops / (ms * 1e-3) / 1e12 : -1.0;
}
