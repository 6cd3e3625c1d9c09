/*
 * Batched L-BFGS-B fit of (c1, c2) on the device, the solver of
 * lbfgsb_core.h (the reference's fit, src/min_saxs.c:153-259).
 * Compiled with -fmad=false so that every objective and solver step rounds
 * like the reference's C code.
 *
 * A block fits `slots` poses at a time.  The solver of a pose is one lane of
 * the first warp, stepped by reverse communication (lb_fit_advance); the
 * objective, ~130 FP64 operations per q and evaluation and nearly all of the
 * work, is evaluated by the whole block for the points that its solvers ask
 * for: threads take (pose, q) pairs for the model, its derivatives and the
 * terms of each sum, and one thread per sum adds a pose's terms in the
 * order of q, so that every sum has the reference's order and every result
 * the bits of a pose fitted by one thread.  A solver that ends hands its
 * slot to the next pose of the block's share.  (With one thread per pose,
 * 10,000 poses at Q = 51 took 41 ms: two warps per SM, each a serial chain
 * with 32 solvers' branches in turn; 1,000 poses took 38 ms, one chain's
 * latency.  Now 4.1 and 2.0 ms, the evaluations ~2.4 ms of FP64 pipe.)
 */
#include "kernels.h"
#include "smem.cuh"
#include "lbfgsb_core.h"

#include <type_traits>

namespace {

__device__ __forceinline__ double cross_at(const double *c, size_t i) { return c[i]; }
__device__ __forceinline__ double cross_at(const float2 *c, size_t i) { return (double)c[i].x + (double)c[i].y; }

#define LB_SLOTS 16      /* poses of a block at most (one lane of the first warp each) */
#define LB_ROWS 6        /* per q and slot: in, its two derivatives, three terms */

/* num / den for den with r = 1/den rounded to nearest, correctly rounded:
 * one Newton step makes the quotient faithful, the second one is Markstein's
 * final step (P. Markstein, IBM J. Res. Dev. 34 (1990)).  Outside the range
 * in which no step can over- or underflow it is divided. */
__device__ __forceinline__ double div_by(double num, double den, double r)
{
	double an = fabs(num);
	if (!(an > 0x1p-800 && an < 0x1p800 && fabs(den) > 0x1p-100 && fabs(den) < 0x1p100))
		return num == 0.0 ? num * r : num / den;
	double q = num * r;
	q = fma(fma(-q, den, num), r, q);
	return fma(fma(-q, den, num), r, q);
}

/* terms added in order from a row of shared memory */
__device__ __forceinline__ double row_sum(const double *w, int Q)
{
	double s = 0.0;
	int i = 0;
	for (; i + 4 <= Q; i += 4) {
		double a = w[i], b = w[i + 1], c = w[i + 2], d = w[i + 3];
		s = s + a;
		s = s + b;
		s = s + c;
		s = s + d;
	}
	for (; i < Q; i++) s = s + w[i];
	return s;
}

/* cross: raw cross terms [npose][6][Q], scaled to the peak (the rescale of
 * src/min_saxs.c:170-188) when rescale != 0. */
template <typename T, int LBT>
__global__ void __launch_bounds__(LBT, 512 / LBT)
k_lbfgsb(const T *__restrict__ cross, int npose, int Q, const double *__restrict__ q, const double *__restrict__ a,
         double mult, double peak, int rescale, int max_eval, int slots, double *__restrict__ chi,
         double *__restrict__ c1, double *__restrict__ c2, double *__restrict__ scale, int *__restrict__ nevals)
{
	extern __shared__ double lsm[];
	__shared__ double sx[LB_SLOTS][2], sk[LB_SLOTS], sg[LB_SLOTS][3], sscale[LB_SLOTS];
	__shared__ int spose[LB_SLOTS], l_any[LB_SLOTS], l_eval[LB_SLOTS];   /* poses; slots with work, with a full evaluation */
	__shared__ unsigned s_eval, s_any;
	const int Qp = Q | 1;                    /* odd row stride: the sums' threads on distinct banks */
	double *qs = lsm, *dq = qs + Q, *rd = dq + Q, *as = rd + Q, *slot = as + 6 * Q;
	int tid = threadIdx.x;
	for (int i = tid; i < Q; i += LBT) {
		double d = q[i] - (i > 0 ? q[i - 1] : -1.0);
		qs[i] = q[i];
		dq[i] = d;
		rd[i] = 1.0 / d;
	}
	for (int i = tid; i < 6 * Q; i += LBT) as[i] = a[i];
	lb_state st;
	int mode = 0, nev = 0;                   /* 0 idle, 1 evaluate, 2 best scale only */
	long pose = (long)blockIdx.x * slots + tid;
	auto begin = [&]() {
		mode = 0;
		if (tid >= slots || pose >= npose) return;
		const T *c = cross + (size_t)pose * 6 * Q;
		double s = 1.0;
		if (rescale) {
			s = cross_at(c, 0) + cross_at(c, 3 * (size_t)Q) + cross_at(c, 5 * (size_t)Q) + cross_at(c, 2 * (size_t)Q) -
			    cross_at(c, Q) - cross_at(c, 4 * (size_t)Q);
			s = peak / s;
		}
		sscale[tid] = s;
		spose[tid] = (int)pose;
		lb_fit_begin(&st);
		mode = 1;
		nev = 0;
	};
	/* warp 0: the points and slots of the next round */
	auto post = [&]() {
		if (mode) {
			sx[tid][0] = st.x[0];
			sx[tid][1] = st.x[1];
		}
		unsigned me = __ballot_sync(0xffffffffu, mode == 1), ma = __ballot_sync(0xffffffffu, mode != 0);
		unsigned below = (1u << tid) - 1u;
		if (mode != 0) l_any[__popc(ma & below)] = tid;
		if (mode == 1) l_eval[__popc(me & below)] = tid;
		if (tid == 0) {
			s_eval = me;
			s_any = ma;
		}
	};
	if (tid < 32) {
		begin();
		post();
	}
	for (;;) {
		__syncthreads();
		unsigned any = s_any, ev = s_eval;
		if (!any) break;
		int nany = __popc(any), nevl = __popc(ev);
		/* the model and its derivatives */
		for (int it = tid; it < nany * Q; it += LBT) {
			int k = it / Q, i = it - k * Q, p = l_any[k];
			double *X = slot + (size_t)p * LB_ROWS * Qp + i;
			double x1 = sx[p][0], x2 = sx[p][1], qc = qs[i], x[6];
			const T *cr = cross + (size_t)spose[p] * 6 * Q + i;
			for (int c = 0; c < 6; c++) {
				x[c] = cross_at(cr, (size_t)c * Q);
				if (rescale) x[c] *= sscale[p];
			}
			double corr = -mult * (x1 * x1 - 1.0);
			double G = x1 * x1 * x1 * exp(corr * qc * qc), Gd = lb_gder(G, x1, mult, qc);
			X[0] = lb_in(x, G, x2);
			X[Qp] = lb_idc1(x, G, Gd, x2);
			X[2 * Qp] = lb_idc2(x, G, x2);
			if (i == 0) sg[p][0] = lb_idc1_first(x, G, Gd, x2);
		}
		__syncthreads();
		for (int it = tid; it < nany * Q; it += LBT) {
			int k = it / Q, i = it - k * Q, p = l_any[k];
			double *X = slot + (size_t)p * LB_ROWS * Qp + i;
			double in = X[0], t[2];
			lb_scale_terms(in, div_by(in - X[-(i > 0)], dq[i], rd[i]), qs[i], as + 6 * i, t);
			X[3 * Qp] = t[0];
			X[4 * Qp] = t[1];
		}
		__syncthreads();
		{
			int p = tid < 2 * nany ? l_any[tid >> 1] : -1;
			double s = p >= 0 ? row_sum(slot + ((size_t)p * LB_ROWS + 3 + (tid & 1)) * Qp, Q) : 0.0;
			double o = __shfl_xor_sync(0xffffffffu, s, 1);
			if (p >= 0 && !(tid & 1)) sk[p] = s / o;
		}
		__syncthreads();
		for (int it = tid; it < nevl * Q; it += LBT) {
			int k = it / Q, i = it - k * Q, p = l_eval[k];
			double *X = slot + (size_t)p * LB_ROWS * Qp + i;
			int b = i > 0;                       /* the previous q's entry; the first q has its own start */
			double in = X[0], i1 = X[Qp], i2 = X[2 * Qp], h = rd[i], t[3];
			double i1p = b ? X[Qp - 1] : sg[p][0];
			lb_grad_terms(sk[p], qs[i], as + 6 * i, in, (in - X[-b]) * h, i1, (i1 - i1p) * h, i2,
			              (i2 - X[2 * Qp - b]) * h, t);
			X[3 * Qp] = t[0];
			X[4 * Qp] = t[1];
			X[5 * Qp] = t[2];
		}
		__syncthreads();
		for (int k = tid; k < 3 * nevl; k += LBT) {
			int p = l_eval[k / 3], c = k % 3;
			sg[p][c] = row_sum(slot + ((size_t)p * LB_ROWS + 3 + c) * Qp, Q);
		}
		__syncthreads();
		if (tid < 32) {
			bool done = mode == 2;
			if (mode == 1) {
				st.g[0] = sg[tid][0];
				st.g[1] = sg[tid][1];
				st.f = sg[tid][2];
				nev++;
				if (!lb_fit_advance(&st, nev == 1, nev, max_eval)) {
					/* the scale of the result: known when the last point
					 * evaluated is the result, else one more sum */
					if (st.x[0] == sx[tid][0] && st.x[1] == sx[tid][1]) done = true;
					else mode = 2;
				}
			}
			if (done) {
				chi[pose] = sqrt(st.f);
				c1[pose] = st.x[0];
				c2[pose] = st.x[1];
				if (scale) scale[pose] = sk[tid];
				if (nevals) nevals[pose] = nev;
				pose += (long)gridDim.x * slots;
				begin();
			}
			__syncwarp();
			post();
		}
	}
}

/* one thread per pose on scaled terms, for q grids whose slots do not fit in
 * shared memory (above 1,900 points) */
__global__ void k_lbfgsb_thread(const double *__restrict__ cross, int npose, int Q, const double *__restrict__ q,
                                const double *__restrict__ a, double mult, int max_eval, double *__restrict__ chi,
                                double *__restrict__ c1, double *__restrict__ c2, double *__restrict__ scale,
                                int *__restrict__ nevals)
{
	int p = blockIdx.x * blockDim.x + threadIdx.x;
	if (p >= npose) return;
	lb_saxs o;
	o.cr = cross + (size_t)p * 6 * Q;
	o.stride = 1;
	o.q = q;
	o.a = a;
	o.mult = mult;
	o.Q = Q;
	double x, y, z, w;
	int ne = lb_saxs_fit(&o, &x, &y, &z, &w, max_eval);
	chi[p] = x;
	c1[p] = y;
	c2[p] = z;
	if (scale) scale[p] = w;
	if (nevals) nevals[p] = ne;
}

#define LB_MAX_EVAL 100000
#define LB_SMEM_MAX (225 * 1024)   /* dynamic; the slots' points and sums have 1.1 KB beside it */

template <typename T, int LBT>
int lbfgsb_launch(const T *cross, int npose, int Q, const double *q, const double *a, double mult, double peak,
                  int rescale, double *chi, double *c1, double *c2, double *scale, int *nevals, int nsm, int slots,
                  size_t smem, cudaStream_t s)
{
	int per = 0;
	auto kern = k_lbfgsb<T, LBT>;
	cudaError_t e = smem_bound(kern, smem, LB_SMEM_MAX);
	if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, LBT, smem);
	if (e) return (int)e;
	if (per < 1) return (int)cudaErrorInvalidConfiguration;
	long want = ((long)npose + slots - 1) / slots, most = (long)nsm * per;
	kern<<<(unsigned)(want < most ? want : most), LBT, smem, s>>>(cross, npose, Q, q, a, mult, peak, rescale, LB_MAX_EVAL,
	                                                              slots, chi, c1, c2, scale, nevals);
	return (int)cudaGetLastError();
}

/* Block shape.  A round is the solver steps of a block's poses (one warp,
 * latency: divisions and square roots; ~110,000 cycles for one pose, 280,000
 * for eight) and their evaluations (the FP64 pipe); more poses per block
 * share the step, more blocks per SM overlap it with other blocks'
 * evaluations.  Measured (fit stage, ms; 10,000 poses at Q = 51 / 20,000 at
 * 101 / 20,000 at 201; one thread per pose took 41.1 for the first): 64
 * threads, 8 poses 7.0 / 25.6 / 43.9, 16 poses 4.1 / 25.4 / 63.7; 128
 * threads, 8 poses 8.3 / 23.6 / 39.9, 16 poses 6.0 / 23.3 / 47.1.  So 16
 * poses while they leave room for two blocks per SM, and 64 threads while
 * four blocks fit; short lists take fewer poses per block, down to one
 * (1,000 poses: 2.0 ms with 1, 3.6 with 16), to spread over the SMs. */
template <typename T>
int lbfgsb_any(const T *cross, int npose, int Q, const double *q, const double *a, double mult, double peak,
               int rescale, double *chi, double *c1, double *c2, double *scale, int *nevals, cudaStream_t s)
{
	int dev = 0, nsm = 0;
	cudaError_t e = cudaGetDevice(&dev);
	if (!e) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
	if (e) return (int)e;
	int slots = LB_SLOTS;
	while (slots > 1 && (long)slots * nsm * 4 > npose) slots >>= 1;
	size_t smem;
	for (;; slots >>= 1) {
		smem = sizeof(double) * (9 * (size_t)Q + (size_t)slots * LB_ROWS * (Q | 1));
		if (smem <= 110 * 1024 || slots == 1) break;
	}
	if (smem > LB_SMEM_MAX) {
		if (rescale || !std::is_same<T, double>::value)
			return (int)cudaErrorInvalidValue;   /* plans have at most 1,024 q */
		k_lbfgsb_thread<<<(npose + 63) / 64, 64, 0, s>>>((const double *)cross, npose, Q, q, a, mult, LB_MAX_EVAL, chi, c1,
		                                                 c2, scale, nevals);
		return (int)cudaGetLastError();
	}
	if (smem <= 56 * 1024)
		return lbfgsb_launch<T, 64>(cross, npose, Q, q, a, mult, peak, rescale, chi, c1, c2, scale, nevals, nsm, slots, smem,
		                            s);
	return lbfgsb_launch<T, 128>(cross, npose, Q, q, a, mult, peak, rescale, chi, c1, c2, scale, nevals, nsm, slots, smem,
	                             s);
}

} // namespace

/* cross: [npose][6][Q] (raw when rescale != 0, already rescaled otherwise),
 * double, or double-float pairs when cross_df */
extern "C" int sxs_fit_lbfgsb_launch(const void *cross, int cross_df, int npose, int Q, const double *q,
                                     const double *a, double mult, double peak, int rescale, double *chi, double *c1,
                                     double *c2, double *scale, int *nevals, cudaStream_t s)
{
	if (npose <= 0) return 0;
	if (cross_df)
		return lbfgsb_any((const float2 *)cross, npose, Q, q, a, mult, peak, rescale, chi, c1, c2, scale, nevals, s);
	return lbfgsb_any((const double *)cross, npose, Q, q, a, mult, peak, rescale, chi, c1, c2, scale, nevals, s);
}
