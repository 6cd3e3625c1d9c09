/* Two-limb fixed point (kernels_fixed.cu): v / 2^e = (h 2^29 + l) 2^-57. */
#ifndef SXS_LIMBS_CUH
#define SXS_LIMBS_CUH

/* the limbs {h, l} of v / 2^e, c28 = 2^(28 - e), |v| <= 2^(e + 1): a sum with
 * 1.5 2^52 leaves the rounded integer in the low word, and the remainder is
 * exact */
__device__ __forceinline__ int2 sxs_limbs(double v, double c28)
{
	const double M = 6755399441055744.0;
	double t = __fma_rn(v, c28, M);
	double r = __fma_rn(v, c28, -__dsub_rn(t, M));
	double u = __fma_rn(r, 536870912.0, M);
	return make_int2(__double2loint(t), __double2loint(u));
}

#endif
