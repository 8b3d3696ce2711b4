/* The functions for arguments of a known range against the general ones, bit
 * for bit, and those against the series they are defined by, over a sweep of
 * [0, 1] (and the quarter circle) with every float near the places where a
 * branch changes.  Prints the number of differences. */
#include <initializer_list>
#include <stdio.h>

#include "kgr_math.h"

using namespace kgr;

static void sincos_by_case(float x, float &s, float &c)
{
	int q;
	float r = reduce_pio2(x, q);
	float sr = sin_kernel(r), cr = cos_kernel(r);
	switch (q) {
	case 0: s = sr; c = cr; break;
	case 1: s = cr; c = -sr; break;
	case 2: s = -sr; c = -cr; break;
	default: s = -cr; c = sr; break;
	}
}

static float atan_by_case(float x)
{
	bool neg = x < 0.0f;
	float a = neg ? -x : x;
	bool inv = a > 1.0f;
	if (inv)
		a = 1.0f / a;
	float r;
	if (a > KGR_TAN_PI12_F)
		r = KGR_PIO6_F + atan_kernel((a * KGR_SQRT3_F - 1.0f) / (a + KGR_SQRT3_F));
	else
		r = atan_kernel(a);
	if (inv)
		r = KGR_PIO2_F - r;
	return neg ? -r : r;
}

static long bad = 0;

static void same(float a, float b) { bad += f2u(a) != f2u(b); }

static void check(float x)
{
	float s0, c0, s1, c1;
	float theta = 2.0f * atan_by_case(ksqrt((1.0f - x) / (1.0f + x)));
	same(kacos_unit(x), theta);
	same(kacos(x), theta);
	sincos_by_case(theta, s0, c0);
	ksincos_quarter(theta, s1, c1);
	same(s0, s1);
	same(c0, c1);
	float q = x * KGR_PIO2_F;
	sincos_by_case(q, s0, c0);
	ksincos_quarter(q, s1, c1);
	same(s0, s1);
	same(c0, c1);
	for (float y : {x, -x, 7.0f * x, -40.0f * x, 1.0f / (x + 1e-30f)}) {
		if (y < 1000.0f) {
			sincos_by_case(y, s0, c0);
			ksincos(y, s1, c1);
			same(s0, s1);
			same(c0, c1);
		}
		same(katan(y), atan_by_case(y));
	}
	f3 seed = mk(x, 1.0f - x, 0.5f * x), at = seed;
	f3 r = pcg3f(at);
	same(fract(r.x), r.x);
	same(fract(r.y), r.y);
	same(fract(r.z), r.z);
}

int main()
{
	const uint32_t one = 0x3f800000u;
	for (uint32_t u = 0; u < one; u += 251u)
		check(u2f(u));
	for (float at : {1.0f, 0.999f, KGR_TAN_PI12_F, 0.5f, 0.70710678f, 0.86602540f, 0.0f})
		for (int32_t o = -5000; o <= 5000; o++) {
			int64_t u = (int64_t)f2u(at) + o;
			if (u >= 0 && u <= (int64_t)one)
				check(u2f((uint32_t)u));
		}
	printf("%ld\n", bad);
	return 0;
}
