// Exact arithmetic shared by the CUDA kernels and their host-side checks.
//
// Everything here is plain binary32 / int64 arithmetic in a fixed order, so the
// same source compiled by nvcc for sm_103a (with -fmad=false) and by a host C++
// compiler (with -ffp-contract=off) gives identical bits.  These are the
// operations the reference renderer performs one pixel at a time; the GPU needs
// them in a form that any thread can evaluate for any pixel independently.
#ifndef DSRG_EXACT_H
#define DSRG_EXACT_H

#include <math.h>
#include <stdint.h>

#if defined(__CUDACC__)
#define DSRG_HD __host__ __device__ __forceinline__
// Large helpers stay out of line on the device so that the kernels fit the instruction cache.
#define DSRG_HD_CALL static __host__ __device__ __noinline__
#else
#define DSRG_HD inline
#define DSRG_HD_CALL inline
#endif

namespace dsrg {

DSRG_HD float fadd(float a, float b) {
#if defined(__CUDA_ARCH__)
	return __fadd_rn(a, b);
#else
	return a + b;
#endif
}
DSRG_HD float fsub(float a, float b) {
#if defined(__CUDA_ARCH__)
	return __fsub_rn(a, b);
#else
	return a - b;
#endif
}
DSRG_HD float fmul(float a, float b) {
#if defined(__CUDA_ARCH__)
	return __fmul_rn(a, b);
#else
	return a * b;
#endif
}
DSRG_HD float fdiv(float a, float b) {
#if defined(__CUDA_ARCH__)
	return __fdiv_rn(a, b);
#else
	return a / b;
#endif
}
// 1 / x correctly rounded: the same value as fdiv(1.0f, x) for every x (IEEE 754 defines both as
// the rounded exact quotient), in fewer instructions on the device.
DSRG_HD float frcp(float x) {
#if defined(__CUDA_ARCH__)
	return __frcp_rn(x);
#else
	return 1.0f / x;
#endif
}
// An estimate of a / b, within 2 ulp on the device for 2^-126 <= |b| <= 2^126, which every nonzero int64
// satisfies and chain_add sees to; beyond it is 0, below (subnormal divisors) it can be infinite.  Integer
// quotients are corrected by exact products afterwards, chain_add leaves room for the error.  A host
// build may define DSRG_HOST_ESTIMATE_ERROR to push its estimates that far off, and out of that range as
// far as they can be, so that host checks exercise what the device does.
DSRG_HD float fdiv_estimate(float a, float b) {
#if defined(__CUDA_ARCH__)
	return __fdividef(a, b);
#elif defined(DSRG_HOST_ESTIMATE_ERROR)
	const float size = b < 0.0f ? -b : b;
	if (a != 0.0f && size < 1.17549435e-38f) return ((a < 0.0f) == (b < 0.0f) ? 1.0f : -1.0f) / 0.0f;
	if (size > 8.50705917e37f) return 0.0f;
	const float q = a / b;
	return q + q * DSRG_HOST_ESTIMATE_ERROR;
#else
	return a / b;
#endif
}
DSRG_HD uint32_t fbits(float f) {
#if defined(__CUDA_ARCH__)
	return __float_as_uint(f);
#else
	union { float f; uint32_t u; } v; v.f = f; return v.u;
#endif
}
DSRG_HD float bitsf(uint32_t u) {
#if defined(__CUDA_ARCH__)
	return __uint_as_float(u);
#else
	union { float f; uint32_t u; } v; v.u = u; return v.f;
#endif
}
DSRG_HD float i64_to_float(int64_t v) {
#if defined(__CUDA_ARCH__)
	return __ll2float_rn(v);
#else
	return (float)v;
#endif
}

// Result of adding d to s, n times in a row, each sum rounded to binary32 nearest-even:
//   for (i = 0; i < n; i++) s = s + d;
// The reference accumulates its depth and vertex weights this way along each
// row pair (implementation/render/shader/fillerTemplates.h:196-244, 339-372).
// Evaluated in O(binades visited) instead of O(n).  Inside one binade [lo, hi) of |s| the
// representable values are the multiples of one ulp U and s + d always has the same remainder
// modulo U, so every step whose exact sum stays in the binade rounds to the same increment; only
// a tie (remainder U / 2) depends on the parity of s / U, and after one such step s / U is even and
// stays even.  So two plain steps inside one binade settle the parity and show the increment
// (their difference, exact in binary32), and the steps that surely stay in the binade are taken at
// once: k times the increment, and the sum with it, are multiples of U below 2^24 U, hence exact.
// Everything is binary32 arithmetic.  An earlier form that worked out the increment and the step
// count in 64-bit integers cost about five times as many instructions per binade, and the running
// sums of long rows were most of the tile pass and of the point lights.
// On a GB300 the change took a frame of 20,000 random triangles at 800x600 from 478 to 402 us, the
// 1080p deferred-light frame from 921 to 752 us and a batch of 32 mixed frames from 13.4 to 12.2 ms.
DSRG_HD_CALL float chain_add(float s, float d, int32_t n) {
	while (n > 0) {
		if (n <= 4) {
			// short chains (small triangles, quads near a row's start, the end of a long one)
			for (; n > 0; n--) s = fadd(s, d);
			return s;
		}
		const float s1 = fadd(s, d), s2 = fadd(s1, d);
		n -= 2;
		const uint32_t b0 = fbits(s), b1 = fbits(s1), b2 = fbits(s2);
		s = s2;
		if (b1 == b2) return s; // a fixed point: d is too small to move s, or an infinity
		if ((((b0 ^ b1) | (b1 ^ b2)) & 0xFF800000u) != 0u) continue; // another binade or sign: only the plain steps
		const uint32_t exponent = b2 & 0x7F800000u;
		// plain steps near overflow, for NaN, and below 2^-103, where the ulp and so the increment can be
		// subnormal, a divisor that the estimate below does not take
		if (exponent - 0x0C000000u >= 0x7F000000u - 0x0C000000u) {
			if (exponent == 0x7F800000u) return s;
			continue;
		}
		const float inc = fsub(s2, s1);
		const float lo = bitsf(exponent), a = bitsf(b2 & 0x7FFFFFFFu), step = bitsf(fbits(inc) & 0x7FFFFFFFu);
		const bool up = ((fbits(inc) ^ b2) >> 31) == 0u;
		// Steps left in the binade: the value after k of them keeps one increment's distance from its
		// end when k <= room / step - 1.  The estimate is 2 ulp off: less than 4 for a quotient below 2^23,
		// less than 1/8 below 2^18.
		const float room = up ? fsub(fadd(lo, lo), a) : fsub(a, lo);
		const float steps = fdiv_estimate(room, step);
		int32_t k = (int32_t)steps - (steps < 262144.0f ? 2 : 5);
		k = k < n ? k : n;
		if (k > 0) {
			s = fadd(s2, fmul((float)k, inc));
			n -= k;
		}
	}
	return s;
}

// min(max(L, (int32_t)(a / b + 1)), R) with C's truncating int64 division, as the
// reference's cutConvexEdge computes each row's bound (implementation/render/ITriangle2D.cpp:122,130).
// A binary32 estimate of the quotient settles the clamp when it is far outside
// [L, R]; near the clamp range an exact int64 remainder check corrects it; only
// quotients beyond +-2^30 (where the int32 cast may wrap) take the 64-bit division.
// Requires b != 0 and -2^20 < L <= R < 2^20.
DSRG_HD int32_t clamp_quotient_plus_one(int64_t a, int64_t b, int32_t L, int32_t R) {
	float qf = fdiv_estimate(i64_to_float(a), i64_to_float(b));
	int32_t v;
	if (qf > -1.0e9f && qf < 1.0e9f) {
		if (qf < -2097152.0f) return L;
		if (qf > 2097152.0f) return R;
		int64_t q = (int64_t)qf;
		// make the divisor positive; truncating and floor quotients are unchanged by negating both
		int64_t aa = a, bb = b;
		if (bb < 0) { aa = -aa; bb = -bb; }
		// floor quotient: q * bb <= aa < (q + 1) * bb
		while (q * bb > aa) q--;
		while ((q + 1) * bb <= aa) q++;
		if (aa < 0 && q * bb != aa) q++; // truncation toward zero
		v = (int32_t)(q + 1);
	} else {
		v = (int32_t)(a / b + 1);
	}
	return v < L ? L : (v > R ? R : v);
}

// One triangle edge in sub-pixel units, from cutConvexEdge (implementation/render/ITriangle2D.cpp:86-148).
struct Edge {
	int64_t sx, sy;      // start corner
	int64_t nx, ny;      // normal: (end.y - start.y, start.x - end.x)
	int64_t threshold;   // -1 or 0 by edge direction
};

DSRG_HD Edge make_edge(int64_t sx, int64_t sy, int64_t ex, int64_t ey) {
	Edge e;
	e.sx = sx; e.sy = sy;
	e.nx = ey - sy;
	e.ny = sx - ex;
	e.threshold = (sx > ex || (sx == ex && sy > ey)) ? -1 : 0;
	return e;
}

// Applies one edge to the interval of pixel row y, clamped to [L, R).
// The per-row limit of cutConvexEdge, limit(y) = threshold - (128 - sx)*nx - (128 + 256*y - sy)*ny,
// does not depend on the clip rectangle's corner, so any row can be cut on its own.
DSRG_HD void cut_row(const Edge &e, int32_t y, int32_t L, int32_t R, int32_t &left, int32_t &right) {
	if (e.nx != 0) {
		int64_t limit = e.threshold - (128 - e.sx) * e.nx - (128 + 256 * (int64_t)y - e.sy) * e.ny;
		int64_t offsetX = e.nx * 256;
		if (e.nx < 0) {
			int32_t side = clamp_quotient_plus_one(limit + 1, offsetX, L, R);
			if (side > left) left = side;
		} else {
			int32_t side = clamp_quotient_plus_one(limit, offsetX, L, R);
			if (side < right) right = side;
		}
	} else if (e.ny != 0) {
		int64_t value = (128 + 256 * (int64_t)y - e.sy) * e.ny;
		if (value > e.threshold) { left = R; right = L; }
	}
}

// cut_row for consecutive rows by exact integer stepping.  For a cutting edge the numerator of
// the quotient changes by the same amount every row, so the floor quotient and its remainder
// advance by a fixed quotient and remainder with at most one carry; truncation toward zero and
// the int32 wrap of (a / b + 1) then give exactly clamp_quotient_plus_one's value.  Two int64
// divisions per edge replace one division per edge and row.
struct EdgeStepper {
	int32_t kind;        // 0: cuts the left end, 1: cuts the right end, 2: empties rows (horizontal), 3: none
	int64_t q, r, B;     // floor(A / B) and A - q * B, B > 0 (A: the numerator with the divisor's sign folded in)
	int64_t qd, rd;      // the same for the change of A per row
	// horizontal edges reuse q as (128 + 256 y - sy) * ny, qd as its change per row and B as the threshold
};

// floor(a / b) and its remainder, b > 0.  Quotients below 2^22 in magnitude (every row crossing
// inside an image) come from a binary32 estimate: a and b round by at most 2^-24 relative and the
// estimated quotient by 2 ulp, so the estimate lies within 2 of a / b, and exact 64-bit products
// step its floor to the answer.  Larger quotients take the 64-bit division.
DSRG_HD void floor_divide(int64_t a, int64_t b, int64_t &q, int64_t &r) {
	const float qf = fdiv_estimate(i64_to_float(a), i64_to_float(b));
	if (qf > -4194304.0f && qf < 4194304.0f) {
		q = (int64_t)floorf(qf);
		r = a - q * b;
		while (r < 0) { q -= 1; r += b; }
		while (r >= b) { q += 1; r -= b; }
		return;
	}
	q = a / b;
	if (a % b != 0 && a < 0) q -= 1;
	r = a - q * b;
}

DSRG_HD EdgeStepper edge_stepper(const Edge &e, int32_t y0) {
	EdgeStepper s;
	s.q = s.r = s.B = s.qd = s.rd = 0;
	if (e.nx != 0) {
		int64_t a = e.threshold - (128 - e.sx) * e.nx - (128 + 256 * (int64_t)y0 - e.sy) * e.ny;
		if (e.nx < 0) a += 1;
		const int64_t b = e.nx * 256, delta = -256 * e.ny;
		const int64_t sign = b > 0 ? 1 : -1;
		s.kind = e.nx < 0 ? 0 : 1;
		s.B = b * sign;
		floor_divide(a * sign, s.B, s.q, s.r);
		floor_divide(delta * sign, s.B, s.qd, s.rd);
	} else if (e.ny != 0) {
		s.kind = 2;
		s.q = (128 + 256 * (int64_t)y0 - e.sy) * e.ny;
		s.qd = 256 * e.ny;
		s.B = e.threshold;
	} else {
		s.kind = 3;
	}
	return s;
}

// Applies the edge to the current row's interval, then moves it to the next row.
DSRG_HD void edge_step(EdgeStepper &s, int32_t L, int32_t R, int32_t &left, int32_t &right) {
	if (s.kind <= 1) {
		const int64_t t = s.q + ((s.q < 0 && s.r != 0) ? 1 : 0); // the quotient truncated toward zero
		int32_t v = (int32_t)(uint32_t)(uint64_t)(t + 1);
		v = v < L ? L : (v > R ? R : v);
		if (s.kind == 0) { if (v > left) left = v; } else { if (v < right) right = v; }
		s.q += s.qd;
		s.r += s.rd;
		if (s.r >= s.B) { s.r -= s.B; s.q += 1; }
	} else if (s.kind == 2) {
		if (s.q > s.B) { left = R; right = L; }
		s.q += s.qd;
	}
}

// The steppers in 32-bit arithmetic, for triangles whose corners lie within NEAR_UNITS sub-pixel units
// (64 pixels) of the pixel corner (left, top) they are taken relative to, and rows within
// NEAR_ROWS of it: every product is then below 2^30.  Taking `left` whole pixels off the corners takes
// exactly `left` off the floor quotient and leaves its remainder, so the quotient of the caller's
// coordinates, which decides the truncation toward zero, is q + left.
static const int32_t NEAR_UNITS = 16384, NEAR_ROWS = 16;

DSRG_HD bool near_corners(const int32_t *flat, int32_t left, int32_t top) {
	for (int i = 0; i < 3; i++) {
		const int64_t x = (int64_t)flat[2 * i] - 256 * (int64_t)left, y = (int64_t)flat[2 * i + 1] - 256 * (int64_t)top;
		if (x < -NEAR_UNITS || x > NEAR_UNITS || y < -NEAR_UNITS || y > NEAR_UNITS) return false;
	}
	return true;
}

struct NearEdge {
	int32_t kind;      // as EdgeStepper
	int32_t q, r, B;
	int32_t qd, rd;
};

DSRG_HD void floor_divide_near(int32_t a, int32_t b, int32_t &q, int32_t &r) {
	q = (int32_t)floorf(fdiv_estimate((float)a, (float)b)); // within 4 of a / b, and b >= 256
	r = a - q * b;
	while (r < 0) { q -= 1; r += b; }
	while (r >= b) { q += 1; r -= b; }
}

// The edge from (sx, sy) to (ex, ey), relative to the pixel corner, at row 0.
DSRG_HD NearEdge near_edge(int32_t sx, int32_t sy, int32_t ex, int32_t ey) {
	NearEdge e;
	e.q = e.r = e.B = e.qd = e.rd = 0;
	const int32_t nx = ey - sy, ny = sx - ex, threshold = (sx > ex || (sx == ex && sy > ey)) ? -1 : 0;
	if (nx != 0) {
		int32_t a = threshold - (128 - sx) * nx - (128 - sy) * ny;
		if (nx < 0) a += 1;
		e.kind = nx < 0 ? 0 : 1;
		e.B = 256 * (nx < 0 ? -nx : nx);
		floor_divide_near(nx < 0 ? -a : a, e.B, e.q, e.r);
		floor_divide_near(nx < 0 ? 256 * ny : -256 * ny, e.B, e.qd, e.rd);
	} else if (ny != 0) {
		e.kind = 2;
		e.q = (128 - sy) * ny;
		e.qd = 256 * ny;
		e.B = threshold;
	} else {
		e.kind = 3;
	}
	return e;
}

// edge_step, `offset` being the pixels the corners were moved by; L and R as there.
DSRG_HD void near_step(NearEdge &e, int32_t offset, int32_t L, int32_t R, int32_t &left, int32_t &right) {
	if (e.kind <= 1) {
		const int32_t t = e.q + offset;
		int32_t v = t + ((t < 0 && e.r != 0) ? 2 : 1); // the quotient truncated toward zero, plus one
		v = v < L ? L : (v > R ? R : v);
		if (e.kind == 0) { if (v > left) left = v; } else { if (v < right) right = v; }
		e.q += e.qd;
		e.r += e.rd;
		if (e.r >= e.B) { e.r -= e.B; e.q += 1; }
	} else if (e.kind == 2) {
		if (e.q > e.B) { left = R; right = L; }
		e.q += e.qd;
	}
}

// Row intervals of rows [y0, y0 + rows) of a triangle, stepped (equal to row_interval of each row).
DSRG_HD void row_intervals_stepped(const int32_t *flat, int32_t y0, int32_t rows, int32_t L, int32_t R, int32_t *lefts, int32_t *rights) {
	const bool degenerate = (flat[0] == flat[2] && flat[1] == flat[3]) || (flat[2] == flat[4] && flat[3] == flat[5]) ||
	                        (flat[4] == flat[0] && flat[5] == flat[1]);
	if (degenerate) {
		for (int32_t k = 0; k < rows; k++) { lefts[k] = R; rights[k] = L; }
		return;
	}
	EdgeStepper s0 = edge_stepper(make_edge(flat[0], flat[1], flat[2], flat[3]), y0);
	EdgeStepper s1 = edge_stepper(make_edge(flat[2], flat[3], flat[4], flat[5]), y0);
	EdgeStepper s2 = edge_stepper(make_edge(flat[4], flat[5], flat[0], flat[1]), y0);
	for (int32_t k = 0; k < rows; k++) {
		int32_t left = L, right = R;
		edge_step(s0, L, R, left, right);
		edge_step(s1, L, R, left, right);
		edge_step(s2, L, R, left, right);
		lefts[k] = left;
		rights[k] = right;
	}
}

// Row interval [left, right) of pixel row y for a triangle with sub-pixel corners,
// clamped to [L, R): rasterizeTriangle (implementation/render/ITriangle2D.cpp:150-169).
DSRG_HD_CALL void row_interval(const int32_t *flat, int32_t y, int32_t L, int32_t R, int32_t &left, int32_t &right) {
	const bool degenerate = (flat[0] == flat[2] && flat[1] == flat[3]) || (flat[2] == flat[4] && flat[3] == flat[5]) ||
	                        (flat[4] == flat[0] && flat[5] == flat[1]);
	if (degenerate) { left = R; right = L; return; }
	left = L; right = R;
	for (int i = 0; i < 3; i++) {
		int j = (i + 1) % 3;
		Edge e = make_edge(flat[i * 2], flat[i * 2 + 1], flat[j * 2], flat[j * 2 + 1]);
		cut_row(e, y, L, R, left, right);
	}
}

} // namespace dsrg

#endif
