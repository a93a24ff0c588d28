// Row arithmetic of the per-row sites for four neighbouring elements per thread ("quads").
//
// A row site is a chain of short dependent phases, so what counts on a decode batch is the number
// of dependent instructions between two block-wide reductions, and on a prefill chunk the number of
// instructions per element. The forms below are the ones sslm_int.cuh defines, with everything that
// depends only on the row hoisted into a few words and the per-element step on 32-bit (or float)
// instructions. Each is exact: a form that covers only part of the operand range says so in a
// row-uniform flag, and a float is used only to FIND an integer that is then known to be the right
// one (or is recomputed with the integer form when it is too close to a rounding tie to know).
#pragma once
#include <cuda_runtime.h>

#include "sslm_types.cuh"

namespace sslm {

// ------------------------------------------------------------- block reductions
// One barrier each: warps reduce with one instruction, post their word, and after the barrier every
// warp reduces the posted words with one more. `bank` alternates between two sets of 32 words, so a
// set is rewritten only after a barrier that all its readers have passed.
struct Bank {
	uint32_t* w;      // 2 x 32 words of shared memory
	int phase;
};
__device__ __forceinline__ uint32_t block_max_u32(uint32_t v, Bank& b) {
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
	uint32_t* w = b.w + b.phase * 32;
	b.phase ^= 1;
	v = __reduce_max_sync(0xffffffffu, v);
	if (lane == 0) w[warp] = v;
	__syncthreads();
	return __reduce_max_sync(0xffffffffu, lane < nw ? w[lane] : 0u);
}
__device__ __forceinline__ uint32_t block_sum_u32(uint32_t v, Bank& b) {
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
	uint32_t* w = b.w + b.phase * 32;
	b.phase ^= 1;
	v = __reduce_add_sync(0xffffffffu, v);
	if (lane == 0) w[warp] = v;
	__syncthreads();
	return __reduce_add_sync(0xffffffffu, lane < nw ? w[lane] : 0u);
}

__device__ __forceinline__ uint32_t abs_u32(int32_t v) { return v < 0 ? 0u - (uint32_t)v : (uint32_t)v; }
__device__ __forceinline__ uint32_t pack4(int a, int b, int c, int d) {
	return __byte_perm(__byte_perm((uint32_t)a, (uint32_t)b, 0x0040u), __byte_perm((uint32_t)c, (uint32_t)d, 0x0040u), 0x5410u);
}
__device__ __forceinline__ int byte_of(uint32_t w, int j) { return (int)(int8_t)(w >> (8 * j)); }

// ------------------------------------------------------------------ requant codes
// code = round_half_away(x * 127 R / 2^E), |x| <= the row's maximum (so |code| <= 127), E = 62 - s.
// v = x * f with f = 127 R / 2^E in float: the three roundings (x, f, the product) put v within
// 127 * 2^-22 < 3.1e-5 of the exact quotient, so unless v is within 1e-4 of a half-integer its
// nearest integer IS the code; one element in 5,000 is not and is recomputed with requant_code.
// Five instructions per element instead of about twenty.
struct QuadCoder {
	float f;
	int64_t r;
	int s;
};
__device__ __forceinline__ QuadCoder make_quad_coder(int64_t r, int s) {
	QuadCoder c;
	c.r = r;
	c.s = s;
	const int e = 62 - s;      // 32..63
	c.f = __ull2float_rn((unsigned long long)r) * 127.0f * __int_as_float((127 - e) << 23);
	return c;
}
constexpr float kRoundMagic = 12582912.0f;      // 1.5 * 2^23: adding it leaves the nearest integer in the low bits
constexpr float kNearTie = 0.4999f;
__device__ __forceinline__ float to_float(int32_t x) { return __int2float_rn(x); }
__device__ __forceinline__ float to_float(int64_t x) { return __ll2float_rn(x); }
template <typename T>
static __device__ __noinline__ uint32_t code_quad_exact(T x0, T x1, T x2, T x3, int64_t r, int s) {
	return pack4(requant_code((int64_t)x0, r, s), requant_code((int64_t)x1, r, s), requant_code((int64_t)x2, r, s),
	             requant_code((int64_t)x3, r, s));
}
// four codes, packed; element j in byte j
template <typename T>
__device__ __forceinline__ uint32_t code_quad(const T (&x)[4], const QuadCoder& c) {
	int t[4];
	float far = 0.0f;
#pragma unroll
	for (int j = 0; j < 4; ++j) {
		const float xf = to_float(x[j]);
		const float m = fmaf(xf, c.f, kRoundMagic);
		t[j] = __float_as_int(m);
		far = fmaxf(far, fabsf(fmaf(xf, c.f, kRoundMagic - m)));
	}
	if (far > kNearTie) return code_quad_exact<T>(x[0], x[1], x[2], x[3], c.r, c.s);
	return pack4(t[0], t[1], t[2], t[3]);
}

// ------------------------------------------------------------------- K/V landing, residual
// LandingRescale with the row's (m_a, r_t, exponent) product hoisted: round_half_away(|code| P / 2^k)
// with P = |m_a| r_t < 2^63, by the 64-bit-word identity landing_rescale states. `fast` when the
// scales are in the range that identity covers.
struct Lander {
	uint32_t hi, lo;
	uint64_t half;      // 2^(k-33)
	int sh;             // k - 32, 1..62
	bool neg, fast;
};
__device__ __forceinline__ Lander make_lander(int64_t m_a, int64_t r_t, int64_t e_a, int64_t e_t) {
	Lander l;
	int64_t k = sat_sub64(62, sat_sub64(e_a, e_t));
	const uint64_t am = m_a < 0 ? (~(uint64_t)m_a + 1u) : (uint64_t)m_a;
	l.fast = k >= 33 && k <= 94 && am < ((uint64_t)1 << 31) && r_t > 0 && (uint64_t)r_t <= ((uint64_t)1 << 32);
	if (!l.fast) k = 33;
	const uint64_t p = am * (uint64_t)r_t;
	l.hi = (uint32_t)(p >> 32);
	l.lo = (uint32_t)p;
	l.half = (uint64_t)1 << (int)(k - 33);
	l.sh = (int)k - 32;
	l.neg = m_a < 0;
	return l;
}
// magnitude of the landed value for |code| = ac <= 2^31
__device__ __forceinline__ uint64_t land_magnitude(uint32_t ac, const Lander& l) {
	return ((uint64_t)ac * l.hi + l.half + __umulhi(ac, l.lo)) >> l.sh;
}

// ---------------------------------------------------------------------- RMSNorm
// floor((h << 32) / root) for |h| <= 127: with 2^32 = Q root + rem it is h Q + floor(h rem / root),
// and mulhi(h rem, Q) is that floor or one beside it. Needs root >= 2^16 (Q <= 2^16, every product
// inside 32 bits): root = floor(2^16 rms), so that is every row whose rms is at least 1.
struct NormDiv {
	int32_t root, q, rem;
	bool fast;
};
// root of RmsNormSite: max(isqrt(floor(ss 2^32 / n)), 1); the inner floor cannot change the outer one.
// n <= 131071 and |h| <= 127 keep (root + 1)^2 n inside 64 bits.
__device__ __forceinline__ NormDiv make_norm_div(uint32_t ss, int n, double inv_n) {
	const uint64_t x = (uint64_t)ss << 32;
	uint32_t r = ss == 0u ? 0u : (uint32_t)sqrt_estimate((double)ss * 4294967296.0 * inv_n);      // within one of the root
	if ((uint64_t)r * r * (uint64_t)n > x) --r;
	if ((uint64_t)(r + 1u) * (r + 1u) * (uint64_t)n <= x) ++r;
	NormDiv d;
	d.fast = r >= 65536u;
	if (r < 65536u) r = 65536u;
	uint32_t q = 0xFFFFFFFFu / r, rem = 0u - q * r;
	if (rem == r) {      // root a power of two
		++q;
		rem = 0u;
	}
	d.root = (int32_t)r;
	d.q = (int32_t)q;
	d.rem = (int32_t)rem;
	return d;
}
__device__ __forceinline__ int32_t norm_quotient(int h, const NormDiv& d) {
	const int32_t t = h * d.rem;
	int32_t e = __mulhi(t, d.q);
	const int32_t r = t - e * d.root;
	if (r < 0) --e;
	if (r >= d.root) ++e;
	return h * d.q + e;
}

// -------------------------------------------------------------------------- RoPE
// one output of rope_pair_clamped: rounding half away from zero is floor((t + 2^29 - [t < 0]) / 2^30)
__device__ __forceinline__ int rope_round(int64_t t) {
	const int32_t q = (int32_t)((t + (((int64_t)1 << 29) - (t < 0 ? 1 : 0))) >> 30);
	return max(-127, min(127, q));
}
// two interleaved pairs: codes in w, table words (c0, c1), (s0, s1)
__device__ __forceinline__ uint32_t rope_quad(uint32_t w, int2 c, int2 s) {
	const int x0 = byte_of(w, 0), y0 = byte_of(w, 1), x1 = byte_of(w, 2), y1 = byte_of(w, 3);
	return pack4(rope_round((int64_t)x0 * c.x - (int64_t)y0 * s.x), rope_round((int64_t)x0 * s.x + (int64_t)y0 * c.x),
	             rope_round((int64_t)x1 * c.y - (int64_t)y1 * s.y), rope_round((int64_t)x1 * s.y + (int64_t)y1 * c.y));
}

// ------------------------------------------------------------- loads of a wide row
// (past the L1: the projection that wrote the row may have been running when this block started)
template <bool W64> struct WideOf { using T = int32_t; };
template <> struct WideOf<true> { using T = int64_t; };
__device__ __forceinline__ void load_quad(const int32_t* p, int32_t (&x)[4]) {
	const int4 v = __ldcg((const int4*)p);
	x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void load_quad(const int64_t* p, int64_t (&x)[4]) {
	const longlong2 a = __ldcg((const longlong2*)p), b = __ldcg((const longlong2*)p + 1);
	x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
}

}  // namespace sslm
