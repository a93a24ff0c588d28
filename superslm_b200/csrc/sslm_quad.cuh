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

// ------------------------------------------------------------------ the funnel's scalars
// funnel_finish for the quads: the carried scale, and for the codes 127 / d as a float instead of the
// normalised reciprocal (R / 2^E = 1 / d up to 2^-32). The reciprocal itself is derived only where an
// element needs the integer form. About a fifth of funnel_finish's instructions, which every warp of
// the block executes on the way from one reduction to the next.
struct QuadFunnel {
	float f, f_lo;     // 127 / d to one rounding, and the rest of it (both of d rounded, above 2^24)
	uint32_t d;        // the row's maximum, at least 1
	Scale out;
	int32_t status;
};
__device__ __forceinline__ QuadFunnel quad_funnel(unsigned long long mx, const FunnelFold& fold) {
	QuadFunnel q;
	const bool wide = mx > (1ull << 31);
	const uint32_t d = wide ? 1u : max((uint32_t)mx, 1u);
	q.d = d;
	const float df = __uint2float_rn(d), rd = __fdividef(1.0f, df), f0 = 127.0f * rd;
	q.f = fmaf(fmaf(-f0, df, 127.0f), rd, f0);
	q.f_lo = fmaf(-q.f, df, 127.0f) * rd;
	const int s = __clz((int)d) - 1;                                   // 30 - floor(log2 d)
	const uint32_t dn = s >= 0 ? d << s : d >> 1;                      // 2^30 <= dn < 2^31
	q.status = fold.fold_status;
	if (fold.run.e > ((int64_t)1 << 61) || fold.run.e < -((int64_t)1 << 61)) {      // exponents that may saturate
		q.out = combine(fold.run, Scale{(int64_t)dn, -(int64_t)s});
		if (!fits_i32(q.out.m)) q.status = kCarriedScaleMantissaOutOfDomain;
	} else {
		// CombineCarriedScale; the doubling high multiply cannot saturate because dn < 2^31
		int32_t m = (int32_t)(((int64_t)(int32_t)fold.run.m * (int64_t)dn + ((int64_t)1 << 30)) >> 31);
		q.out.e = fold.run.e + (31 - s);
		if (m < (1 << 30)) {
			if (m < -(1 << 30)) q.status = kCarriedScaleMantissaOutOfDomain;
			m <<= 1;
			q.out.e -= 1;
		}
		q.out.m = m;
	}
	if (wide) q.status = kChainInputOutOfDomain;
	if (fold.pre_status != kOk) q.status = fold.pre_status;
	return q;
}

// ------------------------------------------------------------------ requant codes
// code = round_half_away(x * 127 R / 2^E), |x| <= the row's maximum d (so |code| <= 127).
// v = x * f with f = 127 / d rounded once. Up to d = 2^24 nothing else rounds and v is within 127 * 2^-24 of the
// exact quotient. Above, x and d round as well. Rounding moves a number of mantissa mu by 2^-24 / mu of itself,
// x moves v by no more than d does, and the mantissa of f is 127/64 / mu (twice that for mu above 127/64): all
// three together move v by 127 * 2^-24 (1/mu + 1/mu + mu / (127/64)) <= 127 * 2^-24 * 2.504 < 1.896e-5, at mu = 1;
// products of roundings, R's own (2^-32) and the rounding of the distance add less than 4e-8. So unless v is
// within 2e-5 of a half-integer its nearest integer IS the code: five instructions per element instead of about
// twenty. One element in 25,000 is closer -- one in most activation rows, and a row waits for its slowest warp --
// so those are settled in place by adding x * f_lo to the distance, and only within 1e-6 of the tie (or in a row
// above 2^24) out of line, at last by requant_code itself.
constexpr float kRoundMagic = 12582912.0f;      // 1.5 * 2^23: adding it leaves the nearest integer in the low bits
constexpr int kRoundMagicBits = 0x4B400000;
constexpr float kNearTie = 0.49998f;
__device__ __forceinline__ float to_float(int32_t x) { return __int2float_rn(x); }
__device__ __forceinline__ float to_float(int64_t x) { return __ll2float_rn(x); }
template <typename T>
static __device__ __noinline__ uint32_t code_quad_exact(T x0, T x1, T x2, T x3, uint32_t d) {
	int64_t dn;
	int s;
	normalize_scale((int64_t)d, &dn, &s);
	const int64_t r = dyn_recip(dn);
	return pack4(requant_code((int64_t)x0, r, s), requant_code((int64_t)x1, r, s), requant_code((int64_t)x2, r, s),
	             requant_code((int64_t)x3, r, s));
}
__device__ __forceinline__ float low_part(int32_t x, float xf) { return (float)((int64_t)x - (int64_t)xf); }
__device__ __forceinline__ float low_part(int64_t x, float xf) { return (float)(x - (int64_t)xf); }
template <typename T>
static __device__ __noinline__ uint32_t code_quad_near_tie(T x0, T x1, T x2, T x3, uint32_t d) {
	// f + f_lo = 127 / d to about 2^-46
	const float df = __uint2float_rn(d), dl = (float)(int)((int64_t)d - (int64_t)df), rd = __fdividef(1.0f, df), f0 = 127.0f * rd;
	const float f = fmaf(fmaf(-f0, df, 127.0f), rd, f0);
	const float f_lo = fmaf(-f, dl, fmaf(-f, df, 127.0f)) * rd;
	const T x[4] = {x0, x1, x2, x3};
	int c[4];
	bool tie = false;
#pragma unroll
	for (int j = 0; j < 4; ++j) {
		const float xf = to_float(x[j]);
		const float q = fmaf(xf, f, kRoundMagic) - kRoundMagic;
		const float off = fmaf(xf, f, -q) + fmaf(xf, f_lo, low_part(x[j], xf) * f);
		tie = tie || fabsf(fabsf(off) - 0.5f) < 1e-6f;
		c[j] = (int)q + (off > 0.5f ? 1 : (off < -0.5f ? -1 : 0));
	}
	if (tie) return code_quad_exact<T>(x0, x1, x2, x3, d);
	return pack4(c[0], c[1], c[2], c[3]);
}
// four codes, each kRoundMagicBits + the code, right unless the value returned (the distance of the farthest
// from its integer) is above kNearTie: then code_quad_settle
template <typename T>
__device__ __forceinline__ float code_quad_try(const T (&x)[4], const QuadFunnel& q, int (&t)[4]) {
	float far = 0.0f;
#pragma unroll
	for (int j = 0; j < 4; ++j) {
		const float xf = to_float(x[j]);
		const float m = fmaf(xf, q.f, kRoundMagic);
		t[j] = __float_as_int(m);
		far = fmaxf(far, fabsf(fmaf(xf, q.f, kRoundMagic - m)));
	}
	return far;
}
template <typename T>
__device__ __forceinline__ void code_quad_settle(const T (&x)[4], const QuadFunnel& q, int (&t)[4]) {
	float far = 1.0f;
#pragma unroll
	for (int j = 0; j < 4; ++j) {
		const float xf = to_float(x[j]);
		const float o = fmaf(xf, q.f_lo, fmaf(xf, q.f, kRoundMagic - __int_as_float(t[j])));
		t[j] += (o > 0.5f ? 1 : 0) - (o < -0.5f ? 1 : 0);
		far = fminf(far, fabsf(fabsf(o) - 0.5f));
	}
	if (far < 1e-6f || q.d > (1u << 24)) {
		const uint32_t c = code_quad_near_tie<T>(x[0], x[1], x[2], x[3], q.d);
#pragma unroll
		for (int j = 0; j < 4; ++j) t[j] = kRoundMagicBits + byte_of(c, j);
	}
}
// four codes, packed; element j in byte j
template <typename T>
__device__ __forceinline__ uint32_t code_quad(const T (&x)[4], const QuadFunnel& q) {
	int t[4];
	if (code_quad_try(x, q, t) > kNearTie) code_quad_settle(x, q, t);
	return pack4(t[0], t[1], t[2], t[3]);
}
// The same for rows of small integers (the residual sums), where a true tie 254 |x| = (2 c + 1) d is
// common: the half of an even maximum usually occurs in the row. On a tie the reference's answer
// depends on which way its reciprocal R = round(2^E / d), E = 32 + floor(log2 d), was rounded: away
// from zero if R d >= 2^E, toward it otherwise (off a tie the distance, at least 1 / (2 d), exceeds
// what R's rounding moves, 63.5 / 2^31). R was rounded up iff floor(2^(E+1) / d) is odd or d is a
// power of two; the quotient's last bit comes from two 16-bit division steps. d < 2^16.
__device__ __forceinline__ uint32_t div_step(uint32_t num, uint32_t d, float rd, uint32_t* rem) {      // num / d <= 2^16
	int32_t q = __float2int_rz(__uint2float_rn(num) * rd), r = (int32_t)(num - (uint32_t)q * d);
	if (r < 0) { --q; r += (int32_t)d; }
	if (r >= (int32_t)d) { ++q; r -= (int32_t)d; }
	*rem = (uint32_t)r;
	return (uint32_t)q;
}
__device__ __forceinline__ bool reciprocal_rounded_up(uint32_t d) {
	const float rd = __fdividef(1.0f, __uint2float_rn(d));
	uint32_t rem;
	div_step(1u << (16 + 31 - __clz((int)d)), d, rd, &rem);      // 2^(p + 16)
	div_step(rem << 16, d, rd, &rem);                            // ... 2^(p + 32)
	return 2u * rem >= d || (d & (d - 1u)) == 0u;                // ... 2^(p + 33)
}
__device__ __forceinline__ uint32_t code_small_near_tie(float x0, float x1, float x2, float x3, float f, uint32_t d) {
	const bool up = reciprocal_rounded_up(d);
	const float x[4] = {x0, x1, x2, x3};
	int c[4];
#pragma unroll
	for (int j = 0; j < 4; ++j) {
		const int a = (int)fabsf(x[j]), k = (int)rintf(fabsf(x[j]) * f);
		const int u = 254 * a - 2 * k * (int)d, dd = (int)d;      // the quotient is k + u / (2 d)
		const int up_by = (u > dd || (u == dd && up)) ? 1 : ((u < -dd || (u == -dd && !up)) ? -1 : 0);
		c[j] = x[j] < 0.0f ? -(k + up_by) : k + up_by;
	}
	return pack4(c[0], c[1], c[2], c[3]);
}
// elements: integers below 2^16 in floats, as is the row's maximum
__device__ __forceinline__ uint32_t code_small_quad(const float (&x)[4], const QuadFunnel& q) {
	int t[4];
	float far = 0.0f;
#pragma unroll
	for (int j = 0; j < 4; ++j) {
		const float m = fmaf(x[j], q.f, kRoundMagic);
		t[j] = __float_as_int(m);
		far = fmaxf(far, fabsf(fmaf(x[j], q.f, kRoundMagic - m)));
	}
	if (far > kNearTie) return code_small_near_tie(x[0], x[1], x[2], x[3], q.f, q.d);
	return pack4(t[0], t[1], t[2], t[3]);
}

// --------------------------------------------------------------------------- K/V landing
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

// ---------------------------------------------------------------------- residual
// A branch code on the stream's scale, LandingRescale(code) = round_half_away(code * rho) with
// rho = m_a r_t / 2^k: like the requant codes, in float with the near-ties settled separately. rho is
// rounded once, so the landed value is known unless it is within 127 rho 2^-23 (+ 1e-6) of a
// half-integer. Sums with the stream stay below 2^16: exact in float.
struct Recip {
	float hi, lo;      // the stream scale's reciprocal r_t as a sum of two floats (0: outside (0, 2^32])
};
__device__ __forceinline__ Recip make_recip(int64_t r_t) {
	Recip r{0.0f, 0.0f};
	if (r_t > 0 && (uint64_t)r_t <= ((uint64_t)1 << 32)) {
		r.hi = __ll2float_rn(r_t);
		r.lo = (float)(r_t - (int64_t)r.hi);
	}
	return r;
}
struct Branch {
	float rho, rho_lo, near_tie;
	bool fast;
};
// bs: the branch's scale, ss: the stream's, r: the reciprocal of its mantissa
__device__ __forceinline__ Branch make_branch(Scale bs, Recip r, Scale ss) {
	Branch b;
	const int64_t k64 = 62 - (bs.e - ss.e);
	const bool e_ok = bs.e < ((int64_t)1 << 61) && bs.e > -((int64_t)1 << 61) && ss.e < ((int64_t)1 << 61) && ss.e > -((int64_t)1 << 61);
	const bool in = e_ok && k64 >= 33 && k64 <= 94 && r.hi > 0.0f;
	const float scale = __int_as_float((127 - (in ? (int)k64 : 33)) << 23);      // 2^-k
	const int32_t m = (int32_t)bs.m;      // (a negative mantissa flips the sign of every landed value)
	const float mh = __int2float_rn(m), ml = (float)((int64_t)m - (int64_t)mh);
	const float p = mh * r.hi, e = fmaf(mh, r.hi, -p) + fmaf(mh, r.lo, ml * r.hi);
	const float rho = p + e;
	b.rho = rho * scale;
	b.rho_lo = ((p - rho) + e) * scale;
	const float top = fabsf(b.rho) * 127.0f;
	b.near_tie = 0.499999f - top * 1.1920928955078125e-07f;      // 2^-23
	b.fast = in && top < 32000.0f;
	return b;
}
static __device__ __noinline__ float land_code_exact(int code, int64_t bs_m, int64_t bs_e, int64_t ss_m, int64_t ss_e) {
	return (float)landing_rescale((int64_t)code, bs_m, dyn_recip(ss_m), bs_e, ss_e, nullptr, nullptr);
}
static __device__ __noinline__ float land_code_near_tie(int code, float rho, float rho_lo, int64_t bs_m, int64_t bs_e, int64_t ss_m,
                                                        int64_t ss_e) {
	const float cf = (float)code, q = fmaf(cf, rho, kRoundMagic) - kRoundMagic;
	const float off = fmaf(cf, rho, -q) + cf * rho_lo;      // within 2^-24 + 127 rho 2^-44
	if (fabsf(fabsf(off) - 0.5f) < 1e-6f) return land_code_exact(code, bs_m, bs_e, ss_m, ss_e);
	return q + (off > 0.5f ? 1.0f : (off < -0.5f ? -1.0f : 0.0f));
}
// w[j] = landed(code j) + stream code j, for four codes packed in c and four in st
__device__ __forceinline__ void join_quad(uint32_t c, uint32_t st, const Branch& b, Scale bs, Scale ss, float (&w)[4]) {
	float far[4], worst = 0.0f;
#pragma unroll
	for (int j = 0; j < 4; ++j) {
		const float cf = (float)byte_of(c, j);
		const float q = fmaf(cf, b.rho, kRoundMagic) - kRoundMagic;
		far[j] = fabsf(fmaf(cf, b.rho, -q));
		worst = fmaxf(worst, far[j]);
		w[j] = q + (float)byte_of(st, j);
	}
	if (worst > b.near_tie) {
#pragma unroll
		for (int j = 0; j < 4; ++j)
			if (far[j] > b.near_tie)
				w[j] = land_code_near_tie(byte_of(c, j), b.rho, b.rho_lo, bs.m, bs.e, ss.m, ss.e) + (float)byte_of(st, j);
	}
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
// A double estimate within one of the root, settled by one exact residual x - r^2 n (n <= 131071 and
// |h| <= 127 keep it inside 64 bits); Q the same way from a float reciprocal (2^32 / root <= 2^16, so
// the estimate is within one).
__device__ __forceinline__ NormDiv make_norm_div(uint32_t ss, int n, double inv_n) {
	const double ms = (double)max(ss, 1u) * 4294967296.0 * inv_n;
	double y;
	asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(ms));
	const double g = ms * y;
	uint32_t r = (uint32_t)__double2int_rz(fma(fma(-g, g, ms), 0.5 * y, g));
	const int64_t left = (int64_t)(((uint64_t)ss << 32) - (uint64_t)r * r * (uint64_t)(uint32_t)n);
	if (left < 0) --r;
	if (left >= (int64_t)(uint64_t)(2u * r + 1u) * n) ++r;
	NormDiv d;
	d.fast = r >= 65536u;
	if (r < 65536u) r = 65536u;
	int32_t q = __float2int_rz(__fdividef(4294967296.0f, __uint2float_rn(r)));
	int32_t rem = (int32_t)(0u - (uint32_t)q * r);
	if (rem < 0) {
		--q;
		rem += (int32_t)r;
	}
	if (rem >= (int32_t)r) {
		++q;
		rem -= (int32_t)r;
	}
	d.root = (int32_t)r;
	d.q = q;
	d.rem = rem;
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

// ---------------------------------------------------------------------- softmax constants
// of one kv head of a row: sm = Combine(S[q], softmax_khead) -> C30 constants -> width gate
__device__ __forceinline__ int32_t softmax_consts(Scale q, Scale kh, uint64_t width, SoftmaxConsts* sc) {
	sc->c = IExpConsts{0, 0, 0};
	sc->peak = 0;
	if (!fits_i32(q.m) || !fits_i32(kh.m)) return kCarriedScaleMantissaOutOfDomain;
	const Scale sm = combine(q, kh);
	if (!fits_i32(sm.m)) return kCarriedScaleMantissaOutOfDomain;
	if (iexp_scale_constants(sm.m, sm.e, &sc->c) != 0) return kIExpScaleDerivationOutOfDomain;
	if (!softmax_width_in_domain(sc->c.q_b, sc->c.q_c, width, &sc->peak)) return kSoftmaxRowWidthOutOfDomain;
	// q_ln2 == 0: every element's construction is refused by the reference (IExpConstruct's q_ln2 >= 1 check) ->
	// SoftmaxKernelRefused. The attention kernels' 32-bit element form also needs q_ln2 <= q_b; that holds for every
	// constant triple iexp_scale_constants returns and needs no test here: q_ln2 = floor(LN2_Q * r / 2^s) and
	// q_b = floor(B_Q * r / 2^s) with the same unsigned reciprocal r and the same shift s, and LN2_Q < B_Q, so the
	// floors are ordered the same way.
	return sc->c.q_ln2 < 1 ? kSoftmaxKernelRefused : kOk;
}

// -------------------------------------------------------------------------- q/k/v bias
// The bias term of one element, false when it leaves int64. A bias code inside 32 bits keeps the
// product with the row's reciprocal (at most 2^32) inside 64; others take the 128-bit composite.
__device__ __forceinline__ bool bias_term(int64_t bias, int64_t r_a, int bexp, int64_t* term) {
	if (bias == (int64_t)(int32_t)bias && r_a > 0 && (uint64_t)r_a <= ((uint64_t)1 << 32)) {
		*term = rdivpot64(bias * r_a, bexp);
		return true;
	}
	return bias_reconcile(bias, r_a, bexp, term);
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
