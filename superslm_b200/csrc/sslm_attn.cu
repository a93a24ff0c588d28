// Integer i-exp softmax attention over the paged int8 KV pool, staged through shared memory, with both
// contractions on the tensor cores (mma.sync m16n8k32, exact int32 accumulation). A row is one token's q heads
// over positions 0..pos, cut by kv head, so that each K / V byte of a sequence leaves HBM once per kv head:
//
//   k_attention        many decode rows: a block owns one kv head of a row and meets nobody
//   k_attention_few    few rows: the row is cut along its width as well; its blocks form a thread-block cluster
//                      and exchange maxima, sums and partial contexts through distributed shared memory
//   k_attention_chunk  prefill chunks: tiles of 32 query rows, wide ones cut over a cluster, scores kept
//   k_attention_tile   prefill chunks: tiles of 64 query rows, the prefix walked three times, nothing kept
//
//   stage 1  scores[g][k] = q_rot[g] . K[k]      A = the group's q rows (heads in the M
//            dimension), B = 8 K rows per MMA straight from the page (16-byte loads; the
//            head-dim order inside an MMA is permuted identically on both operands)
//   stage 2  e_k = second-order integer exp of (score - max); total; p_k = (e_k << 15) /
//            total (SoftmaxRowQ15); p_k is split into two u8 planes, p = 256 ph + pl
//   stage 3  ctx[g][d] = sum_k p_k V[k][d]       A = pl / ph (u8), B = transposed V page
//            words (4 positions of one channel per register), two MMAs per plane, then
//            ctx = acc_l + 256 acc_h, the per-head fold and the row max for the funnel
//
// Every reduction is an integer max or add, so the result does not depend on the order in
// which lanes, warps or blocks contribute. Restates the attention block of RunLayerLoopImpl
// (src/forward/forward_sites.cpp:1858-1897), SoftmaxRowQ15 (src/intmath.cpp:796-901) and
// GemmProbQ15Accumulate (src/matmul.cpp:522-538).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <initializer_list>

#include "sslm_cluster.cuh"
#include "sslm_kernels.h"
#include "sslm_quad.cuh"

namespace sslm {

// One softmax element for constants that passed the gates of k_qkv_post (1 <= q_ln2 <= q_b
// < 2^24, q_c >= 0, peak = q_b^2 + q_c within the width gate): the value iexp_element()
// computes, on 32-bit words and without a branch. dq = max - score (0 <= dq < 2^32).
// z = floor(x / q_ln2) comes from one fused multiply-add that rounds toward zero onto an integer grid, with a
// reciprocal a little too small, so that it is z or z - 1 and the exact remainder tells which.
//
// The reference also refuses an element whose value leaves [0, peak] (SoftmaxRowQ15's per-element
// bound, src/intmath.cpp:870-888). Under the gates above that cannot happen, so the kernels carry
// no such test: 0 <= rem < q_ln2 <= q_b gives 1 <= base = q_b - rem <= q_b, hence
// 0 <= (base^2 + q_c) >> z <= q_b^2 + q_c = peak (and peak >= 1 because q_b >= 1).
struct IExpFast {
	uint32_t ln2, clip;     // q_ln2, 30 * q_ln2
	int32_t qb;
	int64_t qc;
	float inv_ln2;          // (1 - 2^-21) / q_ln2
};
__device__ __forceinline__ IExpFast iexp_fast_prepare(const SoftmaxConsts& k) {
	IExpFast f;
	f.ln2 = (uint32_t)k.c.q_ln2;
	f.clip = 30u * f.ln2;
	f.qb = (int32_t)k.c.q_b;
	f.qc = k.c.q_c;
	f.inv_ln2 = (1.0f / (float)f.ln2) * 0.9999995f;
	return f;
}
// The element by itself: k_attention_tile, which keeps nothing between its walks. (x = z * q_ln2 + rem, rem < q_ln2 < 2^24, z <= 30)
__device__ __forceinline__ int64_t iexp_fast(uint32_t dq, const IExpFast& f) {
	const uint32_t x = min(dq, f.clip);
	uint32_t z = (uint32_t)__float_as_int(__fmaf_rz(__uint2float_rn(x), f.inv_ln2, 8388608.0f)) - 0x4B000000u;
	uint32_t rem = x - z * f.ln2;
	if (rem >= f.ln2) {
		rem -= f.ln2;
		++z;
	}
	const int32_t base = f.qb - (int32_t)rem;
	return (int64_t)((uint64_t)((int64_t)base * (int64_t)base + f.qc) >> z);
}
// Q15 probability floor((e << 15) / tot), 0 <= e <= tot, 1 <= tot < 2^63.
//
// The row's constants scale e to 31 bits; the float product is then within pf 2^-21 + 2^-15 of the
// quotient, and its floor (one add that rounds toward zero) is the answer unless the fraction is that
// close to an integer -- at most one element in some ten thousand, and never below the first integer,
// where nearly all elements of a long row lie. Those take prob_q15.
struct ProbRow {
	unsigned long long tot;
	float c;      // 2^(15 + sh) / tot
	int sh;
};
__device__ __forceinline__ ProbRow prob_row(unsigned long long total) {
	ProbRow r;
	r.tot = total > 1ull ? total : 1ull;
	r.sh = max(0, 33 - __clzll((long long)r.tot));
	r.c = (32768.0f / (float)r.tot) * __int_as_float((127 + r.sh) << 23);
	return r;
}
// the exact form: a float quotient off by at most one, settled by one signed remainder
__device__ __forceinline__ uint32_t prob_q15(int64_t e, unsigned long long tot, float rinv) {
	const unsigned long long num = (unsigned long long)e << 15;
	uint32_t p = min(__float2uint_rz(__ll2float_rn(e) * rinv), 32768u);
	const long long r = (long long)(num - (unsigned long long)p * tot);
	p -= r < 0 ? 1u : 0u;
	p += r >= (long long)tot ? 1u : 0u;
	return p;
}
// bits 0..15 of the result: the probability, unless *unsure came out true
__device__ __forceinline__ uint32_t prob_fast(int64_t e, const ProbRow& r, bool* unsure) {
	const float pf = __uint2float_rn((uint32_t)((uint64_t)e >> r.sh)) * r.c;
	const float t = __fadd_rz(pf, 8388608.0f);
	const float off = fabsf((pf - (t - 8388608.0f)) - 0.5f), eps = fmaf(pf, 4.76837158203125e-07f, 3.2e-05f);
	*unsure = *unsure || (off > 0.5f - eps && pf > eps);
	return (uint32_t)__float_as_int(t);
}
static __device__ __noinline__ uint2 prob_pair_exact(int64_t e0, int64_t e1, unsigned long long tot) {
	const float rinv = 32768.0f / (float)tot;
	return make_uint2(prob_q15(e0, tot, rinv), prob_q15(e1, tot, rinv));
}
// A row's constants of the probability pass. pf = (base^2 + q_c) 2^-z 32768 / total in float is within
// pf 2^-21 (five roundings) + 32768 / total (the element's own floor) of the quotient, so its floor is the
// probability unless the nearest integer from 1 up is that close; those take prob_q15. Below 1 it is 0.
struct ChunkProb {
	float c, qc, eps;
};
__device__ __forceinline__ ChunkProb chunk_prob(unsigned long long total, const IExpFast& f) {
	ChunkProb p;
	p.c = 32768.0f / (float)(total > 1ull ? total : 1ull);
	p.qc = (float)f.qc;
	p.eps = p.c * 1.01f;
	return p;
}
constexpr uint32_t kBaseOfZero = 63u << 24;      // (shift, base) of an element that counts for nothing
// The element of the kernels that keep their scores; *parts, its (shift, base) word, takes the score's place and the
// probability pass reads it instead of dividing again.
__device__ __forceinline__ int64_t chunk_exp(uint32_t dq, const IExpFast& f, uint32_t* parts) {
	const uint32_t x = min(dq, f.clip);
	uint32_t z = (uint32_t)__float_as_int(__fmaf_rz(__uint2float_rn(x), f.inv_ln2, 8388608.0f)) - 0x4B000000u;
	uint32_t rem = x - z * f.ln2;
	if (rem >= f.ln2) {
		rem -= f.ln2;
		++z;
	}
	const uint32_t base = (uint32_t)f.qb - rem;      // 1 .. q_b < 2^24
	*parts = (z << 24) + base;
	return (int64_t)(((uint64_t)base * base + (uint64_t)f.qc) >> z);
}
__device__ __forceinline__ uint32_t chunk_prob_of(uint32_t parts, const ChunkProb& p, float* near) {
	const float bf = __uint2float_rn(parts & 0xFFFFFFu);
	const float pf = fmaf(bf, bf, p.qc) * __int_as_float(__float_as_int(p.c) - (int)((parts >> 24) << 23));
	const float whole = fmaxf((pf + 8388608.0f) - 8388608.0f, 1.0f);
	*near = fminf(*near, fmaf(pf, -4.76837158203125e-07f, fabsf(pf - whole)));
	return (uint32_t)__float_as_int(__fadd_rz(pf, 8388608.0f));      // (low 16 bits)
}
static __device__ __noinline__ uint4 chunk_prob_exact(uint32_t p0, uint32_t p1, uint32_t p2, uint32_t p3, int64_t qc, unsigned long long total) {
	const unsigned long long tot = total > 1ull ? total : 1ull;
	const float rinv = 32768.0f / (float)tot;
	auto one = [&](uint32_t p) {
		const uint64_t base = p & 0xFFFFFFu;
		return (p >> 24) == 63u ? 0u : prob_q15((int64_t)((base * base + (uint64_t)qc) >> (p >> 24)), tot, rinv);
	};
	return make_uint4(one(p0), one(p1), one(p2), one(p3));
}

// bytes 0 (low plane) or 1 (high plane) of four probabilities, packed into one word
__device__ __forceinline__ uint32_t pack_plane(uint32_t p0, uint32_t p1, uint32_t p2, uint32_t p3, int byte) {
	const uint32_t sel = byte ? 0x0051u : 0x0040u;
	return __byte_perm(__byte_perm(p0, p1, sel), __byte_perm(p2, p3, sel), 0x5410u);
}

// D += A(16x32, row) * B(32x8, col); rows 8..15 of A are always zero here (a1 = a3 = 0)
__device__ __forceinline__ void mma_s8s8(int (&c)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
	asm volatile(
	    "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
	    : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
	    : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_u8s8(int (&c)[4], uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
	asm volatile(
	    "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
	    : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
	    : "r"(a0), "r"(0u), "r"(a2), "r"(0u), "r"(b0), "r"(b1));
}

// The HD/16 words of a head-dim row that lane column c (= lane & 3) feeds to the HD/32
// score MMAs: MMA j takes words 2j (k slots 4c..4c+3) and 2j+1 (k slots 16+4c..). Any
// assignment of head-dim bytes to k slots is valid as long as q and K use the same one.
// (Plain loads, not the read-only path: q and the newest K / V rows were written by the kernel
// just before this one, which may still have been running when this block was placed.)
template <int HD>
__device__ __forceinline__ void load_row_words(const int8_t* row, int c, uint32_t (&w)[HD / 16]) {
	if constexpr (HD == 32) {
		const int2 x = *(const int2*)(row + c * 8);
		w[0] = (uint32_t)x.x; w[1] = (uint32_t)x.y;
	} else if constexpr (HD == 128) {
		// one 32-byte load per lane: the four lanes of a position cover its 128-byte row, and a
		// warp's load covers eight whole lines (rows are 128-byte aligned in the pages and in q)
		asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
		             : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
		             : "l"(row + c * 32)
		             : "memory");
	} else {
		const int4 x = *(const int4*)(row + c * 16);
		w[0] = (uint32_t)x.x; w[1] = (uint32_t)x.y; w[2] = (uint32_t)x.z; w[3] = (uint32_t)x.w;
	}
}

// What one block keeps in shared memory. `cp` = positions a block can hold (a multiple of 64).
struct AttnSmem {
	int64_t* pbase;            // [cp/16] byte offset of each of the row's pages inside a plane
	int32_t* sc;               // [G][cp] scores, later (shift, remainder) of each element
	uint8_t* pl;               // [G][cp] low byte of the Q15 probability
	uint8_t* ph;               // [G][cp] high byte
	unsigned long long* sum;   // [8] row total per head
	int32_t* mx;               // [8] row maximum per head
	int32_t* fold;             // [8][3] context fold (identity, multiplier, shift) of this kv head's q heads
	uint32_t* refused;
};
__host__ __device__ inline size_t attn_smem_bytes(int group, int cp) {
	return (size_t)cp / 16 * 8 + (size_t)group * cp * 6 + 8 * 8 + 8 * 4 + 24 * 4 + 16;
}
__device__ __forceinline__ AttnSmem carve(unsigned char* smem, int group, int cp) {
	AttnSmem s;
	s.pbase = (int64_t*)smem;
	s.sum = (unsigned long long*)(s.pbase + cp / 16);
	s.sc = (int32_t*)(s.sum + 8);
	s.pl = (uint8_t*)(s.sc + (size_t)group * cp);
	s.ph = s.pl + (size_t)group * cp;
	s.mx = (int32_t*)(s.ph + (size_t)group * cp);
	s.fold = s.mx + 8;
	s.refused = (uint32_t*)(s.fold + 24);
	return s;
}
// ask for the line at p to be brought into L2; nothing waits for it
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// One attention row = one token of one sequence, all its q heads over the positions 0..pos, cut by kv
// head: a block serves the q heads of one GQA group, so K and V bytes are read once per kv head. Many
// rows (a decode batch, the rows of a prefill chunk) run this way, a block meeting nobody:
//   1  scores (tensor cores) and the row maximum per head
//   2  e_k per element and the row total, then p_k = (e_k << 15) / total
//   3  P.V (tensor cores), per-head context fold, row maximum for the funnel kernel that follows
// HD = head_dim (32, 64 or 128); a warp owns NDB blocks of eight channels, so threads = 4 * HD / NDB.
template <int HD, int NDB>
__global__ void __launch_bounds__(4 * HD / NDB, (HD == 128 ? 2 : 4) * NDB)
k_attention(RowBatch b, Dims d, const __grid_constant__ LayerDev layer, int layer_index, KvPoolDev pool, int cp, int reverse_rows) {
	extern __shared__ __align__(16) unsigned char smem[];
	// blocks start in index order: with reverse_rows the last (widest) rows of a prefill chunk go first
	const int r = reverse_rows ? (int)gridDim.y - 1 - (int)blockIdx.y : (int)blockIdx.y;
	const int kvh = (int)blockIdx.x;
	constexpr int kAttnThreads = 4 * HD / NDB, kAttnWarps = kAttnThreads / 32;
	const int G = d.heads / d.kv_heads;
	const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
	const int g = lane >> 2, c = lane & 3;
	const AttnSmem s = carve(smem, G, cp);
	// Ahead of the kernel that lands this step's K / V rows (it may still be running): the row
	// descriptor and the page table were uploaded before the step's first launch, and every K / V
	// row but the newest was written by earlier steps. So the page offsets are staged now, and
	// the old K rows are asked into L2 while that kernel, which moves little data, finishes.
	const int n = b.rows[r].pos + 1;
	const int n64 = (n + 63) & ~63;
	const int8_t* kplane = pool.base + kv_plane_offset(d, pool, layer_index, kvh, 0);
	const int8_t* vplane = pool.base + kv_plane_offset(d, pool, layer_index, kvh, 1);
	const int npages = (n + kPageTokens - 1) / kPageTokens;
	{
		// entries beyond the row's last page, up to the 64-position group stage 3 reads, repeat
		// that page: their probabilities are zero, so any readable V words will do
		const int32_t* pages = b.rows[r].pages;
		for (int j = t; j < (n64 >> 4); j += kAttnThreads)
			s.pbase[j] = (int64_t)pages[min(j, npages - 1)] * (kPageTokens * HD);
	}
	if (t < 3 * G) s.fold[t] = layer.f_ctx[3 * kvh * G + t];      // (weights: ahead of the wait)
	__syncthreads();
	constexpr int kRowsPerLine = 128 / HD;
	for (int pos = t * kRowsPerLine; pos < n - 1; pos += kAttnThreads * kRowsPerLine)
		prefetch_l2(kplane + s.pbase[pos >> 4] + (pos & 15) * HD);
	pdl_wait();
	pdl_release();
	if (t == 0) *s.refused = __ldcg(&b.status[r]) != 0 ? 1u : 0u;
	if (t < 8) {
		s.mx[t] = INT32_MIN;
		s.sum[t] = 0ull;
	}
	const SoftmaxConsts smc = b.smc[(size_t)r * d.kv_heads + kvh];   // wanted after the scores; asked for now
	__syncthreads();
	if (*s.refused != 0u) return;

	// ---- stage 1: scores, 8 positions per MMA group, groups dealt round-robin to the warps, and the
	// row's maximum per head on the way. Lanes beyond the row's end read its last position again
	// (no predicated loads); their columns are stored as INT32_MIN, which the maximum ignores.
	{
		constexpr int NW = HD / 16;
		uint32_t qw[NW];
		load_row_words<HD>(b.qrot + (size_t)r * d.hidden + (size_t)(kvh * G + min(g, G - 1)) * HD, c, qw);
		const int nblk = (n + 7) >> 3;
		constexpr int U = 4;
		int rmax = INT32_MIN;
		for (int blk0 = warp * U; blk0 < nblk; blk0 += kAttnWarps * U) {
			uint32_t kw[U][NW];
#pragma unroll
			for (int u = 0; u < U; ++u) {
				const int pos = min((blk0 + u) * 8 + g, n - 1);
				load_row_words<HD>(kplane + s.pbase[pos >> 4] + (pos & 15) * HD, c, kw[u]);
			}
#pragma unroll
			for (int u = 0; u < U; ++u) {
				int acc[4] = {0, 0, 0, 0};
#pragma unroll
				for (int j = 0; j < NW / 2; ++j) mma_s8s8(acc, qw[2 * j], qw[2 * j + 1], kw[u][2 * j], kw[u][2 * j + 1]);
				const int k = (blk0 + u) * 8 + c * 2;
				if (g < G && blk0 + u < nblk) {
					const int v0 = k < n ? acc[0] : INT32_MIN, v1 = k + 1 < n ? acc[1] : INT32_MIN;
					*(int2*)&s.sc[(size_t)g * cp + k] = make_int2(v0, v1);
					rmax = max(rmax, max(v0, v1));
				}
			}
		}
		rmax = max(rmax, __shfl_xor_sync(0xffffffffu, rmax, 1));
		rmax = max(rmax, __shfl_xor_sync(0xffffffffu, rmax, 2));
		if (c == 0 && g < G && rmax != INT32_MIN) atomicMax(&s.mx[g], rmax);
	}
	__syncthreads();

	// the softmax below moves no data: ask for the row's V pages (16 lines each) meanwhile
	for (int ln = t; ln < npages * (kPageTokens * HD / 128); ln += kAttnThreads)
			prefetch_l2(vplane + s.pbase[ln / (kPageTokens * HD / 128)] + (ln % (kPageTokens * HD / 128)) * 128);

	// ---- stage 2: softmax. The work is dealt to the warps as (head, 128-position chunk) pairs, so
	// that every warp is busy whatever the width; a lane takes 4 consecutive positions. First the
	// exponentials and their sum per head; the score's place then holds the element's
	// (shift, remainder), which the probability pass rebuilds it from.
	const IExpFast fx = iexp_fast_prepare(smc);
	const int nchunk = (n64 + 127) >> 7;
	{
#pragma unroll 1
		for (int pr = warp; pr < G * nchunk; pr += kAttnWarps) {
			const int h = pr / nchunk, k4 = (pr - h * nchunk) * 128 + lane * 4;
			unsigned long long tot = 0;
			if (k4 < n) {
				int32_t* row = s.sc + (size_t)h * cp;
				const uint32_t m = (uint32_t)s.mx[h];
				const int4 v = *(const int4*)&row[k4];
				uint32_t q0, q1, q2, q3;
				const int64_t e0 = chunk_exp(m - (uint32_t)v.x, fx, &q0);
				int64_t e1 = chunk_exp(m - (uint32_t)v.y, fx, &q1);
				int64_t e2 = chunk_exp(m - (uint32_t)v.z, fx, &q2);
				int64_t e3 = chunk_exp(m - (uint32_t)v.w, fx, &q3);
				if (k4 + 3 >= n) {       // the row's last group: positions beyond its end count for nothing
					if (k4 + 1 >= n) { e1 = 0; q1 = kBaseOfZero; }
					if (k4 + 2 >= n) { e2 = 0; q2 = kBaseOfZero; }
					e3 = 0; q3 = kBaseOfZero;
				}
				tot = (unsigned long long)(e0 + e1) + (unsigned long long)(e2 + e3);
				*(int4*)&row[k4] = make_int4((int)q0, (int)q1, (int)q2, (int)q3);
			}
			// a lane's partial is below 2^50; three 24-bit limbs add up across the warp without
			// leaving 32 bits, one warp-reduce instruction each
			const uint32_t l0 = __reduce_add_sync(0xffffffffu, (uint32_t)tot & 0xFFFFFFu);
			const uint32_t l1 = __reduce_add_sync(0xffffffffu, (uint32_t)(tot >> 24) & 0xFFFFFFu);
			const uint32_t l2 = __reduce_add_sync(0xffffffffu, (uint32_t)(tot >> 48));
			if (lane == 0) atomicAdd(&s.sum[h], (unsigned long long)l0 + ((unsigned long long)l1 << 24) + ((unsigned long long)l2 << 48));
		}
	}
	__syncthreads();
	// probabilities as two u8 planes, zero beyond the row up to the next multiple of 64 (stage 3
	// reads whole 64-position groups)
	{
		const int n4 = (n + 3) & ~3;
#pragma unroll 1
		for (int task = warp; task < G * nchunk; task += kAttnWarps) {
			const int h = task / nchunk, k4 = (task - h * nchunk) * 128 + lane * 4;
			if (k4 < n4) {
				const ChunkProb pr = chunk_prob(s.sum[h], fx);
				const int4 v = *(const int4*)&s.sc[(size_t)h * cp + k4];
				float near = 1.0f;
				uint32_t p0 = chunk_prob_of((uint32_t)v.x, pr, &near), p1 = chunk_prob_of((uint32_t)v.y, pr, &near);
				uint32_t p2 = chunk_prob_of((uint32_t)v.z, pr, &near), p3 = chunk_prob_of((uint32_t)v.w, pr, &near);
				if (near < pr.eps) {
					const uint4 x = chunk_prob_exact((uint32_t)v.x, (uint32_t)v.y, (uint32_t)v.z, (uint32_t)v.w, fx.qc, s.sum[h]);
					p0 = x.x; p1 = x.y; p2 = x.z; p3 = x.w;
				}
				*(uint32_t*)&s.pl[(size_t)h * cp + k4] = pack_plane(p0, p1, p2, p3, 0);
				*(uint32_t*)&s.ph[(size_t)h * cp + k4] = pack_plane(p0, p1, p2, p3, 1);
			} else if (k4 < n64) {
				*(uint32_t*)&s.pl[(size_t)h * cp + k4] = 0u;
				*(uint32_t*)&s.ph[(size_t)h * cp + k4] = 0u;
			}
		}
	}
	__syncthreads();

	// ---- stage 3: ctx = P V. Lane column c owns page 4*grp + c of each
	// 64-position group; its 16-byte row of the transposed page feeds two MMAs (positions 0..7 and
	// 8..15). Nothing is predicated: the page table and the planes are padded to whole groups, and
	// lanes of MMA rows beyond the group's heads read head 0's probabilities (their output rows are
	// never stored).
	int accl[NDB][4], acch[NDB][4];
#pragma unroll
	for (int i = 0; i < NDB; ++i)
#pragma unroll
		for (int j = 0; j < 4; ++j) accl[i][j] = acch[i][j] = 0;
	{
		const int ngrp = n64 >> 6;
		const uint8_t* pl = s.pl + (size_t)(g < G ? g : 0) * cp + c * kPageTokens;
		const uint8_t* ph = s.ph + (size_t)(g < G ? g : 0) * cp + c * kPageTokens;
		const int8_t* vch = vplane + (warp * NDB * 8 + g) * kPageTokens;
		// UG groups' V words are requested before the first of them is used
		constexpr int UG = 4;
		auto group = [&](int grp, const int4 (&vv)[NDB]) {
			const int4 al = *(const int4*)(pl + grp * 64);
			const int4 ah = *(const int4*)(ph + grp * 64);
#pragma unroll
			for (int i = 0; i < NDB; ++i) {
				const int4 v = vv[i];
				mma_u8s8(accl[i], (uint32_t)al.x, (uint32_t)al.y, (uint32_t)v.x, (uint32_t)v.y);
				mma_u8s8(accl[i], (uint32_t)al.z, (uint32_t)al.w, (uint32_t)v.z, (uint32_t)v.w);
				mma_u8s8(acch[i], (uint32_t)ah.x, (uint32_t)ah.y, (uint32_t)v.x, (uint32_t)v.y);
				mma_u8s8(acch[i], (uint32_t)ah.z, (uint32_t)ah.w, (uint32_t)v.z, (uint32_t)v.w);
			}
		};
		int grp0 = 0;
		for (; grp0 + UG <= ngrp; grp0 += UG) {
			int4 vv[UG][NDB];
#pragma unroll
			for (int u = 0; u < UG; ++u) {
				const int64_t pb = s.pbase[(grp0 + u) * 4 + c];
#pragma unroll
				for (int i = 0; i < NDB; ++i) vv[u][i] = *(const int4*)(vch + pb + i * 8 * kPageTokens);
			}
#pragma unroll
			for (int u = 0; u < UG; ++u) group(grp0 + u, vv[u]);
		}
		for (; grp0 < ngrp; ++grp0) {
			int4 vv[NDB];
			const int64_t pb = s.pbase[grp0 * 4 + c];
#pragma unroll
			for (int i = 0; i < NDB; ++i) vv[i] = *(const int4*)(vch + pb + i * 8 * kPageTokens);
			group(grp0, vv);
		}
	}
	{
		// per-head context fold (forward_sites.cpp:1889-1896), store, row maximum for the funnel
		uint32_t smax = 0;
		if (g < G) {
			const int head = kvh * G + g;
			const int32_t fi = s.fold[3 * g], fm = s.fold[3 * g + 1], fs = s.fold[3 * g + 2];
#pragma unroll
			for (int i = 0; i < NDB; ++i) {
				int2 o;
				o.x = fold(accl[i][0] + 256 * acch[i][0], fi, fm, fs);
				o.y = fold(accl[i][1] + 256 * acch[i][1], fi, fm, fs);
				const int ch = (warp * NDB + i) * 8 + c * 2;
				*(int2*)(b.ctxw + (size_t)r * d.hidden + (size_t)head * HD + ch) = o;
				const uint32_t ax = o.x < 0 ? 0u - (uint32_t)o.x : (uint32_t)o.x;
				const uint32_t ay = o.y < 0 ? 0u - (uint32_t)o.y : (uint32_t)o.y;
				smax = max(smax, max(ax, ay));
			}
		}
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) smax = max(smax, __shfl_xor_sync(0xffffffffu, smax, o));
		if (lane == 0 && smax) atomicMax(&b.rowmax[(size_t)r * 4 + 3], (unsigned long long)smax);
	}
}

// ---------------------------------------------------------------- few rows: slices over a cluster
// While rows are few (a handful of conversations decoding), the time of an attention row is one
// block's chain of dependent steps, so the row is cut along its width into slices, one block each; the
// blocks of a row -- all its kv heads when `whole_row`, else those of one kv head -- form a cluster and
// exchange maxima, sums, shares of P.V and, with the whole row, the funnel's maximum (forward_sites.cpp:
// 1898-1903; no separate funnel kernel then). The exact integer softmax needs all of these to be exact:
// an element's exponential depends on the row maximum through floor divisions.
//
// The K / V rows of earlier calls are in place, so with STAGED a block copies those of its slice into
// shared memory (cp.async) ahead of the dependency wait, while the row kernel in front runs; behind the
// wait it fetches only what this call lands: a decode row's own position, a chunk's positions. One row of 2,011 positions, 1.5B widths:
// 13.9 us with four slices per kv head read through L2 and cluster barriers around every exchange.
template <int HD>
struct FewSmem {
	static constexpr int kKStride = HD == 128 ? HD + 16 : HD;      // bytes per staged K row (bank conflicts)
	static constexpr int kVStride = HD * kPageTokens + 32;         // bytes per staged V page
	int64_t* pbase;            // [cp / 16] byte offset of each of the block's pages inside a plane
	int32_t* sc;               // [G][cp] scores, later (shift, remainder) of each element
	uint8_t *pl, *ph;          // [G][cp] low / high byte of the Q15 probability
	unsigned long long* sum;   // [8] this slice's sums
	unsigned long long* rx_sum;      // [16][8] every slice's
	int32_t *rx_max;           // [16][8]
	int32_t* rx_ctx;           // [splits][G * HD / splits] shares of the channels this block reduces
	uint32_t* rx_top;          // [16] every block's largest folded magnitude
	int32_t* mx;               // [8] this slice's maxima
	int32_t* fold;             // [8][3]
	uint32_t* misc;            // [0] this block's largest folded magnitude, [1] refused
	int8_t *ks, *vs;           // staged K rows and V pages
	__host__ __device__ static size_t fixed_bytes() { return 8 * 8 + 16 * 8 * 8 + 16 * 8 * 4 + (size_t)8 * HD * 4 + 16 * 4 + 8 * 4 + 24 * 4 + 4 * 4; }
	__host__ __device__ static size_t bytes(int group, int cp, bool staged) {
		return (size_t)cp / 16 * 8 + (size_t)group * cp * 6 + fixed_bytes() + (staged ? (size_t)cp * kKStride + (size_t)cp / 16 * kVStride + 32 : 0);
	}
	__device__ static FewSmem carve(unsigned char* p, int group, int cp) {
		FewSmem s;
		s.pbase = (int64_t*)p;
		s.sum = (unsigned long long*)(s.pbase + cp / 16);
		s.rx_sum = s.sum + 8;
		s.sc = (int32_t*)(s.rx_sum + 128);
		s.pl = (uint8_t*)(s.sc + (size_t)group * cp);
		s.ph = s.pl + (size_t)group * cp;
		s.rx_ctx = (int32_t*)(s.ph + (size_t)group * cp);
		s.rx_max = s.rx_ctx + 8 * HD;
		s.rx_top = (uint32_t*)(s.rx_max + 128);
		s.mx = (int32_t*)(s.rx_top + 16);
		s.fold = s.mx + 8;
		s.misc = (uint32_t*)(s.fold + 24);
		s.ks = (int8_t*)(((uintptr_t)(s.misc + 4) + 15) & ~(uintptr_t)15);
		s.vs = s.ks + (size_t)cp * kKStride;
		return s;
	}
};
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// the words of load_row_words from a staged K row (plain shared-memory loads)
template <int HD>
__device__ __forceinline__ void shared_row_words(const int8_t* row, int c, uint32_t (&w)[HD / 16]) {
	if constexpr (HD == 32) {
		const int2 x = *(const int2*)(row + c * 8);
		w[0] = (uint32_t)x.x; w[1] = (uint32_t)x.y;
	} else {
#pragma unroll
		for (int h = 0; h < HD / 64; ++h) {
			const int4 x = *(const int4*)(row + c * (HD / 4) + 16 * h);
			w[4 * h] = (uint32_t)x.x; w[4 * h + 1] = (uint32_t)x.y; w[4 * h + 2] = (uint32_t)x.z; w[4 * h + 3] = (uint32_t)x.w;
		}
	}
}

// (Registers: left to itself the compiler takes 56 to 80, and at 64 some forms spill: 24 rows of 500 to
// 1,500 positions at the 1.5B widths, two slices each, took 1,970 us a token then, 1,810 in 80, 1,730 in 100.)
//
// SITE: the q/k/v site of a decode row runs here too (k_qkv_post, which states the reference's lines), so a launch and its
// boundary go and the staging hides behind the projection. Every block codes and rotates its kv head's q rows; the
// one whose slice ends with the row lands K and V, straight into its staged rows as well. All blocks of a row come to the
// same verdict from the same words; rank 0 speaks for it. kSiteBias: a bias joins every element, so the blocks exchange
// their elements' maximum (and whether one of them left its domain) before anything is coded.
enum FewSite { kSiteApart = 0, kSitePlain, kSiteBias };
struct QkvSite {
	const int32_t *rope_cos, *rope_sin;
};
template <int HD, bool STAGED, int SITE, bool W64>
__global__ void __launch_bounds__(2 * HD, 1)
k_attention_few(RowBatch b, Dims d, const __grid_constant__ LayerDev layer, int layer_index, KvPoolDev pool, int cp, int splits,
                int whole_row, int chunk, QkvSite site) {
	static_assert(SITE == kSiteApart || STAGED, "K and V land in the staged rows");
	using S = FewSmem<HD>;
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ __align__(8) unsigned long long s_bars[SITE == kSiteBias ? 5 : 4];
	constexpr int kThreads = 2 * HD, kWarps = kThreads / 32, NW = HD / 16;
	const int r = (int)blockIdx.y, kvh = (int)blockIdx.x / splits, split = (int)blockIdx.x % splits;
	const int G = d.heads / d.kv_heads;
	const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, c = lane & 3;
	const S s = S::carve(smem, G, cp);
	const uint32_t my_rank = cluster_rank(), kv_rank0 = my_rank - (uint32_t)split;      // rank of this kv head's first slice
	const uint32_t cluster_blocks = whole_row ? (uint32_t)(d.kv_heads * splits) : (uint32_t)splits;
	const int per = HD / splits, ch0 = split * per;                  // channels this block reduces
	auto bar = [&](int i) { return cta_addr(&s_bars[i]); };
	if (t == 0) {
		const int held = (blockIdx.x | blockIdx.y) == 0 ? b.debug_withhold : 0;
		auto more = [&](int i) { return held == i + 1 ? 4u : 0u; };
		exchange_init(bar(0), (uint32_t)(splits * G * 4) + more(0));
		exchange_init(bar(1), (uint32_t)(splits * G * 8) + more(1));
		exchange_init(bar(2), (uint32_t)(G * HD * 4) + more(2));
		exchange_init(bar(3), 4u * cluster_blocks + more(3));
		if (SITE == kSiteBias) exchange_init(bar(4), 8u * cluster_blocks + more(4));
		exchange_fence_init();
	}
	// ahead of the kernel that lands this step's K / V rows: the page table, the old rows
	const int width = b.rows[r].pos + 1;
	const int slen = ((width + splits - 1) / splits + 63) & ~63;
	const int p0 = split * slen;                                   // first position of this slice
	const int n = max(0, min(slen, width - p0));                   // positions in it
	const int n64 = (n + 63) & ~63, npages = (n + kPageTokens - 1) / kPageTokens;
	// positions of the slice that were there before this call (the rows of a chunk are consecutive positions)
	const int old = max(0, min(n, (chunk ? b.rows[0].pos : width - 1) - p0)), old_pages = old / kPageTokens;
	const int8_t* kplane = pool.base + kv_plane_offset(d, pool, layer_index, kvh, 0);
	const int8_t* vplane = pool.base + kv_plane_offset(d, pool, layer_index, kvh, 1);
	{
		// entries beyond the slice's last page repeat it: their probabilities are zero, any V words will do
		const int32_t* pages = b.rows[r].pages + p0 / kPageTokens;
		for (int j = t; j < (n64 >> 4); j += kThreads) s.pbase[j] = (int64_t)pages[min(j, npages - 1)] * (kPageTokens * HD);
	}
	if (t < 3 * G) s.fold[t] = layer.f_ctx[3 * kvh * G + t];
	if (t < 8) {
		s.mx[t] = INT32_MIN;
		s.sum[t] = 0ull;
	}
	if (t == 8) s.misc[0] = 0u;
	const FunnelFold fold_ctx = funnel_prefold(nullptr, 0, layer.c_ctx);
	__syncthreads();
	auto stage_k = [&](int from, int to) {
		for (int i = from * (HD / 16) + t; i < to * (HD / 16); i += kThreads) {
			const int pos = i / (HD / 16), piece = i % (HD / 16);
			cp_async16(s.ks + (size_t)pos * S::kKStride + piece * 16, kplane + s.pbase[pos >> 4] + (pos & 15) * HD + piece * 16);
		}
	};
	auto stage_v = [&](int from, int to) {      // pages
		for (int i = from * HD + t; i < to * HD; i += kThreads) {
			const int pg = i / HD, piece = i % HD;
			cp_async16(s.vs + (size_t)pg * S::kVStride + piece * 16, vplane + s.pbase[pg] + piece * 16);
		}
	};
	if (STAGED) {
		stage_k(0, old);
		stage_v(0, SITE != kSiteApart ? npages : old_pages);      // (a new position's byte of the last page follows)
		// (pages between the slice's end and the next group of four are read against zero probabilities)
		for (int i = npages * HD + t; i < (n64 >> 4) * HD; i += kThreads)
			*(int4*)(s.vs + (size_t)(i / HD) * S::kVStride + (i % HD) * 16) = make_int4(0, 0, 0, 0);
	} else {
		constexpr int kRowsPerLine = 128 / HD;
		for (int pos = t * kRowsPerLine; pos < old; pos += kThreads * kRowsPerLine)
			prefetch_l2(kplane + s.pbase[pos >> 4] + (pos & 15) * HD);
	}
	// the q/k/v site, ahead of the projection: the normed row's scale, RoPE words, landing constants, biases
	using T = typename WideOf<W64>::T;
	using Y = typename WideOf<W64 || SITE == kSiteBias>::T;
	__shared__ uint32_t s_bank[SITE != kSiteApart ? 64 : 1];
	__shared__ __align__(16) uint32_t s_q[SITE != kSiteApart ? 2 * HD : 4];
	__shared__ unsigned long long s_biased[16];      // per block: its q elements' maximum, and bit 32: a K / V element without a sum
	__shared__ SoftmaxConsts s_consts;
	__shared__ int32_t s_failed;      // status word of a softmax constant's refusal
	const int H = d.hidden, KV = d.kv_hidden, pos = width - 1, slot = pos % kPageTokens;
	const bool has_q = t < G * (HD / 4), lands = pos >= p0 && pos < p0 + n && t < HD / 2;      // (threads take four elements of either)
	const bool is_k = t < HD / 4;
	const int dd = (4 * t) & (HD - 1);                // channel of both
	const int e_q = kvh * G * HD + 4 * t, e_kv = H + (is_k ? 0 : KV) + kvh * HD + dd;
	Scale ns{0, 0}, kh{0, 0};
	FunnelFold fold_q{};
	int2 rc = make_int2(0, 0), rs = make_int2(0, 0);
	int64_t r_t = 0, e_t = 0, r_a = 0, term_q[4], term_kv[4];
	int bexp = 0;
	bool gate = true;
	uint32_t bad_q = 0, bad_kv = 0;
	const int64_t *bias_q = nullptr, *bias_k = nullptr, *bias_v = nullptr;
	if constexpr (SITE != kSiteApart) {
		ns = b.ns[r];
		fold_q = funnel_prefold(&ns, 1, layer.c_q);
		const size_t at = (size_t)pos * (HD / 2) + (dd >> 1);
		if (has_q || lands) {
			rc = *(const int2*)(site.rope_cos + at);
			rs = *(const int2*)(site.rope_sin + at);
		}
		if (lands) {
			const int64_t* rec = (is_k ? layer.k_recip : layer.v_recip) + 3 * kvh;
			e_t = rec[1];
			r_t = rec[2];
		}
		if (warp == kWarps - 1 && lane < d.kv_heads) kh = Scale{layer.sm_khead[2 * lane], layer.sm_khead[2 * lane + 1]};
		if (t == 0) s_failed = 0;
	}
	if constexpr (SITE == kSiteBias) {
		bias_q = layer.b_q;
		bias_k = layer.b_k;
		bias_v = layer.b_v;
		r_a = dyn_recip(ns.m);
		gate = bias_exponent_in_domain(ns.e, &bexp);
		auto terms = [&](int e, bool in, int64_t (&out)[4], uint32_t& bad) {
			const int64_t* bp = e < H ? bias_q : (e < H + KV ? bias_k : bias_v);
			const int off = e < H ? e : (e < H + KV ? e - H : e - H - KV);
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				out[j] = 0;
				if (in && bp != nullptr && gate && !bias_term(bp[off + j], r_a, bexp, &out[j])) bad = 1;
			}
		};
		terms(e_q, has_q, term_q, bad_q);
		terms(e_kv, lands, term_kv, bad_kv);
	}
	cluster_arrive();
	cluster_wait();
	pdl_wait();
	pdl_release();
	bool live, ok = true;
	int32_t verdict = 0;      // (written behind the last exchange, when every block of the row has read the row's word)
	IExpFast fx;
	uint32_t qw[NW];
	if constexpr (SITE != kSiteApart) {
		const T* row = (const T*)b.wide + (size_t)r * b.wide_ld;
		T xq[4] = {0, 0, 0, 0}, xkv[4] = {0, 0, 0, 0};
		if (has_q) load_quad(row + e_q, xq);
		if (lands) load_quad(row + e_kv, xkv);
		unsigned long long mx = __ldcg(&b.rowmax[(size_t)r * 4]);
		const bool refused = __ldcg(&b.status[r]) != 0;
		Bank bank{s_bank, 0};
		Y yq[4], ykv[4];
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			yq[j] = xq[j];
			ykv[j] = xkv[j];
		}
		int32_t st = kOk;
		int at_site = kSiteQ;
		if constexpr (SITE == kSiteBias) {
			uint32_t top = 0;
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				int64_t sum;
				if (!bias_accumulate((int64_t)xq[j], term_q[j], &sum)) bad_q = 1;
				yq[j] = sum;
				const unsigned long long a = sum < 0 ? ~(unsigned long long)sum + 1ull : (unsigned long long)sum;
				top = max(top, a > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)a);      // (anything above 2^31 is refused alike)
				if (!bias_accumulate((int64_t)xkv[j], term_kv[j], &sum)) bad_kv = 1;
				ykv[j] = sum;
			}
			top = block_max_u32(bad_q != 0u ? 0xFFFFFFFFu : min(top, 0xFFFFFFFEu), bank);
			const bool bad = __syncthreads_or((int)bad_kv) != 0;
			if (t < (int)cluster_blocks) exchange_send(&s_biased[my_rank], bar(4), (uint32_t)t, (unsigned long long)top | (bad ? 1ull << 32 : 0ull));
			ok = exchange_wait(bar(4));
			uint32_t m = 0, any = 0;
			for (uint32_t j = 0; j < cluster_blocks; ++j) {
				m = max(m, (uint32_t)s_biased[j]);
				any |= (uint32_t)(s_biased[j] >> 32);
			}
			bad_kv = any;
			if (bias_q != nullptr) {
				mx = (unsigned long long)m;
				if (!gate) st = kRoundingDivideExponentOutOfDomain;
				else if (m == 0xFFFFFFFFu) st = kBiasReconcileProductOutOfDomain;
			}
		}
		const QuadFunnel fp = quad_funnel(mx, fold_q);
		if constexpr (SITE == kSiteBias) {
			if (st == kOk && (bad_kv != 0u || !gate) && (bias_k != nullptr || bias_v != nullptr) && fp.status == kOk) {
				st = gate ? kBiasReconcileProductOutOfDomain : kRoundingDivideExponentOutOfDomain;
				at_site = kSiteKv;
			}
		}
		if (st == kOk) st = fp.status;
		live = !refused && st == kOk;
		if (!refused) verdict = pack_status(st, at_site, b.layer);
		asm volatile("cp.async.wait_all;" ::: "memory");
		__syncthreads();      // the staged rows and pages are there
		if (live) {
			if (has_q) {
				const uint32_t w = rope_quad(code_quad(yq, fp), rc, rs);
				s_q[t] = w;
				if (split == 0) *(uint32_t*)(b.qrot + (size_t)r * H + e_q) = w;      // (traces read it)
			}
			if (lands) {
				const Lander l = make_lander(ns.m, r_t, ns.e, e_t);
				uint32_t sat = 0;
				int lc[4];
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					const int64_t a = (int64_t)ykv[j];
					const unsigned long long mag = a < 0 ? ~(unsigned long long)a + 1ull : (unsigned long long)a;
					bool s1;
					if (l.fast && mag <= (1ull << 31)) {
						const uint64_t m = land_magnitude((uint32_t)mag, l);
						s1 = m > 127;
						const int c = s1 ? 127 : (int)m;
						lc[j] = ((a < 0) != l.neg) ? -c : c;
					} else {
						lc[j] = (int)clamp127(landing_rescale(a, ns.m, r_t, ns.e, e_t, &s1, nullptr));
					}
					sat += s1 ? 1u : 0u;
				}
				const int64_t page = s.pbase[(pos - p0) >> 4];      // (byte offset)
				if (is_k) {
					const uint32_t w = rope_quad(pack4(lc[0], lc[1], lc[2], lc[3]), rc, rs);
					*(uint32_t*)(s.ks + (size_t)(pos - p0) * S::kKStride + dd) = w;
					*(uint32_t*)(const_cast<int8_t*>(kplane) + page + slot * HD + dd) = w;
				} else {
#pragma unroll
					for (int j = 0; j < 4; ++j) {
						s.vs[(size_t)((pos - p0) >> 4) * S::kVStride + (dd + j) * kPageTokens + slot] = (int8_t)lc[j];
						const_cast<int8_t*>(vplane)[page + (dd + j) * kPageTokens + slot] = (int8_t)lc[j];
					}
				}
				if (sat != 0u) {
					atomicAdd(&b.sat[r], (unsigned long long)sat);
					if (layer_index < b.sat_ld) atomicAdd(&b.sat_layer[(size_t)r * b.sat_ld + layer_index], sat);
				}
			}
			if (warp == kWarps - 1) {
				// softmax constants per kv head, as in k_qkv_post; any head's refusal is the row's
				int32_t cst = kOk;
				if (lane < d.kv_heads) {
					SoftmaxConsts sc;
					cst = softmax_consts(fp.out, kh, (uint64_t)pos + 1, &sc);
					if (lane == kvh) s_consts = sc;
				}
				const uint32_t failing = __ballot_sync(0xffffffffu, cst != kOk);
				if (failing != 0u && lane == __ffs(failing) - 1) s_failed = pack_status(cst, kSiteSoftmaxConsts, b.layer);
			}
		}
		__syncthreads();
		if (live && s_failed != 0) {
			verdict = s_failed;
			live = false;
		}
		fx = iexp_fast_prepare(s_consts);
		shared_row_words<HD>((const int8_t*)s_q + min(g, G - 1) * HD, c, qw);
	} else {
	// A row that an earlier site refused is sat out: zero contributions, but every exchange. (Only this
	// kernel's last step can refuse the row, when every block has long read the word.)
	live = __ldcg(&b.status[r]) == 0;
	fx = iexp_fast_prepare(b.smc[(size_t)r * d.kv_heads + kvh]);
	load_row_words<HD>(b.qrot + (size_t)r * d.hidden + (size_t)(kvh * G + min(g, G - 1)) * HD, c, qw);
	if (STAGED) {
		stage_k(old, n);
		stage_v(old_pages, npages);
		asm volatile("cp.async.wait_all;" ::: "memory");
		__syncthreads();
	}
	}

	// ---- stage 1: scores, 8 positions per MMA group, groups dealt round-robin to the warps; lanes beyond
	// the slice's end read its last position again, their columns are stored as INT32_MIN
	if (live && n > 0) {
		const int nblk = (n + 7) >> 3;
		constexpr int U = 4;
		int rmax = INT32_MIN;
#pragma unroll 1
		for (int blk0 = warp * U; blk0 < nblk; blk0 += kWarps * U) {
			uint32_t kw[U][NW];
#pragma unroll
			for (int u = 0; u < U; ++u) {
				const int pos = min((blk0 + u) * 8 + g, n - 1);
				if (STAGED) shared_row_words<HD>(s.ks + (size_t)pos * S::kKStride, c, kw[u]);
				else load_row_words<HD>(kplane + s.pbase[pos >> 4] + (pos & 15) * HD, c, kw[u]);
			}
#pragma unroll
			for (int u = 0; u < U; ++u) {
				int acc[4] = {0, 0, 0, 0};
#pragma unroll
				for (int j = 0; j < NW / 2; ++j) mma_s8s8(acc, qw[2 * j], qw[2 * j + 1], kw[u][2 * j], kw[u][2 * j + 1]);
				const int k = (blk0 + u) * 8 + c * 2;
				if (g < G && blk0 + u < nblk) {
					const int v0 = k < n ? acc[0] : INT32_MIN, v1 = k + 1 < n ? acc[1] : INT32_MIN;
					*(int2*)&s.sc[(size_t)g * cp + k] = make_int2(v0, v1);
					rmax = max(rmax, max(v0, v1));
				}
			}
		}
		rmax = max(rmax, __shfl_xor_sync(0xffffffffu, rmax, 1));
		rmax = max(rmax, __shfl_xor_sync(0xffffffffu, rmax, 2));
		if (c == 0 && g < G && rmax != INT32_MIN) atomicMax(&s.mx[g], rmax);
	}
	if (!STAGED && live)      // the softmax below moves no data: ask for this slice's V pages meanwhile
		for (int ln = t; ln < npages * (kPageTokens * HD / 128); ln += kThreads)
			prefetch_l2(vplane + s.pbase[ln / (kPageTokens * HD / 128)] + (ln % (kPageTokens * HD / 128)) * 128);
	__syncthreads();
	// ---- exchange 1: every slice's maxima
	for (int i = t; i < splits * G; i += kThreads) exchange_send(&s.rx_max[split * 8 + i % G], bar(0), kv_rank0 + (uint32_t)(i / G), (uint32_t)s.mx[i % G]);
	ok = exchange_wait(bar(0)) && ok;

	// ---- stage 2: softmax, (head, 128-position chunk) pairs dealt to the warps, a lane takes 4 consecutive
	// positions: exponentials and their sums, the score's place then holds the element's (shift, remainder)
	const int nchunk = (n64 + 127) >> 7;
	if (live) {
#pragma unroll 1
		for (int task = warp; task < G * nchunk; task += kWarps) {
			const int h = task / nchunk, k4 = (task - h * nchunk) * 128 + lane * 4;
			unsigned long long tot = 0;
			if (k4 < n) {
				int m = s.rx_max[h];
				for (int j = 1; j < splits; ++j) m = max(m, s.rx_max[j * 8 + h]);
				int32_t* row = s.sc + (size_t)h * cp;
				const int4 v = *(const int4*)&row[k4];
				uint32_t q0, q1, q2, q3;
				const int64_t e0 = chunk_exp((uint32_t)m - (uint32_t)v.x, fx, &q0);
				int64_t e1 = chunk_exp((uint32_t)m - (uint32_t)v.y, fx, &q1);
				int64_t e2 = chunk_exp((uint32_t)m - (uint32_t)v.z, fx, &q2);
				int64_t e3 = chunk_exp((uint32_t)m - (uint32_t)v.w, fx, &q3);
				if (k4 + 3 >= n) {       // the slice's last group: positions beyond its end count for nothing
					if (k4 + 1 >= n) { e1 = 0; q1 = kBaseOfZero; }
					if (k4 + 2 >= n) { e2 = 0; q2 = kBaseOfZero; }
					e3 = 0; q3 = kBaseOfZero;
				}
				tot = (unsigned long long)(e0 + e1) + (unsigned long long)(e2 + e3);
				*(int4*)&row[k4] = make_int4((int)q0, (int)q1, (int)q2, (int)q3);
			}
			// a lane's partial is below 2^50: three 24-bit limbs add up across the warp inside 32 bits
			const uint32_t l0 = __reduce_add_sync(0xffffffffu, (uint32_t)tot & 0xFFFFFFu);
			const uint32_t l1 = __reduce_add_sync(0xffffffffu, (uint32_t)(tot >> 24) & 0xFFFFFFu);
			const uint32_t l2 = __reduce_add_sync(0xffffffffu, (uint32_t)(tot >> 48));
			if (lane == 0) atomicAdd(&s.sum[h], (unsigned long long)l0 + ((unsigned long long)l1 << 24) + ((unsigned long long)l2 << 48));
		}
	}
	__syncthreads();
	// ---- exchange 2: every slice's sums
	for (int i = t; i < splits * G; i += kThreads) exchange_send(&s.rx_sum[split * 8 + i % G], bar(1), kv_rank0 + (uint32_t)(i / G), s.sum[i % G]);
	ok = exchange_wait(bar(1)) && ok;
	// probabilities as two u8 planes, zero beyond the slice up to the next multiple of 64
	if (live) {
		const int n4 = (n + 3) & ~3;
#pragma unroll 1
		for (int task = warp; task < G * nchunk; task += kWarps) {
			const int h = task / nchunk, k4 = (task - h * nchunk) * 128 + lane * 4;
			if (k4 < n4) {
				unsigned long long total = s.rx_sum[h];
				for (int j = 1; j < splits; ++j) total += s.rx_sum[j * 8 + h];
				const ChunkProb pr = chunk_prob(total, fx);
				const int4 v = *(const int4*)&s.sc[(size_t)h * cp + k4];
				float near = 1.0f;
				uint32_t q0 = chunk_prob_of((uint32_t)v.x, pr, &near), q1 = chunk_prob_of((uint32_t)v.y, pr, &near);
				uint32_t q2 = chunk_prob_of((uint32_t)v.z, pr, &near), q3 = chunk_prob_of((uint32_t)v.w, pr, &near);
				if (near < pr.eps) {
					const uint4 x = chunk_prob_exact((uint32_t)v.x, (uint32_t)v.y, (uint32_t)v.z, (uint32_t)v.w, fx.qc, total);
					q0 = x.x; q1 = x.y; q2 = x.z; q3 = x.w;
				}
				*(uint32_t*)&s.pl[(size_t)h * cp + k4] = pack_plane(q0, q1, q2, q3, 0);
				*(uint32_t*)&s.ph[(size_t)h * cp + k4] = pack_plane(q0, q1, q2, q3, 1);
			} else if (k4 < n64) {
				*(uint32_t*)&s.pl[(size_t)h * cp + k4] = 0u;
				*(uint32_t*)&s.ph[(size_t)h * cp + k4] = 0u;
			}
		}
	}
	__syncthreads();

	// ---- stage 3: the slice's share of ctx = P V. Lane column c owns page 4 grp + c of each 64-position
	// group; its 16-byte row of the transposed page feeds two MMAs
	constexpr int NDB = 2;            // 8-channel blocks per warp
	int accl[NDB][4], acch[NDB][4];
#pragma unroll
	for (int i = 0; i < NDB; ++i)
#pragma unroll
		for (int j = 0; j < 4; ++j) accl[i][j] = acch[i][j] = 0;
	if (live) {
		const int ngrp = n64 >> 6;
		const uint8_t* pl = s.pl + (size_t)(g < G ? g : 0) * cp + c * kPageTokens;
		const uint8_t* ph = s.ph + (size_t)(g < G ? g : 0) * cp + c * kPageTokens;
		const int chan = (warp * NDB * 8 + g) * kPageTokens;
#pragma unroll 4
		for (int grp = 0; grp < ngrp; ++grp) {
			const int4 al = *(const int4*)(pl + grp * 64), ah = *(const int4*)(ph + grp * 64);
			const int8_t* vp = STAGED ? s.vs + (size_t)(grp * 4 + c) * S::kVStride + chan : vplane + s.pbase[grp * 4 + c] + chan;
#pragma unroll
			for (int i = 0; i < NDB; ++i) {
				const int4 v = *(const int4*)(vp + i * 8 * kPageTokens);
				mma_u8s8(accl[i], (uint32_t)al.x, (uint32_t)al.y, (uint32_t)v.x, (uint32_t)v.y);
				mma_u8s8(accl[i], (uint32_t)al.z, (uint32_t)al.w, (uint32_t)v.z, (uint32_t)v.w);
				mma_u8s8(acch[i], (uint32_t)ah.x, (uint32_t)ah.y, (uint32_t)v.x, (uint32_t)v.y);
				mma_u8s8(acch[i], (uint32_t)ah.z, (uint32_t)ah.w, (uint32_t)v.z, (uint32_t)v.w);
			}
		}
	}
	// ---- exchange 3: each share goes to the slice that reduces its channels
	if (g < G) {
#pragma unroll
		for (int i = 0; i < NDB; ++i) {
			const int ch = (warp * NDB + i) * 8 + c * 2;
			exchange_send(&s.rx_ctx[(split * G + g) * per + ch % per], bar(2), kv_rank0 + (uint32_t)(ch / per),
			              make_int2(accl[i][0] + 256 * acch[i][0], accl[i][1] + 256 * acch[i][1]));
		}
	}
	ok = exchange_wait(bar(2)) && ok;
	// add the shares, per-head context fold (forward_sites.cpp:1889-1896), row maximum
	uint32_t top = 0;
	constexpr int kMaxMine = 4;                                   // G * per <= 8 HD = 4 threads' worth
	int32_t mine[kMaxMine];
#pragma unroll
	for (int q = 0; q < kMaxMine; ++q) {
		mine[q] = 0;
		const int e = q * kThreads + t;
		if (e < G * per) {
			const int h = e / per, ch = ch0 + e - h * per;
			int32_t sum = 0;
			for (int j = 0; j < splits; ++j) sum += s.rx_ctx[j * G * per + e];
			const int32_t o = fold(sum, s.fold[3 * h], s.fold[3 * h + 1], s.fold[3 * h + 2]);
			mine[q] = o;
			top = max(top, o < 0 ? 0u - (uint32_t)o : (uint32_t)o);
			if (!whole_row && live) b.ctxw[(size_t)r * d.hidden + (size_t)(kvh * G + h) * HD + ch] = o;
		}
	}
	top = __reduce_max_sync(0xffffffffu, top);
	// (every thread has its own limit, so every thread whose wait ran out speaks for the row)
	auto give_up = [&](int exchanges) {
		if (!ok) atomicCAS(&b.status[r], 0, pack_status(kInternalWaitTimeout, kSiteCtx, b.layer));
		__syncwarp();
		exchange_leave(bar(0), exchanges);
	};
	if (!whole_row) {
		if (lane == 0 && top && live) atomicMax(&b.rowmax[(size_t)r * 4 + 3], (unsigned long long)top);
		if (__builtin_expect(!__all_sync(0xffffffffu, ok), 0)) give_up(3);
		return;
	}
	// ---- exchange 4: the cluster holds the whole row, its funnel runs here
	if (lane == 0 && top) atomicMax(&s.misc[0], top);
	__syncthreads();
	if (t < (int)cluster_blocks) exchange_send(&s.rx_top[my_rank], bar(3), (uint32_t)t, s.misc[0]);
	ok = exchange_wait(bar(3)) && ok;
	if (__builtin_expect(!__all_sync(0xffffffffu, ok), 0)) {
		give_up(SITE == kSiteBias ? 5 : 4);
		return;
	}
	if (SITE != kSiteApart && my_rank == 0 && t == 0) {      // (every block has read them)
		b.rowmax[(size_t)r * 4] = 0ull;
		if (verdict != 0) atomicCAS(&b.status[r], 0, verdict);
	}
	if (!live) return;
	for (uint32_t j = 0; j < cluster_blocks; ++j) top = max(top, s.rx_top[j]);
	const QuadFunnel fp = quad_funnel((unsigned long long)top, fold_ctx);
	if (fp.status != kOk) {
		if (my_rank == 0 && t == 0) atomicCAS(&b.status[r], 0, pack_status(fp.status, kSiteCtx, b.layer));
		return;
	}
	const uint32_t codes = code_quad(mine, fp);
#pragma unroll
	for (int q = 0; q < kMaxMine; ++q) {
		const int e = q * kThreads + t;
		if (e < G * per) {
			const int h = e / per, ch = ch0 + e - h * per;
			b.ctx[(size_t)r * d.hidden + (size_t)(kvh * G + h) * HD + ch] = (int8_t)byte_of(codes, q);
		}
	}
	if (my_rank == 0 && t == 0) b.cs[r] = fp.out;
}

// ------------------------------------------------------------ prefill: query-tiled attention
// The rows of a prefill chunk are consecutive positions of ONE sequence, so neighbouring tokens
// read almost the same K / V prefix. A block takes a tile of TQ consecutive tokens of one kv head
// -- TQ * G = up to 64 query rows (token, q head), four 16-row MMA blocks -- and walks the prefix
// in steps of 64 positions staged in shared memory (cp.async, double buffered): every K / V byte
// is fetched once per tile instead of once per token. The exact integer softmax needs the row
// maximum before any exponential and the row total before any probability, so the prefix is
// walked three times: (1) scores -> row maxima, (2) scores -> exponentials -> row totals,
// (3) scores -> probabilities -> P.V. Scores are recomputed each time (tensor-core work, cheap
// beside the integer softmax); nothing of size rows x width is ever stored. The causal limit is
// per row: token i of the tile sees positions <= pos0 + i.
// Warp w works on MMA block w / 2 (16 query rows) and on half w % 2 of each 64-position step
// (scores) respectively half w % 2 of the channels (P.V).
constexpr int kTileRows = 64;
constexpr int kTileKeys = 64;
constexpr int kTileThreads = 256;
constexpr int kTilePStride = 80;      // bytes per row of the probability planes (64 + padding against bank conflicts)

__device__ __forceinline__ void mma_s8s8_full(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                              uint32_t b1) {
	asm volatile(
	    "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
	    : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
	    : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_u8s8_full(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                              uint32_t b1) {
	asm volatile(
	    "mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
	    : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
	    : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int HD>
struct TileSmem {
	static constexpr int kKStride = HD + 16;                       // bytes per staged K row (padding against bank conflicts)
	static constexpr size_t kK = (size_t)2 * kTileKeys * kKStride;
	static constexpr size_t kV = (size_t)2 * kTileKeys * HD;
	static constexpr size_t kP = (size_t)2 * kTileRows * kTilePStride;
	static constexpr size_t kFx = (size_t)kTileRows * sizeof(IExpFast);
	static constexpr size_t kMisc = (size_t)kTileRows * (4 + 2 * 4 + 2 * 8) + 8 * 3 * 4 + 64;
	static constexpr size_t kBytes = kK + kV + kP + kFx + kMisc;
};

template <int HD>
__global__ void __launch_bounds__(kTileThreads, 2)
k_attention_tile(RowBatch b, Dims d, const __grid_constant__ LayerDev layer, int layer_index, KvPoolDev pool, int tq) {
	using L = TileSmem<HD>;
	constexpr int KS = HD / 32;          // MMA steps along the head dimension
	constexpr int NGW = HD / 16;         // 8-channel groups a warp owns in P.V
	extern __shared__ __align__(16) unsigned char smem[];
	int8_t* Ks = (int8_t*)smem;
	int8_t* Vs = (int8_t*)(smem + L::kK);
	uint8_t* Pl = (uint8_t*)(smem + L::kK + L::kV);
	uint8_t* Ph = Pl + (size_t)kTileRows * kTilePStride;
	IExpFast* fxs = (IExpFast*)(smem + L::kK + L::kV + L::kP);
	unsigned long long* wsum = (unsigned long long*)(fxs + kTileRows);      // [2][64]
	int32_t* wmax = (int32_t*)(wsum + 2 * kTileRows);                        // [2][64]
	int32_t* tok_ok = wmax + 2 * kTileRows;                                  // [64] 1: the token takes part
	int32_t* l_fold = tok_ok + kTileRows;                                    // [8][3]

	const int kvh = blockIdx.x;
	const int tile = (int)gridDim.y - 1 - (int)blockIdx.y;      // the last (widest) tiles start first
	const int G = d.heads / d.kv_heads;
	const int r0 = tile * tq, nt = min(tq, b.m - r0);
	const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, c = lane & 3;
	const int mb = warp >> 1, ph = warp & 1;
	// this lane's two query rows (token, head)
	const int rho_a = mb * 16 + g, rho_b = rho_a + 8;
	const int tok_a = rho_a / G, tok_b = rho_b / G;
	const int head_a = rho_a - tok_a * G, head_b = rho_b - tok_b * G;
	// uploaded before the step's first launch: the tile's first position and the sequence's page table
	const int pos0 = b.rows[r0].pos;
	const int32_t* pages = b.rows[r0].pages;
	const int width = pos0 + nt;
	const int nblk = (width + kTileKeys - 1) / kTileKeys;
	const int8_t* kplane = pool.base + kv_plane_offset(d, pool, layer_index, kvh, 0);
	const int8_t* vplane = pool.base + kv_plane_offset(d, pool, layer_index, kvh, 1);
	if (t < 3 * G) l_fold[t] = layer.f_ctx[3 * kvh * G + t];
	pdl_wait();
	pdl_release();
	if (t < kTileRows) {
		int okv = 0;
		if (t < nt) {
			okv = __ldcg(&b.status[r0 + t]) == 0 ? 1 : 0;
			fxs[t] = iexp_fast_prepare(b.smc[(size_t)(r0 + t) * d.kv_heads + kvh]);
		}
		tok_ok[t] = okv;
	}
	__syncthreads();
	const bool in_a = tok_a < nt && tok_ok[tok_a] != 0, in_b = tok_b < nt && tok_ok[tok_b] != 0;
	const int lim_a = in_a ? pos0 + tok_a : -1, lim_b = in_b ? pos0 + tok_b : -1;    // last position each row sees
	// q fragments (A operand) of this warp's MMA block, kept in registers for all three walks
	uint32_t qa[KS][4];
	{
		const int8_t* qpa = b.qrot + (size_t)(r0 + (in_a ? tok_a : 0)) * d.hidden + (size_t)(kvh * G + head_a) * HD;
		const int8_t* qpb = b.qrot + (size_t)(r0 + (in_b ? tok_b : 0)) * d.hidden + (size_t)(kvh * G + head_b) * HD;
#pragma unroll
		for (int ks = 0; ks < KS; ++ks) {
			qa[ks][0] = in_a ? *(const uint32_t*)(qpa + 32 * ks + 4 * c) : 0u;
			qa[ks][1] = in_b ? *(const uint32_t*)(qpb + 32 * ks + 4 * c) : 0u;
			qa[ks][2] = in_a ? *(const uint32_t*)(qpa + 32 * ks + 16 + 4 * c) : 0u;
			qa[ks][3] = in_b ? *(const uint32_t*)(qpb + 32 * ks + 16 + 4 * c) : 0u;
		}
	}
	const IExpFast fa = fxs[in_a ? tok_a : 0], fb = fxs[in_b ? tok_b : 0];

	// stage step `blk` of the prefix: K rows (and V pages) of positions blk * 64 ...; positions
	// beyond the tile's width are left as they are (their scores are masked, their probabilities zero)
	auto load_block = [&](int stage, int blk, bool with_v) {
		int8_t* kd = Ks + (size_t)stage * kTileKeys * L::kKStride;
		for (int idx = t; idx < kTileKeys * (HD / 16); idx += kTileThreads) {
			const int row = idx / (HD / 16), piece = idx - row * (HD / 16);
			const int pos = blk * kTileKeys + row;
			if (pos < width)
				cp_async16(kd + (size_t)row * L::kKStride + piece * 16,
				           kplane + (int64_t)pages[pos >> 4] * (kPageTokens * HD) + (pos & 15) * HD + piece * 16);
		}
		if (with_v) {
			int8_t* vd = Vs + (size_t)stage * kTileKeys * HD;
			for (int idx = t; idx < 4 * HD; idx += kTileThreads) {
				const int pg = idx / HD, piece = idx - pg * HD;
				const int page = blk * 4 + pg;
				if (page * kPageTokens < width)
					cp_async16(vd + (size_t)pg * HD * kPageTokens + piece * 16,
					           vplane + (int64_t)pages[page] * (kPageTokens * HD) + piece * 16);
			}
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	// scores of this warp's 16 rows x 32 positions of the staged step
	auto scores = [&](int stage, int (&acc)[4][4]) {
		const int8_t* kd = Ks + (size_t)stage * kTileKeys * L::kKStride;
#pragma unroll
		for (int j = 0; j < 4; ++j) {
#pragma unroll
			for (int q = 0; q < 4; ++q) acc[j][q] = 0;
			const int8_t* krow = kd + (size_t)(32 * ph + 8 * j + g) * L::kKStride;
#pragma unroll
			for (int ks = 0; ks < KS; ++ks) {
				const uint32_t b0 = *(const uint32_t*)(krow + 32 * ks + 4 * c);
				const uint32_t b1 = *(const uint32_t*)(krow + 32 * ks + 16 + 4 * c);
				mma_s8s8_full(acc[j], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b0, b1);
			}
		}
	};
	// walk the prefix: `body(stage, blk)` runs with step blk staged; the next step loads meanwhile
	auto walk = [&](bool with_v, auto&& body) {
		load_block(0, 0, with_v);
		for (int blk = 0; blk < nblk; ++blk) {
			const int stage = blk & 1;
			if (blk + 1 < nblk) {
				load_block(stage ^ 1, blk + 1, with_v);
				asm volatile("cp.async.wait_group 1;" ::: "memory");
			} else {
				asm volatile("cp.async.wait_group 0;" ::: "memory");
			}
			__syncthreads();
			body(stage, blk);
			__syncthreads();      // the stage (and the probability planes) may be overwritten
		}
	};

	// ---- walk 1: row maxima
	int mx_a = INT32_MIN, mx_b = INT32_MIN;
	walk(false, [&](int stage, int blk) {
		int acc[4][4];
		scores(stage, acc);
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			const int k0 = blk * kTileKeys + 32 * ph + 8 * j + 2 * c;
			if (k0 <= lim_a) mx_a = max(mx_a, acc[j][0]);
			if (k0 + 1 <= lim_a) mx_a = max(mx_a, acc[j][1]);
			if (k0 <= lim_b) mx_b = max(mx_b, acc[j][2]);
			if (k0 + 1 <= lim_b) mx_b = max(mx_b, acc[j][3]);
		}
	});
	mx_a = max(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 1));
	mx_a = max(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 2));
	mx_b = max(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 1));
	mx_b = max(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 2));
	if (c == 0) {
		wmax[ph * kTileRows + rho_a] = mx_a;
		wmax[ph * kTileRows + rho_b] = mx_b;
	}
	__syncthreads();
	mx_a = max(wmax[rho_a], wmax[kTileRows + rho_a]);
	mx_b = max(wmax[rho_b], wmax[kTileRows + rho_b]);

	// ---- walk 2: exponentials and row totals (elements beyond a row's causal limit are computed
	// and dropped by a select: no branch in the element code)
	unsigned long long sum_a = 0, sum_b = 0;
	walk(false, [&](int stage, int blk) {
		int acc[4][4];
		scores(stage, acc);
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			const int k0 = blk * kTileKeys + 32 * ph + 8 * j + 2 * c;
#pragma unroll
			for (int q = 0; q < 2; ++q) {
				const int64_t ea = iexp_fast((uint32_t)mx_a - (uint32_t)acc[j][q], fa);
				const int64_t eb = iexp_fast((uint32_t)mx_b - (uint32_t)acc[j][2 + q], fb);
				sum_a += k0 + q <= lim_a ? (unsigned long long)ea : 0ull;
				sum_b += k0 + q <= lim_b ? (unsigned long long)eb : 0ull;
			}
		}
	});
	sum_a += __shfl_xor_sync(0xffffffffu, sum_a, 1);
	sum_a += __shfl_xor_sync(0xffffffffu, sum_a, 2);
	sum_b += __shfl_xor_sync(0xffffffffu, sum_b, 1);
	sum_b += __shfl_xor_sync(0xffffffffu, sum_b, 2);
	if (c == 0) {
		wsum[ph * kTileRows + rho_a] = sum_a;
		wsum[ph * kTileRows + rho_b] = sum_b;
	}
	__syncthreads();
	sum_a = wsum[rho_a] + wsum[kTileRows + rho_a];
	sum_b = wsum[rho_b] + wsum[kTileRows + rho_b];
	const ProbRow pr_a = prob_row(sum_a), pr_b = prob_row(sum_b);
	const bool go_a = in_a, go_b = in_b;

	// ---- walk 3: probabilities and P.V
	int accl[NGW][4], acch[NGW][4];
#pragma unroll
	for (int i = 0; i < NGW; ++i)
#pragma unroll
		for (int q = 0; q < 4; ++q) accl[i][q] = acch[i][q] = 0;
	walk(true, [&](int stage, int blk) {
		int acc[4][4];
		scores(stage, acc);
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			const int col = 32 * ph + 8 * j + 2 * c;
			const int k0 = blk * kTileKeys + col;
			uint32_t pa[2], pb[2];
			int64_t ea[2], eb[2];
			bool unsure = false;
#pragma unroll
			for (int q = 0; q < 2; ++q) {
				ea[q] = iexp_fast((uint32_t)mx_a - (uint32_t)acc[j][q], fa);
				eb[q] = iexp_fast((uint32_t)mx_b - (uint32_t)acc[j][2 + q], fb);
				// (an element beyond its row's limit may exceed the row's total: it is dropped below, whatever it gives)
				pa[q] = prob_fast(ea[q], pr_a, &unsure);
				pb[q] = prob_fast(eb[q], pr_b, &unsure);
			}
			if (unsure) {
				const uint2 xa = prob_pair_exact(ea[0], ea[1], pr_a.tot), xb = prob_pair_exact(eb[0], eb[1], pr_b.tot);
				pa[0] = xa.x; pa[1] = xa.y; pb[0] = xb.x; pb[1] = xb.y;
			}
#pragma unroll
			for (int q = 0; q < 2; ++q) {
				pa[q] = k0 + q <= lim_a ? pa[q] & 0xFFFFu : 0u;
				pb[q] = k0 + q <= lim_b ? pb[q] & 0xFFFFu : 0u;
			}
			*(uint16_t*)(Pl + (size_t)rho_a * kTilePStride + col) = (uint16_t)((pa[0] & 0xffu) | ((pa[1] & 0xffu) << 8));
			*(uint16_t*)(Ph + (size_t)rho_a * kTilePStride + col) = (uint16_t)((pa[0] >> 8) | ((pa[1] >> 8) << 8));
			*(uint16_t*)(Pl + (size_t)rho_b * kTilePStride + col) = (uint16_t)((pb[0] & 0xffu) | ((pb[1] & 0xffu) << 8));
			*(uint16_t*)(Ph + (size_t)rho_b * kTilePStride + col) = (uint16_t)((pb[0] >> 8) | ((pb[1] >> 8) << 8));
		}
		// the two warps of an MMA block wrote its rows' 64 probabilities between them
		asm volatile("bar.sync %0, 64;" ::"r"(1 + mb) : "memory");
		const int8_t* vd = Vs + (size_t)stage * kTileKeys * HD;
#pragma unroll
		for (int ks = 0; ks < 2; ++ks) {
			const uint8_t* la = Pl + (size_t)rho_a * kTilePStride + 32 * ks + 4 * c;
			const uint8_t* lb = Pl + (size_t)rho_b * kTilePStride + 32 * ks + 4 * c;
			const uint8_t* ha = Ph + (size_t)rho_a * kTilePStride + 32 * ks + 4 * c;
			const uint8_t* hb = Ph + (size_t)rho_b * kTilePStride + 32 * ks + 4 * c;
			const uint32_t l0 = *(const uint32_t*)la, l1 = *(const uint32_t*)lb, l2 = *(const uint32_t*)(la + 16), l3 = *(const uint32_t*)(lb + 16);
			const uint32_t h0 = *(const uint32_t*)ha, h1 = *(const uint32_t*)hb, h2 = *(const uint32_t*)(ha + 16), h3 = *(const uint32_t*)(hb + 16);
#pragma unroll
			for (int i = 0; i < NGW; ++i) {
				const int ch = 8 * (ph * NGW + i) + g;
				const uint32_t b0 = *(const uint32_t*)(vd + (size_t)(2 * ks) * HD * kPageTokens + ch * kPageTokens + 4 * c);
				const uint32_t b1 = *(const uint32_t*)(vd + (size_t)(2 * ks + 1) * HD * kPageTokens + ch * kPageTokens + 4 * c);
				mma_u8s8_full(accl[i], l0, l1, l2, l3, b0, b1);
				mma_u8s8_full(acch[i], h0, h1, h2, h3, b0, b1);
			}
		}
	});

	// ---- per-head context fold (forward_sites.cpp:1889-1896), store, row maximum for the funnel
	uint32_t lm_a = 0, lm_b = 0;
#pragma unroll
	for (int i = 0; i < NGW; ++i) {
		const int ch = 8 * (ph * NGW + i) + 2 * c;
		if (go_a) {
			int2 o;
			o.x = fold(accl[i][0] + 256 * acch[i][0], l_fold[3 * head_a], l_fold[3 * head_a + 1], l_fold[3 * head_a + 2]);
			o.y = fold(accl[i][1] + 256 * acch[i][1], l_fold[3 * head_a], l_fold[3 * head_a + 1], l_fold[3 * head_a + 2]);
			*(int2*)(b.ctxw + (size_t)(r0 + tok_a) * d.hidden + (size_t)(kvh * G + head_a) * HD + ch) = o;
			lm_a = max(lm_a, max(o.x < 0 ? 0u - (uint32_t)o.x : (uint32_t)o.x, o.y < 0 ? 0u - (uint32_t)o.y : (uint32_t)o.y));
		}
		if (go_b) {
			int2 o;
			o.x = fold(accl[i][2] + 256 * acch[i][2], l_fold[3 * head_b], l_fold[3 * head_b + 1], l_fold[3 * head_b + 2]);
			o.y = fold(accl[i][3] + 256 * acch[i][3], l_fold[3 * head_b], l_fold[3 * head_b + 1], l_fold[3 * head_b + 2]);
			*(int2*)(b.ctxw + (size_t)(r0 + tok_b) * d.hidden + (size_t)(kvh * G + head_b) * HD + ch) = o;
			lm_b = max(lm_b, max(o.x < 0 ? 0u - (uint32_t)o.x : (uint32_t)o.x, o.y < 0 ? 0u - (uint32_t)o.y : (uint32_t)o.y));
		}
	}
	lm_a = max(lm_a, __shfl_xor_sync(0xffffffffu, lm_a, 1));
	lm_a = max(lm_a, __shfl_xor_sync(0xffffffffu, lm_a, 2));
	lm_b = max(lm_b, __shfl_xor_sync(0xffffffffu, lm_b, 1));
	lm_b = max(lm_b, __shfl_xor_sync(0xffffffffu, lm_b, 2));
	if (c == 0) {
		if (go_a && lm_a) atomicMax(&b.rowmax[(size_t)(r0 + tok_a) * 4 + 3], (unsigned long long)lm_a);
		if (go_b && lm_b) atomicMax(&b.rowmax[(size_t)(r0 + tok_b) * 4 + 3], (unsigned long long)lm_b);
	}
}

template <int HD>
static cudaError_t launch_attn_tile(const RowBatch& b, const Dims& d, const LayerDev& layer, int layer_index, KvPoolDev pool,
                                    cudaStream_t st) {
	const int G = d.heads / d.kv_heads;
	const int tq = kTileRows / G;
	return launch_pdl(k_attention_tile<HD>, dim3(d.kv_heads, (b.m + tq - 1) / tq), dim3(kTileThreads), TileSmem<HD>::kBytes, st, b,
	                  d, layer, layer_index, pool, tq);
}

// ------------------------------------------------------------ prefill chunks
// The rows of a prefill chunk are consecutive positions of ONE sequence, so neighbouring tokens read
// almost the same K / V prefix. A block takes 32 query rows -- tq consecutive tokens times the q heads of
// one kv head, two 16-row MMA blocks -- and up to 512 positions of their prefix in steps of 128. The exact
// integer softmax needs the row maximum before any exponential and the row total before any probability;
// a block keeps its scores in shared memory, every thread its own elements, so K is multiplied once, V
// once, and the softmax passes touch no other thread's data:
//   1  scores of a step on the tensor cores, masked by each row's causal limit; row maxima
//   2  exponentials and row totals; a score's place then holds the element's (shift, base)
//   3  probabilities, packed in place as the A fragments of P.V (two u8 planes)
//   4  P.V on the tensor cores, a warp per quarter of the channels, context fold
// The K rows of a 16-position group are read in an order (0 1 4 5 8 9 12 13 | 2 3 6 7 10 11 14 15) that
// leaves a lane of the score MMAs with four neighbouring positions, which is what a lane of the P.V MMAs
// holds: probabilities go from one to the other as whole words.
// A tile whose prefix is longer is split over the blocks of a cluster (step s goes to block s mod `sub`),
// which exchange maxima, totals and shares of P.V. Clusters have one size per launch: one takes a single
// wide tile, or two of half the width, or four ... (ChunkPlan). The widest tiles start first.
//
// Bound by the integer instructions of the softmax. One layer, before: the prefix walked three times with
// recomputed scores, 64 rows per block, 186 us for 2,047 positions at the 1.5B widths; one block per row,
// 21 us for 512 positions at the 0.5B widths.
constexpr int kChunkRows = 32, kChunkStep = 128, kChunkThreads = 256, kChunkSteps = 4;
struct ChunkPlan {
	int tq;            // tokens per tile
	int steps;         // steps of 128 positions a block holds at most
	int cluster;       // blocks per cluster, a power of two
	int count[4];      // tiles split `cluster`, cluster / 2, cluster / 4, cluster / 8 ways, widest first
	int cshift;        // log2 cluster
	int ginv;          // ceil(65536 / q heads per kv head): row / heads = row * ginv >> 16 for the rows of a tile
	int tiles;
};

template <int HD>
struct ChunkSmem {
	static constexpr int kKStride = HD + 16;
	static constexpr size_t kStage = (size_t)2 * kChunkStep * kKStride;              // two K steps, or two V steps, or received shares
	static constexpr size_t kScores = (size_t)kChunkRows * kChunkStep * 4;           // per step
	static constexpr size_t kMisc = kChunkRows * sizeof(IExpFast) + kChunkRows * (8 + 4 + 4) + 8 * 3 * 4 + kChunkSteps * 8 * 8 +
	                                8 * kChunkRows * (4 + 8);
	__host__ __device__ static constexpr size_t bytes(int steps) { return kStage + kScores * steps + kMisc; }
};

template <int HD>
__global__ void __launch_bounds__(kChunkThreads, 2)
k_attention_chunk(RowBatch b, Dims d, const __grid_constant__ LayerDev layer, int layer_index, KvPoolDev pool, ChunkPlan pl) {
	using L = ChunkSmem<HD>;
	constexpr int KS = HD / 32;          // MMA steps along the head dimension
	constexpr int NT = HD / 32;          // 8-channel tiles a warp owns in P.V (a quarter of the channels)
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ __align__(8) unsigned long long s_bars[3];
	int8_t* stage = (int8_t*)smem;
	int4* sc = (int4*)(smem + L::kStage);                                     // [step][4][threads]
	IExpFast* fxs = (IExpFast*)(smem + L::kStage + L::kScores * pl.steps);
	unsigned long long* rsum = (unsigned long long*)(fxs + kChunkRows);       // [32]
	unsigned long long* rx_sum = rsum + kChunkRows;                           // [sub][32]
	int64_t* pbase = (int64_t*)(rx_sum + 8 * kChunkRows);                     // [steps * 8] page offsets inside a plane
	int32_t* rmax = (int32_t*)(pbase + kChunkSteps * 8);                      // [32]
	int32_t* rx_max = rmax + kChunkRows;                                      // [sub][32]
	int32_t* tok_ok = rx_max + 8 * kChunkRows;                                // [32] 1: the token takes part
	int32_t* l_fold = tok_ok + kChunkRows;                                    // [8][3]
	int32_t* rx_ctx = (int32_t*)stage;                                        // [sub][32 / sub][HD]

	// which tile, split how many ways
	const int kvh = blockIdx.z, G = d.heads / d.kv_heads;
	const int crank = (int)blockIdx.x;
	int shift = pl.cshift, item = (int)blockIdx.y, before = 0;      // shift = log2 of the ways the tile is split
#pragma unroll
	for (int i = 0; i < 4; ++i) {
		const int per = pl.cshift - shift, clusters = (pl.count[i] + (1 << per) - 1) >> per;
		if (item < clusters || shift == 0 || i == 3) {
			item = (item << per) + (crank >> shift);
			if (item >= pl.count[i]) item = -1;
			break;
		}
		item -= clusters;
		before += pl.count[i];
		--shift;
	}
	const int sub = 1 << shift, rank = crank & (sub - 1), rank0 = crank - rank;      // the group of blocks that share the tile
	const int t = threadIdx.x, warp = t >> 5, lane = t & 31, g = lane >> 2, c = lane & 3;
	if (sub > 1) {
		if (t == 0) {
			const int held = (blockIdx.x | blockIdx.y | blockIdx.z) == 0 ? b.debug_withhold : 0;
			auto more = [&](int i) { return held == i + 1 ? 4u : 0u; };
			exchange_init(cta_addr(&s_bars[0]), (uint32_t)(sub * kChunkRows * 4) + more(0));
			exchange_init(cta_addr(&s_bars[1]), (uint32_t)(sub * kChunkRows * 8) + more(1));
			exchange_init(cta_addr(&s_bars[2]), (uint32_t)(kChunkRows * HD * 4) + more(2));
			exchange_fence_init();
		}
		cluster_arrive();
		cluster_wait();
	}
	if (item < 0) {      // no tile for this block: it only meets the others of its cluster
		if (sub > 1) {
			cluster_arrive();
			cluster_wait();
		}
		return;
	}
	const int tile = pl.tiles - 1 - before - item;
	const int r0 = tile * pl.tq, nt = min(pl.tq, b.m - r0);
	const int rb = warp >> 2, kq = warp & 3;
	const int rho_a = rb * 16 + g, rho_b = rho_a + 8;
	const int tok_a = rho_a * pl.ginv >> 16, tok_b = rho_b * pl.ginv >> 16;
	const int head_a = rho_a - tok_a * G, head_b = rho_b - tok_b * G;
	// uploaded before the call's first launch: the tile's first position and the sequence's page table
	const int pos0 = b.rows[r0].pos, old = b.rows[0].pos;
	const int32_t* pages = b.rows[r0].pages;
	const int width = pos0 + nt;
	const int nsteps = ((width + kChunkStep - 1) / kChunkStep - rank + sub - 1) >> shift;      // this block's: rank, rank + sub, ...
	const int8_t* kplane = pool.base + kv_plane_offset(d, pool, layer_index, kvh, 0);
	const int8_t* vplane = pool.base + kv_plane_offset(d, pool, layer_index, kvh, 1);
	for (int i = t; i < nsteps * 8; i += kChunkThreads) {
		const int page = (rank + (i >> 3) * sub) * 8 + (i & 7);
		pbase[i] = page * kPageTokens < width ? (int64_t)pages[page] * (kPageTokens * HD) : 0;
	}
	if (t < 3 * G) l_fold[t] = layer.f_ctx[3 * kvh * G + t];
	if (t < kChunkRows) {
		rmax[t] = INT32_MIN;
		rsum[t] = 0ull;
	}
	__syncthreads();
	// step i of this block into half i & 1 of the stage; positions beyond the tile's width are left as they are
	// (their scores are masked, their probabilities zero)
	auto load_k = [&](int i) {
		int8_t* kd = stage + (size_t)(i & 1) * kChunkStep * L::kKStride;
		const int base = (rank + i * sub) * kChunkStep;
		for (int idx = t; idx < kChunkStep * (HD / 16); idx += kChunkThreads) {
			const int row = idx / (HD / 16), piece = idx % (HD / 16);
			if (base + row < width)
				cp_async16(kd + (size_t)row * L::kKStride + piece * 16, kplane + pbase[i * 8 + (row >> 4)] + (row & 15) * HD + piece * 16);
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	auto load_v = [&](int i) {
		int8_t* vd = stage + (size_t)(i & 1) * kChunkStep * HD;
		const int base = (rank + i * sub) * kChunkStep;
		for (int idx = t; idx < 8 * HD; idx += kChunkThreads) {
			const int pg = idx / HD, piece = idx % HD;
			if (base + pg * kPageTokens < width)
				cp_async16(vd + (size_t)pg * HD * kPageTokens + piece * 16, vplane + pbase[i * 8 + pg] + piece * 16);
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	// positions of earlier calls are in place: the first step need not wait for the kernel in front
	const bool early = nsteps > 0 && (rank + 1) * kChunkStep <= old;
	if (early) load_k(0);
	pdl_wait();
	pdl_release();
	if (t < kChunkRows) {
		int okv = 0;
		if (t < nt) {
			okv = __ldcg(&b.status[r0 + t]) == 0 ? 1 : 0;
			fxs[t] = iexp_fast_prepare(b.smc[(size_t)(r0 + t) * d.kv_heads + kvh]);
		}
		tok_ok[t] = okv;
	}
	if (nsteps > 0 && !early) load_k(0);
	__syncthreads();
	const bool in_a = tok_a < nt && tok_ok[tok_a] != 0, in_b = tok_b < nt && tok_ok[tok_b] != 0;
	const int lim_a = in_a ? pos0 + tok_a : -1, lim_b = in_b ? pos0 + tok_b : -1;    // last position each row sees
	bool ok = true;

	// ---- pass 1: scores, kept per thread; row maxima. acc[j]: MMA j = 2 * group + half of a 16-position group
	{
		uint32_t qa[KS][4];      // q fragments (A operand) of this warp's rows
		const int8_t* qpa = b.qrot + (size_t)(r0 + (in_a ? tok_a : 0)) * d.hidden + (size_t)(kvh * G + head_a) * HD;
		const int8_t* qpb = b.qrot + (size_t)(r0 + (in_b ? tok_b : 0)) * d.hidden + (size_t)(kvh * G + head_b) * HD;
#pragma unroll
		for (int ks = 0; ks < KS; ++ks) {
			qa[ks][0] = in_a ? *(const uint32_t*)(qpa + 32 * ks + 4 * c) : 0u;
			qa[ks][1] = in_b ? *(const uint32_t*)(qpb + 32 * ks + 4 * c) : 0u;
			qa[ks][2] = in_a ? *(const uint32_t*)(qpa + 32 * ks + 16 + 4 * c) : 0u;
			qa[ks][3] = in_b ? *(const uint32_t*)(qpb + 32 * ks + 16 + 4 * c) : 0u;
		}
		// the K row that matrix row lane & 7 of half h stands for: 4 * (i / 2) + 2 h + (i & 1)
		const int krow = 4 * ((lane & 7) >> 1) + (lane & 1);
		int mx_a = INT32_MIN, mx_b = INT32_MIN;
#pragma unroll 1
		for (int i = 0; i < nsteps; ++i) {
			if (i + 1 < nsteps) {
				load_k(i + 1);
				asm volatile("cp.async.wait_group 1;" ::: "memory");
			} else {
				asm volatile("cp.async.wait_group 0;" ::: "memory");
			}
			__syncthreads();
			const int base = (rank + i * sub) * kChunkStep;
			const bool full = base + kChunkStep - 1 <= pos0;      // every row of the tile sees the whole step
			const uint32_t kd = cta_addr(stage + (size_t)((i & 1) * kChunkStep + kq * 32) * L::kKStride);
			int acc[4][4];
#pragma unroll
			for (int j = 0; j < 4; ++j)
#pragma unroll
				for (int q = 0; q < 4; ++q) acc[j][q] = 0;
			if constexpr (HD == 32) {
#pragma unroll
				for (int j = 0; j < 4; j += 2) {      // both halves of a group in one load
					uint32_t b0, b1, b2, b3;
					ldmatrix4(kd + (8 * j + krow + 2 * (lane >> 4)) * L::kKStride + ((lane >> 3) & 1) * 16, b0, b1, b2, b3);
					mma_s8s8_full(acc[j], qa[0][0], qa[0][1], qa[0][2], qa[0][3], b0, b1);
					mma_s8s8_full(acc[j + 1], qa[0][0], qa[0][1], qa[0][2], qa[0][3], b2, b3);
				}
			} else {
#pragma unroll
				for (int ks = 0; ks < KS; ks += 2) {
#pragma unroll
					for (int j = 0; j < 4; ++j) {
						uint32_t b0, b1, b2, b3;
						ldmatrix4(kd + (16 * (j >> 1) + 2 * (j & 1) + krow) * L::kKStride + 32 * ks + (lane >> 3) * 16, b0, b1, b2, b3);
						mma_s8s8_full(acc[j], qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3], b0, b1);
						mma_s8s8_full(acc[j], qa[ks + 1][0], qa[ks + 1][1], qa[ks + 1][2], qa[ks + 1][3], b2, b3);
					}
				}
			}
			// row a, group p (positions 16 p + 4 c ..): acc[2p][0], acc[2p][1], acc[2p + 1][0], acc[2p + 1][1]; row b: [2], [3]
			if (!full) {
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					const int k0 = base + kq * 32 + 16 * (j >> 1) + 4 * c + 2 * (j & 1);
					acc[j][0] = k0 <= lim_a ? acc[j][0] : INT32_MIN;
					acc[j][1] = k0 + 1 <= lim_a ? acc[j][1] : INT32_MIN;
					acc[j][2] = k0 <= lim_b ? acc[j][2] : INT32_MIN;
					acc[j][3] = k0 + 1 <= lim_b ? acc[j][3] : INT32_MIN;
				}
			}
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				mx_a = max(mx_a, max(acc[j][0], acc[j][1]));
				mx_b = max(mx_b, max(acc[j][2], acc[j][3]));
			}
#pragma unroll
			for (int p = 0; p < 2; ++p) {
				sc[(i * 4 + 2 * p) * kChunkThreads + t] = make_int4(acc[2 * p][0], acc[2 * p][1], acc[2 * p + 1][0], acc[2 * p + 1][1]);
				sc[(i * 4 + 2 * p + 1) * kChunkThreads + t] = make_int4(acc[2 * p][2], acc[2 * p][3], acc[2 * p + 1][2], acc[2 * p + 1][3]);
			}
			__syncthreads();      // the step may be overwritten
		}
		mx_a = max(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 1));
		mx_a = max(mx_a, __shfl_xor_sync(0xffffffffu, mx_a, 2));
		mx_b = max(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 1));
		mx_b = max(mx_b, __shfl_xor_sync(0xffffffffu, mx_b, 2));
		if (c == 0) {
			atomicMax(&rmax[rho_a], mx_a);
			atomicMax(&rmax[rho_b], mx_b);
		}
	}
	// (the stage is free: V arrives during the softmax)
	if (nsteps > 0) load_v(0);
	if (nsteps > 1) load_v(1);
	__syncthreads();
	int mx_a = rmax[rho_a], mx_b = rmax[rho_b];
	if (sub > 1) {
		if (t < sub * kChunkRows) exchange_send(&rx_max[rank * kChunkRows + (t & 31)], cta_addr(&s_bars[0]), (uint32_t)(rank0 + (t >> 5)), (uint32_t)rmax[t & 31]);
		ok = exchange_wait(cta_addr(&s_bars[0]));
		for (int i = 0; i < sub; ++i) {
			mx_a = max(mx_a, rx_max[i * kChunkRows + rho_a]);
			mx_b = max(mx_b, rx_max[i * kChunkRows + rho_b]);
		}
	}

	// ---- pass 2: exponentials and row totals
	const IExpFast fa = fxs[in_a ? tok_a : 0], fb = fxs[in_b ? tok_b : 0];
	{
		unsigned long long sum[2] = {0ull, 0ull};
#pragma unroll 1
		for (int i = 0; i < nsteps; ++i) {
			const bool full = (rank + i * sub) * kChunkStep + kChunkStep - 1 <= pos0;
#pragma unroll
			for (int j = 0; j < 4; ++j) {      // (row j & 1, group j / 2)
				int4* at = &sc[(i * 4 + j) * kChunkThreads + t];
				const int4 v = *at;
				const IExpFast& f = (j & 1) ? fb : fa;
				const uint32_t m = (uint32_t)((j & 1) ? mx_b : mx_a);
				uint32_t p0, p1, p2, p3;
				int64_t e0 = chunk_exp(m - (uint32_t)v.x, f, &p0), e1 = chunk_exp(m - (uint32_t)v.y, f, &p1);
				int64_t e2 = chunk_exp(m - (uint32_t)v.z, f, &p2), e3 = chunk_exp(m - (uint32_t)v.w, f, &p3);
				if (!full) {      // positions beyond a row's limit count for nothing
					if (v.x == INT32_MIN) { e0 = 0; p0 = kBaseOfZero; }
					if (v.y == INT32_MIN) { e1 = 0; p1 = kBaseOfZero; }
					if (v.z == INT32_MIN) { e2 = 0; p2 = kBaseOfZero; }
					if (v.w == INT32_MIN) { e3 = 0; p3 = kBaseOfZero; }
				}
				sum[j & 1] += (unsigned long long)(e0 + e1) + (unsigned long long)(e2 + e3);
				*at = make_int4((int)p0, (int)p1, (int)p2, (int)p3);
			}
		}
#pragma unroll
		for (int h = 0; h < 2; ++h) {
			sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
			sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);
			if (c == 0) atomicAdd(&rsum[h ? rho_b : rho_a], sum[h]);
		}
	}
	__syncthreads();
	unsigned long long tot[2] = {rsum[rho_a], rsum[rho_b]};
	if (sub > 1) {
		if (t < sub * kChunkRows) exchange_send(&rx_sum[rank * kChunkRows + (t & 31)], cta_addr(&s_bars[1]), (uint32_t)(rank0 + (t >> 5)), rsum[t & 31]);
		ok = exchange_wait(cta_addr(&s_bars[1])) && ok;
		tot[0] = tot[1] = 0;
		for (int i = 0; i < sub; ++i) {
			tot[0] += rx_sum[i * kChunkRows + rho_a];
			tot[1] += rx_sum[i * kChunkRows + rho_b];
		}
	}

	// ---- pass 3: probabilities. Slots 0 and 1 of a step then hold this warp's A fragments of P.V, low and high
	// plane: (row a group 0, row b group 0, row a group 1, row b group 1), four positions per word
	{
		const ChunkProb pa = chunk_prob(tot[0], fa), pb = chunk_prob(tot[1], fb);
#pragma unroll 1
		for (int i = 0; i < nsteps; ++i) {
			uint32_t lo[4], hi[4];
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				const int4 v = sc[(i * 4 + j) * kChunkThreads + t];
				const ChunkProb& p = (j & 1) ? pb : pa;
				float near = 1.0f;
				uint32_t p0 = chunk_prob_of((uint32_t)v.x, p, &near), p1 = chunk_prob_of((uint32_t)v.y, p, &near);
				uint32_t p2 = chunk_prob_of((uint32_t)v.z, p, &near), p3 = chunk_prob_of((uint32_t)v.w, p, &near);
				if (near < p.eps) {
					const uint4 x = chunk_prob_exact((uint32_t)v.x, (uint32_t)v.y, (uint32_t)v.z, (uint32_t)v.w, (j & 1) ? fb.qc : fa.qc, tot[j & 1]);
					p0 = x.x; p1 = x.y; p2 = x.z; p3 = x.w;
				}
				lo[j] = pack_plane(p0, p1, p2, p3, 0);
				hi[j] = pack_plane(p0, p1, p2, p3, 1);
			}
			sc[(i * 4) * kChunkThreads + t] = make_int4((int)lo[0], (int)lo[1], (int)lo[2], (int)lo[3]);
			sc[(i * 4 + 1) * kChunkThreads + t] = make_int4((int)hi[0], (int)hi[1], (int)hi[2], (int)hi[3]);
		}
	}

	// ---- pass 4: P.V of this warp's rows and quarter of the channels, over the positions of all four warps
	int accl[NT][4], acch[NT][4];
#pragma unroll
	for (int i = 0; i < NT; ++i)
#pragma unroll
		for (int q = 0; q < 4; ++q) accl[i][q] = acch[i][q] = 0;
#pragma unroll 1
	for (int i = 0; i < nsteps; ++i) {
		if (i + 1 < nsteps) asm volatile("cp.async.wait_group 1;" ::: "memory");
		else asm volatile("cp.async.wait_group 0;" ::: "memory");
		__syncthreads();      // V of the step (and, the first time, everybody's probabilities) are there
		const uint32_t vd = cta_addr(stage + (size_t)(i & 1) * kChunkStep * HD);
#pragma unroll
		for (int ks = 0; ks < kChunkStep / 32; ++ks) {
			const int4 l = sc[(i * 4) * kChunkThreads + (rb * 4 + ks) * 32 + lane], h = sc[(i * 4 + 1) * kChunkThreads + (rb * 4 + ks) * 32 + lane];
			if constexpr (NT == 1) {
				const uint32_t at = vd + (uint32_t)((2 * ks + ((lane >> 3) & 1)) * HD + 8 * kq + (lane & 7)) * kPageTokens;
				uint32_t b0, b1, b2, b3;      // (the upper half of the lanes repeats the lower half's rows)
				ldmatrix4(at, b0, b1, b2, b3);
				mma_u8s8_full(accl[0], l.x, l.y, l.z, l.w, b0, b1);
				mma_u8s8_full(acch[0], h.x, h.y, h.z, h.w, b0, b1);
			} else {
#pragma unroll
				for (int n = 0; n < NT; n += 2) {      // two 8-channel tiles, two pages each
					const uint32_t at = vd + (uint32_t)((2 * ks + ((lane >> 3) & 1)) * HD + 8 * (kq * NT + n + (lane >> 4)) + (lane & 7)) * kPageTokens;
					uint32_t b0, b1, b2, b3;
					ldmatrix4(at, b0, b1, b2, b3);
					mma_u8s8_full(accl[n], l.x, l.y, l.z, l.w, b0, b1);
					mma_u8s8_full(acch[n], h.x, h.y, h.z, h.w, b0, b1);
					mma_u8s8_full(accl[n + 1], l.x, l.y, l.z, l.w, b2, b3);
					mma_u8s8_full(acch[n + 1], h.x, h.y, h.z, h.w, b2, b3);
				}
			}
		}
		__syncthreads();      // the step may be overwritten
		if (i + 2 < nsteps) load_v(i + 2);
	}

	// ---- per-head context fold (forward_sites.cpp:1889-1896), store, row maximum for the funnel
	if (sub == 1) {
		uint32_t top_a = 0, top_b = 0;
#pragma unroll
		for (int n = 0; n < NT; ++n) {
			const int ch = 8 * (kq * NT + n) + 2 * c;
			auto put = [&](int tok, int head, int v0, int v1, uint32_t& top) {
				int2 o;
				o.x = fold(v0, l_fold[3 * head], l_fold[3 * head + 1], l_fold[3 * head + 2]);
				o.y = fold(v1, l_fold[3 * head], l_fold[3 * head + 1], l_fold[3 * head + 2]);
				*(int2*)(b.ctxw + (size_t)(r0 + tok) * d.hidden + (size_t)(kvh * G + head) * HD + ch) = o;
				top = max(top, max(abs_u32(o.x), abs_u32(o.y)));
			};
			if (in_a) put(tok_a, head_a, accl[n][0] + 256 * acch[n][0], accl[n][1] + 256 * acch[n][1], top_a);
			if (in_b) put(tok_b, head_b, accl[n][2] + 256 * acch[n][2], accl[n][3] + 256 * acch[n][3], top_b);
		}
		top_a = max(top_a, __shfl_xor_sync(0xffffffffu, top_a, 1));
		top_a = max(top_a, __shfl_xor_sync(0xffffffffu, top_a, 2));
		top_b = max(top_b, __shfl_xor_sync(0xffffffffu, top_b, 1));
		top_b = max(top_b, __shfl_xor_sync(0xffffffffu, top_b, 2));
		if (c == 0 && top_a) atomicMax(&b.rowmax[(size_t)(r0 + tok_a) * 4 + 3], (unsigned long long)top_a);
		if (c == 0 && top_b) atomicMax(&b.rowmax[(size_t)(r0 + tok_b) * 4 + 3], (unsigned long long)top_b);
		return;
	}
	// the shares go to the blocks that reduce their rows; a peer's stage is free once the peer has got here
	cluster_arrive();
	cluster_wait();
	const int rows = kChunkRows >> shift, rshift = 5 - shift;
	auto send = [&](int rho, int ch, int v0, int v1) {
		exchange_send(&rx_ctx[(rank * rows + (rho & (rows - 1))) * HD + ch], cta_addr(&s_bars[2]), (uint32_t)(rank0 + (rho >> rshift)), make_int2(v0, v1));
	};
#pragma unroll
	for (int n = 0; n < NT; ++n) {
		const int ch = 8 * (kq * NT + n) + 2 * c;
		send(rho_a, ch, accl[n][0] + 256 * acch[n][0], accl[n][1] + 256 * acch[n][1]);
		send(rho_b, ch, accl[n][2] + 256 * acch[n][2], accl[n][3] + 256 * acch[n][3]);
	}
	ok = exchange_wait(cta_addr(&s_bars[2])) && ok;
	for (int e = t; e < rows * HD; e += kChunkThreads) {
		const int rho = rank * rows + e / HD, ch = e % HD, tok = rho * pl.ginv >> 16, head = rho - tok * G;      // (a warp's elements lie in one row)
		int32_t sum = 0;
		for (int i = 0; i < sub; ++i) sum += rx_ctx[i * rows * HD + e];
		const int32_t o = fold(sum, l_fold[3 * head], l_fold[3 * head + 1], l_fold[3 * head + 2]);
		const bool in = tok < nt && tok_ok[tok] != 0;
		if (in) b.ctxw[(size_t)(r0 + tok) * d.hidden + (size_t)(kvh * G + head) * HD + ch] = o;
		const uint32_t top = __reduce_max_sync(0xffffffffu, in ? abs_u32(o) : 0u);
		if (lane == 0 && top) atomicMax(&b.rowmax[(size_t)(r0 + tok) * 4 + 3], (unsigned long long)top);
	}
	if (__builtin_expect(!__all_sync(0xffffffffu, ok), 0)) {      // (the warp's lanes speak for the tile's rows)
		if (lane < nt) atomicCAS(&b.status[r0 + lane], 0, pack_status(kInternalWaitTimeout, kSiteCtx, b.layer));
		__syncwarp();
		exchange_leave(cta_addr(&s_bars[0]), 3);
	}
}

// How a chunk of m rows whose last row is `width` wide is cut: tiles of 32 query rows; a block holds up to
// 512 positions, fewer while twice the blocks still run at once. False when the widest tile needs more
// than the eight blocks of a cluster.
static bool chunk_plan(const Dims& d, int m, int width, ChunkPlan* out) {
	const int G = d.heads / d.kv_heads, tq = kChunkRows / G, tiles = (m + tq - 1) / tq, first = width - m;
	bool found = false;
	for (int steps = kChunkSteps; steps >= 1; steps /= 2) {
		ChunkPlan p{tq, steps, 1, {0, 0, 0, 0}, 0, (65536 + G - 1) / G, tiles};
		auto ways = [&](int tile) {
			const int w = first + std::min((tile + 1) * tq, m);
			int s = 1;
			while (s * steps * kChunkStep < w) s *= 2;
			return s;
		};
		p.cluster = ways(tiles - 1);
		if (p.cluster > 8) break;
		while (1 << p.cshift < p.cluster) ++p.cshift;
		int blocks = 0;
		for (int i = 0; i < tiles; ++i) {
			const int s = ways(i);
			int at = 0;
			while (p.cluster >> at > s) ++at;
			++p.count[at];
			blocks += s * d.kv_heads;
		}
		*out = p;
		found = true;
		if (blocks > sm_count()) break;
	}
	return found;
}
template <int HD>
static cudaError_t launch_attn_chunk(const RowBatch& b, const Dims& d, const LayerDev& layer, int layer_index, KvPoolDev pool,
                                     const ChunkPlan& p, cudaStream_t st) {
	RowBatch rb = b;
	rb.debug_withhold = p.cluster > 1 ? exchange_debug_take(kExchangeAttnChunk) : 0;
	int clusters = 0;
	for (int i = 0, s = p.cluster; i < 4 && s >= 1; ++i, s /= 2) clusters += (p.count[i] + p.cluster / s - 1) / (p.cluster / s);
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(p.cluster, clusters, d.kv_heads);
	cfg.blockDim = dim3(kChunkThreads);
	cfg.dynamicSmemBytes = ChunkSmem<HD>::bytes(p.steps);
	cfg.stream = st;
	cudaLaunchAttribute attr[2];
	attr[0].id = cudaLaunchAttributeClusterDimension;
	attr[0].val.clusterDim.x = (unsigned)p.cluster;
	attr[0].val.clusterDim.y = 1;
	attr[0].val.clusterDim.z = 1;
	attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[1].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = attr;
	cfg.numAttrs = pdl_enabled() ? 2 : 1;
	return cudaLaunchKernelEx(&cfg, k_attention_chunk<HD>, rb, d, layer, layer_index, pool, p);
}

static int pad64(int w) { return (w + 63) / 64 * 64; }
constexpr int kAttnMaxSlice = 2048;      // positions one block holds at most

struct AttnPlan {
	int splits;       // slices along the width (k_attention_few), or 0: whole rows (k_attention)
	int whole_row;    // the cluster spans every kv head of the row (the funnel is fused)
	int cp;           // positions per block (shared-memory capacity)
};
// How a launch over `m` rows of up to `max_width` positions is cut.
static std::atomic<int> g_forced_splits{-1};     // -1: not set yet (the environment decides), 0: automatic
void attn_force_splits(int splits) { g_forced_splits.store(splits < 0 ? 0 : splits); }

static int forced_splits() {
	int forced = g_forced_splits.load();
	if (forced < 0) {      // SSLM_B200_ATTN_SPLITS=n fixes the slices per kv head (tuning, tests)
		const char* e = getenv("SSLM_B200_ATTN_SPLITS");
		forced = e ? atoi(e) : 0;
		g_forced_splits.store(forced < 0 ? 0 : forced);
	}
	return forced;
}
static AttnPlan attn_plan(const Dims& d, int m, int max_width, int forced) {
	AttnPlan p;
	// Clusters of 16 blocks need a GPC to themselves and there are eight: up to six rows get one each.
	// Otherwise a cluster has at most 8 blocks (the portable size).
	const int cluster_max = m <= 6 ? 16 : 8;
	const int per_kv_max = d.kv_heads <= cluster_max ? cluster_max / d.kv_heads : 1;   // slices with the whole row in one cluster
	int splits = 1;
	if (forced > 0) {
		while (splits * 2 <= forced && splits * 2 <= 16) splits *= 2;
	} else {
		// A slice shortens every stage of a block's chain and four exchanges cost under a microsecond, so
		// rows are cut while all blocks still run at once.
		const int blocks = m * d.kv_heads;
		while (splits < 8 && blocks * splits * 2 <= sm_count()) splits *= 2;
		if (splits > per_kv_max) splits = per_kv_max;              // prefer the fused funnel
	}
	while (splits > 1 && splits * 64 > pad64(max_width)) splits /= 2;
	// ... unless the width does not fit the slices: then up to 16 slices of one kv head per cluster
	while (splits < 16 && pad64((max_width + splits - 1) / splits) > kAttnMaxSlice) splits *= 2;
	p.whole_row = splits <= per_kv_max ? 1 : 0;
	p.splits = splits;
	p.cp = pad64((max_width + splits - 1) / splits);
	if (forced <= 0 && splits == 1 && m * d.kv_heads > sm_count() / 2) {      // many rows: a block meets nobody
		p.whole_row = 0;
		p.splits = 0;
	}
	return p;
}
constexpr size_t kFewSmemMax = 223 * 1024;
static size_t few_smem(const Dims& d, int cp) {
	const int G = d.heads / d.kv_heads;
	return d.head_dim == 128 ? FewSmem<128>::bytes(G, cp, true) : (d.head_dim == 64 ? FewSmem<64>::bytes(G, cp, true) : FewSmem<32>::bytes(G, cp, true));
}
// The q/k/v site of decode rows runs inside their attention clusters from two rows on. Apart / inside, ms for 6 or 16 tokens:
// 1.5B 2 rows 6.34 / 6.10, 5 rows 20.0 / 19.7, 12 rows 7.69 / 7.44; 0.5B (biases) 21 rows 18.4 / 17.7, 30 rows 6.78 / 6.75.
// Not for one row (1.5B 18.1 / 18.4, 0.5B 2.69 / 2.91): the streaming projections leave an attention block no registers
// beside them, and without a row kernel in between nothing hides its prologue.
AttnChoice attn_choose(const Dims& d, const LayerDev& h, int m, int max_width, int chunk) {
	AttnChoice c{forced_splits(), kSiteApart};
	if (chunk || m < 2) return c;
	const AttnPlan p = attn_plan(d, m, max_width, c.forced);
	if (p.splits == 0 || p.whole_row == 0 || few_smem(d, p.cp) > kFewSmemMax) return c;
	const bool bias = h.b_q != nullptr || h.b_k != nullptr || h.b_v != nullptr;
	c.site = bias ? kSiteBias : kSitePlain;
	return c;
}

template <int HD>
static cudaError_t launch_attn(const RowBatch& b, const Dims& d, const LayerDev& layer, int layer_index, KvPoolDev pool,
                               const AttnPlan& p, int reverse_rows, int site, const QkvSite& qs, cudaStream_t st) {
	const int G = d.heads / d.kv_heads;
	if (p.splits == 0) {
		// Twice the warps per block for decode rows: the blocks of the widest rows end last, and theirs is a chain. ms for 4 tokens,
		// 2 * head_dim threads / 4 * head_dim: 0.5B 45 rows 5.19 / 4.76, 80 5.75 / 5.44, 250 8.31 / 8.03; 1.5B 100 rows 7.89 / 7.71,
		// 180 9.52 / 9.07. Not with 128 channels and about one block per multiprocessor (64 rows 31.9 / 32.5 for 16
		// tokens, 80 7.22 / 7.32 for 4), nor for the short rows of a prompt (150 rows: 2.32 / 2.39). In 64 registers, with four words spilled from 64 channels on.
		const int blocks = d.kv_heads * b.m;
		const bool wide = reverse_rows == 0 && (HD < 128 || 4 * blocks >= 5 * sm_count());
		return launch_pdl(wide ? k_attention<HD, 1> : k_attention<HD, 2>, dim3(d.kv_heads, b.m), dim3(wide ? 4 * HD : 2 * HD), attn_smem_bytes(G, p.cp), st,
		                  b, d, layer, layer_index, pool, p.cp, reverse_rows);
	}
	const bool staged = FewSmem<HD>::bytes(G, p.cp, true) <= kFewSmemMax;
	RowBatch rb = b;
	rb.debug_withhold = site == kSiteBias && exchange_debug_take(kExchangeAttnSite) ? 5 : exchange_debug_take(kExchangeAttnFew);
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(d.kv_heads * p.splits, b.m);
	cfg.blockDim = dim3(2 * HD);
	cfg.dynamicSmemBytes = FewSmem<HD>::bytes(G, p.cp, staged);
	cfg.stream = st;
	cudaLaunchAttribute attr[2];
	attr[0].id = cudaLaunchAttributeClusterDimension;
	attr[0].val.clusterDim.x = (unsigned)(p.whole_row ? d.kv_heads * p.splits : p.splits);
	attr[0].val.clusterDim.y = 1;
	attr[0].val.clusterDim.z = 1;
	attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[1].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = attr;
	cfg.numAttrs = pdl_enabled() ? 2 : 1;
	auto kernel = staged ? k_attention_few<HD, true, kSiteApart, false> : k_attention_few<HD, false, kSiteApart, false>;
	if (site == kSitePlain) kernel = b.wide64 ? k_attention_few<HD, true, kSitePlain, true> : k_attention_few<HD, true, kSitePlain, false>;
	if (site == kSiteBias) kernel = b.wide64 ? k_attention_few<HD, true, kSiteBias, true> : k_attention_few<HD, true, kSiteBias, false>;
	return cudaLaunchKernelEx(&cfg, kernel, rb, d, layer, layer_index, pool, p.cp, p.splits, p.whole_row, reverse_rows, qs);
}

// (The attributes are the kernel's, not the model's: limits for the largest group, so that mapping one model
// takes nothing from another.)
template <int HD>
static cudaError_t configure_hd() {
	const int group = 8;
	auto set = [](const void* f, int smem, bool big_cluster) {
		cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
		// clusters of 16 blocks are an opt-in size
		if (e == cudaSuccess && big_cluster) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
		// same carve-out as the kernels around it (see rows_configure)
		if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
		return e;
	};
	cudaError_t e = set((const void*)k_attention<HD, 1>, (int)attn_smem_bytes(group, kAttnMaxSlice), false);
	if (e == cudaSuccess) e = set((const void*)k_attention<HD, 2>, (int)attn_smem_bytes(group, kAttnMaxSlice), false);
	for (const void* few : {(const void*)k_attention_few<HD, true, kSiteApart, false>, (const void*)k_attention_few<HD, true, kSitePlain, false>,
	                        (const void*)k_attention_few<HD, true, kSitePlain, true>, (const void*)k_attention_few<HD, true, kSiteBias, false>,
	                        (const void*)k_attention_few<HD, true, kSiteBias, true>})
		if (e == cudaSuccess) e = set(few, (int)kFewSmemMax, true);
	if (e == cudaSuccess)
		e = set((const void*)k_attention_few<HD, false, kSiteApart, false>, (int)FewSmem<HD>::bytes(group, kAttnMaxSlice, false), true);
	if (e == cudaSuccess) e = set((const void*)k_attention_tile<HD>, (int)TileSmem<HD>::kBytes, false);
	if (e == cudaSuccess) e = set((const void*)k_attention_chunk<HD>, (int)ChunkSmem<HD>::bytes(kChunkSteps), false);
	return e;
}

cudaError_t attn_configure(const Dims& d) {
	const int group = d.heads / d.kv_heads;
	if (group < 1 || group > 8 || d.heads % d.kv_heads != 0) return cudaErrorInvalidConfiguration;
	// widest row the plan can serve: 16 slices of kAttnMaxSlice positions
	if (d.context_cap > 16 * kAttnMaxSlice) return cudaErrorInvalidConfiguration;
	if (attn_smem_bytes(group, kAttnMaxSlice) > 225 * 1024) return cudaErrorInvalidConfiguration;
	if (d.head_dim == 128) return configure_hd<128>();
	if (d.head_dim == 64) return configure_hd<64>();
	if (d.head_dim == 32) return configure_hd<32>();
	return cudaErrorInvalidConfiguration;
}

bool launch_attention(const RowBatch& b, const Dims& d, const LayerDev& layer, int layer_index,
                      KvPoolDev pool, int max_width, int reverse_rows, const AttnChoice& choice, const int32_t* cos, const int32_t* sin,
                      cudaStream_t st, cudaError_t* err) {
	// Prefill chunks (rows at consecutive positions of one sequence), by what a whole prompt took with each
	// kernel. Tiles with the scores kept (k_attention_chunk) from 64 rows and 512 positions on: below, a row's
	// own blocks are as fast and a tile's fixed part is not paid back (300 rows of the 28-layer model: 3.3 ms
	// against 3.5; 512: 4.0 for either; 2,000 positions in chunks of 128: 55 against 39). The tiles that walk
	// the prefix three times and keep nothing (k_attention_tile) where a row is wider than a cluster of blocks
	// can hold (beyond 4,096 positions), and for head dimensions up to 64 in chunks of 1,600 rows or more: a
	// walk costs half as much there and its 16 times as many blocks fill the device (24-layer model, 1,400 rows:
	// 6.3 ms against 6.4; 2,047: 9.1 against 8.5).
	static const bool tile_off = [] {
		const char* e = getenv("SSLM_B200_ATTN_TILE");
		return e && e[0] == '0';
	}();
	static const int tile_min = [] {
		const char* e = getenv("SSLM_B200_ATTN_TILE_MIN");      // tuning: the width from which the tiled kernel runs
		return e ? atoi(e) : 1536;
	}();
	const bool tile_ok = reverse_rows && b.m >= 4 && max_width >= tile_min && !tile_off;
	const bool prefer_tile = tile_ok && d.head_dim <= 64 && b.m >= 1600;
	ChunkPlan cp;
	if (reverse_rows && b.m >= 64 && max_width >= 512 && !prefer_tile && chunk_plan(d, b.m, max_width, &cp)) {
		cudaError_t e;
		if (d.head_dim == 128) e = launch_attn_chunk<128>(b, d, layer, layer_index, pool, cp, st);
		else if (d.head_dim == 64) e = launch_attn_chunk<64>(b, d, layer, layer_index, pool, cp, st);
		else e = launch_attn_chunk<32>(b, d, layer, layer_index, pool, cp, st);
		if (err) *err = e;
		return false;
	}
	if (tile_ok) {
		cudaError_t e;
		if (d.head_dim == 128) e = launch_attn_tile<128>(b, d, layer, layer_index, pool, st);
		else if (d.head_dim == 64) e = launch_attn_tile<64>(b, d, layer, layer_index, pool, st);
		else e = launch_attn_tile<32>(b, d, layer, layer_index, pool, st);
		if (err) *err = e;
		return false;
	}
	const AttnPlan p = attn_plan(d, b.m, max_width, choice.forced);
	const QkvSite qs{cos, sin};
	cudaError_t e;
	if (d.head_dim == 128) e = launch_attn<128>(b, d, layer, layer_index, pool, p, reverse_rows, choice.site, qs, st);
	else if (d.head_dim == 64) e = launch_attn<64>(b, d, layer, layer_index, pool, p, reverse_rows, choice.site, qs, st);
	else e = launch_attn<32>(b, d, layer, layer_index, pool, p, reverse_rows, choice.site, qs, st);
	if (err) *err = e;
	return p.whole_row != 0;
}

// ------------------------------------------------------------ primitive sweep (tests)
// The integer primitives of the device library evaluated on arrays of operands ON THE DEVICE, so
// that their device-only halves (rcp.approx / rsqrt.approx estimates, 32-bit short forms) are
// compared with the CPU oracle too. Operand meaning per `which`: see sslm_b200_int_sweep.
__global__ void k_int_sweep(int which, const int64_t* a, const int64_t* b, const int64_t* c, const int64_t* e, long long n,
                            int64_t* out0, int64_t* out1, int64_t* out2) {
	for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
		int64_t o0 = 0, o1 = 0, o2 = 0;
		switch (which) {
		case 0: o0 = dyn_recip(a[i]); break;
		case 1: o0 = isqrt64(a[i]); break;
		case 2: o0 = floor_div_h32((int)a[i], b[i], rcp_estimate((double)b[i])); break;
		case 3: {
			o0 = requant_code(a[i], b[i], (int)c[i]);
			const Coder cd = make_coder(b[i], (int)c[i]);       // the per-row coder the kernels use must agree
			o1 = code_of(a[i], cd);
			o2 = fits_i32(a[i]) ? code_of((int32_t)a[i], cd) : o1;
			break;
		}
		case 4: {
			bool sat = false, ex = false;
			o0 = landing_rescale(a[i], b[i], c[i], e[i] >> 32, (int64_t)(int32_t)(uint32_t)e[i], &sat, &ex);
			o1 = (sat ? 1 : 0) | (ex ? 2 : 0);
			break;
		}
		case 5: o0 = (int64_t)udiv_small_quotient((uint64_t)a[i], (uint64_t)b[i], rcp_estimate((double)b[i])); break;
		case 6: {
			const Scale inc{b[i], c[i]}, site{e[i] >> 32, (int64_t)(int32_t)(uint32_t)e[i]};
			const FunnelParams fp = funnel_params((uint64_t)a[i], &inc, 1, site);
			o0 = fp.out.m;
			o1 = fp.out.e;
			o2 = fp.status;
			break;
		}
		case 7: {      // one softmax element on the attention kernels' 32-bit form; peak in the low half of e
			SoftmaxConsts k;
			k.c = IExpConsts{b[i], c[i], e[i] >> 32};
			k.peak = (int64_t)(uint32_t)e[i] << 16;
			const IExpFast f = iexp_fast_prepare(k);
			const int64_t v = iexp_fast((uint32_t)a[i], f);
			uint32_t word;
			chunk_exp((uint32_t)a[i], f, &word);
			const uint64_t base = word & 0xFFFFFFu;
			o0 = v;
			o1 = (v < 0 || v > k.peak) ? 1 : 0;       // the reference's per-element bound
			o2 = (int64_t)((base * base + (uint64_t)f.qc) >> (word >> 24));
			break;
		}
		case 8: {      // Q15 probability: floor((e << 15) / total), 0 <= e <= total
			const unsigned long long tot = (unsigned long long)b[i];
			const ProbRow pr = prob_row(tot);
			bool unsure = false;
			const uint32_t p = prob_fast(a[i], pr, &unsure) & 0xFFFFu;
			o0 = unsure ? prob_pair_exact(a[i], a[i], pr.tot).x : p;
			o1 = prob_q15(a[i], tot, 32768.0f / (float)tot);      // the exact form by itself
			break;
		}
		case 9: {      // the row kernels' code of x = a in a row of maximum b
			const QuadFunnel q = quad_funnel((unsigned long long)b[i], FunnelFold{Scale{1 << 30, 0}, kOk, kOk});
			const int32_t x32[4] = {(int32_t)a[i], (int32_t)-a[i], 0, (int32_t)a[i]};
			const int64_t x64[4] = {0, a[i], -a[i], 0};
			const uint32_t c32 = code_quad(x32, q), c64 = code_quad(x64, q);
			o0 = byte_of(c32, 0);
			o1 = byte_of(c64, 1);
			o2 = (byte_of(c32, 1) == -o0 && byte_of(c32, 3) == o0 && byte_of(c64, 2) == -o1) ? 0 : 1;
			break;
		}
		case 10: {      // the same for small integers held in floats
			const QuadFunnel q = quad_funnel((unsigned long long)b[i], FunnelFold{Scale{1 << 30, 0}, kOk, kOk});
			const float x[4] = {(float)a[i], (float)-a[i], 0.0f, (float)a[i]};
			const uint32_t c4 = code_small_quad(x, q);
			o0 = byte_of(c4, 0);
			o1 = byte_of(c4, 1);
			break;
		}
		case 11: {      // the residual site's landing of code a: branch scale (b, e >> 32), stream scale (c, low half of e)
			const Scale bs{b[i], e[i] >> 32}, ss{c[i], (int64_t)(int32_t)(uint32_t)e[i]};
			const Branch br = make_branch(bs, make_recip(dyn_recip(ss.m)), ss);
			float w[4] = {0.0f, 0.0f, 0.0f, 0.0f};
			if (br.fast) join_quad((uint32_t)(uint8_t)a[i], 0u, br, bs, ss, w);
			o0 = (int64_t)w[0];
			o1 = br.fast ? 1 : 0;
			break;
		}
		case 12: {      // RMSNorm: floor((a << 32) / root), the root of a row of c elements whose squares add up to b
			const NormDiv nd = make_norm_div((uint32_t)b[i], (int)c[i], rcp_estimate((double)c[i]));
			o0 = norm_quotient((int)a[i], nd);
			o1 = nd.fast ? 1 : 0;
			o2 = nd.root;
			break;
		}
		case 13: {      // the softmax element of the kernels that keep their scores; o1 its (shift, base) word
			SoftmaxConsts k;
			k.c = IExpConsts{b[i], c[i], e[i]};
			k.peak = 0;
			const IExpFast f = iexp_fast_prepare(k);
			uint32_t parts = 0;
			o0 = chunk_exp((uint32_t)a[i], f, &parts);
			o1 = parts;
			break;
		}
		case 14: {      // their Q15 probability of the element with the word a: constant q_c = c, row total b
			IExpFast f{};
			f.qc = c[i];
			const ChunkProb p = chunk_prob((unsigned long long)b[i], f);
			float near = 1.0f;
			o0 = chunk_prob_of((uint32_t)a[i], p, &near) & 0xFFFFu;
			o1 = near < p.eps ? 1 : 0;
			if (o1) o0 = chunk_prob_exact((uint32_t)a[i], kBaseOfZero, kBaseOfZero, kBaseOfZero, f.qc, (unsigned long long)b[i]).x;
			break;
		}
		case 15: {      // K/V landing (operands of case 4), magnitude without the clamp
			const Lander l = make_lander(b[i], c[i], e[i] >> 32, (int64_t)(int32_t)(uint32_t)e[i]);
			const uint64_t ac = a[i] < 0 ? (~(uint64_t)a[i] + 1u) : (uint64_t)a[i];
			o1 = l.fast && ac <= (1ull << 31) ? 1 : 0;
			if (o1) {
				const uint64_t m = land_magnitude((uint32_t)ac, l);
				o0 = ((a[i] < 0) != l.neg) ? -(int64_t)m : (int64_t)m;
			}
			break;
		}
		default: break;
		}
		out0[i] = o0;
		out1[i] = o1;
		out2[i] = o2;
	}
}
void launch_int_sweep(int which, const int64_t* a, const int64_t* b, const int64_t* c, const int64_t* e, long long n, int64_t* out0,
                      int64_t* out1, int64_t* out2, cudaStream_t st) {
	k_int_sweep<<<592, 256, 0, st>>>(which, a, b, c, e, n, out0, out1, out2);
}

// ------------------------------------------------------------ canonical KV export
// Writes `planes` planes of the sequence's K and V, from plane0 on, in the reference's save layout,
// [layer][K|V][kv head][span][head_dim] with zeros past the valid positions, undoing the paging and the
// V-page transposition.
__global__ void k_kv_export(Dims d, KvPoolDev pool, const int32_t* pages, int context_length,
                            int layer_index, int span, int plane0, int planes, int8_t* out) {
	const int hd = d.head_dim, vec = hd / 16;
	const int64_t per_plane = (int64_t)span * vec;
	const int64_t total = planes * per_plane;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
	     i += (int64_t)gridDim.x * blockDim.x) {
		const int64_t nth = i / per_plane, within = i - nth * per_plane, plane = plane0 + nth;
		const int pos = (int)(within / vec), v = (int)(within % vec);
		const int kvh = (int)(plane % d.kv_heads);
		const int is_v = (int)((plane / d.kv_heads) % 2);
		const int layer = (int)(plane / (2 * d.kv_heads));
		// layers already run for the token in flight hold one more position
		const int valid = context_length + (layer < layer_index ? 1 : 0);
		int4 val = make_int4(0, 0, 0, 0);
		if (pos < valid) {
			const int8_t* src = pool.base + kv_plane_offset(d, pool, layer, kvh, is_v) +
			                    (int64_t)pages[pos / kPageTokens] * (kPageTokens * hd);
			const int slot = pos % kPageTokens;
			if (!is_v) {
				val = *((const int4*)(src + slot * hd) + v);
			} else {
				uint32_t w[4] = {0, 0, 0, 0};
				for (int j = 0; j < 16; ++j)
					w[j >> 2] |= (uint32_t)(uint8_t)src[(v * 16 + j) * kPageTokens + slot] << (8 * (j & 3));
				val = make_int4((int)w[0], (int)w[1], (int)w[2], (int)w[3]);
			}
		}
		((int4*)out)[i] = val;
	}
}

void launch_kv_export(const Dims& d, KvPoolDev pool, const int32_t* pages, int context_length,
                      int layer_index, int span, int plane0, int planes, int8_t* out, cudaStream_t st) {
	k_kv_export<<<148 * 4, 256, 0, st>>>(d, pool, pages, context_length, layer_index, span, plane0, planes, out);
}

// The inverse: scatter planes of a canonical block (a save blob's K/V) into the sequence's pages.
// Only the valid positions are written; everything else in the pages is never read.
__global__ void k_kv_import(Dims d, KvPoolDev pool, const int32_t* pages, int context_length,
                            int layer_index, int span, int plane0, int planes, const int8_t* in) {
	const int hd = d.head_dim, vec = hd / 16;
	const int64_t per_plane = (int64_t)span * vec;
	const int64_t total = planes * per_plane;
	for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
	     i += (int64_t)gridDim.x * blockDim.x) {
		const int64_t nth = i / per_plane, within = i - nth * per_plane, plane = plane0 + nth;
		const int pos = (int)(within / vec), v = (int)(within % vec);
		const int kvh = (int)(plane % d.kv_heads);
		const int is_v = (int)((plane / d.kv_heads) % 2);
		const int layer = (int)(plane / (2 * d.kv_heads));
		const int valid = context_length + (layer < layer_index ? 1 : 0);
		if (pos >= valid) continue;
		const int4 val = ((const int4*)in)[i];
		int8_t* dst = pool.base + kv_plane_offset(d, pool, layer, kvh, is_v) +
		              (int64_t)pages[pos / kPageTokens] * (kPageTokens * hd);
		const int slot = pos % kPageTokens;
		if (!is_v) {
			*((int4*)(dst + slot * hd) + v) = val;
		} else {
			const uint32_t w[4] = {(uint32_t)val.x, (uint32_t)val.y, (uint32_t)val.z, (uint32_t)val.w};
			for (int j = 0; j < 16; ++j)
				dst[(v * 16 + j) * kPageTokens + slot] = (int8_t)((w[j >> 2] >> (8 * (j & 3))) & 0xffu);
		}
	}
}

// Block 0 takes over the page ids and the state; the others, one per (layer, kv head, K|V) plane, copy
// the last, partly filled page.
__global__ void k_adopt(Dims d, KvPoolDev pool, AdoptArgs a) {
	if (blockIdx.x == 0) {
		for (int i = threadIdx.x; i < a.full_pages; i += blockDim.x) a.dst_pages[i] = a.src_pages[i];
		if (threadIdx.x == 0 && a.copy_to >= 0) a.dst_pages[a.full_pages] = a.copy_to;
		for (int i = threadIdx.x; i < a.state_bytes / 16; i += blockDim.x) ((int4*)a.dst_state)[i] = ((const int4*)a.src_state)[i];
		return;
	}
	const int64_t page_bytes = (int64_t)kPageTokens * d.head_dim;
	int8_t* plane = pool.base + (int64_t)(blockIdx.x - 1) * (pool.num_pages * page_bytes);
	const int4* src = (const int4*)(plane + (int64_t)a.copy_from * page_bytes);
	int4* dst = (int4*)(plane + (int64_t)a.copy_to * page_bytes);
	for (int i = threadIdx.x; i < (int)(page_bytes / 16); i += blockDim.x) dst[i] = src[i];
}
void launch_adopt(const Dims& d, KvPoolDev pool, const AdoptArgs& a, cudaStream_t st) {
	k_adopt<<<a.copy_from >= 0 ? 1 + d.layers * d.kv_heads * 2 : 1, 128, 0, st>>>(d, pool, a);
}

void launch_kv_import(const Dims& d, KvPoolDev pool, const int32_t* pages, int context_length,
                      int layer_index, int span, int plane0, int planes, const int8_t* in, cudaStream_t st) {
	k_kv_import<<<148 * 4, 256, 0, st>>>(d, pool, pages, context_length, layer_index, span, plane0, planes, in);
}

}  // namespace sslm
