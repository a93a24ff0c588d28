// Per-row sites of the integer forward pass as fused CUDA kernels: one thread block
// (for the wide activation row: one cluster of blocks) owns one row -- one token of one
// sequence -- and carries it through every step that needs only that row: the dynamic-scale
// requant "funnel", RMSNorm, q/k/v post-processing (K/V landing, RoPE, page write, softmax
// constants), the residual reconciliation and the SwiGLU activation.
//
// On a decode batch a row site is bound by the length of its dependent chain, on a prefill chunk
// by the instructions it issues per element. Both are served the same way: a thread keeps its
// elements (NV quads of four neighbours) in registers from the first load to the last store, the
// per-element steps are the short exact forms of sslm_quad.cuh, everything that does not need the
// previous kernel is derived ahead of the dependency wait, and block-wide phases meet in one-barrier
// reductions. Residual site + RMSNorm at hidden 1536, one row: 11,000 cycles with the row staged in
// shared memory and per-row tables of the 255 code values, 2,600 this way (B200, warm code).
#include <cuda_runtime.h>

#include <initializer_list>
#include <type_traits>

#include "sslm_kernels.h"
#include "sslm_cluster.cuh"
#include "sslm_quad.cuh"

namespace sslm {

// per-row lookup tables indexed by an int8 code: 256 int64 values + 256 flag bytes
constexpr int kLutBytes = 256 * 8 + 256;

// ------------------------------------------------------------ block reductions
// Every row kernel is a chain of dependent phases, so a reduction's latency is paid in full
// each time. These cost one barrier: each warp reduces with the warp-reduce instruction and
// posts its value in one of two alternating banks of shared words, and after the barrier
// every thread folds the (at most 32) posted values itself. A bank is rewritten only two
// reductions later, i.e. after a barrier that every reader of its old contents has passed.
constexpr int kRedBank = 32;                   // one slot per warp
constexpr int kRedBytes = 2 * kRedBank * 8;
struct Red {
	unsigned long long* w;
	int phase;
};
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
	const uint32_t hi = (uint32_t)(v >> 32), lo = (uint32_t)v;
	const uint32_t mh = __reduce_max_sync(0xffffffffu, hi);
	const uint32_t ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
	return ((unsigned long long)mh << 32) | ml;
}
__device__ __forceinline__ long long warp_sum_i64(long long v) {
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
	return v;
}
// Every thread gets the result. All threads of the block must call these together.
__device__ __forceinline__ unsigned long long block_max_u64(unsigned long long v, Red& red) {
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
	unsigned long long* bank = red.w + red.phase * kRedBank;
	red.phase ^= 1;
	v = warp_max_u64(v);
	if (lane == 0) bank[warp] = v;
	__syncthreads();
	unsigned long long m = bank[0];
	for (int w = 1; w < nw; ++w) {
		const unsigned long long t = bank[w];
		m = t > m ? t : m;
	}
	return m;
}
__device__ __forceinline__ long long block_sum_i64(long long v, Red& red) {
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
	unsigned long long* bank = red.w + red.phase * kRedBank;
	red.phase ^= 1;
	v = warp_sum_i64(v);
	if (lane == 0) bank[warp] = (unsigned long long)v;
	__syncthreads();
	long long s = (long long)bank[0];
	for (int w = 1; w < nw; ++w) s += (long long)bank[w];
	return s;
}

__device__ __forceinline__ unsigned long long abs_u64(int64_t v) {
	return v < 0 ? (~(unsigned long long)v + 1ull) : (unsigned long long)v;
}
// ------------------------------------------------------------------ the general forms
// What a row takes when its scales leave the ranges the register forms cover (a landing exponent or
// magnitude outside 32 bits, a row whose rms is below 1): the reference's own widths, staged in shared
// memory. Out of line, so that the kernels' common path does not carry it.

// Funnel over a row staged in shared memory (RequantChainChecked,
// src/forward/checked_chain_funnel.cpp:257-364), after the row maximum. Every thread returns the same
// status; on failure nothing is written.
__device__ int32_t block_code(const int64_t* w, int n, unsigned long long mx, const FunnelFold& fold, int8_t* out,
                              Scale* out_scale) {
	const FunnelParams fp = funnel_finish(mx, fold);
	if (fp.status != kOk) return fp.status;
	const Coder cd = make_coder(fp.r, fp.s);
#pragma unroll 1
	for (int i = threadIdx.x; i < n; i += blockDim.x) out[i] = code_of(w[i], cd);
	if (threadIdx.x == 0 && out_scale) *out_scale = fp.out;
	return kOk;
}

// RmsNormSite (src/forward/forward_sites.cpp:410-459) on codes h[n] that this block wrote (or staged):
// root = max(isqrt(floor((sum h^2) << 32 / n)), 1); wide_i = floor((h_i << 32) / root) * g_i;
// funnel with no incoming scale.
__device__ __noinline__ int32_t block_rmsnorm(const int8_t* h, const int8_t* gain, int n, Scale site, int64_t* wide, int8_t* out,
                                              Scale* out_scale, int64_t* lut, Red& red) {
	const double inv_n = rcp_estimate((double)n);
	long long ss = 0;
#pragma unroll 1
	for (int i = threadIdx.x; i < n; i += blockDim.x) {
		const int v = h[i];
		ss += v * v;
	}
	ss = block_sum_i64(ss, red);
	// floor((sum << 32) / n): non-negative operands, an estimated quotient repaired exactly
	int64_t root = isqrt64((int64_t)udiv_small_quotient((uint64_t)ss << 32, (uint64_t)n, inv_n));
	if (root < 1) root = 1;
	// floor((h << 32) / root) depends only on the code: one division per code value, not per element
	const double inv_root = rcp_estimate((double)root);
#pragma unroll 1
	for (int t = threadIdx.x; t < 255; t += blockDim.x) lut[t] = floor_div_h32(t - 127, root, inv_root);
	__syncthreads();
	unsigned long long mx = 0;
#pragma unroll 1
	for (int i = threadIdx.x; i < n; i += blockDim.x) {
		const int64_t v = lut[(int)h[i] + 127] * (int64_t)gain[i];
		wide[i] = v;
		const unsigned long long a = abs_u64(v);
		mx = a > mx ? a : mx;
	}
	mx = block_max_u64(mx, red);   // its barrier also publishes wide[]
	return block_code(wide, n, mx, funnel_prefold(nullptr, 0, site), out, out_scale);
}

// Residual reconciliation (ResidualReconcileSite, forward_sites.cpp:871-989) on branch codes staged in
// shared memory: wide_i = LandingRescale(branch_i, S[branch], Recip(S[stream].m), ...) + stream_i.
__device__ __noinline__ int32_t block_residual(const int8_t* branch, Scale bs, const int8_t* stream, Scale ss, int n, int64_t r_h,
                                               const FunnelFold& fold, int64_t* wide, int8_t* out, Scale* out_scale, int64_t* lut,
                                               Red& red) {
	// the rescaled branch value depends only on the branch code: one LandingRescale per code value.
	// lex marks the codes whose rescaled magnitude left int64 (the site refuses a row that uses one).
	uint8_t* lex = (uint8_t*)(lut + 256);
#pragma unroll 1
	for (int t = threadIdx.x; t < 255; t += blockDim.x) {
		bool ex;
		lut[t] = landing_rescale((int64_t)(t - 127), bs.m, r_h, bs.e, ss.e, nullptr, &ex);
		lex[t] = ex ? 1 : 0;
	}
	__syncthreads();
	// one reduction carries both the row maximum and "some code's rescaled magnitude left
	// int64": no in-range sum has magnitude 2^64 - 1, which stands for the latter
	unsigned long long mx = 0;
#pragma unroll 1
	for (int i = threadIdx.x; i < n; i += blockDim.x) {
		const int c = (int)branch[i] + 127;
		if (lex[c]) {
			mx = ~0ull;
			wide[i] = 0;
		} else {
			const int64_t v = lut[c] + (int64_t)stream[i];
			wide[i] = v;
			const unsigned long long a = abs_u64(v);
			mx = a > mx ? a : mx;
		}
	}
	mx = block_max_u64(mx, red);   // its barrier also publishes wide[]
	if (mx == ~0ull) return kResidualMagnitudeOutOfDomain;
	return block_code(wide, n, mx, fold, out, out_scale);
}
// shared memory of the general forms: reductions, code tables, the int64 staging row, one code row
__host__ __device__ inline size_t general_smem_bytes(int n) { return kRedBytes + kLutBytes + (size_t)n * 9; }

__device__ __forceinline__ void set_status(const RowBatch& b, int row, int32_t st, int site, int layer) {
	if (threadIdx.x == 0 && st != kOk) atomicCAS(&b.status[row], 0, pack_status(st, site, layer));
}

// ------------------------------------------------------------------- kernels
// RMSNorm of the codes in `h` (this thread's NV quads; the block holds the row): sum of squares,
// root, floor((h << 32) / root) * gain, funnel without an incoming scale (RmsNormSite,
// src/forward/forward_sites.cpp:410-459). Returns -1 when the row needs the general form; nothing is
// written then.
template <int NV>
__device__ __forceinline__ int32_t quad_rmsnorm(const uint32_t (&h)[NV], const uint32_t (&g)[NV], int nq, int n, double inv_n,
                                                const FunnelFold& fold, int8_t* out, Scale* out_scale, Bank& bank) {
	uint32_t ss = 0;
#pragma unroll
	for (int v = 0; v < NV; ++v) ss = (uint32_t)__dp4a((int)h[v], (int)h[v], (int)ss);
	ss = block_sum_u32(ss, bank);
	const NormDiv nd = make_norm_div(ss, n, inv_n);
	if (!nd.fast) return -1;
	int32_t w[NV][4];
	uint32_t mx = 0;
#pragma unroll
	for (int v = 0; v < NV; ++v) {
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			w[v][j] = norm_quotient(byte_of(h[v], j), nd) * byte_of(g[v], j);
			mx = max(mx, abs_u32(w[v][j]));
		}
	}
	mx = block_max_u32(mx, bank);
	const QuadFunnel fp = quad_funnel((unsigned long long)mx, fold);
	if (fp.status != kOk) return fp.status;
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		const int q = threadIdx.x + v * blockDim.x;
		const uint32_t c = code_quad(w[v], fp);
		if (q < nq) ((uint32_t*)out)[q] = c;
	}
	if (threadIdx.x == 0) *out_scale = fp.out;
	return kOk;
}

// Start of a call for each row: embed the token (EmbedEntry,
// src/forward/forward_sites.cpp:763-787) or pick up the sequence's stored mid-token
// stream, then the first RMSNorm (gain == nullptr: none).
template <int NV>
__global__ void __launch_bounds__(512)
k_begin(RowBatch b, Dims d, const int8_t* embed, Scale c_embed, const RowSource* src, const int8_t* gain, Scale c_norm, int site_norm) {
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ uint32_t s_bank[64];
	Bank bank{s_bank, 0};
	const int r = blockIdx.x, n = d.hidden, nq = n >> 2;
	uint32_t g[NV];
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		const int q = threadIdx.x + v * blockDim.x;
		g[v] = (gain != nullptr && q < nq) ? ((const uint32_t*)gain)[q] : 0u;
	}
	const FunnelFold fold_e = funnel_prefold(nullptr, 0, c_embed), fold_n = funnel_prefold(nullptr, 0, c_norm);
	const double inv_n = rcp_estimate((double)n);
	pdl_wait();
	pdl_release();
	int8_t* x = b.x + (size_t)r * n;
	if (threadIdx.x == 0) {
		b.status[r] = 0;
		b.sat[r] = 0ull;
		b.done[r] = 0;
		b.best[r] = 0ull;      // the head accumulates its arg-max key here
		const RowDesc& rd = b.rows[r];
		if (rd.new_page >= 0) ((int32_t*)rd.pages)[rd.pos / kPageTokens] = rd.new_page;
	}
	for (int i = threadIdx.x; i < b.sat_ld; i += blockDim.x) b.sat_layer[(size_t)r * b.sat_ld + i] = 0u;
	const RowSource s = src[r];
	const bool fresh = s.hidden == nullptr;
	const uint32_t* from = (const uint32_t*)(fresh ? embed + (size_t)b.rows[r].token * n : s.hidden);
	uint32_t h[NV];
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		const int q = threadIdx.x + v * blockDim.x;
		h[v] = q < nq ? __ldcg(from + q) : 0u;
	}
	int32_t st = kOk;
	int site = kSiteEmbed;
	if (fresh) {
		uint32_t mx = 0;
#pragma unroll
		for (int v = 0; v < NV; ++v)
#pragma unroll
			for (int j = 0; j < 4; ++j) mx = max(mx, abs_u32(byte_of(h[v], j)));
		mx = block_max_u32(mx, bank);
		const QuadFunnel fp = quad_funnel((unsigned long long)mx, fold_e);
		st = fp.status;
		if (st == kOk) {
#pragma unroll
			for (int v = 0; v < NV; ++v) {
				const int32_t w[4] = {byte_of(h[v], 0), byte_of(h[v], 1), byte_of(h[v], 2), byte_of(h[v], 3)};
				h[v] = code_quad(w, fp);
			}
			if (threadIdx.x == 0) b.xs[r] = fp.out;
		}
	} else if (threadIdx.x == 0) {
		b.xs[r] = *s.scale;
	}
	if (st == kOk) {
#pragma unroll
		for (int v = 0; v < NV; ++v) {
			const int q = threadIdx.x + v * blockDim.x;
			if (q < nq) ((uint32_t*)x)[q] = h[v];
		}
		if (gain != nullptr) {
			site = site_norm;
			st = quad_rmsnorm<NV>(h, g, nq, n, inv_n, fold_n, b.nrm + (size_t)r * n, &b.ns[r], bank);
			if (st < 0) {
				Red red{(unsigned long long*)smem, 0};
				int64_t* lut = (int64_t*)(smem + kRedBytes);
				__syncthreads();
				st = block_rmsnorm(x, gain, n, c_norm, (int64_t*)(smem + kRedBytes + kLutBytes), b.nrm + (size_t)r * n, &b.ns[r],
				                   lut, red);
			}
		}
	}
	set_status(b, r, st, site, b.layer);
}

// After the fused q/k/v projection: q funnel (ProjectAndFunnel's tail,
// forward_sites.cpp:1114-1146), K/V landing with the saturation counter (LandTokenKVRow
// :1397-1415, LandingRescale :513-653), RoPE on q and on the landed K (:1748-1787,
// RopeApplySite :663-761), the page write, and the per-kv-head softmax constants with
// their domain gates (:1806-1856).
//
// A quad is two RoPE pairs, so a thread takes its elements from the projection row to their final
// place without meeting another thread. The last warp of the block takes no elements: its first
// lanes derive the softmax constants, a serial scalar chain that needs only the q scale, meanwhile.
template <int NV, bool W64, bool BIAS>
__global__ void __launch_bounds__(NV == 1 ? 704 : (NV == 4 ? 352 : 832), NV == 4 ? 2 : 1)
k_qkv_post(RowBatch b, Dims d, const __grid_constant__ LayerDev lw, int layer_index, KvPoolDev pool, const int32_t* rope_cos,
           const int32_t* rope_sin) {
	using T = typename WideOf<W64>::T;
	__shared__ uint32_t s_bank[64];
	Bank bank{s_bank, 0};
	const int r = blockIdx.x, H = d.hidden, KV = d.kv_hidden, hd = d.head_dim, half = hd >> 1;
	const int hs = __ffs(hd) - 1;                   // head_dim is a power of two
	const int qt = (int)blockDim.x - 32;            // threads that own quads
	const bool scalar_warp = (int)threadIdx.x >= qt;
	const int nq = (H + 2 * KV) >> 2;
	// ahead of the projection: the normed row's scale (written by the previous residual site),
	// the position, its RoPE row and page, the site constants
	const Scale ns = b.ns[r];
	const int pos = b.rows[r].pos;
	const int page = b.rows[r].pages[pos / kPageTokens];
	const int slot = pos % kPageTokens;
	const int64_t *bias_q = BIAS ? lw.b_q : nullptr, *bias_k = BIAS ? lw.b_k : nullptr, *bias_v = BIAS ? lw.b_v : nullptr;
	const FunnelFold fold_q = funnel_prefold(&ns, 1, lw.c_q);
	Scale kh{0, 0};
	const int kv_lane = (int)threadIdx.x - qt;
	if (scalar_warp && kv_lane < d.kv_heads) kh = Scale{lw.sm_khead[2 * kv_lane], lw.sm_khead[2 * kv_lane + 1]};
	// a quad's RoPE words (head_dim divides H, so k's elements sit on the same table words as q's) and
	// landing constants; with one quad per thread they too are fetched ahead of the projection
	auto rope_words = [&](int e, int2& c, int2& s) {
		const size_t at = (size_t)pos * half + ((e & (hd - 1)) >> 1);      // table row = position
		c = *(const int2*)(rope_cos + at);
		s = *(const int2*)(rope_sin + at);
	};
	auto landing = [&](int e, int64_t& r_t, int64_t& e_t) {
		const int64_t* rec = e < H + KV ? lw.k_recip + 3 * ((e - H) >> hs) : lw.v_recip + 3 * ((e - H - KV) >> hs);
		e_t = rec[1];
		r_t = rec[2];
	};
	int2 rc1 = make_int2(0, 0), rs1 = make_int2(0, 0);
	int64_t rt1 = 0, et1 = 0;
	if (NV == 1 && !scalar_warp && (int)threadIdx.x < nq) {
		const int e = (int)threadIdx.x * 4;
		if (e < H + KV) rope_words(e, rc1, rs1);
		if (e >= H) landing(e, rt1, et1);
	}
	// q/k/v bias (BIA1): term_i = round(B_i * Recip(S[x].m) / 2^(92 + S[x].e)) joins the folded
	// accumulator (after the LoRA delta) before the q funnel and before the K/V landing
	// (ApplyBiasReconcileRow, forward_sites.cpp:1015-1036). The exponent gate and R_a are per
	// row; a term or a sum that leaves int64 refuses the row. Biased elements are kept in 64 bits.
	// Only the sum needs the projection.
	int bexp = 0;
	int64_t r_a = 0;
	bool gate = true;
	if (BIAS) {
		r_a = dyn_recip(ns.m);
		gate = bias_exponent_in_domain(ns.e, &bexp);
	}
	auto bias_quad = [&](int q, int64_t (&term)[4], uint32_t& bad) {
		const int e = q * 4;
		const int64_t* bp = e < H ? bias_q : (e < H + KV ? bias_k : bias_v);
		const int off = e < H ? e : (e < H + KV ? e - H : e - H - KV);
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			term[j] = 0;
			if (!scalar_warp && q < nq && bp != nullptr && gate && !bias_term(bp[off + j], r_a, bexp, &term[j])) bad = 1;
		}
	};
	// Many decode rows: their old K pages are asked into L2 while the projection runs, a launch earlier than the
	// attention blocks, which all read K at once, could (78 MB of K and V at 256 rows: 4 % a step; V as well: slower).
	if (b.ask_ahead != 0) {
		const int pages = pos / kPageTokens;      // the full ones: earlier calls filled them
		for (int i = threadIdx.x; i < pages * d.kv_heads; i += blockDim.x) {
			const int h = i / pages;
			const int8_t* at = pool.base + kv_plane_offset(d, pool, layer_index, h, 0) + (int64_t)b.rows[r].pages[i - h * pages] * (kPageTokens * hd);
			asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(at), "r"(kPageTokens * hd) : "memory");
		}
	}
	int64_t term1[4] = {0, 0, 0, 0};
	uint32_t bad1 = 0;
	if (BIAS && NV == 1) bias_quad((int)threadIdx.x, term1, bad1);
	pdl_wait();
	pdl_release();
	const T* row = (const T*)b.wide + (size_t)r * b.wide_ld;
	T x[NV][4];
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		const int q = (int)threadIdx.x + v * qt;
		if (!scalar_warp && q < nq) load_quad(row + 4 * q, x[v]);
		else x[v][0] = x[v][1] = x[v][2] = x[v][3] = 0;
	}
	unsigned long long mx = __ldcg(&b.rowmax[(size_t)r * 4]);
	const bool refused = __ldcg(&b.status[r]) != 0;
	__syncthreads();      // every thread has read the row maximum: zero for its next producer
	if (threadIdx.x == 0) b.rowmax[(size_t)r * 4] = 0ull;
	if (refused) return;

	using Y = typename WideOf<W64 || BIAS>::T;
	Y y[NV][4];
	if constexpr (!BIAS) {
#pragma unroll
		for (int v = 0; v < NV; ++v)
#pragma unroll
			for (int j = 0; j < 4; ++j) y[v][j] = x[v][j];
	} else {
		if (!gate && bias_q != nullptr) {
			set_status(b, r, kRoundingDivideExponentOutOfDomain, kSiteQ, b.layer);
			return;
		}
		uint32_t lmx = 0, bad_q = 0, bad_kv = 0;
#pragma unroll
		for (int v = 0; v < NV; ++v) {
			const int q = (int)threadIdx.x + v * qt, e = q * 4;
			int64_t term[4];
			uint32_t bad = 0;
			if (NV > 1) bias_quad(q, term, bad);
			else bad = bad1;
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				int64_t sum;
				if (!bias_accumulate((int64_t)x[v][j], NV > 1 ? term[j] : term1[j], &sum)) bad = 1;
				y[v][j] = sum;
				if (!scalar_warp && e < H) {
					const unsigned long long a = abs_u64(sum);
					lmx = max(lmx, a > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)a);      // (anything above 2^31 is refused alike)
				}
			}
			if (e < H) bad_q |= bad;
			else bad_kv |= bad;
		}
		if (bias_q != nullptr) {
			// the row maximum the projection reduced does not include the bias: take it here (a q term or
			// sum outside int64 refuses the row first: it votes with a bit no maximum in the domain has)
			const uint32_t m = block_max_u32(bad_q != 0u ? 0xFFFFFFFFu : min(lmx, 0xFFFFFFFEu), bank);
			if (m == 0xFFFFFFFFu) {
				set_status(b, r, kBiasReconcileProductOutOfDomain, kSiteQ, b.layer);
				return;
			}
			mx = (unsigned long long)m;
		}
		// (K / V terms that cannot be formed refuse the row after the q funnel had its say, and before
		// anything lands, so before anything could count as saturated: LandTokenKVRow,
		// forward_sites.cpp:1281-1418)
		if (bias_k != nullptr || bias_v != nullptr) {
			const bool bad = __syncthreads_or((int)bad_kv) != 0;
			if ((bad || !gate) && quad_funnel(mx, fold_q).status == kOk) {
				set_status(b, r, gate ? kBiasReconcileProductOutOfDomain : kRoundingDivideExponentOutOfDomain, kSiteKv, b.layer);
				return;
			}
		}
	}
	const QuadFunnel fp = quad_funnel(mx, fold_q);
	if (fp.status != kOk) {
		set_status(b, r, fp.status, kSiteQ, b.layer);
		return;
	}
	if (scalar_warp) {
		// softmax constants per kv head: sm = Combine(S[q], softmax_khead) -> C30 constants -> width gate
		int32_t st = kOk;
		if (kv_lane < d.kv_heads) {
			SoftmaxConsts sc;
			st = softmax_consts(fp.out, kh, (uint64_t)pos + 1, &sc);
			b.smc[(size_t)r * d.kv_heads + kv_lane] = sc;
		}
		// the first failing head speaks for the row
		const uint32_t failing = __ballot_sync(0xffffffffu, st != kOk);
		if (failing != 0u && kv_lane == __ffs(failing) - 1) atomicCAS(&b.status[r], 0, pack_status(st, kSiteSoftmaxConsts, b.layer));
		return;
	}

	uint32_t sat = 0;
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		const int q = (int)threadIdx.x + v * qt, e = q * 4;
		if (q >= nq) break;
		if (e < H) {      // q: code, rotate
			const uint32_t c = code_quad(y[v], fp);
			if (NV > 1) rope_words(e, rc1, rs1);
			((uint32_t*)(b.qrot + (size_t)r * H))[q] = rope_quad(c, rc1, rs1);
			continue;
		}
		const bool is_k = e < H + KV;
		if (NV > 1) landing(e, rt1, et1);
		const Lander l = make_lander(ns.m, rt1, ns.e, et1);
		int lc[4];
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			const int64_t a = (int64_t)y[v][j];
			const unsigned long long mag = abs_u64(a);
			bool s1;
			if (l.fast && mag <= (1ull << 31)) {
				const uint64_t m = land_magnitude((uint32_t)mag, l);
				s1 = m > 127;
				const int c = s1 ? 127 : (int)m;
				lc[j] = ((a < 0) != l.neg) ? -c : c;
			} else {
				lc[j] = (int)clamp127(landing_rescale(a, ns.m, rt1, ns.e, et1, &s1, nullptr));
			}
			sat += s1 ? 1u : 0u;
		}
		const int kvh = (e - (is_k ? H : H + KV)) >> hs, dd = e & (hd - 1);
		int8_t* plane = pool.base + kv_plane_offset(d, pool, layer_index, kvh, is_k ? 0 : 1);
		if (is_k) {
			if (NV > 1) rope_words(e, rc1, rs1);
			*(uint32_t*)(plane + ((int64_t)page * kPageTokens + slot) * hd + dd) =
			    rope_quad(pack4(lc[0], lc[1], lc[2], lc[3]), rc1, rs1);
		} else {
			// V pages are stored transposed ([head_dim][16 positions]) so that the attention
			// kernel can feed them to the tensor cores as the K-major operand of P.V
#pragma unroll
			for (int j = 0; j < 4; ++j) plane[((int64_t)page * hd + dd + j) * kPageTokens + slot] = (int8_t)lc[j];
		}
	}
	if (sat != 0u) {      // (rare, and nothing in this kernel reads the counters)
		atomicAdd(&b.sat[r], (unsigned long long)sat);
		if (layer_index < b.sat_ld) atomicAdd(&b.sat_layer[(size_t)r * b.sat_ld + layer_index], sat);
	}
}

// Attention-context funnel (forward_sites.cpp:1898-1903): empty incoming, attn_ctx constant.
template <int NV>
__global__ void __launch_bounds__(512)
k_ctx_funnel(RowBatch b, Dims d, Scale c_ctx) {
	const int r = blockIdx.x, n = d.hidden, nq = n >> 2;
	const FunnelFold fold_ctx = funnel_prefold(nullptr, 0, c_ctx);
	pdl_wait();
	pdl_release();
	int32_t x[NV][4];
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		const int q = threadIdx.x + v * blockDim.x;
		if (q < nq) load_quad(b.ctxw + (size_t)r * n + 4 * q, x[v]);
		else x[v][0] = x[v][1] = x[v][2] = x[v][3] = 0;
	}
	const unsigned long long mx = __ldcg(&b.rowmax[(size_t)r * 4 + 3]);
	const bool refused = __ldcg(&b.status[r]) != 0;
	__syncthreads();
	if (threadIdx.x == 0) b.rowmax[(size_t)r * 4 + 3] = 0ull;
	if (refused) return;
	const QuadFunnel fp = quad_funnel(mx, fold_ctx);
	if (fp.status != kOk) {
		set_status(b, r, fp.status, kSiteCtx, b.layer);
		return;
	}
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		const int q = threadIdx.x + v * blockDim.x;
		const uint32_t c = code_quad(x[v], fp);
		if (q < nq) ((uint32_t*)(b.ctx + (size_t)r * n))[q] = c;
	}
	if (threadIdx.x == 0) b.cs[r] = fp.out;
}

// The residual site's general form, from the projection row on (the row's scales left the register
// form's range). Everything it needs is still in global memory.
template <typename T>
__device__ __noinline__ int32_t res_site_general(const T* row, int n, uint32_t peak, int64_t bs_m, int64_t bs_e,
                                                 const int8_t* stream, int64_t ss_m, int64_t ss_e, int64_t site_m, int64_t site_e,
                                                 int8_t* out, Scale* out_scale, unsigned char* smem) {
	Red red{(unsigned long long*)smem, 0};
	int64_t* lut = (int64_t*)(smem + kRedBytes);
	int64_t* wide = (int64_t*)(smem + kRedBytes + kLutBytes);
	int8_t* so = (int8_t*)(wide + n);
	int64_t dn;
	int s;
	normalize_scale((int64_t)peak, &dn, &s);
	const Coder cd = make_coder(dyn_recip(dn), s);
	const Scale ss{ss_m, ss_e};
	__syncthreads();
#pragma unroll 1
	for (int i = threadIdx.x; i < n; i += blockDim.x) so[i] = code_of((int64_t)__ldcg(row + i), cd);
	__syncthreads();
	return block_residual(so, Scale{bs_m, bs_e}, stream, ss, n, dyn_recip(ss.m), funnel_prefold(&ss, 1, Scale{site_m, site_e}), wide, out,
	                      out_scale, lut, red);
}

// A projection's funnel -> residual site -> (RMSNorm): the o projection and the attention residual
// (forward_sites.cpp:1906-1937), or the down projection, the MLP residual and the next layer's
// attention norm (:1968-1987, :1694-1698).
template <int NV, int MAXT, bool W64>
__global__ void __launch_bounds__(MAXT, NV == 1 ? 2 : 1)
k_res(RowBatch b, Dims d, ResSite a) {
	using T = typename WideOf<W64>::T;
	using WideLoad = typename std::conditional<W64, long long, int>::type;
	extern __shared__ __align__(16) unsigned char smem[];
	__shared__ uint32_t s_bank[64];
	Bank bank{s_bank, 0};
	const int r = blockIdx.x, n = d.hidden, nq = n >> 2;
	// ahead of the projection: the stream row and its scale (written two or more launches ago), the
	// scale of the projection's input, the gain and every scalar that needs only those
	uint32_t sx[NV], g[NV];
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		const int q = threadIdx.x + v * blockDim.x;
		sx[v] = q < nq ? __ldcg((const uint32_t*)(a.stream + (size_t)r * n) + q) : 0u;
		g[v] = (a.gain != nullptr && q < nq) ? ((const uint32_t*)a.gain)[q] : 0u;
	}
	const Scale is = a.in_scale[r], ss = a.stream_scale[r];
	const FunnelFold fold_p = funnel_prefold(&is, 1, a.c_proj);
	const FunnelFold fold_res = funnel_prefold(&ss, 1, a.c_res);
	const FunnelFold fold_n = funnel_prefold(nullptr, 0, a.c_norm);
	const int64_t r_h = dyn_recip(ss.m);
	const Recip r_f = make_recip(r_h);
	const double inv_n = rcp_estimate((double)n);
	const T* row = (const T*)b.wide + (size_t)r * b.wide_ld;
	pdl_wait();
	pdl_release();
	T x[NV][4];
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		const int q = threadIdx.x + v * blockDim.x;
		if (q < nq) load_quad(row + 4 * q, x[v]);
		else x[v][0] = x[v][1] = x[v][2] = x[v][3] = 0;
	}
	const unsigned long long pmx = __ldcg(&b.rowmax[(size_t)r * 4]);
	const bool refused = __ldcg(&b.status[r]) != 0;
	const QuadFunnel fp = quad_funnel(pmx, fold_p);
	int32_t st = fp.status;
	int site = a.site_proj, site_layer = b.layer;
	if (refused || st != kOk) {
		__syncthreads();
		if (threadIdx.x == 0) b.rowmax[(size_t)r * 4] = 0ull;
		if (!refused) set_status(b, r, st, site, site_layer);
		return;
	}
	// wide_i = LandingRescale(code_i, S[branch], Recip(S[stream].m), ...) + stream_i, small integers held
	// in floats when the largest landed magnitude allows it
	const Branch br = make_branch(fp.out, r_f, ss);
	site = a.site_res;
	uint32_t h[NV];
	Scale os{0, 0};
	if (br.fast && fits_i32(ss.m)) {
		float w[NV][4], top = 0.0f;
#pragma unroll
		for (int v = 0; v < NV; ++v) {
			const uint32_t c = code_quad(x[v], fp);
			join_quad(c, sx[v], br, fp.out, ss, w[v]);
#pragma unroll
			for (int j = 0; j < 4; ++j) top = fmaxf(top, fabsf(w[v][j]));
		}
		uint32_t mx = (uint32_t)top;
		mx = block_max_u32(mx, bank);
		if (threadIdx.x == 0) b.rowmax[(size_t)r * 4] = 0ull;      // (every thread has read it)
		const QuadFunnel fr = quad_funnel((unsigned long long)mx, fold_res);
		st = fr.status;
		if (st == kOk) {
#pragma unroll
			for (int v = 0; v < NV; ++v) {
				const int q = threadIdx.x + v * blockDim.x;
				h[v] = code_small_quad(w[v], fr);
				if (q < nq) ((uint32_t*)(a.out + (size_t)r * n))[q] = h[v];
			}
			if (threadIdx.x == 0) a.out_scale[r] = fr.out;
			os = fr.out;
		}
	} else {
		if (!fits_i32(ss.m)) st = kCarriedScaleMantissaOutOfDomain;
		else st = res_site_general((const WideLoad*)row, n, fp.d, fp.out.m, fp.out.e, a.stream + (size_t)r * n, ss.m, ss.e,
		                           a.c_res.m, a.c_res.e, a.out + (size_t)r * n, &a.out_scale[r], smem);
		__syncthreads();
		if (threadIdx.x == 0) b.rowmax[(size_t)r * 4] = 0ull;
		if (st == kOk) {
#pragma unroll
			for (int v = 0; v < NV; ++v) {
				const int q = threadIdx.x + v * blockDim.x;
				h[v] = q < nq ? *((volatile const uint32_t*)(a.out + (size_t)r * n) + q) : 0u;      // (this block wrote it)
			}
			if (threadIdx.x == 0) os = a.out_scale[r];
		}
	}
	if (st == kOk) {
		// (of the MLP residual: the layer is complete for this row, whatever the next layer does)
		if (a.done != nullptr && threadIdx.x == 0) a.done[r] = a.done_value;
		if (a.sink != nullptr) {      // the call's last layer: hand the stream back to the sequence
			const RowSink s = a.sink[r];
			if (s.hidden != nullptr) {
#pragma unroll
				for (int v = 0; v < NV; ++v) {
					const int q = threadIdx.x + v * blockDim.x;
					if (q < nq) ((uint32_t*)s.hidden)[q] = h[v];
				}
				if (threadIdx.x == 0) *s.scale = os;
			}
		}
		if (a.gain != nullptr) {
			site = a.site_norm;
			site_layer = a.norm_layer;
			st = quad_rmsnorm<NV>(h, g, nq, n, inv_n, fold_n, b.nrm + (size_t)r * n, &b.ns[r], bank);
			if (st < 0) {
				Red red{(unsigned long long*)smem, 0};
				int64_t* lut = (int64_t*)(smem + kRedBytes);
				__syncthreads();
				st = block_rmsnorm(a.out + (size_t)r * n, a.gain, n, a.c_norm, (int64_t*)(smem + kRedBytes + kLutBytes),
				                   b.nrm + (size_t)r * n, &b.ns[r], lut, red);
			}
		}
	}
	set_status(b, r, st, site, site_layer);
}

// scalars of an activation row
struct ActRow {
	float fg, fg_lo, fu, fu_lo;
	uint32_t dg, du;
	int live;
	FunnelFold fold;
};

// gate / up funnels -> SwiGLU activation site (MlpActSite, forward_sites.cpp:796-864).
//
// The activation row is the longest a row site walks (intermediate width, three codes per element).
// While rows are few its time is one block's chain, so a row is cut over a cluster of `gridDim.x`
// blocks, which meet once, for the maximum of the products; on a prefill chunk two blocks share a row.
// What depends on the row alone (two scale folds, two funnels, the product's fold: a quarter of the instructions) one warp
// derives for the block, while the others wait for their elements: 64 rows of 8,960 1.6 % a step, a prompt of
// 37 3 %. Not with five quads a thread, where it costs registers (prompt of 300: 1.7 % longer). From 16 rows on: a step of 16, 24, 32, 48
// rows 1,503 / 1,480, 1,600 / 1,562, 1,632 / 1,584, 1,793 / 1,764 us apart / shared at the 1.5B widths, 0 to 2 % at 0.5B and 3B; 9 and
// 12 rows take the same time either way.
// DENSE: in 72 registers instead of 80, for one more block per multiprocessor at some widths (launch_act)
template <int NV, bool W64, bool DENSE = false>
__global__ void __launch_bounds__(DENSE ? 288 : (NV == 5 ? 352 : 384), NV == 1 ? 1 : (DENSE ? 3 : 2))
k_act(RowBatch b, Dims d, Scale c_gate, Scale c_up, Scale c_act, const int32_t* silu_table) {
	using T = typename WideOf<W64>::T;
	__shared__ uint32_t s_bank[64];
	__shared__ int32_t table[1025];     // the sigmoid table
	__shared__ int32_t gsil[256];       // g * sigmoid(g) for the 255 gate codes, this row's scale
	__shared__ uint32_t s_peer[8];      // every block's largest product
	__shared__ ActRow s_row;
	__shared__ Scale s_gate;
	__shared__ __align__(8) unsigned long long s_arrived;
	Bank bank{s_bank, 0};
	const int r = blockIdx.y, n = d.inter, nq = n >> 2;
	const uint32_t blocks = gridDim.x, rank = blocks > 1 ? cluster_rank() : 0u;
	const int per = (nq + (int)blocks - 1) / (int)blocks, q0 = (int)rank * per, q1 = min(nq, q0 + per);
	// ahead of the gate/up projection: the normed row's scale (written by the residual site
	// before that projection ran) and the sigmoid table
	const bool shared = NV <= 2 && b.m >= 16;
	const bool scalar_thread = !shared || threadIdx.x < 32;
	for (int i = threadIdx.x; i < 1025; i += blockDim.x) table[i] = silu_table[i];
	FunnelFold fold_g{}, fold_u{};
	if (scalar_thread) {
		const Scale ns = b.ns[r];
		fold_g = funnel_prefold(&ns, 1, c_gate);
		fold_u = funnel_prefold(&ns, 1, c_up);
	}
	const uint32_t arrived = cta_addr(&s_arrived);
	if (blocks > 1) {
		if (threadIdx.x == 0) {
			exchange_init(arrived, 4u * blocks + ((blockIdx.x | blockIdx.y) == 0 && b.debug_withhold != 0 ? 4u : 0u));
			exchange_fence_init();
		}
		cluster_arrive();
		cluster_wait();
	}
	pdl_wait();
	pdl_release();
	const T* grow = (const T*)b.wide + (size_t)r * b.wide_ld;
	T xg[NV][4], xu[NV][4];
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		const int q = q0 + (int)threadIdx.x + v * (int)blockDim.x;
		if (q < q1) {
			load_quad(grow + 4 * q, xg[v]);
			load_quad(grow + n + 4 * q, xu[v]);
		} else {
			xg[v][0] = xg[v][1] = xg[v][2] = xg[v][3] = 0;
			xu[v][0] = xu[v][1] = xu[v][2] = xu[v][3] = 0;
		}
	}
	bool refused = false;
	int32_t st = kOk;
	int site = kSiteGate;
	Scale inc[2] = {Scale{0, 0}, Scale{0, 0}};
	QuadFunnel fg{}, fu{};
	bool live = false;
	if (scalar_thread) {
		const unsigned long long mxg = __ldcg(&b.rowmax[(size_t)r * 4 + 1]), mxu = __ldcg(&b.rowmax[(size_t)r * 4 + 2]);
		refused = __ldcg(&b.status[r]) != 0;
		const QuadFunnel qg = quad_funnel(mxg, fold_g), qu = quad_funnel(mxu, fold_u);
		inc[0] = qg.out;
		inc[1] = qu.out;
		st = qg.status != kOk ? qg.status : qu.status;
		site = qg.status != kOk ? kSiteGate : kSiteUp;
		if (st == kOk && !silu_scale_in_domain(qg.out)) {
			st = kSiluScaleOutOfDomain;
			site = kSiteSilu;
		}
		fg = qg;
		fu = qu;
		live = !refused && st == kOk;
		if (shared && threadIdx.x == 0) {
			s_row.fg = qg.f; s_row.fg_lo = qg.f_lo; s_row.dg = qg.d;
			s_row.fu = qu.f; s_row.fu_lo = qu.f_lo; s_row.du = qu.d;
			s_row.live = live;
			s_gate = qg.out;
		}
	}
	__syncthreads();      // the table and the row's scalars are complete
	if (shared) {
		live = s_row.live != 0;
		fg.f = s_row.fg; fg.f_lo = s_row.fg_lo; fg.d = s_row.dg;
		fu.f = s_row.fu; fu.f_lo = s_row.fu_lo; fu.d = s_row.du;
	}
	if (live) {
		// the sigmoid depends only on the gate code and the row's gate scale: 255 evaluations per
		// block instead of one per element
		const int64_t gm = shared ? s_gate.m : inc[0].m;
		const int ge = (int)(shared ? s_gate.e : inc[0].e);
		for (int t = threadIdx.x; t < 255; t += blockDim.x) gsil[t] = (t - 127) * silu_sigmoid_q15(table, t - 127, gm, ge);
	}
	__syncthreads();
	FunnelFold fold_act{};
	if (scalar_thread) {      // (read behind the barrier of the maximum that it will meet)
		fold_act = funnel_prefold(inc, 2, c_act);
		if (shared && threadIdx.x == 0) s_row.fold = fold_act;
	}
	// products g * sigmoid(g) * u, |.| <= 127 * 2^15 * 127 < 2^29
	int32_t w[NV][4];
	uint32_t mx = 0;
	if (live) {
		#pragma unroll
		for (int v = 0; v < NV; ++v) {
			const uint32_t g = code_quad(xg[v], fg), u = code_quad(xu[v], fu);
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				w[v][j] = gsil[byte_of(g, j) + 127] * byte_of(u, j);
				mx = max(mx, abs_u32(w[v][j]));
			}
		}
	}
	mx = block_max_u32(mx, bank);
	if (blocks > 1) {
		// Every block of the cluster comes through here, refused row or not, so none waits for one
		// that left; and only behind it is the row maximum cleared, so every block saw it.
		if (threadIdx.x < blocks) exchange_send(&s_peer[rank], arrived, threadIdx.x, mx);
		const bool ok = exchange_wait(arrived);
		if (__builtin_expect(!__all_sync(0xffffffffu, ok), 0)) {
			if ((threadIdx.x & 31) == 0) atomicCAS(&b.status[r], 0, pack_status(kInternalWaitTimeout, kSiteAct, b.layer));
			__syncwarp();
			exchange_leave(arrived, 1);
			return;
		}
		for (uint32_t i = 0; i < blocks; ++i) mx = max(mx, s_peer[i]);
	}
	if (rank == 0 && threadIdx.x == 0) {
		b.rowmax[(size_t)r * 4 + 1] = 0ull;
		b.rowmax[(size_t)r * 4 + 2] = 0ull;
	}
	if (!live) {
		if (!refused && rank == 0) set_status(b, r, st, site, b.layer);
		return;
	}
	const QuadFunnel fp = quad_funnel((unsigned long long)mx, shared ? s_row.fold : fold_act);
	if (fp.status != kOk) {
		if (rank == 0) set_status(b, r, fp.status, kSiteAct, b.layer);
		return;
	}
	uint32_t* out = (uint32_t*)(b.act + (size_t)r * n);
#pragma unroll
	for (int v = 0; v < NV; ++v) {
		const int q = q0 + (int)threadIdx.x + v * (int)blockDim.x;
		const uint32_t c = code_quad(w[v], fp);
		if (q < q1) out[q] = c;
	}
	if (rank == 0 && threadIdx.x == 0) b.acts[r] = fp.out;
}

// The activation site of many rows: persistent blocks, one row after another each.
//
// With hundreds of rows the form above is held by what every warp repeats for its row (three scale folds
// and two funnels, the table, 255 sigmoids a block: 840 of its 1,490 instructions) and by a chain of four
// barriers with nothing in flight. Here two warps derive the scalars and the 255 sigmoid products of the
// rows to come; the eight workers stream their elements through shared memory (asynchronous copies,
// each thread its own, kActStages steps ahead and on into the next row, so neither needs a barrier), leave
// the products there and meet once, for their maximum. The loops stay rolled: kept in registers, the
// products took so much code that a fifth of the time went into fetching it. Bound by instruction issue
// (210 a quad and warp, half of the slots): 2,047 rows of 8,960 take 47 us in place of 73, of which the
// 165 MB that move need 26.
constexpr int kActWorkers = 256, kActThreads = kActWorkers + 64, kActStages = 4;
__global__ void __launch_bounds__(kActThreads, 3)
k_act_many(RowBatch b, Dims d, Scale c_gate, Scale c_up, Scale c_act, const int32_t* silu_table) {
	extern __shared__ __align__(128) int4 stage[];      // [kActStages][gate, up][worker], then the products [quads of a row]
	__shared__ uint32_t s_top[2][kActWorkers / 32];
	__shared__ int32_t gsil[2][256];
	__shared__ ActRow s_row[2];
	__shared__ __align__(8) unsigned long long s_full[2], s_empty[2];
	const int n = d.inter, nq = n >> 2, t = threadIdx.x, lane = t & 31;
	if (t == 0) {
		for (int i = 0; i < 2; ++i) {
			ring_init(cta_addr(&s_full[i]), 1);
			ring_init(cta_addr(&s_empty[i]), kActWorkers / 32);
		}
		exchange_fence_init();
	}
	__syncthreads();
	pdl_wait();
	pdl_release();
	if (t >= kActWorkers) {
		const uint32_t slot = (uint32_t)(t - kActWorkers) >> 5;      // the two warps take the rows in turn
		uint32_t turn = 0;
		for (int r = blockIdx.x + (int)(slot * gridDim.x); r < b.m; r += 2 * gridDim.x, ++turn) {
			const unsigned long long mxg = __ldcg(&b.rowmax[(size_t)r * 4 + 1]), mxu = __ldcg(&b.rowmax[(size_t)r * 4 + 2]);
			const bool refused = __ldcg(&b.status[r]) != 0;
			const Scale ns = b.ns[r];
			const QuadFunnel fg = quad_funnel(mxg, funnel_prefold(&ns, 1, c_gate));
			const QuadFunnel fu = quad_funnel(mxu, funnel_prefold(&ns, 1, c_up));
			int32_t st = fg.status != kOk ? fg.status : fu.status;
			int site = fg.status != kOk ? kSiteGate : kSiteUp;
			if (st == kOk && !silu_scale_in_domain(fg.out)) {
				st = kSiluScaleOutOfDomain;
				site = kSiteSilu;
			}
			const bool live = !refused && st == kOk;
			const int freed = turn == 0 || ring_wait(cta_addr(&s_empty[slot]), (turn - 1) & 1);
			if (!__all_sync(0xffffffffu, freed)) return;      // (the workers' wait for the row runs out in turn)
			if (live) {
				const int ge = (int)fg.out.e;
#pragma unroll 4
				for (int c = lane; c < 255; c += 32) gsil[slot][c] = (c - 127) * silu_sigmoid_q15(silu_table, c - 127, fg.out.m, ge);
			}
			const Scale inc[2] = {fg.out, fu.out};
			if (lane == 0) {
				s_row[slot] = ActRow{fg.f, fg.f_lo, fu.f, fu.f_lo, fg.d, fu.d, live, funnel_prefold(inc, 2, c_act)};
				b.rowmax[(size_t)r * 4 + 1] = 0ull;
				b.rowmax[(size_t)r * 4 + 2] = 0ull;
				if (!refused && !live) atomicCAS(&b.status[r], 0, pack_status(st, site, b.layer));
			}
			__syncwarp();
			if (lane == 0) ring_arrive(cta_addr(&s_full[slot]));
		}
		return;
	}
	// A worker's copies run kActStages quads ahead of its arithmetic, on into the block's next row.
	const uint32_t stage0 = cta_addr(stage) + 16u * t;
	constexpr uint32_t kStageBytes = 32u * kActWorkers, kStageMask = kActStages * kStageBytes - 1;
	int ahead_r = t < nq ? (int)blockIdx.x : b.m, ahead_q = t;
	uint32_t ahead_slot = 0, slot_at = 0;
	auto ask = [&]() {
		if (ahead_r < b.m) {
			const int4* src = (const int4*)((const int32_t*)b.wide + (size_t)ahead_r * b.wide_ld) + ahead_q;
			copy16(stage0 + ahead_slot, src);
			copy16(stage0 + ahead_slot + kStageBytes / 2, src + nq);
			ahead_slot = (ahead_slot + kStageBytes) & kStageMask;
			ahead_q += kActWorkers;
			if (ahead_q >= nq) {
				ahead_q = t;
				ahead_r += gridDim.x;
			}
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
#pragma unroll 1
	for (int i = 0; i < kActStages; ++i) ask();
	int4* const kept = stage + kActStages * 2 * kActWorkers;
	uint32_t turn = 0;
	for (int r = blockIdx.x; r < b.m; r += gridDim.x, ++turn) {
		const uint32_t slot = turn & 1;
		const bool ok = ring_wait(cta_addr(&s_full[slot]), turn / 2 & 1);
		const ActRow& a = s_row[slot];
		const bool live = ok && a.live;
		// (of a row that is refused: zeros, whatever its words are)
		QuadFunnel fg{}, fu{};
		fg.f = live ? a.fg : 0.0f; fg.f_lo = a.fg_lo; fg.d = a.dg;
		fu.f = live ? a.fu : 0.0f; fu.f_lo = a.fu_lo; fu.d = a.du;
		const uint32_t products = cta_addr(gsil[slot]) + 4u * 127u - 4u * (uint32_t)kRoundMagicBits;      // + 4 * (biased code)
		uint32_t mx = 0;
#pragma unroll 1
		for (int q = t; q < nq; q += kActWorkers) {
			asm volatile("cp.async.wait_group %0;" ::"n"(kActStages - 1) : "memory");
			const int4 g = *(const int4*)((const char*)(stage + t) + slot_at), u = *(const int4*)((const char*)(stage + t) + slot_at + kStageBytes / 2);
			slot_at = (slot_at + kStageBytes) & kStageMask;
			const int32_t xg[4] = {g.x, g.y, g.z, g.w}, xu[4] = {u.x, u.y, u.z, u.w};
			int cg[4], cu[4], w[4];
			const float far_g = code_quad_try(xg, fg, cg), far_u = code_quad_try(xu, fu, cu);
			if (fmaxf(far_g, far_u) > kNearTie) {
				code_quad_settle(xg, fg, cg);
				code_quad_settle(xu, fu, cu);
			}
			ask();
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				int32_t s;
				asm volatile("ld.shared.s32 %0, [%1];" : "=r"(s) : "r"(products + 4u * (uint32_t)cg[j]));
				w[j] = s * (cu[j] - kRoundMagicBits);
				mx = max(mx, abs_u32(w[j]));
			}
			kept[q] = make_int4(w[0], w[1], w[2], w[3]);
		}
		// products are below 2^29: all ones says that a wait ran out somewhere in the block
		mx = __reduce_max_sync(0xffffffffu, ok ? mx : 0xffffffffu);
		uint32_t* top = s_top[slot];
		if (lane == 0) top[t >> 5] = mx;
		asm volatile("bar.sync 1, %0;" ::"n"(kActWorkers) : "memory");
		mx = __reduce_max_sync(0xffffffffu, lane < kActWorkers / 32 ? top[lane] : 0u);
		if (mx == 0xffffffffu) {
			if (t == 0)
				for (; r < b.m; r += gridDim.x) set_status(b, r, kInternalWaitTimeout, kSiteAct, b.layer);
			break;
		}
		if (live) {
			const QuadFunnel fp = quad_funnel((unsigned long long)mx, a.fold);
			if (fp.status != kOk) {
				set_status(b, r, fp.status, kSiteAct, b.layer);
			} else {
				uint32_t* out = (uint32_t*)(b.act + (size_t)r * n);
#pragma unroll 2
				for (int q = t; q < nq; q += kActWorkers) {
					const int4 k = kept[q];
					const int32_t w[4] = {k.x, k.y, k.z, k.w};
					out[q] = code_quad(w, fp);
				}
				if (t == 0) b.acts[r] = fp.out;
			}
		}
		__syncwarp();
		if (lane == 0) ring_arrive(cta_addr(&s_empty[slot]));
	}
	asm volatile("cp.async.wait_all;" ::: "memory");
}

// ------------------------------------------------------------------ launchers
// Quads per thread. One quad while the rows are few: the kernel's time is then the chain of a block,
// and the shortest chain has one quad per thread. A prefill chunk has hundreds of rows and is bound by
// instruction issue; every thread repeats the row's scalar chains (scale folds, reciprocals, roots), so
// fewer threads with four quads each issue fewer instructions. Widths beyond 4 x 512 quads take eight.
constexpr int kMaxQuadThreads = 512;
static int quads_per_thread(int rows, int nq) {
	static const int min_rows = [] {
		const char* e = getenv("SSLM_B200_ROW_THREADS_MIN_ROWS");      // tuning: batch size from which four quads apply
		return e ? atoi(e) : 512;
	}();
	if (nq > 4 * kMaxQuadThreads) return 8;
	return rows >= min_rows || nq > kMaxQuadThreads ? 4 : 1;
}
static int quad_threads(int nq, int nv) { return ((nq + nv - 1) / nv + 31) / 32 * 32; }

cudaError_t launch_begin(const RowBatch& b, const Dims& d, const int8_t* embed, Scale c_embed, const RowSource* src, const int8_t* gain,
                         Scale c_norm, int site_norm, cudaStream_t st) {
	int refuse = g_refuse_begin.load(std::memory_order_relaxed);
	if (refuse > 0 && g_refuse_begin.compare_exchange_strong(refuse, refuse - 1)) return cudaErrorLaunchOutOfResources;
	const int nq = d.hidden / 4, nv = quads_per_thread(b.m, nq), t = quad_threads(nq, nv);
	const size_t sm = general_smem_bytes(d.hidden);
	auto go = [&](auto kernel) { return launch_pdl(kernel, dim3(b.m), dim3(t), sm, st, b, d, embed, c_embed, src, gain, c_norm, site_norm); };
	if (nv == 1) return go(k_begin<1>);
	return nv == 4 ? go(k_begin<4>) : go(k_begin<8>);
}
void launch_qkv_post(const RowBatch& b, const Dims& d, const LayerDev& h, int layer_index, KvPoolDev pool,
                     const int32_t* cos, const int32_t* sin, cudaStream_t st) {
	const int nq = d.qkv_rows / 4;
	// one more warp than the quads need: it derives the softmax constants (a 704-thread block at most)
	int nv = quads_per_thread(b.m, nq > 672 ? nq : nq / 2);
	if (quad_threads(nq, nv) > (nv == 1 ? 672 : 320)) nv = quad_threads(nq, 4) <= 320 ? 4 : 8;
	const int t = quad_threads(nq, nv) + 32;
	const bool bias = h.b_q != nullptr || h.b_k != nullptr || h.b_v != nullptr;
	auto go = [&](auto kernel) { launch_pdl(kernel, dim3(b.m), dim3(t), 0, st, b, d, h, layer_index, pool, cos, sin); };
	auto pick = [&](auto nvc) {
		constexpr int NV = decltype(nvc)::value;
		if (b.wide64) bias ? go(k_qkv_post<NV, true, true>) : go(k_qkv_post<NV, true, false>);
		else bias ? go(k_qkv_post<NV, false, true>) : go(k_qkv_post<NV, false, false>);
	};
	if (nv == 1) pick(std::integral_constant<int, 1>());
	else if (nv == 4) pick(std::integral_constant<int, 4>());
	else pick(std::integral_constant<int, 8>());
}
void launch_ctx_funnel(const RowBatch& b, const Dims& d, const LayerDev& h, cudaStream_t st) {
	const int nq = d.hidden / 4, nv = quads_per_thread(b.m, nq), t = quad_threads(nq, nv);
	auto go = [&](auto kernel) { launch_pdl(kernel, dim3(b.m), dim3(t), 0, st, b, d, h.c_ctx); };
	if (nv == 1) go(k_ctx_funnel<1>);
	else if (nv == 4) go(k_ctx_funnel<4>);
	else go(k_ctx_funnel<8>);
}
void launch_res(const RowBatch& b, const Dims& d, const ResSite& a, cudaStream_t st) {
	const int nq = d.hidden / 4, nv = quads_per_thread(b.m, nq), t = quad_threads(nq, nv);
	const size_t sm = general_smem_bytes(d.hidden);
	auto go = [&](auto kernel) { launch_pdl(kernel, dim3(b.m), dim3(t), sm, st, b, d, a); };
	// (two blocks of up to 384 threads leave 85 registers per thread, two of 512 only 64, which spill)
	if (nv == 1 && t <= 384) b.wide64 ? go(k_res<1, 384, true>) : go(k_res<1, 384, false>);
	else if (nv == 1) b.wide64 ? go(k_res<1, 512, true>) : go(k_res<1, 512, false>);
	else if (nv == 4) b.wide64 ? go(k_res<4, 512, true>) : go(k_res<4, 512, false>);
	else b.wide64 ? go(k_res<8, 512, true>) : go(k_res<8, 512, false>);
}
// the widest activation row: eight blocks of 352 threads with five quads each
constexpr int kActBlocks = 8, kActQuads = 5, kActBlockThreads = 352;
static int act_many_smem(int nq) { return 16 * (2 * kActStages * kActWorkers + nq); }
constexpr int kActManySmemMax = 200 * 1024;
void launch_act(const RowBatch& b, const Dims& d, const LayerDev& h, const int32_t* silu, cudaStream_t st) {
	const int nq = d.inter / 4;
	// Many rows: from 512 on (28-layer model, whole prompt: 400 rows 3.77 ms against 3.71, 512 4.00 either way,
	// 1,024 6.05 against 6.30, 2,047 12.34 against 13.07). Five blocks per multiprocessor where three fit: what
	// the rows do not divide into evenly is then handed out as blocks leave (3: 6.26 at 1,024 rows; 14: 6.12).
	if (!b.wide64 && b.m >= 512 && act_many_smem(nq) <= kActManySmemMax) {
		const int smem = act_many_smem(nq), per_sm = 5;
		launch_pdl(k_act_many, dim3(std::min(b.m, per_sm * sm_count())), dim3(kActThreads), smem, st, b, d, h.c_gate, h.c_up, h.c_act, silu);
		return;
	}
	// blocks per row: as many (up to 8) as the multiprocessors hold at once, three each
	int blocks = 2;
	while (blocks < kActBlocks && b.m * blocks * 2 <= 3 * sm_count()) blocks *= 2;
	while (blocks < kActBlocks && quad_threads((nq + blocks - 1) / blocks, kActQuads) > kActBlockThreads) blocks *= 2;      // (very wide rows)
	const int per = (nq + blocks - 1) / blocks;
	const int nv = per <= 384 ? 1 : (per <= 2 * 384 ? 2 : 5);
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(blocks, b.m);
	cfg.blockDim = dim3(quad_threads(per, nv));
	cfg.stream = st;
	cudaLaunchAttribute attr[2];
	attr[0].id = cudaLaunchAttributeClusterDimension;
	attr[0].val.clusterDim.x = (unsigned)blocks;
	attr[0].val.clusterDim.y = 1;
	attr[0].val.clusterDim.z = 1;
	attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[1].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = attr;
	cfg.numAttrs = pdl_enabled() ? 2 : 1;
	RowBatch rb = b;
	rb.debug_withhold = exchange_debug_take(kExchangeAct);
	auto go = [&](auto kernel) { cudaLaunchKernelEx(&cfg, kernel, rb, d, h.c_gate, h.c_up, h.c_act, silu); };
	// Registers decide how many blocks a multiprocessor holds: 3 of 224 threads (8,960 elements in two blocks) or 2 of
	// 288 (11,008) with 80 each, one more with 72, which costs a few instructions. The dense form is the faster one
	// where the other leaves blocks for a second wave, whole prompts in ms, dense / other: 8,960 x 28 layers, 256 rows
	// 2.62 / 2.66, 300 3.29 / 3.33, 500 4.00 / 4.04; 11,008 x 4 layers, 215 rows 0.527 / 0.541, 350 0.688 / 0.699.
	// Where all blocks run at once anyway it is not: 215 rows of 8,960 2.558 / 2.528, 140 of 11,008 0.512 / 0.507.
	const int threads = quad_threads(per, nv), plain_per_sm = 65536 / (80 * threads), dense_per_sm = 65536 / (72 * threads);
	const bool dense = threads <= 288 && dense_per_sm > plain_per_sm && b.m * blocks > plain_per_sm * sm_count();
	if (nv == 1) b.wide64 ? go(k_act<1, true>) : go(k_act<1, false>);
	else if (nv == 2) b.wide64 ? go(k_act<2, true>) : go(k_act<2, false>);
	else if (b.wide64) go(k_act<5, true>);
	else if (dense) go(k_act<5, false, true>);
	else go(k_act<5, false>);
}
cudaError_t rows_configure(const Dims& d) {
	// Every kernel of a step asks for the same (largest) shared-memory carve-out as the
	// tensor-core GEMM between them, so consecutive launches never make the SMs re-split
	// their L1 / shared memory.
	// (The limit on dynamic shared memory is the kernel's, not the model's: the most there is, so that mapping
	// a narrow model does not take it from a wider one.)
	const int sm = 226 * 1024;
	if (general_smem_bytes(d.hidden) > (size_t)sm) return cudaErrorInvalidConfiguration;
	// (The hidden width needs no limit of its own here: 128 heads of 128 are 16,384, which eight quads on each of
	// 512 threads hold, and q, k and v together 20,480, which 640 hold.)
	if (quad_threads((d.inter / 4 + kActBlocks - 1) / kActBlocks, kActQuads) > kActBlockThreads) return cudaErrorInvalidConfiguration;
	cudaError_t e = cudaSuccess;
	auto set = [&](const void* f, bool dynamic) {
		if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
		if (e == cudaSuccess && dynamic) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
	};
	for (const void* f : {(const void*)k_begin<1>, (const void*)k_begin<4>, (const void*)k_begin<8>, (const void*)k_res<1, 384, false>,
	                      (const void*)k_res<1, 384, true>, (const void*)k_res<1, 512, false>, (const void*)k_res<1, 512, true>,
	                      (const void*)k_res<4, 512, false>, (const void*)k_res<4, 512, true>, (const void*)k_res<8, 512, false>,
	                      (const void*)k_res<8, 512, true>})
		set(f, true);
	for (const void* f : {(const void*)k_qkv_post<1, false, false>, (const void*)k_qkv_post<1, false, true>,
	                      (const void*)k_qkv_post<1, true, false>, (const void*)k_qkv_post<1, true, true>,
	                      (const void*)k_qkv_post<4, false, false>, (const void*)k_qkv_post<4, false, true>,
	                      (const void*)k_qkv_post<4, true, false>, (const void*)k_qkv_post<4, true, true>,
	                      (const void*)k_qkv_post<8, false, false>, (const void*)k_qkv_post<8, false, true>,
	                      (const void*)k_qkv_post<8, true, false>, (const void*)k_qkv_post<8, true, true>,
	                      (const void*)k_ctx_funnel<1>, (const void*)k_ctx_funnel<4>, (const void*)k_ctx_funnel<8>,
	                      (const void*)k_act<1, false>, (const void*)k_act<1, true>, (const void*)k_act<2, false>,
	                      (const void*)k_act<2, true>, (const void*)k_act<5, false>, (const void*)k_act<5, true>,
	                      (const void*)k_act<5, false, true>})
		set(f, false);
	set((const void*)k_act_many, false);
	if (e == cudaSuccess) e = cudaFuncSetAttribute(k_act_many, cudaFuncAttributeMaxDynamicSharedMemorySize, kActManySmemMax);
	return e;
}

}  // namespace sslm
