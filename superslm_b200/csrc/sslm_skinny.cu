// Linear layers of up to 256 rows (decode batches, short prompts) on the tensor cores, weights first.
//
//   out[m,n] = fold_n( sum_k x[m,k] * w[n,k] ) (+ LoRA delta), per-row max |out| per segment
//
// With few rows the weights are what moves, so they take the M side of tcgen05.mma (128 weight rows
// per tile, one TMEM lane each) and the activation rows, padded to NB = 16 .. 256, the N side: every
// weight byte passes through one multiprocessor once and the activation tile is as small as the batch.
// A lane owning an output channel also makes the epilogue cheap: fold constants in registers, 128
// contiguous bytes per store of a warp, one warp-reduce instruction per row for the row maximum.
//
// While the tiles are fewer than the multiprocessors, K is cut over the blocks of a thread-block
// cluster; a block parks nothing in memory, it sends each peer the accumulator rows that peer
// finishes (st.async into its shared memory) and finishes its own 128 / blocks rows.
//
// The weights are written by no kernel: a block requests its first weight tiles (all of them, at the
// layer widths of a decode step) before the dependency wait, while the row kernel in front runs.
// What remains behind the wait is the activation tile, the MMAs, the exchange and the epilogue.
// q/k/v, o, gate/up, down at the 1.5B widths, 64 rows (B200, in the chain): 7.1, 7.7, 12.0, 11.4 us with
// the activation-major tiles of sslm_gemm_tc.cu.
//
// The epilogues are short rolled loops and the three uses (int32 rows, int64 rows with adapters, the
// head) separate kernels: an epilogue runs once per launch, so what it costs is fetching its
// instructions. Unrolled over the columns with all uses inlined it took 0.5 us per row of x.
//
// Warp roles: warp 0 = TMA producer, warp 1 = TMEM owner + MMA issuer, the rest = epilogue (warp w
// reads TMEM lanes 32 (w % 4) .. +31; with eight of them, two share a lane quarter's columns).
// Every wait on an mbarrier is bounded; a wait that runs out marks the rows with an internal status
// and the block tears down normally.
#include <cuda.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "sslm_cluster.cuh"
#include "sslm_kernels.h"

namespace sslm {
namespace {

constexpr int kWRows = 128, kKBlock = 128, kMmaK = 32;
constexpr int kMaxStages = 12;

template <int NB>
struct SkCfg {
	// Four epilogue warps per 16 columns (each reads a quarter of the lanes), 16 at most: with eight, gate/up of 256 rows at
	// the 1.5B widths spent 8.5 of 14.5 us in its epilogue. A step of 120 rows 13.46 -> 13.05 ms / 5, of 21 rows of 0.5B
	// 18.8 -> 18.25 ms / 15. Eight for 32 columns, against four: a step of 20 to 32 rows of 0.5B 1,175 to 1,230 -> 1,130 to 1,165 us, with
	// adapters 1,821 to 1,865 -> 1,610 to 1,647, at the 1.5B widths the same within 2 % either way; by itself 2,048 x 2,048 10.9 -> 11.6 us, 8,960 x
	// 1,536 14.4 -> 13.3. Not for 64 columns: a clustered block of 16 leaves no registers for a second one beside
	// it (64 rows: 8 % slower), and without clusters it gains nothing.
	static constexpr int kEpiWarps = NB == 64 ? 8 : (NB / 4 < 16 ? NB / 4 : 16);
	static constexpr int kThreads = 64 + 32 * kEpiWarps;
	static constexpr uint32_t kWBytes = kWRows * kKBlock, kXBytes = NB * kKBlock, kStageBytes = kWBytes + kXBytes;
	static constexpr uint32_t kTmemCols = 2 * NB < 32 ? 32 : 2 * NB;      // two accumulator stages
	static constexpr uint32_t kExchangeBytes = kWRows * NB * 4;
	// s8 x s8 -> s32, both K-major, M = 128, N = NB
	static constexpr uint32_t kInstrDesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NB >> 3) << 17) | ((uint32_t)(kWRows >> 4) << 24);
};

__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
	asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) { return bounded_wait<false>(bar, parity); }
// K-major, 128-byte-swizzled operand tile: 8-row groups are 1024 bytes apart
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
	return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
	asm volatile(
	    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
	    ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
	asm volatile(
	    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
	    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
	      "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
	    : "r"(addr));
	asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Maxima of sixteen columns over the warp's lanes: halving exchanges, after which lane l holds column
// l / 2 (one shuffle per column instead of one warp reduction).
__device__ __forceinline__ uint32_t column_max16(uint32_t (&x)[16], int lane) {
#pragma unroll
	for (int half = 8; half > 0; half >>= 1) {
		const bool up = (lane & (2 * half)) != 0;
#pragma unroll
		for (int j = 0; j < half; ++j) {
			const uint32_t keep = up ? x[j + half] : x[j], give = up ? x[j] : x[j + half];
			x[j] = max(keep, __shfl_xor_sync(0xffffffffu, give, 2 * half));
		}
	}
	return max(x[0], __shfl_xor_sync(0xffffffffu, x[0], 1));
}
// the same for (value, channel) pairs, the lower channel winning ties
__device__ __forceinline__ void column_best16(uint32_t (&x)[16], int n, int lane, uint32_t& value, int& channel) {
	int at[16];
#pragma unroll
	for (int j = 0; j < 16; ++j) at[j] = n;
#pragma unroll
	for (int half = 8; half > 0; half >>= 1) {
		const bool up = (lane & (2 * half)) != 0;
#pragma unroll
		for (int j = 0; j < half; ++j) {
			const uint32_t keep = up ? x[j + half] : x[j], give = up ? x[j] : x[j + half];
			const int keep_at = up ? at[j + half] : at[j], give_at = up ? at[j] : at[j + half];
			const uint32_t o = __shfl_xor_sync(0xffffffffu, give, 2 * half);
			const int o_at = __shfl_xor_sync(0xffffffffu, give_at, 2 * half);
			const bool other = o > keep || (o == keep && o_at < keep_at);
			x[j] = other ? o : keep;
			at[j] = other ? o_at : keep_at;
		}
	}
	const uint32_t o = __shfl_xor_sync(0xffffffffu, x[0], 1);
	const int o_at = __shfl_xor_sync(0xffffffffu, at[0], 1);
	const bool other = o > x[0] || (o == x[0] && o_at < at[0]);
	value = other ? o : x[0];
	channel = other ? o_at : at[0];
}
__device__ __forceinline__ void send_quad(uint32_t local, uint32_t bar, uint32_t rank, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
	asm volatile(
	    "{\n\t.reg .b32 ra, rb;\n\tmapa.shared::cluster.u32 ra, %0, %2;\n\tmapa.shared::cluster.u32 rb, %1, %2;\n\t"
	    "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [ra], {%3, %4, %5, %6}, [rb];\n\t}"
	    ::"r"(local), "r"(bar), "r"(rank), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// One output channel: its fold, its segment, its row of the LoRA B matrix for the adapter last met.
struct Channel {
	int n, seg, first;      // channel, segment, first channel of the segment
	bool in, plain;
	int32_t idn, mult, shift;
	uint32_t half;
	const LoraLayerDev* lora;
	const int8_t* brow;
	int32_t df0, df1, df2;
};
__device__ __forceinline__ Channel channel_of(const LinearArgs& a, int n) {
	Channel c;
	c.n = n;
	c.in = n < a.N;
	c.seg = 0;
	while (c.seg + 1 < a.nseg && n >= a.seg_end[c.seg]) ++c.seg;
	c.first = c.seg ? a.seg_end[c.seg - 1] : 0;
	c.idn = 1;
	c.mult = c.shift = 0;
	if (a.fold != nullptr && c.in) {
		const int32_t* f = a.fold + (size_t)n * 3;
		c.idn = __ldg(f);
		c.mult = __ldg(f + 1);
		c.shift = __ldg(f + 2);
	}
	c.plain = a.fold != nullptr && fold_is_plain(c.idn, c.mult, c.shift);
	c.half = c.plain && c.shift > 0 ? 1u << (c.shift - 1) : 0u;
	c.lora = nullptr;
	c.brow = nullptr;
	c.df0 = c.df1 = c.df2 = 0;
	return c;
}
__device__ __forceinline__ int64_t lora_delta(const LinearArgs& a, Channel& c, int m) {
	const LoraLayerDev* ll = a.rows[m].lora;
	if (ll == nullptr || a.seg_lora[c.seg] < 0 || !c.in) return 0;
	const LoraLayerDev& L = ll[a.layer];
	if (c.lora != &L) {      // (rows of one adapter follow one another: its record is read once per channel)
		const LoraProjDev& p = L.p[a.seg_lora[c.seg]];
		c.lora = &L;
		c.brow = nullptr;
		if (p.a != nullptr) {
			const int nl = c.n - c.first;
			c.brow = p.b + (size_t)nl * L.rank;
			c.df0 = p.df[3 * nl];
			c.df1 = p.df[3 * nl + 1];
			c.df2 = p.df[3 * nl + 2];
		}
	}
	if (c.brow == nullptr) return 0;
	const int8_t* u = a.lora_u + ((size_t)m * 3 + c.seg) * kMaxLoraRank;
	int sum = 0;
	if ((L.rank & 3u) == 0u) {
		for (uint32_t t = 0; t < L.rank; t += 4) sum = __dp4a(*(const int*)(c.brow + t), *(const int*)(u + t), sum);
	} else {
		for (uint32_t t = 0; t < L.rank; ++t) sum += (int)c.brow[t] * (int)u[t];
	}
	return (int64_t)amp_fold(sum, c.df0, c.df1, c.df2);
}
// what a launch does with its accumulators
enum Mode { kRows32 = 0, kRows64, kHead };
// Folded accumulator (plus delta) of row m, stored; returns its magnitude for the row maximum, 0 for a
// channel beyond N or a row beyond M. (Magnitudes above 32 bits, possible with a delta, count as
// 2^32 - 1: the funnel refuses everything above 2^31.)
template <int MODE, bool PLAIN>
__device__ __forceinline__ uint32_t finish_value(const LinearArgs& a, Channel& c, int m, int32_t acc) {
	uint32_t mag;
	int32_t v32;
	if (PLAIN) {
		v32 = fold_plain(acc, c.mult, c.shift, c.half, &mag);
	} else {
		v32 = a.fold != nullptr ? fold(acc, c.idn, c.mult, c.shift) : acc;
		mag = v32 < 0 ? 0u - (uint32_t)v32 : (uint32_t)v32;
	}
	const bool keep = c.in && m < a.M;
	if (MODE == kRows32) {
		if (keep) ((int32_t*)a.out)[(size_t)m * a.out_ld + c.n] = v32;
	} else {
		int64_t v = v32;
		if (keep) {
			if (a.rows != nullptr) v += lora_delta(a, c, m);
			((int64_t*)a.out)[(size_t)m * a.out_ld + c.n] = v;
		}
		const unsigned long long ab = v < 0 ? (~(unsigned long long)v + 1ull) : (unsigned long long)v;
		mag = ab > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)ab;
	}
	return keep ? mag : 0u;
}

// (Clustered launches of up to 64 columns count on two blocks per multiprocessor: launch_mode cuts their rings for that. 32-bit rows
// compile to 96 registers and fewer; for 64-bit rows the compiler is told, left to itself it takes 128 to 168: steps of 24 and 48 rows
// with adapters 2.36 and 2.58 ms at the 1.5B widths, 2.15 and 2.34 so, 24 rows with four epilogue warps of 128 registers 2.16.)
template <int NB, int MODE>
__global__ void __launch_bounds__(SkCfg<NB>::kThreads, MODE == kRows64 && NB <= 64 ? 2 : 1)
k_skinny(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, LinearArgs a, int stages, int splits) {
	using Cfg = SkCfg<NB>;
	constexpr int kEpi = 32 * Cfg::kEpiWarps;
	extern __shared__ unsigned char smem_raw[];
	const uint32_t raw = cta_addr(smem_raw);
	const uint32_t base = (raw + 1023u) & ~1023u;            // swizzled tiles want 1024-byte alignment
	unsigned char* smem = smem_raw + (base - raw);
	int32_t* xch = (int32_t*)(smem + (size_t)stages * Cfg::kStageBytes);      // (splits > 1) rows to finish: [source][NB / 4][128 / splits][4]
	__shared__ __align__(8) unsigned long long s_bars[2 * kMaxStages + 5];
	__shared__ uint32_t s_tmem;
	__shared__ volatile int s_timeout;
	__shared__ uint32_t s_max[NB];                 // row maxima of the segment at hand
	__shared__ unsigned long long s_best[MODE == kHead ? NB : 1];
	const uint32_t bars = cta_addr(s_bars);
	auto full_bar = [&](int s) { return bars + 8u * s; };
	auto empty_bar = [&](int s) { return bars + 8u * (kMaxStages + s); };
	auto accf_bar = [&](int s) { return bars + 8u * (2 * kMaxStages + s); };
	auto acce_bar = [&](int s) { return bars + 8u * (2 * kMaxStages + 2 + s); };
	const uint32_t xch_bar = bars + 8u * (2 * kMaxStages + 4);

	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int kblocks = (a.K + kKBlock - 1) / kKBlock;
	const int tiles = (a.N + kWRows - 1) / kWRows;
	// this block's work: with splits, one tile and a slice of its k-blocks; without, every gridDim.x-th tile
	const int rank = splits > 1 ? (int)cluster_rank() : 0;
	const int tile0 = splits > 1 ? (int)blockIdx.x / splits : (int)blockIdx.x;
	const int tile_step = splits > 1 ? tiles : (int)gridDim.x;
	const int kb0 = rank * kblocks / splits, kb1 = (rank + 1) * kblocks / splits, nkb = kb1 - kb0;
	const int ntiles = tile0 < tiles ? (tiles - tile0 + tile_step - 1) / tile_step : 0;
	const int total = ntiles * nkb;                          // stages this block consumes

	// The channel that a thread of a clustered block's epilogue finishes, its fold constants asked for ahead of the weights:
	// behind the exchange the load took half a microsecond, and behind the weights it holds up the dependency wait.
	Channel c{};
	if (warp >= 2 && splits > 1) c = channel_of(a, tile0 * kWRows + rank * (kWRows / splits) + ((int)threadIdx.x - 64) % (kWRows / splits));
	if (threadIdx.x == 0) {
		for (int s = 0; s < stages; ++s) {
			bar_init(full_bar(s), 1);
			bar_init(empty_bar(s), 1);
		}
		for (int s = 0; s < 2; ++s) {
			bar_init(accf_bar(s), 1);
			bar_init(acce_bar(s), Cfg::kEpiWarps);
		}
		s_timeout = 0;
		if (splits > 1) exchange_init(xch_bar, Cfg::kExchangeBytes + (a.debug_withhold == 2 && blockIdx.x == 0 ? 4 : 0));
		exchange_fence_init();
		// the first weight tiles: no kernel writes weights, so they need not wait for anybody
		const int early = total < stages ? total : stages;
		int t = tile0, kb = kb0;
		for (int i = 0; i < early; ++i) {
			bar_expect(full_bar(i), Cfg::kStageBytes);
			// (tests of the bounded waits leave the first request out, once)
			if (!(a.debug_withhold == 1 && blockIdx.x == 0 && i == 0))
				tma_2d(base + i * Cfg::kStageBytes, &map_w, full_bar(i), kb * kKBlock, t * kWRows);
			if (++kb == kb1) { kb = kb0; t += tile_step; }
		}
	}
	for (int i = threadIdx.x; i < NB; i += Cfg::kThreads) {
		s_max[i] = 0u;
		if (MODE == kHead) s_best[i] = 0ull;
	}
	if (warp == 1) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(cta_addr(&s_tmem)), "r"(Cfg::kTmemCols));
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	if (splits > 1) {
		cluster_arrive();
		cluster_wait();
	}
	const uint32_t tmem = s_tmem;
	bool all_in = true;      // (false: a peer may still be sending)

	if (warp == 0) {
		if (lane == 0) {
			// from here on the kernel reads what earlier kernels wrote
			pdl_wait();
			pdl_release();
			int t = tile0, kb = kb0;
			for (int i = 0; i < total && s_timeout == 0; ++i) {
				const int s = i % stages;
				if (i >= stages) {
					if (!bar_wait(empty_bar(s), (uint32_t)(i / stages + 1) & 1u)) { s_timeout = 1; break; }
					bar_expect(full_bar(s), Cfg::kStageBytes);
					tma_2d(base + s * Cfg::kStageBytes, &map_w, full_bar(s), kb * kKBlock, t * kWRows);
				}
				tma_2d(base + s * Cfg::kStageBytes + Cfg::kWBytes, &map_x, full_bar(s), kb * kKBlock, 0);
				if (++kb == kb1) { kb = kb0; t += tile_step; }
			}
		}
	} else if (warp == 1) {
		if (lane == 0) {
			int i = 0;
			for (int tc = 0; tc < ntiles && s_timeout == 0; ++tc) {
				const uint32_t as = tc & 1u;
				if (!bar_wait(acce_bar(as), (((uint32_t)tc >> 1) & 1u) ^ 1u)) { s_timeout = 1; break; }
				asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				for (int k = 0; k < nkb; ++k, ++i) {
					const int s = i % stages;
					if (!bar_wait(full_bar(s), (uint32_t)(i / stages) & 1u)) {
						// the flag must be up before the commit below lets the epilogue look at this tile
						s_timeout = 1;
						__threadfence_block();
						break;
					}
					asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
					const uint64_t dw = smem_desc(base + s * Cfg::kStageBytes), dx = smem_desc(base + s * Cfg::kStageBytes + Cfg::kWBytes);
#pragma unroll
					for (int j = 0; j < kKBlock / kMmaK; ++j)      // (+32 bytes inside the swizzle atom: +2 descriptor units)
						mma_i8(tmem + as * NB, dw + (uint64_t)(2 * j), dx + (uint64_t)(2 * j), Cfg::kInstrDesc, (k | j) != 0 ? 1u : 0u);
					mma_commit(empty_bar(s));
				}
				mma_commit(accf_bar(as));
			}
		}
	} else {
		const int q = warp & 3, part = (warp - 2) >> 2, et = (int)threadIdx.x - 64;
		constexpr int kCols = NB / (Cfg::kEpiWarps / 4);          // columns (rows of x) this warp takes
		const int col0 = part * kCols;
		auto refuse = [&]() {      // (by a whole warp, for all rows)
			for (int m = lane; m < a.M; m += 32) {
				if (a.status != nullptr) atomicCAS(&a.status[m], 0, (int32_t)kInternalWaitTimeout);
				else if (a.rowmax != nullptr) atomicMax(&a.rowmax[(size_t)m * 4], kRowmaxTimeout);
			}
		};
		if (splits == 1) c = channel_of(a, tile0 * kWRows + q * 32 + lane);      // (not ahead of the block's set-up, which would wait for it)
		pdl_wait();
		if (splits > 1) {
			// ---- one tile: send every peer the accumulator rows it finishes, finish 128 / splits of them
			const int rows = kWRows / splits;
			const bool acc_ok = bar_wait(accf_bar(0), 0) && s_timeout == 0;
			asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
			const int wrow = q * 32 + lane;
			const uint32_t to = (uint32_t)(wrow / rows), slot = (uint32_t)(wrow % rows);
#pragma unroll 1
			for (int c0 = 0; c0 < kCols; c0 += 16) {
				uint32_t r[16];
				tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + col0 + c0, r);
#pragma unroll
				for (int j = 0; j < 16; j += 4) {
					const uint32_t unit = ((uint32_t)rank * (NB / 4) + (uint32_t)((col0 + c0 + j) >> 2)) * (uint32_t)rows + slot;
					send_quad(cta_addr(xch) + 16u * unit, xch_bar, to, r[j], r[j + 1], r[j + 2], r[j + 3]);
				}
			}
			const bool ok = exchange_wait(xch_bar);
			all_in = ok;
			if (!__all_sync(0xffffffffu, acc_ok && ok)) refuse();      // (what was sent for a tile given up on is garbage: the rows say so)
			const int my = et % rows;          // (rows divides 128 and the epilogue's thread count: one channel per thread)
			const int first = tile0 * kWRows + rank * rows;
			const bool one_seg = a.nseg == 1 || channel_of(a, first).seg == channel_of(a, min(first + rows, a.N) - 1).seg;
			const int group = rows < 32 ? rows : 32;      // lanes that hold neighbouring channels of the same row
			auto finish = [&](auto plain) {
#pragma unroll 1
				for (int unit = et; unit < rows * (NB / 4); unit += kEpi) {
					const int m0 = (unit / rows) * 4;
					if (((unit - lane) / rows) * 4 >= a.M) break;      // (the warp's first lane decides: later units lie higher)
					int4 sum = make_int4(0, 0, 0, 0);
					for (int s = 0; s < splits; ++s) {
						const int4 p = *(const int4*)&xch[4 * (((size_t)s * (NB / 4) + (m0 >> 2)) * rows + my)];
						sum.x += p.x; sum.y += p.y; sum.z += p.z; sum.w += p.w;
					}
					const int v[4] = {sum.x, sum.y, sum.z, sum.w};
					uint32_t mag[4];
#pragma unroll
					for (int j = 0; j < 4; ++j) mag[j] = finish_value<MODE, decltype(plain)::value>(a, c, m0 + j, v[j]);
					if (one_seg)
						for (int o = 1; o < group; o <<= 1)
#pragma unroll
							for (int j = 0; j < 4; ++j) mag[j] = max(mag[j], __shfl_xor_sync(0xffffffffu, mag[j], o));
					if (a.rowmax != nullptr && a.seg_slot[c.seg] >= 0 && (!one_seg || (lane & (group - 1)) == 0))
#pragma unroll
						for (int j = 0; j < 4; ++j)
							if (mag[j] != 0u) atomicMax(&a.rowmax[(size_t)(m0 + j) * 4 + a.seg_slot[c.seg]], (unsigned long long)mag[j]);
				}
			};
			if (__all_sync(0xffffffffu, c.plain || !c.in)) finish(std::true_type());
			else finish(std::false_type());
		} else {
			// ---- whole tiles: a lane's channel, this warp's columns. Row maxima (arg-max keys) gather in shared
			// memory over the block's tiles and join the global ones at the end, or when the segment changes.
			auto flush = [&](int seg) {
				asm volatile("bar.sync 1, %0;" ::"n"(kEpi) : "memory");
				for (int m = et; m < NB && m < a.M; m += kEpi) {
					if (a.rowmax != nullptr && a.seg_slot[seg] >= 0 && s_max[m] != 0u)
						atomicMax(&a.rowmax[(size_t)m * 4 + a.seg_slot[seg]], (unsigned long long)s_max[m]);
					s_max[m] = 0u;
				}
				asm volatile("bar.sync 1, %0;" ::"n"(kEpi) : "memory");
			};
			int seg = channel_of(a, tile0 * kWRows).seg;      // the segment s_max holds (the same for every warp)
			for (int tc = 0; tc < ntiles; ++tc) {
				const uint32_t as = tc & 1u;
				const int n0 = (tile0 + tc * tile_step) * kWRows;
				bool one_seg = true;
				if (MODE != kHead && a.nseg > 1) {
					const int s0 = channel_of(a, n0).seg;
					one_seg = channel_of(a, min(n0 + kWRows, a.N) - 1).seg == s0;
					if (s0 != seg) {
						flush(seg);
						seg = s0;
					}
				}
				if (tc != 0) c = channel_of(a, n0 + q * 32 + lane);
				const bool acc_ok = __all_sync(0xffffffffu, (s_timeout == 0 && bar_wait(accf_bar(as), ((uint32_t)tc >> 1) & 1u) && s_timeout == 0) ? 1 : 0) != 0;
				asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				if (!acc_ok) {      // (not the tile's accumulators: the rows say so; the loop goes on so that all warps flush alike)
					s_timeout = 1;
					refuse();
				}
				auto columns = [&](auto plain) {
#pragma unroll 1
					for (int c0 = 0; c0 < kCols && col0 + c0 < a.M; c0 += 16) {
						uint32_t r[16];
						tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + as * NB + col0 + c0, r);
						const int mine = col0 + c0 + (lane >> 1);      // the row whose maximum this lane ends up with
						if (MODE == kHead) {
							if (a.row_mask != nullptr) {
								// lane j fetches the mask word of row j for this warp's 32 channels
								uint32_t allowed = 0xFFFFFFFFu;
								const int m = col0 + c0 + lane, w0 = (n0 + q * 32) >> 3;
								if (lane < 16 && m < a.M) {
									const uint8_t* page = a.row_mask[m];
									if (page != nullptr) {
										const int last = (a.N + 7) >> 3;
										allowed = 0u;
#pragma unroll
										for (int b = 0; b < 4; ++b)
											if (w0 + b < last) allowed |= (uint32_t)__ldg(page + w0 + b) << (8 * b);
									}
								}
#pragma unroll
								for (int j = 0; j < 16; ++j)
									if (!((__shfl_sync(0xffffffffu, allowed, j) >> lane) & 1u)) r[j] = 0x80000000u;      // INT32_MIN
							}
							if (a.logits != nullptr) {
#pragma unroll
								for (int j = 0; j < 16; ++j)
									if (col0 + c0 + j < a.M && c.in) a.logits[(size_t)(col0 + c0 + j) * a.N + c.n] = (int32_t)r[j];
							}
							// greedy argmax key, lowest index wins ties
#pragma unroll
							for (int j = 0; j < 16; ++j) r[j] = c.in ? r[j] ^ 0x80000000u : 0u;
							uint32_t value;
							int channel;
							column_best16(r, c.n, lane, value, channel);
							if ((lane & 1) == 0 && mine < a.M && channel < a.N)
								atomicMax(&s_best[mine], ((unsigned long long)value << 32) | (0xFFFFFFFFu - (uint32_t)channel));
						} else {
#pragma unroll
							for (int j = 0; j < 16; ++j) r[j] = finish_value<MODE, decltype(plain)::value>(a, c, col0 + c0 + j, (int32_t)r[j]);
							if (one_seg) {
								const uint32_t top = column_max16(r, lane);
								if ((lane & 1) == 0 && top != 0u) atomicMax(&s_max[mine], top);
							} else if (a.rowmax != nullptr && a.seg_slot[c.seg] >= 0) {
#pragma unroll
								for (int j = 0; j < 16; ++j)
									if (r[j] != 0u) atomicMax(&a.rowmax[(size_t)(col0 + c0 + j) * 4 + a.seg_slot[c.seg]], (unsigned long long)r[j]);
							}
						}
					}
				};
				if (acc_ok) {
					if (MODE == kHead || __all_sync(0xffffffffu, c.plain || !c.in)) columns(std::true_type());
					else columns(std::false_type());
				}
				asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
				__syncwarp();
				if (lane == 0) bar_arrive(acce_bar(as));      // the accumulators may be overwritten
			}
			if (MODE == kHead) {
				asm volatile("bar.sync 1, %0;" ::"n"(kEpi) : "memory");
				for (int m = et; m < NB && m < a.M; m += kEpi)
					if (s_best[m] != 0ull) atomicMax(&a.best[m], s_best[m]);
			} else {
				flush(seg);
			}
		}
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	if (warp == 1) {
		asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::kTmemCols));
	}
	if (__builtin_expect(!__all_sync(0xffffffffu, all_in), 0)) exchange_leave(xch_bar, 1);
}

// How a launch is cut. K slices (the blocks of a cluster): as many, up to 8, as still fit on the
// multiprocessors at once and leave each at least one k-block -- every slice shortens the block's
// stream and its MMAs, and the exchange costs under a microsecond. Ring stages: all of the block's
// k-blocks when they fit, so that its whole weight stream is requested ahead of the wait.
template <int NB, int MODE>
bool launch_mode(const LinearArgs& a_in, cudaStream_t st, int* reason) {
	using Cfg = SkCfg<NB>;
	LinearArgs a = a_in;
	static PerDeviceOnce configured;
	// dynamic share of the 227 KB, beside the barriers and the row words
	constexpr int kSmemMax = 227 * 1024 - ((2 * kMaxStages + 5) * 8 + NB * 4 + (MODE == kHead ? NB * 8 : 8) + 256);
	if (once_per_device(configured, [] {
		    cudaError_t e = cudaFuncSetAttribute(k_skinny<NB, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
		    if (e != cudaSuccess) return e;
		    return cudaFuncSetAttribute(k_skinny<NB, MODE>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
	    }) != cudaSuccess) {
		*reason = 2;
		return false;
	}
	CUtensorMap mw, mx;
	if (!tc_tensor_map(a.w, a.N, a.K, kWRows, a.caller_memory == 0, &mw) || !tc_tensor_map(a.x, a.M, a.K, NB, a.caller_memory == 0, &mx)) {
		*reason = 4;
		return false;
	}
	const int tiles = (a.N + kWRows - 1) / kWRows, kblocks = (a.K + kKBlock - 1) / kKBlock, sms = sm_count();
	int splits = 1;
	if (a.best == nullptr)
		while (splits < 8 && tiles * splits * 2 <= sms && splits * 2 <= kblocks) splits *= 2;
	// The exchange moves 512 bytes per row of x and block: beyond 64 rows it costs more than the
	// activation-major kernel's K slices through L2, except with few tiles and a long K (measured at 128
	// rows: o 8.2 against 8.4 us, down 11.5 against 12.7, but q/k/v, whose sixteen clusters no longer fit
	// side by side, 14.8 against 8.6; at 256 rows 12.2 against 8.6, 16.6 against 15.2). Without slices
	// (gate/up, the head) this kernel is the faster one at every size: 16.1 against 17.6 us at 256 rows.
	if (splits > 1 && NB > 64 && (NB > 128 || tiles > 14)) {
		*reason = 0;
		return false;
	}
	const int nkb = (kblocks + splits - 1) / splits;
	const int per_block = splits > 1 ? nkb : nkb * ((tiles + sms - 1) / sms);
	const size_t fixed = 1024 + (splits > 1 ? Cfg::kExchangeBytes : 0);
	int stages = (int)((kSmemMax - fixed) / Cfg::kStageBytes);
	stages = stages > kMaxStages ? kMaxStages : stages;
	// In clusters, no more than lets two blocks share a multiprocessor: sixteen clusters of eight blocks that take one
	// each do not fit side by side, nor thirty-six of four (the last ones ran alone: K = 11,008 and 2,048 channels,
	// 2 rows 22.6 us in place of 14.4, 64 rows 24.7 / 16.5; 4,608 channels 28.9 / 18.5), and where the clusters fit
	// anyway the shallower ring is as fast (7 to 15 tiles: 0.88 to 1.00 of the time).
	constexpr int kShare = 113 * 1024 - 1024 - (int)((2 * kMaxStages + 5) * 8 + NB * 4 + 8 + 256);
	const int shared = (kShare - (int)fixed) / (int)Cfg::kStageBytes;
	if (splits > 1 && shared >= 2 && stages > shared) stages = shared;
	if (stages > per_block) stages = per_block;
	if (stages < 1) {
		*reason = 2;
		return false;
	}
	a.debug_withhold = tc_debug_take() ? 1 : (splits > 1 && exchange_debug_take(kExchangeLinear) ? 2 : 0);
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = dim3(splits > 1 ? tiles * splits : (tiles < sms ? tiles : sms));
	cfg.blockDim = dim3(Cfg::kThreads);
	cfg.dynamicSmemBytes = fixed + (size_t)stages * Cfg::kStageBytes;
	cfg.stream = st;
	cudaLaunchAttribute attr[2];
	int n = 0;
	if (pdl_enabled() && a.caller_memory == 0) {
		attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
		attr[n++].val.programmaticStreamSerializationAllowed = 1;
	}
	if (splits > 1) {
		attr[n].id = cudaLaunchAttributeClusterDimension;
		attr[n].val.clusterDim.x = (unsigned)splits;
		attr[n].val.clusterDim.y = 1;
		attr[n++].val.clusterDim.z = 1;
	}
	cfg.attrs = attr;
	cfg.numAttrs = n;
	if (cudaLaunchKernelEx(&cfg, k_skinny<NB, MODE>, mw, mx, a, stages, splits) != cudaSuccess) {
		*reason = 5;
		return false;
	}
	return true;
}

}  // namespace

bool launch_linear_skinny(const LinearArgs& a, cudaStream_t st) {
	auto launch = [&](auto nb, int* reason) {
		constexpr int NB = decltype(nb)::value;
		if (a.best != nullptr) return launch_mode<NB, kHead>(a, st, reason);
		return a.out64 ? launch_mode<NB, kRows64>(a, st, reason) : launch_mode<NB, kRows32>(a, st, reason);
	};
	if (a.best != nullptr && a.fold != nullptr) return false;      // (no caller folds logits)
	if (a.M < 1 || a.M > 256) return false;
	int reason = 0;
	bool ok = false;
	if (a.K % 16 != 0 || ((uintptr_t)a.x & 15) || ((uintptr_t)a.w & 15)) reason = 1;
	else if (a.M <= 16) ok = launch(std::integral_constant<int, 16>(), &reason);
	else if (a.M <= 32) ok = launch(std::integral_constant<int, 32>(), &reason);
	else if (a.M <= 64) ok = launch(std::integral_constant<int, 64>(), &reason);
	else if (a.M <= 128) ok = launch(std::integral_constant<int, 128>(), &reason);
	else ok = launch(std::integral_constant<int, 256>(), &reason);
	if (ok || reason != 0) tc_count(ok, reason);      // (reason 0: the other kernel is the better one here)
	return ok;
}

}  // namespace sslm
