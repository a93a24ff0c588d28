// Linear layers of a few rows: a whole projection's weights wait in shared memory.
//
//   out[m,n] = fold_n( sum_k x[m,k] * w[n,k] ) (+ LoRA delta), per-row max |out| per segment
//
// The weights are written by no kernel, so every warp asks for its share of them -- 16 weight rows, a range of K in
// blocks of 128 bytes (TMA, 128-byte swizzle) -- before the dependency wait, while the row kernel in front runs.
// What is left behind the wait is short: the rows of x into shared memory, four multiplications a block
// (mma.sync m16n8k32 s8, fragments by ldmatrix: the weights are the A operand, eight rows of x the B operand, so
// eight rows cost what one does), one exchange of partial sums between the warps that share the 16 rows, the fold.
// Bound by the weights' way into shared memory (gate/up: 27.7 MB, 13 us cold, 9.6 in the chain, where it begins a kernel
// earlier) and by the latencies of that chain (issue slots 7 to 12 % used).
//
// Five rows at the 1.5B widths, behind the wait, on the weights-first tcgen05 kernel (k_skinny) / here: q/k/v 3.1 / 2.7 us,
// o 3.5 / 3.1, gate/up 5.5 / 5.9 (but the row kernel in front 5.4 / 2.9, which its weights no longer crowd out),
// down 5.9 / 3.6; a step 1.43 ms / 1.29. One row is no faster than through k_gemv's rings (0.5B: 4 % slower), and from nine
// rows on a second set of multiplications costs what it gains (12 rows: 2 to 4 % slower; 21 rows of 0.5B: 18 %).
// Weights in registers instead of shared memory (20 % slower): loads that are still out hold up the dependency wait.
// (GemmInt8AccumulateRow + ApplyWeightScaleFold + AddAmplifyingLoraDelta,
//  src/matmul.cpp:455-464, src/forward/forward_sites.cpp:461-470, :1051-1103.)
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <initializer_list>

#include "sslm_cluster.cuh"
#include "sslm_kernels.h"

namespace sslm {
namespace {

constexpr int kFewRows = 8, kTileRows = 16, kBlockBytes = 128, kBoxBytes = kTileRows * kBlockBytes, kMaxWarps = 16;

struct FewPlan {
	int warps_k;      // warps that share 16 weight rows
	int blocks_k;     // 128-byte blocks of K each of them takes
	int tiles;        // of 16 weight rows per block
	int x_stride;     // bytes between rows of x in shared memory (16 more than a multiple of 128: no bank conflicts)
};

__device__ __forceinline__ void copy4(uint32_t dst, const void* src) {
	asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void mma_s8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
	asm volatile(
	    "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
	    : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
	    : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the delta of channel nl of segment seg for row m, AddAmplifyingLoraDelta's second half
__device__ __noinline__ int64_t lora_delta(const LinearArgs& a, int m, int seg, int nl) {
	const LoraLayerDev* ll = a.rows[m].lora;
	if (ll == nullptr) return 0;
	const LoraLayerDev& L = ll[a.layer];
	const LoraProjDev& pj = L.p[a.seg_lora[seg]];
	if (pj.a == nullptr) return 0;
	const int8_t* brow = pj.b + (size_t)nl * L.rank;
	const int8_t* u = a.lora_u + ((size_t)m * 3 + seg) * kMaxLoraRank;
	int sum = 0;
	if ((L.rank & 3u) == 0u) {
		for (uint32_t r = 0; r < L.rank; r += 4) sum = __dp4a(*(const int*)(brow + r), *(const int*)(u + r), sum);
	} else {
		for (uint32_t r = 0; r < L.rank; ++r) sum += (int)brow[r] * (int)u[r];
	}
	return (int64_t)amp_fold(sum, pj.df[3 * nl], pj.df[3 * nl + 1], pj.df[3 * nl + 2]);
}

__global__ void __launch_bounds__(32 * kMaxWarps, 1)
k_linear_few(const __grid_constant__ CUtensorMap map_w, LinearArgs a, FewPlan p) {
	extern __shared__ unsigned char smem_raw[];      // per warp: its weights; then the rows of x
	__shared__ uint32_t s_max[kFewRows * 3];
	__shared__ __align__(8) unsigned long long s_bars[kMaxWarps];
	__shared__ int32_t s_fold[kMaxWarps * kTileRows * 3];
	__shared__ int s_timeout;
	const uint32_t raw = cta_addr(smem_raw), base = (raw + 1023u) & ~1023u;      // swizzled boxes want 1024-byte alignment
	const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
	const int K = a.K, tile = warp / p.warps_k, kb0 = (warp - tile * p.warps_k) * p.blocks_k;
	const int first = blockIdx.x * p.tiles * kTileRows;      // the block's first channel
	const int n0 = first + tile * kTileRows;
	const int nkb = n0 < a.N ? max(0, min(p.blocks_k, (K + kBlockBytes - 1) / kBlockBytes - kb0)) : 0;
	const uint32_t mine = base + (uint32_t)(warp * p.blocks_k) * kBoxBytes, bar = cta_addr(&s_bars[warp]);
	// The block's fold rows, asked for ahead of the weights: behind them they came late, and a load that is still
	// out holds up the dependency wait.
	const int channels = p.tiles * kTileRows;
	for (int i = t; i < 3 * channels; i += blockDim.x)
		if (first + i / 3 < a.N) copy4(cta_addr(s_fold + i), a.fold + (size_t)first * 3 + i);
	__syncthreads();
	if (lane == 0 && nkb > 0) {
		asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
		asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)(nkb * kBoxBytes)) : "memory");
		// (tests of the bounded waits leave one request out)
		for (int i = a.debug_withhold != 0 && (blockIdx.x | warp) == 0 ? 1 : 0; i < nkb; ++i) tma_2d(mine + i * kBoxBytes, &map_w, bar, (kb0 + i) * kBlockBytes, n0);
	}
	// the channel this thread finishes (for every so manyth row), its segment and fold
	const int ch = t % channels, n = first + ch, step = 2 * p.warps_k;
	const int seg = (a.nseg > 1 && n >= a.seg_end[0] ? 1 : 0) + (a.nseg > 2 && n >= a.seg_end[1] ? 1 : 0);
	for (int i = t; i < kFewRows * 3; i += blockDim.x) s_max[i] = 0u;
	if (t == 0) s_timeout = 0;
	const uint32_t xs = base + (uint32_t)((blockDim.x >> 5) * p.blocks_k) * kBoxBytes;
	pdl_wait();
	pdl_release();
	for (int m = 0; m < a.M; ++m)
		for (int i = t; i < (K >> 4); i += blockDim.x) copy16(xs + (uint32_t)(m * p.x_stride + 16 * i), a.x + (size_t)m * K + 16 * i);
	asm volatile("cp.async.wait_all;" ::: "memory");
	__syncthreads();

	// (columns beyond the last row of x repeat it; bytes beyond K meet weights that are zero)
	int acc[4] = {0, 0, 0, 0};
	if (nkb > 0 && !__all_sync(0xffffffffu, bounded_wait<false>(bar, 0))) {
		s_timeout = 1;
		bounded_wait<false>(bar, 0);      // (boxes that are late must not land in a shared memory given up)
	} else {
		const int row = lane & 15;
		const uint32_t wrow = mine + (uint32_t)row * kBlockBytes, sw = (uint32_t)(row & 7), half = (uint32_t)lane >> 4;
		const uint32_t xr = xs + (uint32_t)(min(lane & 7, a.M - 1) * p.x_stride + kb0 * kBlockBytes + (lane >> 3) * 16);
#pragma unroll 2
		for (int k = 0; k < nkb; ++k) {
			uint32_t w[4][4], x0[4], x1[4];
#pragma unroll
			for (int s = 0; s < 4; ++s) ldmatrix4(wrow + (uint32_t)k * kBoxBytes + (((2u * s + half) ^ sw) << 4), w[s][0], w[s][1], w[s][2], w[s][3]);
			ldmatrix4(xr + (uint32_t)k * kBlockBytes, x0[0], x0[1], x0[2], x0[3]);
			ldmatrix4(xr + (uint32_t)k * kBlockBytes + 64u, x1[0], x1[1], x1[2], x1[3]);
			mma_s8(acc, w[0], x0[0], x0[1]);
			mma_s8(acc, w[1], x0[2], x0[3]);
			mma_s8(acc, w[2], x1[0], x1[1]);
			mma_s8(acc, w[3], x1[2], x1[3]);
		}
	}
	// lane (g, c) holds channels g (words 0, 1) and g + 8 (2, 3) of rows 2 c and 2 c + 1; the first of the warp's boxes
	// makes room for them
	__syncwarp();
	int32_t* const part = (int32_t*)(smem_raw + (mine - raw));
#pragma unroll
	for (int q = 0; q < 4; ++q) part[q * 32 + lane] = acc[q];
	__syncthreads();
	if (*(volatile int*)&s_timeout) {
		for (int m = t; m < a.M; m += blockDim.x) {
			if (a.status != nullptr) atomicCAS(&a.status[m], 0, (int32_t)kInternalWaitTimeout);
			else if (a.rowmax != nullptr) atomicMax(&a.rowmax[(size_t)m * 4], kRowmaxTimeout);
		}
		return;
	}

	const int r = ch & 15, apart = p.blocks_k * (kBoxBytes / 4);      // words between two warps' sums
	const int32_t* sums = (const int32_t*)(smem_raw + (base - raw)) + (size_t)(ch >> 4) * p.warps_k * apart + (r >> 3) * 64 + (r & 7) * 4;
	const int32_t f0 = s_fold[3 * ch], f1 = s_fold[3 * ch + 1], f2 = s_fold[3 * ch + 2];      // (beyond N: anything)
	const bool plain = fold_is_plain(f0, f1, f2);
	const uint32_t fhalf = plain && f2 > 0 ? 1u << (f2 - 1) : 0u;
#pragma unroll 1
	for (int m0 = 0; m0 < a.M; m0 += step) {
		const int m = m0 + t / channels;
		const bool in = m < a.M && n < a.N;
		uint32_t mag = 0;
		if (in) {
			const int32_t* q = sums + (m & 1) * 32 + (m >> 1);
			int32_t sum = 0;
#pragma unroll 4
			for (int s = 0; s < p.warps_k; ++s) sum += q[s * apart];
			int32_t v;
			if (plain) {
				v = fold_plain(sum, f1, f2, fhalf, &mag);
			} else {
				v = fold(sum, f0, f1, f2);
				mag = v < 0 ? 0u - (uint32_t)v : (uint32_t)v;
			}
			if (!a.out64) {
				((int32_t*)a.out)[(size_t)m * a.out_ld + n] = v;
			} else {
				int64_t v64 = v;
				if (a.rows != nullptr && a.seg_lora[seg] >= 0) v64 += lora_delta(a, m, seg, n - (seg ? a.seg_end[seg - 1] : 0));
				((int64_t*)a.out)[(size_t)m * a.out_ld + n] = v64;
				// (magnitudes above 32 bits count as 2^32 - 1: the funnel refuses everything above 2^31)
				const unsigned long long ab = v64 < 0 ? (~(unsigned long long)v64 + 1ull) : (unsigned long long)v64;
				mag = ab > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)ab;
			}
		}
		// the 16 lanes of a tile hold one row; where a segment ends inside a tile every lane speaks for itself
		const bool one_seg = __all_sync(0xffffffffu, __shfl_sync(0xffffffffu, seg, lane & 16) == seg);
		if (one_seg) {
#pragma unroll
			for (int o = 8; o > 0; o >>= 1) mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, o));
			if ((lane & 15) != 0) mag = 0u;
		}
		if (mag != 0u) atomicMax(&s_max[m * 3 + seg], mag);
	}
	if (a.rowmax == nullptr) return;
	__syncthreads();
	for (int i = t; i < a.M * 3; i += blockDim.x) {
		const int slot = a.seg_slot[i % 3];
		if (s_max[i] != 0u && slot >= 0) atomicMax(&a.rowmax[(size_t)(i / 3) * 4 + slot], (unsigned long long)s_max[i]);
	}
}

constexpr int kSmemMax = 220 * 1024;
// what a block takes beside its dynamic shared memory, as compiled: registers of a warp (given out in units of 256), shared memory
struct FewCost {
	std::atomic<int> warp_regs, fixed_smem;
};

bool launch(LinearArgs& a, cudaStream_t st) {
	static PerDeviceOnce configured;
	static FewCost costs[kMaxDevices];
	FewCost& cost = costs[current_device_ordinal()];
	if (once_per_device(configured, [&cost] {
		    cudaFuncAttributes f;
		    cudaError_t e = cudaFuncGetAttributes(&f, k_linear_few);
		    if (e == cudaSuccess) {
			    cost.warp_regs = (f.numRegs * 32 + 255) / 256 * 256;
			    cost.fixed_smem = (int)f.sharedSizeBytes + 1024;      // (1 KB is the system's)
		    }
		    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_linear_few, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax);
		    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_linear_few, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
		    return e;
	    }) != cudaSuccess)
		return false;
	// The fewest tiles per block with which all blocks run at once (a second wave of 100 KB blocks began 6 us after the first)
	// beside those of the row kernel in front, which has a block per row and may still hold a multiprocessor each.
	const int kblocks = (a.K + kBlockBytes - 1) / kBlockBytes, tiles = (a.N + kTileRows - 1) / kTileRows, sms = sm_count();
	for (int per = 1; per <= kMaxWarps; ++per) {
		FewPlan p;
		p.tiles = per;
		p.blocks_k = (kblocks + kMaxWarps / per - 1) / (kMaxWarps / per);
		p.warps_k = (kblocks + p.blocks_k - 1) / p.blocks_k;
		p.x_stride = p.warps_k * p.blocks_k * kBlockBytes + 16;
		const int warps = per * p.warps_k, blocks = (tiles + per - 1) / per;
		const int smem = 1024 + warps * p.blocks_k * kBoxBytes + a.M * p.x_stride;
		if (smem > kSmemMax) return false;
		const int resident = std::min({2, 228 * 1024 / (smem + cost.fixed_smem), 65536 / (cost.warp_regs * warps)});
		if (blocks > resident * sms - kFewRows) continue;
		// A projection by itself, its weights asked for ahead of nothing: two blocks on a multiprocessor pay from 1,280 columns
		// and 6,144 channels on. 2, 5, 8 rows, us with the weights-first kernel / here, funnel included: 2,048 x 8,192 12.3 / 12.3,
		// 13.7 / 12.3, 14.4 / 12.4; 1,280 x 6,144 12.3 / 10.3, 12.3 / 10.8, 12.3 / 12.3; below, 896 x 9,728 10.3 / 12.3, 10.8 / 12.3,
		// 11.9 / 12.3, 1,536 x 4,096 10.3 / 11.1, 10.3 / 12.1, 10.3 / 12.3. A block each: 1,536 x 17,920 14.4 / 13.4 to 14.4, and
		// 896 to 11,008 columns of 896 to 2,048 channels 8.2 to 14.4 / 8.2 to 11.8.
		if (a.caller_memory != 0 && blocks > sms && (a.K < 1280 || a.N < 6144)) return false;
		CUtensorMap map;
		if (!tc_tensor_map(a.w, a.N, a.K, kTileRows, a.caller_memory == 0, &map)) return false;
		a.debug_withhold = tc_debug_take() ? 1 : 0;
		if (launch_ordered(a.caller_memory == 0, k_linear_few, dim3(blocks), dim3(32 * warps), smem, st, map, a, p) != cudaSuccess) return false;
		tc_count_few();
		return true;
	}
	return false;
}

}  // namespace

bool launch_linear_few(const LinearArgs& a, cudaStream_t st) {
	if (a.M < 1 || a.M > kFewRows || a.K % 16 != 0 || ((uintptr_t)a.x & 15) || ((uintptr_t)a.w & 15) || a.best != nullptr || a.fold == nullptr)
		return false;
	LinearArgs armed = a;
	return launch(armed, st);
}

}  // namespace sslm
