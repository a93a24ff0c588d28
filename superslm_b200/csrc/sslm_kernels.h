// Launch interface of the CUDA kernels (host side). Every launcher enqueues on the given
// stream and returns immediately; errors surface through cudaGetLastError at the call
// site. Nothing here allocates.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>
#include <utility>

#include "sslm_types.cuh"

namespace sslm {

// ---- programmatic dependent launch
// A step is a chain of ~285 short dependent kernels. Each is launched with the programmatic
// stream-serialization attribute: its blocks may be placed on the SMs, and run whatever does
// not depend on earlier kernels (index arithmetic, barrier and tensor-memory set-up), while
// the previous kernel is still running. Every kernel calls pdl_wait() before its first access
// to global memory -- it returns once the previous kernel has completed and its writes are
// visible -- and then pdl_release(), which lets the NEXT kernel's blocks be placed. Releasing
// only after the wait keeps the look-ahead to one kernel. A kernel launched without the
// attribute (or after a memcpy / memset) sees both calls as no-ops and plain stream order.
#if defined(__CUDACC__)
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif
// SSLM_B200_PDL=0 in the environment turns the attribute off (plain stream order).
inline bool pdl_enabled() {
	static const bool on = [] {
		const char* e = getenv("SSLM_B200_PDL");
		return !(e && e[0] == '0');
	}();
	return on;
}
template <typename... KArgs, typename... Args>
cudaError_t launch_ordered(bool programmatic, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
	cudaLaunchConfig_t cfg = {};
	cfg.gridDim = grid;
	cfg.blockDim = block;
	cfg.dynamicSmemBytes = smem;
	cfg.stream = st;
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = attr;
	cfg.numAttrs = programmatic && pdl_enabled() ? 1 : 0;
	return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
	return launch_ordered(true, kernel, grid, block, smem, st, std::forward<Args>(args)...);
}

// ---- per-device one-time set-up
// cudaFuncSetAttribute and the device attributes apply to the CURRENT device only, and models may
// be mapped on several devices of one process (sslm_b200_set_device): everything a launcher sets
// up once is therefore kept per device ordinal. The set-up calls are idempotent, so two host
// threads racing through the first launch on a device at worst both make them.
constexpr int kMaxDevices = 64;
struct PerDeviceOnce {
	std::atomic<unsigned char> done[kMaxDevices];
};
inline int current_device_ordinal() {
	int dev = 0;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) dev = 0;
	return dev;
}
template <typename F>
cudaError_t once_per_device(PerDeviceOnce& o, F&& setup) {
	const int dev = current_device_ordinal();
	if (o.done[dev].load(std::memory_order_acquire)) return cudaSuccess;
	const cudaError_t e = setup();
	if (e == cudaSuccess) o.done[dev].store(1, std::memory_order_release);
	return e;
}
// multiprocessor count of the current device
inline int sm_count() {
	static std::atomic<int> cached[kMaxDevices];
	const int dev = current_device_ordinal();
	int v = cached[dev].load(std::memory_order_relaxed);
	if (v > 0) return v;
	if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v < 1) v = 148;
	cached[dev].store(v, std::memory_order_relaxed);
	return v;
}

// ---- tests of the bounded waits
// The next launch of one kernel that exchanges words over a cluster arms one of its exchanges, in block 0,
// with four bytes more than will come: that block's wait runs out. One word: 0 for none, else
// kernel << 8 | exchange + 1.
// (4 names no kernel; 5 is the fifth exchange of attention with the q/k/v site of biased rows inside)
enum ExchangeKernel { kExchangeLinear = 0, kExchangeAttnFew, kExchangeAttnChunk, kExchangeAct, kExchangeAttnSite = 5, kExchangeKernels };
inline std::atomic<uint32_t> g_withheld_exchange{0};
inline int exchange_debug_take(ExchangeKernel kernel) {
	uint32_t w = g_withheld_exchange.load(std::memory_order_relaxed);
	if (w == 0 || w >> 8 != (uint32_t)kernel || !g_withheld_exchange.compare_exchange_strong(w, 0)) return 0;
	return (int)(w & 0xFF);
}

// ---- per-row sites (sslm_rows.cu)
cudaError_t rows_configure(const Dims& d);
// (A layer's record travels in the launch parameters: read from memory, its pointers cost a kernel's prologue a trip to HBM
// before the next one could start.)
// first rows of a call: embed or resume, then an RMSNorm with `gain` (nullptr: none)
// (It enters the call's new pages into the page tables: when it is refused, nothing behind it may be launched.)
cudaError_t launch_begin(const RowBatch& b, const Dims& d, const int8_t* embed, Scale c_embed, const RowSource* src, const int8_t* gain,
                         Scale c_norm, int site_norm, cudaStream_t st);
inline std::atomic<int> g_refuse_begin{0};      // tests: the next launches of it that count as refused by the runtime
void launch_qkv_post(const RowBatch& b, const Dims& d, const LayerDev& h, int layer_index, KvPoolDev pool,
                     const int32_t* cos, const int32_t* sin, cudaStream_t st);
void launch_ctx_funnel(const RowBatch& b, const Dims& d, const LayerDev& h, cudaStream_t st);
// A residual site: funnel of the projection row, reconciliation with the stream, and the RMSNorm of
// whatever comes next.
struct ResSite {
	const int8_t* stream;        // [m, hidden] the stream the branch joins, and its scales
	const Scale* stream_scale;
	const Scale* in_scale;       // scales of the projection's input rows
	int8_t* out;                 // [m, hidden] the joined stream, and its scales
	Scale* out_scale;
	const int8_t* gain;          // of the norm that follows into b.nrm / b.ns, nullptr: none
	Scale c_proj, c_res, c_norm;
	int site_proj, site_res, site_norm, norm_layer;
	int32_t* done;               // [m] set to done_value once the stream is joined, or nullptr
	int done_value;
	const RowSink* sink;         // [m] where the joined stream also goes (the call's last layer), or nullptr
};
void launch_res(const RowBatch& b, const Dims& d, const ResSite& a, cudaStream_t st);
void launch_act(const RowBatch& b, const Dims& d, const LayerDev& h, const int32_t* silu, cudaStream_t st);

// ---- int8 linear layers (sslm_gemv.cu, sslm_gemm_tc.cu)
// out[m, n] = fold_n( sum_k x[m,k] * w[n,k] ) (+ LoRA delta), plus the per-row max |out|
// of each column segment, reduced into rowmax[m][slot].
constexpr unsigned long long kRowmaxTimeout = ~0ull;
struct LinearArgs {
	const int8_t* x;      // [M, K] row-major activations
	const int8_t* w;      // [N, K] row-major weights
	const int32_t* fold;  // [N, 3] or nullptr (no fold: logits)
	int M, N, K;
	void* out;            // [M, out_ld] int32, or int64 when out64
	int out_ld;
	int out64;
	unsigned long long* rowmax;  // [M][4] or nullptr
	int nseg;             // column segments (fused projections)
	int seg_end[3];       // exclusive end column of each segment
	int seg_slot[3];      // rowmax slot per segment, -1: none
	int seg_lora[3];      // LoraSlot per segment, -1: projection is never adapted
	const RowDesc* rows;  // per-row adapter pointers (may be nullptr: no LoRA at all)
	int layer;
	const int8_t* lora_u; // [M][3][kMaxLoraRank]
	// head mode: packed argmax keys instead of a stored row (out may be nullptr)
	unsigned long long* best;
	int32_t* logits;      // optional full dump [M, N]
	// head mode, constrained decoding: per row the vocab-bit mask page of the row's DFA state
	// (bit n clear = token n not allowed: its logit counts as INT32_MIN, ApplyMaskAndArgmax,
	// src/forward/forward_sites.cpp:2443-2449), or nullptr for an unconstrained row; the array
	// itself may be nullptr
	const uint8_t* const* row_mask;
	int32_t* status;      // [M] row statuses: a bounded device wait that ran out is reported here, or, where this is
	                      // nullptr, as the row maximum kRowmaxTimeout
	// split-K scratch of the tensor-core path (optional): partial accumulators and one
	// arrival counter per output tile. Counters are zero between launches.
	int32_t* partial;
	size_t partial_bytes;
	unsigned int* tile_counters;
	int n_tile_counters;
	int splits;           // filled in by launch_linear_tc
	int caller_memory;    // 1: operands are a caller's own, on a caller's stream: the weights may have been written by
	                      //    the kernel in front (plain stream order), and no tensor map is kept
	int debug_withhold;   // tests only: 1 block 0 never requests its first weight tile (tc_debug_withhold), 2 it waits for
	                      //    four bytes too many in its exchange (exchange_debug_take)
};
// HBM-bound small-M path: bulk-copy weight streaming through a shared-memory ring, dp4a.
cudaError_t launch_linear_gemv(const LinearArgs& a, cudaStream_t st);
// up to eight rows, the weights waiting in shared memory (sslm_few.cu). Returns false where they do not fit.
bool launch_linear_few(const LinearArgs& a, cudaStream_t st);
// tensor-core path for M > 8 rows (tcgen05 kind::i8, TMA-fed). Returns false when the
// shape is not supported by that kernel (caller then uses the GEMV path).
bool launch_linear_tc(const LinearArgs& a, cudaStream_t st);
// tensor-core path for up to 256 rows, weights on the M side of the MMA (sslm_skinny.cu). Returns false
// where another kernel is the better one as well.
bool launch_linear_skinny(const LinearArgs& a, cudaStream_t st);
// shared by the two tensor-core kernels: [rows, k] int8 map, box 128 bytes x box_rows, 128-byte swizzle
bool tc_tensor_map(const void* ptr, int rows, int k, int box_rows, bool cache, CUtensorMap* out);
void tc_count(bool launched, int reason);      // of the weights-first kernel
void tc_count_few();                           // of launch_linear_few
bool tc_debug_take();      // one launch of those tc_debug_withhold asked for
// Tests of the bounded waits: the next `launches` tensor-core launches arm their first weight-tile
// barrier in block 0 without requesting the tile, so that the wait on it runs out (no fault, no
// endless loop: the rows of that tile end with the internal wait-timeout status).
void tc_debug_withhold(int launches);
// process-wide counters of the tensor-core path: launches, refusals, reason of the last refusal
void tc_stats(unsigned long long* launches, unsigned long long* refusals, int* last_reason);
// launches per kernel variant (tile shape) of the tensor-core path
void tc_variant_counts(unsigned long long* counts, int n);

// u = clamp127(amp_fold(A x)) for up to three projections sharing the input x
// (AddAmplifyingLoraDelta's first half, src/forward/forward_sites.cpp:1062-1080)
void launch_lora_u(const RowBatch& b, const int8_t* x, int k_in, int layer, int nproj,
                   const int* lora_slots, cudaStream_t st);

// ---- attention over the paged KV pool (sslm_attn.cu)
cudaError_t attn_configure(const Dims& d);
// slices per kv head of later attention launches (0: chosen per launch); for tuning and tests
void attn_force_splits(int splits);
// How the attention of m rows will run, decided ahead of the q/k/v site: site != 0 says that it takes that site over
// (launch_qkv_post is then left out).
struct AttnChoice {
	int forced;      // slices per kv head asked for (attn_force_splits), 0: none
	int site;
};
AttnChoice attn_choose(const Dims& d, const LayerDev& h, int m, int max_width, int chunk);
// Returns true when the launch also ran the attention-context funnel (codes in b.ctx, scale in
// b.cs); otherwise b.ctxw / rowmax slot 3 are filled and launch_ctx_funnel must follow.
bool launch_attention(const RowBatch& b, const Dims& d, const LayerDev& layer, int layer_index,
                      KvPoolDev pool, int max_width, int reverse_rows, const AttnChoice& choice, const int32_t* cos, const int32_t* sin,
                      cudaStream_t st, cudaError_t* err);
// gather `planes` planes of a sequence's pages, from plane0 on, into the reference's canonical block layout
// [layer][K|V][kv_head][position][head_dim] with `span` positions per plane; positions beyond
// `valid(layer)` are zero
void launch_kv_export(const Dims& d, KvPoolDev pool, const int32_t* pages, int context_length,
                      int layer_index, int span, int plane0, int planes, int8_t* out, cudaStream_t st);
// tests: the device integer primitives over arrays of operands (device pointers)
void launch_int_sweep(int which, const int64_t* a, const int64_t* b, const int64_t* c, const int64_t* e, long long n, int64_t* out0,
                      int64_t* out1, int64_t* out2, cudaStream_t st);
// What a sequence takes over from a frozen prefix of its pool: the page ids of the full pages, a private
// copy of the last, partly filled one (copy_from < 0: none), the stream state.
struct AdoptArgs {
	const int32_t* src_pages;
	int32_t* dst_pages;
	int full_pages;
	int32_t copy_from, copy_to;
	const int8_t* src_state;
	int8_t* dst_state;
	int state_bytes;      // a multiple of 16
};
void launch_adopt(const Dims& d, KvPoolDev pool, const AdoptArgs& a, cudaStream_t st);
// the inverse: scatter planes of a canonical block into the sequence's pages (valid positions only)
void launch_kv_import(const Dims& d, KvPoolDev pool, const int32_t* pages, int context_length,
                      int layer_index, int span, int plane0, int planes, const int8_t* in, cudaStream_t st);

}  // namespace sslm
