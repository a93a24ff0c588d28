// Exchanges between the blocks of a thread-block cluster.
//
// Values travel as asynchronous stores into the peers' shared memory that complete on an mbarrier
// there (st.async): a block waits for exactly the words it needs and nobody meets at a barrier. A
// max / sum exchange of eight blocks takes 420 cycles this way; remote stores (or loads) around
// barrier.cluster, whose release also waits out the block's global stores, take 1,100 (B200).
//
// Rules. A peer's shared memory may be written once the peer runs, i.e. behind one cluster_arrive /
// cluster_wait pair at the start of the kernel (free: its wait is over before the dependency wait is), and
// until it leaves. A block that has received every word its peers send it may leave: nothing is on its way
// to it any more. Waits are bounded in time (kWaitNs), so a block may also have given up on words that a
// late peer still sends: its warps end in exchange_leave, which outlasts whatever a peer can be late by.
// (Not a second cluster barrier: passed by every block it cost 1 to 2 % of a decode step, and it would have
// to be passed by every block, since a barrier that only the warps that gave up arrived at did not return.)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace sslm {

__device__ __forceinline__ uint32_t cluster_rank() {
	uint32_t r;
	asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
	return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// One mbarrier per exchange, armed with the bytes that will arrive. `bar`: its shared-memory address.
__device__ __forceinline__ uint32_t cta_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void exchange_init(uint32_t bar, uint32_t bytes) {
	asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void exchange_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// v to the place of `local` (an address in this block's shared memory) in block `rank`, counted on its `bar`
__device__ __forceinline__ void exchange_send(const void* local, uint32_t bar, uint32_t rank, uint32_t v) {
	asm volatile(
	    "{\n\t.reg .b32 ra, rb;\n\tmapa.shared::cluster.u32 ra, %0, %2;\n\tmapa.shared::cluster.u32 rb, %1, %2;\n\t"
	    "st.async.shared::cluster.mbarrier::complete_tx::bytes.u32 [ra], %3, [rb];\n\t}" ::"r"(cta_addr(local)), "r"(bar), "r"(rank), "r"(v) : "memory");
}
__device__ __forceinline__ void exchange_send(const void* local, uint32_t bar, uint32_t rank, unsigned long long v) {
	asm volatile(
	    "{\n\t.reg .b32 ra, rb;\n\tmapa.shared::cluster.u32 ra, %0, %2;\n\tmapa.shared::cluster.u32 rb, %1, %2;\n\t"
	    "st.async.shared::cluster.mbarrier::complete_tx::bytes.u64 [ra], %3, [rb];\n\t}" ::"r"(cta_addr(local)), "r"(bar), "r"(rank), "l"(v) : "memory");
}
__device__ __forceinline__ void exchange_send(const void* local, uint32_t bar, uint32_t rank, int2 v) {
	asm volatile(
	    "{\n\t.reg .b32 ra, rb;\n\tmapa.shared::cluster.u32 ra, %0, %2;\n\tmapa.shared::cluster.u32 rb, %1, %2;\n\t"
	    "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.s32 [ra], {%3, %4}, [rb];\n\t}" ::"r"(cta_addr(local)), "r"(bar), "r"(rank), "r"(v.x), "r"(v.y) : "memory");
}
// A wait on an mbarrier: quick polls, then polls with pauses, kWaitNs (%globaltimer) at most. A limit in polls
// is none: 2^22 of them took 1 s for one thread and 17 s for a block. The loop stays rolled: a launch passes
// most of its waits once, so their code is fetched, not run (unrolled, a decode step took 2 to 6 % longer).
constexpr unsigned long long kWaitNs = 250000000ull;
constexpr uint32_t kQuickPolls = 2048;
__device__ __forceinline__ unsigned long long now_ns() {
	unsigned long long t;
	asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
	return t;
}
// PEERS: what peers sent is waited for (the scope of the acquire costs 1 to 3 % of a decode step where only
// this block's own copies and multiplications are)
template <bool PEERS>
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
	uint32_t ok;
	if (PEERS)
		asm volatile(
		    "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
		    : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
	else
		asm volatile(
		    "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
		    : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
	return ok != 0;
}
// false when the limit ran out
template <bool PEERS>
__device__ __forceinline__ bool bounded_wait(uint32_t bar, uint32_t parity) {
	unsigned long long since = 0;
#pragma unroll 1
	for (uint32_t i = 0;; ++i) {
		if (bar_try<PEERS>(bar, parity)) return true;
		if (i < kQuickPolls) continue;
		__nanosleep(64);
		if (i == kQuickPolls) since = now_ns();
		else if (now_ns() - since > kWaitNs) return false;
	}
}
// true once every byte is in
__device__ __forceinline__ bool exchange_wait(uint32_t bar) { return bounded_wait<true>(bar, 0); }
// The end of a warp in which a wait ran out (bar: the first of the block's n exchanges, side by side). The blocks
// of a cluster start together and a peer sends its last words after n waits at most (one more in a kernel that
// waits for its operands), so by this deadline everything that will come has come.
static __device__ __noinline__ void exchange_leave(uint32_t bar, int n) {
	const unsigned long long deadline = now_ns() + (unsigned long long)(n + 2) * kWaitNs;
	for (int i = 0; i < n; ++i)
		while (!bar_try<true>(bar + 8u * (uint32_t)i, 0) && now_ns() < deadline) __nanosleep(64);
}

// ---- tiles: a box of a tensor map (a CUtensorMap in the launch parameters) into shared memory, counted on `bar`; four 8 x 16-byte matrices out of it
__device__ __forceinline__ void tma_2d(uint32_t dst, const void* map, uint32_t bar, int c0, int c1) {
	asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
	             ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}

// ---- slots that some threads fill and others empty, turn by turn
__device__ __forceinline__ void ring_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void ring_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {      // past the L1
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ bool ring_wait(uint32_t bar, uint32_t parity) { return bounded_wait<false>(bar, parity); }

}  // namespace sslm
