// Exchanges between the blocks of a thread-block cluster.
//
// Values travel as asynchronous stores into the peers' shared memory that complete on an mbarrier
// there (st.async): a block waits for exactly the words it needs and nobody meets at a barrier. A
// max / sum exchange of eight blocks takes 420 cycles this way; remote stores (or loads) around
// barrier.cluster, whose release also waits out the block's global stores, take 1,100 (B200).
//
// Rules: a peer's shared memory may be written once the peer runs, i.e. behind one cluster_arrive /
// cluster_wait pair at the start of the kernel (free: its wait is over before the dependency wait is).
// A block leaves only after it has received every word its peers send it, whatever became of its row,
// so no store finds its target gone. Waits are bounded.
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
// true once every byte is in; false when the poll limit (well under a second) ran out
__device__ __forceinline__ bool exchange_wait(uint32_t bar) {
	for (uint32_t i = 0; i < (1u << 22); ++i) {
		uint32_t ok;
		asm volatile(
		    "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
		    : "=r"(ok) : "r"(bar) : "memory");
		if (ok) return true;
		if (i > 2048) __nanosleep(64);
	}
	return false;
}

// ---- slots that some threads fill and others empty, turn by turn
__device__ __forceinline__ void ring_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void ring_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {      // past the L1
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// false when the poll limit (about a second) ran out
__device__ __forceinline__ bool ring_wait(uint32_t bar, uint32_t parity) {
	for (uint32_t i = 0; i < (1u << 23); ++i) {
		uint32_t ok;
		asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
		             : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
		if (ok) return true;
		if (i > 2048) __nanosleep(64);
	}
	return false;
}

}  // namespace sslm
