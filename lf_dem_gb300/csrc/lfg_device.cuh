// lfg_device.cuh -- device helpers shared by the factorisation kernels:
// programmatic dependent launch, scalar/block index arithmetic, shared-memory
// progress flags, and the tcgen05 / mbarrier primitives.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "lfg_internal.h"

namespace lfg {

constexpr unsigned FULL_MASK = 0xffffffffu;

// Programmatic dependent launch.  The factor and solve kernels are launched
// with programmatic stream serialisation (launch_pdl) and call pdl_wait --
// which returns once the previous launch has finished and its writes are
// visible -- before their first access to data an earlier launch writes;
// task lists and indices (written by the symbolic upload, before any of these
// launches) may be read before it.  The solve phases also call pdl_trigger
// first, so the next phase is scheduled as soon as all their CTAs run, and so
// do the panel solves (short launches: the next update's CTAs, the
// diagonal tiles first, are resident when they complete), the Schur products (the
// next level's assembly reads its indices meanwhile: 2 % of a monolayer's step)
// and the assembly.  The updates and diagonal blocks do not (their successors
// would sit resident next to the diagonal-block CTA on the critical path: no
// gain measured), so theirs start when they finish, overlapping only the final
// flush.
//
// Data that an earlier launch writes is never read through a __restrict__ pointer
// that the kernel does not write through (const or not), nor with __ldg: the
// compiler may take such loads as constant and move them ahead of the wait.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Scalar index r of a front or vector with dof unknowns per particle (6, or
// 3 for the in-plane part of a 2D system): its particle (block) and component.
__device__ __forceinline__ int bdiv(int r, int dof) { return dof == 6 ? r/6 : r/3; }
__device__ __forceinline__ int bmod(int r, int dof) { return dof == 6 ? r%6 : r%3; }

// a 16-byte aligned record of read-only memory
template <typename V> __device__ __forceinline__ V load_record(const V *p)
{
	union { int4 q[sizeof(V)/16]; V v; } u;
#pragma unroll
	for (int i = 0; i < (int)(sizeof(V)/16); i++) u.q[i] = __ldg(reinterpret_cast<const int4 *>(p)+i);
	return u.v;
}

template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args)
{
	cudaLaunchConfig_t cfg = {};
	cudaLaunchAttribute attr[1];
	attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr[0].val.programmaticStreamSerializationAllowed = 1;
	cfg.gridDim = grid;
	cfg.blockDim = block;
	cfg.dynamicSmemBytes = smem;
	cfg.stream = st;
	cfg.attrs = attr;
	cfg.numAttrs = 1;
	LFG_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
}

// Progress flags of the diagonal-block pipelines (shared memory): the
// producer warp publishes "columns [0, v) are in Lsh" with a release store
// after the __syncwarp that follows its lanes' stores; a follower warp polls
// with acquire loads.  The wait is bounded: past the limit it records status 0
// (LFG_ERR_TIMEOUT) and goes on, so a broken pipeline cannot hang the SM.
__device__ __forceinline__ void flag_publish(int *p, int v)
{
	asm volatile("st.release.cta.shared::cta.u32 [%0], %1;"
	             :: "r"((unsigned)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}
__device__ __forceinline__ void flag_add(int *p)
{
	asm volatile("red.release.cta.shared::cta.add.u32 [%0], 1;"
	             :: "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ int flag_read(const int *p)
{
	int v;
	asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];"
	             : "=r"(v) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
	return v;
}
constexpr int FLAG_SPIN_LIMIT = 1 << 22;   // ~0.1 s of polls
__device__ __forceinline__ void flag_wait(const int *p, int need, int *fail)
{
	if (!p) return;
	for (int it = 0; it < FLAG_SPIN_LIMIT; it++)
		if (flag_read(p) >= need) return;
	if (fail) atomicMin(fail, 0);
}

// tcgen05 / mbarrier primitives.  Every mbarrier wait is bounded.
namespace umma {
constexpr uint32_t WAIT_LIMIT = 1u << 24;

__device__ inline uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart (stride byte offset), descriptor version 1
__device__ inline uint64_t sdesc(uint32_t a)
{
	return (uint64_t)((a >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
	       ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// The lanes of a warp poll on their own and may leave the loop at different
// turns: a warp-wide (.aligned) instruction that follows a wait needs a
// __syncwarp in between.
__device__ inline bool mbar_wait(uint32_t bar, uint32_t parity)
{
	for (uint32_t it = 0; it < WAIT_LIMIT; it++) {
		uint32_t done;
		asm volatile("{\n\t.reg .pred p;\n\t"
		             "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
		             "selp.u32 %0, 1, 0, p;\n\t}\n"
		             : "=r"(done) : "r"(bar), "r"(parity) : "memory");
		if (done) return true;
	}
	return false;
}

__device__ inline void mbar_init(uint64_t *b, int count)
{
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(saddr(b)), "r"(count));
}
__device__ inline void mbar_arrive(uint64_t *b)
{
	asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" :: "r"(saddr(b)) : "memory");
}
// bulk copies of global memory to shared memory (16-byte aligned, sizes multiples of 16)
__device__ inline void bulk_expect(uint64_t *b, uint32_t bytes)
{
	asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}"
	             :: "r"(saddr(b)), "r"(bytes) : "memory");
}
__device__ inline void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *b)
{
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
	             :: "r"(saddr(dst)), "l"(src), "r"(bytes), "r"(saddr(b)) : "memory");
}
__device__ inline void mma_commit(uint64_t *b)
{
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
	             :: "r"(saddr(b)) : "memory");
}
} // namespace umma

} // namespace lfg
