// lfg_split.cuh -- exact products on the tensor cores: rows scaled to integers
// and cut into signed base-256 digits (FP16 values), digit products summed in
// FP32 accumulators.  Shared by the FP64 and FP32 tile kernels
// (lfg_factor64.cu, lfg_factor32.cu).
#pragma once
#include <cuda_fp16.h>

#include "lfg_device.cuh"

namespace lfg {

namespace split {
using namespace umma;
constexpr int M = 128;                    // tile rows (tensor memory lanes)
constexpr int KS = 16, SLOTS = 4;         // K step of one MMA; ring of SLOTS steps = one 128-byte swizzled row
constexpr int THREADS = 512;              // producers first, all run the epilogue; 16 warps leave 128
                                          // registers a thread (a 17th would leave 96)
constexpr int ROW_BYTES = SLOTS*KS*2;     // 128
constexpr int A_BYTES = M*ROW_BYTES;      // one digit of A

// D = FP32, A = B = FP16, both K-major, M = 128, N = n
__device__ constexpr uint32_t idesc(int n)
{
	return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ inline void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\t"
	             "setp.ne.b32 p, %4, 0;\n\t"
	             "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
	             :: "r"(d), "l"(a), "l"(b), "r"(id), "r"(accumulate));
}

// The byte `sel` of w0 and of w1, each a digit plus 128, as a pair of FP16 values:
// 1024 + byte is an FP16 bit pattern, minus 1152 leaves byte - 128 exactly.
template <int SEL>
__device__ __forceinline__ uint32_t digit_pair(uint32_t w0, uint32_t w1)
{
	uint32_t t = (__byte_perm(w0, w1, SEL | SEL << 4 | (4+SEL) << 8 | (4+SEL) << 12) & 0x00ff00ffu) | 0x64006400u;
	const __half2 h = __hsub2(*reinterpret_cast<__half2 *>(&t), __half2half2(__ushort_as_half(0x6480)));
	return *reinterpret_cast<const uint32_t *>(&h);
}

struct Bars { uint64_t full[SLOTS], empty[SLOTS], done; };

__device__ inline void tmem_ld4(uint32_t ta, uint32_t (&v)[4])
{
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
	             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(ta));
}

} // namespace split

} // namespace lfg
