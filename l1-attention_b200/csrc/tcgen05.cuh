// Tensor-memory and tcgen05 helpers for sm_100a (one CTA, cta_group::1).
//
// Rules kept here: one warp allocates and frees; A and B lie in shared memory with the 128-byte swizzle (rows of 128 bytes, groups of
// eight rows 1024 bytes apart, 16-byte chunk c of row n stored at c ^ (n & 7)) and are both bf16; accumulators are fp32.
#pragma once
#include <stdint.h>
#include "tma.cuh"

namespace l1b {

__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t columns) // a whole warp
{
	asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(columns) : "memory");
	asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t columns) // the same warp
{
	asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(columns) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// arrives on `bar` once every tcgen05.mma that this thread has issued so far is complete
__device__ __forceinline__ void tc_commit(uint64_t *bar)
{
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Shared-memory descriptor of a K-major, 128-byte-swizzled operand (see above); k advances by 32 bytes per step.
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr)
{
	return uint64_t((addr & 0x3ffffu) >> 4) | (1ull << 16) | (uint64_t(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: fp32 accumulators, bf16 operands (16 k a step, 32 bytes), M 128, N n (a multiple of 16).  b_mn: B lies with its n
// contiguous -- rows of k, 128 bytes of n each, swizzled alike; k advances by 2048 bytes per 16 rows.
constexpr uint32_t tc_idesc_bf16(int n, bool b_mn)
{
	return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn ? 1u << 16 : 0u) | (uint32_t(n / 8) << 17) | (uint32_t(128 / 16) << 24);
}
__device__ __forceinline__ uint64_t tc_desc_mn(uint32_t addr) // one block of 64 n; groups of eight k rows 1024 bytes apart
{
	return uint64_t((addr & 0x3ffffu) >> 4) | (uint64_t(1024 >> 4) << 16) | (uint64_t(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// d[128 lanes][n columns] (+)= a[128 rows][16] * b^T; one thread issues
__device__ __forceinline__ void tc_mma_bf16_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
		     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(uint32_t(accumulate))
		     : "memory");
}
// Operands of the products are split times 2^24.  The last bit of a float lies at 2^-149 or above, that of its 2^24-fold at 2^-125: no
// piece is subnormal and none is lost.  Below 2^36 the sum of 64 products of two such operands stays below 2^126; larger ones have no pieces.
constexpr float PIECE_SCALE = 0x1p24f, PIECE_LIMIT = 0x1p36f, PIECE_UNSCALE = 0x1p-48f;
// a and b (times PIECE_SCALE) as three bf16 each, exactly: truncations of the value and of what they leave
__device__ __forceinline__ void split_bf16(float a, float b, uint32_t (&piece)[3])
{
#pragma unroll
	for (int i = 0; i < 3; i++) {
		asm("prmt.b32 %0, %1, %2, 0x7632;" : "=r"(piece[i]) : "r"(__float_as_uint(a)), "r"(__float_as_uint(b)));
		a -= __uint_as_float(__float_as_uint(a) & 0xffff0000u);
		b -= __uint_as_float(__float_as_uint(b) & 0xffff0000u);
	}
}
// The same with a leading piece of 6 bits and a second of 8, both rounded (the rest, signed, fits 8 bits): products of such leading pieces reach less
// far down, so that the adder, which truncates, loses less of their sum.  Mean loss of 64 products of one sign, emulated: 1.8 to 3.9e-8 of the
// sum with leading pieces of 8 bits, 0.1 to 0.7e-8 of 6, 0.6 to 2.1e-8 with one of each (in two sums of 32).
__device__ __forceinline__ float round_bits(float x, uint32_t drop)
{
	return __uint_as_float((__float_as_uint(x) + (1u << (drop - 1))) & ~((1u << drop) - 1));
}
__device__ __forceinline__ void split_bf16_short(float a, float b, uint32_t (&piece)[3])
{
#pragma unroll
	for (int i = 0; i < 3; i++) {
		const float pa = i == 0 ? round_bits(a, 18) : round_bits(a, 16), pb = i == 0 ? round_bits(b, 18) : round_bits(b, 16);
		asm("prmt.b32 %0, %1, %2, 0x7632;" : "=r"(piece[i]) : "r"(__float_as_uint(i < 2 ? pa : a)), "r"(__float_as_uint(i < 2 ? pb : b)));
		a -= pa;
		b -= pb;
	}
}
// 16 (8) columns at three places, of the calling warp's 32 lanes, complete on return (one wait for the three: 1 % of the fused forward)
__device__ __forceinline__ void tmem_load3(uint32_t tr, uint32_t tx, uint32_t ty, float (&r)[16], float (&x)[16], float (&y)[16])
{
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%48];\n\t"
		     "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%49];\n\t"
		     "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, [%50];\n\t"
		     "tcgen05.wait::ld.sync.aligned;"
		     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
		       "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]),
		       "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7]),
		       "=f"(x[8]), "=f"(x[9]), "=f"(x[10]), "=f"(x[11]), "=f"(x[12]), "=f"(x[13]), "=f"(x[14]), "=f"(x[15]),
		       "=f"(y[0]), "=f"(y[1]), "=f"(y[2]), "=f"(y[3]), "=f"(y[4]), "=f"(y[5]), "=f"(y[6]), "=f"(y[7]),
		       "=f"(y[8]), "=f"(y[9]), "=f"(y[10]), "=f"(y[11]), "=f"(y[12]), "=f"(y[13]), "=f"(y[14]), "=f"(y[15])
		     : "r"(tr), "r"(tx), "r"(ty)
		     : "memory");
}
__device__ __forceinline__ void tmem_load3(uint32_t tr, uint32_t tx, uint32_t ty, float (&r)[8], float (&x)[8], float (&y)[8])
{
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%24];\n\t"
		     "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%25];\n\t"
		     "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%26];\n\t"
		     "tcgen05.wait::ld.sync.aligned;"
		     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
		       "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]), "=f"(x[4]), "=f"(x[5]), "=f"(x[6]), "=f"(x[7]),
		       "=f"(y[0]), "=f"(y[1]), "=f"(y[2]), "=f"(y[3]), "=f"(y[4]), "=f"(y[5]), "=f"(y[6]), "=f"(y[7])
		     : "r"(tr), "r"(tx), "r"(ty)
		     : "memory");
}

// mbar_wait() without its call of the clocked loop: a call keeps what lives across it in half of the registers, and warps that hold
// a whole tile of operands have none to spare.  `polls` failed polls (2 FAST_POLLS: a second or two), then it gives up the same way.
__device__ __forceinline__ bool mbar_wait_inline(uint64_t *bar, uint32_t parity, int *err, uint32_t polls = 2 * FAST_POLLS)
{
	const uint32_t a = smem_u32(bar);
	for (uint32_t i = 0; i < polls; i++)
		if (mbar_try(a, parity))
			return true;
	*reinterpret_cast<volatile int *>(err) = 1;
	if (int *host = *reinterpret_cast<int *volatile *>(err + ERROR_HOST_WORD))
		*reinterpret_cast<volatile int *>(host) = 1;
	return false;
}

} // namespace l1b
