// Tensor-memory and tcgen05 helpers for sm_100a (one CTA, cta_group::1).
//
// Rules kept here: one warp allocates and frees; A comes from tensor memory (written by tcgen05.st, lane = row of the tile, four
// 8-bit integers of consecutive k per column), B from shared memory in the K-major layout with the 128-byte swizzle (rows of 128
// bytes, groups of eight rows 1024 bytes apart, 16-byte chunk c of row n stored at c ^ (n & 7)).
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
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
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
// Instruction descriptor: int32 accumulators, signed 8-bit operands, M 128, N n (a multiple of 16).
constexpr uint32_t tc_idesc_s8(int n) { return (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n / 8) << 17) | (uint32_t(128 / 16) << 24); }

// d[128 lanes][n columns] (+)= a[128 lanes][32] * b[n rows][32]^T; one thread issues
__device__ __forceinline__ void tc_mma_s8(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
		     "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(uint32_t(accumulate))
		     : "memory");
}

// The same for bf16 operands that both lie in shared memory (16 k a step, 32 bytes) and fp32 accumulators.  b_mn: B lies with its n
// contiguous -- rows of k, 128 bytes of n each, swizzled alike; k advances by 2048 bytes per 16 rows.
constexpr uint32_t tc_idesc_bf16(int n, bool b_mn)
{
	return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn ? 1u << 16 : 0u) | (uint32_t(n / 8) << 17) | (uint32_t(128 / 16) << 24);
}
__device__ __forceinline__ uint64_t tc_desc_mn(uint32_t addr) // one block of 64 n; groups of eight k rows 1024 bytes apart
{
	return uint64_t((addr & 0x3ffffu) >> 4) | (uint64_t(1024 >> 4) << 16) | (uint64_t(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tc_mma_bf16_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
		     "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(uint32_t(accumulate))
		     : "memory");
}
// a and b as three bf16 each, exactly (but for what lies below 2^-133): truncations of the value and of what they leave
__device__ __forceinline__ void split_bf16(float a, float b, uint32_t (&piece)[3])
{
#pragma unroll
	for (int i = 0; i < 3; i++) {
		asm("prmt.b32 %0, %1, %2, 0x7632;" : "=r"(piece[i]) : "r"(__float_as_uint(a)), "r"(__float_as_uint(b)));
		a -= __uint_as_float(__float_as_uint(a) & 0xffff0000u);
		b -= __uint_as_float(__float_as_uint(b) & 0xffff0000u);
	}
}
__device__ __forceinline__ void tmem_load(uint32_t t, float (&r)[16])
{
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
		     "tcgen05.wait::ld.sync.aligned;"
		     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]),
		       "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
		     : "r"(t)
		     : "memory");
}
__device__ __forceinline__ void tmem_load(uint32_t t, float (&r)[8])
{
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\ttcgen05.wait::ld.sync.aligned;"
		     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
		     : "r"(t)
		     : "memory");
}

// 32 columns of the calling warp's 32 lanes
__device__ __forceinline__ void tmem_store32(uint32_t t, const uint32_t (&r)[32])
{
	asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
		     "%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(t),
		     "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
		     "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
		     "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
		     : "memory");
}
// four columns, complete on return
__device__ __forceinline__ void tmem_load4(uint32_t t, int (&r)[4])
{
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n\ttcgen05.wait::ld.sync.aligned;"
		     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
		     : "r"(t)
		     : "memory");
}

// mbar_wait() without its call of the clocked loop: a call keeps what lives across it in half of the registers, and warps that hold
// a whole tile of operands have none to spare.  2 FAST_POLLS failed polls, a second or two, then it gives up the same way.
__device__ __forceinline__ bool mbar_wait_inline(uint64_t *bar, uint32_t parity, int *err)
{
	const uint32_t a = smem_u32(bar);
	for (uint32_t i = 0; i < 2 * FAST_POLLS; i++)
		if (mbar_try(a, parity))
			return true;
	*reinterpret_cast<volatile int *>(err) = 1;
	if (int *host = *reinterpret_cast<int *volatile *>(err + ERROR_HOST_WORD))
		*reinterpret_cast<volatile int *>(host) = 1;
	return false;
}

// untiled bulk copy global -> shared: addresses and size multiples of 16 bytes
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes),
		     "r"(smem_u32(bar))
		     : "memory");
}

} // namespace l1b
