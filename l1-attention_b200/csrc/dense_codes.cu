// Order codes of q and k for the tensor-core backward (dense_codes.h).
//
// A CTA takes 16 columns of one (batch, head) and one block of up to 1024 keys: a warp sorts a column in registers (bitonic network,
// element lane * EPT + r: 40 of its 55 steps stay inside a lane), the sorted columns go to shared memory, and every thread ranks
// tokens of q (all of them), then of k (the block's own), by binary search, eight independent searches at a time: the tables' 16-byte
// vectors.  Bound by the shared-memory pipe: 11 gathered loads per value whose lanes hit random banks below the top levels.  The
// columns' pitch is 1 modulo 32 (odd for smaller blocks), so that lanes at the same depth of different columns read different banks.
#include "common.cuh"
#include "dense_codes.h"

namespace l1b {
namespace {

constexpr int COLS = 16, NTHREADS = 512;

// index of sorted element i: one word of padding per 32
__device__ __forceinline__ int padded(int i) { return i + (i >> 5); }

// the key `WORD` words behind a shared address
template <int WORD> __device__ __forceinline__ float load_key(unsigned at)
{
	float v;
	asm volatile("ld.shared.f32 %0, [%1 + %2];" : "=f"(v) : "r"(at), "n"(WORD * 4));
	return v;
}
// lower bounds of eight values among 2 STEP sorted keys (padded): one instruction per step beside load and comparison
template <int STEP> __device__ __forceinline__ void search(unsigned (&at)[8], const float (&x)[8])
{
	if constexpr (STEP >= 1) {
#pragma unroll
		for (int e = 0; e < 8; e++)
			if (load_key<STEP - 1 + (STEP - 1) / 32>(at[e]) < x[e])
				at[e] += (STEP + STEP / 32) * 4;
		search<STEP / 2>(at, x);
	}
}

template <int EPT> __device__ __forceinline__ void sort_column(float (&v)[EPT], int lane)
{
	constexpr int N = 32 * EPT;
#pragma unroll
	for (int size = 2; size <= N; size *= 2) {
		// first step of a merge: element i against its mirror image in the group of `size`
		if (size <= EPT) {
#pragma unroll
			for (int r = 0; r < EPT; r++) {
				const int m = r ^ (size - 1);
				if (m > r) {
					const float lo = fminf(v[r], v[m]), hi = fmaxf(v[r], v[m]);
					v[r] = lo;
					v[m] = hi;
				}
			}
		} else {
			const int mask = size / EPT - 1;
			const bool low = (lane & (size / EPT / 2)) == 0;
			float o[EPT];
#pragma unroll
			for (int r = 0; r < EPT; r++)
				o[r] = __shfl_xor_sync(0xffffffffu, v[EPT - 1 - r], mask);
#pragma unroll
			for (int r = 0; r < EPT; r++)
				v[r] = low ? fminf(v[r], o[r]) : fmaxf(v[r], o[r]);
		}
#pragma unroll
		for (int d = size / 4; d >= 1; d /= 2) {
			if (d < EPT) {
#pragma unroll
				for (int r = 0; r < EPT; r++)
					if ((r & d) == 0) {
						const float lo = fminf(v[r], v[r + d]), hi = fmaxf(v[r], v[r + d]);
						v[r] = lo;
						v[r + d] = hi;
					}
			} else {
				const bool low = (lane & (d / EPT)) == 0;
#pragma unroll
				for (int r = 0; r < EPT; r++) {
					const float o = __shfl_xor_sync(0xffffffffu, v[r], d / EPT);
					v[r] = low ? fminf(v[r], o) : fmaxf(v[r], o);
				}
			}
		}
	}
}

template <int EPT>
__global__ void __launch_bounds__(NTHREADS, 2)
dense_codes_kernel(const float *__restrict__ q, const float *__restrict__ k, int *__restrict__ hdr, uint4 *__restrict__ kc, uint4 *__restrict__ qc,
		   size_t q_block, int n_tok, int n_heads, int width, int t8, int ncg)
{
	constexpr int CAP = 32 * EPT, PITCH = CAP + CAP / 32 + 1;
	extern __shared__ float sm[]; // [COLS][PITCH]
	__shared__ unsigned tied[COLS][EPT]; // a bit per sorted key: some q equals it (set at the first of equal keys)
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 0)
		hdr[CODE_HDR_EXACT] = 0;
	const int w0 = int(blockIdx.x % ncg) * COLS, h = int(blockIdx.x / ncg) % n_heads, b = int(blockIdx.x / ncg) / n_heads;
	const int j = blockIdx.y, s0 = j * CODE_BLOCK, len = min(CODE_BLOCK, n_tok - s0);
	const size_t row = size_t(n_heads) * width, base = size_t(b) * n_tok * row + size_t(h) * width + w0;
	const int col = tid % COLS, ncol = min(COLS, width - w0);

	for (int i = tid; i < COLS * EPT; i += NTHREADS)
		(&tied[0][0])[i] = 0;
	for (int s = tid / COLS; s < CAP; s += NTHREADS / COLS) { // (a NaN sorts above all keys: it is below nothing)
		float x = INFINITY;
		if (s < len && col < ncol) {
			x = k[base + size_t(s0 + s) * row + col];
			x = x == x ? x : INFINITY;
		}
		sm[col * PITCH + s] = x;
	}
	__syncthreads();
	{
		float v[EPT];
		float *c = sm + warp * PITCH;
#pragma unroll
		for (int r = 0; r < EPT; r++)
			v[r] = c[r * 32 + lane];
		__syncwarp();
		sort_column<EPT>(v, lane);
#pragma unroll
		for (int r = 0; r < EPT; r++)
			c[padded(lane * EPT + r)] = v[r];
	}
	__syncthreads();
	const unsigned c_addr = unsigned(__cvta_generic_to_shared(sm + col * PITCH));
	auto rank_groups = [&](bool is_k, const float *values, int first, int groups) {
		for (int g = tid / COLS; g < groups; g += NTHREADS / COLS) {
			const int t = first + g * 8; // first of eight tokens
			const float *src = values + base + size_t(t) * row + col;
			float x[8];
			unsigned at[8]; // shared address of the first of the keys that may still be at or above x
#pragma unroll
			for (int e = 0; e < 8; e++) {
				x[e] = t + e < n_tok ? src[size_t(e) * row] : NAN;
				at[e] = c_addr;
			}
			search<CAP / 2>(at, x);
			unsigned code[8];
#pragma unroll
			for (int e = 0; e < 8; e++) {
				const float key = load_key<0>(at[e]);
				const int word = int(at[e] - c_addr) >> 2, p = word - word / 33; // (padding out)
				const int rank = p + (key < x[e]);                               // (above the block's last key)
				if (is_k) {
					code[e] = 0x8000 - 4 * (2 * rank + 1) + (tied[col][p >> 5] >> (p & 31) & 1u);
					if (x[e] != x[e])
						code[e] = 0x8000 - 4 * NAN_CODE;
				} else {
					const bool tie = key == x[e] && p < len;
					if (tie)
						atomicOr(&tied[col][p >> 5], 1u << (p & 31));
					code[e] = 8 * rank + (tie ? 5 : 0);
				}
			}
			const size_t out = ((size_t(b) * n_heads + h) * t8 + t / 8) * width + w0 + col;
			(is_k ? kc : qc + size_t(j) * (q_block / 16))[out] =
				make_uint4(code[0] | code[1] << 16, code[2] | code[3] << 16, code[4] | code[5] << 16, code[6] | code[7] << 16);
		}
	};
	if (col < ncol)
		rank_groups(false, q, 0, t8);
	__syncthreads();
	if (col < ncol)
		rank_groups(true, k, s0, (len + 7) / 8);
}

template <int EPT>
int launch(const float *q, const float *k, unsigned char *scratch, const CodeTables &ct, int bs, int n_tok, int n_heads, int width, cudaStream_t st)
{
	constexpr int CAP = 32 * EPT;
	const int ncg = (width + COLS - 1) / COLS;
	const long long gx = (long long)bs * n_heads * ncg;
	if (gx > 0x7fffffffLL || ct.nb > 65535)
		return 1;
	auto kern = dense_codes_kernel<EPT>;
	constexpr int smem = COLS * (CAP + CAP / 32 + 1) * 4;
	L1B_SHARED_MEMORY(kern, smem);
	kern<<<dim3(unsigned(gx), unsigned(ct.nb)), NTHREADS, smem, st>>>(q, k, reinterpret_cast<int *>(scratch + ct.hdr), reinterpret_cast<uint4 *>(scratch + ct.k),
									  reinterpret_cast<uint4 *>(scratch + ct.q), ct.q_block, n_tok, n_heads, width, ct.t8, ncg);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

} // namespace

// Fills the tables and clears the header.  scratch: code_tables().bytes, 256-byte aligned.  Returns 1 when nothing was launched.
int dense_codes_launch(const float *q, const float *k, void *scratch, int bs, int n_tok, int n_heads, int width, cudaStream_t st)
{
	const CodeTables ct = code_tables(bs, n_tok, n_heads, width);
	unsigned char *sc = static_cast<unsigned char *>(scratch);
	return n_tok <= 64    ? launch<2>(q, k, sc, ct, bs, n_tok, n_heads, width, st)
	       : n_tok <= 128 ? launch<4>(q, k, sc, ct, bs, n_tok, n_heads, width, st)
	       : n_tok <= 256 ? launch<8>(q, k, sc, ct, bs, n_tok, n_heads, width, st)
	       : n_tok <= 512 ? launch<16>(q, k, sc, ct, bs, n_tok, n_heads, width, st)
			      : launch<32>(q, k, sc, ct, bs, n_tok, n_heads, width, st);
}

} // namespace l1b
