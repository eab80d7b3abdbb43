// Dense L1 scores, backward, for sets of at most 48 tokens (fp32) or 32 (fp64), any width, head count and alignment.
//
// A warp owns one head and 32 width columns (a lane each) of one batch item and holds every query row of its column in
// registers: both gradients of a term come from ONE visit, d_k of a source row is complete at the end of its row, and the
// sign is exact (zero where q == k), so there is no tie list, no scratch and no second kernel.  The head's scores'
// gradients lie [s][t] in shared memory and are read as broadcasts, 16 bytes at a time.
//
// Bound by instruction issue, and by its one launch where the batch is small: [512,16,8,32] 18 us, [200,30,8,64] 41 us, [200,48,6,33]
// 91 us (the tiled kernels 224).  The
// tiled kernels spent their time on padding (an item is 128 query rows), on the tie detector and, with padded sets, on the exact
// two-pass kernel: 1.3 ms (padded) and 225 us for the same.
#include "common.cuh"
#include "dense_bwd_tiles.h"

namespace l1b {
namespace {

// sign(d) * g with the reference's sign: also a difference of equal infinities (NaN in fp32) has none, as where ties are listed
__device__ __forceinline__ float term(float d, float g)
{
	const float sg = __uint_as_float(__float_as_uint(g) ^ (__float_as_uint(d) & 0x80000000u));
	return fabsf(d) > 0.f ? sg : 0.f;
}
__device__ __forceinline__ double term(double d, double g) { return sign_apply(d, g); }

// TN >= n_tok query rows per thread; NW warps per CTA: consecutive (head, 32 columns) units of one batch item
template <typename T, int TN, int NW>
__global__ void __launch_bounds__(NW * 32)
dense_bwd_small_kernel(const T *__restrict__ g, const T *__restrict__ q, const T *__restrict__ k, T *__restrict__ d_q,
		       T *__restrict__ d_k, int n_tok, int n_heads, int width, T scale, int nws, int cpb)
{
	constexpr int VEC = 16 / sizeof(T);
	using V = Pack<T, VEC>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	T *G = reinterpret_cast<T *>(smem_raw); // [head of this CTA][s][t], rows of TN; a head's pitch puts 8 heads on 8 bank groups
	const int pitch = (n_tok * TN + 31) / 32 * 32 + VEC;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int b = blockIdx.x / cpb, u0 = (blockIdx.x % cpb) * NW;
	const int nu = n_heads * nws, h_lo = u0 / nws, h_hi = min(nu - 1, u0 + NW - 1) / nws; // at most NW heads
	const size_t tok0 = size_t(b) * n_tok;
	{
		const int hh = tid & (NW - 1);
		const T *src = g + tok0 * n_tok * n_heads + h_lo + hh;
		if (h_lo + hh <= h_hi)
			for (int i = tid / NW; i < n_tok * TN; i += 32) {
				const int s = i / TN, t = i % TN; // query rows past the end: gradient 0
				G[hh * pitch + i] = t < n_tok ? src[size_t(s * n_tok + t) * n_heads] : T(0);
			}
	}
	__syncthreads();
	const int u = u0 + warp;
	if (u >= nu)
		return;
	const int h = u / nws, w = (u % nws) * 32 + lane;
	if (w >= width)
		return;
	const size_t row = size_t(n_heads) * width, off = tok0 * row + size_t(h) * width + w;
	T a[TN], acc[TN];
#pragma unroll
	for (int t = 0; t < TN; t++) {
		a[t] = t < n_tok ? q[off + t * row] : T(0);
		acc[t] = T(0);
	}
	const V *Gh = reinterpret_cast<const V *>(G + (h - h_lo) * pitch);
	T kv = k[off];
	for (int s = 0; s < n_tok; s++) {
		const T kn = s + 1 < n_tok ? k[off + (s + 1) * row] : T(0);
		T sum = T(0);
#pragma unroll
		for (int i = 0; i < TN / VEC; i++) {
			const V gv = Gh[s * (TN / VEC) + i];
#pragma unroll
			for (int e = 0; e < VEC; e++) {
				const T x = term(a[i * VEC + e] - kv, gv.v[e]);
				acc[i * VEC + e] += x;
				sum += x;
			}
		}
		d_k[off + s * row] = -scale * sum;
		kv = kn;
	}
#pragma unroll
	for (int t = 0; t < TN; t++)
		if (t < n_tok)
			d_q[off + t * row] = scale * acc[t];
}

template <typename T, int TN, int NW = 8>
int launch(const T *g, const T *q, const T *k, T *d_q, T *d_k, int bs, int n_tok, int n_heads, int width, cudaStream_t st)
{
	const int nws = (width + 31) / 32;
	const long long nu = (long long)n_heads * nws, cpb = (nu + NW - 1) / NW, grid = bs * cpb;
	if (nu > 0x7fffffffLL || grid > 0x7fffffffLL)
		return L1ATTN_ERR_SHAPE;
	const size_t smem = NW * ((size_t(n_tok) * TN + 31) / 32 * 32 + 16 / sizeof(T)) * sizeof(T);
	auto kern = dense_bwd_small_kernel<T, TN, NW>;
	L1B_SHARED_MEMORY(kern, int(smem));
	kern<<<unsigned(grid), NW * 32, smem, st>>>(g, q, k, d_q, d_k, n_tok, n_heads, width, T(-1.0 / sqrt(double(width))), nws, int(cpb));
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

template <typename T>
int pick(const void *g, const void *q, const void *k, void *d_q, void *d_k, int bs, int n_tok, int n_heads, int width, cudaStream_t st)
{
	if (n_tok <= 16)
		return launch<T, 16>((const T *)g, (const T *)q, (const T *)k, (T *)d_q, (T *)d_k, bs, n_tok, n_heads, width, st);
	if (sizeof(T) == 4 && n_tok > 32) {
		// two warps per CTA while eight would leave SMs without one ([4,48,8,64] 28 us, 37 with eight)
		const bool few = (long long)bs * n_heads * ((width + 31) / 32) < 8 * 148;
		auto go = few ? launch<float, 48, 2> : launch<float, 48, 8>;
		return go((const float *)g, (const float *)q, (const float *)k, (float *)d_q, (float *)d_k, bs, n_tok, n_heads, width, st);
	}
	return launch<T, 32>((const T *)g, (const T *)q, (const T *)k, (T *)d_q, (T *)d_k, bs, n_tok, n_heads, width, st);
}

} // namespace

int dense_bwd_small_launch(const void *d_attn, const void *q, const void *k, void *d_q, void *d_k, int bs, int n_tok, int n_heads,
			   int width, int dtype, cudaStream_t st)
{
	if (dtype == L1ATTN_F32)
		return pick<float>(d_attn, q, k, d_q, d_k, bs, n_tok, n_heads, width, st);
	return pick<double>(d_attn, q, k, d_q, d_k, bs, n_tok, n_heads, width, st);
}

} // namespace l1b
