// Dense L1 scores, backward:
//   d_q[b][t][h][w] =  scale * sum_s sign(q[b][t][h][w] - k[b][s][h][w]) * g[b][s][t][h]
//   d_k[b][s][h][w] = -scale * sum_t sign(q[b][t][h][w] - k[b][s][h][w]) * g[b][s][t][h]
// with sign(0) = 0.  Both are instances of
//   out[x][h][w] = scale * sum_y sign(a[x][h][w] - b[y][h][w]) * G(x, y, h)
// (d_q: a=q, b=k, G(t,s)=g[s][t];  d_k: a=k, b=q, G(s,t)=g[s][t]), so one kernel serves both
// and one launch runs the two passes side by side (blockIdx decides).  Each CTA owns an x tile,
// 8 heads and a slice of the width, keeps its `a` values and accumulators in registers and
// streams y in tiles through shared memory.  Every output element is produced by exactly one
// thread in a fixed order: no atomics, bit-reproducible.
#include <cstdlib>
#include "common.cuh"
#include "dense_bwd_tiles.h"

namespace l1b {
namespace {

constexpr int HG = 8;  // heads per CTA = lanes along heads
constexpr int LW = 4;  // lanes along the width (16-byte vectors)
constexpr int TY = 16; // y rows per shared-memory tile
constexpr int NCH = 8; // 16-byte chunks per shared row (both tiles)

// one element, global -> shared, asynchronously; !ok: zero
template <typename T> __device__ __forceinline__ void copy_element(T *dst, const T *src, bool ok)
{
	const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
	asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(sizeof(T)), "r"(ok ? int(sizeof(T)) : 0) : "memory");
}

// One source-side row for a thread: acc[i][e] += sign(a[i][e] - b[e]) * g[i].
template <int TM, int VEC>
__device__ __forceinline__ void row_terms(const float (&a)[TM][VEC], const float (&b)[VEC], const float (&g)[TM], float (&acc)[TM][VEC], bool)
{
#pragma unroll
	for (int i = 0; i < TM; i++)
#pragma unroll
		for (int e = 0; e < VEC; e++)
			acc[i][e] += sign_apply(a[i][e] - b[e], g[i]);
}
// fp64: two instructions of the FP64 pipe per term (subtract, add) instead of four -- the comparisons of the exact sign run on that
// pipe too, and it takes two cycles each.  The sign bit of the difference flips g's in the integer pipe, and the high words of
// a thread's eight differences are searched for a zero (a tie, or a difference below 2^-1042); then, and where an operand is
// not finite (odd), the row's terms take the exact form.  a holds no negative zeros, so equal values differ by +0.
// [2,512,8,128]: 420 us for the backward, 558 with the exact sign everywhere and tiles loaded one after the other.
template <int TM, int VEC>
__device__ __forceinline__ void row_terms(const double (&a)[TM][VEC], const double (&b)[VEC], const double (&g)[TM], double (&acc)[TM][VEC], bool odd)
{
	double d[TM][VEC];
	unsigned least = 0xffffffffu;
	bool exact = odd;
#pragma unroll
	for (int e = 0; e < VEC; e++)
		exact = exact || (__double2hiint(b[e]) & 0x7ff00000) == 0x7ff00000;
#pragma unroll
	for (int i = 0; i < TM; i++)
#pragma unroll
		for (int e = 0; e < VEC; e++) {
			d[i][e] = a[i][e] - b[e];
			least = min(least, unsigned(__double2hiint(d[i][e])));
		}
	if (exact || least == 0u) {
#pragma unroll
		for (int i = 0; i < TM; i++)
#pragma unroll
			for (int e = 0; e < VEC; e++)
				acc[i][e] += sign_apply(d[i][e], g[i]);
		return;
	}
#pragma unroll
	for (int i = 0; i < TM; i++)
#pragma unroll
		for (int e = 0; e < VEC; e++)
			acc[i][e] += __hiloint2double(__double2hiint(g[i]) ^ (__double2hiint(d[i][e]) & int(0x80000000)), __double2loint(g[i]));
}
__device__ __forceinline__ bool not_finite(float) { return false; }
__device__ __forceinline__ bool not_finite(double x) { return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000; }

template <typename T, int TM, int NWX, int NWW>
__global__ void __launch_bounds__(NWX *NWW * 32, 2)
dense_bwd_kernel(const T *__restrict__ g, const T *__restrict__ q, const T *__restrict__ k,
		 T *__restrict__ d_q, T *__restrict__ d_k, int n_tok, int n_heads, int width, T scale,
		 int vec_ok, int nxt, int nwt, int nhg, int bs, const int *__restrict__ tie_hdr, int g_pitch)
{ // g_pitch: 0, or g lies [b][h][s][t] in rows of that many elements
	if (tie_hdr && tie_hdr[BWD_HDR_OVERFLOW] == 0)
		return; // the single-visit kernel (dense_bwd_svr.cu) has computed this call
	constexpr int VEC = 16 / sizeof(T);
	constexpr int TX = NWX * TM;       // x tile
	constexpr int WR = NWW * LW * VEC; // width slice per CTA
	constexpr int NT = NWX * NWW * 32;
	static_assert(TX / VEC == NCH && WR / VEC == NCH, "tile rows must be 8 chunks of 16 bytes");
	static_assert(TM % VEC == 0, "TM must be whole vectors");
	using V = Pack<T, VEC>;
	extern __shared__ __align__(16) unsigned char smem_raw[];
	V *stages = reinterpret_cast<V *>(smem_raw); // [2]: b[y][h][w chunk], chunk ^= h; then G[y][h][x chunk], chunk ^= h

	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int lane_h = lane & 7, lane_w = lane >> 3;
	const int wx = warp % NWX, ww = warp / NWX;
	long long bid = blockIdx.x;
	const int x0 = int(bid % nxt) * TX;
	bid /= nxt;
	const int w0 = int(bid % nwt) * WR;
	bid /= nwt;
	const int h0 = int(bid % nhg) * HG;
	bid /= nhg;
	const int b = int(bid % bs);
	const int pass = int(bid / bs); // 0: d_q, 1: d_k

	const size_t row = size_t(n_heads) * width;
	const T *av = (pass == 0 ? q : k) + size_t(b) * n_tok * row;
	const T *bv = (pass == 0 ? k : q) + size_t(b) * n_tok * row;
	T *out = (pass == 0 ? d_q : d_k) + size_t(b) * n_tok * row;
	const T *gb = g + size_t(b) * n_tok * n_heads * (g_pitch > 0 ? g_pitch : n_tok);
	const size_t gst = g_pitch > 0 ? 1 : n_heads, gss = g_pitch > 0 ? size_t(g_pitch) : size_t(n_tok) * n_heads;
	const size_t gsh = g_pitch > 0 ? size_t(n_tok) * g_pitch : 1;
	const size_t gsx = pass == 0 ? gst : gss, gsy = pass == 0 ? gss : gst;

	const int h = h0 + lane_h;
	const int wv = ww * LW + lane_w; // this thread's 16-byte chunk within the slice
	const int w = w0 + wv * VEC;

	T a[TM][VEC], acc[TM][VEC];
	bool odd = false; // a value of a is not finite
#pragma unroll
	for (int i = 0; i < TM; i++) {
		const int x = x0 + wx * TM + i;
#pragma unroll
		for (int e = 0; e < VEC; e++) {
			const bool ok = x < n_tok && h < n_heads && w + e < width;
			a[i][e] = ok ? av[size_t(x) * row + size_t(h) * width + w + e] + T(0) : T(1); // (past the end: anything that ties with nothing)
			odd = odd || not_finite(a[i][e]);
			acc[i][e] = T(0);
		}
	}

	// one tile's copies, asynchronous: they land while the tile before is worked on
	auto load_tile = [&](int y0) {
		V *Bt = stages + (y0 / TY & 1) * (2 * TY * HG * NCH), *Gt = Bt + TY * HG * NCH;
		// b tile: [TY][HG][WR]
		for (int v = tid; v < TY * HG * NCH; v += NT) {
			const int c = v % NCH, hh = (v / NCH) % HG, y = v / (NCH * HG);
			const int gy = y0 + y, gh = h0 + hh, gw = w0 + c * VEC;
			V *dst = &Bt[(y * HG + hh) * NCH + (c ^ hh)];
			const bool ok = gy < n_tok && gh < n_heads;
			const T *src = ok ? bv + size_t(gy) * row + size_t(gh) * width + gw : bv;
			if (ok && vec_ok && gw + VEC <= width) {
				cp_async16(dst, src);
			} else {
#pragma unroll
				for (int e = 0; e < VEC; e++)
					copy_element(&dst->v[e], ok && gw + e < width ? src + e : bv, ok && gw + e < width);
			}
		}
		// G tile: [TY][HG][TX], heads fastest in global memory
		T *Gs = reinterpret_cast<T *>(Gt);
		for (int idx = tid; idx < TY * HG * TX; idx += NT) {
			const int hh = idx % HG;
			int x, y;
			if (pass == 0) { // x = t is the contiguous token axis of g
				x = (idx / HG) % TX;
				y = idx / (HG * TX);
			} else { // y = t is
				y = (idx / HG) % TY;
				x = idx / (HG * TY);
			}
			const int gx = x0 + x, gy = y0 + y, gh = h0 + hh;
			const bool ok = gx < n_tok && gy < n_tok && gh < n_heads;
			copy_element(&Gs[((y * HG + hh) * NCH + ((x / VEC) ^ hh)) * VEC + (x % VEC)],
				     ok ? gb + size_t(gx) * gsx + size_t(gy) * gsy + gh * gsh : gb, ok);
		}
	};
	load_tile(0);
	cp_async_commit();
	for (int y0 = 0; y0 < n_tok; y0 += TY) {
		if (y0 + TY < n_tok)
			load_tile(y0 + TY);
		cp_async_commit();
		cp_async_wait<1>();
		__syncthreads();
		const V *Bt = stages + (y0 / TY & 1) * (2 * TY * HG * NCH), *Gt = Bt + TY * HG * NCH;
#pragma unroll 4
		for (int y = 0; y < TY; y++) {
			const V bvec = Bt[(y * HG + lane_h) * NCH + (wv ^ lane_h)];
			T gv[TM];
#pragma unroll
			for (int m = 0; m < TM / VEC; m++) {
				const V t = Gt[(y * HG + lane_h) * NCH + ((wx * TM / VEC + m) ^ lane_h)];
#pragma unroll
				for (int e = 0; e < VEC; e++)
					gv[m * VEC + e] = t.v[e];
			}
			row_terms<TM, VEC>(a, bvec.v, gv, acc, odd);
		}
		__syncthreads();
	}

	if (h < n_heads) {
#pragma unroll
		for (int i = 0; i < TM; i++) {
			const int x = x0 + wx * TM + i;
			if (x >= n_tok)
				continue;
			T *dst = out + size_t(x) * row + size_t(h) * width + w;
			if (vec_ok && w + VEC <= width) {
				V o;
#pragma unroll
				for (int e = 0; e < VEC; e++)
					o.v[e] = acc[i][e] * scale;
				*reinterpret_cast<V *>(dst) = o;
			} else {
#pragma unroll
				for (int e = 0; e < VEC; e++)
					if (w + e < width)
						dst[e] = acc[i][e] * scale;
			}
		}
	}
}

template <typename T, int TM, int NWX, int NWW>
int launch(const T *g, const T *q, const T *k, T *d_q, T *d_k, int bs, int n_tok, int n_heads, int width,
	   const int *tie_hdr, int g_pitch, cudaStream_t st)
{
	constexpr int VEC = 16 / sizeof(T);
	constexpr int TX = NWX * TM, WR = NWW * LW * VEC;
	const int nxt = (n_tok + TX - 1) / TX, nwt = (width + WR - 1) / WR, nhg = (n_heads + HG - 1) / HG;
	const long long nblk = 2LL * bs * nhg * nwt * nxt;
	if (nblk > 0x7fffffffLL)
		return L1ATTN_ERR_SHAPE;
	const int vec_ok = (width % VEC == 0) && aligned(q, 16) && aligned(k, 16) && aligned(d_q, 16) && aligned(d_k, 16);
	const T scale = T(-1.0 / sqrt(double(width)));
	auto kern = dense_bwd_kernel<T, TM, NWX, NWW>;
	constexpr int smem = 2 * 2 * TY * HG * NCH * 16;
	L1B_SHARED_MEMORY(kern, smem);
	kern<<<unsigned(nblk), NWX * NWW * 32, smem, st>>>(
		g, q, k, d_q, d_k, n_tok, n_heads, width, scale, vec_ok, nxt, nwt, nhg, bs, tie_hdr, g_pitch);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

} // namespace

size_t dense_bwd_scratch_bytes(int bs, int n_tok, int n_heads, int width, int dtype)
{
	if (dtype != L1ATTN_F32 || bs <= 0 || n_tok <= 0 || n_heads <= 0 || width <= 0)
		return 16;
	return bwd_scratch_layout(bs, n_tok, n_heads, width).bytes; // tie flags, tie header, tie list, shares of d_k
}

size_t dense_bwd_scratch_bytes_upto(int bs, int n_tok, int n_heads, int width, int dtype)
{
	if (dtype != L1ATTN_F32 || bs < 1 || n_tok < 1 || n_heads < 1 || width < 1)
		return dense_bwd_scratch_bytes(bs, n_tok, n_heads, width, dtype);
	return bwd_scratch_bytes_upto(bs, n_tok, n_heads, width);
}

// The single-visit kernel for rows of any pitch, between the tie detector and the repair of the listed ties, and the exact kernel in
// case the list overflowed.  Returns 1 when nothing was computed (token index beyond 24 bits, too many items).
int dense_bwd_listed_launch(const void *d_attn, int g_pitch, const void *q, const void *k, void *d_q, void *d_k, void *scratch, int bs,
			    int n_tok, int n_heads, int width, cudaStream_t st)
{
	const float *g = (const float *)d_attn, *qf = (const float *)q, *kf = (const float *)k;
	int rc = dense_ties_launch(qf, kf, (unsigned char *)scratch, d_k, bs, n_tok, n_heads, width, 1, st);
	if (!rc)
		rc = dense_bwd_svr_launch(d_attn, g_pitch, 0, q, k, d_q, d_k, scratch, bs, n_tok, n_heads, width, st);
	if (!rc)
		rc = dense_bwd_partsum_launch(d_q, d_k, scratch, bs, n_tok, n_heads, width, st);
	if (rc)
		return rc;
	const int *tie_hdr = (const int *)((const unsigned char *)scratch + bwd_scratch_layout(bs, n_tok, n_heads, width).hdr);
	rc = launch<float, 8, 4, 2>(g, qf, kf, (float *)d_q, (float *)d_k, bs, n_tok, n_heads, width, tie_hdr, g_pitch, st);
	return rc ? rc : dense_tiefix_launch(d_attn, g_pitch, d_q, d_k, (const unsigned char *)scratch, bs, n_tok, n_heads, width, -1, st);
}

int dense_bwd_launch(const void *d_attn, const void *q, const void *k, void *d_q, void *d_k, void *scratch, int bs,
		     int n_tok, int n_heads, int width, int dtype, cudaStream_t st)
{
	if (bs == 0 || n_tok == 0 || n_heads == 0 || width == 0)
		return L1ATTN_OK;
	if (n_tok <= bwd_small_tokens(dtype == L1ATTN_F32))
		return dense_bwd_small_launch(d_attn, q, k, d_q, d_k, bs, n_tok, n_heads, width, dtype, st);
	static const bool no_tma = getenv("L1ATTN_NO_TMA") != nullptr; // debugging aid: force the generic kernel
	static const bool no_sv = getenv("L1ATTN_NO_SV") != nullptr;   // debugging aid: force the two-pass kernel
	// With scratch the tie detector runs first: it lists every exact tie q == k (and marks tiles, for the case
	// that the list overflows -- a device-side fact, no host round trip).  Then a single-visit kernel computes
	// both gradients with the compare form and the listed terms are repaired afterwards.  If the list overflowed
	// that kernel returns at once and an exact one, gated on the same word, does the call: the two-pass kernel with its
	// exact loop where flagged tiles meet, or the any-shape kernel.  Without scratch (or when the detector does not apply)
	// every tile takes the exact loop.
	const bool listed = scratch && dtype == L1ATTN_F32 && aligned(scratch, 256);
	bool tma = !no_tma && dtype == L1ATTN_F32 && width % 4 == 0 && n_heads % 4 == 0; // row pitches that TMA can address
	for (const void *p : {d_attn, q, k, (const void *)d_q, (const void *)d_k})
		tma = tma && aligned(p, 16);
	const float *qf = (const float *)q, *kf = (const float *)k;
	if (tma) {
		unsigned char *flags = nullptr;
		const int *tie_hdr = nullptr;
		int sv = 0;
		if (listed) {
			const BwdScratchLayout sl = bwd_scratch_layout(bs, n_tok, n_heads, width);
			// Both fast kernels are persistent with equal-sized work items, so the last wave of items decides how
			// full the GPU stays: the single-visit kernel (4 heads x 32 columns x 128 query rows per item, ~8 %
			// faster per term) runs unless its item count leaves the SMs markedly emptier than the two-pass
			// kernel's (8 heads x 64 columns x 32 rows per item and gradient) would.
			int sms = 148;
			if (const int rc = multiprocessors(&sms))
				return rc;
			auto fill = [&](double items) { return bwd_wave_fill(items, sms); };
			const double it_sv = double(bs) * ((n_heads + 3) / 4) * ((width + 31) / 32) * ((n_tok + 127) / 128) * sl.ns;
			const double it_tp = 2.0 * bs * ((n_heads + 7) / 8) * ((width + 63) / 64) * ((n_tok + 31) / 32);
			// (and an item of either kernel is only as busy as its head group is full: 4 heads leave half of an
			// 8-head item's lanes idle)
			const double hf_sv = double(n_heads) / (4.0 * ((n_heads + 3) / 4)), hf_tp = double(n_heads) / (8.0 * ((n_heads + 7) / 8));
			const bool want_sv = !no_sv && 1.08 * fill(it_sv) * hf_sv >= fill(it_tp) * hf_tp;
			const int trc = dense_ties_launch(qf, kf, (unsigned char *)scratch, d_k, bs, n_tok, n_heads, width, want_sv, st);
			if (trc < 0)
				return trc;
			if (trc == 0) {
				flags = (unsigned char *)scratch + sl.flags;
				tie_hdr = (const int *)((unsigned char *)scratch + sl.hdr);
				if (want_sv) {
					const int frc = dense_bwd_sv_launch(d_attn, q, k, d_q, d_k, scratch, bs, n_tok, n_heads, width, dtype, st);
					if (frc < 0)
						return frc;
					sv = frc == 0;
					if (!sv) // zero rows are not in the list: the exact loops everywhere
						flags = nullptr, tie_hdr = nullptr;
				}
			}
		}
		const int rc = dense_bwd_tma_launch(d_attn, q, k, d_q, d_k, bs, n_tok, n_heads, width, dtype, flags, tie_hdr, sv, st);
		if (rc < 0)
			return rc;
		if (rc == 0)
			return tie_hdr ? dense_tiefix_launch(d_attn, 0, d_q, d_k, (const unsigned char *)scratch, bs, n_tok, n_heads,
							     width, sv ? -1 : 1, st)
				       : L1ATTN_OK;
		if (sv)
			return L1ATTN_ERR_CUDA; // cannot happen: both fast kernels accept the same shapes and alignments
	} else if (listed && !no_tma && !no_sv) {
		const int rc = dense_bwd_listed_launch(d_attn, 0, q, k, d_q, d_k, scratch, bs, n_tok, n_heads, width, st);
		if (rc <= 0)
			return rc;
	}
	if (dtype == L1ATTN_F32)
		return launch<float, 8, 4, 2>((const float *)d_attn, qf, kf, (float *)d_q, (float *)d_k, bs, n_tok, n_heads, width, nullptr, 0, st);
	return launch<double, 4, 4, 2>((const double *)d_attn, (const double *)q, (const double *)k, (double *)d_q,
				       (double *)d_k, bs, n_tok, n_heads, width, nullptr, 0, st);
}

} // namespace l1b
