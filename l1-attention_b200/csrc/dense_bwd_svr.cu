// Dense L1 scores, backward, single visit per term -- rows of any pitch (fp32).
//
// The arithmetic of dense_bwd_sv.cu (one compare and two predicated adds per term for both gradients, ties repaired
// from the detector's list) for the shapes whose rows TMA cannot address: widths or head counts that are not multiples
// of 4, pointers that are aligned to the element only.  What differs is how the operands arrive and how heads are grouped:
//   * every element of d_attn and k comes by a 4-byte asynchronous copy.  That removes the transposition pass: the
//     copies drop d_attn straight into the [s][h][t] order the math reads (row pitch 512/HG + 32/HG floats, so that the
//     32 lanes of a copy, HG heads x 32/HG query rows, hit 32 banks).  16 + HG copies per thread and tile of
//     16 source rows stand against ~1800 instructions of math;
//   * a work item is HG heads x 512/HG query rows x 32 columns, HG = 4, 2 or 1, whichever pads the head and token counts
//     least (bwd_heads_per_item): six heads of 201 tokens are 3 x 2 heads x 256 rows, not 2 x 4 heads x 2 x 128.
// A CTA walks ONE item (or one of its ns ranges of source rows); three operand stages, one CTA barrier per tile.
// d_k: the row groups' partial sums of a tile meet in shared memory one tile behind the math, in a fixed order; an
// item's share goes to scratch and the shares are added in order (no atomics: bit-reproducible).
// A gradient that is not finite makes 2 sum p g - sum g NaN where a signed sum would be infinite.  A sum that is not finite sets a word of
// its own in the header (this kernel's CTAs must agree on the overflow word); dense_bwd_partsum_launch() turns it into the overflow
// word, and the exact kernel behind it computes the call.
//
// Bound by instruction issue, as dense_bwd_sv.cu.  [48,201,6,65]: 268 us (any-shape kernel 1247), [8,512,1,64]: 57 us (736).
#include "common.cuh"
#include "dense_bwd_tiles.h"

namespace l1b {
namespace {

constexpr int TY = 16;      // source rows per tile = warps (each copies one row of every tile)
constexpr int XR = 32;      // query rows per thread
constexpr int NTHREADS = TY * 32;
constexpr int G_FLOATS = TY * (512 + 32);
constexpr int NSTAGE = 3;
// The sums of d_q are folded every 4 to 32 source rows: acc - (sum of g) / 2, half the signed sum so far.  A plain sum of the g where
// q > k grows with the rows even where the signed sum does not, and rounds accordingly; short sets are folded more often, where a
// tile is most of the sum.  Error of d_q against float64, relative to that of one signed sum over all source rows (the exact
// kernel), k N(0,1), q N(0,1) / q 0.3 N(0,1) with gradients 1 + 0.1 N(0,1), without the folding in brackets: 64 tokens
// 0.97 / 1.00 (2.1), 100 tokens 0.92 / 0.96 (2.5), 201 tokens 0.86 / 0.90 (2.6), 333 tokens 0.84 / 0.91 (2.8), 1040 tokens
// 0.37 / 0.22 (0.40).  It costs 1 to 3 % of this kernel.  d_k is such a difference per group of 32 query rows: 0.97 / 0.88,
// 0.79 / 0.56, 0.57 / 0.32, 0.46 / 0.23, 0.27 / 0.13.
__device__ __forceinline__ int fold_mask(int n_tok) { return n_tok <= 64 ? 0 : n_tok <= 128 ? 1 : n_tok <= 256 ? 3 : 7; } // fold behind the quarters of tiles whose number has these bits
template <int HG> struct Stage {
	static constexpr int TX = 512 / HG, PITCH = 544 / HG, B_FLOATS = TY * HG * 32, FLOATS = G_FLOATS + B_FLOATS;
};
constexpr int PK_FLOATS = TY * TY * 32; // [warp][s][lane]
template <int HG> constexpr size_t smem_bytes() { return sizeof(float) * (NSTAGE * Stage<HG>::FLOATS + 2 * PK_FLOATS + 2 * TY * TY + TY * 32); }

struct Items {
	unsigned nws, ntb, nhg, ns;
	int nt; // tiles of TY source rows per item
};

struct Item {
	int b, h0, tb, sh, w0; // batch item, first head, block of query rows, range of source rows, first column
};
template <int HG> __device__ __forceinline__ Item item_at(unsigned r, const Items &wk)
{
	Item x;
	x.w0 = int(r % wk.nws) * 32;
	r /= wk.nws;
	x.sh = int(r % wk.ns);
	r /= wk.ns;
	x.tb = int(r % wk.ntb);
	r /= wk.ntb;
	x.h0 = int(r % wk.nhg) * HG;
	x.b = int(r / wk.nhg);
	return x;
}

__device__ __forceinline__ size_t opaque(size_t x)
{
	asm volatile("" : "+l"(x));
	return x;
}

__device__ __forceinline__ void copy4(float *dst, const float *src, bool ok)
{
	const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
	asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(ok ? 4 : 0) : "memory");
}

// 16 bytes, of which the first n exist (0..4 floats; the others become zeros)
__device__ __forceinline__ void copy16(float *dst, const float *src, int n)
{
	const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(4 * n) : "memory");
}

// HST: the scores' gradients lie [b][h][s][t] with rows of g_pitch floats (a multiple of 4, 16-byte aligned), as the fused operator's
// backward writes them for this kernel: 4 copies of 16 bytes per thread and tile in the place of 16 of 4, and pairs of equal
// rows need no dropping (their gradients are zero already).  K16: k rows are made of 16-byte vectors too.
template <int HG, bool HST, bool K16>
__global__ void __launch_bounds__(NTHREADS, 1)
dense_bwd_svr_kernel(const float *__restrict__ g, int g_pitch, const float *__restrict__ q, const float *__restrict__ k, float *__restrict__ d_q,
		     size_t dq_stride, float *__restrict__ part, int *__restrict__ tie_hdr,
		     const unsigned char *__restrict__ zero_q, const unsigned char *__restrict__ zero_k, int bs, int n_tok, int n_heads, int width, float scale, Items wk, int only_zeros)
{
	using St = Stage<HG>;
	const bool zeros = !HST && tie_hdr[BWD_HDR_ZERO_Q] != 0 && tie_hdr[BWD_HDR_ZERO_K] != 0;
	if (tie_hdr[BWD_HDR_OVERFLOW] != 0 || (only_zeros != 0 && !zeros))
		return; // too many ties to list: the exact kernel computes this call (or dense_bwd_sv_kernel has)
	extern __shared__ __align__(16) float sm[];
	float *pk = sm + NSTAGE * St::FLOATS;   // [tile & 1][warp][s][lane]
	float *cs = pk + 2 * PK_FLOATS;          // [tile & 1][s][h][group]: sum over the group's query rows of g
	float *rowsum = cs + 2 * TY * TY;        // [warp][lane]
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int xg = warp / HG, h = warp % HG;  // math: group of 32 query rows, head
	const Item it = item_at<HG>(blockIdx.x, wk);
	const int w0 = it.w0, sh = it.sh, tb = it.tb, h0 = it.h0, b = it.b;
	const int t0 = tb * St::TX, s_first = sh * wk.nt * TY;
	const size_t row = size_t(n_heads) * width;
	const size_t tok0 = size_t(b) * n_tok;

	// copies of this thread: source row s_first + tile * TY + warp; d_attn elements (t = tl + 32/HG * i, head hl)
	const int hl = lane % HG, tl = lane / HG;
	const float *gp = g + ((tok0 + s_first + warp) * n_tok + t0 + tl) * n_heads + h0 + hl;
	unsigned zq = 0; // bit i: query row t = tl + 32/HG * i of head hl is zero in every column
	if (zeros && h0 + hl < n_heads)
#pragma unroll
		for (int i = 0; i < 16; i++) {
			const int t = t0 + tl + 32 / HG * i;
			if (t < n_tok && zero_q[(tok0 + t) * n_heads + h0 + hl])
				zq |= 1u << i;
		}
	auto load_tile = [&](int m) { // m < wk.nt
		float *st = sm + (m % NSTAGE) * St::FLOATS;
		const int s = s_first + m * TY + warp;
		const bool s_ok = s < n_tok;
		float *bd = st + G_FLOATS + warp * HG * 32;
		const float *ks = k + (tok0 + (s_ok ? s : 0)) * row + size_t(h0) * width + w0;
		if (K16) { // lane: head lane / 8, columns 4 * (lane % 8) ..
			const int j = lane / 8, c = lane % 8 * 4;
			if (j < HG) {
				const int left = s_ok && h0 + j < n_heads ? min(max(width - w0 - c, 0), 4) : 0;
				copy16(bd + j * 32 + c, left > 0 ? ks + size_t(j) * width + c : k, left);
			}
		} else {
#pragma unroll
			for (int j = 0; j < HG; j++) {
				const bool ok = s_ok && h0 + j < n_heads && w0 + lane < width;
				copy4(bd + j * 32 + lane, ok ? ks + size_t(j) * width + lane : k, ok);
			}
		}
		if (HST) {
			constexpr int CPH = St::TX / 4; // 16-byte pieces of a head's row
#pragma unroll
			for (int i = 0; i < 4; i++) {
				const int hh = (lane + 32 * i) / CPH, c = (lane + 32 * i) % CPH * 4;
				const int left = s_ok && h0 + hh < n_heads ? min(max(n_tok - t0 - c, 0), 4) : 0;
				const float *src = g + ((size_t(b) * n_heads + h0 + hh) * n_tok + s) * g_pitch + t0 + c;
				copy16(st + (warp * HG + hh) * St::PITCH + c, left > 0 ? src : g, left);
			}
			return;
		}
		// a zero query row and a zero source row differ in no column: that score's gradient reaches neither
		const unsigned drop = (zq != 0 && s_ok && zero_k[(tok0 + s) * n_heads + h0 + hl]) ? zq : 0u;
		float *dst = st + (warp * HG + hl) * St::PITCH + tl;
		const int t_left = s_ok && h0 + hl < n_heads ? n_tok - t0 - tl : 0;
		const float *src = gp + size_t(m) * TY * n_tok * n_heads;
#pragma unroll
		for (int i = 0; i < 16; i++) {
			const bool ok = 32 / HG * i < t_left && !(drop >> i & 1u);
			copy4(dst + 32 / HG * i, ok ? src + size_t(32 / HG * i) * n_heads : g, ok);
		}
	};
	load_tile(0);
	cp_async_commit();
	if (wk.nt > 1)
		load_tile(1);
	cp_async_commit();

	float a[XR], acc[XR], rsq = 0.f;
	const bool col_ok = h0 + h < n_heads && w0 + lane < width;
	const int rows_ok = col_ok ? n_tok - t0 - xg * XR : 0; // query rows of this thread that exist: i < rows_ok
	const size_t qoff = (tok0 + t0 + xg * XR) * row + size_t(h0 + h) * width + w0 + lane;
#pragma unroll
	for (int i = 0; i < XR; i++) {
		a[i] = i < rows_ok ? q[qoff + i * row] : 0.f;
		acc[i] = 0.f;
	}
	// the tile before the one at hand: its share of d_k for source row `warp` of the tile and every head of the item
	auto reduce = [&](int m) {
		const float *P = pk + (m & 1) * PK_FLOATS + warp * 32 + lane;
		const int s = s_first + m * TY + warp;
		float *out = part + ((size_t(tb) * bs + b) * n_tok + s) * row + size_t(h0) * width + w0 + lane;
		float all = 0.f; // (rows and columns that do not exist add zeros)
#pragma unroll
		for (int j = 0; j < HG; j++) {
			const float4 *C = reinterpret_cast<const float4 *>(cs + ((m & 1) * TY + warp) * TY + j * (TY / HG));
			float v = 0.f;
#pragma unroll
			for (int x = 0; x < TY / HG; x += 4) {
				const float4 c = C[x / 4];
				v += (fmaf(2.f, P[(x * HG + j) * (TY * 32)], -c.x) + fmaf(2.f, P[((x + 1) * HG + j) * (TY * 32)], -c.y)) +
				     (fmaf(2.f, P[((x + 2) * HG + j) * (TY * 32)], -c.z) + fmaf(2.f, P[((x + 3) * HG + j) * (TY * 32)], -c.w));
			}
			if (s < n_tok && h0 + j < n_heads && w0 + lane < width)
				out[size_t(j) * width] = v;
			all += v;
		}
		if (!(fabsf(all) < INFINITY))
			tie_hdr[BWD_HDR_NOT_FINITE] = 1;
	};

	// acc -= (row sum) / 2 over the source rows since the last call; the row sum of query row i sits in lane i
	auto fold = [&]() {
		float *rs = rowsum + warp * 32;
		rs[lane] = rsq;
		__syncwarp();
#pragma unroll
		for (int i4 = 0; i4 < XR / 4; i4++) {
			const float4 x = reinterpret_cast<const float4 *>(rs)[i4];
			acc[i4 * 4] = fmaf(-0.5f, x.x, acc[i4 * 4]);
			acc[i4 * 4 + 1] = fmaf(-0.5f, x.y, acc[i4 * 4 + 1]);
			acc[i4 * 4 + 2] = fmaf(-0.5f, x.z, acc[i4 * 4 + 2]);
			acc[i4 * 4 + 3] = fmaf(-0.5f, x.w, acc[i4 * 4 + 3]);
		}
		rsq = 0.f;
		__syncwarp();
	};
	const int fold_at = fold_mask(n_tok);

	for (int m = 0; m < wk.nt; m++) {
		cp_async_wait<1>(); // this thread's copies of tile m have landed ...
		__syncthreads();     // ... everyone's have; and all are done with the math of tile m - 1 and the sums of tile m - 2
		if (m + 2 < wk.nt)
			load_tile(m + 2);
		cp_async_commit();
		const float *st = sm + (m % NSTAGE) * St::FLOATS;
		const float4 *GT = reinterpret_cast<const float4 *>(st + h * St::PITCH + xg * XR);
		const float *GL = st + h * St::PITCH + xg * XR + lane;
		const float *B = st + G_FLOATS + h * 32 + lane;
		float *pkw = pk + (m & 1) * PK_FLOATS + warp * (TY * 32) + lane;
#pragma unroll 1
		for (int quarter = 0; quarter < 4; quarter++) {
#pragma unroll
			for (int sq = 0; sq < TY / 4; sq++) {
				const int s = quarter * (TY / 4) + sq;
				const float bv = B[s * (HG * 32)];
				float p = 0.f;
#pragma unroll
				for (int i4 = 0; i4 < XR / 4; i4++) {
					const float4 gv = GT[s * (HG * St::PITCH / 4) + i4];
					bwd_sv_terms(acc[i4 * 4], acc[i4 * 4 + 1], acc[i4 * 4 + 2], acc[i4 * 4 + 3], p, a[i4 * 4], a[i4 * 4 + 1],
						     a[i4 * 4 + 2], a[i4 * 4 + 3], bv, gv);
				}
				pkw[s * 32] = p;
				rsq += GL[s * (HG * St::PITCH)]; // lane l sums g of query row l of the group
			}
			if (((m * 4 + quarter) & fold_at) == fold_at)
				fold();
		}
		if (m > 0)
			reduce(m - 1);
		// sums over groups of 32 query rows of source row `warp`, per head: eight lanes hold a group
		const float4 *R = reinterpret_cast<const float4 *>(st + warp * HG * St::PITCH);
#pragma unroll
		for (int j = 0; j < HG; j++)
#pragma unroll
			for (int i = 0; i < St::TX / 128; i++) {
				const float4 x = R[j * (St::PITCH / 4) + i * 32 + lane];
				float c = (x.x + x.y) + (x.z + x.w);
#pragma unroll
				for (int o = 4; o > 0; o >>= 1)
					c += __shfl_xor_sync(0xffffffffu, c, o);
				if (lane % 8 == 0)
					cs[((m & 1) * TY + warp) * TY + j * (TY / HG) + i * 4 + lane / 8] = c;
			}
	}
	fold();
	__syncthreads();
	reduce(wk.nt - 1);
	// (the item is decoded anew, and the 32 addresses one after the other: what is kept over the hot loop spills)
	unsigned block;
	asm volatile("mov.u32 %0, %%ctaid.x;" : "=r"(block));
	const Item o = item_at<HG>(block, wk);
	const int first = o.tb * St::TX + xg * XR, left = o.h0 + h < n_heads && o.w0 + lane < width ? n_tok - first : 0;
	size_t off = opaque(size_t(o.sh) * dq_stride + (size_t(o.b) * n_tok + first) * row + size_t(o.h0 + h) * width + o.w0 + lane);
#pragma unroll
	for (int i = 0; i < XR; i++) {
		if (i < left) {
			const float x = 2.f * scale * acc[i];
			*reinterpret_cast<volatile float *>(d_q + off) = x;
			if (!(fabsf(x) < INFINITY))
				tie_hdr[BWD_HDR_NOT_FINITE] = 1;
		}
		off = opaque(off + row);
	}
}

template <int HG, bool HST, bool K16>
int launch(const float *g, int g_pitch, int only_zeros, const float *q, const float *k, float *d_q, float *d_k, unsigned char *scratch, const BwdScratchLayout &sl,
	   int bs, int n_tok, int n_heads, int width, cudaStream_t st)
{
	Items wk;
	wk.nws = (width + 31) / 32;
	wk.ntb = unsigned(sl.ntb);
	wk.nhg = (n_heads + HG - 1) / HG;
	wk.ns = unsigned(sl.ns);
	wk.nt = ((n_tok + TY - 1) / TY + sl.ns - 1) / sl.ns;
	const long long total = (long long)bs * wk.nhg * wk.ntb * wk.nws * wk.ns;
	if (total > 0x7fffffffLL)
		return 1;
	int *hdr = reinterpret_cast<int *>(scratch + sl.hdr);
	float *part = reinterpret_cast<float *>(scratch + sl.part), *dqp = reinterpret_cast<float *>(scratch + sl.dqpart);
	const size_t n = size_t(bs) * n_tok * n_heads * width;
	const float scale = float(-1.0 / sqrt(double(width)));
	const BwdZeroRows z = bwd_zero_rows_in(d_k, bs, n_tok, n_heads);
	auto kern = dense_bwd_svr_kernel<HG, HST, K16>;
	L1B_SHARED_MEMORY(kern, int(smem_bytes<HG>()));
	kern<<<unsigned(total), NTHREADS, smem_bytes<HG>(), st>>>(g, g_pitch, q, k, sl.ns > 1 ? dqp : d_q, sl.ns > 1 ? n : size_t(0), part, hdr,
								  z.q, z.k, bs, n_tok, n_heads, width, scale, wk, only_zeros);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

} // namespace

// Enqueue after dense_ties_launch() on the same stream, and dense_bwd_partsum_launch() after it.  only_zeros: compute only if the call has pairs
// of zero rows to drop (dense_bwd_sv_kernel does the others).  g_pitch: 0 for d_attn's own layout, else [b][h][s][t] rows of that many floats.
// Returns L1ATTN_OK, a negative error, or 1 when nothing was launched.
int dense_bwd_svr_launch(const void *d_attn, int g_pitch, int only_zeros, const void *q, const void *k, void *d_q, void *d_k, void *scratch, int bs,
			 int n_tok, int n_heads, int width, cudaStream_t st)
{
	const BwdScratchLayout sl = bwd_scratch_layout(bs, n_tok, n_heads, width);
	const float *g = (const float *)d_attn, *qf = (const float *)q, *kf = (const float *)k;
	float *dq = (float *)d_q, *dk = (float *)d_k;
	unsigned char *sc = (unsigned char *)scratch;
	const bool k16 = width % 4 == 0 && aligned(k, 16);
#define L1B_SVR(HG, HST, K16)                    \
	if (sl.hg == HG && (g_pitch > 0) == HST && (!HST || k16 == K16)) \
		return launch<HG, HST, K16>(g, g_pitch, only_zeros, qf, kf, dq, dk, sc, sl, bs, n_tok, n_heads, width, st);
	L1B_SVR(4, false, false) L1B_SVR(2, false, false) L1B_SVR(1, false, false)
	L1B_SVR(4, true, true) L1B_SVR(2, true, true) L1B_SVR(1, true, true)
	L1B_SVR(4, true, false) L1B_SVR(2, true, false) L1B_SVR(1, true, false)
#undef L1B_SVR
	return 1;
}

} // namespace l1b
