// Work-item geometry shared by the fast dense backward (dense_bwd_tma.cu) and the tie detector
// (dense_ties.cu): both must number the (pass, batch, head group, width slice, x tile) items alike.
#pragma once
#include <stddef.h>
#include <cuda_runtime.h>
#include <stdint.h>
namespace l1b {
constexpr int BWD_HG = 8;  // heads per work item
constexpr int BWD_TX = 32; // x rows (tokens) per work item
constexpr int BWD_WS = 64; // width columns per work item
constexpr int BWD_TY = 16; // y rows (tokens of the other side) per pipeline stage

constexpr int BWD_XF = 4;  // x rows per x flag: the rows one warp of the backward owns
constexpr int BWD_WF = 32; // width columns per flag group: the columns one warp of the backward owns,
                           // i.e. those of a 64-wide slice with the same (w % 32) / 16

// Tie flags, one byte each, for G = bs * head groups * width groups (two per width slice):
//   xflag[pass][G][nxf]  rows [4i, 4i+4) of the x side hold a value that ties with some row of the other side
//   yflag[pass][G][ny]   the y tile holds such a row of the other side
// A warp of the backward (4 x rows, 8 heads, 32 width columns) needs the exact loop for a y tile only
// if both flags are set.
struct BwdFlagLayout {
	size_t groups, nxf, ny, nhg, nwf;
	__host__ __device__ size_t group(int b, int h, int w) const { return (size_t(b) * nhg + size_t(h) / BWD_HG) * nwf + size_t(w) / BWD_WS * 2 + size_t(w) % 32 / 16; }
	__host__ __device__ size_t xoff(int pass) const { return size_t(pass) * groups * nxf; }
	__host__ __device__ size_t yoff(int pass) const { return 2 * groups * nxf + size_t(pass) * groups * ny; }
	__host__ __device__ size_t bytes() const { return 2 * groups * (nxf + ny); }
};
inline BwdFlagLayout bwd_flag_layout(int bs, int n_tok, int n_heads, int width)
{
	BwdFlagLayout l;
	l.nhg = (n_heads + BWD_HG - 1) / BWD_HG;
	l.nwf = size_t((width + BWD_WS - 1) / BWD_WS) * (BWD_WS / BWD_WF); // padded to whole width slices
	l.groups = size_t(bs) * l.nhg * l.nwf;
	l.nxf = size_t((n_tok + BWD_TX - 1) / BWD_TX) * (BWD_TX / BWD_XF); // padded to whole x tiles
	l.ny = (n_tok + BWD_TY - 1) / BWD_TY;
	return l;
}

// ---- listed ties, single-visit backward ----
constexpr int BWD_TIE_CAP = 4096; // listed ties per call; more set the overflow word and the flagged exact loops run
constexpr int BWD_SV_TX = 128;    // query rows per work item of the single-visit kernel: d_k leaves it as ceil(n_tok / 128) shares

// The single-visit kernel's work items are (batch, 4 heads, 32 columns, 128 query rows); each walks all source
// rows, or -- when that many items would leave much of the last wave of SMs empty (long context, small batch, a
// shard of a multi-GPU run) -- one of `ns` equal ranges of them, leaving `ns` partial d_q that the summing kernel
// adds.  The choice depends on the shape alone (the SM count is taken as B200's 148) so that the scratch size can
// be stated without a device.  An item's fixed cost (its q rows in, its d_q rows out) is taken as 0.4 tiles.
constexpr int BWD_SV_SMS = 148;
inline double bwd_wave_fill(double items, int sms)
{
	const double waves = double((long long)((items + sms - 1) / sms));
	return waves > 0 ? items / (waves * sms) : 0.0;
}
inline int bwd_sv_splits(int bs, int n_tok, int n_heads, int width, int hg)
{
	const double items = double(bs) * ((n_heads + hg - 1) / hg) * ((width + 31) / 32) * ((n_tok + 512 / hg - 1) / (512 / hg));
	const int tiles = (n_tok + 15) / 16;
	int best = 1;
	double best_eff = bwd_wave_fill(items, BWD_SV_SMS) * tiles / (tiles + 0.4);
	for (int ns = 2; ns <= 8; ns *= 2) {
		const double tp = double((tiles + ns - 1) / ns);
		if (tp < 8)
			break;
		const double eff = bwd_wave_fill(items * ns, BWD_SV_SMS) * tp / (tp + 0.4);
		if (eff > best_eff * 1.02) { // (not for a percent or two: a split costs one more pass over d_q)
			best = ns;
			best_eff = eff;
		}
	}
	return best;
}

// Heads per work item of the single-visit kernels: 4 x 128 query rows where TMA reads d_attn and k (both row pitches are
// multiples of 16 bytes), else 4 x 128, 2 x 256 or 1 x 512, whichever pads the head and the token count least.
inline int bwd_heads_per_item(int n_tok, int n_heads, int width)
{
	if (n_heads % 4 == 0 && width % 4 == 0)
		return 4;
	int best = 4;
	long long least = 0;
	for (int hg = 4; hg >= 1; hg /= 2) {
		const long long tx = 512 / hg, padded = ((n_heads + hg - 1) / hg * (long long)hg) * ((n_tok + tx - 1) / tx * tx);
		if (hg == 4 || padded < least) {
			best = hg;
			least = padded;
		}
	}
	return best;
}

// The tie header: listed ties; set when not every tie is listed; set when some q (k) row is zero in every column; set by
// dense_bwd_svr_kernel when a sum of its is not finite
constexpr int BWD_HDR_COUNT = 0, BWD_HDR_OVERFLOW = 1, BWD_HDR_ZERO_Q = 2, BWD_HDR_ZERO_K = 3, BWD_HDR_NOT_FINITE = 4;

// Caller-provided scratch of the dense backward, in this order (every part 256-byte aligned):
//   tie flags | tie header | tie list uint4[BWD_TIE_CAP] | shares of d_k | partial d_q (if split)
// The flags and the header are adjacent so that one memset clears both.
struct BwdScratchLayout {
	size_t flags, hdr, ties, part, dqpart, bytes; // offsets, total
	int ntb, ns, hg;
};
inline BwdScratchLayout bwd_scratch_layout(int bs, int n_tok, int n_heads, int width)
{
	auto pad = [](size_t n) { return (n + 255) / 256 * 256; };
	BwdScratchLayout l;
	l.flags = 0;
	l.hdr = pad(bwd_flag_layout(bs, n_tok, n_heads, width).bytes());
	l.ties = l.hdr + 256;
	l.part = l.ties + size_t(BWD_TIE_CAP) * 16;
	l.hg = bwd_heads_per_item(n_tok, n_heads, width);
	l.ntb = (n_tok + 512 / l.hg - 1) / (512 / l.hg);
	l.ns = bwd_sv_splits(bs, n_tok, n_heads, width, l.hg);
	const size_t n = size_t(bs) * n_tok * n_heads * width * 4;
	l.dqpart = l.part + pad(size_t(l.ntb) * n);
	l.bytes = l.dqpart + (l.ns > 1 ? pad(size_t(l.ns) * n) : 0);
	return l;
}

// Scratch for any call of 1 .. bs items.  That can be more than a call of bs items needs: fewer items may split their source rows
// over more ranges, and every range has a partial d_q of its own (600 tokens, 16 heads, 64 columns: 135 MB for 11 items,
// 221 MB for 10).
inline size_t bwd_scratch_bytes_upto(int bs, int n_tok, int n_heads, int width)
{
	size_t most = bwd_scratch_layout(bs, n_tok, n_heads, width).bytes;
	if ((n_tok + 15) / 16 <= 14)
		return most; // too few tiles to be split: the layout grows with the items
	for (int c = bs - 1; c >= 1; c--) {
		const BwdScratchLayout l = bwd_scratch_layout(c, n_tok, n_heads, width);
		most = l.bytes > most ? l.bytes : most;
		if (most >= l.dqpart + size_t(8) * c * n_tok * n_heads * width * 4 + 256)
			break; // as much as c items in eight ranges need, and fewer items need less than that
	}
	return most;
}

// Which rows of q and k are zero in every column (padded tokens), a byte per (batch, token, head) of q, then of k: the detector
// leaves them in d_k, which nothing writes before the single-visit kernel is through (its shares are summed into d_k
// by the kernel behind it).  2 bytes a row, where d_k has width * 4.
struct BwdZeroRows {
	unsigned char *q, *k;
};
inline BwdZeroRows bwd_zero_rows_in(void *d_k, int bs, int n_tok, int n_heads)
{
	unsigned char *p = static_cast<unsigned char *>(d_k);
	return BwdZeroRows{p, p + size_t(bs) * n_tok * n_heads};
}

// The tie detector's bitmaps, one for each of the BWD_TIE_COLS columns of a CTA: 64 bits per token, 32 Kbit at least (a false candidate
// costs a small set more than clearing does: with 4 Kbit at least the detector took 17 us instead of 12 at [8,256,8,64];
// 32 KiB per CTA at 1024 tokens: seven CTAs per SM hide the load latency; 128 bits per token held three and took twice the time for
// 1/4 of the false candidates) up to 4096 tokens, fewer beyond: more false candidates to prove, and past ~16k tokens the list
// overflows into the conservative marking.
constexpr int BWD_TIE_COLS = 4;
inline int bwd_bitmap_log2bits(int n_tok)
{
	int log2bits = 15;
	while (log2bits < 18 && (1 << log2bits) < 64 * n_tok)
		log2bits++;
	return log2bits;
}
inline size_t bwd_bitmap_bytes(int n_tok) { return size_t(BWD_TIE_COLS) << bwd_bitmap_log2bits(n_tok) >> 3; }
// The detector's pass over the zeros keeps two mask bytes per token where the bitmaps were, in whole 8-byte entries: up to 65536 tokens
// fit.  Beyond, zeros are candidates like any other value.
inline size_t bwd_zero_mask_bytes(int n_tok) { return (2 * size_t(n_tok) + 7) / 8 * 8; }
inline bool bwd_zeros_apart(int n_tok) { return bwd_zero_mask_bytes(n_tok) <= bwd_bitmap_bytes(n_tok); }

// Token counts that take one exact kernel without scratch (dense_bwd_small.cu).  fp32, 33 to 48 tokens: the single-visit kernels' sums
// of up to 32 gradients, of which half the total is taken away, round up to 1.7 times as much as one signed sum of so few (33 tokens,
// gradients 1 + 0.1 N(0,1)), and most of an item of 128 query rows is padding.  With fp64 more rows do not fit the registers.
inline int bwd_small_tokens(bool f32) { return f32 ? 48 : 32; }

#ifdef __CUDACC__
// Four terms of the single-visit backward: four compares, then the eight predicated adds they feed -- the query rows'
// sums and p, the source row's.
__device__ __forceinline__ void bwd_sv_terms(float &acc0, float &acc1, float &acc2, float &acc3, float &p, float a0, float a1, float a2,
					     float a3, float bv, const float4 &g)
{
	asm("{\n\t.reg .pred p0, p1, p2, p3;\n\t"
	    "setp.gt.f32 p0, %5, %9;\n\tsetp.gt.f32 p1, %6, %9;\n\tsetp.gt.f32 p2, %7, %9;\n\tsetp.gt.f32 p3, %8, %9;\n\t"
	    "@p0 add.f32 %0, %0, %10;\n\t@p1 add.f32 %1, %1, %11;\n\t@p2 add.f32 %2, %2, %12;\n\t@p3 add.f32 %3, %3, %13;\n\t"
	    "@p0 add.f32 %4, %4, %10;\n\t@p1 add.f32 %4, %4, %11;\n\t@p2 add.f32 %4, %4, %12;\n\t@p3 add.f32 %4, %4, %13;\n\t}"
	    : "+f"(acc0), "+f"(acc1), "+f"(acc2), "+f"(acc3), "+f"(p)
	    : "f"(a0), "f"(a1), "f"(a2), "f"(a3), "f"(bv), "f"(g.x), "f"(g.y), "f"(g.z), "f"(g.w));
}
#endif
} // namespace l1b
