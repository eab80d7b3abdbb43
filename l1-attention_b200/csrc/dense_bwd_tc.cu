// Dense L1 scores, backward, on the tensor cores (fp32, widths up to 128).
//
//   out[x][h][w] = scale * sum_y sign(a[x][h][w] - b[y][h][w]) * G(x, y, h)      pass 0: d_q (x = t, y = s), pass 1: d_k (x = s, y = t)
//
// For one (x, h) this is a product of a [w][y] matrix of signs with the vector G(x, ., h), and the signs are the whole cost: with
// comparisons and predicated adds of fp32 values a term takes three instructions for both gradients.  Here the values are replaced
// by their order codes (dense_codes.h): one 32-bit addition compares two pairs, one byte permutation turns the sign bits of four into
// the bytes -1 (q >= k) and 0, and tcgen05.mma (8-bit integers) does the sums: sum_y sign * G = 2 sum_y [q >= k] G - sum_y G.  Where
// a warp's columns hold a value with a tie in the block of keys at hand, it adds [q > k] to [q >= k] instead of doubling it: ties
// are exact, however many.
//
// Exact sums.  Per (x, h) and tile of 128 y the gradients are written as integers of 30 bits, G = u n with u a power of two, n in four
// signed bytes; the tensor cores' int32 sums of bytes are exact.  So a tile's signed sum is exact up to its own rounding to fp32 (what a
// gradient loses is below 2^-30 of the tile's largest), and the tiles are added in order: no larger an error than a signed sum over
// all rows has, and no atomics.  Gradients that are not finite or above 2^100 set a word, and an exact kernel behind this one
// computes the call.
//
// Rows of an MMA tile (128) are four quarters of 32 columns of one x each; its N = 16 columns are the four bytes of four x, so the
// NC = ceil(width / 32) tiles of a group of four x share one B operand.  Roles of a CTA's 16 warps, one CTA per SM, persistent:
//   0-7     two sets of four: codes of 128 y of their column in registers (64), reused for every x; per tile 64 additions and 32
//           permutations into tensor memory, signal; RING tiles later, the MMAs done, read the four sums and fold them
//   8-11    digits: gradients by plain loads (any pitch, any layout), largest of a row by shuffles, bytes to shared memory (B)
//   12, 14  issue the MMAs of a set each      13  brings codes in by bulk copies      15  nothing (registers move between warpgroups)
// A work item is four (head, x block) pairs, 4 NG x per block: heads innermost in d_attn means four heads are 16 bytes of a sector; with
// fewer heads the pairs are x blocks of the same head.  Set 0 works on pairs 0 and 2, set 1 on 1 and 3.
#include "common.cuh"
#include "dense_codes.h"
#include "tcgen05.cuh"

namespace l1b {
namespace {

constexpr int TY = 128;      // y per tile
constexpr int NPAIR = 4;     // (head, x block) pairs per item
constexpr int NTHREADS = 512;
// registers per thread of the four warpgroups, from 128 at the launch: the sum stays within 4 x 128
constexpr int REGS_SIGNS = 176, REGS_DIGITS = 112, REGS_REST = 48;
static_assert(2 * REGS_SIGNS + REGS_DIGITS + REGS_REST <= 512, "more than the block was launched with");
constexpr int RING = 3;      // MMA tiles in flight per set
constexpr int B_TILE = 2048; // B operand of four x: 16 rows x 128 bytes

struct Args {
	const float *g;
	GradStrides gs;
	const unsigned char *kc, *qc; // code tables
	size_t q_block;
	float *d_q, *d_k;
	int *hdr, *err;
	int bs, n_tok, n_heads, width, t8, hgi; // hgi: heads per item
	unsigned nxt, nhg, per_pass, total;
	float scale;
};
struct Item {
	int pass, b, h0, x0;
};

template <int NC, int NG> struct Plan {
	static constexpr int X = 4 * NG, NT = NC * NG;
	static constexpr int B_PAIR = NG * B_TILE, B_STAGE = NPAIR * B_PAIR;
	static constexpr int XGROUPS = (X + 7) / 8;
	static constexpr int INFO = NPAIR * X;             // int4 per stage
	static constexpr int TPR = 32 / X, YPT = TY / TPR; // threads per row of G, y per thread
	static __host__ __device__ int codes_bytes(int width) { return (TY / 8 + XGROUPS) * width * 16; }
	static __host__ __device__ size_t smem(int width) { return 1024 + size_t(2) * B_STAGE + size_t(4) * codes_bytes(width) + 2 * INFO * 16 + 2 * NT * 1024; }
};

struct Bars {
	uint64_t codes_full[2][2], codes_empty[2][2], b_full[2], b_empty[2], a_full[2][RING], a_done[2][RING];
	uint32_t tmem;
};

template <int X> __device__ __forceinline__ Item item_at(const Args &A, unsigned r)
{
	Item it;
	it.pass = r >= A.per_pass;
	r -= it.pass ? A.per_pass : 0u;
	it.h0 = int(r % A.nhg) * A.hgi; // neighbours in time share the sectors of d_attn
	r /= A.nhg;
	it.x0 = int(r % A.nxt) * (NPAIR / A.hgi * X);
	it.b = int(r / A.nxt);
	return it;
}

// bytes of four terms: -1 where the comparison of a pair holds (bit 15 of a half), else 0
__device__ __forceinline__ uint32_t four_signs(uint32_t x, uint32_t y01, uint32_t y23)
{
	uint32_t r;
	asm volatile("{\n\t.reg .b32 a, b;\n\tadd.u32 a, %1, %2;\n\tadd.u32 b, %1, %3;\n\tprmt.b32 %0, a, b, 0xfdb9;\n\t}"
		     : "=r"(r)
		     : "r"(x), "r"(y01), "r"(y23)); // (volatile: in order, 32 results live at a time)
	return r;
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel)
{
	uint32_t r;
	asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
	return r;
}

template <int NC, int NG>
__global__ void __launch_bounds__(NTHREADS, 1)
dense_bwd_tc_kernel(const __grid_constant__ Args A)
{
	using P = Plan<NC, NG>;
	constexpr int X = P::X, NT = P::NT;
	extern __shared__ unsigned char smem_raw[];
	__shared__ __align__(8) Bars bars;
	unsigned char *Bs = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u); // (by offset: it stays a shared-memory pointer)
	unsigned char *Cs = Bs + 2 * P::B_STAGE;
	const int codes_bytes = P::codes_bytes(A.width);
	int4 *info = reinterpret_cast<int4 *>(Cs + 4 * codes_bytes); // [stage][pair][x]: sums of the upper and the lower two bytes, u
	float *accs = reinterpret_cast<float *>(info + 2 * P::INFO);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int ny = (A.n_tok + TY - 1) / TY;

	if (warp == 12)
		tmem_alloc(&bars.tmem, 512);
	if (tid == 0) {
		for (int i = 0; i < 2; i++) {
			for (int j = 0; j < 2; j++) {
				mbar_init(&bars.codes_full[i][j], 1);
				mbar_init(&bars.codes_empty[i][j], 4);
			}
			for (int j = 0; j < RING; j++) {
				mbar_init(&bars.a_full[i][j], 4);
				mbar_init(&bars.a_done[i][j], 1);
			}
			mbar_init(&bars.b_full[i], 128);
			mbar_init(&bars.b_empty[i], 8);
		}
		mbar_fence_init();
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = bars.tmem;
	// tensor memory: A tiles of 32 columns [set][slot], then accumulators of 16 columns [set][slot]
	constexpr uint32_t D0 = 2 * RING * 32;

	if (warp < 8) { // ---- signs, and the sums back from the tensor cores
		asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_SIGNS));
		const int set = warp >> 2, quarter = warp & 3;
		const uint32_t lanes = tmem + (uint32_t(quarter * 32) << 16);
		uint32_t slot = 0, wrap = 0; // of the tile at hand
		uint32_t cst = 0, cpar = 0;  // codes stage, its parity
		uint32_t sc = 0;             // y tiles so far
		uint32_t tied = 0;           // bit i: the tile i tiles ago added [q > k]
		bool dead = false;
		float *acc = accs + tid; // [tile of a y tile][thread]: in shared memory, so that the loop over tiles stays one body
		uint4 yc[TY / 8];
		// tile `lin` of a y tile, of the stage with parity sp, in `at_slot`, `ago` tiles ago: its sums into acc
		auto flush = [&](int lin, uint32_t sp, uint32_t at_slot, uint32_t parity, int ago) {
			if (!dead && !mbar_wait_inline(&bars.a_done[set][at_slot], parity, A.err))
				dead = true;
			tc_fence_after();
			const int l = lin % NT, xg = (l / NG * 4 + quarter) / NC; // x within the group of four
			int d[4];
			tmem_load4(lanes + D0 + (set * RING + at_slot) * 16 + 4 * xg, d);
			const int4 f = info[sp * P::INFO + (set + 2 * (lin / NT)) * X + l % NG * 4 + xg];
			const int sh = (tied >> ago & 1u) ? 0 : 1;
			const int lo = -((d[1] * 256 + d[0]) << sh) - f.y, hi = -((d[3] * 256 + d[2]) << sh) - f.x; // below 2^24: exact as floats
			acc[lin * 256] = fmaf(fmaf(float(hi), 65536.f, float(lo)), __int_as_float(f.z), acc[lin * 256]);
		};
		for (unsigned item = blockIdx.x; item < A.total; item += gridDim.x) {
			const Item it = item_at<X>(A, item);
			const int xb = NPAIR / A.hgi;
#pragma unroll 1
			for (int lin = 0; lin < 2 * NT; lin++)
				acc[lin * 256] = 0.f;
			for (int yt = 0; yt < ny; yt++, sc++) {
				const uint32_t sp = sc & 1;
				const unsigned char *ys = Cs, *xs = Cs;
#pragma unroll 1
				for (int lin = 0; lin < 2 * NT; lin++) {
					const int hh = lin / NT, l = lin % NT, i = l / NG, gi = l % NG;
					const int chunk = (i * 4 + quarter) % NC, xg = (i * 4 + quarter) / NC;
					const int w = min(chunk * 32 + lane, A.width - 1);
					if (l == 0) {
						if (!dead && !mbar_wait_inline(&bars.codes_full[set][cst], cpar, A.err))
							dead = true;
						ys = Cs + (set * 2 + cst) * codes_bytes;
						xs = ys + (TY / 8) * A.width * 16; // x codes behind the y codes
						if (X < 8) // an x block of 4 may be the upper half of its group of eight
							xs += (it.x0 + (set + 2 * hh) % xb * X) % 8 * 2;
					}
					if (NC == 3 ? gi == 0 : l == 0) { // (NC 1, 2, 4: a quarter keeps its columns)
#pragma unroll
						for (int y = 0; y < TY / 8; y++)
							yc[y] = *reinterpret_cast<const uint4 *>(ys + (y * A.width + w) * 16);
					}
					// the tile RING tiles ago: of this y tile, or of the last one
					if (lin == RING && !dead && !mbar_wait_inline(&bars.b_full[sp], (sc >> 1) & 1, A.err))
						dead = true; // (its info)
					if (lin >= RING || yt > 0)
						flush(lin >= RING ? lin - RING : lin + 2 * NT - RING, lin >= RING ? sp : sp ^ 1, slot, wrap ^ 1, RING - 1);
					if (lin == RING - 1 && yt > 0) { // the last y tile's stage is read
						__syncwarp();
						if (lane == 0)
							mbar_arrive(&bars.b_empty[sp ^ 1]);
					}
					const int x = gi * 4 + xg;
					uint32_t xx = *reinterpret_cast<const unsigned short *>(xs + ((x >> 3) * A.width + w) * 16 + (x & 7) * 2);
					xx |= xx << 16;
					uint32_t o[32];
#pragma unroll
					for (int y = 0; y < TY / 8; y++) {
						o[y * 2] = four_signs(xx, yc[y].x, yc[y].y);
						o[y * 2 + 1] = four_signs(xx, yc[y].z, yc[y].w);
					}
					const bool tie = __any_sync(0xffffffffu, xx & 1u);
					tied = tied << 1 | uint32_t(tie);
					if (tie) { // -2 where q > k, -1 where they are equal
						const uint32_t above = xx - 0x00030003u;
#pragma unroll
						for (int y = 0; y < TY / 8; y++) {
							o[y * 2] &= ~(four_signs(above, yc[y].x, yc[y].y) & 0x01010101u);
							o[y * 2 + 1] &= ~(four_signs(above, yc[y].z, yc[y].w) & 0x01010101u);
						}
					}
					tmem_store32(lanes + (set * RING + slot) * 32, o);
					tc_wait_st();
					tc_fence_before();
					__syncwarp();
					if (lane == 0) {
						mbar_arrive(&bars.a_full[set][slot]);
						if (l == NT - 1)
							mbar_arrive(&bars.codes_empty[set][cst]);
					}
					slot = slot == RING - 1 ? 0 : slot + 1;
					wrap ^= slot == 0;
					if (l == NT - 1) {
						cst ^= 1;
						cpar ^= cst == 0;
					}
				}
			}
			{ // the last tiles
				uint32_t ds = slot, dw = wrap;
				const uint32_t sp = (sc - 1) & 1;
#pragma unroll 1
				for (int i = 0; i < RING; i++) {
					flush(2 * NT - RING + i, sp, ds, dw ^ 1, RING - 1 - i);
					ds = ds == RING - 1 ? 0 : ds + 1;
					dw ^= ds == 0;
				}
				tc_fence_before();
				__syncwarp();
				if (lane == 0)
					mbar_arrive(&bars.b_empty[sp]);
			}
			float *out = it.pass == 0 ? A.d_q : A.d_k;
			const float scale = it.pass == 0 ? A.scale : -A.scale;
#pragma unroll 1
			for (int lin = 0; lin < 2 * NT; lin++) {
				const int v = set + 2 * (lin / NT), l = lin % NT, i = l / NG;
				const int w = (i * 4 + quarter) % NC * 32 + lane, x = it.x0 + v % xb * X + l % NG * 4 + (i * 4 + quarter) / NC;
				if (x < A.n_tok && w < A.width)
					out[((size_t(it.b) * A.n_tok + x) * A.n_heads + it.h0 + v / xb) * A.width + w] = acc[lin * 256] * scale;
			}
		}
	} else if (warp < 12) { // ---- digits of the gradients
		asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_DIGITS));
		constexpr int TPR = P::TPR, YPT = P::YPT;
		const int tc = tid - 256, v = tc & 3, part = (tc >> 2) % TPR, xl = tc / (4 * TPR);
		const int xb = NPAIR / A.hgi;
		uint32_t sc = 0;
		bool dead = false;
		for (unsigned item = blockIdx.x; item < A.total; item += gridDim.x) {
			const Item it = item_at<X>(A, item);
			const int x = it.x0 + v % xb * X + xl;
			const bool row_ok = x < A.n_tok;
			const long long sx = it.pass == 0 ? A.gs.t : A.gs.s, sy = it.pass == 0 ? A.gs.s : A.gs.t;
			const float *gp = A.g + it.b * A.gs.b + (it.h0 + v / xb) * A.gs.h + (row_ok ? x : 0) * sx + (long long)(part * YPT) * sy;
			for (int yt = 0; yt < ny; yt++, sc++, gp += TY * sy) {
				const uint32_t sp = sc & 1;
				const int left = row_ok ? A.n_tok - yt * TY - part * YPT : 0;
				float g[YPT];
				if (left >= YPT) {
					const float *p = gp;
#pragma unroll
					for (int i = 0; i < YPT; i++, p += sy)
						g[i] = __ldg(p);
				} else {
#pragma unroll
					for (int i = 0; i < YPT; i++)
						g[i] = i < left ? __ldg(gp + i * sy) : 0.f;
				}
				float most = 0.f, chk = 0.f;
#pragma unroll
				for (int i = 0; i < YPT; i++) {
					most = fmaxf(most, fabsf(g[i]));
					chk = fmaf(g[i], 0.f, chk); // NaN if anything is not finite
				}
#pragma unroll
				for (int o = 4; o < 4 * TPR; o *= 2)
					most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
				// |G| < 2^(e - 126), e the exponent field: integers n = G 2^(156 - e) below 2^30, u = 2^(e - 156)
				int e = int(__float_as_uint(most) >> 23);
				if (e >= 127 + 100 || !(chk == 0.f))
					A.hdr[CODE_HDR_EXACT] = 1;
				e = max(min(e, 254), 8);
				const float u = __uint_as_float(e < 30 ? 1u << (e - 7) : uint32_t(e - 29) << 23); // (may be subnormal)
				int lift = 0;
				if (e < 30) { // (the factor would overflow: in two steps)
					lift = 64;
#pragma unroll
					for (int i = 0; i < YPT; i++)
						g[i] *= 18446744073709551616.f; // 2^64
				}
				const float to_int = __uint_as_float(uint32_t(283 - e - lift) << 23);
				if (!dead && !mbar_wait_inline(&bars.b_empty[sp], ((sc >> 1) & 1) ^ 1, A.err))
					dead = true;
				unsigned char *B = Bs + sp * P::B_STAGE + v * P::B_PAIR + (xl / 4) * B_TILE;
				const int n = xl % 4 * 4;
				int sum[4] = {0, 0, 0, 0};
#pragma unroll
				for (int c = 0; c < YPT / 16; c++) {
					uint32_t o[4][4];
#pragma unroll
					for (int p = 0; p < 4; p++) {
						uint32_t b[4];
#pragma unroll
						for (int z = 0; z < 4; z++) // (bytes of n, the lower three as signed digits)
							b[z] = (uint32_t(__float2int_rn(g[c * 16 + p * 4 + z] * to_int)) + 0x00808080u) ^ 0x00808080u;
						const uint32_t l01 = prmt(b[0], b[1], 0x5140), h01 = prmt(b[0], b[1], 0x7362);
						const uint32_t l23 = prmt(b[2], b[3], 0x5140), h23 = prmt(b[2], b[3], 0x7362);
						o[0][p] = prmt(l01, l23, 0x5410);
						o[1][p] = prmt(l01, l23, 0x7632);
						o[2][p] = prmt(h01, h23, 0x5410);
						o[3][p] = prmt(h01, h23, 0x7632);
#pragma unroll
						for (int z = 0; z < 4; z++)
							sum[z] = __dp4a(int(o[z][p]), 0x01010101, sum[z]);
					}
					const int y16 = part * (YPT / 16) + c; // chunk of 16 y
#pragma unroll
					for (int z = 0; z < 4; z++)
						*reinterpret_cast<uint4 *>(B + (n + z) * 128 + ((y16 ^ ((n + z) & 7)) << 4)) = make_uint4(o[z][0], o[z][1], o[z][2], o[z][3]);
				}
				int hi = sum[3] * 256 + sum[2], lo = sum[1] * 256 + sum[0];
#pragma unroll
				for (int o = 4; o < 4 * TPR; o *= 2) {
					hi += __shfl_xor_sync(0xffffffffu, hi, o);
					lo += __shfl_xor_sync(0xffffffffu, lo, o);
				}
				if (part == 0)
					info[sp * P::INFO + v * X + xl] = make_int4(hi, lo, __float_as_int(u), 0);
				fence_proxy_async_smem();
				mbar_arrive(&bars.b_full[sp]);
			}
		}
	} else { // ---- MMAs, codes
		asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_REST));
		if ((warp == 12 || warp == 14) && lane == 0) {
			constexpr uint32_t idesc = tc_idesc_s8(16);
			const int set = warp == 14;
			const uint64_t bdesc = tc_desc(smem_u32(Bs)) + ((set * P::B_PAIR) >> 4);
			uint32_t slot = 0, wrap = 0, sc = 0;
			bool dead = false;
			for (unsigned item = blockIdx.x; item < A.total && !dead; item += gridDim.x)
				for (int yt = 0; yt < ny && !dead; yt++, sc++) {
					const uint32_t sp = sc & 1;
					dead = !mbar_wait_inline(&bars.b_full[sp], (sc >> 1) & 1, A.err);
					for (int lin = 0; lin < 2 * NT && !dead; lin++) {
						if (!mbar_wait_inline(&bars.a_full[set][slot], wrap, A.err)) {
							dead = true;
							break;
						}
						tc_fence_after();
						const uint64_t b = bdesc + ((sp * P::B_STAGE + lin / NT * 2 * P::B_PAIR + lin % NG * B_TILE) >> 4);
						const uint32_t a = tmem + (set * RING + slot) * 32, d = tmem + D0 + (set * RING + slot) * 16;
#pragma unroll
						for (int kk = 0; kk < 4; kk++)
							tc_mma_s8(d, a + kk * 8, b + kk * 2, idesc, kk > 0);
						tc_commit(&bars.a_done[set][slot]);
						slot = slot == RING - 1 ? 0 : slot + 1;
						wrap ^= slot == 0;
					}
				}
		}
		if (warp == 13 && lane == 0) {
			const int xb = NPAIR / A.hgi;
			uint32_t st = 0, par = 1;
			bool dead = false;
			for (unsigned item = blockIdx.x; item < A.total && !dead; item += gridDim.x) {
				const Item it = item_at<X>(A, item);
				for (int yt = 0; yt < ny && !dead; yt++)
					for (int hh = 0; hh < 2 && !dead; hh++) {
						for (int set = 0; set < 2; set++) {
							const int v = set + 2 * hh;
							const int x0 = it.x0 + v % xb * X;
							const size_t bh = (size_t(it.b) * A.n_heads + it.h0 + v / xb) * A.t8;
							const unsigned char *q = A.qc + size_t((it.pass == 0 ? yt * TY : x0 < A.n_tok ? x0 : 0) / CODE_BLOCK) * A.q_block;
							const unsigned char *ysrc = it.pass == 0 ? A.kc : q, *xsrc = it.pass == 0 ? q : A.kc;
							const int yg = yt * (TY / 8), ny8 = min(TY / 8, A.t8 - yg);
							const int xg = x0 / 8, nx8 = max(min(P::XGROUPS, A.t8 - xg), 0);
							const uint32_t ybytes = uint32_t(ny8) * A.width * 16, xbytes = uint32_t(nx8) * A.width * 16;
							unsigned char *dst = Cs + (set * 2 + st) * codes_bytes;
							if (!mbar_wait_inline(&bars.codes_empty[set][st], par, A.err)) {
								dead = true;
								break;
							}
							mbar_expect_tx(&bars.codes_full[set][st], ybytes + xbytes);
							bulk_load(dst, ysrc + (bh + yg) * A.width * 16, ybytes, &bars.codes_full[set][st]);
							if (xbytes)
								bulk_load(dst + (TY / 8) * A.width * 16, xsrc + (bh + xg) * A.width * 16, xbytes, &bars.codes_full[set][st]);
						}
						st ^= 1;
						par ^= st == 0;
					}
			}
		}
		__syncwarp();
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 12)
		tmem_free(tmem, 512);
}

template <int NC, int NG>
int launch(Args &A, int sms, cudaStream_t st)
{
	using P = Plan<NC, NG>;
	const int span = NPAIR / A.hgi * P::X;
	A.nxt = unsigned((A.n_tok + span - 1) / span);
	const long long per_pass = (long long)A.bs * A.nhg * A.nxt;
	if (2 * per_pass > 0x7fffffffLL)
		return 1;
	A.per_pass = unsigned(per_pass);
	A.total = unsigned(2 * per_pass);
	auto kern = dense_bwd_tc_kernel<NC, NG>;
	L1B_SHARED_MEMORY(kern, int(P::smem(NC * 32)));
	kern<<<A.total < unsigned(sms) ? A.total : unsigned(sms), NTHREADS, P::smem(A.width), st>>>(A);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

} // namespace

// Enqueue behind dense_codes_launch() on the same stream, with the same scratch.  Returns L1ATTN_OK, a negative error, or 1 when
// nothing was launched.
int dense_bwd_tc_launch(const float *g, GradStrides gs, float *d_q, float *d_k, void *scratch, int bs, int n_tok, int n_heads, int width, cudaStream_t st)
{
	const CodeTables ct = code_tables(bs, n_tok, n_heads, width);
	const unsigned char *sc = static_cast<const unsigned char *>(scratch);
	Args A;
	A.g = g;
	A.gs = gs;
	A.kc = sc + ct.k;
	A.qc = sc + ct.q;
	A.q_block = ct.q_block;
	A.d_q = d_q;
	A.d_k = d_k;
	A.hdr = reinterpret_cast<int *>(static_cast<unsigned char *>(scratch) + ct.hdr);
	A.err = device_error_word();
	if (!A.err)
		return 1;
	A.bs = bs;
	A.n_tok = n_tok;
	A.n_heads = n_heads;
	A.width = width;
	A.t8 = ct.t8;
	A.hgi = n_heads % 4 == 0 ? 4 : n_heads % 2 == 0 ? 2 : 1;
	A.nhg = unsigned(n_heads / A.hgi);
	A.scale = float(-1.0 / sqrt(double(width)));
	int sms = 0;
	if (const int rc = multiprocessors(&sms))
		return rc;
	const int nc = (width + 31) / 32;
	// Groups of four x per pair: as many as fit, fewer where the items would not fill the SMs (an item's fixed cost is about one group).
	auto cost = [&](int ng) {
		const long long span = NPAIR / A.hgi * 4 * ng, items = 2LL * bs * A.nhg * ((n_tok + span - 1) / span);
		return double((items + sms - 1) / sms) * (ng + 1.0 / ((n_tok + TY - 1) / TY));
	};
	int ng = nc <= 2 ? 4 : 2;
	for (int c = ng / 2; c >= (nc == 1 ? 2 : 1); c /= 2)
		if (cost(c) < cost(ng) * 0.97)
			ng = c;
#define L1B_TC(NC, NG)            \
	if (nc == NC && ng == NG) \
		return launch<NC, NG>(A, sms, st);
	L1B_TC(1, 4) L1B_TC(1, 2) L1B_TC(2, 4) L1B_TC(2, 2) L1B_TC(2, 1) L1B_TC(3, 2) L1B_TC(3, 1) L1B_TC(4, 2) L1B_TC(4, 1)
#undef L1B_TC
	return 1;
}

} // namespace l1b
