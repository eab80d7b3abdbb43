// Tie detector for the fast dense backward.
//
// The two-instruction form of the backward (dense_bwd_tma.cu) is valid for a stretch of work only
// if none of its `a` values equals a `b` value of the same (batch, head, width index): sign(0) must
// be 0, and the compare form cannot see a tie.  This kernel finds every token row that takes part
// in such a tie and marks the row groups that contain one (layout: dense_bwd_tiles.h); a warp of the
// backward runs its exact loop where its marked x rows meet a marked y tile and the short loop elsewhere.
//
// Exact, in two steps.  One CTA handles NC width columns of one (batch, head):
//   1. filter: every k value sets three bits of one hashed word of its column's bitmap in shared
//      memory; a q value whose three bits are all set is a candidate.  With 64 bits per token (up to
//      4096 tokens) the false-candidate rate is ~1/1000 per value: about four candidates per CTA;
//   2. proof: every candidate value is compared, bit pattern against bit pattern, with all k values
//      of its column (held in registers by the threads that loaded them).  Matching k rows and
//      the candidate's q row are the rows that tie.
// Values are canonical bit patterns (-0 becomes +0); NaNs are skipped because they equal nothing.
// If a CTA finds more candidates than its list holds (heavy ties: q == k, a coarse grid of values) it falls
// back to marking conservatively, without the proof: its candidate q rows and every k row of the
// group.  Marking too much only costs speed, never correctness; proving 512 candidates against every k value first
// took 12 ms at [4,1024,8,64] with a quarter of the tokens padded, where the backward takes 0.8.
// Padded tokens -- rows of q and k that are zero in every column -- tie in every column with each other.  Where the kernel that
// follows drops those pairs itself (they differ in no column: the score's gradient counts as zero) they are not
// candidates, and such calls keep the fast path.
#include <cooperative_groups.h>
#include "common.cuh"
#include "dense_bwd_tiles.h"

namespace l1b {
namespace {

constexpr int NT_MAX = 1024; // threads per CTA: 256..1024, chosen so that one batch of TB tokens per thread covers n_tok when possible
constexpr int TB = 4;    // tokens per thread per batch
constexpr int CAP = 512; // candidate list entries per CTA

__device__ __forceinline__ unsigned canon(float x) { return __float_as_uint(x + 0.0f); }
// The three filter bits of a value lie in ONE 32-bit word of its column's bitmap: the word comes from the top bits of
// one hash, the bit positions from a second one.  One shared-memory atomic per k value and one load per q value (bits
// in two words cost twice that, and the shared-memory atomics and the proof loop over the candidates are what
// bounds this kernel; two bits in one word gave three times the false candidates and a 35 % slower kernel).
__device__ __forceinline__ unsigned hash_word(unsigned b, int sh) { return (b * 0x9E3779B1u) >> sh; } // sh = 32 - log2(words)
__device__ __forceinline__ unsigned hash_bits(unsigned b)
{
	const unsigned x = (b ^ (b >> 15)) * 0xC2B2AE3Du;
	return (1u << (x >> 27)) | (1u << ((x >> 22) & 31u)) | (1u << ((x >> 17) & 31u));
}

template <int NC>
__device__ __forceinline__ void load_batch(const float *base, size_t row, int t0, int n_tok, int ncol, bool vec, float (&v)[TB][NC])
{
	const int NT = blockDim.x;
#pragma unroll
	for (int i = 0; i < TB; i++) {
		const int t = t0 + i * NT;
		if (NC == 4 && vec && ncol == 4) {
			float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
			if (t < n_tok)
				x = *reinterpret_cast<const float4 *>(base + size_t(t) * row);
			v[i][0] = x.x;
			v[i][1 % NC] = x.y;
			v[i][2 % NC] = x.z;
			v[i][3 % NC] = x.w;
		} else {
#pragma unroll
			for (int j = 0; j < NC; j++)
				v[i][j] = (t < n_tok && j < ncol) ? base[size_t(t) * row + j] : 0.f;
		}
	}
}

// What a launch works on.
struct ZeroArgs {
	const float *q, *k;
	unsigned char *zero_q, *zero_k; // tables to be filled (a byte per row), or null: zero rows are no special case
	unsigned char *flags;
	int *hdr;
	BwdFlagLayout fl;
	int n_tok, n_heads, width, ncg; // ncg: CTAs (groups of NC columns) per (batch, head)
	int apart;                      // zeros have a pass of their own (bwd_zeros_apart())
};

// The ties between zeros in the CTA's columns, where both q and k hold some: padded tokens tie with one another in every column, and each
// zero among the values of another row ties with all of them.  A pass of its own, out of line, behind the hot loops: with the test for
// zero rows inside these, even as a call, the kernel took 150 us instead of 103 at [16,1024,16,64].
//   1. per token: which columns are zero, and is the whole row?  (the CTAs of the first columns write the tables)
//   2. the zeros of rows that are not zero throughout, a short list on either side
//   3. every q zero against the k zeros of that list, every q zero of that list against the zero k rows.
// smem: `room` uint2, of which the first (2 n_tok + 7) / 8 hold the tokens' masks (bwd_zeros_apart(): they fit).
template <int NC>
__device__ __noinline__ void zero_ties(const ZeroArgs &z, uint2 *smem, int room, uint4 *tie_list, int &n_hits, int &hit_base)
{
	constexpr int SHORT = 256;
	constexpr unsigned ROW = 0x80u;
	__shared__ unsigned zlist[2][SHORT]; // {column << 24 | token}: of k, of q
	__shared__ int n_short[2], found[2];
	const int NT = blockDim.x, n_tok = z.n_tok;
	const int w0 = int(blockIdx.x % z.ncg) * NC, h = int(blockIdx.x / z.ncg % z.n_heads), b = int(blockIdx.x / z.ncg / z.n_heads);
	const int ncol = min(NC, z.width - w0);
	const bool drop = z.zero_q != nullptr;
	unsigned char *mask = reinterpret_cast<unsigned char *>(smem); // of k, then of q
	uint2 *hits = smem + (2 * n_tok + 7) / 8;
	room -= (2 * n_tok + 7) / 8;
	if (threadIdx.x < 2)
		n_short[threadIdx.x] = found[threadIdx.x] = 0;
	if (threadIdx.x == 0)
		n_hits = 0;
	__syncthreads();
	for (int side = 0; side < 2; side++)
		for (int t = threadIdx.x; t < n_tok; t += NT) {
			const size_t r = (size_t(b) * n_tok + t) * z.n_heads + h;
			const float *row = (side == 0 ? z.k : z.q) + r * z.width;
			unsigned m = 0u;
			for (int j = 0; j < ncol; j++)
				m |= unsigned(row[w0 + j] == 0.f) << j;
			if (drop && m == (1u << ncol) - 1u) {
				bool zero = true;
				for (int w = 0; w < z.width && zero; w += 8) { // (eight loads in flight)
					float x = 0.f;
#pragma unroll
					for (int e = 0; e < 8; e++)
						x = w + e < z.width && !(row[w + e] == 0.f) ? 1.f : x;
					zero = x == 0.f;
				}
				if (zero) {
					m |= ROW;
					found[side] = 1;
				}
			}
			mask[side * n_tok + t] = (unsigned char)m;
			if (drop && w0 == 0)
				(side == 0 ? z.zero_k : z.zero_q)[r] = (m & ROW) != 0u;
			if (m != 0u) { // for the exact loops, should the list overflow
				const size_t g = z.fl.group(b, h, w0); // (the CTA's columns share a flag group)
				z.flags[z.fl.xoff(side == 0 ? 1 : 0) + g * z.fl.nxf + t / BWD_XF] = 1;
				z.flags[z.fl.yoff(side == 0 ? 0 : 1) + g * z.fl.ny + t / BWD_TY] = 1;
			}
			if ((m & ROW) == 0u)
				for (int j = 0; j < ncol; j++)
					if (m >> j & 1u) {
						const int i = atomicAdd(&n_short[side], 1);
						if (i < SHORT)
							zlist[side][i] = unsigned(j) << 24 | unsigned(t);
					}
		}
	__syncthreads();
	if (threadIdx.x == 0 && found[0])
		z.hdr[BWD_HDR_ZERO_K] = 1;
	if (threadIdx.x == 0 && found[1])
		z.hdr[BWD_HDR_ZERO_Q] = 1;
	bool lost = n_short[0] > SHORT || n_short[1] > SHORT;
	for (int side = 0; side < 2 && !lost; side++)
		for (int i = 0; i < n_short[side]; i++) {
			const unsigned e = zlist[side][i];
			const int j = int(e >> 24), t = int(e & 0xffffffu);
			for (int o = threadIdx.x; o < n_tok; o += NT) {
				const unsigned m = mask[(1 - side) * n_tok + o];
				if ((m >> j & 1u) && (side == 0 || (m & ROW))) {
					const int x = atomicAdd(&n_hits, 1);
					if (x < room) // {column << 24 | query row, source row}
						hits[x] = side == 0 ? make_uint2(unsigned(j) << 24 | unsigned(o), unsigned(t)) : make_uint2(e, unsigned(o));
				}
			}
		}
	__syncthreads();
	const int nh = min(n_hits, room);
	if (threadIdx.x == 0 && nh > 0)
		hit_base = atomicAdd(&z.hdr[BWD_HDR_COUNT], nh);
	__syncthreads();
	lost = lost || n_hits > room || (nh > 0 && hit_base + nh > BWD_TIE_CAP);
	if (threadIdx.x == 0 && lost)
		z.hdr[BWD_HDR_OVERFLOW] = 1;
	for (int i = threadIdx.x; i < nh; i += NT)
		if (hit_base + i < BWD_TIE_CAP)
			tie_list[hit_base + i] = make_uint4((unsigned(b) * z.n_heads + h) * z.width + w0 + int(hits[i].x >> 24), hits[i].x & 0xffffffu,
							    hits[i].y, 0u);
}

// grid: bs * n_heads * ceil(width / NC) CTAs.  smem: NC bitmaps of (1 << log2bits) bits.
template <int NC>
__global__ void __launch_bounds__(NT_MAX) dense_ties_kernel(const __grid_constant__ ZeroArgs z, int log2bits, uint4 *tie_list, int vec_ok)
{
	const float *__restrict__ q = z.q, *__restrict__ k = z.k;
	unsigned char *flags = z.flags;
	int *tie_hdr = z.hdr;
	const BwdFlagLayout &fl = z.fl;
	const int n_tok = z.n_tok, n_heads = z.n_heads, width = z.width;
	extern __shared__ unsigned bitmap[]; // [NC][words]
	__shared__ unsigned cand_bits[CAP];  // candidate value
	__shared__ unsigned cand_where[CAP]; // (column << 24) | q token
	__shared__ unsigned char cand_hit[CAP];
	__shared__ int n_cand, overflow, zero_cand, n_hits, hit_base;
	const int NT = blockDim.x;
	const unsigned words = 1u << (log2bits - 5);
	const int sh = 32 - (log2bits - 5);
	const int ncg = (width + NC - 1) / NC;
	unsigned r = blockIdx.x;
	const int w0 = int(r % ncg) * NC;
	r /= ncg;
	const int h = int(r % n_heads);
	const int b = int(r / n_heads);
	const int ncol = min(NC, width - w0);
	{
		uint4 *bm4 = reinterpret_cast<uint4 *>(bitmap);
		for (unsigned i = threadIdx.x; i < NC * words / 4; i += NT)
			bm4[i] = make_uint4(0u, 0u, 0u, 0u);
		for (int i = threadIdx.x; i < CAP; i += NT)
			cand_hit[i] = 0;
		if (threadIdx.x == 0) {
			n_cand = 0;
			n_hits = 0;
			overflow = 0;
			zero_cand = 0;
		}
	}
	__syncthreads();
	const size_t row = size_t(n_heads) * width;
	const float *qb = q + size_t(b) * n_tok * row + size_t(h) * width + w0;
	const float *kb = k + size_t(b) * n_tok * row + size_t(h) * width + w0;
	unsigned char *xq = flags + fl.xoff(0), *xk = flags + fl.xoff(1), *yk = flags + fl.yoff(0), *yq = flags + fl.yoff(1);
	const bool one_batch = n_tok <= NT * TB, vec = vec_ok != 0;
	float v[TB][NC];

	// 1a. k values -> bitmaps
	for (int t0 = threadIdx.x; t0 < n_tok; t0 += NT * TB) {
		load_batch<NC>(kb, row, t0, n_tok, ncol, vec, v);
#pragma unroll
		for (int i = 0; i < TB; i++)
#pragma unroll
			for (int j = 0; j < NC; j++) {
				const float x = v[i][j];
				if (t0 + i * NT < n_tok && j < ncol && x == x) {
					const unsigned bits = canon(x);
					atomicOr(&bitmap[j * words + hash_word(bits, sh)], hash_bits(bits));
				}
			}
	}
	__syncthreads();
	// 1b. q values that pass the filter -> candidate list
	{
		float qv[TB][NC];
		for (int t0 = threadIdx.x; t0 < n_tok; t0 += NT * TB) {
			load_batch<NC>(qb, row, t0, n_tok, ncol, vec, qv);
#pragma unroll
			for (int i = 0; i < TB; i++)
#pragma unroll
				for (int j = 0; j < NC; j++) {
					const float x = qv[i][j];
					const int t = t0 + i * NT;
					if (t < n_tok && j < ncol && x == x) {
						const unsigned bits = canon(x), want = hash_bits(bits);
						if ((bitmap[j * words + hash_word(bits, sh)] & want) == want) {
							if (bits == 0u && z.apart) {
								zero_cand = 1;
							} else {
								const int idx = atomicAdd(&n_cand, 1);
								if (idx < CAP) {
									cand_bits[idx] = bits;
									cand_where[idx] = (unsigned(j) << 24) | unsigned(t);
								} else { // list full: mark this q row without proof
									const size_t g = fl.group(b, h, w0 + j);
									xq[g * fl.nxf + t / BWD_XF] = 1;
									yq[g * fl.ny + t / BWD_TY] = 1;
									overflow = 1;
									tie_hdr[BWD_HDR_OVERFLOW] = 1; // not every tie of this call gets listed
								}
							}
						}
					}
				}
		}
	}
	__syncthreads();
	// the bitmaps are done with: the proven ties {candidate, k token} on their way to the call's list (4 * n_tok at least)
	uint2 *hits = reinterpret_cast<uint2 *>(bitmap);
	const int hit_room = int(NC * words / 2);
	const int nc = min(n_cand, CAP);
	if (w0 == 0 && z.zero_q && !zero_cand) // (the pass over the zeros fills the tables otherwise)
		for (int t = threadIdx.x; t < n_tok; t += NT) {
			const size_t i = (size_t(b) * n_tok + t) * n_heads + h;
			z.zero_q[i] = 0;
			z.zero_k[i] = 0;
		}
	if (nc == 0 && !overflow) {
		if (zero_cand)
			zero_ties<NC>(z, hits, hit_room, tie_list, n_hits, hit_base);
		return;
	}
	// 2. proof: candidates against every k value of their column (k batch still in v when one_batch)
	for (int t0 = threadIdx.x; t0 < n_tok; t0 += NT * TB) {
		if (!one_batch && !overflow)
			load_batch<NC>(kb, row, t0, n_tok, ncol, vec, v);
		for (int ci = 0; ci < nc && !overflow; ci++) {
			const unsigned bits = cand_bits[ci];
			const int col = int(cand_where[ci] >> 24);
#pragma unroll
			for (int i = 0; i < TB; i++) {
				const int t = t0 + i * NT;
#pragma unroll
				for (int j = 0; j < NC; j++)
					if (j == col && t < n_tok && v[i][j] == v[i][j] && canon(v[i][j]) == bits) {
						const size_t g = fl.group(b, h, w0 + j);
						xk[g * fl.nxf + t / BWD_XF] = 1; // k row t equals a q value
						yk[g * fl.ny + t / BWD_TY] = 1;
						cand_hit[ci] = 1;
						const int idx = atomicAdd(&n_hits, 1);
						if (idx < hit_room)
							hits[idx] = make_uint2(unsigned(ci), unsigned(t));
					}
			}
		}
		if (overflow) { // unlisted candidates may match any k row: mark them all
#pragma unroll
			for (int i = 0; i < TB; i++) {
				const int t = t0 + i * NT;
				if (t < n_tok)
					for (int j = 0; j < ncol; j++) {
						const size_t g = fl.group(b, h, w0 + j);
						xk[g * fl.nxf + t / BWD_XF] = 1;
						yk[g * fl.ny + t / BWD_TY] = 1;
					}
			}
		}
	}
	__syncthreads();
	// one reservation in the call's list per CTA
	const int nh = min(n_hits, hit_room);
	if (threadIdx.x == 0 && nh > 0)
		hit_base = atomicAdd(&tie_hdr[BWD_HDR_COUNT], nh);
	__syncthreads();
	if (threadIdx.x == 0 && (n_hits > hit_room || (nh > 0 && hit_base + nh > BWD_TIE_CAP)))
		tie_hdr[BWD_HDR_OVERFLOW] = 1;
	for (int i = threadIdx.x; i < nh; i += NT) {
		const unsigned wv = cand_where[hits[i].x];
		if (hit_base + i < BWD_TIE_CAP) // (batch, head, column), query row, source row
			tie_list[hit_base + i] = make_uint4((unsigned(b) * n_heads + h) * width + w0 + int(wv >> 24), wv & 0xffffffu, hits[i].y, 0u);
	}
	for (int ci = threadIdx.x; ci < nc; ci += NT)
		if (cand_hit[ci] || overflow) { // proven: this q row equals some k value (or not worth a proof any more)
			const unsigned wv = cand_where[ci];
			const int t = int(wv & 0xffffffu), j = int(wv >> 24);
			const size_t g = fl.group(b, h, w0 + j);
			xq[g * fl.nxf + t / BWD_XF] = 1;
			yq[g * fl.ny + t / BWD_TY] = 1;
		}
	if (zero_cand) {
		__syncthreads();
		zero_ties<NC>(z, hits, hit_room, tie_list, n_hits, hit_base);
	}
}

template <int NC>
int launch_nc(ZeroArgs z, int bs, int log2bits, uint4 *tie_list, int vec_ok, cudaStream_t st)
{
	static_assert(NC == BWD_TIE_COLS, "bwd_bitmap_bytes() counts that many bitmaps");
	z.ncg = (z.width + NC - 1) / NC;
	const long long grid = (long long)bs * z.n_heads * z.ncg;
	if (grid > 0x7fffffffLL)
		return 1;
	const size_t smem = bwd_bitmap_bytes(z.n_tok);
	L1B_SHARED_MEMORY(dense_ties_kernel<NC>, int(smem));
	int nt = 256;
	while (nt < NT_MAX && nt * TB < z.n_tok)
		nt *= 2;
	dense_ties_kernel<NC><<<unsigned(grid), nt, smem, st>>>(z, log2bits, tie_list, vec_ok);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

// Repairs the listed ties after the compare-form backward.  That form counts a term as +g where a > b and as -g
// otherwise, so a tie q == k (which must contribute nothing) has put -scale * g into d_q[b][t][h][w]: it gets
// scale * g[b][s][t][h] back.  d_k[b][s][h][w] received -scale * g from the two-pass kernel (which compares k > q
// for it) and +scale * g from the single-visit kernel (one compare q > k for both): dk_sign = +1 / -1.
// One cluster.  The list arrives in no particular order (the detector appends with an atomic counter), so it is
// ranked first -- by (column, query row, source row) for d_q, by (column, source row, query row) for d_k -- and
// every run of entries that hit the same output element is summed by one thread in rank order: the result
// does not depend on the order of arrival.  The ranking compares every entry with every other: the threads of eight CTAs
// take an entry each and leave it, with its term, at its rank in the first CTA's shared memory (d_q) and in the
// second's (d_k), which sum the runs.  One CTA took 153 us for the ~2500 ties of [4,1024,8,64] with padded tokens.
namespace cg = cooperative_groups;
constexpr int FIX_CTAS = 8, FIX_THREADS = 1024; // 8192 threads >= BWD_TIE_CAP

struct FixEntry {
	unsigned col, row; // (batch, head, column); query row (d_q) or source row (d_k)
	float g;
};

__global__ void __cluster_dims__(FIX_CTAS, 1, 1) __launch_bounds__(FIX_THREADS)
dense_tiefix_kernel(const int *__restrict__ tie_hdr, const uint4 *__restrict__ ties, const float *__restrict__ g, int g_pitch,
		    float *__restrict__ d_q, float *__restrict__ d_k, int n_tok, int n_heads, int width, float scale, float dk_scale)
{
	static_assert(FIX_CTAS * FIX_THREADS >= BWD_TIE_CAP, "an entry per thread");
	extern __shared__ __align__(16) unsigned char fix_smem[];
	const int n = min(tie_hdr[BWD_HDR_COUNT], BWD_TIE_CAP);
	if (tie_hdr[BWD_HDR_OVERFLOW] != 0 || n == 0)
		return; // list incomplete (the backward ran its exact loops instead), or no ties
	cg::cluster_group cluster = cg::this_cluster();
	uint4 *e = reinterpret_cast<uint4 *>(fix_smem);                                                     // {column, query row, source row, -}
	FixEntry *sorted = reinterpret_cast<FixEntry *>(fix_smem + size_t(BWD_TIE_CAP) * sizeof(uint4)); // used in the first two CTAs
	for (int i = threadIdx.x; i < n; i += FIX_THREADS)
		e[i] = ties[i];
	cluster.sync(); // the list is complete, and the first two CTAs run: their shared memory may be written from now on
	const unsigned hwn = unsigned(n_heads) * unsigned(width);
	// entry i of this thread: spread over the CTAs first, so that short lists use all of them
	const int i = int(threadIdx.x) * FIX_CTAS + int(cluster.block_rank());
	if (i < n) {
		const uint4 a = e[i];
		const unsigned b = a.x / hwn, hh = (a.x % hwn) / unsigned(width);
		const float gv = g[g_pitch > 0 ? ((size_t(b) * n_heads + hh) * n_tok + a.z) * g_pitch + a.y
					       : ((size_t(b) * n_tok + a.z) * n_tok + a.y) * n_heads + hh];
		int rq = 0, rk = 0;
#pragma unroll 4
		for (int j = 0; j < n; j++) {
			const uint4 c = e[j];
			const bool col_lt = c.x < a.x, col_eq = c.x == a.x;
			rq += (col_lt || (col_eq && (c.y < a.y || (c.y == a.y && c.z < a.z)))) ? 1 : 0;
			rk += (col_lt || (col_eq && (c.z < a.z || (c.z == a.z && c.y < a.y)))) ? 1 : 0;
		}
		// entries are distinct (column, query row, source row) triples: the ranks are a permutation
		cluster.map_shared_rank(sorted, 0)[rq] = FixEntry{a.x, a.y, gv};
		cluster.map_shared_rank(sorted, 1)[rk] = FixEntry{a.x, a.z, gv};
	}
	cluster.sync();
	if (cluster.block_rank() > 1)
		return;
	float *out = cluster.block_rank() == 0 ? d_q : d_k;
	const float factor = cluster.block_rank() == 0 ? scale : dk_scale;
	for (int p = threadIdx.x; p < n; p += FIX_THREADS) {
		const FixEntry a = sorted[p];
		if (p > 0 && sorted[p - 1].col == a.col && sorted[p - 1].row == a.row)
			continue;
		float sum = 0.f;
		for (int pp = p; pp < n && sorted[pp].col == a.col && sorted[pp].row == a.row; pp++)
			sum += sorted[pp].g;
		out[(size_t(a.col / hwn) * n_tok + a.row) * (size_t(n_heads) * width) + a.col % hwn] += factor * sum;
	}
}

} // namespace

// Fills the flag arrays, the tie header and the tie list in `scratch` (device, laid out by bwd_scratch_layout(); the shares
// behind them are not touched), and the zero rows in d_k (bwd_zero_rows_in()).  drop_zero_rows: the kernel that follows drops the pairs
// of zero rows itself, they are not listed.  Returns L1ATTN_OK, a negative error, or 1 when the detector does
// not apply (token index beyond 24 bits); the caller then runs every tile with the exact loop.
int dense_ties_launch(const float *q, const float *k, unsigned char *scratch, void *d_k, int bs, int n_tok, int n_heads, int width,
		      int drop_zero_rows, cudaStream_t st)
{
	if (n_tok >= (1 << 24))
		return 1;
	// four columns as one 16-byte vector where the rows are made of such; the C ABI only promises element alignment
	const int vec_ok = width % 4 == 0 && aligned(q, 16) && aligned(k, 16);
	// four columns per CTA keep the global loads 16 bytes wide
	if ((unsigned long long)bs * n_heads * width > 0xffffffffull)
		return 1; // a tie entry holds the (batch, head, column) index in 32 bits
	const BwdFlagLayout fl = bwd_flag_layout(bs, n_tok, n_heads, width);
	const BwdScratchLayout sl = bwd_scratch_layout(bs, n_tok, n_heads, width);
	L1B_CUDA(cudaMemsetAsync(scratch, 0, sl.hdr + 256, st)); // flags and header
	const BwdZeroRows zr = bwd_zero_rows_in(d_k, bs, n_tok, n_heads);
	const ZeroArgs z{q, k, drop_zero_rows ? zr.q : nullptr, drop_zero_rows ? zr.k : nullptr, scratch + sl.flags,
			 reinterpret_cast<int *>(scratch + sl.hdr), fl, n_tok, n_heads, width, 0, bwd_zeros_apart(n_tok)};
	return launch_nc<BWD_TIE_COLS>(z, bs, bwd_bitmap_log2bits(n_tok), reinterpret_cast<uint4 *>(scratch + sl.ties), vec_ok, st);
}

// Enqueue after the compare-form backward: adds the listed ties' terms back (no-op when the list overflowed).
int dense_tiefix_launch(const void *d_attn, int g_pitch, void *d_q, void *d_k, const unsigned char *scratch, int bs, int n_tok,
			int n_heads, int width, int dk_sign, cudaStream_t st)
{
	const BwdScratchLayout sl = bwd_scratch_layout(bs, n_tok, n_heads, width);
	const size_t smem = size_t(BWD_TIE_CAP) * (sizeof(uint4) + sizeof(FixEntry));
	L1B_SHARED_MEMORY(dense_tiefix_kernel, int(smem));
	dense_tiefix_kernel<<<FIX_CTAS, FIX_THREADS, smem, st>>>(reinterpret_cast<const int *>(scratch + sl.hdr),
						   reinterpret_cast<const uint4 *>(scratch + sl.ties), (const float *)d_attn, g_pitch,
						   (float *)d_q, (float *)d_k, n_tok, n_heads, width,
						   float(-1.0 / sqrt(double(width))), float(-dk_sign / sqrt(double(width))));
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

} // namespace l1b
