// Dense L1 scores, forward -- the B200 fast path.
//
//   attn[b][s][t][h] = scale * sum_w |q[b][t][h][w] - k[b][s][h][w]|
//
// Persistent, warp-specialised kernel: one CTA per SM walks a list of (batch, head-group of 8,
// query tile of 64, key tile of 32) work items.
//   * warp 8 is the producer: one lane issues TMA tensor copies (cp.async.bulk.tensor, no
//     multicast) -- per stage the 64-byte-wide width chunk of the q tile and of the k tile, as
//     [token][head][16 B chunk] boxes with the 64-byte hardware swizzle -- into a ring of NSTAGE
//     shared-memory stages, each guarded by a full/empty mbarrier pair.  It runs ahead across
//     work items, so the next item's tiles land while the current one is still being reduced;
//   * warps 0..7 compute: lanes = 8 heads x 4 query rows, each thread keeps an 8 x 8 (query, key)
//     register tile of its head, reads operands with conflict-free 16-byte shared loads (the
//     swizzle spreads the 8 head-lanes over 8 bank groups) and spends 1.5 issue slots per
//     term (packed sub.f32x2 for two differences; scalar add with |.| as a source modifier).  Eight compute warps with ~160
//     registers each (no spills) measured faster than sixteen with 128;
//   * results leave through shared memory: the compute warps drop their scaled tiles into a
//     [key][query][head] staging buffer (each warp store is one 128-byte row) and one thread issues
//     a single TMA tensor store of the 32 x 64 x 8 box; scattered 4-byte global stores from the
//     register tiles cost over 20 % of the kernel when measured.  When the head count is not a
//     multiple of 4 (row pitch not 16-byte aligned) the tiles are stored directly instead: the 8
//     head-lanes then write 32 contiguous bytes per (s, t), whole sectors either way;
//   * no [b,h,t,w] copy of q/k is ever made (the reference transposes both first).
// Out-of-range rows/heads/width are zero-filled by TMA (|0-0| adds nothing) and masked at the store; 16-byte chunks of
// the last stage that lie past the width altogether are not computed.
//   * rows that TMA cannot address (a width that is no multiple of 4, a base aligned to the element only) are fetched by
//     FOUR producer warps with 4-byte asynchronous copies into the same places; everything else is the same.
// Every mbarrier wait is bounded (tma.cuh); on a timeout the CTA stops and the error word is set.
#include "common.cuh"
#include "tma.cuh"

namespace l1b {
namespace {

// A work item is HG heads x TT query rows x TS key rows with HG * TT = 512: HG = 8 (TT = 64) or, for head counts
// that leave fewer idle lanes in smaller groups (4, 12, 20 ... heads, a head-group shard of a multi-GPU run: 4; 6 or 2 heads: 2;
// 1 or 3: 1), HG = 4, 2, 1 (TT = 128, 256, 512).  The lanes of a warp are the 32 consecutive (query row, head) rows of the q
// tile in any case.
constexpr int CH = 4;       // 16-byte chunks per (token, head) row per stage
constexpr int NCW = 8;      // compute warps: 2 (query halves) x 4 (key groups)
constexpr int NSTAGE = 3;
constexpr int TS = 32;
constexpr int TM = 8, TN = 8;
constexpr int Q_BYTES = 512 * CH * 16;           // 32768: TT * HG rows of 64 bytes
constexpr int K_BYTES_MAX = TS * 8 * CH * 16;    // 16384 (HG = 8; half of it with HG = 4)
constexpr int STAGE_BYTES = Q_BYTES + K_BYTES_MAX; // 49152
constexpr int OUT_BYTES = TS * 512 * 4;          // 65536: staging tile [s][t][h] of the TMA store
constexpr int producer_warps(bool tma) { return tma ? 1 : 4; } // four: one per scheduler, 12 warps of 168 registers

struct Work {
	unsigned ntt, nst, nhg, total;
};

struct Item {
	int t0, s0, h0, b;
};
template <int HG> __device__ __forceinline__ Item decode_item(const Work &wk, unsigned r)
{
	constexpr int TT = 512 / HG;
	Item x;
	x.t0 = int(r % wk.ntt) * TT;
	r /= wk.ntt;
	x.s0 = int(r % wk.nst) * TS;
	r /= wk.nst;
	x.h0 = int(r % wk.nhg) * HG;
	x.b = int(r / wk.nhg);
	return x;
}

// A producer thread's copies of one stage's rows: `rows` consecutive (token, head) rows of 16 columns.  Sixteen lanes cover
// the columns of a row; the four warps take eight rows at a time, so a thread keeps its head and its swizzle (chunk ^=
// row >> 1 & 3 = its warp) and steps a constant number of tokens.
template <int HG>
__device__ __forceinline__ void copy_rows(unsigned char *dst, const float *base, size_t pitch, int rows, int tok, int n_tok, bool ok, int pw, int lane)
{
	const int r = pw * 2 + (lane >> 4), e = lane & 15;
	const float *src = base + size_t(tok + r / HG) * pitch;
	uint32_t d = smem_u32(dst) + r * 64 + (((e >> 2) ^ pw) << 4) + (e & 3) * 4;
	int left = ok ? n_tok - tok - r / HG : 0;
#pragma unroll 4
	for (int i = 0; i < rows / 8; i++) {
		const bool in = left > 0;
		asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(in ? src : base), "r"(in ? 4 : 0) : "memory");
		src += (8 / HG) * pitch;
		d += 512;
		left -= 8 / HG;
	}
}

// T: instantiated for float only: the packed subtract below is fp32.  FULL: the width is a multiple of the stage's 16 columns.
template <typename T, int HG, bool TMA, bool FULL>
__global__ void __launch_bounds__((NCW + producer_warps(TMA)) * 32, 1)
dense_fwd_tma_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
		     const __grid_constant__ CUtensorMap omap, int tma_store, const T *__restrict__ q, const T *__restrict__ k,
		     T *__restrict__ attn, int n_tok, int n_heads, int width, T scale, Work wk, int *err)
{
	constexpr int VEC = 16 / sizeof(T);
	constexpr int WC = CH * VEC;
	constexpr int LT = 32 / HG;  // lanes along the query axis
	constexpr int TT = 512 / HG; // query rows per item
	extern __shared__ __align__(1024) unsigned char smem_raw[];
	// 1024-byte alignment by OFFSET into the shared array: a pointer rebuilt from an integer loses its
	// address space and every access through it becomes a generic load, which measured ~2x slower here
	unsigned char *stages = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
	__shared__ __align__(8) uint64_t full_bar[NSTAGE], empty_bar[NSTAGE];

	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	if (tid == 0) {
		for (int s = 0; s < NSTAGE; s++) {
			mbar_init(&full_bar[s], TMA ? 1 : producer_warps(TMA) * 32);
			mbar_init(&empty_bar[s], NCW);
		}
		mbar_fence_init();
	}
	__syncthreads();

	const int nchunk = (width + WC - 1) / WC;

	if (!TMA && warp >= NCW) {
		// ---------------- producer warps: every thread copies its elements of a stage and arrives when they have landed
		const int pw = warp - NCW;
		const size_t row = size_t(n_heads) * width;
		int st = 0;
		uint32_t ph = 1;
		for (unsigned item = blockIdx.x; item < wk.total; item += gridDim.x) {
			const Item x = decode_item<HG>(wk, item);
			const int head = x.h0 + (pw * 2 + (lane >> 4)) % HG;
			const size_t off = size_t(x.b) * n_tok * row + size_t(head < n_heads ? head : 0) * width;
			for (int ci = 0; ci < nchunk; ci++) {
				if (!mbar_wait_relaxed(&empty_bar[st], ph, err))
					return;
				unsigned char *dst = stages + size_t(st) * STAGE_BYTES;
				const int col = ci * WC + (lane & 15);
				const bool ok = head < n_heads && col < width;
				const size_t o = off + (ok ? col : 0);
				copy_rows<HG>(dst, q + o, row, 512, x.t0, n_tok, ok, pw, lane);
				copy_rows<HG>(dst + Q_BYTES, k + o, row, TS * HG, x.s0, n_tok, ok, pw, lane);
				asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&full_bar[st])) : "memory");
				if (++st == NSTAGE) {
					st = 0;
					ph ^= 1;
				}
			}
		}
		asm volatile("cp.async.wait_all;" ::: "memory");
		return;
	}
	if (TMA && warp == NCW) {
		// ---------------- producer warp: one lane feeds the ring
		if (lane == 0) {
			int st = 0;
			uint32_t ph = 1; // a fresh barrier reads as "previous phase (parity 1) complete"
			for (unsigned item = blockIdx.x; item < wk.total; item += gridDim.x) {
				const Item x = decode_item<HG>(wk, item);
				for (int ci = 0; ci < nchunk; ci++) {
					if (!mbar_wait_relaxed(&empty_bar[st], ph, err))
						return;
					unsigned char *dst = stages + size_t(st) * STAGE_BYTES;
					mbar_expect_tx(&full_bar[st], Q_BYTES + TS * HG * CH * 16);
					tma_load_4d(dst, &qmap, &full_bar[st], ci * WC, x.h0, x.t0, x.b);
					if (HG == 1) // (a box has at most 256 rows along an axis)
						tma_load_4d(dst + Q_BYTES / 2, &qmap, &full_bar[st], ci * WC, x.h0, x.t0 + TT / 2, x.b);
					tma_load_4d(dst + Q_BYTES, &kmap, &full_bar[st], ci * WC, x.h0, x.s0, x.b);
					if (++st == NSTAGE) {
						st = 0;
						ph ^= 1;
					}
				}
			}
		}
		return;
	}

	// ---------------- compute warps
	const int lane_h = lane & (HG - 1), lane_t = lane / HG;
	const int wt = warp & 1, ws = warp >> 1; // 2 query halves x 4 key groups
	// TMA 64-byte swizzle: chunk ^= address bits 7..8 = (row >> 1) & 3, row = token * HG + head within the box.  The
	// q rows of a warp load are base + lane with base a multiple of 32; the k rows are (ws * TN + j) * HG + head,
	// where j contributes to those bits when HG < 8
	const int sw = (lane >> 1) & 3;
	const int swk = (lane_h >> 1) & 3;
	const int qoff = ((wt * (TT / 2) + lane_t) * HG + lane_h) * CH;
	const int koff = Q_BYTES / 16 + ((ws * TN) * HG + lane_h) * CH;
	int st = 0;
	uint32_t ph = 0;
	bool dead = false;
	for (unsigned item = blockIdx.x; item < wk.total; item += gridDim.x) {
		T acc[TM][TN];
#pragma unroll
		for (int i = 0; i < TM; i++)
#pragma unroll
			for (int j = 0; j < TN; j++)
				acc[i][j] = T(0);

		for (int ci = 0; ci < nchunk; ci++) {
			// after a timeout the warp keeps walking its items without waiting (results are
			// invalid and the error word says so) so that it still meets the others at the barriers
			if (!dead && !mbar_wait(&full_bar[st], ph, err))
				dead = true;
			const ulonglong2 *S = reinterpret_cast<const ulonglong2 *>(stages + size_t(st) * STAGE_BYTES);
			const ulonglong2 *qp = S + qoff, *kp = S + koff;
			auto chunk = [&](int c) {
				const int pc = c ^ sw, pk0 = c ^ swk;
				// Each 16-byte operand is two register pairs; the subtraction is the packed
				// sub.f32x2 (one issue slot for two differences), the |.|-accumulation stays
				// scalar because its abs is a free source modifier only there.
				ulonglong2 kv[TN];
#pragma unroll
				for (int j = 0; j < TN; j++)
					kv[j] = kp[j * HG * CH + (pk0 ^ (HG == 8 ? 0 : HG == 4 ? (2 * j) & 3 : HG == 2 ? j & 3 : (j >> 1) & 3))];
#pragma unroll
				for (int i = 0; i < TM; i++) {
					const ulonglong2 qv = qp[i * LT * HG * CH + pc];
#pragma unroll
					for (int j = 0; j < TN; j++) {
						unsigned long long d0, d1;
						float x0, x1, x2, x3;
						asm("sub.f32x2 %0, %1, %2;" : "=l"(d0) : "l"(qv.x), "l"(kv[j].x));
						asm("sub.f32x2 %0, %1, %2;" : "=l"(d1) : "l"(qv.y), "l"(kv[j].y));
						asm("mov.b64 {%0, %1}, %2;" : "=f"(x0), "=f"(x1) : "l"(d0));
						asm("mov.b64 {%0, %1}, %2;" : "=f"(x2), "=f"(x3) : "l"(d1));
						acc[i][j] += fabsf(x0);
						acc[i][j] += fabsf(x1);
						acc[i][j] += fabsf(x2);
						acc[i][j] += fabsf(x3);
					}
				}
			};
			if (FULL || (ci + 1) * WC <= width) {
#pragma unroll
				for (int c = 0; c < CH; c++)
					chunk(c);
			} else {
				const int nc = (width - ci * WC + VEC - 1) / VEC;
#pragma unroll 1
				for (int c = 0; c < nc; c++)
					chunk(c);
			}
			__syncwarp();
			if (lane == 0)
				mbar_arrive(&empty_bar[st]);
			if (++st == NSTAGE) {
				st = 0;
				ph ^= 1;
			}
		}

		const Item x = decode_item<HG>(wk, item);
		if (tma_store) {
			T *stage_out = reinterpret_cast<T *>(stages + size_t(NSTAGE) * STAGE_BYTES);
			if (tid == 0)
				tma_store_wait_read(); // the previous item's store has drained the staging tile
			named_barrier(1, NCW * 32);
			T *o = stage_out + ((ws * TN) * TT + wt * (TT / 2) + lane_t) * HG + lane_h;
#pragma unroll
			for (int j = 0; j < TN; j++)
#pragma unroll
				for (int i = 0; i < TM; i++)
					o[(j * TT + LT * i) * HG] = acc[i][j] * scale;
			fence_proxy_async_smem();
			named_barrier(1, NCW * 32);
			if (tid == 0) {
				tma_store_4d(&omap, stage_out, x.h0, x.t0, x.s0, x.b);
				tma_store_commit();
			}
			continue;
		}
		const int h = x.h0 + lane_h;
		if (h < n_heads) {
			T *ab = attn + size_t(x.b) * n_tok * n_tok * n_heads + h;
#pragma unroll
			for (int j = 0; j < TN; j++) {
				const int s = x.s0 + ws * TN + j;
				if (s >= n_tok)
					continue;
				T *row = ab + size_t(s) * n_tok * n_heads;
#pragma unroll
				for (int i = 0; i < TM; i++) {
					const int t = x.t0 + wt * (TT / 2) + lane_t + LT * i;
					if (t < n_tok)
						row[size_t(t) * n_heads] = acc[i][j] * scale;
				}
			}
		}
	}
	if (tma_store && tid == 0)
		tma_store_wait_read(); // shared memory must outlive the last store's reads
}

template <typename T> CUtensorMapDataType tmap_dtype();
template <> CUtensorMapDataType tmap_dtype<float>() { return CU_TENSOR_MAP_DATA_TYPE_FLOAT32; }

template <typename T, int HG, bool TMA, bool FULL>
int launch(const T *q, const T *k, T *attn, int bs, int n_tok, int n_heads, int width, cudaStream_t st)
{
	constexpr int VEC = 16 / sizeof(T);
	constexpr int TT = 512 / HG;
	// tensor [bs][n_tok][n_heads][width], innermost first; one stage row is CH*VEC elements = 64 bytes
	const uint64_t dims[4] = {uint64_t(width), uint64_t(n_heads), uint64_t(n_tok), uint64_t(bs)};
	const uint64_t strides[3] = {uint64_t(width) * sizeof(T), uint64_t(n_heads) * width * sizeof(T),
				     uint64_t(n_tok) * n_heads * width * sizeof(T)};
	const uint32_t qbox[4] = {CH * VEC, HG, TT < 256 ? TT : 256, 1}, kbox[4] = {CH * VEC, HG, TS, 1};
	CUtensorMap qmap{}, kmap{};
	if (TMA && (!encode_tmap_4d(&qmap, tmap_dtype<T>(), q, dims, strides, qbox, CU_TENSOR_MAP_SWIZZLE_64B) ||
	    !encode_tmap_4d(&kmap, tmap_dtype<T>(), k, dims, strides, kbox, CU_TENSOR_MAP_SWIZZLE_64B)))
		return 1; // caller falls back to the kernel without tensor maps
	int *err = device_error_word();
	if (!err)
		return 1;
	// output [bs][s][t][h] as a tensor for the TMA store; needs a 16-byte row pitch and base
	CUtensorMap omap = qmap;
	int tma_store = 0;
	if (HG >= 4 && (size_t(n_heads) * sizeof(T)) % 16 == 0 && aligned(attn, 16)) {
		const uint64_t odims[4] = {uint64_t(n_heads), uint64_t(n_tok), uint64_t(n_tok), uint64_t(bs)};
		const uint64_t ostr[3] = {uint64_t(n_heads) * sizeof(T), uint64_t(n_tok) * n_heads * sizeof(T),
					  uint64_t(n_tok) * n_tok * n_heads * sizeof(T)};
		const uint32_t obox[4] = {HG, TT, TS, 1};
		tma_store = encode_tmap_4d(&omap, tmap_dtype<T>(), attn, odims, ostr, obox, CU_TENSOR_MAP_SWIZZLE_NONE) ? 1 : 0;
	}
	Work wk;
	wk.ntt = (n_tok + TT - 1) / TT;
	wk.nst = (n_tok + TS - 1) / TS;
	wk.nhg = (n_heads + HG - 1) / HG;
	const long long total = (long long)bs * wk.nhg * wk.ntt * wk.nst;
	if (total > 0x7fffffffLL)
		return L1ATTN_ERR_SHAPE;
	wk.total = unsigned(total);
	int sms = 0;
	if (const int rc = multiprocessors(&sms))
		return rc;
	const unsigned grid = wk.total < unsigned(sms) ? wk.total : unsigned(sms);
	const size_t smem = size_t(NSTAGE) * STAGE_BYTES + OUT_BYTES + 1024;
	auto kern = dense_fwd_tma_kernel<T, HG, TMA, FULL>;
	L1B_SHARED_MEMORY(kern, int(smem));
	const T scale = T(-1.0 / sqrt(double(width)));
	kern<<<unsigned(grid), (NCW + producer_warps(TMA)) * 32, smem, st>>>(qmap, kmap, omap, tma_store, q, k, attn, n_tok, n_heads, width, scale, wk, err);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

} // namespace

// Returns L1ATTN_OK, a negative error, or 1 when this path does not apply (fp64, no tensor-map support) and the caller should
// use the generic kernel.
int dense_fwd_tma_launch(const void *q, const void *k, void *attn, int bs, int n_tok, int n_heads, int width,
			 int dtype, cudaStream_t st)
{
	if (dtype != L1ATTN_F32)
		return 1; // an 8 x 8 tile of doubles does not fit the register file; fp64 uses the generic kernel
	const bool tma = width % 4 == 0 && aligned(q, 16) && aligned(k, 16);
	// the group of heads (x 512 / HG query rows) that leaves the fewest lanes idle, larger groups first: their rows of
	// the output are longer
	int hg = 8;
	long long least = 0;
	for (int c = 8; c >= 1; c /= 2) {
		const long long tt = 512 / c, work = ((n_heads + c - 1) / c * (long long)c) * ((n_tok + tt - 1) / tt * tt);
		if (c == 8 || work < least) {
			hg = c;
			least = work;
		}
	}
#define L1B_FWD(HG_)                                                                                                               \
	if (hg == HG_) {                                                                                                           \
		if (tma && width % 16 == 0)                                                                                        \
			return launch<float, HG_, true, true>((const float *)q, (const float *)k, (float *)attn, bs, n_tok, n_heads, width, st);  \
		if (tma)                                                                                                           \
			return launch<float, HG_, true, false>((const float *)q, (const float *)k, (float *)attn, bs, n_tok, n_heads, width, st); \
		return launch<float, HG_, false, false>((const float *)q, (const float *)k, (float *)attn, bs, n_tok, n_heads, width, st);        \
	}
	L1B_FWD(8) L1B_FWD(4) L1B_FWD(2) L1B_FWD(1)
#undef L1B_FWD
	return 1;
}

} // namespace l1b
