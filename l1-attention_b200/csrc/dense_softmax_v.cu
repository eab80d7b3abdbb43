// Fused consumer of the dense L1 scores: softmax over the source tokens and the value product,
// without ever writing the [bs, n_tok, n_tok, n_heads] score tensor.
//
//   x[b][s][t][h]  = scale * sum_w |q[b][t][h][w] - k[b][s][h][w]|          scale = -1/sqrt(width)
//   a              = softmax of x over s                                    (mode SOFTMAX)
//                  | exp(x) / (1 + sum_s exp(x))   "one more all-zero row"  (mode SOFTMAX_PLUS_ONE)
//                  | exp(x)                                                 (mode EXP)
//   vo[b][t][h][:] = sum_s a[b][s][t][h] * v[b][s][h][:]
//
// This is what every dense caller of the reference does right after L1Attn
// (README.md:64-66: F.softmax(a, 1) then einsum 'bsdh,bshw->bdhw'); the "+1" forms are the dense
// equivalents of the sparse operator's normalisation (python/l1attn_sparse.py:491-502).
//
// Three kernels forward (and as many, with the roles swapped, for the first step of the backward):
//   * softmax_v_kernel: any shape, fp32/fp64.  One CTA per (b, t, h) keeps the n_tok scores of its row
//     in shared memory: scores, max, exp/sum, value product, each in a fixed order.
//   * softmax_v_tile_kernel (fp32, width and v_width up to 128): one CTA per (b, h, tile of 64 or 128 query
//     rows) streams the keys and values of its head in tiles of 64 through a ring and keeps running
//     max / sum / output rows in registers (online softmax).  The ring is filled by TMA where rows are whole
//     16-byte vectors, else by 4-byte asynchronous copies of all threads; columns past the end of a row read as zeros.
//   * softmax_v_tc_kernel (fp32, width and v_width up to 64, where CTAs of 128 rows fill the SMs well): the same with the value product
//     on the tensor cores.
// sv_plan() and sv_bwd_plan() choose.
#include <math.h>
#include <stdlib.h>
#include "common.cuh"
#include "tma.cuh"
#include "tcgen05.cuh"
#include "dense_bwd_tiles.h"

namespace l1b {
namespace {

// ------------------------------------------------------------------------------------------------
// generic kernel
// ------------------------------------------------------------------------------------------------
constexpr int GEN_NT = 128;

template <typename T> __device__ __forceinline__ T block_reduce(T v, T *red, bool is_max)
{
	// fixed tree: lanes by shuffle, then warp results in warp order by thread 0
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) {
		const T u = __shfl_xor_sync(0xffffffffu, v, o);
		v = is_max ? (u > v ? u : v) : v + u;
	}
	__syncthreads(); // red may still be read from the previous reduction
	if ((threadIdx.x & 31) == 0)
		red[threadIdx.x >> 5] = v;
	__syncthreads();
	T r = red[0];
	for (int i = 1; i < GEN_NT / 32; i++)
		r = is_max ? (red[i] > r ? red[i] : r) : r + red[i];
	return r;
}

template <typename T>
__global__ void __launch_bounds__(GEN_NT)
softmax_v_kernel(const T *__restrict__ q, const T *__restrict__ k, const T *__restrict__ v, T *__restrict__ vo,
		 T *__restrict__ lse, int n_tok, int n_heads, int width, int v_width, T scale, int mode)
{
	extern __shared__ __align__(16) unsigned char gsm[];
	T *sc = reinterpret_cast<T *>(gsm); // [n_tok] scores, then weights
	T *qrow = sc + n_tok;               // [width]
	T *red = qrow + width;              // [GEN_NT / 32]
	unsigned r = blockIdx.x;
	const int h = int(r % unsigned(n_heads));
	r /= unsigned(n_heads);
	const int t = int(r % unsigned(n_tok));
	const int b = int(r / unsigned(n_tok));
	const size_t row = size_t(n_heads) * width, vrow = size_t(n_heads) * v_width;
	const T *qp = q + (size_t(b) * n_tok + t) * row + size_t(h) * width;
	const T *kb = k + size_t(b) * n_tok * row + size_t(h) * width;
	const T *vb = v + size_t(b) * n_tok * vrow + size_t(h) * v_width;
	for (int w = threadIdx.x; w < width; w += GEN_NT)
		qrow[w] = qp[w];
	__syncthreads();
	T lmax = -INFINITY;
	for (int s = threadIdx.x; s < n_tok; s += GEN_NT) {
		const T *kp = kb + size_t(s) * row;
		T acc = T(0);
		for (int w = 0; w < width; w++)
			acc += absdiff(qrow[w], kp[w]);
		const T x = acc * scale;
		sc[s] = x;
		lmax = x > lmax ? x : lmax;
	}
	T m = T(0); // the "+1" and exp forms do not shift (the reference's sparse operator does not either)
	if (mode == L1ATTN_SV_SOFTMAX)
		m = block_reduce(lmax, red, true);
	T lsum = T(0);
	for (int s = threadIdx.x; s < n_tok; s += GEN_NT) {
		const T e = exp_t(sc[s] - m);
		sc[s] = e;
		lsum += e;
	}
	T denom = block_reduce(lsum, red, false); // also publishes sc[] to every thread
	if (mode == L1ATTN_SV_SOFTMAX_PLUS_ONE)
		denom += T(1);
	if (mode == L1ATTN_SV_EXP)
		denom = T(1);
	if (lse && threadIdx.x == 0) // weight of (s, t) = exp(x - lse)
		lse[(size_t(b) * n_tok + t) * n_heads + h] = m + log(denom);
	T *op = vo + (size_t(b) * n_tok + t) * vrow + size_t(h) * v_width;
	for (int c = threadIdx.x; c < v_width; c += GEN_NT) {
		T o = T(0);
		for (int s = 0; s < n_tok; s++)
			o += sc[s] * vb[size_t(s) * vrow + c];
		op[c] = o / denom;
	}
}

template <typename T>
int launch_generic(const T *q, const T *k, const T *v, T *vo, T *lse, int bs, int n_tok, int n_heads, int width,
		   int v_width, int mode, cudaStream_t st)
{
	const long long grid = (long long)bs * n_tok * n_heads;
	const size_t smem = (size_t(n_tok) + width + GEN_NT / 32) * sizeof(T);
	if (grid > 0x7fffffffLL || smem > 200 * 1024)
		return L1ATTN_ERR_SHAPE;
	auto kern = softmax_v_kernel<T>;
	L1B_SHARED_MEMORY(kern, int(smem));
	kern<<<unsigned(grid), GEN_NT, smem, st>>>(q, k, v, vo, lse, n_tok, n_heads, width, v_width,
						    T(-1.0 / sqrt(double(width))), mode);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

// ------------------------------------------------------------------------------------------------
// TMA kernel (fp32)
// ------------------------------------------------------------------------------------------------
// CTA = NW warps = 2 NW half-warps.  Half-warp `tg` owns TI query rows (t = i*2*NW + tg) and is
// self-contained: for every key tile its 16 lanes first each compute TI x 4 scores (keys
// s = j*16 + lane), reduce the row maxima and sums by shuffles, park the weights in a private slice
// of shared memory, and then each accumulate TI x NV output values (lane = value columns
// [lane*NV, lane*NV+NV)).  Only the key/value ring is shared by the CTA.
// Shared operand rows are 128 bytes (one 32-float slice of the width per TMA box, 128-byte swizzle),
// so the 16 lanes of a half-warp read 16 different key rows without bank conflicts.
constexpr int TS = 64;     // keys per ring stage
constexpr int PP = TS + 4; // row pitch (floats) of the weight tile: the two half-warps of a warp land on different banks
constexpr int MAX_STAGE = 3;

struct SvShape {
	int n_tok, n_heads, width, v_width, nwb, nstage, ntt, mode;
	int dx_pitch; // backward: 0 = dx as d_attn lies, [b][s][t][h]; else [b][h][s][t] in rows of that many floats
	float scale;
};

// Rows that TMA cannot address (a row pitch or base that is no multiple of 16 bytes): the CTA's warps copy `rows` token
// rows, 32 columns at a time, with 4-byte asynchronous copies into the place and order a TMA box would leave them in.
// `base` is the head's row of token 0.  Slices of 32 columns: [slice][row] of 128 bytes, SWZ: 16-byte chunk ^= row & 7;
// !SWZ: [row][32 * slices].  Columns >= width and tokens >= n_tok become zeros.  The copies are ~16 per thread and tile against
// ~2500 instructions of math: [4,300,5,33], values 21 wide, takes 31 us forward and 38 us backward (dx, dv), [4,333,6,48],
// values 40 wide, through TMA 34 and 48 us (the whole pass with the any-shape kernels 1633 us, with these 373).
template <int NW, bool SWZ>
__device__ __forceinline__ void copy_rows(unsigned char *dst, const float *base, size_t pitch, int t0, int rows, int nslice, int width, int n_tok)
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (int sl = 0; sl < nslice; sl++) {
		const int col = sl * 32 + lane;
		for (int r = warp; r < rows; r += NW) {
			const bool ok = col < width && t0 + r < n_tok;
			const float *src = base + (ok ? size_t(t0 + r) * pitch + col : 0);
			const uint32_t d = smem_u32(dst) + (SWZ ? (sl * rows + r) * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4
								: (r * nslice * 32 + col) * 4);
			asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(ok ? 4 : 0) : "memory");
		}
	}
}
// this thread's arrival on `bar` once its asynchronous copies so far have landed
__device__ __forceinline__ void copy_arrive(uint64_t *bar)
{
	asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <int NV, int TI, int NW, bool TMA, bool FULL>
__global__ void __launch_bounds__(NW * 32, 1)
softmax_v_tile_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
		      const __grid_constant__ CUtensorMap vmap, const float *__restrict__ q, const float *__restrict__ k,
		      const float *__restrict__ v, float *__restrict__ vo, float *__restrict__ lse, SvShape sh, int *err)
{
	constexpr int TT = 2 * NW * TI; // query rows of the CTA: a half-warp owns TI of them (t = i*2*NW + tg)
	constexpr int NTH = NW * 32;
	constexpr int VW = 16 * NV; // v_width
	constexpr int V_BYTES = TS * VW * 4;
	extern __shared__ __align__(1024) unsigned char smem_raw[];
	unsigned char *base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
	__shared__ __align__(8) uint64_t q_bar, full_bar[MAX_STAGE], empty_bar[MAX_STAGE];
	const int q_bytes = sh.nwb * TT * 128, k_bytes = sh.nwb * TS * 128, stage_bytes = k_bytes + V_BYTES;
	unsigned char *Qs = base;
	unsigned char *stages = base + q_bytes;
	float *Ps = reinterpret_cast<float *>(stages + size_t(sh.nstage) * stage_bytes);

	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	unsigned r = blockIdx.x;
	const int t0 = int(r % unsigned(sh.ntt)) * TT;
	r /= unsigned(sh.ntt);
	const int h = int(r % unsigned(sh.n_heads));
	const int b = int(r / unsigned(sh.n_heads));
	const int ns = (sh.n_tok + TS - 1) / TS;

	if (tid == 0) {
		mbar_init(&q_bar, TMA ? 1 : NTH);
		for (int s = 0; s < MAX_STAGE; s++) {
			mbar_init(&full_bar[s], TMA ? 1 : NTH);
			mbar_init(&empty_bar[s], NTH / 32);
		}
		mbar_fence_init();
	}
	__syncthreads();

	const size_t krow = size_t(sh.n_heads) * sh.width, vrow = size_t(sh.n_heads) * sh.v_width;
	const size_t qk0 = size_t(b) * sh.n_tok * krow + size_t(h) * sh.width, v0 = size_t(b) * sh.n_tok * vrow + size_t(h) * sh.v_width;
	// key/value tile m goes to stage m % nstage; the caller has made sure the stage is free (TMA: one thread asks;
	// otherwise every thread copies its part and arrives when it has landed)
	auto load_tile = [&](int m) {
		const int st = m % sh.nstage;
		unsigned char *dst = stages + size_t(st) * stage_bytes;
		if (!TMA) {
			copy_rows<NW, true>(dst, k + qk0, krow, m * TS, TS, sh.nwb, sh.width, sh.n_tok);
			copy_rows<NW, false>(dst + k_bytes, v + v0, vrow, m * TS, TS, VW / 32, sh.v_width, sh.n_tok);
			copy_arrive(&full_bar[st]);
			return;
		}
		mbar_expect_tx(&full_bar[st], uint32_t(stage_bytes));
		for (int wb = 0; wb < sh.nwb; wb++)
			tma_load_4d(dst + wb * TS * 128, &kmap, &full_bar[st], wb * 32, h, m * TS, b);
		tma_load_4d(dst + k_bytes, &vmap, &full_bar[st], 0, h, m * TS, b);
	};
	if (!TMA || tid == 0) {
		if (TMA) {
			mbar_expect_tx(&q_bar, uint32_t(q_bytes));
			for (int wb = 0; wb < sh.nwb; wb++)
				tma_load_4d(Qs + wb * TT * 128, &qmap, &q_bar, wb * 32, h, t0, b);
		} else {
			copy_rows<NW, true>(Qs, q + qk0, krow, t0, TT, sh.nwb, sh.width, sh.n_tok);
			copy_arrive(&q_bar);
		}
		for (int m = 0; m < sh.nstage - 1 && m < ns; m++)
			load_tile(m);
	}

	const int sg = lane & 15, tg = warp * 2 + (lane >> 4);
	const bool softmax = sh.mode == L1ATTN_SV_SOFTMAX;
	float o[TI][NV], mrow[TI], lrow[TI];
#pragma unroll
	for (int i = 0; i < TI; i++) {
		mrow[i] = softmax ? -INFINITY : 0.f;
		lrow[i] = sh.mode == L1ATTN_SV_SOFTMAX_PLUS_ONE ? 1.f : 0.f; // the extra all-zero row weighs exp(0)
#pragma unroll
		for (int e = 0; e < NV; e++)
			o[i][e] = 0.f;
	}
	bool dead = false;
	if (!mbar_wait(&q_bar, 0, err))
		dead = true;
	float *Pw = Ps + tg * PP; // weight rows of this half-warp: row i at Pw + i*16*PP

	for (int m = 0; m < ns; m++) {
		// one lane asks for the tile that will be needed nstage-1 tiles from now; its stage held tile
		// m-1, which every warp must have released (the duty rotates so that no warp is always late)
		if ((!TMA || (warp == m % NW && lane == 0)) && m + sh.nstage - 1 < ns && !dead) {
			const int mm = m + sh.nstage - 1;
			if (mbar_wait(&empty_bar[mm % sh.nstage], ((unsigned(mm) / unsigned(sh.nstage)) & 1u) ^ 1u, err))
				load_tile(mm);
			else
				dead = true;
		}
		__syncwarp();
		const int st = m % sh.nstage;
		if (!dead && !mbar_wait(&full_bar[st], (unsigned(m) / unsigned(sh.nstage)) & 1u, err))
			dead = true; // keep walking without waiting; the error word reports the failure
		const unsigned char *Ks = stages + size_t(st) * stage_bytes;
		const float *Vs = reinterpret_cast<const float *>(Ks + k_bytes);

		// ---- scores of TI query rows x 4 keys
		float acc[TI][4];
#pragma unroll
		for (int i = 0; i < TI; i++)
#pragma unroll
			for (int j = 0; j < 4; j++)
				acc[i][j] = 0.f;
		for (int wb = 0; wb < sh.nwb; wb++) {
			const ulonglong2 *Qb = reinterpret_cast<const ulonglong2 *>(Qs + wb * TT * 128);
			const ulonglong2 *Kb = reinterpret_cast<const ulonglong2 *>(Ks + wb * TS * 128);
			const int nc = FULL ? 8 : min(8, ((sh.width - wb * 32 + 7) >> 3) * 2); // 16-byte chunks of this slice, to a pair
#pragma unroll 2
			for (int c = 0; c < nc; c++) {
				ulonglong2 kv[4];
#pragma unroll
				for (int j = 0; j < 4; j++) // row j*16+sg, chunk c ^ (row & 7)
					kv[j] = Kb[(j * 16 + sg) * 8 + (c ^ (sg & 7))];
#pragma unroll
				for (int i = 0; i < TI; i++) {
					const ulonglong2 qv = Qb[(i * (2 * NW) + tg) * 8 + (c ^ (tg & 7))];
#pragma unroll
					for (int j = 0; j < 4; j++) {
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
			}
		}

		// ---- weights: running max / sum per query row, rescale of the output rows
#pragma unroll
		for (int i = 0; i < TI; i++) {
			float x[4], mx = -INFINITY;
#pragma unroll
			for (int j = 0; j < 4; j++) {
				x[j] = (m * TS + j * 16 + sg < sh.n_tok) ? acc[i][j] * sh.scale : -INFINITY; // keys past the end weigh nothing
				mx = fmaxf(mx, x[j]);
			}
			float mnew = mrow[i], shift = mnew;
			if (softmax) {
#pragma unroll
				for (int d = 8; d > 0; d >>= 1)
					mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
				mnew = fmaxf(mrow[i], mx);
				shift = mnew == -INFINITY ? 0.f : mnew; // all keys so far infinitely far (masked): they weigh nothing
			}
			float ps = 0.f;
#pragma unroll
			for (int j = 0; j < 4; j++) {
				const float p = expf(x[j] - shift);
				Pw[i * (2 * NW) * PP + j * 16 + sg] = p;
				ps += p;
			}
#pragma unroll
			for (int d = 8; d > 0; d >>= 1)
				ps += __shfl_xor_sync(0xffffffffu, ps, d);
			if (softmax) {
				const float alpha = expf(mrow[i] - shift); // exp(-inf) = 0 on the first tile
				lrow[i] = lrow[i] * alpha + ps;
#pragma unroll
				for (int e = 0; e < NV; e++)
					o[i][e] *= alpha;
				mrow[i] = mnew;
			} else {
				lrow[i] += ps;
			}
		}
		__syncwarp();

		// ---- output rows += weights x values; this lane owns value columns [sg*NV, sg*NV+NV)
#pragma unroll 2
		for (int s4 = 0; s4 < TS / 4; s4++) {
			float4 p[TI];
#pragma unroll
			for (int i = 0; i < TI; i++)
				p[i] = *reinterpret_cast<const float4 *>(Pw + i * (2 * NW) * PP + s4 * 4);
#pragma unroll
			for (int ss = 0; ss < 4; ss++) {
				float vv[NV];
				const float *vp = Vs + (s4 * 4 + ss) * VW + sg * NV;
				if (NV == 2) {
					const float2 t2 = *reinterpret_cast<const float2 *>(vp);
					vv[0] = t2.x;
					vv[1] = t2.y;
				} else {
#pragma unroll
					for (int e = 0; e < NV; e += 4) {
						const float4 t4 = *reinterpret_cast<const float4 *>(vp + e);
						vv[e] = t4.x;
						vv[(e + 1) % NV] = t4.y;
						vv[(e + 2) % NV] = t4.z;
						vv[(e + 3) % NV] = t4.w;
					}
				}
#pragma unroll
				for (int i = 0; i < TI; i++) {
					const float pi = ss == 0 ? p[i].x : ss == 1 ? p[i].y : ss == 2 ? p[i].z : p[i].w;
#pragma unroll
					for (int e = 0; e < NV; e++)
						o[i][e] = fmaf(pi, vv[e], o[i][e]);
				}
			}
		}
		__syncwarp(); // the weight slice is rewritten by the next tile
		if (lane == 0)
			mbar_arrive(&empty_bar[st]);
	}

#pragma unroll
	for (int i = 0; i < TI; i++) {
		const int t = t0 + i * (2 * NW) + tg;
		if (t >= sh.n_tok)
			continue;
		const float inv = sh.mode == L1ATTN_SV_EXP ? 1.f : 1.f / lrow[i];
		if (lse && sg == 0) // weight of (s, t) = exp(x - lse)
			lse[(size_t(b) * sh.n_tok + t) * sh.n_heads + h] = sh.mode == L1ATTN_SV_EXP ? 0.f : mrow[i] + logf(lrow[i]);
		float *op = vo + v0 + size_t(t) * vrow + sg * NV;
#pragma unroll
		for (int e = 0; e < NV; e++)
			if (FULL || sg * NV + e < sh.v_width)
				op[e] = o[i][e] * inv;
	}
}

// acc += |q row - k row| over one slice of 32 columns: TI query rows (i * 2 NW + tg) x 4 keys (j * 16 + sg), nc 16-byte chunks of it
template <int TI, int NW, bool FULL>
__device__ __forceinline__ void score_slice(const unsigned char *Qslice, const unsigned char *Kslice, int tg, int sg, int nc, float (&acc)[TI][4])
{
	const ulonglong2 *Qb = reinterpret_cast<const ulonglong2 *>(Qslice);
	const ulonglong2 *Kb = reinterpret_cast<const ulonglong2 *>(Kslice);
#pragma unroll 2
	for (int c = 0; c < (FULL ? 8 : nc); c++) {
		ulonglong2 kv[4];
#pragma unroll
		for (int j = 0; j < 4; j++) // row j*16+sg, chunk c ^ (row & 7)
			kv[j] = Kb[(j * 16 + sg) * 8 + (c ^ (sg & 7))];
#pragma unroll
		for (int i = 0; i < TI; i++) {
			const ulonglong2 qv = Qb[(i * (2 * NW) + tg) * 8 + (c ^ (tg & 7))];
#pragma unroll
			for (int j = 0; j < 4; j++) {
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
	}
}

// ------------------------------------------------------------------------------------------------
// Forward with the value product on the tensor cores (fp32, 128-row CTAs, width <= 64, v_width <= 64)
// ------------------------------------------------------------------------------------------------
// The scores, the softmax and who owns what are those of softmax_v_tile_kernel<.., 4, 16, ..>; the value product -- a third of that
// kernel's instructions -- is done by tcgen05.mma.  Weights and values, times 2^24, are written as sums of three bf16 each (exact: 3 x 8
// bits of 24, none of them subnormal), nine products in three fp32 sums per key tile (see mma_pieces); they are read back,
// rescaled and added in fp32 registers, a tile behind the scores.  Warps:
//   0-15   scores and weights; the weights' pieces to shared memory (A, [query row][key]), keys in the order 4 * (s % 16) + s / 16, so
//          that a lane's four weights are neighbours; sums of the tile before: warp = 32 rows x v_width / 4 columns
//   16     issues the MMAs       17, 18  values' pieces to shared memory (B, [column][key])        19  nothing
// [16,1024,16,64], values 64 wide: 2.11 ms, softmax_v_tile_kernel 2.27; error against float64 0.85-1.0 of that kernel's.  Bound: FP32 pipe
// of the scores (two lane-cycles per term) with the shared loads of a 4 x 4 tile beside it.
// Values without pieces (not finite, or 2^36 and more) are added by FMAs to the sums of their tile, from the weights' pieces and the values in
// global memory (one such value in every head: 2.14 ms).
constexpr int TC_NW = 16, TC_ROWS = 128, TC_THREADS = (TC_NW + 4) * 32;
constexpr int TC_REGS = 104, TC_REGS_REST = 64, TC_REGS_LAUNCH = 96; // registers per thread; the launcher asks whether the kernel was built with the last
static_assert(4 * TC_REGS + TC_REGS_REST <= 5 * TC_REGS_LAUNCH, "more than the block was launched with");
constexpr int TC_MAINS = 2;                        // sums of the leading products (see mma_pieces), each 64 columns of tensor memory
constexpr int TC_SUM = 64 * (1 + TC_MAINS), TC_COLUMNS = 256, TC_BWD_COLUMNS = 512;
static_assert(TC_SUM <= TC_COLUMNS && 2 * TC_SUM <= TC_BWD_COLUMNS, "tensor memory");
constexpr int TC_A_PIECE = TC_ROWS * 128;          // 64 bf16 a row
constexpr size_t TC_SMEM = 227 * 1024 - 3072;      // per CTA, less the static part
// Widest rows of q, k.  More do not fit the backward; a forward on the tensor cores before a backward that is not gained nothing ([1,512,37,96], values
// 64 wide: 120 us either way) and cost precision: dp - delta no longer cancels what is left of the adder's one-sided error in vo.
constexpr int TC_WIDTH = 64;

struct TcBars {
	uint64_t own, full[MAX_STAGE], empty[MAX_STAGE], p_full, v_full, done, done2, patched;
	uint32_t tmem;
	uint32_t own_without[TC_ROWS / 32];           // rows of the CTA's own values that hold some without pieces
	__align__(16) uint32_t without[2][2][2];      // [tile & 1][warp - 17]: tokens of the streamed tile that do, by 32
};

// Values that are not finite have no pieces (inf - inf), and very large ones get none, for the range of the sums.  The products are
// done without them, and the tile is marked.
__device__ __forceinline__ bool has_pieces(float x) { return fabsf(x) < PIECE_LIMIT; }
__device__ __forceinline__ float take(float x, bool &all)
{
	const bool ok = has_pieces(x);
	all = all && ok;
	return ok ? x * PIECE_SCALE : 0.f;
}
__device__ __forceinline__ unsigned long long tile_without(const TcBars &bars, int m)
{
	uint32_t a, b, c, d;
	asm volatile("ld.volatile.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(smem_u32(bars.without[m & 1])) : "memory");
	return (unsigned long long)(b | d) << 32 | (a | c);
}
// o[e] += weight x rows[token][e], e < left, for the values of tile m without pieces; they are of the tokens in `which`.  The weights come from their
// pieces, so all sixteen warps wait for one another before any of them writes the next tile's.  False: a wait has run out.
template <int NO> __device__ __forceinline__ bool add_without(float (&o)[NO], unsigned long long which, const unsigned char *pieces, int row, const float *rows,
							      size_t pitch, int m, int n_tok, int left, TcBars &bars, int &patches, int *err)
{
	bool ok = mbar_wait_inline(&bars.p_full, m & 1, err); // (the weights are there: complete already, and seen by this thread)
#pragma unroll 1
	for (; which; which &= which - 1) {
		const int i = __ffsll(which) - 1, place = 4 * (i % 16) + i / 16;
		const unsigned char *a = pieces + row * 128 + (((place >> 3) ^ (row & 7)) << 4) + (place & 7) * 2;
		float p = 0.f;
#pragma unroll
		for (int j = 2; j >= 0; j--)
			p += __uint_as_float(uint32_t(*reinterpret_cast<const unsigned short *>(a + j * TC_A_PIECE)) << 16);
#pragma unroll
		for (int e = 0; e < NO; e++) {
			const float x = e < left && m * TS + i < n_tok ? rows[size_t(m * TS + i) * pitch + e] : 0.f;
			if (!has_pieces(x))
				o[e] = fmaf(p * (1.f / PIECE_SCALE), x, o[e]);
		}
	}
	__syncwarp();
	if ((threadIdx.x & 31) == 0)
		mbar_arrive(&bars.patched);
	ok = ok && mbar_wait_inline(&bars.patched, patches & 1, err);
	patches++;
	return ok;
}

// this lane's four weights of row r (keys 4 sg .. in the order above), as three pieces
__device__ __forceinline__ void store_weights(unsigned char *pieces, int r, int sg, const float (&p)[4])
{
	uint32_t a[3], b[3];
	split_bf16(p[0] * PIECE_SCALE, p[1] * PIECE_SCALE, a);
	split_bf16(p[2] * PIECE_SCALE, p[3] * PIECE_SCALE, b);
	unsigned char *d = pieces + r * 128 + (((sg >> 1) ^ (r & 7)) << 4) + (sg & 1) * 8;
#pragma unroll
	for (int i = 0; i < 3; i++)
		*reinterpret_cast<uint2 *>(d + i * TC_A_PIECE) = make_uint2(a[i], b[i]);
}

// All products of the pieces, STEPS of 16 k.  The tensor core adds to its fp32 sums by truncation, which for values of one sign is an error of one
// sign.  So the leading products go to two sums of their own, a half of the k each (at d + 64, d + 128), the eight others, 2^-6 of them and less,
// to a third (at d, smallest first), and the three are added with rounding.  (All in one sum: vo and dv of positive values 4.5e-8 too small.)
template <int STEPS> __device__ __forceinline__ void mma_pieces(uint32_t d, uint64_t a, uint32_t a_piece, uint64_t b, uint32_t b_piece, uint32_t b_step, uint32_t idesc)
{
	static_assert(STEPS % TC_MAINS == 0, "every sum gets products");
	bool more = false;
#pragma unroll 1
	for (int i = 8; i > 0; i--) { // i = 3 * piece of a + piece of b: (2,2), (2,1), ... (0,1)
		const uint64_t ai = a + i / 3 * (a_piece >> 4), bi = b + i % 3 * (b_piece >> 4);
#pragma unroll
		for (int k = 0; k < STEPS; k++) {
			tc_mma_bf16_ss(d, ai + k * 2, bi + k * (b_step >> 4), idesc, more);
			more = true;
		}
	}
#pragma unroll
	for (int k = 0; k < STEPS; k++)
		tc_mma_bf16_ss(d + 64 * (1 + k * TC_MAINS / STEPS), a + k * 2, b + k * (b_step >> 4), idesc, k * TC_MAINS % STEPS != 0);
}
// this lane's row of them: d + 64, d + 128 and d
template <int N> __device__ __forceinline__ void load_sums(uint32_t d, float (&r)[N])
{
	float x[N], y[N];
	tmem_load3(d + 64, d + 128, d, r, x, y);
#pragma unroll
	for (int e = 0; e < N; e++)
		r[e] = r[e] + x[e] + y[e];
}

template <int NV, bool TMA, bool FULL>
__global__ void __launch_bounds__(TC_THREADS, 1)
softmax_v_tc_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
		    const __grid_constant__ CUtensorMap vmap, const float *__restrict__ q, const float *__restrict__ k,
		    const float *__restrict__ v, float *__restrict__ vo, float *__restrict__ lse, SvShape sh, int *err)
{
	constexpr int NW = TC_NW, TI = 4, TT = TC_ROWS, VW = 16 * NV, V_BYTES = TS * VW * 4, NO = VW / 4;
	constexpr int V_PIECE = VW * 128;
	extern __shared__ __align__(1024) unsigned char smem_raw[];
	unsigned char *base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
	__shared__ __align__(8) TcBars bars;
	__shared__ float row_corr[2][TT], row_inv[TT];
	const int q_bytes = sh.nwb * TT * 128, k_bytes = sh.nwb * TS * 128, stage_bytes = k_bytes + V_BYTES;
	unsigned char *Pp = base, *Vp = Pp + 3 * TC_A_PIECE, *Qs = Vp + 3 * V_PIECE, *stages = Qs + q_bytes;

	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	unsigned r = blockIdx.x;
	const int t0 = int(r % unsigned(sh.ntt)) * TT;
	r /= unsigned(sh.ntt);
	const int h = int(r % unsigned(sh.n_heads));
	const int b = int(r / unsigned(sh.n_heads));
	const int ns = (sh.n_tok + TS - 1) / TS;

	if (warp == 16)
		tmem_alloc(&bars.tmem, TC_COLUMNS);
	if (tid == 0) {
		mbar_init(&bars.own, TMA ? 1 : NW * 32);
		for (int s = 0; s < MAX_STAGE; s++) {
			mbar_init(&bars.full[s], TMA ? 1 : NW * 32);
			mbar_init(&bars.empty[s], NW + 2);
		}
		mbar_init(&bars.p_full, NW);
		mbar_init(&bars.v_full, 2);
		mbar_init(&bars.done, 1);
		mbar_init(&bars.patched, NW);
		mbar_fence_init();
	}
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = bars.tmem;
	const size_t krow = size_t(sh.n_heads) * sh.width, vrow = size_t(sh.n_heads) * sh.v_width;
	const size_t qk0 = size_t(b) * sh.n_tok * krow + size_t(h) * sh.width, v0 = size_t(b) * sh.n_tok * vrow + size_t(h) * sh.v_width;

	if (warp < NW) {
		asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TC_REGS));
		auto load_tile = [&](int m) {
			const int st = m % sh.nstage;
			unsigned char *dst = stages + size_t(st) * stage_bytes;
			if (!TMA) {
				copy_rows<NW, true>(dst, k + qk0, krow, m * TS, TS, sh.nwb, sh.width, sh.n_tok);
				copy_rows<NW, false>(dst + k_bytes, v + v0, vrow, m * TS, TS, VW / 32, sh.v_width, sh.n_tok);
				copy_arrive(&bars.full[st]);
				return;
			}
			mbar_expect_tx(&bars.full[st], uint32_t(stage_bytes));
			for (int wb = 0; wb < sh.nwb; wb++)
				tma_load_4d(dst + wb * TS * 128, &kmap, &bars.full[st], wb * 32, h, m * TS, b);
			tma_load_4d(dst + k_bytes, &vmap, &bars.full[st], 0, h, m * TS, b);
		};
		if (!TMA || tid == 0) {
			if (TMA) {
				mbar_expect_tx(&bars.own, uint32_t(q_bytes));
				for (int wb = 0; wb < sh.nwb; wb++)
					tma_load_4d(Qs + wb * TT * 128, &qmap, &bars.own, wb * 32, h, t0, b);
			} else {
				copy_rows<NW, true>(Qs, q + qk0, krow, t0, TT, sh.nwb, sh.width, sh.n_tok);
				copy_arrive(&bars.own);
			}
			for (int m = 0; m < sh.nstage - 1 && m < ns; m++)
				load_tile(m);
		}

		const int sg = lane & 15, tg = warp * 2 + (lane >> 4);
		const int orow = (warp & 3) * 32 + lane, ocol = (warp >> 2) * NO; // this thread's part of the output
		const uint32_t d_at = tmem + (uint32_t((warp & 3) * 32) << 16) + ocol;
		const bool softmax = sh.mode == L1ATTN_SV_SOFTMAX;
		float o[NO], mrow[TI], lrow[TI];
#pragma unroll
		for (int i = 0; i < TI; i++) {
			mrow[i] = softmax ? -INFINITY : 0.f;
			lrow[i] = sh.mode == L1ATTN_SV_SOFTMAX_PLUS_ONE ? 1.f : 0.f; // the extra all-zero row weighs exp(0)
		}
#pragma unroll
		for (int e = 0; e < NO; e++)
			o[e] = 0.f;
		bool dead = !mbar_wait_inline(&bars.own, 0, err);
		int patches = 0;
		// the sums of tile m, once its MMAs are done, onto the output, which goes to that tile's shift first
		auto collect = [&](int m) {
			if (!dead && !(mbar_wait_inline(&bars.p_full, m & 1, err) && mbar_wait_inline(&bars.done, m & 1, err)))
				dead = true;
			tc_fence_after();
			float d[NO];
			load_sums(d_at, d);
			const float c = row_corr[m & 1][orow];
#pragma unroll
			for (int e = 0; e < NO; e++)
				o[e] = fmaf(o[e], c, d[e] * PIECE_UNSCALE);
			const unsigned long long which = tile_without(bars, m);
			if (__all_sync(0xffffffffu, which != 0 && !dead)) // (a warp as one, also after a timeout)
				dead = !add_without(o, which, Pp, orow, v + v0 + ocol, vrow, m, sh.n_tok, sh.v_width - ocol, bars, patches, err);
		};

		for (int m = 0; m < ns; m++) {
			if ((!TMA || (warp == m % NW && lane == 0)) && m + sh.nstage - 1 < ns && !dead) {
				const int mm = m + sh.nstage - 1;
				if (mbar_wait_inline(&bars.empty[mm % sh.nstage], ((unsigned(mm) / unsigned(sh.nstage)) & 1u) ^ 1u, err))
					load_tile(mm);
				else
					dead = true;
			}
			__syncwarp();
			const int st = m % sh.nstage;
			if (!dead && !mbar_wait_inline(&bars.full[st], (unsigned(m) / unsigned(sh.nstage)) & 1u, err))
				dead = true; // keep walking without waiting; the error word reports the failure
			const unsigned char *Ks = stages + size_t(st) * stage_bytes;

			float acc[TI][4];
#pragma unroll
			for (int i = 0; i < TI; i++)
#pragma unroll
				for (int j = 0; j < 4; j++)
					acc[i][j] = 0.f;
			for (int wb = 0; wb < sh.nwb; wb++) {
				const int nc = FULL ? 8 : min(8, ((sh.width - wb * 32 + 7) >> 3) * 2);
				score_slice<TI, NW, FULL>(Qs + wb * TT * 128, Ks + wb * TS * 128, tg, sg, nc, acc);
			}
			__syncwarp();
			if (lane == 0)
				mbar_arrive(&bars.empty[st]);

			float corr[TI];
#pragma unroll
			for (int i = 0; i < TI; i++) {
				float mx = -INFINITY;
#pragma unroll
				for (int j = 0; j < 4; j++) {
					acc[i][j] = (m * TS + j * 16 + sg < sh.n_tok) ? acc[i][j] * sh.scale : -INFINITY; // keys past the end weigh nothing
					mx = fmaxf(mx, acc[i][j]);
				}
				float shift = mrow[i];
				corr[i] = 1.f;
				if (softmax) {
#pragma unroll
					for (int d = 8; d > 0; d >>= 1)
						mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
					const float mnew = fmaxf(mrow[i], mx);
					shift = mnew == -INFINITY ? 0.f : mnew; // all keys so far infinitely far (masked): they weigh nothing
					corr[i] = expf(mrow[i] - shift);        // exp(-inf) = 0 on the first tile
					mrow[i] = mnew;
				}
				float ps = 0.f;
#pragma unroll
				for (int j = 0; j < 4; j++) {
					acc[i][j] = expf(acc[i][j] - shift);
					ps += acc[i][j];
				}
#pragma unroll
				for (int d = 8; d > 0; d >>= 1)
					ps += __shfl_xor_sync(0xffffffffu, ps, d);
				lrow[i] = lrow[i] * corr[i] + ps;
			}
			if (m > 0)
				collect(m - 1); // (and the pieces of tile m - 1 are read)
#pragma unroll
			for (int i = 0; i < TI; i++) {
				store_weights(Pp, i * (2 * NW) + tg, sg, acc[i]);
				if (sg == 0)
					row_corr[m & 1][i * (2 * NW) + tg] = corr[i];
			}
			fence_proxy_async_smem();
			tc_fence_before();
			__syncwarp();
			if (lane == 0)
				mbar_arrive(&bars.p_full);
		}
		collect(ns - 1);
#pragma unroll
		for (int i = 0; i < TI; i++) {
			const int row = i * (2 * NW) + tg, t = t0 + row;
			if (sg == 0) {
				row_inv[row] = sh.mode == L1ATTN_SV_EXP ? 1.f : 1.f / lrow[i];
				if (lse && t < sh.n_tok) // weight of (s, t) = exp(x - lse)
					lse[(size_t(b) * sh.n_tok + t) * sh.n_heads + h] = sh.mode == L1ATTN_SV_EXP ? 0.f : mrow[i] + logf(lrow[i]);
			}
		}
		named_barrier(1, NW * 32);
		if (t0 + orow < sh.n_tok) {
			float *op = vo + v0 + size_t(t0 + orow) * vrow + ocol;
			const float inv = row_inv[orow];
#pragma unroll
			for (int e = 0; e < NO; e++)
				if (FULL || ocol + e < sh.v_width)
					op[e] = o[e] * inv;
		}
	} else {
		asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TC_REGS_REST));
		if (warp == 16 && lane == 0) {
			const uint64_t a = tc_desc(smem_u32(Pp)), bd = tc_desc(smem_u32(Vp));
			bool dead = false;
			int m = 0;
			for (; m < ns && !dead; m++) {
				dead = !(mbar_wait_inline(&bars.v_full, m & 1, err) && mbar_wait_inline(&bars.p_full, m & 1, err));
				tc_fence_after();
				if (!dead)
					mma_pieces<4>(tmem, a, TC_A_PIECE, bd, V_PIECE, 32, tc_idesc_bf16(VW, false));
				tc_commit(&bars.done);
			}
			mbar_wait_inline(&bars.done, (m - 1) & 1, err); // no product is in flight when the tensor memory goes, also after a timeout
		}
		if (warp == 17 || warp == 18) { // a column per thread (VW 32: half of the threads)
			const int c = (warp - 17) * 32 + lane;
			bool dead = false;
			for (int m = 0; m < ns; m++) {
				const int st = m % sh.nstage;
				if (!dead && !mbar_wait_inline(&bars.full[st], (unsigned(m) / unsigned(sh.nstage)) & 1u, err))
					dead = true;
				if (m > 0 && !dead && !mbar_wait_inline(&bars.done, (m - 1) & 1, err))
					dead = true;
				const float *Vs = reinterpret_cast<const float *>(stages + size_t(st) * stage_bytes + k_bytes);
				bool all = true;
				if (c < VW) {
#pragma unroll 2
					for (int g = 0; g < 8; g++) { // keys at places 8 g .. 8 g + 7
						uint32_t o[3][4];
#pragma unroll
						for (int e = 0; e < 4; e++) {
							const int s = (e & 1) * 32 + 2 * g + (e >> 1); // places 8 g + 2 e, + 1: keys s, s + 16
							uint32_t pc[3];
							split_bf16_short(take(Vs[s * VW + c], all), take(Vs[(s + 16) * VW + c], all), pc);
#pragma unroll
							for (int i = 0; i < 3; i++)
								o[i][e] = pc[i];
						}
#pragma unroll
						for (int i = 0; i < 3; i++)
							*reinterpret_cast<uint4 *>(Vp + i * V_PIECE + c * 128 + ((g ^ (c & 7)) << 4)) = make_uint4(o[i][0], o[i][1], o[i][2], o[i][3]);
					}
				}
				uint32_t which[2] = {0, 0};
				if (!__all_sync(0xffffffffu, all))
					for (int s = 0; s < TS; s++)
						which[s >> 5] |= uint32_t(__any_sync(0xffffffffu, c < VW && !has_pieces(Vs[s * VW + c]))) << (s & 31);
				fence_proxy_async_smem();
				__syncwarp();
				if (lane == 0) {
					bars.without[m & 1][warp - 17][0] = which[0];
					bars.without[m & 1][warp - 17][1] = which[1];
					mbar_arrive(&bars.v_full);
					mbar_arrive(&bars.empty[st]);
				}
			}
		}
		__syncwarp();
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 16)
		tmem_free(tmem, TC_COLUMNS);
}

size_t sv_tc_smem(int nwb, int nv, int nstage)
{
	return size_t(3) * TC_A_PIECE + size_t(3) * nv * 16 * 128 + size_t(nwb) * TC_ROWS * 128 + size_t(nstage) * (size_t(nwb) * TS * 128 + size_t(TS) * nv * 64) + 1024;
}

// (query rows per half-warp, warps, ring stages) of the tiled kernels.  4 x 16 and 8 x 8 make a 128-row CTA, 4 x 8 a 64-row
// one.  Sixteen warps of 128 registers measured 7 % faster than eight of 168 (four warps per scheduler hide the
// shared-memory and arithmetic latencies); with 128 value columns the thread state does not fit 128 registers.  A 64-row CTA is taken
// where the rows do not fit shared memory otherwise, or where its finer grid fills the SMs better (few rows in all, or few left over for the
// last wave): its waves count `short_cta` each.  Measured, a wave of 64-row CTAs (half of two) against one of 128-row CTAs, us at [1,512,37,w]:
// forward, width 64 50 / 86, 48 (values 40) 45 / 71, 33 (21) 39 / 70, 96 (64) 61 / 106, 32 (32) 28 / 57; backward on the tensor cores 64 / 94,
// 53 / 79, 51 / 76, -, 38 / 61, without (width 96) 75 / 140.  From 36 to 450 CTAs of 128 rows, ten widths, the rule is within 7 % of the better form in
// the forward, 4 % in the backward.
struct TilePlan {
	int ti, nw, nstage; // nstage 0: no form fits
	size_t smem;
	bool tc; // products on the tensor cores
};
double sv_short_cta(int width, int v_width) { return width <= 32 && v_width <= 32 ? 0.48 : 0.6; }
double sv_bwd_short_cta(bool tc) { return tc ? 0.67 : 0.54; }
template <typename F, typename G> TilePlan plan_tile(int nv, long long groups, int n_tok, double short_cta, F smem_of, G tc_smem_of)
{
	const size_t limit = 227 * 1024 - 256; // per-CTA maximum minus the static barriers
	const bool nw16 = nv <= 4;
	const int cand[2][2] = {{nw16 ? 4 : 8, nw16 ? TC_NW : 8}, {4, 8}};
	TilePlan best{0, 0, 0, 0, false};
	double best_cost = 0;
	for (const auto &c : cand)
		for (int ns : {3, 2}) {
			const int tt = 2 * c[0] * c[1];
			const size_t smem = smem_of(tt, ns);
			if (smem > limit)
				continue;
			const long long ctas = groups * ((n_tok + tt - 1) / tt);
			const double cost = double((ctas + 147) / 148) * (tt == 64 ? short_cta : 1.0);
			if (!best.nstage || cost < best_cost) {
				best = {c[0], c[1], ns, smem, false};
				best_cost = cost;
			}
			break; // the deeper ring that fits
		}
	if (best.nw == TC_NW)
		for (int ns : {2, 3}) // (the deeper ring that fits)
			if (tc_smem_of(ns) <= TC_SMEM) {
				best.nstage = ns;
				best.smem = tc_smem_of(ns);
				best.tc = true;
			}
	return best;
}

template <int NV, int TI, int NW, bool TMA, bool FULL>
int launch_tile(const float *q, const float *k, const float *v, float *vo, float *lse, int bs, int n_tok, int n_heads,
		int width, int v_width, int mode, const TilePlan &plan, cudaStream_t st)
{
	constexpr int TT = 2 * NW * TI, VW = 16 * NV, NTH = NW * 32;
	const uint64_t dims[4] = {uint64_t(width), uint64_t(n_heads), uint64_t(n_tok), uint64_t(bs)};
	const uint64_t str[3] = {uint64_t(width) * 4, uint64_t(n_heads) * width * 4, uint64_t(n_tok) * n_heads * width * 4};
	const uint64_t vdims[4] = {uint64_t(v_width), uint64_t(n_heads), uint64_t(n_tok), uint64_t(bs)};
	const uint64_t vstr[3] = {uint64_t(v_width) * 4, uint64_t(n_heads) * v_width * 4, uint64_t(n_tok) * n_heads * v_width * 4};
	const uint32_t qbox[4] = {32, 1, TT, 1}, kbox[4] = {32, 1, TS, 1}, vbox[4] = {VW, 1, TS, 1};
	CUtensorMap qmap{}, kmap{}, vmap{};
	if (TMA && (!encode_tmap_4d(&qmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, q, dims, str, qbox, CU_TENSOR_MAP_SWIZZLE_128B) ||
	    !encode_tmap_4d(&kmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, k, dims, str, kbox, CU_TENSOR_MAP_SWIZZLE_128B) ||
	    !encode_tmap_4d(&vmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, v, vdims, vstr, vbox, CU_TENSOR_MAP_SWIZZLE_NONE)))
		return 1;
	int *err = device_error_word();
	if (!err)
		return 1;
	SvShape sh;
	sh.n_tok = n_tok;
	sh.n_heads = n_heads;
	sh.width = width;
	sh.v_width = v_width;
	sh.nwb = (width + 31) / 32;
	sh.nstage = plan.nstage;
	sh.ntt = (n_tok + TT - 1) / TT;
	sh.mode = mode;
	sh.scale = float(-1.0 / sqrt(double(width)));
	const long long grid = (long long)bs * n_heads * sh.ntt;
	if (grid > 0x7fffffffLL)
		return L1ATTN_ERR_SHAPE;
	if constexpr (NW == TC_NW)
		if (plan.tc) {
			auto kern = softmax_v_tc_kernel<NV, TMA, FULL>;
			L1B_SHARED_MEMORY(kern, int(plan.smem));
			L1B_REGISTERS(kern, TC_REGS_LAUNCH);
			kern<<<unsigned(grid), TC_THREADS, plan.smem, st>>>(qmap, kmap, vmap, q, k, v, vo, lse, sh, err);
			L1B_LAUNCH_CHECK();
			return L1ATTN_OK;
		}
	auto kern = softmax_v_tile_kernel<NV, TI, NW, TMA, FULL>;
	L1B_SHARED_MEMORY(kern, int(plan.smem));
	kern<<<unsigned(grid), NTH, plan.smem, st>>>(qmap, kmap, vmap, q, k, v, vo, lse, sh, err);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

// shared memory of one CTA: query tile + ring + weight tile + alignment slack
size_t sv_smem(int nwb, int nv, int tt_rows, int nstage)
{
	const size_t tt = size_t(tt_rows);
	return size_t(nwb) * tt * 128 + size_t(nstage) * (size_t(nwb) * TS * 128 + size_t(TS) * nv * 64) + tt * PP * 4 + 1024;
}

int sv_nv(int v_width) { return v_width <= 32 ? 2 : v_width <= 64 ? 4 : 8; } // value columns per lane
TilePlan sv_plan(int bs, int n_tok, int n_heads, int width, int v_width)
{
	if (width < 1 || width > 128 || v_width < 1 || v_width > 128)
		return {0, 0, 0, 0, false};
	const int nwb = (width + 31) / 32, nv = sv_nv(v_width);
	return plan_tile(nv, (long long)bs * n_heads, n_tok, sv_short_cta(width, v_width), [&](int tt, int ns) { return sv_smem(nwb, nv, tt, ns); },
			 [&](int ns) { return width <= TC_WIDTH ? sv_tc_smem(nwb, nv, ns) : TC_SMEM + 1; });
}

// Returns L1ATTN_OK, a negative error, or 1 when the shape is outside this kernel's set.
int softmax_v_tile(const float *q, const float *k, const float *v, float *vo, float *lse, int bs, int n_tok, int n_heads,
		   int width, int v_width, int mode, cudaStream_t st)
{
	const TilePlan p = sv_plan(bs, n_tok, n_heads, width, v_width);
	if (!p.nstage)
		return 1;
	const bool tma = width % 4 == 0 && v_width % 4 == 0 && aligned(q, 16) && aligned(k, 16) && aligned(v, 16);
	const int nv = sv_nv(v_width);
	const bool full = width % 32 == 0 && v_width == 16 * nv; // no padded columns
#define L1B_SV_RUN(NV_, TI_, NW_, TMA_, FULL_) \
	launch_tile<NV_, TI_, NW_, TMA_, FULL_>(q, k, v, vo, lse, bs, n_tok, n_heads, width, v_width, mode, p, st)
#define L1B_SV(NV_, TI_, NW_)                                                                                                  \
	if (nv == NV_ && p.ti == TI_ && p.nw == NW_) {                                                                         \
		const int rc = !tma ? 1 : full ? L1B_SV_RUN(NV_, TI_, NW_, true, true) : L1B_SV_RUN(NV_, TI_, NW_, true, false); \
		return rc <= 0 ? rc : L1B_SV_RUN(NV_, TI_, NW_, false, false);                                                  \
	}
	L1B_SV(2, 4, 8) L1B_SV(4, 4, 8) L1B_SV(8, 4, 8) L1B_SV(8, 8, 8) L1B_SV(2, 4, 16) L1B_SV(4, 4, 16)
#undef L1B_SV
#undef L1B_SV_RUN
	return 1;
}

// ------------------------------------------------------------------------------------------------
// backward, step 1: score gradients dx and value gradients dv
// ------------------------------------------------------------------------------------------------
// With lse[b][t][h] from the forward (weight of (s, t) = exp(x - lse)) and
// delta[b][t][h] = <dvo[b][t][h][:], vo[b][t][h][:]> (zeros for the exp form):
//   p  = exp(x[b][s][t][h] - lse[b][t][h])
//   dx[b][s][t][h] = p * (<v[b][s][h][:], dvo[b][t][h][:]> - delta[b][t][h])
//   dv[b][s][h][:] = sum_t p * dvo[b][t][h][:]
// dx has the layout of the dense operator's d_attn, so l1attn_dense_bwd(dx, q, k) finishes the job
// (d_q, d_k).  Callers bound memory by running a few batch items at a time.

template <typename T>
__global__ void __launch_bounds__(GEN_NT)
softmax_v_bwd_kernel(const T *__restrict__ q, const T *__restrict__ k, const T *__restrict__ v, const T *__restrict__ dvo,
		     const T *__restrict__ lse, const T *__restrict__ delta, T *__restrict__ dx, T *__restrict__ dv,
		     int n_tok, int n_heads, int width, int v_width, T scale)
{
	extern __shared__ __align__(16) unsigned char gsm[];
	T *pw = reinterpret_cast<T *>(gsm); // [n_tok] weights of this source row
	T *krow = pw + n_tok;               // [width]
	T *vrow = krow + width;             // [v_width]
	unsigned r = blockIdx.x;
	const int h = int(r % unsigned(n_heads));
	r /= unsigned(n_heads);
	const int s = int(r % unsigned(n_tok));
	const int b = int(r / unsigned(n_tok));
	const size_t row = size_t(n_heads) * width, vr = size_t(n_heads) * v_width;
	const T *kp = k + (size_t(b) * n_tok + s) * row + size_t(h) * width;
	const T *vp = v + (size_t(b) * n_tok + s) * vr + size_t(h) * v_width;
	for (int w = threadIdx.x; w < width; w += GEN_NT)
		krow[w] = kp[w];
	for (int c = threadIdx.x; c < v_width; c += GEN_NT)
		vrow[c] = vp[c];
	__syncthreads();
	const T *qb = q + size_t(b) * n_tok * row + size_t(h) * width;
	const T *gb = dvo + size_t(b) * n_tok * vr + size_t(h) * v_width;
	for (int t = threadIdx.x; t < n_tok; t += GEN_NT) {
		const T *qp = qb + size_t(t) * row, *gp = gb + size_t(t) * vr;
		T acc = T(0), dp = T(0);
		for (int w = 0; w < width; w++)
			acc += absdiff(qp[w], krow[w]);
		for (int c = 0; c < v_width; c++)
			dp += vrow[c] * gp[c];
		const size_t st = (size_t(b) * n_tok + t) * n_heads + h;
		const T p = exp_t(acc * scale - lse[st]);
		pw[t] = p;
		dx[((size_t(b) * n_tok + s) * n_tok + t) * n_heads + h] = p * (dp - delta[st]);
	}
	__syncthreads();
	T *op = dv + (size_t(b) * n_tok + s) * vr + size_t(h) * v_width;
	for (int c = threadIdx.x; c < v_width; c += GEN_NT) {
		T o = T(0);
		for (int t = 0; t < n_tok; t++)
			o += pw[t] * gb[size_t(t) * vr + c];
		op[c] = o;
	}
}

template <typename T>
int launch_bwd_generic(const T *q, const T *k, const T *v, const T *dvo, const T *lse, const T *delta, T *dx, T *dv, int bs,
		       int n_tok, int n_heads, int width, int v_width, cudaStream_t st)
{
	const long long grid = (long long)bs * n_tok * n_heads;
	const size_t smem = (size_t(n_tok) + width + v_width) * sizeof(T);
	if (grid > 0x7fffffffLL || smem > 200 * 1024)
		return L1ATTN_ERR_SHAPE;
	auto kern = softmax_v_bwd_kernel<T>;
	L1B_SHARED_MEMORY(kern, int(smem));
	kern<<<unsigned(grid), GEN_NT, smem, st>>>(q, k, v, dvo, lse, delta, dx, dv, n_tok, n_heads, width, v_width,
						    T(-1.0 / sqrt(double(width))));
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

// Tiled variant: the forward kernel with the roles swapped.  The CTA owns TT source rows (their key and
// value rows stay in shared memory) and streams the query and dvo rows in tiles of 64; a half-warp
// owns TI source rows, a lane 4 query columns for the scores and the <v, dvo> products, and NV value
// columns for dv.  Every operand row is kept as 128-byte slices with the 128-byte swizzle.
template <int NV, int TI, int NW, bool TMA, bool FULL>
__global__ void __launch_bounds__(NW * 32, 1)
softmax_v_bwd_tile_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
			 const __grid_constant__ CUtensorMap vmap, const __grid_constant__ CUtensorMap gmap,
			 const float *__restrict__ q, const float *__restrict__ k, const float *__restrict__ v,
			 const float *__restrict__ dvo, const float *__restrict__ lse, const float *__restrict__ delta,
			 float *__restrict__ dx, float *__restrict__ dv, SvShape sh, int *err)
{
	constexpr int TT = 2 * NW * TI; // source rows of the CTA
	constexpr int NTH = NW * 32;
	constexpr int VW = 16 * NV;
	constexpr int NVB = VW / 32; // 128-byte slices per value row
	extern __shared__ __align__(1024) unsigned char smem_raw[];
	unsigned char *base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
	__shared__ __align__(8) uint64_t own_bar, full_bar[MAX_STAGE], empty_bar[MAX_STAGE];
	const int k_bytes = sh.nwb * TT * 128, v_bytes = NVB * TT * 128;
	const int q_bytes = sh.nwb * TS * 128, g_bytes = NVB * TS * 128, stage_bytes = q_bytes + g_bytes;
	unsigned char *Ks = base, *Vs = base + k_bytes;
	unsigned char *stages = Vs + v_bytes;
	float *Ps = reinterpret_cast<float *>(stages + size_t(sh.nstage) * stage_bytes);

	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	unsigned r = blockIdx.x;
	const int s0 = int(r % unsigned(sh.ntt)) * TT;
	r /= unsigned(sh.ntt);
	const int h = int(r % unsigned(sh.n_heads));
	const int b = int(r / unsigned(sh.n_heads));
	const int nt = (sh.n_tok + TS - 1) / TS;

	if (tid == 0) {
		mbar_init(&own_bar, TMA ? 1 : NTH);
		for (int s = 0; s < MAX_STAGE; s++) {
			mbar_init(&full_bar[s], TMA ? 1 : NTH);
			mbar_init(&empty_bar[s], NTH / 32);
		}
		mbar_fence_init();
	}
	__syncthreads();

	const size_t krow = size_t(sh.n_heads) * sh.width, vrow = size_t(sh.n_heads) * sh.v_width;
	const size_t qk0 = size_t(b) * sh.n_tok * krow + size_t(h) * sh.width, v0 = size_t(b) * sh.n_tok * vrow + size_t(h) * sh.v_width;
	auto load_tile = [&](int m) {
		const int st = m % sh.nstage;
		unsigned char *dst = stages + size_t(st) * stage_bytes;
		if (!TMA) {
			copy_rows<NW, true>(dst, q + qk0, krow, m * TS, TS, sh.nwb, sh.width, sh.n_tok);
			copy_rows<NW, true>(dst + q_bytes, dvo + v0, vrow, m * TS, TS, NVB, sh.v_width, sh.n_tok);
			copy_arrive(&full_bar[st]);
			return;
		}
		mbar_expect_tx(&full_bar[st], uint32_t(stage_bytes));
		for (int wb = 0; wb < sh.nwb; wb++)
			tma_load_4d(dst + wb * TS * 128, &qmap, &full_bar[st], wb * 32, h, m * TS, b);
		for (int vb = 0; vb < NVB; vb++)
			tma_load_4d(dst + q_bytes + vb * TS * 128, &gmap, &full_bar[st], vb * 32, h, m * TS, b);
	};
	if (!TMA || tid == 0) {
		if (TMA) {
			mbar_expect_tx(&own_bar, uint32_t(k_bytes + v_bytes));
			for (int wb = 0; wb < sh.nwb; wb++)
				tma_load_4d(Ks + wb * TT * 128, &kmap, &own_bar, wb * 32, h, s0, b);
			for (int vb = 0; vb < NVB; vb++)
				tma_load_4d(Vs + vb * TT * 128, &vmap, &own_bar, vb * 32, h, s0, b);
		} else {
			copy_rows<NW, true>(Ks, k + qk0, krow, s0, TT, sh.nwb, sh.width, sh.n_tok);
			copy_rows<NW, true>(Vs, v + v0, vrow, s0, TT, NVB, sh.v_width, sh.n_tok);
			copy_arrive(&own_bar);
		}
		for (int m = 0; m < sh.nstage - 1 && m < nt; m++)
			load_tile(m);
	}

	const int sg = lane & 15, tg = warp * 2 + (lane >> 4);
	float o[TI][NV];
#pragma unroll
	for (int i = 0; i < TI; i++)
#pragma unroll
		for (int e = 0; e < NV; e++)
			o[i][e] = 0.f;
	bool dead = false;
	if (!mbar_wait(&own_bar, 0, err))
		dead = true;
	float *Pw = Ps + tg * PP;
	const size_t hstride = size_t(sh.n_heads);
	const size_t dx_t = sh.dx_pitch > 0 ? 1 : hstride, dx_s = sh.dx_pitch > 0 ? size_t(sh.dx_pitch) : hstride * sh.n_tok;
	const size_t dx0 = sh.dx_pitch > 0 ? (size_t(b) * sh.n_heads + h) * sh.n_tok * sh.dx_pitch : size_t(b) * sh.n_tok * sh.n_tok * hstride + h;

	for (int m = 0; m < nt; m++) {
		if ((!TMA || (warp == m % NW && lane == 0)) && m + sh.nstage - 1 < nt && !dead) {
			const int mm = m + sh.nstage - 1;
			if (mbar_wait(&empty_bar[mm % sh.nstage], ((unsigned(mm) / unsigned(sh.nstage)) & 1u) ^ 1u, err))
				load_tile(mm);
			else
				dead = true;
		}
		__syncwarp();
		// per-query statistics of this lane's 4 columns (global loads issued before the wait)
		float lj[4], dj[4];
#pragma unroll
		for (int j = 0; j < 4; j++) {
			const int t = m * TS + j * 16 + sg;
			const bool ok = t < sh.n_tok;
			const size_t st = (size_t(b) * sh.n_tok + (ok ? t : 0)) * hstride + h;
			lj[j] = ok ? lse[st] : INFINITY; // exp(x - inf) = 0: query rows past the end weigh nothing
			dj[j] = ok ? delta[st] : 0.f;
		}
		const int st = m % sh.nstage;
		if (!dead && !mbar_wait(&full_bar[st], (unsigned(m) / unsigned(sh.nstage)) & 1u, err))
			dead = true;
		const unsigned char *Qs = stages + size_t(st) * stage_bytes;
		const unsigned char *Gs = Qs + q_bytes;

		float acc[TI][4], dp[TI][4];
#pragma unroll
		for (int i = 0; i < TI; i++)
#pragma unroll
			for (int j = 0; j < 4; j++) {
				acc[i][j] = 0.f;
				dp[i][j] = 0.f;
			}
		for (int wb = 0; wb < sh.nwb; wb++) {
			const ulonglong2 *Kb = reinterpret_cast<const ulonglong2 *>(Ks + wb * TT * 128);
			const ulonglong2 *Qb = reinterpret_cast<const ulonglong2 *>(Qs + wb * TS * 128);
			const int nc = FULL ? 8 : min(8, ((sh.width - wb * 32 + 7) >> 3) * 2);
#pragma unroll 2
			for (int c = 0; c < nc; c++) {
				ulonglong2 qv[4];
#pragma unroll
				for (int j = 0; j < 4; j++)
					qv[j] = Qb[(j * 16 + sg) * 8 + (c ^ (sg & 7))];
#pragma unroll
				for (int i = 0; i < TI; i++) {
					const ulonglong2 kv = Kb[(i * (2 * NW) + tg) * 8 + (c ^ (tg & 7))];
#pragma unroll
					for (int j = 0; j < 4; j++) {
						unsigned long long d0, d1;
						float x0, x1, x2, x3;
						asm("sub.f32x2 %0, %1, %2;" : "=l"(d0) : "l"(kv.x), "l"(qv[j].x));
						asm("sub.f32x2 %0, %1, %2;" : "=l"(d1) : "l"(kv.y), "l"(qv[j].y));
						asm("mov.b64 {%0, %1}, %2;" : "=f"(x0), "=f"(x1) : "l"(d0));
						asm("mov.b64 {%0, %1}, %2;" : "=f"(x2), "=f"(x3) : "l"(d1));
						acc[i][j] += fabsf(x0);
						acc[i][j] += fabsf(x1);
						acc[i][j] += fabsf(x2);
						acc[i][j] += fabsf(x3);
					}
				}
			}
		}
#pragma unroll
		for (int vb = 0; vb < NVB; vb++) {
			const float4 *Vb = reinterpret_cast<const float4 *>(Vs + vb * TT * 128);
			const float4 *Gb = reinterpret_cast<const float4 *>(Gs + vb * TS * 128);
			const int nc = FULL ? 8 : min(8, ((sh.v_width - vb * 32 + 7) >> 3) * 2);
#pragma unroll 2
			for (int c = 0; c < nc; c++) {
				float4 gv[4];
#pragma unroll
				for (int j = 0; j < 4; j++)
					gv[j] = Gb[(j * 16 + sg) * 8 + (c ^ (sg & 7))];
#pragma unroll
				for (int i = 0; i < TI; i++) {
					const float4 vv = Vb[(i * (2 * NW) + tg) * 8 + (c ^ (tg & 7))];
#pragma unroll
					for (int j = 0; j < 4; j++) {
						dp[i][j] = fmaf(vv.x, gv[j].x, dp[i][j]);
						dp[i][j] = fmaf(vv.y, gv[j].y, dp[i][j]);
						dp[i][j] = fmaf(vv.z, gv[j].z, dp[i][j]);
						dp[i][j] = fmaf(vv.w, gv[j].w, dp[i][j]);
					}
				}
			}
		}

		// weights, score gradients (stored), weights parked for the dv product
#pragma unroll
		for (int i = 0; i < TI; i++) {
			const int s = s0 + i * (2 * NW) + tg;
			float *dxr = dx + dx0 + size_t(s < sh.n_tok ? s : 0) * dx_s;
#pragma unroll
			for (int j = 0; j < 4; j++) {
				const int t = m * TS + j * 16 + sg;
				const float p = expf(acc[i][j] * sh.scale - lj[j]);
				Pw[i * (2 * NW) * PP + j * 16 + sg] = p;
				// (equal rows: the distance has no slope in any column, so its gradient reaches neither)
				if (s < sh.n_tok && t < sh.n_tok)
					dxr[size_t(t) * dx_t] = sh.dx_pitch > 0 && acc[i][j] == 0.f ? 0.f : p * (dp[i][j] - dj[j]);
			}
		}
		__syncwarp();

		// dv rows += weights x dvo rows; this lane owns value columns [sg*NV, sg*NV+NV)
#pragma unroll 2
		for (int t4 = 0; t4 < TS / 4; t4++) {
			float4 p[TI];
#pragma unroll
			for (int i = 0; i < TI; i++)
				p[i] = *reinterpret_cast<const float4 *>(Pw + i * (2 * NW) * PP + t4 * 4);
#pragma unroll
			for (int tt = 0; tt < 4; tt++) {
				const int trow = t4 * 4 + tt;
				float gvv[NV];
#pragma unroll
				for (int e = 0; e < NV; e += (NV < 4 ? NV : 4)) {
					const int col = sg * NV + e; // float column within the value row
					const unsigned char *gp = Gs + (col >> 5) * TS * 128 + trow * 128 + ((((col & 31) >> 2) ^ (trow & 7)) << 4);
					if (NV == 2) {
						const float2 t2 = *reinterpret_cast<const float2 *>(gp + (col & 3) * 4);
						gvv[0] = t2.x;
						gvv[1 % NV] = t2.y;
					} else {
						const float4 t4v = *reinterpret_cast<const float4 *>(gp);
						gvv[e] = t4v.x;
						gvv[(e + 1) % NV] = t4v.y;
						gvv[(e + 2) % NV] = t4v.z;
						gvv[(e + 3) % NV] = t4v.w;
					}
				}
#pragma unroll
				for (int i = 0; i < TI; i++) {
					const float pi = tt == 0 ? p[i].x : tt == 1 ? p[i].y : tt == 2 ? p[i].z : p[i].w;
#pragma unroll
					for (int e = 0; e < NV; e++)
						o[i][e] = fmaf(pi, gvv[e], o[i][e]);
				}
			}
		}
		__syncwarp();
		if (lane == 0)
			mbar_arrive(&empty_bar[st]);
	}

#pragma unroll
	for (int i = 0; i < TI; i++) {
		const int s = s0 + i * (2 * NW) + tg;
		if (s >= sh.n_tok)
			continue;
		float *op = dv + v0 + size_t(s) * vrow + sg * NV;
#pragma unroll
		for (int e = 0; e < NV; e++)
			if (FULL || sg * NV + e < sh.v_width)
				op[e] = o[i][e];
	}
}


// The same with both products on the tensor cores (128-row CTAs, width and v_width <= 64): dp = <v, dvo> in D1, dv in D2, operands as
// three bf16 pieces each (see softmax_v_tc_kernel).  The pieces of dvo lie [query][column], queries in the order 4 * (t % 16) + t / 16:
// for dp that is B with its columns along k, for dv B with its queries along k (n contiguous).  Per tile: dp is computed as soon as its
// pieces are there, beside the scores; it goes through shared memory from the tensor memory's rows to the lanes that hold the scores, in
// the place of the weights' pieces, which are written behind it.  Whole backward of [8,1024,16,64], values 64 wide, d_q and d_k included: 2.56 ms,
// with softmax_v_bwd_tile_kernel 3.00.  Bound: FP32 pipe of the scores (55 % of the active cycles, issue 64 %), the two barriers per tile beside it.
template <int NV, bool TMA, bool FULL>
__global__ void __launch_bounds__(TC_THREADS, 1)
softmax_v_bwd_tc_kernel(const __grid_constant__ CUtensorMap qmap, const __grid_constant__ CUtensorMap kmap,
			const __grid_constant__ CUtensorMap gmap, const float *__restrict__ q, const float *__restrict__ k,
			const float *__restrict__ v, const float *__restrict__ dvo, const float *__restrict__ lse,
			const float *__restrict__ delta, float *__restrict__ dx, float *__restrict__ dv, SvShape sh, int *err)
{
	constexpr int NW = TC_NW, TI = 4, TT = TC_ROWS, VW = 16 * NV, NVB = VW / 32, NO = VW / 4;
	constexpr int G_PIECE = TS * 128; // 64 queries of 64 bf16 (VW 32: half of them unused)
	extern __shared__ __align__(1024) unsigned char smem_raw[];
	unsigned char *base = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
	__shared__ __align__(8) TcBars bars;
	const int k_bytes = sh.nwb * TT * 128, q_bytes = sh.nwb * TS * 128, g_bytes = NVB * TS * 128, stage_bytes = q_bytes + g_bytes;
	unsigned char *Vp = base, *Pp = Vp + 3 * TC_A_PIECE, *Gp = Pp + 3 * TC_A_PIECE, *Ks = Gp + 3 * G_PIECE, *stages = Ks + k_bytes;

	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	unsigned r = blockIdx.x;
	const int s0 = int(r % unsigned(sh.ntt)) * TT;
	r /= unsigned(sh.ntt);
	const int h = int(r % unsigned(sh.n_heads));
	const int b = int(r / unsigned(sh.n_heads));
	const int nt = (sh.n_tok + TS - 1) / TS;
	const size_t krow = size_t(sh.n_heads) * sh.width, vrow = size_t(sh.n_heads) * sh.v_width;
	const size_t qk0 = size_t(b) * sh.n_tok * krow + size_t(h) * sh.width, v0 = size_t(b) * sh.n_tok * vrow + size_t(h) * sh.v_width;

	if (warp == 16)
		tmem_alloc(&bars.tmem, TC_BWD_COLUMNS);
	if (tid == 0) {
		mbar_init(&bars.own, TMA ? 1 : NW * 32);
		for (int s = 0; s < MAX_STAGE; s++) {
			mbar_init(&bars.full[s], TMA ? 1 : NW * 32);
			mbar_init(&bars.empty[s], NW + 2);
		}
		mbar_init(&bars.p_full, NW);
		mbar_init(&bars.v_full, 2); // (the pieces of dvo)
		mbar_init(&bars.done, 1);   // D1
		mbar_init(&bars.done2, 1);  // D2
		mbar_init(&bars.patched, NW);
		for (int i = 0; i < TT / 32; i++)
			bars.own_without[i] = 0;
		mbar_fence_init();
	}
	__syncthreads();
	// the CTA's own value rows as pieces [source row][column]
	for (int i = tid; i < TT * (VW / 2); i += TC_THREADS) {
		const int row = i / (VW / 2), c = i % (VW / 2) * 2;
		const float *vp = v + v0 + size_t(s0 + row < sh.n_tok ? s0 + row : 0) * vrow + c;
		bool all = true;
		const float x = take(s0 + row < sh.n_tok && c < sh.v_width ? vp[0] : 0.f, all), y = take(s0 + row < sh.n_tok && c + 1 < sh.v_width ? vp[1] : 0.f, all);
		if (!all)
			atomicOr(&bars.own_without[row >> 5], 1u << (row & 31));
		uint32_t pc[3];
		split_bf16_short(x, y, pc);
		unsigned char *d = Vp + row * 128 + (((c >> 3) ^ (row & 7)) << 4) + (c & 7) * 2;
#pragma unroll
		for (int e = 0; e < 3; e++)
			*reinterpret_cast<uint32_t *>(d + e * TC_A_PIECE) = pc[e];
	}
	fence_proxy_async_smem();
	tc_fence_before();
	__syncthreads();
	tc_fence_after();
	const uint32_t tmem = bars.tmem, D1 = 0, D2 = TC_SUM;
	const size_t hstride = size_t(sh.n_heads);
	const size_t dx_t = sh.dx_pitch > 0 ? 1 : hstride, dx_s = sh.dx_pitch > 0 ? size_t(sh.dx_pitch) : hstride * sh.n_tok;
	const size_t dx0 = sh.dx_pitch > 0 ? (size_t(b) * sh.n_heads + h) * sh.n_tok * sh.dx_pitch : size_t(b) * sh.n_tok * sh.n_tok * hstride + h;

	if (warp < NW) {
		asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(TC_REGS));
		auto load_tile = [&](int m) {
			const int st = m % sh.nstage;
			unsigned char *dst = stages + size_t(st) * stage_bytes;
			if (!TMA) {
				copy_rows<NW, true>(dst, q + qk0, krow, m * TS, TS, sh.nwb, sh.width, sh.n_tok);
				copy_rows<NW, true>(dst + q_bytes, dvo + v0, vrow, m * TS, TS, NVB, sh.v_width, sh.n_tok);
				copy_arrive(&bars.full[st]);
				return;
			}
			mbar_expect_tx(&bars.full[st], uint32_t(stage_bytes));
			for (int wb = 0; wb < sh.nwb; wb++)
				tma_load_4d(dst + wb * TS * 128, &qmap, &bars.full[st], wb * 32, h, m * TS, b);
			for (int vb = 0; vb < NVB; vb++)
				tma_load_4d(dst + q_bytes + vb * TS * 128, &gmap, &bars.full[st], vb * 32, h, m * TS, b);
		};
		if (!TMA || tid == 0) {
			if (TMA) {
				mbar_expect_tx(&bars.own, uint32_t(k_bytes));
				for (int wb = 0; wb < sh.nwb; wb++)
					tma_load_4d(Ks + wb * TT * 128, &kmap, &bars.own, wb * 32, h, s0, b);
			} else {
				copy_rows<NW, true>(Ks, k + qk0, krow, s0, TT, sh.nwb, sh.width, sh.n_tok);
				copy_arrive(&bars.own);
			}
			for (int m = 0; m < sh.nstage - 1 && m < nt; m++)
				load_tile(m);
		}

		const int sg = lane & 15, tg = warp * 2 + (lane >> 4);
		const int orow = (warp & 3) * 32 + lane, part = warp >> 2; // this thread's part of D1 and D2: a row, a quarter of the columns
		const uint32_t d_at = tmem + (uint32_t((warp & 3) * 32) << 16);
		float o[NO];
#pragma unroll
		for (int e = 0; e < NO; e++)
			o[e] = 0.f;
		bool dead = !mbar_wait_inline(&bars.own, 0, err);
		const bool any_own = (bars.own_without[0] | bars.own_without[1] | bars.own_without[2] | bars.own_without[3]) != 0;
		int patches = 0;
		auto collect = [&](int m) { // dv of tile m
			if (!dead && !mbar_wait_inline(&bars.done2, m & 1, err))
				dead = true;
			tc_fence_after();
			float d[NO];
			load_sums(d_at + D2 + part * NO, d);
#pragma unroll
			for (int e = 0; e < NO; e++)
				o[e] = fmaf(d[e], PIECE_UNSCALE, o[e]);
			const unsigned long long which = tile_without(bars, m);
			if (__all_sync(0xffffffffu, which != 0 && !dead)) // (a warp as one, also after a timeout)
				dead = !add_without(o, which, Pp, orow, dvo + v0 + part * NO, vrow, m, sh.n_tok, sh.v_width - part * NO, bars, patches, err);
		};

		for (int m = 0; m < nt; m++) {
			if ((!TMA || (warp == m % NW && lane == 0)) && m + sh.nstage - 1 < nt && !dead) {
				const int mm = m + sh.nstage - 1;
				if (mbar_wait_inline(&bars.empty[mm % sh.nstage], ((unsigned(mm) / unsigned(sh.nstage)) & 1u) ^ 1u, err))
					load_tile(mm);
				else
					dead = true;
			}
			__syncwarp();
			const int st = m % sh.nstage;
			if (!dead && !mbar_wait_inline(&bars.full[st], (unsigned(m) / unsigned(sh.nstage)) & 1u, err))
				dead = true;
			const unsigned char *Qs = stages + size_t(st) * stage_bytes;
			float acc[TI][4];
#pragma unroll
			for (int i = 0; i < TI; i++)
#pragma unroll
				for (int j = 0; j < 4; j++)
					acc[i][j] = 0.f;
			for (int wb = 0; wb < sh.nwb; wb++) {
				const int nc = FULL ? 8 : min(8, ((sh.width - wb * 32 + 7) >> 3) * 2);
				score_slice<TI, NW, FULL>(Ks + wb * TT * 128, Qs + wb * TS * 128, tg, sg, nc, acc);
			}
			__syncwarp();
			if (lane == 0)
				mbar_arrive(&bars.empty[st]);
			// per-query statistics of this lane's 4 columns (in flight while the products are collected)
			float lj[4], dj[4];
#pragma unroll
			for (int j = 0; j < 4; j++) {
				const int t = m * TS + j * 16 + sg;
				const bool ok = t < sh.n_tok;
				const size_t at = (size_t(b) * sh.n_tok + (ok ? t : 0)) * hstride + h;
				lj[j] = ok ? lse[at] : INFINITY; // exp(x - inf) = 0: query rows past the end weigh nothing
				dj[j] = ok ? delta[at] : 0.f;
			}
			if (m > 0)
				collect(m - 1); // (and the weights' pieces of tile m - 1 are read)
			if (!dead && !mbar_wait_inline(&bars.done, m & 1, err))
				dead = true;
			tc_fence_after();
			{ // dp: a row and 16 places of it per thread to [row][place], 16-byte chunk ^= row & 15
				float d[16];
				load_sums(d_at + D1 + part * 16, d);
#pragma unroll
				for (int e = 0; e < 16; e++)
					d[e] *= PIECE_UNSCALE;
#pragma unroll
				for (int e = 0; e < 4; e++)
					*reinterpret_cast<float4 *>(Pp + orow * 256 + (((part * 4 + e) ^ (orow & 15)) << 4)) =
						make_float4(d[e * 4], d[e * 4 + 1], d[e * 4 + 2], d[e * 4 + 3]);
				const unsigned long long which = tile_without(bars, m);
				if (which != 0 || any_own) { // this thread's part again: the terms with a factor that has no pieces
					const float *vr = v + v0 + size_t(s0 + orow) * vrow, *gr = dvo + v0 + size_t(m) * TS * vrow;
					auto token = [&](int i) { return i % 4 * 16 + part * 4 + i / 4; }; // of place part * 16 + i
					auto add = [&](int i, float x, float y) {
						float *cell = reinterpret_cast<float *>(Pp + orow * 256 + (((part * 4 + i / 4) ^ (orow & 15)) << 4)) + i % 4;
						*cell = fmaf(x, y, *cell);
					};
					if (bars.own_without[orow >> 5] >> (orow & 31) & 1) // the factor of v
#pragma unroll 1
						for (int c = 0; c < sh.v_width; c++)
							if (!has_pieces(vr[c]))
#pragma unroll 1
								for (int i = 0; i < 16; i++)
									if (m * TS + token(i) < sh.n_tok)
										add(i, vr[c], gr[size_t(token(i)) * vrow + c]);
					if (which != 0 && s0 + orow < sh.n_tok) // the factor of dvo alone
#pragma unroll 1
						for (int i = 0; i < 16; i++)
							if ((which >> token(i) & 1) && m * TS + token(i) < sh.n_tok)
#pragma unroll 1
								for (int c = 0; c < sh.v_width; c++)
									if (!has_pieces(gr[size_t(token(i)) * vrow + c]) && has_pieces(vr[c]))
										add(i, vr[c], gr[size_t(token(i)) * vrow + c]);
				}
			}
			named_barrier(1, NW * 32);
#pragma unroll
			for (int i = 0; i < TI; i++) {
				const int row = i * (2 * NW) + tg, s = s0 + row;
				const float4 dp = *reinterpret_cast<const float4 *>(Pp + row * 256 + ((sg ^ (row & 15)) << 4));
				float *dxr = dx + dx0 + size_t(s < sh.n_tok ? s : 0) * dx_s;
				const float dpj[4] = {dp.x, dp.y, dp.z, dp.w};
#pragma unroll
				for (int j = 0; j < 4; j++) {
					const int t = m * TS + j * 16 + sg;
					const float p = expf(acc[i][j] * sh.scale - lj[j]);
					// (equal rows: the distance has no slope in any column, so its gradient reaches neither)
					if (s < sh.n_tok && t < sh.n_tok)
						dxr[size_t(t) * dx_t] = sh.dx_pitch > 0 && acc[i][j] == 0.f ? 0.f : p * (dpj[j] - dj[j]);
					acc[i][j] = p;
				}
			}
			named_barrier(1, NW * 32); // (dp is read)
#pragma unroll
			for (int i = 0; i < TI; i++)
				store_weights(Pp, i * (2 * NW) + tg, sg, acc[i]);
			fence_proxy_async_smem();
			tc_fence_before();
			__syncwarp();
			if (lane == 0)
				mbar_arrive(&bars.p_full);
		}
		collect(nt - 1);
		if (s0 + orow < sh.n_tok) {
			float *op = dv + v0 + size_t(s0 + orow) * vrow + part * NO;
#pragma unroll
			for (int e = 0; e < NO; e++)
				if (FULL || part * NO + e < sh.v_width)
					op[e] = o[e];
		}
	} else {
		asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(TC_REGS_REST));
		if (warp == 16 && lane == 0) {
			const uint64_t va = tc_desc(smem_u32(Vp)), pa = tc_desc(smem_u32(Pp)), gk = tc_desc(smem_u32(Gp)), gn = tc_desc_mn(smem_u32(Gp));
			bool dead = false;
			int m = 0;
			for (; m < nt && !dead; m++) {
				dead = !mbar_wait_inline(&bars.v_full, m & 1, err);
				tc_fence_after();
				if (!dead)
					mma_pieces<VW / 16>(tmem + D1, va, TC_A_PIECE, gk, G_PIECE, 32, tc_idesc_bf16(TS, false));
				tc_commit(&bars.done);
				dead = dead || !mbar_wait_inline(&bars.p_full, m & 1, err);
				tc_fence_after();
				if (!dead)
					mma_pieces<TS / 16>(tmem + D2, pa, TC_A_PIECE, gn, G_PIECE, 2048, tc_idesc_bf16(VW, true));
				tc_commit(&bars.done2);
			}
			mbar_wait_inline(&bars.done2, (m - 1) & 1, err); // no product is in flight when the tensor memory goes, also after a timeout
		}
		if (warp == 17 || warp == 18) { // a query row per thread
			const int t = (warp - 17) * 32 + lane, place = 4 * (t % 16) + t / 16;
			bool dead = false;
			for (int m = 0; m < nt; m++) {
				const int st = m % sh.nstage;
				if (!dead && !mbar_wait_inline(&bars.full[st], (unsigned(m) / unsigned(sh.nstage)) & 1u, err))
					dead = true;
				if (m > 0 && !dead && !mbar_wait_inline(&bars.done2, (m - 1) & 1, err))
					dead = true;
				const unsigned char *Gs = stages + size_t(st) * stage_bytes + q_bytes;
				bool all = true;
#pragma unroll 2
				for (int g = 0; g < VW / 8; g++) { // columns 8 g .. 8 g + 7: two chunks of the row's 128-byte slice
					uint32_t o[3][4];
#pragma unroll
					for (int e = 0; e < 2; e++) {
						const float4 x = *reinterpret_cast<const float4 *>(Gs + (g >> 2) * TS * 128 + t * 128 + ((((g & 3) * 2 + e) ^ (t & 7)) << 4));
						uint32_t pa[3], pb[3];
						split_bf16_short(take(x.x, all), take(x.y, all), pa);
						split_bf16_short(take(x.z, all), take(x.w, all), pb);
#pragma unroll
						for (int i = 0; i < 3; i++) {
							o[i][e * 2] = pa[i];
							o[i][e * 2 + 1] = pb[i];
						}
					}
#pragma unroll
					for (int i = 0; i < 3; i++)
						*reinterpret_cast<uint4 *>(Gp + i * G_PIECE + place * 128 + ((g ^ (place & 7)) << 4)) = make_uint4(o[i][0], o[i][1], o[i][2], o[i][3]);
				}
				const uint32_t which = __ballot_sync(0xffffffffu, !all);
				fence_proxy_async_smem();
				__syncwarp();
				if (lane == 0) {
					bars.without[m & 1][warp - 17][warp - 17] = which;
					bars.without[m & 1][warp - 17][18 - warp] = 0;
					mbar_arrive(&bars.v_full);
					mbar_arrive(&bars.empty[st]);
				}
			}
		}
		__syncwarp();
	}
	tc_fence_before();
	__syncthreads();
	if (warp == 16)
		tmem_free(tmem, TC_BWD_COLUMNS);
}

size_t sv_bwd_tc_smem(int nwb, int nv, int nstage)
{
	return size_t(6) * TC_A_PIECE + size_t(3) * TS * 128 + size_t(nwb) * TC_ROWS * 128 + size_t(nstage) * (size_t(nwb) + nv / 2) * TS * 128 + 1024;
}

size_t sv_bwd_smem(int nwb, int nv, int tt_rows, int nstage)
{
	const size_t tt = size_t(tt_rows), nvb = size_t(nv) / 2;
	return (size_t(nwb) + nvb) * tt * 128 + size_t(nstage) * (size_t(nwb) + nvb) * TS * 128 + tt * PP * 4 + 1024;
}

template <int NV, int TI, int NW, bool TMA, bool FULL>
int launch_bwd_tile(const float *q, const float *k, const float *v, const float *dvo, const float *lse, const float *delta,
		    float *dx, int dx_pitch, float *dv, int bs, int n_tok, int n_heads, int width, int v_width, const TilePlan &plan, cudaStream_t st)
{
	constexpr int TT = 2 * NW * TI, NTH = NW * 32;
	const uint64_t dims[4] = {uint64_t(width), uint64_t(n_heads), uint64_t(n_tok), uint64_t(bs)};
	const uint64_t str[3] = {uint64_t(width) * 4, uint64_t(n_heads) * width * 4, uint64_t(n_tok) * n_heads * width * 4};
	const uint64_t vdims[4] = {uint64_t(v_width), uint64_t(n_heads), uint64_t(n_tok), uint64_t(bs)};
	const uint64_t vstr[3] = {uint64_t(v_width) * 4, uint64_t(n_heads) * v_width * 4, uint64_t(n_tok) * n_heads * v_width * 4};
	const uint32_t own[4] = {32, 1, TT, 1}, stream[4] = {32, 1, TS, 1};
	CUtensorMap qmap{}, kmap{}, vmap{}, gmap{};
	const auto f32 = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
	const auto swz = CU_TENSOR_MAP_SWIZZLE_128B;
	if (TMA && (!encode_tmap_4d(&qmap, f32, q, dims, str, stream, swz) || !encode_tmap_4d(&kmap, f32, k, dims, str, own, swz) ||
	    !encode_tmap_4d(&vmap, f32, v, vdims, vstr, own, swz) || !encode_tmap_4d(&gmap, f32, dvo, vdims, vstr, stream, swz)))
		return 1;
	int *err = device_error_word();
	if (!err)
		return 1;
	SvShape sh;
	sh.n_tok = n_tok;
	sh.n_heads = n_heads;
	sh.width = width;
	sh.v_width = v_width;
	sh.nwb = (width + 31) / 32;
	sh.nstage = plan.nstage;
	sh.ntt = (n_tok + TT - 1) / TT;
	sh.mode = 0;
	sh.dx_pitch = dx_pitch;
	sh.scale = float(-1.0 / sqrt(double(width)));
	const long long grid = (long long)bs * n_heads * sh.ntt;
	if (grid > 0x7fffffffLL)
		return L1ATTN_ERR_SHAPE;
	if constexpr (NW == TC_NW)
		if (plan.tc) {
			auto kern = softmax_v_bwd_tc_kernel<NV, TMA, FULL>;
			L1B_SHARED_MEMORY(kern, int(plan.smem));
			L1B_REGISTERS(kern, TC_REGS_LAUNCH);
			kern<<<unsigned(grid), TC_THREADS, plan.smem, st>>>(qmap, kmap, gmap, q, k, v, dvo, lse, delta, dx, dv, sh, err);
			L1B_LAUNCH_CHECK();
			return L1ATTN_OK;
		}
	auto kern = softmax_v_bwd_tile_kernel<NV, TI, NW, TMA, FULL>;
	L1B_SHARED_MEMORY(kern, int(plan.smem));
	kern<<<unsigned(grid), NTH, plan.smem, st>>>(qmap, kmap, vmap, gmap, q, k, v, dvo, lse, delta, dx, dv, sh, err);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

TilePlan sv_bwd_plan(int bs, int n_tok, int n_heads, int width, int v_width)
{
	if (width < 1 || width > 128 || v_width < 1 || v_width > 128)
		return {0, 0, 0, 0, false};
	const int nwb = (width + 31) / 32, nv = sv_nv(v_width);
	return plan_tile(nv, (long long)bs * n_heads, n_tok, sv_bwd_short_cta(nv <= 4 && width <= TC_WIDTH), [&](int tt, int ns) { return sv_bwd_smem(nwb, nv, tt, ns); },
			 [&](int ns) { return width <= TC_WIDTH ? sv_bwd_tc_smem(nwb, nv, ns) : TC_SMEM + 1; });
}

int softmax_v_bwd_tile(const float *q, const float *k, const float *v, const float *dvo, const float *lse, const float *delta,
		       float *dx, int dx_pitch, float *dv, int bs, int n_tok, int n_heads, int width, int v_width, cudaStream_t st)
{
	const TilePlan p = sv_bwd_plan(bs, n_tok, n_heads, width, v_width);
	if (!p.nstage)
		return 1;
	const bool tma = width % 4 == 0 && v_width % 4 == 0 && aligned(q, 16) && aligned(k, 16) && aligned(v, 16) && aligned(dvo, 16);
	const int nv = sv_nv(v_width);
	const bool full = width % 32 == 0 && v_width == 16 * nv; // no padded columns
#define L1B_SVB_RUN(NV_, TI_, NW_, TMA_, FULL_) \
	launch_bwd_tile<NV_, TI_, NW_, TMA_, FULL_>(q, k, v, dvo, lse, delta, dx, dx_pitch, dv, bs, n_tok, n_heads, width, v_width, p, st)
#define L1B_SVB(NV_, TI_, NW_)                                                                                                   \
	if (nv == NV_ && p.ti == TI_ && p.nw == NW_) {                                                                           \
		const int rc = !tma ? 1 : full ? L1B_SVB_RUN(NV_, TI_, NW_, true, true) : L1B_SVB_RUN(NV_, TI_, NW_, true, false); \
		return rc <= 0 ? rc : L1B_SVB_RUN(NV_, TI_, NW_, false, false);                                                   \
	}
	L1B_SVB(2, 4, 8) L1B_SVB(4, 4, 8) L1B_SVB(8, 4, 8) L1B_SVB(8, 8, 8) L1B_SVB(2, 4, 16) L1B_SVB(4, 4, 16)
#undef L1B_SVB
#undef L1B_SVB_RUN
	return 1;
}

} // namespace

// The kernel that a float32 call of these sizes takes: 0 one for any shape, else the rows of a CTA, and one more where the products are on the tensor cores
int dense_softmax_v_form(int bs, int n_tok, int n_heads, int width, int v_width, int backward)
{
	const TilePlan p = backward ? sv_bwd_plan(bs, n_tok, n_heads, width, v_width) : sv_plan(bs, n_tok, n_heads, width, v_width);
	return p.nstage ? 2 * p.ti * p.nw + p.tc : 0;
}

int dense_softmax_v_launch(const void *q, const void *k, const void *v, void *vo, void *lse, int bs, int n_tok, int n_heads,
			   int width, int v_width, int mode, int dtype, cudaStream_t st)
{
	if (bs == 0 || n_tok == 0 || n_heads == 0 || v_width == 0)
		return L1ATTN_OK;
	static const bool no_tma = getenv("L1ATTN_NO_TMA") != nullptr; // debugging aid: force the generic kernel
	if (dtype == L1ATTN_F32 && !no_tma && width > 0) {
		const int rc = softmax_v_tile((const float *)q, (const float *)k, (const float *)v, (float *)vo, (float *)lse, bs, n_tok,
					     n_heads, width, v_width, mode, st);
		if (rc <= 0)
			return rc;
	}
	if (dtype == L1ATTN_F32)
		return launch_generic((const float *)q, (const float *)k, (const float *)v, (float *)vo, (float *)lse, bs, n_tok,
				      n_heads, width, v_width, mode, st);
	return launch_generic((const double *)q, (const double *)k, (const double *)v, (double *)vo, (double *)lse, bs, n_tok,
			      n_heads, width, v_width, mode, st);
}

int dense_softmax_v_bwd_dx_launch(const void *q, const void *k, const void *v, const void *dvo, const void *lse,
				  const void *delta, void *dx, void *dv, int bs, int n_tok, int n_heads, int width, int v_width,
				  int dtype, cudaStream_t st)
{
	if (bs == 0 || n_tok == 0 || n_heads == 0 || v_width == 0)
		return L1ATTN_OK;
	static const bool no_tma = getenv("L1ATTN_NO_TMA") != nullptr;
	if (dtype == L1ATTN_F32 && !no_tma && width > 0) {
		const int rc = softmax_v_bwd_tile((const float *)q, (const float *)k, (const float *)v, (const float *)dvo,
						 (const float *)lse, (const float *)delta, (float *)dx, 0, (float *)dv, bs, n_tok, n_heads,
						 width, v_width, st);
		if (rc <= 0)
			return rc;
	}
	if (dtype == L1ATTN_F32)
		return launch_bwd_generic((const float *)q, (const float *)k, (const float *)v, (const float *)dvo,
					  (const float *)lse, (const float *)delta, (float *)dx, (float *)dv, bs, n_tok, n_heads, width,
					  v_width, st);
	return launch_bwd_generic((const double *)q, (const double *)k, (const double *)v, (const double *)dvo,
				  (const double *)lse, (const double *)delta, (double *)dx, (double *)dv, bs, n_tok, n_heads, width,
				  v_width, st);
}

// Workspace of the whole backward: dx, then the dense backward's scratch.  Its size serves every call of up to bs items (a batch is
// walked in chunks, the last of them smaller).
static size_t sv_dx_bytes(int bs, int n_tok, int n_heads, int dtype)
{
	const size_t es = dtype == L1ATTN_F64 ? 8 : 4, pitch = (size_t(n_tok) + 3) / 4 * 4; // rows of dx as the tiled kernels write them
	return (size_t(bs) * n_heads * n_tok * pitch * es + 255) / 256 * 256;
}
size_t dense_softmax_v_bwd_bytes(int bs, int n_tok, int n_heads, int width, int, int dtype)
{
	return sv_dx_bytes(bs, n_tok, n_heads, dtype) + dense_bwd_scratch_bytes_upto(bs, n_tok, n_heads, width, dtype);
}

// dx lies [b][h][s][t] between its two kernels: the tiled kernel that makes it owns one head, and in d_attn's order, heads innermost, each of
// its 4-byte stores touched a sector of its own (32 sectors per warp store, about as many cycles of the load/store pipe as its shared
// reads take); the kernel that consumes it reads 16 bytes of a row at once and has nothing to transpose.
int dense_softmax_v_bwd_launch(const void *q, const void *k, const void *v, const void *dvo, const void *lse, const void *delta,
			       void *dq, void *dk, void *dv, void *work, int bs, int n_tok, int n_heads, int width, int v_width,
			       int dtype, cudaStream_t st)
{
	if (bs == 0 || n_tok == 0 || n_heads == 0)
		return L1ATTN_OK;
	static const bool no_tma = getenv("L1ATTN_NO_TMA") != nullptr, no_sv = getenv("L1ATTN_NO_SV") != nullptr;
	void *scratch = static_cast<unsigned char *>(work) + sv_dx_bytes(bs, n_tok, n_heads, dtype);
	if (dtype == L1ATTN_F32 && !no_tma && !no_sv && n_tok > bwd_small_tokens(true) && n_tok < (1 << 24)) {
		const int pitch = (n_tok + 3) / 4 * 4;
		int rc = softmax_v_bwd_tile((const float *)q, (const float *)k, (const float *)v, (const float *)dvo, (const float *)lse,
					    (const float *)delta, (float *)work, pitch, (float *)dv, bs, n_tok, n_heads, width, v_width, st);
		if (!rc)
			rc = dense_bwd_listed_launch(work, pitch, q, k, dq, dk, scratch, bs, n_tok, n_heads, width, st);
		if (rc <= 0)
			return rc;
	}
	const int rc = dense_softmax_v_bwd_dx_launch(q, k, v, dvo, lse, delta, work, dv, bs, n_tok, n_heads, width, v_width, dtype, st);
	return rc ? rc : dense_bwd_launch(work, q, k, dq, dk, scratch, bs, n_tok, n_heads, width, dtype, st);
}

} // namespace l1b
