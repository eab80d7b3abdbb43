// Integer graph preprocessing: expandCoo on the GPU and the edge index of the sparse kernels.
//
// Both need, for every row i of a key column, rank_i = #{j < i : key_j == key_i} -- the running
// per-key counter of the reference's Python loop (cuda/l1attn_sparse_cuda.py:70-91).  The order
// is part of the result (bit-exact contract).  rank_cluster_kernel splits the rows into one contiguous
// chunk per warp of a cluster of CTAs: histogram of every chunk, exclusive sums over the chunks, then every
// warp ranks its own chunk in order, 32 rows at a time (lanes holding the same key find each other with
// match.any, take consecutive ranks after the key's running count and the highest such lane writes the count
// back).  rank_by_key_kernel is the same walk by ONE warp over all rows, for few rows or many keys.
// The dst and src columns are independent and run as separate CTAs / clusters.
#include <cooperative_groups.h>
#include "common.cuh"

namespace l1b {
namespace {

constexpr int SMEM_KEYS = 50 * 1024; // int32 counters that fit beside nothing else in 227 KB

// keys[i*stride], i < n; rows whose key is outside [key_lo, key_lo+n_keys) get rank -1 and are
// not counted.  rank_out[i*rstride] may alias keys (each row's key is read before its rank is
// written, and rows are prefetched strictly ahead).  blockIdx.x selects the column: pointers
// advance by `col_step` elements, counts by n_keys, max_out by 1.  key_out (optional) receives the keys as
// int32 beside the ranks (same stride and column step).
template <typename K>
__global__ void __launch_bounds__(32) rank_by_key_kernel(const K *keys, int stride, int n, long long key_lo,
							  long long n_keys, int32_t *rank_out, int rstride,
							  int32_t *counts, int32_t *max_out, int col_step,
							  int use_smem, int32_t *key_out)
{
	extern __shared__ int32_t scnt[];
	const int lane = threadIdx.x;
	keys += size_t(blockIdx.x) * col_step;
	rank_out += size_t(blockIdx.x) * col_step;
	if (key_out)
		key_out += size_t(blockIdx.x) * col_step;
	int32_t *cnt = use_smem ? scnt : counts + size_t(blockIdx.x) * n_keys;
	if (use_smem)
		for (long long i = lane; i < n_keys; i += 32)
			scnt[i] = 0;
	__syncwarp();
	int mx = 0; // the reference starts its maxima at 0, so an empty list reports length 1
	long long nxt = 0;
	if (lane < n)
		nxt = (long long)keys[size_t(lane) * stride];
	for (int base = 0; base < n; base += 32) {
		const int i = base + lane;
		const long long key = nxt - key_lo;
		if (i + 32 < n)
			nxt = (long long)keys[size_t(i + 32) * stride];
		const bool valid = i < n && key >= 0 && key < n_keys;
		const unsigned act = __ballot_sync(0xffffffffu, valid);
		int rank = -1;
		if (valid) {
			const unsigned m = __match_any_sync(act, key);
			const int seen = cnt[key]; // every lane of the group reads the counter ...
			__syncwarp(act);           // ... before its highest lane overwrites it
			rank = seen + __popc(m & ((1u << lane) - 1u));
			if (lane == 31 - __clz(m))
				cnt[key] = rank + 1;
		}
		__syncwarp();
		if (i < n) {
			rank_out[size_t(i) * rstride] = rank;
			if (key_out)
				key_out[size_t(i) * rstride] = int32_t(key + key_lo);
		}
		mx = max(mx, rank);
	}
	for (int o = 16; o > 0; o >>= 1)
		mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
	if (max_out && lane == 0)
		max_out[blockIdx.x] = mx + 1;
	if (use_smem && counts) { // hand the final counts to the caller (index build needs them)
		__syncwarp();
		int32_t *gc = counts + size_t(blockIdx.x) * n_keys;
		for (long long i = lane; i < n_keys; i += 32)
			gc[i] = scnt[i];
	}
}

// The same ranks, by a cluster of RC CTAs per column.  Chunk c = CTA rank * nwarp + warp holds rows
// [c * per, (c + 1) * per).  Shared memory of a CTA: cnt[nwarp][n_keys] (a chunk's histogram, then its running
// counts) and tot[n_keys] (the CTA's histogram, read by the CTAs after it through distributed shared memory).
// Bound by the latency of the ranked walk (one match + shared read + write per 32 rows, in order): RC * nwarp walks
// of n / (RC * nwarp) rows side by side instead of one of n.  Both columns of 75000 rows with 1024 ids: 20.5 us
// (one warp per column: 989 us), 400000 rows: 74 us (5.2 ms); with 8192 ids, where clearing and summing the six copies of the
// counters that fit weighs more, 44 us (1.0 ms).
namespace cg = cooperative_groups;
constexpr int RC = 8;            // CTAs per cluster (the portable maximum)
constexpr int RANK_THREADS = 512; // 16 warps; the first `nwarp` of them own a chunk, all share the per-key sums
constexpr int RANK_SMEM = 208 * 1024;

template <typename K>
__device__ __forceinline__ void rank_chunks(int32_t *rsm, int32_t &smax, int col, const K *keys, int stride, int n, long long key_lo, int n_keys, int32_t *rank_out, int rstride,
		    int32_t *counts, int32_t *max_out, int col_step, int nwarp, int32_t *key_out)
{
	cg::cluster_group cluster = cg::this_cluster();
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int crank = int(cluster.block_rank());
	keys += size_t(col) * col_step;
	rank_out += size_t(col) * col_step;
	if (key_out)
		key_out += size_t(col) * col_step;
	int32_t *tot = rsm + size_t(nwarp) * n_keys;
	for (int i = tid; i < nwarp * n_keys; i += RANK_THREADS)
		rsm[i] = 0;
	if (tid == 0)
		smax = 0;
	__syncthreads();

	const long long per = (((long long)n + RC * nwarp - 1) / (RC * nwarp) + 31) / 32 * 32;
	const long long lo = (long long)(crank * nwarp + warp) * per;
	const int begin = int(lo < n ? lo : n), end = int(lo + per < n ? lo + per : n);
	int32_t *cnt = rsm + size_t(warp) * n_keys; // (warps >= nwarp own no chunk and never touch it)
	if (warp < nwarp) {
#pragma unroll 4
		for (int i = begin + lane; i < end; i += 32) {
			const long long key = (long long)keys[size_t(i) * stride] - key_lo;
			if (key >= 0 && key < n_keys)
				atomicAdd(&cnt[key], 1);
		}
	}
	__syncthreads();
	for (int x = tid; x < n_keys; x += RANK_THREADS) {
		int32_t s = 0;
		for (int w = 0; w < nwarp; w++)
			s += rsm[size_t(w) * n_keys + x];
		tot[x] = s;
	}
	cluster.sync();
	int mx = 0;
	for (int x = tid; x < n_keys; x += RANK_THREADS) {
		int32_t run = 0;
		for (int r = 0; r < crank; r++)
			run += cluster.map_shared_rank(tot, r)[x];
		for (int w = 0; w < nwarp; w++) {
			const int32_t c = rsm[size_t(w) * n_keys + x];
			rsm[size_t(w) * n_keys + x] = run;
			run += c;
		}
		if (crank == RC - 1) { // the last chunk's end: the key's count over all rows
			if (counts)
				counts[size_t(col) * n_keys + x] = run;
			mx = max(mx, run);
		}
	}
	for (int o = 16; o > 0; o >>= 1)
		mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
	if (lane == 0 && mx > 0)
		atomicMax(&smax, mx);
	cluster.sync(); // the other CTAs have read this one's tot; every thread sees the chunk's running counts
	if (max_out && crank == RC - 1 && tid == 0)
		max_out[col] = max(smax, 1); // longest list; an empty column reports 1, as the reference does

	if (warp >= nwarp)
		return;
	long long nxt = begin + lane < end ? (long long)keys[size_t(begin + lane) * stride] : 0;
	for (int base = begin; base < end; base += 32) {
		const int i = base + lane;
		const long long key = nxt - key_lo;
		if (i + 32 < end)
			nxt = (long long)keys[size_t(i + 32) * stride];
		const bool valid = i < end && key >= 0 && key < n_keys;
		const unsigned act = __ballot_sync(0xffffffffu, valid);
		int rank = -1;
		if (valid) {
			const unsigned m = __match_any_sync(act, unsigned(key)); // n_keys fits 32 bits
			const int seen = cnt[key];
			__syncwarp(act);
			rank = seen + __popc(m & ((1u << lane) - 1u));
			if (lane == 31 - __clz(m))
				cnt[key] = rank + 1;
		}
		__syncwarp();
		if (i < end) {
			rank_out[size_t(i) * rstride] = rank;
			if (key_out)
				key_out[size_t(i) * rstride] = int32_t(key + key_lo);
		}
	}
}

template <typename K>
__global__ void __cluster_dims__(RC, 1, 1) __launch_bounds__(RANK_THREADS)
rank_cluster_kernel(const K *keys, int stride, int n, long long key_lo, int n_keys, int32_t *rank_out, int rstride,
		    int32_t *counts, int32_t *max_out, int col_step, int nwarp, int32_t *key_out)
{
	extern __shared__ int32_t rsm[];
	__shared__ int32_t smax;
	rank_chunks(rsm, smax, int(blockIdx.x) / RC, keys, stride, n, key_lo, n_keys, rank_out, rstride, counts, max_out, col_step, nwarp,
		    key_out);
}

__host__ __device__ inline int rank_warps(long long n_keys) // chunks per CTA whose counters fit, one array for the sums left over
{
	const long long fit = RANK_SMEM / (n_keys * 4) - 1;
	return int(fit < RANK_THREADS / 32 ? fit : RANK_THREADS / 32);
}

// expandCoo as ONE kernel: the range of the ids, then (where it fits) the ranks of both columns, a cluster each.  The host learns range
// and list lengths from one copy; with the range found first, by a kernel of its own, it had to wait for the device twice.
// result: lowest id, highest id, length of the longest dst list, of the longest src list -- or 0, 0 when the counters of so
// many ids (or ids beyond int32) do not fit and nothing else was written.
__global__ void __cluster_dims__(RC, 1, 1) __launch_bounds__(RANK_THREADS)
expand_cluster_kernel(const int64_t *co, int n, int32_t *coo, long long *result)
{
	extern __shared__ int32_t rsm[];
	__shared__ int32_t smax;
	__shared__ int32_t longest[2];
	__shared__ long long slo[RANK_THREADS / 32], shi[RANK_THREADS / 32], range[2];
	cg::cluster_group cluster = cg::this_cluster();
	const int tid = threadIdx.x, crank = int(cluster.block_rank()), col = int(blockIdx.x) / RC;
	long long lo = INT64_MAX, hi = INT64_MIN;
#pragma unroll 4
	for (long long i = (long long)crank * RANK_THREADS + tid; i < 2LL * n; i += RC * RANK_THREADS) {
		const long long v = co[i];
		lo = min(lo, v);
		hi = max(hi, v);
	}
	for (int o = 16; o > 0; o >>= 1) {
		lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
		hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
	}
	if ((tid & 31) == 0) {
		slo[tid >> 5] = lo;
		shi[tid >> 5] = hi;
	}
	__syncthreads();
	if (tid == 0) {
		for (int w = 1; w < RANK_THREADS / 32; w++) {
			lo = min(lo, slo[w]);
			hi = max(hi, shi[w]);
		}
		range[0] = lo;
		range[1] = hi;
	}
	cluster.sync();
	for (int r = 0; r < RC; r++) {
		const long long *other = cluster.map_shared_rank(range, r);
		lo = min(lo, other[0]);
		hi = max(hi, other[1]);
	}
	const bool fits = lo >= INT32_MIN && hi <= INT32_MAX && 2 * (hi - lo + 1) * 4 <= RANK_SMEM; // the same in every thread
	if (fits) {
		const int n_keys = int(hi - lo + 1);
		// (max_out: shared memory of this CTA, written by the last CTA of the cluster only)
		rank_chunks(rsm, smax, col, co, 2, n, lo, n_keys, coo + 2, 4, nullptr, longest, 1, rank_warps(n_keys), coo);
	} else {
		cluster.sync(); // shared memory must outlive the others' reads (rank_chunks has such a barrier too)
	}
	if (crank == RC - 1 && tid == 0) {
		if (col == 0) {
			result[0] = lo;
			result[1] = hi;
		}
		result[2 + col] = fits ? longest[col] : 0;
	}
}

// Smallest and largest of x, by one cluster (no scratch, no second launch).
__global__ void __cluster_dims__(RC, 1, 1) __launch_bounds__(1024) minmax_kernel(const int64_t *x, long long n, int64_t *out)
{
	__shared__ long long slo[32], shi[32];
	cg::cluster_group cluster = cg::this_cluster();
	long long lo = INT64_MAX, hi = INT64_MIN;
#pragma unroll 4
	for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
		const long long v = x[i];
		lo = min(lo, v);
		hi = max(hi, v);
	}
	for (int o = 16; o > 0; o >>= 1) {
		lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
		hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
	}
	if ((threadIdx.x & 31) == 0) {
		slo[threadIdx.x >> 5] = lo;
		shi[threadIdx.x >> 5] = hi;
	}
	cluster.sync();
	if (cluster.block_rank() == 0 && threadIdx.x < 32) {
		for (int r = 0; r < RC; r++) {
			lo = min(lo, cluster.map_shared_rank(slo, r)[threadIdx.x]);
			hi = max(hi, cluster.map_shared_rank(shi, r)[threadIdx.x]);
		}
		for (int o = 16; o > 0; o >>= 1) {
			lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
			hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
		}
		if (threadIdx.x == 0) {
			out[0] = lo;
			out[1] = hi;
		}
	}
	cluster.sync(); // shared memory must outlive the first CTA's reads
}

// ---- sparse edge index ------------------------------------------------------------------

__global__ void idx_init_kernel(int32_t *slot_src, long long nslot, int32_t *cnt, int n_tok, int32_t *status)
{
	const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (i < nslot)
		slot_src[i] = -1;
	if (i < n_tok)
		cnt[i] = 0;
	if (i == 0 && status)
		*status = 0;
}

// slot table + the key column for the src ranking (invalid rows: key -1)
__global__ void idx_scatter_kernel(const int32_t *coo, int cl, int n_tok, int dm, int32_t *slot_src,
				   int32_t *key, int32_t *status)
{
	const int c = blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= cl)
		return;
	const int dst = coo[4 * size_t(c)], src = coo[4 * size_t(c) + 1], r = coo[4 * size_t(c) + 2];
	const bool ok = dst >= 0 && dst < n_tok && src >= 0 && src < n_tok && r >= 0 && r < dm;
	if (ok) {
		slot_src[size_t(dst) * dm + r] = src;
	} else if (status) {
		*status = L1ATTN_ERR_INDEX;
	}
	key[c] = ok ? src : -1;
}

// exclusive scan of cnt[0..n) into off[0..n], one CTA
__global__ void __launch_bounds__(1024) idx_scan_kernel(const int32_t *cnt, int32_t *off, int n)
{
	__shared__ int32_t wsum[32];
	__shared__ int32_t carry_s;
	if (threadIdx.x == 0)
		carry_s = 0;
	__syncthreads();
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (int base = 0; base < n; base += 1024) {
		const int i = base + threadIdx.x;
		const int v = i < n ? cnt[i] : 0;
		int x = v;
		for (int o = 1; o < 32; o <<= 1) {
			const int y = __shfl_up_sync(0xffffffffu, x, o);
			if (lane >= o)
				x += y;
		}
		if (lane == 31)
			wsum[warp] = x;
		__syncthreads();
		if (warp == 0) {
			int s = wsum[lane];
			for (int o = 1; o < 32; o <<= 1) {
				const int y = __shfl_up_sync(0xffffffffu, s, o);
				if (lane >= o)
					s += y;
			}
			wsum[lane] = s; // inclusive over warps
		}
		__syncthreads();
		const int carry = carry_s;
		const int incl = x + (warp ? wsum[warp - 1] : 0) + carry;
		if (i < n)
			off[i] = incl - v;
		__syncthreads();
		if (threadIdx.x == 1023)
			carry_s = incl;
		__syncthreads();
	}
	if (threadIdx.x == 0)
		off[n] = carry_s;
}

__global__ void idx_fill_kernel(const int32_t *coo, const int32_t *rank, const int32_t *off, int32_t *csc_slot,
				int cl, int dm)
{
	const int c = blockIdx.x * blockDim.x + threadIdx.x;
	if (c >= cl)
		return;
	const int rk = rank[c];
	if (rk < 0)
		return;
	const int dst = coo[4 * size_t(c)], src = coo[4 * size_t(c) + 1], r = coo[4 * size_t(c) + 2];
	csc_slot[off[src] + rk] = dst * dm + r;
}

size_t pad16(size_t n_int) { return ((n_int * 4 + 15) / 16) * 16; }

template <typename K>
int launch_rank(const K *keys, int stride, int n, long long key_lo, long long n_keys, int32_t *rank_out,
		int rstride, int32_t *counts, int32_t *max_out, int col_step, int ncol, int32_t *key_out, cudaStream_t st)
{
	// A cluster unless one warp is done sooner or its counters do not fit (nwarp + 1 arrays of n_keys).  One warp takes
	// 13 ns a row, the cluster 7 us and 1.5 ns a key before its walk.  Measured, one warp against the cluster: 1024 rows of
	// 8192 ids 18.5 / 19.2 us, 2048 rows 32.8 / 20.5; 2048 rows of 20000 ids 33.9 / 36.9, 8192 rows 116 / 47;
	// 64 rows of 1024 ids 11.3 / 6.7.
	if (8LL * n >= n_keys && n > 0 && n_keys > 0 && 2 * n_keys * 4 <= RANK_SMEM) {
		const int nwarp = rank_warps(n_keys);
		const size_t smem = size_t(nwarp + 1) * n_keys * 4;
		auto kern = rank_cluster_kernel<K>;
		L1B_SHARED_MEMORY(kern, int(smem));
		kern<<<ncol * RC, RANK_THREADS, smem, st>>>(keys, stride, n, key_lo, int(n_keys), rank_out, rstride, counts, max_out,
							    col_step, nwarp, key_out);
		L1B_LAUNCH_CHECK();
		return L1ATTN_OK;
	}
	const int use_smem = n_keys <= SMEM_KEYS;
	if (!use_smem && !counts)
		return L1ATTN_ERR_ARG;
	auto kern = rank_by_key_kernel<K>;
	size_t smem = use_smem ? size_t(n_keys) * 4 : 0;
	if (smem > 48 * 1024)
		L1B_SHARED_MEMORY(kern, int(smem));
	if (!use_smem)
		L1B_CUDA(cudaMemsetAsync(counts, 0, size_t(ncol) * n_keys * 4, st));
	kern<<<ncol, 32, smem, st>>>(keys, stride, n, key_lo, n_keys, rank_out, rstride, counts, max_out, col_step,
				     use_smem, key_out);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

} // namespace

SparseIndex sparse_index_view(void *base, int cl, int n_tok, int dst_mxlen)
{
	SparseIndex ix;
	unsigned char *p = static_cast<unsigned char *>(base);
	size_t o = 0;
	ix.slot_src = reinterpret_cast<int32_t *>(p + o);
	o += pad16(size_t(n_tok) * dst_mxlen);
	ix.csc_off = reinterpret_cast<int32_t *>(p + o);
	o += pad16(size_t(n_tok) + 1);
	ix.csc_slot = reinterpret_cast<int32_t *>(p + o);
	o += pad16(size_t(cl));
	ix.cnt = reinterpret_cast<int32_t *>(p + o);
	o += pad16(size_t(n_tok));
	ix.rank = reinterpret_cast<int32_t *>(p + o);
	o += pad16(size_t(cl));
	ix.bytes = o ? o : 16;
	return ix;
}

} // namespace l1b

using namespace l1b;

extern "C" size_t l1attn_sparse_index_bytes(int cl, int n_tok, int dst_mxlen)
{
	if (cl < 0 || n_tok < 0 || dst_mxlen < 0)
		return 0;
	return sparse_index_view(nullptr, cl, n_tok, dst_mxlen).bytes;
}

extern "C" int l1attn_sparse_build_index(const int32_t *coo, int cl, int n_tok, int dst_mxlen, void *index,
					  int32_t *status, void *stream)
{
	if (cl < 0 || n_tok < 0 || dst_mxlen < 0 || !index || (cl > 0 && !coo))
		return L1ATTN_ERR_ARG;
	if ((long long)n_tok * dst_mxlen > 0x7fffffffLL)
		return L1ATTN_ERR_SHAPE;
	cudaStream_t st = static_cast<cudaStream_t>(stream);
	SparseIndex ix = sparse_index_view(index, cl, n_tok, dst_mxlen);
	const long long nslot = (long long)n_tok * dst_mxlen;
	const long long ninit = nslot > n_tok ? nslot : n_tok;
	idx_init_kernel<<<unsigned((ninit + 255) / 256 + 1), 256, 0, st>>>(ix.slot_src, nslot, ix.cnt, n_tok, status);
	L1B_LAUNCH_CHECK();
	if (cl > 0) {
		idx_scatter_kernel<<<(cl + 255) / 256, 256, 0, st>>>(coo, cl, n_tok, dst_mxlen, ix.slot_src, ix.rank, status);
		L1B_LAUNCH_CHECK();
		int rc = launch_rank<int32_t>(ix.rank, 1, cl, 0, n_tok, ix.rank, 1, ix.cnt, nullptr, 0, 1, nullptr, st);
		if (rc)
			return rc;
	}
	idx_scan_kernel<<<1, 1024, 0, st>>>(ix.cnt, ix.csc_off, n_tok);
	L1B_LAUNCH_CHECK();
	if (cl > 0) {
		idx_fill_kernel<<<(cl + 255) / 256, 256, 0, st>>>(coo, ix.rank, ix.csc_off, ix.csc_slot, cl, dst_mxlen);
		L1B_LAUNCH_CHECK();
	}
	return L1ATTN_OK;
}

extern "C" size_t l1attn_expand_coo_scratch_bytes(long long n_keys)
{
	if (n_keys <= SMEM_KEYS)
		return 0;
	return size_t(n_keys) * 2 * 4;
}

extern "C" int l1attn_expand_coo(const int64_t *co, int cl, int32_t *coo, int32_t *mxlen, long long key_lo,
				  long long n_keys, void *counters, void *stream)
{
	if (cl < 0 || !mxlen || n_keys < 0 || (cl > 0 && (!co || !coo)))
		return L1ATTN_ERR_ARG;
	if (n_keys > 0x7fffffffLL)
		return L1ATTN_ERR_SHAPE;
	cudaStream_t st = static_cast<cudaStream_t>(stream);
	// column 0 -> ranks into coo[:,2], column 1 -> coo[:,3]; with cl == 0 the kernel still writes mxlen = 1
	int32_t *cnt = n_keys > SMEM_KEYS ? static_cast<int32_t *>(counters) : nullptr;
	return launch_rank<int64_t>(co, 2, cl, key_lo, n_keys, coo ? coo + 2 : nullptr, 4, cnt, mxlen, 1, 2, coo, st);
}

extern "C" int l1attn_expand_coo_once(const int64_t *co, int cl, int32_t *coo, int64_t *result, void *stream)
{
	if (cl < 1 || !co || !coo || !result)
		return L1ATTN_ERR_ARG;
	L1B_SHARED_MEMORY(expand_cluster_kernel, RANK_SMEM);
	expand_cluster_kernel<<<2 * RC, RANK_THREADS, RANK_SMEM, static_cast<cudaStream_t>(stream)>>>(co, cl, coo, reinterpret_cast<long long *>(result));
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}

extern "C" int l1attn_i64_minmax(const int64_t *x, long long n, int64_t *out, void *stream)
{
	if (n < 0 || !out || (n > 0 && !x))
		return L1ATTN_ERR_ARG;
	minmax_kernel<<<RC, 1024, 0, static_cast<cudaStream_t>(stream)>>>(x, n, out);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}
