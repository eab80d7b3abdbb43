// Host side of the TMA helpers: tensor-map encoding through the driver entry point (no link
// against libcuda), and the sticky device error word.
#include <atomic>
#include <cstddef>
#include <mutex>
#include "common.cuh"
#include "tma.cuh"
#include "tcgen05.cuh"

namespace l1b {

namespace {
struct KernelError {
	int word, pad;
	int *host;
};
__device__ KernelError l1b_kernel_error;
static_assert(offsetof(KernelError, host) == ERROR_HOST_WORD * sizeof(int), "layout");
constexpr int MAX_DEVICES = 64;
std::atomic<int *> g_error_addr[MAX_DEVICES], g_error_host[MAX_DEVICES];
std::atomic<int> g_sms[MAX_DEVICES];
std::mutex g_error_mu;

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
				  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
				  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
std::once_flag g_once;

void resolve()
{
	void *fn = nullptr;
	cudaDriverEntryPointQueryResult qres;
	if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess &&
	    qres == cudaDriverEntryPointSuccess)
		g_encode = reinterpret_cast<EncodeTiledFn>(fn);
	else
		(void)cudaGetLastError();
}
} // namespace

bool encode_tmap_4d(CUtensorMap *out, CUtensorMapDataType dt, const void *base, const uint64_t dims[4],
		    const uint64_t strides_bytes[3], const uint32_t box[4], CUtensorMapSwizzle swz)
{
	std::call_once(g_once, resolve);
	if (!g_encode)
		return false;
	cuuint64_t d[4], s[3];
	cuuint32_t b[4], es[4] = {1, 1, 1, 1};
	for (int i = 0; i < 4; i++) {
		d[i] = dims[i];
		b[i] = box[i];
	}
	for (int i = 0; i < 3; i++)
		s[i] = strides_bytes[i];
	const CUresult r = g_encode(out, dt, 4, const_cast<void *>(base), d, s, b, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
				    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
	return r == CUDA_SUCCESS;
}

int *device_error_word()
{
	int dev = 0;
	KernelError *p = nullptr;
	if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) {
		(void)cudaGetLastError();
		return nullptr;
	}
	if (int *known = g_error_addr[dev].load(std::memory_order_acquire))
		return known;
	if (cudaGetSymbolAddress(reinterpret_cast<void **>(&p), l1b_kernel_error) != cudaSuccess) {
		(void)cudaGetLastError();
		return nullptr;
	}
	g_error_addr[dev].store(&p->word, std::memory_order_release);
	return &p->word;
}

int multiprocessors(int *out)
{
	int dev = 0, n = 0;
	L1B_CUDA(cudaGetDevice(&dev));
	const bool slot = dev >= 0 && dev < MAX_DEVICES;
	if (slot && (n = g_sms[dev].load(std::memory_order_relaxed)) > 0) {
		*out = n;
		return L1ATTN_OK;
	}
	L1B_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
	if (slot)
		g_sms[dev].store(n, std::memory_order_relaxed);
	*out = n;
	return L1ATTN_OK;
}

} // namespace l1b

// Reads (and clears, with the host's copy of it) the sticky error word set by a kernel whose bounded wait ran out.
extern "C" int l1attn_device_status(void)
{
	int v = 0, dev = 0;
	int *p = l1b::device_error_word();
	if (!p)
		return L1ATTN_ERR_CUDA;
	L1B_CUDA(cudaMemcpy(&v, p, sizeof(int), cudaMemcpyDeviceToHost));
	if (v) {
		L1B_CUDA(cudaMemset(p, 0, sizeof(int)));
		L1B_CUDA(cudaGetDevice(&dev)); // (device_error_word() has found it in range)
		if (volatile int *host = l1b::g_error_host[dev].load(std::memory_order_acquire))
			*host = 0; // reported: the next look at the host word must not report it again
		return L1ATTN_ERR_TIMEOUT;
	}
	return L1ATTN_OK;
}

// The current device's host word: pinned memory that a kernel of this library sets to 1 when it gives up a bounded wait, at once and
// without a copy on any stream.  The caller clears it.  Null when it cannot be had now (the first call on a device needs
// to allocate and copy: not while a stream of the process captures in global mode).
extern "C" int *l1attn_device_status_word(void)
{
	using namespace l1b;
	int dev = 0, *err = device_error_word(), *host = nullptr;
	if (!err || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES)
		return nullptr;
	if ((host = g_error_host[dev].load(std::memory_order_acquire)))
		return host;
	std::lock_guard<std::mutex> lock(g_error_mu);
	if ((host = g_error_host[dev].load(std::memory_order_relaxed)))
		return host;
	cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed; // this thread's calls below belong to no capture
	cudaStream_t st = nullptr;
	if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) {
		(void)cudaGetLastError();
		return nullptr;
	}
	bool ok = cudaHostAlloc(reinterpret_cast<void **>(&host), 64, cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess;
	if (ok) {
		host[0] = host[1] = 0;
		ok = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess &&
		     cudaMemcpyAsync(err + ERROR_HOST_WORD, &host, sizeof host, cudaMemcpyHostToDevice, st) == cudaSuccess &&
		     cudaMemcpyAsync(&host[1], err, sizeof(int), cudaMemcpyDeviceToHost, st) == cudaSuccess &&
		     cudaStreamSynchronize(st) == cudaSuccess;
		if (ok && host[1])
			*reinterpret_cast<volatile int *>(host) = 1; // a kernel has given up before there was a host word
		if (st)
			(void)cudaStreamDestroy(st);
		if (!ok)
			(void)cudaFreeHost(host);
	}
	(void)cudaThreadExchangeStreamCaptureMode(&mode);
	if (!ok) {
		(void)cudaGetLastError();
		return nullptr;
	}
	g_error_host[dev].store(host, std::memory_order_release);
	return host;
}

// Copies the error word to *host_word on `stream` without waiting and without clearing it.  With host_word in
// pinned memory a caller can look at the word before its next launch and call l1attn_device_status() only when
// it is set.
extern "C" int l1attn_device_status_async(int *host_word, void *stream)
{
	int *p = l1b::device_error_word();
	if (!p || !host_word)
		return L1ATTN_ERR_ARG;
	L1B_CUDA(cudaMemcpyAsync(host_word, p, sizeof(int), cudaMemcpyDeviceToHost, static_cast<cudaStream_t>(stream)));
	return L1ATTN_OK;
}

namespace l1b {
namespace {
// One warp waits on a barrier that nothing ever completes, with a short limit: the wait runs out, the error word
// is set and the kernel returns.  Nothing faults and nothing hangs; it exists so that the give-up path of
// mbar_wait and the error word's set / read / clear cycle can be exercised.  limit_polls: the wait that counts its polls instead.
__global__ void wait_timeout_probe_kernel(unsigned long long limit_ns, unsigned limit_polls, int *err, int *returned)
{ // returned[0]: 1 = the wait gave up, 2 = it succeeded (cannot happen); returned[1]: failed polls of thread 0
	__shared__ __align__(8) uint64_t bar;
	if (threadIdx.x == 0) {
		mbar_init(&bar, 1);
		mbar_fence_init();
	}
	__syncthreads();
	unsigned polls = limit_polls;
	const bool ok = limit_polls ? mbar_wait_inline(&bar, 0, err, limit_polls) : mbar_wait_timed(&bar, 0, err, limit_ns, &polls);
	if (threadIdx.x == 0) {
		returned[0] = ok ? 2 : 1;
		returned[1] = int(polls);
	}
}
} // namespace
} // namespace l1b

static int wait_timeout_probe(int limit_us, int limit_polls, int *returned_dev, void *stream)
{
	const int limit = limit_us + limit_polls; // one of them is 0
	if (limit < 1 || limit > 100000 || !returned_dev)
		return L1ATTN_ERR_ARG;
	int *err = l1b::device_error_word();
	if (!err)
		return L1ATTN_ERR_CUDA;
	l1b::wait_timeout_probe_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(1000ull * limit_us, unsigned(limit_polls), err, returned_dev);
	L1B_LAUNCH_CHECK();
	return L1ATTN_OK;
}
extern "C" int l1attn_test_wait_timeout(int limit_us, int *returned_dev, void *stream) { return wait_timeout_probe(limit_us, 0, returned_dev, stream); }
extern "C" int l1attn_test_wait_polls(int polls, int *returned_dev, void *stream) { return wait_timeout_probe(0, polls, returned_dev, stream); }
