#include "pg_runtime.h"

#include <algorithm>
#include <mutex>
#include <set>
#include <utility>

namespace pg
{

namespace
{
thread_local std::string t_last_error;
}

void set_last_error(const std::string& message)
{
	t_last_error = message;
}

const char* last_error()
{
	return t_last_error.c_str();
}

void require_device()
{
	int n = 0;
	const cudaError_t err = cudaGetDeviceCount(&n);
	if(err != cudaSuccess || n == 0)
	{
		throw Error(PG_ERR_NO_DEVICE,
			std::string("no CUDA device available (") + cudaGetErrorString(err) +
			"); the B200 path-tracing core has no CPU fallback");
	}
}

int current_device()
{
	int dev = -1;
	PG_CUDA_CHECK(cudaGetDevice(&dev));
	if(dev < 0 || dev >= kMaxDevices)
	{
		throw Error(PG_ERR_INVALID_ARGUMENT, "device index " + std::to_string(dev) + " out of range");
	}
	return dev;
}

cudaStream_t library_stream()
{
	static std::mutex mutex;
	static cudaStream_t streams[kMaxDevices] = {};
	const int dev = current_device();
	std::lock_guard<std::mutex> lock(mutex);
	if(!streams[dev])
	{
		const cudaError_t status = cudaStreamCreateWithFlags(&streams[dev], cudaStreamNonBlocking);
		if(status != cudaSuccess)
		{
			streams[dev] = nullptr;
			cudaGetLastError();
			throw Error(PG_ERR_CUDA, std::string("cudaStreamCreate: ") + cudaGetErrorString(status));
		}
	}
	return streams[dev];
}

namespace
{

std::mutex g_scratch_mutex;
struct ScratchPool
{
	cudaMemPool_t pool = nullptr;
	std::size_t live = 0;   // bytes of the buffers in use
	std::size_t high = 0;   // the most that were in use since the pool was last cut back
};
ScratchPool g_scratch[kMaxDevices];

// (the mutex is held)
cudaMemPool_t make_scratch_pool(int dev)
{
	cudaMemPoolProps props{};
	props.allocType = cudaMemAllocationTypePinned;
	props.location.type = cudaMemLocationTypeDevice;
	props.location.id = dev;
	cudaMemPool_t pool = nullptr;
	PG_CUDA_CHECK(cudaMemPoolCreate(&pool, &props));
	uint64_t kept = kScratchKept;
	const cudaError_t status = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &kept);
	if(status != cudaSuccess)
	{
		cudaMemPoolDestroy(pool);
		cudaGetLastError();
		throw Error(PG_ERR_CUDA, std::string("cudaMemPoolSetAttribute: ") + cudaGetErrorString(status));
	}
	return pool;
}

}// end anonymous namespace

void* scratch_alloc(std::size_t bytes)
{
	const int dev = current_device();
	ScratchPool& scratch = g_scratch[dev];
	{
		std::lock_guard<std::mutex> lock(g_scratch_mutex);
		if(!scratch.pool)
		{
			scratch.pool = make_scratch_pool(dev);
		}
	}
	void* p = nullptr;
	PG_CUDA_CHECK(cudaMallocFromPoolAsync(&p, bytes, scratch.pool, library_stream()));
	std::lock_guard<std::mutex> lock(g_scratch_mutex);
	scratch.live += bytes;
	scratch.high = std::max(scratch.high, scratch.live);
	return p;
}

void scratch_free(void* p, std::size_t bytes) noexcept
{
	// (device, pool and stream exist: the allocation was made from them)
	try
	{
		cudaStream_t s = library_stream();
		cudaFreeAsync(p, s);
		ScratchPool& scratch = g_scratch[current_device()];
		{
			std::lock_guard<std::mutex> lock(g_scratch_mutex);
			scratch.live -= bytes;
			if(scratch.high <= kScratchKept || scratch.live > kScratchKept)
			{
				return;
			}
			scratch.high = scratch.live;
		}
		// The release threshold acts at a synchronize only, and a call's last one is before its buffers are freed:
		// what a large call took beyond the threshold would stay until somebody synchronizes again.
		cudaStreamSynchronize(s);
		cudaMemPoolTrimTo(scratch.pool, kScratchKept);
	}
	catch(...)
	{
	}
}

void trim_scratch()
{
	const int dev = current_device();
	if(g_scratch[dev].pool)
	{
		cudaStreamSynchronize(library_stream());   // buffers count as freed once the host has seen the stream pass them
	}
	std::lock_guard<std::mutex> lock(g_scratch_mutex);
	for(const ScratchPool& scratch : g_scratch)
	{
		if(scratch.pool)
		{
			cudaMemPoolTrimTo(scratch.pool, 0);
		}
	}
}

void* device_alloc(std::size_t bytes)
{
	void* p = nullptr;
	cudaError_t status = cudaMalloc(&p, bytes);
	if(status == cudaErrorMemoryAllocation)
	{
		(void)cudaGetLastError();
		trim_scratch();
		status = cudaMalloc(&p, bytes);
	}
	PG_CUDA_CHECK(status);
	return p;
}

unsigned char* pinned_stage()
{
	struct Stage
	{
		void* p = nullptr;
		~Stage() { if(p) { cudaFreeHost(p); } }
	};
	static thread_local Stage stage;
	if(!stage.p)
	{
		PG_CUDA_CHECK(cudaHostAlloc(&stage.p, kPinnedStage, cudaHostAllocPortable));
	}
	return static_cast<unsigned char*>(stage.p);
}

void check_same_device(int owner_device, int current, const char* what)
{
	if(current != owner_device)
	{
		throw Error(PG_ERR_INVALID_ARGUMENT, std::string(what) + " lives on device " + std::to_string(owner_device) +
		            " but device " + std::to_string(current) + " is current; make its device current first");
	}
}

void require_same_device(int owner_device, const char* what)
{
	check_same_device(owner_device, current_device(), what);
}

void check_render_end(uint32_t device_errors, bool done)
{
	if(device_errors & PG_DEV_ERR_STACK)
	{
		throw Error(PG_ERR_STACK_OVERFLOW, "render: BVH traversal stack overflow");
	}
	if(device_errors & PG_DEV_ERR_QUEUE)
	{
		throw Error(PG_ERR_QUEUE_OVERFLOW, "render: the queues ran empty before all paths finished");
	}
	if(!done)
	{
		throw Error(PG_ERR_ITERATION_LIMIT, "render: iteration limit reached before all paths finished");
	}
}

void allow_shared_memory(const void* kernel, int bytes)
{
	static std::mutex mutex;
	static std::set<std::pair<const void*, int>> allowed;
	const auto key = std::make_pair(kernel, current_device());
	std::lock_guard<std::mutex> lock(mutex);
	if(allowed.count(key) == 0)
	{
		PG_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
		allowed.insert(key);
	}
}

int sm_count()
{
	int dev = 0;
	PG_CUDA_CHECK(cudaGetDevice(&dev));
	int n = 0;
	PG_CUDA_CHECK(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
	return n;
}

}// end namespace pg
