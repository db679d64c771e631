// A training step whose network kernels reported an error: the sums of a failed CTA are missing from
// the workspace (here: NaN), so neither the plain gradient nor Adam may take them up.
#include "guide_image.cuh"
#include "guide_mlp.h"
#include "pg_runtime.h"

#include <cstdio>
#include <cstring>
#include <limits>
#include <vector>

using namespace pg;

namespace
{

template<typename T>
std::vector<T> host(const DeviceBuffer<T>& d, cudaStream_t s)
{
	std::vector<T> h(d.size());
	PG_CUDA_CHECK(cudaMemcpyAsync(h.data(), d.get(), d.bytes(), cudaMemcpyDeviceToHost, s));
	PG_CUDA_CHECK(cudaStreamSynchronize(s));
	return h;
}

template<typename T>
bool same(const std::vector<T>& a, const std::vector<T>& b)
{
	return std::memcmp(a.data(), b.data(), a.size() * sizeof(T)) == 0;
}

template<typename T>
void fill(const DeviceBuffer<T>& d, T value, cudaStream_t s)
{
	const std::vector<T> h(d.size(), value);
	PG_CUDA_CHECK(cudaMemcpyAsync(d.get(), h.data(), d.bytes(), cudaMemcpyHostToDevice, s));
	PG_CUDA_CHECK(cudaStreamSynchronize(s));
}

int check(uint32_t error_word, bool changes)
{
	constexpr uint32_t n = 128;
	cudaStream_t s = library_stream();
	DeviceBuffer<float> params(guide::kNumParams), m(guide::kNumParams), v(guide::kNumParams), partials(guide::partial_floats(n));
	DeviceBuffer<unsigned char> image(guide::image_bytes());
	DeviceBuffer<uint32_t> step(1), error(1);
	fill(params, 0.25f, s);
	fill(m, 0.0f, s);
	fill(v, 0.0f, s);
	fill(step, 3u, s);
	fill(error, error_word, s);
	fill(partials, changes ? 0.5f : std::numeric_limits<float>::quiet_NaN(), s);
	guide::pack_image(params.get(), image.get(), s);
	const auto p0 = host(params, s), m0 = host(m, s), v0 = host(v, s);
	const auto i0 = host(image, s);
	const auto s0 = host(step, s);
	guide::launch_adam(params.get(), partials.get(), n, nullptr, m.get(), v.get(), step.get(), image.get(), 1e-2f, error.get(), s);
	const bool kept = same(p0, host(params, s)) && same(m0, host(m, s)) && same(v0, host(v, s)) && same(i0, host(image, s)) &&
	                  same(s0, host(step, s));
	if(kept == changes)
	{
		std::printf("Adam with error word %u: state %s\n", error_word, kept ? "kept" : "changed");
		return 1;
	}
	// a plain gradient of n samples: added to what is there, unless the batch failed
	DeviceBuffer<float> feat(n * 8), raw(n * guide::kOut), grads(guide::kNumParams), scalars(2);
	DeviceBuffer<float4> dirw(n);
	DeviceBuffer<__nv_bfloat16> acts(n * guide::kHiddenLayers * guide::kHidden);
	fill(feat, 0.5f, s);
	fill(dirw, make_float4(0.0f, 0.0f, 1.0f, 1.0f), s);
	fill(grads, 7.0f, s);
	fill(scalars, 0.0f, s);
	const auto g0 = host(grads, s);
	guide::launch_gradients(params.get(), image.get(), feat.get(), dirw.get(), n, raw.get(), acts.get(), partials.get(),
	                        grads.get(), scalars.get(), scalars.get() + 1, error.get(), s);
	if(same(g0, host(grads, s)) == changes)
	{
		std::printf("gradient with error word %u: %s\n", error_word, changes ? "not added" : "added");
		return 1;
	}
	return 0;
}

}// end anonymous namespace

int main()
{
	if(check(PG_DEV_ERR_GUIDE_WAIT, false) != 0 || check(0u, true) != 0)
	{
		return 1;
	}
	std::puts("ok");
	return 0;
}
