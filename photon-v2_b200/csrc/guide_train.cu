// Guiding network training: loss gradient, backward pass and Adam.
//
// A training batch is n samples (features, sampled direction, weight). The forward pass runs on
// the tensor cores (guide_mlp.cu) and keeps the BF16 hidden activations; this file computes
//   loss = -sum_i w_i log q(d_i | x_i) / sum_i w_i
// (the KL divergence to the target density up to a constant, Mueller et al. 2019) and its gradient
// with respect to every parameter, then applies Adam to the FP32 master parameters.
//
// FP32 backward pass (the cross-check of the tensor-core one below): one block of 128 threads per 128
// samples, thread = sample. Each thread turns its raw outputs into d loss / d raw (the analytic derivative of the vMF mixture's log density) and
// back-propagates through the layers with the same BF16-rounded weights the forward pass used.
// Per layer, the block stages the layer inputs and pre-activation gradients of its 128 samples in
// shared memory and reduces the weight gradient sum_t x[t][i] dz[t][o] over them (FP32), adding
// the block's partial to the global gradient with one atomic per weight.
#include "guide_image.cuh"
#include "guide_mlp.h"

#include "pg_runtime.h"
#include "tcgen05.cuh"
#include "../../include/photon_gpu.h"

#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <vector>

namespace pg
{
namespace guide
{

namespace
{

constexpr int kBlock = 128;
constexpr int kPitch = kHidden + 1;   // shared-memory row pitch (floats), avoids bank conflicts

__device__ __forceinline__ float bf16r(float x)
{
	return __bfloat162float(__float2bfloat16_rn(x));
}

__global__ void weight_sum_kernel(const float4* __restrict__ dirw, uint32_t n_max, const uint32_t* __restrict__ d_n,
                                  float* __restrict__ total)
{
	const uint32_t n = d_n ? min(*d_n, n_max) : n_max;
	float s = 0.0f;
	for(uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		s += dirw[i].w;
	}
	for(int o = 16; o > 0; o >>= 1)
	{
		s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
	}
	if((threadIdx.x & 31) == 0)
	{
		atomicAdd(total, s);
	}
}

// Caps every sample weight at factor x the batch's mean weight (the sum in *total), in place.
__global__ void clamp_weights_kernel(float4* __restrict__ dirw, uint32_t n_max, const uint32_t* __restrict__ d_n,
                                     const float* __restrict__ total, float factor)
{
	const uint32_t n = d_n ? min(*d_n, n_max) : n_max;
	if(n == 0u)
	{
		return;
	}
	const float cap = factor * *total / static_cast<float>(n);
	for(uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
	{
		dirw[i].w = fminf(dirw[i].w, cap);
	}
}

// d loss / d raw for one sample (40 values) and its loss term.
__device__ void output_gradient(const float* raw, V3 d, float scale, float* g, float* loss_term)
{
	Mixture m = decode(raw);
	float v[kLobes];
	float q = 0.0f;
	#pragma unroll
	for(int j = 0; j < kLobes; ++j)
	{
		v[j] = vmf_pdf(m.mu[j], m.kappa[j], d);
		q += m.w[j] * v[j];
	}
	q = fmaxf(q, 1e-30f);
	*loss_term = scale * logf(q);   // scale = -w / total
	#pragma unroll
	for(int j = 0; j < kLobes; ++j)
	{
		const float r = m.w[j] * v[j] / q;
		const float k = m.kappa[j];
		const float cosv = dot(m.mu[j], d);
		g[5 * j + 0] = scale * (r - m.w[j]);
		const float e = expf(-2.0f * k);
		const float dlogv_dk = 1.0f / k - 2.0f * e / (1.0f - e) + (cosv - 1.0f);
		const float k_raw = expf(raw[5 * j + 4]);
		const bool inside = k_raw > kMinKappa && k_raw < kMaxKappa;
		g[5 * j + 4] = inside ? scale * r * dlogv_dk * k : 0.0f;
		const V3 mraw = v3(raw[5 * j + 1], raw[5 * j + 2], raw[5 * j + 3]);
		const float norm = fmaxf(sqrtf(dot(mraw, mraw)), 1e-30f);
		const float c = scale * r * k / norm;
		g[5 * j + 1] = c * (d.x - cosv * m.mu[j].x);
		g[5 * j + 2] = c * (d.y - cosv * m.mu[j].y);
		g[5 * j + 3] = c * (d.z - cosv * m.mu[j].z);
	}
}

// Adds sum_t x[t][i] * dz[t][o] over the block's samples to grad[i * out_dim + o] (i < in_rows).
__device__ void reduce_weight_grad(const float* sx, const float* sd, int in_rows, int out_dim, float* grad)
{
	for(int e = threadIdx.x; e < in_rows * out_dim; e += kBlock)
	{
		const int i = e / out_dim, o = e % out_dim;
		float acc = 0.0f;
		for(int t = 0; t < kBlock; ++t)
		{
			acc += sx[t * kPitch + i] * sd[t * kPitch + o];
		}
		if(acc != 0.0f)
		{
			atomicAdd(grad + e, acc);
		}
	}
}

__device__ void reduce_bias_grad(const float* sd, int out_dim, float* grad)
{
	for(int o = threadIdx.x; o < out_dim; o += kBlock)
	{
		float acc = 0.0f;
		for(int t = 0; t < kBlock; ++t)
		{
			acc += sd[t * kPitch + o];
		}
		if(acc != 0.0f)
		{
			atomicAdd(grad + o, acc);
		}
	}
}

__global__ void __launch_bounds__(kBlock)
backward_kernel(const float* __restrict__ params, const float* __restrict__ features,
                const float4* __restrict__ dirw, const float* __restrict__ raw_out,
                const __nv_bfloat16* __restrict__ acts, uint32_t n_max, const uint32_t* __restrict__ d_n,
                const float* __restrict__ total_weight, float* __restrict__ grads, float* __restrict__ loss)
{
	const uint32_t n = d_n ? min(*d_n, n_max) : n_max;
	if(blockIdx.x * kBlock >= n)
	{
		return;   // whole block past the live samples (uniform exit before any barrier)
	}
	extern __shared__ float smem_f[];   // sx, sd: [kBlock][kPitch] each (dynamic, 66 KB)
	float* sx = smem_f;
	float* sd = smem_f + kBlock * kPitch;
	__shared__ float sloss[kBlock / 32];
	const int tid = threadIdx.x;
	const uint32_t row = blockIdx.x * kBlock + tid;
	const bool valid = row < n;

	// ---- d loss / d out
	float g[kOut];
	float loss_term = 0.0f;
	if(valid)
	{
		float raw[kOut];
		#pragma unroll
		for(int i = 0; i < kOut; ++i)
		{
			raw[i] = raw_out[static_cast<size_t>(row) * kOut + i];
		}
		const float4 dw = dirw[row];
		const float scale = -dw.w / fmaxf(*total_weight, 1e-30f);
		output_gradient(raw, v3(dw.x, dw.y, dw.z), scale, g, &loss_term);
	}
	else
	{
		#pragma unroll
		for(int i = 0; i < kOut; ++i)
		{
			g[i] = 0.0f;
		}
	}
	for(int o = 16; o > 0; o >>= 1)
	{
		loss_term += __shfl_xor_sync(0xFFFFFFFFu, loss_term, o);
	}
	if((tid & 31) == 0)
	{
		sloss[tid >> 5] = loss_term;
	}

	// layer inputs x_l of this sample (x_1..x_4: BF16 activations of the forward pass)
	auto load_act = [&](int layer, float* x)
	{
		#pragma unroll
		for(int c = 0; c < kHidden; ++c)
		{
			x[c] = valid ? __bfloat162float(acts[(static_cast<size_t>(row) * kHiddenLayers + layer) * kHidden + c]) : 0.0f;
		}
	};

	// ---- output layer: dW4 = x4^T g, db4 = sum g, dx4 = W4 g
	float x[kHidden], dz[kHidden];
	load_act(3, x);
	#pragma unroll
	for(int c = 0; c < kHidden; ++c)
	{
		sx[tid * kPitch + c] = x[c];
		sd[tid * kPitch + c] = c < kOut ? g[c] : 0.0f;
	}
	__syncthreads();
	if(tid == 0)
	{
		float s = 0.0f;
		for(int w = 0; w < kBlock / 32; ++w)
		{
			s += sloss[w];
		}
		atomicAdd(loss, s);
	}
	reduce_weight_grad(sx, sd, kHidden, kOut, grads + kOffW4);
	reduce_bias_grad(sd, kOut, grads + kOffB4);
	#pragma unroll 4
	for(int i = 0; i < kHidden; ++i)
	{
		float acc = 0.0f;
		#pragma unroll
		for(int o = 0; o < kOut; ++o)
		{
			acc += bf16r(__ldg(params + kOffW4 + i * kOut + o)) * g[o];
		}
		dz[i] = x[i] > 0.0f ? acc : 0.0f;   // through the ReLU that produced x4
	}

	// ---- hidden layers 3, 2, 1, then the input layer 0
	const int w_off[4] = {kOffW0, kOffW1, kOffW2, kOffW3};
	const int b_off[4] = {kOffB0, kOffB1, kOffB2, kOffB3};
	for(int l = 3; l >= 1; --l)
	{
		load_act(l - 1, x);   // x_l, the input of layer l
		__syncthreads();      // previous reductions are done with sx / sd
		#pragma unroll
		for(int c = 0; c < kHidden; ++c)
		{
			sx[tid * kPitch + c] = x[c];
			sd[tid * kPitch + c] = dz[c];
		}
		__syncthreads();
		reduce_weight_grad(sx, sd, kHidden, kHidden, grads + w_off[l]);
		reduce_bias_grad(sd, kHidden, grads + b_off[l]);
		// dz of the layer below, reading this layer's dz back from shared memory
		const float* my_dz = sd + tid * kPitch;
		#pragma unroll 4
		for(int i = 0; i < kHidden; ++i)
		{
			float acc = 0.0f;
			#pragma unroll 8
			for(int o = 0; o < kHidden; ++o)
			{
				acc += bf16r(__ldg(params + w_off[l] + i * kHidden + o)) * my_dz[o];
			}
			dz[i] = x[i] > 0.0f ? acc : 0.0f;
		}
	}

	// input layer: x_0 is the one-blob encoding, recomputed in 64-column chunks
	__syncthreads();
	#pragma unroll
	for(int c = 0; c < kHidden; ++c)
	{
		sd[tid * kPitch + c] = dz[c];
	}
	float f[kInputs];
	#pragma unroll
	for(int i = 0; i < kInputs; ++i)
	{
		f[i] = valid ? features[static_cast<size_t>(row) * 8 + i] : 0.0f;
	}
	for(int chunk = 0; chunk * kHidden < kIn; ++chunk)
	{
		const int cols = min(kHidden, kIn - chunk * kHidden);
		__syncthreads();
		for(int c = 0; c < cols; ++c)
		{
			const int k = chunk * kHidden + c;
			sx[tid * kPitch + c] = valid ? bf16r(one_blob(f[k / kBins], k % kBins)) : 0.0f;
		}
		__syncthreads();
		reduce_weight_grad(sx, sd, cols, kHidden, grads + kOffW0 + chunk * kHidden * kHidden);
		if(chunk == 0)
		{
			reduce_bias_grad(sd, kHidden, grads + kOffB0);
		}
	}
}

// ---------------------------------------------------------------------------------------------
// Backward pass on the tensor cores (tcgen05, BF16 operands, FP32 accumulators in TMEM).
//
// Per 128-sample tile and layer l (4 down to 0), with G_l = d loss / d z_l [128 x out_l] and
// X_l the layer's input [128 x in_l]:
//   dW_l += X_l^T G_l      MMA M = 128 (the layer's inputs, padded; one extra row of ones gives
//                           the bias gradient sum_t G_l[t]), N = out_l, K = 128 samples;
//   dX_l  = G_l W_l^T      MMA M = 128 samples, N = in_l = 64, K = out_l (layers 4..1);
//   G_l-1 = dX_l where X_l > 0 (the ReLU that produced X_l).
// The weight gradients stay in tensor memory across all tiles a CTA processes; each CTA then writes
// its sums to a row of its own in `partials`, which the next kernel (Adam, or the reduction of a
// plain gradient) adds up. Operands: G_l as sample rows (K = out_l) for dX, and the transposed
// X_l^T / G_l^T (K = samples) for dW, written by each thread for its own sample; the transposed
// buffers' K-chunk stride carries 16 bytes of padding so that the 8 sample groups a warp writes
// land in different banks.
//
// A step of 16,384 samples is one tile per CTA, a serial chain of six rounds of staging, MMAs and
// read-back: what counts is the latency of each. Two threads share a sample (part 0: columns 0..31
// and lobes 0..3, part 1: the rest; thread t and t + 128 on sample t), the next layer's activations
// are loaded while a round's MMAs run, and the input layer's two halves go through one round. The
// CTAs' 3.8 M atomics on 29,480 addresses, four bytes each with every lane on a line of its own, had
// been part of the 145 us that the kernel took at one thread per sample. 32 steps of 16,384 samples through
// pgpu_guide_train went from 4.87 to 2.30 ms with this kernel and the fused Adam step, and to 2.36 ms with
// every bin of the input layer encoded by its own exponential.

namespace tcb
{

using namespace tc;

constexpr int kThreads = 256;
constexpr int kCols = kHidden / 2;                     // hidden columns per thread
constexpr uint32_t kLboG = kTile * 16u;                // G rows (samples) x K = outputs: 2048
constexpr uint32_t kLboXT = kTile * 16u + 16u;         // X^T: 128 rows x K = samples, padded: 2064
constexpr uint32_t kLboGT = kHidden * 16u + 16u;       // G^T: 64 rows x K = samples, padded: 1040
constexpr uint32_t kLboW = kHidden * 16u;              // W_l: 64 rows (inputs) x K = outputs: 1024

constexpr int kBwHidden = kHidden * kHidden * 2;       // 8,192
constexpr int kXtBytes = (kTile / 8) * static_cast<int>(kLboXT);          // 33,024
constexpr int kOffBw = 0;                              // W1, W2, W3, W4 (W4: K = 48)
constexpr int kOffG = kOffBw + 3 * kBwHidden + kHidden * kOutPad * 2;     // 30,720
constexpr int kOffXT = kOffG + kTile * kHidden * 2;                       // 47,104; two buffers
constexpr int kOffGT = kOffXT + 2 * kXtBytes;                             // 113,152
constexpr int kOffXch = kOffGT + (kTile / 8) * static_cast<int>(kLboGT);  // 129,792: [part][sample] float3
constexpr int kOffBar = kOffXch + 2 * kTile * 12;
constexpr int kOffSlot = kOffBar + 8;
// More than half an SM's shared memory: one CTA per SM, so that each CTA's 512 TMEM columns are free.
constexpr int kSmemBytes = kOffSlot + 8;
static_assert(kSmemBytes > 114 * 1024 && kSmemBytes <= 227 * 1024, "shared memory");
static_assert(kOffG % 16 == 0 && kOffXT % 16 == 0 && kOffGT % 16 == 0 && kOffXch % 16 == 0 && kOffBar % 8 == 0, "alignment");

// TMEM columns: the dX accumulator, then the weight gradients of every layer (rows = the layer's
// inputs, columns = its outputs).
constexpr uint32_t kColAcc = 0;
constexpr uint32_t kColW0a = 64;    // inputs 0..127 of layer 0
constexpr uint32_t kColW0b = 128;   // inputs 128..223 of layer 0, bias in row 96
// layer l >= 1: 192, 256, 320, 384 (bias in row 64)
PG_HD constexpr uint32_t col_w(int l) { return l == 0 ? kColW0a : 128u + 64u * static_cast<uint32_t>(l); }
constexpr uint32_t kTmemColsB = 512;

__device__ __forceinline__ void st_bf16(unsigned char* base, uint32_t off, float v)
{
	*reinterpret_cast<__nv_bfloat16*>(base + off) = __float2bfloat16_rn(v);
}

__device__ __forceinline__ uint4 pack8(const float* v)
{
	return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
}

// 8 floats to a 32-byte aligned address.
__device__ __forceinline__ void st_global8(float* p, const float* v)
{
	asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
	             :: "l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]) : "memory");
}

// d loss / d raw for this thread's four lobes of a sample (20 values) and, on part 0, the loss term.
// The two threads of a sample exchange the softmax's maximum and sum and the mixture density through
// xch. `valid` is the same for both.
__device__ __forceinline__ void output_gradient_half(const float* raw, V3 d, float scale, bool valid, uint32_t part,
                                                     float* mine, const float* other, float* g, float* loss_term)
{
	float mx = raw[0];
	#pragma unroll
	for(int j = 1; j < 4; ++j)
	{
		mx = fmaxf(mx, raw[5 * j]);
	}
	mine[0] = mx;
	__syncthreads();
	mx = fmaxf(mx, other[0]);
	float w[4], k[4], v[4], cosv[4], sum = 0.0f, q = 0.0f;
	V3 mu[4];
	#pragma unroll
	for(int j = 0; j < 4; ++j)
	{
		w[j] = expf(raw[5 * j] - mx);
		sum += w[j];
		const V3 m = v3(raw[5 * j + 1], raw[5 * j + 2], raw[5 * j + 3]);
		const float l2 = dot(m, m);
		mu[j] = l2 > 1e-20f ? m * (1.0f / sqrtf(l2)) : v3(0.0f, 0.0f, 1.0f);
		k[j] = fminf(fmaxf(expf(raw[5 * j + 4]), kMinKappa), kMaxKappa);
		v[j] = vmf_pdf(mu[j], k[j], d);
		cosv[j] = dot(mu[j], d);
		q += w[j] * v[j];
	}
	mine[1] = sum;
	mine[2] = q;
	__syncthreads();
	sum += other[1];
	q = fmaxf((q + other[2]) / sum, 1e-30f);
	*loss_term = part == 0u && valid ? scale * logf(q) : 0.0f;   // scale = -w / total
	#pragma unroll
	for(int j = 0; j < 4; ++j)
	{
		const float wj = w[j] / sum;
		const float r = wj * v[j] / q;
		const float e = expf(-2.0f * k[j]);
		const float dlogv_dk = 1.0f / k[j] - 2.0f * e / (1.0f - e) + (cosv[j] - 1.0f);
		const float k_raw = expf(raw[5 * j + 4]);
		const bool inside = k_raw > kMinKappa && k_raw < kMaxKappa;
		const V3 m = v3(raw[5 * j + 1], raw[5 * j + 2], raw[5 * j + 3]);
		const float c = scale * r * k[j] / fmaxf(sqrtf(dot(m, m)), 1e-30f);
		g[5 * j + 0] = valid ? scale * (r - wj) : 0.0f;
		g[5 * j + 1] = valid ? c * (d.x - cosv[j] * mu[j].x) : 0.0f;
		g[5 * j + 2] = valid ? c * (d.y - cosv[j] * mu[j].y) : 0.0f;
		g[5 * j + 3] = valid ? c * (d.z - cosv[j] * mu[j].z) : 0.0f;
		g[5 * j + 4] = valid && inside ? scale * r * dlogv_dk * k[j] : 0.0f;
	}
}

__global__ void __launch_bounds__(kThreads, 1)
backward_tc_kernel(const float* __restrict__ params, const float* __restrict__ features,
                   const float4* __restrict__ dirw, const float* __restrict__ raw_out,
                   const __nv_bfloat16* __restrict__ acts, uint32_t n_max, const uint32_t* __restrict__ d_n,
                   const float* __restrict__ total_weight, float* __restrict__ partials, float* __restrict__ loss,
                   uint32_t* __restrict__ error)
{
	const uint32_t n = d_n ? min(*d_n, n_max) : n_max;
	const uint32_t num_tiles = (n + kTile - 1) / kTile;
	if(blockIdx.x >= num_tiles)
	{
		return;   // uniform per CTA, before any barrier or tensor-memory use
	}
	extern __shared__ __align__(128) unsigned char smem[];
	const uint32_t tid = threadIdx.x;
	const uint32_t warp = tid >> 5;
	const uint32_t r = tid & (kTile - 1);   // the sample (row) this thread works on
	const uint32_t part = tid / kTile;      // which half of its columns / lobes
	const uint32_t c0 = part * kCols;

	// W_1..W_4 as B operands of dX: [64 rows = layer inputs][K = layer outputs], BF16 as the
	// forward pass rounds them, 8 outputs at a time
	for(uint32_t e = tid; e < 3u * kHidden * (kHidden / 8) + kHidden * (kOutPad / 8); e += kThreads)
	{
		const bool last = e >= 3u * kHidden * (kHidden / 8);
		const uint32_t f = last ? e - 3u * kHidden * (kHidden / 8) : e % (kHidden * (kHidden / 8));
		const uint32_t l = last ? 4u : 1u + e / (kHidden * (kHidden / 8));
		const uint32_t i = last ? f / (kOutPad / 8) : f / (kHidden / 8);
		const uint32_t o = (last ? f % (kOutPad / 8) : f % (kHidden / 8)) * 8u;
		const int w_off[5] = {kOffW0, kOffW1, kOffW2, kOffW3, kOffW4};
		float w[8] = {};
		if(!last || o < static_cast<uint32_t>(kOut))
		{
			const float4* src = reinterpret_cast<const float4*>(params + w_off[l] + i * (last ? kOut : kHidden) + o);
			const float4 a = __ldg(src), b = __ldg(src + 1);
			w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
			w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
		}
		*reinterpret_cast<uint4*>(smem + kOffBw + (l - 1u) * kBwHidden + core_offset_lbo(i, o, kLboW)) = pack8(w);
	}
	const uint32_t bar = smem_u32(smem + kOffBar);
	uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffSlot);
	if(tid == 0)
	{
		mbar_init(bar, 1);
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if(warp == 0)
	{
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
		             :: "r"(smem_u32(tmem_slot)), "r"(kTmemColsB) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
	}
	fence_async_smem();
	fence_before_sync();
	__syncthreads();
	fence_after_sync();
	const uint32_t tmem = *tmem_slot;
	const uint32_t tmem_row = tmem + (((warp & 3u) * 32u) << 16);

	unsigned char* gbuf = smem + kOffG;
	unsigned char* xt = smem + kOffXT;
	unsigned char* gt = smem + kOffGT;
	float* xch = reinterpret_cast<float*>(smem + kOffXch);
	const uint32_t a_g = smem_u32(gbuf), a_gt = smem_u32(gt);

	uint32_t phase = 0;
	bool failed = false;
	// one dW chain: X^T buffer `x` and G^T into TMEM column col (thread 0)
	auto weight_chain = [&](const unsigned char* x, uint32_t col, uint32_t n_out, bool accumulate)
	{
		const uint32_t a_xt = smem_u32(x);
		const uint32_t idesc = instr_desc(kTile, n_out);
		for(uint32_t ks = 0; ks < kTile / 16u; ++ks)
		{
			mma_bf16(tmem + col, smem_desc(a_xt + ks * 2u * kLboXT, kLboXT, 128u),
			         smem_desc(a_gt + ks * 2u * kLboGT, kLboGT, 128u), idesc, (accumulate || ks > 0) ? 1u : 0u);
		}
	};
	// the staged operands -> the round's chains, committed and awaited: layers 4..1 dX (first, the next
	// round waits for it) and dW; layer 0 the dW of both halves of its inputs
	auto run = [&](int layer, uint32_t n_out, bool acc_w) -> bool
	{
		fence_async_smem();
		fence_before_sync();
		__syncthreads();
		if(tid == 0)
		{
			fence_after_sync();
			if(layer >= 1)
			{
				const uint32_t idesc_x = instr_desc(kTile, kHidden);
				const uint32_t w_base = smem_u32(smem + kOffBw + (layer - 1) * kBwHidden);
				for(uint32_t ks = 0; ks < n_out / 16u; ++ks)
				{
					mma_bf16(tmem + kColAcc, smem_desc(a_g + ks * 2u * kLboG, kLboG, 128u),
					         smem_desc(w_base + ks * 2u * kLboW, kLboW, 128u), idesc_x, ks > 0 ? 1u : 0u);
				}
				weight_chain(xt, col_w(layer), n_out, acc_w);
			}
			else
			{
				weight_chain(xt, kColW0a, kHidden, acc_w);
				weight_chain(xt + kXtBytes, kColW0b, kHidden, acc_w);
			}
			mma_commit(bar);
		}
		// one thread polls the barrier; the others wait at the block barrier, which issues no
		// instructions while the MMAs run
		const bool ok = tid == 0 ? mbar_wait(bar, phase) : true;
		if(__syncthreads_or(ok ? 0 : 1))
		{
			if(!ok)
			{
				mbar_wait(bar, phase);   // bounded: do not free TMEM under running MMAs
			}
			return false;
		}
		phase ^= 1u;
		fence_after_sync();
		return true;
	};

	bool first = true;
	for(uint32_t tile = blockIdx.x; tile < num_tiles && !failed; tile += gridDim.x, first = false)
	{
		const uint32_t row = tile * kTile + r;
		const bool valid = row < n;

		// this thread's columns of X_l (l = layer + 1: the activations of hidden layer `layer`)
		auto load_x = [&](int layer, uint4* q)
		{
			const uint4* src = reinterpret_cast<const uint4*>(acts + (static_cast<size_t>(row) * kHiddenLayers + layer) * kHidden + c0);
			#pragma unroll
			for(int c = 0; c < kCols / 8; ++c)
			{
				q[c] = valid ? __ldg(src + c) : make_uint4(0u, 0u, 0u, 0u);
			}
		};
		uint4 xq[kCols / 8];
		load_x(3, xq);
		float f7[kInputs];
		#pragma unroll
		for(int i = 0; i < kInputs; ++i)
		{
			f7[i] = valid ? __ldg(features + static_cast<size_t>(row) * 8 + i) : 0.0f;
		}

		// ---- d loss / d raw outputs: columns 20 part .. 20 part + 19 of 48 (the last 8 zero)
		float loss_term = 0.0f;
		{
			float raw[20], g[20];
			V3 d = v3(0.0f, 0.0f, 1.0f);
			float scale = 0.0f;
			#pragma unroll
			for(int c = 0; c < 5; ++c)
			{
				const float4 q = valid ? __ldg(reinterpret_cast<const float4*>(raw_out + static_cast<size_t>(row) * kOut + 20u * part) + c)
				                       : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
				raw[4 * c] = q.x; raw[4 * c + 1] = q.y; raw[4 * c + 2] = q.z; raw[4 * c + 3] = q.w;
			}
			if(valid)
			{
				const float4 dw = __ldg(dirw + row);
				d = v3(dw.x, dw.y, dw.z);
				scale = -dw.w / fmaxf(*total_weight, 1e-30f);
			}
			output_gradient_half(raw, d, scale, valid, part, xch + 3u * (part * kTile + r), xch + 3u * ((1u - part) * kTile + r),
			                     g, &loss_term);
			#pragma unroll
			for(int o = 0; o < 20; ++o)
			{
				st_bf16(gt, core_offset_lbo(20u * part + static_cast<uint32_t>(o), r, kLboGT), g[o]);
			}
			if(part == 1u)
			{
				#pragma unroll
				for(int o = kOut; o < kOutPad; ++o)
				{
					st_bf16(gt, core_offset_lbo(static_cast<uint32_t>(o), r, kLboGT), 0.0f);
				}
			}
			// the sample's row of G, 4 columns at a time (20 is not a multiple of 8)
			#pragma unroll
			for(int c = 0; c < 5; ++c)
			{
				*reinterpret_cast<uint2*>(gbuf + core_offset_lbo(r, 20u * part + 4u * c, kLboG)) =
					make_uint2(pack_bf16x2(g[4 * c], g[4 * c + 1]), pack_bf16x2(g[4 * c + 2], g[4 * c + 3]));
			}
			if(part == 1u)
			{
				*reinterpret_cast<uint4*>(gbuf + core_offset_lbo(r, kOut, kLboG)) = make_uint4(0u, 0u, 0u, 0u);
			}
		}
		for(int o = 16; o > 0; o >>= 1)
		{
			loss_term += __shfl_xor_sync(0xFFFFFFFFu, loss_term, o);
		}
		if((tid & 31u) == 0u && loss_term != 0.0f)
		{
			atomicAdd(loss, loss_term);
		}

		// ---- layers 4..1: dX_l and dW_l together
		for(int l = 4; l >= 1; --l)
		{
			const uint32_t n_out = l == 4 ? static_cast<uint32_t>(kOutPad) : static_cast<uint32_t>(kHidden);
			// X_l^T (+ the ones row); a BF16 activation is positive where its bits are neither 0 nor a sign
			uint32_t positive = 0u;
			#pragma unroll
			for(int c = 0; c < kCols / 8; ++c)
			{
				const uint32_t w4[4] = {xq[c].x, xq[c].y, xq[c].z, xq[c].w};
				#pragma unroll
				for(int j = 0; j < 8; ++j)
				{
					const uint16_t bits = static_cast<uint16_t>(w4[j / 2] >> (16 * (j & 1)));
					const int f = 8 * c + j;
					*reinterpret_cast<uint16_t*>(xt + core_offset_lbo(c0 + static_cast<uint32_t>(f), r, kLboXT)) = bits;
					positive |= (bits != 0u && bits < 0x8000u) ? 1u << f : 0u;
				}
			}
			if(part == 0u)
			{
				st_bf16(xt, core_offset_lbo(kHidden, r, kLboXT), 1.0f);
			}
			if(l > 1)
			{
				load_x(l - 2, xq);   // the next round's, in flight while this one's MMAs run
			}
			if(!run(l, n_out, !first))
			{
				failed = true;
				break;
			}
			// G_l-1 = dX_l through the ReLU that produced X_l, staged for the next round
			float g[kCols];
			tmem_ld16(tmem_row + kColAcc + c0, g);
			tmem_ld16(tmem_row + kColAcc + c0 + 16u, g + 16);
			tmem_wait_ld();
			#pragma unroll
			for(int c = 0; c < kCols; ++c)
			{
				g[c] = (positive >> c) & 1u ? g[c] : 0.0f;
				st_bf16(gt, core_offset_lbo(c0 + static_cast<uint32_t>(c), r, kLboGT), g[c]);
			}
			#pragma unroll
			for(int c = 0; c < kCols / 8; ++c)
			{
				*reinterpret_cast<uint4*>(gbuf + core_offset_lbo(r, c0 + 8u * c, kLboG)) = pack8(g + 8 * c);
			}
		}
		if(failed)
		{
			break;
		}

		// ---- layer 0: dW_0 of its 224 one-blob inputs, each bin by its own exponential (the forward pass's
		//      recurrence over a chunk of bins loses those of a chunk whose first one underflows); part 0
		//      inputs 0, 2, 4 and 6, part 1 the others (unrolled so that f7 stays in registers)
		#pragma unroll
		for(int i = 0; i < kInputs; ++i)
		{
			if((i & 1) == static_cast<int>(part))
			{
				#pragma unroll 8
				for(int b = 0; b < kBins; ++b)
				{
					const uint32_t k = static_cast<uint32_t>(i * kBins + b);
					st_bf16(i < 4 ? xt : xt + kXtBytes, core_offset_lbo(k & 127u, r, kLboXT), valid ? one_blob(f7[i], b) : 0.0f);
				}
			}
		}
		if(part == 1u)
		{
			st_bf16(xt + kXtBytes, core_offset_lbo(static_cast<uint32_t>(kIn - 128), r, kLboXT), 1.0f);
		}
		if(!run(0, kHidden, !first))
		{
			failed = true;
			break;
		}
	}

	if(!failed)
	{
		// ---- the CTA's weight gradients: thread t and t + 128 hold row t of each block, half of its
		//      columns each
		float* const out = partials + static_cast<size_t>(blockIdx.x) * kNumParams;
		auto flush = [&](uint32_t col, int w_off, int b_off, uint32_t rows, uint32_t bias_row, uint32_t first_input,
		                 uint32_t out_stride)
		{
			float v[kCols];
			tmem_ld16(tmem_row + col + c0, v);
			tmem_ld16(tmem_row + col + c0 + 16u, v + 16);
			tmem_wait_ld();
			float* const dst = r < rows ? out + w_off + (first_input + r) * out_stride : out + b_off;
			if(r < rows || r == bias_row)
			{
				#pragma unroll
				for(uint32_t c = 0; c < kCols; c += 8u)
				{
					if(c0 + c < out_stride)
					{
						st_global8(dst + c0 + c, v + c);
					}
				}
			}
		};
		flush(kColW0a, kOffW0, kOffB0, 128u, 0xFFFFFFFFu, 0u, kHidden);
		flush(kColW0b, kOffW0, kOffB0, static_cast<uint32_t>(kIn - 128), static_cast<uint32_t>(kIn - 128), 128u, kHidden);
		flush(col_w(1), kOffW1, kOffB1, kHidden, kHidden, 0u, kHidden);
		flush(col_w(2), kOffW2, kOffB2, kHidden, kHidden, 0u, kHidden);
		flush(col_w(3), kOffW3, kOffB3, kHidden, kHidden, 0u, kHidden);
		flush(col_w(4), kOffW4, kOffB4, kHidden, kHidden, 0u, kOut);
	}
	else if(tid == 0)
	{
		atomicOr(error, PG_DEV_ERR_GUIDE_WAIT);
	}
	fence_before_sync();
	__syncthreads();
	if(warp == 0)
	{
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(kTmemColsB) : "memory");
	}
}

}// end namespace tcb

// CTAs of the backward kernel that had a tile, each with a row of gradient sums in `partials`.
__device__ __forceinline__ uint32_t partial_rows(uint32_t n_max, const uint32_t* d_n, uint32_t grid)
{
	const uint32_t n = d_n ? min(*d_n, n_max) : n_max;
	return min((n + kTile - 1u) / kTile, grid);
}

// The gradient of parameter i: the CTAs' sums, in their order (eight loads in flight).
__device__ __forceinline__ float sum_partials(const float* __restrict__ partials, uint32_t rows, uint32_t i)
{
	float s = 0.0f;
	uint32_t b = 0;
	for(; b + 8u <= rows; b += 8u)
	{
		float v[8];
		#pragma unroll
		for(uint32_t k = 0; k < 8u; ++k)
		{
			v[k] = __ldg(partials + static_cast<size_t>(b + k) * kNumParams + i);
		}
		s += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
	}
	for(; b < rows; ++b)
	{
		s += __ldg(partials + static_cast<size_t>(b) * kNumParams + i);
	}
	return s;
}

// A CTA of the backward kernel that gave up waiting on its tensor cores left no row in `partials`: with
// the error word set, the rows are not summed and the state stays as it was before the step.

__global__ void reduce_partials_kernel(const float* __restrict__ partials, uint32_t n_max, const uint32_t* __restrict__ d_n,
                                       uint32_t grid, const uint32_t* __restrict__ error, float* __restrict__ grads)
{
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i < kNumParams && *error == 0u)
	{
		grads[i] += sum_partials(partials, partial_rows(n_max, d_n, grid), i);
	}
}

// Adds up the step's gradient, applies Adam and writes the new weight to the packed image the network
// kernels read, in one launch.
__global__ void adam_kernel(float* __restrict__ params, const float* __restrict__ partials, uint32_t n_max,
                            const uint32_t* __restrict__ d_n, uint32_t grid, float* __restrict__ m,
                            float* __restrict__ v, float lr, float beta1, float beta2, float eps,
                            const uint32_t* __restrict__ step, const uint32_t* __restrict__ error,
                            unsigned char* __restrict__ image)
{
	const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i >= kNumParams || *error != 0u)
	{
		return;
	}
	const float t = static_cast<float>(*step + 1u);
	const float bias1 = 1.0f - powf(beta1, t);
	const float bias2 = 1.0f - powf(beta2, t);
	const float g = sum_partials(partials, partial_rows(n_max, d_n, grid), i);
	const float mi = beta1 * m[i] + (1.0f - beta1) * g;
	const float vi = beta2 * v[i] + (1.0f - beta2) * g * g;
	m[i] = mi;
	v[i] = vi;
	const float w = params[i] - lr * (mi / bias1) / (sqrtf(vi / bias2) + eps);
	params[i] = w;
	store_image(image, i, w);
}

__global__ void step_kernel(uint32_t* step, const uint32_t* error)
{
	*step += *error == 0u ? 1u : 0u;
}

uint32_t backward_grid(uint32_t n)
{
	// one CTA per SM: a batch of up to one tile per SM runs in one round of tiles; larger batches keep
	// their weight gradients in TMEM across each CTA's tiles
	return std::max(1u, std::min((n + kTile - 1u) / kTile, static_cast<uint32_t>(sm_count())));
}

}// end anonymous namespace

std::size_t partial_floats(uint32_t n)
{
	return static_cast<std::size_t>(backward_grid(n)) * kNumParams;
}

void launch_gradients(const float* d_params, const unsigned char* d_image, const float* d_features,
                      const float4* d_dirw, uint32_t n, float* d_raw, __nv_bfloat16* d_acts, float* d_partials,
                      float* d_grads, float* d_loss, float* d_total, uint32_t* d_error, cudaStream_t s,
                      const uint32_t* d_n, float clamp_factor, bool tensor_cores)
{
	if(n == 0)
	{
		return;
	}
	PG_CUDA_CHECK(cudaMemsetAsync(d_total, 0, sizeof(float), s));
	weight_sum_kernel<<<64, 256, 0, s>>>(d_dirw, n, d_n, d_total);
	PG_CUDA_CHECK(cudaGetLastError());
	if(clamp_factor > 0.0f)
	{
		// rare, very bright samples would otherwise dominate single steps
		clamp_weights_kernel<<<64, 256, 0, s>>>(const_cast<float4*>(d_dirw), n, d_n, d_total, clamp_factor);
		PG_CUDA_CHECK(cudaMemsetAsync(d_total, 0, sizeof(float), s));
		weight_sum_kernel<<<64, 256, 0, s>>>(d_dirw, n, d_n, d_total);
		PG_CUDA_CHECK(cudaGetLastError());
	}
	launch_forward(d_image, d_features, n, d_raw, d_acts, d_error, s, d_n);
	if(tensor_cores)
	{
		allow_shared_memory(reinterpret_cast<const void*>(tcb::backward_tc_kernel), tcb::kSmemBytes);
		const uint32_t grid = backward_grid(n);
		tcb::backward_tc_kernel<<<grid, tcb::kThreads, tcb::kSmemBytes, s>>>(d_params, d_features, d_dirw, d_raw, d_acts,
		                                                                     n, d_n, d_total, d_partials, d_loss, d_error);
		PG_CUDA_CHECK(cudaGetLastError());
		if(d_grads)
		{
			reduce_partials_kernel<<<(kNumParams + 127) / 128, 128, 0, s>>>(d_partials, n, d_n, grid, d_error, d_grads);
			PG_CUDA_CHECK(cudaGetLastError());
		}
		return;
	}
	constexpr int smem_bytes = 2 * kBlock * kPitch * sizeof(float);
	allow_shared_memory(reinterpret_cast<const void*>(backward_kernel), smem_bytes);
	backward_kernel<<<(n + kBlock - 1) / kBlock, kBlock, smem_bytes, s>>>(d_params, d_features, d_dirw, d_raw, d_acts,
	                                                                     n, d_n, d_total, d_grads, d_loss);
	PG_CUDA_CHECK(cudaGetLastError());
}

void launch_adam(float* d_params, const float* d_partials, uint32_t n, const uint32_t* d_n, float* d_m, float* d_v,
                 uint32_t* d_step, unsigned char* d_image, float lr, const uint32_t* d_error, cudaStream_t s)
{
	adam_kernel<<<(kNumParams + 127) / 128, 128, 0, s>>>(d_params, d_partials, n, d_n, backward_grid(n), d_m, d_v, lr, 0.9f,
	                                                     0.999f, 1e-8f, d_step, d_error, d_image);
	PG_CUDA_CHECK(cudaGetLastError());
	step_kernel<<<1, 1, 0, s>>>(d_step, d_error);
	PG_CUDA_CHECK(cudaGetLastError());
}

}// end namespace guide
}// end namespace pg

using namespace pg;

extern "C" {

int pgpu_guide_gradients(const float* params, const float* features, const float* dirs, const float* weights,
                         uint64_t n, float* out_loss, float* out_grads)
{
	return pgpu_guide_gradients_ex(params, features, dirs, weights, n, 0u, out_loss, out_grads);
}

int pgpu_guide_gradients_ex(const float* params, const float* features, const float* dirs, const float* weights,
                            uint64_t n, uint32_t flags, float* out_loss, float* out_grads)
{
	return guarded([&]
	{
		if(!params || !out_grads || n == 0 || !features || !dirs || !weights)
		{
			throw Error(PG_ERR_INVALID_ARGUMENT, "pgpu_guide_gradients: empty batch or null pointer");
		}
		if(n > (1u << 24))
		{
			throw Error(PG_ERR_INVALID_ARGUMENT, "pgpu_guide_gradients: batch too large");
		}
		require_device();
		cudaStream_t s = library_stream();
		ScratchBuffer<float> d_params(guide::kNumParams), d_grads(guide::kNumParams);
		ScratchBuffer<unsigned char> d_image(guide::image_bytes());
		ScratchBuffer<float> d_feat(n * 8), d_raw(n * guide::kOut), d_scalars(2);
		ScratchBuffer<float4> d_dirw(n);
		ScratchBuffer<float> d_partials(guide::partial_floats(static_cast<uint32_t>(n)));
		ScratchBuffer<__nv_bfloat16> d_acts(n * guide::kHiddenLayers * guide::kHidden);
		ScratchBuffer<uint32_t> d_err(1);
		PG_CUDA_CHECK(cudaMemsetAsync(d_err.get(), 0, sizeof(uint32_t), s));
		PG_CUDA_CHECK(cudaMemsetAsync(d_grads.get(), 0, d_grads.bytes(), s));
		PG_CUDA_CHECK(cudaMemsetAsync(d_scalars.get(), 0, d_scalars.bytes(), s));
		PG_CUDA_CHECK(cudaMemcpyAsync(d_params.get(), params, d_params.bytes(), cudaMemcpyHostToDevice, s));
		guide::upload_rows(features, dirs, weights, n, d_feat.get(), d_dirw.get(), s);
		guide::pack_image(d_params.get(), d_image.get(), s);
		guide::launch_gradients(d_params.get(), d_image.get(), d_feat.get(), d_dirw.get(), static_cast<uint32_t>(n),
		                        d_raw.get(), d_acts.get(), d_partials.get(), d_grads.get(), d_scalars.get(), d_scalars.get() + 1,
		                        d_err.get(), s, nullptr, 0.0f, (flags & PG_GUIDE_BACKWARD_CUDA_CORES) == 0u);
		float scalars[2] = {0.0f, 0.0f};
		uint32_t err = 0;
		PG_CUDA_CHECK(cudaMemcpyAsync(out_grads, d_grads.get(), d_grads.bytes(), cudaMemcpyDeviceToHost, s));
		PG_CUDA_CHECK(cudaMemcpyAsync(scalars, d_scalars.get(), sizeof(scalars), cudaMemcpyDeviceToHost, s));
		PG_CUDA_CHECK(cudaMemcpyAsync(&err, d_err.get(), sizeof(err), cudaMemcpyDeviceToHost, s));
		PG_CUDA_CHECK(cudaStreamSynchronize(s));
		if(err)
		{
			throw Error(PG_ERR_CUDA, "guiding network: tensor-core wait timed out");
		}
		if(out_loss) { *out_loss = scalars[0]; }
	});
}

int pgpu_guide_train(float* params, const float* features, const float* dirs, const float* weights,
                     uint64_t n, uint32_t steps, uint32_t batch, float lr, float* out_losses)
{
	return guarded([&]
	{
		if(!params || n == 0 || !features || !dirs || !weights || steps == 0 || batch == 0)
		{
			throw Error(PG_ERR_INVALID_ARGUMENT, "pgpu_guide_train: empty input");
		}
		if(n > (1u << 24))
		{
			throw Error(PG_ERR_INVALID_ARGUMENT, "pgpu_guide_train: data set too large");
		}
		require_device();
		cudaStream_t s = library_stream();
		const uint32_t b = static_cast<uint32_t>(std::min<uint64_t>(batch, n));
		ScratchBuffer<float> d_params(guide::kNumParams), d_partials(guide::partial_floats(b)), d_m(guide::kNumParams),
			d_v(guide::kNumParams);
		ScratchBuffer<unsigned char> d_image(guide::image_bytes());
		ScratchBuffer<float> d_feat(n * 8), d_raw(static_cast<std::size_t>(b) * guide::kOut), d_scalars(2 * static_cast<std::size_t>(steps));
		ScratchBuffer<float4> d_dirw(n);
		ScratchBuffer<__nv_bfloat16> d_acts(static_cast<size_t>(b) * guide::kHiddenLayers * guide::kHidden);
		ScratchBuffer<uint32_t> d_err(1), d_step(1);
		PG_CUDA_CHECK(cudaMemsetAsync(d_err.get(), 0, sizeof(uint32_t), s));
		PG_CUDA_CHECK(cudaMemsetAsync(d_step.get(), 0, sizeof(uint32_t), s));
		PG_CUDA_CHECK(cudaMemsetAsync(d_m.get(), 0, d_m.bytes(), s));
		PG_CUDA_CHECK(cudaMemsetAsync(d_v.get(), 0, d_v.bytes(), s));
		PG_CUDA_CHECK(cudaMemsetAsync(d_scalars.get(), 0, d_scalars.bytes(), s));
		PG_CUDA_CHECK(cudaMemcpyAsync(d_params.get(), params, d_params.bytes(), cudaMemcpyHostToDevice, s));
		guide::upload_rows(features, dirs, weights, n, d_feat.get(), d_dirw.get(), s);
		guide::pack_image(d_params.get(), d_image.get(), s);
		for(uint32_t step = 0; step < steps; ++step)
		{
			const uint32_t first = static_cast<uint32_t>((static_cast<uint64_t>(step) * b) % n);
			const uint32_t count = std::min<uint32_t>(b, static_cast<uint32_t>(n - first));
			guide::launch_gradients(d_params.get(), d_image.get(), d_feat.get() + static_cast<size_t>(first) * 8,
			                        d_dirw.get() + first, count, d_raw.get(), d_acts.get(), d_partials.get(), nullptr,
			                        d_scalars.get() + 2 * step, d_scalars.get() + 2 * step + 1, d_err.get(), s);
			guide::launch_adam(d_params.get(), d_partials.get(), count, nullptr, d_m.get(), d_v.get(), d_step.get(),
			                   d_image.get(), lr, d_err.get(), s);
		}
		std::vector<float> scalars(2 * static_cast<std::size_t>(steps));
		uint32_t err = 0;
		// (through the stage: the caller's parameters stay as they are if a step failed)
		static_assert(guide::kNumParams * sizeof(float) <= kPinnedStage, "page-locked stage");
		const unsigned char* const trained = pinned_stage();
		PG_CUDA_CHECK(cudaMemcpyAsync(pinned_stage(), d_params.get(), d_params.bytes(), cudaMemcpyDeviceToHost, s));
		PG_CUDA_CHECK(cudaMemcpyAsync(scalars.data(), d_scalars.get(), d_scalars.bytes(), cudaMemcpyDeviceToHost, s));
		PG_CUDA_CHECK(cudaMemcpyAsync(&err, d_err.get(), sizeof(err), cudaMemcpyDeviceToHost, s));
		PG_CUDA_CHECK(cudaStreamSynchronize(s));
		if(err)
		{
			throw Error(PG_ERR_CUDA, "guiding network: tensor-core wait timed out");
		}
		std::memcpy(params, trained, d_params.bytes());
		if(out_losses)
		{
			for(uint32_t i = 0; i < steps; ++i)
			{
				out_losses[i] = scalars[2 * i];
			}
		}
	});
}

}// extern "C"
