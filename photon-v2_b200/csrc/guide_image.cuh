// The guiding network's weight image: BF16 W^T of every layer in the K-major core-matrix layout of the
// MMA operands, and the FP32 biases; what the forward kernel copies into shared memory.
#pragma once

#include "guide.cuh"
#include "tcgen05.cuh"

namespace pg
{
namespace guide
{

constexpr int kW0Bytes = kHidden * kIn * 2;         // 28,672
constexpr int kWhBytes = kHidden * kHidden * 2;     //  8,192
constexpr int kW4Bytes = kOutPad * kHidden * 2;     //  6,144
constexpr int kOffImgW0 = 0;
constexpr int kOffImgW1 = kOffImgW0 + kW0Bytes;
constexpr int kOffImgW2 = kOffImgW1 + kWhBytes;
constexpr int kOffImgW3 = kOffImgW2 + kWhBytes;
constexpr int kOffImgW4 = kOffImgW3 + kWhBytes;
constexpr int kOffImgBias = kOffImgW4 + kW4Bytes;   // FP32 biases: 4 x 64 + 48
constexpr int kBiasCount = kHiddenLayers * kHidden + kOutPad;
constexpr int kImageBytes = kOffImgBias + kBiasCount * 4;   // 60,576


#ifdef __CUDACC__

// Writes parameter i of the packed FP32 order (guide.cuh) to its place in the image.
__device__ __forceinline__ void store_image(unsigned char* image, uint32_t i, float w)
{
	auto weight = [&](int img, int off, uint32_t outs, uint32_t rows)
	{
		const uint32_t e = i - static_cast<uint32_t>(off);
		*reinterpret_cast<__nv_bfloat16*>(image + img + tc::core_offset(e % outs, e / outs, rows)) = __float2bfloat16_rn(w);
	};
	auto bias = [&](int layer, int off)
	{
		reinterpret_cast<float*>(image + kOffImgBias)[layer * kHidden + static_cast<int>(i) - off] = w;
	};
	if(i < kOffB0) { weight(kOffImgW0, kOffW0, kHidden, kHidden); }
	else if(i < kOffW1) { bias(0, kOffB0); }
	else if(i < kOffB1) { weight(kOffImgW1, kOffW1, kHidden, kHidden); }
	else if(i < kOffW2) { bias(1, kOffB1); }
	else if(i < kOffB2) { weight(kOffImgW2, kOffW2, kHidden, kHidden); }
	else if(i < kOffW3) { bias(2, kOffB2); }
	else if(i < kOffB3) { weight(kOffImgW3, kOffW3, kHidden, kHidden); }
	else if(i < kOffW4) { bias(3, kOffB3); }
	else if(i < kOffB4) { weight(kOffImgW4, kOffW4, kOut, kOutPad); }
	else { bias(4, kOffB4); }
}

#endif

}// end namespace guide
}// end namespace pg
