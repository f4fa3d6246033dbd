// step_io.cuh — the first and the last kernel of a step whose inputs and logits lie in pinned host memory, for calls that wait for it.  A copy's node in the graph, and the
// change from it to a kernel and back, take longer than a kernel more (the engine's copies of 16 bytes and 128 KB: about 4 and 10 us of a step, these two 2 and 4).
#pragma once
#include "common.cuh"

namespace xalm {

// a token's parameters, before the kernels that read them ahead of their dependency waits
static __global__ void step_in_kernel(const int* in, int* out) { out[threadIdx.x] = in[threadIdx.x]; }
static __global__ void logits_out_kernel(const float* logits, float* host, int n) { // four logits a thread
	pdl_enter();
	const int i = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
	if (i + 4 <= n) *reinterpret_cast<float4*>(host + i) = __ldcg(reinterpret_cast<const float4*>(logits + i));
	else
		for (int k = i; k < n; k++) host[k] = __ldcg(logits + k);
}

} // namespace xalm
