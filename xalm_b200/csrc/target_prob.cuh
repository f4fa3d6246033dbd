// target_prob.cuh — Sampler::sample_prob (sampler.cpp:18-33) for many rows of logits: softmax(row)[target], a CTA per row.
//
// Bound: one read of the rows.  Every thread keeps a running maximum and the sum of exp(v - maximum) over its share, 16 values at a time (four
// 16-byte loads in flight), so that a row is read once; the threads' pairs are joined at the end.  (A pass for the maximum and a pass for the sum
// with one 4-byte load in flight per thread took 499 us for 4096 rows of 32000; 1024 rows take 30 us here.)
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "common.cuh"

namespace xalm {

constexpr int TARGET_PROB_THREADS = 512;

// seed: where the maximum starts (FLT_MIN in the reference's sampler, -infinity for a plain softmax)
static __global__ void __launch_bounds__(TARGET_PROB_THREADS) target_prob_kernel(const float* __restrict__ logits, int vocab, float seed,
                                                                                const int* __restrict__ targets, float* __restrict__ probs) {
	__shared__ float red_m[32], red_s[32];
	const float* l = logits + (size_t) blockIdx.x * vocab;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
	float m = seed, s = 0.f;
	// While m is -infinity no value above it has been met: such values count 0, a NaN stays a NaN
	auto add = [&](const float* v, int n) {
		float top = m;
		for (int i = 0; i < n; i++) top = fmaxf(top, v[i]);
		if (top > m) {
			if (m != -INFINITY) s *= expf(m - top);
			m = top;
		}
		const float at = m == -INFINITY ? 0.f : m;
		for (int i = 0; i < n; i++) s += expf(v[i] - at);
	};
	int done = 0;
	if ((vocab & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0) {
		const int n4 = vocab >> 2;
		const float4* l4 = reinterpret_cast<const float4*>(l);
		int i = threadIdx.x;
		for (; i + 3 * TARGET_PROB_THREADS < n4; i += 4 * TARGET_PROB_THREADS) {
			float v[16];
#pragma unroll
			for (int u = 0; u < 4; u++) {
				const float4 t = l4[i + u * TARGET_PROB_THREADS];
				v[4 * u] = t.x; v[4 * u + 1] = t.y; v[4 * u + 2] = t.z; v[4 * u + 3] = t.w;
			}
			add(v, 16);
		}
		for (; i < n4; i += TARGET_PROB_THREADS) {
			const float4 t = l4[i];
			const float v[4] = {t.x, t.y, t.z, t.w};
			add(v, 4);
		}
		done = vocab;
	}
	for (int i = done + threadIdx.x; i < vocab; i += TARGET_PROB_THREADS) {
		const float v = l[i];
		add(&v, 1);
	}
	auto weight = [](float mine, float all) { return mine == -INFINITY ? 1.f : expf(mine - all); };
	float top = warp_max(m);
	s = warp_sum(s * weight(m, top));
	if (lane == 0) { red_m[warp] = top; red_s[warp] = s; }
	__syncthreads();
	if (threadIdx.x == 0) {
		float tot = 0.f;
		top = red_m[0];
		for (int i = 1; i < nw; i++) top = fmaxf(top, red_m[i]);
		for (int i = 0; i < nw; i++) tot += red_s[i] * weight(red_m[i], top);
		probs[blockIdx.x] = expf(l[targets[blockIdx.x]] - (top == -INFINITY ? 0.f : top)) / tot;
	}
}

} // namespace xalm
