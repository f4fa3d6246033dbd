// quantize.cpp — host-side writers for the weight formats: fp32 rows -> on-disk bytes.
//
// Needed by the synthetic-checkpoint generator (the benchmark's are random-init models that must be produced
// where the reference's Python is not available) and by Tensor::convert_to on the C++ host side.
// Each quantiser reproduces quants.py *byte for byte* (tests/test_quantize.py checks that against
// fixtures generated by quants.py itself):
//   Q8_0  quants.py:444-456   d = max|x|/127, round half away from zero (np_roundf, :108-112)
//   Q4_0  quants.py:283-300   d = x[argmax|x|] / -8, trunc(float32(double(x)*double(1/d) + 8.5)), clip 0..15
//   Q4_1  quants.py:318-335   d = (max-min)/15, trunc((x-min)*(1/d) + 0.5) in fp32
//   Q5_0  quants.py:355-374   like Q4_0 with 16 / 16.5 / clip 31, fifth bits packed LSB-first into a u32
//   Q5_1  quants.py:398-417   like Q4_1 with 31
//   TQ1_0 quants.py:640-662   d = max|x|, ternary round, base-3 pack, (v*256 + 242) / 243
//   BF16  quants.py:265-274   round to nearest even, NaNs quieted (== types.h:327-335 f32_to_bf16)
//   F16   numpy astype(float16): IEEE round to nearest even
//   Q8    types.h:458-463     clamp(round(x*100), -128, 127)   (C++-only format)
// Also a counter-based normal generator so a 7B-parameter checkpoint can be produced in seconds on all cores,
// independent of the thread count.
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#ifdef _OPENMP
#include <omp.h>
#endif

#include "../../../include/xalm_cuda.h"

namespace {

inline uint16_t f32_to_f16_bits(float f) {
	_Float16 h = (_Float16) f;
	uint16_t b;
	memcpy(&b, &h, 2);
	return b;
}
inline void put_f16(uint8_t* p, float f) {
	const uint16_t b = f32_to_f16_bits(f);
	p[0] = (uint8_t) (b & 0xFF);
	p[1] = (uint8_t) (b >> 8);
}
inline float np_roundf(float n) { // quants.py:108-112
	const float a = fabsf(n);
	const float floored = floorf(a);
	const float b = floored + floorf(2 * (a - floored));
	return n > 0 ? b : (n < 0 ? -b : 0.0f * n);
}
inline float inv_or_zero(float d) { return d == 0 ? 0.f : 1.0f / d; }

void q8_0_block(const float* x, uint8_t* o) {
	float amax = 0.f;
	for (int j = 0; j < 32; j++) amax = std::max(amax, fabsf(x[j]));
	const float d = amax / 127;
	const float id = inv_or_zero(d);
	put_f16(o, d);
	for (int j = 0; j < 32; j++) o[2 + j] = (uint8_t) (int8_t) np_roundf(x[j] * id);
}

// first index of the largest |x| (numpy argmax semantics)
inline float signed_absmax(const float* x) {
	int im = 0;
	float am = fabsf(x[0]);
	for (int j = 1; j < 32; j++)
		if (fabsf(x[j]) > am) { am = fabsf(x[j]); im = j; }
	return x[im];
}
inline uint8_t q_trunc_f64(float x, float id, double off, int hi) {
	const float v = (float) ((double) x * (double) id + off); // computed in double, cast to fp32, then truncated
	int q = (int) (uint8_t) truncf(v);
	return (uint8_t) std::min(q, hi);
}

void q4_0_block(const float* x, uint8_t* o) {
	const float d = signed_absmax(x) / -8;
	const float id = inv_or_zero(d);
	uint8_t q[32];
	for (int j = 0; j < 32; j++) q[j] = q_trunc_f64(x[j], id, 8.5, 15);
	put_f16(o, d);
	for (int j = 0; j < 16; j++) o[2 + j] = (uint8_t) (q[j] | (q[j + 16] << 4));
}

void q5_0_block(const float* x, uint8_t* o) {
	const float d = signed_absmax(x) / -16;
	const float id = inv_or_zero(d);
	uint8_t q[32];
	for (int j = 0; j < 32; j++) q[j] = q_trunc_f64(x[j], id, 16.5, 31);
	uint32_t qh = 0;
	for (int j = 0; j < 32; j++) qh |= (uint32_t) (q[j] >> 4) << j;
	put_f16(o, d);
	memcpy(o + 2, &qh, 4);
	for (int j = 0; j < 16; j++) o[6 + j] = (uint8_t) ((q[j] & 0x0F) | (q[j + 16] << 4));
}

inline void minmax32(const float* x, float* mn, float* mx) {
	*mn = *mx = x[0];
	for (int j = 1; j < 32; j++) { *mn = std::min(*mn, x[j]); *mx = std::max(*mx, x[j]); }
}
inline uint8_t q_trunc_f32(float x, float mn, float id, int hi) {
	volatile float t = (x - mn) * id; // two separately rounded fp32 ops, as numpy evaluates it
	const float v = t + 0.5f;
	int q = (int) (uint8_t) truncf(v);
	return (uint8_t) std::min(q, hi);
}

void q4_1_block(const float* x, uint8_t* o) {
	float mn, mx;
	minmax32(x, &mn, &mx);
	const float d = (mx - mn) / 15;
	const float id = inv_or_zero(d);
	uint8_t q[32];
	for (int j = 0; j < 32; j++) q[j] = q_trunc_f32(x[j], mn, id, 15);
	put_f16(o, d);
	put_f16(o + 2, mn);
	for (int j = 0; j < 16; j++) o[4 + j] = (uint8_t) (q[j] | (q[j + 16] << 4));
}

void q5_1_block(const float* x, uint8_t* o) {
	float mn, mx;
	minmax32(x, &mn, &mx);
	const float d = (mx - mn) / 31;
	const float id = inv_or_zero(d);
	uint8_t q[32];
	for (int j = 0; j < 32; j++) q[j] = q_trunc_f32(x[j], mn, id, 31);
	uint32_t qh = 0;
	for (int j = 0; j < 32; j++) qh |= (uint32_t) (q[j] >> 4) << j;
	put_f16(o, d);
	put_f16(o + 2, mn);
	memcpy(o + 4, &qh, 4);
	for (int j = 0; j < 16; j++) o[8 + j] = (uint8_t) ((q[j] & 0x0F) | (q[j + 16] << 4));
}

void tq1_0_block(const float* x, uint8_t* o) {
	float d = 0.f;
	for (int j = 0; j < 256; j++) d = std::max(d, fabsf(x[j]));
	const float id = inv_or_zero(d);
	uint8_t t[256];
	for (int j = 0; j < 256; j++) t[j] = (uint8_t) ((int8_t) np_roundf(x[j] * id) + 1);
	static const int w5[5] = {81, 27, 9, 3, 1};
	uint8_t packed[52];
	for (int B = 0; B < 32; B++) {
		int v = 0;
		for (int k = 0; k < 5; k++) v += t[k * 32 + B] * w5[k];
		packed[B] = (uint8_t) v;
	}
	for (int B = 0; B < 16; B++) {
		int v = 0;
		for (int k = 0; k < 5; k++) v += t[160 + k * 16 + B] * w5[k];
		packed[32 + B] = (uint8_t) v;
	}
	for (int B = 0; B < 4; B++) {
		int v = 0;
		for (int k = 0; k < 4; k++) v += t[240 + k * 4 + B] * w5[k];
		packed[48 + B] = (uint8_t) v;
	}
	for (int B = 0; B < 52; B++) o[B] = (uint8_t) (((int) packed[B] * 256 + 242) / 243);
	put_f16(o + 52, d);
}

inline uint16_t f32_to_bf16_bits(float s) { // types.h:327-335 / quants.py:265-274
	uint32_t i;
	memcpy(&i, &s, 4);
	if ((i & 0x7fffffff) > 0x7f800000) return (uint16_t) ((i >> 16) | 64);
	return (uint16_t) ((i + (0x7fff + ((i >> 16) & 1))) >> 16);
}

// splitmix64 finaliser: a stateless hash of (seed, stream, index)
inline uint64_t mix64(uint64_t z) {
	z += 0x9E3779B97F4A7C15ull;
	z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
	z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
	return z ^ (z >> 31);
}

} // namespace

extern "C" {

// torchrun exports OMP_NUM_THREADS=1 before any code runs; let the host side ask for its share of the cores explicitly.
void xalm_host_set_threads(int n) {
#ifdef _OPENMP
	if (n > 0) omp_set_num_threads(n);
#else
	(void) n;
#endif
}

// n_rows x n_cols fp32 (row-major) -> on-disk bytes of `type_id`.  Returns 0, or 1 for an unsupported type /
// a row length that is not a multiple of the block size.
int xalm_host_quantize(int type_id, const float* src, long long n_rows, long long n_cols, uint8_t* dst) {
	int bs = 1, ts = 0;
	switch (type_id) {
		case XALM_F32: ts = 4; break;
		case XALM_F16: case XALM_BF16: ts = 2; break;
		case XALM_Q8: ts = 1; break;
		case XALM_Q8_0: bs = 32; ts = 34; break;
		case XALM_Q4_0: bs = 32; ts = 18; break;
		case XALM_Q4_1: bs = 32; ts = 20; break;
		case XALM_Q5_0: bs = 32; ts = 22; break;
		case XALM_Q5_1: bs = 32; ts = 24; break;
		case XALM_TQ1_0: bs = 256; ts = 54; break;
		default: return 1;
	}
	if (n_cols % bs) return 1;
	const long long nb = n_rows * n_cols / bs;
#pragma omp parallel for schedule(static)
	for (long long b = 0; b < nb; b++) {
		const float* x = src + b * bs;
		uint8_t* o = dst + b * ts;
		switch (type_id) {
			case XALM_F32: memcpy(o, x, 4); break;
			case XALM_F16: put_f16(o, *x); break;
			case XALM_BF16: { const uint16_t h = f32_to_bf16_bits(*x); o[0] = (uint8_t) (h & 0xFF); o[1] = (uint8_t) (h >> 8); break; }
			case XALM_Q8: { // types.h:458-463
				float v = roundf(*x * 100.f);
				v = std::min(127.f, std::max(-128.f, v));
				*o = (uint8_t) (int8_t) v;
				break;
			}
			case XALM_Q8_0: q8_0_block(x, o); break;
			case XALM_Q4_0: q4_0_block(x, o); break;
			case XALM_Q4_1: q4_1_block(x, o); break;
			case XALM_Q5_0: q5_0_block(x, o); break;
			case XALM_Q5_1: q5_1_block(x, o); break;
			case XALM_TQ1_0: tq1_0_block(x, o); break;
		}
	}
	return 0;
}

// out[i] = mean + std * z_i,  z ~ N(0,1) from a counter-based generator keyed by (seed, stream): element i depends on
// nothing but (seed, stream, i), so the result is the same for any thread count and any chunking.
void xalm_host_normal(uint64_t seed, uint64_t stream, long long n, float mean, float std, float* out) {
	const uint64_t key = mix64(seed * 0x100000001B3ull ^ mix64(stream));
	const long long pairs = (n + 1) / 2;
#pragma omp parallel for schedule(static)
	for (long long p = 0; p < pairs; p++) {
		const uint64_t h = mix64(key + (uint64_t) p);
		const float u1 = ((float) (uint32_t) (h >> 40) + 1.0f) * (1.0f / 16777216.0f); // (0,1]
		const float u2 = (float) (uint32_t) ((h >> 8) & 0xFFFFFF) * (1.0f / 16777216.0f); // [0,1)
		const float r = sqrtf(-2.0f * logf(u1));
		float sn, cs;
		sincosf(6.28318530717958647692f * u2, &sn, &cs);
		out[2 * p] = mean + std * r * cs;
		if (2 * p + 1 < n) out[2 * p + 1] = mean + std * r * sn;
	}
}

// The same stream restricted to rows [r0, r1) x columns [c0, c1) of an (n_rows x n_cols) row-major matrix, written densely:
// out[(r - r0) * (c1 - c0) + (c - c0)] = element r * n_cols + c of xalm_host_normal(seed, stream, n_rows * n_cols, ...).
// A tensor-parallel rank generates only the shard it keeps (n_cols, c0 and c1 must be even: elements come in Box-Muller pairs).
int xalm_host_normal_block(uint64_t seed, uint64_t stream, long long n_cols, long long r0, long long r1, long long c0, long long c1, float mean,
                           float std, float* out) {
	if ((n_cols | c0 | c1) & 1) return 1;
	const uint64_t key = mix64(seed * 0x100000001B3ull ^ mix64(stream));
	const long long w = c1 - c0, pw = w / 2;
#pragma omp parallel for schedule(static)
	for (long long r = r0; r < r1; r++) {
		float* o = out + (r - r0) * w;
		const long long p0 = (r * n_cols + c0) / 2;
		for (long long p = 0; p < pw; p++) {
			const uint64_t h = mix64(key + (uint64_t) (p0 + p));
			const float u1 = ((float) (uint32_t) (h >> 40) + 1.0f) * (1.0f / 16777216.0f);
			const float u2 = (float) (uint32_t) ((h >> 8) & 0xFFFFFF) * (1.0f / 16777216.0f);
			const float rr = sqrtf(-2.0f * logf(u1));
			float sn, cs;
			sincosf(6.28318530717958647692f * u2, &sn, &cs);
			o[2 * p] = mean + std * rr * cs;
			o[2 * p + 1] = mean + std * rr * sn;
		}
	}
	return 0;
}

} // extern "C"
