// swa_mma.cu — the attention of mix_ops.cuh (window, kept first positions, chunks, soft cap, distance biases, sink, gate; no mixing of heads) for passes
// of many tokens over a bf16 cache, on the tensor cores in fp32 grade.
//
// Queries and probabilities are fp32 values: each enters as three bf16 planes (hi + mid + lo = its 24 bits), keys and values as the bf16 the cache
// holds, so that every product is exact and only the fp32 sums round.  The tensor cores sum 16 products (of the small planes first) from zero; sums of more
// are added in round-to-nearest, since the tensor cores' own additions truncate: chained over a head's channels and a key block, the result was
// twice as far from float64 as the fp32 FMA kernel's.
// A CTA takes 16 queries of one head per warp and, where few CTAs would run (swa_mma_splits), a share of the keys, whose parts swa_merge_kernel joins;
// 64 keys and their values at a time come through a two-deep cp.async ring; queries stay in shared memory as planes, scores, probabilities and output in
// registers (m16n8k16 fragments).
// Bound: latency, one or two warps per scheduler (115 KB a CTA) going through chains of three products, adds, exponentials and splits: at 1024 tokens of 16
// heads over 1024 keys the mma.sync pipe is active 20 % and 26 % of the issue slots are used.  Against the fp32
// FMA tiles of mix_ops.cuh, caches flushed: 1024 tokens of 16 heads of 128 over up to 2048 keys 1978 -> 215 us, of 8 heads in a window of 512 268 -> 69 us;
// 256 tokens of 8 heads over up to 256 keys 93 -> 31 us (four splits).  Distance from float64 at 128 channels and 1500 keys: 2.6e-7, the FMA kernel 4.4e-7.
#define XALM_SECONDARY_TU
#include "common.cuh"
#include "family.h"
#include "mix_ops.cuh"

namespace xalm {
namespace mix {

constexpr int SMM_KEYS = SWA_MMA_KEYS, SMM_STAGES = 2;

__device__ __forceinline__ void smm_ldsm4(uint32_t (&r)[4], uint32_t addr) {
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void smm_ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void smm_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
	asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
	             : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
	             : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the three planes of A times two pairs of fragments of B (four tiles of 8 columns), small planes first; four sums at a time, so that a product does not wait
// for the one before it
__device__ __forceinline__ void smm_planes(float (&part)[4][4], const uint32_t (&a)[3][4], const uint32_t (&b)[2][4]) {
#pragma unroll
	for (int pl = 2; pl >= 0; pl--)
#pragma unroll
		for (int x = 0; x < 4; x++) smm_mma(part[x], a[pl], b[x >> 1][2 * (x & 1)], b[x >> 1][2 * (x & 1) + 1]);
}
// two fp32 values as three pairs of bf16 whose sums are the values
__device__ __forceinline__ void smm_split(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
	const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
	const float xr = x - __low2float(h), yr = y - __high2float(h);
	const __nv_bfloat162 m = __floats2bfloat162_rn(xr, yr);
	const __nv_bfloat162 l = __floats2bfloat162_rn(xr - __low2float(m), yr - __high2float(m));
	hi = *reinterpret_cast<const uint32_t*>(&h);
	mid = *reinterpret_cast<const uint32_t*>(&m);
	lo = *reinterpret_cast<const uint32_t*>(&l);
}
// rows of D bf16 in 16-byte pieces, piece p of row r at place p ^ (r % 8): the eight rows of a fragment's 8x8 matrix fall on different banks
template <int D>
__device__ __forceinline__ uint32_t smm_at(int row, int piece) {
	return (uint32_t) (row * (D * 2) + ((piece ^ (row & 7)) << 4));
}
__host__ __device__ constexpr size_t smm_smem(int dq, int dv, int warps) {
	return (size_t) 3 * 16 * warps * dq * 2 + (size_t) SMM_STAGES * SMM_KEYS * (dq + dv) * 2 + (size_t) SMM_STAGES * SMM_KEYS * 4;
}

__device__ __forceinline__ bool smm_seen(const SwaArgs& a, int i, int j) {
	return j <= i && (a.window >= 0x7fffffff || i - j < a.window || j < a.keep_first) && (a.mask_chunk <= 0 || j >= i - i % a.mask_chunk);
}
// scale, soft cap and distance biases of the raw score of positions i and j; slope, b1, b2: the head's
__device__ __forceinline__ float smm_score(const SwaArgs& a, float x, int i, int j, float slope, float b1, float b2) {
	x *= a.scale;
	if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
	const float dist = (float) max(i - j, 0);
	if (a.r1) x -= b1 * log1pf(b2 * dist);
	if (a.slope) x -= slope * dist;
	return x;
}
// row t's value of column col of head h, or split sp's part of it
__device__ __forceinline__ void smm_store(const SwaArgs& a, int t, int h, int sp, int col, float o, float l, float m) {
	if (a.n_splits > 1) { // swa_merge_kernel joins them
		a.part_o[((size_t) t * a.n_splits + sp) * (a.H * a.dv) + (size_t) h * a.dv + col] = o;
		if (col == 0) {
			float* pml = a.part_ml + ((size_t) t * a.n_splits + sp) * (a.H * 2) + 2 * h;
			pml[0] = m;
			pml[1] = l;
		}
		return;
	}
	float v = swa_finish(a, h, o, l, m);
	if (a.gate) v *= swa_gate(a, t, h, col);
	a.out[(size_t) t * (a.ldo ? a.ldo : a.H * a.dv) + (size_t) h * a.dv + col] = v;
}
// Rows first, first + step, ... of a tile from shared memory (row r at os + r * LDS_, its l and m at lm[2 r]) to their places, a warp a row, four neighbouring
// columns a lane; place(r, t, h) says whose row it is.  What a row's columns share (the softmax's denominator with the sink, a head's gate) is worked out
// once.  (swa_mma_kernel's rows of 128 channels at most are no faster this way.)
template <int LDS_, typename Place>
__device__ __forceinline__ void smm_store_rows(const SwaArgs& a, const float* os, const float* lm, int first, int step, int nrows, int sp, Place place) {
	const int lane = threadIdx.x & 31, dv = a.dv, ldo = a.ldo ? a.ldo : a.H * dv;
	float* out = a.n_splits > 1 ? a.part_o : a.out;
	const bool wide = ((ldo | dv) & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
#pragma unroll 1
	for (int r = first; r < nrows; r += step) {
		int t, h;
		place(r, t, h);
		const float l = lm[2 * r], m = lm[2 * r + 1];
		float c = 1.f, den = 1.f, g = 1.f;
		size_t at;
		if (a.n_splits > 1) { // swa_merge_kernel joins them
			at = ((size_t) t * a.n_splits + sp) * (a.H * dv) + (size_t) h * dv;
			if (lane == 0) {
				float* pml = a.part_ml + ((size_t) t * a.n_splits + sp) * (a.H * 2) + 2 * h;
				pml[0] = m;
				pml[1] = l;
			}
		} else { // as swa_finish
			at = (size_t) t * ldo + (size_t) h * dv;
			den = l;
			if (a.sink) {
				const float sk = a.sink[h];
				if (sk > m) {
					c = expf(m - sk);
					den = fmaf(den, c, 1.f);
				} else den += expf(sk - m);
			}
			if (a.gate && a.gate_per_head) g = swa_gate(a, t, h, 0);
		}
#pragma unroll 1
		for (int col = lane * 4; col < dv; col += 128) {
			const float4 x = *reinterpret_cast<const float4*>(os + r * LDS_ + col);
			float o[4] = {x.x, x.y, x.z, x.w};
			if (a.n_splits <= 1) {
#pragma unroll
				for (int e = 0; e < 4; e++) {
					o[e] = o[e] * c / den;
					if (a.out_scale != 0.f) o[e] *= a.out_scale;
					if (a.gate) o[e] *= a.gate_per_head ? g : swa_gate(a, t, h, col + e);
				}
			}
			if (wide) *reinterpret_cast<float4*>(out + at + col) = make_float4(o[0], o[1], o[2], o[3]);
			else
#pragma unroll
				for (int e = 0; e < 4; e++) out[at + col + e] = o[e];
		}
	}
}
// A query by fp32 FMAs on one warp, keys that it does not see left out: for infinities and NaN, whose planes are not finite and whose product with a masked
// key's weight of zero is NaN.  t: its row, i: its position; DV: the value channels rounded up
template <int DV>
__device__ __forceinline__ void smm_nonfinite_row(const SwaArgs& a, const SwaKeys& km, const __nv_bfloat16* kc, const __nv_bfloat16* vc, int ldk, int ldv, int t, int i,
                                                  int h, int sp, int jb, int je, float slope, float b1, float b2) {
	const int lane = threadIdx.x & 31;
	const float* q = a.q + (size_t) t * a.ldq + a.q_off + (size_t) h * a.d;
	float m = -INFINITY, l = 0.f, o[DV / 32] = {};
	for (int j0 = jb; j0 < je; j0 += 32) {
		const int x = min(j0 + lane, je - 1), j = km.pos(x);
		const bool seen = j0 + lane < je && smm_seen(a, i, j);
		const __nv_bfloat16* k = kc + (size_t) km.slot(x) * ldk;
		float s = 0.f;
		for (int c = 0; c < a.d; c++) s = fmaf(q[c], __bfloat162float(k[c]), s);
		s = seen ? smm_score(a, s, i, j, slope, b1, b2) : -INFINITY;
		const float top = fmaxf(m, warp_max(s)), at = top == -INFINITY ? 0.f : top, keep = m == -INFINITY ? 0.f : expf(m - at), p = expf(s - at);
		l = fmaf(l, keep, warp_sum(p));
		m = top;
#pragma unroll
		for (int c = 0; c < DV / 32; c++) o[c] *= keep;
		const unsigned sees = __ballot_sync(0xffffffffu, seen);
		for (int y = 0; y < 32; y++) {
			const float w = __shfl_sync(0xffffffffu, p, y);
			if (!(sees >> y & 1)) continue;
			const __nv_bfloat16* v = vc + (size_t) km.slot(j0 + y) * ldv;
#pragma unroll
			for (int c = 0; c < DV / 32; c++)
				if (c * 32 + lane < a.dv) o[c] = fmaf(w, __bfloat162float(v[c * 32 + lane]), o[c]);
		}
	}
#pragma unroll
	for (int c = 0; c < DV / 32; c++)
		if (c * 32 + lane < a.dv) smm_store(a, t, h, sp, c * 32 + lane, o[c], l, m);
}
// the CTA's nq queries, a warp per query
template <int DV, int WARPS>
__device__ __noinline__ void smm_nonfinite(const SwaArgs a, const SwaKeys km, const __nv_bfloat16* kc, const __nv_bfloat16* vc, int ldk, int ldv, int t0, int nq,
                                              int i_lo, int h, int sp, int jb, int je, float slope, float b1, float b2) {
	for (int row = threadIdx.x >> 5; row < nq; row += WARPS) smm_nonfinite_row<DV>(a, km, kc, vc, ldk, ldv, t0 + row, i_lo + row, h, sp, jb, je, slope, b1, b2);
}

// DQ, DV: the channel counts rounded up to 64 or 128 (the rest is zero); WARPS * 16 queries
template <int DQ, int DV, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) swa_mma_kernel(SwaArgs a) {
	extern __shared__ __align__(128) uint8_t smem[];
	constexpr int NTH = WARPS * 32, ROWS = WARPS * 16;
	uint8_t* qs = smem;                                  // 3 planes x ROWS x DQ
	uint8_t* ks = qs + (size_t) 3 * ROWS * DQ * 2;       // stages x SMM_KEYS x DQ
	uint8_t* vs = ks + (size_t) SMM_STAGES * SMM_KEYS * DQ * 2;
	int* kp = reinterpret_cast<int*>(vs + (size_t) SMM_STAGES * SMM_KEYS * DV * 2); // stages x SMM_KEYS positions (0x7fffffff: no key)
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quad = lane >> 2, ql = lane & 3;
	const int n = a.step->n, pos0 = a.step->pos0, H = a.H, G = a.G, d = a.d, dv = a.dv;
	const int t0 = ((int) gridDim.x - 1 - (int) blockIdx.x) * ROWS, h = blockIdx.y, g = h / (H / G); // the last queries see the most keys: they start first
	const int nq = min(ROWS, n - t0);
	if (nq <= 0) return;
	const int i_lo = pos0 + t0, i_hi = i_lo + nq - 1;
	const SwaKeys km = swa_keys(a, i_lo);
	const int nk = km.ks + i_hi - km.j_first + 1;
	const int per = ((nk + a.n_splits - 1) / a.n_splits + SMM_KEYS - 1) / SMM_KEYS * SMM_KEYS, sp = blockIdx.z; // whole key blocks for every split but the last
	const int jb = min(nk, sp * per), je = min(nk, jb + per);
	const int ldk = a.ldk ? a.ldk : G * d, ldv = a.ldv ? a.ldv : G * dv;
	const __nv_bfloat16* kc = reinterpret_cast<const __nv_bfloat16*>(a.kc) + (size_t) g * d;
	const __nv_bfloat16* vc = reinterpret_cast<const __nv_bfloat16*>(a.vc) + (size_t) g * dv;

	auto stage = [&](int j0, int buf) {
		const uint32_t kb = smem_u32(ks) + (uint32_t) buf * SMM_KEYS * DQ * 2, vb = smem_u32(vs) + (uint32_t) buf * SMM_KEYS * DV * 2;
		// PER threads share a key, whose slot is worked out once, and take alternate 16-byte pieces; size 0 writes zeros (beyond the last key or channel)
		constexpr int PER = NTH / SMM_KEYS;
		const int row = tid / PER, j = min(j0 + row, je - 1), first = tid % PER;
		const bool in = j0 + row < je;
		const size_t slot = km.slot(j);
		if (first == 0) kp[buf * SMM_KEYS + row] = in ? km.pos(j) : 0x7fffffff;
		const __nv_bfloat16 *kr = kc + slot * ldk, *vr = vc + slot * ldv;
#pragma unroll
		for (int p = 0; p < DQ / 8; p += PER) {
			const int ok = in && (p + first) * 8 < d;
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(kb + smm_at<DQ>(row, p + first)), "l"(kr + (ok ? (p + first) * 8 : 0)), "r"(ok ? 16 : 0) : "memory");
		}
#pragma unroll
		for (int p = 0; p < DV / 8; p += PER) {
			const int ok = in && (p + first) * 8 < dv;
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(vb + smm_at<DV>(row, p + first)), "l"(vr + (ok ? (p + first) * 8 : 0)), "r"(ok ? 16 : 0) : "memory");
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	if (jb < je) stage(jb, 0);
	// queries, as planes
	for (int x = tid; x < ROWS * (DQ / 8); x += NTH) {
		const int row = x / (DQ / 8), p = x % (DQ / 8);
		float v[8] = {};
		if (row < nq && p * 8 < d) ld8(a.q + (size_t) (t0 + row) * a.ldq + a.q_off + (size_t) h * d + p * 8, v);
		uint32_t w[3][4];
#pragma unroll
		for (int e = 0; e < 4; e++) smm_split(v[2 * e], v[2 * e + 1], w[0][e], w[1][e], w[2][e]);
#pragma unroll
		for (int pl = 0; pl < 3; pl++)
			*reinterpret_cast<uint4*>(qs + (size_t) pl * ROWS * DQ * 2 + smm_at<DQ>(row, p)) = make_uint4(w[pl][0], w[pl][1], w[pl][2], w[pl][3]);
	}
	float o[DV / 8][4] = {}, m[2] = {-INFINITY, -INFINITY}, l[2] = {};
	const int r0 = warp * 16 + quad; // this thread's rows: r0 and r0 + 8 of the CTA's
	const float slope = a.slope ? a.slope[h] : 0.f, b1 = a.r1 ? a.r1[h] : 0.f, b2 = a.r1 ? a.r2[h] : 0.f;
	const int blocks = (je - jb + SMM_KEYS - 1) / SMM_KEYS;
	const bool plain = !(a.softcap > 0.f) && !a.r1 && !a.slope, one_run = a.mask_chunk <= 0 || i_lo / a.mask_chunk == i_hi / a.mask_chunk;
	for (int blk = 0; blk < blocks; blk++) {
		const int buf = blk % SMM_STAGES, j0 = jb + blk * SMM_KEYS;
		if (blk + 1 < blocks) {
			stage(j0 + SMM_KEYS, (blk + 1) % SMM_STAGES);
			asm volatile("cp.async.wait_group 1;" ::: "memory");
		} else asm volatile("cp.async.wait_group 0;" ::: "memory");
		__syncthreads();
		const uint32_t kb = smem_u32(ks) + (uint32_t) buf * SMM_KEYS * DQ * 2, vb = smem_u32(vs) + (uint32_t) buf * SMM_KEYS * DV * 2;
		// ---- scores ----
		float s[SMM_KEYS / 8][4] = {};
#pragma unroll
		for (int k = 0; k < DQ / 16; k++) {
			uint32_t qa[3][4];
#pragma unroll
			for (int pl = 0; pl < 3; pl++) smm_ldsm4(qa[pl], smem_u32(qs) + (uint32_t) pl * ROWS * DQ * 2 + smm_at<DQ>(warp * 16 + (lane & 15), 2 * k + (lane >> 4)));
#pragma unroll
			for (int c = 0; c < SMM_KEYS / 16; c += 2) { // 32 keys
				uint32_t b[2][4];
				float part[4][4] = {};
#pragma unroll
				for (int x = 0; x < 2; x++) smm_ldsm4(b[x], kb + smm_at<DQ>((c + x) * 16 + (lane & 7) + ((lane >> 4) << 3), 2 * k + ((lane >> 3) & 1)));
				smm_planes(part, qa, b);
#pragma unroll
				for (int x = 0; x < 4; x++)
#pragma unroll
					for (int e = 0; e < 4; e++) s[2 * c + x][e] += part[x][e];
			}
		}
		// ---- scale, soft cap, biases, mask ----
		const int* pos = kp + buf * SMM_KEYS;
		float top[2] = {m[0], m[1]};
		const int p_lo = km.pos(j0), p_hi = km.pos(min(j0 + SMM_KEYS, je) - 1);
		if (plain && j0 + SMM_KEYS <= je && p_hi <= i_lo && (a.window >= 0x7fffffff || i_hi - p_lo < a.window || p_hi < a.keep_first) && one_run) {
			// every query sees every key of the block, and the score is only scaled
#pragma unroll
			for (int c = 0; c < SMM_KEYS / 8; c++)
#pragma unroll
				for (int e = 0; e < 4; e++) {
					s[c][e] *= a.scale;
					top[e >> 1] = fmaxf(top[e >> 1], s[c][e]);
				}
		} else
#pragma unroll
		for (int c = 0; c < SMM_KEYS / 8; c++)
#pragma unroll
			for (int e = 0; e < 4; e++) {
				const int i = i_lo + r0 + (e >> 1) * 8, j = pos[c * 8 + ql * 2 + (e & 1)];
				s[c][e] = smm_seen(a, i, j) ? smm_score(a, s[c][e], i, j, slope, b1, b2) : -INFINITY;
				top[e >> 1] = fmaxf(top[e >> 1], s[c][e]);
			}
		// ---- softmax weights ----
#pragma unroll
		for (int r = 0; r < 2; r++) {
			top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 1));
			top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], 2));
			const float at = top[r] == -INFINITY ? 0.f : top[r], keep = m[r] == -INFINITY ? 0.f : expf(m[r] - at);
			float sum = 0.f;
#pragma unroll
			for (int c = 0; c < SMM_KEYS / 8; c++)
#pragma unroll
				for (int e = 0; e < 2; e++) {
					s[c][2 * r + e] = expf(s[c][2 * r + e] - at);
					sum += s[c][2 * r + e];
				}
			l[r] = fmaf(l[r], keep, sum); // this lane's keys; joined at the end
			m[r] = top[r];
#pragma unroll
			for (int c = 0; c < DV / 8; c++)
#pragma unroll
				for (int e = 0; e < 2; e++) o[c][2 * r + e] *= keep;
		}
		uint32_t p[SMM_KEYS / 16][3][4];
#pragma unroll
		for (int c = 0; c < SMM_KEYS / 16; c++)
#pragma unroll
			for (int e = 0; e < 4; e++) smm_split(s[2 * c + (e >> 1)][(e & 1) * 2], s[2 * c + (e >> 1)][(e & 1) * 2 + 1], p[c][0][e], p[c][1][e], p[c][2][e]);
		// ---- values ----
#pragma unroll
		for (int c = 0; c < DV / 16; c += 2) { // 32 value channels
#pragma unroll
			for (int k = 0; k < SMM_KEYS / 16; k++) {
				uint32_t b[2][4];
				float part[4][4] = {};
#pragma unroll
				for (int x = 0; x < 2; x++) smm_ldsm4_t(b[x], vb + smm_at<DV>(k * 16 + (lane & 15), 2 * (c + x) + (lane >> 4)));
				smm_planes(part, p[k], b);
#pragma unroll
				for (int x = 0; x < 4; x++)
#pragma unroll
					for (int e = 0; e < 4; e++) o[2 * c + x][e] += part[x][e];
			}
		}
		__syncthreads(); // the block's buffer is read
	}
	bool finite = true;
#pragma unroll
	for (int r = 0; r < 2; r++) {
		l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
		l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
		if (r0 + r * 8 >= nq) continue;
		finite &= isfinite(l[r]);
#pragma unroll
		for (int c = 0; c < DV / 8; c++) finite &= isfinite(o[c][2 * r]) && isfinite(o[c][2 * r + 1]);
	}
	if (__syncthreads_or(!finite)) {
		smm_nonfinite<DV, WARPS>(a, km, kc, vc, ldk, ldv, t0, nq, i_lo, h, sp, jb, je, slope, b1, b2);
		return;
	}
	// Through shared memory, a warp its own rows: with the store's code once per value of a thread, fetching it took 45 us of a CTA's time (16 tokens of 8
	// heads over 1024 keys, one split: 139 -> 94 us)
	constexpr int LDO = DV + 8; // floats: the eight rows of a fragment on different banks
	float *os = reinterpret_cast<float*>(smem) + warp * 16 * LDO, *ls = reinterpret_cast<float*>(smem) + ROWS * LDO + warp * 32;
#pragma unroll
	for (int r = 0; r < 2; r++) {
#pragma unroll
		for (int c = 0; c < DV / 8; c++) *reinterpret_cast<float2*>(os + (quad + r * 8) * LDO + c * 8 + ql * 2) = make_float2(o[c][2 * r], o[c][2 * r + 1]);
		if (ql == 0) *reinterpret_cast<float2*>(ls + (quad + r * 8) * 2) = make_float2(l[r], m[r]);
	}
	__syncwarp();
	for (int row = 0; row < min(16, nq - warp * 16); row++)
#pragma unroll 1
		for (int col = lane; col < dv; col += 32) smm_store(a, t0 + warp * 16 + row, h, sp, col, os[row * LDO + col], ls[row * 2], ls[row * 2 + 1]);
}
static_assert(4 * (64 * (64 + 8) + 4 * 32) <= smm_smem(64, 64, 4) && 4 * (64 * (128 + 8) + 4 * 32) <= smm_smem(64, 128, 4), "the output's rows fit where queries and keys lay");

// ---- a latent: one head of up to 576 channels of keys, whose first channels are the values, for all query heads -------------------------------
// Rows of a tile are (query, head) pairs, 32 a CTA.  Two groups of W warps, 16 rows each: for the scores a warp takes a W-th of the channels (its queries'
// planes stay in registers) and all 64 keys of a block, for the output a W-th of the value channels.  The parts of the scores meet in shared memory, where a
// warp makes its share of the rows' weights of them.  Products and sums as above.
// Bound: latency of a scheduler's four warps (1024 tokens of 8 heads of 256: issue slots 30 %, mma.sync pipe 17 %); at 512 channels the pipe is next (3072
// products of 16 x 8 x 16 per 64 keys).  Registers are short: at the 128 of two CTAs per SM the queries' planes of 256 channels spill in part (7 % of the warp
// instructions are spill stores and loads), a few of the instances for 512 and 576 channels too.  W = 8 where W = 4 would
// leave two warps per scheduler (256 tokens of 16 heads of 512 over 256 to 777 keys 93 -> 72 us).  The instance for up to 320 channels with values of 256 against
// the one for 512 (320 and 328 channels, 64 tokens of 8 heads over 4000 keys): 69 us, 79; 33 tokens over 33 keys 26, 26.  The fp32 FMA tiles of mix_ops.cuh, which took these passes
// before, and this kernel, caches flushed: 256 tokens of 16 heads of 512 496 -> 72 us, 9 tokens of them over 777 keys 244 -> 24 + 6 us (twelve splits and their join), 1024 tokens of 8 heads of 256
// in a window of 512 357 -> 110 us.  Distance from float64 at 512 channels and 764 keys: within 5 % of the FMA kernel's.
constexpr int SML_ROWS = SWA_LATENT_ROWS, SML_LDS = SMM_KEYS + 4; // floats of a row of scores
template <int W, int NK, int NV>
struct SmlCfg { // NK, NV: 16 channels of keys and of values per warp
	static constexpr int TH = 2 * W * 32, DQ = W * NK * 16, DV = W * NV * 16, RPW = SML_ROWS / (2 * W); // RPW: rows whose weights a warp makes
	static constexpr size_t SMEM = (size_t) SMM_STAGES * SMM_KEYS * DQ * 2 + (size_t) W * SML_ROWS * SML_LDS * 4 + (size_t) 3 * SML_ROWS * SMM_KEYS * 2 +
	                               (size_t) SMM_STAGES * SMM_KEYS * 4 + 4 * SML_ROWS * 4;
	static constexpr int PER_SM = 2 * (SMEM + 1024) <= 228 * 1024 && TH <= 256 ? 2 : 1;
};
template <int DV, int TH>
__device__ __noinline__ void sml_nonfinite(const SwaArgs a, const SwaKeys km, const __nv_bfloat16* kc, int ldk, int row0, int nrows, int pos0, int sp, int jb, int je) {
	for (int row = threadIdx.x >> 5; row < nrows; row += TH / 32) {
		const int t = (row0 + row) / a.H, h = (row0 + row) % a.H;
		smm_nonfinite_row<DV>(a, km, kc, kc, ldk, ldk, t, pos0 + t, h, sp, jb, je, a.slope ? a.slope[h] : 0.f, a.r1 ? a.r1[h] : 0.f, a.r1 ? a.r2[h] : 0.f);
	}
}

template <int W, int NK, int NV>
__global__ void __launch_bounds__(SmlCfg<W, NK, NV>::TH, SmlCfg<W, NK, NV>::PER_SM) swa_latent_kernel(SwaArgs a) {
	using Cfg = SmlCfg<W, NK, NV>;
	extern __shared__ __align__(128) uint8_t smem[];
	constexpr int TH = Cfg::TH, DQ = Cfg::DQ, DV = Cfg::DV, RPW = Cfg::RPW, LDO = DV + 8;
	static_assert((size_t) SML_ROWS * LDO * 4 <= (size_t) SMM_STAGES * SMM_KEYS * DQ * 2, "the output's rows fit where the keys lay");
	uint8_t* ks = smem;                                                                       // stages x SMM_KEYS x DQ
	float* sc = reinterpret_cast<float*>(ks + (size_t) SMM_STAGES * SMM_KEYS * DQ * 2);       // W parts x SML_ROWS x SML_LDS
	uint8_t* ps = reinterpret_cast<uint8_t*>(sc + W * SML_ROWS * SML_LDS);                    // 3 planes x SML_ROWS x SMM_KEYS
	int* kp = reinterpret_cast<int*>(ps + (size_t) 3 * SML_ROWS * SMM_KEYS * 2);              // stages x SMM_KEYS positions (0x7fffffff: no key)
	float *keeps = reinterpret_cast<float*>(kp + SMM_STAGES * SMM_KEYS), *lm = keeps + SML_ROWS;
	int* at_row = reinterpret_cast<int*>(lm + 2 * SML_ROWS); // rows' positions
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quad = lane >> 2, ql = lane & 3, rg = warp / W, qt = warp % W;
	const int n = a.step->n, pos0 = a.step->pos0, H = a.H, d = a.d, dv = a.dv;
	const int row0 = ((int) gridDim.x - 1 - (int) blockIdx.x) * SML_ROWS, nrows = min(SML_ROWS, n * H - row0);
	if (nrows <= 0) return;
	const int i_lo = pos0 + row0 / H, i_hi = pos0 + (row0 + nrows - 1) / H;
	const SwaKeys km = swa_keys(a, i_lo);
	const int nk = km.ks + i_hi - km.j_first + 1;
	const int per = ((nk + a.n_splits - 1) / a.n_splits + SMM_KEYS - 1) / SMM_KEYS * SMM_KEYS, sp = blockIdx.y;
	const int jb = min(nk, sp * per), je = min(nk, jb + per);
	const int ldk = a.ldk ? a.ldk : d;
	const __nv_bfloat16* kc = reinterpret_cast<const __nv_bfloat16*>(a.kc);
	auto stage = [&](int j0, int buf) {
		const uint32_t kb = smem_u32(ks) + (uint32_t) buf * SMM_KEYS * DQ * 2;
		constexpr int PER = TH / SMM_KEYS;
		const int row = tid / PER, first = tid % PER;
		const bool in = j0 + row < je;
		const int j = min(j0 + row, je - 1);
		if (first == 0) kp[buf * SMM_KEYS + row] = in ? km.pos(j) : 0x7fffffff;
		const __nv_bfloat16* kr = kc + (size_t) km.slot(j) * ldk;
#pragma unroll
		for (int p = 0; p < DQ / 8; p += PER) {
			const int ok = in && (p + first) * 8 < d;
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(kb + smm_at<DQ>(row, p + first)), "l"(kr + (ok ? (p + first) * 8 : 0)), "r"(ok ? 16 : 0) : "memory");
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	if (jb < je) stage(jb, 0);
	uint32_t qf[NK][3][4]; // this warp's rows and channels as operand fragments, three planes
#pragma unroll
	for (int k = 0; k < NK; k++)
#pragma unroll
		for (int e = 0; e < 4; e++) {
			const int row = rg * 16 + quad + (e & 1) * 8, col = (qt * NK + k) * 16 + ql * 2 + (e >> 1) * 8;
			float2 v = make_float2(0.f, 0.f);
			if (row < nrows && col < d) v = *reinterpret_cast<const float2*>(a.q + (size_t) ((row0 + row) / H) * a.ldq + a.q_off + (size_t) ((row0 + row) % H) * d + col);
			smm_split(v.x, v.y, qf[k][0][e], qf[k][1][e], qf[k][2][e]);
		}
	float o[2 * NV][4] = {}; // rows quad, quad + 8 of the group; value channels (qt * NV + ..) * 16 ..
	float m[RPW], l[RPW]; // of rows RPW warp .. (l: this lane's keys)
#pragma unroll
	for (int r = 0; r < RPW; r++) { m[r] = -INFINITY; l[r] = 0.f; }
	const bool biased = a.r1 || a.slope;
	if (tid < SML_ROWS) at_row[tid] = pos0 + (row0 + min(tid, nrows - 1)) / H;
	const int blocks = (je - jb + SMM_KEYS - 1) / SMM_KEYS;
	for (int blk = 0; blk < blocks; blk++) {
		const int buf = blk % SMM_STAGES, j0 = jb + blk * SMM_KEYS;
		asm volatile("cp.async.wait_group 0;" ::: "memory");
		__syncthreads(); // the block's keys are there, and nobody reads the block before it any more
		if (blk + 1 < blocks) stage(j0 + SMM_KEYS, (blk + 1) % SMM_STAGES);
		const uint32_t kb = smem_u32(ks) + (uint32_t) buf * SMM_KEYS * DQ * 2;
		{ // ---- scores over this warp's channels ----
#pragma unroll 1
			for (int half = 0; half < SMM_KEYS; half += 32) {
				float s[4][4] = {};
#pragma unroll
				for (int k = 0; k < NK; k++) {
					uint32_t b[2][4];
					float part[4][4] = {};
#pragma unroll
					for (int x = 0; x < 2; x++) smm_ldsm4(b[x], kb + smm_at<DQ>(half + x * 16 + (lane & 7) + ((lane >> 4) << 3), 2 * (qt * NK + k) + ((lane >> 3) & 1)));
					smm_planes(part, qf[k], b);
#pragma unroll
					for (int x = 0; x < 4; x++)
#pragma unroll
						for (int e = 0; e < 4; e++) s[x][e] += part[x][e];
				}
				float* dst = sc + ((size_t) qt * SML_ROWS + rg * 16 + quad) * SML_LDS + half + ql * 2;
#pragma unroll
				for (int c = 0; c < 4; c++)
#pragma unroll
					for (int r = 0; r < 2; r++) *reinterpret_cast<float2*>(dst + r * 8 * SML_LDS + c * 8) = make_float2(s[c][2 * r], s[c][2 * r + 1]);
			}
		}
		__syncthreads();
		// ---- weights: a lane takes two neighbouring keys ----
#pragma unroll
		for (int r = 0; r < RPW; r++) {
			const int row = warp * RPW + r;
			float z[2] = {};
#pragma unroll
			for (int q = 0; q < W; q++) {
				const float2 v = *reinterpret_cast<const float2*>(sc + ((size_t) q * SML_ROWS + row) * SML_LDS + lane * 2);
				z[0] += v.x; z[1] += v.y;
			}
			const int2 j = *reinterpret_cast<const int2*>(kp + buf * SMM_KEYS + lane * 2);
			const int i = at_row[row];
			float slope = 0.f, b1 = 0.f, b2 = 0.f;
			if (biased) {
				const int h = (row0 + min(row, nrows - 1)) % H;
				if (a.slope) slope = a.slope[h];
				if (a.r1) { b1 = a.r1[h]; b2 = a.r2[h]; }
			}
			z[0] = smm_seen(a, i, j.x) ? smm_score(a, z[0], i, j.x, slope, b1, b2) : -INFINITY;
			z[1] = smm_seen(a, i, j.y) ? smm_score(a, z[1], i, j.y, slope, b1, b2) : -INFINITY;
			const float top = fmaxf(m[r], warp_max(fmaxf(z[0], z[1]))), at = top == -INFINITY ? 0.f : top, keep = m[r] == -INFINITY ? 0.f : expf(m[r] - at);
			const float p0 = expf(z[0] - at), p1 = expf(z[1] - at);
			l[r] = fmaf(l[r], keep, p0 + p1);
			m[r] = top;
			if (lane == 0) keeps[row] = keep;
			uint32_t pl[3];
			smm_split(p0, p1, pl[0], pl[1], pl[2]);
#pragma unroll
			for (int x = 0; x < 3; x++) *reinterpret_cast<uint32_t*>(ps + (size_t) x * SML_ROWS * SMM_KEYS * 2 + smm_at<SMM_KEYS>(row, lane >> 2) + (lane & 3) * 4) = pl[x];
		}
		__syncthreads();
		// ---- values ----
		const float k0 = keeps[rg * 16 + quad], k1 = keeps[rg * 16 + quad + 8];
#pragma unroll
		for (int c = 0; c < 2 * NV; c++) { o[c][0] *= k0; o[c][1] *= k0; o[c][2] *= k1; o[c][3] *= k1; }
#pragma unroll 1
		for (int k = 0; k < SMM_KEYS / 16; k++) {
			uint32_t pa[3][4];
#pragma unroll
			for (int pl = 0; pl < 3; pl++) smm_ldsm4(pa[pl], smem_u32(ps) + (uint32_t) pl * SML_ROWS * SMM_KEYS * 2 + smm_at<SMM_KEYS>(rg * 16 + (lane & 15), 2 * k + (lane >> 4)));
#pragma unroll
			for (int c = 0; c < NV; c += 2) { // 32 value channels
				uint32_t b[2][4];
				float part[4][4] = {};
#pragma unroll
				for (int x = 0; x < 2; x++) smm_ldsm4_t(b[x], kb + smm_at<DQ>(k * 16 + (lane & 15), 2 * (qt * NV + c + x) + (lane >> 4)));
				smm_planes(part, pa, b);
#pragma unroll
				for (int x = 0; x < 4; x++)
#pragma unroll
					for (int e = 0; e < 4; e++) o[2 * c + x][e] += part[x][e];
			}
		}
	}
	bool finite = true;
#pragma unroll
	for (int r = 0; r < RPW; r++) {
		l[r] = warp_sum(l[r]);
		if (warp * RPW + r < nrows) finite &= isfinite(l[r]);
		if (lane == 0) *reinterpret_cast<float2*>(lm + 2 * (warp * RPW + r)) = make_float2(l[r], m[r]);
	}
#pragma unroll
	for (int r = 0; r < 2; r++)
		if (rg * 16 + quad + r * 8 < nrows)
#pragma unroll
			for (int c = 0; c < 2 * NV; c++) finite &= isfinite(o[c][2 * r]) && isfinite(o[c][2 * r + 1]);
	if (__syncthreads_or(!finite)) {
		sml_nonfinite<DV, TH>(a, km, kc, ldk, row0, nrows, pos0, sp, jb, je);
		return;
	}
	float* os = reinterpret_cast<float*>(smem);
#pragma unroll
	for (int r = 0; r < 2; r++)
#pragma unroll
		for (int c = 0; c < 2 * NV; c++)
			*reinterpret_cast<float2*>(os + (rg * 16 + quad + r * 8) * LDO + (qt * NV * 2 + c) * 8 + ql * 2) = make_float2(o[c][2 * r], o[c][2 * r + 1]);
	__syncthreads();
	smm_store_rows<LDO>(a, os, lm, warp, TH / 32, nrows, sp, [&](int r, int& t, int& h) { t = (row0 + r) / H; h = (row0 + r) % H; });
}

template <int W, int NK, int NV>
static int launch_swa_latent_inst(const SwaArgs& a, int rows, cudaStream_t s) {
	using Cfg = SmlCfg<W, NK, NV>;
	XALM_CUDA_CHECK(cudaFuncSetAttribute(swa_latent_kernel<W, NK, NV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) Cfg::SMEM));
	swa_latent_kernel<W, NK, NV><<<dim3((unsigned) (((long long) rows * a.H + SML_ROWS - 1) / SML_ROWS), a.n_splits), Cfg::TH, Cfg::SMEM, s>>>(a);
	return launch_check("swa_latent");
}
int launch_swa_latent(const SwaArgs& a, int rows, cudaStream_t s) {
	if (a.d <= 256) return launch_swa_latent_inst<4, 4, 4>(a, rows, s);
	if (a.d <= 320 && a.dv <= 256) return launch_swa_latent_inst<4, 5, 4>(a, rows, s);
	return a.d <= 512 ? launch_swa_latent_inst<8, 4, 4>(a, rows, s) : launch_swa_latent_inst<4, 9, 8>(a, rows, s);
}

template <int DQ, int DV>
static int launch_swa_mma_inst(const SwaArgs& a, int rows, cudaStream_t s) {
	// Fewer warps per CTA for passes of 16 and 32 tokens, and two for twice the CTAs, copied every key block for fewer queries and were slower
	constexpr int WARPS = SWA_MMA_ROWS / 16;
	XALM_CUDA_CHECK(cudaFuncSetAttribute(swa_mma_kernel<DQ, DV, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smm_smem(DQ, DV, WARPS)));
	swa_mma_kernel<DQ, DV, WARPS><<<dim3((rows + WARPS * 16 - 1) / (WARPS * 16), a.H, a.n_splits), WARPS * 32, smm_smem(DQ, DV, WARPS), s>>>(a);
	return launch_check("swa_mma");
}

int launch_swa_mma(const SwaArgs& a, int rows, cudaStream_t s) {
	if (a.d <= 64) return a.dv <= 64 ? launch_swa_mma_inst<64, 64>(a, rows, s) : launch_swa_mma_inst<64, 128>(a, rows, s);
	return a.dv <= 64 ? launch_swa_mma_inst<128, 64>(a, rows, s) : launch_swa_mma_inst<128, 128>(a, rows, s);
}

} // namespace mix
} // namespace xalm
