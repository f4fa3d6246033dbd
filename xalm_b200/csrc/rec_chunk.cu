// rec_chunk.cu — the gated linear recurrence of mix_ops.cuh (every mode of Hgrn2Args) for passes of many tokens, REC_L tokens at a time:
//
//   S_t = diag(f_t) S_{t-1} + g_t v_t^T,   o_t = S_t^T q_t
//
// With F_t the product of the decays from the chunk's start to t, and E_s of those behind s to its end,
//   rec_local_kernel   per chunk and head: A[t, s] = sum_i q_t[i] g_s[i] prod_{s < r <= t} f_r[i] for s <= t, o = A v, the chunk's own state
//                      (g E)^T v, the queries q F and the decay F over the whole chunk
//   rec_carry_kernel   chunk after chunk, the state every chunk starts from, and the one the pass leaves
//   rec_output_kernel  per chunk and head: o += (q F)^T S, then the per-head norm and the gate
// All of it in fp32 FMAs.  A decay only ever multiplies (A is built by walking t with g_s and its decays in registers): quotients of products of decays,
// which would make A a plain product of two matrices, overflow where a decay is small.  A product with s > t is not formed, so that an infinity
// or a NaN stays with the tokens that see it.
//
// Bound: latency and issue slots, 56 thousand warp instructions per chunk and head at 64 x 128 (a third the walk over t, half the two products with v), 29 % of
// the slots used at 1024 tokens of 8 heads.  Two CTAs of rec_local_kernel fit an SM at up to 64 key channels (100 KB each), one at 128 (149 KB).  The scan of
// hgrn2_cols_kernel takes token after token on a warp per scheduler, 0.4 to 0.6 us each (8 and 16 heads of 64 x 128); here all chunks and heads are there at
// once.  1024 tokens of 16 heads of 64 x 128: 505 us as a scan, 38 + 8 + 21 us as the three kernels (caches flushed).
#define XALM_SECONDARY_TU
#include "common.cuh"
#include "family.h"
#include "mix_ops.cuh"

namespace xalm {
namespace mix {

constexpr int REC_L = 64, REC_DV = 128, REC_TH = 256; // tokens of a chunk, value channels (the rest is zero), threads
constexpr int REC_LDA = REC_L + 4;

__host__ __device__ constexpr size_t rec_local_smem(int D) { return sizeof(float) * (3 * (size_t) REC_L * D + (size_t) REC_L * REC_LDA + (size_t) REC_L * REC_DV + 2 * REC_L); }
__host__ __device__ constexpr size_t rec_output_smem(int D) { return sizeof(float) * ((size_t) REC_L * (D + 4) + (size_t) D * REC_DV); }
static inline int rec_dim(int d) { return d <= 64 ? 64 : 128; }

// workspace: chunk states (chunks, H, D, REC_DV) | chunk decays (chunks, H, D) | queries (tokens, H, D)
struct RecWs {
	float *s, *f, *q;
};
__host__ __device__ inline RecWs rec_ws(float* ws, int chunks, int H, int D) {
	RecWs w;
	w.s = ws;
	w.f = w.s + (size_t) chunks * H * D * REC_DV;
	w.q = w.f + (size_t) chunks * H * D;
	return w;
}
size_t hgrn2_chunk_floats(int H, int d, int dv, int rows) {
	if (d > 128 || dv > REC_DV || rows < HG_CHUNK_ROWS) return 0;
	const size_t chunks = (rows + REC_L - 1) / REC_L, D = rec_dim(d);
	return chunks * H * D * REC_DV + chunks * H * D + chunks * REC_L * H * D;
}

__device__ __forceinline__ float4 rec_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// grid (chunks, H)
template <int D>
__global__ void __launch_bounds__(REC_TH) rec_local_kernel(Hgrn2Args a, int chunks) {
	extern __shared__ __align__(16) float sm[];
	float *qs = sm, *fs = qs + REC_L * D, *gs = fs + REC_L * D; // (token, channel)
	float* At = gs + REC_L * D;         // (s, t)
	float* vs = At + REC_L * REC_LDA;   // (token, value channel)
	float *sf = vs + REC_L * REC_DV, *sd = sf + REC_L;
	const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	const int n = a.step->n, t0 = c * REC_L, nt = min(REC_L, n - t0), d = a.d, dv = a.dv;
	if (nt <= 0) return;
	const int hk = a.keyed ? h / max(a.qk_rep, 1) : h;
	const float* rows = a.proj + (size_t) t0 * a.ld;
	if (a.keyed == 2) { // one step size and decay per token
		if (tid < REC_L) {
			const float dt = tid < nt ? softplusf_(rows[(size_t) tid * a.ld + a.dt_off + h] + a.dt_bias[h]) : 0.f;
			sd[tid] = dt;
			sf[tid] = expf(-expf(a.A_log[h]) * dt);
		}
		__syncthreads();
	}
	for (int x = tid; x < REC_L * (D / 4); x += REC_TH) {
		const int t = x / (D / 4), i = x % (D / 4) * 4;
		float f[4] = {1.f, 1.f, 1.f, 1.f}, g[4] = {}, q[4] = {}; // beyond the last token or channel: the state stays and nothing is read
		if (t < nt && i < d) {
			const float* row = rows + (size_t) t * a.ld;
			const float4 rq = rec_ld4(row + a.q_off + hk * d + i);
			const float zq[4] = {rq.x, rq.y, rq.z, rq.w};
			if (a.keyed || a.decay) {
				const float4 rk = rec_ld4(row + a.k_off + hk * d + i);
				const float k[4] = {rk.x, rk.y, rk.z, rk.w};
				float4 rf = make_float4(0.f, 0.f, 0.f, 0.f);
				if (a.keyed == 1) rf = rec_ld4(row + a.f_off + h * d + i);
				const float z[4] = {rf.x, rf.y, rf.z, rf.w};
#pragma unroll
				for (int e = 0; e < 4; e++) {
					f[e] = a.keyed == 1 ? z[e] : a.keyed == 2 ? sf[t] : a.decay[h];
					g[e] = a.keyed == 1 ? k[e] : a.keyed == 2 ? k[e] * sd[t] : k[e] * a.k_scale;
					q[e] = a.keyed && a.q_scale != 0.f ? zq[e] * a.q_scale : zq[e];
				}
			} else {
				const float4 rf = rec_ld4(row + a.f_off + h * d + i);
				const float z[4] = {rf.x, rf.y, rf.z, rf.w};
#pragma unroll
				for (int e = 0; e < 4; e++) {
					if (a.activated) { f[e] = z[e]; q[e] = zq[e]; }
					else {
						const float lo = a.lower ? a.lower[h * d + i + e] : 0.f;
						f[e] = lo + (1.f - lo) * sigmoidf_(z[e] + (a.f_bias ? a.f_bias[h * d + i + e] : 0.f));
						q[e] = zq[e] * sigmoidf_(zq[e]);
					}
					g[e] = 1.f - f[e];
				}
			}
		}
		*reinterpret_cast<float4*>(qs + t * D + i) = make_float4(q[0], q[1], q[2], q[3]);
		*reinterpret_cast<float4*>(fs + t * D + i) = make_float4(f[0], f[1], f[2], f[3]);
		*reinterpret_cast<float4*>(gs + t * D + i) = make_float4(g[0], g[1], g[2], g[3]);
	}
	for (int x = tid; x < REC_L * (REC_DV / 4); x += REC_TH) {
		const int t = x / (REC_DV / 4), i = x % (REC_DV / 4) * 4;
		*reinterpret_cast<float4*>(vs + t * REC_DV + i) = t < nt && i < dv ? rec_ld4(rows + (size_t) t * a.ld + a.v_off + h * dv + i) : make_float4(0.f, 0.f, 0.f, 0.f);
	}
	__syncthreads();
	// ---- A: a warp takes eight s, four lanes an s with every fourth four of its channels, and walks t.  The first warps walk farthest: two turns of
	// four warps, the second with the s from the other end ----
	{
		const int s_warp = (warp < 4 ? warp : 11 - warp) * 8, s = s_warp + (lane >> 2), part = lane & 3;
		float w[D / 4];
#pragma unroll
		for (int j = 0; j < D / 4; j++) w[j] = 0.f;
		auto step = [&](int t, bool first) { // first: some lane's s may be t
			float sum[4] = {};
			const float* by = first && t == s ? gs + t * D : fs + t * D;
#pragma unroll
			for (int j = 0; j < D / 16; j++) {
				const float4 f = rec_ld4(by + (j * 4 + part) * 4), q = rec_ld4(qs + t * D + (j * 4 + part) * 4);
				if (first && t == s) { w[4 * j] = f.x; w[4 * j + 1] = f.y; w[4 * j + 2] = f.z; w[4 * j + 3] = f.w; }
				else { w[4 * j] *= f.x; w[4 * j + 1] *= f.y; w[4 * j + 2] *= f.z; w[4 * j + 3] *= f.w; }
				sum[0] = fmaf(q.x, w[4 * j], sum[0]); sum[1] = fmaf(q.y, w[4 * j + 1], sum[1]); sum[2] = fmaf(q.z, w[4 * j + 2], sum[2]); sum[3] = fmaf(q.w, w[4 * j + 3], sum[3]);
			}
			float o = (sum[0] + sum[1]) + (sum[2] + sum[3]);
			o += __shfl_xor_sync(0xffffffffu, o, 1);
			o += __shfl_xor_sync(0xffffffffu, o, 2);
			if (part == 0 && (!first || t >= s)) At[s * REC_LDA + t] = first && t == s && a.skip ? o + a.skip[h] : o;
		};
		for (int t = s_warp; t < s_warp + 8; t++) step(t, true);
#pragma unroll 4
		for (int t = s_warp + 8; t < REC_L; t++) step(t, false);
	}
	__syncthreads();
	// ---- queries times the decays before them, keys times the decays behind them ----
	if (tid < 2 * D) {
		const bool fwd = tid < D;
		const int i = fwd ? tid : tid - D;
		float* by = fwd ? qs : gs;
		float F = 1.f;
		for (int t8 = 0; t8 < REC_L; t8 += 8) {
			float f[8], x[8];
#pragma unroll
			for (int u = 0; u < 8; u++) {
				const int t = fwd ? t8 + u : REC_L - 1 - t8 - u;
				f[u] = fs[t * D + i];
				x[u] = by[t * D + i];
			}
#pragma unroll
			for (int u = 0; u < 8; u++) {
				const int t = fwd ? t8 + u : REC_L - 1 - t8 - u;
				if (fwd) F *= f[u];
				by[t * D + i] = x[u] * F;
				if (!fwd) F *= f[u];
			}
		}
		if (fwd) rec_ws(a.ws, chunks, a.H, D).f[((size_t) c * a.H + h) * D + i] = F;
	}
	__syncthreads();
	const RecWs ws = rec_ws(a.ws, chunks, a.H, D);
	for (int x = tid; x < nt * (D / 4); x += REC_TH) {
		const int t = x / (D / 4), i = x % (D / 4) * 4;
		*reinterpret_cast<float4*>(ws.q + ((size_t) (t0 + t) * a.H + h) * D + i) = rec_ld4(qs + t * D + i);
	}
	// ---- the two products with v: D / 16 (state) and 4 (output) rows of a thread, value channels 4 tx .. and 64 + 4 tx .. ----
	const int ty = tid >> 4, tx = tid & 15;
	{
		constexpr int R = D / 16;
		float acc[R][8] = {};
#pragma unroll 4
		for (int s = 0; s < REC_L; s++) {
			const float4 v0 = rec_ld4(vs + s * REC_DV + tx * 4), v1 = rec_ld4(vs + s * REC_DV + 64 + tx * 4);
#pragma unroll
			for (int r4 = 0; r4 < R; r4 += 4) {
				const float4 k = rec_ld4(gs + s * D + ty * R + r4);
				const float kk[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
				for (int r = 0; r < 4; r++) {
					float* o = acc[r4 + r];
					o[0] = fmaf(kk[r], v0.x, o[0]); o[1] = fmaf(kk[r], v0.y, o[1]); o[2] = fmaf(kk[r], v0.z, o[2]); o[3] = fmaf(kk[r], v0.w, o[3]);
					o[4] = fmaf(kk[r], v1.x, o[4]); o[5] = fmaf(kk[r], v1.y, o[5]); o[6] = fmaf(kk[r], v1.z, o[6]); o[7] = fmaf(kk[r], v1.w, o[7]);
				}
			}
		}
		float* dst = ws.s + (((size_t) c * a.H + h) * D + ty * R) * REC_DV + tx * 4;
#pragma unroll
		for (int r = 0; r < R; r++) {
			*reinterpret_cast<float4*>(dst + (size_t) r * REC_DV) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
			*reinterpret_cast<float4*>(dst + (size_t) r * REC_DV + 64) = make_float4(acc[r][4], acc[r][5], acc[r][6], acc[r][7]);
		}
	}
	{
		const int tr = ty * 4; // rows tr .. tr + 3: every s up to tr, then those of the diagonal
		float acc[4][8] = {};
		auto add = [&](int s, int from) {
			const float4 v0 = rec_ld4(vs + s * REC_DV + tx * 4), v1 = rec_ld4(vs + s * REC_DV + 64 + tx * 4), k = rec_ld4(At + s * REC_LDA + tr);
			const float kk[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
			for (int r = 0; r < 4; r++) {
				if (r < from) continue;
				float* o = acc[r];
				o[0] = fmaf(kk[r], v0.x, o[0]); o[1] = fmaf(kk[r], v0.y, o[1]); o[2] = fmaf(kk[r], v0.z, o[2]); o[3] = fmaf(kk[r], v0.w, o[3]);
				o[4] = fmaf(kk[r], v1.x, o[4]); o[5] = fmaf(kk[r], v1.y, o[5]); o[6] = fmaf(kk[r], v1.z, o[6]); o[7] = fmaf(kk[r], v1.w, o[7]);
			}
		};
#pragma unroll 4
		for (int s = 0; s < tr; s++) add(s, 0);
#pragma unroll
		for (int j = 0; j < 4; j++) add(tr + j, j);
#pragma unroll
		for (int r = 0; r < 4; r++) {
			if (tr + r >= nt) continue;
			float* orow = a.out + (size_t) (t0 + tr + r) * (a.H * dv) + h * dv;
			if (tx * 4 < dv) *reinterpret_cast<float4*>(orow + tx * 4) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
			if (64 + tx * 4 < dv) *reinterpret_cast<float4*>(orow + 64 + tx * 4) = make_float4(acc[r][4], acc[r][5], acc[r][6], acc[r][7]);
		}
	}
}

// A thread takes four value channels of one key channel through the chunks and leaves, where a chunk's own state was, the state it starts from
template <int D>
__global__ void __launch_bounds__(128) rec_carry_kernel(Hgrn2Args a, int chunks) {
	const int x = blockIdx.x * 128 + threadIdx.x, per_head = D * (REC_DV / 4);
	const int h = x / per_head, i = x % per_head / (REC_DV / 4), col = x % (REC_DV / 4) * 4;
	if (h >= a.H || i >= a.d || col >= a.dv) return;
	const RecWs ws = rec_ws(a.ws, chunks, a.H, D);
	const int used = (a.step->n + REC_L - 1) / REC_L;
	float* st = a.state + ((size_t) h * a.d + i) * a.dv + col;
	float4 S = rec_ld4(st);
	constexpr int AHEAD = 8;
	for (int c0 = 0; c0 < used; c0 += AHEAD) {
		float4 own[AHEAD];
		float f[AHEAD];
#pragma unroll
		for (int u = 0; u < AHEAD; u++)
			if (c0 + u < used) {
				own[u] = rec_ld4(ws.s + (((size_t) (c0 + u) * a.H + h) * D + i) * REC_DV + col);
				f[u] = ws.f[((size_t) (c0 + u) * a.H + h) * D + i];
			}
#pragma unroll
		for (int u = 0; u < AHEAD; u++)
			if (c0 + u < used) {
				*reinterpret_cast<float4*>(ws.s + (((size_t) (c0 + u) * a.H + h) * D + i) * REC_DV + col) = S;
				S = make_float4(fmaf(f[u], S.x, own[u].x), fmaf(f[u], S.y, own[u].y), fmaf(f[u], S.z, own[u].z), fmaf(f[u], S.w, own[u].w));
			}
	}
	*reinterpret_cast<float4*>(st) = S;
}

// grid (chunks, H)
template <int D>
__global__ void __launch_bounds__(REC_TH) rec_output_kernel(Hgrn2Args a, int chunks) {
	extern __shared__ __align__(16) float sm[];
	constexpr int LDQ = D + 4;
	float *qs = sm, *Ss = qs + REC_L * LDQ;
	const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
	const int t0 = c * REC_L, nt = min(REC_L, a.step->n - t0), d = a.d, dv = a.dv;
	if (nt <= 0) return;
	const RecWs ws = rec_ws(a.ws, chunks, a.H, D);
	for (int x = tid; x < REC_L * (D / 4); x += REC_TH) {
		const int t = x / (D / 4), i = x % (D / 4) * 4;
		*reinterpret_cast<float4*>(qs + t * LDQ + i) = t < nt ? rec_ld4(ws.q + ((size_t) (t0 + t) * a.H + h) * D + i) : make_float4(0.f, 0.f, 0.f, 0.f);
	}
	const float* src = ws.s + ((size_t) c * a.H + h) * D * REC_DV;
	for (int x = tid; x < D * (REC_DV / 4); x += REC_TH) { // beyond the head's channels the workspace holds nothing
		const int i = x / (REC_DV / 4), col = x % (REC_DV / 4) * 4;
		*reinterpret_cast<float4*>(Ss + i * REC_DV + col) = i < d && col < dv ? rec_ld4(src + i * REC_DV + col) : make_float4(0.f, 0.f, 0.f, 0.f);
	}
	float acc[4][8] = {}, z[4][8] = {}, nw[8]; // the sums so far, gates, norm weights: all on their way before the first use
#pragma unroll
	for (int r = 0; r < 4; r++) {
		const int t = ty * 4 + r;
		if (t >= nt) continue;
		const float* orow = a.out + (size_t) (t0 + t) * (a.H * dv) + h * dv;
		const float* grow = a.gate ? a.gate + (size_t) (t0 + t) * a.ldg + a.g_off + h * dv : nullptr;
#pragma unroll
		for (int e = 0; e < 8; e += 4)
			if (e * 16 + tx * 4 < dv) {
				const float4 o = rec_ld4(orow + e * 16 + tx * 4);
				acc[r][e] = o.x; acc[r][e + 1] = o.y; acc[r][e + 2] = o.z; acc[r][e + 3] = o.w;
#pragma unroll
				for (int u = 0; u < 4; u++)
					if (grow) z[r][e + u] = grow[e * 16 + tx * 4 + u];
			}
	}
#pragma unroll
	for (int e = 0; e < 8; e++) nw[e] = a.norm_w && (e / 4) * 64 + tx * 4 + e % 4 < dv ? a.norm_w[(e / 4) * 64 + tx * 4 + e % 4] : 1.f;
	__syncthreads();
#pragma unroll 2
	for (int i = 0; i < D; i += 4) {
		float q[4][4];
#pragma unroll
		for (int r = 0; r < 4; r++) {
			const float4 v = rec_ld4(qs + (ty * 4 + r) * LDQ + i);
			q[r][0] = v.x; q[r][1] = v.y; q[r][2] = v.z; q[r][3] = v.w;
		}
#pragma unroll
		for (int e = 0; e < 4; e++) {
			const float4 s0 = rec_ld4(Ss + (i + e) * REC_DV + tx * 4), s1 = rec_ld4(Ss + (i + e) * REC_DV + 64 + tx * 4);
#pragma unroll
			for (int r = 0; r < 4; r++) {
				float* o = acc[r];
				o[0] = fmaf(q[r][e], s0.x, o[0]); o[1] = fmaf(q[r][e], s0.y, o[1]); o[2] = fmaf(q[r][e], s0.z, o[2]); o[3] = fmaf(q[r][e], s0.w, o[3]);
				o[4] = fmaf(q[r][e], s1.x, o[4]); o[5] = fmaf(q[r][e], s1.y, o[5]); o[6] = fmaf(q[r][e], s1.z, o[6]); o[7] = fmaf(q[r][e], s1.w, o[7]);
			}
		}
	}
	const bool normed = a.norm_w || a.norm_plain;
#pragma unroll
	for (int r = 0; r < 4; r++) {
		float scale = 1.f;
		if (normed) {
			float ss = 0.f;
#pragma unroll
			for (int e = 0; e < 8; e++) ss = fmaf(acc[r][e], acc[r][e], ss);
#pragma unroll
			for (int w = 1; w < 16; w <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, w);
			scale = 1.f / sqrtf(ss / (float) dv + a.eps);
		}
		const int t = ty * 4 + r;
		if (t >= nt) continue;
		float* orow = a.out + (size_t) (t0 + t) * (a.H * dv) + h * dv;
#pragma unroll
		for (int e = 0; e < 8; e += 4) {
			const int col = e * 16 + tx * 4;
			if (col >= dv) continue;
			float o[4];
#pragma unroll
			for (int u = 0; u < 4; u++) {
				o[u] = acc[r][e + u] * scale * nw[e + u];
				if (a.gate) o[u] *= z[r][e + u] * sigmoidf_(z[r][e + u]);
			}
			*reinterpret_cast<float4*>(orow + col) = make_float4(o[0], o[1], o[2], o[3]);
		}
	}
}

template <int D>
static int launch_chunks(const Hgrn2Args& a, cudaStream_t s) {
	XALM_CUDA_CHECK(cudaFuncSetAttribute(rec_local_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) rec_local_smem(D)));
	XALM_CUDA_CHECK(cudaFuncSetAttribute(rec_output_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) rec_output_smem(D)));
	const int chunks = (a.rows + REC_L - 1) / REC_L;
	rec_local_kernel<D><<<dim3(chunks, a.H), REC_TH, rec_local_smem(D), s>>>(a, chunks);
	XALM_TRY(launch_check("rec_local"));
	rec_carry_kernel<D><<<(a.H * D * (REC_DV / 4) + 127) / 128, 128, 0, s>>>(a, chunks);
	XALM_TRY(launch_check("rec_carry"));
	rec_output_kernel<D><<<dim3(chunks, a.H), REC_TH, rec_output_smem(D), s>>>(a, chunks);
	return launch_check("rec_output");
}
int launch_hgrn2_chunks(const Hgrn2Args& a, cudaStream_t s) { return a.d <= 64 ? launch_chunks<64>(a, s) : launch_chunks<128>(a, s); }

} // namespace mix
} // namespace xalm
