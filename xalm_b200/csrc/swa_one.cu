// swa_one.cu — the attention of mix_ops.cuh (window, kept first positions, chunks, soft cap, distance biases, sink, gate; no mixing of heads) for
// steps of one to four tokens.
//
// Bound: latency.  A step's keys are a few MB (0.3 to 1.3 us of memory time), so what counts is the chain of dependent trips: query -> keys and
// values -> softmax -> join, and the instructions' own way to the SM: a step runs this code once, from cold.  A cluster of 8 CTAs takes HB heads of one
// key/value group and a CTA an eighth of the keys; a unit of LPK lanes takes KB keys at a time (8 channels per lane and chunk, NCH chunks), with the
// keys' and the first values' rows requested together.  The KB * HB dot products are summed over the lanes by halving both (15 shuffles for 16 sums),
// which leaves each lane one score to finish.  The eight CTAs are joined through distributed shared memory in the same launch.
// In a step's graph at position 1000 (before: all heads of a row in one CTA, barriers between the phases of a 32-key block, a kernel for the join):
// 32 heads over 8 of 128, window 2048, 10.3 us (27.1 + 5.0); 16 over 4, chunks of 1024, 9.0 us (16.4 + 4.0); 16 heads of a latent of 512, 16.1 us
// (26.5 + 4.6); at position 300, 8 heads over 2, 9.3 us (11.5 + 3.6).  Keeping scores and a running softmax in registers with every loop unrolled
// took 22 us: thousands of instructions fetched for one trip through them.
#include <cooperative_groups.h>

#define XALM_SECONDARY_TU
#include "common.cuh"
#include "family.h"
#include "mix_ops.cuh"

namespace xalm {
namespace mix {

constexpr int SWO_CTAS = 8, SWO_KEYS = 512; // CTAs per cluster; keys a CTA scores before it takes their values

template <typename CT>
struct SwoRow; // eight channels as they lie in the cache
template <>
struct SwoRow<__nv_bfloat16> {
	uint4 r;
	__device__ __forceinline__ void load(const __nv_bfloat16* p) { r = *reinterpret_cast<const uint4*>(p); }
	__device__ __forceinline__ void clear() { r = make_uint4(0, 0, 0, 0); }
	__device__ __forceinline__ void get(float* x) const {
		x[0] = __uint_as_float(r.x << 16); x[1] = __uint_as_float(r.x & 0xffff0000u);
		x[2] = __uint_as_float(r.y << 16); x[3] = __uint_as_float(r.y & 0xffff0000u);
		x[4] = __uint_as_float(r.z << 16); x[5] = __uint_as_float(r.z & 0xffff0000u);
		x[6] = __uint_as_float(r.w << 16); x[7] = __uint_as_float(r.w & 0xffff0000u);
	}
};
template <>
struct SwoRow<float> {
	float4 a, b;
	__device__ __forceinline__ void load(const float* p) { a = *reinterpret_cast<const float4*>(p); b = *reinterpret_cast<const float4*>(p + 4); }
	__device__ __forceinline__ void clear() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
	__device__ __forceinline__ void get(float* x) const {
		x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
	}
};

__host__ __device__ constexpr int swo_threads(int nch) { return nch == 1 ? 512 : 256; } // registers: query and output take 16 * HB * NCH
__host__ __device__ constexpr size_t swo_smem_floats(int lpk, int nch, int hb) {
	const size_t dp = (size_t) lpk * 8 * nch;
	return (swo_threads(nch) / 32) * hb * dp + hb * dp + (size_t) hb * SWO_KEYS + 3 * hb; // warps' outputs | the CTA's | scores | m, l, alpha
}

template <typename CT, int LPK, int NCH, int HB>
__global__ void __launch_bounds__(swo_threads(NCH)) swa_one_kernel(SwaArgs a) {
	pdl_enter();
	namespace cg = cooperative_groups;
	constexpr int DP = LPK * 8 * NCH, NTH = swo_threads(NCH), UNITS = NTH / LPK, KB = sizeof(CT) == 2 ? (NCH <= 2 ? 4 : 2) : (NCH == 1 ? 2 : 1), NV = KB * HB;
	extern __shared__ __align__(16) float sm[];
	float* wo = sm;                        // NTH / 32 * HB * DP
	float* co = wo + NTH / 32 * HB * DP;   // HB * DP
	float* sc = co + HB * DP;              // HB * SWO_KEYS
	float* cm = sc + HB * SWO_KEYS;        // HB
	float* cl = cm + HB;
	float* ca = cl + HB;
	cg::cluster_group cluster = cg::this_cluster();
	const int rank = (int) cluster.block_rank(), sp = blockIdx.x / SWO_CTAS, t = blockIdx.z;
	const int H = a.H, G = a.G, d = a.d, dv = a.dv, rep = H / G, hgroups = (rep + HB - 1) / HB;
	const int g = blockIdx.y / hgroups, h0 = g * rep + blockIdx.y % hgroups * HB, nh = min(HB, (g + 1) * rep - h0);
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, unit = tid / LPK, ln = tid % LPK;
	if (t >= a.step->n) return; // the whole cluster leaves
	const int i = a.step->pos0 + t;
	const SwaKeys km = swa_keys(a, i);
	const int nk = km.ks + i - km.j_first + 1, parts = a.n_splits * SWO_CTAS, per = (nk + parts - 1) / parts;
	const int jb = min(nk, (sp * SWO_CTAS + rank) * per), je = min(nk, jb + per);
	const int ldk = a.ldk ? a.ldk : G * d, ldv = a.ldv ? a.ldv : G * dv;
	const CT* kc = reinterpret_cast<const CT*>(a.kc) + (size_t) g * d;
	const CT* vc = reinterpret_cast<const CT*>(a.vc) + (size_t) g * dv;
	auto load = [&](SwoRow<CT>(&r)[KB][NCH], const CT* base, int ld, int width, int j0) {
#pragma unroll
		for (int b = 0; b < KB; b++) {
			const CT* p = base + (size_t) km.slot(min(j0 + b * UNITS, je - 1)) * ld;
#pragma unroll
			for (int c = 0; c < NCH; c++) {
				const int col = (c * LPK + ln) * 8;
				if (col < width) r[b][c].load(p + col);
				else r[b][c].clear();
			}
		}
	};

	SwoRow<CT> kr[KB][NCH], vr[KB][NCH];
	if (jb < je) {
		load(kr, kc, ldk, d, jb + unit);
		load(vr, vc, ldv, dv, jb + unit);
	}
	float q[HB][NCH * 8], o[HB][NCH * 8] = {};
#pragma unroll
	for (int u = 0; u < HB; u++)
#pragma unroll
		for (int c = 0; c < NCH; c++) {
			const int col = (c * LPK + ln) * 8;
			SwoRow<float> x;
			if (col < d) x.load(a.q + (size_t) t * a.ldq + a.q_off + (size_t) (h0 + min(u, nh - 1)) * d + col);
			else x.clear();
			x.get(&q[u][c * 8]);
		}
	if (tid < HB) { cm[tid] = -INFINITY; cl[tid] = 0.f; }
	__syncthreads();

	for (int blk = jb; blk < je; blk += SWO_KEYS) {
		const int end = min(je, blk + SWO_KEYS);
		if (blk != jb) load(vr, vc, ldv, dv, blk + unit);
		for (int jj = blk; jj < end; jj += UNITS * KB) { // the same trips for every lane of a warp
			if (jj != jb) load(kr, kc, ldk, d, jj + unit);
			float v[NV];
#pragma unroll
			for (int b = 0; b < KB; b++) {
#pragma unroll
				for (int u = 0; u < HB; u++) v[b * HB + u] = 0.f;
#pragma unroll
				for (int c = 0; c < NCH; c++) {
					float x[8];
					kr[b][c].get(x);
#pragma unroll
					for (int u = 0; u < HB; u++)
#pragma unroll
						for (int e = 0; e < 8; e++) v[b * HB + u] = fmaf(q[u][c * 8 + e], x[e], v[b * HB + u]);
				}
			}
			int cnt = NV, first = 0; // this lane keeps the sums first .. first + cnt - 1
#pragma unroll
			for (int w = LPK / 2; w >= 1; w >>= 1) {
				if (cnt > 1) {
					cnt >>= 1;
					const bool up = ln & w;
#pragma unroll
					for (int x = 0; x < NV / 2; x++)
						if (x < cnt) {
							const float give = up ? v[x] : v[x + cnt], keep = up ? v[x + cnt] : v[x];
							v[x] = keep + __shfl_xor_sync(0xffffffffu, give, w);
						}
					if (up) first += cnt;
				} else v[0] += __shfl_xor_sync(0xffffffffu, v[0], w);
			}
#pragma unroll
			for (int x = 0; x < NV; x++)
				if (x < cnt) {
					const int u = (first + x) % HB, j = jj + unit + (first + x) / HB * UNITS, h = h0 + min(u, nh - 1);
					if (j < end) {
						float z = v[x] * a.scale;
						const float dist = (float) (i - km.pos(j));
						if (a.softcap > 0.f) z = a.softcap * tanhf(z / a.softcap);
						if (a.r1) z -= a.r1[h] * log1pf(a.r2[h] * dist);
						if (a.slope) z -= a.slope[h] * dist;
						sc[u * SWO_KEYS + j - blk] = z;
					}
				}
		}
		__syncthreads();
		if (warp < HB) { // softmax weights of the block, a warp per head
			float* s = sc + warp * SWO_KEYS;
			const int n = end - blk;
			float top = cm[warp];
#pragma unroll 4
			for (int x = lane; x < n; x += 32) top = fmaxf(top, s[x]);
			top = warp_max(top);
			const float at = top == -INFINITY ? 0.f : top;
			float sum = 0.f;
#pragma unroll 4
			for (int x = lane; x < n; x += 32) {
				const float p = expf(s[x] - at);
				s[x] = p;
				sum += p;
			}
			sum = warp_sum(sum);
			if (lane == 0) {
				const float keep = cm[warp] == -INFINITY ? 0.f : expf(cm[warp] - at);
				cl[warp] = fmaf(cl[warp], keep, sum);
				cm[warp] = top;
				ca[warp] = keep;
			}
		}
		__syncthreads();
		if (blk != jb)
#pragma unroll
			for (int u = 0; u < HB; u++)
#pragma unroll
				for (int e = 0; e < NCH * 8; e++) o[u][e] *= ca[u];
		for (int jj = blk; jj < end; jj += UNITS * KB) {
			if (jj != blk) load(vr, vc, ldv, dv, jj + unit);
#pragma unroll
			for (int b = 0; b < KB; b++) {
				const int j = jj + unit + b * UNITS;
				float p[HB];
#pragma unroll
				for (int u = 0; u < HB; u++) p[u] = j < end ? sc[u * SWO_KEYS + j - blk] : 0.f;
				if (j < end) // a row beyond the last key is a copy of it, which may hold an infinity
#pragma unroll
					for (int c = 0; c < NCH; c++) {
						float x[8];
						vr[b][c].get(x);
#pragma unroll
						for (int u = 0; u < HB; u++)
#pragma unroll
							for (int e = 0; e < 8; e++) o[u][c * 8 + e] = fmaf(p[u], x[e], o[u][c * 8 + e]);
					}
			}
		}
		__syncthreads(); // the scores are read
	}
	// ---- join the units of the CTA, which share their maximum ----
#pragma unroll
	for (int u = 0; u < HB; u++)
#pragma unroll
		for (int c = 0; c < NCH; c++) {
#pragma unroll
			for (int e = 0; e < 8; e++)
#pragma unroll
				for (int w = LPK; w < 32; w <<= 1) o[u][c * 8 + e] += __shfl_xor_sync(0xffffffffu, o[u][c * 8 + e], w);
			if (lane < LPK) {
				float4* dst = reinterpret_cast<float4*>(wo + ((size_t) warp * HB + u) * DP + (c * LPK + ln) * 8);
				dst[0] = make_float4(o[u][c * 8], o[u][c * 8 + 1], o[u][c * 8 + 2], o[u][c * 8 + 3]);
				dst[1] = make_float4(o[u][c * 8 + 4], o[u][c * 8 + 5], o[u][c * 8 + 6], o[u][c * 8 + 7]);
			}
		}
	__syncthreads();
	for (int x = tid; x < nh * DP; x += NTH) {
		float v = 0.f;
#pragma unroll 8
		for (int y = 0; y < NTH / 32; y++) v += wo[(size_t) y * HB * DP + x];
		co[x] = v;
	}
	cluster.sync();
	// ---- join the CTAs of the cluster: each writes its share of the heads' columns ----
	const int total = nh * dv, share = (total + SWO_CTAS - 1) / SWO_CTAS;
	for (int x = rank * share + tid; x < min(total, (rank + 1) * share); x += NTH) {
		const int u = x / dv, c = x % dv, h = h0 + u;
		float ms[SWO_CTAS], ls[SWO_CTAS], os[SWO_CTAS], top = -INFINITY, num = 0.f, den = 0.f;
#pragma unroll
		for (int r = 0; r < SWO_CTAS; r++) {
			ms[r] = cluster.map_shared_rank(cm, r)[u];
			ls[r] = cluster.map_shared_rank(cl, r)[u];
			os[r] = cluster.map_shared_rank(co, r)[u * DP + c];
			top = fmaxf(top, ms[r]);
		}
		const float at = top == -INFINITY ? 0.f : top;
#pragma unroll 2
		for (int r = 0; r < SWO_CTAS; r++) {
			const float w = expf(ms[r] - at);
			num = fmaf(w, os[r], num);
			den = fmaf(w, ls[r], den);
		}
		if (a.n_splits == 1) {
			float v = swa_finish(a, h, num, den, top);
			if (a.gate) v *= swa_gate(a, t, h, c);
			a.out[(size_t) t * (a.ldo ? a.ldo : H * dv) + (size_t) h * dv + c] = v;
		} else {
			a.part_o[((size_t) t * a.n_splits + sp) * (H * dv) + (size_t) h * dv + c] = num;
			if (c == 0) {
				float* pml = a.part_ml + ((size_t) t * a.n_splits + sp) * (H * 2) + 2 * h;
				pml[0] = top;
				pml[1] = den;
			}
		}
	}
	cluster.sync(); // no CTA leaves while another reads its shared memory
}

template <typename CT, int LPK, int NCH, int HB>
static int launch_swa_one_inst(const SwaArgs& a, int rows, cudaStream_t s) {
	const size_t smem = swo_smem_floats(LPK, NCH, HB) * 4;
	if (smem > 48 * 1024) XALM_CUDA_CHECK(cudaFuncSetAttribute(swa_one_kernel<CT, LPK, NCH, HB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
	cudaLaunchConfig_t cfg = {};
	const int rep = a.H / a.G;
	cfg.gridDim = dim3((unsigned) (SWO_CTAS * a.n_splits), (unsigned) (a.G * ((rep + HB - 1) / HB)), (unsigned) rows);
	cfg.blockDim = dim3(swo_threads(NCH));
	cfg.dynamicSmemBytes = smem;
	cfg.stream = s;
	cudaLaunchAttribute at[2];
	at[0].id = cudaLaunchAttributeClusterDimension;
	at[0].val.clusterDim.x = SWO_CTAS; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
	at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at[1].val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = at;
	cfg.numAttrs = rows == 1 && pdl_next(s) ? 2 : 1;
	const cudaError_t e = cudaLaunchKernelEx(&cfg, swa_one_kernel<CT, LPK, NCH, HB>, a);
	if (e != cudaSuccess) return set_error(XALM_ERR_CUDA, "swa_one launch failed: %s", cudaGetErrorString(e));
	return launch_check("swa_one");
}

// lanes per key, chunks and heads by the wider of d and dv, and by the heads of a group
template <typename CT>
static int launch_swa_one_typed(const SwaArgs& a, int rows, cudaStream_t s) {
	const int w = std::max(a.d, a.dv), rep = a.H / a.G;
#define XALM_SWO(LPK_, NCH_, HB_) return launch_swa_one_inst<CT, LPK_, NCH_, HB_>(a, rows, s)
	if (w > 512) { if (rep >= 2) XALM_SWO(32, 3, 2); XALM_SWO(32, 3, 1); }
	if (w > 256) { if (rep >= 2) XALM_SWO(32, 2, 2); XALM_SWO(32, 2, 1); }
	if (w > 128) { if (rep >= 3) XALM_SWO(32, 1, 4); if (rep == 2) XALM_SWO(32, 1, 2); XALM_SWO(32, 1, 1); }
	if (w > 64) { if (rep >= 3) XALM_SWO(16, 1, 4); if (rep == 2) XALM_SWO(16, 1, 2); XALM_SWO(16, 1, 1); }
	if (rep >= 3) XALM_SWO(8, 1, 4);
	if (rep == 2) XALM_SWO(8, 1, 2);
	XALM_SWO(8, 1, 1);
#undef XALM_SWO
}

int launch_swa_one(const SwaArgs& a, int rows, bool cache_f32, cudaStream_t s) {
	return cache_f32 ? launch_swa_one_typed<float>(a, rows, s) : launch_swa_one_typed<__nv_bfloat16>(a, rows, s);
}

} // namespace mix
} // namespace xalm
