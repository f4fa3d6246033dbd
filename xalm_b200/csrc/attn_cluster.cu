// attn_cluster.cu — attention of one query token over the fp16 KV ring (the semantics of attention.cuh) on the tensor cores: a cluster of CTAs per kv head.
//
// Bound: latency.  A step's keys and values are 1 to 17 MB a layer (0.2 to 2.6 us of memory time) that the projection before has pulled into L2.  The split
// kernel of attention.cuh walks them with fp32 FMAs (24 instructions per key and head for 128 channels, 177 registers) and joins its splits by a store, a fence, a
// ticket and the last CTA's loads.  Here a warp takes 16 slots at a time with ldmatrix and m16n8k16: one product covers all query heads of the kv head, about
// 250 instructions for 16 keys of four heads; the slots go round the cluster's warps, so that short contexts use all of them; what this step does not write is fetched
// before the kernel waits for the projection; and the parts are pushed to the CTA that owns their channels through distributed shared memory, one barrier in all.
// Queries and probabilities are fp32 values: each enters as three fp16 planes, scaled by powers of two, whose products with the cache's fp16 are exact.  Sums
// of 16 products start from zero and are added in round-to-nearest as a tree, since the tensor cores' own additions truncate.  Distance from float64 over
// 20 to 3002 keys and queries of deviation 0.3, 1 and 3: 0.99 times the split kernel's (0.86 to 1.13).  A warp that meets a score or a sum that is not finite
// does its keys again in fp32 FMAs, so that an infinity goes where it goes there (its zero planes would spread it); a NaN score, wherever its key lies, makes its head NaN.
// Per token, with the split kernel and with this one: 32 layers of q8_0 of width 4096 at position 3001 1854 -> 1800 us, 8 of q4_0 at 700 398 -> 374, 6 of bf16 at width 2048
// and position 1777 267 -> 249, 4 of q8_0 at width 1024 116 -> 108.  Tried and not faster: rings of the neighbouring products cut so that this kernel's CTAs fit beside
// them (no difference).
#define XALM_SECONDARY_TU
#include "attention.cuh"
#include "family.h"

namespace xalm {

constexpr int AC_NW = 4, AC_KEYS = 16, AC_MAX_CTAS = 16; // warps per CTA; slots of a unit (one product's keys); most CTAs of a cluster
constexpr float AC_PSCALE = 16384.f;                     // probabilities enter the tensor cores times 2^14: their third fp16 plane stays above the subnormals' step
__host__ __device__ constexpr int ac_stages(int hd) { return hd >= 256 ? 1 : hd == 128 ? 2 : 4; } // units a warp holds: 64 KB a CTA at most
__host__ __device__ constexpr size_t ac_ring_bytes(int hd) { return (size_t) AC_NW * ac_stages(hd) * 2 * AC_KEYS * hd * 2; }
__host__ __device__ constexpr size_t ac_smem_bytes(int hd, int gp) {
	return ac_ring_bytes(hd) + (size_t) 4 * gp * hd * 2 + ((size_t) hd * gp + AC_MAX_CTAS * 8) * 4 + (size_t) AC_MAX_CTAS * gp * 8 + (size_t) AC_NW * gp * 8 + gp * 4;
}

__device__ __forceinline__ void ac_ldsm4(uint32_t (&r)[4], uint32_t addr) {
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ac_ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ac_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
	asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
	    : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
	    : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// a fp32 value as three fp16 whose sum it is (down to 2^-25)
__device__ __forceinline__ void ac_split(float x, __half& hi, __half& mid, __half& lo) {
	hi = __float2half_rn(x);
	const float r = x - __half2float(hi);
	mid = __float2half_rn(r);
	lo = __float2half_rn(r - __half2float(mid));
}
__device__ __forceinline__ uint32_t ac_pack(__half a, __half b) {
	const __half2 h = __halves2half2(a, b);
	return *reinterpret_cast<const uint32_t*>(&h);
}
// byte offset of 16-byte piece `piece` of row `row` (HD fp16): the eight rows of an 8 x 8 matrix fall on different banks
template <int HD>
__device__ __forceinline__ uint32_t ac_at(int row, int piece) {
	return HD >= 64 ? (uint32_t) (row * HD * 2 + ((piece ^ (row & 7)) << 4)) : (uint32_t) (row * HD * 2 + ((piece ^ ((row >> 1) & 3)) << 4));
}
__device__ __forceinline__ void ac_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void ac_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t ac_peer(const void* p, int rank) {
	uint32_t r;
	asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
	return r;
}
template <int N>
__device__ __forceinline__ void ac_cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

enum { AC_EARLY = 0, AC_LATE = 1, AC_ALL = 2 }; // rows that this step's QKV kernel does not write | those it does | all

template <int HD, int GP, bool TL> // GP: query heads of a kv head; TL: with stamps of the in-kernel timeline, as the split kernel's (code of their own: looked up at every launch they took 0.2 us a layer)
__global__ void __launch_bounds__(AC_NW * 32, 4) attn_cluster_kernel(const AttnArgs a) {
	constexpr int NW = AC_NW, NST = ac_stages(HD), KEYS = AC_KEYS, NTH = NW * 32, PIECES = HD / 8, TILE = KEYS * HD; // TILE: halves of a unit's keys
	extern __shared__ __align__(128) uint8_t smem[];
	__half* ring = reinterpret_cast<__half*>(smem);                    // [NW][NST][K | V][KEYS][HD]
	__half* qp = ring + (size_t) NW * NST * 2 * TILE;                  // [4 GP][HD]: the queries' planes
	float* cpart = reinterpret_cast<float*>(qp + 4 * GP * HD);         // [C][HD / C * GP (+ 8)]: the cluster's parts of this CTA's channels
	float* cml = cpart + HD * GP + AC_MAX_CTAS * 8;                    // [C][GP][2]
	float* wml = cml + AC_MAX_CTAS * GP * 2;                           // [NW][GP][2]
	float* qsc = wml + NW * GP * 2;                                    // [GP]

	pdl_launch_dependents();
	ac_cluster_arrive(); // (1) every CTA of the cluster runs
	const int C = gridDim.x, rank = blockIdx.x, kvh = blockIdx.y; // one cluster per kv head
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
	__shared__ unsigned long long tl_sm[TL ? 2 : 1]; // the start, the wait's end (no registers are left)
	if (TL && (tid | rank | kvh) == 0) tl_sm[0] = gtime();
	if (tid == 0) l2_prefetch_slice(a.pf_ptr, a.pf_bytes, kvh * C + rank, C * (int) gridDim.y);

	const bool fixed = a.kv_len_fixed >= 0;
	const int kv_len = fixed ? a.kv_len_fixed : a.step->kv_len, kv_pos = fixed ? -1 : a.step->kv_pos, kv_sink = fixed ? 0 : a.step->kv_sink;
	const int nu = (kv_len + KEYS - 1) / KEYS, u0 = rank + C * warp, du = C * NW; // this warp's units: u0, u0 + du, ...
	const int kv_stride = a.n_kv_heads * HD;
	const __half* kbase = a.k_cache + (size_t) kvh * HD;
	const __half* vbase = a.v_cache + (size_t) kvh * HD;
	auto fetch = [&](int u, int stage, int what) {
		const uint32_t dst = smem_u32(ring + (size_t) (warp * NST + stage) * 2 * TILE);
#pragma unroll 4
		for (int i = 0; i < 2 * KEYS * PIECES / 32; i++) {
			const int x = i * 32 + lane, kv = x / (KEYS * PIECES), row = x / PIECES % KEYS, piece = x % PIECES, slot = u * KEYS + row;
			const bool late = slot == kv_pos || slot < kv_sink;
			if (what != AC_ALL && late != (what == AC_LATE)) continue;
			const __half* src = (kv ? vbase : kbase) + (size_t) min(slot, kv_len - 1) * kv_stride + piece * 8;
			asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + kv * TILE * 2 + ac_at<HD>(row, piece)), "l"(src), "r"(slot < kv_len ? 16 : 0) : "memory");
		}
	};
	auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
	// What the running QKV kernel does not write is fetched before this kernel waits for it (the step's parameters were written before the token began)
#pragma unroll
	for (int j = 0; j < NST; j++)
		if (u0 + j * du < nu) fetch(u0 + j * du, j, AC_EARLY);
	commit();

	pdl_wait();
	if (TL && (tid | rank | kvh) == 0) tl_sm[1] = gtime();
#pragma unroll
	for (int j = 0; j < NST; j++) {
		const int u = u0 + j * du;
		if (u < nu && (kv_pos / KEYS == u || u * KEYS < kv_sink)) fetch(u, j, AC_LATE);
	}
	commit();

	// ---- queries: scaled by a power of two to [2^13, 2^14) at most, three fp16 planes (rows plane * GP + head; the fourth is zero) ----
	for (int h = warp; h < GP; h += NW) {
		constexpr int E = HD / 32;
		float q[E];
		uint32_t top = 0;
#pragma unroll
		for (int e = 0; e < E; e++) {
			q[e] = __ldcg(a.q + (size_t) (kvh * GP + h) * HD + lane + 32 * e);
			top = max(top, __float_as_uint(q[e]) & 0x7fffffffu);
		}
		top = __reduce_max_sync(0xffffffffu, top) >> 23;
		const int ex = top >= 254 ? 140 : max((int) top, 14); // (not finite, or nearly: as it is; the scores say so below)
		const float up = __uint_as_float((uint32_t) (267 - ex) << 23);
		if (lane == 0) qsc[h] = __uint_as_float((uint32_t) (ex - 13) << 23);
#pragma unroll
		for (int e = 0; e < E; e++) {
			const int dim = lane + 32 * e;
			__half pl[4];
			ac_split(q[e] * up, pl[0], pl[1], pl[2]);
			pl[3] = __ushort_as_half(0);
#pragma unroll
			for (int p = 0; p < 4; p++) *reinterpret_cast<__half*>(reinterpret_cast<uint8_t*>(qp) + ac_at<HD>(p * GP + h, dim / 8) + dim % 8 * 2) = pl[p];
		}
	}
	__syncthreads();

	const float inv_sqrt = 1.0f / sqrtf((float) HD);
	const float scale = qsc[g % GP];
	const int mid = lane >> 3, mr = lane & 7; // ldmatrix: this lane names row mr of matrix mid
	const uint32_t qa = smem_u32(qp);
	float m = -CUDART_INF_F, l = 0.f, acc[HD / 16][4];
#pragma unroll
	for (int i = 0; i < HD / 16; i++)
#pragma unroll
		for (int e = 0; e < 4; e++) acc[i][e] = 0.f;
	bool bad = false; // a score or a sum that is not finite
	for (int j = 0, u = u0; u < nu; j++, u += du) {
		if (j == 0) ac_cp_wait<0>();
		else if (j >= NST) ac_cp_wait<NST - 1>();
		__syncwarp();
		const uint32_t ka = smem_u32(ring + (size_t) (warp * NST + j % NST) * 2 * TILE), va = ka + TILE * 2;
		// ---- scores: (planes x heads) . keys, 16 channels at a time from zero, added in round-to-nearest (the tensor cores' own additions truncate) as a tree ----
		constexpr int KS = HD / 16;
		float s[2][4], sum[4][2][4], s2[2][4] = {}; // sum[i]: a pending sum of 2^i steps
#pragma unroll
		for (int ks = 0; ks < KS; ks++) {
			uint32_t qf[4], kf[4];
			ac_ldsm4(kf, ka + ac_at<HD>((mid >> 1) * 8 + mr, 2 * ks + (mid & 1)));
			ac_ldsm4(qf, qa + ac_at<HD>((mid & 1) * 8 + mr, 2 * ks + (mid >> 1)));
#pragma unroll
			for (int n = 0; n < 2; n++) {
				float d[4] = {};
				ac_mma(d, qf, kf[2 * n], kf[2 * n + 1]);
				int lev = 0;
#pragma unroll
				for (; lev < 4 && (ks >> lev & 1); lev++)
#pragma unroll
					for (int e = 0; e < 4; e++) d[e] += sum[lev][n][e];
#pragma unroll
				for (int e = 0; e < 4; e++) {
					if (ks == KS - 1) s[n][e] = d[e];
					else sum[lev][n][e] = d[e];
				}
			}
			if (GP == 8) {
				ac_ldsm4(qf, qa + ac_at<HD>(16 + (mid & 1) * 8 + mr, 2 * ks + (mid >> 1)));
#pragma unroll
				for (int n = 0; n < 2; n++) {
					float d[4] = {};
					ac_mma(d, qf, kf[2 * n], kf[2 * n + 1]);
#pragma unroll
					for (int e = 0; e < 2; e++) s2[n][e] += d[e];
				}
			}
		}
		// this lane: head g % GP, keys 8 n + 2 t + e
		float p[2][2], top = m;
#pragma unroll
		for (int n = 0; n < 2; n++)
#pragma unroll
			for (int e = 0; e < 2; e++) {
				float v;
				if (GP == 8) v = s[n][e] + (s[n][e + 2] + s2[n][e]);
				else { // lanes g < 4 hold the hi and lo planes, the others the mid one: small planes first
					const float x = g < 4 ? s[n][e + 2] : s[n][e], other = __shfl_xor_sync(0xffffffffu, s[n][e], 16);
					v = (x + __shfl_xor_sync(0xffffffffu, x, 16)) + (g < 4 ? s[n][e] : other);
				}
				v = v * scale * inv_sqrt;
				const bool in = u * KEYS + 8 * n + 2 * t + e < kv_len;
				bad |= in && !(fabsf(v) < CUDART_INF_F);
				p[n][e] = in ? v : -CUDART_INF_F;
				top = fmaxf(top, p[n][e]);
			}
		top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
		top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
		const float corr = expf(m - top);
		m = top;
		l *= corr;
		uint32_t ph[2], pm[2], pl[2];
#pragma unroll
		for (int n = 0; n < 2; n++) {
			__half hi[2], mi[2], lo[2];
#pragma unroll
			for (int e = 0; e < 2; e++) {
				const float x = expf(p[n][e] - top);
				l += x;
				ac_split(x * AC_PSCALE, hi[e], mi[e], lo[e]);
			}
			ph[n] = ac_pack(hi[0], hi[1]);
			pm[n] = ac_pack(mi[0], mi[1]);
			pl[n] = ac_pack(lo[0], lo[1]);
		}
		if (__any_sync(0xffffffffu, corr != 1.f)) { // columns 2 t and 2 t + 1 of the output: heads of lanes 8 t and 8 t + 4
			const float c0 = __shfl_sync(0xffffffffu, corr, 8 * t), c1 = __shfl_sync(0xffffffffu, corr, 8 * t + 4);
#pragma unroll
			for (int i = 0; i < HD / 16; i++) { acc[i][0] *= c0; acc[i][1] *= c1; acc[i][2] *= c0; acc[i][3] *= c1; }
		}
		if (GP == 4) { // columns 0-3: heads' hi planes, 4-7: their mid planes; the lo planes in a product of their own
#pragma unroll
			for (int n = 0; n < 2; n++) {
				if (g >= 4) { ph[n] = pm[n]; pl[n] = 0; }
			}
		}
		// ---- values: (channels x keys) . (keys x heads), small planes first ----
#pragma unroll
		for (int i = 0; i < HD / 16; i++) {
			uint32_t vf[4];
			ac_ldsm4_t(vf, va + ac_at<HD>((mid >> 1) * 8 + mr, 2 * i + (mid & 1)));
			float d[4] = {};
			ac_mma(d, vf, pl[0], pl[1]);
			if (GP == 8) ac_mma(d, vf, pm[0], pm[1]);
			ac_mma(d, vf, ph[0], ph[1]);
#pragma unroll
			for (int e = 0; e < 4; e++) acc[i][e] += d[e];
		}
		__syncwarp();
		if (u + NST * du < nu) fetch(u + NST * du, j % NST, AC_ALL);
		commit();
	}
	ac_cp_wait<0>();
	l += __shfl_xor_sync(0xffffffffu, l, 1);
	l += __shfl_xor_sync(0xffffffffu, l, 2);
#pragma unroll
	for (int i = 0; i < HD / 16; i++)
#pragma unroll
		for (int e = 0; e < 4; e++) bad |= !(fabsf(acc[i][e]) < CUDART_INF_F);

	// ---- the warp's part: [channel][head] floats where its keys lay, maxima and sums ----
	float* wp = reinterpret_cast<float*>(ring + (size_t) warp * NST * 2 * TILE);
	__syncwarp();
	if (__any_sync(0xffffffffu, bad)) { // again in fp32 products, so that an infinity or a NaN goes where it goes there
		constexpr int E = HD / 32;
#pragma unroll 1
		for (int h = 0; h < GP; h++) {
			float o[E] = {}, mh = -CUDART_INF_F, lh = 0.f;
#pragma unroll 1
			for (int u = u0; u < nu; u += du)
#pragma unroll 1
				for (int slot = u * KEYS; slot < min(kv_len, (u + 1) * KEYS); slot++) {
					float x = 0.f;
#pragma unroll
					for (int e = 0; e < E; e++)
						x += __ldcg(a.q + (size_t) (kvh * GP + h) * HD + lane + 32 * e) * __half2float(__ldcg(kbase + (size_t) slot * kv_stride + lane + 32 * e));
					x = warp_sum(x) * inv_sqrt;
					const float mn = fmaxf(mh, x); // (-inf also where the first score is a NaN)
					const float corr = mh == mn ? 1.f : expf(mh - mn), pr = x == -CUDART_INF_F ? 0.f : expf(x - mn);
					lh = lh * corr + pr;
					mh = mn;
#pragma unroll
					for (int e = 0; e < E; e++) o[e] = o[e] * corr + pr * __half2float(__ldcg(vbase + (size_t) slot * kv_stride + lane + 32 * e));
				}
#pragma unroll
			for (int e = 0; e < E; e++) wp[(lane + 32 * e) * GP + h] = o[e] * AC_PSCALE;
			if (lane == 0) { wml[(warp * GP + h) * 2] = mh; wml[(warp * GP + h) * 2 + 1] = lh; }
		}
	} else {
		if (GP == 4) { // the planes joined: lanes t < 2 keep channel g, the others channel g + 8, of heads 2 (t % 2) and the next
#pragma unroll
			for (int i = 0; i < HD / 16; i++) {
				const bool up = t >= 2;
				const float k0 = (up ? acc[i][2] : acc[i][0]) + __shfl_xor_sync(0xffffffffu, up ? acc[i][0] : acc[i][2], 2);
				const float k1 = (up ? acc[i][3] : acc[i][1]) + __shfl_xor_sync(0xffffffffu, up ? acc[i][1] : acc[i][3], 2);
				*reinterpret_cast<float2*>(wp + (16 * i + g + (up ? 8 : 0)) * 4 + 2 * (t & 1)) = make_float2(k0, k1);
			}
		} else {
#pragma unroll
			for (int i = 0; i < HD / 16; i++) {
				*reinterpret_cast<float2*>(wp + (16 * i + g) * GP + 2 * t) = make_float2(acc[i][0], acc[i][1]);
				*reinterpret_cast<float2*>(wp + (16 * i + g + 8) * GP + 2 * t) = make_float2(acc[i][2], acc[i][3]);
			}
		}
		if (t == 0 && g < GP) { wml[(warp * GP + g) * 2] = m; wml[(warp * GP + g) * 2 + 1] = l; }
	}
	__syncthreads();
	// ---- the CTA's part, sent to the CTAs that own its channels ----
	ac_cluster_wait(); // (1)
	const int own = HD / C, stride = own * GP + 8; // channels of a CTA; floats between two CTAs' parts of them
	auto weight = [](float mw, float top) { return mw == -CUDART_INF_F ? 0.f : expf(mw - top); };
	for (int x = tid; x < HD * GP / 4; x += NTH) {
		const int dim = x / (GP / 4), h0 = x % (GP / 4) * 4;
		float v[4];
#pragma unroll
		for (int h = 0; h < 4; h++) {
			float mw[NW], top = -CUDART_INF_F;
#pragma unroll
			for (int w = 0; w < NW; w++) { mw[w] = wml[(w * GP + h0 + h) * 2]; top = fmaxf(top, mw[w]); }
			v[h] = 0.f;
#pragma unroll
			for (int w = 0; w < NW; w++) v[h] += weight(mw[w], top) * reinterpret_cast<const float*>(ring + (size_t) w * NST * 2 * TILE)[dim * GP + h0 + h];
		}
		asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(ac_peer(cpart + rank * stride + dim % own * GP + h0, dim / own)), "f"(v[0]), "f"(v[1]), "f"(v[2]),
		             "f"(v[3])
		             : "memory");
	}
	for (int x = tid; x < C * GP; x += NTH) {
		const int h = x % GP;
		float top = -CUDART_INF_F, sum = 0.f;
#pragma unroll
		for (int w = 0; w < NW; w++) top = fmaxf(top, wml[(w * GP + h) * 2]);
#pragma unroll
		for (int w = 0; w < NW; w++) sum += weight(wml[(w * GP + h) * 2], top) * wml[(w * GP + h) * 2 + 1];
		asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(ac_peer(cml + (rank * GP + h) * 2, x / GP)), "f"(top), "f"(sum) : "memory");
	}
	ac_cluster_arrive(); // (2) every part has arrived; nothing of this CTA's is read by another after it
	ac_cluster_wait();
	// ---- the cluster's parts joined: four lanes per output ----
	for (int x0 = 0; x0 < own * GP; x0 += NTH / 4) {
		const int x = x0 + tid / 4, h = x % GP, part = tid % 4;
		const bool in = x < own * GP;
		float top = -CUDART_INF_F, num = 0.f, den = 0.f;
		for (int c = part; in && c < C; c += 4) top = fmaxf(top, cml[(c * GP + h) * 2]);
		top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
		top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
		for (int c = part; in && c < C; c += 4) {
			const float w = weight(cml[(c * GP + h) * 2], top);
			num += w * cpart[c * stride + x];
			den += w * cml[(c * GP + h) * 2 + 1];
		}
		num += __shfl_xor_sync(0xffffffffu, num, 1);
		den += __shfl_xor_sync(0xffffffffu, den, 1);
		num += __shfl_xor_sync(0xffffffffu, num, 2);
		den += __shfl_xor_sync(0xffffffffu, den, 2);
		if (in && part == 0) a.out[(size_t) (kvh * GP + h) * HD + rank * own + x / GP] = num * (1.f / AC_PSCALE) / den;
	}
	if (TL && (tid | rank | kvh) == 0 && a.tl->buf) {
		const unsigned int slot = atomicAdd(&a.tl->count, 1u);
		unsigned long long* r = a.tl->buf + 4 * (size_t) slot;
		if (slot < a.tl->cap) { r[0] = 300; r[1] = tl_sm[0]; r[2] = tl_sm[1]; r[3] = gtime(); }
	}
}

template <int HD, int GP, bool TL = false>
static cudaError_t ac_config(int n_kv, int C, cudaStream_t s, bool pdl, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
	auto kern = attn_cluster_kernel<HD, GP, TL>;
	cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) ac_smem_bytes(HD, GP));
	if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
	*cfg = {};
	cfg->gridDim = dim3((unsigned) C, (unsigned) n_kv);
	cfg->blockDim = dim3(AC_NW * 32);
	cfg->dynamicSmemBytes = ac_smem_bytes(HD, GP);
	cfg->stream = s;
	at[0].id = cudaLaunchAttributeClusterDimension;
	at[0].val.clusterDim.x = (unsigned) C; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
	at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	at[1].val.programmaticStreamSerializationAllowed = 1;
	cfg->attrs = at;
	cfg->numAttrs = pdl ? 2 : 1;
	return e;
}
template <int HD, int GP>
static int ac_size(int n_kv) {
	int sms = 148, dev = 0;
	if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
	for (int C = AC_MAX_CTAS; C >= 4 && n_kv > 0; C /= 2) {
		if (C * n_kv > sms) continue;
		cudaLaunchConfig_t cfg;
		cudaLaunchAttribute at[2];
		int n = 0;
		if (ac_config<HD, GP>(n_kv, C, 0, false, &cfg, at) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, attn_cluster_kernel<HD, GP, false>, &cfg) != cudaSuccess) {
			cudaGetLastError();
			continue;
		}
		if (n >= n_kv) return C;
	}
	return 0;
}

#define XALM_AC_CASES(CALL)                                                              \
	if (G == 4 && head_dim == 32) { CALL(32, 4); }                                       \
	if (G == 4 && head_dim == 64) { CALL(64, 4); }                                       \
	if (G == 4 && head_dim == 128) { CALL(128, 4); }                                     \
	if (G == 8 && head_dim == 32) { CALL(32, 8); }                                       \
	if (G == 8 && head_dim == 64) { CALL(64, 8); }                                       \
	if (G == 8 && head_dim == 128) { CALL(128, 8); }                                     \
	if (G == 8 && head_dim == 256) { CALL(256, 8); }

// CTAs per kv head so that all clusters run at once on the current device; 0: the split kernel is the faster one for these heads.  Alone, back to back, buffers
// beyond L2 (split kernel / this one, us): four heads of 128 over 8 kv heads 10.3 / 8.2 at 500 keys, 14.4 / 12.4 at 4096, 28.7 / 28.7 at 16384, 47 / 51 at 32768;
// eight heads 14.4 / 10.3, 20.5 / 16.1, 49 / 35, 84 / 59; two heads 8.3 / 8.3, 12.4 / 12.3, 22.6 / 28.7; one head 10.1 / 10.3, 22.6 / 22.6.  Of 256 channels: eight
// heads 26.6 / 14.4, 41 / 29, four 14.4 / 11.4, 20.5 / 22.6.  Operands in L2, 1 to 32 kv heads of 32 and 64 channels: four heads 0.55 to 0.95 of the split kernel's
// time up to 4096 keys, 0.88 to 1.1 at 16384; eight heads 0.4 to 0.9.  The line for four heads is one of capacity, since a captured step serves every position.
// From 38 kv heads on a cluster has one or two CTAs, 4 or 8 warps, and short contexts lose (100 keys, 128 channels, four heads: 74 kv heads 7.0 / 8.2, 80 7.0 / 12.2;
// eight heads 10.6 / 12.5, 10.4 / 19.9): the split kernel's.
int attn_cluster_size(int head_dim, int G, int n_kv_heads, int max_kv_len) {
	if (G == 4 && max_kv_len > 16384) return 0;
#define XALM_AC_SIZE(HD_, GP_) return ac_size<HD_, GP_>(n_kv_heads)
	XALM_AC_CASES(XALM_AC_SIZE)
#undef XALM_AC_SIZE
	return 0;
}

// C: attn_cluster_size's answer
int launch_attn_cluster(const AttnArgs& a, int head_dim, int G, int C, cudaStream_t s, bool pdl) {
	cudaError_t e = cudaErrorInvalidValue;
	cudaLaunchConfig_t cfg;
	cudaLaunchAttribute at[2];
#define XALM_AC_LAUNCH_TL(HD_, GP_, TL_)                                                \
	e = ac_config<HD_, GP_, TL_>(a.n_kv_heads, C, s, pdl, &cfg, at);                    \
	if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, attn_cluster_kernel<HD_, GP_, TL_>, a);
#define XALM_AC_LAUNCH(HD_, GP_)                                                        \
	if (a.tl) { XALM_AC_LAUNCH_TL(HD_, GP_, true) }                                     \
	else { XALM_AC_LAUNCH_TL(HD_, GP_, false) }
	XALM_AC_CASES(XALM_AC_LAUNCH)
#undef XALM_AC_LAUNCH
#undef XALM_AC_LAUNCH_TL
	if (e != cudaSuccess) return set_error(XALM_ERR_CUDA, "attention launch failed: %s", cudaGetErrorString(e));
	return XALM_OK;
}

} // namespace xalm
