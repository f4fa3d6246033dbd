// delta_chunk.cu — the gated delta rule of delta_ops.cuh for passes of many tokens, DC_L tokens at a time.
//
//   S_t = g_t S_{t-1} + k_t u_t^T,   u_t = beta_t (v_t - g_t S_{t-1}^T k_t),   o_t = S_t^T q_t
//
// With D[t, s] = prod_{s < r <= t} g_r inside a chunk, G_t = prod_{r <= t} g_r and S_0 the state before the chunk
//   u_t = U_t - S_0^T W_t:   U_t = beta_t v_t - sum_{s < t} A[t, s] U_s,   W_t = beta_t G_t k_t - sum_{s < t} A[t, s] W_s,   A[t, s] = beta_t D[t, s] k_t . k_s
//   o_t = G_t S_0^T q_t + sum_{s <= t} P[t, s] u_s,   P[t, s] = D[t, s] q_t . k_s,   S = G_L S_0 + sum_s D[L, s] k_s u_s^T
// (the rule's products of Householder-like steps written as one triangular system: Yang et al., "Parallelizing linear transformers with the delta rule over
// sequence length", 2024).
//   delta_local_kernel    per chunk and head: A, P, then U and W by forward substitution, a thread per column
//   delta_states_kernel   per head and group of value channels, chunk after chunk: u, o and the state as products of small matrices in shared memory
//   delta_finish_kernel   per-head norm and gate of o; the convolutions' state
// All in fp32 FMAs, decays as products (no quotients, no logarithms).  Products with s > t are not formed, so that an infinity or a NaN stays with the
// tokens that see it.
//
// Bound: the chain over the chunks in delta_states_kernel, 4 us (8 heads of 64 x 128) to 7 us (16 of 128 x 128) a chunk for three products with a barrier
// each; then the FMAs.  Scan -> the three kernels, caches flushed: 1024 tokens of 8 heads of 64 x 128 509 -> 18 + 65 + 7 us, 1000 tokens of 16 heads of
// 128 x 128 777 -> 36 + 111 + 7 us.
#define XALM_SECONDARY_TU
#include "common.cuh"
#include "family.h"
#include "delta_ops.cuh"

namespace xalm {
namespace mix {

constexpr int DC_L = 64, DC_DV = 128, DC_TH = 256; // tokens of a chunk, value channels (the rest is zero), threads

static inline int dc_dim(int d) { return d <= 64 ? 64 : 128; }
struct DcWs { // per chunk and head: U (DC_L, DC_DV) | W (DC_L, D) | P (DC_L, DC_L) | G, then D[L, s] (2 DC_L)
	float *u, *w, *p, *g;
};
__host__ __device__ inline DcWs dc_ws(float* ws, int chunks, int H, int D) {
	const size_t n = (size_t) chunks * H;
	DcWs w;
	w.u = ws;
	w.w = w.u + n * DC_L * DC_DV;
	w.p = w.w + n * DC_L * D;
	w.g = w.p + n * DC_L * DC_L;
	return w;
}
size_t delta_chunk_floats(int H, int d, int dv, int rows) {
	if (d > 128 || dv > DC_DV || rows < DELTA_CHUNK_ROWS) return 0;
	return (size_t) ((rows + DC_L - 1) / DC_L) * H * (DC_L * (DC_DV + dc_dim(d) + DC_L) + 2 * DC_L);
}

__device__ __forceinline__ float4 dc_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void dc_cp16(float* dst, const float* src, bool in) { // zeros where there is nothing
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
#define DC_COMMIT() asm volatile("cp.async.commit_group;" ::: "memory")
#define DC_WAIT(n_) asm volatile("cp.async.wait_group %0;" ::"n"(n_) : "memory")

// two CTAs per SM at D = 128: 114 KB each
__host__ __device__ constexpr size_t dc_local_smem(int D) { return sizeof(float) * (2 * (size_t) DC_L * D + (size_t) DC_L * DC_L + (size_t) DC_L * DC_DV + 3 * DC_L); }

// grid (chunks, H)
template <int D>
__global__ void __launch_bounds__(DC_TH, 2) delta_local_kernel(DeltaArgs a, int chunks) {
	extern __shared__ __align__(16) float sm[];
	float *ks = sm, *qs = ks + DC_L * D;    // (token, channel), 16-byte pieces of a row in places piece ^ (row % 8)
	float* M = qs + DC_L * D;               // (t, s): decays, then A
	float* xu = M + DC_L * DC_L;            // (token, value channel): v, then U.  W takes the place of the queries (in order)
	float *be = xu + DC_L * DC_DV, *gg = be + DC_L, *G = gg + DC_L;
	const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
	const int t0 = c * DC_L, nt = min(DC_L, a.step->n - t0), d = a.d, dv = a.dv;
	if (nt <= 0) return;
	const int hk = h / (a.H / a.G), nq = a.G * d, Cc = 2 * nq + a.H * dv;
	const float* rows = a.prep + (size_t) t0 * a.ldp;
	for (int x = tid; x < DC_L * (D / 4); x += DC_TH) {
		const int t = x / (D / 4), p = x % (D / 4);
		const bool in = t < nt && p * 4 < d;
		const float* src = rows + (size_t) (in ? t : 0) * a.ldp + hk * d + (in ? p * 4 : 0);
		dc_cp16(ks + t * D + (p ^ (t & 7)) * 4, src + nq, in);
		dc_cp16(qs + t * D + (p ^ (t & 7)) * 4, src, in);
	}
	for (int x = tid; x < DC_L * (DC_DV / 4); x += DC_TH) {
		const int t = x / (DC_DV / 4), p = x % (DC_DV / 4);
		const bool in = t < nt && p * 4 < dv;
		dc_cp16(xu + t * DC_DV + p * 4, rows + (size_t) (in ? t : 0) * a.ldp + 2 * nq + h * dv + (in ? p * 4 : 0), in);
	}
	DC_COMMIT();
	if (tid < DC_L) { // beyond the last token: nothing is written, nothing decays
		be[tid] = tid < nt ? rows[(size_t) tid * a.ldp + Cc + h] : 0.f;
		gg[tid] = tid < nt ? rows[(size_t) tid * a.ldp + Cc + a.H + h] : 1.f;
	}
	__syncthreads();
	const DcWs ws = dc_ws(a.ws, chunks, a.H, D);
	const size_t at = (size_t) c * a.H + h;
	if (tid < DC_L) { // column s of the decays
		float p = 1.f;
		for (int t8 = tid & ~7; t8 < DC_L; t8 += 8) {
			float f[8];
#pragma unroll
			for (int u = 0; u < 8; u++) f[u] = gg[t8 + u];
#pragma unroll
			for (int u = 0; u < 8; u++) {
				const int t = t8 + u;
				if (t > tid) p *= f[u];
				if (t >= tid) M[t * DC_L + tid] = p;
			}
		}
		ws.g[at * 2 * DC_L + DC_L + tid] = p;
	} else if (tid == DC_L) {
		float p = 1.f;
		for (int t8 = 0; t8 < DC_L; t8 += 8) {
			float f[8];
#pragma unroll
			for (int u = 0; u < 8; u++) f[u] = gg[t8 + u];
#pragma unroll
			for (int u = 0; u < 8; u++) {
				p *= f[u];
				G[t8 + u] = p;
				ws.g[at * 2 * DC_L + t8 + u] = p;
			}
		}
	}
	DC_WAIT(0);
	__syncthreads();
	// ---- k_t . k_s and q_t . k_s: rows t = 4 ty .., columns s = tx + 16 b ----
	{
		const int ty = tid >> 4, tx = tid & 15;
		float kk[4][4] = {}, qk[4][4] = {};
#pragma unroll 2
		for (int p = 0; p < D / 4; p++) {
			float4 kt[4], qt[4];
#pragma unroll
			for (int r = 0; r < 4; r++) {
				const int t = ty * 4 + r;
				kt[r] = dc_ld4(ks + t * D + (p ^ (t & 7)) * 4);
				qt[r] = dc_ld4(qs + t * D + (p ^ (t & 7)) * 4);
			}
#pragma unroll
			for (int b = 0; b < 4; b++) {
				const int s = tx + 16 * b;
				const float4 k = dc_ld4(ks + s * D + (p ^ (s & 7)) * 4);
#pragma unroll
				for (int r = 0; r < 4; r++) {
					kk[r][b] = fmaf(kt[r].x, k.x, kk[r][b]); kk[r][b] = fmaf(kt[r].y, k.y, kk[r][b]);
					kk[r][b] = fmaf(kt[r].z, k.z, kk[r][b]); kk[r][b] = fmaf(kt[r].w, k.w, kk[r][b]);
					qk[r][b] = fmaf(qt[r].x, k.x, qk[r][b]); qk[r][b] = fmaf(qt[r].y, k.y, qk[r][b]);
					qk[r][b] = fmaf(qt[r].z, k.z, qk[r][b]); qk[r][b] = fmaf(qt[r].w, k.w, qk[r][b]);
				}
			}
		}
#pragma unroll
		for (int r = 0; r < 4; r++)
#pragma unroll
			for (int b = 0; b < 4; b++) {
				const int t = ty * 4 + r, s = tx + 16 * b;
				const float f = s <= t ? M[t * DC_L + s] : 0.f;
				ws.p[at * DC_L * DC_L + t * DC_L + s] = s <= t ? f * qk[r][b] : 0.f;
				M[t * DC_L + s] = s < t ? be[t] * (f * kk[r][b]) : 0.f;
			}
	}
	__syncthreads();
	// ---- U and W: a thread's column, eight rows at a time ----
	if (tid < DC_DV + D) {
		const bool is_u = tid < DC_DV;
		const int col = is_u ? tid : tid - DC_DV, ldx = is_u ? DC_DV : D;
		float* X = is_u ? xu : qs;
		float* dst = (is_u ? ws.u + at * DC_L * DC_DV : ws.w + at * DC_L * D) + col;
		for (int r0 = 0; r0 < DC_L; r0 += 8) {
			float x[8];
#pragma unroll
			for (int r = 0; r < 8; r++) {
				const int t = r0 + r;
				x[r] = be[t] * (is_u ? X[t * ldx + col] : G[t] * ks[t * D + (((col >> 2) ^ (t & 7)) << 2) + (col & 3)]);
			}
#pragma unroll 2
			for (int s = 0; s < r0; s += 4) {
				float y[4];
#pragma unroll
				for (int e = 0; e < 4; e++) y[e] = X[(s + e) * ldx + col];
#pragma unroll
				for (int r = 0; r < 8; r++) {
					const float4 m = dc_ld4(M + (r0 + r) * DC_L + s);
					x[r] = fmaf(-m.x, y[0], x[r]); x[r] = fmaf(-m.y, y[1], x[r]); x[r] = fmaf(-m.z, y[2], x[r]); x[r] = fmaf(-m.w, y[3], x[r]);
				}
			}
#pragma unroll
			for (int r = 0; r < 8; r++) {
#pragma unroll
				for (int s = 0; s < r; s++) x[r] = fmaf(-M[(r0 + r) * DC_L + r0 + s], x[s], x[r]);
				X[(r0 + r) * ldx + col] = x[r];
				dst[(size_t) (r0 + r) * ldx] = x[r];
			}
		}
	}
}

// sixteen partial sums of a tile, spread over KS neighbouring lanes: every lane ends with 16 / KS of the totals, from the returned one on
template <int KS>
__device__ __forceinline__ int dc_join(float (&v)[16], int lane) {
	int first = 0, cnt = 16;
#pragma unroll
	for (int w = KS / 2; w >= 1; w >>= 1) {
		cnt >>= 1;
		const bool up = lane & w;
#pragma unroll
		for (int x = 0; x < 8; x++)
			if (x < cnt) {
				const float give = up ? v[x] : v[x + cnt], keep = up ? v[x + cnt] : v[x];
				v[x] = keep + __shfl_xor_sync(0xffffffffu, give, w);
			}
		if (up) first += cnt;
	}
	return first;
}
template <int D, int CG>
struct DcCfg {
	static constexpr int KA = 32 / CG, KB = 64 / CG, KC = 4096 / (D * CG); // lanes that share a tile's sum in the three products
	static constexpr int LDW = D + 4 * KA, LDK = D + 16, LDP = DC_L + 16, LDC = CG + 4;
	static constexpr size_t FLOATS = 2 * (size_t) DC_L * LDW + (size_t) DC_L * LDK + (size_t) DC_L * LDP + (size_t) DC_L * CG + 3 * (size_t) DC_L * LDC + (size_t) D * LDC + 4 * DC_L;
};

// grid (groups of CG value channels, H)
template <int D, int CG>
__global__ void __launch_bounds__(DC_TH) delta_states_kernel(DeltaArgs a, int chunks) {
	using Cfg = DcCfg<D, CG>;
	constexpr int KA = Cfg::KA, KB = Cfg::KB, KC = Cfg::KC, LDW = Cfg::LDW, LDK = Cfg::LDK, LDP = Cfg::LDP, LDC = Cfg::LDC, NC = CG / 4;
	extern __shared__ __align__(16) float sm[];
	float* wq = sm;                 // rows 0 .. 63: W, 64 .. 127: q
	float* ks = wq + 2 * DC_L * LDW;
	float* P = ks + DC_L * LDK;
	float* U = P + DC_L * LDP;
	float *us = U + DC_L * CG, *eu = us + DC_L * LDC, *os = eu + DC_L * LDC; // u, D[L, s] u, G S_0^T q
	float* S = os + DC_L * LDC;
	float* ge = S + D * LDC;        // two chunks' G and D[L, s]
	const int c0 = blockIdx.x * CG, h = blockIdx.y, tid = threadIdx.x;
	const int n = a.step->n, used = (n + DC_L - 1) / DC_L, d = a.d, dv = a.dv;
	const int hk = h / (a.H / a.G), nq = a.G * d;
	const DcWs ws = dc_ws(a.ws, chunks, a.H, D);
	float* st = a.state + (size_t) h * d * dv;
	for (int x = tid; x < D * CG; x += DC_TH) {
		const int i = x / CG, col = x % CG;
		S[i * LDC + col] = i < d && c0 + col < dv ? st[(size_t) i * dv + c0 + col] : 0.f;
	}
	auto stage_a = [&](int c) { // what the first product reads
		const size_t at = (size_t) c * a.H + h;
		const float* rows = a.prep + (size_t) c * DC_L * a.ldp;
		const int nt = n - c * DC_L;
		for (int x = tid; x < DC_L * (D / 4); x += DC_TH) {
			const int t = x / (D / 4), i = x % (D / 4) * 4;
			const bool in = t < nt && i < d;
			dc_cp16(wq + t * LDW + i, ws.w + at * DC_L * D + t * D + i, true);
			dc_cp16(wq + (DC_L + t) * LDW + i, rows + (in ? (size_t) t * a.ldp + hk * d + i : 0), in);
		}
		for (int x = tid; x < DC_L * NC; x += DC_TH) dc_cp16(U + x * 4, ws.u + at * DC_L * DC_DV + x / NC * DC_DV + c0 + x % NC * 4, true);
		if (tid < 2 * DC_L / 4) dc_cp16(ge + (c & 1) * 2 * DC_L + tid * 4, ws.g + at * 2 * DC_L + tid * 4, true);
		DC_COMMIT();
	};
	auto stage_b = [&](int c) { // what the other two read
		const size_t at = (size_t) c * a.H + h;
		const float* rows = a.prep + (size_t) c * DC_L * a.ldp;
		const int nt = n - c * DC_L;
		for (int x = tid; x < DC_L * (D / 4); x += DC_TH) {
			const int t = x / (D / 4), i = x % (D / 4) * 4;
			const bool in = t < nt && i < d;
			dc_cp16(ks + t * LDK + i, rows + (in ? (size_t) t * a.ldp + nq + hk * d + i : 0), in);
		}
		for (int x = tid; x < DC_L * (DC_L / 4); x += DC_TH) dc_cp16(P + x / (DC_L / 4) * LDP + x % (DC_L / 4) * 4, ws.p + at * DC_L * DC_L + x * 4, true);
		DC_COMMIT();
	};
	if (used > 0) { stage_a(0); stage_b(0); }
	for (int c = 0; c < used; c++) {
		const float *G = ge + (c & 1) * 2 * DC_L, *E = G + DC_L;
		DC_WAIT(1);
		__syncthreads();
		{ // [W; q] S: rows rg + 32 r, four columns
			const int k = tid % KA, cg = tid / KA % NC * 4, rg = tid / (KA * NC);
			float acc[16] = {};
#pragma unroll 2
			for (int j = 0; j < D / 4 / KA; j++) {
				const int i = (j * KA + k) * 4;
				float4 w[4], s[4];
#pragma unroll
				for (int r = 0; r < 4; r++) w[r] = dc_ld4(wq + (rg + 32 * r) * LDW + i);
#pragma unroll
				for (int e = 0; e < 4; e++) s[e] = dc_ld4(S + (i + e) * LDC + cg);
#pragma unroll
				for (int r = 0; r < 4; r++) {
					const float x[4] = {w[r].x, w[r].y, w[r].z, w[r].w};
#pragma unroll
					for (int e = 0; e < 4; e++) {
						acc[4 * r] = fmaf(x[e], s[e].x, acc[4 * r]); acc[4 * r + 1] = fmaf(x[e], s[e].y, acc[4 * r + 1]);
						acc[4 * r + 2] = fmaf(x[e], s[e].z, acc[4 * r + 2]); acc[4 * r + 3] = fmaf(x[e], s[e].w, acc[4 * r + 3]);
					}
				}
			}
			const int first = dc_join<KA>(acc, tid);
#pragma unroll
			for (int x = 0; x < 16 / KA; x++) {
				const int row = rg + 32 * ((first + x) >> 2), col = cg + ((first + x) & 3), t = row & (DC_L - 1);
				if (row < DC_L) {
					const float u = U[t * CG + col] - acc[x];
					us[t * LDC + col] = u;
					eu[t * LDC + col] = E[t] * u;
				} else os[t * LDC + col] = G[t] * acc[x];
			}
		}
		DC_WAIT(0);
		__syncthreads();
		if (c + 1 < used) stage_a(c + 1);
		{ // o = G S_0^T q + P u: rows rg + 16 r
			const int k = tid % KB, cg = tid / KB % NC * 4, rg = tid / (KB * NC);
			float acc[16] = {};
#pragma unroll 2
			for (int j = 0; j < DC_L / 4 / KB; j++) {
				const int s0 = (j * KB + k) * 4;
				float4 p[4], u[4];
#pragma unroll
				for (int r = 0; r < 4; r++) p[r] = dc_ld4(P + (rg + 16 * r) * LDP + s0);
#pragma unroll
				for (int e = 0; e < 4; e++) u[e] = dc_ld4(us + (s0 + e) * LDC + cg);
#pragma unroll
				for (int r = 0; r < 4; r++) {
					const float x[4] = {p[r].x, p[r].y, p[r].z, p[r].w};
#pragma unroll
					for (int e = 0; e < 4; e++)
						if (s0 + e <= rg + 16 * r) {
							acc[4 * r] = fmaf(x[e], u[e].x, acc[4 * r]); acc[4 * r + 1] = fmaf(x[e], u[e].y, acc[4 * r + 1]);
							acc[4 * r + 2] = fmaf(x[e], u[e].z, acc[4 * r + 2]); acc[4 * r + 3] = fmaf(x[e], u[e].w, acc[4 * r + 3]);
						}
				}
			}
			const int first = dc_join<KB>(acc, tid);
#pragma unroll
			for (int x = 0; x < 16 / KB; x++) {
				const int t = rg + 16 * ((first + x) >> 2), col = cg + ((first + x) & 3);
				if (c * DC_L + t < n && c0 + col < dv) a.out[(size_t) (c * DC_L + t) * (a.H * dv) + h * dv + c0 + col] = os[t * LDC + col] + acc[x];
			}
		}
		{ // S = G_L S_0 + k^T (D[L, s] u): channels 4 rg ..
			const int k = tid % KC, cg = tid / KC % NC * 4, rg = tid / (KC * NC);
			float acc[16] = {};
#pragma unroll 4
			for (int j = 0; j < DC_L / KC; j++) {
				const int s = j * KC + k;
				const float4 kv = dc_ld4(ks + s * LDK + rg * 4), u = dc_ld4(eu + s * LDC + cg);
				const float x[4] = {kv.x, kv.y, kv.z, kv.w};
#pragma unroll
				for (int r = 0; r < 4; r++) {
					acc[4 * r] = fmaf(x[r], u.x, acc[4 * r]); acc[4 * r + 1] = fmaf(x[r], u.y, acc[4 * r + 1]);
					acc[4 * r + 2] = fmaf(x[r], u.z, acc[4 * r + 2]); acc[4 * r + 3] = fmaf(x[r], u.w, acc[4 * r + 3]);
				}
			}
			const int first = dc_join<KC>(acc, tid);
#pragma unroll
			for (int x = 0; x < 16 / KC; x++) {
				float* s = S + (rg * 4 + ((first + x) >> 2)) * LDC + cg + ((first + x) & 3);
				*s = fmaf(G[DC_L - 1], *s, acc[x]);
			}
		}
		__syncthreads();
		if (c + 1 < used) stage_b(c + 1);
	}
	for (int x = tid; x < D * CG; x += DC_TH) {
		const int i = x / CG, col = x % CG;
		if (i < d && c0 + col < dv) st[(size_t) i * dv + c0 + col] = S[i * LDC + col];
	}
}

// a warp per token and head; then the inputs of the last taps - 1 positions (a pass has more tokens) become the convolutions' state
__global__ void __launch_bounds__(256) delta_finish_kernel(DeltaArgs a) {
	const int n = a.step->n, lane = threadIdx.x & 31, x = blockIdx.x * 8 + (threadIdx.x >> 5), t = x / a.H, h = x % a.H, dv = a.dv;
	if (t < n) {
		float* row = a.out + (size_t) t * (a.H * dv) + h * dv;
		const float* gate = a.proj + (size_t) t * a.ld + a.g_off + h * dv;
		float o[DC_DV / 32], z[DC_DV / 32], ss = 0.f, r = 1.f;
#pragma unroll
		for (int j = 0; j < DC_DV / 32; j++) {
			const bool in = j * 32 + lane < dv;
			o[j] = in ? row[j * 32 + lane] : 0.f;
			z[j] = in ? gate[j * 32 + lane] : 0.f;
			ss = fmaf(o[j], o[j], ss);
		}
		if (a.norm_w) r = 1.f / sqrtf(warp_sum(ss) / (float) dv + a.eps);
#pragma unroll
		for (int j = 0; j < DC_DV / 32; j++)
			if (j * 32 + lane < dv) row[j * 32 + lane] = o[j] * r * (a.norm_w ? a.norm_w[j * 32 + lane] : 1.f) * (z[j] * sigmoidf_(z[j]));
	}
	const int nq = a.G * a.d, Cc = 2 * nq + a.H * dv, keep = a.taps - 1;
	for (int y = blockIdx.x * 256 + threadIdx.x; y < keep * Cc; y += gridDim.x * 256) {
		const int r = y / Cc, cc = y % Cc, sec = cc < nq ? 0 : cc < 2 * nq ? 1 : 2, lc = cc - (sec == 0 ? 0 : sec == 1 ? nq : 2 * nq);
		a.conv_state[y] = a.proj[(size_t) (n - keep + r) * a.ld + (sec == 0 ? a.q_off : sec == 1 ? a.k_off : a.v_off) + lc];
	}
}

template <int D, int CG>
static int launch_states(const DeltaArgs& a, int chunks, cudaStream_t s) {
	const size_t smem = DcCfg<D, CG>::FLOATS * 4;
	XALM_CUDA_CHECK(cudaFuncSetAttribute(delta_states_kernel<D, CG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem));
	delta_states_kernel<D, CG><<<dim3((a.dv + CG - 1) / CG, a.H), DC_TH, smem, s>>>(a, chunks);
	return launch_check("delta_states");
}
template <int D>
static int launch_chunks(const DeltaArgs& a, int rows, cudaStream_t s) {
	const int chunks = (rows + DC_L - 1) / DC_L;
	XALM_CUDA_CHECK(cudaFuncSetAttribute(delta_local_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) dc_local_smem(D)));
	delta_local_kernel<D><<<dim3(chunks, a.H), DC_TH, dc_local_smem(D), s>>>(a, chunks);
	XALM_TRY(launch_check("delta_local"));
	// eight value channels per CTA where sixteen would leave a third of the SMs idle: every CTA of a head reads the head's W, q, k and P.  All kernels of a pass, us
	// with 8 -> 16 channels: 1024 tokens of 8 heads of 64 x 128 (64 CTAs of 16) 120 -> 138, of 16 of 64 x 64 (64) 151 -> 169, of 12 of 64 x 128 (96) 183 -> 159,
	// of 12 of 128 x 128 (96) 261 -> 196, of 24 of 64 x 64 (96) 224 -> 202; 64 and 256 tokens likewise
	if (a.H * ((a.dv + 15) / 16) >= 96) XALM_TRY((launch_states<D, 16>(a, chunks, s)));
	else XALM_TRY((launch_states<D, 8>(a, chunks, s)));
	delta_finish_kernel<<<(rows * a.H + 7) / 8, 256, 0, s>>>(a);
	return launch_check("delta_finish");
}
int launch_delta_chunks(const DeltaArgs& a, int rows, cudaStream_t s) { return a.d <= 64 ? launch_chunks<64>(a, rows, s) : launch_chunks<128>(a, rows, s); }

} // namespace mix
} // namespace xalm
