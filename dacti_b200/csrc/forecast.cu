// Regrid forecaster network: a multilayer perceptron n_in -> 64 -> 64 -> 1 (ReLU, logistic output)
// that predicts, from per-leaf features, whether the refinement indicator will fire at that place a
// few global steps ahead. No counterpart in the reference. Training keeps FP32 master weights with Adam
// moments; inference reads BF16 copies of the weights, refreshed after every optimiser step.
//
// Parameter layout (FP32 master and BF16 copies alike): W1[H][n_in], b1[H], W2[H][H], b2[H], W3[H], b3.
// Loss: binary cross-entropy on the logit z with a weight on the positive class,
//   l = pw y softplus(-z) + (1 - y) softplus(z),   dl/dz = sigmoid(z) (pw y + 1 - y) - pw y.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "dacti_gpu.h"
#include "mem.cuh"

namespace {

constexpr int H      = 64;   // hidden width
constexpr int MAX_IN = 32;   // largest input width
constexpr int TPB    = 128;  // threads per block (one sample each)

thread_local std::string g_mlp_error;

struct Layout {
	int nin;
	long long w1, b1, w2, b2, w3, b3, n;
	explicit Layout(int in) : nin(in) {
		w1 = 0;
		b1 = w1 + (long long) H * nin;
		w2 = b1 + H;
		b2 = w2 + (long long) H * H;
		w3 = b2 + H;
		b3 = w3 + H;
		n  = b3 + 1;
	}
};

__device__ __forceinline__ float softplus(float z) { return z > 0.f ? z + log1pf(expf(-z)) : log1pf(expf(z)); }
__device__ __forceinline__ float sigmoidf(float z) { return 1.f / (1.f + expf(-z)); }

// Forward pass of one sample with weights `w` (shared memory, FP32); leaves the hidden activations in
// a1/a2 and returns the logit.
__device__ __forceinline__ float forward(const float *w, const Layout &L, const float *x, float *a1, float *a2) {
#pragma unroll
	for (int j = 0; j < H; ++j) {
		float z = w[L.b1 + j];
		for (int i = 0; i < L.nin; ++i) z += w[L.w1 + j * L.nin + i] * x[i];
		a1[j] = fmaxf(z, 0.f);
	}
#pragma unroll 4
	for (int k = 0; k < H; ++k) {
		float z = w[L.b2 + k];
#pragma unroll
		for (int j = 0; j < H; ++j) z += w[L.w2 + k * H + j] * a1[j];
		a2[k] = fmaxf(z, 0.f);
	}
	float z = w[L.b3];
#pragma unroll
	for (int k = 0; k < H; ++k) z += w[L.w3 + k] * a2[k];
	return z;
}

__global__ void k_predict(const __nv_bfloat16 *wb, Layout L, const float *x, long long n, float *prob) {
	extern __shared__ float sw[];
	for (long long p = threadIdx.x; p < L.n; p += blockDim.x) sw[p] = __bfloat162float(wb[p]);
	__syncthreads();
	float a1[H], a2[H], xi[MAX_IN];
	for (long long s = (long long) blockIdx.x * blockDim.x + threadIdx.x; s < n; s += (long long) gridDim.x * blockDim.x) {
		for (int i = 0; i < L.nin; ++i) xi[i] = x[s * L.nin + i];
		prob[s] = sigmoidf(forward(sw, L, xi, a1, a2));
	}
}

// ---- loss and gradient over tiles of 32 samples -----------------------------------------------------
//
// A block of 256 threads takes 32 samples through the network and back with all operands in shared memory:
// in the forward pass and in the backward pass through the layers a lane is a sample and a warp has eight
// of the 64 units; the weight gradients are 32-term products of activations and deltas, 4 x 4 of the second
// layer's per thread. What bounds it is the latency of that chain.
//
// Every value is rounded as one thread per sample and one warp reduction per weight would round it: products
// before they are added (a unit within rounding of zero is on or off by that), units in ascending order, the 32
// samples of a tile in the pairs of a butterfly, four tiles to a block sum. A gradient's sign decides a
// step of Adam, so another rounding is another network.

constexpr int GT   = 256;  // threads
constexpr int TS   = 32;   // samples of a tile
constexpr int TB   = 4;    // tiles of a block sum
constexpr int ROW  = 68;   // row stride of [sample][unit] arrays: 16-byte rows that start in different banks
constexpr int XMAX = TS * MAX_IN / GT;  // inputs of a tile per thread
static_assert(H == 64 && GT == 256 && TS == 32 && TB * TS == TPB, "the thread mapping below is for these sizes");

struct TileMem {
	float *W, *G, *X, *A1, *A2, *D1, *D2, *A1T, *D2T, *dz, *y;
	static __host__ __device__ int pad(long long n) { return (int) ((n + 3) / 4 * 4); }
	static __host__ __device__ size_t floats(const Layout &L) {
		return 3 * (size_t) pad(L.n) + 2 * pad((long long) TS * L.nin) + 4 * TS * ROW + 2 * H * TS + TS + 2 * TS;
	}
	__device__ TileMem(float *m, const Layout &L) {
		auto take = [&](size_t n) {
			float *r = m;
			m += n;
			return r;
		};
		W = take(pad(L.n)), G = take(2 * pad(L.n)), X = take(2 * pad((long long) TS * L.nin));
		A1 = take(TS * ROW), A2 = take(TS * ROW), D1 = take(TS * ROW), D2 = take(TS * ROW);
		A1T = take(H * TS), D2T = take(H * TS), dz = take(TS), y = take(2 * TS);
	}
};

// A thread's share of the gradient: 4 x 4 of W2, a quarter of a row of W1, and one of b2, W3, b1, b3.
struct GradShare {
	float w2[16], w1[MAX_IN / 4], one;
	__device__ void zero() {
#pragma unroll
		for (float &v: w2) v = 0.f;
#pragma unroll
		for (float &v: w1) v = 0.f;
		one = 0.f;
	}
	// Where the thread's values stand in the parameter vector: f(index, value).
	template<class F>
	__device__ void each(const Layout &L, F f) const {
		const int t = threadIdx.x, k0 = 4 * (t >> 4), j0 = 4 * (t & 15);
#pragma unroll
		for (int a = 0; a < 4; ++a)
#pragma unroll
			for (int b = 0; b < 4; ++b) f(L.w2 + (k0 + a) * H + j0 + b, w2[4 * a + b]);
#pragma unroll
		for (int c = 0; c < MAX_IN / 4; ++c)
			if ((t & 3) + 4 * c < L.nin) f(L.w1 + (long long) (t >> 2) * L.nin + (t & 3) + 4 * c, w1[c]);
		if (t < 64) f(L.b2 + t, one);
		else if (t < 128) f(L.w3 + t - 64, one);
		else if (t < 192) f(L.b1 + t - 128, one);
		else if (t == 192) f(L.b3, one);
	}
};

// The inputs of samples [first, first + TS) of the order `perm` (identity when null) into registers; samples
// from `end` on are zero. The labels come with the first TS threads.
__device__ __forceinline__ void fetch_tile(const Layout &L, const float *x, const float *y, const int *perm, long long first,
                                           long long end, float *xr, float &yr) {
#pragma unroll
	for (int c = 0; c < XMAX; ++c) {
		const int e = threadIdx.x + GT * c;
		xr[c]       = 0.f;
		if (e < TS * L.nin) {
			const long long t = first + e / L.nin;
			if (t < end) xr[c] = x[(perm ? (long long) perm[t] : t) * L.nin + e % L.nin];
		}
	}
	yr = 0.f;
	if (threadIdx.x < TS && first + threadIdx.x < end) {
		const long long t = first + threadIdx.x;
		yr                = y[perm ? (long long) perm[t] : t];
	}
}
__device__ __forceinline__ void store_tile(const Layout &L, float *X, float *y, const float *xr, float yr) {
#pragma unroll
	for (int c = 0; c < XMAX; ++c) {
		const int e = threadIdx.x + GT * c;
		if (e < TS * L.nin) X[e] = xr[c];
	}
	if (threadIdx.x < TS) y[threadIdx.x] = yr;
}

// The sums over a tile's samples of N values each, v(sample, out): node HALF of the butterfly that pairs the samples
// 16 apart, then 8, 4, 2 and 1.
template<int N, int HALF, class V>
__device__ __forceinline__ void sum_samples(int q, const V &v, float (&out)[N]) {
	if constexpr (HALF == TS) {
		v(q, out);
	} else {
		float b[N];
		sum_samples<N, 2 * HALF>(q, v, out);
		sum_samples<N, 2 * HALF>(q + HALF, v, b);
#pragma unroll
		for (int k = 0; k < N; ++k) out[k] += b[k];
	}
}

// Adds a tile's gradient to `g` and its loss to `loss_sum`. X and y of the tile are in shared memory (stored before a
// barrier); `live` samples count.
__device__ __forceinline__ void tile_grad(const TileMem &m, const Layout &L, const float *X, const float *y, int live, float pw,
                                          GradShare &g, double *loss_sum) {
	const int t = threadIdx.x, lane = t & 31, u0 = 8 * (t >> 5);
	float a1[8], a2[8];
#pragma unroll
	for (int c = 0; c < 8; ++c) a1[c] = m.W[L.b1 + u0 + c];
	for (int i = 0; i < L.nin; ++i) {
		const float v = X[lane * L.nin + i];
#pragma unroll
		for (int c = 0; c < 8; ++c) a1[c] += m.W[L.w1 + (u0 + c) * L.nin + i] * v;
	}
#pragma unroll
	for (int c = 0; c < 8; ++c) {
		a1[c]                      = fmaxf(a1[c], 0.f);
		m.A1T[(u0 + c) * TS + lane] = a1[c];
	}
#pragma unroll
	for (int c = 0; c < 8; c += 4) *(float4 *) (m.A1 + lane * ROW + u0 + c) = make_float4(a1[c], a1[c + 1], a1[c + 2], a1[c + 3]);
	__syncthreads();
#pragma unroll
	for (int c = 0; c < 8; ++c) a2[c] = m.W[L.b2 + u0 + c];
#pragma unroll 4
	for (int j = 0; j < H; j += 4) {
		float v[4];
#pragma unroll
		for (int q = 0; q < 4; ++q) v[q] = m.A1T[(j + q) * TS + lane];
#pragma unroll
		for (int c = 0; c < 8; ++c) {
			const float4 w = *(const float4 *) (m.W + L.w2 + (u0 + c) * H + j);
			a2[c] += w.x * v[0];
			a2[c] += w.y * v[1];
			a2[c] += w.z * v[2];
			a2[c] += w.w * v[3];
		}
	}
#pragma unroll
	for (int c = 0; c < 8; ++c) a2[c] = fmaxf(a2[c], 0.f);
#pragma unroll
	for (int c = 0; c < 8; c += 4) *(float4 *) (m.A2 + lane * ROW + u0 + c) = make_float4(a2[c], a2[c + 1], a2[c + 2], a2[c + 3]);
	__syncthreads();
	// the logit, on every warp alike: a sum in the units' order
	float z = m.W[L.b3];
#pragma unroll 4
	for (int k = 0; k < H; k += 4) {
		const float4 a = *(const float4 *) (m.A2 + lane * ROW + k), w = *(const float4 *) (m.W + L.w3 + k);
		z += w.x * a.x;
		z += w.y * a.y;
		z += w.z * a.z;
		z += w.w * a.w;
	}
	const float yt = y[lane];
	float dz       = sigmoidf(z) * (pw * yt + 1.f - yt) - pw * yt;
	if (lane >= live) dz = 0.f;
	if (t < TS) {
		m.dz[lane] = dz;
		double l   = lane < live ? (double) (pw * yt * softplus(-z) + (1.f - yt) * softplus(z)) : 0.0;
		for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
		if (t == 0) atomicAdd(loss_sum, l);
	}
	float d[8];
#pragma unroll
	for (int c = 0; c < 8; ++c) {
		d[c]                       = a2[c] > 0.f ? dz * m.W[L.w3 + u0 + c] : 0.f;
		m.D2T[(u0 + c) * TS + lane] = d[c];
	}
#pragma unroll
	for (int c = 0; c < 8; c += 4) *(float4 *) (m.D2 + lane * ROW + u0 + c) = make_float4(d[c], d[c + 1], d[c + 2], d[c + 3]);
	__syncthreads();
#pragma unroll
	for (int c = 0; c < 8; ++c) d[c] = 0.f;
#pragma unroll 4
	for (int k = 0; k < H; ++k) {
		const float v   = m.D2T[k * TS + lane];
		const float4 wa = *(const float4 *) (m.W + L.w2 + k * H + u0), wb = *(const float4 *) (m.W + L.w2 + k * H + u0 + 4);
		d[0] += wa.x * v, d[1] += wa.y * v, d[2] += wa.z * v, d[3] += wa.w * v;
		d[4] += wb.x * v, d[5] += wb.y * v, d[6] += wb.z * v, d[7] += wb.w * v;
	}
#pragma unroll
	for (int c = 0; c < 8; ++c) d[c] = a1[c] > 0.f ? d[c] : 0.f;
#pragma unroll
	for (int c = 0; c < 8; c += 4) *(float4 *) (m.D1 + lane * ROW + u0 + c) = make_float4(d[c], d[c + 1], d[c + 2], d[c + 3]);
	const int k0 = 4 * (t >> 4), j0 = 4 * (t & 15);
	float s2[16];
	sum_samples<16, 1>(0, [&](int q, float (&o)[16]) {
		const float4 dk = *(const float4 *) (m.D2 + q * ROW + k0), aj = *(const float4 *) (m.A1 + q * ROW + j0);
		const float dv[4] = {dk.x, dk.y, dk.z, dk.w}, av[4] = {aj.x, aj.y, aj.z, aj.w};
#pragma unroll
		for (int a = 0; a < 4; ++a)
#pragma unroll
			for (int b = 0; b < 4; ++b) o[4 * a + b] = dv[a] * av[b];
	}, s2);
#pragma unroll
	for (int q = 0; q < 16; ++q) g.w2[q] += s2[q];
	float one[1] = {0.f};
	if (t < 64) {
		sum_samples<1, 1>(0, [&](int q, float (&o)[1]) { o[0] = m.D2[q * ROW + t]; }, one);
	} else if (t < 128) {
		sum_samples<1, 1>(0, [&](int q, float (&o)[1]) { o[0] = m.dz[q] * m.A2[q * ROW + t - 64]; }, one);
	} else if (t == 192) {
		sum_samples<1, 1>(0, [&](int q, float (&o)[1]) { o[0] = m.dz[q]; }, one);
	}
	__syncthreads();
	float s1[MAX_IN / 4];
	sum_samples<MAX_IN / 4, 1>(0, [&](int q, float (&o)[MAX_IN / 4]) {
		const float v = m.D1[q * ROW + (t >> 2)];
#pragma unroll
		for (int c = 0; c < MAX_IN / 4; ++c) o[c] = (t & 3) + 4 * c < L.nin ? v * X[q * L.nin + (t & 3) + 4 * c] : 0.f;
	}, s1);
#pragma unroll
	for (int c = 0; c < MAX_IN / 4; ++c) g.w1[c] += s1[c];
	if (t >= 128 && t < 192) sum_samples<1, 1>(0, [&](int q, float (&o)[1]) { o[0] = m.D1[q * ROW + t - 128]; }, one);
	g.one += one[0];
}

// Sums of the loss and of its gradient over all n samples into loss_sum / grad. A block sums the tiles of TPB samples
// in their order, the blocks add to the gradient as they end.
__global__ void __launch_bounds__(GT) k_grad(const float *w, Layout L, const float *x, const float *y, long long n, float pw,
                                             float *grad, double *loss_sum) {
	extern __shared__ __align__(16) float sm[];
	const TileMem m(sm, L);
	for (int p = threadIdx.x; p < L.n; p += GT) m.W[p] = w[p];
	GradShare g;
	g.zero();
	for (long long base = (long long) blockIdx.x * TPB; base < n; base += (long long) gridDim.x * TPB) {
		for (long long first = base; first < min(n, base + TPB); first += TS) {
			float xr[XMAX], yr;
			fetch_tile(L, x, y, nullptr, first, n, xr, yr);
			__syncthreads();  // the previous tile's readers are done
			store_tile(L, m.X, m.y, xr, yr);
			__syncthreads();
			tile_grad(m, L, m.X, m.y, (int) min((long long) TS, n - first), pw, g, loss_sum);
		}
	}
	g.each(L, [&](long long p, float v) { atomicAdd(grad + p, v); });
}

// One epoch of Adam in one launch of one thread-block cluster. A round takes a tile of the minibatch on each block; the
// blocks leave their gradients in shared memory, and each block sums its share of the parameters over the cluster,
// four tiles to a block sum. After a minibatch's rounds it steps those parameters (moments and weights
// stay in registers for the whole epoch) and writes them into every block's copy of the weights. A cluster barrier a round
// and one a step take the place of two launches and a pass over the gradient in global memory. The gradients have two
// buffers: a block writes one while others may still read the other. A call of 24 steps of 512 samples takes 0.52 ms
// (18.0 with two launches a step and a reduction and an atomic per weight and warp). bc[step] holds Adam's bias
// corrections.
__global__ void __launch_bounds__(GT) k_epoch(float *w, __nv_bfloat16 *wb, float *mom, float *var, Layout L, const float *x,
                                              const float *y, const int *perm, long long n, long long batch, float pw, float lr,
                                              const float2 *bc, double *loss_sum) {
	constexpr float B1 = 0.9f, B2 = 0.999f, EPS = 1e-8f;
	constexpr int MINE = 4;         // parameters of a thread, at least the largest network's over eight blocks
	constexpr int MOST_BLOCKS = 16;
	extern __shared__ __align__(16) float sm[];
	const TileMem m(sm, L);
	cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
	const int rank = (int) cl.block_rank(), blocks = (int) cl.num_blocks();
	const int share = (int) ((L.n + blocks - 1) / blocks), p0 = rank * share;
	for (int p = threadIdx.x; p < L.n; p += GT) m.W[p] = w[p];
	float pw_[MINE], pm[MINE], pv[MINE];
	int at[MINE];
#pragma unroll
	for (int c = 0; c < MINE; ++c) {
		const int o = threadIdx.x + GT * c;
		at[c]       = o < share && p0 + o < L.n ? p0 + o : -1;
		pw_[c] = at[c] < 0 ? 0.f : w[at[c]];
		pm[c]  = at[c] < 0 ? 0.f : mom[at[c]];
		pv[c]  = at[c] < 0 ? 0.f : var[at[c]];
	}
	const int xn = TileMem::pad((long long) TS * L.nin), gn = TileMem::pad(L.n);
	int buf = 0, gbuf = 0;
	float xr[XMAX], yr;
	// the tile of this block that follows tile `tile` of the minibatch at `first`
	auto next = [&](long long &first, long long &tile) {
		tile += blocks;
		while (first < n && tile * TS >= min(batch, n - first)) {
			first += batch;
			tile = rank;
		}
		return first < n;
	};
	long long nf = 0, nt = rank - blocks;
	bool more = next(nf, nt);
	if (more) {
		fetch_tile(L, x, y, perm, nf + nt * TS, nf + min(batch, n - nf), xr, yr);
		store_tile(L, m.X, m.y, xr, yr);
	}
	__syncthreads();
	int step = 0;
	for (long long first = 0; first < n; first += batch, ++step) {
		const long long cnt = min(batch, n - first), tiles = (cnt + TS - 1) / TS;
		float sum[MINE];
#pragma unroll
		for (float &v: sum) v = 0.f;
		for (long long t0 = 0; t0 < tiles; t0 += blocks, gbuf ^= 1) {
			const long long tile = t0 + rank;
			float *G             = m.G + gbuf * gn;
			if (tile < tiles) {
				GradShare g;
				g.zero();
				more = next(nf, nt);
				if (more) fetch_tile(L, x, y, perm, nf + nt * TS, nf + min(batch, n - nf), xr, yr);
				tile_grad(m, L, m.X + buf * xn, m.y + buf * TS, (int) min((long long) TS, cnt - tile * TS), pw, g, loss_sum);
				buf ^= 1;
				if (more) store_tile(L, m.X + buf * xn, m.y + buf * TS, xr, yr);
				g.each(L, [&](long long p, float v) { G[p] = v; });
			}
			cl.sync();
			const int live = (int) min((long long) blocks, tiles - t0);
#pragma unroll
			for (int c = 0; c < MINE; ++c) {
				if (at[c] < 0) continue;
#pragma unroll
				for (int r0 = 0; r0 < MOST_BLOCKS; r0 += TB) {
					if (r0 >= live) break;
					float s = 0.f;
#pragma unroll
					for (int r = r0; r < r0 + TB; ++r) s += r < live ? cl.map_shared_rank(G, r)[at[c]] : 0.f;
					sum[c] += s;
				}
			}
		}
		const float2 c2   = bc[step];
		const float scale = 1.f / (float) cnt;
#pragma unroll
		for (int c = 0; c < MINE; ++c) {
			if (at[c] < 0) continue;
			const float gr = sum[c] * scale;
			pm[c]          = B1 * pm[c] + (1.f - B1) * gr;
			pv[c]          = B2 * pv[c] + (1.f - B2) * gr * gr;
			pw_[c] -= lr * (pm[c] / c2.x) / (sqrtf(pv[c] / c2.y) + EPS);
			for (int r = 0; r < blocks; ++r) cl.map_shared_rank(m.W, r)[at[c]] = pw_[c];
		}
		cl.sync();
	}
#pragma unroll
	for (int c = 0; c < MINE; ++c)
		if (at[c] >= 0) {
			w[at[c]]   = pw_[c];
			mom[at[c]] = pm[c];
			var[at[c]] = pv[c];
			wb[at[c]]  = __float2bfloat16(pw_[c]);
		}
}

__global__ void k_to_bf16(const float *w, __nv_bfloat16 *wb, long long n) {
	for (long long p = (long long) blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long) gridDim.x * blockDim.x)
		wb[p] = __float2bfloat16(w[p]);
}

uint64_t splitmix(uint64_t &s) {
	uint64_t z = (s += 0x9E3779B97F4A7C15ull);
	z          = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
	z          = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
	return z ^ (z >> 31);
}
double uniform01(uint64_t &s) { return (splitmix(s) >> 11) * (1.0 / 9007199254740992.0); }

int grid_of(long long n) {
	long long b = (n + TPB - 1) / TPB;
	return (int) (b < 1 ? 1 : (b > 148 * 8 ? 148 * 8 : b));
}

}  // namespace

struct dg_mlp {
	dg::MemoryUser memory;
	Layout L{1};
	int device = 0;
	cudaStream_t st = nullptr;
	cudaEvent_t copied = nullptr;  // an epoch's order and bias corrections are on the device
	float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
	__nv_bfloat16 *wb = nullptr;
	double *loss = nullptr;
	int t = 0;
	int cluster = 8;  // blocks of a training launch
};

namespace {

int fail(int code, const std::string &msg) {
	g_mlp_error = msg;
	return code;
}

#define MLP_CUDA(call)                                                                        \
	do {                                                                                      \
		cudaError_t e_ = (call);                                                              \
		if (e_ != cudaSuccess) return fail(DG_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
	} while (0)

size_t smem_predict(const Layout &L) { return sizeof(float) * L.n; }
size_t smem_grad(const Layout &L) { return sizeof(float) * TileMem::floats(L); }
// The limit of a kernel's shared memory holds for the device, not for a network: it is the widest network's.
int smem_limit_predict() { return (int) smem_predict(Layout(MAX_IN)); }
int smem_limit_grad() { return (int) smem_grad(Layout(MAX_IN)); }

// Device copies of host arrays on the network's stream, given back on scope exit.
struct DevBuf {
	cudaStream_t st;
	void *p = nullptr;
	explicit DevBuf(cudaStream_t s) : st(s) {}
	~DevBuf() { dg::mem_free(p, st); }
};

}  // namespace

extern "C" {

const char *dg_mlp_last_error(void) { return g_mlp_error.c_str(); }

static int mlp_create_steps(dg_mlp *h, int n_in, unsigned long long seed) {
	h->L = Layout(n_in);
	const long long n = h->L.n;
	MLP_CUDA(cudaGetDevice(&h->device));
	MLP_CUDA(cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking));
	MLP_CUDA(cudaEventCreateWithFlags(&h->copied, cudaEventDisableTiming));
	MLP_CUDA(cudaMalloc(&h->w, sizeof(float) * n));
	MLP_CUDA(cudaMalloc(&h->g, sizeof(float) * n));
	MLP_CUDA(cudaMalloc(&h->m, sizeof(float) * n));
	MLP_CUDA(cudaMalloc(&h->v, sizeof(float) * n));
	MLP_CUDA(cudaMalloc(&h->wb, sizeof(__nv_bfloat16) * n));
	MLP_CUDA(cudaMalloc(&h->loss, sizeof(double)));
	MLP_CUDA(cudaFuncSetAttribute(k_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_limit_grad()));
	MLP_CUDA(cudaFuncSetAttribute(k_epoch, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_limit_grad()));
	MLP_CUDA(cudaFuncSetAttribute(k_epoch, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
	{
		// sixteen blocks where the device can place such a cluster, else the portable eight
		cudaLaunchConfig_t cfg{};
		cudaLaunchAttribute at[1];
		at[0].id               = cudaLaunchAttributeClusterDimension;
		at[0].val.clusterDim.x = 16;
		at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
		cfg.gridDim            = 16;
		cfg.blockDim           = GT;
		cfg.dynamicSmemBytes   = smem_grad(h->L);
		cfg.attrs              = at;
		cfg.numAttrs           = 1;
		int fit                = 0;
		if (cudaOccupancyMaxActiveClusters(&fit, k_epoch, &cfg) != cudaSuccess) {
			cudaGetLastError();
			fit = 0;
		}
		h->cluster = fit > 0 ? 16 : 8;
	}
	MLP_CUDA(cudaFuncSetAttribute(k_predict, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_limit_predict()));
	// He-uniform hidden layers, Glorot-uniform output layer, zero biases
	std::vector<float> w(n, 0.f);
	uint64_t s = seed;
	auto fill = [&](long long off, long long cnt, double lim) {
		for (long long k = 0; k < cnt; ++k) w[off + k] = (float) ((2.0 * uniform01(s) - 1.0) * lim);
	};
	fill(h->L.w1, (long long) H * n_in, std::sqrt(6.0 / n_in));
	fill(h->L.w2, (long long) H * H, std::sqrt(6.0 / H));
	fill(h->L.w3, H, std::sqrt(6.0 / (H + 1)));
	return dg_mlp_set_params(h, w.data());
}

int dg_mlp_create(int n_in, unsigned long long seed, dg_mlp **out) {
	if (!out || n_in < 1 || n_in > MAX_IN) return fail(DG_ERR_ARG, "dg_mlp_create: n_in must be in [1, 32]");
	*out = nullptr;
	dg_mlp *h = new dg_mlp();
	const int rc = mlp_create_steps(h, n_in, seed);
	if (rc != DG_OK) {
		// release whatever the failed step left allocated; the error text of the failure is kept
		const std::string msg = g_mlp_error;
		dg_mlp_destroy(h);
		g_mlp_error = msg;
		return rc;
	}
	*out = h;
	return DG_OK;
}

int dg_mlp_param_count(dg_mlp *h, long long *n) {
	if (!h || !n) return fail(DG_ERR_ARG, "dg_mlp_param_count: null argument");
	*n = h->L.n;
	return DG_OK;
}

int dg_mlp_set_params(dg_mlp *h, const float *params) {
	if (!h || !params) return fail(DG_ERR_ARG, "dg_mlp_set_params: null argument");
	const long long n = h->L.n;
	MLP_CUDA(cudaSetDevice(h->device));
	MLP_CUDA(cudaMemcpyAsync(h->w, params, sizeof(float) * n, cudaMemcpyHostToDevice, h->st));
	MLP_CUDA(cudaMemsetAsync(h->g, 0, sizeof(float) * n, h->st));
	MLP_CUDA(cudaMemsetAsync(h->m, 0, sizeof(float) * n, h->st));
	MLP_CUDA(cudaMemsetAsync(h->v, 0, sizeof(float) * n, h->st));
	k_to_bf16<<<grid_of(n), TPB, 0, h->st>>>(h->w, h->wb, n);
	MLP_CUDA(cudaGetLastError());
	MLP_CUDA(cudaStreamSynchronize(h->st));
	h->t = 0;
	return DG_OK;
}

int dg_mlp_get_params(dg_mlp *h, float *params) {
	if (!h || !params) return fail(DG_ERR_ARG, "dg_mlp_get_params: null argument");
	MLP_CUDA(cudaSetDevice(h->device));
	MLP_CUDA(cudaMemcpyAsync(params, h->w, sizeof(float) * h->L.n, cudaMemcpyDeviceToHost, h->st));
	MLP_CUDA(cudaStreamSynchronize(h->st));
	return DG_OK;
}

int dg_mlp_predict(dg_mlp *h, const float *x, long long n, float *prob) {
	if (!h || (!x && n > 0) || (!prob && n > 0) || n < 0) return fail(DG_ERR_ARG, "dg_mlp_predict: bad argument");
	if (n == 0) return DG_OK;
	MLP_CUDA(cudaSetDevice(h->device));
	DevBuf dx(h->st), dp(h->st);
	MLP_CUDA(dg::mem_alloc(&dx.p, sizeof(float) * n * h->L.nin, h->st));
	MLP_CUDA(dg::mem_alloc(&dp.p, sizeof(float) * n, h->st));
	MLP_CUDA(cudaMemcpyAsync(dx.p, x, sizeof(float) * n * h->L.nin, cudaMemcpyHostToDevice, h->st));
	k_predict<<<grid_of(n), TPB, smem_predict(h->L), h->st>>>(h->wb, h->L, (const float *) dx.p, n, (float *) dp.p);
	MLP_CUDA(cudaGetLastError());
	MLP_CUDA(cudaMemcpyAsync(prob, dp.p, sizeof(float) * n, cudaMemcpyDeviceToHost, h->st));
	MLP_CUDA(cudaStreamSynchronize(h->st));
	return DG_OK;
}

int dg_mlp_loss_grad(dg_mlp *h, const float *x, const float *y, long long n, float pos_weight, float *grad,
                     double *loss) {
	if (!h || !x || !y || !grad || !loss || n <= 0) return fail(DG_ERR_ARG, "dg_mlp_loss_grad: bad argument");
	MLP_CUDA(cudaSetDevice(h->device));
	DevBuf dx(h->st), dy(h->st);
	MLP_CUDA(dg::mem_alloc(&dx.p, sizeof(float) * n * h->L.nin, h->st));
	MLP_CUDA(dg::mem_alloc(&dy.p, sizeof(float) * n, h->st));
	MLP_CUDA(cudaMemcpyAsync(dx.p, x, sizeof(float) * n * h->L.nin, cudaMemcpyHostToDevice, h->st));
	MLP_CUDA(cudaMemcpyAsync(dy.p, y, sizeof(float) * n, cudaMemcpyHostToDevice, h->st));
	MLP_CUDA(cudaMemsetAsync(h->g, 0, sizeof(float) * h->L.n, h->st));
	MLP_CUDA(cudaMemsetAsync(h->loss, 0, sizeof(double), h->st));
	k_grad<<<grid_of(n), GT, smem_grad(h->L), h->st>>>(h->w, h->L, (const float *) dx.p, (const float *) dy.p, n, pos_weight, h->g,
	                                                   h->loss);
	MLP_CUDA(cudaGetLastError());
	MLP_CUDA(cudaMemcpyAsync(grad, h->g, sizeof(float) * h->L.n, cudaMemcpyDeviceToHost, h->st));
	MLP_CUDA(cudaMemcpyAsync(loss, h->loss, sizeof(double), cudaMemcpyDeviceToHost, h->st));
	MLP_CUDA(cudaMemsetAsync(h->g, 0, sizeof(float) * h->L.n, h->st));
	MLP_CUDA(cudaStreamSynchronize(h->st));
	return DG_OK;
}

int dg_mlp_train(dg_mlp *h, const float *x, const float *y, long long n, int epochs, int batch, float lr,
                 float pos_weight, unsigned long long seed, double *mean_loss) {
	if (!h || !x || !y || n <= 0 || epochs < 1 || batch < 1 || lr <= 0.f)
		return fail(DG_ERR_ARG, "dg_mlp_train: bad argument");
	MLP_CUDA(cudaSetDevice(h->device));
	const long long steps = (n + batch - 1) / batch;
	DevBuf dx(h->st), dy(h->st), dperm(h->st), dbc(h->st);
	MLP_CUDA(dg::mem_alloc(&dx.p, sizeof(float) * n * h->L.nin, h->st));
	MLP_CUDA(dg::mem_alloc(&dy.p, sizeof(float) * n, h->st));
	MLP_CUDA(dg::mem_alloc(&dperm.p, sizeof(int) * n, h->st));
	MLP_CUDA(dg::mem_alloc(&dbc.p, sizeof(float2) * steps, h->st));
	MLP_CUDA(cudaMemcpyAsync(dx.p, x, sizeof(float) * n * h->L.nin, cudaMemcpyHostToDevice, h->st));
	MLP_CUDA(cudaMemcpyAsync(dy.p, y, sizeof(float) * n, cudaMemcpyHostToDevice, h->st));
	std::vector<int> perm(n);
	for (long long k = 0; k < n; ++k) perm[k] = (int) k;
	std::vector<float2> bc(steps);
	struct Drain {  // the arrays outlive their copies, on an error too
		cudaStream_t st;
		~Drain() { cudaStreamSynchronize(st); }
	} drain{h->st};
	cudaLaunchConfig_t cfg{};
	cudaLaunchAttribute at[1];
	at[0].id               = cudaLaunchAttributeClusterDimension;
	at[0].val.clusterDim.x = h->cluster;
	at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
	cfg.gridDim            = h->cluster;
	cfg.blockDim           = GT;
	cfg.dynamicSmemBytes   = smem_grad(h->L);
	cfg.stream             = h->st;
	cfg.attrs              = at;
	cfg.numAttrs           = 1;
	uint64_t s = seed;
	for (int e = 0; e < epochs; ++e) {
		// the host draws the next epoch's order while the GPU runs this one, once this one's has left the host's arrays
		if (e > 0) MLP_CUDA(cudaEventSynchronize(h->copied));
		for (long long k = n - 1; k > 0; --k) std::swap(perm[k], perm[(long long) (splitmix(s) % (uint64_t) (k + 1))]);
		for (long long k = 0; k < steps; ++k) {
			h->t++;
			bc[k] = make_float2(1.f - std::pow(0.9f, (float) h->t), 1.f - std::pow(0.999f, (float) h->t));
		}
		MLP_CUDA(cudaMemcpyAsync(dperm.p, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, h->st));
		MLP_CUDA(cudaMemcpyAsync(dbc.p, bc.data(), sizeof(float2) * steps, cudaMemcpyHostToDevice, h->st));
		MLP_CUDA(cudaEventRecord(h->copied, h->st));
		MLP_CUDA(cudaMemsetAsync(h->loss, 0, sizeof(double), h->st));
		MLP_CUDA(cudaLaunchKernelEx(&cfg, k_epoch, h->w, h->wb, h->m, h->v, h->L, (const float *) dx.p, (const float *) dy.p,
		                            (const int *) dperm.p, n, (long long) batch, pos_weight, lr, (const float2 *) dbc.p, h->loss));
	}
	double sum = 0.0;
	MLP_CUDA(cudaMemcpyAsync(&sum, h->loss, sizeof(double), cudaMemcpyDeviceToHost, h->st));
	MLP_CUDA(cudaStreamSynchronize(h->st));
	const double last = sum / (double) n;
	if (mean_loss) *mean_loss = last;
	return DG_OK;
}

int dg_mlp_destroy(dg_mlp *h) {
	if (!h) return DG_OK;
	cudaSetDevice(h->device);
	if (h->st) cudaStreamSynchronize(h->st);
	cudaFree(h->w);
	cudaFree(h->g);
	cudaFree(h->m);
	cudaFree(h->v);
	cudaFree(h->wb);
	cudaFree(h->loss);
	if (h->copied) cudaEventDestroy(h->copied);
	if (h->st) cudaStreamDestroy(h->st);
	delete h;
	return DG_OK;
}

}  // extern "C"
