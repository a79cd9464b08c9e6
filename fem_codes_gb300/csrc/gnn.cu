// Learned preconditioner: a mesh graph network on the graph of the CSR
// matrix, with hand-written forward and backward kernels (no reference
// counterpart; the CPU restatement used by the tests is the oracle's
// gnn_oracle.py).
//
//   s = rms(r), dbar = mean|a_ii|, x_i = [r_i/s, (r_i/s) dbar / a_ii]
//   h0 = relu(We^T x + be)
//   3 layers: m1_i = sum_j (a_ij/a_ii) h_j, m2_i = sum_j (a_ji/a_jj) h_j,
//             h <- h + relu(Wh^T h + W1^T m1 + W2^T m2 + b)
//   z_i = s (Wd . h_i + bd) dbar / a_ii
//
// Weights FP32; activations (h, m1, m2) stored as TA = bf16 (or FP32 for
// exact checks), every accumulation in FP32.  Layout of activations:
// node-major [n][32], one 64-byte (bf16) row per node, so a warp gathers a
// neighbour's row with one coalesced access.  A bf16 layer is one kernel: a
// tile's messages are gathered into shared memory and go to the tensor cores
// from there; a layer's backward pass is one kernel too.  Weight gradients are
// reduced per block into partial sums, then over blocks in a fixed order
// (deterministic).
#include <algorithm>
#include <type_traits>

#include <cuda_bf16.h>

#include "fg_common.cuh"
#include "fg_div.cuh"
#include "fg_gnn.h"

#define W 32
#define TILE 64
#define UPD_TPB 256
#define PAD (3 * W + 1)

template <typename TA> __device__ __forceinline__ float ld_act(const TA *p);
template <> __device__ __forceinline__ float ld_act<float>(const float *p) { return *p; }
template <> __device__ __forceinline__ float ld_act<__nv_bfloat16>(const __nv_bfloat16 *p)
{
	return __bfloat162float(*p);
}
template <typename TA> __device__ __forceinline__ TA st_act(float v);
template <> __device__ __forceinline__ float st_act<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 st_act<__nv_bfloat16>(float v)
{
	return __float2bfloat16_rn(v);
}

// ------------------------------------------------------------ graph set-up
// Off-diagonal graph of a CSR matrix with exactly one diagonal entry per row:
// gptr[i] = IA[i] - i; for each off-diagonal (i, j): col j, wA = a_ij / a_ii,
// wT = a_ji / a_jj (the transposed entry found by binary search in row j).
__global__ void k_gnn_graph(int n, const int *IA, const int *JA, const double *AA, int *gptr, int *gcol,
                            float *wA, float *wT, double *d, int *err)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		int lo = IA[i], hi = IA[i + 1], o = lo - i, nd = 0;
		double di = 0.0;
		for (int p = lo; p < hi; p++) if (JA[p] == i) { di = AA[p]; nd++; }
		gptr[i] = o;
		if (i == n - 1) gptr[n] = IA[n] - n;
		d[i] = di;
		if (nd != 1 || di == 0.0) { fg_set_err(err, FEMGPU_E_MESH); continue; }
		for (int p = lo; p < hi; p++) {
			int j = JA[p];
			if (j == i) continue;
			int a = IA[j], b = IA[j + 1] - 1, q = -1;
			while (a <= b) {
				int mid = (a + b) >> 1, c = JA[mid];
				if (c == i) { q = mid; break; }
				if (c < i) a = mid + 1; else b = mid - 1;
			}
			double dj = 0.0;
			for (int t = IA[j]; t < IA[j + 1]; t++) if (JA[t] == j) dj = AA[t];
			gcol[o] = j;
			wA[o] = (float)(AA[p] / di);
			wT[o] = (q >= 0 && dj != 0.0) ? (float)(AA[q] / dj) : 0.0f;
			if (q < 0) fg_set_err(err, FEMGPU_E_MESH);
			o++;
		}
	}
}

// --------------------------------------------------- small deterministic sums
#define RTPB 256
__device__ __forceinline__ double blk_sum(double v, double *sh)
{
	v = fg_warp_sum(v);
	int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
	if (lane == 0) sh[wid] = v;
	__syncthreads();
	double r = 0.0;
	if (wid == 0) {
		r = (lane < (int)(blockDim.x >> 5)) ? sh[lane] : 0.0;
		r = fg_warp_sum(r);
	}
	__syncthreads();
	return r;
}

// Per-block partial sums: part[2b] = sum a_i^2 (or |a_i| when absval),
// part[2b+1] = sum (b_i - a_i)^2 when b != NULL; then one thread adds the
// partials in block order (deterministic).
__global__ void __launch_bounds__(RTPB) k_gnn_psums(int n, const double *a, const double *b, int absval,
                                                    double *part, const int *active)
{
	if (active && !*active) return;
	__shared__ double sh[32];
	double s0 = 0.0, s1 = 0.0;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		double v = a[i];
		s0 += absval ? fabs(v) : v * v;
		if (b) { double e = b[i] - v; s1 += e * e; }
	}
	s0 = blk_sum(s0, sh);
	s1 = blk_sum(s1, sh);
	if (threadIdx.x == 0) { part[2 * blockIdx.x] = s0; part[2 * blockIdx.x + 1] = s1; }
}

// One block of 256 threads: thread t adds partials t, t+256, ... in order,
// then a fixed shuffle tree (deterministic for a given block count).
__global__ void __launch_bounds__(RTPB) k_gnn_fsums(int nblk, const double *part, double *out, const int *active)
{
	if (active && !*active) return;
	__shared__ double sh[32];
	double s0 = 0.0, s1 = 0.0;
	for (int b = threadIdx.x; b < nblk; b += blockDim.x) { s0 += part[2 * b]; s1 += part[2 * b + 1]; }
	s0 = blk_sum(s0, sh);
	s1 = blk_sum(s1, sh);
	if (threadIdx.x == 0) { out[0] = s0; out[1] = s1; }
}

// stats[0] = s = rms(r) (1 if zero), stats[2] = 1 / s, out[0] = sum r_i^2: the
// partial sums of k_gnn_psums (eight loads in flight, the same order of
// additions), the last block to finish adding them up as k_gnn_fsums does.
#define RMS_UNR 8
__global__ void __launch_bounds__(RTPB) k_gnn_rms(int n, const double *__restrict__ r, double *part, unsigned *ticket,
                                                  double *out, double *stats, const int *active)
{
	if (active && !*active) return;
	__shared__ double sh[32];
	__shared__ bool last;
	double s0 = 0.0;
	const long long st = (long long)gridDim.x * blockDim.x;
	for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += RMS_UNR * st) {
		double v[RMS_UNR];
#pragma unroll
		for (int u = 0; u < RMS_UNR; u++) v[u] = i + u * st < n ? __ldg(&r[i + u * st]) : 0.0;
#pragma unroll
		for (int u = 0; u < RMS_UNR; u++) s0 += v[u] * v[u];
	}
	s0 = blk_sum(s0, sh);
	if (threadIdx.x == 0) {
		part[2 * blockIdx.x] = s0;
		__threadfence();
		last = atomicAdd(ticket, 1u) == gridDim.x - 1;
	}
	__syncthreads();
	if (!last) return;
	double t = 0.0;
	for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) t += __ldcg(&part[2 * b]);
	t = blk_sum(t, sh);
	if (threadIdx.x == 0) {
		double s = sqrt(t / n);
		if (!(s > 0.0)) s = 1.0;
		out[0] = t;
		stats[0] = s;
		stats[2] = 1.0 / s;
		*ticket = 0u;
	}
}

// ------------------------------------------------------------------ forward
// stats: [0] = s (rms of r, 1 if zero), [1] = dbar, [2] = 1 / s.
// A warp takes 32 consecutive nodes: lane q computes node q's scaled inputs
// (the FP64 arithmetic once per node), then a half warp computes one node's
// features, two a lane, so a warp stores two rows at a time.  Bound by the
// FP64 quotient (5 operations a node, see fg_div) and the 64-byte rows written:
// 20.5 us at 1M nodes (32 us with the general quotient and one feature a lane).
__device__ __forceinline__ unsigned spread16(unsigned x)   // bit k to bit 2k
{
	x = (x | (x << 8)) & 0x00ff00ffu;
	x = (x | (x << 4)) & 0x0f0f0f0fu;
	x = (x | (x << 2)) & 0x33333333u;
	return (x | (x << 1)) & 0x55555555u;
}
template <typename TA>
__global__ void k_gnn_encode(int n, const double *r, const double *stats, const double *d,
                             const float *__restrict__ th, TA *h0, unsigned *mask0, float2 *x, const int *active)
{
	if (active && !*active) return;
	struct __align__(2 * sizeof(TA)) Pair { TA a, b; };
	const int lane = threadIdx.x & 31, half = lane >> 4, f = (lane & 15) * 2;
	const float wa0 = th[GNN_OFF_WE + f], wa1 = th[GNN_OFF_WE + W + f], ba = th[GNN_OFF_BE + f];
	const float wb0 = th[GNN_OFF_WE + f + 1], wb1 = th[GNN_OFF_WE + W + f + 1], bb = th[GNN_OFF_BE + f + 1];
	const double s = stats[0], dbar = stats[1], rs = stats[2];
	int warps = (gridDim.x * blockDim.x) >> 5;
	for (int g0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; g0 < n; g0 += warps * 32) {
		int i = g0 + lane;
		float rh = 0.0f, x1 = 0.0f;
		if (i < n) {
			rh = (float)fg_div(r[i], s, rs);
			x1 = rh * (float)dbar / (float)d[i];
			if (x) x[i] = make_float2(rh, x1);
		}
		unsigned mine = 0;
		#pragma unroll 4
		for (int q = 0; q < 32; q += 2) {
			float a = __shfl_sync(0xffffffffu, rh, q + half), c = __shfl_sync(0xffffffffu, x1, q + half);
			float pa = a * wa0 + c * wa1 + ba, pb = a * wb0 + c * wb1 + bb;
			if (mask0) {
				const unsigned ma = __ballot_sync(0xffffffffu, pa > 0.0f), mb = __ballot_sync(0xffffffffu, pb > 0.0f);
				const int sh = (lane & 1) * 16;              // node q's bits, node q + 1's
				if ((lane & ~1) == q) mine = spread16((ma >> sh) & 0xffffu) | spread16((mb >> sh) & 0xffffu) << 1;
			}
			if (g0 + q + half < n) {
				Pair o = { st_act<TA>(pa > 0.0f ? pa : 0.0f), st_act<TA>(pb > 0.0f ? pb : 0.0f) };
				*reinterpret_cast<Pair *>(&h0[(size_t)(g0 + q + half) * W + f]) = o;
			}
		}
		if (mask0 && i < n) mask0[i] = mine;
	}
}

// m1_i = sum wA h_j, m2_i = sum wT h_j: one warp per node, lane = feature.
// Quarter-warp per node (four nodes in flight per warp): lane l of group
// l/8 owns features 4*(l%8) .. +4 and gathers them with one 8-byte (bf16) or
// 16-byte (FP32) load per neighbour.
template <typename TA>
__global__ void k_gnn_agg(int n, const int *__restrict__ gptr, const int *__restrict__ gcol,
                          const float *__restrict__ wA, const float *__restrict__ wT, const TA *__restrict__ h,
                          TA *m1, TA *m2, const int *active)
{
	if (active && !*active) return;
	typedef typename std::conditional<sizeof(TA) == 2, uint2, uint4>::type V4;
	const int lane = threadIdx.x & 31, sub = lane >> 3, fl = (lane & 7) * 4;
	int groups = (gridDim.x * blockDim.x) >> 3;
	for (int i = ((blockIdx.x * blockDim.x + threadIdx.x) >> 3); i - sub < n; i += groups) {
		float a1[4] = {0.0f, 0.0f, 0.0f, 0.0f}, a2[4] = {0.0f, 0.0f, 0.0f, 0.0f};
		if (i < n) {
			int lo = __ldg(&gptr[i]), hi = __ldg(&gptr[i + 1]);
			#pragma unroll 2
			for (int p = lo; p < hi; p++) {
				int j = __ldg(&gcol[p]);
				float wa = __ldg(&wA[p]), wt = __ldg(&wT[p]);
				V4 raw = __ldg(reinterpret_cast<const V4 *>(&h[(size_t)j * W + fl]));
				const TA *v = reinterpret_cast<const TA *>(&raw);
				#pragma unroll
				for (int q = 0; q < 4; q++) {
					float hv = ld_act(&v[q]);
					a1[q] += wa * hv;
					a2[q] += wt * hv;
				}
			}
			V4 o1, o2;
			TA *p1 = reinterpret_cast<TA *>(&o1), *p2 = reinterpret_cast<TA *>(&o2);
			#pragma unroll
			for (int q = 0; q < 4; q++) { p1[q] = st_act<TA>(a1[q]); p2[q] = st_act<TA>(a2[q]); }
			*reinterpret_cast<V4 *>(&m1[(size_t)i * W + fl]) = o1;
			*reinterpret_cast<V4 *>(&m2[(size_t)i * W + fl]) = o2;
		}
	}
}

// h_out = h + relu(Wh^T h + W1^T m1 + W2^T m2 + b) on tiles of UTILE = 128
// nodes; thread t computes outputs 8*(t%4) .. +8 of nodes t/4 + 64 q (q < 2),
// so each shared-memory weight load feeds two nodes.  Inputs are staged as
// FP32 rows of 96 (+1 pad) in shared memory with 16-byte global loads.
#define UTILE 128
#define UNODE (UTILE / (UPD_TPB / 4))
template <typename TA>
__global__ void __launch_bounds__(UPD_TPB) k_gnn_update(int n, const float *__restrict__ th, const TA *h,
		const TA *m1, const TA *m2, TA *hout, unsigned *mask, const int *active)
{
	if (active && !*active) return;
	extern __shared__ __align__(16) float dyn[];
	float *sW = dyn;                                   // [3*W*W + W]
	float *sin_ = dyn + 3 * W * W + W;                 // [UTILE][PAD]
	for (int k = threadIdx.x; k < 3 * W * W + W; k += blockDim.x) sW[k] = th[k];
	const int t = threadIdx.x, node = t >> 2, fo = (t & 3) * 8;
	constexpr int VEC = 16 / sizeof(TA);               // elements per 16-byte load
	int ntile = (n + UTILE - 1) / UTILE;
	for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
		int base = tile * UTILE;
		__syncthreads();
		for (int e = t; e < UTILE * 3 * W / VEC; e += blockDim.x) {
			int nd = e / (3 * W / VEC), kv = (e - nd * (3 * W / VEC)) * VEC, i = base + nd;
			const TA *src = kv < W ? h : (kv < 2 * W ? m1 : m2);
			float *dst = &sin_[nd * PAD + kv];
			if (i < n) {
				uint4 raw = *reinterpret_cast<const uint4 *>(&src[(size_t)i * W + (kv & (W - 1))]);
				const TA *v = reinterpret_cast<const TA *>(&raw);
				#pragma unroll
				for (int q = 0; q < VEC; q++) dst[q] = ld_act(&v[q]);
			} else {
				#pragma unroll
				for (int q = 0; q < VEC; q++) dst[q] = 0.0f;
			}
		}
		__syncthreads();
		float acc[UNODE][8];
		#pragma unroll
		for (int q = 0; q < UNODE; q++)
			#pragma unroll
			for (int j = 0; j < 8; j++) acc[q][j] = sW[3 * W * W + fo + j];
		#pragma unroll 4
		for (int k = 0; k < 3 * W; k++) {
			const float4 *wr = reinterpret_cast<const float4 *>(&sW[k * W + fo]);
			float4 w0 = wr[0], w1 = wr[1];
			#pragma unroll
			for (int q = 0; q < UNODE; q++) {
				float v = sin_[(node + 64 * q) * PAD + k];
				acc[q][0] += v * w0.x; acc[q][1] += v * w0.y; acc[q][2] += v * w0.z; acc[q][3] += v * w0.w;
				acc[q][4] += v * w1.x; acc[q][5] += v * w1.y; acc[q][6] += v * w1.z; acc[q][7] += v * w1.w;
			}
		}
		#pragma unroll
		for (int q = 0; q < UNODE; q++) {
			int nd = node + 64 * q, i = base + nd;
			const float *in = &sin_[nd * PAD];
			unsigned bits = 0;
			#pragma unroll
			for (int j = 0; j < 8; j++) {
				float u = acc[q][j];
				bits |= (u > 0.0f ? 1u : 0u) << (fo + j);
				if (i < n) hout[(size_t)i * W + fo + j] = st_act<TA>(in[fo + j] + (u > 0.0f ? u : 0.0f));
			}
			bits |= __shfl_xor_sync(0xffffffffu, bits, 1);
			bits |= __shfl_xor_sync(0xffffffffu, bits, 2);
			if (mask && i < n && (t & 3) == 0) mask[i] = bits;
		}
	}
}

// One layer on bf16 activations in one kernel: messages, update and, for the
// last layer, the decoder.  A block gathers the messages of a tile of 256 nodes
// into shared memory beside their own activations (rows [h, m1, m2] of MPAD
// bf16), multiplies there and goes on to its next tile, so m1 and m2 are
// written and read back by no inference (a training pass stores them for the
// backward one), and the gathers of one block run beside another's products.
//
// Messages: four lanes per node (lane l owns features 8l .. 8l+7, one 16-byte
// load of a neighbour's row).  The lanes fetch eight edges of the node after
// the current one and hand them round, so a node's neighbour rows are all in
// flight together; sums run in edge order, two FP32 products an instruction.
// Update: tensor cores (mma.sync m16n8k16, bf16 operands, FP32 accumulation).
// Each FP32 weight is split into bf16 parts w = hi + lo (|w - hi - lo| <= 2^-16
// |w|) and both parts are multiplied, so the product keeps the FP32 weights; the
// activations are bf16 already.  Warp w of 8 takes nodes 32w..32w+31 (two
// fragments of 16 against each load of the weights) and all 32 outputs over K =
// 96 in 6 steps.  The row stride of 104 elements (52 words) puts the 8 rows of a
// fragment tile in 8 distinct groups of 4 banks.
// Decoder: z_i = s (Wd . h_i + bd) dbar / d_i; the dot product in k_gnn_decode's
// order (its shuffle tree over 32 lanes, here over the fragment's columns), the
// FP64 scaling one node a thread.
//
// At 1M nodes (1024 x 1024, six neighbours) one layer takes 102 us, 112 us with
// the decoder; the aggregation and update kernels it replaces 85 + 85 us, the
// decoder 63 us.  It is bound by the L1 data path (71 % busy: the gathered rows,
// the weights' fragments, the edges handed round), then by instruction issue
// (45 %); DRAM is at 22 %.  Eight lanes a node, 128-node tiles and fragment
// loads by word: 154 us.
#define LTILE 256
#define MPAD (3 * W + 8)
#define LAYER_OCC 3
#define MMA_SMEM ((2 * W * MPAD + LTILE * MPAD) * (int)sizeof(__nv_bfloat16) + (2 * W + LTILE) * (int)sizeof(float))
__device__ __forceinline__ void ld_matrix4(unsigned (&r)[4], const __nv_bfloat16 *p)
{
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
	             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                         unsigned b0, unsigned b1)
{
	asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
	             "{%0,%1,%2,%3};"
	             : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
	             : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Two FP32 values in a register pair: acc += w * v, each rounded as fmaf.
__device__ __forceinline__ unsigned long long pair2(float lo, float hi)
{
	unsigned long long r;
	asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
	return r;
}
__device__ __forceinline__ void fma2(unsigned long long &acc, unsigned long long w, unsigned long long v)
{
	asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(w), "l"(v));
}
// The bf16 pair x as FP32.
__device__ __forceinline__ unsigned long long unpack2(unsigned x)
{
	return pair2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u));
}
__device__ __forceinline__ unsigned round2(unsigned long long v)
{
	float lo, hi;
	asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
	const __nv_bfloat162 o = __floats2bfloat162_rn(lo, hi);
	return *reinterpret_cast<const unsigned *>(&o);
}
// Up to four edges of each of the warp's eight nodes (cnt of the lane's node,
// `most' of any): the neighbours' rows, then their weighted sums in edge order.
// Edges a node does not have add zero times zero.
__device__ __forceinline__ void rows4(uint4 (&row)[4], const __nv_bfloat16 *h, int ec, int cnt, int most, int fl)
{
#pragma unroll
	for (int q = 0; q < 4; q++) {
		row[q] = make_uint4(0u, 0u, 0u, 0u);
		if (q < most) {                                   // uniform
			const int j = __shfl_sync(0xffffffffu, ec, q, 4);
			if (q < cnt) row[q] = __ldg(reinterpret_cast<const uint4 *>(&h[(size_t)j * W + fl]));
		}
	}
}
__device__ __forceinline__ void sum4(unsigned long long (&a1)[4], unsigned long long (&a2)[4], const uint4 (&row)[4],
                                     float ea, float et, int most)
{
#pragma unroll
	for (int q = 0; q < 4; q++) {
		if (q < most) {                                   // uniform
			const float wa = __shfl_sync(0xffffffffu, ea, q, 4), wt = __shfl_sync(0xffffffffu, et, q, 4);
			const unsigned long long pa = pair2(wa, wa), pt = pair2(wt, wt);
			const unsigned x[4] = {row[q].x, row[q].y, row[q].z, row[q].w};
#pragma unroll
			for (int f = 0; f < 4; f++) {
				const unsigned long long v = unpack2(x[f]);
				fma2(a1[f], pa, v);
				fma2(a2[f], pt, v);
			}
		}
	}
}
struct LayerArgs {
	int n;
	const int *gptr, *gcol;
	const float *wA, *wT, *th, *theta;    // the layer's weights, the whole parameter vector
	const __nv_bfloat16 *h;
	__nv_bfloat16 *m1, *m2, *hout;        // m1, m2: training only; hout: not by an inference's last layer
	unsigned *mask;                       // training only
	const double *stats, *d;              // last layer
	double *z;
	const int *active;
};
// The first eight edges of a node, two in each of its four lanes.
__device__ __forceinline__ void edges8(const LayerArgs &a, int lo, int hi, int el, int (&ec)[2], float (&ea)[2],
                                       float (&et)[2])
{
#pragma unroll
	for (int x = 0; x < 2; x++) {
		const int p = lo + 4 * x + el;
		ec[x] = 0;
		ea[x] = et[x] = 0.0f;
		if (p < hi) { ec[x] = __ldg(&a.gcol[p]); ea[x] = __ldg(&a.wA[p]); et[x] = __ldg(&a.wT[p]); }
	}
}
template <bool TRAIN, bool LAST>
__global__ void __launch_bounds__(UPD_TPB, LAYER_OCC) k_gnn_layer_mma(LayerArgs a)
{
	if (a.active && !*a.active) return;
	extern __shared__ __align__(16) unsigned char dynb[];
	__nv_bfloat16 *sWh = reinterpret_cast<__nv_bfloat16 *>(dynb);   // [W][MPAD]: W^T, row = output
	__nv_bfloat16 *sWl = sWh + W * MPAD;
	__nv_bfloat16 *sA = sWl + W * MPAD;                              // [LTILE][MPAD]: [h, m1, m2]
	float *sB = reinterpret_cast<float *>(sA + LTILE * MPAD);       // bias [W]
	float *sD = sB + W;                                             // decoder weights [W]
	float *sY = sD + W;                                             // decoder sums [LTILE]
	const int n = a.n;
	for (int e = threadIdx.x; e < 3 * W * W; e += blockDim.x) {
		int k = e / W, o = e - k * W;
		float w = a.th[e];
		__nv_bfloat16 hi = __float2bfloat16_rn(w);
		sWh[o * MPAD + k] = hi;
		sWl[o * MPAD + k] = __float2bfloat16_rn(w - __bfloat162float(hi));
	}
	if (threadIdx.x < W) {
		sB[threadIdx.x] = a.th[3 * W * W + threadIdx.x];
		if (LAST) sD[threadIdx.x] = a.theta[GNN_OFF_WD + threadIdx.x];
	}
	const int t = threadIdx.x, lane = t & 31, warp = t >> 5, g = lane >> 2, c = (lane & 3) * 2;
	const int el = lane & 3, fl = el * 8;
	// the two nodes a quarter warp stores together are four rows apart: 16 banks
	const int nl = warp * 8 + ((lane >> 2) & 1) * 4 + (lane >> 3);
	constexpr int NN = LTILE / (UPD_TPB / 4);              // nodes of four lanes, 64 rows apart
	const int ntile = (n + LTILE - 1) / LTILE;
	for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
		const int base = tile * LTILE;
		__syncthreads();                                  // the tile before is done with sA (and sY)
		// edge range of the node after the next, edges of the next, rows of this one
		int lo = 0, hi = 0, nlo = 0, nhi = 0, ec[2] = {0, 0};
		float ea[2] = {0.0f, 0.0f}, et[2] = {0.0f, 0.0f};     // edges 0-3, 4-7
		if (base + nl < n) { lo = __ldg(&a.gptr[base + nl]); hi = __ldg(&a.gptr[base + nl + 1]); }
		if (base + nl + UPD_TPB / 4 < n) {
			nlo = __ldg(&a.gptr[base + nl + UPD_TPB / 4]);
			nhi = __ldg(&a.gptr[base + nl + UPD_TPB / 4 + 1]);
		}
		edges8(a, lo, hi, el, ec, ea, et);
#pragma unroll 1
		for (int m = 0; m < NN; m++) {
			const int nd = nl + m * (UPD_TPB / 4), i = base + nd, cnt = hi - lo;
			const int most = __reduce_max_sync(0xffffffffu, cnt);
			uint4 own = make_uint4(0u, 0u, 0u, 0u), row[2][4];
			if (i < n) own = *reinterpret_cast<const uint4 *>(&a.h[(size_t)i * W + fl]);
			unsigned long long a1[4] = {0ull, 0ull, 0ull, 0ull}, a2[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
			for (int x = 0; x < 2; x++) rows4(row[x], a.h, ec[x], cnt - 4 * x, most - 4 * x, fl);
			int nc[2], flo = 0, fhi = 0;
			float na[2], nt_[2];
			edges8(a, nlo, nhi, el, nc, na, nt_);
			if (m + 2 < NN && i + 2 * (UPD_TPB / 4) < n) {
				flo = __ldg(&a.gptr[i + 2 * (UPD_TPB / 4)]);
				fhi = __ldg(&a.gptr[i + 2 * (UPD_TPB / 4) + 1]);
			}
#pragma unroll
			for (int x = 0; x < 2; x++) sum4(a1, a2, row[x], ea[x], et[x], most - 4 * x);
			for (int p = 8; p < most; p += 4) {               // more than eight edges
				int c4 = 0;
				float wa = 0.0f, wt = 0.0f;
				if (p + el < cnt) {
					c4 = __ldg(&a.gcol[lo + p + el]);
					wa = __ldg(&a.wA[lo + p + el]);
					wt = __ldg(&a.wT[lo + p + el]);
				}
				rows4(row[0], a.h, c4, cnt - p, most - p, fl);
				sum4(a1, a2, row[0], wa, wt, most - p);
			}
			lo = nlo; hi = nhi; nlo = flo; nhi = fhi;
#pragma unroll
			for (int x = 0; x < 2; x++) { ec[x] = nc[x]; ea[x] = na[x]; et[x] = nt_[x]; }
			const uint4 o1 = make_uint4(round2(a1[0]), round2(a1[1]), round2(a1[2]), round2(a1[3]));
			const uint4 o2 = make_uint4(round2(a2[0]), round2(a2[1]), round2(a2[2]), round2(a2[3]));
			__nv_bfloat16 *dst = sA + nd * MPAD + fl;
			*reinterpret_cast<uint4 *>(dst) = own;
			*reinterpret_cast<uint4 *>(dst + W) = o1;
			*reinterpret_cast<uint4 *>(dst + 2 * W) = o2;
			if (TRAIN && i < n) {
				*reinterpret_cast<uint4 *>(&a.m1[(size_t)i * W + fl]) = o1;
				*reinterpret_cast<uint4 *>(&a.m2[(size_t)i * W + fl]) = o2;
			}
		}
		__syncthreads();
		float acc[2][4][4];
		#pragma unroll
		for (int mt = 0; mt < 2; mt++)
			#pragma unroll
			for (int nt = 0; nt < 4; nt++) {
				acc[mt][nt][0] = acc[mt][nt][2] = sB[nt * 8 + c];
				acc[mt][nt][1] = acc[mt][nt][3] = sB[nt * 8 + c + 1];
			}
		// fragments by ldmatrix: lane l names row l of the four 8x8 tiles of a load
		const __nv_bfloat16 *ra = sA + (warp * 32 + (lane & 15)) * MPAD + (lane >> 4) * 8;
		const int bo = ((lane >> 4) * 8 + (lane & 7)) * MPAD + ((lane >> 3) & 1) * 8;
		#pragma unroll
		for (int ks = 0; ks < 3 * W / 16; ks++) {
			unsigned fa[2][4];
			ld_matrix4(fa[0], ra + ks * 16);
			ld_matrix4(fa[1], ra + 16 * MPAD + ks * 16);
			#pragma unroll
			for (int o = 0; o < 2; o++) {                     // outputs 16 o .. 16 o + 15
				unsigned fh[4], fw[4];
				ld_matrix4(fh, sWh + o * 16 * MPAD + bo + ks * 16);
				ld_matrix4(fw, sWl + o * 16 * MPAD + bo + ks * 16);
				#pragma unroll
				for (int mt = 0; mt < 2; mt++)
					#pragma unroll
					for (int q = 0; q < 2; q++) {
						float (&ac)[4] = acc[mt][2 * o + q];
						mma_bf16(ac, fa[mt][0], fa[mt][1], fa[mt][2], fa[mt][3], fh[2 * q], fh[2 * q + 1]);
						mma_bf16(ac, fa[mt][0], fa[mt][1], fa[mt][2], fa[mt][3], fw[2 * q], fw[2 * q + 1]);
					}
			}
		}
		#pragma unroll
		for (int rr = 0; rr < 4; rr++) {
			const int nd = warp * 32 + g + 8 * rr, i = base + nd;
			const __nv_bfloat16 *in = sA + nd * MPAD;
			unsigned bits = 0;
			float hv[4][2];                               // the new activations, as stored
			#pragma unroll
			for (int nt = 0; nt < 4; nt++) {
				int col = nt * 8 + c;
				float u0 = acc[rr >> 1][nt][2 * (rr & 1)], u1 = acc[rr >> 1][nt][2 * (rr & 1) + 1];
				if (TRAIN) {
					bits |= (u0 > 0.0f ? 1u : 0u) << col;
					bits |= (u1 > 0.0f ? 1u : 0u) << (col + 1);
				}
				__nv_bfloat162 o;
				o.x = __float2bfloat16_rn(__bfloat162float(in[col]) + (u0 > 0.0f ? u0 : 0.0f));
				o.y = __float2bfloat16_rn(__bfloat162float(in[col + 1]) + (u1 > 0.0f ? u1 : 0.0f));
				if ((TRAIN || !LAST) && i < n) *reinterpret_cast<__nv_bfloat162 *>(&a.hout[(size_t)i * W + col]) = o;
				hv[nt][0] = __bfloat162float(o.x);
				hv[nt][1] = __bfloat162float(o.y);
			}
			if (TRAIN) {
				bits |= __shfl_xor_sync(0xffffffffu, bits, 1);
				bits |= __shfl_xor_sync(0xffffffffu, bits, 2);
				if (i < n && (lane & 3) == 0) a.mask[i] = bits;
			}
			if (LAST) {
				// features f and f + 16, then + 8, 4, 2, 1, as the lanes of k_gnn_decode
				float y[2];
				#pragma unroll
				for (int x = 0; x < 2; x++) {
					float v[2];
					#pragma unroll
					for (int nt = 0; nt < 2; nt++)
						v[nt] = __fadd_rn(__fmul_rn(hv[nt][x], sD[nt * 8 + c + x]),
						                  __fmul_rn(hv[nt + 2][x], sD[(nt + 2) * 8 + c + x]));
					y[x] = v[0] + v[1];
				}
				#pragma unroll
				for (int o = 2; o > 0; o >>= 1)
					#pragma unroll
					for (int x = 0; x < 2; x++) y[x] += __shfl_xor_sync(0xffffffffu, y[x], o);
				if ((lane & 3) == 0) sY[nd] = y[0] + y[1];
			}
		}
		if (LAST) {
			__syncwarp();                                 // a warp's own 32 nodes
			const int i = base + t;
			if (i < n) a.z[i] = a.stats[0] * (double)(sY[t] + __ldg(&a.theta[GNN_OFF_BD])) * a.stats[1] / a.d[i];
		}
	}
}

// z_i = s (Wd . h_i + bd) dbar / d_i: a warp reduces the rows of 32
// consecutive nodes (lane = feature), lane q keeps node q's sum and does its
// FP64 scaling (once per node).
template <typename TA>
__global__ void k_gnn_decode(int n, const TA *h, const float *__restrict__ th, const double *stats,
                             const double *d, double *z, const int *active)
{
	if (active && !*active) return;
	const int lane = threadIdx.x & 31;
	const float wd = th[GNN_OFF_WD + lane], bd = th[GNN_OFF_BD];
	const double s = stats[0], dbar = stats[1];
	int warps = (gridDim.x * blockDim.x) >> 5;
	for (int g0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; g0 < n; g0 += warps * 32) {
		int cnt = min(32, n - g0);
		float mine = 0.0f;
		for (int q = 0; q < cnt; q++) {
			float y = fg_warp_sumf(ld_act(&h[(size_t)(g0 + q) * W + lane]) * wd);
			if (lane == q) mine = y;
		}
		int i = g0 + lane;
		if (i < n) z[i] = s * (double)(mine + bd) * dbar / d[i];
	}
}

// Loss gradients dL/dz: supervised (ILU target) 2 (z - t) / sum t^2, and
// residual 2 A^T (A z - v) / sum v^2 with A = diag(d) (I + W) from the graph
// (a_ij = d_i wA_ij; (A^T y)_j = d_j y_j + sum_q wT[q] d_col y_col).
__global__ void k_gnn_gz_sup(int n, const double *z, const double *t, const double *sums, double *gz)
{
	const double T2 = sums[0];
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
		gz[i] = 2.0 * (z[i] - t[i]) / T2;
}

// res = A z - v and the loss sums out[0] = sum v_i^2, out[1] = sum res_i^2: each
// thread sums what it computes, in k_gnn_psums's order, and the last block to
// finish adds the partial sums up as k_gnn_fsums does.  65k nodes: 9.7 us; six
// launches (the residual, two sums of two kernels, a copy) took 21 and ten of
// gaps, the residual part of dL/dz in a kernel before k_gnn_decode_bwd six more.
__global__ void __launch_bounds__(RTPB) k_gnn_resid(int n, const int *__restrict__ gptr, const int *__restrict__ gcol,
                            const float *__restrict__ wA, const double *d, const double *z, const double *v,
                            double *res, double *part, unsigned *ticket, double *out)
{
	__shared__ double sh[32];
	__shared__ bool last;
	double s0 = 0.0, s1 = 0.0;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		const double vi = v[i];
		double s = z[i];
		for (int p = gptr[i]; p < gptr[i + 1]; p++) s += (double)wA[p] * z[gcol[p]];
		const double e = d[i] * s - vi;
		res[i] = e;
		s0 += vi * vi;
		s1 += e * e;
	}
	s0 = blk_sum(s0, sh);
	s1 = blk_sum(s1, sh);
	if (threadIdx.x == 0) {
		part[2 * blockIdx.x] = s0;
		part[2 * blockIdx.x + 1] = s1;
		__threadfence();
		last = atomicAdd(ticket, 1u) == gridDim.x - 1;
	}
	__syncthreads();
	if (!last) return;
	double t0 = 0.0, t1 = 0.0;
	for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) {
		t0 += __ldcg(&part[2 * b]);
		t1 += __ldcg(&part[2 * b + 1]);
	}
	t0 = blk_sum(t0, sh);
	t1 = blk_sum(t1, sh);
	if (threadIdx.x == 0) { out[0] = t0; out[1] = t1; *ticket = 0u; }
}

// The residual loss's part of dL/dz (see k_gnn_gz_sup): its graph and A z - v.
struct ResGrad { const int *gptr, *gcol; const float *wT; const double *res, *sums; };

// gh = gy Wd with gy = gz s dbar / d; partials of gWd (32), gbd (1).  A warp
// takes 32 nodes, lane q forming node q's gy (FP64) and lane f then feature f of
// every node, so each row is one coalesced access and a lane keeps one sum.
// SUP: gz has the supervised part; RES: the residual part is formed here.
template <typename TA, bool SUP, bool RES>
__global__ void __launch_bounds__(RTPB) k_gnn_decode_bwd(int n, const double *gzv, ResGrad rg, const double *stats,
		const double *d, const TA *h, const float *__restrict__ th, float *gh, float *part)
{
	__shared__ float sacc[RTPB / 32][W], sbd[RTPB / 32];
	const double s = stats[0], dbar = stats[1];
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = (gridDim.x * blockDim.x) >> 5;
	const float wd = th[GNN_OFF_WD + lane];
	const double c = RES ? 2.0 / rg.sums[0] : 0.0;
	float acc = 0.0f, accb = 0.0f;
	for (int g0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; g0 < n; g0 += warps * 32) {
		const int i = g0 + lane, cnt = min(32, n - g0);
		float mine = 0.0f;
		if (i < n) {
			double gz = SUP ? gzv[i] : 0.0;
			const double di = d[i];
			if (RES) {
				double r = di * rg.res[i];
				for (int q = __ldg(&rg.gptr[i]); q < __ldg(&rg.gptr[i + 1]); q++) {
					const int k = __ldg(&rg.gcol[q]);
					r += (double)__ldg(&rg.wT[q]) * d[k] * rg.res[k];
				}
				gz = SUP ? gz + c * r : c * r;
			}
			mine = (float)(gz * s * dbar / di);
		}
		accb += mine;
		#pragma unroll 8
		for (int q = 0; q < cnt; q++) {
			const float gy = __shfl_sync(0xffffffffu, mine, q);
			const size_t o = (size_t)(g0 + q) * W + lane;
			gh[o] = gy * wd;
			acc += gy * ld_act(&h[o]);
		}
	}
	accb = fg_warp_sumf(accb);
	sacc[wid][lane] = acc;
	if (lane == 0) sbd[wid] = accb;
	__syncthreads();
	if (threadIdx.x <= W) {
		float v = 0.0f;
		for (int w = 0; w < RTPB / 32; w++) v += threadIdx.x < W ? sacc[w][threadIdx.x] : sbd[w];
		part[(size_t)blockIdx.x * (W + 1) + threadIdx.x] = v;
	}
}

// One layer backward, gathers and products in one kernel, on tiles of 64 nodes:
//   gu = gh_out * [u > 0]
//   gh_in_j = gh_out_j + Wh gu_j + W1 sum_q wT[q] gu_col + W2 sum_q wA[q] gu_col
//   partials: gWh, gW1, gW2 (sum over nodes of input (x) gu), gb (sum gu).
// The transposed aggregation and the weight products commute, so one row of gu
// per neighbour is gathered instead of the two rows W1 gu and W2 gu, and those
// are never stored.  Both products run in FP32 from shared memory on register
// tiles (8 nodes x 4 inputs, 12 inputs x 4 outputs, a quarter of the block each
// taking a quarter of the sum): they bound the kernel, 6.1k FMA a node against
// the shared-memory words they read, 2.7 and 3 FMA a word.  65k nodes: 36 us a
// layer; the separate update and aggregation kernels took 103 + 15.5 us.
template <typename TA> __device__ __forceinline__ float4 ld_act4(const TA *p);
template <> __device__ __forceinline__ float4 ld_act4<float>(const float *p) { return *reinterpret_cast<const float4 *>(p); }
template <> __device__ __forceinline__ float4 ld_act4<__nv_bfloat16>(const __nv_bfloat16 *p)
{
	const uint2 raw = *reinterpret_cast<const uint2 *>(p);
	const __nv_bfloat16 *v = reinterpret_cast<const __nv_bfloat16 *>(&raw);
	return make_float4(__bfloat162float(v[0]), __bfloat162float(v[1]), __bfloat162float(v[2]), __bfloat162float(v[3]));
}
__device__ __forceinline__ void gather_rows4(float4 (&row)[8], const float *g, int ec, int cnt, int fl)
{
	#pragma unroll
	for (int q = 0; q < 8; q++) {
		const int j = __shfl_sync(0xffffffffu, ec, q, 8);
		row[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
		if (q < cnt) row[q] = __ldg(reinterpret_cast<const float4 *>(&g[(size_t)j * W + fl]));
	}
}
__device__ __forceinline__ void add_rows4(float (&a1)[4], float (&a2)[4], const float4 (&row)[8], float e1, float e2,
                                          unsigned em, int cnt, int fl)
{
	#pragma unroll
	for (int q = 0; q < 8; q++) {
		const float w1 = __shfl_sync(0xffffffffu, e1, q, 8), w2 = __shfl_sync(0xffffffffu, e2, q, 8);
		const unsigned mk = __shfl_sync(0xffffffffu, em, q, 8) >> fl;
		if (q < cnt) {
			const float v[4] = {row[q].x, row[q].y, row[q].z, row[q].w};
			#pragma unroll
			for (int f = 0; f < 4; f++) {
				const float gv = (mk >> f) & 1u ? v[f] : 0.0f;
				a1[f] = fmaf(w1, gv, a1[f]);
				a2[f] = fmaf(w2, gv, a2[f]);
			}
		}
	}
}
#define XPAD (TILE + 2)
#define GPAD (W + 4)
#define IPAD (3 * W + 4)
#define BWD_SMEM ((3 * W * W + 3 * W * XPAD + TILE * IPAD + 5 * TILE * GPAD) * (int)sizeof(float))
template <typename TA>
__global__ void __launch_bounds__(UPD_TPB, 2) k_gnn_layer_bwd(int n, const int *__restrict__ gptr,
		const int *__restrict__ gcol, const float *__restrict__ wA, const float *__restrict__ wT,
		const float *__restrict__ th, const TA *h, const TA *m1, const TA *m2, const unsigned *__restrict__ mask,
		const float *__restrict__ gh_out, float *gh_in, float *part)
{
	extern __shared__ __align__(16) float dynf[];
	float *sW = dynf;                                  // [3W][W]: row (m, f), column k: W_m[k][f]
	float *sX = sW + 3 * W * W;                        // [3W][XPAD]: gu and its two aggregates, transposed
	float *sIn = sX + 3 * W * XPAD;                    // [TILE][IPAD]: h, m1, m2
	float *sG = sIn + TILE * IPAD;                     // [TILE][GPAD]: gu
	float *sP = sG + TILE * GPAD;                      // [4][TILE][GPAD]: the quarters' input gradients
	for (int e = threadIdx.x; e < 3 * W * W; e += blockDim.x) {
		int m = e / (W * W), r = e - m * W * W, f = r / W, k = r - f * W;
		sW[e] = th[m * W * W + k * W + f];
	}
	const int t = threadIdx.x, el = t & 7, fl = el * 4;
	const int qt = t >> 6, og = (t >> 3) & 7;
	float acc[12][4], accb[4];
	#pragma unroll
	for (int q = 0; q < 4; q++) {
		#pragma unroll
		for (int k = 0; k < 12; k++) acc[k][q] = 0.0f;
		accb[q] = 0.0f;
	}
	const int ntile = (n + TILE - 1) / TILE;
	for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
		const int base = tile * TILE;
		__syncthreads();
		constexpr int NN = TILE / (UPD_TPB / 8);
		int lo[NN], hi[NN], ec[NN];
		unsigned em[NN], bits[NN];
		float ea[NN], et[NN];
		float4 own[NN];
		#pragma unroll
		for (int k = 0; k < NN; k++) {
			const int i = base + (t >> 3) + k * (UPD_TPB / 8);
			lo[k] = hi[k] = 0;
			bits[k] = 0u;
			own[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
			if (i < n) {
				lo[k] = __ldg(&gptr[i]);
				hi[k] = __ldg(&gptr[i + 1]);
				own[k] = *reinterpret_cast<const float4 *>(&gh_out[(size_t)i * W + fl]);
				bits[k] = __ldg(&mask[i]) >> fl;
			}
		}
		#pragma unroll
		for (int k = 0; k < NN; k++) {
			ec[k] = 0;
			em[k] = 0u;
			ea[k] = et[k] = 0.0f;
			if (lo[k] + el < hi[k]) {
				ec[k] = __ldg(&gcol[lo[k] + el]);
				ea[k] = __ldg(&wA[lo[k] + el]);
				et[k] = __ldg(&wT[lo[k] + el]);
				em[k] = __ldg(&mask[ec[k]]);
			}
		}
		// the inputs, while the neighbours' rows are on their way
		#pragma unroll
		for (int k = 0; k < NN; k++) {
			const int nd = (t >> 3) + k * (UPD_TPB / 8), i = base + nd;
			float4 row[8];
			gather_rows4(row, gh_out, ec[k], hi[k] - lo[k], fl);
			#pragma unroll
			for (int m = 0; m < 3; m++) {
				const TA *src = m == 0 ? h : (m == 1 ? m1 : m2);
				float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
				if (i < n) v = ld_act4(&src[(size_t)i * W + fl]);
				*reinterpret_cast<float4 *>(&sIn[nd * IPAD + m * W + fl]) = v;
			}
			float a1[4] = {0.0f, 0.0f, 0.0f, 0.0f}, a2[4] = {0.0f, 0.0f, 0.0f, 0.0f};
			add_rows4(a1, a2, row, et[k], ea[k], em[k], hi[k] - lo[k], fl);
			for (int p = lo[k] + 8; __any_sync(0xffffffffu, p < hi[k]); p += 8) {    // more than eight edges
				int c8 = 0;
				unsigned m8 = 0u;
				float wa = 0.0f, wt = 0.0f;
				if (p + el < hi[k]) {
					c8 = __ldg(&gcol[p + el]);
					wa = __ldg(&wA[p + el]);
					wt = __ldg(&wT[p + el]);
					m8 = __ldg(&mask[c8]);
				}
				gather_rows4(row, gh_out, c8, hi[k] - p, fl);
				add_rows4(a1, a2, row, wt, wa, m8, hi[k] - p, fl);
			}
			const float o[4] = {own[k].x, own[k].y, own[k].z, own[k].w};
			float gu[4];
			#pragma unroll
			for (int f = 0; f < 4; f++) {
				gu[f] = (bits[k] >> f) & 1u ? o[f] : 0.0f;
				sX[(fl + f) * XPAD + nd] = gu[f];
				sX[(W + fl + f) * XPAD + nd] = a1[f];
				sX[(2 * W + fl + f) * XPAD + nd] = a2[f];
			}
			*reinterpret_cast<float4 *>(&sG[nd * GPAD + fl]) = make_float4(gu[0], gu[1], gu[2], gu[3]);
		}
		__syncthreads();
		// input gradients: a quarter of the block takes 24 of the 96 rows, a
		// thread 8 nodes x features fl .. fl+3 of them
		{
			float v[8][4];
			#pragma unroll
			for (int q = 0; q < 8; q++)
				#pragma unroll
				for (int f = 0; f < 4; f++) v[q][f] = 0.0f;
			#pragma unroll 4
			for (int r = 24 * qt; r < 24 * qt + 24; r++) {
				const float4 w = *reinterpret_cast<const float4 *>(&sW[r * W + fl]);
				#pragma unroll
				for (int q = 0; q < 8; q += 2) {
					const float2 x = *reinterpret_cast<const float2 *>(&sX[r * XPAD + 8 * og + q]);
					v[q][0] += x.x * w.x; v[q][1] += x.x * w.y; v[q][2] += x.x * w.z; v[q][3] += x.x * w.w;
					v[q + 1][0] += x.y * w.x; v[q + 1][1] += x.y * w.y; v[q + 1][2] += x.y * w.z; v[q + 1][3] += x.y * w.w;
				}
			}
			#pragma unroll
			for (int q = 0; q < 8; q++)
				*reinterpret_cast<float4 *>(&sP[(qt * TILE + 8 * og + q) * GPAD + fl]) =
					make_float4(v[q][0], v[q][1], v[q][2], v[q][3]);
		}
		// weight gradients: a quarter of the block takes 16 of the 64 nodes, a
		// thread rows 12 og .. +11 of the 96 x outputs fl .. fl+3
		#pragma unroll 2
		for (int nd = 16 * qt; nd < 16 * qt + 16; nd++) {
			const float4 gv = *reinterpret_cast<const float4 *>(&sG[nd * GPAD + fl]);
			#pragma unroll
			for (int k = 0; k < 12; k += 4) {
				const float4 x = *reinterpret_cast<const float4 *>(&sIn[nd * IPAD + 12 * og + k]);
				const float xs[4] = {x.x, x.y, x.z, x.w};
				#pragma unroll
				for (int m = 0; m < 4; m++) {
					acc[k + m][0] += xs[m] * gv.x; acc[k + m][1] += xs[m] * gv.y;
					acc[k + m][2] += xs[m] * gv.z; acc[k + m][3] += xs[m] * gv.w;
				}
			}
			if (og == 0) { accb[0] += gv.x; accb[1] += gv.y; accb[2] += gv.z; accb[3] += gv.w; }
		}
		__syncthreads();
		#pragma unroll
		for (int k = 0; k < TILE / (UPD_TPB / 8); k++) {
			const int nd = (t >> 3) + k * (UPD_TPB / 8), i = base + nd;
			if (i >= n) continue;
			float4 o = *reinterpret_cast<const float4 *>(&gh_out[(size_t)i * W + fl]);
			#pragma unroll
			for (int q = 0; q < 4; q++) {
				const float4 x = *reinterpret_cast<const float4 *>(&sP[(q * TILE + nd) * GPAD + fl]);
				o.x += x.x; o.y += x.y; o.z += x.z; o.w += x.w;
			}
			*reinterpret_cast<float4 *>(&gh_in[(size_t)i * W + fl]) = o;
		}
	}
	// the quarters' weight gradients, added in their order
	float *pb = part + (size_t)blockIdx.x * (3 * W * W + W);
	for (int q = 0; q < 4; q++) {
		__syncthreads();
		if (qt != q) continue;
		#pragma unroll
		for (int k = 0; k < 13; k++) {                        // row 12: the bias gradient
			if (k == 12 && og) continue;
			const int at = (k < 12 ? 12 * og + k : 3 * W) * W + fl;
			const float *v = k < 12 ? acc[k < 12 ? k : 0] : accb;
			float4 o = make_float4(v[0], v[1], v[2], v[3]);
			if (q) {
				const float4 x = *reinterpret_cast<const float4 *>(&sP[at]);
				o.x += x.x; o.y += x.y; o.z += x.z; o.w += x.w;
			}
			*reinterpret_cast<float4 *>(q < 3 ? &sP[at] : &pb[at]) = o;
		}
	}
}

// gpre = gh * [pre > 0]; partials gWe (2 x 32), gbe (32).  Lanes as in
// k_gnn_decode_bwd.
__global__ void __launch_bounds__(RTPB) k_gnn_encode_bwd(int n, const float2 *x, const unsigned *mask0,
                                                         const float *gh, float *part)
{
	__shared__ float sacc[RTPB / 32][3 * W];
	const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = (gridDim.x * blockDim.x) >> 5;
	float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f;
	for (int g0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; g0 < n; g0 += warps * 32) {
		const int i = g0 + lane, cnt = min(32, n - g0);
		const float2 mine = i < n ? x[i] : make_float2(0.0f, 0.0f);
		const unsigned mk = i < n ? mask0[i] : 0u;
		#pragma unroll 8
		for (int q = 0; q < cnt; q++) {
			const float xa = __shfl_sync(0xffffffffu, mine.x, q), xb = __shfl_sync(0xffffffffu, mine.y, q);
			const unsigned m = __shfl_sync(0xffffffffu, mk, q);
			const float v = gh[(size_t)(g0 + q) * W + lane], g = (m >> lane) & 1u ? v : 0.0f;
			s0 += xa * g;
			s1 += xb * g;
			s2 += g;
		}
	}
	sacc[wid][lane] = s0;
	sacc[wid][W + lane] = s1;
	sacc[wid][2 * W + lane] = s2;
	__syncthreads();
	for (int f = threadIdx.x; f < 3 * W; f += blockDim.x) {
		float v = 0.0f;
		for (int w = 0; w < RTPB / 32; w++) v += sacc[w][f];
		part[(size_t)blockIdx.x * 3 * W + f] = v;
	}
}

// Every stage's partial sums into the gradient in one launch: 32 entries a
// block, eight slices of the stage's blocks beside each other (a warp reads 32
// neighbouring entries), the slices added in order.
struct RedStage { const float *part; float *grad; int nblk, cnt, first; };   // first: of its blocks
struct RedArgs { RedStage st[GNN_LAYERS + 2]; };
__global__ void __launch_bounds__(256) k_gnn_reduce(RedArgs a, int accumulate)
{
	__shared__ float sl[8][32];
	int s = 0;
	while (s + 1 < GNN_LAYERS + 2 && (int)blockIdx.x >= a.st[s + 1].first) s++;
	const RedStage r = a.st[s];
	const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5, e = ((int)blockIdx.x - r.first) * 32 + lane;
	float v = 0.0f;
	if (e < r.cnt)
		for (int b = slice; b < r.nblk; b += 8) v += r.part[(size_t)b * r.cnt + e];
	sl[slice][lane] = v;
	__syncthreads();
	if (slice == 0 && e < r.cnt) {
		float t = 0.0f;
		for (int q = 0; q < 8; q++) t += sl[q][lane];
		r.grad[e] = accumulate ? r.grad[e] + t : t;
	}
}

__global__ void k_gnn_adam(int P, float *th, const float *g, float *m, float *v, float lr, float b1, float b2,
                           float eps, float c1, float c2, float gscale)
{
	for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < P; k += gridDim.x * blockDim.x) {
		float gk = g[k] * gscale;
		float mk = b1 * m[k] + (1.0f - b1) * gk;
		float vk = b2 * v[k] + (1.0f - b2) * gk * gk;
		m[k] = mk;
		v[k] = vk;
		th[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
	}
}

__global__ void k_gnn_dbar(const double *sums, int n, double *stats) { stats[1] = sums[0] / n; }

// ---------------------------------------------------------------- launchers
#define UPD_SMEM ((3 * W * W + W + UTILE * PAD) * (int)sizeof(float))

static int update_attrs()
{
	static int done = 0;
	if (!done) {
		FG_TRY(cudaFuncSetAttribute(k_gnn_update<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, UPD_SMEM));
		FG_TRY(cudaFuncSetAttribute(k_gnn_update<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                            UPD_SMEM));
		FG_TRY(cudaFuncSetAttribute(k_gnn_layer_mma<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MMA_SMEM));
		FG_TRY(cudaFuncSetAttribute(k_gnn_layer_mma<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MMA_SMEM));
		FG_TRY(cudaFuncSetAttribute(k_gnn_layer_mma<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, MMA_SMEM));
		FG_TRY(cudaFuncSetAttribute(k_gnn_layer_mma<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, MMA_SMEM));
		FG_TRY(cudaFuncSetAttribute(k_gnn_layer_bwd<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM));
		FG_TRY(cudaFuncSetAttribute(k_gnn_layer_bwd<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                            BWD_SMEM));
		done = 1;
	}
	return 0;
}
// bf16 activations take the tensor-core update unless FEMGPU_GNN_MMA=0
// (read at every launch: the FP32-core form stays available for comparison)
static bool update_mma()
{
	const char *e = getenv("FEMGPU_GNN_MMA");
	return !(e && e[0] == '0');
}
static int nb(long long n, int tpb, int cap)
{
	return (int)std::max<long long>(1, std::min<long long>((n + tpb - 1) / tpb, cap));
}

static void sums(fg_gnn *g, int n, const double *a, const double *b, int absval, double *out,
                 const int *active = nullptr)
{
	k_gnn_psums<<<GNN_RED_BLOCKS, RTPB, 0, g->stream>>>(n, a, b, absval, g->rpart, active);
	k_gnn_fsums<<<1, RTPB, 0, g->stream>>>(GNN_RED_BLOCKS, g->rpart, out, active);
}

extern "C" int fg_gnn_graph(fg_gnn *g, int n, const int *IA, const int *JA, const double *AA)
{
	k_gnn_graph<<<nb(n, 256, 16 * FG_SMS), 256, 0, g->stream>>>(n, IA, JA, AA, g->gptr, g->gcol, g->wA, g->wT, g->d,
	                                                          &g->err[0]);
	FG_TRY(cudaGetLastError());
	sums(g, n, g->d, nullptr, 1, g->sums);
	k_gnn_dbar<<<1, 1, 0, g->stream>>>(g->sums, n, g->stats);
	return (int)cudaGetLastError();
}

template <typename TA>
static int forward_t(fg_gnn *g, const double *r, double *z, int train, const int *active)
{
	cudaStream_t s = g->stream;
	int n = g->n;
	TA **H = (TA **)g->h, **M1 = (TA **)g->m1, **M2 = (TA **)g->m2;
	FG_TRY((cudaError_t)update_attrs());
	k_gnn_rms<<<GNN_RED_BLOCKS, RTPB, 0, s>>>(n, r, g->rpart, g->ticket, g->sums, g->stats, active);
	k_gnn_encode<TA><<<nb(n, 256, 16 * FG_SMS), 256, 0, s>>>(n, r, g->stats, g->d, g->theta, H[0],
	                                                         train ? g->mask[0] : nullptr,
	                                                         train ? (float2 *)g->x : nullptr, active);
	const bool mma = std::is_same<TA, __nv_bfloat16>::value && update_mma();
	for (int l = 0; l < GNN_LAYERS; l++) {
		int cur = train ? l : (l & 1), nxt = train ? l + 1 : ((l + 1) & 1);
		int ml = train ? l : 0;
		if (mma) {
			LayerArgs a;
			a.n = n; a.gptr = g->gptr; a.gcol = g->gcol; a.wA = g->wA; a.wT = g->wT;
			a.th = g->theta + GNN_OFF_L(l); a.theta = g->theta;
			a.h = (const __nv_bfloat16 *)g->h[cur]; a.hout = (__nv_bfloat16 *)g->h[nxt];
			a.m1 = (__nv_bfloat16 *)g->m1[ml]; a.m2 = (__nv_bfloat16 *)g->m2[ml];
			a.mask = g->mask[l + 1]; a.stats = g->stats; a.d = g->d; a.z = z; a.active = active;
			const int grid = nb(n, LTILE, LAYER_OCC * FG_SMS);
			const bool last = l == GNN_LAYERS - 1;
			if (train && last) k_gnn_layer_mma<true, true><<<grid, UPD_TPB, MMA_SMEM, s>>>(a);
			else if (train) k_gnn_layer_mma<true, false><<<grid, UPD_TPB, MMA_SMEM, s>>>(a);
			else if (last) k_gnn_layer_mma<false, true><<<grid, UPD_TPB, MMA_SMEM, s>>>(a);
			else k_gnn_layer_mma<false, false><<<grid, UPD_TPB, MMA_SMEM, s>>>(a);
			continue;
		}
		k_gnn_agg<TA><<<nb(8LL * n, 256, 32 * FG_SMS), 256, 0, s>>>(n, g->gptr, g->gcol, g->wA, g->wT, H[cur],
		                                                            M1[ml], M2[ml], active);
		k_gnn_update<TA><<<nb(n, UTILE, 4 * FG_SMS), UPD_TPB, UPD_SMEM, s>>>(n, g->theta + GNN_OFF_L(l), H[cur],
		                                                                   M1[ml], M2[ml], H[nxt],
		                                                                   train ? g->mask[l + 1] : nullptr, active);
	}
	if (!mma)
		k_gnn_decode<TA><<<nb(n, 256, 16 * FG_SMS), 256, 0, s>>>(n, H[train ? GNN_LAYERS : (GNN_LAYERS & 1)], g->theta,
		                                                         g->stats, g->d, z, active);
	return (int)cudaGetLastError();
}

extern "C" int fg_gnn_forward(fg_gnn *g, const double *r, double *z, int train, const int *active)
{
	return g->bf16 ? forward_t<__nv_bfloat16>(g, r, z, train, active)
	               : forward_t<float>(g, r, z, train, active);
}

template <typename TA>
static int backward_t(fg_gnn *g, const double *r, const double *z, const double *t, int accumulate)
{
	cudaStream_t s = g->stream;
	int n = g->n;
	TA **H = (TA **)g->h, **M1 = (TA **)g->m1, **M2 = (TA **)g->m2;
	const int PL = 3 * W * W + W;
	int gn = nb(n, 256, 16 * FG_SMS);
	// loss sums in g->lsums: [0] = normaliser, [1] = squared error (loss = [1]/[0])
	ResGrad rg = { nullptr, nullptr, nullptr, nullptr, nullptr };
	if (g->loss_kind != GNN_LOSS_RESIDUAL) {
		sums(g, n, t, z, 0, g->lsums);            // sum t^2, sum (z - t)^2
		k_gnn_gz_sup<<<gn, 256, 0, s>>>(n, z, t, g->lsums, g->gz);
	}
	if (g->loss_kind != GNN_LOSS_SUPERVISED) {
		double *ls = g->loss_kind == GNN_LOSS_RESIDUAL ? g->lsums : g->lsums2;
		k_gnn_resid<<<GNN_RED_BLOCKS, RTPB, 0, s>>>(n, g->gptr, g->gcol, g->wA, g->d, z, r, g->res, g->rpart, g->ticket, ls);
		rg = ResGrad{g->gptr, g->gcol, g->wT, g->res, ls};
	}
	// partial sums of the stages, one after another in g->part
	RedArgs red;
	float *pt = g->part;
	int blocks = 0;
	auto stage = [&](int k, int nblk, int cnt, int off) {
		red.st[k] = RedStage{pt, g->grad + off, nblk, cnt, blocks};
		pt += ((size_t)nblk * cnt + 3) & ~(size_t)3;         // the next stage's 16-byte stores
		blocks += (cnt + 31) / 32;
		return red.st[k].part;
	};
	int gd = nb(n, RTPB, GNN_BWD_BLOCKS);
	float *pd = (float *)stage(0, gd, W + 1, GNN_OFF_WD);
#define DECODE_BWD(S, R) k_gnn_decode_bwd<TA, S, R><<<gd, RTPB, 0, s>>>(n, g->gz, rg, g->stats, g->d, H[GNN_LAYERS], \
	g->theta, g->gh[0], pd)
	if (g->loss_kind == GNN_LOSS_RESIDUAL) DECODE_BWD(false, true);
	else if (g->loss_kind == GNN_LOSS_SUPERVISED) DECODE_BWD(true, false);
	else DECODE_BWD(true, true);
#undef DECODE_BWD
	int cur = 0;
	int gu = nb(n, TILE, GNN_BWD_BLOCKS);
	for (int l = GNN_LAYERS - 1; l >= 0; l--) {
		k_gnn_layer_bwd<TA><<<gu, UPD_TPB, BWD_SMEM, s>>>(n, g->gptr, g->gcol, g->wA, g->wT, g->theta + GNN_OFF_L(l),
		                                                 H[l], M1[l], M2[l], g->mask[l + 1], g->gh[cur],
		                                                 g->gh[cur ^ 1],
		                                                 (float *)stage(GNN_LAYERS - l, gu, PL, GNN_OFF_L(l)));
		cur ^= 1;
	}
	k_gnn_encode_bwd<<<gd, RTPB, 0, s>>>(n, (const float2 *)g->x, g->mask[0], g->gh[cur],
	                                     (float *)stage(GNN_LAYERS + 1, gd, 3 * W, GNN_OFF_WE));
	k_gnn_reduce<<<blocks, 256, 0, s>>>(red, accumulate);
	return (int)cudaGetLastError();
}

extern "C" int fg_gnn_backward(fg_gnn *g, const double *r, const double *z, const double *t, int accumulate)
{
	return g->bf16 ? backward_t<__nv_bfloat16>(g, r, z, t, accumulate)
	               : backward_t<float>(g, r, z, t, accumulate);
}

extern "C" int fg_gnn_adam(fg_gnn *g, float lr, float gscale)
{
	const float b1 = 0.9f, b2 = 0.999f;
	g->step++;
	float c1 = 1.0f - powf(b1, (float)g->step), c2 = 1.0f - powf(b2, (float)g->step);
	k_gnn_adam<<<nb(GNN_NPARAMS, 256, 64), 256, 0, g->stream>>>(GNN_NPARAMS, g->theta, g->grad, g->am, g->av, lr, b1,
	                                                            b2, 1e-8f, c1, c2, gscale);
	return (int)cudaGetLastError();
}
