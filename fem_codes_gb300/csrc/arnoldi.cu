// The small dense side of a Krylov step and, for vectors that fit the device's
// registers, the whole orthogonalisation of an Arnoldi step in one launch.
//
//   * k_givens / k_backsolve: the Givens update of a Hessenberg column
//     (pgmres.c:123-163) and the back substitution (pgmres.c:165-175), one warp.
//   * k_orth_mgs / k_orth_cgs: w against v_0 .. v_i (modified Gram-Schmidt as
//     pgmres.c:107-121, or one or two passes of classical Gram-Schmidt), its
//     norm, v_(i+1) = w / norm and the column's Givens update.
//
// A step on a small system was a chain of launches: i + 2 fused dot products for
// MGS, or multi-dot, finish and update, then the scaling and the Givens kernel,
// each waiting for the last.  In one launch w stays in registers and the sums
// over the device go through L2 (fg_dataflow.cuh): every block publishes its
// parts and every block polls them, adding them in one order, 0.36 us a trip.
// The launch is cooperative, so its blocks are resident together.  An extra
// block without rows rotates the column while the others go on.  Every sum is
// taken in the separate kernels' order (linalg.cu: 304 blocks of 256 threads),
// so a step has the same bits either way, whichever its size selects.
#include <math.h>

#include "fg_common.cuh"
#include "fg_dataflow.cuh"
#include "fg_div.cuh"

#define OR_TPB 256                    // threads of a block here and there
#define OR_VB (2 * FG_SMS)            // blocks of the separate reductions; two of them to a block here
#define OR_S 2                        // most entries a thread of those takes
#define OR_J 8                        // basis vectors of a CGS multi-dot at a time

// ------------------------------------------------------ Givens, solve ----
// The last step of column i: the rotation of (hii, hi1), the right-hand side,
// the status and, for the host, how far the cycle is.
__device__ __forceinline__ void finish_column(double hii, double hi1, double *H, int ldh, double *cs, double *sn,
                                              double *ge, int i, int kmax, fg_status *st, int *step)
{
	const double r = sqrt(__dadd_rn(__dmul_rn(hii, hii), __dmul_rn(hi1, hi1)));
	const double q = ((threadIdx.x & 31) ? hi1 : hii) / r;           // lane 0 the cosine, the others the sine
	const double c = __shfl_sync(0xffffffffu, q, 0), s = __shfl_sync(0xffffffffu, q, 1);
	if ((threadIdx.x & 31) == 0) {
		cs[i] = c;
		sn[i] = s;
		H[i * ldh + i] = r;
		H[(i + 1) * ldh + i] = 0.0;
		const double g = ge[i], g1 = __dmul_rn(-s, g), rho = fabs(g1);
		ge[i + 1] = g1;
		ge[i] = __dmul_rn(c, g);
		st->rho = rho;
		st->inner = i + 1;
		st->total += 1;
		int done = 0;
		if (!(rho > st->eps) || i + 1 >= kmax) done = 1;
		if (!(rho == rho)) { done = 1; fg_set_err(&st->err, FEMGPU_E_BREAKDOWN); }
		if (done) st->active = 0;
		*(volatile int *)step = (i + 1) | (done ? FG_STEP_DONE : 0);
	}
}

// The rotations of columns 0 .. i-1 applied to hc[0 .. i] (one warp, shared
// memory); the products that do not wait for the running entry are formed side
// by side, so a rotation costs two dependent operations.  Returns entry i.
__device__ __forceinline__ double rotate_column(const double *hc, double *pre, double *neg, double *run,
                                                const double *cs, const double *sn, double *H, int ldh, int i)
{
	const int lane = threadIdx.x & 31;
	for (int j = lane; j < i; j += 32) {
		neg[j] = -sn[j];
		pre[j] = __dmul_rn(cs[j], hc[j + 1]);
	}
	__syncwarp();
	double x = hc[0];
	for (int j = 0; j < i; j++) {
		if (lane == 0) run[j] = x;
		x = __dadd_rn(__dmul_rn(neg[j], x), pre[j]);
	}
	__syncwarp();
	for (int j = lane; j < i; j += 32)
		H[j * ldh + i] = __dadd_rn(__dmul_rn(cs[j], run[j]), __dmul_rn(sn[j], hc[j + 1]));
	return x;
}

// work: 4 (kmax + 1) words of global memory, or NULL: shared memory.
__global__ void __launch_bounds__(32) k_givens(double *H, int ldh, double *cs, double *sn, double *ge, int i, int kmax,
                                               fg_status *st, int *step, double *work)
{
	if (!st->active) return;
	extern __shared__ double sh[];
	double *hc = work ? work : sh, *pre = hc + kmax + 1, *neg = pre + kmax + 1, *run = neg + kmax + 1;
	for (int j = threadIdx.x; j <= i; j += 32) hc[j] = H[j * ldh + i];
	__syncwarp();
	const double hii = rotate_column(hc, pre, neg, run, cs, sn, H, ldh, i);
	finish_column(hii, H[(i + 1) * ldh + i], H, ldh, cs, sn, ge, i, kmax, st, step);
}

// H y = g from the last row up, each row's products added in ascending order
// (pgmres.c:165-175).  The products are formed side by side and the quotient
// comes from a reciprocal formed beforehand, which leaves the additions: 104 us
// for 80 rows (one thread walking them 186 us).
__global__ void __launch_bounds__(32) k_backsolve(const double *H, int ldh, const double *ge, double *gy, fg_status *st,
                                                  double *work)
{
	extern __shared__ double sh[];
	const int m = st->inner, lane = threadIdx.x;
	double *y = work ? work : sh, *rd = y + m, *pr = rd + m;
	for (int j = lane; j < m; j += 32) rd[j] = 1.0 / H[j * ldh + j];
	__syncwarp();
	for (int j = m - 1; j >= 0; j--) {
		const double g = ge[j], hjj = H[j * ldh + j];
		for (int k = j + 1 + lane; k < m; k += 32) pr[k] = __dmul_rn(H[j * ldh + k], y[k]);
		__syncwarp();
		double s = 0.0;
#pragma unroll 8
		for (int k = j + 1; k < m; k++) s = __dadd_rn(s, pr[k]);
		const double v = fg_div(j + 1 < m ? __dadd_rn(g, -s) : g, hjj, rd[j]);
		__syncwarp();
		if (lane == 0) { y[j] = v; gy[j] = v; }
		__syncwarp();
	}
}

// Up to OR_SMALL basis vectors the columns fit in shared memory as it comes;
// beyond, the context's scratch (the tail of fg_krylov.orth) takes its place.
#define OR_SMALL 256
static double *orth_tail(const fg_krylov *k);

extern "C" int fg_kry_givens(const fg_krylov *k, int i)
{
	const bool small = k->kmax <= OR_SMALL;
	k_givens<<<1, 32, small ? 4 * sizeof(double) * ((size_t)k->kmax + 1) : 0, k->stream>>>(
		k->H, k->kmax + 1, k->cs, k->sn, k->ge, i, k->kmax, k->st, &k->st_host->step, small ? nullptr : orth_tail(k) + 1);
	return (int)cudaGetLastError();
}

extern "C" int fg_kry_backsolve(const fg_krylov *k)
{
	const bool small = k->kmax <= OR_SMALL;
	k_backsolve<<<1, 32, small ? 3 * sizeof(double) * (size_t)k->kmax : 0, k->stream>>>(
		k->H, k->kmax + 1, k->ge, k->gy, k->st, small ? nullptr : orth_tail(k) + 1);
	return (int)cudaGetLastError();
}

// ------------------------------------------------- one-launch steps ----
struct OrthArgs {
	double *V;
	size_t ldv;
	int n, i, kmax, ldh, passes, G, nvb;  // G: blocks with rows; nvb: reduction blocks with rows
	double *H, *cs, *sn, *ge;
	double *slot, *next;                  // this step's sums, and the next one's (marked unset here)
	long long nnext;
	fg_ticket *tk;                        // abort word
	fg_status *st;
	int *step;
	int poll0;                            // fg_poll0
};

__device__ __forceinline__ void reset_next(const OrthArgs &a)
{
	for (long long q = blockIdx.x * (long long)OR_TPB + threadIdx.x; q < a.nnext; q += (long long)gridDim.x * OR_TPB)
		a.next[q] = __longlong_as_double((long long)FG_UNSET);
}

// Polls slot[first + 32 k'] ... of a lane: NQ words `stride' apart below end,
// all there on return (a warp); false when the wait gave up.
template <int NQ>
__device__ __forceinline__ bool poll_words(unsigned long long (&x)[NQ], const double *slot, int first, int stride, int end,
                                           const OrthArgs &a)
{
#pragma unroll
	for (int q = 0; q < NQ; q++) x[q] = first + q * stride < end ? fg_ld_poll(&slot[first + q * stride]) : 0ull;
	for (int it = a.poll0;; it++) {
		bool w = false;
#pragma unroll
		for (int q = 0; q < NQ; q++) w |= x[q] == FG_UNSET;
		if (!__any_sync(0xffffffffu, w)) return true;
#pragma unroll
		for (int q = 0; q < NQ; q++)
			if (x[q] == FG_UNSET) x[q] = fg_ld_poll(&slot[first + q * stride]);
		if (!fg_keep_polling(it, a.tk, &a.st->err)) return false;
	}
}

// Eight warps' sums as linalg.cu's block_sum adds them (its shuffle tree), lane
// 8 g + w holding warp w's sum of group g.  Three FP64 operations of one warp:
// every thread adding the eight up for itself is seven of eight warps, 900
// clocks of the four FP64 pipes for each of MGS's sums (64x64 transport, ten
// sums a step on average: 19.5 us a step that way, 14.3 now).
__device__ __forceinline__ double tree8_lanes(double s)
{
	s += __shfl_xor_sync(0xffffffffu, s, 4);
	s += __shfl_xor_sync(0xffffffffu, s, 2);
	return s + __shfl_xor_sync(0xffffffffu, s, 1);
}

// The total of nb published parts as last_block_total adds them: thread t takes
// parts t, t + 256, .., then block_sum.  Every thread of the block calls.
template <int NQ>
__device__ __forceinline__ bool block_total(const double *slot, int nb, const OrthArgs &a, double *sw, int *fail,
                                            double *tot)
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	double v = 0.0;
	if (32 * warp < nb) {                                 // (uniform; the others' sums are zeros)
		unsigned long long x[NQ];
		const bool ok = poll_words<NQ>(x, slot, threadIdx.x, OR_TPB, nb, a);
#pragma unroll
		for (int q = 0; q < NQ; q++) if (q == 0 || q * OR_TPB < nb) v += __longlong_as_double((long long)x[q]);
		v = fg_warp_sum(v);
		if (lane == 0 && !ok) *fail = 1;
	}
	if (nb <= 32) {                                       // the first warp's sum is the total
		if (threadIdx.x == 0) sw[0] = v;
		__syncthreads();
		*tot = sw[0];
		return *fail == 0;
	}
	if (lane == 0) sw[warp] = v;
	__syncthreads();
	*tot = tree8_lanes(sw[lane & 7]);
	return *fail == 0;
}

// NV reduction blocks (blockIdx.x, blockIdx.x + G) of this block, S entries a
// thread of each: entry s of block b, thread t is b 256 + t + s 304 256.
#define OR_AT(v, s) (((int)blockIdx.x + (v) * a.G) * OR_TPB + (int)threadIdx.x + (s) * OR_VB * OR_TPB)
#define OR_ON(v, s) ((int)blockIdx.x + (v) * a.G < a.nvb && OR_AT(v, s) < a.n)

template <int NV, int S>
__global__ void __launch_bounds__(OR_TPB) k_orth_mgs(OrthArgs a)
{
	if (!a.st->active) return;
	__shared__ double sw[NV][8], sv[2][8];
	__shared__ int fail;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, i = a.i;
	if (tid == 0) fail = 0;
	reset_next(a);
	__syncthreads();
	if ((int)blockIdx.x == a.G) {                         // the column, rotated as its entries come
		double x = 0.0, tot;
		for (int j = 0; j <= i + 1; j++) {
			if (!block_total<2>(a.slot + (size_t)j * a.nvb, a.nvb, a, sv[j & 1], &fail, &tot)) return;
			if (warp) continue;
			if (j == 0) { x = tot; continue; }
			if (j == i + 1) {
				finish_column(x, sqrt(tot), a.H, a.ldh, a.cs, a.sn, a.ge, i, a.kmax, a.st, a.step);
				continue;
			}
			const double c = a.cs[j - 1], s = a.sn[j - 1];
			if (tid == 0) a.H[(j - 1) * a.ldh + i] = __dadd_rn(__dmul_rn(c, x), __dmul_rn(s, tot));
			x = __dadd_rn(__dmul_rn(-s, x), __dmul_rn(c, tot));
		}
		return;
	}
	double *wv = a.V + (size_t)(i + 1) * a.ldv;
	double w[NV][S], v[NV][S], u[NV][S];
#pragma unroll
	for (int q = 0; q < NV; q++)
#pragma unroll
		for (int s = 0; s < S; s++) {
			w[q][s] = OR_ON(q, s) ? wv[OR_AT(q, s)] : 0.0;
			v[q][s] = OR_ON(q, s) ? a.V[OR_AT(q, s)] : 0.0;
			u[q][s] = 0.0;
		}
	double h = 0.0;
	for (int j = 0; j <= i + 1; j++) {
		double *slot = a.slot + (size_t)j * a.nvb;
#pragma unroll
		for (int q = 0; q < NV; q++) {
			double part = 0.0;
#pragma unroll
			for (int s = 0; s < S; s++) {
				if (j > 0) w[q][s] = __dadd_rn(w[q][s], __dmul_rn(-h, u[q][s]));
				part += j <= i ? v[q][s] * w[q][s] : w[q][s] * w[q][s];
				u[q][s] = v[q][s];
				if (j < i && OR_ON(q, s)) v[q][s] = a.V[(size_t)(j + 1) * a.ldv + OR_AT(q, s)];  // on its way during the sum
			}
			part = fg_warp_sum(part);
			if (lane == 0) sw[q][warp] = part;
		}
		__syncthreads();
		if (warp == 0) {
			const int g = lane >> 3;
			const double t = tree8_lanes(g < NV ? sw[g][lane & 7] : 0.0);
			if (g < NV && !(lane & 7) && (int)blockIdx.x + g * a.G < a.nvb) fg_st_value(&slot[blockIdx.x + g * a.G], t);
		}
		if (!block_total<2>(slot, a.nvb, a, sv[j & 1], &fail, &h)) return;
	}
	const double sc = 1.0 / sqrt(h);
#pragma unroll
	for (int q = 0; q < NV; q++)
#pragma unroll
		for (int s = 0; s < S; s++)
			if (OR_ON(q, s)) wv[OR_AT(q, s)] = __dmul_rn(sc, w[q][s]);
}

// Slots of a CGS step with m basis vectors: per pass the blocks' parts of each
// product [m][nvb] and the products [m], then the parts of the norm, one for
// each 256 entries (the update's blocks).
template <int NV, int S>
__global__ void __launch_bounds__(OR_TPB) k_orth_cgs(OrthArgs a)
{
	if (!a.st->active) return;
	extern __shared__ double dyn[];
	__shared__ double sw[NV * S][8], sv[8];
	__shared__ int fail;
	const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, i = a.i, m = i + 1, nvb = a.nvb;
	const int nb = (a.n + OR_TPB - 1) / OR_TPB;
	const size_t plen = (size_t)m * (nvb + 1);
	double *norm = a.slot + a.passes * plen;
	if (tid == 0) fail = 0;
	reset_next(a);
	__syncthreads();
	if ((int)blockIdx.x == a.G) {                         // the column
		double *hc = dyn, *pre = hc + m + 1, *neg = pre + m + 1, *run = neg + m + 1, tot, hii = 0.0;
		if (warp == 0) {
			for (int p = 0; p < a.passes; p++) {
				const double *res = a.slot + p * plen + (size_t)m * nvb;
				for (int j0 = 0; j0 < m; j0 += 32) {
					unsigned long long x[1];
					if (!poll_words<1>(x, res, j0 + lane, 32, m, a)) { fail = 1; break; }
					const double t = __longlong_as_double((long long)x[0]);
					if (j0 + lane < m) hc[j0 + lane] = p ? hc[j0 + lane] + t : t;
				}
			}
			__syncwarp();
			hii = rotate_column(hc, pre, neg, run, a.cs, a.sn, a.H, a.ldh, i);
		}
		if (!block_total<3>(norm, nb, a, sv, &fail, &tot)) return;
		if (warp == 0) finish_column(hii, sqrt(tot), a.H, a.ldh, a.cs, a.sn, a.ge, i, a.kmax, a.st, a.step);
		return;
	}
	double *ws = dyn, *hs = dyn + NV * 8 * (size_t)m;     // the warps' parts [NV][8][m], the products [m]
	double *wv = a.V + (size_t)(i + 1) * a.ldv;
	double w[NV][S];
#pragma unroll
	for (int q = 0; q < NV; q++)
#pragma unroll
		for (int s = 0; s < S; s++) w[q][s] = OR_ON(q, s) ? wv[OR_AT(q, s)] : 0.0;
	for (int p = 0; p < a.passes; p++) {
		double *part = a.slot + p * plen, *res = part + (size_t)m * nvb;
		for (int jb = 0; jb < m; jb += OR_J)
#pragma unroll
			for (int q = 0; q < NV; q++) {
				double acc[OR_J];
#pragma unroll
				for (int x = 0; x < OR_J; x++) acc[x] = 0.0;
#pragma unroll
				for (int s = 0; s < S; s++) {
					double v[OR_J];
#pragma unroll
					for (int x = 0; x < OR_J; x++)
						v[x] = jb + x < m && OR_ON(q, s) ? a.V[(size_t)(jb + x) * a.ldv + OR_AT(q, s)] : 0.0;
#pragma unroll
					for (int x = 0; x < OR_J; x++) acc[x] += v[x] * w[q][s];
				}
				// k_mdot's eight sums over the warp
#pragma unroll
				for (int o = 4; o > 0; o >>= 1)
#pragma unroll
					for (int x = 0; x < o; x++) {
						const bool hi = lane & (4 * o);
						const double keep = hi ? acc[x + o] : acc[x], give = hi ? acc[x] : acc[x + o];
						acc[x] = keep + __shfl_xor_sync(0xffffffffu, give, 4 * o);
					}
				acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
				acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
				const int j = jb + ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
				if ((lane & 3) == 0 && j < m) ws[(q * 8 + warp) * m + j] = acc[0];
			}
		__syncthreads();
		for (int e = tid; e < NV * m; e += OR_TPB) {
			const int q = NV == 1 ? 0 : e / m, j = e - q * m, b = blockIdx.x + q * a.G;
			double t = 0.0;
#pragma unroll
			for (int x = 0; x < 8; x++) t += ws[(q * 8 + x) * m + j];
			if (b < nvb) fg_st_value(&part[(size_t)j * nvb + b], t);
		}
		// product j is added up by block j (mod G), a warp each, as k_mdot_fin does
		for (int j = blockIdx.x + warp * a.G; j < m; j += 8 * a.G) {
			unsigned long long x[10];
			if (!poll_words<10>(x, part + (size_t)j * nvb, lane, 32, nvb, a)) fail = 1;
			double t = 0.0;
#pragma unroll
			for (int y = 0; y < 10; y++) if (32 * y < nvb) t += __longlong_as_double((long long)x[y]);
			t = fg_warp_sum(t);
			if (lane == 0) fg_st_value(&res[j], t);
		}
		for (int j0 = 32 * warp; j0 < m; j0 += OR_TPB) {
			unsigned long long x[1];
			if (!poll_words<1>(x, res, j0 + lane, 32, m, a)) fail = 1;
			if (j0 + lane < m) hs[j0 + lane] = __longlong_as_double((long long)x[0]);
		}
		__syncthreads();
		if (fail) return;
#pragma unroll
		for (int q = 0; q < NV; q++)
#pragma unroll
			for (int s = 0; s < S; s++) {
				if (!OR_ON(q, s)) continue;
				const double *Vk = a.V + OR_AT(q, s);
				double x = w[q][s];
				int j = 0;
				for (; j + OR_J <= m; j += OR_J) {
					double v[OR_J];
#pragma unroll
					for (int y = 0; y < OR_J; y++) v[y] = Vk[(size_t)(j + y) * a.ldv];
#pragma unroll
					for (int y = 0; y < OR_J; y++) x -= hs[j + y] * v[y];
				}
				for (; j < m; j++) x -= hs[j] * Vk[(size_t)j * a.ldv];
				w[q][s] = x;
			}
		__syncthreads();                                  // ws, hs are written again by the next pass
	}
#pragma unroll
	for (int q = 0; q < NV; q++)
#pragma unroll
		for (int s = 0; s < S; s++) {
			const double t = fg_warp_sum(w[q][s] * w[q][s]);
			if (lane == 0) sw[q * S + s][warp] = t;
		}
	__syncthreads();
	if (warp == 0) {
		static_assert(NV * S <= 4, "a group of eight lanes each");
		const int g = lane >> 3, q = g / S, s = g - q * S, b = blockIdx.x + q * a.G + s * OR_VB;
		const double t = tree8_lanes(g < NV * S ? sw[g][lane & 7] : 0.0);
		if (g < NV * S && !(lane & 7) && (int)blockIdx.x + q * a.G < nvb && b < nb) fg_st_value(&norm[b], t);
	}
	double tot;
	if (!block_total<3>(norm, nb, a, sv, &fail, &tot)) return;
	const double sc = 1.0 / sqrt(tot);
#pragma unroll
	for (int q = 0; q < NV; q++)
#pragma unroll
		for (int s = 0; s < S; s++)
			if (OR_ON(q, s)) wv[OR_AT(q, s)] = __dmul_rn(sc, w[q][s]);
}

__global__ void k_orth_begin(double *slot, long long n, fg_ticket *tk)
{
	const long long q0 = blockIdx.x * (long long)blockDim.x + threadIdx.x;
	if (q0 == 0) { tk->next = 0u; tk->abort = 0u; }
	for (long long q = q0; q < n; q += (long long)gridDim.x * blockDim.x) slot[q] = __longlong_as_double((long long)FG_UNSET);
}

static int orth_nvb(int n)
{
	const int b = (n + OR_TPB - 1) / OR_TPB;
	return b < OR_VB ? b : OR_VB;
}

// Words of one step's sums; a context keeps two sets, the abort word and 4 (kmax
// + 1) words of scratch.
static size_t orth_words(int m, int nvb, int mgs)
{
	return mgs ? (size_t)(m + 1) * nvb : 2 * (size_t)m * (nvb + 1) + OR_S * OR_VB;
}
extern "C" size_t fg_kry_orth_bytes(int kmax)
{
	return sizeof(double) * (2 * orth_words(kmax + 1, OR_VB, 0) + 1 + 4 * ((size_t)kmax + 1));
}
static double *orth_tail(const fg_krylov *k) { return k->orth + 2 * orth_words(k->kmax + 1, OR_VB, 0); }

// Whether a step runs in one launch: w has to fit the registers (155,648
// unknowns at most); beyond, the separate kernels are bound by the FP64 pipes
// and the launches between them no longer count.  Measured, whole solves with
// the launches of converged steps gone too: 64x64 transport, GMRES(30), a Picard
// iteration 6.2 -> 3.4 ms (a step's orthogonalisation 19 us, now 14, of 10 dot
// products on average, each a launch of 2.3 us and a gap before); Euler 256x64, FGMRES(50),
// a time step 19.7 -> 10.8 ms (35 us a step, half of them two passes; multi-dot
// 13, finish 2, update 7, scaling 2 and Givens 8 us before, gaps apart).
extern "C" int fg_kry_orth_fits(const fg_krylov *k)
{
	return k->n <= OR_S * OR_VB * OR_TPB && k->kmax <= OR_SMALL && k->nblk == OR_VB;
}

extern "C" int fg_kry_orth_begin(const fg_krylov *k)
{
	k_orth_begin<<<4, 256, 0, k->stream>>>(k->orth, (long long)orth_words(1, OR_VB, 0), (fg_ticket *)orth_tail(k));
	return (int)cudaGetLastError();
}

// Step i on w = V[i+1]: passes 0 MGS, else that many passes of CGS.
extern "C" int fg_kry_orth(const fg_krylov *k, int i, int passes)
{
	const size_t half = orth_words(k->kmax + 1, OR_VB, 0);
	OrthArgs a;
	a.V = k->V; a.ldv = k->ldv; a.n = k->n; a.i = i; a.kmax = k->kmax; a.ldh = k->kmax + 1; a.passes = passes;
	a.nvb = orth_nvb(k->n);
	a.G = a.nvb < FG_SMS ? a.nvb : FG_SMS;
	a.H = k->H; a.cs = k->cs; a.sn = k->sn; a.ge = k->ge; a.st = k->st; a.step = &k->st_host->step;
	a.slot = k->orth + (i & 1) * half;
	a.next = k->orth + ((i + 1) & 1) * half;
	a.nnext = (long long)orth_words(i + 2, a.nvb, passes == 0);
	a.tk = (fg_ticket *)orth_tail(k);
	a.poll0 = fg_poll0(k->wait1);
	const int nv = a.nvb > a.G ? 2 : 1, f = nv - 1 + (k->n > OR_VB * OR_TPB ? 1 : 0);
	static void *const mgs[3] = { (void *)k_orth_mgs<1, 1>, (void *)k_orth_mgs<2, 1>, (void *)k_orth_mgs<2, 2> };
	static void *const cgs[3] = { (void *)k_orth_cgs<1, 1>, (void *)k_orth_cgs<2, 1>, (void *)k_orth_cgs<2, 2> };
	void *args[] = { &a };
	const size_t smem = passes ? sizeof(double) * (8 * (size_t)nv + 1) * ((size_t)i + 2) : 0;
	return (int)cudaLaunchCooperativeKernel(passes ? cgs[f] : mgs[f], dim3((unsigned)a.G + 1), dim3(OR_TPB), args, smem,
	                                        k->stream);
}
