// V-cycle of the double-pairwise AMG preconditioner
// (00_CommonFiles/Solvers_and_Preconditioners/CSR/AMG/amg_dpa.c:485-506).
//
// Per smoothed level l (even levels; odd levels are only the intermediate of
// the double pairwise step): SOR_relax (amg_solvers.c:3-17) forward nr times,
// residual r = f - A u (amg_util.c:44-48 with mat_vec, amg_matrix.c:276-282),
// restriction twice (dpa_fine2coarse, amg_dpa.c:394-401), zero coarse u; at
// the coarsest level SOR forward nr + reverse nr times; on the way up
// prolongation twice (dpa_coarse2fine_pure then dpa_coarse2fine,
// amg_dpa.c:403-422) and SOR_relax_rev (amg_solvers.c:19-33) nr times.
//
// GB300 mapping.  The Gauss-Seidel sweeps run as a dataflow (fg_dataflow.cuh):
// every sweep writes an iterate of its own, marked unset beforehand, and a row
// polls the values it reads -- this sweep's for the rows before it, the
// previous one's for the others -- so each row sees exactly the values the
// sequential sweep sees and the result is the reference's bit for bit (this
// translation unit is compiled without FMA contraction; sums run in CSR
// order).  Two sweeps run in one launch, the second a few levels behind the
// first.  The residual and both restrictions are one kernel (one thread per
// level-(l+2) row recomputes its <= 4 fine residual rows, r is never stored),
// and both prolongations are one kernel through the composite aggregate map.
//
// A sweep is bound by its chain of levels: per level one trip of a value
// through L2 (0.36 us) and the FP64 operations behind it (a dependent one takes
// 31 ns on this part): the last product, the sum's rest, the quotient, the
// relaxation.  A chain of single rows measures 0.95 us a row, the levels of a
// 300x200 transport mesh 1.5 us (499 levels, 200 rows wide) to 1.9 us (its
// coarse levels).  One V-cycle on it (2 + 2 sweeps, 4 smoothed levels): 18.3 ms
// with one thread block walking the levels between barriers, one sweep after
// another (3.7 us a level), 4.3 ms now.
#include <cuda_runtime.h>

#include "fg_amg.h"
#include "fg_dataflow.cuh"
#include "fg_div.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kSorThreads = 128;      // four warps: one per FP64 pipe
constexpr int kSorAhead = 4;          // levels whose warps are resident: a row's pattern, values and
                                      // the iterate it starts from load while earlier levels run

__device__ __forceinline__ bool skip(const int *active) { return active && !*active; }

struct SorArgs {
	const int *ptr, *col;
	const double *val, *diag, *rdiag, *f;
	const double *b0;             // input iterate (NULL: zero)
	double *b1, *b2;              // after the first and the second sweep
	const int *item;
	unsigned nwarp;
	int reverse, relax;           // relax: omega is not 1 (1.0 * x is x)
	double omega;
	fg_ticket *tk;
	int *err;
	const int *active;
	int poll0;                    // BOUND: fg_poll0
};

// SOR_relax / SOR_relax_rev, L lanes per row update (the row's entries side by
// side, L at a time), 32 / L updates of one level a warp.  A lane whose value is
// not there yet polls it again whenever any entry of the warp is waited for, so
// a row whose last values come together pays one trip through L2, not one for
// each.  The row's sum runs over the lanes in CSR order as far as the values go.
// BOUND: the waits' bound is the context's own (as an argument of every launch
// it costs 0.6 % of a cycle).
template <int L, bool BOUND>
__global__ void __launch_bounds__(kSorThreads) k_sor(SorArgs a)
{
	if (skip(a.active)) return;
	constexpr int R = 32 / L;
	const int lane = threadIdx.x & 31, q = lane & (L - 1), l0 = lane & ~(L - 1);
	for (;;) {
		const unsigned t = fg_take(a.tk, a.nwarp);
		if (t >= a.nwarp) return;
		const int it0 = __ldg(&a.item[(long long)R * t + lane / L]);
		const bool on = it0 >= 0, second = on && (it0 >> 30);
		const int i = on ? it0 & 0x3fffffff : 0;
		const double *old = second ? a.b1 : a.b0;
		double *nw = second ? a.b2 : a.b1;
		const int k0 = on ? __ldg(&a.ptr[i]) : 0, len = on ? __ldg(&a.ptr[i + 1]) - k0 : 0;
		const int most = __reduce_max_sync(0xffffffffu, len);
		const double fi = on ? __ldg(&a.f[i]) : 1.0, di = on ? __ldg(&a.diag[i]) : 1.0, ri = on ? __ldg(&a.rdiag[i]) : 1.0;
		unsigned long long own = on && old ? fg_ld_poll(&old[i]) : 0ull;
		double sum = 0.0;
		for (int base = 0; base < most; base += L) {
			const bool in = base + q < len;
			const int c = in ? __ldg(&a.col[k0 + base + q]) : i;
			const double v = in ? __ldg(&a.val[k0 + base + q]) : 0.0;
			const bool e = c != i, n = a.reverse ? c > i : c < i;
			const double *src = n ? nw : old;
			unsigned long long x = e && src ? fg_ld_poll(&src[c]) : 0ull;
			double p = v * __longlong_as_double((long long)x);
			const unsigned used = __ballot_sync(0xffffffffu, e) >> l0;
			unsigned there = __ballot_sync(0xffffffffu, x != FG_UNSET) >> l0;
#pragma unroll
			for (int k = 0; k < L; k++) {
				if (base + k >= most) break;                      // uniform
				if (!__all_sync(0xffffffffu, there >> k & 1u)) {
					for (int it = BOUND ? a.poll0 : 0;; it++) {
						if (!fg_keep_polling(it, a.tk, a.err)) return;
						if (x == FG_UNSET) x = fg_ld_poll(&src[c]);
						there = __ballot_sync(0xffffffffu, x != FG_UNSET) >> l0;
						if (__all_sync(0xffffffffu, there >> k & 1u)) break;
					}
					p = v * __longlong_as_double((long long)x);
				}
				if (!__any_sync(0xffffffffu, used >> k & 1u)) continue;
				const double s = sum + __shfl_sync(0xffffffffu, p, l0 + k);
				if (used >> k & 1u) sum = s;
			}
		}
		for (int it = BOUND ? a.poll0 : 0;; it++) {
			const bool w = own == FG_UNSET;
			if (!__any_sync(0xffffffffu, w)) break;
			if (!fg_keep_polling(it, a.tk, a.err)) return;
			if (w) own = fg_ld_poll(&old[i]);
		}
		const double uo = __longlong_as_double((long long)own);
		double step = fg_div(fi - sum, di, ri) - uo;
		if (a.relax) step = a.omega * step;
		if (on && q == 0) fg_st_value(&nw[i], uo + step);
	}
}

__device__ __forceinline__ double resid_row(const int *__restrict__ ptr, const int *__restrict__ col,
                                            const double *__restrict__ val, const double *__restrict__ f,
                                            const double *__restrict__ u, int i)
{
	double p = 0.0;
	for (int k = ptr[i]; k < ptr[i + 1]; k++) p += val[k] * u[col[k]];
	return f[i] - p;
}

// f2[k] = (r[a] + r[b]) + (r[c] + r[d]) with absent members dropped, r = f - A u
// on level l.
__global__ void k_restrict2(const int *__restrict__ ptr, const int *__restrict__ col,
                            const double *__restrict__ val, const double *__restrict__ f,
                            const double *__restrict__ u, const int4 *__restrict__ quad, int nc2,
                            double *__restrict__ f2, const int *active)
{
	if (skip(active)) return;
	int k = blockIdx.x * blockDim.x + threadIdx.x;
	if (k >= nc2) return;
	int4 q = quad[k];
	double s1 = resid_row(ptr, col, val, f, u, q.x);
	if (q.y >= 0) s1 = s1 + resid_row(ptr, col, val, f, u, q.y);
	if (q.z >= 0) {
		double s2 = resid_row(ptr, col, val, f, u, q.z);
		if (q.w >= 0) s2 = s2 + resid_row(ptr, col, val, f, u, q.w);
		s1 = s1 + s2;
	}
	f2[k] = s1;
}

// u[i] += u2[agg2[i]]
__global__ void k_prolong2(const int *__restrict__ agg2, const double *__restrict__ u2, double *__restrict__ u,
                           int n, const int *active)
{
	if (skip(active)) return;
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) u[i] += u2[agg2[i]];
}

__global__ void k_copy(const double *__restrict__ src, double *__restrict__ dst, int n, const int *active)
{
	if (skip(active)) return;
	int i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) dst[i] = src[i];
}

// Marks up to two iterates unset and readies the launches' tickets.
__global__ void k_unset(double *x, long long nx, double *y, long long ny, fg_ticket *tk, int ntk, const int *active)
{
	if (skip(active)) return;
	const long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, st = (long long)gridDim.x * blockDim.x;
	const double unset = __longlong_as_double((long long)FG_UNSET);
	for (long long i = i0; i < ntk; i += st) tk[i] = fg_ticket{0u, 0u};
	for (long long i = i0; i < nx; i += st) x[i] = unset;
	for (long long i = i0; i < ny; i += st) y[i] = unset;
}

inline unsigned blocks(int n) { return (unsigned)((n + kThreads - 1) / kThreads); }

// nr SOR sweeps on level L from the iterate `in' (NULL: zero), two to a launch;
// *out: the last iterate (z when given).  With nr <= 2 the iterates were
// marked unset when the cycle began.  err: where a wait that runs out is told.
int sor(const femgpu_amg *g, const fg_amg_level *L, const double *in, double *z, int reverse, fg_ticket **tk,
        const int *active, int *err, double **out)
{
	const double *cur = in;
	for (int left = g->nr; left > 0;) {
		const int two = left > 1;
		left -= 1 + two;
		double *mid = L->w[reverse ? 2 : 0], *end = L->w[reverse ? 3 : 1];
		if (g->nr > 2) {                                  // two vectors that do not hold cur
			int k = 0;
			mid = L->w[k] == cur ? L->w[++k] : L->w[k];
			k++;
			end = L->w[k] == cur ? L->w[++k] : L->w[k];
		}
		if (z && !left) end = z;
		fg_ticket *q = (*tk)++;
		if (g->nr > 2)
			k_unset<<<fg_grid(L->n), kThreads, 0, g->stream>>>(mid, L->n, end, L->n, q, 1, active);
		const fg_amg_sched *S = reverse ? &L->bw[two] : &L->fw[two];
		const int lanes = L->longest <= 8 ? 8 : (L->longest <= 16 ? 16 : 32), rows = 32 / lanes;
		SorArgs a = { L->ptr, L->col, L->val, L->diag, L->rdiag, L->f, cur, two ? mid : end, end, S->item,
		              (unsigned)(S->nitem / rows), reverse, g->omega != 1.0, g->omega, q, err, active,
		              fg_poll0(g->wait1) };
		const int per = kSorThreads / 32 * rows, want = (int)(((long long)kSorAhead * S->wide + per - 1) / per);
		const int grid = want < 1 ? 1 : (want > 4 * FG_SMS ? 4 * FG_SMS : want);
#define SOR(L) do { if (g->wait1) k_sor<L, true><<<grid, kSorThreads, 0, g->stream>>>(a); \
	else k_sor<L, false><<<grid, kSorThreads, 0, g->stream>>>(a); } while (0)
		if (lanes == 8) SOR(8);
		else if (lanes == 16) SOR(16);
		else SOR(32);
#undef SOR
		cur = end;
	}
	*out = (double *)cur;
	return (int)cudaGetLastError();
}

}  // namespace

extern "C" int fg_amg_vcycle(femgpu_amg *g, const double *q, double *z, const int *active, int *err)
{
	int top = g->nlevels - 1, l, rc;
	fg_amg_level *lv = g->lv;
	int n0 = lv[0].n;
	fg_ticket *tk = (fg_ticket *)g->ticket;
	if (q == z) {
		k_copy<<<blocks(n0), kThreads, 0, g->stream>>>(q, g->qcopy, n0, active);
		q = g->qcopy;
	}
	lv[0].f = (double *)q;           // level 0 works on the caller's vectors
	if (g->nr <= 2)
		k_unset<<<fg_grid(g->narena), kThreads, 0, g->stream>>>(g->arena, g->narena, z, n0, tk, g->nticket, active);
	for (l = 0; l < top; l += 2) {
		fg_amg_level *L = &lv[l], *C = &lv[l + 2];
		if ((rc = sor(g, L, nullptr, nullptr, 0, &tk, active, err, &L->u))) return rc;
		k_restrict2<<<blocks(L->nc2), kThreads, 0, g->stream>>>(L->ptr, L->col, L->val, L->f, L->u, L->quad,
		                                                          L->nc2, C->f, active);
	}
	if ((rc = sor(g, &lv[top], nullptr, nullptr, 0, &tk, active, err, &lv[top].u))) return rc;
	if ((rc = sor(g, &lv[top], lv[top].u, nullptr, 1, &tk, active, err, &lv[top].u))) return rc;
	for (l = top; l > 0; l -= 2) {
		fg_amg_level *F = &lv[l - 2];
		k_prolong2<<<blocks(F->n), kThreads, 0, g->stream>>>(F->agg2, lv[l].u, F->u, F->n, active);
		if ((rc = sor(g, F, F->u, l == 2 ? z : nullptr, 1, &tk, active, err, &F->u))) return rc;
	}
	lv[0].f = nullptr;
	lv[0].u = nullptr;
	return (int)cudaGetLastError();
}
