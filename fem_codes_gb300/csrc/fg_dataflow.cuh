// Self-synchronising FP64 values in global memory: a kernel whose warps
// compute values other warps of the same launch wait for marks every such
// value "not yet written" beforehand, and a reader polls the value itself.
// An 8-byte store is one access, so no flag and no fence stands between a
// producer and its readers: one trip through L2 (about 0.36 us from the store
// to the poll that sees it, whichever SMs hold the two warps) instead of a
// fence, a flag and then the data.
//
// The mark is a NaN no FP64 instruction produces; a value that carries these
// very bits (only a copied input can) is stored as the ordinary quiet NaN.
// Work is handed out by a ticket counter in an order in which every value
// comes after those it needs.  The lowest unfinished ticket is always held by
// a running warp that waits for nothing, so the launch finishes however few
// of its blocks the device holds at once.  Every wait is bounded all the same:
// a warp that gives up raises the abort word, which the others look at while
// they wait and before they take more work.
#pragma once
#include "fg_common.cuh"

#define FG_UNSET 0xffffffffffffffffull
#define FG_POLL_LIMIT (1 << 22)       // polls of one wait (about 1.5 s) unless the context says otherwise

// A context's bound on a wait (wait1 = bound + 1, 0 the default) as the count a
// wait starts at, so that the loops compare with a constant.
static inline int fg_poll0(int wait1) { return wait1 > 0 ? FG_POLL_LIMIT - (wait1 - 1) : 0; }

// Control words of one launch, zeroed before it: next ticket, abort.
struct fg_ticket { unsigned next, abort; };

__device__ __forceinline__ unsigned long long fg_ld_poll(const double *p)
{
	unsigned long long v;
	asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
	return v;
}

__device__ __forceinline__ void fg_st_value(double *p, double x)
{
	unsigned long long v = (unsigned long long)__double_as_longlong(x);
	if (v == FG_UNSET) v = 0x7ff8000000000000ull;
	asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(v) : "memory");
}

// The warp's next unit of work, the same in every lane; at least `end' once
// the work or, after an abort, the launch is over.
__device__ __forceinline__ unsigned fg_take(fg_ticket *tk, unsigned end)
{
	unsigned t = 0;
	if ((threadIdx.x & 31) == 0) {
		t = atomicAdd(&tk->next, 1u);
		if (*(volatile unsigned *)&tk->abort) t = end;
	}
	return __shfl_sync(0xffffffffu, t, 0);
}

// One more poll of a wait (the same count in every lane, from fg_poll0 on):
// false when the bound is reached or another warp gave up.
__device__ __forceinline__ bool fg_keep_polling(int it, fg_ticket *tk, int *err)
{
	if (it >= FG_POLL_LIMIT) {
		if ((threadIdx.x & 31) == 0) {
			*(volatile unsigned *)&tk->abort = 1u;
			fg_set_err(err, FEMGPU_E_TIMEOUT);
		}
		return false;
	}
	return (it & 255) != 255 || !__any_sync(0xffffffffu, *(volatile unsigned *)&tk->abort != 0u);
}
