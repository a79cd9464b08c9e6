// ILU(0) on the device (ILUp_precond_setup.c:66-167 at level of fill 0,
// ILUp_precond.c:26-46).
//
// The triangular sweeps have ~2.5*nx dependency levels after SYMRCM (5118
// for a 2048x1024 grid) of a few hundred rows each, so they are bound by
// per-level latency, not bandwidth.  Each matrix block is swept by ONE
// thread block:
//   * at set-up, each sweep is compiled into a "program": every level is cut
//     into sub-blocks of at most SW_SUB rows, 16-byte aligned -- one record
//     per row (dependency codes, output slot, factor values, the inverted
//     pivot backward; k_sweep_df / k_sweep_rec) when no row has more than 16
//     dependencies, else ELL arrays (k_sweep); factor values are refreshed
//     after every factorisation;
//   * records: chunks of up to 32 rows are dealt to the warps in turn; each
//     warp streams its chunks (and their slice of the input vector) into
//     shared-memory stages of its own with TMA bulk copies and polls the values
//     its rows read in a shared-memory ring (k_sweep_df, k_sweep_fb);
//   * ELL arrays and FEMGPU_SWEEP_SYNC=barrier: one producer warp streams the
//     sub-blocks into a ring of stages (cp.async.bulk, completion on a "full"
//     mbarrier; stage reuse gated by an "empty" mbarrier), consumer warps
//     compute a level, publish its values in a shared-memory ring indexed by
//     level-order position and meet at one named barrier per level (k_sweep,
//     k_sweep_rec);
//   * dependencies older than the ring are re-read from global memory.
// Rows are computed in the reference's order (ascending columns) and the
// FP64 variant rounds each operation separately, so its results are
// bit-identical to the reference's sweeps; FGMRES uses the fused
// multiply-subtract variant.
//
// Block ILU(0) (ilu_blocks = P > 1): the rows are cut into P contiguous runs
// of the (reordered) numbering (make_blocks: by default at equal spans of the
// full factor's dependency levels) and couplings between runs are dropped, so
// each block factorises and sweeps independently: its levels form a
// contiguous run of the program (levels are numbered block by block) and one
// thread block per matrix block runs them, P thread blocks at once.  The
// factorisation runs all blocks' rows as one dataflow over the device.  Every
// wait is bounded: on timeout the block records FEMGPU_E_TIMEOUT, waits (bounded) for
// the copies it has in flight and returns.
#include "fg_common.cuh"
#include "fg_dataflow.cuh"
#include <string.h>
#include <vector>
#include <algorithm>

#ifndef FG_SW2_CW
#define FG_SW2_CW 16
#endif
#define SW_SUB (FG_SW2_CW * 32)       // max rows of a sub-block
#define SW_MAXW 8                     // dependencies per row on the unrolled path
#define SW_RPT 4                      // rows per consumer thread per pass
#define SW_RING 4096                  // ring slots (power of two)
#define SW_RING_WIDE 8192             // ... of dataflow programs whose stages leave room
#define SW_NEAR 0x80000000u           // dependency code: ring slot (dataflow programs: global position)
#define SW_WAIT_LIMIT (1 << 24)
#define SW_MAXD 12                    // max stages
#define SW_BAR_BYTES (2 * SW_MAXD * 8)
#define SW_SMEM_CAP (226 * 1024)
#define SW_HDR 32

// ------------------------------------------------------------ PTX helpers
__device__ __forceinline__ unsigned smem_u32(const void *p)
{
	return (unsigned)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count)
{
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes)
{
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
	             :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *bar)
{
	asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
	             :: "r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity)
{
	unsigned ok;
	asm volatile("{\n\t.reg .pred p;\n\t"
	             "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
	             "selp.u32 %0, 1, 0, p;\n\t}"
	             : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
	return ok != 0;
}

__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity)
{
	for (int i = 0; i < SW_WAIT_LIMIT; i++)
		if (mbar_try_wait(bar, parity)) return true;
	return false;
}

// Wait for a phase, giving up when the bound is hit or another warp failed.
__device__ __forceinline__ bool mbar_wait_or_fail(unsigned long long *bar, unsigned parity, volatile int *failed)
{
	for (int i = 0; i < SW_WAIT_LIMIT; i++) {
		if (mbar_try_wait(bar, parity)) return true;
		if (*failed) return false;
	}
	return false;
}

// The same for a whole warp, the answer the same in every lane: lanes that saw
// the failure while others saw the phase end would leave the others at the next
// warp barrier.
__device__ __forceinline__ bool mbar_wait_warp(unsigned long long *bar, unsigned parity, volatile int *failed)
{
	for (int i = 0; i < SW_WAIT_LIMIT; i++) {
		if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
		if (__any_sync(0xffffffffu, *failed != 0)) return false;
	}
	return false;
}

__device__ __forceinline__ void fence_proxy_async()
{
	asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void fence_mbar_init()
{
	asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Release store / acquire load of a shared-memory flag (CTA scope).
__device__ __forceinline__ void st_release_cta(int *p, int v)
{
	asm volatile("st.release.cta.shared.s32 [%0], %1;" :: "r"(smem_u32(p)), "r"(v) : "memory");
}

__device__ __forceinline__ int ld_acquire_cta(const int *p)
{
	int v;
	asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
	return v;
}

// Synchronise the CW consumer warps (shared-memory ordering included).
template <int CW>
__device__ __forceinline__ void consumer_sync()
{
	if (CW == 1) __syncwarp();
	else asm volatile("bar.sync 1, %0;" :: "r"(CW * 32) : "memory");
}

template <typename T> __device__ __forceinline__ T fms(T x, T a, T b);   // x - a*b
template <> __device__ __forceinline__ double fms(double x, double a, double b)
{
	return __dsub_rn(x, __dmul_rn(a, b));
}
template <> __device__ __forceinline__ float fms(float x, float a, float b) { return x - a * b; }
template <typename T> __device__ __forceinline__ T mul(T a, T b);
template <> __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
template <> __device__ __forceinline__ float mul(float a, float b) { return a * b; }

// x - a*b: separately rounded (bit-identical to the reference) or fused.
template <typename T, bool FMA> __device__ __forceinline__ T fmsub(T x, T a, T b)
{
	if (FMA) return fma(-a, b, x);
	return fms(x, a, b);
}

// ---------------------------------------------------- double-single values
// (fg_ds.cuh): the sweeps' values, multipliers and ring in float pairs.
#include "fg_ds.cuh"

template <> __device__ __forceinline__ dsf fmsub<dsf, true>(dsf x, dsf a, dsf b) { return ds_fma(ds_neg(a), b, x); }
template <> __device__ __forceinline__ dsf mul(dsf a, dsf b) { return ds_mul(a, b); }

// zero, FP64 -> T, and the cache-global load / warp shuffle of a T
template <typename T> __device__ __forceinline__ T zero_t() { return T(0); }
template <> __device__ __forceinline__ dsf zero_t<dsf>() { return dsf{ 0.0f, 0.0f }; }
template <typename T> __device__ __forceinline__ T from_d(double v) { return (T)v; }
template <> __device__ __forceinline__ dsf from_d<dsf>(double v) { return ds_from(v); }
template <typename T> __device__ __forceinline__ T ld_cg(const T *p) { return __ldcg(p); }
template <> __device__ __forceinline__ dsf ld_cg<dsf>(const dsf *p)
{
	const float2 v = __ldcg((const float2 *)p);
	return dsf{ v.x, v.y };
}
template <typename T> __device__ __forceinline__ T shfl_up_t(T v, int d) { return __shfl_up_sync(0xffffffffu, v, d); }
template <> __device__ __forceinline__ dsf shfl_up_t<dsf>(dsf v, int d)
{
	return dsf{ __shfl_up_sync(0xffffffffu, v.hi, d), __shfl_up_sync(0xffffffffu, v.lo, d) };
}

// Sub-block: 32-byte header, dep[w*cp] (int), out[cp] (int), pad to 16,
// val[w*cp] (T), and for the backward sweep dinv[cp] (T); the stage then
// holds the sub-block's slice of the input vector.  Header: rows c, ELL
// width w, level-order position of the first row, padded rows cp, number of
// sub-blocks of the level, a flag set when some dependency is older than the
// ring holds (read from global memory instead), and the byte offsets of the
// values and of the input slice.
struct LevHdr { int c, w, start, cp, nsub, hasfar, voff, boff; };

static inline __host__ __device__ long long al16(long long x) { return (x + 15) & ~15LL; }

template <typename T, bool UPPER>
__host__ __device__ __forceinline__ long long blk_bytes(int w, int cp)
{
	long long voff = al16(SW_HDR + (long long)(w + 1) * cp * 4);
	return al16(voff + (long long)w * cp * (long long)sizeof(T) + (UPPER ? (long long)cp * sizeof(T) : 0));
}

struct SweepArgs {
	const unsigned char *prog;
	const long long *blk_off;     // [nsb+1] byte offset of each sub-block
	const int *sb_in;             // [nsb] padded start of the sub-block's input slice
	const int *sb_inb;            // [nsb] bytes of that slice
	int nlev, nsb, D, stage_bytes;
	int *err;
	const int *active;
	const int *chunk_sb;          // [P+1] first sub-block of each matrix block (NULL: one block)
	const int *chunk_lev;         // [P+1] first level of each matrix block
	int bvo, cmax;                // record layout: input slice offset, most rows of a sub-block
	int ring, look;               // dataflow: ring slots (power of two), chunks a warp may run ahead
	int wait;                     // spins of a warp waiting for the rows it depends on
};

// The producer warp of the barrier sweeps: streams this thread block's
// sub-blocks [sb0, sb1) and their input slices into the D-stage ring with
// cp.async.bulk (completion on full[s]), reusing a stage once the consumers
// have released it (empty[s]); stops when a consumer has failed.  The input
// slice lands at the stage's fixed offset a.bvo (record layouts,
// slice_at_bvo) or right after the sub-block (ELL layout).
template <typename T>
__device__ __forceinline__ void sweep_producer(const SweepArgs &a, const T *in, unsigned char *stages,
                                               unsigned sbytes, unsigned long long *full,
                                               unsigned long long *empty, int D, int sb0, int sb1, int lane,
                                               volatile int *vfailed, int *issued, int *pdone, bool slice_at_bvo)
{
	bool stop = false;
	int s = 0;
	unsigned ph = 0;                                      // phase of empty[s] to wait for
	for (int base = sb0; base < sb1 && !stop; base += 32) {
		// each lane fetches the offsets of one upcoming sub-block
		int i = base + lane;
		long long b0 = 0, b1 = 0;
		int p0 = 0, vb = 0;
		if (i < sb1) { b0 = a.blk_off[i]; b1 = a.blk_off[i + 1]; p0 = a.sb_in[i]; vb = a.sb_inb[i]; }
		for (int j = 0; j < 32 && base + j < sb1; j++) {
			long long B0 = __shfl_sync(0xffffffffu, b0, j), B1 = __shfl_sync(0xffffffffu, b1, j);
			int P0 = __shfl_sync(0xffffffffu, p0, j), VB = __shfl_sync(0xffffffffu, vb, j);
			int sb = base + j - sb0;                      // local sub-block index
			int go = 1;
			if (lane == 0) {
				if (sb >= D && !mbar_wait_or_fail(&empty[s], ph, vfailed)) go = 0;
				if (*vfailed) go = 0;
				if (go) {
					unsigned bb = (unsigned)(B1 - B0);
					unsigned char *dst = stages + (unsigned)s * sbytes;
					fence_proxy_async();
					mbar_expect_tx(&full[s], bb + (unsigned)VB);
					bulk_g2s(dst, a.prog + B0, bb, &full[s]);
					if (VB) bulk_g2s(dst + (slice_at_bvo ? (unsigned)a.bvo : bb), in + P0, (unsigned)VB, &full[s]);
					*(volatile int *)issued = sb + 1;
				}
			}
			go = __shfl_sync(0xffffffffu, go, 0);
			if (!go) { stop = true; break; }
			if (++s == D) { s = 0; if (sb >= D) ph ^= 1u; else if (sb == D - 1) ph = 0; }
		}
	}
	if (lane == 0) {
		__threadfence_block();                            // `issued' is final before `pdone'
		*(volatile int *)pdone = 1;
	}
}

// After a consumer failed (one thread): record the timeout, let the producer
// stop, then wait (bounded) for the copies it issued beyond the `done' stages
// this thread consumed, so no copy lands in shared memory after the exit.
__device__ __forceinline__ void sweep_drain(const SweepArgs &a, unsigned long long *full, int D, int done,
                                            int *issued, int *pdone)
{
	fg_set_err(a.err, FEMGPU_E_TIMEOUT);
	for (int i = 0; i < SW_WAIT_LIMIT && !*(volatile int *)pdone; i++) __nanosleep(64);
	__threadfence_block();
	int last = *(volatile int *)issued;
	for (int q = done; q < last; q++) (void)mbar_wait(&full[q % D], (unsigned)((q / D) & 1));
}

// CW consumer warps (warps 0..CW-1) and one producer warp (warp CW).
template <typename T, bool UPPER, int CW, bool FMA>
__global__ void __launch_bounds__((CW + 1) * 32, 1)
k_sweep(SweepArgs a, const T *__restrict__ in, T *out)
{
	if (a.active && !*a.active) return;
	extern __shared__ __align__(128) unsigned char sm[];
	const unsigned ring_b = (unsigned)al16((SW_RING + 1) * sizeof(T));
	T *ring = (T *)sm;
	unsigned long long *full = (unsigned long long *)(sm + ring_b);
	unsigned long long *empty = full + SW_MAXD;
	unsigned char *stages = sm + ((ring_b + SW_BAR_BYTES + 127) & ~127u);
	__shared__ int failed, issued, pdone;
	volatile int *vfailed = &failed;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, D = a.D;
	const unsigned sbytes = (unsigned)a.stage_bytes;
	// this thread block's run of sub-blocks and levels
	const int sb0 = a.chunk_sb ? a.chunk_sb[blockIdx.x] : 0, sb1 = a.chunk_sb ? a.chunk_sb[blockIdx.x + 1] : a.nsb;
	const int l0 = a.chunk_lev ? a.chunk_lev[blockIdx.x] : 0, l1 = a.chunk_lev ? a.chunk_lev[blockIdx.x + 1] : a.nlev;

	if (tid == 0) {
		failed = 0; issued = 0; pdone = 0;
		ring[SW_RING] = T(0);
		for (int s = 0; s < D; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
		fence_mbar_init();
	}
	__syncthreads();

	if (warp == CW) {                                     // ---- producer warp
		sweep_producer(a, in, stages, sbytes, full, empty, D, sb0, sb1, lane, vfailed, &issued, &pdone, false);
		return;
	}

	const int ctid = tid;                                 // ---- consumer warps
	int sb = 0, s = 0;
	unsigned ph = 0;                                      // phase of full[s] to wait for
	for (int l = l0; l < l1; l++) {
		int nsub = 1, j = 0, s0 = s;
		for (; j < nsub; j++) {
			bool ok = mbar_wait_warp(&full[s], ph, vfailed);
			if (!ok) { *vfailed = 1; break; }
			const unsigned char *st = stages + (unsigned)s * sbytes;
			const LevHdr h = *(const LevHdr *)st;
			if (j == 0) nsub = h.nsub;
			const int *dep = (const int *)(st + SW_HDR);
			const int *outp = dep + h.w * h.cp;
			const T *val = (const T *)(st + h.voff);
			const T *dinv = val + h.w * h.cp;
			const T *bv = (const T *)(st + h.boff);
			if (!h.hasfar) {
				// every dependency is in the ring
				for (int r = ctid; r < h.c; r += CW * 32) {
					T x = bv[r];
					for (int k = 0; k < h.w; k++)
						x = fmsub<T, FMA>(x, ring[(unsigned)dep[k * h.cp + r] & ~SW_NEAR], val[k * h.cp + r]);
					if (UPPER) x = mul(x, dinv[r]);
					ring[(h.start + r) & (SW_RING - 1)] = x;
					out[outp[r]] = x;
				}
			} else {
				for (int r = ctid; r < h.c; r += CW * 32) {
					T x = bv[r];
					for (int k = 0; k < h.w; k++) {
						unsigned d = (unsigned)dep[k * h.cp + r];
						T xd = (d & SW_NEAR) ? ring[d & ~SW_NEAR] : __ldcg(&out[d]);
						x = fmsub<T, FMA>(x, xd, val[k * h.cp + r]);
					}
					if (UPPER) x = mul(x, dinv[r]);
					ring[(h.start + r) & (SW_RING - 1)] = x;
					out[outp[r]] = x;
				}
			}
			if (++s == D) { s = 0; ph ^= 1u; }
		}
		consumer_sync<CW>();
		// every consumer is done with the level's stages: release them
		if (ctid == 0) {
			int q = s0;
			for (int c = 0; c < j; c++) { mbar_arrive(&empty[q]); if (++q == D) q = 0; }
		}
		sb += j;
		if (*vfailed) break;
	}
	if (*vfailed && ctid == 0) sweep_drain(a, full, D, sb, &issued, &pdone);
}

// ------------------------------------------------ record layout (fixed width)
// When every row of a sweep has at most 16 dependencies, each sub-block is a
// 16-byte header {rows, sub-blocks of the level, level-order position of the
// first row, far flag} followed by one record per row: W dependency codes and
// the output slot (ints, padded to 16 bytes), then W factor values and, in
// the backward sweep, the inverted pivot (padded to 16 bytes).  Rows with
// fewer dependencies are padded with the zero ring slot and a zero value,
// after their real terms, so the order of the real operations is unchanged.
// A record is an odd number of 16-byte words (a quarter warp's 16-byte loads
// then fall in distinct banks), and the input slice sits at the same offset
// of every stage: a consumer thread issues all loads of its row before the
// header arrives, which shortens the per-level chain of dependent loads.
__host__ __device__ constexpr int rec_ib(int w) { return ((w + 1) * 4 + 15) & ~15; }
__host__ __device__ constexpr int rec_vb(int w, bool upper, int ts) { return ((w + (upper ? 1 : 0)) * ts + 15) & ~15; }
__host__ __device__ constexpr int rec_bytes(int w, bool upper, int ts)
{
	return (((rec_ib(w) + rec_vb(w, upper, ts)) / 16) & 1) ? rec_ib(w) + rec_vb(w, upper, ts)
	                                                        : rec_ib(w) + rec_vb(w, upper, ts) + 16;
}
#define SW2_CW FG_SW2_CW              // consumer warps of the record-layout sweep (SW_SUB rows)

template <typename T, bool UPPER, bool FMA, int W>
__global__ void __launch_bounds__((SW2_CW + 1) * 32, 1)
k_sweep_rec(SweepArgs a, const T *__restrict__ in, T *out)
{
	constexpr int CW = SW2_CW;
	constexpr int IB = rec_ib(W), VB = rec_vb(W, UPPER, (int)sizeof(T)), RB = rec_bytes(W, UPPER, (int)sizeof(T));
	static_assert(SW_SUB == CW * 32, "one row per consumer thread and sub-block");
	if (a.active && !*a.active) return;
	extern __shared__ __align__(128) unsigned char sm[];
	const unsigned ring_b = (unsigned)al16((SW_RING + 1) * sizeof(T));
	T *ring = (T *)sm;
	unsigned long long *full = (unsigned long long *)(sm + ring_b);
	unsigned long long *empty = full + SW_MAXD;
	unsigned char *stages = sm + ((ring_b + SW_BAR_BYTES + 127) & ~127u);
	__shared__ int failed, issued, pdone;
	volatile int *vfailed = &failed;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, D = a.D;
	const unsigned sbytes = (unsigned)a.stage_bytes;
	const int sb0 = a.chunk_sb ? a.chunk_sb[blockIdx.x] : 0, sb1 = a.chunk_sb ? a.chunk_sb[blockIdx.x + 1] : a.nsb;
	const int l0 = a.chunk_lev ? a.chunk_lev[blockIdx.x] : 0, l1 = a.chunk_lev ? a.chunk_lev[blockIdx.x + 1] : a.nlev;

	if (tid == 0) {
		failed = 0; issued = 0; pdone = 0;
		ring[SW_RING] = T(0);
		for (int s = 0; s < D; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
		fence_mbar_init();
	}
	__syncthreads();

	if (warp == CW) {                                     // ---- producer warp
		sweep_producer(a, in, stages, sbytes, full, empty, D, sb0, sb1, lane, vfailed, &issued, &pdone, true);
		return;
	}

	const int ctid = tid;                                 // ---- consumer warps
	// the record this thread reads in every stage (clamped into the staged rows;
	// rows past a sub-block's count are read but not used)
	const unsigned roff = 16u + (unsigned)(ctid < a.cmax ? ctid : a.cmax - 1) * RB;
	const unsigned boff = (unsigned)a.bvo + (unsigned)(ctid < a.cmax ? ctid : a.cmax - 1) * sizeof(T);
	int sb = 0, s = 0;
	unsigned ph = 0;
	for (int l = l0; l < l1; l++) {
		int nsub = 1, j = 0, s0 = s;
		for (; j < nsub; j++) {
			bool ok = mbar_wait_warp(&full[s], ph, vfailed);
			if (!ok) { *vfailed = 1; break; }
			const unsigned char *st = stages + (unsigned)s * sbytes;
			union { int4 q[IB / 16]; int i[IB / 4]; } ci;
			union { int4 q[VB / 16]; T v[VB / sizeof(T)]; } cv;
#pragma unroll
			for (int q = 0; q < IB / 16; q++) ci.q[q] = ((const int4 *)(st + roff))[q];
#pragma unroll
			for (int q = 0; q < VB / 16; q++) cv.q[q] = ((const int4 *)(st + roff + IB))[q];
			T x = *(const T *)(st + boff);
			const int4 h = *(const int4 *)st;         // rows, sub-blocks, start, far flag
			if (j == 0) nsub = h.y;
			T d[W];
#pragma unroll
			for (int k = 0; k < W; k++) {
				unsigned c = (unsigned)ci.i[k] & ~SW_NEAR;
				d[k] = ring[c < SW_RING ? c : SW_RING];
			}
			if (ctid < h.x) {
				if (h.w) {
#pragma unroll
					for (int k = 0; k < W; k++)
						if (!((unsigned)ci.i[k] & SW_NEAR)) d[k] = __ldcg(&out[ci.i[k]]);
				}
#pragma unroll
				for (int k = 0; k < W; k++) x = fmsub<T, FMA>(x, d[k], cv.v[k]);
				if (UPPER) x = mul(x, cv.v[W]);
				ring[(h.z + ctid) & (SW_RING - 1)] = x;
				out[ci.i[W]] = x;
			}
			if (++s == D) { s = 0; ph ^= 1u; }
		}
		consumer_sync<CW>();
		if (ctid == 0) {
			int q = s0;
			for (int c = 0; c < j; c++) { mbar_arrive(&empty[q]); if (++q == D) q = 0; }
		}
		sb += j;
		if (*vfailed) break;
	}
	if (*vfailed && ctid == 0) sweep_drain(a, full, D, sb, &issued, &pdone);
}

// ------------------------------------------- dataflow sweep (record layout)
// The same records without barriers or a producer warp.  A level is cut into
// chunks of up to 32 rows and the chunks of a matrix block are dealt to the
// block's warps in turn, so consecutive levels go to different warps: a warp
// stages its own chunks (bulk copies into D stages of its own, one mbarrier
// each), takes its next record and its rows' older dependencies while other
// warps compute the levels before, and only the newest value's arrival and the
// operations on it stand between two levels.  (With level l's rows always on
// warps 0, 1, ... a level took one warp's whole turn, about 980 clocks, the
// values it waited for being there long before it looked.)
//
// Ring slots hold the mark "not yet written" (all ones: a NaN no arithmetic
// produces; a value with these bits is stored as the ordinary NaN) until their
// value is there, and a row polls the values it reads: one trip through shared
// memory from a producer to its readers.  A row's terms are taken in order,
// each as soon as its value is there.
//
// Ring slot of lane t of chunk c: 32 c + t modulo the ring (R chunks).  Slots
// are marked again by the writers: chunk c marks chunk c - (R - X - 1).  Warps
// publish their progress (prog[warp]: all its chunks below are done; release)
// and chunk c starts only when all chunks below c - X are done.  A chunk reads
// from the ring at most R - 2 X - 2 chunks back, so nobody still reads what is
// marked, and the chunk that takes the slot next (X + 1 past c) starts only
// when c is done and its marks are known.  Older dependencies come from global
// memory: a warp stores a chunk's outputs after publishing it, so they are
// there once the warp has published its next one; the chunk's header holds
// what it has to wait for (1 + its last chunk with such a dependency, 0: none;
// the program keeps them more than one turn of all warps back).
// Header: {rows, 0, 0, far}, then the records.
//
// Both sweeps of an application, before (per-warp progress flags, rows of a
// level always on the first warps) and now: 64x64 cells, 2 x 127 levels, FP64:
// 117 us, 67; 400x300 cells, 2 x 1098 levels, FP64: 1.50 ms, 0.80; 2048x1024
// cells in 32 blocks, double-single chains, the largest block 9106 chunks:
// 0.70 ms, 0.45.  FP64: a level is a poll (about 100 clocks) and the newest
// values' multiplications and subtractions, 64 clocks each on a warp; four
// chunks a level and more keep the four FP64 pipes (6 or 7 such operations a
// chunk) half busy.  Double-single: issue slots, about 130 FP32 operations a
// chunk of some 380 slots.
#define DF_HDR 16
#define DF_WARPS 24                   // most warps of a block
#define DF_MAXD 8                     // ... stages of a warp
#define DF_BARS 128                   // most stages of a block
#define DF_DONE 0x7fffffff
// Warps: rows in FP64 wait for their level (20 or 24 warps gain nothing over
// 16); a chain chunk is a long run of dependent FP32 operations, so the narrow
// ones, whose registers allow it, take 24 (2048x1024, 32 blocks: 667 us an
// application with 16, 586 with 20, 554 with 24 before their chunks lay side by
// side, 448 now).  Rows of 16 do not fit the registers of 16 warps.
__host__ __device__ constexpr int df_warps(bool cs, int w) { return cs && w <= 4 ? 24 : w > 12 ? 12 : 16; }

// How a row waits for values that are late.  Narrow rows, and FP64 ones of any
// width, go on term by term, each as soon as its value is there.  Wide rows in
// FP32 or double-single arithmetic wait for all of them and run their terms then
// without a vote between: a term costs less than its vote.  Looking at every
// value still missing while one is late takes code that grows with the square
// of the width, which for 12 and 16 was no longer unrolled (values in local
// memory): a look at the next three is enough.  An application at 400x300 with
// ILU(4) (12 wide) and ILU(6) (16), squares / next three / all:
// FP64 rows 19.6 / 8.11 / 8.52 and 42.5 / 13.8 / 14.3 ms, double-single chains
// 13.1 / 4.22 / 3.56 and 17.8 / 6.24 / 4.70, FP32 chains 3.91 / 2.66 / 1.50 and
// 16.9 / 4.15 / 2.03; Navier-Stokes 256x256 (12 wide), an FGMRES iteration 6.04
// / 2.17 / 1.95 ms.
template <typename T> __host__ __device__ constexpr bool sweep_all(int w) { return w > 8; }
template <> __host__ __device__ constexpr bool sweep_all<double>(int) { return false; }

// Ring values: polled loads, stores, the mark.
template <typename T> __device__ __forceinline__ bool ring_unset(T v)
{
	if (sizeof(T) == 8) {
		const uint2 u = *(const uint2 *)&v;
		return (u.x & u.y) == ~0u;
	}
	return *(const unsigned *)&v == ~0u;
}
template <typename T> __device__ __forceinline__ T ring_ld(unsigned p)      // p: a shared-memory address
{
	T v;
	if (sizeof(T) == 8) {
		unsigned long long u;
		asm volatile("ld.relaxed.cta.shared.u64 %0, [%1];" : "=l"(u) : "r"(p) : "memory");
		*(unsigned long long *)&v = u;
	} else {
		unsigned u;
		asm volatile("ld.relaxed.cta.shared.u32 %0, [%1];" : "=r"(u) : "r"(p) : "memory");
		*(unsigned *)&v = u;
	}
	return v;
}
template <typename T> __device__ __forceinline__ void ring_st(unsigned p, T v)
{
	if (sizeof(T) == 8)
		asm volatile("st.relaxed.cta.shared.u64 [%0], %1;" :: "r"(p), "l"(*(const unsigned long long *)&v) : "memory");
	else
		asm volatile("st.relaxed.cta.shared.u32 [%0], %1;" :: "r"(p), "r"(*(const unsigned *)&v) : "memory");
}
template <typename T> __device__ __forceinline__ T ring_mark()
{
	T v;
	if (sizeof(T) == 8) *(unsigned long long *)&v = ~0ull;
	else *(unsigned *)&v = ~0u;
	return v;
}
template <typename T> __device__ __forceinline__ T ring_value(T v)       // never the mark
{
	if (ring_unset(v)) {
		if (sizeof(T) == 8) *(unsigned long long *)&v = 0x7ff8000000000000ull;
		else *(unsigned *)&v = 0x7fc00000u;
	}
	return v;
}
template <> __device__ __forceinline__ dsf ring_value(dsf v)
{
	if (ring_unset(v)) v.hi = __uint_as_float(0x7fc00000u);
	return v;
}
// ------------------------------------------------ chain-scan sweep (records)
// After SYMRCM the rows of a matrix block form fronts, and along a front every
// row depends on its predecessor in the sweep order: y_i = a_i + b_i y_pred,
// with a_i the row's other terms (backward: times the inverted pivot) and b_i
// its coupling to the predecessor -- a first-order linear recurrence.  The
// program groups up to 32 chained rows into a segment, gives segments (not
// rows) dependency levels, and packs each level's segments into 32-slot
// chunks, one per warp (a segment never straddles two chunks; unused slots are
// padding).  A warp computes a_i for its 32 slots from earlier levels, then
// solves its segments' recurrences with a Kogge-Stone scan over the lanes:
// five steps a_t += M_k,t a_{t-2^k}, the multipliers (products of b along the
// segment, zero across a segment start) precompiled from the factor by
// k_chain_mult.  At 2048x1024 with 16 blocks the deepest block falls from
// 1340 row levels to 349 segment levels.  The scan reassociates the
// recurrence, so results agree with the row-by-row sweeps to rounding, not bit
// for bit: it serves the fused-arithmetic (FGMRES) and FP32 sweeps only.
// Records: W dependency codes (the predecessor excluded) and the output slot
// (-1: padding), then W values, the inverted pivot (backward) and M_0..M_4.
// Staging, ring and bounded waits are the dataflow sweep's.
__host__ __device__ constexpr int rec_vb_cs(int w, bool upper, int ts) { return ((w + (upper ? 1 : 0) + 5) * ts + 15) & ~15; }

template <typename T> __device__ __forceinline__ T fma_t(T a, T b, T c);
template <> __device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }
template <> __device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }
template <> __device__ __forceinline__ dsf fma_t(dsf a, dsf b, dsf c) { return ds_fma(a, b, c); }

// A row's record in registers.  Row programs: the rows' records one after the
// other; chain programs (32 rows to a chunk always): the lanes' 16-byte words
// side by side, without the padding that keeps whole records off each other's
// banks.
template <typename T, bool UPPER, bool CS, int W> struct SweepRec {
	static constexpr int IB = rec_ib(W), VB = CS ? rec_vb_cs(W, UPPER, (int)sizeof(T)) : rec_vb(W, UPPER, (int)sizeof(T));
	static constexpr int FIRST = CS ? 16 : rec_bytes(W, UPPER, (int)sizeof(T)), STEP = CS ? 512 : 16;
	int i[IB / 4];
	T v[VB / sizeof(T)];
	T x0;
	int rows, far;
	__device__ __forceinline__ void load(const unsigned char *st, unsigned roff, unsigned boff)
	{
#pragma unroll
		for (int k = 0; k < IB / 16; k++) {
			const int4 q = *(const int4 *)(st + roff + k * STEP);
			i[4 * k] = q.x; i[4 * k + 1] = q.y; i[4 * k + 2] = q.z; i[4 * k + 3] = q.w;
		}
#pragma unroll
		for (int k = 0; k < VB / 16; k++) {
			union { int4 q; T t[16 / sizeof(T)]; } u;
			u.q = *(const int4 *)(st + roff + (IB / 16 + k) * STEP);
#pragma unroll
			for (int j = 0; j < (int)(16 / sizeof(T)); j++) v[k * (16 / sizeof(T)) + j] = u.t[j];
		}
		x0 = *(const T *)(st + boff);
		rows = CS ? 32 : *(const int *)st;
		far = *(const int *)(st + 12);
	}
};

// One sweep of this thread block's matrix block with the barriers `full' (D a
// warp); every thread returns after a block barrier, true when a wait gave up.
// CS: a chain-scan program.
template <typename T, bool UPPER, bool FMA, bool CS, int W>
__device__ __forceinline__ bool sweep_run(const SweepArgs &a, const T *__restrict__ in, T *out, unsigned char *sm,
                                          unsigned long long *full, int *failed, int *prog)
{
	typedef SweepRec<T, UPPER, CS, W> Rec;
	constexpr bool ALL = sweep_all<T>(W);
	const unsigned rb = smem_u32(sm), zero = rb + (unsigned)a.ring * (unsigned)sizeof(T);
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, D = a.D, nw = blockDim.x >> 5;
	const int sb0 = a.chunk_sb[blockIdx.x], cnt = a.chunk_sb[blockIdx.x + 1] - sb0;
	unsigned char *stages = sm + (((unsigned)al16((a.ring + 1) * sizeof(T)) + 2 * DF_BARS * 8 + 127) & ~127u) +
	                        (unsigned)(warp * D) * (unsigned)a.stage_bytes;
	volatile int *vfailed = failed;
	full += warp * D;

	if (tid == 0) *failed = 0;
	if (lane == 0) {
		for (int s = 0; s < D; s++) mbar_init(&full[s], 1);
		fence_mbar_init();
		prog[warp] = warp < cnt ? warp : DF_DONE;
	}
	for (int q = tid; q <= a.ring; q += blockDim.x) ((T *)sm)[q] = q < a.ring ? ring_mark<T>() : zero_t<T>();
	__syncthreads();

	// row programs: lane k: where turn tb + k's chunk and its input slice lie (and, mn, turn tb + 32 + k's)
	struct Meta { long long off; int len, p0, vb; } m, mn;
	auto meta = [&](int turn) {
		Meta r = { 0, 0, 0, 0 };
		const long long c = warp + (long long)turn * nw;
		if (c < cnt) {
			const int i = sb0 + (int)c;
			r.off = __ldg(&a.blk_off[i]);
			r.len = (int)(__ldg(&a.blk_off[i + 1]) - r.off);
			r.p0 = __ldg(&a.sb_in[i]);
			r.vb = __ldg(&a.sb_inb[i]);
		}
		return r;
	};
	int tb = 0;
	if (!CS) { m = meta(lane); mn = meta(32 + lane); }
	// chain programs: whole chunks, one after the other
	const unsigned char *gp = a.prog + (long long)(sb0 + warp) * a.bvo;
	const T *ip = in + 32LL * (sb0 + warp);
	auto issue = [&](int turn, int s) {                   // turn's chunk into stage s (turns in order)
		int len = a.bvo, vb = 32 * (int)sizeof(T);
		if (!CS) {
			if (turn == tb + 32) { tb += 32; m = mn; mn = meta(tb + 32 + lane); }
			const int k = turn - tb;
			gp = a.prog + __shfl_sync(0xffffffffu, m.off, k);
			ip = in + __shfl_sync(0xffffffffu, m.p0, k);
			len = __shfl_sync(0xffffffffu, m.len, k);
			vb = __shfl_sync(0xffffffffu, m.vb, k);
		}
		if (lane == 0) {
			unsigned char *dst = stages + (unsigned)s * (unsigned)a.stage_bytes;
			fence_proxy_async();
			mbar_expect_tx(&full[s], (unsigned)(len + vb));
			bulk_g2s(dst, gp, (unsigned)len, &full[s]);
			bulk_g2s(dst + (unsigned)a.bvo, ip, (unsigned)vb, &full[s]);
		}
		if (CS) { gp += (long long)nw * a.bvo; ip += 32 * nw; }
	};
	const int turns = warp < cnt ? (cnt - warp + nw - 1) / nw : 0;
	int issued = 0, waited = 0;
	for (; issued < D && issued < turns; issued++) issue(issued, issued);

	const int rl = lane < a.cmax ? lane : a.cmax - 1;     // rows past a chunk's count are read but not used
	const unsigned roff = (unsigned)DF_HDR + (unsigned)rl * Rec::FIRST, boff = (unsigned)a.bvo + (unsigned)rl * sizeof(T);
	int s = 0, known = -DF_DONE;
	unsigned ph = 0;
	bool fail = false;
	// byte offsets of the chunk's slot and of the one it marks
	const unsigned bytes = (unsigned)a.ring * (unsigned)sizeof(T) - 1, step = 32u * (unsigned)nw * (unsigned)sizeof(T);
	unsigned pos = (32u * (unsigned)warp + (unsigned)lane) * (unsigned)sizeof(T) & bytes,
	         next = (pos + 32u * (unsigned)(a.look + 1) * (unsigned)sizeof(T)) & bytes;
	for (int t = 0; t < turns && !fail; t++) {
		const int c = warp + t * nw;
		if (!mbar_wait_warp(&full[s], ph, vfailed)) { fail = true; break; }
		waited++;
		Rec cur;
		cur.load(stages + (unsigned)s * (unsigned)a.stage_bytes, roff, boff);
		__syncwarp();                                     // the chunk is in registers: its stage takes the next
		if (issued < turns) { issue(issued, s); issued++; }
		if (++s == D) { s = 0; ph ^= 1u; }
		// every chunk below c - X, and a far dependency's warp past its next chunk
		const int far = cur.far, want = max(c - a.look, far ? far + nw : 0);
		for (int it = 0; known < want && it < a.wait; it++) {
			known = __reduce_min_sync(0xffffffffu, lane < nw && lane != warp ? ld_acquire_cta(&prog[lane]) : DF_DONE);
			if (known < want && (it & 63) == 63 && __any_sync(0xffffffffu, *vfailed != 0)) break;
		}
		if (known < want) { fail = true; break; }
		__syncwarp();                                     // the lanes' acquires order every lane's reads
		const bool on = CS || lane < cur.rows;
		unsigned src[W];
		T d[W], y = cur.x0;
#pragma unroll
		for (int k = 0; k < W; k++) src[k] = on ? rb + (unsigned)cur.i[k] : zero;
		if (far) {
#pragma unroll
			for (int k = 0; k < W; k++)                   // read back from global memory (below), zero meanwhile
				if (on && ((unsigned)cur.i[k] & SW_NEAR)) src[k] = zero;
		}
		bool miss = false;
#pragma unroll
		for (int k = 0; k < W; k++) d[k] = ring_ld<T>(src[k]);
		if (far) {
#pragma unroll
			for (int k = 0; k < W; k++)
				if (on && ((unsigned)cur.i[k] & SW_NEAR)) d[k] = ld_cg(&out[(unsigned)cur.i[k] & ~SW_NEAR]);
		}
#pragma unroll
		for (int k = 0; k < W; k++) miss = miss || ring_unset(d[k]);
		bool late = __any_sync(0xffffffffu, miss);
		if (ALL && late) {
			int it = 0;
			do {
				if (it >= a.wait || ((it & 63) == 63 && __any_sync(0xffffffffu, *vfailed != 0))) { fail = true; break; }
				it++;
				miss = false;
#pragma unroll
				for (int k = 0; k < W; k++) {
					if (ring_unset(d[k])) d[k] = ring_ld<T>(src[k]);
					miss = miss || ring_unset(d[k]);
				}
			} while (__any_sync(0xffffffffu, miss));
			if (fail) break;
			late = false;
		}
		if (!late) {
#pragma unroll
			for (int k = 0; k < W; k++) y = fmsub<T, FMA>(y, d[k], cur.v[k]);
		} else {
#pragma unroll
			for (int k = 0; k < W; k++) {
				if (__any_sync(0xffffffffu, ring_unset(d[k]))) {
					int it = 0;
					do {
						if (it >= a.wait || ((it & 63) == 63 && __any_sync(0xffffffffu, *vfailed != 0))) { fail = true; break; }
						it++;
						if (ring_unset(d[k])) d[k] = ring_ld<T>(src[k]);
					} while (__any_sync(0xffffffffu, ring_unset(d[k])));
					if (fail) break;
#pragma unroll
					for (int q = k + 1; q < W && (W <= 8 || q < k + 4); q++)   // the others may have come meanwhile
						if (ring_unset(d[q])) d[q] = ring_ld<T>(src[q]);
				}
				y = fmsub<T, FMA>(y, d[k], cur.v[k]);
			}
			if (fail) break;
		}
		if (UPPER) y = mul(y, cur.v[W]);
		if (CS) {
			// the segments' recurrences across the warp's lanes
#pragma unroll
			for (int k = 0; k < 5; k++) {
				const T up = shfl_up_t(y, 1 << k);
				if (lane >= (1 << k)) y = fma_t(cur.v[W + (UPPER ? 1 : 0) + k], up, y);
			}
		}
		if (on) y = ring_value(y);
		if (on) ring_st(rb + pos, y);
		ring_st(rb + next, ring_mark<T>());
		pos = (pos + step) & bytes;
		next = (next + step) & bytes;
		__syncwarp();
		if (lane == 0) st_release_cta(&prog[warp], c + nw);
		if (on && cur.i[W] >= 0) out[cur.i[W]] = y;
	}
	if (fail) {
		// record the timeout, wait (bounded) for this warp's copies in flight
		*vfailed = 1;
		if (lane == 0) {
			fg_set_err(a.err, FEMGPU_E_TIMEOUT);
			for (int q = waited; q < issued; q++) (void)mbar_wait(&full[q % D], (unsigned)((q / D) & 1));
		}
	}
	__syncwarp();
	if (lane == 0) st_release_cta(&prog[warp], DF_DONE);  // its last outputs are stored
	__syncthreads();
	return *vfailed != 0;
}

#define DF_SMEM(ring) (sm + (unsigned)al16(((ring) + 1) * sizeof(T)))
template <typename T, bool UPPER, bool FMA, bool CS, int W>
__global__ void __launch_bounds__(df_warps(CS, W) * 32, 1)
k_sweep_df(SweepArgs a, const T *__restrict__ in, T *out)
{
	if (a.active && !*a.active) return;
	extern __shared__ __align__(128) unsigned char sm[];
	__shared__ int failed, prog[DF_WARPS];
	(void)sweep_run<T, UPPER, FMA, CS, W>(a, in, out, sm, (unsigned long long *)DF_SMEM(a.ring), &failed, prog);
}

// Both sweeps of one preconditioner application in one launch: each thread
// block sweeps its matrix block forward (in -> y) and then backward (y ->
// out), keeping its SM between the two (a block's backward sweep reads only
// its own forward results).  The forward sweep's global stores of y are
// ordered before the bulk copies of y by an async-proxy fence and the block
// barrier; the backward sweep runs on barriers of its own.  Dynamic shared
// memory: the larger of the two sweeps' layouts.
template <typename T, bool FMA, bool CS, int W>
__global__ void __launch_bounds__(df_warps(CS, W) * 32, 1)
k_sweep_fb(SweepArgs al, SweepArgs au, const T *__restrict__ in, T *y, T *out)
{
	if (al.active && !*al.active) return;
	extern __shared__ __align__(128) unsigned char sm[];
	__shared__ int failed, prog[DF_WARPS];
	if (sweep_run<T, false, FMA, CS, W>(al, in, y, sm, (unsigned long long *)DF_SMEM(al.ring), &failed, prog)) return;
	asm volatile("fence.proxy.async.global;" ::: "memory");
	__syncthreads();
	(void)sweep_run<T, true, FMA, CS, W>(au, y, out, sm, (unsigned long long *)DF_SMEM(au.ring) + DF_BARS, &failed, prog);
}

// Scan multipliers of a chain-scan program from the factor, one warp per
// 32-slot chunk: b = -L(row, pred) forward, -Dinv[row] U(row, pred) backward
// (0 at a segment start and in padding); M_0 = b and, as the scan composes
// the recurrences, M_{k+1,t} = M_k,t M_k,t-2^k for t >= 2^k (else M_k,t).
template <typename T, bool UPPER>
__global__ void k_chain_mult(unsigned char *prog, const long long *voff, const int *src, const int *row, int nslot, int mo,
                             const double *LU, const double *Dinv)
{
	const int lane = threadIdx.x & 31;
	const int w0 = (int)((blockIdx.x * (unsigned)blockDim.x + threadIdx.x) >> 5);
	const int nw = (int)((gridDim.x * (unsigned)blockDim.x) >> 5);
	for (int c = w0; c * 32 < nslot; c += nw) {          // uniform per warp
		const int i = c * 32 + lane;
		const int sr = i < nslot ? src[i] : -1;
		double m = 0.0;
		if (sr >= 0) m = UPPER ? -(Dinv[row[i]] * LU[sr]) : -LU[sr];
		double M[5];
		M[0] = m;
#pragma unroll
		for (int k = 0; k < 4; k++) {
			const double up = __shfl_up_sync(0xffffffffu, M[k], 1 << k);
			M[k + 1] = lane >= (1 << k) ? M[k] * up : M[k];
		}
		const long long o = i < nslot ? voff[i] : -1;
		if (o >= 0) {
			constexpr int PER = 16 / (int)sizeof(T);     // value v of a slot: word v / PER of its lane
#pragma unroll
			for (int k = 0; k < 5; k++)
				((T *)(prog + o + (mo + k) / PER * 512))[(mo + k) % PER] = from_d<T>(M[k]);
		}
	}
}

// Gather the sweep input into padded level order: in[ppos[i]] = (T) p[rows[i]].
template <typename T, typename TI>
__global__ void k_perm_in(const TI *__restrict__ p, const int *__restrict__ rows,
                          const int *__restrict__ ppos, int n, T *in)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
		in[ppos[i]] = (T)p[rows[i]];
}

// The same gather into double-single values, and back from double-single
// (the backward sweep's natural-order output) to FP64.
__global__ void k_perm_in_ds(const double *__restrict__ p, const int *__restrict__ rows,
                             const int *__restrict__ ppos, int n, dsf *in)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
		in[ppos[i]] = ds_from(p[rows[i]]);
}

__global__ void k_perm_in_dsds(const dsf *__restrict__ p, const int *__restrict__ rows,
                               const int *__restrict__ ppos, int n, dsf *in, const int *active)
{
	if (active && !*active) return;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
		in[ppos[i]] = p[rows[i]];
}

// dpos[rows[i]] = ppos[i]: where the gather of the double-single apply puts
// natural row r, for a product that writes the gathered input itself.
__global__ void k_inv_gather(const int *__restrict__ rows, const int *__restrict__ ppos, int n, int *dpos)
{
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dpos[rows[i]] = ppos[i];
}

__global__ void k_ds_to_double(const dsf *__restrict__ x, int n, double *z, const int *active)
{
	if (active && !*active) return;
	for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
		const dsf v = x[i];
		z[i] = (double)v.hi + (double)v.lo;
	}
}

// Refresh the value slots of a program from the factor (after every factorisation).
template <typename T>
__global__ void k_refresh(unsigned char *prog, const long long *val_off, const int *val_src, long long nval,
                          const double *LU, const double *Dinv)
{
	for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nval;
	     i += (long long)gridDim.x * blockDim.x) {
		int s = val_src[i];
		double v = (s >= 0) ? LU[s] : (s == -1 ? 0.0 : Dinv[-2 - s]);
		*(T *)(prog + val_off[i]) = from_d<T>(v);
	}
}

// ---------------------------------------------------------- factor ------
// IKJ ILU(0) as a dataflow of rows (fg_dataflow.cuh): L lanes per row (8, 16
// or 32, the smallest that holds the longest row), lane q keeping entry q.  A
// warp takes the next 32 / L rows of one dependency level, and for each lower
// entry in ascending column order waits for the values of row k it reads --
// the pivot's inverse in lane "group", U(k, .) in the lanes of the columns both
// rows have -- and updates its entries, the operations and their order those
// of ILUp_precond_setup.c:119-139.  What each lane reads is precompiled, so a
// row needs no pattern searches.
//
// The program takes 16 + 8 L + L L bytes a row, 144, 400 or 1296 for rows of up
// to 8, 16 and 32 entries (the longest row's L for all), on the device and, while
// it is built, on the host: transport 144, ILU(1) and ILU(2) of it 400,
// Navier-Stokes (21 entries) and Euler (28) 1296.  Programs of operand lists took
// 212, 312, 297, 724 and 1291.
//
// What bounds it is the chain of levels: per level one trip of a value
// through L2 (0.36 us), two dependent rows' groups (three FP64 operations of 31
// ns each; a warp's FP64 instruction holds this part's FP64 pipe for 64
// clocks) and the pivot's reciprocal (0.19 us); measured 1.3 us a level.
// Before it, levels were split over the CTAs of a thread-block cluster with a
// cluster barrier after each (4.6 us a level), or, for rows of more than 64
// program words, walked by one CTA (17 us a level).  Measured, before and now:
// 400x300 transport, one block (1098 levels) 4.80 -> 1.42 ms; 2048x1024 in 32
// blocks 5.81 -> 1.96 ms; Navier-Stokes 96x96 (27k rows of up to 21 entries)
// 17.0 -> 0.96 ms.  (Polling one operand at a time, each missing one costs a
// trip of its own: 1.65 and 1.11 ms.)
#define FAC_CAP 32                    // entries of a row
#define FAC_TPB 128                   // four warps: one per FP64 pipe
#define FAC_AHEAD 6                   // levels whose warps are resident (3, 6 and 12 measure within 3 %)
#define FAC_NONE 0xff                 // position codes: the group leaves the lane's entry alone,
#define FAC_MULT 0xfe                 // the lane's entry is the group's own (the multiplier)

__global__ void k_ilu0_factor_init(double *LU, long long nnz, double *Dinv, int n, fg_ticket *tk)
{
	const long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, st = (long long)gridDim.x * blockDim.x;
	if (i0 == 0) { tk->next = 0u; tk->abort = 0u; }
	for (long long i = i0; i < nnz; i += st) LU[i] = __longlong_as_double((long long)FG_UNSET);
	for (long long i = i0; i < n; i += st) Dinv[i] = __longlong_as_double((long long)FG_UNSET);
}

__device__ __forceinline__ unsigned fac_code(uint2 c, int k) { return ((k < 4 ? c.x : c.y) >> (8 * (k & 3))) & 255u; }

template <int L>
__global__ void __launch_bounds__(FAC_TPB)
k_ilu0_factor_df(const double *__restrict__ AA, const int4 *__restrict__ head, const int2 *__restrict__ grp,
                 const uint2 *__restrict__ pos, int nslot, double *LU, double *Dinv, fg_ticket *tk, int *err, int poll0)
{
	constexpr int R = 32 / L, NB = L / 8;
	const int lane = threadIdx.x & 31, q = lane & (L - 1), l0 = lane & ~(L - 1);
	const unsigned end = (unsigned)(nslot / R);          // slots are padded to whole warps
	for (;;) {
		const unsigned t = fg_take(tk, end);
		if (t >= end) return;
		const long long sl = (long long)t * R + lane / L;
		const int4 h = __ldcs(&head[sl]);
		const int2 g = __ldcs(&grp[sl * L + q]);
		uint2 code[NB];
#pragma unroll
		for (int b = 0; b < NB; b++) code[b] = __ldcs(&pos[(sl * L + q) * NB + b]);
		const int len = h.y & 255, dpos = (h.y >> 8) & 255, ng = h.y >> 16;
		const int most = __reduce_max_sync(0xffffffffu, ng);
		double v = q < len ? __ldcs(&AA[h.x + q]) : 1.0;   // (a padding slot's 1/d stays ordinary)
		unsigned long long piv = q < ng ? fg_ld_poll(&Dinv[g.x]) : 0ull;
#pragma unroll
		for (int b = 0; b < NB; b++) {
			const double *at[8];
			unsigned long long u[8];
#pragma unroll
			for (int k = 0; k < 8; k++) {
				const unsigned c = 8 * b < most ? fac_code(code[b], k) : FAC_NONE;
				at[k] = LU + (__shfl_sync(0xffffffffu, g.y, l0 + 8 * b + k) + (int)c);
				u[k] = c < FAC_MULT ? fg_ld_poll(at[k]) : 0ull;
			}
#pragma unroll
			for (int k = 0; k < 8; k++) {
				const int gi = 8 * b + k;
				if (gi < most) {                              // uniform
					const unsigned c = fac_code(code[b], k);
					const unsigned own = (__ballot_sync(0xffffffffu, c == FAC_MULT) >> l0) & (0xffffffffu >> (32 - L));
					const int from = own ? l0 + __ffs(own) - 1 : lane;
					// everything still missing is polled again together: operands
					// that come at the same time cost one trip, not one each
					for (int it = poll0;; it++) {
						if (!__any_sync(0xffffffffu, u[k] == FG_UNSET || (q == gi && piv == FG_UNSET))) break;
						if (piv == FG_UNSET) piv = fg_ld_poll(&Dinv[g.x]);
#pragma unroll
						for (int m = k; m < 8; m++)
							if (u[m] == FG_UNSET) u[m] = fg_ld_poll(at[m]);
						if (!fg_keep_polling(it, tk, err)) return;
					}
					const double lq = __dmul_rn(__shfl_sync(0xffffffffu, v, from),
					                            __shfl_sync(0xffffffffu, __longlong_as_double((long long)piv), l0 + gi));
					const double w = __dsub_rn(v, __dmul_rn(lq, __longlong_as_double((long long)u[k])));
					v = c == FAC_MULT ? lq : c == FAC_NONE ? v : w;
				}
			}
		}
		if (q < len) fg_st_value(&LU[h.x + q], v);
		const double d = __shfl_sync(0xffffffffu, v, l0 + dpos);
		const bool zero = ((unsigned long long)__double_as_longlong(d) << 1) == 0ull;   // no FP64 compare
		const double inv = 1.0 / d;
		if (q == dpos && h.z >= 0) {
			fg_st_value(&Dinv[h.z], zero ? 0.0 : inv);
			if (zero) fg_set_err(err, FEMGPU_E_ZERO_PIVOT);
		}
	}
}

// ------------------------------------------------------- host: programs
struct HostLevels {
	int nlev;
	std::vector<int> start, pstart, rows, pos, ppos;   // pos/ppos indexed by row
};

// Matrix block of a row: P contiguous runs of the numbering (P = 0: one).
struct Blocks {
	int P = 0;
	std::vector<int> id;                                  // block of each row (P > 0)
	int of(int r) const { return P ? id[r] : 0; }
	bool same(int r, int c) const { return !P || id[r] == id[c]; }
};

// Block ILU(0) cuts: P contiguous runs of the numbering; couplings between
// runs are dropped.  The P thread blocks of a sweep run side by side, so the
// slowest run (its chunks, and its depth in levels counted with the couplings
// dropped) sets its time, while where the cuts fall sets how many FGMRES
// iterations the weaker preconditioner costs.  After SYMRCM every front is a
// dependency chain about as long as the front is wide, so equal row counts
// leave the middle runs deepest.  FEMGPU_ILU_BLOCK_CUT selects:
//   levels (default)  run b starts at the first row where the running maximum
//                     of the full factor's forward level reaches
//                     ceil(b * levels / P): equal spans of fronts;
//   depth             the smallest budget T for which the greedy scan (open a
//                     new run at the row whose level would reach T) makes at
//                     most P runs (bisection), the runs with the most rows then
//                     halved until there are P: the shallowest deepest run;
//   rows              row r in run floor(r * P / n).
// Measured with FGMRES(80) to 1e-8 on the double-single chain sweeps, an
// application and the iterations of three Picard steps, levels / rows / depth:
// 2048x1024, P=32: 500 us 47 109 100 / 502 us 53 136 142 / 808 us 58 205 272;
// 1023x1023, P=32: 318 us 56 110 341 / 337 us 63 150 293 / 711 us 83 409 625;
// 1023x511, P=16: 271 us 57 57 61 / 328 us 58 62 65 / 396 us 58 64 67.  The
// row cut's largest run has half as many chunks at 2048x1024 (4996 against
// 9106) but more levels: no faster, and more iterations.
static std::vector<int> greedy_runs(const int *IA, const int *JA, int n, int T, std::vector<int> &lev)
{
	std::vector<int> first(1, 0);
	int start = 0;
	for (int i = 0; i < n; i++) {
		int L = 0;
		for (int k = IA[i]; k < IA[i + 1] && JA[k] < i; k++)
			if (JA[k] >= start) L = std::max(L, lev[JA[k]] + 1);
		if (L >= T) { start = i; L = 0; first.push_back(i); }
		lev[i] = L;
	}
	first.push_back(n);
	return first;
}

static Blocks make_blocks(const int *IA, const int *JA, int n, int P, std::vector<int> *first_out)
{
	Blocks B;
	if (P <= 1 || n <= 1) { if (first_out) *first_out = { 0, n }; return B; }
	P = std::min(P, n);
	std::vector<int> cut;
	const char *e = getenv("FEMGPU_ILU_BLOCK_CUT");
	if (e && !strcmp(e, "rows")) {
		cut.assign(P + 1, n);
		for (int b = 0; b < P; b++) cut[b] = (int)(((long long)b * n + P - 1) / P);
	} else if (!e || strcmp(e, "depth")) {
		std::vector<int> lev(n, 0), run(n, 0);
		int top = 0;
		for (int i = 0; i < n; i++) {
			int L = 0;
			for (int k = IA[i]; k < IA[i + 1] && JA[k] < i; k++) L = std::max(L, lev[JA[k]] + 1);
			lev[i] = L;
			top = std::max(top, L);
			run[i] = top;
		}
		const long long nl = (long long)top + 1;
		cut.assign(P + 1, n);
		cut[0] = 0;
		for (int b = 1, i = 0; b < P; b++) {
			const long long fl = (nl * b + P - 1) / P;
			while (i < n && run[i] < fl) i++;
			cut[b] = i;
		}
		for (int b = 1; b < P; b++) cut[b] = std::max(cut[b], cut[b - 1] + 1);     // no empty run
		for (int b = P - 1; b >= 1; b--) cut[b] = std::min(cut[b], cut[b + 1] - 1);
	} else {
		std::vector<int> lev(n, 0);
		int lo = 1, hi = n;                       // T = n always gives one run
		while (lo < hi) {
			int T = lo + (hi - lo) / 2;
			if ((int)greedy_runs(IA, JA, n, T, lev).size() - 1 <= P) hi = T;
			else lo = T + 1;
		}
		cut = greedy_runs(IA, JA, n, lo, lev);
		while ((int)cut.size() - 1 < P) {          // halve the run with the most rows
			int bb = 0;
			for (int b = 1; b + 1 < (int)cut.size(); b++)
				if (cut[b + 1] - cut[b] > cut[bb + 1] - cut[bb]) bb = b;
			cut.insert(cut.begin() + bb + 1, cut[bb] + (cut[bb + 1] - cut[bb]) / 2);
		}
	}
	B.P = P;
	B.id.assign(n, 0);
	for (int b = 0; b < P; b++)
		for (int r = cut[b]; r < cut[b + 1]; r++) B.id[r] = b;
	if (first_out) *first_out = cut;
	return B;
}

// Dependency levels of the forward (lower) or backward sweep; with blocks,
// levels are numbered block by block (block b's levels follow block b-1's),
// and clev [P+1] receives each block's first level.
static HostLevels host_levels(const int *IA, const int *JA, int n, bool lower, const Blocks &B,
                              std::vector<int> *clev = nullptr)
{
	HostLevels H;
	std::vector<int> lev(n, 0);
	int P = B.P ? B.P : 1;
	std::vector<int> bl(P, 0);                 // levels of each block
	if (lower) {
		for (int i = 0; i < n; i++) {
			int L = 0;
			for (int k = IA[i]; k < IA[i + 1] && JA[k] < i; k++)
				if (B.same(i, JA[k])) L = std::max(L, lev[JA[k]] + 1);
			lev[i] = L; bl[B.of(i)] = std::max(bl[B.of(i)], L + 1);
		}
	} else {
		for (int i = n - 1; i >= 0; i--) {
			int L = 0;
			for (int k = IA[i]; k < IA[i + 1]; k++) if (JA[k] > i && B.same(i, JA[k])) L = std::max(L, lev[JA[k]] + 1);
			lev[i] = L; bl[B.of(i)] = std::max(bl[B.of(i)], L + 1);
		}
	}
	std::vector<int> boff(P + 1, 0);
	for (int b = 0; b < P; b++) boff[b + 1] = boff[b] + bl[b];
	for (int i = 0; i < n; i++) lev[i] += boff[B.of(i)];
	if (clev) *clev = boff;
	int nlev = boff[P];
	H.nlev = nlev;
	H.start.assign(nlev + 1, 0);
	H.pstart.assign(nlev + 1, 0);
	for (int i = 0; i < n; i++) H.start[lev[i] + 1]++;
	for (int l = 0; l < nlev; l++) {
		int c = H.start[l + 1];
		H.start[l + 1] += H.start[l];
		H.pstart[l + 1] = H.pstart[l] + ((c + 3) & ~3);      // 16-byte aligned level slices
	}
	std::vector<int> fill(H.start.begin(), H.start.end() - 1);
	H.rows.assign(n, 0);
	H.pos.assign(n, 0);
	H.ppos.assign(n, 0);
	for (int i = 0; i < n; i++) {
		int p = fill[lev[i]]++;
		H.rows[p] = i;
		H.pos[i] = p;
		H.ppos[i] = H.pstart[lev[i]] + (p - H.start[lev[i]]);
	}
	return H;
}

template <typename X>
static int up_vec(X **d, const std::vector<X> &h)
{
	FG_TRY(cudaMalloc((void **)d, sizeof(X) * (h.size() + 1)));
	if (!h.empty()) FG_TRY(cudaMemcpy(*d, h.data(), sizeof(X) * h.size(), cudaMemcpyHostToDevice));
	return 0;
}

// Width of the record layout for a sweep whose widest row has w dependencies
// (0: the ELL sub-block layout, used above 16 or when FEMGPU_SWEEP_LAYOUT=ell).
static int rec_width(int w)
{
	const char *e = getenv("FEMGPU_SWEEP_LAYOUT");
	if (e && !strcmp(e, "ell")) return 0;
	static const int widths[] = { 2, 3, 4, 6, 8, 12, 16 };
	for (int v : widths) if (w <= v) return v;
	return 0;
}

// Dependencies at most this many level-order positions before the end of
// their row's level are read from the shared-memory ring, older ones from
// global memory.  FEMGPU_SWEEP_NEAR lowers the limit (1..SW_RING) so that
// small systems exercise the global-memory path too.
static int sweep_near_limit(void)
{
	const char *e = getenv("FEMGPU_SWEEP_NEAR");
	int v = e ? atoi(e) : SW_RING;
	return (v >= 1 && v <= SW_RING) ? v : SW_RING;
}

// Record-layout sweeps run as dataflow (k_sweep_df) unless
// FEMGPU_SWEEP_SYNC=barrier asks for one barrier per level (k_sweep_rec).
static bool sweep_dataflow(void)
{
	const char *e = getenv("FEMGPU_SWEEP_SYNC");
	return !(e && !strcmp(e, "barrier"));
}

// Chain-scan programs for the fused and FP32 sweeps (FEMGPU_SWEEP_CHAIN=0
// keeps the row-by-row programs for them too).
static bool sweep_chain(void)
{
	const char *e = getenv("FEMGPU_SWEEP_CHAIN");
	return !(e && !strcmp(e, "0"));
}

// Double-single chain sweeps for the fused FP64 (FGMRES) applications
// (FEMGPU_SWEEP_DS=0: FP64 chain sweeps).
static bool sweep_ds(void)
{
	const char *e = getenv("FEMGPU_SWEEP_DS");
	return !(e && !strcmp(e, "0"));
}

// Chunks a dataflow warp may run ahead of the slowest one: 8 times
// FEMGPU_SWEEP_SKEW (1..64; default 4, two turns of 16 warps).
static int sweep_look(void)
{
	const char *e = getenv("FEMGPU_SWEEP_SKEW");
	int v = e ? atoi(e) : 4;
	return 8 * ((v >= 1 && v <= 64) ? v : 4);
}

// Layout of a dataflow program whose chunks take `stage' bytes: warps (at most
// `most', fewer until two stages of each fit), stages a warp, ring (the wide one
// if it fits with all of `most'), lookahead X and the ring's reach in chunks.
// False when nothing fits.
struct DfFit { int ring, look, reach, warps, D; };
static bool df_stages(int ring, long long stage, long long tsize, int warps, int *D)
{
	const long long fixed = (al16(((long long)ring + 1) * tsize) + 2 * DF_BARS * 8 + 127) & ~127LL;
	*D = (int)std::min<long long>((SW_SMEM_CAP - fixed) / (warps * al16(stage)), std::min(DF_MAXD, DF_BARS / warps));
	return *D >= 2;
}
static bool df_fit(int most, long long stage, long long tsize, DfFit &f)
{
	f.ring = SW_RING_WIDE;
	f.warps = most;
	if (!df_stages(f.ring, stage, tsize, f.warps, &f.D)) {
		f.ring = SW_RING;
		while (f.warps >= 4 && !df_stages(f.ring, stage, tsize, f.warps, &f.D)) f.warps -= 4;
		if (f.warps < 4) return false;
	}
	const int R = f.ring / 32;
	f.look = std::min(sweep_look() * (f.ring / SW_RING), (R - 2 - f.warps) / 3);
	// a lowered reach (FEMGPU_SWEEP_NEAR): a dependency read back from global
	// memory must be more than a turn of all warps back
	f.reach = std::min(R - 2 * f.look - 2, std::max((sweep_near_limit() + 31) / 32, f.warps + 1));
	return true;
}

// One sweep program.  Forward (lower): L part, outputs to the backward
// sweep's padded level order (target = the U levels' ppos).  Backward: U part
// and pivots, outputs in natural order.
template <typename T, bool UPPER>
static int build_prog(const int *IA, const int *JA, int n, const HostLevels &H, const HostLevels *target,
                      const Blocks &B, const std::vector<int> &clev, fg_sweep &sw)
{
	const bool lower = !UPPER;
	const long long tsize = sizeof(T);
	int near_lim = sweep_near_limit();
	int nlev = H.nlev;
	// sub-blocks: (level, first row within the level, rows, width)
	struct Sub { int l, j0, c, w; };
	std::vector<Sub> subs;
	subs.reserve(nlev + 16);
	int wmax = 0, lmax = 1;
	for (int r = 0; r < n; r++) {
		int cnt = 0;
		for (int k = IA[r]; k < IA[r + 1]; k++)
			if ((lower ? JA[k] < r : JA[k] > r) && B.same(r, JA[k])) cnt++;
		wmax = std::max(wmax, cnt);
	}
	for (int l = 0; l < nlev; l++) lmax = std::max(lmax, H.start[l + 1] - H.start[l]);
	int rw = rec_width(wmax);                                         // 0: ELL sub-blocks
	const long long RB0 = rw ? rec_bytes(rw, UPPER, (int)tsize) : 0;
	DfFit fit = { SW_RING, 0, 0, 0, 0 };
	const int widest = std::min(lmax, 32);
	const bool df = rw && sweep_dataflow() && 
	                df_fit(df_warps(false, rw), DF_HDR + widest * RB0 + al16((long long)((widest + 3) & ~3) * tsize), tsize, fit);
	const int sub = df ? 32 : SW_SUB;
	for (int l = 0; l < nlev; l++) {
		int c = H.start[l + 1] - H.start[l];
		for (int j0 = 0; j0 < c; j0 += sub) {
			int cc = std::min(sub, c - j0), w = 0;
			for (int p = H.start[l] + j0; p < H.start[l] + j0 + cc; p++) {
				int r = H.rows[p], cnt = 0;
				for (int k = IA[r]; k < IA[r + 1]; k++)
					if ((lower ? JA[k] < r : JA[k] > r) && B.same(r, JA[k])) cnt++;
				w = std::max(w, cnt);
			}
			subs.push_back({ l, j0, cc, w });
		}
	}
	int nsb = (int)subs.size();
	int cmax = 1;
	for (const Sub &S : subs) cmax = std::max(cmax, S.c);
	if (rw && !df) {
		// wide records must still leave room for two stages of the widest sub-block
		const long long fixed = (al16((SW_RING + 1) * tsize) + SW_BAR_BYTES + 127) & ~127LL;
		const long long stage = 16 + (long long)cmax * RB0 + al16((long long)((cmax + 3) & ~3) * tsize);
		if (fixed + 2 * ((stage + 127) & ~127LL) > SW_SMEM_CAP) rw = 0;
	}
	const long long RB = rw ? RB0 : 0;
	const long long hdrb = 16;
	// dataflow: chunk of each level-order position, counted from its matrix block's first
	std::vector<int> chunk(df ? n : 0), lane(df ? n : 0), cfirst(df ? nsb : 0);
	if (df) {
		size_t b = 0;
		int first = 0;
		for (int i = 0; i < nsb; i++) {
			while (b + 1 < clev.size() && subs[i].l >= clev[b + 1]) { b++; first = i; }
			cfirst[i] = i - first;
			for (int j = 0; j < subs[i].c; j++) {
				chunk[H.start[subs[i].l] + subs[i].j0 + j] = i - first;
				lane[H.start[subs[i].l] + subs[i].j0 + j] = j;
			}
		}
	}
	std::vector<long long> off(nsb + 1, 0);
	std::vector<int> sb_in(nsb), sb_inb(nsb);
	long long maxblk = 0, bvo = 0, maxin = 0;
	for (int i = 0; i < nsb; i++) {
		int cp = (subs[i].c + 3) & ~3;
		long long bb = rw ? hdrb + (long long)subs[i].c * RB : blk_bytes<T, UPPER>(subs[i].w, cp);
		off[i + 1] = off[i] + bb;
		sb_in[i] = H.pstart[subs[i].l] + subs[i].j0;                 // j0 is a multiple of 4
		sb_inb[i] = (int)al16((long long)cp * tsize);
		maxblk = std::max(maxblk, bb + sb_inb[i]);
		bvo = std::max(bvo, bb);
		maxin = std::max(maxin, (long long)sb_inb[i]);
	}
	if (rw) maxblk = bvo + maxin;                                     // input slice at a fixed offset
	std::vector<unsigned char> prog((size_t)off[nsb] + 16, 0);
	std::vector<long long> val_off;
	std::vector<int> val_src;
	val_off.reserve((size_t)IA[n] + n);
	val_src.reserve((size_t)IA[n] + n);
	for (int i = 0; i < nsb; i++) {
		const Sub &S = subs[i];
		int l = S.l, c = S.c, w = S.w, cp = (c + 3) & ~3, start = H.start[l] + S.j0;
		int end = H.start[l + 1];
		int nsub = (H.start[l + 1] - H.start[l] + sub - 1) / sub;
		unsigned char *b = prog.data() + off[i];
		int hasfar = 0;
		auto near = [&](int p) { return df ? cfirst[i] - chunk[p] <= fit.reach : end - p <= near_lim; };
		auto ring_slot = [&](int p) {
			return (unsigned)(df ? (32 * chunk[p] + lane[p]) & (fit.ring - 1) : p & (SW_RING - 1));
		};
		// dataflow: the ring slot's byte offset, or the global position and the top bit
		auto code = [&](bool ring, unsigned at) {
			return (int)(df ? (ring ? at * (unsigned)tsize : SW_NEAR | at) : (ring ? SW_NEAR | at : at));
		};
		for (int j = 0; j < c; j++) {
			int r = H.rows[start + j];
			for (int q = IA[r]; q < IA[r + 1]; q++) {
				int col = JA[q];
				if ((lower ? col < r : col > r) && B.same(r, col) && !near(H.pos[col]))
					hasfar = df ? std::max(hasfar, chunk[H.pos[col]] + 1) : 1;
			}
		}
		if (rw) {
			const int hh[4] = { c, df ? 0 : nsub, df ? 0 : start, hasfar };
			memcpy(b, hh, sizeof hh);
			for (int j = 0; j < c; j++) {
				int *ri = (int *)(b + hdrb + (size_t)j * RB), r = H.rows[start + j], k = 0;
				long long vo = off[i] + hdrb + (long long)j * RB + rec_ib(rw);
				for (int q = 0; q < rw; q++) ri[q] = code(true, (unsigned)fit.ring);   // the zero slot
				ri[rw] = lower ? target->ppos[r] : r;
				for (int q = IA[r]; q < IA[r + 1]; q++) {
					int col = JA[q];
					if ((lower ? !(col < r) : !(col > r)) || !B.same(r, col)) continue;
					int p = H.pos[col];
					ri[k] = near(p) ? code(true, ring_slot(p)) : code(false, (unsigned)(lower ? target->ppos[col] : col));
					val_off.push_back(vo + k * tsize);
					val_src.push_back(q);
					k++;
				}
				for (; k < rw; k++) { val_off.push_back(vo + k * tsize); val_src.push_back(-1); }
				if (!lower) { val_off.push_back(vo + rw * tsize); val_src.push_back(-2 - r); }
			}
			continue;
		}
		LevHdr h = { c, w, start, cp, nsub, hasfar, (int)al16(SW_HDR + (long long)(w + 1) * cp * 4),
		             (int)blk_bytes<T, UPPER>(w, cp) };
		memcpy(b, &h, sizeof h);
		int *dep = (int *)(b + SW_HDR), *outp = dep + (size_t)w * cp;
		long long voff = al16(SW_HDR + (long long)(w + 1) * cp * 4);
		for (int k = 0; k < w * cp; k++) dep[k] = (int)(SW_NEAR | SW_RING);       // the zero slot
		for (int j = 0; j < c; j++) {
			int r = H.rows[start + j], k = 0;
			outp[j] = lower ? target->ppos[r] : r;
			for (int q = IA[r]; q < IA[r + 1]; q++) {
				int col = JA[q];
				if ((lower ? !(col < r) : !(col > r)) || !B.same(r, col)) continue;
				int p = H.pos[col];
				unsigned code = (end - p <= near_lim) ? (SW_NEAR | (unsigned)(p & (SW_RING - 1)))
				                                     : (unsigned)(lower ? target->ppos[col] : col);
				dep[(size_t)k * cp + j] = (int)code;
				val_off.push_back(off[i] + voff + ((long long)k * cp + j) * tsize);
				val_src.push_back(q);
				k++;
			}
			for (; k < w; k++) {
				val_off.push_back(off[i] + voff + ((long long)k * cp + j) * tsize);
				val_src.push_back(-1);
			}
			if (!lower) {
				val_off.push_back(off[i] + voff + ((long long)w * cp + j) * tsize);
				val_src.push_back(-2 - r);
			}
		}
	}
	// first sub-block of each matrix block (its first level's first sub-block)
	std::vector<int> csb(clev.size(), nsb);
	for (size_t b = 0, i = 0; b < clev.size(); b++) {
		while (i < (size_t)nsb && subs[i].l < clev[b]) i++;
		csb[b] = (int)i;
	}
	sw.nchunk = (int)clev.size() - 1;
	sw.rw = rw;
	sw.df = df;
	sw.ring = fit.ring;
	sw.look = fit.look;
	sw.warps = fit.warps;
	sw.bvo = (int)bvo;
	sw.cmax = cmax;
	sw.nlev = nlev;
	sw.nsb = nsb;
	sw.bytes = off[nsb];
	sw.maxblk = maxblk;
	sw.nval = (long long)val_off.size();
	sw.npad = H.pstart[nlev];
	int rc;
	FG_TRY(cudaMalloc((void **)&sw.prog, prog.size()));
	FG_TRY(cudaMemcpy(sw.prog, prog.data(), prog.size(), cudaMemcpyHostToDevice));
	if ((rc = up_vec(&sw.blk_off, off))) return rc;
	if ((rc = up_vec(&sw.sb_in, sb_in))) return rc;
	if ((rc = up_vec(&sw.sb_inb, sb_inb))) return rc;
	if ((rc = up_vec(&sw.rows, H.rows))) return rc;
	std::vector<int> ppos_by_pos(n);
	for (int p = 0; p < n; p++) ppos_by_pos[p] = H.ppos[H.rows[p]];
	if ((rc = up_vec(&sw.ppos, ppos_by_pos))) return rc;
	if ((rc = up_vec(&sw.val_off, val_off))) return rc;
	if ((rc = up_vec(&sw.val_src, val_src))) return rc;
	if ((rc = up_vec(&sw.chunk_sb, csb))) return rc;
	if ((rc = up_vec(&sw.chunk_lev, clev))) return rc;
	return 0;
}

// ------------------------------------------- host: chain-scan programs
// Segments of one chain-scan sweep: rows in sweep order
// (forward ascending, backward descending) within their matrix block; a row
// joins the current segment when it depends on its sweep predecessor, the
// segment has fewer than 32 rows and the row's other dependencies are all on
// earlier levels than the segment's -- otherwise it starts a new segment,
// whose level is one past its dependencies' (the predecessor among them).
// This cut keeps segments of consecutive fronts aligned, so a block's depth
// is about its fronts plus a front's chunk count, not fronts plus front width.
// Each level's segments are packed, in order, into 32-slot chunks.
struct ChainLevels {
	int nlev = 0, nslot = 0, maxw = 0;
	std::vector<int> lstart;   // [nlev+1] first slot of each level (multiples of 32)
	std::vector<int> slot_row; // [nslot] row in each slot (-1 padding)
	std::vector<int> slot_pred; // [nslot] CSR position of the chain coefficient (-1: segment start, padding)
	std::vector<int> slot;     // [n] slot of each row
	std::vector<int> clev;     // [P+1] first level of each matrix block
	int rowlev_max = 0;        // deepest block in row levels (for the choice of program)
};

static ChainLevels host_chain_levels(const int *IA, const int *JA, int n, bool lower, const Blocks &B)
{
	ChainLevels H;
	const int P = B.P ? B.P : 1;
	std::vector<int> seg_of(n), seg_lev, seg_blk, seg_first, seg_pred_pos(n, -1), rowlev(n, 0);
	std::vector<int> bl(P, 0), blrow(P, 0);
	int cur = -1, run = 0;
	for (int s = 0; s < n; s++) {
		const int i = lower ? s : n - 1 - s, pred = lower ? i - 1 : i + 1, b = B.of(i);
		int elev = 0, ppos = -1, rl = 0, nd = 0;
		for (int k = IA[i]; k < IA[i + 1]; k++) {
			const int c = JA[k];
			if (!(lower ? c < i : c > i) || !B.same(i, c)) continue;
			rl = std::max(rl, rowlev[c] + 1);
			if (c == pred) { ppos = k; continue; }
			elev = std::max(elev, seg_lev[seg_of[c]] + 1);
			nd++;
		}
		rowlev[i] = rl;
		blrow[b] = std::max(blrow[b], rl + 1);
		bool chain = ppos >= 0 && cur >= 0 && seg_blk[cur] == b && run < 32 && elev <= seg_lev[cur] &&
		             seg_of[pred] == cur;
		if (chain) {
			seg_of[i] = cur;
			seg_pred_pos[i] = ppos;
			run++;
		} else {
			if (ppos >= 0) { elev = std::max(elev, seg_lev[seg_of[pred]] + 1); nd++; }
			seg_lev.push_back(elev);
			seg_blk.push_back(b);
			seg_first.push_back(i);
			cur = (int)seg_lev.size() - 1;
			seg_of[i] = cur;
			run = 1;
			bl[b] = std::max(bl[b], elev + 1);
		}
		H.maxw = std::max(H.maxw, nd);
	}
	for (int b = 0; b < P; b++) H.rowlev_max = std::max(H.rowlev_max, blrow[b]);
	std::vector<int> boff(P + 1, 0);
	for (int b = 0; b < P; b++) boff[b + 1] = boff[b] + bl[b];
	H.clev = boff;
	H.nlev = boff[P];
	const int nseg = (int)seg_lev.size();
	// segments by global level, in creation order; their rows in sweep order
	std::vector<int> lcount(H.nlev + 1, 0), seg_len(nseg, 0), order(nseg);
	for (int g = 0; g < nseg; g++) lcount[seg_lev[g] + boff[seg_blk[g]] + 1]++;
	for (int l = 0; l < H.nlev; l++) lcount[l + 1] += lcount[l];
	{
		std::vector<int> fill(lcount.begin(), lcount.end() - 1);
		for (int g = 0; g < nseg; g++) order[fill[seg_lev[g] + boff[seg_blk[g]]]++] = g;
	}
	for (int i = 0; i < n; i++) seg_len[seg_of[i]]++;
	std::vector<int> seg_slot(nseg);
	H.lstart.assign(H.nlev + 1, 0);
	int slot = 0;
	for (int l = 0; l < H.nlev; l++) {
		H.lstart[l] = slot;
		int used = 32;                                    // lanes used in the current chunk
		for (int q = lcount[l]; q < lcount[l + 1]; q++) {
			const int g = order[q];
			if (used + seg_len[g] > 32) { if (used < 32) slot += 32 - used; used = 0; }
			seg_slot[g] = slot;
			slot += seg_len[g];
			used += seg_len[g];
		}
		if (used < 32) slot += 32 - used;
	}
	H.lstart[H.nlev] = slot;
	H.nslot = slot;
	H.slot_row.assign(slot, -1);
	H.slot_pred.assign(slot, -1);
	H.slot.assign(n, 0);
	std::vector<int> next(seg_slot);
	for (int s = 0; s < n; s++) {
		const int i = lower ? s : n - 1 - s, g = seg_of[i], sl = next[g]++;
		H.slot[i] = sl;
		H.slot_row[sl] = i;
		H.slot_pred[sl] = seg_pred_pos[i];
	}
	return H;
}

// The chain-scan program of one sweep: chunks of 32 slots of one level, the
// dataflow header, one record per slot (the lanes' 16-byte words side by side),
// the input slice at a fixed stage offset.  Forward: L part, outputs to the
// backward program's slots; backward: U part and pivots, outputs in natural
// order.  Returns FEMGPU_E_MESH when its stages do not fit (the caller keeps
// the row-by-row programs then).
template <typename T, bool UPPER>
static int build_prog_chain(const int *IA, const int *JA, int n, const ChainLevels &H, const ChainLevels *target,
                            const Blocks &B, fg_sweep &sw)
{
	const bool lower = !UPPER;
	const long long tsize = sizeof(T);
	const int nlev = H.nlev;
	int rw = rec_width(std::max(H.maxw, 1));
	if (!rw) return FEMGPU_E_MESH;
	const long long IBy = rec_ib(rw), RB = IBy + rec_vb_cs(rw, UPPER, (int)tsize);
	// int q and value v of a chunk's slot j, from the chunk's start
	auto iat = [](int q, int j) { return (long long)DF_HDR + q / 4 * 512 + 16 * j + q % 4 * 4; };
	auto vat = [&](int v, int j) {
		const int per = 16 / (int)tsize;
		return DF_HDR + 32 * IBy + v / per * 512 + 16 * j + v % per * tsize;
	};
	struct Sub { int l, j0, c; };
	std::vector<Sub> subs;
	for (int l = 0; l < nlev; l++) {
		const int c = H.lstart[l + 1] - H.lstart[l];
		for (int j0 = 0; j0 < c; j0 += 32) subs.push_back({ l, j0, 32 });
	}
	const int nsb = (int)subs.size();
	const int cmax = 32;
	DfFit fit;
	if (!df_fit(df_warps(true, rw), DF_HDR + cmax * RB + cmax * tsize, tsize, fit)) return FEMGPU_E_MESH;
	std::vector<int> cfirst(nsb);                        // chunks before each chunk in its matrix block
	for (size_t i = 0, bk = 0, first = 0; i < (size_t)nsb; i++) {
		while (bk + 1 < H.clev.size() && subs[i].l >= H.clev[bk + 1]) { bk++; first = i; }
		cfirst[i] = (int)(i - first);
	}
	std::vector<long long> off(nsb + 1, 0);
	long long bvo = 0;
	const long long inb = al16(cmax * tsize);            // bytes of a chunk's input slice
	for (int i = 0; i < nsb; i++) {
		const long long bb = DF_HDR + (long long)subs[i].c * RB;
		off[i + 1] = off[i] + bb;
		bvo = std::max(bvo, bb);
	}
	std::vector<unsigned char> prog((size_t)off[nsb] + 16, 0);
	std::vector<long long> val_off, cs_voff(H.nslot, -1);
	std::vector<int> val_src, cs_src(H.nslot, -1), cs_row(H.nslot, 0);
	val_off.reserve((size_t)H.nslot * (rw + 1));
	val_src.reserve((size_t)H.nslot * (rw + 1));
	for (int i = 0; i < nsb; i++) {
		const Sub &S = subs[i];
		const int l = S.l, c = S.c, start = H.lstart[l] + S.j0;
		unsigned char *b = prog.data() + off[i];
		int hasfar = 0;
		for (int j = 0; j < c; j++) {
			const int r = H.slot_row[start + j];
			if (r < 0) continue;
			for (int q = IA[r]; q < IA[r + 1]; q++) {
				const int col = JA[q];
				if ((lower ? col < r : col > r) && B.same(r, col) && q != H.slot_pred[start + j] &&
				    i - H.slot[col] / 32 > fit.reach) hasfar = std::max(hasfar, cfirst[H.slot[col] / 32] + 1);
			}
		}
		const int hh[4] = { c, 0, 0, hasfar };
		memcpy(b, hh, sizeof hh);
		for (int j = 0; j < c; j++) {
			const int r = H.slot_row[start + j];
			int k = 0;
			auto ri = [&](int q) -> int & { return *(int *)(b + iat(q, j)); };
			cs_voff[start + j] = off[i] + vat(0, j);
			for (int q = 0; q < rw; q++) ri(q) = fit.ring * (int)tsize;        // the zero slot
			if (r < 0) {                                                       // padding (multipliers zero)
				ri(rw) = -1;
				for (int q = 0; q < rw + (UPPER ? 1 : 0); q++) { val_off.push_back(off[i] + vat(q, j)); val_src.push_back(-1); }
				continue;
			}
			ri(rw) = lower ? target->slot[r] : r;
			for (int q = IA[r]; q < IA[r + 1]; q++) {
				const int col = JA[q];
				if ((lower ? !(col < r) : !(col > r)) || !B.same(r, col) || q == H.slot_pred[start + j]) continue;
				const int p = H.slot[col];
				ri(k) = (int)(i - p / 32 <= fit.reach
				                  ? (unsigned)((32 * cfirst[p / 32] + p % 32) & (fit.ring - 1)) * (unsigned)tsize
				                  : SW_NEAR | (unsigned)(lower ? target->slot[col] : col));
				val_off.push_back(off[i] + vat(k, j));
				val_src.push_back(q);
				k++;
			}
			for (; k < rw; k++) { val_off.push_back(off[i] + vat(k, j)); val_src.push_back(-1); }
			if (!lower) { val_off.push_back(off[i] + vat(rw, j)); val_src.push_back(-2 - r); }
			cs_src[start + j] = H.slot_pred[start + j];
			cs_row[start + j] = r;
		}
	}
	// every index the kernel will follow stays inside its array: dependency
	// codes (ring slots or output positions), output positions, input slices
	{
		const long long nout = lower ? target->nslot : n;
		for (int i = 0; i < nsb; i++) {
			const unsigned char *b = prog.data() + off[i];
			const int c = subs[i].c;
			const int at = H.lstart[subs[i].l] + subs[i].j0;          // its input slice
			if (at != 32 * i || c != 32 || (long long)at + c > H.nslot) return FEMGPU_E_MESH;
			for (int j = 0; j < c; j++) {
				auto ri = [&](int q) { return *(const int *)(b + iat(q, j)); };
				for (int q = 0; q < rw; q++) {
					const unsigned code = (unsigned)ri(q);
					if (code & SW_NEAR) { if ((long long)(code & ~SW_NEAR) >= nout) return FEMGPU_E_MESH; }
					else if (code > (unsigned)(fit.ring * tsize)) return FEMGPU_E_MESH;
				}
				if (ri(rw) < -1 || ri(rw) >= nout) return FEMGPU_E_MESH;
			}
		}
		for (size_t q = 0; q < cs_voff.size(); q++)
			if (cs_voff[q] < 0 || cs_voff[q] - vat(0, 0) + vat(rw + (UPPER ? 1 : 0) + 4, 0) + tsize > off[nsb]) return FEMGPU_E_MESH;
		for (size_t q = 0; q < val_off.size(); q++)
			if (val_off[q] < 0 || val_off[q] + tsize > off[nsb]) return FEMGPU_E_MESH;
	}
	std::vector<int> csb(H.clev.size(), nsb);
	for (size_t bk = 0, i = 0; bk < H.clev.size(); bk++) {
		while (i < (size_t)nsb && subs[i].l < H.clev[bk]) i++;
		csb[bk] = (int)i;
	}
	// real rows in slot order (the gather of the sweep input)
	std::vector<int> rows, ppos;
	rows.reserve(n);
	ppos.reserve(n);
	for (int q = 0; q < H.nslot; q++)
		if (H.slot_row[q] >= 0) { rows.push_back(H.slot_row[q]); ppos.push_back(q); }
	sw.nchunk = (int)H.clev.size() - 1;
	sw.rw = rw;
	sw.df = 1;
	sw.cs = 1;
	sw.ring = fit.ring;
	sw.look = fit.look;
	sw.warps = fit.warps;
	sw.bvo = (int)bvo;
	sw.cmax = cmax;
	sw.nlev = nlev;
	sw.nsb = nsb;
	sw.bytes = off[nsb];
	sw.maxblk = bvo + inb;
	sw.nval = (long long)val_off.size();
	sw.npad = H.nslot;
	sw.nslot = H.nslot;
	int rc;
	FG_TRY(cudaMalloc((void **)&sw.prog, prog.size()));
	FG_TRY(cudaMemcpy(sw.prog, prog.data(), prog.size(), cudaMemcpyHostToDevice));
	if ((rc = up_vec(&sw.rows, rows))) return rc;
	if ((rc = up_vec(&sw.ppos, ppos))) return rc;
	if ((rc = up_vec(&sw.val_off, val_off))) return rc;
	if ((rc = up_vec(&sw.val_src, val_src))) return rc;
	if ((rc = up_vec(&sw.chunk_sb, csb))) return rc;
	if ((rc = up_vec(&sw.cs_voff, cs_voff))) return rc;
	if ((rc = up_vec(&sw.cs_src, cs_src))) return rc;
	if ((rc = up_vec(&sw.cs_row, cs_row))) return rc;
	return 0;
}

// Elimination program of every row for k_ilu0_factor_df: the sequence of
// updates of ILUp_precond_setup.c:119-139, resolved against the pattern once
// (couplings between matrix blocks dropped).  Slots run over the levels of all
// matrix blocks side by side (level l of every block, then level l + 1), so the
// blocks advance together, each level padded to whole warps.
static int build_factor_prog(const int *IA, const int *JA, int n, const HostLevels &Lo, const Blocks &B,
                             const std::vector<int> &clev, fg_ilu_sweeps &S)
{
	int longest = 0, depth = 0;
	for (int r = 0; r < n; r++) longest = std::max(longest, IA[r + 1] - IA[r]);
	if (longest > FAC_CAP) return FEMGPU_E_MESH;
	const int L = longest <= 8 ? 8 : (longest <= 16 ? 16 : 32), R = 32 / L, P = (int)clev.size() - 1;
	for (int b = 0; b < P; b++) depth = std::max(depth, clev[b + 1] - clev[b]);
	std::vector<int> slot;                               // row of each slot, -1 padding
	slot.reserve((size_t)n + (size_t)depth * (R - 1));
	S.fac_wide = 0;
	for (int l = 0; l < depth; l++) {
		const size_t s0 = slot.size();
		for (int b = 0; b < P; b++)
			if (clev[b] + l < clev[b + 1])
				slot.insert(slot.end(), Lo.rows.begin() + Lo.start[clev[b] + l],
				            Lo.rows.begin() + Lo.start[clev[b] + l + 1]);
		while (slot.size() % R) slot.push_back(-1);
		S.fac_wide = std::max(S.fac_wide, (int)(slot.size() - s0));
	}
	const size_t ns = slot.size();
	std::vector<int> head(4 * ns, 0), grp(2 * ns * L, 0);
	std::vector<unsigned char> pos(ns * L * L, FAC_NONE);
	for (size_t s = 0; s < ns; s++) {
		const int r = slot[s];
		head[4 * s + 2] = r;
		if (r < 0) continue;
		const int rb = IA[r], len = IA[r + 1] - rb;
		int dpos = -1, ng = 0;
		for (int q = 0; q < len; q++) if (JA[rb + q] == r) dpos = q;
		if (dpos < 0) return FEMGPU_E_ZERO_PIVOT;        // no diagonal entry
		unsigned char *ps = &pos[s * L * L];              // [lane][group]
		for (int q = 0; q < len && JA[rb + q] < r; q++) {
			const int jrow = JA[rb + q];
			if (!B.same(r, jrow)) continue;
			grp[2 * (s * L + ng)] = jrow;
			grp[2 * (s * L + ng) + 1] = IA[jrow];
			ps[q * L + ng] = FAC_MULT;
			for (int k = IA[jrow]; k < IA[jrow + 1]; k++) {
				const int col = JA[k];
				if (col <= jrow || !B.same(r, col)) continue;
				for (int m = 0; m < len; m++)
					if (JA[rb + m] == col) { ps[m * L + ng] = (unsigned char)(k - IA[jrow]); break; }
			}
			ng++;
		}
		head[4 * s] = rb;
		head[4 * s + 1] = len | (dpos << 8) | (ng << 16);
	}
	S.fac_lanes = L;
	S.fac_nslot = (int)ns;
	int rc;
	if ((rc = up_vec(&S.fac_head, head))) return rc;
	if ((rc = up_vec(&S.fac_grp, grp))) return rc;
	if ((rc = up_vec(&S.fac_pos, pos))) return rc;
	FG_TRY(cudaMalloc(&S.fac_ticket, sizeof(fg_ticket)));
	return 0;
}

#define SW_SET(T, U, CW, F) FG_TRY(cudaFuncSetAttribute(k_sweep<T, U, CW, F>, \
	cudaFuncAttributeMaxDynamicSharedMemorySize, SW_SMEM_CAP))
#define SW_SET_CW(CW) SW_SET(double, false, CW, false); SW_SET(double, true, CW, false); \
	SW_SET(double, false, CW, true); SW_SET(double, true, CW, true); \
	SW_SET(float, false, CW, false); SW_SET(float, true, CW, false)
#define SR_SET(T, U, F, W) FG_TRY(cudaFuncSetAttribute(k_sweep_rec<T, U, F, W>, \
	cudaFuncAttributeMaxDynamicSharedMemorySize, SW_SMEM_CAP))
#define SD_SET(T, U, F, C, W) FG_TRY(cudaFuncSetAttribute(k_sweep_df<T, U, F, C, W>, \
	cudaFuncAttributeMaxDynamicSharedMemorySize, SW_SMEM_CAP))
#define SF_SET(T, F, C, W) FG_TRY(cudaFuncSetAttribute(k_sweep_fb<T, F, C, W>, \
	cudaFuncAttributeMaxDynamicSharedMemorySize, SW_SMEM_CAP))
#define SD_BOTH(T, F, C, W) SD_SET(T, false, F, C, W); SD_SET(T, true, F, C, W); SF_SET(T, F, C, W)
#define SR_SET_W(W) SD_BOTH(double, true, true, W); SD_BOTH(float, true, true, W); SD_BOTH(dsf, true, true, W); \
	SD_BOTH(double, false, false, W); SD_BOTH(double, true, false, W); SD_BOTH(float, false, false, W); \
	SR_SET(double, false, false, W); SR_SET(double, true, false, W); \
	SR_SET(double, false, true, W); SR_SET(double, true, true, W); \
	SR_SET(float, false, false, W); SR_SET(float, true, false, W)
static int sweep_attrs(void)
{
	SW_SET_CW(4);
	SW_SET_CW(8);
	SW_SET_CW(16);
	SR_SET_W(2);
	SR_SET_W(3);
	SR_SET_W(4);
	SR_SET_W(6);
	SR_SET_W(8);
	SR_SET_W(12);
	SR_SET_W(16);
	return 0;
}

// Consumer warps per sweep (4, 8 or 16; FEMGPU_SWEEP_WARPS overrides).
static int sweep_cw(void)
{
	static int cw = 0;
	if (!cw) {
		const char *e = getenv("FEMGPU_SWEEP_WARPS");
		int v = e ? atoi(e) : 16;
		cw = (v == 4 || v == 8 || v == 16) ? v : 16;
	}
	return cw;
}

// fma: fused multiply-subtract in the FP64 sweeps (the FGMRES solves); the
// separately rounded form reproduces the reference bit for bit.
#define DF_CASES(RUN) switch (rw) { case 2: RUN(2); break; case 3: RUN(3); break; case 4: RUN(4); break; \
	case 6: RUN(6); break; case 8: RUN(8); break; case 12: RUN(12); break; default: RUN(16); break; }
template <typename T, bool UPPER, bool FMA, bool CS>
static void launch_df(const SweepArgs &a, int rw, int grid, int warps, int bytes, cudaStream_t s, const T *in, T *out)
{
#define RUN(W) k_sweep_df<T, UPPER, FMA, CS, W><<<grid, 32 * warps, bytes, s>>>(a, in, out)
	DF_CASES(RUN)
#undef RUN
}
template <typename T, bool FMA, bool CS>
static void launch_fb(const SweepArgs &al, const SweepArgs &au, int rw, int grid, int warps, int bytes, cudaStream_t s,
                      const T *in, T *y, T *out)
{
#define RUN(W) k_sweep_fb<T, FMA, CS, W><<<grid, 32 * warps, bytes, s>>>(al, au, in, y, out)
	DF_CASES(RUN)
#undef RUN
}

template <typename T, bool UPPER, bool FMA>
static void launch_rec(const SweepArgs &a, int rw, int grid, int bytes, cudaStream_t s, const T *in, T *out)
{
	const int nt = (SW2_CW + 1) * 32;
	switch (rw) {
	case 2: k_sweep_rec<T, UPPER, FMA, 2><<<grid, nt, bytes, s>>>(a, in, out); break;
	case 3: k_sweep_rec<T, UPPER, FMA, 3><<<grid, nt, bytes, s>>>(a, in, out); break;
	case 4: k_sweep_rec<T, UPPER, FMA, 4><<<grid, nt, bytes, s>>>(a, in, out); break;
	case 6: k_sweep_rec<T, UPPER, FMA, 6><<<grid, nt, bytes, s>>>(a, in, out); break;
	case 8: k_sweep_rec<T, UPPER, FMA, 8><<<grid, nt, bytes, s>>>(a, in, out); break;
	case 12: k_sweep_rec<T, UPPER, FMA, 12><<<grid, nt, bytes, s>>>(a, in, out); break;
	default: k_sweep_rec<T, UPPER, FMA, 16><<<grid, nt, bytes, s>>>(a, in, out); break;
	}
}

template <typename T, bool UPPER>
static void launch_sweep(const SweepArgs &a, int rw, int grid, int bytes, cudaStream_t s, const T *in, T *out, bool fma)
{
	if (rw) {
		if (fma && sizeof(T) == 8) launch_rec<T, UPPER, true>(a, rw, grid, bytes, s, in, out);
		else launch_rec<T, UPPER, false>(a, rw, grid, bytes, s, in, out);
		return;
	}
	int cw = sweep_cw();
	if (fma && sizeof(T) == 8) {
		if (cw == 4) k_sweep<T, UPPER, 4, true><<<grid, 160, bytes, s>>>(a, in, out);
		else if (cw == 8) k_sweep<T, UPPER, 8, true><<<grid, 288, bytes, s>>>(a, in, out);
		else k_sweep<T, UPPER, 16, true><<<grid, 544, bytes, s>>>(a, in, out);
	} else {
		if (cw == 4) k_sweep<T, UPPER, 4, false><<<grid, 160, bytes, s>>>(a, in, out);
		else if (cw == 8) k_sweep<T, UPPER, 8, false><<<grid, 288, bytes, s>>>(a, in, out);
		else k_sweep<T, UPPER, 16, false><<<grid, 544, bytes, s>>>(a, in, out);
	}
}

static int sweep_smem(const fg_sweep &sw, size_t tsize, int *D, int *stage_bytes, int warps = 0)
{
	if (sw.df) {
		const int w = warps ? warps : sw.warps;
		*stage_bytes = (int)al16(sw.maxblk);
		if (!df_stages(sw.ring, sw.maxblk, (long long)tsize, w, D)) return FEMGPU_E_MESH;
		return (int)((al16((sw.ring + 1LL) * (long long)tsize) + 2 * DF_BARS * 8 + 127) & ~127LL) + w * *D * *stage_bytes;
	}
	size_t fixed = ((al16((SW_RING + 1) * tsize) + SW_BAR_BYTES + 127) & ~(size_t)127);
	size_t sb = (size_t)((sw.maxblk + 127) & ~127LL);
	if (fixed + 2 * sb > SW_SMEM_CAP) return FEMGPU_E_MESH;   // a sub-block too wide to stage
	int d = (int)((SW_SMEM_CAP - fixed) / sb);
	if (d > SW_MAXD) d = SW_MAXD;
	*D = d;
	*stage_bytes = (int)sb;
	return (int)(fixed + (size_t)d * sb);
}

// Host only (no device call): the block ILU(0) cut of a CSR pattern, as
// fg_ilu_prepare computes it.  first receives R + 1 row boundaries, R =
// max(min(P, n), 1); cap is the room in first.  The pattern is checked first
// (IA[0] == 0, IA non-decreasing, every column in 0..n-1, columns ascending in
// each row): the cut's level scan indexes by column and stops at the first
// column at or past the row.
extern "C" int femgpu_ilu_block_cut(int n, const int *IA, const int *JA, int P, int *first, int cap)
{
	if (n <= 0 || !IA || !JA || !first) return FEMGPU_E_ARG;
	const int R = std::max(std::min(P, n), 1);
	if (cap < R + 1) return FEMGPU_E_ARG;
	if (IA[0] != 0) return FEMGPU_E_ARG;
	for (int i = 0; i < n; i++) {
		if (IA[i + 1] < IA[i]) return FEMGPU_E_ARG;
		for (int k = IA[i]; k < IA[i + 1]; k++) {
			if (JA[k] < 0 || JA[k] >= n) return FEMGPU_E_ARG;
			if (k > IA[i] && JA[k] <= JA[k - 1]) return FEMGPU_E_ARG;
		}
	}
	std::vector<int> f;
	(void)make_blocks(IA, JA, n, P, &f);
	if ((int)f.size() > cap) return FEMGPU_E_ARG;
	memcpy(first, f.data(), sizeof(int) * f.size());
	return (int)f.size() - 1;
}

// Host only (no device call): the chain-scan segmentation of one ILU(0)
// sweep of a CSR pattern with P blocks, as fg_ilu_prepare computes it.
extern "C" int femgpu_ilu_chain_segments(int n, const int *IA, const int *JA, int P, int lower, int *info,
                                         int *slot_row, int *slot_pred, int *lstart, int cap_slots, int cap_levels)
{
	if (n <= 0 || !IA || !JA || !info) return FEMGPU_E_ARG;
	if (IA[0] != 0) return FEMGPU_E_ARG;
	for (int i = 0; i < n; i++) {
		if (IA[i + 1] < IA[i]) return FEMGPU_E_ARG;
		for (int k = IA[i]; k < IA[i + 1]; k++)
			if (JA[k] < 0 || JA[k] >= n || (k > IA[i] && JA[k] <= JA[k - 1])) return FEMGPU_E_ARG;
	}
	Blocks B = make_blocks(IA, JA, n, P, nullptr);
	ChainLevels H = host_chain_levels(IA, JA, n, lower != 0, B);
	int deep = 0;
	for (size_t b = 0; b + 1 < H.clev.size(); b++) deep = std::max(deep, H.clev[b + 1] - H.clev[b]);
	info[0] = H.nlev;
	info[1] = deep;
	info[2] = H.rowlev_max;
	info[3] = H.maxw;
	if (slot_row || slot_pred || lstart) {
		if (cap_slots < H.nslot || cap_levels < H.nlev + 1) return FEMGPU_E_ARG;
		if (slot_row) memcpy(slot_row, H.slot_row.data(), sizeof(int) * H.nslot);
		if (slot_pred) memcpy(slot_pred, H.slot_pred.data(), sizeof(int) * H.nslot);
		if (lstart) memcpy(lstart, H.lstart.data(), sizeof(int) * (H.nlev + 1));
	}
	return H.nslot;
}

extern "C" int fg_ilu_prepare(femgpu_transport *t, const int *hIA, const int *hJA)
{
	int n = t->neq, rc, D, sb;
	fg_ilu_sweeps &S = t->sweeps;
	std::vector<int> first;
	Blocks B = make_blocks(hIA, hJA, n, t->o.ilu_blocks, &first);
	free(S.block_first);
	S.block_first = (int *)malloc(sizeof(int) * first.size());
	if (!S.block_first) return FEMGPU_E_NOMEM;
	memcpy(S.block_first, first.data(), sizeof(int) * first.size());
	S.nblocks = (int)first.size() - 1;
	std::vector<int> clo, cup;
	HostLevels Lo = host_levels(hIA, hJA, n, true, B, &clo), Up = host_levels(hIA, hJA, n, false, B, &cup);
	if ((rc = build_prog<double, true>(hIA, hJA, n, Up, nullptr, B, cup, S.up64))) return rc;
	if ((rc = build_prog<double, false>(hIA, hJA, n, Lo, &Up, B, clo, S.lo64))) return rc;
	if ((rc = build_prog<float, true>(hIA, hJA, n, Up, nullptr, B, cup, S.up32))) return rc;
	if ((rc = build_prog<float, false>(hIA, hJA, n, Lo, &Up, B, clo, S.lo32))) return rc;
	if ((rc = build_factor_prog(hIA, hJA, n, Lo, B, clo, S))) return rc;
	S.chain = 0;
	S.ds = 0;
	size_t nb = (size_t)std::max(Lo.pstart[Lo.nlev], Up.pstart[Up.nlev]) + 64;
	if (sweep_chain()) {
		ChainLevels CL = host_chain_levels(hIA, hJA, n, true, B), CU = host_chain_levels(hIA, hJA, n, false, B);
		int deepL = 0, deepU = 0;
		for (size_t b = 0; b + 1 < CL.clev.size(); b++) deepL = std::max(deepL, CL.clev[b + 1] - CL.clev[b]);
		for (size_t b = 0; b + 1 < CU.clev.size(); b++) deepU = std::max(deepU, CU.clev[b + 1] - CU.clev[b]);
		// worth it only when the segments remove most of the levels
		if (4 * (deepL + deepU) <= 3 * (CL.rowlev_max + CU.rowlev_max)) {
			int r1 = build_prog_chain<double, true>(hIA, hJA, n, CU, nullptr, B, S.up64c);
			int r2 = r1 ? r1 : build_prog_chain<double, false>(hIA, hJA, n, CL, &CU, B, S.lo64c);
			int r3 = r2 ? r2 : build_prog_chain<float, true>(hIA, hJA, n, CU, nullptr, B, S.up32c);
			int r4 = r3 ? r3 : build_prog_chain<float, false>(hIA, hJA, n, CL, &CU, B, S.lo32c);
			if (r4 && r4 != FEMGPU_E_MESH) return r4;
			S.chain = r4 == 0;
			if (S.chain) {
				nb = std::max(nb, (size_t)std::max(CL.nslot, CU.nslot) + 64);
				const fg_sweep *cs[4] = { &S.lo64c, &S.up64c, &S.lo32c, &S.up32c };
				for (int i = 0; i < 4; i++) {
					rc = sweep_smem(*cs[i], i < 2 ? sizeof(double) : sizeof(float), &D, &sb);
					if (rc < 0) { S.chain = 0; break; }
				}
			}
			if (S.chain && sweep_ds()) {
				// the FP64 programs' bytes (codes and offsets are the same;
				// the refresh rewrites the values as double-single)
				const size_t bl = (size_t)S.lo64c.bytes + 16, bu = (size_t)S.up64c.bytes + 16;
				FG_TRY(cudaMalloc((void **)&S.prog_lo_ds, bl));
				FG_TRY(cudaMalloc((void **)&S.prog_up_ds, bu));
				FG_TRY(cudaMemcpy(S.prog_lo_ds, S.lo64c.prog, bl, cudaMemcpyDeviceToDevice));
				FG_TRY(cudaMemcpy(S.prog_up_ds, S.up64c.prog, bu, cudaMemcpyDeviceToDevice));
				FG_TRY(cudaMalloc((void **)&S.dpos, sizeof(int) * (size_t)n));
				k_inv_gather<<<fg_grid(n), FG_TPB, 0, t->stream>>>(S.lo64c.rows, S.lo64c.ppos, n, S.dpos);
				FG_TRY(cudaGetLastError());
				S.ds = 1;
			}
		}
	}
	FG_TRY(cudaMalloc((void **)&S.bl64, sizeof(double) * nb));
	FG_TRY(cudaMalloc((void **)&S.y64, sizeof(double) * nb));
	FG_TRY(cudaMalloc((void **)&S.bl32, sizeof(float) * nb));
	FG_TRY(cudaMalloc((void **)&S.y32, sizeof(float) * nb));
	FG_TRY(cudaMemset(S.bl64, 0, sizeof(double) * nb));
	FG_TRY(cudaMemset(S.y64, 0, sizeof(double) * nb));
	if (S.ds) {
		FG_TRY(cudaMalloc((void **)&S.o64, sizeof(double) * nb));
		FG_TRY(cudaMemset(S.o64, 0, sizeof(double) * nb));
	}
	FG_TRY(cudaMemset(S.bl32, 0, sizeof(float) * nb));
	FG_TRY(cudaMemset(S.y32, 0, sizeof(float) * nb));
	FG_TRY(cudaMalloc((void **)&S.dpos64, sizeof(int) * (size_t)std::max(n, 1)));
	k_inv_gather<<<fg_grid(n), FG_TPB, 0, t->stream>>>(S.lo64.rows, S.lo64.ppos, n, S.dpos64);
	FG_TRY(cudaGetLastError());
	const fg_sweep *all[4] = { &S.lo64, &S.up64, &S.lo32, &S.up32 };
	for (int i = 0; i < 4; i++) {
		rc = sweep_smem(*all[i], i < 2 ? sizeof(double) : sizeof(float), &D, &sb);
		if (rc < 0) return rc;
	}
	return sweep_attrs();
}

// ILU(p): the matrix's values onto the filled pattern (fill entries zero).
__global__ void k_fill_scatter(const double *__restrict__ A, const int *__restrict__ map, int nnz, double *fA)
{
	for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += gridDim.x * blockDim.x) fA[map[k]] = A[k];
}

extern "C" int fg_ilu0_factor(femgpu_transport *t)
{
	cudaStream_t s = t->stream;
	fg_ilu_sweeps &S = t->sweeps;
	const double *A = t->A;
	if (S.fill) {
		FG_TRY(cudaMemsetAsync(S.fA, 0, sizeof(double) * ((size_t)S.fnnz + 1), s));
		k_fill_scatter<<<fg_grid(t->nnz), FG_TPB, 0, s>>>(t->A, S.fmap, t->nnz, S.fA);
		A = S.fA;
	}
	// enough warps for FAC_AHEAD levels: a warp takes its rows, their program
	// and matrix values while the levels before are computed
	const int R = 32 / S.fac_lanes, per = FAC_TPB / 32 * R;
	const long long want = ((long long)FAC_AHEAD * S.fac_wide + per - 1) / per;
	const int grid = (int)std::min<long long>(std::max<long long>(want, 1), 4 * FG_SMS);
	fg_ticket *tk = (fg_ticket *)S.fac_ticket;
	k_ilu0_factor_init<<<fg_grid(t->ilu.nnz), FG_TPB, 0, s>>>(t->ilu.LU, t->ilu.nnz, t->ilu.Dinv, t->neq, tk);
#define FAC_RUN(L) k_ilu0_factor_df<L><<<grid, FAC_TPB, 0, s>>>(A, (const int4 *)S.fac_head, (const int2 *)S.fac_grp, \
	(const uint2 *)S.fac_pos, S.fac_nslot, t->ilu.LU, t->ilu.Dinv, tk, &t->st->err, fg_poll0(t->sweep_wait1))
	if (S.fac_lanes == 8) FAC_RUN(8);
	else if (S.fac_lanes == 16) FAC_RUN(16);
	else FAC_RUN(32);
#undef FAC_RUN
	// the double-single chain programs (the FGMRES sweeps) take the new
	// values now, the others when an application first uses them
	S.stale = S.chain ? 0xFF : 0x0F;
	if (S.ds) {
		const fg_sweep &L = S.lo64c, &U = S.up64c;
		k_refresh<dsf><<<fg_grid(L.nval), FG_TPB, 0, s>>>(S.prog_lo_ds, L.val_off, L.val_src, L.nval, t->ilu.LU,
		                                                  t->ilu.Dinv);
		k_refresh<dsf><<<fg_grid(U.nval), FG_TPB, 0, s>>>(S.prog_up_ds, U.val_off, U.val_src, U.nval, t->ilu.LU,
		                                                  t->ilu.Dinv);
		k_chain_mult<dsf, false><<<fg_grid((long long)L.nslot), FG_TPB, 0, s>>>(S.prog_lo_ds, L.cs_voff, L.cs_src,
		                                                                      L.cs_row, L.nslot, L.rw, t->ilu.LU,
		                                                                      t->ilu.Dinv);
		k_chain_mult<dsf, true><<<fg_grid((long long)U.nslot), FG_TPB, 0, s>>>(S.prog_up_ds, U.cs_voff, U.cs_src,
		                                                                     U.cs_row, U.nslot, U.rw + 1, t->ilu.LU,
		                                                                     t->ilu.Dinv);
	}
	return (int)cudaGetLastError();
}

// Program pair i0, i0 + 1 (0: lo64/up64, 2: lo32/up32, 4: lo64c/up64c,
// 6: lo32c/up32c) given the current factor's values (and, for the chain
// programs, their scan multipliers) if the factorisation left it stale; on
// the context's stream, ahead of the application that uses it.
static int refresh_pair(femgpu_transport *t, int i0)
{
	fg_ilu_sweeps &S = t->sweeps;
	cudaStream_t s = t->stream;
	fg_sweep *pr[8] = { &S.lo64, &S.up64, &S.lo32, &S.up32, &S.lo64c, &S.up64c, &S.lo32c, &S.up32c };
	for (int i = i0; i < i0 + 2; i++) {
		if (!(S.stale & (1 << i))) continue;
		const fg_sweep &c = *pr[i];
		const bool f64 = (i & 2) == 0, up = (i & 1) != 0;
		const int g = fg_grid(c.nval);
		if (f64) k_refresh<double><<<g, FG_TPB, 0, s>>>(c.prog, c.val_off, c.val_src, c.nval, t->ilu.LU, t->ilu.Dinv);
		else k_refresh<float><<<g, FG_TPB, 0, s>>>(c.prog, c.val_off, c.val_src, c.nval, t->ilu.LU, t->ilu.Dinv);
		if (i >= 4) {
			const int gc = fg_grid((long long)c.nslot);
			if (f64 && up) k_chain_mult<double, true><<<gc, FG_TPB, 0, s>>>(c.prog, c.cs_voff, c.cs_src, c.cs_row,
			                                                               c.nslot, c.rw + (up ? 1 : 0), t->ilu.LU, t->ilu.Dinv);
			else if (f64) k_chain_mult<double, false><<<gc, FG_TPB, 0, s>>>(c.prog, c.cs_voff, c.cs_src, c.cs_row,
			                                                               c.nslot, c.rw + (up ? 1 : 0), t->ilu.LU, t->ilu.Dinv);
			else if (up) k_chain_mult<float, true><<<gc, FG_TPB, 0, s>>>(c.prog, c.cs_voff, c.cs_src, c.cs_row,
			                                                            c.nslot, c.rw + (up ? 1 : 0), t->ilu.LU, t->ilu.Dinv);
			else k_chain_mult<float, false><<<gc, FG_TPB, 0, s>>>(c.prog, c.cs_voff, c.cs_src, c.cs_row,
			                                                     c.nslot, c.rw + (up ? 1 : 0), t->ilu.LU, t->ilu.Dinv);
		}
		S.stale &= ~(1 << i);
	}
	return (int)cudaGetLastError();
}

// The dependency-wait bound of the sweep warps: the context's override
// (sweep_wait1 = bound + 1) or SW_WAIT_LIMIT.  Stage waits and the drain after
// a timeout always keep SW_WAIT_LIMIT, so no bulk copy outlives its block.
static int sweep_wait(const femgpu_transport *t)
{
	return t->sweep_wait1 > 0 ? t->sweep_wait1 - 1 : SW_WAIT_LIMIT;
}

static int sweep_args(const femgpu_transport *t, const fg_sweep &sw, const unsigned char *prog, size_t tsize,
                      const int *active, int warps, SweepArgs &a)
{
	a.err = &t->st->err;
	a.active = active;
	a.wait = sweep_wait(t);
	a.prog = prog; a.blk_off = sw.blk_off; a.sb_in = sw.sb_in; a.sb_inb = sw.sb_inb;
	a.nlev = sw.nlev; a.nsb = sw.nsb;
	a.chunk_sb = sw.chunk_sb; a.chunk_lev = sw.chunk_lev; a.bvo = sw.bvo; a.cmax = sw.cmax;
	a.ring = sw.ring; a.look = sw.look;
	return sweep_smem(sw, tsize, &a.D, &a.stage_bytes, warps);
}

// Both sweeps of a dataflow program pair, in one launch when the two have the
// same record width and blocks (FEMGPU_SWEEP_FB=0: always two).
template <typename T, bool FMA, bool CS>
static int run_df(femgpu_transport *t, const fg_sweep &lo, const fg_sweep &up, const unsigned char *plo,
                  const unsigned char *pup, const int *active, const T *in, T *y, T *out)
{
	SweepArgs a, b;
	const char *e = getenv("FEMGPU_SWEEP_FB");
	const bool fb = !(e && e[0] == '0') && lo.rw == up.rw && lo.nchunk == up.nchunk;
	const int w = std::min(lo.warps, up.warps);
	const int bl = sweep_args(t, lo, plo, sizeof(T), active, fb ? w : lo.warps, a);
	if (bl < 0) return bl;
	const int bu = sweep_args(t, up, pup, sizeof(T), active, fb ? w : up.warps, b);
	if (bu < 0) return bu;
	if (fb) launch_fb<T, FMA, CS>(a, b, lo.rw, lo.nchunk, w, std::max(bl, bu), t->stream, in, y, out);
	else {
		launch_df<T, false, FMA, CS>(a, lo.rw, lo.nchunk, lo.warps, bl, t->stream, in, y);
		launch_df<T, true, FMA, CS>(b, up.rw, up.nchunk, up.warps, bu, t->stream, y, out);
	}
	return (int)cudaGetLastError();
}

template <typename T, typename TI, typename TO>
static int apply_t(femgpu_transport *t, const fg_sweep &lo, const fg_sweep &up, T *bl, T *y,
                   const TI *p, TO *z, const int *active, bool fma)
{
	cudaStream_t s = t->stream;
	const int n = t->neq;
	if (p) k_perm_in<T, TI><<<fg_grid(n), FG_TPB, 0, s>>>(p, lo.rows, lo.ppos, n, bl);
	if (lo.cs) return run_df<T, true, true>(t, lo, up, lo.prog, up.prog, active, bl, y, (T *)z);
	fma = fma && sizeof(T) == 8;
	if (lo.df && up.df)
		return fma ? run_df<T, sizeof(T) == 8, false>(t, lo, up, lo.prog, up.prog, active, bl, y, (T *)z)
		           : run_df<T, false, false>(t, lo, up, lo.prog, up.prog, active, bl, y, (T *)z);
	SweepArgs a;
	int bytes = sweep_args(t, lo, lo.prog, sizeof(T), active, 0, a);
	if (bytes < 0) return bytes;
	if (lo.df) {
		if (fma) launch_df<T, false, sizeof(T) == 8, false>(a, lo.rw, lo.nchunk, lo.warps, bytes, s, bl, y);
		else launch_df<T, false, false, false>(a, lo.rw, lo.nchunk, lo.warps, bytes, s, bl, y);
	} else launch_sweep<T, false>(a, lo.rw, lo.nchunk, bytes, s, bl, y, fma);
	bytes = sweep_args(t, up, up.prog, sizeof(T), active, 0, a);
	if (bytes < 0) return bytes;
	if (up.df) {
		if (fma) launch_df<T, true, sizeof(T) == 8, false>(a, up.rw, up.nchunk, up.warps, bytes, s, y, (T *)z);
		else launch_df<T, true, false, false>(a, up.rw, up.nchunk, up.warps, bytes, s, y, (T *)z);
	} else launch_sweep<T, true>(a, up.rw, up.nchunk, bytes, s, y, (T *)z, fma);
	return (int)cudaGetLastError();
}

// FGMRES sweeps (fused arithmetic) and FP32 sweeps take the chain-scan
// programs when the factor has them; the reference's left-preconditioned
// GMRES keeps the row-by-row programs, bit-identical to its ILUp_precond.
// The double-single chain sweeps: gather into double-single slots, the
// forward and backward chain-scan programs with double-single values, the
// backward output (natural order, in the gather buffer) back to FP64.
static int sweeps_ds(femgpu_transport *t, const int *active);
static int apply_ds(femgpu_transport *t, const double *p, const dsf *p_ds, double *z, const int *active)
{
	fg_ilu_sweeps &S = t->sweeps;
	const fg_sweep &lo = S.lo64c;
	cudaStream_t s = t->stream;
	const int n = t->neq;
	dsf *bl = (dsf *)S.bl64;
	if (p_ds) k_perm_in_dsds<<<fg_grid(n), FG_TPB, 0, s>>>(p_ds, lo.rows, lo.ppos, n, bl, active);
	else k_perm_in_ds<<<fg_grid(n), FG_TPB, 0, s>>>(p, lo.rows, lo.ppos, n, bl);
	const int rc = sweeps_ds(t, active);
	if (rc) return rc;
	k_ds_to_double<<<fg_grid(n), FG_TPB, 0, s>>>((const dsf *)S.o64, n, z, active);
	return (int)cudaGetLastError();
}

// The two double-single chain sweeps on the gathered input in the gather
// buffer; the backward sweep writes its output, in natural order, to o64 (not
// back into the gather buffer: in the one-launch form a block's backward sweep
// may run while another block's forward sweep still reads its input there).
static int sweeps_ds(femgpu_transport *t, const int *active)
{
	fg_ilu_sweeps &S = t->sweeps;
	return run_df<dsf, true, true>(t, S.lo64c, S.up64c, S.prog_lo_ds, S.prog_up_ds, active, (const dsf *)S.bl64,
	                               (dsf *)S.y64, (dsf *)S.o64);
}

extern "C" int fg_ilu0_sweeps_gathered(femgpu_transport *t, const int *active)
{
	if (!t->sweeps.ds) return FEMGPU_E_ARG;
	return sweeps_ds(t, active);
}

extern "C" int fg_ilu0_apply64(femgpu_transport *t, const double *p, double *z, const int *active)
{
	fg_ilu_sweeps &S = t->sweeps;
	const bool fma = t->o.solver == FEMGPU_FGMRES;
	if (fma && S.ds) return apply_ds(t, p, NULL, z, active);
	const int pair = (fma && S.chain) ? 4 : 0;
	const int rc = refresh_pair(t, pair);
	if (rc) return rc;
	if (pair) return apply_t<double, double, double>(t, S.lo64c, S.up64c, S.bl64, S.y64, p, z, active, true);
	return apply_t<double, double, double>(t, S.lo64, S.up64, S.bl64, S.y64, p, z, active, fma);
}

// z = M^-1 p by the separately rounded sweeps, p already in bl64 as lo64 takes it
// (at dpos64[row]).
extern "C" int fg_ilu0_apply64_gathered(femgpu_transport *t, double *z, const int *active)
{
	fg_ilu_sweeps &S = t->sweeps;
	const int rc = refresh_pair(t, 0);
	if (rc) return rc;
	return apply_t<double, double, double>(t, S.lo64, S.up64, S.bl64, S.y64, nullptr, z, active, false);
}

// The double-single sweeps with a double-single input (the Krylov basis of
// the double-single Arnoldi); available when fg_ilu0_ds_ready says so.
extern "C" int fg_ilu0_ds_ready(const femgpu_transport *t)
{
	return t->sweeps.ds ? 1 : 0;
}

extern "C" int fg_ilu0_apply64_dsin(femgpu_transport *t, const void *p, double *z, const int *active)
{
	if (!t->sweeps.ds) return FEMGPU_E_NOT_BUILT;
	return apply_ds(t, NULL, (const dsf *)p, z, active);
}

extern "C" int fg_ilu0_apply32(femgpu_transport *t, const double *p, float *z, const int *active)
{
	fg_ilu_sweeps &S = t->sweeps;
	const int rc = refresh_pair(t, S.chain ? 6 : 2);
	if (rc) return rc;
	if (S.chain) return apply_t<float, double, float>(t, S.lo32c, S.up32c, S.bl32, S.y32, p, z, active, false);
	return apply_t<float, double, float>(t, S.lo32, S.up32, S.bl32, S.y32, p, z, active, false);
}

extern "C" void fg_ilu_free(femgpu_transport *t)
{
	fg_ilu_sweeps &S = t->sweeps;
	fg_sweep *all[8] = { &S.lo64, &S.up64, &S.lo32, &S.up32, &S.lo64c, &S.up64c, &S.lo32c, &S.up32c };
	for (int i = 0; i < 8; i++) {
		void *p[] = { all[i]->prog, all[i]->blk_off, all[i]->sb_in, all[i]->sb_inb,
		              all[i]->rows, all[i]->ppos, all[i]->val_off, all[i]->val_src, all[i]->chunk_sb,
		              all[i]->chunk_lev, all[i]->cs_voff, all[i]->cs_src, all[i]->cs_row };
		for (void *q : p) if (q) cudaFree(q);
		memset(all[i], 0, sizeof(fg_sweep));
	}
	S.chain = 0;
	void *v[] = { S.bl64, S.y64, S.o64, S.bl32, S.y32, S.fac_head, S.fac_grp, S.fac_pos, S.fac_ticket, S.fIA, S.fJA,
	              S.fmap, S.fA };
	for (void *q : v) if (q) cudaFree(q);
	S.bl64 = S.y64 = S.o64 = nullptr;
	S.bl32 = S.y32 = nullptr;
	S.fIA = S.fJA = S.fmap = nullptr;
	S.fA = nullptr;
	S.fill = 0;
	if (S.dpos) cudaFree(S.dpos);
	if (S.dpos64) cudaFree(S.dpos64);
	S.dpos = S.dpos64 = nullptr;
	if (S.prog_lo_ds) cudaFree(S.prog_lo_ds);
	if (S.prog_up_ds) cudaFree(S.prog_up_ds);
	S.prog_lo_ds = S.prog_up_ds = nullptr;
	S.ds = 0;
	free(S.block_first);
	S.block_first = nullptr;
	S.nblocks = 0;
}
