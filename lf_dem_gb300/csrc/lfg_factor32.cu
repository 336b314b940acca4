// lfg_factor32.cu -- FP32 trailing updates of large fronts on the tensor cores,
// C -= A B^T over an outer block of four panels at a time, in the manner of the
// FP64 tiles (lfg_factor64.cu).  Over the block's 256 columns a row is scaled by a power of
// two to 30-bit integers and cut into 4 signed base-256 digits (FP16); the
// digit products of order i + j = q < 4 are summed in FP32, integers of at most
// 4 x 256 x 2^14 = 2^24, so exactly.  What is dropped (orders 4 to 6) lies
// 2^-26 under the product of the rows' largest entries per term, at most 2^-18 over a
// block whatever the signs and typically 2^-24; one rounding per block replaces one
// per term, where a chain of 256 FP32 multiply-adds may lose 2^-16.  Measured against
// the FP64 factor: L b of suspensions of 3500 to 16384 particles 2.9e-6 with either;
// dense fronts whose updates cancel the entries from 100 to 6, 3402 and 3840 columns:
// 6.5e-3 and 7.1e-3, 1.4e-2 and 1.6e-2 by multiply-adds.
#include <mutex>

#include "lfg_split.cuh"

namespace lfg {

namespace split32 {
using namespace split;
constexpr int DIGITS = 4;
constexpr int TN = 128;                   // tile columns: 4 orders fill the tensor memory
constexpr int KB = 256;                   // K block: one scale per row, one flush of the accumulators
constexpr int PANEL = 64;                 // panel width
constexpr int OUTER = KB/PANEL;           // panels per outer block
constexpr int GROUP = 2*M, GROUPS = 2;    // producer threads: a row of A (first 128) or of B each; the groups
                                          // take alternate K steps (one alone took 1200 cycles a step, half
                                          // of it waiting: twice the MMAs' 640)
constexpr int PRODUCERS = GROUPS*GROUP, MMA_WARP = PRODUCERS/32, LOAD_WARP = MMA_WARP+1;
constexpr int THREADS = PRODUCERS+64;
constexpr int STAGES = 4;                 // K steps of scaled rows in flight
constexpr int STEP_BYTES = KS*4;          // a row's K step
constexpr int STAGE_BYTES = 2*M*STEP_BYTES;
constexpr int SMEM = 2*DIGITS*A_BYTES+STAGES*STAGE_BYTES+1024;
constexpr int MIN_EXP = 32;               // rows below 2^-95 are scaled as if that large
constexpr uint32_t BIAS = 0x80808080u;    // the scaled zero

// x (its bits) scaled to a 30-bit signed integer against the row's largest
// biased exponent e (times 2^(156 - e), rounded to nearest) plus 128 in every
// byte: digit i of the integer is byte 3 - i minus 128
__device__ __forceinline__ uint32_t scale_entry(uint32_t b, int e)
{
	const unsigned ex = (b >> 23) & 0xffu;
	const unsigned d = min((unsigned)e-ex, 31u);
	const uint32_t y = (((((b & 0x007fffffu) | 0x00800000u) << 7) >> d)+1) >> 1;
	const uint32_t s = (uint32_t)((int32_t)b >> 31);
	return (y ^ s)+(BIAS-s);
}

// Scaled rows in memory: K step q (16 columns) of row r of a front is a 64-byte
// record at 16 (q ld + r), the rows of a step one after another, so a tile's 128
// rows are one bulk copy.  The record's 16-byte chunks are permuted by the row
// (chunk c at c ^ ((r >> 1) & 3)): eight lanes of consecutive rows then read
// theirs from all 32 shared-memory banks.
__device__ __forceinline__ int64_t record(int q, int ld, int row) { return ((int64_t)q*ld+row)*KS; }
__device__ __forceinline__ int chunk(int c, int row) { return 4*(c ^ ((row >> 1) & 3)); }

// digit I of the 16 scaled entries of a row's K step: two 16-byte chunks,
// swizzled by the row (m7 = row & 7)
template <int I>
__device__ __forceinline__ void store_digits(const uint32_t (&y)[16], unsigned char *row, int slot, int m7)
{
	if constexpr (I < DIGITS) {
#pragma unroll
		for (int h = 0; h < 2; h++) {
			uint32_t w[4];
#pragma unroll
			for (int p = 0; p < 4; p++) w[p] = digit_pair<3-I>(y[8*h+2*p], y[8*h+2*p+1]);
			*reinterpret_cast<uint4 *>(row+I*A_BYTES+(((2*slot+h) ^ m7) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
		}
		store_digits<I+1>(y, row, slot, m7);
	}
}

// the smaller and the larger of two scales; NaN if either is
__device__ __forceinline__ float min_scale(float a, float b)
{
	float r;
	asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
	return r;
}
__device__ __forceinline__ float max_scale(float a, float b)
{
	float r;
	asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
	return r;
}

__device__ inline void tmem_ld8(uint32_t ta, uint32_t (&v)[8])
{
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
	             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
	             : "r"(ta));
}

} // namespace split32

// One 128 x 128 tile per CTA of the pivot columns that remain after panel k, the
// last of an outer block.  The rows arrive scaled (ybuf, yexp) from the panel
// solves.
//
// One thread copies the scaled rows of a K step (8 KB each of A and B, bulk
// copies) into a ring of four stages; two groups of eight warps take alternate
// steps, a thread a row of A or of B, and cut it into a ring of four K steps
// behind full/empty mbarriers; one warp multiplies (digit i of A with digits 0..3-i of B, N = 128 or 256 columns an
// instruction, onto the accumulators of orders i..3).  Then the producers
// join the four sums (three multiply-adds) and subtract them from C.  Rows past
// the tile's limits are cut from whatever is there; their results are not stored.
//
// Bound: the 10 digit products of a K step take 640 tensor cycles, and shared
// memory (65 KB of operands read by the MMAs, 64 KB through the rings) a thousand;
// measured 1200 a step and 31k cycles a tile, 15 us a wave of 152 tiles (64 us for
// the four right-looking CUDA-core updates of the same columns).  N = 16384: 41.1
// -> 33.2 ms per step.
__global__ void __launch_bounds__(split32::THREADS, 1)
k_tile32(const int4 *__restrict__ tasks, const int *__restrict__ sn_n, const int *__restrict__ sn_m,
         const int *__restrict__ sn_ld, const int64_t *__restrict__ sn_off, float *__restrict__ arena,
         const unsigned short *yexp, const uint32_t *ybuf,
         const int64_t *__restrict__ split_off, int *fail, int dof)
{
	using namespace split32;
	extern __shared__ unsigned char smem_s32[];
	__shared__ __align__(8) Bars bars;
	__shared__ __align__(8) uint64_t yfull[STAGES], yempty[STAGES];
	__shared__ uint32_t tmem_slot;
	__shared__ int exps[2*M];   // rows of A, rows of B
	unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_s32)+1023) &
	                                                      ~static_cast<uintptr_t>(1023));
	const int tid = threadIdx.x, warp = tid/32, lane = tid%32;
	const int4 tk = tasks[blockIdx.x];
	const int s = tk.x, r0 = tk.y, c0 = tk.z, k = tk.w;
	const int n6 = dof*sn_n[s], F6 = n6+dof*sn_m[s], ld = sn_ld[s];
	const int t0 = min((k+1)*PANEL, n6);
	const int k0 = k/OUTER*KB, k1 = t0;   // one whole K block
	const bool extra = r0 >= F6;          // identity rows
	const int rlim = extra ? F6+t0 : F6, clim = n6;
	float *base = arena+sn_off[s];
	const unsigned short *etab = yexp+split_off[3*s+1];
	const uint32_t *src = ybuf+split_off[3*s+2];
	bool ok = true;
	pdl_wait();   // before the tensor-memory allocation, too
	asm volatile("fence.proxy.async.global;" ::: "memory");   // the bulk copies see the panel solve's stores
	if (warp == 0) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
		             :: "r"(saddr(&tmem_slot)), "r"(DIGITS*TN));
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
		asm volatile("tcgen05.fence::before_thread_sync;");
	}
	if (tid == 32) {
		for (int q = 0; q < SLOTS; q++) {
			mbar_init(&bars.full[q], GROUP);
			mbar_init(&bars.empty[q], 1);
		}
		for (int q = 0; q < STAGES; q++) {
			mbar_init(&yfull[q], 1);
			mbar_init(&yempty[q], GROUP);
		}
		mbar_init(&bars.done, 1);
		asm volatile("fence.mbarrier_init.release.cluster;");
	}
	// producer role: a row of A or B
	const bool producer = tid < PRODUCERS, isA = tid % GROUP < M;
	const int grp = tid/GROUP, m = tid & (M-1), row = (isA ? r0 : c0)+m;
	const bool live = producer && row < (isA ? rlim : clim);
	unsigned char *rowp = sm+(isA ? 0 : DIGITS*A_BYTES)+(m >> 3)*1024+(m & 7)*128;
	unsigned char *stages = sm+2*DIGITS*A_BYTES;
	int g = 0;   // K steps so far (loader: copied, producers: cut, MMA warp: multiplied)
	auto stage = [&]() {
		const int slot = g % SLOTS, st = g % STAGES;
		if (ok && !mbar_wait(saddr(&yfull[st]), (g/STAGES) & 1)) ok = false;
		const uint32_t *rec = reinterpret_cast<const uint32_t *>(stages+st*STAGE_BYTES)+tid%GROUP*KS;
		uint32_t x[16];
#pragma unroll
		for (int c = 0; c < 4; c++) {
			const uint4 q = *reinterpret_cast<const uint4 *>(rec+chunk(c, row));
			x[4*c] = q.x; x[4*c+1] = q.y; x[4*c+2] = q.z; x[4*c+3] = q.w;
		}
		if (g >= SLOTS && ok && !mbar_wait(saddr(&bars.empty[slot]), ((g/SLOTS)-1) & 1)) ok = false;
		store_digits<0>(x, rowp, slot, m & 7);
		asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // visible to the tensor cores
		asm volatile("tcgen05.fence::before_thread_sync;");
		mbar_arrive(&bars.full[slot]);
		// not before the digits were formed: an arrive may overtake shared loads
		// that are still on their way
		mbar_arrive(&yempty[st]);
	};
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;");
	const uint32_t tmem = tmem_slot;
	// epilogue role: row er, columns c0 + eg + [0, 32)
	const int el = 32*(warp & 3)+lane, er = r0+el, eg = 32*(warp >> 2 & 3);
	if (grp == 0) exps[tid] = live ? max((int)etab[(int64_t)(k0/KB)*ld+row], MIN_EXP) : MIN_EXP;
	__syncwarp();
	if (producer) asm volatile("bar.sync 1, 512;" ::: "memory");   // producers: the exponents are in
	if (producer) {
		for (int t = k0; t < k1; t += KS, g++)
			if ((g & 1) == grp) stage();
	} else if (warp == MMA_WARP) {
		if (lane == 0) {
			const uint32_t sa = saddr(sm), sb = sa+DIGITS*A_BYTES;
			for (int t = k0; t < k1; t += KS, g++) {
				const int slot = g % SLOTS;
				if (ok && !mbar_wait(saddr(&bars.full[slot]), (g/SLOTS) & 1)) ok = false;
				if (!ok) break;
				asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
				for (int i = 0; i < DIGITS; i++)
#pragma unroll
					for (int j = 0; j < DIGITS-i; j += 2) {
						const int cnt = DIGITS-i-j < 2 ? 1 : 2;
						mma_f16(tmem+(i+j)*TN, sdesc(sa+i*A_BYTES+32*slot), sdesc(sb+j*A_BYTES+32*slot),
						        idesc(TN*cnt), (t > k0 || i > 0) ? 1u : 0u);
					}
				mma_commit(&bars.empty[slot]);
			}
			mma_commit(&bars.done);   // everything issued so far
		}
		__syncwarp();
	} else if (warp == LOAD_WARP) {
		if (lane == 0) {
			for (int t = k0; t < k1; t += KS, g++) {
				const int st = g % STAGES;
				if (g >= STAGES && ok && !mbar_wait(saddr(&yempty[st]), ((g/STAGES)-1) & 1)) ok = false;
				if (!ok) break;
				bulk_expect(&yfull[st], STAGE_BYTES);
				bulk_load(stages+st*STAGE_BYTES, src+record(t/KS, ld, r0), M*STEP_BYTES, &yfull[st]);
				bulk_load(stages+st*STAGE_BYTES+M*STEP_BYTES, src+record(t/KS, ld, c0), M*STEP_BYTES, &yfull[st]);
			}
			for (int q = max(0, g-STAGES); q < g; q++)   // no copy in flight when the CTA ends
				if (!mbar_wait(saddr(&yfull[q % STAGES]), (q/STAGES) & 1)) ok = false;
		}
		__syncwarp();
	}
	// epilogue, 16 columns at a time: the old values first, the first of them in
	// flight while the MMAs finish
#pragma unroll 1
	for (int j1 = producer ? 0 : 32; j1 < 32; j1 += 16) {
		float C[16];
		unsigned in = 0;
		float *pc = base+(int64_t)(c0+eg+j1)*ld+er;
#pragma unroll
		for (int j = 0; j < 16; j++) {
			const int c = c0+eg+j1+j;
			const bool own = er < rlim && c < clim && (extra || er >= c);
			C[j] = own ? pc[(int64_t)j*ld] : 0.f;
			in |= (unsigned)own << j;
		}
		if (j1 == 0) {
			if (ok && !mbar_wait(saddr(&bars.done), 0)) ok = false;
			__syncwarp();
			asm volatile("tcgen05.fence::after_thread_sync;");
		}
		// exponents ea, eb: the sum of order 0 is in units of 2^(ea + eb - 264).  The
		// smaller of the rows' scales first: nothing overflows that the product does not
		const int ea = exps[el];
		const float sa = __int_as_float(ea < 0xff ? (ea-5) << 23 : 0x7fc00000);   // NaN for a row with an inf or NaN
#pragma unroll
		for (int j0 = 0; j0 < 16; j0 += 8) {
			uint32_t a[DIGITS][8];
#pragma unroll
			for (int q = 0; q < DIGITS; q++)
				tmem_ld8(tmem+((uint32_t)(32*(warp & 3)) << 16)+(uint32_t)(q*TN+eg+j1+j0), a[q]);
			asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
			for (int j = 0; j < 8; j++) {
				float x = 0.f;
#pragma unroll
				for (int q = DIGITS-1; q >= 0; q--) {
					asm volatile("" : "+r"(a[q][j]));   // not used before the wait
					x = fmaf(x, 1.f/256, __uint_as_float(a[q][j]));
				}
				const int eb = exps[M+eg+j1+j0+j];
				const float sb = __int_as_float(eb < 0xff ? (eb-5) << 23 : 0x7fc00000);
				C[j0+j] = fmaf(-(x*min_scale(sa, sb)), max_scale(sa, sb), C[j0+j]);
			}
		}
		if (ok)
#pragma unroll
			for (int j = 0; j < 16; j++)
				if (in >> j & 1) pc[(int64_t)j*ld] = C[j];
	}
	asm volatile("tcgen05.fence::before_thread_sync;");
	ok = __syncthreads_and(ok);
	if (warp == 0)
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(DIGITS*TN));
	if (!ok && tid == 0 && fail) atomicMin(fail, 0);
}

// Panel solve X = A Linv_kk^T of up to 64 rows per CTA, as k_trsm
// (lfg_factor.cu) and with its results bit for bit, for the levels that hold a
// front that is updated two-level.  Such a front's (split_off >= 0) also record each row's
// largest exponent in the panel and, after the last panel of a K block that has
// columns after it, leave the rows' entries in the block as scaled integers for k_tile32.
__global__ void __launch_bounds__(256) k_trsm_split(const int4 *__restrict__ tasks, const int *__restrict__ sn_n,
                                                    const int *__restrict__ sn_m, const int *__restrict__ sn_ld,
                                                    const int64_t *__restrict__ sn_off, float *__restrict__ arena,
                                                    const float *linv, int nsn, int dof,
                                                    unsigned short *rexp, unsigned short *yexp, uint32_t *ybuf,
                                                    const int64_t *__restrict__ split_off)
{
	using namespace split32;
	constexpr int NB = PANEL, CW = NB/8, R = 64;
	__shared__ __align__(16) float Vt[NB*NB];   // Linv^T, row-major
	__shared__ float As[R*NB];                  // row r, column t at r*NB + (t ^ (r & 31))
	__shared__ int rmax[R];
	const int4 tk = tasks[blockIdx.x];
	const int s = tk.x, row0 = tk.y, k = tk.z, nrows = tk.w, tid = threadIdx.x;
	const int ld = sn_ld[s], n6 = dof*sn_n[s], F6 = n6+dof*sn_m[s];
	const int p0 = k*NB, w = min(NB, n6-p0), kp = k/OUTER*OUTER;
	const int64_t ro = split_off[3*s];
	const bool two = ro >= 0;   // of a front that is updated two-level
	const bool block_end = two && k-kp == OUTER-1 && p0+w < n6;   // columns are left
	float *base = arena+sn_off[s];
	const float *vt = linv+((int64_t)(k & 1)*nsn+s)*NB*NB;
	unsigned short *rt = rexp+ro;
	if (tid < R) rmax[tid] = 0;
	pdl_trigger();   // the next update's CTAs wait resident while this short launch runs
	pdl_wait();
	{
		float lv[NB*NB/256], av[R*NB/256];
#pragma unroll
		for (int u = 0; u < NB*NB/256; u++) lv[u] = vt[tid+256*u];
#pragma unroll
		for (int u = 0; u < R*NB/256; u++) {
			const int e = tid+256*u, r = e%R, t = e/R;   // coalesced over rows
			av[u] = r < nrows && t < w ? base[(int64_t)(p0+t)*ld+row0+r] : 0.f;
		}
#pragma unroll
		for (int u = 0; u < NB*NB/256; u++) Vt[tid+256*u] = lv[u];
#pragma unroll
		for (int u = 0; u < R*NB/256; u++) {
			const int e = tid+256*u, r = e%R, t = e/R;
			As[r*NB+(t ^ (r & 31))] = av[u];
		}
	}
	__syncthreads();
	// thread: row r, column chunks g and 7 - g (equal work per thread: chunk c
	// has (c + 1) CW terms per entry)
	const int g = tid/R, r = tid%R, sw = r & 31;
	const float *a0 = As+r*NB;
	float x[2][CW];
	int emax = 0;
#pragma unroll
	for (int h = 0; h < 2; h++) {
		const int j0 = (h ? 7-g : g)*CW;
#pragma unroll
		for (int q = 0; q < CW; q++) x[h][q] = 0.f;
#pragma unroll 4
		for (int t = 0; t < j0+CW; t++) {
			const float4 v0 = *reinterpret_cast<const float4 *>(Vt+t*NB+j0);
			const float4 v1 = *reinterpret_cast<const float4 *>(Vt+t*NB+j0+4);
			const float u = a0[t ^ sw];
			x[h][0] += u*v0.x; x[h][1] += u*v0.y; x[h][2] += u*v0.z; x[h][3] += u*v0.w;
			x[h][4] += u*v1.x; x[h][5] += u*v1.y; x[h][6] += u*v1.z; x[h][7] += u*v1.w;
		}
#pragma unroll
		for (int q = 0; q < CW; q++)
			if (j0+q < w) {
				if (r < nrows) base[(int64_t)(p0+j0+q)*ld+row0+r] = x[h][q];
				emax = max(emax, (__float_as_int(x[h][q]) >> 23) & 0xff);
			}
	}
	if (!two) return;
	atomicMax(&rmax[r], emax);
	__syncthreads();
	if (tid < nrows) rt[(int64_t)k*ld+row0+tid] = (unsigned short)rmax[tid];
	if (!block_end) return;
	if (tid < nrows) {
		// the row's exponent in the block (identity row i is zero in panels that end before it)
		int e = max(rmax[tid], MIN_EXP);
		const int i = row0+tid-F6;
		for (int p = kp; p < k; p++)
			if (i < (p+1)*NB) e = max(e, (int)rt[(int64_t)p*ld+row0+tid]);
		rmax[tid] = e;
		yexp[split_off[3*s+1]+(int64_t)(k/OUTER)*ld+row0+tid] = (unsigned short)e;
	}
	__syncthreads();
	if (r >= nrows) return;
	const int e = rmax[r];
	uint32_t *yb = ybuf+split_off[3*s+2];
	const uint32_t *xb = reinterpret_cast<const uint32_t *>(base)+row0+r;
	// earlier panels: chunks of 4 columns, g first, 4 chunks loaded at a time
	for (int t0 = kp*NB+4*g; t0 < p0; t0 += 64) {
		uint32_t y[16];
#pragma unroll
		for (int u = 0; u < 16; u++) y[u] = xb[(int64_t)(t0+16*(u/4)+u%4)*ld];
#pragma unroll
		for (int u = 0; u < 16; u += 4)
			*reinterpret_cast<uint4 *>(yb+record(t0/KS+u/4, ld, row0+r)+chunk(g, row0+r)) =
				make_uint4(scale_entry(y[u], e), scale_entry(y[u+1], e), scale_entry(y[u+2], e), scale_entry(y[u+3], e));
	}
	// this panel's (a whole one: columns are left)
#pragma unroll
	for (int h = 0; h < 2; h++)
#pragma unroll
		for (int q = 0; q < CW; q += 4) {
			const int j = (h ? 7-g : g)*CW+q;
			uint32_t y[4];
#pragma unroll
			for (int u = 0; u < 4; u++) y[u] = scale_entry(__float_as_uint(x[h][q+u]), e);
			*reinterpret_cast<uint4 *>(yb+record((p0+j)/KS, ld, row0+r)+chunk(j/4%4, row0+r)) =
				make_uint4(y[0], y[1], y[2], y[3]);
		}
}

void tile32_setup()
{
	static std::once_flag once;
	std::call_once(once, [] {
		LFG_CUDA(cudaFuncSetAttribute(k_tile32, cudaFuncAttributeMaxDynamicSharedMemorySize, split32::SMEM));
	});
}

int tile32_kblock() { return split32::KB; }
int trsm_split_rows() { return 64; }   // four threads a row

// scaled entries of a front's K blocks; the slack lets a tile's copy run past the last rows
int64_t tile32_ybuf(int kblocks, int ld)
{
	return ((int64_t)kblocks*(split32::KB/split32::KS)*ld+split32::M)*split32::KS;
}

void tile32_launch(const DevSymbolic &D, int64_t off, int count, DevFactor<float> &F, cudaStream_t st)
{
	launch_pdl(k_tile32, count, split32::THREADS, split32::SMEM, st, (const int4 *)D.tile_tasks+off, (const int *)D.sn_n,
	           (const int *)D.sn_m, (const int *)D.sn_ld, (const int64_t *)D.sn_off, F.arena,
	           (const unsigned short *)F.yexp, (const uint32_t *)F.ybuf, (const int64_t *)D.split_off, F.status, D.dof);
}

void trsm_split_launch(const DevSymbolic &D, int64_t off, int count, DevFactor<float> &F, cudaStream_t st)
{
	launch_pdl(k_trsm_split, count, 256, 0, st, (const int4 *)D.panel_tasks+off, (const int *)D.sn_n,
	           (const int *)D.sn_m, (const int *)D.sn_ld, (const int64_t *)D.sn_off, F.arena, (const float *)F.linv,
	           D.nsn, D.dof, F.rexp, F.yexp, (uint32_t *)F.ybuf, (const int64_t *)D.split_off);
}

} // namespace lfg
