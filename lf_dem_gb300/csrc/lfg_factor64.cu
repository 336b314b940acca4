// lfg_factor64.cu -- FP64 products of the multifrontal factorisation on the
// tensor cores (the plain FP64 form; replaces the dense part of CHOLMOD's
// supernodal cholmod_factorize, LF_DEM/StokesSolver.cpp:950-978).
//
// GB300 has 2 FP64 multiply-adds per cycle and SM and no FP64 tensor path, so
// C -= A B^T runs as exact integer products (the error-free splitting of
// Ozaki, Ogita, Oishi, Rump 2012).  Per K block of 128 every row of A and of B
// is scaled by a power of two to 62-bit integers and cut into 8 signed
// base-256 digits, each an FP16 value.  tcgen05.mma multiplies digit matrices
// into FP32 accumulators, one per digit order i + j = 0..7: integer sums of at
// most 8 x 128 x 2^14 = 2^24, so exact for any input.  The epilogue joins the
// eight sums into one 96-bit integer, rounds it once to FP64 and subtracts it
// from C.
//
// Error: what is dropped (below the last digit, and orders above 7) lies 2^-57
// under the product of the two rows' largest entries in the block per term, at
// most 2^-50 over a block whatever the signs and typically 2^-56, and one
// rounding per K block replaces one per term (128 terms in FP64 may lose 2^-46).
// 7 digits (256 times that) were not enough: the rows' large entries are several
// times their typical ones, and the solver's error against 128-bit solutions grew
// by a fifth.
#include <mutex>

#include "lfg_diag64.cuh"
#include "lfg_split.cuh"

namespace lfg {

namespace split64 {
using namespace split;
constexpr int DIGITS = 8;
constexpr int KB = 128;                   // K block: one scale per row, one flush of the accumulators
constexpr int PANEL = 32;                 // panel width
constexpr int OUTER = 4;                  // panels per outer block of the trailing updates
static_assert(OUTER*PANEL == KB, "an outer block is a K block");
constexpr int MMA_WARP = 12;              // issues the MMAs and nothing else: the issue waits for the tensor
                                          // pipe, and a warp that also cut entries held everyone up
constexpr int MIN_EXP = 64;               // rows below 2^-959 are scaled as if that large

template <int TN> struct Tile {
	static constexpr int B_BYTES = TN*ROW_BYTES;
	static constexpr int SMEM = DIGITS*(A_BYTES+B_BYTES)+1024;
	static constexpr int COLS = DIGITS*TN <= 256 ? 256 : 512;   // tensor memory columns
	static constexpr int CPW = TN/4;                            // epilogue columns per warp
	static constexpr int PRODUCERS = 2*M+2*TN;                  // threads: 8 entries of a row each per K step
};

// x scaled to a 62-bit signed integer against the row's largest biased
// exponent e (times 2^(1084 - e), rounded to nearest) plus 128 in every byte:
// digit i of the integer is byte 7 - i of the result minus 128.  Zeros and
// entries far below the row's scale shift out.
constexpr uint64_t BIAS = 0x8080808080808080ull;   // the scaled zero
__device__ __forceinline__ uint64_t scale_entry(uint64_t b, int e)   // b: the bits of x
{
	const unsigned ex = (unsigned)(b >> 52) & 0x7ffu;
	const unsigned d = min((unsigned)e-ex, 63u);
	const uint64_t m = ((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 10;
	const uint64_t y = ((m >> d)+1) >> 1;
	const uint64_t s = (uint64_t)((int64_t)b >> 63);
	return (y ^ s)+(BIAS-s);
}

// digit I of N scaled entries of one row as FP16 values
template <int I, int N>
__device__ __forceinline__ void digit(const uint64_t (&y)[N], uint32_t (&out)[N/2])
{
	constexpr int byte = 7-I, sel = byte & 3;
#pragma unroll
	for (int p = 0; p < N/2; p++) {
		const uint32_t w0 = byte >= 4 ? (uint32_t)(y[2*p] >> 32) : (uint32_t)y[2*p];
		const uint32_t w1 = byte >= 4 ? (uint32_t)(y[2*p+1] >> 32) : (uint32_t)y[2*p+1];
		out[p] = digit_pair<sel>(w0, w1);
	}
}

template <int I>
__device__ __forceinline__ void store_digits(const uint64_t (&y)[8], unsigned char *p, int stride)
{
	if constexpr (I < DIGITS) {
		uint32_t w[4];
		digit<I>(y, w);
		*reinterpret_cast<uint4 *>(p+I*stride) = make_uint4(w[0], w[1], w[2], w[3]);
		store_digits<I+1>(y, p, stride);
	}
}

// The largest biased exponent of row r of a front over the panels
// [p0, p1): the panel solves record it per row and panel.  An identity row
// (i = r - F6 >= 0) is zero in panels that end at or before column i.
__device__ __forceinline__ int row_exponent(const unsigned short *tab, int ld, int r, int F6, int n6, int p0, int p1)
{
	int e = MIN_EXP;
	const int i = r-F6;
#pragma unroll 8
	for (int p = p0; p < p1; p++) {
		if (i >= 0 && i >= min((p+1)*PANEL, n6)) continue;
		e = max(e, (int)tab[(int64_t)p*ld+r]);
	}
	return e;
}

// 2^(e - 2168) sum_q a[q] 256^(14 - q), rounded once (half up): the product sum
// of two rows whose exponents add up to e.
//
// The integer pipe is half as wide as the FP32 one and a warp's FP64 operation
// takes 64 cycles, so the carries are propagated in FP32 (exactly: every value
// is an integer below 2^25), a digit at a time from the last order up; three
// 24-bit groups are left to convert and to join.  The last digit itself, 2^-63
// under the largest product, only passes its carry on.
__device__ __forceinline__ double join_orders(const uint32_t (&a)[DIGITS], int e)
{
	constexpr float R = 3221225472.f;   // 1.5 2^31: x + R rounds x to a multiple of 256
	float l[DIGITS], carry = 0.f;
#pragma unroll
	for (int q = DIGITS-1; q > 0; q--) {
		const float x = fmaf(carry, 1.f/256, __uint_as_float(a[q]));
		carry = __fsub_rn(__fadd_rn(x, R), R);
		l[q] = x-carry;
	}
	const int top = __float2int_rn(fmaf(carry, 1.f/256, __uint_as_float(a[0])));
	const int mid = __float2int_rn(fmaf(fmaf(l[1], 256.f, l[2]), 256.f, l[3]));
	const int low = __float2int_rn(fmaf(fmaf(l[4], 256.f, l[5]), 256.f, l[6]));
	// top 2^48 + mid 2^24 + low = h 2^32 + l: sign and magnitude (below 2^70)
	const int64_t p = (int64_t)mid*16777216+low;
	const int64_t h = (int64_t)top*65536+(p >> 32);
	const uint64_t sg = (uint64_t)(h >> 63);
	const uint32_t lu = ((uint32_t)p ^ (uint32_t)sg)-(uint32_t)sg;
	const uint64_t hu = ((uint64_t)h ^ sg)+(lu == 0 ? sg & 1 : 0);
	uint32_t w2 = (uint32_t)(hu >> 6), w1 = (uint32_t)hu << 26 | lu >> 6, w0 = lu << 26;
	int f = e-1012;
	if (w2 == 0) {   // rare but for exact zeros
		w2 = w1; w1 = w0; w0 = 0; f -= 32;
		if (w2 == 0) { w2 = w1; w1 = 0; f -= 32; }
		if (w2 == 0) return 0.0;
	}
	const int lz = __clz(w2);
	f -= lz;
	const uint64_t m = (uint64_t)__funnelshift_l(w1, w2, lz) << 32 | __funnelshift_l(w0, w1, lz);
	uint64_t b = ((uint64_t)(f-1) << 52)+((m >> 11)+((m >> 10) & 1));
	if (__builtin_expect((unsigned)(f-1) >= 2046u, 0))   // infinite, or below the normal numbers
		b = f > 0 ? 0x7ff0000000000000ull : f >= -52 ? ((m >> (11-f))+1) >> 1 : 0;
	return __longlong_as_double((long long)(b | (sg & 0x8000000000000000ull)));
}

// Linv slot of supernode s for panel k: two slots per supernode, by the parity
// of k (the update launch of panel k writes panel k + 1's)
template <typename P> __device__ inline P *linv64_slot(P *linv, int nsn, int s, int k)
{
	return linv+((int64_t)(k & 1)*nsn+s)*PANEL*PANEL;
}

__device__ inline void tmem_ld2(uint32_t ta, uint32_t (&v)[2])
{
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(ta));
}

// digit I of 4 entries of a row, to the row's place in B's tile and in the four
// row quarters of A's
template <int I>
__device__ __forceinline__ void store_diag_digits(const uint64_t (&y)[4], unsigned char *pa, unsigned char *pb)
{
	if constexpr (I < DIGITS) {
		uint32_t w[2];
		digit<I>(y, w);
#pragma unroll
		for (int rep = 0; rep < 4; rep++) *reinterpret_cast<uint2 *>(pa+I*A_BYTES+rep*4096) = make_uint2(w[0], w[1]);
		*reinterpret_cast<uint2 *>(pb+I*4096) = make_uint2(w[0], w[1]);
		store_diag_digits<I+1>(y, pa, pb);
	}
}

// The next panel's w1 x w1 diagonal block (rows and columns t0 + [0, 32)),
// updated over the front's columns [k0, k1), at most KB of them, into Ls
// (stride 33, identity-padded), by the whole CTA.  It is on the chain of the
// panels, so it is a tile of its own: 32 rows instead of 128, cut once for A
// and B, and stored four times in A, once for each quarter of the tensor
// memory's lanes, so that all 16 warps can read it: a lane per row, two columns
// per warp.  (A warp reaches its own quarter only.)
__device__ inline bool diag_tile(const double *base, int ld, int t0, int w1, int k0, int k1, int F6, int n6,
                                 const unsigned short *rexp, unsigned char *sm, uint64_t *done, uint32_t tmem,
                                 int *exps, double *Ls)
{
	const int warp = threadIdx.x/32, lane = threadIdx.x%32, row = t0+lane;
	const bool live = lane < w1;
	bool ok = true;
	uint64_t v[4];
	auto load = [&](int t) {   // columns t + 4 warp + [0, 4) of a half of 64
		const uint64_t *p = reinterpret_cast<const uint64_t *>(base)+(int64_t)(t+4*warp)*ld+row;
#pragma unroll
		for (int i = 0; i < 4; i++) v[i] = live && t+4*warp+i < k1 ? p[(int64_t)i*ld] : 0;
	};
	load(k0);
	double C[2];
#pragma unroll
	for (int j = 0; j < 2; j++) {
		const int c = 2*warp+j;
		C[j] = live && lane >= c ? base[(int64_t)(t0+c)*ld+row] : 0.0;
	}
	const int e = live ? row_exponent(rexp, ld, row, F6, n6, k0/PANEL, (k1+PANEL-1)/PANEL) : MIN_EXP;
	if (warp == 0) exps[lane] = e;
	unsigned char *pa = sm+(lane >> 3)*1024+(lane & 7)*128+(((warp >> 1) ^ (lane & 7)) << 4)+8*(warp & 1);
	unsigned char *pb = pa+DIGITS*A_BYTES;
	int h = 0;
	for (int t = k0; t < k1; t += SLOTS*KS, h++) {
		uint64_t y[4];
#pragma unroll
		for (int i = 0; i < 4; i++) y[i] = scale_entry(v[i], e);
		load(t+SLOTS*KS);
		if (h > 0 && ok && !mbar_wait(saddr(done), (h-1) & 1)) ok = false;   // the tiles are free again
		store_diag_digits<0>(y, pa, pb);
		asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
		asm volatile("tcgen05.fence::before_thread_sync;");
		ok = __syncthreads_and(ok);
		if (threadIdx.x == 32*MMA_WARP && ok) {
			asm volatile("tcgen05.fence::after_thread_sync;");
			const uint32_t sa = saddr(sm), sb = sa+DIGITS*A_BYTES;
			for (int q = 0; t+q*KS < min(k1, t+SLOTS*KS); q++)
#pragma unroll
				for (int i = 0; i < DIGITS; i++)
					mma_f16(tmem+32*i, sdesc(sa+i*A_BYTES+32*q), sdesc(sb+32*q), idesc(32*(DIGITS-i)),
					        (h > 0 || q > 0 || i > 0) ? 1u : 0u);
			mma_commit(done);
		}
	}
	if (ok && !mbar_wait(saddr(done), (h-1) & 1)) ok = false;
	__syncwarp();
	asm volatile("tcgen05.fence::after_thread_sync;");
	uint32_t a[DIGITS][2];
#pragma unroll
	for (int q = 0; q < DIGITS; q++) tmem_ld2(tmem+((uint32_t)(32*(warp & 3)) << 16)+(uint32_t)(32*q+2*warp), a[q]);
	asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
	for (int j = 0; j < 2; j++) {
		uint32_t o[DIGITS];
#pragma unroll
		for (int q = 0; q < DIGITS; q++) {
			asm volatile("" : "+r"(a[q][j]));   // not used before the wait
			o[q] = a[q][j];
		}
		const int c = 2*warp+j, eb = exps[c];
		const double r = join_orders(o, e+eb);
		C[j] -= max(e, eb) >= 0x7ff ? __longlong_as_double(0x7ff8000000000000ll) : r;   // inf, NaN
		Ls[33*lane+c] = lane < c ? 0.0 : live ? C[j] : lane == c ? 1.0 : 0.0;
	}
	asm volatile("tcgen05.fence::before_thread_sync;");
	return ok;
}

} // namespace split64

// One tile of rows r0 + [0, 128) x columns c0 + [0, TN) per CTA (all THREADS):
// C -= A B^T over the front's columns [k0, k1), A and B rows of the same
// column-major front.  schur: the update matrix, over all pivot columns.
// Otherwise the trailing update after panel k, two-level: inside an outer
// block of OUTER panels only the next panel's columns, over the block's panels
// so far (TN = 32); after its last panel all remaining pivot columns, over the
// whole block (TN = 64).  The launch's first CTAs (c0 < 0), one per front, update
// panel k + 1's diagonal block (diag_tile) and factor and invert it (diag64); the
// tiles leave that block alone.
//
// Producer threads take one row and 8 K entries per K step, scale and cut them
// and write the digits to the step's slot of the 128-byte-swizzled K-major
// shared tiles (a ring of four K steps behind full/empty mbarriers), the next
// step's entries already loading.  One warp multiplies: digit i of A with
// digits 0..7-i of B in one or two instructions (B's digit tiles follow one
// another, so N = TN (8 - i) columns of B land on the accumulators of orders
// i..7).  After a K block all warps read the accumulators, join them and
// subtract from C, in place in the front.
//
// Bound: per K step and 128 x 64 tile the 36 digit products take 1152 tensor
// cycles and read 123 KB of shared memory, the splitting about 900 issue slots
// per scheduler; a K block's epilogue takes about 5k cycles.
template <int TN>
__global__ void __launch_bounds__(split64::THREADS, 1)
k_tile64(const int4 *__restrict__ tasks, const int *__restrict__ sn_n, const int *__restrict__ sn_m,
         const int *__restrict__ sn_ld, const int64_t *__restrict__ sn_off, double *__restrict__ arena,
         const unsigned short *rexp, const unsigned short *yexp, const uint64_t *ybuf,
         const int64_t *__restrict__ split_off, int *fail, int dof, bool schur,
         const int *__restrict__ sn_first, double *__restrict__ linv, int nsn)
{
	using namespace split64;
	constexpr bool SCALED = TN == 64;   // whole K blocks: the panel solves left them scaled
	static_assert(THREADS == DIAG64_THREADS, "diag64 runs in this CTA");
	typedef Tile<TN> T;
	extern __shared__ unsigned char smem_s64[];
	__shared__ __align__(8) Bars bars;
	__shared__ uint32_t tmem_slot;
	__shared__ int expA[2][M], expB[2][TN];
	unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_s64)+1023) &
	                                                      ~static_cast<uintptr_t>(1023));
	// diag64's block and work space, over the digit tiles
	double *Ls = reinterpret_cast<double *>(sm), *ul = Ls+33*32, *zr = ul+2048;
	int *flags = reinterpret_cast<int *>(zr+1056);
	const int tid = threadIdx.x, warp = tid/32, lane = tid%32;
	const int4 tk = tasks[blockIdx.x];
	const int s = tk.x, r0 = tk.y, c0 = tk.z;
	const int n6 = dof*sn_n[s], F6 = n6+dof*sn_m[s], ld = sn_ld[s];
	const int k = tk.w, t0 = min((k+1)*PANEL, n6);   // columns before t0 are solved
	const int k0 = schur ? 0 : k/OUTER*OUTER*PANEL, k1 = schur ? n6 : t0;
	const bool extra = !schur && r0 >= F6;           // identity rows
	const int rlim = extra ? F6+t0 : F6;
	const int clim = schur ? F6 : (k+1) % OUTER ? min(n6, t0+PANEL) : n6;
	const bool diag = c0 < 0, corner = !schur && r0 == t0 && c0 == t0;
	const int w1 = min(PANEL, n6-t0);                // width of panel k + 1
	double *base = arena+sn_off[s];
	const unsigned short *etab = SCALED ? yexp+split_off[3*s+1] : rexp+split_off[3*s];
	const uint64_t *src = SCALED ? ybuf+split_off[3*s+2] : reinterpret_cast<const uint64_t *>(base);
	const int nblk = (k1-k0+KB-1)/KB;
	bool ok = true;
	if (schur) pdl_trigger();   // the next level's assembly reads its indices during the last wave
	pdl_wait();   // before the tensor-memory allocation, too
	if (warp == 0) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
		             :: "r"(saddr(&tmem_slot)), "r"(T::COLS));
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
		asm volatile("tcgen05.fence::before_thread_sync;");
	}
	if (tid == 32) {
		for (int q = 0; q < SLOTS; q++) {
			mbar_init(&bars.full[q], T::PRODUCERS);
			mbar_init(&bars.empty[q], 1);
		}
		mbar_init(&bars.done, 1);
		asm volatile("fence.mbarrier_init.release.cluster;");
	}
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;");
	const uint32_t tmem = tmem_slot;

	// digit products of K step q of a block, once every warp's digits are in
	int gm = 0;   // K steps multiplied so far (MMA warp)
	auto multiply = [&](bool first) {
		if (lane == 0) {
			const uint32_t sa = saddr(sm), sb = sa+DIGITS*A_BYTES;
			const int slot = gm % SLOTS;
			if (ok && !mbar_wait(saddr(&bars.full[slot]), (gm/SLOTS) & 1)) ok = false;
			if (ok) {
				asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
				for (int i = 0; i < DIGITS; i++) {
					const uint64_t da = sdesc(sa+i*A_BYTES+32*slot);
					constexpr int NMAX = 256/TN;   // digits of B per instruction
#pragma unroll
					for (int j = 0; j < DIGITS-i; j += NMAX) {
						const int cnt = DIGITS-i-j < NMAX ? DIGITS-i-j : NMAX;
						mma_f16(tmem+(i+j)*TN, da, sdesc(sb+j*T::B_BYTES+32*slot), idesc(TN*cnt),
						        (!first || i > 0) ? 1u : 0u);
					}
				}
				mma_commit(&bars.empty[slot]);
			}
		}
		gm++;
		__syncwarp();
	};
	if (diag)
		ok = diag_tile(base, ld, t0, w1, k0, k1, F6, n6, rexp+split_off[3*s], sm, &bars.done, tmem, expA[0], Ls);
	else {
		// epilogue role: row er, columns ec + [0, CPW)
		const int er = r0+32*(warp & 3)+lane, el = 32*(warp & 3)+lane, eg = (warp >> 2)*T::CPW, ec = c0+eg;
		// producer role: one row, 8 consecutive K entries of each step
		const bool isA = warp < 2*M/32, producer = tid < T::PRODUCERS;
		const int pt = isA ? tid : tid-2*M;
		const int m = isA ? pt & (M-1) : pt & (TN-1);
		const int kofs = 8*(isA ? pt/M : pt/TN);
		const int row = (isA ? r0 : c0)+m;
		const bool live = producer && row < (isA ? rlim : clim);
		uint64_t v[8];
		auto load = [&](int t) {   // entries of the K step that starts at column t
			const uint64_t *p = src+(int64_t)(t+kofs)*ld+row;
			const int nk = live ? k1-(t+kofs) : 0;
#pragma unroll
			for (int k = 0; k < 8; k++)
				v[k] = k < nk ? p[(int64_t)k*ld] : SCALED ? BIAS : 0;
		};
		// this thread's 16-byte chunk of a slot: chunk column 2 slot + kofs / 8,
		// swizzled by the row
		unsigned char *rowp = (isA ? sm : sm+DIGITS*A_BYTES)+(m >> 3)*1024+(m & 7)*128;
		load(k0);
		int g = 0;   // K steps so far
		for (int kb = 0; kb < nblk; kb++) {
			const int kk0 = k0+kb*KB, kk1 = min(k1, kk0+KB);
			const int e = !live ? MIN_EXP : SCALED ? etab[(int64_t)(kk0/KB)*ld+row]
			                                       : row_exponent(etab, ld, row, F6, n6, kk0/PANEL, (kk1+PANEL-1)/PANEL);
			if (producer && kofs == 0) {
				if (isA) expA[kb & 1][m] = e;
				else expB[kb & 1][m] = e;
			}
			__syncwarp();
			asm volatile("bar.sync 1, 512;" ::: "memory");   // the block's exponents are in
			if (producer)
				for (int t = kk0; t < kk1; t += KS, g++) {
					const int slot = g % SLOTS;
					uint64_t y[8];
#pragma unroll
					for (int k = 0; k < 8; k++) y[k] = SCALED ? v[k] : scale_entry(v[k], e);
					load(t+KS);
					if (g >= SLOTS && ok && !mbar_wait(saddr(&bars.empty[slot]), ((g/SLOTS)-1) & 1)) ok = false;
					store_digits<0>(y, rowp+(((2*slot+(kofs >> 3)) ^ (m & 7)) << 4), isA ? A_BYTES : T::B_BYTES);
					asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // visible to the tensor cores
					asm volatile("tcgen05.fence::before_thread_sync;");
					mbar_arrive(&bars.full[slot]);
				}
			else if (warp == MMA_WARP) {
				for (int t = kk0; t < kk1; t += KS) multiply(t == kk0);
				if (lane == 0) mma_commit(&bars.done);   // everything issued so far
				__syncwarp();
			}
			// epilogue of the block: the old values first, in flight while the
			// MMAs finish
			double C[T::CPW];
			bool in[T::CPW];
#pragma unroll
			for (int j = 0; j < T::CPW; j++) {
				const int c = ec+j;
				in[j] = er < rlim && c < clim && (extra || er >= c) && !(corner && el < w1 && eg+j < w1);
				C[j] = in[j] ? base[(int64_t)c*ld+er] : 0.0;
			}
			if (ok && !mbar_wait(saddr(&bars.done), kb & 1)) ok = false;
			__syncwarp();
			asm volatile("tcgen05.fence::after_thread_sync;");
			const int ea = expA[kb & 1][el];
#pragma unroll
			for (int j0 = 0; j0 < T::CPW; j0 += 4) {
				uint32_t a[DIGITS][4];
#pragma unroll
				for (int q = 0; q < DIGITS; q++)
					tmem_ld4(tmem+((uint32_t)(32*(warp & 3)) << 16)+(uint32_t)(q*TN+eg+j0), a[q]);
				asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
				for (int j = 0; j < 4; j++) {
					uint32_t o[DIGITS];
#pragma unroll
					for (int q = 0; q < DIGITS; q++) {
						asm volatile("" : "+r"(a[q][j]));   // not used before the wait
						o[q] = a[q][j];
					}
					const int eb = expB[kb & 1][eg+j0+j];
					const double r = join_orders(o, ea+eb);
					C[j0+j] -= max(ea, eb) >= 0x7ff ? __longlong_as_double(0x7ff8000000000000ll) : r;   // inf, NaN
				}
			}
			asm volatile("tcgen05.fence::before_thread_sync;");
			if (ok)
#pragma unroll
				for (int j = 0; j < T::CPW; j++)
					if (in[j]) base[(int64_t)(ec+j)*ld+er] = C[j];
		}
	}
	ok = __syncthreads_and(ok);
	if (warp == 0)
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(T::COLS));
	if (!ok && tid == 0 && fail) atomicMin(fail, 0);
	if (diag) {
		if (tid < DIAG64_FLAGS) flags[tid] = 0;
		__syncthreads();
		diag64(base, ld, t0, w1, dof*sn_first[s]+t0, fail, Ls, linv64_slot(linv, nsn, s, k+1), ul, zr, flags);
	}
}

// diagonal block of panel 0 of every front of a level
__global__ void __launch_bounds__(DIAG64_THREADS, 1) k_diag64(const int4 *__restrict__ tasks, const int *__restrict__ sn_first,
                                                const int *__restrict__ sn_ld, const int64_t *__restrict__ sn_off,
                                                double *__restrict__ arena, double *__restrict__ linv, int nsn, int *fail,
                                                int dof)
{
	__shared__ double Ls[33*32], ul[2048], zr[1056];
	__shared__ int flags[DIAG64_FLAGS];
	const int4 tk = tasks[blockIdx.x];
	const int s = tk.x, w = tk.w, ld = sn_ld[s];
	double *base = arena+sn_off[s];
	if (threadIdx.x < DIAG64_FLAGS) flags[threadIdx.x] = 0;
	pdl_wait();
#pragma unroll
	for (int e = threadIdx.x; e < 1024; e += 512) {
		const int i = e%32, j = e/32;
		Ls[33*i+j] = j > i ? 0.0 : i < w ? base[(int64_t)j*ld+i] : i == j ? 1.0 : 0.0;
	}
	__syncthreads();
	diag64(base, ld, 0, w, dof*sn_first[s], fail, Ls, split64::linv64_slot(linv, nsn, s, 0), ul, zr, flags);
}

// Rows below the diagonal block of panel k: X = A Linv_kk^T for up to 16 rows
// per CTA (real and identity rows), in place, and the rows' largest exponents.
// Thread (r, j) takes the entries j and 31 - j of row r: 33 terms together, so
// the eight warps' FP64 instructions (34 each, 64 cycles apiece) are equal.
// Bound by those, 264 cycles a row and SM: 16 rows a CTA put the ~2500 rows of a
// large front on all SMs (64 rows: 40 CTAs of 17k cycles).
constexpr int TRSM64_ROWS = 16;

__global__ void __launch_bounds__(256) k_trsm64(const int4 *__restrict__ tasks, const int *__restrict__ sn_n,
                                                const int *__restrict__ sn_m, const int *__restrict__ sn_ld,
                                                const int64_t *__restrict__ sn_off,
                                                double *__restrict__ arena, const double *linv, int nsn, int dof,
                                                unsigned short *rexp, unsigned short *yexp, uint64_t *ybuf,
                                                const int64_t *__restrict__ split_off)
{
	using namespace split64;
	constexpr int R = TRSM64_ROWS, PREV = (OUTER-1)*PANEL*R/256;   // entries of earlier panels per thread
	__shared__ double Vt[PANEL*PANEL];   // Linv^T, row-major
	__shared__ double As[R][PANEL+1];
	__shared__ int rmax[R];
	const int4 tk = tasks[blockIdx.x];
	const int s = tk.x, row0 = tk.y, k = tk.z, nrows = tk.w;
	const int ld = sn_ld[s], p0 = k*PANEL, w = min(PANEL, dof*sn_n[s]-p0), tid = threadIdx.x;
	double *base = arena+sn_off[s];
	const double *vt = linv64_slot(linv, nsn, s, k);
	if (tid < R) rmax[tid] = 0;
	pdl_trigger();   // the next update's CTAs wait resident while this short launch runs
	pdl_wait();
	// last panel of a K block: its rows' entries in the block's earlier panels,
	// and their exponents (identity rows are zero in panels before their own)
	const int n6 = dof*sn_n[s], kp = k/OUTER*OUTER;
	const bool block_end = k-kp == OUTER-1 || p0+w == n6;
	uint64_t prev[PREV];
	int pe = MIN_EXP;
	if (block_end) {
#pragma unroll
		for (int u = 0; u < PREV; u++) {
			const int t = tid/R+16*u;
			prev[u] = tid%R < nrows && t < (k-kp)*PANEL
			          ? *reinterpret_cast<const uint64_t *>(base+(int64_t)(kp*PANEL+t)*ld+row0+tid%R) : 0;
		}
		if (tid < nrows) pe = row_exponent(rexp+split_off[3*s], ld, row0+tid, n6+dof*sn_m[s], n6, kp, k);
	}
	{
		double lv[4], av[2];
#pragma unroll
		for (int u = 0; u < 4; u++) lv[u] = vt[tid+256*u];
#pragma unroll
		for (int u = 0; u < 2; u++) {
			const int r = tid%R, t = tid/R+16*u;
			av[u] = r < nrows && t < w ? base[(int64_t)(p0+t)*ld+row0+r] : 0.0;
		}
#pragma unroll
		for (int u = 0; u < 4; u++) Vt[tid+256*u] = lv[u];
#pragma unroll
		for (int u = 0; u < 2; u++) As[tid%R][tid/R+16*u] = av[u];
	}
	__syncthreads();
	const int r = tid%R, j = tid/R, i = PANEL-1-j;
	double x = 0, y = 0;
	const int jw = j | 1;   // of the warp's two columns the later one: past its own, Linv^T is zero
#pragma unroll 4
	for (int t = 0; t <= jw; t++) x += As[r][t]*Vt[PANEL*t+j];
#pragma unroll 4
	for (int t = 0; t <= (i | 1); t++) y += As[r][t]*Vt[PANEL*t+i];
	int e = 0;
	if (j < w) e = (__double2hiint(x) >> 20) & 0x7ff;
	if (i < w) e = max(e, (__double2hiint(y) >> 20) & 0x7ff);
	if (r < nrows) {
		if (j < w) base[(int64_t)(p0+j)*ld+row0+r] = x;
		if (i < w) base[(int64_t)(p0+i)*ld+row0+r] = y;
	}
	e = max(e, __shfl_xor_sync(FULL_MASK, e, 16));
	if (tid%32 < R) atomicMax(&rmax[r], e);
	__syncthreads();
	if (tid < nrows) rexp[split_off[3*s]+(int64_t)k*ld+row0+tid] = (unsigned short)rmax[tid];
	if (!block_end) return;
	// the rows of the whole K block as scaled integers, for the trailing update
	// and the Schur complement (scaled once here, not by every tile)
	if (tid < nrows) {
		pe = max(pe, rmax[tid]);
		rmax[tid] = pe;
		yexp[split_off[3*s+1]+(int64_t)(k/OUTER)*ld+row0+tid] = (unsigned short)pe;
	}
	__syncthreads();
	if (r >= nrows) return;
	e = rmax[r];
	uint64_t *yb = ybuf+split_off[3*s+2]+row0+r;
#pragma unroll
	for (int u = 0; u < PREV; u++) {
		const int t = tid/R+16*u;
		if (t < (k-kp)*PANEL) yb[(int64_t)(kp*PANEL+t)*ld] = scale_entry(prev[u], e);
	}
	if (j < w) yb[(int64_t)(p0+j)*ld] = scale_entry((uint64_t)__double_as_longlong(x), e);
	if (i < w) yb[(int64_t)(p0+i)*ld] = scale_entry((uint64_t)__double_as_longlong(y), e);
}

using split64::Tile;

void tile64_setup()
{
	static std::once_flag once;
	std::call_once(once, [] {
		LFG_CUDA(cudaFuncSetAttribute(k_tile64<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<64>::SMEM));
		LFG_CUDA(cudaFuncSetAttribute(k_tile64<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<32>::SMEM));
	});
}

int trsm64_rows() { return TRSM64_ROWS; }

int tile64_kblock() { return split64::KB; }

int tile64_cols(int k) { return (k+1) % split64::OUTER ? 32 : 64; }

void tile64_launch(const DevSymbolic &D, int64_t off, int count, int cols, bool schur, DevFactor<double> &F,
                   cudaStream_t st)
{
	launch_pdl(cols == 32 ? k_tile64<32> : k_tile64<64>, count, split64::THREADS,
	           cols == 32 ? Tile<32>::SMEM : Tile<64>::SMEM, st, (const int4 *)D.tile_tasks+off, (const int *)D.sn_n,
	           (const int *)D.sn_m, (const int *)D.sn_ld, (const int64_t *)D.sn_off, F.arena,
	           (const unsigned short *)F.rexp, (const unsigned short *)F.yexp, (const uint64_t *)F.ybuf,
	           (const int64_t *)D.split_off, F.status, D.dof, schur,
	           (const int *)D.sn_first, F.linv, D.nsn);
}

void trsm64_launch(const DevSymbolic &D, int64_t off, int count, DevFactor<double> &F, cudaStream_t st)
{
	launch_pdl(k_trsm64, count, 256, 0, st, (const int4 *)D.panel_tasks+off, (const int *)D.sn_n, (const int *)D.sn_m,
	           (const int *)D.sn_ld, (const int64_t *)D.sn_off, F.arena, (const double *)F.linv, D.nsn, D.dof, F.rexp, F.yexp,
	           (uint64_t *)F.ybuf,
	           (const int64_t *)D.split_off);
}

void diag64_launch(const DevSymbolic &D, int64_t off, int count, DevFactor<double> &F, cudaStream_t st)
{
	launch_pdl(k_diag64, count, 512, 0, st, (const int4 *)D.diag_tasks+off, (const int *)D.sn_first,
	           (const int *)D.sn_ld, (const int64_t *)D.sn_off, F.arena, F.linv, D.nsn, F.status, D.dof);
}

} // namespace lfg
