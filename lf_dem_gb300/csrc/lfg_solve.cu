// lfg_solve.cu -- solves and products with the multifrontal factor
// (cholmod_solve2, LF_DEM/StokesSolver.cpp:671-703; compute_LTRHS, 627-669).
//
// Solve: forward (leaves first) and backward (root first) sweeps over the
// levels of the assembly tree, for K <= 4 right-hand sides (RHS-major:
// v[r*6n + i], permuted order).  Per level, forward:
//   gather  : v_top (own columns, in xp) = b + children's update vectors;
//             w_s (update rows) = children's update vectors
//   cols 0  : y = E^T v_top            (E = L11^-T, upper triangular)
//   rows 0  : w_s -= L21 y              (+ ordered sum of column chunks)
// backward:
//   cols 1  : z = y - L21^T x[rows of s]
//   rows 1  : x = E z                   (+ ordered sum of column chunks)
// Product y = P^T L P b: per level gather, then x_top += L11 b_top and
// w += L21 b_top in one phase.
// A phase table built with the symbolic analysis lists the phases of a
// sweep; each runs as one launch of k_solve_phase with one CTA per work
// unit, about 1.7 us apart on small systems, so phases are kept few: a front of
// at most SOLVE_WARP_ROWS columns has no gather (its column products gather v_top,
// its row products w), b is read and x written (or added to) in the caller's
// order where the values arise.  Column products take ColsLarge columns per CTA (8
// warps split the rows) or SOLVE_CB per warp, row products 32 rows x SOLVE_JC columns
// (lanes own rows, warps split the columns; the last chunk of a row block to
// finish, found with a per-block counter, adds the chunks' partial sums).  Every
// sum runs in a fixed order: results are bitwise reproducible.  (One launch of
// resident CTAs per sweep was measured slower in FP32: with grid barriers, and
// with units that wait on counters of the units they depend on -- N = 4096 191 us
// against 190, N = 16384 770 us against 605 per iteration.)

// Solve phases read their indices and the first batch of their factor
// entries before pdl_wait, overlapping the previous phase.  A sweep's first phase
// is an ordinary launch: it starts when the factorisation is complete, so the
// factor is constant while any phase runs and its entries may be read through
// the read-only path (a programmatic launch would start while the
// factorisation's last kernel still writes).  Every other access to vectors follows the
// wait (b apart: no launch of a sweep before the backward phases writes it).
#include <algorithm>
#include <type_traits>
#include <vector>
#include <cuda_runtime.h>

#include "lfg_device.cuh"

namespace lfg {

constexpr int SOLVE_WARPS = 8, SOLVE_THREADS = 32*SOLVE_WARPS;
constexpr int SOLVE_CB = 4;      // columns per warp of the column products of few rows
// columns per CTA of the others (FP64: fewer, its products take the FP64 pipe 64 cycles a warp)
template <typename T> struct ColsLarge { static constexpr int CB = sizeof(T) == 4 ? 8 : 4; };
constexpr int SOLVE_JC = 256;    // columns per chunk of the row products
constexpr int SOLVE_WARP_ROWS = 256;   // column products with at most this many rows: one warp per SOLVE_CB columns
// ... and this many such groups per CTA (FP64: one warp per scheduler, whose
// FP64 pipe it fills)
template <typename T> struct ColGroups { static constexpr int G = sizeof(T) == 4 ? 8 : 4; };

enum { SP_GATHER, SP_COLS0, SP_ROWS0, SP_COLS1, SP_ROWS1, SP_MUL_GATHER, SP_MUL_TOP, SP_MUL_UPD };

template <typename T> struct SolveArgs {
	const FrontRec *fronts;
	const ChildRec *childs;
	const int *rows, *cinv, *perm;
	const T *arena;
	T *w, *xp, *yp, *part;
	int *tally;
	int64_t wstride, pstride, w_elems;
	int n, n6tot, dof;   // particles, scalar unknowns (dof n), unknowns per particle
	int add;             // x += solution instead of x = solution
	const double *b;
	double *x;
};

// a CTA's share of a phase: row block or column group bx of front by of the
// level, column chunk bz of nchunk
struct SolveUnit { int bx, by, bz; };

static_assert(SOLVE_WARP_ROWS == SOLVE_THREADS, "a thread gathers a row");
template <typename T> union SolveShared {
	T red_c[SOLVE_WARPS][ColsLarge<T>::CB*4];
	T xs[4*SOLVE_WARP_ROWS];
	T red_r[SOLVE_WARPS][4][32];
};

// particle and component (of 6) of scalar unknown g
template <typename T>
__device__ __forceinline__ int caller_index(const SolveArgs<T> &A, int g)
{
	const int i = __ldg(A.perm+bdiv(g, A.dof)), d = bmod(g, A.dof);
	return 6*i+(A.dof == 6 ? d : 2*d);
}

// b and x keep 6 values per particle; with dof 3 only components 0, 2, 4 (x, z
// translation, y rotation) are unknowns: the others of b are not read and
// those of x are written as 0.
template <typename T>
__device__ __forceinline__ void store_x(const SolveArgs<T> &A, int q, int c, T a)
{
	double *x = A.x+(int64_t)q*6*A.n+c;
	if (A.add) *x += (double)a;
	else {
		*x = (double)a;
		if (A.dof == 3) x[1] = 0.0;
	}
}

// The children's update vectors summed at row r of a front, in child order.
// The first children's source positions (symbolic) are read before the wait.
template <typename T, int K> struct ChildSum {
	static constexpr int CPRE = 2;
	int64_t src[CPRE];
	__device__ __forceinline__ void prefetch(const SolveArgs<T> &A, const FrontRec &f, int r, bool valid)
	{
		const int rb = bdiv(r, A.dof), rr = bmod(r, A.dof);
#pragma unroll
		for (int c = 0; c < CPRE; c++) {
			src[c] = -1;
			if (valid && f.ca+c < f.cz) src[c] = source(A, f.ca+c, rb, rr);
		}
	}
	__device__ __forceinline__ void add(const SolveArgs<T> &A, const FrontRec &f, int r, bool valid, T (&acc)[K]) const
	{
#pragma unroll
		for (int q = 0; q < K; q++) acc[q] = 0;
#pragma unroll
		for (int c = 0; c < CPRE; c++)
			if (src[c] >= 0)
#pragma unroll
				for (int q = 0; q < K; q++) acc[q] += A.w[q*A.wstride+src[c]];
		if (!valid) return;
		for (int c = f.ca+CPRE; c < f.cz; c++) {
			const int64_t sc = source(A, c, bdiv(r, A.dof), bmod(r, A.dof));
			if (sc < 0) continue;
#pragma unroll
			for (int q = 0; q < K; q++) acc[q] += A.w[q*A.wstride+sc];
		}
	}
	static __device__ __forceinline__ int64_t source(const SolveArgs<T> &A, int ch, int rb, int rr)
	{
		const ChildRec g = load_record(A.childs+ch);
		const int ic = __ldg(A.cinv+g.cinv_off+rb);
		return ic < 0 ? -1 : g.woff+A.dof*(ic-g.n)+rr;
	}
};

template <typename T, int K, bool MUL>
__device__ void unit_gather(const SolveArgs<T> &A, const FrontRec &f, const SolveUnit &u)
{
	const int n6 = f.n6, r = u.bx*SOLVE_THREADS+threadIdx.x;
	if (!MUL && n6 > 0 && n6 <= SOLVE_WARP_ROWS) return;   // gathered by its column and row products
	const bool valid = r < f.n6+f.m6;
	ChildSum<T, K> cs;
	cs.prefetch(A, f, r, valid);
	T acc[K], top[K];
	if (r < n6) {
		const int c = caller_index(A, f.f6+r);
#pragma unroll
		for (int q = 0; q < K; q++) top[q] = (T)A.b[(int64_t)q*6*A.n+c];
	}
	pdl_wait();   // before the first access to what earlier phases write
	cs.add(A, f, r, valid, acc);
	if (valid) {
#pragma unroll
		for (int q = 0; q < K; q++) {
			if (r >= n6) A.w[q*A.wstride+f.woff+(r-n6)] = acc[q];
			else {
				const int64_t g = (int64_t)q*A.n6tot+f.f6+r;
				A.xp[g] = MUL ? acc[q] : top[q]+acc[q];
				if (MUL) A.yp[g] = top[q];
			}
		}
	}
}

// MODE 0: y_j = sum_{i <= j} E[i][j] x_i;  MODE 1: z_j -= sum_t L21[t][j] x[rows(t)]
// A thread takes U rows of CB columns per batch: all their loads are
// issued before the first multiply-add (the units are latency-bound: one
// round trip per batch), those of the first batch before the wait; each thread
// adds its rows in increasing order.
template <typename T, int K, int CB> struct SolveUnroll {
	static constexpr int U = (sizeof(T) == 4 ? 32 : 16)/CB/(K == 1 ? 1 : 2);   // rows of a column product
	static constexpr int RU = sizeof(T) == 8 && K == 1 ? 16 : 8;                                              // columns of a row product
};

// one batch of a column product's rows: their positions in xp or, where the
// sums read xs (a front's own rows), in xs (g < 0 past the rows), and factor
// entries
template <typename T, int U, int CB, int MODE>
__device__ __forceinline__ void cols_batch(int i0, int nrow, int g0, const int *R, const T *M, int ld, int j0, int jn,
                                           int dof, int (&g)[U], T (&e)[U][CB], int stride)
{
#pragma unroll
	for (int u = 0; u < U; u++) {
		int i = i0+u*stride;
		g[u] = i >= nrow ? -1 : MODE == 0 ? g0+i : dof*R[bdiv(i, dof)]+bmod(i, dof);
#pragma unroll
		for (int c = 0; c < CB; c++)
			e[u][c] = (i >= nrow || c >= jn || (MODE == 0 && i > j0+c)) ? T(0) : __ldg(&M[(int64_t)c*ld+i]);
	}
}

// The sums of CB columns over rows first, first + stride, ... of a front.
// xs: its own rows are in shared memory once ready() has returned, otherwise
// in xp.
template <typename T, int K, int CB, int MODE, typename Ready>
__device__ __forceinline__ void cols_sums(const SolveArgs<T> &A, const FrontRec &f, int j0, int first, int stride,
                                          T (&acc)[CB*K], const T *xs, const Ready &ready)
{
	constexpr int U = SolveUnroll<T, K, CB>::U;
	const int dof = A.dof;
	const int jn = min(CB, f.n6-j0);   // <= 0: a warp past the columns
	const T *M = A.arena+f.off+(MODE == 0 ? f.n6+f.m6 : f.n6)+(int64_t)j0*f.ld;
	const int *R = A.rows+f.rows_off;
	const int nrow = jn <= 0 ? 0 : MODE == 0 ? j0+jn : f.m6, g0 = xs ? 0 : f.f6;
#pragma unroll
	for (int v = 0; v < CB*K; v++) acc[v] = 0;
	int g[U];
	T e[U][CB];
	cols_batch<T, U, CB, MODE>(first, nrow, g0, R, M, f.ld, j0, jn, dof, g, e, stride);
	ready();
	for (int i0 = first; i0 < nrow; i0 += U*stride) {
		T v[U][K];
#pragma unroll
		for (int u = 0; u < U; u++)
#pragma unroll
			for (int q = 0; q < K; q++)
				v[u][q] = g[u] < 0 ? T(0) : xs ? xs[q*SOLVE_WARP_ROWS+g[u]] : A.xp[(int64_t)q*A.n6tot+g[u]];
#pragma unroll
		for (int u = 0; u < U; u++) {
			if (g[u] < 0) continue;
			int i = i0+u*stride;
#pragma unroll
			for (int c = 0; c < CB; c++) {
				if (c >= jn || (MODE == 0 && i > j0+c)) continue;
#pragma unroll
				for (int q = 0; q < K; q++) acc[c*K+q] += e[u][c]*v[u][q];
			}
		}
		int i1 = i0+U*stride;
		if (i1 < nrow) cols_batch<T, U, CB, MODE>(i1, nrow, g0, R, M, f.ld, j0, jn, dof, g, e, stride);
	}
}

// The NV sums of a warp's lanes, sum i in lanes i LG ... (LG = SumLanes):
// a butterfly reduce-scatter over the lane bits from the highest down; while a
// lane holds several values it keeps the half whose index bit matches its lane
// bit.  A sum's order does not depend on NV.
template <int NV> struct SumLanes { static constexpr int LG = 32/(NV <= 4 ? 4 : NV <= 8 ? 8 : NV <= 16 ? 16 : 32); };

template <typename T, int NV>
__device__ __forceinline__ T warp_scatter_sums(const T (&v)[NV], int lane)
{
	constexpr int LG = SumLanes<NV>::LG, NVP = 32/LG;   // padded to a power of two
	static_assert(NV <= 32, "one sum per lane");
	T acc[NVP];
#pragma unroll
	for (int i = 0; i < NVP; i++) acc[i] = i < NV ? v[i < NV ? i : 0] : T(0);
#pragma unroll
	for (int t = 0; t < 5; t++) {
		const int w = 16 >> t, h = NVP >> (t+1);
		const bool upper = (lane & w) != 0;
		if (h == 0) acc[0] += __shfl_xor_sync(FULL_MASK, acc[0], w);
#pragma unroll
		for (int i = 0; i < NVP/2; i++)
			if (i < h) {
				T mine = upper ? acc[i+h] : acc[i];
				T other = upper ? acc[i] : acc[i+h];
				acc[i] = mine+__shfl_xor_sync(FULL_MASK, other, w);
			}
	}
	return acc[0];
}

template <typename T, int MODE>
__device__ __forceinline__ void cols_apply(const SolveArgs<T> &A, int q, int j, T a)
{
	T *o = A.yp+(int64_t)q*A.n6tot+j;
	if (MODE == 0) *o = a;
	else *o = *o-a;
}

template <typename T, int K, int MODE>
__device__ void unit_cols(const SolveArgs<T> &A, const FrontRec &f, const SolveUnit &un, SolveShared<T> &sh)
{
	const int j0 = un.bx*ColsLarge<T>::CB, jn = min(ColsLarge<T>::CB, f.n6-j0);
	if (j0 >= f.n6) return;
	T acc[ColsLarge<T>::CB*K];
	cols_sums<T, K, ColsLarge<T>::CB, MODE>(A, f, j0, threadIdx.x, SOLVE_THREADS, acc, nullptr, [&]() { pdl_wait(); });
	const int warp = threadIdx.x/32, lane = threadIdx.x%32;
	const T a = warp_scatter_sums(acc, lane);
	constexpr int LG = SumLanes<ColsLarge<T>::CB*K>::LG;
	if (lane%LG == 0 && lane/LG < ColsLarge<T>::CB*K) sh.red_c[warp][lane/LG] = a;
	__syncthreads();
	if (warp) return;
	if (lane < ColsLarge<T>::CB*K && lane/K < jn) {
		T b = 0;
#pragma unroll
		for (int u = 0; u < SOLVE_WARPS; u++) b += sh.red_c[u][lane];
		cols_apply<T, MODE>(A, lane%K, f.f6+j0+lane/K, b);
	}
}

// The same column products with one warp per SOLVE_CB columns, COL_GROUPS such
// groups of a front per unit, for fronts whose products have few rows (at most
// SOLVE_WARP_ROWS).  Forward, such a front has no gather of its own: the unit
// gathers v_top into shared memory, the row products gather w.
template <typename T, int K, int MODE>
__device__ void unit_cols_warp(const SolveArgs<T> &A, const FrontRec &f, const SolveUnit &un, SolveShared<T> &sh)
{
	const int warp = threadIdx.x/32, lane = threadIdx.x%32;
	if (un.bx*ColGroups<T>::G*SOLVE_CB >= f.n6 || (MODE == 1 && f.m6 == 0)) return;
	const int j0 = warp < ColGroups<T>::G ? (un.bx*ColGroups<T>::G+warp)*SOLVE_CB : f.n6;
	T acc[SOLVE_CB*K];
	ChildSum<T, K> cs;
	T top[K];
	const int r = threadIdx.x;
	const bool own = MODE == 0 && r < f.n6;
	if (MODE == 0) {
		cs.prefetch(A, f, r, own);
		const int c = own ? caller_index(A, f.f6+r) : 0;
#pragma unroll
		for (int q = 0; q < K; q++) top[q] = own ? (T)A.b[(int64_t)q*6*A.n+c] : T(0);
	}
	cols_sums<T, K, SOLVE_CB, MODE>(A, f, j0, lane, 32, acc, MODE == 0 ? sh.xs : nullptr, [&]() {
		pdl_wait();
		if (MODE == 0) {
			T v[K];
			cs.add(A, f, r, own, v);
#pragma unroll
			for (int q = 0; q < K; q++) sh.xs[q*SOLVE_WARP_ROWS+r] = top[q]+v[q];
			__syncthreads();
		}
	});
	const T a = warp_scatter_sums(acc, lane);
	constexpr int LG = SumLanes<SOLVE_CB*K>::LG;
	const int v = lane/LG;
	if (lane%LG == 0 && v < SOLVE_CB*K && j0+v/K < f.n6) cols_apply<T, MODE>(A, v%K, f.f6+j0+v/K, a);
}

// a row product's result for row r of a front's update rows (w0: what they
// hold before) or own rows
template <typename T, int TYPE>
__device__ inline void rows_apply(const SolveArgs<T> &A, const FrontRec &f, int q, int r, int c, T w0, T a)
{
	if (TYPE == SP_ROWS0 || TYPE == SP_MUL_UPD) A.w[q*A.wstride+f.woff+r] = TYPE == SP_ROWS0 ? w0-a : w0+a;
	else {
		T *x = A.xp+(int64_t)q*A.n6tot+f.f6+r;
		if (TYPE == SP_MUL_TOP) a += *x;
		else *x = a;
		store_x(A, q, c, a);
	}
}

// SP_ROWS0: w_t -= sum_j L21[t][j] y_j;  SP_ROWS1: x_i = sum_{j >= i} E[i][j] z_j
// (product with L, y in yp): SP_MUL_TOP: x_i += sum_{j <= i} L11[i][j] y_j;
// SP_MUL_UPD: w_t += sum_j L21[t][j] y_j
// A CTA takes 32 rows (a lane each) and SOLVE_JC columns (split over its warps).
template <typename T, int K, int TYPE>
__device__ void unit_rows(const SolveArgs<T> &A, const FrontRec &f, const SolveUnit &un, SolveShared<T> &sh)
{
	constexpr bool UPD = TYPE == SP_ROWS0 || TYPE == SP_MUL_UPD;   // rows of the update block (w)
	const int warp = threadIdx.x/32, lane = threadIdx.x%32, r0 = un.bx*32;
	const int nrows = UPD ? f.m6 : f.n6;
	const int ncol = TYPE == SP_ROWS1 ? f.n6-r0 : TYPE == SP_MUL_TOP ? min(r0+32, f.n6) : f.n6;
	const int nchunk = (ncol+SOLVE_JC-1)/SOLVE_JC;
	if (r0 >= nrows || un.bz >= nchunk) return;
	const int jlo = (TYPE == SP_ROWS1 ? r0 : 0)+un.bz*SOLVE_JC;
	const int jhi = min(f.n6, jlo+SOLVE_JC);
	const T *M = A.arena+f.off+(UPD ? f.n6 : TYPE == SP_ROWS1 ? f.n6+f.m6 : 0);
	const int r = r0+lane, ld = f.ld;
	T acc[K];
#pragma unroll
	for (int q = 0; q < K; q++) acc[q] = 0;
	// RU columns of a warp per batch, the factor entries of the first batch
	// before the wait, loads ahead of the multiply-adds (see cols_sums).
	// Unmasked by the triangle: column j < n6 of a front is allocated down
	// to its last row (the masked product skips it).
	constexpr int RU = SolveUnroll<T, K, SOLVE_CB>::RU;
	T e[RU];
	int jb = jlo+warp;
#pragma unroll
	for (int u = 0; u < RU; u++) {
		int j = jb+u*SOLVE_WARPS;
		e[u] = (r < nrows && j < jhi) ? __ldg(&M[(int64_t)j*ld+r]) : T(0);
	}
	const bool mine = warp == 0 && r < nrows, inl = TYPE == SP_ROWS0 && f.n6 <= SOLVE_WARP_ROWS;
	const int c = !UPD && mine ? caller_index(A, f.f6+r) : 0;
	ChildSum<T, K> cs;
	cs.prefetch(A, f, f.n6+r, inl && mine);
	pdl_wait();
	T w0[K];
	cs.add(A, f, f.n6+r, inl && mine, w0);
	if (UPD && !inl && mine)
#pragma unroll
		for (int q = 0; q < K; q++) w0[q] = A.w[q*A.wstride+f.woff+r];
	if (r < nrows) {
		for (int j0 = jb; j0 < jhi; j0 += RU*SOLVE_WARPS) {
			T y[RU][K];
#pragma unroll
			for (int u = 0; u < RU; u++) {
				int j = j0+u*SOLVE_WARPS;
#pragma unroll
				for (int q = 0; q < K; q++) y[u][q] = j < jhi ? A.yp[(int64_t)q*A.n6tot+f.f6+j] : T(0);
			}
#pragma unroll
			for (int u = 0; u < RU; u++) {
				int j = j0+u*SOLVE_WARPS;
				if (j >= jhi || (TYPE == SP_ROWS1 && j < r) || (TYPE == SP_MUL_TOP && j > r)) continue;
#pragma unroll
				for (int q = 0; q < K; q++) acc[q] += e[u]*y[u][q];
			}
			int j1 = j0+RU*SOLVE_WARPS;
			if (j1 < jhi)
#pragma unroll
				for (int u = 0; u < RU; u++) {
					int j = j1+u*SOLVE_WARPS;
					e[u] = j < jhi ? __ldg(&M[(int64_t)j*ld+r]) : T(0);
				}
		}
	}
#pragma unroll
	for (int q = 0; q < K; q++) sh.red_r[warp][q][lane] = acc[q];
	__syncthreads();
	if (warp) return;
	if (mine)
#pragma unroll
		for (int q = 0; q < K; q++)
#pragma unroll
			for (int u = 1; u < SOLVE_WARPS; u++) acc[q] += sh.red_r[u][q][lane];
	if (nchunk > 1) {
		// The chunk that completes this row block adds the chunks' partial
		// sums in chunk order (the count releases this chunk's partial sums
		// and acquires the others').
		const int64_t row = UPD ? f.woff+r : A.w_elems+f.f6+r;
		if (mine)
#pragma unroll
			for (int q = 0; q < K; q++) A.part[((int64_t)q*nchunk+un.bz)*A.pstride+row] = acc[q];
		__syncwarp();
		int last = 0;
		if (lane == 0) {
			int *cnt = A.tally+(int64_t)un.by*gridDim.x+blockIdx.x;
			asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(last) : "l"(cnt) : "memory");
			last = last == nchunk-1;
			if (last) *cnt = 0;   // ready for the next phase of row products
		}
		if (!__shfl_sync(FULL_MASK, last, 0)) return;
		if (mine)
#pragma unroll
			for (int q = 0; q < K; q++) {
				acc[q] = 0;
#pragma unroll 8
				for (int ch = 0; ch < nchunk; ch++) acc[q] += __ldcg(&A.part[((int64_t)q*nchunk+ch)*A.pstride+row]);
			}
	}
	if (mine)
#pragma unroll
		for (int q = 0; q < K; q++) rows_apply<T, TYPE>(A, f, q, r, c, w0[q], acc[q]);
}


// One phase as its own launch; one instantiation per phase type, so each gets
// its own register budget.  CTAS resident per SM: fewer leave the compiler the
// registers to issue a batch's loads together, more keep the large levels' memory
// traffic up.  A solve at 2, at (4 for K = 1, 3 otherwise), left to the compiler:
// FP32 K = 1 N = 16384 1650, 1572, 1534 us, K = 4 N = 2047 676, 681, 814, N = 4096
// 1144, 1140, 1422, N = 16384 3486, 3265, 3483; FP64 K = 1 N = 4096 368 at 2, 392
// left to the compiler, K = 4 840, 874.
template <typename T, int K> struct SolveBound { static constexpr int CTAS = sizeof(T) == 8 ? 2 : K == 1 ? 4 : 3; };

template <typename T, int K, int TYPE>
__global__ void __launch_bounds__(SOLVE_THREADS, SolveBound<T, K>::CTAS) k_solve_phase(SolveArgs<T> A, SolvePhase ph)
{
	__shared__ SolveShared<T> sh;
	const SolveUnit u{(int)blockIdx.x, (int)blockIdx.y, (int)blockIdx.z};
	pdl_trigger();
	const FrontRec f = load_record(A.fronts+ph.lev_off+u.by);
	if (TYPE == SP_GATHER) unit_gather<T, K, false>(A, f, u);
	if (TYPE == SP_COLS0) {
		if (f.n6 <= SOLVE_WARP_ROWS) unit_cols_warp<T, K, 0>(A, f, u, sh);
		else unit_cols<T, K, 0>(A, f, u, sh);
	}
	if (TYPE == SP_COLS1) {
		if (f.m6 <= SOLVE_WARP_ROWS) unit_cols_warp<T, K, 1>(A, f, u, sh);
		else unit_cols<T, K, 1>(A, f, u, sh);
	}
	if (TYPE == SP_ROWS0) unit_rows<T, K, SP_ROWS0>(A, f, u, sh);
	if (TYPE == SP_ROWS1) unit_rows<T, K, SP_ROWS1>(A, f, u, sh);
	if (TYPE == SP_MUL_GATHER) unit_gather<T, K, true>(A, f, u);
	if (TYPE == SP_MUL_TOP) {   // ph.split row blocks of the update rows, then the own rows
		SolveUnit v = u;
		v.bx -= ph.split;
		if (v.bx >= 0) unit_rows<T, K, SP_MUL_TOP>(A, f, v, sh);
		else unit_rows<T, K, SP_MUL_UPD>(A, f, u, sh);
	}
}

template <typename T, int K>
static void launch_phase(const SolveArgs<T> &A, const SolvePhase &p, cudaStream_t st)
{
	const dim3 g(p.gx, p.gy, p.gz), t(SOLVE_THREADS);
	auto launch = [&](auto kern) {
		if (p.first) kern<<<g, t, 0, st>>>(A, p);
		else launch_pdl(kern, g, t, 0, st, A, p);
	};
	switch (p.type) {
	case SP_GATHER: launch(k_solve_phase<T, K, SP_GATHER>); break;
	case SP_COLS0: launch(k_solve_phase<T, K, SP_COLS0>); break;
	case SP_ROWS0: launch(k_solve_phase<T, K, SP_ROWS0>); break;
	case SP_COLS1: launch(k_solve_phase<T, K, SP_COLS1>); break;
	case SP_ROWS1: launch(k_solve_phase<T, K, SP_ROWS1>); break;
	case SP_MUL_GATHER: launch(k_solve_phase<T, K, SP_MUL_GATHER>); break;
	default: launch(k_solve_phase<T, K, SP_MUL_TOP>); break;
	}
}

// Phase tables of a solve (forward levels leaves first, backward levels root
// first) and of a product; a phase's grid covers the largest extents of its
// level's fronts.
void solve_plan_build(DevSymbolic &D, const Symbolic &S, int precision)
{
	const int dof = S.dof, groups = precision == LFG_PREC_FP64 ? ColGroups<double>::G : ColGroups<float>::G;
	const int large = precision == LFG_PREC_FP64 ? ColsLarge<double>::CB : ColsLarge<float>::CB;
	auto cdiv = [](int a, int b) { return (a+b-1)/b; };
	auto cols = [&](int n6, int rows) { return cdiv(n6, rows <= SOLVE_WARP_ROWS ? SOLVE_CB*groups : large); };
	struct Level { int off, cnt, gather, mgather, cols0, cols1, rows0, rows1, chunks; };
	std::vector<Level> lev;
	for (int l = 0; l < S.nlevels; l++) {
		Level v{S.level_off[l], S.level_off[l+1]-S.level_off[l], 0, 0, 0, 0, 0, 0, 0};
		for (int t = 0; t < v.cnt; t++) {
			const int s = S.level_sn[v.off+t], n6 = dof*S.sn_n[s], m6 = dof*S.sn_m[s];
			v.mgather = std::max(v.mgather, cdiv(n6+m6, SOLVE_THREADS));
			if (n6 == 0 || n6 > SOLVE_WARP_ROWS) v.gather = std::max(v.gather, cdiv(n6+m6, SOLVE_THREADS));
			v.cols0 = std::max(v.cols0, cols(n6, n6));
			if (m6 > 0) v.cols1 = std::max(v.cols1, cols(n6, m6));
			if (n6 > 0) v.rows0 = std::max(v.rows0, cdiv(m6, 32));
			v.rows1 = std::max(v.rows1, cdiv(n6, 32));
			v.chunks = std::max(v.chunks, cdiv(n6, SOLVE_JC));
		}
		lev.push_back(v);
	}
	std::vector<SolvePhase> *P;
	auto add = [&](int type, const Level &v, int gx, int gz, int split = 0) {
		if (gx > 0 && v.cnt > 0 && gz > 0) P->push_back(SolvePhase{type, v.off, gx, v.cnt, gz, P->empty() ? 1 : 0, split});
	};
	P = &D.h_solve_phases;
	for (const Level &v : lev) {
		add(SP_GATHER, v, v.gather, 1);
		add(SP_COLS0, v, v.cols0, 1);
		add(SP_ROWS0, v, v.rows0, v.chunks);
	}
	for (auto v = lev.rbegin(); v != lev.rend(); ++v) {
		add(SP_COLS1, *v, v->cols1, 1);
		add(SP_ROWS1, *v, v->rows1, v->chunks);
	}
	P = &D.h_mul_phases;
	for (const Level &v : lev) {
		add(SP_MUL_GATHER, v, v.mgather, 1);
		add(SP_MUL_TOP, v, v.rows0+v.rows1, v.chunks, v.rows0);
	}
}

template <typename T> void solve_alloc(DevFactor<T> &F, const DevSymbolic &D, int kmax)
{
	// partial sums of the update rows, then of the own rows
	F.pstride = D.w_elems+(int64_t)D.dof*D.nblk;
	device_grow(F.part, F.part_cap, (int64_t)kmax*((D.max_n6+SOLVE_JC-1)/SOLVE_JC)*F.pstride);
	int64_t tneed = 1;
	for (const auto *tab : {&D.h_solve_phases, &D.h_mul_phases})
		for (const SolvePhase &p : *tab)
			if (p.gz > 1) tneed = std::max<int64_t>(tneed, (int64_t)p.gx*p.gy);
	if (F.tally_cap < tneed) {
		device_grow(F.tally, F.tally_cap, tneed);
		LFG_CUDA(cudaMemset(F.tally, 0, sizeof(int)*tneed));
	}
}

template <typename T, int K>
static int sweep(DevFactor<T> &F, const DevSymbolic &D, const std::vector<SolvePhase> &phases, const double *b, double *x,
                 bool add, cudaStream_t st)
{
	SolveArgs<T> A;
	A.fronts = D.fronts;
	A.childs = D.child_recs; A.rows = D.rows; A.cinv = D.cinv; A.perm = D.perm;
	A.arena = F.arena; A.w = F.w; A.xp = F.xp; A.yp = F.yp; A.part = F.part; A.tally = F.tally;
	A.wstride = A.w_elems = D.w_elems; A.pstride = F.pstride; A.n = D.nblk; A.n6tot = D.dof*D.nblk; A.dof = D.dof;
	A.add = add; A.b = b; A.x = x;
	for (const SolvePhase &p : phases) launch_phase<T, K>(A, p, st);
	LFG_CUDA(cudaGetLastError());
	return (int)phases.size();
}

template <typename T>
static int run_sweeps(DevFactor<T> &F, const DevSymbolic &D, const std::vector<SolvePhase> &ph, int k, const double *b,
                      double *x, bool add, cudaStream_t st)
{
	int launches = 0;
	for (int r0 = 0; r0 < k; r0 += 4) {
		const double *bb = b+(int64_t)r0*6*D.nblk;
		double *xx = x+(int64_t)r0*6*D.nblk;
		switch (std::min(4, k-r0)) {
		case 1: launches += sweep<T, 1>(F, D, ph, bb, xx, add, st); break;
		case 2: launches += sweep<T, 2>(F, D, ph, bb, xx, add, st); break;
		case 3: launches += sweep<T, 3>(F, D, ph, bb, xx, add, st); break;
		default: launches += sweep<T, 4>(F, D, ph, bb, xx, add, st); break;
		}
	}
	return launches;
}

template <typename T>
int factor_solve(DevFactor<T> &F, const DevSymbolic &D, int k, const double *b, double *x, bool add, cudaStream_t st)
{
	return run_sweeps(F, D, D.h_solve_phases, k, b, x, add, st);
}

// y = L b with the factor (R = L L^T in the caller's order): StokesSolver::
// compute_LTRHS (StokesSolver.cpp:627-669) for the Brownian force
template <typename T>
int factor_multiply(DevFactor<T> &F, const DevSymbolic &D, int k, const double *b, double *x, cudaStream_t st)
{
	return run_sweeps(F, D, D.h_mul_phases, k, b, x, false, st);
}

template void solve_alloc<double>(DevFactor<double> &, const DevSymbolic &, int);
template void solve_alloc<float>(DevFactor<float> &, const DevSymbolic &, int);
template int factor_solve<double>(DevFactor<double> &, const DevSymbolic &, int, const double *, double *, bool, cudaStream_t);
template int factor_solve<float>(DevFactor<float> &, const DevSymbolic &, int, const double *, double *, bool, cudaStream_t);
template int factor_multiply<double>(DevFactor<double> &, const DevSymbolic &, int, const double *, double *, cudaStream_t);
template int factor_multiply<float>(DevFactor<float> &, const DevSymbolic &, int, const double *, double *, cudaStream_t);

} // namespace lfg
