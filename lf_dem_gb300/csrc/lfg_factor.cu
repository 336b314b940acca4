// lfg_factor.cu -- device multifrontal Cholesky of R_FU (replaces CHOLMOD's
// supernodal cholmod_factorize, LF_DEM/StokesSolver.cpp:950-978), in FP64 ("plain
// form") or FP32 (factor of the FP32 + FP64-refinement form): the assembly of both
// (FP64 panels: lfg_factor64.cu), the FP32 panels and Schur complements (two-level
// updates of large fronts: lfg_factor32.cu), and the refinement's FP64 residual.
//
// Front layout: supernode s with n (own) and m (below) block columns has a
// dense column-major front of 6F x ... (F = n + m) with leading dimension
// ld = 6F + 6n.  Rows [6F, 6F + 6n) are an appended identity block: the same
// panel triangular solves that produce L21 = A21 L11^-T turn it into
// E = L11^-T, so both triangular solves become parallel matrix-vector
// products.  Columns [0, 6n) hold L after factorisation; the lower triangle
// of rows/columns [6n, 6F) holds the update (Schur complement) matrix that the
// parent gathers.
//
// Per level of the assembly tree (leaves first):
//   assemble  : gather children's update matrices (fixed child order), add the
//               compact D / OD blocks of the level's columns,
//   diag      : factor and invert panel 0's diagonal block (one CTA per front);
//               panel k + 1's is done inside update k by the tile that holds it,
//   trsm k    : rows below it (real rows and identity rows) times Linv^T,
//   update k  : trailing rank-w update of the front's own columns (tiles),
//   syrk      : the update (Schur complement) matrix, one deep-K product.
// Atomics touch the failure flag, exponents' maxima and progress counters only,
// never a sum, so results are bitwise reproducible run to run.
#include <atomic>
#include <type_traits>
#include <cstdio>
#include <mutex>
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "lfg_device.cuh"

namespace lfg {

template <typename T> struct Cfg;
// NB: panel width; TILE/TPT: trailing-update tile edge / outputs per thread
// per dimension
template <> struct Cfg<double> { static constexpr int NB = 32; };
template <> struct Cfg<float>  { static constexpr int NB = 64, TILE = 64, TPT = 4; };

// ---------------------------------------------------------------------------
// compact blocks (StokesSolver.cpp:154-231)
// ---------------------------------------------------------------------------
// Dense position r*6+c of a compact block: 0 = structural zero, otherwise
// +-(index+1) into the compact storage.  DSYM is the full symmetric diagonal
// block of the 15-value storage, ODENSE the 18-value off-diagonal block.
__constant__ signed char c_dsym[36] = {1, 2, 3, 0, 4, 5, 2, 6, 7, -4, 0, 8, 3, 7, 9, -5, -8, 0,
                                       0, -4, -5, 10, 11, 12, 4, 0, -8, 11, 13, 14, 5, 8, 0, 12, 14, 15};
__constant__ signed char c_odense[36] = {1, 2, 3, 0, -10, -11, 2, 6, 7, 10, 0, -15, 3, 7, 9, 11, 15, 0,
                                         0, -4, -5, 12, 13, 14, 4, 0, -8, 13, 16, 17, 5, 8, 0, 14, 17, 18};

// ---------------------------------------------------------------------------
// assembly
// ---------------------------------------------------------------------------
// A front's own and update columns: the sum over its children, in child order, of
// the update-matrix entries that land there, plus R's blocks; identity rows below.
// One CTA (blockIdx.y: of several that share it) per block column of DOF scalar
// columns; a thread takes ASM_ROWS rows of it per pass.  A row's source in a child
// is found through the parent -> child map, so a pass is one round trip for the
// indices and one for the entries of two children, all in flight together, and
// nothing is staged.  (One CTA or warp per scalar column, adding the children's
// columns up in shared memory, and a launch of its own for R's blocks were bound by
// the chains of index loads: 31 + 3 us a level at N = 4096.)
constexpr int ASM_THREADS = 128, ASM_ROWS = 2;

template <typename T, int DOF>
__global__ void __launch_bounds__(ASM_THREADS)
k_assemble(const int2 *__restrict__ tasks, const FrontRec *__restrict__ fronts, const ChildRec *__restrict__ childs,
           const int *__restrict__ cinv, const int *__restrict__ perm, const int *__restrict__ col_off,
           const int *__restrict__ col_e, const int *__restrict__ col_br, const double *dbl, const double *odbl, T *arena,
           int *status)
{
	pdl_trigger();   // the next launch (the level's diagonal blocks) is short of CTAs: they wait resident
	const int2 task = __ldg(tasks+blockIdx.x);
	const FrontRec f = load_record(fronts+task.x);
	const int cb = task.y, c0 = DOF*cb, F6 = f.n6+f.m6;
	const bool own = c0 < f.n6;
	const int q = f.f6/DOF+cb, a0 = own ? __ldg(col_off+q) : 0, a1 = own ? __ldg(col_off+q+1) : 0;
	const int particle = own ? __ldg(perm+q) : 0;
	T *col = arena+f.off+(int64_t)c0*f.ld;
	// where this pass's rows come from in children ch, ch + 1 (row 0 of their
	// columns; front blocks jc of the column, ir of the rows); the first pass's
	// before the wait
	struct { const T *src; int ld, jc, ir[ASM_ROWS]; } loc[2];
	auto locate = [&](int ch, int r0) {
#pragma unroll
		for (int k = 0; k < 2; k++) {
			const bool there = ch+k < f.cz;
			const ChildRec g = load_record(childs+(there ? ch+k : ch));
			const int *map = cinv+g.cinv_off;
			loc[k].ld = g.ld;
			loc[k].jc = there ? __ldg(map+cb) : -1;   // uniform
			loc[k].src = arena+g.off+(int64_t)DOF*loc[k].jc*g.ld;
#pragma unroll
			for (int u = 0; u < ASM_ROWS; u++) {
				const int r = r0+u*ASM_THREADS;
				loc[k].ir[u] = there && r < F6 ? __ldg(map+r/DOF) : -1;
			}
		}
	};
	const int first = c0+blockIdx.y*ASM_ROWS*ASM_THREADS+threadIdx.x;
	if (f.ca < f.cz) locate(f.ca, first);
	pdl_wait();
	if (status && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *status = 0x7fffffff;   // before any pivot
	for (int r0 = first; r0 < F6; r0 += gridDim.y*ASM_ROWS*ASM_THREADS) {
		T acc[ASM_ROWS][DOF];
		int rb[ASM_ROWS], rr[ASM_ROWS], entry[ASM_ROWS];
#pragma unroll
		for (int u = 0; u < ASM_ROWS; u++) {
			const int r = r0+u*ASM_THREADS;
			rb[u] = r < F6 ? r/DOF : -1;
			rr[u] = r%DOF;
			entry[u] = -1;
#pragma unroll
			for (int c = 0; c < DOF; c++) acc[u][c] = 0;
		}
		for (int ch = f.ca; ch < f.cz; ch += 2) {
			if (ch != f.ca || r0 != first) locate(ch, r0);
			T v[2][ASM_ROWS][DOF];
#pragma unroll
			for (int k = 0; k < 2; k++)
#pragma unroll
				for (int u = 0; u < ASM_ROWS; u++) {
					const int ir = loc[k].ir[u], jc = loc[k].jc;
#pragma unroll
					for (int c = 0; c < DOF; c++)   // the child's lower triangle
						v[k][u][c] = jc >= 0 && (ir > jc || (ir == jc && rr[u] >= c)) ? loc[k].src[(int64_t)c*loc[k].ld+DOF*ir+rr[u]] : T(0);
				}
#pragma unroll
			for (int k = 0; k < 2; k++)
#pragma unroll
				for (int u = 0; u < ASM_ROWS; u++)
#pragma unroll
					for (int c = 0; c < DOF; c++) acc[u][c] += v[k][u][c];
		}
		for (int t = a0; t < a1; t++) {
			const int br = __ldg(col_br+t);
#pragma unroll
			for (int u = 0; u < ASM_ROWS; u++)
				if (br == rb[u]) entry[u] = __ldg(col_e+t);
		}
#pragma unroll
		for (int u = 0; u < ASM_ROWS; u++) {
			const bool diag = own && rb[u] == cb;
			if (!diag && entry[u] < 0) continue;
			const double *m = diag ? dbl+15*(int64_t)particle : odbl+18*(int64_t)(entry[u]/2);
#pragma unroll
			for (int c = 0; c < DOF; c++) {
				const int i = DOF == 6 ? rr[u] : 2*rr[u], j = DOF == 6 ? c : 2*c;   // DOF 3: components 0, 2, 4
				const int p = diag ? c_dsym[6*i+j] : c_odense[entry[u] & 1 ? 6*j+i : 6*i+j];
				const double e = p == 0 ? 0.0 : m[(p < 0 ? -p : p)-1];
				acc[u][c] += (T)(p < 0 ? -e : e);
			}
		}
#pragma unroll
		for (int u = 0; u < ASM_ROWS; u++)
#pragma unroll
			for (int c = 0; c < DOF; c++)
				if (rb[u] > cb || (rb[u] == cb && rr[u] >= c)) col[(int64_t)c*f.ld+r0+u*ASM_THREADS] = acc[u][c];
	}
	if (own)
		for (int r = blockIdx.y*ASM_THREADS+threadIdx.x; r < f.n6; r += gridDim.y*ASM_THREADS)
#pragma unroll
			for (int c = 0; c < DOF; c++) col[(int64_t)c*f.ld+F6+r] = r == c0+c ? T(1) : T(0);
}

// CTAs that share a block column: one per ASM_SPLIT rows of the level's largest
// front
constexpr int ASM_SPLIT = 1024;

// ---------------------------------------------------------------------------
// FP32 diagonal block of panel k: one CTA (256 threads) per front factors and
// inverts the 64 x 64 block (diag_factor), so the rows below it are solved by
// k_trsm as a product with Linv^T, which goes to the front's slot of the Linv
// workspace.  k_diag is the launch for panel 0's.
// ---------------------------------------------------------------------------

// pivot reciprocal square root: the hardware approximation (the FP32 factor is
// refined in FP64 anyway; no denormal handling on the chain)
__device__ __forceinline__ float pivot_rsqrt(float x)
{
	float r;
	asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
	return r;
}

// 1 / d on the pivot chain: the hardware's approximation, whose results below 2^-126
// are 0; LARGE: pivots above LARGE_PIVOT may come (the block's diagonal bounds them)
constexpr float LARGE_PIVOT = 0x1p126f;
template <bool LARGE> __device__ __forceinline__ float pivot_rcp(float d)
{
	const float s = LARGE && d > LARGE_PIVOT ? 0.25f : 1.f;
	float r;
	asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(LARGE ? d*s : d));
	return LARGE ? r*s : r;
}

constexpr int DIAG_ZLD = 68;   // row stride of the inverse (rows 16-byte aligned)
constexpr int DIAG_FLAGS = 16;
constexpr int DIAG_FLAGS_AT = 64*64+64*DIAG_ZLD+128;   // in floats
constexpr size_t DIAG_SMEM = sizeof(float)*(DIAG_FLAGS_AT+DIAG_FLAGS);

// rows [8b, 8b + 8) of the inverse to vt
__device__ __forceinline__ void diag_out(float *vt, const float *zr, const float *dv, int b, int tid, int nthr)
{
	for (int e = tid; e < 512; e += nthr) {
		const int i = 8*b+e%8, j = e/8;
		const float d = dv[i], y = pivot_rsqrt(d);
		vt[64*j+i] = zr[DIAG_ZLD*i+j]*fmaf(d*y, 0.f, y);
	}
}

// diag_factor's chain of pivots, by one warp
template <bool LARGE>
__device__ __forceinline__ void diag_chain(float *base, int ld, int p0, int w, int gcol0, int *fail, float *S, float *rp,
                                           float *dv, int *fp, int *ca, int lane)
{
	float a0[8], a1[8];   // rows lane, lane + 32 of sub-panel b
#pragma unroll
	for (int q = 0; q < 8; q++) {
		a0[q] = S[64*q+lane];
		a1[q] = S[64*q+32+lane];
	}
	float d = __shfl_sync(FULL_MASK, a0[0], 0);
#pragma unroll 1
	for (int b = 0; b < 8; b++) {
		float l0[8], l1[8];
		const int s0 = (8*b) & 31;
		int bad = 64;
#pragma unroll
		for (int t = 0; t < 8; t++) {
			const int j = 8*b+t;
			const float u0 = a0[t], u1 = a1[t], us = b >= 4 ? u1 : u0;
			float uq[8];
#pragma unroll
			for (int q = t+1; q < 8; q++) uq[q] = __shfl_sync(FULL_MASK, us, s0+q);
			if (!(d > 0.f)) bad = min(bad, j);
			d = d > 0.f ? d : 1.f;
			const float r = pivot_rcp<LARGE>(d);
			l0[t] = u0*r;
			l1[t] = u1*r;
			const float dj = d;
			if (t < 7) {   // the next pivot first
				a0[min(t+1, 7)] -= l0[t]*uq[min(t+1, 7)];
				a1[min(t+1, 7)] -= l1[t]*uq[min(t+1, 7)];
				d = __shfl_sync(FULL_MASK, b >= 4 ? a1[min(t+1, 7)] : a0[min(t+1, 7)], s0+t+1);
			}
			S[64*j+lane] = u0;
			S[64*j+32+lane] = u1;
			rp[j] = r;
			dv[j] = dj;
			{   // L = U D^-1/2 (NaN for an infinite pivot)
				const float y = pivot_rsqrt(dj), rs = fmaf(dj*y, 0.f, y);
				float *o = base+(int64_t)(p0+j)*ld+p0+lane;
				if (lane >= j && lane < w) o[0] = (lane == j ? dj : u0)*rs;
				if (lane+32 >= j && lane+32 < w) o[32] = (lane+32 == j ? dj : u1)*rs;
			}
#pragma unroll
			for (int q = t+2; q < 8; q++) {
				a0[q] -= l0[t]*uq[q];
				a1[q] -= l1[t]*uq[q];
			}
		}
		__syncwarp();
		if (lane == 0) flag_publish(fp, b+1);
		if (bad < w && lane == 0 && fail) atomicMin(fail, gcol0+bad+1);
		if (b == 7) break;
		// the next sub-panel, up to date but for this one
		if (b) flag_wait(ca+b-1, 2, fail);
#pragma unroll
		for (int q = 0; q < 8; q++) {
			a0[q] = S[64*(8*b+8+q)+lane];
			a1[q] = S[64*(8*b+8+q)+32+lane];
		}
#pragma unroll
		for (int t = 0; t < 8; t++) {
			const float4 x = *reinterpret_cast<const float4 *>(S+64*(8*b+t)+8*b+8);
			const float4 y = *reinterpret_cast<const float4 *>(S+64*(8*b+t)+8*b+12);
			const float u[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
			for (int q = 0; q < 8; q++) {
				a0[q] -= l0[t]*u[q];
				a1[q] -= l1[t]*u[q];
			}
		}
		d = __shfl_sync(FULL_MASK, b >= 3 ? a1[0] : a0[0], (8*b+8) & 31);
	}
}

// Factor and invert a 64 x 64 diagonal block with the calling CTA (256 threads):
// L goes to the front at (p0, p0), L^-T (row-major) to vt.  sm: DIAG_SMEM bytes of
// shared memory, the block in its first 64 x 64 floats (column-major, lower part,
// identity-padded past the panel width w, zero above the diagonal) and the flags
// zeroed, both before a __syncthreads that precedes the call.  A non-positive
// pivot is replaced by 1 and reported (global scalar column + 1).
//
// The block is on the chain of the panels, bound by the latency from column to
// column, so one warp does nothing else.  LDL^T: a reciprocal, a product and a
// multiply-add lead from a pivot to the next (the square roots come with the
// stores: L = U D^-1/2, L^-1 = D^-1/2 (unit L)^-1).
//  warp 0, the chain: 8-column sub-panels in registers, rows lane and lane + 32;
//    brings the next sub-panel up to date with this one by itself;
//  warps 1-3, 5-7: the columns from two sub-panels on, and the rows of the
//    inverse below, four columns at a time in registers, a finished sub-panel
//    (rank 8) at a time;
//  warp 4: the inverse's rows of a sub-panel, behind the chain.
// Alone, warm: 13.4k cycles; 20.1k for two 32 x 32 halves, each column of which one
// warp factored and applied to all others (157 cycles a column, now 95).
__device__ void diag_factor(float *base, int ld, int p0, int w, int gcol0, int *fail, float *sm, float *vt)
{
	constexpr int ZLD = DIAG_ZLD;
	float *S = sm, *zr = S+64*64, *rp = zr+64*ZLD, *dv = rp+64;   // rp: reciprocals, dv: pivots
	int *flags = reinterpret_cast<int *>(sm+DIAG_FLAGS_AT);
	// sub-panels factored; their inverse rows solved; columns of sub-panel b + 2
	// ready (two quads); inverse rows of sub-panel b + 1 ready (six warps)
	int *fp = flags, *fz = flags+1, *ca = flags+2, *cr = flags+9;
	const int warp = threadIdx.x/32, lane = threadIdx.x%32;
	if (warp == 0) {
		const bool large = __any_sync(FULL_MASK, fmaxf(S[65*lane], S[65*(lane+32)]) > LARGE_PIVOT);
		if (__builtin_expect(!large, 1)) diag_chain<false>(base, ld, p0, w, gcol0, fail, S, rp, dv, fp, ca, lane);
		else diag_chain<true>(base, ld, p0, w, gcol0, fail, S, rp, dv, fp, ca, lane);
	} else if (warp == 4) {   // the inverse's rows of a sub-panel
#pragma unroll 1
		for (int b = 0; b < 8; b++) {
			if (b) flag_wait(cr+b-1, 6, fail);
			float z0[8], z1[8];
#pragma unroll
			for (int q = 0; q < 8; q++) {
				const int i = 8*b+q;
				z0[q] = lane < 8*b ? zr[ZLD*i+lane] : lane == i ? 1.f : 0.f;
				z1[q] = lane+32 < 8*b ? zr[ZLD*i+lane+32] : lane+32 == i ? 1.f : 0.f;
			}
			flag_wait(fp, b+1, fail);
			float l[8][8];
#pragma unroll
			for (int t = 0; t < 7; t++) {
				const float r = rp[8*b+t];
#pragma unroll
				for (int q = t+1; q < 8; q++) l[t][q] = S[64*(8*b+t)+8*b+q]*r;
			}
#pragma unroll
			for (int t = 0; t < 8; t++) {
#pragma unroll
				for (int q = t+1; q < 8; q++) {
					z0[q] -= l[t][q]*z0[t];
					z1[q] -= l[t][q]*z1[t];
				}
				zr[ZLD*(8*b+t)+lane] = z0[t];
				zr[ZLD*(8*b+t)+lane+32] = z1[t];
			}
			__syncwarp();
			if (lane == 0) flag_publish(fz, b+1);
		}
	} else {
		const int k = warp < 4 ? warp-1 : warp-2;   // 0..5
		// rows lane, lane + 32 of four columns each: trailing quads 4 + k, 10 + k
		// (columns 16 + 4k.., 40 + 4k..), inverse quads k, k + 6, k + 12
		float a[2][2][4], r[3][2][4];
#pragma unroll
		for (int x = 0; x < 2; x++)
#pragma unroll
			for (int c = 0; c < 4; c++) {
				const float *col = S+64*(16+4*k+24*x+c);
				a[x][0][c] = col[lane];
				a[x][1][c] = col[lane+32];
			}
#pragma unroll
		for (int x = 0; x < 3; x++)
#pragma unroll
			for (int c = 0; c < 4; c++) r[x][0][c] = r[x][1][c] = 0.f;
#pragma unroll 1
		for (int b = 0; b < 7; b++) {
			flag_wait(fp, b+1, fail);
			const float *U = S+64*8*b;
			float l0[8], l1[8];
#pragma unroll
			for (int t = 0; t < 8; t++) {
				const float q = rp[8*b+t];
				l0[t] = U[64*t+lane]*q;
				l1[t] = U[64*t+lane+32]*q;
			}
#pragma unroll
			for (int x = 0; x < 2; x++) {
				const int c0 = 16+4*k+24*x;
				if (c0 < 8*(b+2)) continue;
#pragma unroll
				for (int t = 0; t < 8; t++) {
					const float4 u = *reinterpret_cast<const float4 *>(U+64*t+c0);
					a[x][0][0] -= l0[t]*u.x; a[x][0][1] -= l0[t]*u.y; a[x][0][2] -= l0[t]*u.z; a[x][0][3] -= l0[t]*u.w;
					a[x][1][0] -= l1[t]*u.x; a[x][1][1] -= l1[t]*u.y; a[x][1][2] -= l1[t]*u.z; a[x][1][3] -= l1[t]*u.w;
				}
				if (c0 < 8*(b+3)) {   // of sub-panel b + 2: complete but for b + 1
#pragma unroll
					for (int c = 0; c < 4; c++) {
						S[64*(c0+c)+lane] = a[x][0][c];
						S[64*(c0+c)+lane+32] = a[x][1][c];
					}
					__syncwarp();
					if (lane == 0) flag_add(ca+b);
				}
			}
			flag_wait(fz, b+1, fail);
#pragma unroll
			for (int x = 0; x < 3; x++) {
				const int c0 = 4*k+24*x;
				if (c0 >= 8*(b+1)) continue;
#pragma unroll
				for (int t = 0; t < 8; t++) {
					const float4 z = *reinterpret_cast<const float4 *>(zr+ZLD*(8*b+t)+c0);
					r[x][0][0] -= l0[t]*z.x; r[x][0][1] -= l0[t]*z.y; r[x][0][2] -= l0[t]*z.z; r[x][0][3] -= l0[t]*z.w;
					r[x][1][0] -= l1[t]*z.x; r[x][1][1] -= l1[t]*z.y; r[x][1][2] -= l1[t]*z.z; r[x][1][3] -= l1[t]*z.w;
				}
				// rows of sub-panel b + 1
				const int h = b+1 >= 4, i = 8*(b+1)-32*h;
				if (lane >= i && lane < i+8)
					*reinterpret_cast<float4 *>(zr+ZLD*(lane+32*h)+c0) =
						h ? make_float4(r[x][1][0], r[x][1][1], r[x][1][2], r[x][1][3])
						  : make_float4(r[x][0][0], r[x][0][1], r[x][0][2], r[x][0][3]);
			}
			__syncwarp();
			if (lane == 0) flag_add(cr+b);
			diag_out(vt, zr, dv, b, k*32+lane, 192);
		}
	}
	__syncthreads();
	diag_out(vt, zr, dv, 7, threadIdx.x, 256);
}

// Linv slot of supernode s for panel k: two slots per supernode, by the
// parity of k, so the update launch of panel k can write panel k + 1's while
// the panel-k solve of other fronts still reads panel k's
template <typename P> __device__ inline P *linv_slot(P *linv, int nsn, int s, int k)
{
	constexpr int NB = Cfg<float>::NB;
	return linv+((int64_t)(k & 1)*nsn+s)*NB*NB;
}

// diagonal block of panel 0 of every front of a level (later panels' blocks
// are factored by the update launch of the previous panel)
__global__ void __launch_bounds__(256) k_diag(const int4 *__restrict__ tasks, const int *__restrict__ sn_first,
                                              const int *__restrict__ sn_ld, const int64_t *__restrict__ sn_off,
                                              float *__restrict__ arena, float *__restrict__ linv, int nsn, int *fail, int dof)
{
	__shared__ __align__(16) unsigned char smem_diag[DIAG_SMEM];
	float *sm = reinterpret_cast<float *>(smem_diag);
	int4 tk = tasks[blockIdx.x];
	int s = tk.x, p0 = tk.y, k = tk.z, w = tk.w, ld = sn_ld[s];
	float *base = arena+sn_off[s];
	if (threadIdx.x < DIAG_FLAGS) reinterpret_cast<int *>(sm)[DIAG_FLAGS_AT+threadIdx.x] = 0;
	pdl_wait();
	{
		float v[16];
#pragma unroll
		for (int u = 0; u < 16; u++) {
			const int e = threadIdx.x+256*u, i = e%64, j = e/64;   // coalesced over rows
			v[u] = j > i ? 0.f : i < w ? base[(int64_t)(p0+j)*ld+p0+i] : i == j ? 1.f : 0.f;
		}
#pragma unroll
		for (int u = 0; u < 16; u++) sm[threadIdx.x+256*u] = v[u];
	}
	__syncthreads();
	diag_factor(base, ld, p0, w, dof*sn_first[s]+p0, fail, sm, linv_slot(linv, nsn, s, k));
}

// ---------------------------------------------------------------------------
// rows below the diagonal block of panel k (k_trsm): X = A Linv_kk^T for up
// to R rows per CTA (real rows [t0, 6F) and identity rows [6F, 6F + t0)), in
// place.  256 threads in GROUPS groups: thread (g, r) computes row r for two
// column chunks of equal work together (column j needs t <= j).  Linv^T sits in shared memory row-major, so a
// chunk's coefficients for one t are one or two vector loads (a broadcast).
// ---------------------------------------------------------------------------
template <int CW>
__device__ inline void lds_chunk(const float *p, float (&v)[CW])
{
	static_assert(CW % 4 == 0, "chunk width");
#pragma unroll
	for (int q = 0; q < CW/4; q++) {
		const float4 x = reinterpret_cast<const float4 *>(p)[q];
		v[4*q] = x.x; v[4*q+1] = x.y; v[4*q+2] = x.z; v[4*q+3] = x.w;
	}
}

template <int R>
__global__ void __launch_bounds__(256) k_trsm(const int4 *__restrict__ tasks, const int *__restrict__ sn_n,
                                              const int *__restrict__ sn_ld, const int64_t *__restrict__ sn_off,
                                              float *__restrict__ arena, const float *linv, int nsn, int dof)
{
	constexpr int NB = Cfg<float>::NB, GROUPS = 256/R, CW = NB/(2*GROUPS);
	__shared__ __align__(16) float Vt[NB*NB];
	__shared__ float As[R*NB];   // row r, column t at r*NB + (t ^ (r & 31)): a warp's rows on distinct banks
	static_assert(R == 32 || R == 64, "a group's warps whole");
	int4 tk = tasks[blockIdx.x];
	int s = tk.x, row0 = tk.y, k = tk.z, nrows = tk.w;
	int ld = sn_ld[s];
	int p0 = k*NB;
	int w = min(NB, dof*sn_n[s]-p0);   // panel width: columns p0 + w and later are not touched
	float *base = arena+sn_off[s];
	const float *vt = linv_slot(linv, nsn, s, k);
	pdl_trigger();   // the next update's CTAs wait resident while this short launch runs
	pdl_wait();
	// all of a thread's loads are issued before its shared stores (256
	// threads: NB*NB/256 entries of Linv^T, R*NB/256 of the panel)
	{
		constexpr int PV = NB*NB/256, PA = R*NB/256;
		float lv[PV], av[PA];
#pragma unroll
		for (int u = 0; u < PV; u++) lv[u] = vt[threadIdx.x+256*u];
#pragma unroll
		for (int u = 0; u < PA; u++) {
			int e = threadIdx.x+256*u;
			int r = e%R, t = e/R;   // coalesced over rows
			av[u] = (r < nrows && t < w) ? base[(int64_t)(p0+t)*ld+row0+r] : float(0);
		}
#pragma unroll
		for (int u = 0; u < PV; u++) Vt[threadIdx.x+256*u] = lv[u];
#pragma unroll
		for (int u = 0; u < PA; u++) {
			int e = threadIdx.x+256*u;
			int r = e%R, t = e/R;
			As[r*NB+(t ^ (r & 31))] = av[u];
		}
	}
	__syncthreads();
	// thread: row r, column chunks g and 2 GROUPS - 1 - g (equal work per thread:
	// chunk c has (c + 1) CW terms per entry)
	int g = threadIdx.x/R, r = threadIdx.x%R;
	const float *a0 = As+r*NB;
	const int sw = r & 31;
#pragma unroll
	for (int h = 0; h < 2; h++) {
		int c = h ? 2*GROUPS-1-g : g;
		int j0 = c*CW;
		float x0[CW];
#pragma unroll
		for (int q = 0; q < CW; q++) x0[q] = float(0);
#pragma unroll 4
		for (int t = 0; t < j0+CW; t++) {
			float v[CW];
			lds_chunk<CW>(Vt+t*NB+j0, v);
			float u0 = a0[t ^ sw];
#pragma unroll
			for (int q = 0; q < CW; q++) x0[q] += u0*v[q];
		}
#pragma unroll
		for (int q = 0; q < CW; q++) {
			if (j0+q >= w) continue;
			if (r < nrows) base[(int64_t)(p0+j0+q)*ld+row0+r] = x0[q];
		}
	}
}

// trailing update: CTA = one tile (sn, r0, c0, k) of the front's own columns.
// The tile at (t0, t0) holds panel k + 1's diagonal block: after its update it
// factors and inverts that block (diag_factor), so the next panel needs no
// separate diagonal launch.  (Solving panel k + 1's rows in this launch as
// well -- column-t0 tiles waiting on a flag the diagonal CTA publishes, tasks
// in ticket order -- was measured slower than the separate solve launch.)
__global__ void __launch_bounds__(256, 2) k_update(const int4 *__restrict__ tasks, const int *__restrict__ sn_first,
                                                const int *__restrict__ sn_n, const int *__restrict__ sn_m,
                                                const int *__restrict__ sn_ld, const int64_t *__restrict__ sn_off,
                                                float *__restrict__ arena, float *__restrict__ linv, int nsn, int *fail,
                                                int dof)
{
	constexpr int NB = Cfg<float>::NB, TL = Cfg<float>::TILE, TPT = Cfg<float>::TPT;
	constexpr int TD = TL/TPT; // threads per dimension (16)
	extern __shared__ __align__(16) unsigned char smem_upd[];
	float (*As)[TL] = reinterpret_cast<float (*)[TL]>(smem_upd);
	float (*Bs)[TL] = reinterpret_cast<float (*)[TL]>(smem_upd+sizeof(float)*NB*TL);
	int4 tk = tasks[blockIdx.x];
	int s = tk.x, r0 = tk.y, cc0 = tk.z, k = tk.w;
	int n6 = dof*sn_n[s], F6 = n6+dof*sn_m[s], ld = sn_ld[s];
	int p0 = k*NB, w = min(NB, n6-p0), t0 = p0+w;
	float *base = arena+sn_off[s];
	bool extra = r0 >= F6;
	int rlim = extra ? F6+t0 : F6;
	int clim = n6;   // own columns only; the update matrix is k_syrk_tc's
	int tx = threadIdx.x%TD, ty = threadIdx.x/TD;
	pdl_wait();
	// the tile's old values, loaded first: their latency overlaps the panel
	// loads and the products
	float old[TPT][TPT];
#pragma unroll
	for (int b = 0; b < TPT; b++) {
		int c = cc0+ty+TD*b;
#pragma unroll
		for (int a = 0; a < TPT; a++) {
			int r = r0+tx+TD*a;
			bool in = c < clim && r < rlim && (extra || r >= c);
			old[a][b] = in ? base[(int64_t)c*ld+r] : float(0);
		}
	}
	// load panel rows of the tile rows and tile columns
	{
		constexpr int PU = NB*TL/256;   // entries of each panel per thread, all loaded before the stores
		float av[PU], bv[PU];
#pragma unroll
		for (int u = 0; u < PU; u++) {
			int e = threadIdx.x+256*u;
			int t = e/TL, i = e%TL;
			int ra = r0+i, rb = cc0+i;
			av[u] = (t < w && ra < rlim) ? base[(int64_t)(p0+t)*ld+ra] : float(0);
			bv[u] = (t < w && rb < clim) ? base[(int64_t)(p0+t)*ld+rb] : float(0);
		}
		// row i = x + TD a of the tile (thread x's a-th row) goes to position
		// TPT x + a, so a thread's TPT values of one t are one vector load
#pragma unroll
		for (int u = 0; u < PU; u++) {
			int e = threadIdx.x+256*u;
			int i = e%TL, pi = TPT*(i%TD)+i/TD;
			As[e/TL][pi] = av[u];
			Bs[e/TL][pi] = bv[u];
		}
	}
	__syncthreads();
	float acc[TPT][TPT];
#pragma unroll
	for (int a = 0; a < TPT; a++)
#pragma unroll
		for (int b = 0; b < TPT; b++) acc[a][b] = 0;
	// unrolled: the loads of later columns ahead of the products (N = 4096 step 6.84 -> 6.74 ms)
#pragma unroll 8
	for (int t = 0; t < w; t++) {
		float av[TPT], bv[TPT];
		lds_chunk<TPT>(&As[t][TPT*tx], av);
		lds_chunk<TPT>(&Bs[t][TPT*ty], bv);
#pragma unroll
		for (int a = 0; a < TPT; a++)
#pragma unroll
			for (int b = 0; b < TPT; b++) acc[a][b] += av[a]*bv[b];
	}
	const bool diag = !extra && r0 == t0 && cc0 == t0;
	float *sm = reinterpret_cast<float *>(smem_upd);   // the diagonal block's work space (over As, Bs)
	const int w1 = min(NB, n6-t0);   // width of panel k + 1
	// The diagonal tile is panel k + 1's diagonal block (NB == TL): its entries
	// in the block's rows go to shared memory (diag_factor writes them back), the
	// rows below it to the front.
	static_assert(NB == TL, "the diagonal tile is the next diagonal block");
	if (diag) __syncthreads();   // As, Bs are no longer read
#pragma unroll
	for (int b = 0; b < TPT; b++) {
		int c = cc0+ty+TD*b;
#pragma unroll
		for (int a = 0; a < TPT; a++) {
			int r = r0+tx+TD*a;
			float v = old[a][b]-acc[a][b];
			if (diag) {
				int i = tx+TD*a, j = ty+TD*b;
				float l = 0.f;
				if (j <= i) {
					if (i < w1) l = v;
					else if (i == j) l = 1.f;
				}
				sm[64*j+i] = l;
				if (i < w1) continue;
			}
			if (c < clim && r < rlim && (extra || r >= c)) base[(int64_t)c*ld+r] = v;
		}
	}
	if (diag) {
		if (threadIdx.x < DIAG_FLAGS) reinterpret_cast<int *>(sm)[DIAG_FLAGS_AT+threadIdx.x] = 0;
		__syncthreads();   // the updated block is in place
		diag_factor(base, ld, t0, w1, dof*sn_first[s]+t0, fail, sm, linv_slot(linv, nsn, s, k+1));
	}
}


// ---------------------------------------------------------------------------
// FP32 Schur complement on the tensor cores: k_syrk_tc.  tcgen05.mma
// (kind::tf32) with a 3xTF32 split: x = hi + lo with hi the TF32 part of x
// (the MMA reads only the upper 19 bits, so hi is x itself) and lo = x -
// hi exactly, so A B^T ~ Ahi Bhi^T + Ahi Blo^T + Alo Bhi^T keeps FP32-level
// accuracy for the refinement.  One CTA (544 threads) per 128 x 128 tile of
// the update matrix; the accumulator lives in tensor memory (128 columns).
// K is walked in chunks of 32 (one 128-byte row of TF32): the threads
// transpose the chunk's column-major front data into K-major,
// 128-byte-swizzled shared-memory tiles in a ring of 4 stages, one thread
// issues 4 K-steps x 3 MMAs per chunk and commits them to the stage's
// mbarrier, and staging of the next chunks overlaps the MMAs.  Every mbarrier
// wait is bounded: on a timeout the CTA stops issuing, waits (bounded) for
// what it issued, frees its tensor memory and records the timeout (status 0)
// in *fail.
// ---------------------------------------------------------------------------
namespace umma {
constexpr int M = 128, N = 128, KC = 32, STAGES = 4;
constexpr int GROUP = 256;                // threads of a producer group (8 warps)
constexpr int GROUPS = 2;                 // group g stages the chunks ch = g (mod GROUPS)
constexpr int PRODUCERS = GROUPS*GROUP;   // warps 0-15: staging and epilogue
constexpr int THREADS = PRODUCERS+32;     // + warp 16: MMA issue
constexpr int TILE_BYTES = M*KC*4;           // one operand part (16 KB)
constexpr int STAGE_BYTES = 2*TILE_BYTES;    // B hi, B lo (A's parts are in tensor memory)
constexpr int SMEM_BYTES = STAGES*STAGE_BYTES+1024;
// tensor memory: the accumulator in columns [0, N), stage b's A hi / lo in
// columns ACOL + 2 KC b + [0, KC) / + KC + [0, KC)
constexpr int ACOL = N;
constexpr int TMEM_COLS = 512;
static_assert(ACOL+STAGES*2*KC <= TMEM_COLS, "tensor memory columns");
// instruction descriptor: D = F32, A = B = TF32, both K-major, N = 128, M = 128
constexpr uint32_t IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) |
                           ((uint32_t)(M >> 4) << 24);

__device__ inline float tf32_lo(float x) { return x-__uint_as_float(__float_as_uint(x) & 0xffffe000u); }

// D (tensor memory) += A (tensor memory, lane = row, one column per K
// element) B^T (shared memory descriptor)
__device__ inline void mma_tf32(uint32_t dt, uint32_t at, uint64_t b, uint32_t accumulate)
{
	asm volatile("{\n\t.reg .pred p;\n\t"
	             "setp.ne.b32 p, %4, 0;\n\t"
	             "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}\n"
	             :: "r"(dt), "r"(at), "l"(b), "r"(IDESC), "r"(accumulate));
}
__device__ inline void tmem_st16(uint32_t ta, const uint32_t (&v)[16])
{
	asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
	             "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
	             :: "r"(ta), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
	                "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
	                "r"(v[15]) : "memory");
}

} // namespace umma

// Barriers of a tensor-core tile: per ring stage "full" (the producers'
// stores are in) and "empty" (the stage's MMAs are complete), and "done" (all
// MMAs complete).
struct TcBars { uint64_t full[umma::STAGES], empty[umma::STAGES], done; };

// One 128 x 128 tile C -= A B^T on the tensor cores, for the calling CTA
// (umma::THREADS threads): rows r0 + [0, 128) of A and c0 + [0, 128) of B
// taken from the front's columns [k0, k1) (A and B are rows of the same
// column-major front), C[r][c] at base[c ld + r] for r < rlim, c < clim and,
// when lower_only, r >= c.  tmem: this CTA's tensor memory; bars: fresh
// (phase 0).  Returns false if a wait timed out.
//
// Warp-specialised: two producer groups of 8 warps take alternate K chunks.
// A producer thread (row m, K half h) loads its chunk's values of A row m
// and B row m into registers one chunk of its group ahead, writes A's TF32
// hi / lo parts to tensor memory (tcgen05.st: a warp owns the 32 lanes =
// rows of its quarter) and B's parts to the swizzled shared stage, then
// arrives on the stage's full barrier.  The MMA warp waits on that, issues
// the stage's three products per K step (A hi B hi, A hi B lo, A lo B hi)
// and commits them to the stage's empty barrier, which the producers wait on
// before they reuse the stage.  No CTA-wide barrier in the K loop.  Then the
// producer warps run the epilogue (old values first, TMEM, stores).
__device__ bool tc_tile_update(float *base, int ld, int r0, int c0, int k0, int k1, int rlim, int clim,
                               bool lower_only, unsigned char *sm, TcBars &bars, uint32_t tmem)
{
	using namespace umma;
	const int tid = threadIdx.x, warp = tid/32, lane = tid%32;
	const int nchunk = (k1-k0+KC-1)/KC;
	constexpr int PW = PRODUCERS/32;
	bool ok = true;
	if (warp < PW) {
		const int g = warp/(GROUP/32), gt = tid-GROUP*g;
		const int m = gt & (M-1), h = gt >> 7, q = warp & 3;
		const int ra = r0+m, rb = c0+m;
		const bool va = ra < rlim, vb = rb < clim;
		auto load = [&](int ch, float (&a)[16], float (&b)[16]) {
			int tb = k0+ch*KC+16*h;
			const float *pa = base+(int64_t)tb*ld+ra, *pb = base+(int64_t)tb*ld+rb;
			int nk = ch < nchunk ? min(16, k1-tb) : 0;
#pragma unroll
			for (int k = 0; k < 16; k++) {
				a[k] = (k < nk && va) ? *pa : 0.f;
				b[k] = (k < nk && vb) ? *pb : 0.f;
				pa += ld;
				pb += ld;
			}
		};
		float av[16], bv[16];
		load(g, av, bv);
		for (int ch = g; ch < nchunk; ch += GROUPS) {
			int b = ch % STAGES;
			if (ch >= STAGES && !mbar_wait(saddr(&bars.empty[b]), ((ch/STAGES)-1) & 1)) ok = false;
			// B: 16-byte chunks (4 consecutive K); the 8 lanes of a quarter
			// warp (consecutive m) land on 8 distinct rows and swizzled chunk
			// columns, i.e. on all 32 banks
			unsigned char *stg = sm+b*STAGE_BYTES;
#pragma unroll
			for (int c4 = 0; c4 < 4; c4++) {
				int ck = 4*h+c4;
				uint32_t off = (uint32_t)((m >> 3)*1024+(m & 7)*128+((ck ^ (m & 7)) << 4));
				const float *bq = bv+4*c4;
				*reinterpret_cast<float4 *>(stg+0*TILE_BYTES+off) = make_float4(bq[0], bq[1], bq[2], bq[3]);
				*reinterpret_cast<float4 *>(stg+1*TILE_BYTES+off) =
					make_float4(tf32_lo(bq[0]), tf32_lo(bq[1]), tf32_lo(bq[2]), tf32_lo(bq[3]));
			}
			// A: lane = row of the warp's quarter, 16 columns = this K half
			uint32_t hi[16], lo[16];
#pragma unroll
			for (int k = 0; k < 16; k++) {
				hi[k] = __float_as_uint(av[k]);
				lo[k] = __float_as_uint(tf32_lo(av[k]));
			}
			__syncwarp();
			uint32_t ta = tmem+((uint32_t)(32*q) << 16)+(uint32_t)(ACOL+2*KC*b+16*h);
			tmem_st16(ta, hi);
			tmem_st16(ta+KC, lo);
			asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
			asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // B visible to the tensor cores
			asm volatile("tcgen05.fence::before_thread_sync;");
			mbar_arrive(&bars.full[b]);
			load(ch+GROUPS, av, bv);
		}
	} else if (warp == PW && lane == 0) {
		for (int ch = 0; ch < nchunk; ch++) {
			int b = ch % STAGES;
			if (!mbar_wait(saddr(&bars.full[b]), (ch/STAGES) & 1)) { ok = false; break; }
			asm volatile("tcgen05.fence::after_thread_sync;");
			uint32_t sa = saddr(sm+b*STAGE_BYTES);
			uint32_t at = tmem+(uint32_t)(ACOL+2*KC*b);
#pragma unroll
			for (int kk = 0; kk < KC/8; kk++) {
				uint64_t bhi = sdesc(sa+0*TILE_BYTES+32*kk), blo = sdesc(sa+1*TILE_BYTES+32*kk);
				mma_tf32(tmem, at+8*kk, bhi, (ch > 0 || kk > 0) ? 1u : 0u);
				mma_tf32(tmem, at+8*kk, blo, 1u);
				mma_tf32(tmem, at+KC+8*kk, bhi, 1u);
			}
			mma_commit(&bars.empty[b]);
		}
		mma_commit(&bars.done);   // every MMA issued above is complete
	}
	if (warp < PW) {
		if (!mbar_wait(saddr(&bars.done), 0)) ok = false;
		asm volatile("tcgen05.fence::after_thread_sync;");
	}
	ok = __syncthreads_and(ok);
	if (ok && nchunk > 0 && warp < PW) {
		// warp w reads TMEM lanes 32 (w % 4) .. +32 (rows) and CPW columns
		constexpr int CPW = N/(PW/4);
		int q = warp & 3, grp = warp >> 2;
		int r = r0+32*q+lane;
		// the thread's old values, loaded before any store (the stores
		// would otherwise serialise the loads: the addresses may alias)
		float old[CPW];
		const float *po = base+(int64_t)(c0+CPW*grp)*ld+r;
#pragma unroll
		for (int j = 0; j < CPW; j++) {
			int c = c0+CPW*grp+j;
			old[j] = (r < rlim && c < clim && (!lower_only || r >= c)) ? *po : 0.f;
			po += ld;
		}
#pragma unroll
		for (int cb = CPW*grp; cb < CPW*grp+CPW; cb += 16) {
			uint32_t v[16];
			uint32_t ta = tmem+((uint32_t)(32*q) << 16)+(uint32_t)cb;
			asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
			             "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
			             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
			               "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
			               "=r"(v[14]), "=r"(v[15])
			             : "r"(ta));
			asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
			for (int j = 0; j < 16; j++) {
				int c = c0+cb+j;
				if (r < rlim && c < clim && (!lower_only || r >= c))
					base[(int64_t)c*ld+r] = old[cb-CPW*grp+j]-__uint_as_float(v[j]);
			}
		}
	}
	asm volatile("tcgen05.fence::before_thread_sync;");
	__syncthreads();
	return ok;
}

// tensor memory (all TMEM_COLS columns: one CTA per SM) and the barriers of a
// tensor-core CTA
__device__ inline uint32_t tc_setup(uint32_t *tmem_slot, TcBars &bars)
{
	using namespace umma;
	if (threadIdx.x/32 == 0) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
		             :: "r"(saddr(tmem_slot)), "r"(TMEM_COLS));
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
		asm volatile("tcgen05.fence::before_thread_sync;");
	}
	if (threadIdx.x == 0) {
		for (int q = 0; q < STAGES; q++) {
			mbar_init(&bars.full[q], GROUP);
			mbar_init(&bars.empty[q], 1);
		}
		mbar_init(&bars.done, 1);
		asm volatile("fence.mbarrier_init.release.cluster;");
	}
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;");
	return *tmem_slot;
}

__device__ inline void tc_teardown(uint32_t tmem)
{
	if (threadIdx.x/32 == 0)
		asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(umma::TMEM_COLS));
}

// Schur complement tile: U[r][c] -= sum_{t < 6n} L[r][t] L[c][t], lower part of [6n, 6F)^2
__global__ void __launch_bounds__(umma::THREADS, 1) k_syrk_tc(const int4 *__restrict__ tasks,
                                                              const int *__restrict__ sn_n,
                                                              const int *__restrict__ sn_m,
                                                              const int *__restrict__ sn_ld,
                                                              const int64_t *__restrict__ sn_off,
                                                              float *__restrict__ arena, int *fail, int dof)
{
	extern __shared__ unsigned char smem_tc[];
	__shared__ __align__(8) TcBars bars;
	__shared__ uint32_t tmem_slot;
	unsigned char *sm = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_tc)+1023) &
	                                                      ~static_cast<uintptr_t>(1023));
	int4 tk = tasks[blockIdx.x];
	int s = tk.x, r0 = tk.y, c0 = tk.z;
	int n6 = dof*sn_n[s], F6 = n6+dof*sn_m[s], ld = sn_ld[s];
	pdl_trigger();   // the next level's assembly reads its indices during the last wave
	pdl_wait();   // before the tensor-memory allocation, too
	uint32_t tmem = tc_setup(&tmem_slot, bars);
	bool ok = tc_tile_update(arena+sn_off[s], ld, r0, c0, 0, n6, F6, F6, true, sm, bars, tmem);
	tc_teardown(tmem);
	if (!ok && threadIdx.x == 0 && fail) atomicMin(fail, 0);
}

// ---------------------------------------------------------------------------
// allocation and launch
// ---------------------------------------------------------------------------


static size_t update_smem()
{
	// the tile's two panels, or the diagonal block's work space
	return std::max(sizeof(float)*2*Cfg<float>::NB*Cfg<float>::TILE, DIAG_SMEM);
}

// FP32 update launches of at most UPDATE_SOLO_TILES tiles (two waves at one CTA per
// SM) ask for more shared memory than two CTAs can share, so the CTA that factors
// the next diagonal block -- the launch's critical path -- has its SM to
// itself.  Step at N = 4096 with 304, 480, 760: 6.77, 6.79, 7.04 ms (at 760 the
// tiles' waves outlast the diagonal block); at N = 200 the same.
constexpr int UPDATE_SOLO_TILES = 304;
constexpr size_t UPDATE_SOLO_SMEM = 120*1024;

static void set_update_smem()
{
	static std::once_flag once;
	std::call_once(once, [] {
		LFG_CUDA(cudaFuncSetAttribute(k_update, cudaFuncAttributeMaxDynamicSharedMemorySize,
		                              (int)std::max(update_smem(), UPDATE_SOLO_SMEM)));
		LFG_CUDA(cudaFuncSetAttribute(k_syrk_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, umma::SMEM_BYTES));
		tile32_setup();
	});
}

// Larger fronts (29056 rows in FP64, 58112 in FP32) are refused: no kernel has
// been run on one.
constexpr size_t MAX_COLUMN_BYTES = 227*1024;

template <typename T> void factor_alloc(DevFactor<T> &F, const DevSymbolic &D, int kmax)
{
	if (sizeof(T)*(size_t)D.max_F > MAX_COLUMN_BYTES)
		throw Error{LFG_ERR_BAD_ARG, (int)D.max_F, "front too large for the assembly kernel"};
	device_grow(F.arena, F.arena_cap, D.arena_elems);
	device_grow(F.w, F.w_cap, D.w_elems*kmax);
	const int64_t xneed = (int64_t)6*D.nblk*kmax;
	device_grow(F.xp, F.xp_cap, xneed);
	device_grow(F.yp, F.yp_cap, xneed);
	device_grow(F.linv, F.linv_cap, (int64_t)2*D.nsn*Cfg<T>::NB*Cfg<T>::NB);
	solve_alloc(F, D, kmax);
	const int64_t ybytes = (int64_t)sizeof(T)*D.ybuf_elems;
	device_grow(F.ybuf, F.split_cap, ybytes+(int64_t)sizeof(short)*(D.rexp_elems+D.yexp_elems));
	F.rexp = reinterpret_cast<unsigned short *>(F.ybuf+ybytes);
	F.yexp = F.rexp+D.rexp_elems;
	if (!F.status) LFG_CUDA(cudaMalloc((void **)&F.status, sizeof(int)*4));
	if (std::is_same<T, double>::value) tile64_setup();
	else set_update_smem();
}

template <typename T> void factor_free(DevFactor<T> &F)
{
	if (F.arena) cudaFree(F.arena);
	if (F.w) cudaFree(F.w);
	if (F.xp) cudaFree(F.xp);
	if (F.yp) cudaFree(F.yp);
	if (F.status) cudaFree(F.status);
	if (F.linv) cudaFree(F.linv);
	if (F.part) cudaFree(F.part);
	if (F.tally) cudaFree(F.tally);
	if (F.ybuf) cudaFree(F.ybuf);
	F = DevFactor<T>();
}

template <typename T>
int factor_numeric(DevFactor<T> &F, const DevSymbolic &D, const double *dbl, const double *odbl,
                   cudaStream_t st)
{
	int launches = 0;
	bool first = true;
	for (const auto &L : D.factor_plan) {
		if (L.count <= 0) continue;
		switch (L.kind) {
		case PLAN_ASSEMBLE: {
			auto assemble = [&](auto kern) {
				launch_pdl(kern, dim3(L.count, (D.h_level_maxF6[L.level]+ASM_SPLIT-1)/ASM_SPLIT), ASM_THREADS, 0, st,
				           (const int2 *)D.col_tasks+L.off, (const FrontRec *)D.fronts, (const ChildRec *)D.child_recs,
				           (const int *)D.cinv, (const int *)D.perm, (const int *)D.col_off, (const int *)D.col_e,
				           (const int *)D.col_br, dbl, odbl, F.arena, first ? F.status : (int *)nullptr);
			};
			if (D.dof == 6) assemble(k_assemble<T, 6>);
			else assemble(k_assemble<T, 3>);
			first = false;
			break;
		}
		case PLAN_DIAG:
			if constexpr (std::is_same<T, double>::value) diag64_launch(D, L.off, L.count, F, st);
			else
				launch_pdl(k_diag, L.count, 256, 0, st, (const int4 *)D.diag_tasks+L.off, (const int *)D.sn_first,
				           (const int *)D.sn_ld, (const int64_t *)D.sn_off, F.arena, F.linv, D.nsn, F.status, D.dof);
			break;
		case PLAN_PANEL: case PLAN_PANEL_64:
			if constexpr (std::is_same<T, double>::value) trsm64_launch(D, L.off, L.count, F, st);
			else
				launch_pdl(L.kind == PLAN_PANEL ? k_trsm<32> : k_trsm<64>, L.count, 256, 0, st,
				           (const int4 *)D.panel_tasks+L.off, (const int *)D.sn_n, (const int *)D.sn_ld,
				           (const int64_t *)D.sn_off, F.arena, (const float *)F.linv, D.nsn, D.dof);
			break;
		case PLAN_UPDATE:
			if constexpr (std::is_same<T, double>::value)
				tile64_launch(D, L.off, L.count, tile64_cols(L.k), false, F, st);
			else
				launch_pdl(k_update, L.count, 256, L.count <= UPDATE_SOLO_TILES ? UPDATE_SOLO_SMEM : update_smem(), st,
				           (const int4 *)D.tile_tasks+L.off, (const int *)D.sn_first, (const int *)D.sn_n,
				           (const int *)D.sn_m, (const int *)D.sn_ld, (const int64_t *)D.sn_off, F.arena, F.linv, D.nsn,
				           F.status, D.dof);
			break;
		case PLAN_SYRK:
			if constexpr (std::is_same<T, double>::value)
				tile64_launch(D, L.off, L.count, factor_syrk_cols(LFG_PREC_FP64), true, F, st);
			else
				launch_pdl(k_syrk_tc, L.count, umma::THREADS, umma::SMEM_BYTES, st, (const int4 *)D.tile_tasks+L.off,
				           (const int *)D.sn_n, (const int *)D.sn_m, (const int *)D.sn_ld, (const int64_t *)D.sn_off,
				           F.arena, F.status, D.dof);
			break;
		case PLAN_PANEL_SPLIT:
			if constexpr (std::is_same<T, float>::value) trsm_split_launch(D, L.off, L.count, F, st);
			break;
		case PLAN_TRAIL_SPLIT:
			if constexpr (std::is_same<T, float>::value) tile32_launch(D, L.off, L.count, F, st);
			break;
		}
		launches++;
	}
	LFG_CUDA(cudaGetLastError());
	return launches;
}

// ---------------------------------------------------------------------------
// FP64 block residual r = b - A x (row-block gather, deterministic)
// ---------------------------------------------------------------------------
// r = b - A x, one warp per block row i, five blocks of the row at a time:
// lane 6 t + a takes row a of the t-th block, straight from the compact storage
// (row a's structural zero is column (a + 3) % 6: five products).  Positions,
// entries and x of two rounds of five blocks are loaded before their products:
// the kernel is bound by those loads' latency (one block per round trip took 27
// us at N = 2047, 34 us at 4096, 90 us at 16384 with 4 right-hand sides).  The
// blocks are ordered diagonal, row i's lower blocks, its upper blocks, and the
// five partial sums added in a fixed order: the result is reproducible.
constexpr int RES_WARPS = 4, RES_BLOCKS = 5, RES_ROUNDS = 2;

template <int K>
__global__ void __launch_bounds__(32*RES_WARPS) k_residual(int n, const double *__restrict__ dbl,
                           const double *__restrict__ odbl, const int *__restrict__ od_row,
                           const int *__restrict__ od_col, const int *__restrict__ lo_ptr,
                           const int *__restrict__ lo_idx, const int *__restrict__ up_ptr,
                           const int *__restrict__ up_idx, const double *__restrict__ b,
                           const double *__restrict__ x, double *__restrict__ r, int dof)
{
	const int i = blockIdx.x*RES_WARPS+threadIdx.x/32, lane = threadIdx.x%32;
	if (i >= n) return;
	const int t = lane/6, a = lane%6;
	// compact positions of the block row: diagonal, lower, upper (transposed)
	signed char pd[5], pl[5], pu[5];
#pragma unroll
	for (int m = 0; m < 5; m++) {
		const int c = (a+4+m)%6;
		pd[m] = c_dsym[6*a+c];
		pl[m] = c_odense[6*a+c];
		pu[m] = c_odense[6*c+a];
	}
	const int l0 = lo_ptr[i], nl = lo_ptr[i+1]-l0, u0 = up_ptr[i], nblk = 1+nl+up_ptr[i+1]-u0;
	double acc[K];
#pragma unroll
	for (int q = 0; q < K; q++) acc[q] = 0;
	for (int s0 = 0; s0 < nblk; s0 += RES_ROUNDS*RES_BLOCKS) {
		const double *M[RES_ROUNDS];
		int kind[RES_ROUNDS], j[RES_ROUNDS];
#pragma unroll
		for (int u = 0; u < RES_ROUNDS; u++) {
			const int s = s0+u*RES_BLOCKS+t;
			kind[u] = t >= RES_BLOCKS || s >= nblk ? -1 : s == 0 ? 0 : s <= nl ? 1 : 2;
			j[u] = i;
			M[u] = dbl+15*(int64_t)i;
			if (kind[u] > 0) {
				const int e = kind[u] == 1 ? lo_idx[l0+s-1] : up_idx[u0+s-1-nl];
				j[u] = kind[u] == 1 ? od_col[e] : od_row[e];
				M[u] = odbl+18*(int64_t)e;
			}
		}
		double m[RES_ROUNDS][5], v[RES_ROUNDS][5][K];
#pragma unroll
		for (int u = 0; u < RES_ROUNDS; u++)
#pragma unroll
			for (int c = 0; c < 5; c++) {
				const int p = kind[u] == 0 ? pd[c] : kind[u] == 1 ? pl[c] : pu[c];
				const double e = kind[u] < 0 ? 0.0 : M[u][(p < 0 ? -p : p)-1];
				m[u][c] = p < 0 ? -e : e;
#pragma unroll
				for (int q = 0; q < K; q++) v[u][c][q] = x[(int64_t)q*6*n+6*j[u]+(a+4+c)%6];
			}
#pragma unroll
		for (int u = 0; u < RES_ROUNDS; u++) {
			if (s0+u*RES_BLOCKS >= nblk) break;
#pragma unroll
			for (int c = 0; c < 5; c++)
#pragma unroll
				for (int q = 0; q < K; q++)
					if (kind[u] >= 0) acc[q] += m[u][c]*v[u][c][q];
		}
	}
	// blocks 0 + 1, 2 + 3, the two pairs, then 4, in the lanes of block 0
#pragma unroll
	for (int q = 0; q < K; q++) {
		const double p = acc[q]+__shfl_down_sync(FULL_MASK, acc[q], 6);
		const double s = p+__shfl_down_sync(FULL_MASK, p, 12)+__shfl_down_sync(FULL_MASK, acc[q], 24);
		// dof 3: only components 0, 2, 4 are unknowns of the system (the
		// out-of-plane ones are neither solved nor part of the residual)
		const int64_t o = (int64_t)q*6*n+6*i+a;
		if (lane < 6) r[o] = (dof == 3 && (a & 1)) ? 0.0 : b[o]-s;
	}
}

void block_residual(const DevBlockMatrix &A, int k, const double *b, const double *x, double *r,
                    cudaStream_t st)
{
	const int grid = (A.n+RES_WARPS-1)/RES_WARPS;
	for (int q0 = 0; q0 < k; q0 += 4) {
		const int64_t o = (int64_t)q0*6*A.n;
		auto run = [&](auto kern) {
			kern<<<grid, 32*RES_WARPS, 0, st>>>(A.n, A.dblocks, A.odblocks, A.od_row, A.od_col, A.lo_ptr, A.lo_idx,
			                                    A.up_ptr, A.up_idx, b+o, x+o, r+o, A.dof);
		};
		switch (std::min(4, k-q0)) {
		case 1: run(k_residual<1>); break;
		case 2: run(k_residual<2>); break;
		case 3: run(k_residual<3>); break;
		default: run(k_residual<4>); break;
		}
	}
}

// Squared norms of r and b per right-hand side and segment: segment q of a
// right-hand side is entries [seg[q], seg[q+1]) (one segment, [0, n6), when
// seg is null); out[2 (rh nseg + q)] = |r|^2, then |b|^2.  A cluster of NORM_CTAS
// CTAs shares a segment and its first adds their sums up through distributed
// shared memory; every sum in a fixed order (per thread, warps by shuffles, warps,
// CTAs).  CTA 0's shared memory may be written once that CTA has started: all
// arrive on the cluster's barrier when they start and wait for it after their
// sums, so the wait costs nothing.  With one CTA per right-hand side: 13 us at N =
// 2047, 21 us at 4096, 64 us at 16384.
constexpr int NORM_CTAS = 8, NORM_THREADS = 512;

__global__ void __cluster_dims__(NORM_CTAS, 1, 1) __launch_bounds__(NORM_THREADS)
k_norms(int n6, const double *__restrict__ r, const double *__restrict__ b, const int *__restrict__ seg, double *out)
{
	namespace cg = cooperative_groups;
	__shared__ double sums[2][NORM_THREADS/32], total[NORM_CTAS][2];
	cg::cluster_group cluster = cg::this_cluster();
	cluster.barrier_arrive();
	const int rank = blockIdx.x%NORM_CTAS, rh = blockIdx.x/NORM_CTAS, q = blockIdx.y, nseg = gridDim.y;
	const int lo = seg ? seg[q] : 0, hi = seg ? seg[q+1] : n6;
	double a = 0, c = 0;
#pragma unroll 4
	for (int i = lo+rank*NORM_THREADS+threadIdx.x; i < hi; i += NORM_CTAS*NORM_THREADS) {
		double u = r[(int64_t)rh*n6+i], v = b[(int64_t)rh*n6+i];
		a += u*u;
		c += v*v;
	}
	for (int o = 16; o > 0; o >>= 1) {
		a += __shfl_down_sync(FULL_MASK, a, o);
		c += __shfl_down_sync(FULL_MASK, c, o);
	}
	const int w = threadIdx.x/32, l = threadIdx.x%32;
	if (l == 0) { sums[0][w] = a; sums[1][w] = c; }
	__syncthreads();
	cluster.barrier_wait();
	if (threadIdx.x < 2) {
		a = 0;
		for (int t = 0; t < NORM_THREADS/32; t++) a += sums[threadIdx.x][t];
		*cluster.map_shared_rank(&total[rank][threadIdx.x], 0) = a;
	}
	cluster.sync();
	if (rank == 0 && threadIdx.x < 2) {
		a = 0;
		for (int t = 0; t < NORM_CTAS; t++) a += total[t][threadIdx.x];
		out[2*(rh*nseg+q)+threadIdx.x] = a;
	}
}

void residual_norms(int n6, int k, const double *r, const double *b, double *out, cudaStream_t st,
                    const int *seg, int nseg)
{
	k_norms<<<dim3(k*NORM_CTAS, seg ? nseg : 1), NORM_THREADS, 0, st>>>(n6, r, b, seg, out);
}

int factor_tile_size() { return Cfg<float>::TILE; }
int factor_syrk_cols(int precision) { return precision == LFG_PREC_FP64 ? 64 : 128; }
int factor_panel_width(int precision) { return precision == LFG_PREC_FP64 ? Cfg<double>::NB : Cfg<float>::NB; }

template void factor_alloc<double>(DevFactor<double> &, const DevSymbolic &, int);
template void factor_alloc<float>(DevFactor<float> &, const DevSymbolic &, int);
template void factor_free<double>(DevFactor<double> &);
template void factor_free<float>(DevFactor<float> &);
template int factor_numeric<double>(DevFactor<double> &, const DevSymbolic &, const double *, const double *, cudaStream_t);
template int factor_numeric<float>(DevFactor<float> &, const DevSymbolic &, const double *, const double *, cudaStream_t);

} // namespace lfg
