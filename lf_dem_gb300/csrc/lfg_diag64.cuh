// lfg_diag64.cuh -- FP64 diagonal block of a panel: factor and invert a 32 x
// 32 block with one CTA.
#pragma once
#include "lfg_device.cuh"

namespace lfg {

// 1 / d on the pivot chain: the hardware's 20-bit approximation and one
// third-order Householder step (e = 1 - d y; y (1 + e + e^2), error e^3), three
// dependent FP64 operations instead of a division's five or six.  Comparisons
// are made on the bits: an FP64 compare costs as much as a multiply-add.
__device__ __forceinline__ double pivot_rcp(double d)
{
	const unsigned ex = ((unsigned)__double2hiint(d) >> 20)-4u;
	if (ex > 2038u) {   // negative, or a biased exponent outside [4, 2042]
		const double r = 1.0/d;
		return d*r*r;   // NaN for an infinite pivot, as d rsqrt(d) is
	}
	double y;
	asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
	const double e = fma(-d, y, 1.0);
	return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ bool pivot_positive(double d)
{
	const long long b = __double_as_longlong(d);
	return b > 0 && b <= 0x7ff0000000000000ll;
}

constexpr int DIAG64_THREADS = 512, DIAG64_FLAGS = 8;

// The block arrives in S (lower part, row-major, stride 33, identity-padded
// past the panel width w, zero above the diagonal) and is overwritten; L goes
// to the front at (p0, p0) and L^-T, row-major, to vt.  All 512 threads of the
// CTA call.  ul: 2048, zr: 1056 doubles and flags: DIAG64_FLAGS zeroed ints of
// shared memory, ordered before the call by a __syncthreads.
//
// A warp's FP64 instruction occupies its scheduler's FP64 unit for 64 cycles
// whatever its active lanes (measured), so the block is bound by the number of
// FP64 instructions and how they spread over the four schedulers.  LDL^T keeps
// square roots off the chain (one reciprocal, one product, one multiply-add per
// column; the 32 square roots follow at the end in one instruction sequence,
// and the stores scale: L = U D^-1/2, L^-1 = D^-1/2 (unit L)^-1).
//  warp 0 (alone on its scheduler) is the chain: 8-column sub-panels, a lane
//    per row, a finished column published at once;
//  11 warps of the other schedulers hold the entries right of the first
//    sub-panel (A groups) and the updated identity rows of the inverse (R
//    groups), 32 entries packed into a warp's lanes whatever their shape, and
//    apply each published column to those still active;
//  warp 15 solves the inverse's rows of a sub-panel behind the chain.
// Alone, warm: 30.5k cycles; with one warp per role (columns and rows dealt out
// to 4 + 4 or 8 + 8 warps, full 32-lane columns) 55k, of which FP64 compares
// on the chain 7k.
inline __device__ void diag64(double *base, int ld, int p0, int w, int gcol0, int *fail, double *S, double *vt, double *ul,
                              double *zr, int *flags)
{
	constexpr int LD = 33;
	double *uc = ul, *lc = ul+1024, *rs = zr+1024;
	int *fp = flags, *fz = flags+1, *ca = flags+2, *cr = flags+5;   // ca[b], cr[b], b = 0..2
	const int warp = threadIdx.x/32, lane = threadIdx.x%32;
	if (warp == 0) {
#pragma unroll 1
		for (int b = 0; b < 4; b++) {
			if (b) flag_wait(ca+b-1, 8-2*b, fail);
			double a[8];
#pragma unroll
			for (int q = 0; q < 8; q++) a[q] = S[lane*LD+8*b+q];
#pragma unroll
			for (int t = 0; t < 8; t++) {
				const int j = 8*b+t;
				const double u = a[t];
				double d = __shfl_sync(FULL_MASK, u, j);
				if (!pivot_positive(d)) {
					if (lane == 0 && j < w && fail) atomicMin(fail, gcol0+j+1);
					d = 1;
				}
				double ub[8];
#pragma unroll
				for (int q = t+1; q < 8; q++) ub[q] = __shfl_sync(FULL_MASK, u, 8*b+q);
				uc[32*j+lane] = lane == j ? d : u;
				const double l = u*pivot_rcp(d);
				if (t < 7) a[min(t+1, 7)] -= l*ub[min(t+1, 7)];   // the next column first
				lc[32*j+lane] = l;
				__syncwarp();
				if (lane == 0) flag_publish(fp, j+1);
#pragma unroll
				for (int q = t+2; q < 8; q++) a[q] -= l*ub[q];
			}
		}
	} else if (warp == 15) {   // rows of the inverse of unit L
#pragma unroll 1
		for (int b = 0; b < 4; b++) {
			if (b) flag_wait(cr+b-1, 2*b, fail);
			double z[8];
#pragma unroll
			for (int q = 0; q < 8; q++) z[q] = lane < 8*b ? zr[32*(8*b+q)+lane] : lane == 8*b+q ? 1.0 : 0.0;
#pragma unroll
			for (int t = 0; t < 8; t++) {
				const int j = 8*b+t;
				zr[32*j+lane] = z[t];
				__syncwarp();
				if (lane == 0) flag_publish(fz, j+1);
				if (t < 7) {
					flag_wait(fp, j+1, fail);
#pragma unroll
					for (int q = t+1; q < 8; q++) z[q] -= lc[32*j+8*b+q]*z[t];
				}
			}
		}
	} else if (warp & 3) {
		// bulk warps k = 0..10 on schedulers 1-3; groups k and, for k = 0 / 1, A / R group 11
		const int k = 3*(warp >> 2)+(warp & 3)-1;
		double a[2] = {0, 0}, r[2] = {0, 0};
		int ai[2], ac[2], ag[2], ri[2], rc[2], rb[2];
#pragma unroll
		for (int x = 0; x < 2; x++) {
			const int ga = x == 0 ? k : k == 0 ? 11 : -1, gr = x == 0 ? k : k == 1 ? 11 : -1;
			ag[x] = ga < 0 ? 0 : ga < 6 ? 1 : ga < 10 ? 2 : 3;
			const int e = 32*(ga-(ag[x] == 1 ? 0 : ag[x] == 2 ? 6 : 10))+lane, rows = 32-8*ag[x];
			ai[x] = 8*ag[x]+e%rows; ac[x] = 8*ag[x]+e/rows;
			if (ga < 0) { ai[x] = ac[x] = 0; }
			else a[x] = S[ai[x]*LD+ac[x]];
			rb[x] = gr < 0 ? 0 : gr < 2 ? 1 : gr < 6 ? 2 : 3;
			const int f = 32*(gr-(rb[x] == 1 ? 0 : rb[x] == 2 ? 2 : 6))+lane, cols = max(8*rb[x], 1);
			ri[x] = 8*rb[x]+f/cols; rc[x] = f%cols;
			if (gr < 0) ri[x] = rc[x] = 0;
		}
#pragma unroll 1
		for (int j = 0; j < 24; j++) {
			const int b = j >> 3;
			flag_wait(fp, j+1, fail);
#pragma unroll
			for (int x = 0; x < 2; x++)
				if (ag[x] > b) a[x] -= lc[32*j+ai[x]]*uc[32*j+ac[x]];
			if ((j & 7) == 7) {
#pragma unroll
				for (int x = 0; x < 2; x++)
					if (ag[x] == b+1) {
						S[ai[x]*LD+ac[x]] = a[x];
						__syncwarp();
						if (lane == 0) flag_add(ca+b);
					}
			}
			if (rb[0] > b || rb[1] > b) {
				flag_wait(fz, j+1, fail);
#pragma unroll
				for (int x = 0; x < 2; x++)
					if (rb[x] > b && rc[x] < 8*b+8) r[x] -= lc[32*j+ri[x]]*zr[32*j+rc[x]];
				if ((j & 7) == 7) {
#pragma unroll
					for (int x = 0; x < 2; x++)
						if (rb[x] == b+1) {
							zr[32*ri[x]+rc[x]] = r[x];
							__syncwarp();
							if (lane == 0) flag_add(cr+b);
						}
				}
			}
		}
	}
	__syncthreads();
	if (warp == 0) {
		const double d = uc[33*lane], y = rsqrt(d);
		rs[lane] = fma(d*y, 0.0, y);   // NaN for an infinite pivot
	}
	__syncthreads();
	for (int e = threadIdx.x; e < 1024; e += blockDim.x) {
		const int i = e%32, j = e/32;
		if (i >= j && i < w) base[(int64_t)(p0+j)*ld+p0+i] = uc[32*j+i]*rs[j];
		vt[j*32+i] = zr[32*i+j]*rs[i];
	}
}

} // namespace lfg
