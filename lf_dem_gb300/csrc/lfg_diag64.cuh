// lfg_diag64.cuh -- FP64 diagonal block of a panel: factor and invert a 32 x
// 32 block with one CTA.
#pragma once
#include "lfg_device.cuh"

namespace lfg {

// 1 / d on the pivot chain: the hardware's 20-bit approximation and one
// third-order Householder step (e = 1 - d y; y (1 + e + e^2), error e^3), three
// dependent FP64 operations instead of a division's five or six.
__device__ __forceinline__ double pivot_rcp(double d)
{
	if (!(d < 0x1p1020 && d > 0x1p-1020)) {
		const double r = 1.0/d;
		return d*r*r;   // NaN for an infinite pivot, as d rsqrt(d) is
	}
	double y;
	asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
	const double e = fma(-d, y, 1.0);
	return fma(y, fma(e, e, e), y);
}

// The block arrives in Ls (lower part, row-major, stride 33, identity-padded
// past the panel width w); L goes to the front at (p0, p0) and L^-T,
// row-major, to vt.  The first 2 W warps of the CTA work, all threads call.
// ul: 2048, zr: 1056 doubles and flags: 2 zeroed ints of shared memory, ordered
// before the call by a __syncthreads.
//
// A warp's FP64 instruction occupies its scheduler's FP64 unit for 64 cycles
// whatever its active lanes (measured), so one warp alone would need 32 x 31 / 2
// of them for the factor and as many for the inverse, 64k cycles.  Here the
// columns of the factor (warps 0..W-1, lane = row) and the rows of the inverse
// (warps W..2W-1, lane = column) are dealt out to the warps of all four
// schedulers, which follow each other through shared-memory flags.  The chain
// is column to column: LDL^T, so it holds one reciprocal (and no square root),
// one product and one multiply-add; the square roots of all pivots follow at
// the end in one warp instruction sequence, and L = U D^-1/2, L^-1 = D^-1/2
// (unit L)^-1 in the stores.  Against the single-warp
// routines before it (W = 4): FP64 factor + solve at N = 60 0.94 -> 0.70 ms, at
// N = 500 3.99 -> 2.85 ms, about 30 us less per 32 columns of the chain.
template <int W>
__device__ void diag64(double *base, int ld, int p0, int w, int gcol0, int *fail, const double *Ls, double *vt,
                       double *ul, double *zr, int *flags)
{
	constexpr int LD = 33, C = 32/W;
	double *uc = ul, *lc = ul+1024, *rs = zr+1024;
	const int warp = threadIdx.x/32, lane = threadIdx.x%32;
	if (warp < W) {
		double a[C];   // columns warp + W q of the trailing block
#pragma unroll
		for (int q = 0; q < C; q++) a[q] = Ls[lane*LD+warp+W*q];
#pragma unroll
		for (int jq = 0; jq < C; jq++)
#pragma unroll 1
			for (int jo = 0; jo < W; jo++) {
				const int j = jq*W+jo;
				double l;
				if (warp == jo) {
					const double u = a[jq];
					double d = __shfl_sync(FULL_MASK, u, j);
					if (!(d > 0)) {
						if (lane == 0 && j < w && fail) atomicMin(fail, gcol0+j+1);
						d = 1;
					}
					l = lane > j ? u*pivot_rcp(d) : 0.0;
					uc[32*j+lane] = lane == j ? d : u;
					lc[32*j+lane] = l;
					__syncwarp();
					if (lane == 0) flag_publish(flags, j+1);
				} else {
					flag_wait(flags, j+1, fail);
					l = lc[32*j+lane];
				}
#pragma unroll
				for (int q = jq; q < C; q++)
					if (q > jq || warp > jo) a[q] -= l*uc[32*j+warp+W*q];
			}
	} else if (warp < 2*W) {
		const int iw = warp-W;
		double z[C];   // rows iw + W q of the inverse of unit L
#pragma unroll
		for (int q = 0; q < C; q++) z[q] = iw+W*q == lane ? 1.0 : 0.0;
#pragma unroll
		for (int tq = 0; tq < C; tq++)
#pragma unroll 1
			for (int to = 0; to < W; to++) {
				const int t = tq*W+to;
				double zt;
				if (iw == to) {
					zt = z[tq];
					zr[32*t+lane] = zt;
					__syncwarp();
					if (lane == 0) flag_publish(flags+1, t+1);
				} else {
					flag_wait(flags+1, t+1, fail);
					zt = zr[32*t+lane];
				}
				flag_wait(flags, t+1, fail);
#pragma unroll
				for (int q = tq; q < C; q++)
					if (q > tq || iw > to) z[q] -= lc[32*t+iw+W*q]*zt;
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
