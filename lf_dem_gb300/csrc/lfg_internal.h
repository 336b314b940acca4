// lfg_internal.h -- internal declarations shared by the host driver (C++) and
// the CUDA translation units of the GB300 engine.  Not part of the C ABI.
#pragma once

#include <array>
#include <cstdint>
#include <exception>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/lfdem_gb300.h"

namespace lfg {

// ---------------------------------------------------------------------------
// error handling: every CUDA call in the host driver goes through LFG_CUDA,
// which throws lfg::Error; the C-ABI layer converts it to a status code.
// ---------------------------------------------------------------------------
struct Error {
	int code;
	int info;
	std::string msg;
};

#define LFG_CUDA(call)                                                                     \
	do {                                                                                   \
		cudaError_t e_ = (call);                                                       \
		if (e_ != cudaSuccess) {                                                       \
			cudaGetLastError();   /* or a later check of launches would find it */ \
			throw ::lfg::Error{e_ == cudaErrorMemoryAllocation ? LFG_ERR_OOM : LFG_ERR_CUDA, \
			                   (int)e_, std::string(#call) + ": " + cudaGetErrorString(e_)}; \
		}                                                                              \
	} while (0)

// Device buffer of at least `need` elements (old contents are not kept).  When
// the allocation fails the buffer is gone and its capacity 0.
template <typename V> inline void device_grow(V *&p, int64_t &cap, int64_t need)
{
	if (cap >= need) return;
	if (p) cudaFree(p);
	p = nullptr;
	cap = 0;
	LFG_CUDA(cudaMalloc((void **)&p, sizeof(V)*need));
	cap = need;
}

// Ordinary host memory that a scope's asynchronous copies read or write is not
// given back before they are done (a copy may read it as late as it runs): the
// scope waits for the stream at its end, and this guard, declared after that
// memory, waits when an exception leaves it.
struct StreamDrain {
	cudaStream_t st;
	~StreamDrain() { if (std::uncaught_exceptions()) cudaStreamSynchronize(st); }
};

// ---------------------------------------------------------------------------
// Symbolic analysis of the block matrix (nested dissection + multifrontal
// assembly tree).  Computed on the host, mirrored to the device.
// ---------------------------------------------------------------------------
struct Symbolic {
	int nblk = 0;                 // particles (dof x dof blocks)
	int dof = 6;                  // scalar unknowns per particle: 6, or 3 for the in-plane part of a 2D system
	std::vector<int> perm;        // perm[k] = particle at permuted position k
	std::vector<int> iperm;       // iperm[particle] = permuted position
	// supernodes, in postorder (children before parents)
	int nsn = 0;
	std::vector<int> sn_first, sn_n, sn_m, sn_parent, sn_level;
	std::vector<int> sn_rows_off;     // into rows[] (m entries each, permuted block ids)
	std::vector<int> rows;
	std::vector<int64_t> sn_off;      // front arena offsets (elements)
	std::vector<int> sn_ld;           // front leading dimension = 6F + 6n
	std::vector<int64_t> sn_woff;     // forward-solve update vector offsets (elements)
	// children and inverse maps: for child c of parent p, inv[cinv_off[c] + b]
	// (b in [0, F_p)) = child front block index or -1
	std::vector<int> child_off, children;   // CSR over supernodes
	std::vector<int64_t> cinv_off;
	std::vector<int> cinv;
	// levels (0 = leaves)
	int nlevels = 0;
	std::vector<int> level_off, level_sn;   // CSR: supernodes of each level
	// off-diagonal blocks of R by block column (permuted position q, CSR):
	// 2 e + (1: transposed) for the caller's block e, and its row block in the
	// front that owns column q
	std::vector<int> col_off, col_e, col_br;
	int64_t arena_elems = 0;
	int64_t w_elems = 0;
	int max_F = 0;
	int64_t nnz_L = 0;
	double flops = 0;
};

// Build the symbolic analysis.  od_row/od_col: nb lower off-diagonal blocks
// (the pattern).  pos (3 * nblk, may be null) drives a geometric nested
// dissection; otherwise a breadth-first level-set dissection is used.
// dof: scalar unknowns per particle (6; 3 for the in-plane x, z translation
// and y rotation of a 2D system); it scales the front sizes only.
void symbolic_analyze(Symbolic &S, int nblk, int nb, const int32_t *od_row,
                      const int32_t *od_col, const double *pos, double lx, double ly, double lz,
                      int leaf_size, int dof = 6);

// The joint analysis of independent systems (the block-diagonal matrix of
// all of them): parts concatenated, levels of their assembly trees merged
// from the leaves.
void symbolic_concat(Symbolic &J, const std::vector<const Symbolic *> &parts);

// ---------------------------------------------------------------------------
// Device-side multifrontal factor (one precision per instance).
// ---------------------------------------------------------------------------
// A front, and a child of one, as the assembly and the solves read them.
struct alignas(16) FrontRec {
	int n6, m6, ld, f6;          // own scalars, update rows, leading dimension, first own scalar
	int rows_off, ca, cz, pad;   // into rows; its children [ca, cz)
	int64_t off, woff;           // into the arena and w
};
struct alignas(16) ChildRec {
	int64_t off, cinv_off, woff;   // its front, its inverse map, its update vector
	int ld, n;                     // leading dimension, own columns (particles)
};
static_assert(sizeof(FrontRec) == 48 && sizeof(ChildRec) == 32, "read by 16-byte loads");

// One phase of a solve sweep: gx x gy x gz CTAs of one type (lfg_solve.cu) over
// the gy fronts from lev_off of one level; the sweep's first phase; where the
// type has two parts, the first part's share of gx.
struct SolvePhase { int type, lev_off, gx, gy, gz, first, split; };

// Launch kinds of the factor plan (built by dev_symbolic_upload, run by
// factor_numeric).
enum { PLAN_ASSEMBLE, PLAN_PANEL, PLAN_PANEL_64, PLAN_PANEL_SPLIT, PLAN_UPDATE, PLAN_TRAIL_SPLIT, PLAN_SYRK, PLAN_DIAG };

struct DevSymbolic {
	int nblk = 0, nsn = 0, nlevels = 0;
	int dof = 6;                   // scalar unknowns per particle (6 or 3)
	int *perm = nullptr;
	int *sn_first = nullptr, *sn_n = nullptr, *sn_m = nullptr, *sn_ld = nullptr;
	int *rows = nullptr;
	int64_t *sn_off = nullptr;
	int *cinv = nullptr;
	int *col_off = nullptr, *col_e = nullptr, *col_br = nullptr;   // blocks of R by column (Symbolic)
	FrontRec *fronts = nullptr;       // in level order
	ChildRec *child_recs = nullptr;   // of every front, as Symbolic::children
	// per-level / per-panel task lists
	int2 *col_tasks = nullptr;     // (front in level order, block column) of the assembly
	int4 *panel_tasks = nullptr;   // (sn, row0, k, nrows)
	int4 *tile_tasks = nullptr;    // (sn, row0, col0, k)
	int4 *diag_tasks = nullptr;    // (sn, col0, k, width) of each panel's diagonal block
	// digit-split tile products (FP64; FP32 fronts updated two-level, -1 for others): per
	// supernode three offsets into DevFactor's tables (rows are front rows,
	// entry = offset + column or panel x ld + row):
	// 0  rexp: largest biased exponent of a row per panel
	// 1  yexp: the same per K block of the tile products
	// 2  ybuf: the row's entries as scaled integers (columns [0, 6n); FP32: in
	//    records of 16 columns, see lfg_factor32.cu)
	// The last two hold one level at a time.
	int64_t *split_off = nullptr;
	int64_t rexp_elems = 0, yexp_elems = 0, ybuf_elems = 0;
	std::vector<SolvePhase> h_solve_phases;   // phase table of a solve sweep
	std::vector<SolvePhase> h_mul_phases;     // ... of the product with L
	// host-side launch plan
	struct Launch { int kind; int level; int k; int64_t off; int count; };
	std::vector<Launch> factor_plan;
	std::vector<int> h_level_maxF6;   // per-level maximum front order dof (n + m) (scalar)
	int64_t arena_elems = 0, w_elems = 0;
	int max_F = 0;
	int max_n6 = 0;
	double flops = 0;
	int64_t nnz_L = 0;
};

// Tile edge and panel width the factor kernels use for a precision; the
// launch plan built by dev_symbolic_upload must use the same values.
int factor_tile_size();                   // FP32 trailing-update tiles
int factor_syrk_cols(int precision);      // Schur complement tiles: 128 rows x this
int factor_panel_width(int precision);

void dev_symbolic_upload(DevSymbolic &D, const Symbolic &S, int precision, cudaStream_t st);
void dev_symbolic_free(DevSymbolic &D);
// builds the phase tables of the solves (lfg_solve.cu)
void solve_plan_build(DevSymbolic &D, const Symbolic &S, int precision);

// Factor arenas and launchers (lfg_factor.cu).
template <typename T> struct DevFactor {
	T *arena = nullptr;   // fronts
	T *w = nullptr;       // forward-solve update vectors
	T *xp = nullptr, *yp = nullptr; // permuted solve workspaces (k * 6n)
	T *linv = nullptr;    // per supernode: Linv^T of its current panel's diagonal block
	char *ybuf = nullptr;             // scaled integers (as wide as T), rexp and yexp (DevSymbolic::split_off)
	unsigned short *rexp = nullptr, *yexp = nullptr;   // behind ybuf, in its allocation
	T *part = nullptr;    // solve: partial row sums per column chunk
	int *tally = nullptr; // solve: chunks done per row block of a row-product phase (0 between phases)
	int64_t pstride = 0;
	int64_t arena_cap = 0, w_cap = 0, xp_cap = 0, yp_cap = 0, linv_cap = 0, part_cap = 0, tally_cap = 0, split_cap = 0;
	int *status = nullptr; // device: first non-positive pivot column + 1; 0 = a bounded wait gave up;
	                       // 0x7fffffff = ok
};

template <typename T> void factor_alloc(DevFactor<T> &F, const DevSymbolic &D, int kmax);
template <typename T> void factor_free(DevFactor<T> &F);
template <typename T> void solve_alloc(DevFactor<T> &F, const DevSymbolic &D, int kmax);   // by factor_alloc

// Numeric factorisation from compact blocks (dblocks n x 15, odblocks nb x 18,
// both FP64 device arrays).  Launches only; status left in F.status.
template <typename T>
int factor_numeric(DevFactor<T> &F, const DevSymbolic &D, const double *d_dblocks,
                   const double *d_odblocks, cudaStream_t st);

// FP64 kernels (lfg_factor64.cu): tile products on the tensor cores for the
// tasks tile_tasks[off ... off + count), tiles of `cols` columns (32 or 64):
// Schur complements, or the update after a panel, which covers tile64_cols(k)
// columns at a time; the panel solves panel_tasks[off ... off + count); panel
// 0's diagonal blocks
void tile64_setup();
int tile64_kblock();     // columns of a K block
int tile64_cols(int k);
int trsm64_rows();
void tile64_launch(const DevSymbolic &D, int64_t off, int count, int cols, bool schur, DevFactor<double> &F,
                   cudaStream_t st);
void trsm64_launch(const DevSymbolic &D, int64_t off, int count, DevFactor<double> &F, cudaStream_t st);
void diag64_launch(const DevSymbolic &D, int64_t off, int count, DevFactor<double> &F, cudaStream_t st);

// FP32 fronts that are updated two-level (lfg_factor32.cu): tile products, panel solves
void tile32_setup();
int tile32_kblock();
int trsm_split_rows();
int64_t tile32_ybuf(int kblocks, int ld);
void tile32_launch(const DevSymbolic &D, int64_t off, int count, DevFactor<float> &F, cudaStream_t st);
void trsm_split_launch(const DevSymbolic &D, int64_t off, int count, DevFactor<float> &F, cudaStream_t st);

// Solve with k right-hand sides: b, x device arrays k x 6n, FP64 (x may alias
// b); add: x += solution.
template <typename T>
int factor_solve(DevFactor<T> &F, const DevSymbolic &D, int k, const double *b, double *x, bool add,
                 cudaStream_t st);
// x = P^T L P b (k vectors; x may not alias b)
template <typename T>
int factor_multiply(DevFactor<T> &F, const DevSymbolic &D, int k, const double *b, double *x,
                    cudaStream_t st);

// y = A x for the compact block matrix (FP64), k vectors, and r = b - A x.
// Lower/upper adjacency lists for the per-block-row gather.
struct DevBlockMatrix {
	int n = 0, nb = 0;
	int dof = 6;                 // unknowns per particle of the solved system (6, or 3: components 0, 2, 4)
	double *dblocks = nullptr;   // n x 15
	double *odblocks = nullptr;  // nb x 18
	int *od_row = nullptr, *od_col = nullptr;
	int *lo_ptr = nullptr, *lo_idx = nullptr;   // for row block i: OD entries with row == i
	int *up_ptr = nullptr, *up_idx = nullptr;   // OD entries with col == i
};
void block_residual(const DevBlockMatrix &A, int k, const double *b, const double *x, double *r,
                    cudaStream_t st);

// Everything the output writers read from a simulation (lfg_output.cpp),
// gathered by sim_output_snapshot (lfg_sim.cpp) at the current state.
struct OutputSnapshot {
	int n = 0, twodim = 0, lubrication = 0, repulsion = 0, control = 0;
	double lx = 0, ly = 0, lz = 0;
	double time = 0, strain = 0, shear_rate = 0, avg_dt = 0, max_velocity = 0;
	double shear_disp[2] = {0, 0}, shear_strain[3] = {0, 0, 0}, Einf[6] = {0}, vel_diff[3] = {0, 0, 0};
	double kn = 0, kt = 0, kr = 0, interaction_range = 0;
	double total_stress[6] = {0};
	std::vector<std::string> groups;          // System::total_stress_groups, in key order
	std::vector<std::array<double, 6>> group_stress;
	std::vector<double> radius, pos, vel, ang, na, na_disp, angle;   // n, 3n, 3n, 3n, 6n, 3n, n
	std::vector<double> pairs;                // OUT_W doubles per interaction, sorted by (p0, p1)
	int out_w = 0;
	// per-particle stresslets of every stress slot (NSC x 6n) and which slots
	// the run declares; filled only when want_particle_stress is set
	bool want_particle_stress = false;
	std::vector<double> particle_stress;
	std::vector<char> slot_declared;
};

// Fused batch (lfg_sim.cpp): suspensions stepping in lockstep through one
// joint solver.  fused_add creates a member simulation (owned by the caller,
// destroyed with lfg_sim_destroy after the group).
class FusedGroup;
FusedGroup *fused_create(int device, int precision);
void fused_destroy(FusedGroup *g);
int fused_add(FusedGroup *g, const lfg_params *p, const lfg_options *opt, int n, const double *pos,
              const double *radius, double lx, double ly, double lz, const double *le_disp, lfg_sim **out,
              lfg_status *st);
void fused_run(FusedGroup *g, int nsteps);
void fused_advance(FusedGroup *g, const double *strain_end);
void fused_set_leaf_size(FusedGroup *g, int leaf);
void fused_stats(const FusedGroup *g, int64_t *kernels, int *joint_runs, double *flops, int *iters);

// per-RHS squared norms of r and b, written to out[2k] (device); with a
// segment table seg (nseg + 1 offsets into each right-hand side, device), per
// right-hand side and segment: out[2 (rh nseg + q)]
void residual_norms(int n6, int k, const double *r, const double *b, double *out, cudaStream_t st,
                    const int *seg = nullptr, int nseg = 1);

} // namespace lfg
