// lfg_solver.cpp -- the resistance solve behind LF_DEM's StokesSolver
// (StokesSolver.h:198-285), as a device object: compact block matrix in HBM,
// symbolic analysis on pattern change only (StokesSolver.cpp:955-962),
// multifrontal factorisation in FP64 or FP32, solves with k right-hand sides,
// FP64 iterative refinement for the FP32 form.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>

#include "lfg_solver.h"

namespace lfg {
int fail(lfg_status *st, int code, int info, const char *msg);

Solver::Solver(int n, const lfg_options &o, cudaStream_t st, int dof, bool analysis_only)
    : n_(n), dof_(dof), analysis_only_(analysis_only), opt_(o), st_(st)
{
	if (dof != 6 && dof != 3) throw Error{LFG_ERR_BAD_ARG, dof, "degrees of freedom per particle must be 6 or 3"};
	A_.n = n;
	A_.dof = dof;
	// pinned: staged values, norms, status (one allocation)
	LFG_CUDA(cudaMallocHost((void **)&h_pinned_, STAGE_BYTES+sizeof(double)*64+sizeof(int)*4));
	h_norms_ = reinterpret_cast<double *>(h_pinned_+STAGE_BYTES);
	h_status_ = reinterpret_cast<int *>(h_norms_+64);
	LFG_CUDA(cudaMalloc((void **)&d_norms_, sizeof(double)*64));
}

Solver::~Solver()
{
	dev_symbolic_free(D_);
	factor_free(F64_);
	factor_free(F32_);
	void *p[] = {block_mem_, d_norms_, ref_x_, ref_r_, hb_, hx_, d_seg_};
	for (void *q : p) if (q) cudaFree(q);
	if (h_segnorms_) cudaFreeHost(h_segnorms_);
	if (h_pinned_) cudaFreeHost(h_pinned_);
	for (auto &g : graphs_) if (g.exec) cudaGraphExecDestroy(g.exec);
}

void Solver::set_pattern(int nb, const int32_t *row, const int32_t *col, const double *pos, double lx,
                         double ly, double lz, bool device_ptrs)
{
	std::vector<int32_t> r(nb), c(nb);
	if (device_ptrs) {
		if (nb) {
			LFG_CUDA(cudaMemcpyAsync(r.data(), row, sizeof(int32_t)*nb, cudaMemcpyDeviceToHost, st_));
			LFG_CUDA(cudaMemcpyAsync(c.data(), col, sizeof(int32_t)*nb, cudaMemcpyDeviceToHost, st_));
			LFG_CUDA(cudaStreamSynchronize(st_));
		}
	} else {
		std::copy(row, row+nb, r.begin());
		std::copy(col, col+nb, c.begin());
	}
	for (int e = 0; e < nb; e++)
		if (r[e] <= c[e] || r[e] >= n_ || c[e] < 0)
			throw Error{LFG_ERR_BAD_ARG, e, "off-diagonal block must have n > row > col >= 0"};
	nb_ = nb;
	pat_r_ = r;
	pat_c_ = c;
	pat_pos_.assign(pos ? pos : nullptr, pos ? pos+3*(size_t)n_ : nullptr);
	pat_box_[0] = lx; pat_box_[1] = ly; pat_box_[2] = lz;
	drop_analysis();
	symbolic_analyze(S_, n_, nb, r.data(), c.data(), pos, lx, ly, lz, opt_.leaf_size, dof_);
	if (analysis_only_) {
		analyzed_ = true;
		symbolic_runs_++;
		return;
	}
	upload(r, c);
}

// A symbolic analysis made elsewhere (a joint analysis of several
// suspensions) for the pattern (row, col): upload and allocate as set_pattern.
void Solver::install(Symbolic &&S, int nb, const int32_t *row, const int32_t *col)
{
	if (S.nblk != n_ || S.dof != dof_) throw Error{LFG_ERR_BAD_ARG, S.nblk, "symbolic analysis of another system"};
	std::vector<int32_t> r(row, row+nb), c(col, col+nb);
	nb_ = nb;
	pat_r_ = r;
	pat_c_ = c;
	pat_pos_.clear();
	drop_analysis();
	S_ = std::move(S);
	upload(r, c);
}

// Before the tables and workspaces of an analysis change: until the new ones are
// complete (an analysis may be refused, an allocation fail) nothing is launched
// over them, and no graph that holds the old addresses stays.
void Solver::drop_analysis()
{
	analyzed_ = false;
	for (auto &g : graphs_) if (g.exec) cudaGraphExecDestroy(g.exec);
	graphs_.clear();
}

void Solver::require_analysis() const
{
	if (!analyzed_) throw Error{LFG_ERR_BAD_ARG, 0, "solve before set_blocks"};
}

void Solver::upload(const std::vector<int32_t> &r, const std::vector<int32_t> &c)
{
	const int nb = nb_;
	dev_symbolic_upload(D_, S_, opt_.precision, st_);
	if (opt_.precision == LFG_PREC_FP64) factor_alloc(F64_, D_, 4);
	else factor_alloc(F32_, D_, 4);
	// one allocation: block values (diagonal blocks padded to an even count), then
	// the pattern and its row adjacency for the residual, copied at once
	A_.nb = nb;
	const int64_t values = dvalues()+18*(int64_t)nb;
	std::vector<int> pattern(4*(size_t)nb+2*((size_t)n_+1), 0);
	device_grow(block_mem_, block_cap_, (int64_t)sizeof(double)*values+(int64_t)(sizeof(int)*pattern.size()));
	A_.dblocks = reinterpret_cast<double *>(block_mem_);
	A_.odblocks = A_.dblocks+dvalues();
	A_.od_row = reinterpret_cast<int *>(A_.dblocks+values);
	A_.od_col = A_.od_row+nb; A_.lo_idx = A_.od_col+nb; A_.up_idx = A_.lo_idx+nb;
	A_.lo_ptr = A_.up_idx+nb; A_.up_ptr = A_.lo_ptr+n_+1;
	int *li = pattern.data()+2*nb, *ui = li+nb, *lp = ui+nb, *upp = lp+n_+1;
	std::copy(r.begin(), r.end(), pattern.begin());
	std::copy(c.begin(), c.end(), pattern.begin()+nb);
	for (int e = 0; e < nb; e++) { lp[r[e]+1]++; upp[c[e]+1]++; }
	for (int i = 0; i < n_; i++) { lp[i+1] += lp[i]; upp[i+1] += upp[i]; }
	{
		std::vector<int> f1(lp, lp+n_), f2(upp, upp+n_);
		for (int e = 0; e < nb; e++) { li[f1[r[e]]++] = e; ui[f2[c[e]]++] = e; }
	}
	StreamDrain drain{st_};
	LFG_CUDA(cudaMemcpyAsync(A_.od_row, pattern.data(), sizeof(int)*pattern.size(), cudaMemcpyHostToDevice, st_));
	LFG_CUDA(cudaStreamSynchronize(st_));
	analyzed_ = true;
	symbolic_runs_++;
}

void Solver::reanalyze(int leaf_size)
{
	if (!analyzed_) throw Error{LFG_ERR_BAD_ARG, 0, "reanalyze before the first analysis"};
	if (leaf_size < 1) throw Error{LFG_ERR_BAD_ARG, leaf_size, "leaf size must be positive"};
	opt_.leaf_size = leaf_size;
	std::vector<int32_t> r = pat_r_, c = pat_c_;
	std::vector<double> pos = pat_pos_;
	set_pattern(nb_, r.data(), c.data(), pos.empty() ? nullptr : pos.data(), pat_box_[0], pat_box_[1], pat_box_[2],
	            false);
}

// The caller's arrays are its own again when this returns: small ones are staged
// in pinned memory and copied at once, the copies of others waited for (7 us more at N = 60, where
// the factorisation's launches otherwise overlap them; none at N = 500).
void Solver::set_values_host(const double *dblocks, const double *odblocks)
{
	const size_t bd = sizeof(double)*15*(size_t)n_, bo = sizeof(double)*18*(size_t)nb_, od = sizeof(double)*dvalues();
	if (od+bo <= STAGE_BYTES) {
		if (staged_) LFG_CUDA(cudaStreamSynchronize(st_));   // the copy of the values before
		staged_ = true;
		std::memcpy(h_pinned_, dblocks, bd);
		if (nb_) std::memcpy(h_pinned_+od, odblocks, bo);
		LFG_CUDA(cudaMemcpyAsync(A_.dblocks, h_pinned_, od+bo, cudaMemcpyHostToDevice, st_));
		return;
	}
	StreamDrain drain{st_};
	LFG_CUDA(cudaMemcpyAsync(A_.dblocks, dblocks, bd, cudaMemcpyHostToDevice, st_));
	if (nb_) LFG_CUDA(cudaMemcpyAsync(A_.odblocks, odblocks, bo, cudaMemcpyHostToDevice, st_));
	LFG_CUDA(cudaStreamSynchronize(st_));
}

// Launch the factorisation; with graphs, the launch sequence is captured once
// per symbolic analysis and replayed.
void Solver::factorize_async()
{
	if (!analyzed_) throw Error{LFG_ERR_BAD_ARG, 0, "factorize before set_blocks"};
	auto body = [&]() {
		if (opt_.precision == LFG_PREC_FP64) launches_factor_ = factor_numeric(F64_, D_, A_.dblocks, A_.odblocks, st_);
		else launches_factor_ = factor_numeric(F32_, D_, A_.dblocks, A_.odblocks, st_);
		return launches_factor_;
	};
	run_graph(0, 0, A_.dblocks, A_.odblocks, body);
}

// body launches its work and returns the number of kernels.  The first call of a
// kind and shape after an analysis launches directly, the second captures, later
// ones replay: a pattern that is factored once does not pay for a graph (3 us a
// launch to capture and instantiate; direct launches run ahead of the device).
void Solver::run_graph(int kind, int k, const void *b, const void *x, const std::function<int()> &body)
{
	if (!opt_.use_graphs) {
		kernels_ += body();
		return;
	}
	size_t at = 0;
	while (at < graphs_.size() && !(graphs_[at].kind == kind && graphs_[at].k == k && graphs_[at].b == b && graphs_[at].x == x))
		at++;
	if (at == graphs_.size()) {
		kernels_ += body();
		GraphEntry e;
		e.kind = kind; e.k = k; e.b = b; e.x = x;
		graphs_.push_back(e);
		return;
	}
	GraphEntry &e = graphs_[at];
	if (e.exec) {
		LFG_CUDA(cudaGraphLaunch(e.exec, st_));
		kernels_ += e.nodes;
		return;
	}
	auto t0 = std::chrono::steady_clock::now();
	cudaGraph_t graph;
	LFG_CUDA(cudaStreamBeginCapture(st_, cudaStreamCaptureModeThreadLocal));
	try {
		body();
	} catch (...) {
		cudaStreamEndCapture(st_, &graph);
		throw;
	}
	LFG_CUDA(cudaStreamEndCapture(st_, &graph));
	size_t nn = 0;
	LFG_CUDA(cudaGraphGetNodes(graph, nullptr, &nn));
	std::vector<cudaGraphNode_t> nodes(nn);
	if (nn) LFG_CUDA(cudaGraphGetNodes(graph, nodes.data(), &nn));
	e.nodes = 0;   // kernel nodes only (memsets and copies are not launches)
	for (size_t q = 0; q < nn; q++) {
		cudaGraphNodeType t;
		LFG_CUDA(cudaGraphNodeGetType(nodes[q], &t));
		if (t == cudaGraphNodeTypeKernel) e.nodes++;
	}
	LFG_CUDA(cudaGraphInstantiate(&e.exec, graph, 0));
	cudaGraphDestroy(graph);
	capture_ms_ += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now()-t0).count();
	LFG_CUDA(cudaGraphLaunch(e.exec, st_));
	kernels_ += e.nodes;
}

int Solver::check_factor(lfg_status *st)
{
	int *dst = opt_.precision == LFG_PREC_FP64 ? F64_.status : F32_.status;
	LFG_CUDA(cudaMemcpyAsync(h_status_, dst, sizeof(int), cudaMemcpyDeviceToHost, st_));
	LFG_CUDA(cudaStreamSynchronize(st_));
	staged_ = false;
	if (*h_status_ == 0) return fail(st, LFG_ERR_TIMEOUT, 0, "a bounded device wait gave up");
	if (*h_status_ != 0x7fffffff) {
		int q = *h_status_-1;
		// scalar column of the caller's 6-per-particle numbering (dof 3:
		// components 0, 2, 4)
		int orig = dof_ == 6 ? S_.perm[q/6]*6+q%6 : S_.perm[q/3]*6+2*(q%3);
		if (st) {
			st->code = LFG_ERR_NOT_SPD;
			st->info = orig+1;
			snprintf(st->msg, sizeof st->msg, "non-positive pivot at column %d (particle %d)", orig, orig/6);
		}
		return LFG_ERR_NOT_SPD;
	}
	return LFG_OK;
}

void Solver::ensure_refine_ws(int k)
{
	int64_t need = (int64_t)6*n_*std::max(k, 1);
	if (std::min(refx_cap_, refr_cap_) >= need) return;
	// graphs of refinement iterations hold these vectors' addresses
	for (size_t q = 0; q < graphs_.size();) {
		if (graphs_[q].kind != 2) { q++; continue; }
		if (graphs_[q].exec) cudaGraphExecDestroy(graphs_[q].exec);
		graphs_.erase(graphs_.begin()+q);
	}
	device_grow(ref_x_, refx_cap_, need);
	device_grow(ref_r_, refr_cap_, need);
}

// k RHS on the device.  FP64: one direct solve.  FP32: x = 0, repeat
// { d = (L L^T)_32^-1 r ; x += d ; r = b - A x } until max relative residual
// <= refine_tol.
int Solver::solve_device(int k, const double *b, double *x, lfg_status *st, bool sync_check)
{
	if (k <= 0) return LFG_OK;
	require_analysis();
	if (opt_.precision == LFG_PREC_FP64) {
		run_graph(1, k, b, x, [&]() { return launches_solve_ = factor_solve(F64_, D_, k, b, x, false, st_); });
		last_iters_ = 0;
		last_resid_ = 0;
		return LFG_OK;
	}
	refine_begin(k, b);
	int it = 0;
	double worst = 0;
	int batch = std::max(1, std::min(pred_iters_, opt_.refine_max_iter));
	while (it < opt_.refine_max_iter) {
		int j = std::min(batch, opt_.refine_max_iter-it);
		run_graph(2, k*64+j, b, nullptr, [&]() { return refine_iterations(k, b, j); });
		it += j;
		worst = refine_worst(k);
		if (worst <= opt_.refine_tol) break;
		batch = 1;
	}
	pred_iters_ = it;
	return refine_finish(k, x, it, worst, st);
}

// FP32 refinement in pieces.  refine_begin: x = 0, r = b.  refine_iterations:
// j times { x += (L L^T)_32^-1 r, solved in FP32; r = b - A x in FP64 }, then
// the squared norms of r and b per right-hand side (and per segment); these
// only launch work, so a caller may capture them in its own graph.
// refine_worst: waits and returns the largest relative residual.
// refine_finish: copies x out and records the counts.
void Solver::refine_begin(int k, const double *b)
{
	ensure_refine_ws(k);
	int64_t tot = (int64_t)6*n_*k;
	LFG_CUDA(cudaMemsetAsync(ref_x_, 0, sizeof(double)*tot, st_));
	LFG_CUDA(cudaMemcpyAsync(ref_r_, b, sizeof(double)*tot, cudaMemcpyDeviceToDevice, st_));
}

int Solver::refine_iterations(int k, const double *b, int j)
{
	for (int q = 0; q < j; q++) {
		launches_solve_ = factor_solve(F32_, D_, k, ref_r_, ref_x_, true, st_);
		block_residual(A_, k, b, ref_x_, ref_r_, st_);
	}
	residual_norms(6*n_, k, ref_r_, b, d_norms_, st_, seg_.empty() ? nullptr : d_seg_, (int)seg_.size()-1);
	return j*(launches_solve_+(k+3)/4)+1;   // sweeps and residuals, norms
}

double Solver::refine_worst(int k)
{
	int nseg = seg_.empty() ? 1 : (int)seg_.size()-1;
	LFG_CUDA(cudaMemcpyAsync(h_norms_, d_norms_, sizeof(double)*2*k*nseg, cudaMemcpyDeviceToHost, st_));
	LFG_CUDA(cudaStreamSynchronize(st_));
	double worst = 0;
	for (int r = 0; r < k*nseg; r++) {
		double rb = h_norms_[2*r+1] > 0 ? std::sqrt(h_norms_[2*r]/h_norms_[2*r+1]) : std::sqrt(h_norms_[2*r]);
		if (!(rb == rb)) rb = INFINITY;
		worst = std::max(worst, rb);
	}
	return worst;
}

int Solver::refine_finish(int k, double *x, int iters, double worst, lfg_status *st)
{
	int64_t tot = (int64_t)6*n_*k;
	last_iters_ = iters;
	last_resid_ = worst;
	LFG_CUDA(cudaMemcpyAsync(x, ref_x_, sizeof(double)*tot, cudaMemcpyDeviceToDevice, st_));
	if (st) { st->refine_iters = last_iters_; st->refine_residual = worst; }
	if (!(worst <= opt_.refine_tol)) {
		if (st) {
			st->code = LFG_ERR_NOT_CONVERGED;
			snprintf(st->msg, sizeof st->msg, "FP32 refinement reached %.3e after %d iterations", worst, last_iters_);
		}
		return LFG_ERR_NOT_CONVERGED;
	}
	return LFG_OK;
}

// Per-suspension segments of a joint system (particle offsets, nseg + 1):
// the refinement's convergence test takes the largest relative residual over
// the segments, so every suspension meets the tolerance on its own.
void Solver::set_segments(const std::vector<int> &particle_off)
{
	seg_.resize(particle_off.size());
	for (size_t q = 0; q < particle_off.size(); q++) seg_[q] = 6*particle_off[q];
	if (d_seg_) cudaFree(d_seg_);
	d_seg_ = nullptr;
	LFG_CUDA(cudaMalloc((void **)&d_seg_, sizeof(int)*std::max<size_t>(seg_.size(), 1)));
	LFG_CUDA(cudaMemcpyAsync(d_seg_, seg_.data(), sizeof(int)*seg_.size(), cudaMemcpyHostToDevice, st_));
	size_t need = 2*8*std::max<size_t>(seg_.size(), 2);
	if (need > norms_cap_) {
		if (h_segnorms_) cudaFreeHost(h_segnorms_);
		if (d_norms_) cudaFree(d_norms_);
		h_norms_ = h_segnorms_ = nullptr; d_norms_ = nullptr;
		norms_cap_ = 0;
		LFG_CUDA(cudaMallocHost((void **)&h_segnorms_, sizeof(double)*need));
		LFG_CUDA(cudaMalloc((void **)&d_norms_, sizeof(double)*need));
		h_norms_ = h_segnorms_;
		norms_cap_ = need;
	}
	LFG_CUDA(cudaStreamSynchronize(st_));
}

// StokesSolver::compute_LTRHS (StokesSolver.cpp:627-669): the Brownian
// force's L psi, with this factor's L (any L with L L^T = R gives the same
// statistics; the reference's CHOLMOD factor is another one)
void Solver::multiply_device(int k, const double *b, double *x)
{
	if (k <= 0) return;
	require_analysis();
	run_graph(3, k, b, x, [&]() {
		return opt_.precision == LFG_PREC_FP64 ? factor_multiply(F64_, D_, k, b, x, st_)
		                                       : factor_multiply(F32_, D_, k, b, x, st_);
	});
}

int Solver::multiply_host(int k, const double *rhs, double *x, lfg_status *st)
{
	int64_t tot = (int64_t)6*n_*k;
	device_grow(hb_, hb_cap_, tot);
	device_grow(hx_, hx_cap_, tot);
	StreamDrain drain{st_};
	LFG_CUDA(cudaMemcpyAsync(hb_, rhs, sizeof(double)*tot, cudaMemcpyHostToDevice, st_));
	multiply_device(k, hb_, hx_);
	LFG_CUDA(cudaMemcpyAsync(x, hx_, sizeof(double)*tot, cudaMemcpyDeviceToHost, st_));
	LFG_CUDA(cudaStreamSynchronize(st_));
	(void)st;
	return LFG_OK;
}

int Solver::solve_host(int k, const double *rhs, double *x, lfg_status *st)
{
	int64_t tot = (int64_t)6*n_*k;
	device_grow(hb_, hb_cap_, tot);
	device_grow(hx_, hx_cap_, tot);
	StreamDrain drain{st_};
	LFG_CUDA(cudaMemcpyAsync(hb_, rhs, sizeof(double)*tot, cudaMemcpyHostToDevice, st_));
	int rc = solve_device(k, hb_, hx_, st, true);
	LFG_CUDA(cudaMemcpyAsync(x, hx_, sizeof(double)*tot, cudaMemcpyDeviceToHost, st_));
	int *dst = opt_.precision == LFG_PREC_FP64 ? F64_.status : F32_.status;
	LFG_CUDA(cudaMemcpyAsync(h_status_+1, dst, sizeof(int), cudaMemcpyDeviceToHost, st_));
	LFG_CUDA(cudaStreamSynchronize(st_));
	if (h_status_[1] == 0) return fail(st, LFG_ERR_TIMEOUT, 0, "a bounded device wait gave up");
	return rc;
}

void Solver::stats(lfg_solver_stats *o) const
{
	std::memset(o, 0, sizeof *o);
	o->n_blocks = S_.nblk;
	o->n_supernodes = S_.nsn;
	o->n_levels = S_.nlevels;
	o->max_front = S_.max_F;
	o->nnz_L = S_.nnz_L;
	o->flops_factor = S_.flops;
	o->front_bytes = S_.arena_elems*(opt_.precision == LFG_PREC_FP64 ? 8 : 4);
	o->n_factor_launches = launches_factor_;
	o->n_solve_launches = launches_solve_;
}

} // namespace lfg
