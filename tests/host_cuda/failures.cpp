// failures.cpp -- a pattern whose allocation fails part way (see fake_cudart.cpp):
// nothing is launched over half-replaced tables and workspaces, and the next
// pattern finds every buffer it needs
#include <cstdio>
#include <cstring>
#include <vector>

#include "lfdem_gb300.h"

extern "C" void fake_fail_malloc(long at);
extern "C" long fake_launches();
extern "C" long fake_live();

static int bad = 0;
#define CHECK(c) do { if (!(c)) { printf("%s:%d: %s\n", __FILE__, __LINE__, #c); bad++; } } while (0)

static const int N = 300;

static lfg_solver *solver(int precision)
{
	lfg_options o;
	lfg_default_options(&o);
	o.precision = precision;
	lfg_solver *s = nullptr;
	lfg_status st;
	CHECK(lfg_solver_create(N, 6, &o, &s, &st) == LFG_OK);
	return s;
}

// every particle coupled to the `band` before it
static int set_blocks(lfg_solver *s, int band)
{
	std::vector<int32_t> r, c;
	for (int i = 0; i < N; i++)
		for (int j = i-band < 0 ? 0 : i-band; j < i; j++) { r.push_back(i); c.push_back(j); }
	std::vector<double> d(15*N, 1.0), od(18*r.size(), 0.1);
	lfg_status st;
	return lfg_solver_set_blocks(s, d.data(), (int)r.size(), r.data(), c.data(), od.data(), 1, nullptr, &st);
}

// refused, and nothing launched
static void refused(lfg_solver *s, bool factorize)
{
	std::vector<double> b(6*N, 1.0), x(6*N);
	lfg_status st;
	const long before = fake_launches();
	if (factorize) CHECK(lfg_solver_factorize(s, &st) == LFG_ERR_BAD_ARG);
	CHECK(lfg_solver_solve(s, 1, b.data(), x.data(), &st) == LFG_ERR_BAD_ARG);
	CHECK(lfg_solver_multiply_factor(s, 1, b.data(), x.data(), &st) == LFG_ERR_BAD_ARG);
	CHECK(fake_launches() == before);
}

int main()
{
	lfg_status st;
	for (int precision : {LFG_PREC_FP64, LFG_PREC_FP32_REFINE}) {
		lfg_solver *f = solver(precision);
		refused(f, true);
		const long empty = fake_live();
		set_blocks(f, 2);
		const long fresh = fake_live()-empty;
		lfg_solver_destroy(f);
		int failed = 0;
		for (int at = 0; ; at++) {
			lfg_solver *s = solver(precision);
			std::vector<double> b(24*N, 1.0), x(24*N);
			const long none = fake_live();
			CHECK(set_blocks(s, 2) == LFG_OK);
			for (int turn = 0; turn < 3; turn++) {   // the third replays graphs
				lfg_solver_factorize(s, &st);
				lfg_solver_solve(s, 1, b.data(), x.data(), &st);
			}
			fake_fail_malloc(at);
			const int rc = set_blocks(s, 40);
			fake_fail_malloc(-1);
			if (rc != LFG_OK) {
				failed++;
				CHECK(rc == LFG_ERR_OOM);
				refused(s, true);
				CHECK(set_blocks(s, 2) == LFG_OK);
				CHECK(fake_live()-none >= fresh);
				const long before = fake_launches();
				CHECK(lfg_solver_factorize(s, &st) != LFG_ERR_OOM);   // not the error of before
				CHECK(fake_launches() > before);
			}
			lfg_solver_destroy(s);
			if (rc == LFG_OK) break;
		}
		CHECK(failed > 20);
		for (int at = 0; at < 4; at++) {   // the vectors of a solve
			lfg_solver *s = solver(precision);
			std::vector<double> b(24*N, 1.0), x(24*N);
			set_blocks(s, 2);
			lfg_solver_factorize(s, &st);
			lfg_solver_solve(s, 1, b.data(), x.data(), &st);
			const long one = fake_live();
			fake_fail_malloc(at);
			lfg_solver_solve(s, 4, b.data(), x.data(), &st);
			fake_fail_malloc(-1);
			lfg_solver_solve(s, 1, b.data(), x.data(), &st);
			CHECK(fake_live() >= one);
			lfg_solver_destroy(s);
		}
	}
	// a fused batch's member has no blocks of its own to assemble into
	lfg_params p;
	memset(&p, 0, sizeof p);
	p.kn = 1e4; p.kt = 5e3; p.lubrication_model = 2; p.lub_reduce_parameter = 1e-3; p.lub_max_gap = 0.5;
	p.interaction_range = -1; p.sd_coeff = 1; p.contact_relaxation_time = 1e-3; p.contact_relaxation_time_tan = -1;
	p.disp_max = 1e-3; p.dt = 1e-4; p.dt_max = p.dt_min = -1; p.integration_method = 1; p.shear_rate = 1;
	p.friction_model = 1; p.mu_static = p.mu_dynamic = 1; p.Ehat[2] = 0.5; p.Ohat[1] = 0.5;
	std::vector<double> pos(3*N), rad(N, 1.0), d(15*N), od(18*N);
	for (int i = 0; i < 3*N; i++) pos[i] = 40.0*i/(3*N);
	std::vector<int32_t> r(N), c(N);
	lfg_batch *batch = nullptr;
	int slot = -1, nb = 0;
	CHECK(lfg_batch_create_fused(0, LFG_PREC_FP64, &batch, &st) == LFG_OK);
	CHECK(lfg_batch_add(batch, &p, nullptr, N, pos.data(), rad.data(), 40, 40, 40, nullptr, &slot, &st) == LFG_OK);
	const long before = fake_launches();
	CHECK(lfg_sim_assemble(lfg_batch_sim(batch, slot), d.data(), r.data(), c.data(), od.data(), N, &nb) == LFG_ERR_BAD_ARG);
	CHECK(fake_launches() == before);
	lfg_batch_destroy(batch);
	printf("%d\n", bad);
	return bad != 0;
}
