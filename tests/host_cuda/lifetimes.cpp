// lifetimes.cpp -- host memory handed to asynchronous copies lives until they are
// done (see fake_cudart.cpp); argument: which path
#include <cstdio>
#include <cstring>
#include <list>
#include <string>
#include <vector>

#include "lfdem_gb300.h"

static lfg_solver *solver(int n, int precision, lfg_status *st)
{
	lfg_options o;
	lfg_default_options(&o);
	o.precision = precision;
	lfg_solver *s = nullptr;
	if (lfg_solver_create(n, 6, &o, &s, st)) printf("create: %s\n", st->msg);
	return s;
}

// new values, from memory that is gone when this returns or (keep) stays
static void set_blocks(lfg_solver *s, int n, int changed, bool keep, lfg_status *st)
{
	static std::list<std::vector<double>> kept;
	std::vector<double> d(15*n, 1.0), od(18*(n-1), 0.1);
	std::vector<int32_t> r(n-1), c(n-1);
	for (int i = 1; i < n; i++) { r[i-1] = i; c[i-1] = i-1; }
	if (lfg_solver_set_blocks(s, d.data(), n-1, r.data(), c.data(), od.data(), changed, nullptr, st))
		printf("set_blocks: %s\n", st->msg);
	if (!keep) return;
	kept.push_back(std::move(d));
	kept.push_back(std::move(od));
}

int main(int argc, char **argv)
{
	const std::string what = argc > 1 ? argv[1] : "";
	lfg_status st;
	memset(&st, 0, sizeof st);
	if (what == "analysis" || what == "values") {
		for (int precision : {LFG_PREC_FP64, LFG_PREC_FP32_REFINE})
			for (int n : {2, 60, 700}) {
				lfg_solver *s = solver(n, precision, &st);
				set_blocks(s, n, 1, what == "analysis", &st);
				if (what == "values")
					for (int turn = 0; turn < 3; turn++) set_blocks(s, n, 0, false, &st);
				lfg_solver_factorize(s, &st);   // waits
				lfg_solver_destroy(s);
			}
	} else if (what == "superset") {
		// a member of a fused batch only analyses its pattern
		lfg_params p;
		memset(&p, 0, sizeof p);
		p.kn = 1e4; p.kt = 5e3; p.lubrication_model = 2; p.lub_reduce_parameter = 1e-3; p.lub_max_gap = 0.5;
		p.interaction_range = -1; p.sd_coeff = 1; p.contact_relaxation_time = 1e-3; p.contact_relaxation_time_tan = -1;
		p.disp_max = 1e-3; p.dt = 1e-4; p.dt_max = p.dt_min = -1; p.integration_method = 1; p.shear_rate = 1;
		p.friction_model = 1; p.mu_static = p.mu_dynamic = 1; p.Ehat[2] = 0.5; p.Ohat[1] = 0.5;
		const int n = 40;
		std::vector<double> pos(3*n), rad(n, 1.0);
		for (int i = 0; i < 3*n; i++) pos[i] = 20.0*i/(3*n);
		lfg_options o;
		lfg_default_options(&o);
		lfg_batch *b = nullptr;
		int slot = -1;
		if (lfg_batch_create_fused(0, LFG_PREC_FP64, &b, &st)) printf("create: %s\n", st.msg);
		if (lfg_batch_add(b, &p, &o, n, pos.data(), rad.data(), 20, 20, 20, nullptr, &slot, &st)) printf("add: %s\n", st.msg);
		lfg_batch_destroy(b);
	} else return 2;
	printf("done %s\n", what.c_str());
	return 0;
}
