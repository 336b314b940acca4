// plans.cpp -- which FP32 fronts are updated two-level, and what the launch plan and
// the workspace hold for them (on fake_cudart.cpp: device tables are host memory)
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../lf_dem_gb300/csrc/lfg_internal.h"

using namespace lfg;

static int bad = 0;
#define CHECK(c) do { if (!(c)) { printf("%s:%d: %s\n", __FILE__, __LINE__, #c); bad++; } } while (0)

static cudaStream_t st;

// a cubic lattice of m^3 particles, each coupled to its 26 neighbours
static Symbolic lattice(int m, int leaf)
{
	std::vector<int32_t> r, c;
	std::vector<double> pos;
	for (int i = 0; i < m*m*m; i++) {
		const int x = i/(m*m), y = i/m%m, z = i%m;
		for (double v : {x+0.5, y+0.5, z+0.5}) pos.push_back(v);
		for (int j = 0; j < i; j++)
			if (abs(j/(m*m)-x) < 2 && abs(j/m%m-y) < 2 && abs(j%m-z) < 2) { r.push_back(i); c.push_back(j); }
	}
	Symbolic S;
	symbolic_analyze(S, m*m*m, (int)r.size(), r.data(), c.data(), pos.data(), 100, 100, 100, leaf, 6);
	return S;
}

// two cliques of a and b particles, both coupled to all of a third of s between them:
// fronts of (a, s), (b, s) and (s, 0) particles
static Symbolic cliques(int a, int b, int s)
{
	std::vector<int32_t> r, c;
	std::vector<double> pos;
	auto part = [&](int i) { return i < a ? 0 : i < a+s ? 1 : 2; };
	for (int i = 0; i < a+b+s; i++) {
		for (double v : {10.0*part(i)+1+1e-3*i, 1.0, 1.0}) pos.push_back(v);
		for (int j = 0; j < i; j++)
			if (part(i)-part(j) < 2) { r.push_back(i); c.push_back(j); }
	}
	Symbolic S;
	symbolic_analyze(S, a+b+s, (int)r.size(), r.data(), c.data(), pos.data(), 100, 100, 100, a > b ? a : b, 6);
	return S;
}

struct Plan { DevSymbolic D; int panel_split = 0, trail_split = 0; };

static Plan plan(const Symbolic &S)
{
	Plan p;
	dev_symbolic_upload(p.D, S, LFG_PREC_FP32_REFINE, st);
	for (const auto &L : p.D.factor_plan)
		if (L.count > 0) {
			p.panel_split += L.kind == PLAN_PANEL_SPLIT;
			p.trail_split += L.kind == PLAN_TRAIL_SPLIT;
		}
	return p;
}

static bool two(const Plan &p, int s) { return p.D.split_off && p.D.split_off[3*s] >= 0; }

int main()
{
	cudaStreamCreateWithFlags(&st, 0);
	// a batch of many small suspensions: thousands of tiles in its leaf level, but no
	// front with more than one outer block
	std::vector<Symbolic> parts;
	for (int q = 0; q < 48; q++) parts.push_back(lattice(6+q%6, 32));
	std::vector<const Symbolic *> ptr;
	for (const Symbolic &P : parts) ptr.push_back(&P);
	Symbolic J;
	symbolic_concat(J, ptr);
	Plan small = plan(J);
	CHECK(small.panel_split == 0 && small.trail_split == 0);
	CHECK(small.D.ybuf_elems == 0 && small.D.rexp_elems == 0);

	// fronts of 4080 rows (2580 columns) and 3300 rows (1800 columns) in one level
	Symbolic A = cliques(430, 300, 250);
	CHECK(A.nsn == 3 && A.nlevels == 2 && A.max_F == 680*6);
	Plan pa = plan(A);
	int large = -1;
	for (int s = 0; s < A.nsn; s++)
		if (A.sn_n[s] == 430) large = s;
	CHECK(large >= 0);
	for (int s = 0; s < A.nsn; s++) CHECK(two(pa, s) == (s == large));
	// 41 panels, ten of them before the last end an outer block
	CHECK(pa.trail_split == 10);
	CHECK(pa.D.rexp_elems == (int64_t)41*A.sn_ld[large]);
	CHECK(pa.D.yexp_elems == (int64_t)10*A.sn_ld[large]);
	CHECK(pa.D.ybuf_elems == (int64_t)16*(10*16*(int64_t)A.sn_ld[large]+128));

	// the same among others: the same fronts
	ptr.insert(ptr.begin()+7, &A);
	Symbolic K;
	symbolic_concat(K, ptr);
	Plan pk = plan(K);
	int count = 0, found = 0;
	for (int s = 0; s < K.nsn; s++) {
		count += two(pk, s);
		found += K.sn_n[s] == 430 && two(pk, s);
	}
	CHECK(count == 1 && found == 1);
	CHECK(pk.trail_split == 10 && pk.D.ybuf_elems == pa.D.ybuf_elems);

	// columns a multiple of the outer block: none are left after the last one
	Symbolic W = cliques(768, 1, 1);
	Plan pw = plan(W);
	for (int s = 0; s < W.nsn; s++)
		if (two(pw, s)) CHECK(pw.D.yexp_elems == (int64_t)((6*W.sn_n[s]-1)/256)*W.sn_ld[s]);
	for (Plan *p : {&small, &pa, &pk, &pw}) dev_symbolic_free(p->D);
	printf("%d\n", bad);
	return bad != 0;
}
