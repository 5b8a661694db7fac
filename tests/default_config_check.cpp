// The FP64 configuration of a new handle by sector: with the fused form and,
// for the same sectors, where that form cannot run (fused_bn = 0).
// Prints "ok" or "FAIL <case>".
#include "kron_plan.h"

#include <cstdio>

using namespace dmrgpp;

int main()
{
	struct Case {
		size_t    np;
		long long l, r;
		double    f_alg;
		bool      fused;
		int       cfg, without; // two-pass configuration (without the fused form)
	};
	const Case cases[] = {
		{ 1, 1, 1, 4.0, true, 0, 1 },             // one state
		{ 21, 101, 101, 1.3e8, true, 0, 1 },      // microbench sector
		{ 40, 128, 400, 3.9e8, true, 0, 1 },      // the edges of the fused rule ...
		{ 41, 128, 400, 3.9e8, false, 1, 1 },     // ... and one step past each
		{ 40, 129, 400, 3.9e8, false, 1, 1 },
		{ 40, 128, 400, 4e8, false, 1, 1 },
		{ 200, 300, 320, 6e8, false, 0, 0 },
		{ 200, 300, 320, 5.9e8, false, 1, 1 },
		{ 300, 500, 500, 2.5e10, false, 2, 2 },
		{ 300, 500, 500, 2.4e10, false, 0, 0 },
	};
	int n = 0;
	for (const Case& c : cases) {
		KronPlan plan;
		plan.np = c.np;
		plan.l.assign(c.np, 1);
		plan.r.assign(c.np, 1);
		plan.l.back() = c.l;
		plan.r.back() = c.r;
		plan.f_alg    = c.f_alg;
		const DefaultConfig a = default_config(plan, 128), b = default_config(plan, 0);
		if (a.fused != c.fused || (!a.fused && a.cfg != c.cfg) || a.items_per_cta != (c.fused ? 1 : 2) || b.fused
		    || b.cfg != c.without || b.items_per_cta != 2) {
			std::printf("FAIL %d\n", n);
			return 1;
		}
		++n;
	}
	std::printf("ok\n");
	return 0;
}
