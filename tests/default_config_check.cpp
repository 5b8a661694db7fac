// The FP64 configuration of a new handle by sector, on both sides of every
// line of the rule, and where the fused form cannot run (no cluster resident).
// Prints "ok" or "FAIL <case>".
#include "kron_plan.h"

#include <cstdio>

using namespace dmrgpp;

int main()
{
	struct Case {
		size_t    np;
		long long l, r; // every patch
		double    f_alg;
		int       clusters; // resident
		bool      fused;
		int       cfg; // of two passes
	};
	const Case cases[] = {
		{ 1, 1, 1, 4.0, 33, true, 1 },        // one state
		{ 1, 1, 1, 4.0, 0, false, 1 },        // ... no cluster fits
		{ 21, 101, 101, 1.3e8, 33, true, 1 }, // 84 tiles: 11 clusters without terms
		{ 21, 101, 101, 1.3e8, 11, true, 1 },
		{ 21, 101, 101, 1.3e8, 10, false, 1 }, // a second round
		{ 40, 128, 32, 3.9e8, 33, true, 1 },
		{ 41, 128, 32, 3.9e8, 33, false, 1 },
		{ 40, 129, 32, 3.9e8, 33, false, 1 },
		{ 40, 128, 32, 4e8, 33, false, 1 },
		{ 2, 16, 256, 1e7, 33, true, 1 },
		{ 2, 16, 257, 1e7, 33, false, 1 },
		{ 200, 300, 320, 6e8, 33, false, 0 },
		{ 200, 300, 320, 5.9e8, 33, false, 1 },
		{ 300, 500, 500, 2.5e10, 33, false, 2 },
		{ 300, 500, 500, 2.4e10, 33, false, 0 },
	};
	int n = 0;
	for (const Case& c : cases) {
		KronPlan plan;
		plan.np = c.np;
		plan.l.assign(c.np, c.l);
		plan.r.assign(c.np, c.r);
		for (size_t p = 0; p <= c.np; ++p)
			plan.xy_start.push_back((long long)p * c.l * c.r);
		plan.f_alg            = c.f_alg;
		const DefaultConfig d = default_config(plan, 32, 128, 64, 8, c.clusters);
		if (d.fused != c.fused || (!d.fused && d.cfg != c.cfg) || d.items_per_cta != (c.fused ? 1 : 2)) {
			std::printf("FAIL %d\n", n);
			return 1;
		}
		++n;
	}
	std::printf("ok\n");
	return 0;
}
