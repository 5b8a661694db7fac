// Host emulation of the persistent and fused FP64 H*x on sectors with identity blocks,
// whose terms skip pass 1 (kSegXA, kSegXB in kron_plan.h), against H*x from the
// caller's blocks with every identity multiplied out.
// Usage: identity_schedule_check seed npatches max_size
// Prints "ok <max relative error> <identity terms>" or "FAIL <reason>".
#include "kron_plan.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <map>
#include <random>
#include <vector>

using namespace dmrgpp;

namespace {
int fail(const std::string& why)
{
	std::printf("FAIL %s\n", why.c_str());
	return 1;
}
const double kNaN = std::numeric_limits<double>::quiet_NaN();
} // namespace

int main(int argc, char** argv)
{
	if (argc < 4)
		return fail("usage");
	std::mt19937_64                        rng{ unsigned(std::atoi(argv[1])) };
	const size_t                           np = size_t(std::atoi(argv[2])), nop = 5;
	std::uniform_int_distribution<size_t>  size(1, size_t(std::atoi(argv[3])));
	std::uniform_real_distribution<double> val(-1.0, 1.0), coin(0.0, 1.0);
	std::vector<size_t>                    l(np), r(np);
	for (size_t p = 0; p < np; ++p) { // some equal sizes: identities off the diagonal too
		l[p] = p > 0 && coin(rng) < 0.3 ? l[p - 1] : size(rng);
		r[p] = p > 0 && coin(rng) < 0.3 ? r[p - 1] : size(rng);
	}
	const size_t                     nt = np * np * nop;
	std::vector<std::vector<double>> store;
	std::vector<const double*>       A(nt, nullptr), B(nt, nullptr);
	std::vector<size_t>              ldA(nt, 0), ldB(nt, 0);
	store.reserve(2 * nt);
	int idents = 0;
	for (size_t k = 0; k < nop; ++k)
		for (size_t j = 0; j < np; ++j)
			for (size_t i = 0; i < np; ++i) {
				if (i != j && coin(rng) < 0.5)
					continue;
				const size_t t = i + j * np + k * np * np;
				bool         id = false;
				auto         block = [&](size_t rows, size_t cols, bool eye, size_t& ld) {
                    ld = rows + (coin(rng) < 0.3 ? 2 : 0);
                    store.emplace_back(ld * cols, 7.0);
                    for (size_t c = 0; c < cols; ++c)
                        for (size_t q = 0; q < rows; ++q)
                            store.back()[q + c * ld] = eye ? (q == c ? 1.0 : 0.0) : val(rng);
                    id = id || eye;
                    return store.back().data();
				};
				// almost an identity is none: one off-diagonal entry
				const bool near = coin(rng) < 0.1 && l[i] > 1;
				A[t] = block(l[i], l[j], (k == 0 || k == 2) && l[i] == l[j] && coin(rng) < 0.8, ldA[t]);
				if (near && id && l[i] == l[j])
					store.back()[1] = 1e-30;
				B[t] = block(r[i], r[j], (k == 1 || k == 2) && r[i] == r[j] && coin(rng) < 0.8, ldB[t]);
			}
	KronPlan          plan;
	PackBuffer        pack;
	const std::string msg
	    = build_kron_plan(nop, np, l.data(), r.data(), A.data(), ldA.data(), B.data(), ldB.data(), 64, 64, plan, &pack);
	if (!msg.empty())
		return fail(msg);
	for (int id : plan.ident)
		idents += id != 0;
	const size_t        D = size_t(plan.dim());
	std::vector<double> x(D), ref(D, 0.0);
	for (double& v : x)
		v = val(rng);
	for (size_t t = 0; t < plan.triples.size(); ++t) {
		const size_t    i = size_t(plan.triples[t].i), j = size_t(plan.triples[t].j);
		const BlockRef& b = plan.blocks[t];
		for (size_t c = 0; c < l[j]; ++c)
			for (size_t q = 0; q < r[i]; ++q) {
				double s = 0.0;
				for (size_t k = 0; k < r[j]; ++k)
					s += b.B[q + k * b.ldB] * x[size_t(plan.xy_start[j]) + k + c * r[j]];
				for (size_t n = 0; n < l[i]; ++n)
					ref[size_t(plan.xy_start[i]) + q + n * r[i]] += s * b.A[n + c * b.ldA];
			}
	}
	double scale = 1e-300, e64 = 0.0;
	for (double v : ref)
		scale = std::max(scale, std::fabs(v));

	for (int tile : { 32, 64 })
		for (int ipc : { 1, 4 }) {
			build_tile_lists(plan, tile, tile);
			build_persistent_schedule(plan, 16, 444, ipc);
			const std::string verdict = validate_persistent_schedule(plan, tile);
			if (!verdict.empty())
				return fail("validator: " + verdict);
			std::vector<double> bx(size_t(plan.bx_elems) + 1, kNaN), y(D, 0.0);
			std::vector<int>    written(D, 0);
			for (const KronItem& w : plan.items)
				for (int n = w.n0; n < std::min(w.n0 + tile, w.N); ++n)
					for (int m = w.m0; m < std::min(w.m0 + tile, w.M); ++m) {
						double s = 0.0;
						for (int e = w.seg_begin; e < w.seg_end; ++e) {
							const GemmSeg& g = w.kind == 0 ? plan.seg1[size_t(e)] : plan.pseg2[size_t(e)];
							const double*  a = w.kind == 0 || g.dep == kSegXB ? pack.data()
							                  : g.dep == kSegXA               ? x.data()
							                                                  : bx.data();
							const double*  b = w.kind == 0 || g.dep == kSegXB ? x.data() : pack.data();
							for (int k = 0; k < g.K; ++k)
								s += a[g.a_off + m + (long long)k * g.lda] * b[g.b_off + k + (long long)n * g.ldb];
						}
						const size_t at = size_t(w.c_off + m + (long long)n * w.ldc);
						if (w.kind == 0) {
							bx[at] = s;
						} else {
							y[at] += s;
							written[at] += w.kind == 1 || w.part == 0;
						}
					}
			for (size_t q = 0; q < D; ++q) {
				if (written[q] != 1)
					return fail("y element not written once");
				if (!(std::fabs(y[q] - ref[q]) <= 1e-12 * scale))
					return fail("FP64 H*x differs");
				e64 = std::max(e64, std::fabs(y[q] - ref[q]) / scale);
			}
		}

	// the fused form's units (its tiles 32 rows high, 64 or 128 columns wide)
	for (int bn : { 64, 128 }) {
		build_fused_schedule(plan, 32, bn, 64, 8, 2, 1184);
		const std::string verdict = validate_fused_schedule(plan, 32, bn, 8);
		if (!verdict.empty())
			return fail("fused validator: " + verdict);
		std::vector<double> y(D, 0.0);
		for (const FusedItem& it : plan.fitems) {
			if (it.nparts == 0)
				continue;
			for (int n = it.n0; n < std::min(it.n0 + bn, it.N); ++n)
				for (int m = it.m0; m < std::min(it.m0 + 32, it.M); ++m) {
					double s = 0.0;
					for (int u = it.u_begin; u < it.u_end; ++u) {
						const FusedUnit& d = plan.funits[size_t(u)];
						for (int c = 0; c < d.cw; ++c) {
							double t = 0.0;
							if (d.kind == kSegXA) {
								t = x.at(size_t(d.x_off + m + (long long)c * d.rj));
							} else if (d.kind == kSegXB) {
								s += pack.at(size_t(d.b_off + m + (long long)c * d.ldb))
								    * x.at(size_t(d.x_off + c + (long long)n * d.rj));
								continue;
							} else {
								for (int k = 0; k < d.rj; ++k)
									t += pack.at(size_t(d.b_off + m + (long long)k * d.ldb))
									    * x.at(size_t(d.x_off + k + (long long)c * d.rj));
							}
							s += t * pack.at(size_t(d.at_off + c + (long long)n * d.lj));
						}
					}
					y[size_t(it.y_off + m + (long long)n * it.M)] += s;
				}
		}
		for (size_t q = 0; q < D; ++q)
			if (!(std::fabs(y[q] - ref[q]) <= 1e-12 * scale))
				return fail("fused H*x differs");
	}
	std::printf("ok %.2e %d\n", e64, idents);
	return 0;
}
