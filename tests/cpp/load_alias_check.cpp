// The device loads' pointer arguments do not overlap: circuit.cpp with its calls of the
// loads replaced by ones that compare the spans.  Prints "0 failure(s)" on
// success.
#include "host/circuit.hpp"
#include "kernels/bsim4_model.cuh"
#include "kernels/mos1_model.cuh"

#include <cstdio>
#include <utility>
#include <vector>

namespace {
int failures = 0, loads = 0;

// spans of P, rec, s0, s1, s2 and t, in doubles
template <int kStates>
void compare(const double* P, const double* rec, const double* s0, const double* s1,
             const double* s2, const double* t) {
    const std::pair<const double*, int> span[] = {{P, 1},        {rec, nsg::kMosRec}, {s0, kStates},
                                                  {s1, kStates}, {s2, kStates},
                                                  {t, nsg::kMosTerms}};
    ++loads;
    for (int i = 0; i < 6; ++i)
        for (int j = 0; j < i; ++j)
            if (span[i].first < span[j].first + span[j].second &&
                span[j].first < span[i].first + span[i].second) {
                std::printf("failed: arguments %d and %d overlap (%d states)\n", j, i, kStates);
                ++failures;
            }
}
}  // namespace

namespace nsg {
void checked_mos1(const double* P, double* rec, double* s0, double* s1, const double* s2, int mode,
                  const Mos1Integ& ic, double gmin, const double v[4], double* t) {
    compare<kMosStates>(P, rec, s0, s1, s2, t);
    mos1_load(P, rec, s0, s1, s2, mode, ic, gmin, v, t);
}
void checked_bsim4(const double* P, double* rec, double* s0, double* s1, const double* s2,
                   int mode, const Mos1Integ& ic, double gmin, double reltol, double abstol,
                   const double v[4], double* t) {
    compare<kB4States>(P, rec, s0, s1, s2, t);
    bsim4_load(P, rec, s0, s1, s2, mode, ic, gmin, reltol, abstol, v, t);
}
}  // namespace nsg

#define mos1_load checked_mos1
#define bsim4_load checked_bsim4
#include "host/circuit.cpp"
#undef mos1_load
#undef bsim4_load

int main() {
    nsg::Circuit c(4);
    nsg::Mos1Card m1;
    m1.params = {{"VTO", 0.7}, {"KP", 1e-4}};
    const int32_t mod = c.add_mos1_model(m1);
    const int32_t b4 = c.add_bsim4_model(nsg::Bsim4Card{});
    c.add_vsource(0, -1, 1.8);
    c.add_resistor(0, 1, 1e3);
    c.add_resistor(0, 2, 1e3);
    c.add_resistor(0, 3, 1e3);
    c.add_mosfet(1, 0, -1, -1, mod, 1e-6, 1e-7);
    c.add_mosfet(2, 1, 3, -1, mod, 2e-6, 1e-7);
    c.add_bsim4(2, 1, -1, -1, b4, 1e-6, 1e-7, 0.0);
    c.add_bsim4(3, 2, 1, -1, b4, 1e-6, 1e-7, 0.0);
    c.finalize();
    std::vector<double> a, rhs;
    c.initjct_values(a, rhs, 1e-12);
    const std::vector<double> x(c.num_vars(), 0.1);
    std::vector<double> states(3 * c.num_states(), 0.0), rec(4 * nsg::kMosRec, 0.0);
    const nsg::Mos1Integ ic{0, 0, 0, 0, 0, 0, 1, 0};
    c.eval_values(nsg::kM1DcOp | nsg::kM1InitJct, x.data(), ic, 0.0, 1e-12, 1e-3, 1e-12,
                  states.data(), rec.data(), a, rhs);
    if (loads != 8) ++failures;
    std::printf("%d loads, %d failure(s)\n", loads, failures);
    return failures == 0 ? 0 : 1;
}
