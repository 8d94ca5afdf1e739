// Level programs against the column-wise refactor and row-wise sweeps.  For
// seeded sparse matrices of many sizes (1 unknown up to the program's bound
// and past it), the packed program is run step after step the way a kernel
// runs it (every lane's operands read before any lane stores) and must give
// the column-wise factor, pivots, solution and transposed solution bit for bit;
// every index must lie in its array, every step hold at most 32 entries, and
// no entry of a step read what an entry of the step writes.  Prints
// "0 failure(s)" on success.
#include "host/plan.hpp"
#include "host/sparse_order.hpp"

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <set>
#include <vector>

namespace {

int failures = 0;

void fail(const char* what, int n, int seed) {
    if (++failures < 20) std::printf("%s (n %d, seed %d)\n", what, n, seed);
}

bool same(double a, double b) { return std::memcmp(&a, &b, sizeof a) == 0; }

// Unfused, separately rounded multiply and subtract.
double msub(double t, double a, double b) {
    volatile double p = a * b;
    volatile double r = t - p;
    return r;
}

void run_steps(const nsg::TopologyPlan& p, int section, std::vector<double>& V, int seed) {
    const int32_t words = static_cast<int32_t>(p.lp.size());
    const int32_t limit = section < 2 ? p.lp_core : words;
    const int32_t values = p.lp_doubles();
    for (int r = section ? p.lp_steps[section - 1] : 0; r < p.lp_steps[section]; ++r) {
        nsg::LevelStep d;
        if (4 * (r + 1) > words) return fail("step index", p.n, seed);
        std::memcpy(&d, p.lp.data() + 4 * r, sizeof d);
        const int w = static_cast<int>(d.last) + 1;
        if (w < 1 || w > 32 || d.entries % 4 || d.terms % 8) return fail("step", p.n, seed);
        if (static_cast<int32_t>(d.entries / 4) + w > limit ||
            static_cast<int32_t>(d.terms / 4) + 2 * nsg::kLevelTerms * w > limit)
            return fail("section bounds", p.n, seed);
        std::vector<std::pair<int32_t, double>> out;
        std::set<int32_t> writes, reads;
        bool pivots = false;
        for (int e = 0; e < w; ++e) {
            const uint32_t x = static_cast<uint32_t>(p.lp[d.entries / 4 + e]);
            const int32_t target = (x & 0xfff8) / 8, aux = (x >> 16) / 8;
            if (target >= p.nnz_lu + p.n || aux >= values || (x >> 16) % 8)
                return fail("operand", p.n, seed);
            double t = V[target];
            if (section == 1 && t != 0.0) t *= V[aux];
            for (int k = 0; k < nsg::kLevelTerms; ++k) {
                const int32_t at = static_cast<int32_t>(d.terms / 4) + 2 * (k * w + e);
                const uint32_t y = static_cast<uint32_t>(p.lp[at]);
                const uint32_t y2 = static_cast<uint32_t>(p.lp[at + 1]);
                const int32_t a = (y & 0xffff) / 8, s = (y >> 16) / 8, b = y2 / 8;
                if (a >= values || s >= values || b >= values || (y & 7) || (y >> 16) % 8 || y2 % 8)
                    return fail("term", p.n, seed);
                for (int32_t v : {a, s, b}) reads.insert(v);
                volatile double u = V[a] * V[s];
                if (section == 0 && (x & nsg::kLevelSkip) && (V[a] == 0.0 || u == 0.0)) continue;
                if (section == 2 && V[b] == 0.0) continue;
                t = msub(t, u, V[b]);
            }
            if (section == 0 && (x & nsg::kLevelPivot)) {
                pivots = true;
                out.push_back({aux, t});
                writes.insert(aux);
                t = 1.0 / t;
            }
            if (section == 3) t *= V[aux];
            if (section == 1 || section == 3) reads.insert(aux);
            if (!writes.insert(target).second) fail("two writers in a step", p.n, seed);
            out.push_back({target, t});
        }
        if (pivots != (d.pivots != 0)) fail("pivot flag", p.n, seed);
        for (int32_t x : writes)
            if (reads.count(x)) fail("operand written in its step", p.n, seed);
        for (const auto& o : out) V[o.first] = o.second;
    }
}

void check(const nsg::TopologyPlan& p, const std::vector<double>& a, std::mt19937_64& g, int seed) {
    const int n = p.n;
    std::vector<double> lu(p.nnz_lu), piv(n);
    for (int q = 0; q < p.nnz_lu; ++q) lu[q] = p.lu_src[q] >= 0 ? a[p.lu_src[q]] : 0.0;
    for (int j = 0; j < n; ++j) {
        for (int q = p.col_ptr[j]; q < p.diag_pos[j]; ++q) {
            const int r = p.row_idx[q];
            lu[q] *= lu[p.diag_pos[r]];
            for (int k = p.diag_pos[r] + 1; k < p.col_ptr[r + 1]; ++k) {
                const int d = p.col_ptr[j] + p.upd_dst[p.upd_start[q] + k - p.diag_pos[r] - 1];
                lu[d] = msub(lu[d], lu[q], lu[k]);
            }
        }
        piv[j] = lu[p.diag_pos[j]];
        lu[p.diag_pos[j]] = 1.0 / piv[j];
    }
    std::vector<double> b(n), x(n), xt(n), w(n);
    std::normal_distribution<double> nd;
    for (double& v : b) v = (g() % 4 == 0) ? 0.0 : nd(g);
    for (int i = 0; i < n; ++i) {
        double t = b[p.perm_row[i]];
        for (int k = p.lrow_ptr[i]; k < p.lrow_ptr[i + 1]; ++k)
            if (w[p.lrow_col[k]] != 0.0) t = msub(t, w[p.lrow_col[k]], lu[p.lrow_pos[k]]);
        w[i] = t != 0.0 ? t * lu[p.diag_pos[i]] : t;
    }
    for (int i = n - 1; i >= 0; --i)
        for (int k = p.urow_ptr[i]; k < p.urow_ptr[i + 1]; ++k)
            w[i] = msub(w[i], lu[p.urow_pos[k]], w[p.urow_col[k]]);
    for (int i = 0; i < n; ++i) x[p.perm_col[i]] = w[i];
    for (int c = 0; c < n; ++c) {
        w[c] = b[p.perm_col[c]];
        for (int q = p.col_ptr[c]; q < p.diag_pos[c]; ++q)
            if (w[p.row_idx[q]] != 0.0) w[c] = msub(w[c], w[p.row_idx[q]], lu[q]);
    }
    for (int i = n - 1; i >= 0; --i) {
        for (int q = p.diag_pos[i] + 1; q < p.col_ptr[i + 1]; ++q)
            w[i] = msub(w[i], lu[q], w[p.row_idx[q]]);
        w[i] *= lu[p.diag_pos[i]];
    }
    for (int i = 0; i < n; ++i) xt[p.perm_row[i]] = w[i];

    const uint16_t* src = reinterpret_cast<const uint16_t*>(p.lp.data() + p.lp_src);
    const uint16_t* perm = reinterpret_cast<const uint16_t*>(p.lp.data() + p.lp_perm);
    std::vector<double> V(p.lp_doubles(), 0.0);
    V.back() = 1.0;
    for (int q = 0; q < p.nnz_lu; ++q) V[q] = src[q] != 0xffff ? a[src[q]] : 0.0;
    for (int i = 0; i < n; ++i) V[p.nnz_lu + i] = b[perm[i]];
    run_steps(p, 0, V, seed);
    run_steps(p, 1, V, seed);
    for (int j = 0; j < n; ++j)  // U unscaled, else as the column-wise factor
        for (int q = p.col_ptr[j]; q < p.col_ptr[j + 1]; ++q) {
            const double v = q < p.diag_pos[j] ? V[q] * V[p.diag_pos[p.row_idx[q]]] : V[q];
            if (!same(v, lu[q])) return fail("factor", n, seed);
        }
    for (int i = 0; i < n; ++i) {
        if (!same(V[p.nnz_lu + n + i], piv[i])) return fail("pivot", n, seed);
        if (!same(V[p.nnz_lu + i], x[perm[n + i]])) return fail("solution", n, seed);
    }
    for (int i = 0; i < n; ++i) V[p.nnz_lu + i] = b[perm[n + i]];
    run_steps(p, 2, V, seed);
    run_steps(p, 3, V, seed);
    for (int i = 0; i < n; ++i)
        if (!same(V[p.nnz_lu + i], xt[perm[i]])) return fail("transposed solution", n, seed);
}

}  // namespace

int main() {
    int with = 0, without = 0;
    for (int seed = 0; seed < 400; ++seed) {
        std::mt19937_64 g(seed);
        static const int sizes[] = {1, 2, 3, 31, 32, 33, 64, 100, 127, 129, 300, 700, 1500};
        const int n = sizes[seed % 13];
        const int extra = static_cast<int>(g() % (seed % 5 == 0 ? 12 : 3));
        std::vector<std::set<int>> cols(n);
        for (int j = 0; j < n; ++j) {
            cols[j].insert(j);
            if (j > 0) {  // a tree, a chain or scattered couplings
                const int o = (seed % 3 == 0) ? j - 1 : static_cast<int>(g() % j);
                cols[j].insert(o);
                cols[o].insert(j);
            }
        }
        for (int k = 0; k < extra * n / 2; ++k) cols[g() % n].insert(static_cast<int>(g() % n));
        std::vector<int32_t> cp(1, 0), ri;
        std::vector<double> a;
        std::normal_distribution<double> nd;
        for (int j = 0; j < n; ++j) {
            for (int r : cols[j]) {
                ri.push_back(r);
                a.push_back(r == j ? 8.0 + nd(g) : nd(g));
            }
            cp.push_back(static_cast<int32_t>(ri.size()));
        }
        nsg::MarkowitzOrder mo(n);
        std::vector<int32_t> elem(ri.size());
        for (int j = 0; j < n; ++j)
            for (int k = cp[j]; k < cp[j + 1]; ++k) elem[k] = mo.get_element(ri[k] + 1, j + 1);
        mo.clear_fillins();
        for (size_t k = 0; k < elem.size(); ++k) mo.value(elem[k]) = a[k];
        mo.mna_preorder();
        if (mo.order_and_factor(1e-3, 1e-13, true) != nsg::OrderStatus::ok) continue;
        nsg::TopologyPlan p = nsg::build_plan(mo, elem);
        nsg::build_level_program(p);
        if (p.lp.empty()) {
            ++without;
            continue;
        }
        ++with;
        std::vector<double> b(a);
        for (double& v : b) v *= 1.0 + 0.01 * nd(g);
        check(p, b, g, seed);
    }
    if (with < 100 || without < 10) fail("both sides of the bound were to be seen", with, without);
    std::printf("%d programs, %d plans without\n%d failure(s)\n", with, without, failures);
    return failures == 0 ? 0 : 1;
}
