#include "plan.hpp"

#include "amd_lu.hpp"
#include "sparse_order.hpp"
#include "threads.hpp"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <functional>
#include <queue>
#include <stdexcept>
#include <string>
#include <thread>

namespace nsg {

namespace {
std::atomic<int64_t> g_update_map_limit{int64_t{1} << 30};
}  // namespace

int64_t update_map_limit() { return g_update_map_limit.load(); }
void set_update_map_limit(int64_t words) { g_update_map_limit.store(words); }

namespace {

// Counting sort of items by level; returns (ptr over levels, members).
void level_sort(const std::vector<int32_t>& level, std::vector<int32_t>& ptr,
                std::vector<int32_t>& members) {
    int32_t nlev = 0;
    for (int32_t l : level) nlev = std::max(nlev, l + 1);
    ptr.assign(nlev + 1, 0);
    for (int32_t l : level) ++ptr[l + 1];
    for (int32_t l = 0; l < nlev; ++l) ptr[l + 1] += ptr[l];
    members.assign(level.size(), 0);
    std::vector<int32_t> fill(ptr.begin(), ptr.end() - 1);
    for (int32_t i = 0; i < static_cast<int32_t>(level.size()); ++i)
        members[fill[level[i]]++] = i;
}

// Bounds of a level program: what it works in and its packed words stay small
// enough for several CTAs per SM, and its entries' operand chains short (a
// denser factor has entries with long sums that one lane would walk alone).
// Inverter chains, BSIM4v7 rings and interconnect trees have 1 to 10 updates
// per unknown; the 257-unknown mesh has 83 and its columns keep 16 warps busy.
constexpr int32_t kLevelMaxDoubles = 6144;
constexpr int64_t kLevelMaxUpdatesPerRow = 32;
constexpr size_t kLevelMaxWords = 16384;
constexpr int64_t kPlanStageWords = 4096;  // of a plan without a program

// One section of a level program: entries scheduled into steps of up to 32
// whose operands were all finished in earlier steps.
struct LevelBuilder {
    struct Term {
        int32_t first, scale, second;
    };
    struct Entry {
        int32_t target, aux, nterms;
        uint32_t flags;
        Term terms[kLevelTerms];
    };
    std::vector<Entry> entries;

    // The sum over terms[0 .. n - 1] into `target`, as one entry or several:
    // first_aux goes to the first of them, last_aux and last_flags to the
    // last, `one` to the others' aux, flags to all.
    void sum(int32_t target, const Term* terms, int32_t n, int32_t one, int32_t first_aux,
             int32_t last_aux, uint32_t flags, uint32_t last_flags) {
        for (int32_t k = 0; k == 0 || k < n; k += kLevelTerms) {
            const bool last = k + kLevelTerms >= n;
            Entry e{target, one, std::min(kLevelTerms, n - k), flags, {}};
            if (k == 0 && first_aux != one) e.aux = first_aux;
            if (last && last_aux != one) e.aux = last_aux;
            if (last) e.flags |= last_flags;
            for (int32_t u = 0; u < e.nterms; ++u) e.terms[u] = terms[k + u];
            entries.push_back(e);
        }
    }

    // Longest remaining chain first (cycles on a B200: about 120 for a step, 110
    // more for a reciprocal).  values: size of the value space; zero: its
    // zero.  Appends entry and term words and the steps (offsets relative to
    // the appended words).
    void schedule(int32_t values, int32_t zero, std::vector<LevelStep>& steps,
                  std::vector<uint32_t>& entry_words, std::vector<uint32_t>& term_words) const {
        const int32_t m = static_cast<int32_t>(entries.size());
        // the last entry of each value, and of each entry the one before it
        std::vector<int32_t> maker(values, -1), before(m, -1);
        for (int32_t e = 0; e < m; ++e) {
            before[e] = maker[entries[e].target];
            maker[entries[e].target] = e;
        }
        std::vector<int32_t> missing(m, 0), ptr(m + 1, 0);
        auto operands = [&](int32_t e, auto&& f) {
            const Entry& x = entries[e];
            if (before[e] >= 0) f(before[e]);
            for (int32_t k = 0; k < x.nterms; ++k)
                for (int32_t v : {x.terms[k].first, x.terms[k].scale, x.terms[k].second})
                    if (maker[v] >= 0) f(maker[v]);
        };
        for (int32_t e = 0; e < m; ++e)
            operands(e, [&](int32_t o) {
                ++ptr[o + 1];
                ++missing[e];
            });
        for (int32_t e = 0; e < m; ++e) ptr[e + 1] += ptr[e];
        std::vector<int32_t> users(ptr[m]), fill(ptr.begin(), ptr.end() - 1);
        for (int32_t e = 0; e < m; ++e) operands(e, [&](int32_t o) { users[fill[o]++] = e; });
        std::vector<int32_t> topo, left(missing);
        topo.reserve(m);
        for (int32_t e = 0; e < m; ++e)
            if (left[e] == 0) topo.push_back(e);
        for (size_t k = 0; k < topo.size(); ++k)
            for (int32_t u = ptr[topo[k]]; u < ptr[topo[k] + 1]; ++u)
                if (--left[users[u]] == 0) topo.push_back(users[u]);
        if (static_cast<int32_t>(topo.size()) != m)
            throw std::logic_error("plan: level program has a cycle");
        std::vector<int32_t> height(m, 0);
        for (int32_t k = m - 1; k >= 0; --k) {
            const int32_t e = topo[k];
            int32_t h = 0;
            for (int32_t u = ptr[e]; u < ptr[e + 1]; ++u) h = std::max(h, height[users[u]]);
            height[e] = h + 120 + ((entries[e].flags & kLevelPivot) ? 110 : 0);
        }
        std::priority_queue<std::pair<int32_t, int32_t>> ready;
        for (int32_t e = 0; e < m; ++e)
            if (missing[e] == 0) ready.push({height[e], -e});
        std::vector<int32_t> step;
        while (!ready.empty()) {
            step.clear();
            while (!ready.empty() && step.size() < 32) {
                step.push_back(-ready.top().second);
                ready.pop();
            }
            uint32_t pivots = 0;
            const uint32_t entry_at = static_cast<uint32_t>(4 * entry_words.size());
            for (int32_t e : step) {
                pivots |= entries[e].flags & kLevelPivot;
                entry_words.push_back(static_cast<uint32_t>(8 * entries[e].target) |
                                      entries[e].flags |
                                      (static_cast<uint32_t>(8 * entries[e].aux) << 16));
            }
            steps.push_back({entry_at, static_cast<uint32_t>(4 * term_words.size()),
                             static_cast<uint32_t>(step.size()) - 1, pivots});
            for (int32_t k = 0; k < kLevelTerms; ++k)
                for (int32_t e : step) {
                    const Term t = k < entries[e].nterms ? entries[e].terms[k]
                                                         : Term{zero, zero, zero};
                    term_words.push_back(static_cast<uint32_t>(8 * t.first) |
                                         (static_cast<uint32_t>(8 * t.scale) << 16));
                    term_words.push_back(static_cast<uint32_t>(8 * t.second));
                }
            for (int32_t e : step)
                for (int32_t u = ptr[e]; u < ptr[e + 1]; ++u)
                    if (--missing[users[u]] == 0) ready.push({height[users[u]], -users[u]});
        }
    }
};

// Derive everything from the CSC LU pattern (col_ptr/row_idx/lu_src set).
void finish(TopologyPlan& p) {
    const int32_t n = p.n;
    p.nnz_lu = static_cast<int32_t>(p.row_idx.size());
    p.diag_pos.assign(n, -1);
    for (int32_t j = 0; j < n; ++j) {
        for (int32_t q = p.col_ptr[j]; q < p.col_ptr[j + 1]; ++q) {
            if (p.kind == kPlanKindMarkowitz && q > p.col_ptr[j] &&
                p.row_idx[q] <= p.row_idx[q - 1])
                throw std::invalid_argument("plan: rows not ascending in column " +
                                            std::to_string(j));
            if (p.row_idx[q] == j) p.diag_pos[j] = q;
        }
        if (p.diag_pos[j] < 0)
            throw std::invalid_argument("plan: no pivot in column " + std::to_string(j));
        for (int32_t q = p.col_ptr[j]; q < p.col_ptr[j + 1]; ++q) {
            const int32_t r = p.row_idx[q];
            if (r < 0 || r >= n || (q < p.diag_pos[j] && r >= j) || (q > p.diag_pos[j] && r <= j))
                throw std::invalid_argument("plan: U/L rows out of place in column " +
                                            std::to_string(j));
        }
    }

    // Update map for the left-looking refactor: for U(r, j), the positions
    // in column j of the rows of L(:, r).  Counted first (upd_start), then
    // filled column by column — on several host threads for large plans.
    p.upd_start.assign(p.nnz_lu, 0);
    int64_t total = 0;
    for (int32_t j = 0; j < n; ++j)
        for (int32_t q = p.col_ptr[j]; q < p.diag_pos[j]; ++q) {
            const int32_t r = p.row_idx[q];
            total += p.col_ptr[r + 1] - p.diag_pos[r] - 1;
        }
    p.has_update_map = total <= update_map_limit();
    if (p.has_update_map) {
        int64_t start = 0;
        for (int32_t j = 0; j < n; ++j)
            for (int32_t q = p.col_ptr[j]; q < p.diag_pos[j]; ++q) {
                p.upd_start[q] = static_cast<int32_t>(start);
                const int32_t r = p.row_idx[q];
                start += p.col_ptr[r + 1] - p.diag_pos[r] - 1;
            }
    }
    p.upd_dst.clear();
    if (p.has_update_map) p.upd_dst.resize(static_cast<size_t>(total));  // every entry written below
    // First failing column of each kind (duplicate row / fill not closed),
    // so that the error does not depend on the thread schedule.
    std::atomic<int32_t> bad_dup{INT32_MAX}, bad_fill{INT32_MAX};
    auto fill_columns = [&](std::atomic<int32_t>& next_col, int32_t chunk) {
        std::vector<int32_t> where(n, -1);
        for (;;) {
            const int32_t j0 = next_col.fetch_add(chunk);
            if (j0 >= n) break;
            const int32_t j1 = std::min(n, j0 + chunk);
            for (int32_t j = j0; j < j1; ++j) {
                bool dup = false;
                for (int32_t q = p.col_ptr[j]; q < p.col_ptr[j + 1]; ++q) {
                    if (where[p.row_idx[q]] >= 0) dup = true;
                    where[p.row_idx[q]] = q;
                }
                bool open = false;
                if (!dup) {
                    for (int32_t q = p.col_ptr[j]; q < p.diag_pos[j] && !open; ++q) {
                        const int32_t r = p.row_idx[q];
                        int32_t* out = p.upd_dst.data() + p.upd_start[q];
                        for (int32_t k = p.diag_pos[r] + 1; k < p.col_ptr[r + 1]; ++k) {
                            const int32_t d = where[p.row_idx[k]];
                            if (d < 0) {
                                open = true;
                                break;
                            }
                            *out++ = d - p.col_ptr[j];  // relative to column j
                        }
                    }
                }
                for (int32_t q = p.col_ptr[j]; q < p.col_ptr[j + 1]; ++q) where[p.row_idx[q]] = -1;
                auto lower = [](std::atomic<int32_t>& a, int32_t v) {
                    int32_t cur = a.load();
                    while (v < cur && !a.compare_exchange_weak(cur, v)) {
                    }
                };
                if (dup) lower(bad_dup, j);
                if (open) lower(bad_fill, j);
            }
        }
    };
    if (p.has_update_map) {
        std::atomic<int32_t> next_col{0};
        const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
        const int nthreads = total >= (int64_t{1} << 25) ? static_cast<int>(std::min(hw, 16u)) : 1;
        on_threads(nthreads, [&] { fill_columns(next_col, nthreads == 1 ? n : 64); });
    }
    const int32_t first_bad = std::min(bad_dup.load(), bad_fill.load());
    if (first_bad != INT32_MAX) {
        if (bad_dup.load() == first_bad)
            throw std::invalid_argument("plan: duplicate row in column " + std::to_string(first_bad));
        throw std::invalid_argument("plan: fill pattern not closed at column " +
                                    std::to_string(first_bad));
    }
    p.updates = total;
    p.max_col = 0;
    for (int32_t j = 0; j < n; ++j) p.max_col = std::max(p.max_col, p.col_ptr[j + 1] - p.col_ptr[j]);

    // Row-wise L and U.
    std::vector<int32_t> lcount(n + 1, 0), ucount(n + 1, 0);
    for (int32_t j = 0; j < n; ++j)
        for (int32_t q = p.col_ptr[j]; q < p.col_ptr[j + 1]; ++q) {
            const int32_t i = p.row_idx[q];
            if (i > j) ++lcount[i + 1];
            else if (i < j) ++ucount[i + 1];
        }
    for (int32_t i = 0; i < n; ++i) {
        lcount[i + 1] += lcount[i];
        ucount[i + 1] += ucount[i];
    }
    p.lrow_ptr = lcount;
    p.urow_ptr = ucount;
    p.lrow_pos.assign(lcount[n], 0);
    p.lrow_col.assign(lcount[n], 0);
    p.urow_pos.assign(ucount[n], 0);
    p.urow_col.assign(ucount[n], 0);
    std::vector<int32_t> lf(lcount.begin(), lcount.end() - 1), uf(ucount.begin(), ucount.end() - 1);
    for (int32_t j = 0; j < n; ++j)  // columns ascending -> rows get ascending columns
        for (int32_t q = p.col_ptr[j]; q < p.col_ptr[j + 1]; ++q) {
            const int32_t i = p.row_idx[q];
            if (i > j) {
                p.lrow_pos[lf[i]] = q;
                p.lrow_col[lf[i]++] = j;
            } else if (i < j) {
                p.urow_pos[uf[i]] = q;
                p.urow_col[uf[i]++] = j;
            }
        }

    // next[r]: the column r' whose L rows follow it in L(:, r), if L(:, r) is r'
    // and then L(:, r') -- neighbours in a run of equal structure.
    std::vector<int32_t> next(n, -1);
    for (int32_t r = 0; r < n; ++r) {
        const int32_t l0 = p.diag_pos[r] + 1, cnt = p.col_ptr[r + 1] - l0;
        if (cnt == 0) continue;
        const int32_t r2 = p.row_idx[l0], m0 = p.diag_pos[r2] + 1;
        if (p.col_ptr[r2 + 1] - m0 == cnt - 1 &&
            std::equal(p.row_idx.begin() + m0, p.row_idx.begin() + m0 + cnt - 1,
                       p.row_idx.begin() + l0 + 1))
            next[r] = r2;
    }
    p.umeta.assign(4 * static_cast<size_t>(p.nnz_lu), 0);
    for (int32_t j = 0; j < n; ++j)
        for (int32_t q = p.col_ptr[j]; q < p.diag_pos[j]; ++q) {
            const int32_t r = p.row_idx[q];
            p.umeta[4 * q] = r;
            p.umeta[4 * q + 1] = p.diag_pos[r];
            p.umeta[4 * q + 2] = p.col_ptr[r + 1] - p.diag_pos[r] - 1;
            if (q + 1 < p.diag_pos[j] && next[r] == p.row_idx[q + 1]) p.umeta[4 * q + 2] |= kRunBit;
            p.umeta[4 * q + 3] = p.upd_start[q];
        }
    p.rowcopy_pos.assign(p.nnz_lu, -1);
    for (int32_t i = 0; i < n; ++i) {
        for (int32_t k = p.lrow_ptr[i]; k < p.lrow_ptr[i + 1]; ++k) p.rowcopy_pos[p.lrow_pos[k]] = k;
        for (int32_t k = p.urow_ptr[i]; k < p.urow_ptr[i + 1]; ++k) p.rowcopy_pos[p.urow_pos[k]] = k;
    }

    // Level schedules.
    std::vector<int32_t> lev(n, 0);
    for (int32_t j = 0; j < n; ++j) {
        int32_t l = 0;
        for (int32_t q = p.col_ptr[j]; q < p.diag_pos[j]; ++q)
            l = std::max(l, lev[p.row_idx[q]] + 1);
        lev[j] = l;
    }
    level_sort(lev, p.col_lev_ptr, p.col_lev);
    for (int32_t i = 0; i < n; ++i) {
        int32_t l = 0;
        for (int32_t k = p.lrow_ptr[i]; k < p.lrow_ptr[i + 1]; ++k)
            l = std::max(l, lev[p.lrow_col[k]] + 1);
        lev[i] = l;
    }
    level_sort(lev, p.fwd_lev_ptr, p.fwd_lev);
    for (int32_t i = n - 1; i >= 0; --i) {
        int32_t l = 0;
        for (int32_t k = p.urow_ptr[i]; k < p.urow_ptr[i + 1]; ++k)
            l = std::max(l, lev[p.urow_col[k]] + 1);
        lev[i] = l;
    }
    level_sort(lev, p.bwd_lev_ptr, p.bwd_lev);
    for (int32_t i = n - 1; i >= 0; --i) {
        int32_t l = 0;
        for (int32_t q = p.diag_pos[i] + 1; q < p.col_ptr[i + 1]; ++q)
            l = std::max(l, lev[p.row_idx[q]] + 1);
        lev[i] = l;
    }
    level_sort(lev, p.tbw_lev_ptr, p.tbw_lev);

    p.a_to_lu.assign(p.nnz_a, -1);
    for (int32_t q = 0; q < p.nnz_lu; ++q)
        if (p.lu_src[q] >= 0) p.a_to_lu[p.lu_src[q]] = q;
    for (int32_t k = 0; k < p.nnz_a; ++k)
        if (p.a_to_lu[k] < 0)
            throw std::invalid_argument("plan: caller slot without an element");
}

}  // namespace

// The level program of a Markowitz plan (see TopologyPlan::lp), for factors
// within the bounds above that have an update map.  An entry of the factor
// receives its updates in ascending pivot order, a row of a sweep its columns in
// the order of the row-wise sweeps, so every value is the one the column-wise
// refactor and the sweeps compute.
void build_level_program(TopologyPlan& p) {
    p.lp.clear();
    p.lp_core = 0;
    const int32_t n = p.n, nlu = p.nnz_lu;
    const int32_t vec = nlu, pivots = nlu + n, zero = nlu + 2 * n, one = zero + 1;
    static_assert(8 * kLevelMaxDoubles <= 0xffff, "value offsets are 16 bits");
    if (p.kind != kPlanKindMarkowitz || !p.has_update_map || one >= kLevelMaxDoubles ||
        p.updates > kLevelMaxUpdatesPerRow * n || p.nnz_a >= 0xffff)
        return;
    // updates of each LU position, ascending in the source column
    std::vector<int32_t> upd_ptr(nlu + 1, 0);
    auto each_update = [&](auto&& f) {
        for (int32_t j = 0; j < n; ++j)
            for (int32_t q = p.col_ptr[j]; q < p.diag_pos[j]; ++q) {
                const int32_t r = p.row_idx[q], cnt = p.col_ptr[r + 1] - p.diag_pos[r] - 1;
                for (int32_t k = 0; k < cnt; ++k)
                    f(p.col_ptr[j] + p.upd_dst[p.upd_start[q] + k],
                      LevelBuilder::Term{q, p.diag_pos[r], p.diag_pos[r] + 1 + k});
            }
    };
    each_update([&](int32_t d, const LevelBuilder::Term&) { ++upd_ptr[d + 1]; });
    for (int32_t q = 0; q < nlu; ++q) upd_ptr[q + 1] += upd_ptr[q];
    std::vector<LevelBuilder::Term> upd(upd_ptr[nlu]);
    std::vector<int32_t> at(upd_ptr.begin(), upd_ptr.end() - 1);
    each_update([&](int32_t d, const LevelBuilder::Term& t) { upd[at[d]++] = t; });
    LevelBuilder factor, backward, over_u, over_l;
    for (int32_t j = 0; j < n; ++j)
        for (int32_t q = p.col_ptr[j]; q < p.col_ptr[j + 1]; ++q) {
            const LevelBuilder::Term* t = upd.data() + upd_ptr[q];
            const int32_t cnt = upd_ptr[q + 1] - upd_ptr[q];
            if (q == p.diag_pos[j]) factor.sum(q, t, cnt, one, one, pivots + j, 0, kLevelPivot);
            else if (cnt > 0) factor.sum(q, t, cnt, one, one, one, 0, 0);
        }
    std::vector<LevelBuilder::Term> row;
    for (int32_t i = 0; i < n; ++i) {
        const int32_t di = p.diag_pos[i];
        row.clear();
        for (int32_t k = p.lrow_ptr[i]; k < p.lrow_ptr[i + 1]; ++k)
            row.push_back({vec + p.lrow_col[k], p.diag_pos[p.lrow_col[k]], p.lrow_pos[k]});
        if (!row.empty())
            factor.sum(vec + i, row.data(), static_cast<int32_t>(row.size()), one, one, one,
                       kLevelSkip, 0);
        row.clear();
        for (int32_t k = p.urow_ptr[i]; k < p.urow_ptr[i + 1]; ++k)
            row.push_back({p.urow_pos[k], di, vec + p.urow_col[k]});
        backward.sum(vec + i, row.data(), static_cast<int32_t>(row.size()), one, di, one, 0, 0);
        row.clear();
        for (int32_t q = p.col_ptr[i]; q < di; ++q)
            row.push_back({q, p.diag_pos[p.row_idx[q]], vec + p.row_idx[q]});
        if (!row.empty())
            over_u.sum(vec + i, row.data(), static_cast<int32_t>(row.size()), one, one, one, 0, 0);
        row.clear();
        for (int32_t q = di + 1; q < p.col_ptr[i + 1]; ++q)
            row.push_back({q, one, vec + p.row_idx[q]});
        over_l.sum(vec + i, row.data(), static_cast<int32_t>(row.size()), one, one, di, 0, 0);
    }
    std::vector<LevelStep> steps;
    std::vector<uint32_t> ent[4], trm[4];
    const LevelBuilder* section[4] = {&factor, &backward, &over_u, &over_l};
    for (int s = 0; s < 4; ++s) {
        section[s]->schedule(one + 1, zero, steps, ent[s], trm[s]);
        p.lp_steps[s] = static_cast<int32_t>(steps.size());
    }
    std::vector<int32_t>& lp = p.lp;
    lp.assign(4 * steps.size(), 0);
    p.lp_src = static_cast<int32_t>(lp.size());
    p.lp_perm = p.lp_src + (nlu + 1) / 2;
    lp.resize(p.lp_perm + n, 0);
    for (int32_t q = 0; q < nlu; ++q) {
        const uint32_t v = p.lu_src[q] < 0 ? 0xffffu : static_cast<uint32_t>(p.lu_src[q]);
        lp[p.lp_src + q / 2] |= static_cast<int32_t>(v << (16 * (q % 2)));
    }
    for (int32_t i = 0; i < 2 * n; ++i) {
        const uint32_t v = static_cast<uint32_t>(i < n ? p.perm_row[i] : p.perm_col[i - n]);
        lp[p.lp_perm + i / 2] |= static_cast<int32_t>(v << (16 * (i % 2)));
    }
    for (int s = 0; s < 4; ++s) {
        if (lp.size() % 2) lp.push_back(0);
        const uint32_t t0 = static_cast<uint32_t>(4 * lp.size());
        const uint32_t e0 = t0 + static_cast<uint32_t>(4 * trm[s].size());
        for (int32_t r = s == 0 ? 0 : p.lp_steps[s - 1]; r < p.lp_steps[s]; ++r) {
            steps[r].entries += e0;
            steps[r].terms += t0;
        }
        lp.insert(lp.end(), trm[s].begin(), trm[s].end());
        lp.insert(lp.end(), ent[s].begin(), ent[s].end());
        if (s == 1) p.lp_core = static_cast<int32_t>(lp.size());
    }
    std::memcpy(lp.data(), steps.data(), sizeof(LevelStep) * steps.size());
    if (lp.size() > kLevelMaxWords) lp.clear();
}

// Order of the arrays in the device pool; must match PlanArrays in the
// kernels' header.
#define NSG_PLAN_ARRAYS(X)                                                      \
    X(perm_row) X(perm_col) X(col_ptr) X(row_idx) X(diag_pos) X(lu_src)         \
    X(upd_start) X(upd_dst) X(lrow_ptr) X(lrow_pos) X(lrow_col) X(urow_ptr)     \
    X(urow_pos) X(urow_col) X(col_lev_ptr) X(col_lev) X(fwd_lev_ptr) X(fwd_lev) \
    X(bwd_lev_ptr) X(bwd_lev) X(tbw_lev_ptr) X(tbw_lev) X(rowcopy_pos) X(umeta) \
    X(piv_rank) X(gmin_pos) X(lp)

namespace {
template <class V>
bool is_update_map(const TopologyPlan& p, const V& v) {
    return static_cast<const void*>(&v) == static_cast<const void*>(&p.upd_dst);
}

// v's values (each below 65,536) as consecutive uint16, in ceil(|v| / 2)
// words; the last half word of an odd count is zero.
template <class V>
void append_packed16(std::vector<int32_t>& pool, const V& v) {
    const size_t at = pool.size();
    pool.resize(at + (v.size() + 1) / 2, 0);
    char* out = reinterpret_cast<char*>(pool.data() + at);
    uint16_t chunk[4096];
    for (size_t k0 = 0; k0 < v.size(); k0 += 4096) {
        const size_t m = std::min<size_t>(4096, v.size() - k0);
        for (size_t k = 0; k < m; ++k) chunk[k] = static_cast<uint16_t>(v[k0 + k]);
        std::memcpy(out + 2 * k0, chunk, 2 * m);
    }
}
}  // namespace

int32_t TopologyPlan::stage_words(bool transposed) const {
    if (!lp.empty()) return transposed ? static_cast<int32_t>(lp.size()) : lp_core;
    return n <= 128 && device_words() <= kPlanStageWords ? static_cast<int32_t>(device_words()) : 0;
}

void PlanStage::add(const TopologyPlan& p, bool transposed) {
    const bool one_warp = one_warp_factor(p.n, p.nnz_lu);
    doubles = std::max({doubles, p.lp_doubles(), one_warp ? p.nnz_lu + p.n : 0});
    words = std::max(words, p.stage_words(transposed));
    programs = programs || !p.lp.empty();
    dataflow = dataflow || (p.lp.empty() && !one_warp);
}

// A packed update map takes one int32 word per two positions.
int64_t TopologyPlan::device_words() const {
    int64_t w = 0;
#define NSG_COUNT(name)                                                          \
    w += (is_update_map(*this, name) && map16() ? (static_cast<int64_t>(name.size()) + 1) / 2 \
                                                 : static_cast<int64_t>(name.size())) +       \
         4;  // 16 B align
    NSG_PLAN_ARRAYS(NSG_COUNT)
#undef NSG_COUNT
    return w;
}

void TopologyPlan::append_to(std::vector<int32_t>& pool, int64_t* off) const {
    int idx = 0;
    const bool pack = map16();
#define NSG_APPEND(name)                                          \
    while (pool.size() % 4) pool.push_back(0);                    \
    off[idx++] = static_cast<int64_t>(pool.size());               \
    if (pack && is_update_map(*this, name)) {                     \
        append_packed16(pool, name);                              \
    } else {                                                      \
        pool.insert(pool.end(), name.begin(), name.end());        \
    }
    NSG_PLAN_ARRAYS(NSG_APPEND)
#undef NSG_APPEND
}

TopologyPlan build_plan(const MarkowitzOrder& mo, const std::vector<int32_t>& slot_elem) {
    TopologyPlan p;
    p.n = mo.size();
    p.nnz_a = static_cast<int32_t>(slot_elem.size());
    p.perm_row.resize(p.n);
    p.perm_col.resize(p.n);
    for (int32_t i = 1; i <= p.n; ++i) {
        p.perm_row[i - 1] = mo.int_to_ext_row()[i] - 1;
        p.perm_col[i - 1] = mo.int_to_ext_col()[i] - 1;
    }
    std::vector<int32_t> slot_of(mo.element_count(), -1);
    for (int32_t k = 0; k < p.nnz_a; ++k) slot_of[slot_elem[k]] = k;
    p.col_ptr.assign(p.n + 1, 0);
    for (int32_t j = 1; j <= p.n; ++j) {
        for (int32_t e = mo.first_in_col(j); e >= 0; e = mo.next_in_col(e)) {
            p.row_idx.push_back(mo.row_of(e) - 1);
            p.lu_src.push_back(slot_of[e]);
        }
        p.col_ptr[j] = static_cast<int32_t>(p.row_idx.size());
    }
    finish(p);
    return p;
}

TopologyPlan build_plan_amd(const AmdLuFactor& f) {
    if (!f.factored()) throw std::logic_error("build_plan_amd: engine not factored");
    TopologyPlan p;
    p.kind = kPlanKindAmdLu;
    p.n = f.size();
    p.nnz_a = f.nnz();
    const int32_t n = p.n;
    const auto& q = f.q();
    const auto& pinv = f.pinv();
    const auto& acp = f.col_ptr();
    const auto& ari = f.row_idx();
    p.perm_row.assign(n, -1);
    for (int32_t r = 0; r < n; ++r) p.perm_row[pinv[r]] = r;
    p.perm_col = q;
    p.piv_rank = f.piv_rank();
    p.gmin_pos.assign(n, -1);
    p.col_ptr.assign(n + 1, 0);
    p.row_idx.reserve(f.Li().size() + f.Ui().size());
    p.lu_src.reserve(f.Li().size() + f.Ui().size());
    std::vector<int32_t> slot_at(n, -1);  // pivot-step row -> A slot of this column
    for (int32_t k = 0; k < n; ++k) {
        const int32_t col = q[k];
        for (int32_t a = acp[col]; a < acp[col + 1]; ++a) slot_at[pinv[ari[a]]] = a;
        const int32_t c0 = static_cast<int32_t>(p.row_idx.size());
        auto push = [&](int32_t s) {
            if (s == pinv[col]) p.gmin_pos[k] = static_cast<int32_t>(p.row_idx.size()) - c0;
            p.row_idx.push_back(s);
            p.lu_src.push_back(slot_at[s]);
        };
        // U(:, k) above the pivot in replay order, the pivot (stored last in
        // U(:, k) by the reference), then L(:, k) after its unit diagonal.
        for (int32_t u = f.Up()[k]; u < f.Up()[k + 1] - 1; ++u) push(f.Ui()[u]);
        push(k);
        for (int32_t l = f.Lp()[k] + 1; l < f.Lp()[k + 1]; ++l) push(f.Li()[l]);
        for (int32_t a = acp[col]; a < acp[col + 1]; ++a) slot_at[pinv[ari[a]]] = -1;
        p.col_ptr[k + 1] = static_cast<int32_t>(p.row_idx.size());
    }
    finish(p);
    return p;
}

TopologyPlan build_plan_from_structure(int32_t n, int32_t nnz_a,
                                       const int32_t* int_to_ext_row,
                                       const int32_t* int_to_ext_col,
                                       int32_t n_elem, const int32_t* elem_row,
                                       const int32_t* elem_col,
                                       const int32_t* slot_to_elem) {
    if (n <= 0 || nnz_a <= 0 || n_elem < nnz_a)
        throw std::invalid_argument("plan: bad sizes");
    TopologyPlan p;
    p.n = n;
    p.nnz_a = nnz_a;
    p.perm_row.resize(n);
    p.perm_col.resize(n);
    for (int32_t i = 0; i < n; ++i) {
        if (int_to_ext_row[i] < 1 || int_to_ext_row[i] > n || int_to_ext_col[i] < 1 ||
            int_to_ext_col[i] > n)
            throw std::invalid_argument("plan: permutation out of range");
        p.perm_row[i] = int_to_ext_row[i] - 1;
        p.perm_col[i] = int_to_ext_col[i] - 1;
    }
    std::vector<int32_t> slot_of(n_elem, -1);
    for (int32_t k = 0; k < nnz_a; ++k) {
        if (slot_to_elem[k] < 0 || slot_to_elem[k] >= n_elem)
            throw std::invalid_argument("plan: slot map out of range");
        slot_of[slot_to_elem[k]] = k;
    }
    p.col_ptr.assign(n + 1, 0);
    p.row_idx.resize(n_elem);
    p.lu_src.resize(n_elem);
    for (int32_t e = 0; e < n_elem; ++e) {
        if (elem_col[e] < 1 || elem_col[e] > n || elem_row[e] < 1 || elem_row[e] > n ||
            (e > 0 && elem_col[e] < elem_col[e - 1]))
            throw std::invalid_argument("plan: element list not column ordered");
        ++p.col_ptr[elem_col[e]];
        p.row_idx[e] = elem_row[e] - 1;
        p.lu_src[e] = slot_of[e];
    }
    for (int32_t j = 0; j < n; ++j) p.col_ptr[j + 1] += p.col_ptr[j];
    finish(p);
    return p;
}

}  // namespace nsg
