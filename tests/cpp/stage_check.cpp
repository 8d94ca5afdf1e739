// What a launch stages of an instance's workspace is what its kernels work in:
// the regions of a DcDesc follow one another from x_off to x_off + stage_len
// with no space between them.  Prints "0 failure(s)" on success.
#include "capi_internal.hpp"
#include "host/sparse_order.hpp"
#include "kernels/dc_device.cuh"

#include <algorithm>
#include <cstdio>
#include <utility>
#include <vector>

int main() {
    int failures = 0;
    for (int n : {1, 2, 3, 4, 5, 37, 100, 257}) {
        nsg::Circuit c(n);
        for (int k = 1; k < n; ++k) c.add_resistor(k - 1, k, 100.0);
        c.add_resistor(0, -1, 50.0);
        c.add_isource(-1, n - 1, 1e-3);
        for (int k = 0; k < n; k += 3) c.add_diode(k, -1, 1e-14, 1.0);
        for (int k = 1; k < n; k += 2) c.add_capacitor(k, -1, 1e-12, false, 0.0);
        c.finalize();
        std::vector<double> a, rhs;
        c.initjct_values(a, rhs, 1e-12);
        nsg::MarkowitzOrder mo(c.num_vars());
        std::vector<int32_t> elem;
        for (int j = 0; j < c.num_vars(); ++j)
            for (int q = c.col_ptr()[j]; q < c.col_ptr()[j + 1]; ++q)
                elem.push_back(mo.get_element(c.row_idx()[q] + 1, j + 1));
        mo.clear_fillins();
        for (size_t k = 0; k < elem.size(); ++k) mo.value(elem[k]) = a[k];
        mo.mna_preorder();
        if (mo.order_and_factor(1e-3, 1e-13, true) != nsg::OrderStatus::ok) ++failures;
        const nsg::TopologyPlan p = nsg::build_plan(mo, elem);
        nsg::DcDesc d{};
        std::vector<int32_t> prog;
        int64_t work = 0;
        nsg_internal::fill_instance(d, c, p, prog, work);
        std::vector<std::pair<int64_t, int64_t>> r = {
            {d.x_off, d.n},
            {d.xold_off, d.n},
            {d.a_off, d.nnz},
            {d.lu_off, p.nnz_lu},
            {d.lrows_off, p.lrow_ptr[p.n]},
            {d.urows_off, p.urow_ptr[p.n]},
            {d.tv_off, c.n_terms()},
            {d.dconst_off, 3 * d.n_diodes},
            {d.state_off, 4 * int64_t{d.n_states}},
            {d.mrec_off, nsg::kMosRecCount * int64_t{d.n_mos}},
        };
        std::sort(r.begin(), r.end());
        int64_t end = d.x_off;
        for (auto [off, len] : r) {
            if (off != end) {
                std::printf("failed: n %d, %lld doubles unused before %lld\n", n,
                            static_cast<long long>(off - end), static_cast<long long>(off));
                ++failures;
            }
            end = (off + len + 3) & ~int64_t{3};
        }
        if (end != d.x_off + d.stage_len) ++failures;
    }
    std::printf("%d failure(s)\n", failures);
    return failures == 0 ? 0 : 1;
}
