// Launch shapes of the Newton kernels without a GPU: the library's own launch
// functions run against stand-ins for the runtime calls they make, which record
// each launch.  Prints "0 failure(s)" on success.
//   shapes: transients of circuits with level programs or one-warp factors run
//     in CTAs of 128 or 256 threads, denser factors on 512 threads, whatever
//     the batch's size; and a launch has room for every path its plans take.
//   failures: a runtime call that fails once fails that launch only.
#include "host/plan.hpp"
#include "host/sparse_order.hpp"
#include "kernels/tran_device.cuh"

#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <random>
#include <set>
#include <vector>

namespace {
int launches = 0, threads = 0, failures = 0;
size_t smem = 0;
cudaError_t attribute_result = cudaSuccess;

void expect(bool ok, const char* what, int a = 0, int b = 0) {
    if (!ok && ++failures < 20) std::printf("failed: %s (%d, %d)\n", what, a, b);
}
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return attribute_result; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3 block, void**, size_t bytes, cudaStream_t) {
    ++launches;
    threads = static_cast<int>(block.x);
    smem = bytes;
    return cudaSuccess;
}
}

namespace nsg {
bool register_wait_limit_setter(cudaError_t (*)(int)) { return true; }
cudaError_t launch_transient(const PlanDesc*, const int32_t*, const DcDesc*, const TranDesc*,
                             const int32_t*, int, const int32_t*, const double*, const double*,
                             double*, const double*, const int32_t*, double*, double*, int32_t*,
                             int32_t*, int32_t*, TranCtl*, const TranOptions&, const TranShape&,
                             StepRecord*, double*, cudaStream_t);
cudaError_t launch_newton_dc(const PlanDesc*, const int32_t*, const DcDesc*, const int32_t*, int,
                             const int32_t*, const double*, double*, double*, int32_t*, int32_t*,
                             DcCtl*, const NewtonOptions&, int, int, const int64_t*, int, int, int,
                             int32_t*, cudaStream_t);
}  // namespace nsg

namespace {

// The plan of a symmetric pattern, diagonally dominant.
nsg::TopologyPlan plan_of(const std::vector<std::pair<int, int>>& edges, int n) {
    std::vector<std::set<int>> cols(n);
    for (int j = 0; j < n; ++j) cols[j].insert(j);
    for (auto [a, b] : edges) {
        cols[a].insert(b);
        cols[b].insert(a);
    }
    std::mt19937_64 g(n);
    std::uniform_real_distribution<double> u(0.5, 1.5);
    nsg::MarkowitzOrder mo(n);
    std::vector<int32_t> elem;
    std::vector<double> a;
    for (int j = 0; j < n; ++j)
        for (int r : cols[j]) {
            elem.push_back(mo.get_element(r + 1, j + 1));
            a.push_back(r == j ? 4.0 * n : -u(g));
        }
    mo.clear_fillins();
    for (size_t k = 0; k < elem.size(); ++k) mo.value(elem[k]) = a[k];
    mo.mna_preorder();
    expect(mo.order_and_factor(1e-3, 1e-13, true) == nsg::OrderStatus::ok, "ordering", n);
    nsg::TopologyPlan p = nsg::build_plan(mo, elem);
    nsg::build_level_program(p);
    return p;
}

nsg::TopologyPlan chain(int n) {
    std::vector<std::pair<int, int>> e;
    for (int k = 1; k < n; ++k) e.push_back({k - 1, k});
    return plan_of(e, n);
}
nsg::TopologyPlan mesh(int side) {
    std::vector<std::pair<int, int>> e;
    for (int y = 0; y < side; ++y)
        for (int x = 0; x < side; ++x) {
            if (x + 1 < side) e.push_back({y * side + x, y * side + x + 1});
            if (y + 1 < side) e.push_back({y * side + x, (y + 1) * side + x});
        }
    return plan_of(e, side * side);
}
nsg::TopologyPlan band(int n, int width) {
    std::vector<std::pair<int, int>> e;
    for (int a = 0; a < n; ++a)
        for (int b = a + 1; b <= a + width && b < n; ++b) e.push_back({a, b});
    return plan_of(e, n);
}
nsg::TopologyPlan coupled(int n) {
    std::vector<std::pair<int, int>> e;
    for (int a = 0; a < n; ++a)
        for (int b = 0; b < a; ++b) e.push_back({b, a});
    return plan_of(e, n);
}

void transient(const char* what, const std::vector<nsg::TopologyPlan>& plans, int devices,
               int count, int want_threads) {
    nsg::TranShape sh{};
    for (const auto& p : plans) {
        sh.max_col = std::max(sh.max_col, p.max_col);
        sh.max_n = std::max(sh.max_n, p.n);
        sh.plans.add(p, false);
    }
    sh.stage_lens.assign(count, 4096);
    sh.max_devices = devices;
    nsg::TranOptions o{};
    threads = 0;
    expect(nsg::launch_transient(nullptr, nullptr, nullptr, nullptr, nullptr, count, nullptr,
                                 nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr,
                                 nullptr, nullptr, nullptr, nullptr, o, sh, nullptr, nullptr,
                                 nullptr) == cudaSuccess, what, count);
    if (threads != want_threads) std::printf("%s: %d threads\n", what, threads);
    expect(threads == want_threads, what, count, want_threads);
    // the largest factor one warp, a level program or the column buffers take
    const size_t flow = sizeof(double) * (threads / 32) * ((sh.max_col + 31) / 32 * 32) +
                        sizeof(int32_t) * sh.max_n;
    expect(smem >= flow && smem >= sizeof(double) * sh.plans.doubles, "room", count, threads);
    for (const auto& p : plans)
        if (nsg::one_warp_factor(p.n, p.nnz_lu))
            expect(smem >= sizeof(double) * (p.nnz_lu + p.n), "one-warp room", p.n, threads);
}

cudaError_t dc(int count) {
    const std::vector<int64_t> lens(count, 4096);
    return nsg::launch_newton_dc(nullptr, nullptr, nullptr, nullptr, count, nullptr, nullptr,
                                 nullptr, nullptr, nullptr, nullptr, nullptr, nsg::NewtonOptions{},
                                 100, 500, lens.data(), count, 0, 0, nullptr, nullptr);
}

void one_failure(int count) {
    attribute_result = cudaErrorMemoryAllocation;
    launches = 0;
    expect(dc(count) == cudaErrorMemoryAllocation && launches == 0, "failing attribute", count);
    attribute_result = cudaSuccess;
    expect(dc(count) == cudaSuccess && launches == 1, "launch after a failure", count);
}

}  // namespace

int main() {
    one_failure(1);
    one_failure(600);
    expect(!chain(100).lp.empty() && !mesh(8).lp.empty() && !band(128, 4).lp.empty(), "programs");
    expect(mesh(11).lp.empty() && band(128, 6).lp.empty() && coupled(12).lp.empty(), "no programs");
    for (int count : {1, 148, 149, 296, 297, 1200}) {
        const bool alone = count <= 148;
        transient("chain", {chain(100)}, 100, count, alone ? 256 : 128);
        transient("chain, many devices", {chain(100)}, 200, count, 256);
        transient("chain, most devices", {chain(100)}, 300, count, 512);
        transient("mesh with a program", {mesh(8)}, 60, count, alone ? 256 : 128);
        transient("program too large for four CTAs", {band(128, 4)}, 100, count, 256);
        transient("band without a program", {band(128, 6)}, 100, count, 512);
        transient("coupled, one warp", {coupled(12), coupled(22)}, 20, count, alone ? 256 : 128);
        transient("coupled, dataflow", {coupled(23)}, 20, count, 512);
        transient("coupled, largest", {coupled(128)}, 120, count, 512);
        transient("mesh without a program", {mesh(11)}, 120, count, 512);
        transient("chain beside a mesh", {chain(40), mesh(11)}, 120, count, 512);
        transient("large tree", {chain(500)}, 120, count, 512);
    }
    std::printf("%d failure(s)\n", failures);
    return failures == 0 ? 0 : 1;
}
