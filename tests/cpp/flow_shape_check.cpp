// Launch shapes of a batch's dataflow kernels without a GPU: the library's own
// launch functions run against stand-ins for the runtime calls they make.
// And which plans are solved with a thread per row, which transposed and complex
// solves run level after level in a workspace.  Prints "0 failure(s)" on success.
#include "kernels/flow_shape.cuh"
#include "kernels/lu_device.cuh"

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <set>
#include <utility>

namespace {
int threads = 0, failures = 0;

void expect(const char* what, int n, int count, int want) {
    if (threads != want && ++failures < 20)
        std::printf("failed: %s of %d, %d instances: %d threads\n", what, n, count, threads);
}
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3 block, void**, size_t, cudaStream_t) {
    threads = static_cast<int>(block.x);
    return cudaSuccess;
}
}

namespace nsg {
bool register_wait_limit_setter(cudaError_t (*)(int)) { return true; }
bool transposed_levels_pay(const FlowBatch&);
bool complex_levels_pay(const FlowBatch&, const double*);
cudaError_t launch_refactor(const PlanDesc*, const int32_t*, const InstDesc*, const FlowBatch&,
                            const double*, double*, double, int, double, int32_t*, int32_t*, bool,
                            double*, double*, cudaStream_t);
cudaError_t launch_solve(const PlanDesc*, const int32_t*, const InstDesc*, const FlowBatch&,
                         const double*, double*, double*, bool, const double*, const double*,
                         cudaStream_t);
cudaError_t launch_complex_refactor(const PlanDesc*, const int32_t*, const InstDesc*,
                                    const FlowBatch&, const double*, double*, int32_t*,
                                    cudaStream_t);
cudaError_t launch_complex_solve(const PlanDesc*, const int32_t*, const InstDesc*,
                                 const FlowBatch&, const double*, double*, double*, cudaStream_t);
}  // namespace nsg

namespace {

const double* const kRows = reinterpret_cast<const double*>(64);
double* const kLu = reinterpret_cast<double*>(64);

void check(int n, int col, double level_rows, int refactor, int solve, int complex_refactor,
           int complex_solve) {
    for (int count : {1, 148, 149, 296, 297, 444, 445, 592, 1500}) {
        const nsg::FlowBatch b{count, col, n, level_rows};
        auto want = [&](int many) { return count <= 296 ? 512 : many; };
        nsg::launch_refactor(nullptr, nullptr, nullptr, b, nullptr, kLu, 0.0, 0, 0.0, nullptr,
                             nullptr, true, nullptr, nullptr, nullptr);
        // three CTAs do where they hold the whole batch
        const bool three = nsg::ctas_per_sm(8 * 8 * ((col + 31) / 32 * 32) + 4 * n) == 3;
        expect("refactor", n, count, three && count <= 444 ? want(256) : want(refactor));
        for (bool transposed : {false, true}) {
            nsg::launch_solve(nullptr, nullptr, nullptr, b, kLu, nullptr, nullptr, transposed,
                              transposed ? nullptr : kRows, kRows, nullptr);
            expect(transposed ? "transposed solve" : "solve", n, count, want(solve));
        }
        nsg::launch_complex_refactor(nullptr, nullptr, nullptr, b, nullptr, kLu, nullptr, nullptr);
        expect("complex refactor", n, count, want(complex_refactor));
        nsg::launch_complex_solve(nullptr, nullptr, nullptr, b, kLu, nullptr, nullptr, nullptr);
        expect("complex solve", n, count, want(complex_solve));
    }
}

// n unknowns, off-diagonal entries a row of a sweep, rows a level
void wide(int n, double entries, double level_rows, bool want) {
    nsg::PlanDesc pd{};
    pd.n = n;
    pd.nnz_lu = n + static_cast<int>(2 * entries * n);
    pd.n_fwd_lev = static_cast<int>(n / level_rows);
    if (nsg::wide_levels(pd) != want) {
        std::printf("failed: %d unknowns, %g entries, %g rows\n", n, entries, level_rows);
        ++failures;
    }
}

// the instances of n unknowns with which each solve runs level after level
void levels(int n, double level_rows, double entries, bool wide, std::set<int> transposed,
            std::set<int> complex) {
    for (int count : {1, 148, 149, 296, 297, 592, 740, 741, 1184}) {
        const nsg::FlowBatch b{count, 32, n, level_rows, entries, wide};
        if (nsg::transposed_levels_pay(b) != (transposed.count(count) == 1) ||
            nsg::complex_levels_pay(b, kLu) != (complex.count(count) == 1)) {
            std::printf("failed: levels of %d, %d instances\n", n, count);
            ++failures;
        }
        // with a workspace the general kernel (256 threads), without one the sweeps
        double* const w = reinterpret_cast<double*>(64);
        nsg::launch_complex_solve(nullptr, nullptr, nullptr, b, kLu, nullptr, w, nullptr);
        if (complex.count(count)) expect("complex levels", n, count, 256);
        nsg::launch_solve(nullptr, nullptr, nullptr, b, kLu, nullptr, w, true, nullptr, nullptr,
                          nullptr);
        if (transposed.count(count)) expect("transposed levels", n, count, 256);
    }
}

}  // namespace

int main() {
    for (auto [count, want] : {std::pair<int, int>{592, 256}, {700, 512}, {888, 512}, {1184, 256}}) {
        const nsg::FlowBatch b{count, 64, 577, 7.0, 9.0, false};  // a mesh's last pass
        nsg::launch_complex_refactor(nullptr, nullptr, nullptr, b, nullptr, kLu, nullptr, nullptr);
        expect("complex refactor", 577, count, want);
    }
    const std::set<int> all = {149, 296, 297, 592, 740, 741, 1184};
    levels(300, 1.0, 1.0, false, {740}, {740});     // a chain: four CTAs hold 592
    levels(10000, 1.0, 1.0, false, all, all);       // one CTA
    levels(10000, 10.0, 1.0, false, all, all);      // a tree of short branches
    levels(10000, 500.0, 1.0, true, {}, {});        // wide levels
    levels(9000, 1.0, 6.0, false, {}, {592, 740, 1184});  // a band: two CTAs and one
    levels(9217, 18.0, 20.0, false, {}, {});        // meshes
    levels(16385, 21.0, 24.0, false, {}, {});
    // meshes (rows of a level from 2.5 to 20), at the sizes where fewer CTAs fit
    check(37, 12, 2.5, 256, 256, 256, 256);
    check(1601, 96, 10.0, 256, 256, 256, 256);
    check(2816, 352, 15.0, 256, 256, 512, 256);  // complex vector: four CTAs up to 2816
    check(2817, 192, 15.0, 256, 256, 256, 512);
    check(6314, 224, 15.0, 256, 256, 512, 512);  // vector and flags: three CTAs up to 6314
    check(6315, 224, 15.0, 256, 512, 512, 512);
    check(8101, 448, 18.0, 512, 512, 512, 512);    // three refactors
    check(10000, 600, 20.0, 512, 512, 512, 512);   // two
    // chains
    check(300, 2, 1.0, 256, 256, 256, 256);
    check(9000, 13, 1.0, 256, 256, 256, 256);
    check(10000, 2, 1.0, 256, 256, 256, 256);
    wide(10002, 1.0, 500.0, true);  // trees of random branches
    wide(502, 1.0, 36.0, true);
    wide(202, 1.0, 16.8, true);
    wide(202, 1.0, 15.0, false);
    wide(1, 0.0, 1.0, true);        // no entries at all
    wide(3000, 1.0, 10.0, false);   // a tree of short branches
    wide(10000, 1.0, 1.0, false);   // a chain
    wide(16385, 24.0, 21.0, false); // meshes
    wide(37, 3.4, 2.5, false);
    wide(20000000, 25.0, 20.0, false);
    std::printf("%d failure(s)\n", failures);
    return failures == 0 ? 0 : 1;
}
