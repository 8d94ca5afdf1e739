// Batched DC operating point: solve_dc (src/core/dc.cpp:53-175; newton_solve,
// src/core/newton.cpp:51-419) with its direct attempt and the gmin-stepping
// aids, for one circuit instance per CTA, all instances in a single launch.
// Each iteration: device loads, matrix and right-hand-side assembly from the
// stamp program, fixed-pivot refactor (dataflow), forward/backward solve, the
// NIiter convergence test and the INITJCT -> INITFIX -> INITFLOAT cascade.
// Instances converge and stop independently (per-instance convergence mask =
// its CTA leaving the loop).
#include "dc_op.cuh"

#include <cuda_runtime.h>

namespace nsg {

// kBlocks CTAs of kThreads threads per SM.  subset (optional)
// lists the descriptor positions to run, one per block.  ctls[index] is the
// instance's operating-point controller: zeroed by the host for a fresh run,
// kept across launches when an instance stopped with kStatusReorder.
template <int kThreads, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks)
newton_dc_kernel(const PlanDesc* __restrict__ plans, const int32_t* __restrict__ lu_pool,
                 const DcDesc* __restrict__ descs, const int32_t* __restrict__ subset,
                 const int32_t* __restrict__ prog, const double* __restrict__ params,
                 double* __restrict__ work, double* __restrict__ solutions,
                 int32_t* __restrict__ status, int32_t* __restrict__ iterations,
                 DcCtl* __restrict__ ctls, NewtonOptions opt, int colbuf, int scratch_doubles,
                 int stage_doubles, int plan_words, int32_t* rmaps, int64_t rmap_stride) {
    extern __shared__ double smem[];
    const DcDesc d = descs[subset ? subset[blockIdx.x] : blockIdx.x];
    __shared__ PlanDesc s_pd;
    const int32_t* pool = stage_plan(
        plans[d.plan], lu_pool,
        plan_words > 0 ? reinterpret_cast<int32_t*>(smem + scratch_doubles + stage_doubles) : nullptr,
        plan_words, &s_pd);
    const PlanDesc& pd = s_pd;
    double* stage = (d.stage_len <= stage_doubles) ? smem + scratch_doubles : nullptr;
    stage_copy(d, work, stage, true);
    // Per-thread views (not a shared copy as in the transient kernel): the
    // dataflow scratch of large meshes fills the shared memory of two CTAs
    // per SM to within a few hundred bytes.
    Inst v = make_inst(d, prog, params, work, stage);
    static_assert(kThreads <= 32 * kDcMaxWarps, "the host sizes the row maps for kDcMaxWarps");
    if (rmaps) {
        v.rmaps = rmaps + static_cast<int64_t>(blockIdx.x) * kDcMaxWarps * rmap_stride;
        v.rmap_stride = rmap_stride;
    }
    __shared__ IntegCtx ctx;
    __shared__ SolverState solver;
    __shared__ int32_t s_fresh;
    DcCtl* ctl = ctls + d.index;
    constexpr int kFirst = kModeDcOp | kModeInitJct, kCont = kModeDcOp | kModeInitFloat;

    if (threadIdx.x == 0) s_fresh = (ctl->active == 0);
    __syncthreads();
    const bool fresh = s_fresh != 0;
    if (fresh) {
        for (int32_t k = threadIdx.x; k < kMosRecCount * v.n_mos; k += blockDim.x) v.mrec[k] = 0.0;
        for (int32_t k = threadIdx.x; k < 4 * d.n_states; k += blockDim.x) v.st[0][k] = 0.0;
        for (int32_t i = threadIdx.x; i < v.n; i += blockDim.x) v.x[i] = 0.0;
    }
    if (threadIdx.x == 0) {
        if (fresh) dc_op_start(ctl, kFirst, opt.first_aid);
        ctx = IntegCtx{};
        ctx.order = 1;
        ctx.time = 0.0;
        solver.factored = fresh ? 0 : 1;
    }
    __syncthreads();
    // solve_dc (dc.cpp:53-175): direct attempt, true gmin stepping, gmin stepping
    const int32_t code = dc_operating_point(v, d.n_states, pd, pool, &ctx, &solver, ctl, opt,
                                            kFirst, kCont, true, work + d.dcsave_off, smem, colbuf,
                                            scratch_doubles);

    stage_copy(d, work, stage, false);
    double* out = solutions + d.sol_off;
    for (int32_t i = threadIdx.x; i < v.n; i += blockDim.x) out[i] = v.x[i];
    if (threadIdx.x == 0) {
        status[d.index] = code;
        iterations[d.index] = ctl->total;
    }
}

namespace {

size_t dc_scratch_bytes(int max_col, int max_n, int warps) {
    const int colbuf = (max_col + 31) & ~31;
    const size_t a = flow_smem_bytes(colbuf, max_n, warps);
    const size_t b = flow_solve_smem_bytes(max_n);
    return a > b ? a : b;
}

int dc_sm_count() {
    static const int sms = [] {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        return n > 0 ? n : 1;
    }();
    return sms;
}

}  // namespace

size_t dc_smem_bytes(int max_col, int max_n) {
    return dc_scratch_bytes(max_col, max_n, kFlowWarps);
}

// Launch shape: up to one instance per SM, one CTA of 24 warps has the SM's
// registers (80 a thread) to itself; more instances run as CTAs of 16 warps,
// two per SM (64 registers).  One 2305-unknown mesh took 12.8 ms with the
// first and 16.3 ms with the second shape, 148 of 5185 unknowns 41.7 and
// 55.0 ms, 600 of 257 to 1601 unknowns 18.1 and 14.1 ms.  stage_lens: the
// instances' stage_len, ascending.
cudaError_t launch_newton_dc(const PlanDesc* plans, const int32_t* lu_pool, const DcDesc* descs,
                             const int32_t* subset, int count, const int32_t* prog,
                             const double* params, double* work, double* solutions,
                             int32_t* status, int32_t* iterations, DcCtl* ctls,
                             const NewtonOptions& opt, int max_col, int max_n,
                             const int64_t* stage_lens, int n_stage, int lu_doubles,
                             int plan_words, int32_t* rmaps, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    const int colbuf = (max_col + 31) & ~31;
    const bool wide = count <= dc_sm_count() &&
                      dc_scratch_bytes(max_col, max_n, kDcMaxWarps) <= 200 * 1024;
    const size_t small = sizeof(double) * static_cast<size_t>(lu_doubles);
    const size_t flow = dc_scratch_bytes(max_col, max_n, wide ? kDcMaxWarps : kFlowWarps);
    const size_t scratch = ((flow > small ? flow : small) + 15) & ~size_t{15};
    size_t plan = (sizeof(int32_t) * static_cast<size_t>(plan_words) + 15) & ~size_t{15};
    if (scratch + plan > kStageCapBytes) plan = 0;  // read from global memory instead
    const size_t stage = stage_bytes_for(scratch + plan, stage_lens, n_stage);
    const size_t smem = scratch + stage + plan;
    if (smem > 200 * 1024) return cudaErrorInvalidValue;
    const int scratch_d = static_cast<int>(scratch / sizeof(double));
    const int stage_d = static_cast<int>(stage / sizeof(double));
    const int plan_w = static_cast<int>(plan / sizeof(int32_t));
    auto launch = [&](auto kernel, int threads) -> cudaError_t {
        const cudaError_t e = cudaFuncSetAttribute(
            kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        if (e != cudaSuccess) return e;
        kernel<<<count, threads, smem, stream>>>(plans, lu_pool, descs, subset, prog, params, work,
                                                 solutions, status, iterations, ctls, opt, colbuf,
                                                 scratch_d, stage_d, plan_w, rmaps, max_n);
        return cudaGetLastError();
    };
    constexpr int kWide = 32 * kDcMaxWarps;
    return wide ? launch(newton_dc_kernel<kWide, 1>, kWide)
                : launch(newton_dc_kernel<kFlowThreads, 2>, kFlowThreads);
}

}  // namespace nsg
