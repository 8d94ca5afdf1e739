// Device-side descriptors shared by the host batch code and the kernels.
#pragma once
#include <cstdint>

namespace nsg {

// Index of each plan array in PlanDesc::off; order matches the host's
// NSG_PLAN_ARRAYS list in plan.cpp.
enum PlanArray : int {
    PA_perm_row, PA_perm_col, PA_col_ptr, PA_row_idx, PA_diag_pos, PA_lu_src,
    PA_upd_start, PA_upd_dst, PA_lrow_ptr, PA_lrow_pos, PA_lrow_col, PA_urow_ptr,
    PA_urow_pos, PA_urow_col, PA_col_lev_ptr, PA_col_lev, PA_fwd_lev_ptr, PA_fwd_lev,
    PA_bwd_lev_ptr, PA_bwd_lev, PA_tbw_lev_ptr, PA_tbw_lev, PA_rowcopy_pos, PA_umeta,
    PA_piv_rank, PA_gmin_pos, PA_lp, PA_COUNT
};

struct PlanDesc {
    int32_t n, nnz_a, nnz_lu;
    int32_t n_col_lev, n_fwd_lev, n_bwd_lev, n_tbw_lev;
    int32_t max_col;  // longest LU column
    int32_t nnz_l, nnz_u;  // strictly lower / upper entries
    int32_t kind;          // kPlanMarkowitz or kPlanAmdLu
    int32_t has_map;       // 1: PA_upd_start / PA_upd_dst hold the update map
    int32_t map16;         // 1: the update map is packed as uint16 positions
                           // (every column is shorter than 65,537 rows)
    int64_t off[PA_COUNT];  // int32-word offsets into the plan pool
    int64_t words;          // words from off[0] that hold all of the plan's arrays
    // Level program (PA_lp; lp_words 0: none): section ends in steps and
    // word offsets of its parts (TopologyPlan); lp_at: its copy in shared
    // memory, set by a kernel that made one.
    int32_t lp_words, lp_core, lp_steps[4], lp_src, lp_perm;
    const int32_t* lp_at;
};

// Whether a plan's levels hold so many rows for the entries of each that a thread
// per row and a barrier per level solve it faster than a warp per row: 16 times
// as many rows in a level as entries in a row (an interconnect tree of random
// branches: one entry, 10 rows a level at 100 unknowns, 500 at 10,000; meshes,
// bands and chains at most 2 rows per entry).  A warp has one lane at work in a row
// of one entry: 592 solves of 1502-unknown trees took 0.27 ms, 0.07 here, of
// 10,002 5.2 and 0.58 ms, one transient of 3000 nodes 100 and 80 ms; 592 of 102
// unknowns (10 rows a level, a warp per row) 0.04 ms either way.
#ifdef __CUDACC__
__host__ __device__
#endif
inline bool wide_levels(const PlanDesc& pd) {
    const long long n = pd.n;
    return 8LL * (pd.nnz_lu - pd.n) * pd.n_fwd_lev <= n * n;
}

#ifdef __CUDACC__
// Entry k of a plan's update map: the position in column j that update k
// of U(r, j) writes.  Packed plans (map16) hold it in 16 bits, halving the
// map reads of the refactor; the values are the same.
__device__ __forceinline__ int32_t upd_at(const int32_t* upd_dst, int32_t map16, int64_t k) {
    return map16 ? static_cast<int32_t>(reinterpret_cast<const uint16_t*>(upd_dst)[k])
                 : upd_dst[k];
}
#endif

#ifdef __CUDACC__
// U entry q of a plan's umeta without its run bit (kRunBit of the third word).
__device__ __forceinline__ int4 u_entry(const int4* umeta, int32_t q) {
    int4 m = umeta[q];
    m.z &= 0x7fffffff;
    return m;
}
#endif

struct InstDesc {
    int32_t plan;   // index into the PlanDesc array
    int32_t index;  // the instance's position in the caller's arrays
    int64_t a_off;   // into the caller's A values (doubles)
    int64_t lu_off;  // into the batch's LU values
    int64_t x_off;   // into the caller's rhs / solution vectors
    int64_t w_off;   // into the batch's sweep workspace
    int64_t lrows_off;  // into the batch's row-major L copy
    int64_t urows_off;  // into the batch's row-major U copy
};

// Engine whose factorization a plan replays.
//   kPlanMarkowitz: SparseMatrix::factor (src/solver/factor.cpp:980-1052).
//     U(r, j) = a(r, j) * (1 / p_r), L unscaled, the pivot stored as its
//     reciprocal; U entries applied in ascending row order.
//   kPlanAmdLu: AmdLuSolver::refactor_replay_ (src/core/amd_lu_solver.cpp:
//     214-271).  U unscaled, L(i, k) = x_i / u_kk, the pivot stored as is; U
//     entries applied in the stored (reach) order.
enum : int32_t { kPlanMarkowitz = 0, kPlanAmdLu = 1 };

// What a refactor checks beyond an exact zero pivot.
//   kCheckNone:     nothing (spFactor; a replay whose pivots the host chose).
//   kCheckNumeric:  a numeric() on an already factored solver.  Markowitz:
//     the pivot re-validation of order_and_factor (factor.cpp:929-947).
//     AMD-LU: factor_'s threshold pivot choice (amd_lu_solver.cpp:134-157)
//     must pick the plan's pivot row.  Failure -> kStatusReorder.
//   kCheckRefactor: a refactorize().  Markowitz: as kCheckNone.  AMD-LU: the
//     replay's pivot-growth test (amd_lu_solver.cpp:256-259); failure ->
//     kStatusReorder (the reference falls back to a full factor_).
enum : int { kCheckNone = 0, kCheckNumeric = 1, kCheckRefactor = 2 };

// Per-instance status codes written by the refactor.
enum : int32_t {
    kStatusOk = 0,
    kStatusSingular = 102,  // exact zero pivot (SparseError::ZeroDiag)
    kStatusReorder = 103,   // pivot failed the relative threshold
    kStatusTimeout = 104,   // a bounded dependency wait gave up (no result)
    kStatusNeedOrder = 105, // a solver's first numeric(): the host orders on this matrix
};

}  // namespace nsg
