// Device plan of one factored topology: the LU pattern in pivot (internal)
// order plus everything the batched refactor and the four triangular sweeps
// need, as flat int32 arrays ready to upload.
#pragma once
#include <cstdint>
#include <memory>
#include <utility>
#include <vector>

namespace nsg {

// Largest update map a plan carries (int32 words; default 2^30, 4 GiB),
// process-wide (nsg_set_update_map_limit).
int64_t update_map_limit();
void set_update_map_limit(int64_t words);

// An allocator whose resize() leaves new int32 elements uninitialised: the
// refactor's update map (one word per multiply-subtract, gigabytes for large
// grids) is written entirely by the threads that fill it, so each thread
// first-touches its own pages instead of one thread zeroing them all.
template <class T>
struct UninitAllocator : std::allocator<T> {
    template <class U>
    struct rebind {
        using other = UninitAllocator<U>;
    };
    UninitAllocator() = default;
    template <class U>
    UninitAllocator(const UninitAllocator<U>&) noexcept {}
    template <class U>
    void construct(U* p) noexcept {
        ::new (static_cast<void*>(p)) U;
    }
    template <class U, class... Args>
    void construct(U* p, Args&&... args) {
        ::new (static_cast<void*>(p)) U(std::forward<Args>(args)...);
    }
};

class MarkowitzOrder;
class AmdLuFactor;

constexpr int32_t kRunBit = INT32_MIN;  // of TopologyPlan::umeta's third words

// Whether a Newton kernel runs a factor without a level program on one warp in
// shared memory (cta_refactor_small) rather than on the dataflow kernels: at
// most 128 unknowns and 512 entries.  A property of the plan alone, so that a
// circuit runs alike beside any others and in any launch shape.  The line:
// transients of n fully coupled RC nodes, 400 instances, take 14.6 ms on one
// warp and 17.4 ms on the dataflow kernels with n = 12, 17.1 and 19.0 with 16,
// 20.8 and 20.9 with 20 (484 entries), 25.4 and 24.0 with 24 (676), 71 and 37
// with 40; MOS networks of 60 nodes (936 entries) 430 and 156 ms.  One instance
// alone is faster on the dataflow kernels from n = 12 on (4.3 and 3.1 ms).
constexpr int32_t kOneWarpEntries = 512;
constexpr bool one_warp_factor(int32_t n, int32_t nnz_lu) {
    return n <= 128 && nnz_lu <= kOneWarpEntries;
}

// Engines whose pivot sequence a plan replays.
enum PlanKindHost : int32_t {
    kPlanKindMarkowitz = 0,  // SparseMatrix (Sparse 1.3): U scaled by 1/pivot
    kPlanKindAmdLu = 1,      // AmdLuSolver: L scaled by 1/pivot
};

struct TopologyPlan {
    int32_t kind = kPlanKindMarkowitz;
    int32_t n = 0;
    int32_t nnz_a = 0;   // slots of the caller's CSC pattern
    int32_t nnz_lu = 0;  // originals + fill-ins
    int32_t max_col = 0; // longest LU column

    // internal index i (0-based) -> external row / column (0-based).
    std::vector<int32_t> perm_row, perm_col;

    // LU in CSC, internal order.  In column j: positions
    // col_ptr[j]..diag_pos[j]-1 are U (rows < j), diag_pos[j] is the pivot,
    // diag_pos[j]+1..col_ptr[j+1]-1 are L (rows > j).  Markowitz plans keep
    // rows ascending; AMD-LU plans keep the U rows in the order the
    // refactor must apply them (the reach's topological order) and the L
    // rows in the reference's stored order.
    std::vector<int32_t> col_ptr, row_idx, diag_pos;

    // Load map: per LU position, the caller's CSC slot, or -1 for a fill-in.
    std::vector<int32_t> lu_src;
    // Inverse: per caller slot, its LU position.
    std::vector<int32_t> a_to_lu;

    // Refactor update map.  For the U entry at position q = (r, j):
    // upd_start[q] indexes upd_dst, where the |L(:, r)| destinations of
    // L(:, r)'s rows are stored in L(:, r)'s order, as positions relative to
    // the start of column j.
    std::vector<int32_t> upd_start;
    std::vector<int32_t, UninitAllocator<int32_t>> upd_dst;
    // False when the map would exceed update_map_limit(): upd_start is then
    // all zero, upd_dst empty, and the grid-wide refactor finds each
    // destination through a per-warp row -> position map instead.
    bool has_update_map = true;

    // L by rows (strictly lower, columns ascending) and U by rows (strictly
    // upper, columns ascending): LU position and column of each entry.
    std::vector<int32_t> lrow_ptr, lrow_pos, lrow_col;
    std::vector<int32_t> urow_ptr, urow_pos, urow_col;
    // Per LU position: its index in the row-major copy of L (rows > column)
    // or of U (rows < column), which the refactor writes alongside the
    // column-major values so the sweeps read contiguous rows; -1 for pivots.
    std::vector<int32_t> rowcopy_pos;
    // Per LU position q of a U entry (r, j): {r, diag_pos[r], |L(:, r)|,
    // upd_start[q]} packed as four int32 (zeros elsewhere), so one 16-byte
    // load gives the refactor everything it needs to apply entry q.  The third
    // has its top bit (kRunBit) set when entry q + 1 = (r', j) continues a
    // run: L(:, r) is r' followed by L(:, r') in stored order.
    std::vector<int32_t> umeta;

    // Level schedules (ptr over levels, then members sorted by level).
    //   col:  column j after every r with U(r, j) != 0  (refactor and the
    //         forward sweep of the transposed solve)
    //   fwd:  row i after every c with L(i, c) != 0      (forward solve)
    //   bwd:  row i after every c with U(i, c) != 0      (backward solve)
    //   tbw:  column i after every r with L(r, i) != 0   (transposed backward)
    std::vector<int32_t> col_lev_ptr, col_lev;
    std::vector<int32_t> fwd_lev_ptr, fwd_lev;
    std::vector<int32_t> bwd_lev_ptr, bwd_lev;
    std::vector<int32_t> tbw_lev_ptr, tbw_lev;

    // AMD-LU plans only (empty otherwise), per column k: the pivot's rank
    // among the candidate rows (pivot + L rows, in reach order; -1 when the
    // pivot was outside the reach), and the position, relative to the
    // column start, of the entry that receives diag_gmin (the row of the
    // column's own diagonal element of A), or -1 when the column has none.
    std::vector<int32_t> piv_rank, gmin_pos;

    // Level program (build_level_program; empty when the plan has none): the
    // refactor and the sweeps of a small sparse factor as steps of up to 32
    // independent entries, packed into words that a kernel keeps in shared
    // memory.  It works on unscaled values (a U entry is multiplied by its
    // pivot's reciprocal where it is used), named by their byte offset in the
    // kernel's space: the LU positions, the vector (n), the pivots (n), a zero,
    // a one.  An entry subtracts up to kLevelTerms terms from one value; longer
    // sums are several entries, one after another.  Layout in words: LevelStep
    // of every step (four words); lu_src (uint16 per LU position, 0xffff for a
    // fill-in), perm_row and perm_col (uint16); per section the terms (two
    // words each: first | scale << 16, second) and entries (one word each:
    // target | LevelFlag bits, aux << 16) of its steps; lp_core words up to
    // the transposed sections.  Of a step of w entries, term k of entry e is
    // at k * w + e, short entries padded with (zero, zero, zero), which
    // subtracts +0.0.
    std::vector<int32_t> lp;
    int32_t lp_core = 0;
    // Step ends: factor and forward sweep, backward sweep, transposed sweep
    // over U, over L.
    int32_t lp_steps[4] = {0, 0, 0, 0};
    int32_t lp_src = 0, lp_perm = 0;   // word offsets
    // Doubles of shared memory the program works in.
    int32_t lp_doubles() const { return lp.empty() ? 0 : nnz_lu + 2 * n + 2; }
    // Words of the plan that a kernel keeps in shared memory: the level
    // program (with the transposed section if asked for), else all arrays of a
    // plan of at most 128 unknowns, else none.
    int32_t stage_words(bool transposed) const;

    // Algorithmic work: multiply-subtract updates of one refactor (each is
    // 2 flops), and the reciprocal pivots.
    int64_t updates = 0;

    int64_t refactor_flops() const { return 2 * updates + n; }
    // Compulsory bytes of one refactor: read A, write LU, the index stream
    // (update map + LU pattern), the reciprocal diagonal.
    int64_t refactor_bytes() const {
        return 8LL * nnz_a + 8LL * nnz_lu + (map16() ? 2LL : 4LL) * updates +
               4LL * (nnz_lu + n) + 8LL * n;
    }
    // The device copy of the update map is packed as uint16 positions when
    // every column is short enough for them.
    bool map16() const { return has_update_map && max_col <= 65536; }
    int64_t solve_bytes() const { return 12LL * nnz_lu + 16LL * n; }

    // Total int32 words this plan occupies on the device.
    int64_t device_words() const;
    // Append all arrays to pool; offsets (in int32 words) go to off[].
    void append_to(std::vector<int32_t>& pool, int64_t* off) const;
};

// One step of a level program: byte offsets of its entries and terms from the
// program's start, entries - 1, and whether any entry is a pivot.
struct LevelStep {
    uint32_t entries, terms, last, pivots;
};
constexpr int32_t kLevelTerms = 2;

// An entry computes t = value - sum (first * scale) * second over its terms, in
// order, and stores t.  The backward sweep starts from value * aux's value
// unless value is zero; the transposed sweep over L stores t * aux's value
// (aux is the one where an entry has no such factor).  In the factor section:
enum LevelFlag : uint32_t {
    kLevelPivot = 1,  // t itself to aux, 1 / t to the target
    kLevelSkip = 2,   // forward sweep: terms with first or first * scale zero are left out
};

// Shared memory the plans of a batch ask of a Newton kernel: the largest space
// of a level program or one-warp factor (doubles) and the largest staged part
// of a plan (words); and whether any plan has a level program, or has none and
// runs on the dataflow kernels.
struct PlanStage {
    int32_t doubles = 0, words = 0;
    bool programs = false, dataflow = false;
    void add(const TopologyPlan& p, bool transposed);
};

// Build from the host ordering engine after order_and_factor.  slot_elem[k]
// is the engine element of caller CSC slot k.
TopologyPlan build_plan(const MarkowitzOrder& mo, const std::vector<int32_t>& slot_elem);

// Build from the AMD-LU engine after a successful factor(): the pivot
// sequence, L/U structure and replay order of AmdLuSolver::factor_.
TopologyPlan build_plan_amd(const AmdLuFactor& f);

// Give a plan its level program (TopologyPlan::lp) if it is a small sparse
// Markowitz plan with an update map; clears it otherwise.  The batches of
// circuits call it for each distinct plan they keep.
void build_level_program(TopologyPlan& p);

// Build from an exported structure (the reference's own NeoSolver state):
// elements column by column in internal order (1-based rows/cols), the slot
// map and 1-based permutations.  Throws std::invalid_argument on a malformed
// structure.
TopologyPlan build_plan_from_structure(int32_t n, int32_t nnz_a,
                                       const int32_t* int_to_ext_row,
                                       const int32_t* int_to_ext_col,
                                       int32_t n_elem, const int32_t* elem_row,
                                       const int32_t* elem_col,
                                       const int32_t* slot_to_elem);

}  // namespace nsg
