// CTA-level building blocks: one thread block refactors / solves one
// instance.  Used by the standalone batched kernels (lu_kernels.cu) and by the
// fused Newton kernel (newton_dc.cu).
//
// Rounding order.  Every value is produced by the same sequence of IEEE
// double operations as the reference's SparseMatrix::factor / solve /
// solve_transposed (src/solver/factor.cpp:980-1052, solve.cpp:6-47,
// :102-141): updates into one entry are applied in ascending pivot order, one
// at a time, with separately rounded multiply and subtract (__dmul_rn,
// __dsub_rn: no FMA contraction).  Results are therefore bit-identical to the
// reference under the same pivot sequence.
#pragma once
#include "host/plan.hpp"
#include "lu_device.cuh"

#include <cuda_runtime.h>

namespace nsg {

constexpr int kFlowWarps = 16;
constexpr int kFlowThreads = kFlowWarps * 32;

// Polls a bounded dependency wait makes before it gives up and its instance
// reports kStatusTimeout (a wait that finds its flag set at the first look
// makes no poll; a limit of 0 gives up at the first wait that has to poll).
// Every translation unit that includes this header keeps its own copy in
// constant memory and registers a setter; nsg_set_wait_limit writes all of
// them on the current device.
constexpr int kDefaultWaitLimit = 1 << 22;
static __constant__ int c_wait_limit = kDefaultWaitLimit;

// Host: keep `set` in the list nsg_set_wait_limit walks (defined in capi.cpp).
bool register_wait_limit_setter(cudaError_t (*set)(int polls));

namespace {
cudaError_t set_wait_limit_here(int polls) {
    return cudaMemcpyToSymbol(c_wait_limit, &polls, sizeof(int));
}
const bool wait_limit_setter_registered = register_wait_limit_setter(&set_wait_limit_here);
}  // namespace
// Rounds of 32 L(:, r) rows the dataflow refactor loads before applying them.
constexpr int kColChunk = 2;
// Entries whose completion flags a refactoring warp looks at together, entries
// of a run it applies together, and other entries whose operands it loads
// together.  More of each (8, 8, 4) costs registers: at 64 a thread the
// spills took back more than the longer runs gave.
constexpr int kRunLanes = 4;
constexpr int kRun = 4;
constexpr int kGroup = 2;

__device__ __forceinline__ double lu_mul(double x, double y) { return __dmul_rn(x, y); }
__device__ __forceinline__ double lu_sub(double x, double y) { return __dsub_rn(x, y); }

// Completion flags in shared memory: the producer publishes with a release
// store after writing its values, the consumer reads with an acquire load
// before reading them (PTX ld.acquire / st.release at CTA scope).
__device__ __forceinline__ int32_t flag_acquire(const volatile int32_t* f) {
    int32_t v;
    const unsigned addr = static_cast<unsigned>(__cvta_generic_to_shared(const_cast<int32_t*>(f)));
    asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

__device__ __forceinline__ void flag_release(volatile int32_t* f, int32_t v) {
    const unsigned addr = static_cast<unsigned>(__cvta_generic_to_shared(const_cast<int32_t*>(f)));
    asm volatile("st.release.cta.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Verdict on column k of an AMD-LU replay, computed by one warp from the
// column's values after all its U updates (col: relative to the column
// start; dj: the pivot's position; colmax: the largest |U(r, k)| applied).
//   growth_fail (kCheckRefactor only): refactor_replay_'s growth test
//     (amd_lu_solver.cpp:250-259), u_kk == 0 or |u_kk| < 1e-3 *
//     max(colmax, |u_kk|).  On any such column the reference abandons the
//     replay and runs a full factor_ on the same values.
//   code (kCheckNumeric and kCheckRefactor): whether factor_ on these
//     values (amd_lu_solver.cpp:134-157) would pick the plan's pivot row --
//     the first candidate of largest |x| in reach order, unless the row of
//     the column's own diagonal is a candidate within 1e-3 of that maximum;
//     no candidate above zero -> kStatusSingular, another row ->
//     kStatusReorder.  When every column agrees, factor_ reproduces the
//     replay's values bit for bit, so a failed growth test costs nothing.
//   kCheckNone: code is kStatusSingular for u_kk == 0.
// Ends with __syncwarp(): the caller may overwrite the column afterwards.
struct AmdColumn {
    int32_t code;
    bool growth_fail;
};

// The pivot candidate search of amd_column_status, split so a whole CTA can
// run it: each thread scans positions dj + start, dj + start + stride, ...
// and the partial results merge in any order (largest |x|, then lowest
// rank: a total order, since ranks are distinct).
struct AmdCand {
    double best;
    int32_t rank, pos;
};

__device__ __forceinline__ void amd_cand_merge(AmdCand& a, double ob, int32_t orank,
                                               int32_t opos) {
    if (ob > a.best || (ob == a.best && orank < a.rank)) {
        a.best = ob;
        a.rank = orank;
        a.pos = opos;
    }
}

__device__ inline AmdCand amd_cand_scan(const double* col, int32_t dj, int32_t len,
                                        int32_t piv_rank, int start, int stride) {
    AmdCand c{-1.0, INT32_MAX, -1};
    for (int32_t t = dj + start; t < len; t += stride) {
        int32_t rank;
        if (t == dj) {
            if (piv_rank < 0) continue;  // the pivot was not in the reach
            rank = piv_rank;
        } else {
            const int32_t m = t - dj - 1;
            rank = (piv_rank >= 0 && m >= piv_rank) ? m + 1 : m;
        }
        amd_cand_merge(c, fabs(col[t]), rank, t);
    }
    return c;
}

__device__ __forceinline__ AmdCand amd_cand_warp(AmdCand c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, c.best, o);
        const int32_t orank = __shfl_xor_sync(0xffffffffu, c.rank, o);
        const int32_t opos = __shfl_xor_sync(0xffffffffu, c.pos, o);
        amd_cand_merge(c, ob, orank, opos);
    }
    return c;
}

// The verdict from the column's pivot, colmax and (for kCheckNumeric /
// kCheckRefactor) the merged candidate.
__device__ inline AmdColumn amd_verdict(const double* col, int32_t dj, double colmax, int check,
                                        int32_t gpos, const AmdCand& c) {
    const double piv = col[dj];
    AmdColumn r{(piv == 0.0) ? kStatusSingular : kStatusOk, false};
    if (check == kCheckRefactor) {
        const double a = fabs(piv);
        const double cm = a > colmax ? a : colmax;
        r.growth_fail = (piv == 0.0 || (cm > 0.0 && a < 1e-3 * cm));
    }
    if (check == kCheckNumeric || check == kCheckRefactor) {
        if (c.pos < 0 || c.best <= 0.0) {
            r.code = kStatusSingular;
        } else {
            int32_t chosen = c.pos;
            if (gpos >= dj && fabs(col[gpos]) >= c.best * 1e-3) chosen = gpos;
            r.code = (chosen != dj) ? kStatusReorder : (piv == 0.0 ? kStatusSingular : kStatusOk);
        }
    }
    return r;
}

__device__ inline AmdColumn amd_column_status(const double* col, int32_t dj, int32_t len,
                                              double colmax, int check, int32_t piv_rank,
                                              int32_t gpos, int lane) {
    AmdCand c{-1.0, INT32_MAX, -1};
    if (check == kCheckNumeric || check == kCheckRefactor)
        c = amd_cand_warp(amd_cand_scan(col, dj, len, piv_rank, lane, 32));
    const AmdColumn r = amd_verdict(col, dj, colmax, check, gpos, c);
    __syncwarp();
    return r;
}

// Outcome of an AMD-LU refactor from the first column verdict that failed
// (packed by fail_key, ~0 if none) and whether any growth test failed.  A
// refactorize() whose growth tests all pass keeps the replay; otherwise, as
// for a numeric(), the first failing verdict decides.
__device__ __forceinline__ bool amd_verdict_counts(int check, bool any_growth_fail) {
    return check != kCheckRefactor || any_growth_fail;
}

// Value stored at relative position t of a finished column (pivot at dj):
// Markowitz keeps L as eliminated and stores 1 / pivot; AMD-LU divides L by
// the pivot and keeps the pivot.
__device__ __forceinline__ double lu_store_value(bool amd, double v, int32_t t, int32_t dj,
                                                 double piv) {
    if (amd) return t > dj ? __ddiv_rn(v, piv) : v;
    return t == dj ? 1.0 / piv : v;
}

// First failing column and its status, packed for one atomicMin.
__device__ __forceinline__ unsigned long long fail_key(int32_t step, int32_t code) {
    return (static_cast<unsigned long long>(static_cast<uint32_t>(step)) << 32) |
           static_cast<uint32_t>(code);
}

// Dynamic shared memory a kernel may use without asking: 48 KB less its static
// shared memory, for which 1 KB is left.
constexpr size_t kUnaskedSmem = 47 * 1024;

// Shared memory of the dataflow refactor: a column buffer of colbuf doubles per
// warp, then n int32 completion flags.
__host__ __device__ inline size_t flow_smem_bytes(int colbuf, int n, int warps = kFlowWarps) {
    return sizeof(double) * warps * colbuf + sizeof(int32_t) * n;
}

struct RefactorResult {
    int32_t code;  // kStatus*
    int32_t step;  // failing pivot step or -1
};

// Outcome of one column of the dataflow refactor.
struct ColumnResult {
    int32_t code;      // kStatusOk / kStatusSingular / kStatusReorder verdict
    bool growth_fail;  // AMD-LU kCheckRefactor: the replay's growth test failed
    bool timed_out;    // a bounded dependency wait gave up
};

// Loads of another column's factor values: through L1 when one SM owns the
// whole instance, L2-only (ld.global.cg) when columns are finished by other
// SMs and an L1 line could hold values from before their completion.
template <bool kCrossSm>
__device__ __forceinline__ double lu_peer(const double* p) {
    if constexpr (kCrossSm) return __ldcg(p);
    return *p;
}

// Where a column's update destinations come from: the packed update map, or
// per-warp row maps.
enum DestKind : int { kDestMap16 = 0, kDestRowMap = 1 };

// kRun consecutive U entries (r_0, j), (r_1, j), ... of column j that form a
// run -- L(:, r_i) is r_(i+1) and then L(:, r_(i+1)) -- at positions q .. q +
// kRun - 1 of the column in buf, applied together by one warp.  Entry i's
// updates of the other entries of the run are a small triangle, done in
// registers (lane i holds entry i); below it all kRun columns have the same
// rows, so a row's value is read and written once, receives its kRun updates in
// ascending order, and its kRun factors are independent loads in flight
// together.  Of a mesh's updates nine in ten lie in such runs.  dp:
// diag_pos[r_(lane % kRun)]; cnt, us: |L(:, r)| and upd_start of the last
// entry.  Ends with __syncwarp().
template <bool kCrossSm, class Dest>
__device__ __forceinline__ void run_step(bool amd, const double* lu, double* buf, int32_t q,
                                         int32_t dp, int32_t cnt, int32_t us, Dest dest,
                                         double& colmax) {
    const int lane = threadIdx.x & 31;
    int32_t at[kRun];  // diag_pos of each entry's column
#pragma unroll
    for (int i = 0; i < kRun; ++i) at[i] = __shfl_sync(0xffffffffu, dp, i);
    const int32_t l0 = at[kRun - 1] + 1;
    double x = lane < kRun ? buf[q + lane] : 0.0;
    const double rd = (lane < kRun && !amd) ? lu_peer<kCrossSm>(lu + dp) : 0.0;
    double tri[kRun], l[kRun], u[kRun];
    int32_t d;
#pragma unroll
    for (int i = 0; i < kRun - 1; ++i)
        tri[i] = (lane > i && lane < kRun) ? lu_peer<kCrossSm>(lu + at[i] + lane - i) : 0.0;
    auto load = [&](int32_t t) {
        d = t < cnt ? dest(us, l0, t) : 0;
#pragma unroll
        for (int i = 0; i < kRun; ++i)
            l[i] = t < cnt ? lu_peer<kCrossSm>(lu + at[i] + (kRun - i) + t) : 0.0;
    };
    load(lane);
#pragma unroll
    for (int i = 0; i < kRun; ++i) {
        const double v = amd ? x : lu_mul(x, rd);
        u[i] = __shfl_sync(0xffffffffu, v, i);
        if (lane == i) x = v;
        if (i < kRun - 1 && lane > i) x = lu_sub(x, lu_mul(u[i], tri[i]));
        colmax = fmax(colmax, fabs(u[i]));
    }
    if (lane < kRun) buf[q + lane] = x;
    for (int32_t t = lane; t < cnt + lane; t += 32) {
        if (t >= 32) load(t);
        if (t < cnt) {
            double v = buf[d];
#pragma unroll
            for (int i = 0; i < kRun; ++i) v = lu_sub(v, lu_mul(u[i], l[i]));
            buf[d] = v;
        }
    }
    __syncwarp();
}

// Column j of the left-looking dataflow refactor, by one warp.  buf holds the
// column while it is eliminated (shared memory, or the column's own place in
// lu); probe(r) reads column r's completion flag (acquire).  Loads A
// (through lu_src, diag_gmin added), applies every U entry in stored order
// after column r is done, judges the pivot (check_pivots, kCheck*), and
// writes the column (and its row-major copies) to lu.  Ends with
// __syncwarp(); the caller publishes completion.  The position in column j
// of each row of L(:, r) comes from the plan's update map, or, when rmap is
// given (always for plans without a map, pd.has_map == 0), from rmap: this
// warp's row -> position scratch (pd.n words), written for column j's rows
// first.  The row map reads L(:, r)'s row indices, which every consumer
// column of r shares, instead of a map entry per update.
template <bool kCrossSm, int kPlan, int kDest, int kChunk = kColChunk, int kGroupN = kGroup,
          class Probe, class Publish>
__device__ __forceinline__ void refactor_column(
    const PlanDesc& pd, const int32_t* __restrict__ pool, const double* __restrict__ a,
    double* lu, double diag_gmin, int check_pivots, double rel_threshold, int32_t j, double* buf,
    double* __restrict__ lrows, double* __restrict__ urows, Probe probe, Publish publish,
    int32_t* rmap = nullptr) {
    const int32_t* col_ptr = pool + pd.off[PA_col_ptr];
    const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
    const int32_t* lu_src = pool + pd.off[PA_lu_src];
    const int32_t* upd_dst = pool + pd.off[PA_upd_dst];
    const int32_t map16 = kDest == kDestMap16 ? 1 : pd.map16;
    const bool amd = kPlan < 0 ? pd.kind == kPlanAmdLu : kPlan == kPlanAmdLu;
    const int32_t* piv_rank = pool + pd.off[PA_piv_rank];
    const int32_t* gmin_pos = pool + pd.off[PA_gmin_pos];
    constexpr int kLanes = kGroupN > kRunLanes ? kGroupN : kRunLanes;
    const int lane = threadIdx.x & 31;

    const int32_t c0 = col_ptr[j];
    const int32_t len = col_ptr[j + 1] - c0;
    const int32_t dj = diag_pos[j] - c0;
    const int32_t gp = amd ? gmin_pos[j] : dj;
    const int32_t* row_idx = pool + pd.off[PA_row_idx];
    const bool mapped = kDest < 0 ? rmap == nullptr : kDest == kDestMap16;
    for (int32_t t = lane; t < len; t += 32) {
        const int32_t s = lu_src[c0 + t];
        double v = (s >= 0) ? a[s] : 0.0;
        if (t == gp && diag_gmin != 0.0) v = __dadd_rn(v, diag_gmin);
        buf[t] = v;
        if (!mapped) rmap[row_idx[c0 + t]] = t;
    }
    __syncwarp();
    // Position in column j of entry t of L(:, r) (its k-th update).
    auto dest = [&](int32_t us, int32_t l0, int32_t t) -> int32_t {
        return mapped ? upd_at(upd_dst, map16, us + t) : rmap[row_idx[l0 + t]];
    };
    double colmax = 0.0;  // AMD-LU: largest |U(r, j)| applied
    // U-entry metadata {r, diag_pos[r], |L(:,r)|, upd_start} is held 32
    // entries at a time in registers (lane k holds entry base + k) and
    // broadcast by shuffle; chain: bit k says that entry base + k + 1 continues
    // entry base + k's run.
    const int4* umeta = reinterpret_cast<const int4*>(pool + pd.off[PA_umeta]) + c0;
    bool timed_out = false;
    int32_t base = 0;
    int4 meta;
    unsigned chain;
    auto window = [&](int32_t at) {
        base = at;
        meta = at + lane < dj ? umeta[at + lane] : make_int4(0, 0, 0, 0);
        chain = __ballot_sync(0xffffffffu, meta.z < 0);
    };
    window(0);
    for (int32_t q = 0; q < dj;) {
        if (q - base > 32 - kLanes && base + 32 < dj) window(q);
        const int32_t k0 = q - base;
        // How many of the next entries' source columns are done, at least one.
        const int32_t ahead = min(min(kLanes, dj - q), 32 - k0);
        const int32_t src = __shfl_sync(0xffffffffu, meta.x, k0 + (lane & (kLanes - 1)));
        int32_t ready = 0;
        for (int spins = 0;;) {
            const bool open = lane < ahead && probe(src) == 0;
            const unsigned mask = __ballot_sync(0xffffffffu, open);
            ready = mask ? __ffs(mask) - 1 : ahead;
            if (ready > 0) break;
            if (++spins > c_wait_limit) {
                timed_out = true;
                break;
            }
            __nanosleep(64);
        }
        if (timed_out) break;
        __syncwarp();
        // entries of q's run in the window
        const int32_t run = __ffs(~(chain >> k0));
        const int32_t both = min(run, ready);
        if (both >= kRun) {
            const int32_t last = k0 + kRun - 1;
            run_step<kCrossSm>(amd, lu, buf, q,
                               __shfl_sync(0xffffffffu, meta.y, k0 + (lane & (kRun - 1))),
                               __shfl_sync(0xffffffffu, meta.z, last) & 0x7fffffff,
                               __shfl_sync(0xffffffffu, meta.w, last), dest, colmax);
            q += kRun;
        } else {
            // Up to kGroup entries of any structure: the first 32 rows of
            // every L(:, r), their destinations and the pivot reciprocals
            // are loaded together, then applied one entry after another.
            const int32_t count = min(kGroupN, ready);
            int32_t l0[kGroupN], cnt[kGroupN], us[kGroupN], dd[kGroupN];
            double rd[kGroupN], ll[kGroupN];
#pragma unroll
            for (int g = 0; g < kGroupN; ++g) {
                const int32_t k = k0 + min(g, count - 1);
                const int32_t dp = __shfl_sync(0xffffffffu, meta.y, k);
                l0[g] = dp + 1;
                cnt[g] = __shfl_sync(0xffffffffu, meta.z, k) & 0x7fffffff;
                if (g >= count) cnt[g] = 0;
                us[g] = __shfl_sync(0xffffffffu, meta.w, k);
                rd[g] = (amd || g >= count) ? 0.0 : lu_peer<kCrossSm>(lu + dp);
                ll[g] = lane < cnt[g] ? lu_peer<kCrossSm>(lu + l0[g] + lane) : 0.0;
                dd[g] = lane < cnt[g] ? dest(us[g], l0[g], lane) : 0;
            }
#pragma unroll
            for (int g = 0; g < kGroupN; ++g) {
                if (g < count) {
                    const double u = amd ? buf[q + g] : lu_mul(buf[q + g], rd[g]);
                    colmax = fmax(colmax, fabs(u));
                    __syncwarp();
                    if (lane == 0) buf[q + g] = u;
                    if (lane < cnt[g]) buf[dd[g]] = lu_sub(buf[dd[g]], lu_mul(u, ll[g]));
                    // rows beyond the first 32, kChunk rounds at a time (the
                    // destinations of one entry are distinct, so the order
                    // among them does not matter)
                    for (int32_t t0 = 32; t0 < cnt[g]; t0 += 32 * kChunk) {
                        int32_t d[kChunk];
                        double l[kChunk];
#pragma unroll
                        for (int k = 0; k < kChunk; ++k) {
                            const int32_t t = t0 + 32 * k + lane;
                            d[k] = (t < cnt[g]) ? dest(us[g], l0[g], t) : 0;
                            l[k] = (t < cnt[g]) ? lu_peer<kCrossSm>(lu + l0[g] + t) : 0.0;
                        }
#pragma unroll
                        for (int k = 0; k < kChunk; ++k)
                            if (t0 + 32 * k + lane < cnt[g])
                                buf[d[k]] = lu_sub(buf[d[k]], lu_mul(u, l[k]));
                    }
                    __syncwarp();
                }
            }
            q += count;
        }
    }
    timed_out = __shfl_sync(0xffffffffu, timed_out, 0);
    const double piv = buf[dj];
    ColumnResult res{kStatusOk, false, timed_out};
    if (amd) {
        const AmdColumn v = amd_column_status(buf, dj, len, colmax, check_pivots, piv_rank[j],
                                              gmin_pos[j], lane);
        res.code = v.code;
        res.growth_fail = v.growth_fail;
    } else if (check_pivots == kCheckNumeric) {
        double largest = 0.0;
        for (int32_t t = dj + 1 + lane; t < len; t += 32) largest = fmax(largest, fabs(buf[t]));
        largest = warp_max(largest);
        res.code = !(largest * rel_threshold < fabs(piv)) ? kStatusReorder : kStatusOk;
    } else {
        res.code = (piv == 0.0) ? kStatusSingular : kStatusOk;
    }
    // The column's values, then its completion: the row-major copies, which
    // only the sweeps read, follow off the other columns' critical path.
    const double inv = amd ? piv : 1.0 / piv;
    for (int32_t t = lane; t < len; t += 32) {
        double v = buf[t];
        if (amd ? t > dj : t == dj) v = amd ? __ddiv_rn(v, piv) : inv;
        lu[c0 + t] = v;
        buf[t] = v;
    }
    __syncwarp();
    publish(res);
    if (lrows) {
        const int32_t* rowcopy = pool + pd.off[PA_rowcopy_pos];
        for (int32_t t = lane; t < len; t += 32) {
            if (t < dj) urows[rowcopy[c0 + t]] = buf[t];
            else if (t > dj) lrows[rowcopy[c0 + t]] = buf[t];
        }
    }
    __syncwarp();
}

// Dataflow refactor of one instance by the whole CTA (blockDim.x ==
// kFlowThreads).  Warps claim columns in pivot order from a shared counter;
// before using column r a warp waits for done[r], so independent columns
// overlap and the dense trailing block pipelines as a wavefront.  Column j
// stays in a per-warp shared buffer from its load (A gathered through lu_src,
// diag_gmin added) to its write-back.  check_pivots is a kCheck* mode: for
// Markowitz plans kCheckNumeric applies the re-validation test of
// SparseMatrix::order_and_factor (factor.cpp:929-947), otherwise only an
// exact zero pivot fails, as in SparseMatrix::factor; AMD-LU plans follow
// amd_column_status.  Every
// wait is bounded: past c_wait_limit polls the instance reports kStatusTimeout
// and the warp moves on, so the CTA always finishes.  Begins and ends with
// __syncthreads().
// When lrows/urows are given, every L and U entry is also written to its
// position in the row-major copies the dataflow sweeps read.
template <int kPlan, int kDest>
static __device__ __noinline__ RefactorResult cta_refactor_flow_as(const PlanDesc& pd, const int32_t* __restrict__ pool,
                                                   const double* __restrict__ a, double* __restrict__ lu,
                                                   double diag_gmin, int check_pivots,
                                                   double rel_threshold, double* smem, int colbuf,
                                                   double* __restrict__ lrows,
                                                   double* __restrict__ urows, int32_t* rmaps,
                                                   int64_t rmap_stride) {
    const int32_t n = pd.n;
    const bool amd = kPlan == kPlanAmdLu;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    double* buf = smem + warp * colbuf;
    volatile int32_t* done =
        reinterpret_cast<volatile int32_t*>(smem + (blockDim.x >> 5) * colbuf);
    int32_t* rmap = rmaps ? rmaps + warp * rmap_stride : nullptr;

    __shared__ int32_t s_next, s_timeout, s_growth;
    __shared__ unsigned long long s_fail;
    __syncthreads();
    for (int32_t j = threadIdx.x; j < n; j += blockDim.x) done[j] = 0;
    if (threadIdx.x == 0) {
        s_next = 0;
        s_timeout = 0;
        s_growth = 0;
        s_fail = ~0ull;
    }
    __syncthreads();

    for (;;) {
        int32_t j = 0;
        if (lane == 0) j = atomicAdd(&s_next, 1);
        j = __shfl_sync(0xffffffffu, j, 0);
        if (j >= n) break;
        refactor_column<false, kPlan, kDest>(
            pd, pool, a, lu, diag_gmin, check_pivots, rel_threshold, j, buf, lrows, urows,
            [&](int32_t r) { return flag_acquire(done + r); },
            [&](const ColumnResult& c) {
                if (lane != 0) return;
                if (c.timed_out) s_timeout = 1;
                else if (c.code != kStatusOk) atomicMin(&s_fail, fail_key(j, c.code));
                if (c.growth_fail) s_growth = 1;
                flag_release(done + j, 1);
            },
            rmap);
    }
    __syncthreads();
    RefactorResult res;
    if (s_timeout) {
        res.code = kStatusTimeout;
        res.step = -1;
    } else if (s_fail == ~0ull || (amd && !amd_verdict_counts(check_pivots, s_growth != 0))) {
        res.code = kStatusOk;
        res.step = -1;
    } else {
        res.code = static_cast<int32_t>(s_fail & 0xffffffffu);
        res.step = static_cast<int32_t>(s_fail >> 32);
    }
    __syncthreads();
    return res;
}

// The dataflow refactor compiled for the plan's engine and for the way its
// update destinations are found (a column that fits shared memory has a packed
// update map unless row maps were asked for).
static __device__ __forceinline__ RefactorResult cta_refactor_flow(
    const PlanDesc& pd, const int32_t* pool, const double* a, double* lu, double diag_gmin,
    int check_pivots, double rel_threshold, double* smem, int colbuf, double* lrows = nullptr,
    double* urows = nullptr, int32_t* rmaps = nullptr, int64_t rmap_stride = 0) {
    if (pd.kind == kPlanAmdLu) {
        if (rmaps)
            return cta_refactor_flow_as<kPlanAmdLu, kDestRowMap>(
                pd, pool, a, lu, diag_gmin, check_pivots, rel_threshold, smem, colbuf, lrows, urows,
                rmaps, rmap_stride);
        return cta_refactor_flow_as<kPlanAmdLu, kDestMap16>(
            pd, pool, a, lu, diag_gmin, check_pivots, rel_threshold, smem, colbuf, lrows, urows,
            nullptr, 0);
    }
    if (rmaps)
        return cta_refactor_flow_as<kPlanMarkowitz, kDestRowMap>(
            pd, pool, a, lu, diag_gmin, check_pivots, rel_threshold, smem, colbuf, lrows, urows,
            rmaps, rmap_stride);
    return cta_refactor_flow_as<kPlanMarkowitz, kDestMap16>(
        pd, pool, a, lu, diag_gmin, check_pivots, rel_threshold, smem, colbuf, lrows, urows, nullptr,
        0);
}

// x <- A^{-1} x (SparseMatrix::solve, or AmdLuSolver::solve,
// amd_lu_solver.cpp:303-344, for AMD-LU plans) by the whole CTA; w is an
// n-vector of scratch.  Level-synchronous, a thread per row.  Each row
// applies its updates in the order the reference's column-oriented sweeps
// reach it: forward columns ascending; backward ascending for Markowitz
// (row dot product, solve.cpp:30-44), descending for AMD-LU.  Begins and ends
// with __syncthreads().
__device__ inline void cta_solve(const PlanDesc& pd, const int32_t* __restrict__ pool,
                                 const double* __restrict__ lu, double* __restrict__ x,
                                 double* __restrict__ w) {
    const int32_t n = pd.n;
    const bool amd = pd.kind == kPlanAmdLu;
    const int32_t* perm_row = pool + pd.off[PA_perm_row];
    const int32_t* perm_col = pool + pd.off[PA_perm_col];
    const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
    __syncthreads();
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) w[i] = x[perm_row[i]];
    __syncthreads();
    {   // forward: L with the reciprocal pivot, row-oriented gather
        const int32_t* lp = pool + pd.off[PA_lrow_ptr];
        const int32_t* lpos = pool + pd.off[PA_lrow_pos];
        const int32_t* lcol = pool + pd.off[PA_lrow_col];
        const int32_t* lev_ptr = pool + pd.off[PA_fwd_lev_ptr];
        const int32_t* lev = pool + pd.off[PA_fwd_lev];
        for (int32_t l = 0; l < pd.n_fwd_lev; ++l) {
            for (int32_t k = lev_ptr[l] + threadIdx.x; k < lev_ptr[l + 1]; k += blockDim.x) {
                const int32_t i = lev[k];
                double t = w[i];
                if (amd) {
                    for (int32_t e = lp[i]; e < lp[i + 1]; ++e)
                        t = lu_sub(t, lu_mul(lu[lpos[e]], w[lcol[e]]));
                    w[i] = t;
                    continue;
                }
                for (int32_t e = lp[i]; e < lp[i + 1]; ++e) {
                    const double xc = w[lcol[e]];
                    if (xc != 0.0) t = lu_sub(t, lu_mul(xc, lu[lpos[e]]));
                }
                w[i] = (t != 0.0) ? lu_mul(t, lu[diag_pos[i]]) : t;
            }
            __syncthreads();
        }
    }
    {   // backward: Markowitz unit-diagonal U, row dot products in ascending
        // column order; AMD-LU columns descending, then the pivot division
        const int32_t* up = pool + pd.off[PA_urow_ptr];
        const int32_t* upos = pool + pd.off[PA_urow_pos];
        const int32_t* ucol = pool + pd.off[PA_urow_col];
        const int32_t* lev_ptr = pool + pd.off[PA_bwd_lev_ptr];
        const int32_t* lev = pool + pd.off[PA_bwd_lev];
        for (int32_t l = 0; l < pd.n_bwd_lev; ++l) {
            for (int32_t k = lev_ptr[l] + threadIdx.x; k < lev_ptr[l + 1]; k += blockDim.x) {
                const int32_t i = lev[k];
                double t = w[i];
                if (amd) {
                    for (int32_t e = up[i + 1] - 1; e >= up[i]; --e)
                        t = lu_sub(t, lu_mul(lu[upos[e]], w[ucol[e]]));
                    w[i] = __ddiv_rn(t, lu[diag_pos[i]]);
                    continue;
                }
                for (int32_t e = up[i]; e < up[i + 1]; ++e)
                    t = lu_sub(t, lu_mul(lu[upos[e]], w[ucol[e]]));
                w[i] = t;
            }
            __syncthreads();
        }
    }
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) x[perm_col[i]] = w[i];
    __syncthreads();
}

// cta_solve out of line, for kernels that reach it only for wide levels or where a
// bounded wait of their dataflow sweeps gave up.
static __device__ __noinline__ void cta_solve_levels(const PlanDesc& pd,
                                                     const int32_t* __restrict__ pool,
                                                     const double* __restrict__ lu,
                                                     double* __restrict__ x,
                                                     double* __restrict__ w) {
    cta_solve(pd, pool, lu, x, w);
}

// Dynamic shared memory of a Newton kernel launch: the LU scratch (flow or
// small path) followed by an optional stage for instance workspaces, capped
// so that two CTAs still fit on an SM.
constexpr size_t kStageCapBytes = 100 * 1024;
// lens: the instances' staged doubles, ascending.  The stage holds the largest
// instance that fits, provided that half of the batch does: shared memory that
// few instances use is better left to L1 (a batch of meshes too large for the
// stage ran 1.4 times slower with the room reserved for it).
inline size_t stage_bytes_for(size_t scratch_bytes, const int64_t* lens, int count) {
    if (scratch_bytes >= kStageCapBytes || count <= 0) return 0;
    const int64_t room = static_cast<int64_t>((kStageCapBytes - scratch_bytes) / sizeof(double));
    int fit = 0;
    while (fit < count && lens[fit] <= room) ++fit;
    return 2 * fit >= count ? sizeof(double) * static_cast<size_t>(lens[fit - 1]) : 0;
}

// Level programs.  A small sparse factor (an inverter chain, a BSIM4v7 ring, an
// interconnect tree: a few updates per unknown) is bound by its longest chain
// of dependent operations, not by their number, and on one warp alone by the
// instructions between two links of the chain.  Column after column, every
// link paid for the index loads, branches and barriers of everything beside
// it.  The host therefore schedules single LU entries and sweep rows into
// steps (longest remaining chain first, up to 32 independent ones a step;
// long sums in pieces, which run as their operands become ready), and one warp
// runs the steps, a lane per entry, with values and program in shared memory:
// a step is one batch of loads by precomputed byte offsets, two terms, a store
// and a warp barrier, without a branch (a reciprocal aside); the next step's
// words are already in registers.  U entries stay unscaled and are multiplied
// by their pivot's reciprocal where they are used, so a column waits for one
// step per pivot before it, and the forward sweep is part of the factor's
// steps (a right-hand side is one more column).
// Measured on a B200 at 1965 MHz: refactor and solve of the 32-stage inverter
// chain 77,000 -> 17,800 cycles a Newton iteration (the steps 12,500 of them);
// a pass of one transient of it (0.3 ns) 50.3 -> 25.0 ms, of 300 BSIM4v7 ring +
// NAND instances (0.06 ns) 224 -> 103 ms, of transient and adjoint of 64
// 500-node trees (0.1 ns) 119 -> 34.5 ms, all in CTAs of 512 threads.
// Every entry applies its updates in the order of the column-wise refactor,
// with the same rounded operations, so all values are bit-identical.
// The space: pd.nnz_lu LU values, the vector (pd.n), the unscaled pivots (pd.n),
// 0.0, 1.0, at the start of the dynamic shared memory.
__device__ __forceinline__ double* level_space() {
    extern __shared__ __align__(16) double smem[];
    return smem;
}

// Whether an instance runs its level program: it has one, in shared memory
// (stage_plan), and the kernel's scratch holds its space.
__device__ __forceinline__ bool level_ready(const PlanDesc& pd, int smem_doubles) {
    return pd.lp_at != nullptr && pd.nnz_lu + 2 * pd.n + 2 <= smem_doubles;
}

enum LevelSection : int { kLevelFactor = 0, kLevelBackward, kLevelOverU, kLevelOverL };

// The program's words do not change, so these loads may move freely; kPinned
// keeps them where they stand.  Pinned before a step's arithmetic they are 25 %
// faster in the short steps of the sweeps and 10 % slower in the factor's.
template <bool kPinned>
__device__ __forceinline__ uint32_t lds32(uint32_t at) {
    uint32_t v;
    if constexpr (kPinned) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at));
    else asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at));
    return v;
}

template <bool kPinned>
__device__ __forceinline__ uint2 lds64(uint32_t at) {
    uint2 v;
    if constexpr (kPinned)
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(at));
    else asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(at));
    return v;
}

template <bool kPinned>
__device__ __forceinline__ uint4 lds128(uint32_t at) {
    uint4 v;
    if constexpr (kPinned)
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "r"(at));
    else
        asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
            : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
            : "r"(at));
    return v;
}

// Steps first .. end - 1 (of section kSection) by one whole warp.  Ends with
// __syncwarp().
template <int kSection>
__device__ __forceinline__ void level_steps(const PlanDesc& pd, int32_t first, int32_t end) {
    if (first >= end) return;
    constexpr bool kPinned = kSection != kLevelFactor;
    char* const V = reinterpret_cast<char*>(level_space());
    auto val = [&](uint32_t off) -> double& { return *reinterpret_cast<double*>(V + off); };
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t lp = static_cast<uint32_t>(__cvta_generic_to_shared(pd.lp_at));
    uint32_t at = lp + sizeof(LevelStep) * first;
    const uint32_t last = lp + sizeof(LevelStep) * (end - 1);
    static_assert(kLevelTerms == 2 && sizeof(LevelStep) == 16, "the loads below");
    // idle lanes repeat the step's last entry and do not store
    uint4 d = lds128<kPinned>(at);
    uint32_t mine = min(lane, d.z);
    uint32_t ent = lds32<kPinned>(lp + d.x + 4 * mine);
    uint2 t0 = lds64<kPinned>(lp + d.y + 8 * mine);
    uint2 t1 = lds64<kPinned>(lp + d.y + 8 * (mine + d.z + 1));
    uint4 dn = lds128<kPinned>(min(at + 16, last));
    for (; at <= last; at += 16) {
        const double a0 = val(t0.x & 0xffffu), s0 = val(t0.x >> 16), b0 = val(t0.y);
        const double a1 = val(t1.x & 0xffffu), s1 = val(t1.x >> 16), b1 = val(t1.y);
        double t = val(ent & 0xfff8u);
        const double f = (kSection == kLevelBackward || kSection == kLevelOverL) ? val(ent >> 16)
                                                                                 : 1.0;
        // the next step's entry and terms, and the bounds of the one after
        const uint32_t nmine = min(lane, dn.z);
        const uint32_t nent = lds32<kPinned>(lp + dn.x + 4 * nmine);
        const uint2 n0 = lds64<kPinned>(lp + dn.y + 8 * nmine);
        const uint2 n1 = lds64<kPinned>(lp + dn.y + 8 * (nmine + dn.z + 1));
        const uint4 dnn = lds128<kPinned>(min(at + 32, last));
        const bool skip = (ent & kLevelSkip) != 0;
        // a term that is left out subtracts +0.0, which keeps t
        auto term = [&](double a, double s, double b) {
            const double u = lu_mul(a, s);
            const double v = lu_mul(u, b);
            if (kSection == kLevelFactor) return (skip && (a == 0.0 || u == 0.0)) ? 0.0 : v;
            if (kSection == kLevelOverU) return b == 0.0 ? 0.0 : v;
            return v;
        };
        if (kSection == kLevelBackward) {
            const double u = lu_mul(t, f);
            t = t == 0.0 ? t : u;
        }
        t = lu_sub(t, term(a0, s0, b0));
        t = lu_sub(t, term(a1, s1, b1));
        const bool live = lane <= d.z;
        double res = kSection == kLevelOverL ? lu_mul(t, f) : t;
        if (kSection == kLevelFactor && d.w != 0) {
            const bool pivot = (ent & kLevelPivot) != 0;
            const double r = __drcp_rn(t);
            if (pivot) res = r;
            if (live && pivot) val(ent >> 16) = t;
        }
        if (live) val(ent & 0xfff8u) = res;
        __syncwarp();
        d = dn;
        dn = dnn;
        mine = nmine;
        ent = nent;
        t0 = n0;
        t1 = n1;
    }
}

// Refactor a (through lu_src, diag_gmin added) into the level space and, when
// x is given and the factor is accepted, x <- A^{-1} x.  check_pivots as in
// cta_refactor_flow for Markowitz plans.  Begins and ends with __syncthreads().
static __device__ __noinline__ RefactorResult cta_level_factor(
    const PlanDesc& pd, const int32_t* __restrict__ pool, const double* __restrict__ a,
    double* __restrict__ x, double diag_gmin, int check_pivots, double rel_threshold) {
    const int32_t n = pd.n, nlu = pd.nnz_lu;
    const int32_t* lp = pd.lp_at;
    double* V = level_space();
    const uint16_t* src = reinterpret_cast<const uint16_t*>(lp + pd.lp_src);
    const uint16_t* perm = reinterpret_cast<const uint16_t*>(lp + pd.lp_perm);
    double* z = V + nlu;
    const double* pivots = z + n;
    __shared__ int32_t s_fail_step;
    __syncthreads();
    for (int32_t q = threadIdx.x; q < nlu; q += blockDim.x)
        V[q] = src[q] != 0xffffu ? a[src[q]] : 0.0;
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) z[i] = x ? x[perm[i]] : 0.0;
    if (threadIdx.x == 0) {
        s_fail_step = INT32_MAX;
        z[2 * n] = 0.0;
        z[2 * n + 1] = 1.0;
    }
    if (diag_gmin != 0.0) {
        const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
        __syncthreads();
        for (int32_t j = threadIdx.x; j < n; j += blockDim.x)
            V[diag_pos[j]] = __dadd_rn(V[diag_pos[j]], diag_gmin);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        // with the backward sweep where a solution is wanted; a rejected
        // factor's solution is computed too and dropped below
        level_steps<kLevelFactor>(pd, 0, pd.lp_steps[0]);
        if (x) level_steps<kLevelBackward>(pd, pd.lp_steps[0], pd.lp_steps[1]);
    }
    __syncthreads();
    if (check_pivots == kCheckNumeric) {
        const int32_t* col_ptr = pool + pd.off[PA_col_ptr];
        const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
        for (int32_t j = threadIdx.x; j < n; j += blockDim.x) {
            double largest = 0.0;
            for (int32_t q = diag_pos[j] + 1; q < col_ptr[j + 1]; ++q)
                largest = fmax(largest, fabs(V[q]));
            if (!(largest * rel_threshold < fabs(pivots[j]))) atomicMin(&s_fail_step, j);
        }
    } else {
        for (int32_t j = threadIdx.x; j < n; j += blockDim.x)
            if (pivots[j] == 0.0) atomicMin(&s_fail_step, j);
    }
    __syncthreads();
    RefactorResult res{kStatusOk, -1};
    if (s_fail_step != INT32_MAX) {
        res.code = check_pivots == kCheckNumeric ? kStatusReorder : kStatusSingular;
        res.step = s_fail_step;
    } else if (x) {
        for (int32_t i = threadIdx.x; i < n; i += blockDim.x) x[perm[n + i]] = z[i];
    }
    __syncthreads();
    return res;
}

// x <- A^{-T} x from the factor cta_level_factor left in the level space.
// Begins and ends with __syncthreads().
static __device__ __noinline__ void cta_level_solve_transposed(const PlanDesc& pd,
                                                               double* __restrict__ x) {
    const int32_t n = pd.n;
    const uint16_t* perm = reinterpret_cast<const uint16_t*>(pd.lp_at + pd.lp_perm);
    double* z = level_space() + pd.nnz_lu;
    __syncthreads();
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) z[i] = x[perm[n + i]];
    __syncthreads();
    if (threadIdx.x < 32) {
        level_steps<kLevelOverU>(pd, pd.lp_steps[1], pd.lp_steps[2]);
        level_steps<kLevelOverL>(pd, pd.lp_steps[2], pd.lp_steps[3]);
    }
    __syncthreads();
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) x[perm[i]] = z[i];
    __syncthreads();
}

// Small instances without a level program (AMD-LU plans, or a factor denser
// than the program's bounds): the LU in shared memory, one column after another
// on warp 0.  Every column's A values are scattered by the whole CTA before
// the elimination starts, U entries whose L(:, r) is short are applied by
// lane 0 alone with no warp barrier, longer ones by the warp, and the sweeps
// run row after row on lane 0 in pivot order.  Same operations in the same
// order per entry as cta_refactor_flow / cta_solve_flow, so the values are
// bit-identical.  lu_s: pd.nnz_lu doubles; w_s: pd.n.

// U entries whose L(:, r) has at most this many rows are applied by lane 0
// alone; longer ones by the whole warp.
constexpr int kSmallSerialRows = 4;

// Refactor into lu_s (and lu, written back at the end).  Begins and ends with
// __syncthreads().
static __device__ __noinline__ RefactorResult cta_refactor_small(
    const PlanDesc& pd, const int32_t* __restrict__ pool, const double* __restrict__ a,
    double* __restrict__ lu, double diag_gmin, int check_pivots, double rel_threshold,
    double* lu_s) {
    const int32_t n = pd.n;
    const int32_t* col_ptr = pool + pd.off[PA_col_ptr];
    const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
    const int32_t* lu_src = pool + pd.off[PA_lu_src];
    const int32_t* upd_dst = pool + pd.off[PA_upd_dst];
    const int32_t map16 = pd.map16;
    const int4* umeta = reinterpret_cast<const int4*>(pool + pd.off[PA_umeta]);
    const bool amd = pd.kind == kPlanAmdLu;
    const int32_t* piv_rank = pool + pd.off[PA_piv_rank];
    const int32_t* gmin_pos = pool + pd.off[PA_gmin_pos];
    const int lane = threadIdx.x & 31;
    __shared__ int32_t s_fail_step, s_fail_code;
    __syncthreads();
    // A values of every column at once (the scatter does not depend on the
    // elimination), then diag_gmin on each column's gmin row.
    for (int32_t t = threadIdx.x; t < pd.nnz_lu; t += blockDim.x) {
        const int32_t src = lu_src[t];
        lu_s[t] = (src >= 0) ? a[src] : 0.0;
    }
    if (diag_gmin != 0.0) {
        __syncthreads();
        for (int32_t j = threadIdx.x; j < n; j += blockDim.x) {
            const int32_t gp = amd ? gmin_pos[j] : diag_pos[j] - col_ptr[j];
            if (gp >= 0) lu_s[col_ptr[j] + gp] = __dadd_rn(lu_s[col_ptr[j] + gp], diag_gmin);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) s_fail_step = INT32_MAX;
    if (threadIdx.x < 32 && n > 0) {
        int32_t fail_step = INT32_MAX, fail_code = kStatusOk;
        bool any_growth = false;
        const bool lane0_pivots = !amd && check_pivots != kCheckNumeric;
        int32_t nc0 = col_ptr[0], nc1 = col_ptr[1], ndp = diag_pos[0];
        for (int32_t j = 0; j < n; ++j) {
            const int32_t c0 = nc0, len = nc1 - nc0, dj = ndp - nc0;
            if (j + 1 < n) {  // the next column's bounds, off the dependency chain
                nc0 = nc1;
                nc1 = col_ptr[j + 2];
                ndp = diag_pos[j + 1];
            }
            double colmax = 0.0;  // AMD-LU: largest |U(r, j)| applied (lane 0)
            for (int32_t q = 0; q < dj; ++q) {
                const int4 m = u_entry(umeta, c0 + q);  // r, diag_pos[r], |L(:, r)|, upd_start
                if (m.z <= kSmallSerialRows) {
                    if (lane == 0) {
                        const double u = amd ? lu_s[c0 + q] : lu_mul(lu_s[c0 + q], lu_s[m.y]);
                        colmax = fmax(colmax, fabs(u));
                        lu_s[c0 + q] = u;
                        for (int32_t t = 0; t < m.z; ++t) {
                            const int32_t d = c0 + upd_at(upd_dst, map16, m.w + t);
                            lu_s[d] = lu_sub(lu_s[d], lu_mul(u, lu_s[m.y + 1 + t]));
                        }
                    }
                } else {
                    __syncwarp();  // lane 0's serial updates visible to the warp
                    double u = 0.0;
                    if (lane == 0) {
                        u = amd ? lu_s[c0 + q] : lu_mul(lu_s[c0 + q], lu_s[m.y]);
                        colmax = fmax(colmax, fabs(u));
                        lu_s[c0 + q] = u;
                    }
                    u = __shfl_sync(0xffffffffu, u, 0);
                    for (int32_t t = lane; t < m.z; t += 32) {
                        const int32_t d = c0 + upd_at(upd_dst, map16, m.w + t);
                        lu_s[d] = lu_sub(lu_s[d], lu_mul(u, lu_s[m.y + 1 + t]));
                    }
                    __syncwarp();
                }
            }
            int32_t code = kStatusOk;
            if (lane0_pivots) {
                // refactorize(): a zero pivot fails; the reciprocal is stored.
                if (lane == 0) {
                    const double piv = lu_s[c0 + dj];
                    code = (piv == 0.0) ? kStatusSingular : kStatusOk;
                    lu_s[c0 + dj] = __drcp_rn(piv);
                }
            } else {
                __syncwarp();
                const double piv = lu_s[c0 + dj];
                if (amd) {
                    colmax = __shfl_sync(0xffffffffu, colmax, 0);
                    const AmdColumn v = amd_column_status(lu_s + c0, dj, len, colmax,
                                                          check_pivots, piv_rank[j], gmin_pos[j],
                                                          lane);
                    code = v.code;
                    any_growth = any_growth || v.growth_fail;
                    for (int32_t t = dj + 1 + lane; t < len; t += 32)
                        lu_s[c0 + t] = __ddiv_rn(lu_s[c0 + t], piv);
                } else {
                    double largest = 0.0;
                    for (int32_t t = dj + 1 + lane; t < len; t += 32)
                        largest = fmax(largest, fabs(lu_s[c0 + t]));
                    largest = warp_max(largest);
                    code = !(largest * rel_threshold < fabs(piv)) ? kStatusReorder : kStatusOk;
                    __syncwarp();
                    if (lane == 0) lu_s[c0 + dj] = __drcp_rn(piv);
                }
                __syncwarp();
            }
            if (lane == 0 && code != kStatusOk && j < fail_step) {
                fail_step = j;
                fail_code = code;
            }
        }
        if (amd && !amd_verdict_counts(check_pivots, any_growth)) fail_step = INT32_MAX;
        if (lane == 0) {
            s_fail_step = fail_step;
            s_fail_code = fail_code;
        }
    }
    __syncthreads();
    for (int32_t k = threadIdx.x; k < pd.nnz_lu; k += blockDim.x) lu[k] = lu_s[k];
    RefactorResult res;
    res.step = s_fail_step == INT32_MAX ? -1 : s_fail_step;
    res.code = s_fail_step == INT32_MAX ? kStatusOk : s_fail_code;
    __syncthreads();
    return res;
}

// x <- A^{-1} x from the LU in lu_s: lane 0, row after row in pivot order
// (forward: ascending, backward: descending), each row's entries in the
// order of the level-scheduled sweeps.  The next row's bounds and pivot are
// fetched while the current row is computed, so only the values carry the
// dependency from row to row.  Begins and ends with __syncthreads().
static __device__ __noinline__ void cta_solve_small(const PlanDesc& pd,
                                                    const int32_t* __restrict__ pool,
                                                    const double* __restrict__ lu_s,
                                                    double* __restrict__ x,
                                                    double* __restrict__ w) {
    const int32_t n = pd.n;
    const int32_t* perm_row = pool + pd.off[PA_perm_row];
    const int32_t* perm_col = pool + pd.off[PA_perm_col];
    const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
    const bool amd = pd.kind == kPlanAmdLu;
    __syncthreads();
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) w[i] = x[perm_row[i]];
    __syncthreads();
    if (threadIdx.x == 0 && n > 0) {
        {   // forward: L (Markowitz: skip zero operands, then the reciprocal pivot)
            const int32_t* lp = pool + pd.off[PA_lrow_ptr];
            const int32_t* lpos = pool + pd.off[PA_lrow_pos];
            const int32_t* lcol = pool + pd.off[PA_lrow_col];
            int32_t e = lp[0], e1 = lp[1];
            double piv = amd ? 0.0 : lu_s[diag_pos[0]];
            for (int32_t i = 0; i < n; ++i) {
                const bool more = i + 1 < n;
                const int32_t e1n = more ? lp[i + 2] : 0;
                const double pivn = (more && !amd) ? lu_s[diag_pos[i + 1]] : 0.0;
                double t = w[i];
                if (amd) {
                    for (; e < e1; ++e) t = lu_sub(t, lu_mul(lu_s[lpos[e]], w[lcol[e]]));
                    w[i] = t;
                } else {
                    for (; e < e1; ++e) {
                        const double l = lu_s[lpos[e]];
                        const double xc = w[lcol[e]];
                        if (xc != 0.0) t = lu_sub(t, lu_mul(xc, l));
                    }
                    w[i] = (t != 0.0) ? lu_mul(t, piv) : t;
                }
                e1 = e1n;
                piv = pivn;
            }
        }
        {   // backward: U row dot products (AMD-LU: columns descending, then
            // the pivot division)
            const int32_t* up = pool + pd.off[PA_urow_ptr];
            const int32_t* upos = pool + pd.off[PA_urow_pos];
            const int32_t* ucol = pool + pd.off[PA_urow_col];
            int32_t e0 = up[n - 1], e1 = up[n];
            double piv = amd ? lu_s[diag_pos[n - 1]] : 0.0;
            for (int32_t i = n - 1; i >= 0; --i) {
                const bool more = i > 0;
                const int32_t e0n = more ? up[i - 1] : 0;
                const double pivn = (more && amd) ? lu_s[diag_pos[i - 1]] : 0.0;
                double t = w[i];
                if (amd) {
                    for (int32_t e = e1 - 1; e >= e0; --e)
                        t = lu_sub(t, lu_mul(lu_s[upos[e]], w[ucol[e]]));
                    w[i] = __ddiv_rn(t, piv);
                } else {
                    for (int32_t e = e0; e < e1; ++e)
                        t = lu_sub(t, lu_mul(lu_s[upos[e]], w[ucol[e]]));
                    w[i] = t;
                }
                e1 = e0;
                e0 = e0n;
                piv = pivn;
            }
        }
    }
    __syncthreads();
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) x[perm_col[i]] = w[i];
    __syncthreads();
}

// Shared memory of the dataflow solve: the n-vector and n completion flags.
__host__ __device__ inline size_t flow_solve_smem_bytes(int n) {
    return (sizeof(double) + sizeof(int32_t)) * static_cast<size_t>(n);
}

// One triangular sweep of the dataflow solves: row i of `order` (a level
// order) becomes t = w[i] - sum val * w[idx] over its entries, one rounded
// multiply and subtract at a time in stored order, then
//   kFinalMul        t * pivot value
//   kFinalMulNonzero t * pivot value unless t is zero (SparseMatrix::solve's
//                    forward sweep, solve.cpp:14-27)
//   kFinalDiv        t / pivot value
// kSkipZero leaves out entries whose operand is zero (their product is
// replaced by +0.0, which subtracts to the same value); kDescending runs a
// row's entries from the last to the first.
enum SweepFinal : int { kFinalNone = 0, kFinalMul, kFinalMulNonzero, kFinalDiv };

struct SweepRows {
    const int32_t* order;    // rows, level after level
    const int32_t* beg;      // row i's entries: beg[i] + beg_add .. end[i] - 1
    const int32_t* end;
    int32_t beg_add;
    const int32_t* idx;
    const double* val;
    const int32_t* piv_pos;  // position of row i's pivot in piv
    const double* piv;
};

// What bounds a sweep is the chain of rows that wait for one another and, in
// front of it, the index and value loads of each row; its bytes and
// operations are a few microseconds' worth.  So a warp takes a whole row: its
// lanes load 32 entries and look at their 32 flags at once, the products are
// formed in parallel as their operands become final, and only the
// subtractions run one after another (in every lane, from shuffles).  A row of
// the dense trailing block has all but its last entries summed by the time
// its predecessor is done.  The row numbers, bounds and pivots of a warp's
// next 32 rows come in with one load each, and the next row's first 32
// entries are in flight while a row waits.  A thread per row, walking its
// entries and their flags alone, spent 2.0 ms on the two sweeps of a 2305-
// unknown mesh where this takes 0.48 ms (B200, 1965 MHz).
// Rows are dealt to warps in level order, and a row waits only on rows at
// earlier positions, so every wait ends; waits are bounded all the same
// (c_wait_limit polls in vain within 32 entries, then the warp runs on with
// what it has and the sweep reports false).
template <int kFinal, bool kSkipZero, bool kDescending>
__device__ __forceinline__ bool sweep_rows(const SweepRows& s, int32_t n, double* w,
                                           volatile int32_t* done, int32_t target) {
    const int lane = threadIdx.x & 31;
    const int32_t warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int limit = c_wait_limit;
    bool ok = true;
    for (int32_t base = warp; base < n; base += 32 * nwarps) {
        const int32_t at = base + lane * nwarps;
        int32_t row = 0, beg = 0, end = 0;
        double piv = 0.0;
        if (at < n) {
            row = s.order[at];
            beg = s.beg[row] + s.beg_add;
            end = s.end[row];
            if (kFinal != kFinalNone) piv = s.piv[s.piv_pos[row]];
        }
        const int32_t rows = min(32, (n - base + nwarps - 1) / nwarps);
        // entries m0 .. m0 + 31 of the row e0 .. e1 - 1, in the sweep's order
        auto load = [&](int32_t e0, int32_t e1, int32_t m0, int32_t& c, double& v) {
            const int32_t e = kDescending ? e1 - 1 - m0 - lane : e0 + m0 + lane;
            const bool in = kDescending ? e >= e0 : e < e1;
            c = in ? s.idx[e] : 0;
            v = in ? s.val[e] : 0.0;
        };
        int32_t e0 = __shfl_sync(0xffffffffu, beg, 0), e1 = __shfl_sync(0xffffffffu, end, 0);
        int32_t c;
        double v;
        load(e0, e1, 0, c, v);
        for (int32_t r = 0; r < rows; ++r) {
            const int32_t i = __shfl_sync(0xffffffffu, row, r);
            const int32_t ne0 = __shfl_sync(0xffffffffu, beg, (r + 1) & 31);
            const int32_t ne1 = __shfl_sync(0xffffffffu, end, (r + 1) & 31);
            int32_t nc = 0;
            double nv = 0.0;
            if (r + 1 < rows) load(ne0, ne1, 0, nc, nv);
            const int32_t len = e1 - e0;
            double t = w[i];
            for (int32_t m0 = 0; m0 < len; m0 += 32) {
                int32_t cc = c;
                double vv = v;
                if (m0 + 32 < len) load(e0, e1, m0 + 32, c, v);
                const int32_t m = min(32, len - m0);
                bool ready = lane >= m;
                double p = 0.0;
                int32_t k = 0;  // entries of this chunk subtracted so far
                int spins = 0;
                while (k < m) {
                    if (!ready && (flag_acquire(done + cc) >= target || !ok)) {
                        ready = true;
                        const double x = w[cc];
                        p = (!kSkipZero || x != 0.0) ? lu_mul(vv, x) : 0.0;
                    }
                    const unsigned open = __ballot_sync(0xffffffffu, !ready);
                    const int32_t stop = open ? min(m, __ffs(open) - 1) : m;
                    if (stop == k) {
                        if (++spins > limit) ok = false;
                        else if (spins > 4) __nanosleep(20);
                        continue;
                    }
                    for (; k + 4 <= stop; k += 4) {
                        const double p0 = __shfl_sync(0xffffffffu, p, k);
                        const double p1 = __shfl_sync(0xffffffffu, p, k + 1);
                        const double p2 = __shfl_sync(0xffffffffu, p, k + 2);
                        const double p3 = __shfl_sync(0xffffffffu, p, k + 3);
                        t = lu_sub(lu_sub(lu_sub(lu_sub(t, p0), p1), p2), p3);
                    }
                    for (; k < stop; ++k) t = lu_sub(t, __shfl_sync(0xffffffffu, p, k));
                }
            }
            if (kFinal != kFinalNone) {
                const double d = __shfl_sync(0xffffffffu, piv, r);
                if (kFinal == kFinalDiv) t = __ddiv_rn(t, d);
                else if (kFinal == kFinalMul || t != 0.0) t = lu_mul(t, d);
            }
            if (lane == 0) {
                w[i] = t;
                flag_release(done + i, target);
            }
            e0 = ne0;
            e1 = ne1;
            c = nc;
            v = nv;
        }
    }
    return ok;
}

// The two sweeps of a dataflow solve with the vector and its flags in shared
// memory (flow_solve_smem_bytes): gather through perm_in, first sweep (flags
// to 1), second sweep (flags to 2), scatter through perm_out.  Returns false,
// with x as it was, if a bounded wait gave up.  Begins and ends with
// __syncthreads().
template <class First, class Second>
__device__ __forceinline__ bool sweep_pair(int32_t n, const int32_t* perm_in,
                                           const int32_t* perm_out, double* __restrict__ x,
                                           double* smem, First first, Second second) {
    double* w = smem;
    volatile int32_t* done = reinterpret_cast<volatile int32_t*>(smem + n);
    __shared__ int32_t s_ok;
    __syncthreads();
    if (threadIdx.x == 0) s_ok = 1;
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) {
        w[i] = x[perm_in[i]];
        done[i] = 0;
    }
    __syncthreads();
    bool ok = first(w, done);
    __syncthreads();
    ok = second(w, done) && ok;
    if (!ok) s_ok = 0;
    __syncthreads();
    const bool all_ok = (s_ok != 0);
    if (all_ok)
        for (int32_t i = threadIdx.x; i < n; i += blockDim.x) x[perm_out[i]] = w[i];
    __syncthreads();
    return all_ok;
}

// x <- A^{-1} x (SparseMatrix::solve) by the whole CTA: L forward with the
// reciprocal pivot, U backward (AMD-LU: unit L, then U columns descending and
// the pivot division), on the row-major copies the refactor wrote.  Same
// arithmetic, in the same order per row, as cta_solve.  any_wide: false where no
// plan of the launch has wide levels, which saves the look at the plan (0.2 of a
// 37-unknown refactor and solve's 34.7 us).
static __device__ __noinline__ bool cta_solve_flow(const PlanDesc& pd, const int32_t* __restrict__ pool,
                                      const double* __restrict__ lu,
                                      const double* __restrict__ lrows,
                                      const double* __restrict__ urows, double* __restrict__ x,
                                      double* smem, bool any_wide = true) {
    if (any_wide && wide_levels(pd)) {
        cta_solve_levels(pd, pool, lu, x, smem);
        return true;
    }
    const int32_t n = pd.n;
    const bool amd = pd.kind == kPlanAmdLu;
    const int32_t* lp = pool + pd.off[PA_lrow_ptr];
    const int32_t* up = pool + pd.off[PA_urow_ptr];
    const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
    const SweepRows fwd{pool + pd.off[PA_fwd_lev], lp, lp + 1, 0, pool + pd.off[PA_lrow_col],
                        lrows, diag_pos, lu};
    const SweepRows bwd{pool + pd.off[PA_bwd_lev], up, up + 1, 0, pool + pd.off[PA_urow_col],
                        urows, diag_pos, lu};
    return sweep_pair(
        n, pool + pd.off[PA_perm_row], pool + pd.off[PA_perm_col], x, smem,
        [&](double* w, volatile int32_t* done) {
            return amd ? sweep_rows<kFinalNone, false, false>(fwd, n, w, done, 1)
                       : sweep_rows<kFinalMulNonzero, true, false>(fwd, n, w, done, 1);
        },
        [&](double* w, volatile int32_t* done) {
            return amd ? sweep_rows<kFinalDiv, false, true>(bwd, n, w, done, 2)
                       : sweep_rows<kFinalNone, false, false>(bwd, n, w, done, 2);
        });
}

// x <- A^{-T} x (SparseMatrix::solve_transposed) by the whole CTA on the
// column-major factors: U^T forward (zero operands left out), then L^T with the
// reciprocal pivot (AMD-LU: A^T = Q U^T L^T P, U^T with the pivot division, then
// unit L^T).  Same arithmetic, in the same order per row, as
// cta_solve_transposed: 592 transposed solves of 145 to 577 unknowns took
// 0.67 ms with a thread per row and a barrier per level, 0.36 ms here.  If a
// bounded wait gave up, those sweeps, which wait for nothing but barriers, give
// the result (the vector in smem).
static __device__ __noinline__ void cta_solve_transposed_levels(const PlanDesc& pd,
                                                                const int32_t* __restrict__ pool,
                                                                const double* __restrict__ lu,
                                                                double* __restrict__ x,
                                                                double* __restrict__ w);
static __device__ __noinline__ void cta_solve_transposed_flow(const PlanDesc& pd,
                                                              const int32_t* __restrict__ pool,
                                                              const double* __restrict__ lu,
                                                              double* __restrict__ x,
                                                              double* smem,
                                                              bool any_wide = true) {
    if (any_wide && wide_levels(pd)) {
        cta_solve_transposed_levels(pd, pool, lu, x, smem);
        return;
    }
    const int32_t n = pd.n;
    const bool amd = pd.kind == kPlanAmdLu;
    const int32_t* cp = pool + pd.off[PA_col_ptr];
    const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
    const int32_t* row_idx = pool + pd.off[PA_row_idx];
    const SweepRows over_u{pool + pd.off[PA_col_lev], cp, diag_pos, 0, row_idx, lu, diag_pos, lu};
    const SweepRows over_l{pool + pd.off[PA_tbw_lev], diag_pos, cp + 1, 1, row_idx, lu, diag_pos, lu};
    const bool ok = sweep_pair(
        n, pool + pd.off[PA_perm_col], pool + pd.off[PA_perm_row], x, smem,
        [&](double* w, volatile int32_t* done) {
            return amd ? sweep_rows<kFinalDiv, true, false>(over_u, n, w, done, 1)
                       : sweep_rows<kFinalNone, true, false>(over_u, n, w, done, 1);
        },
        [&](double* w, volatile int32_t* done) {
            return amd ? sweep_rows<kFinalNone, false, false>(over_l, n, w, done, 2)
                       : sweep_rows<kFinalMul, false, false>(over_l, n, w, done, 2);
        });
    if (!ok) cta_solve_transposed_levels(pd, pool, lu, x, smem);
}

// The same level after level, a thread per row; w is an n-vector of scratch: for
// instances whose vector and flags exceed shared memory, and where a wait gave
// up.
// x <- A^{-T} x (SparseMatrix::solve_transposed) by the whole CTA.  AMD-LU
// plans (the reference's AmdLuSolver has no transposed solve) use
// A^T = Q U^T L^T P: U^T forward with the pivot division, then unit L^T.
__device__ inline void cta_solve_transposed(const PlanDesc& pd, const int32_t* __restrict__ pool,
                                            const double* __restrict__ lu, double* __restrict__ x,
                                            double* __restrict__ w) {
    const int32_t n = pd.n;
    const int32_t* perm_row = pool + pd.off[PA_perm_row];
    const int32_t* perm_col = pool + pd.off[PA_perm_col];
    const int32_t* col_ptr = pool + pd.off[PA_col_ptr];
    const int32_t* row_idx = pool + pd.off[PA_row_idx];
    const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
    const bool amd = pd.kind == kPlanAmdLu;
    __syncthreads();
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) w[i] = x[perm_col[i]];
    __syncthreads();
    {   // forward over U^T: column c gathers its U entries in stored order
        // (AMD-LU: then divides by the pivot)
        const int32_t* lev_ptr = pool + pd.off[PA_col_lev_ptr];
        const int32_t* lev = pool + pd.off[PA_col_lev];
        for (int32_t l = 0; l < pd.n_col_lev; ++l) {
            for (int32_t k = lev_ptr[l] + threadIdx.x; k < lev_ptr[l + 1]; k += blockDim.x) {
                const int32_t c = lev[k];
                double t = w[c];
                for (int32_t q = col_ptr[c]; q < diag_pos[c]; ++q) {
                    const double xr = w[row_idx[q]];
                    if (xr != 0.0) t = lu_sub(t, lu_mul(xr, lu[q]));
                }
                w[c] = amd ? __ddiv_rn(t, lu[diag_pos[c]]) : t;
            }
            __syncthreads();
        }
    }
    {   // backward over L^T (Markowitz: then the reciprocal pivot)
        const int32_t* lev_ptr = pool + pd.off[PA_tbw_lev_ptr];
        const int32_t* lev = pool + pd.off[PA_tbw_lev];
        for (int32_t l = 0; l < pd.n_tbw_lev; ++l) {
            for (int32_t k = lev_ptr[l] + threadIdx.x; k < lev_ptr[l + 1]; k += blockDim.x) {
                const int32_t i = lev[k];
                double t = w[i];
                for (int32_t q = diag_pos[i] + 1; q < col_ptr[i + 1]; ++q)
                    t = lu_sub(t, lu_mul(lu[q], w[row_idx[q]]));
                w[i] = amd ? t : lu_mul(t, lu[diag_pos[i]]);
            }
            __syncthreads();
        }
    }
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) x[perm_row[i]] = w[i];
    __syncthreads();
}

static __device__ __noinline__ void cta_solve_transposed_levels(const PlanDesc& pd,
                                                                const int32_t* __restrict__ pool,
                                                                const double* __restrict__ lu,
                                                                double* __restrict__ x,
                                                                double* __restrict__ w) {
    cta_solve_transposed(pd, pool, lu, x, w);
}

}  // namespace nsg
