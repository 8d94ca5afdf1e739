// Batched complex refactor and solve for AC sweeps: every instance of a batch
// (typically one frequency point of G + jwC, or one circuit) refactored with
// the fixed pivot order of the plan -- SparseMatrix::factor_complex
// (src/solver/factor.cpp:1054-1141) -- and swept -- solve_complex
// (src/solver/solve.cpp:49-100).  Values are interleaved (re, im) per matrix
// slot / LU position / unknown.  Every complex product keeps the reference's
// grouping (re = a*c - b*d, im = a*d + b*c, one rounding each), and every
// entry receives its updates in ascending pivot order, so the factors and
// solutions are bit-identical to the reference's under the same pivots.
#include "flow_shape.cuh"
#include "lu_cta.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

namespace nsg {

namespace {

constexpr int kCplxWarps = 8;
constexpr int kCplxThreads = kCplxWarps * 32;

// complex_ops::reciprocal (src/solver/element.hpp:42-54).
__device__ __forceinline__ void c_recip(double den_r, double den_i, double& out_r,
                                        double& out_i) {
    if ((den_r >= den_i && den_r > -den_i) || (den_r < den_i && den_r <= -den_i)) {
        const double r = __ddiv_rn(den_i, den_r);
        out_r = __ddiv_rn(1.0, __dadd_rn(den_r, __dmul_rn(r, den_i)));
        out_i = __dmul_rn(-r, out_r);
    } else {
        const double r = __ddiv_rn(den_r, den_i);
        out_i = __ddiv_rn(-1.0, __dadd_rn(den_i, __dmul_rn(r, den_r)));
        out_r = __dmul_rn(-r, out_i);
    }
}

// a*c - b*d and a*d + b*c with separately rounded products.
__device__ __forceinline__ double c_re(double a, double b, double c, double d) {
    return __dsub_rn(__dmul_rn(a, c), __dmul_rn(b, d));
}
__device__ __forceinline__ double c_im(double a, double b, double c, double d) {
    return __dadd_rn(__dmul_rn(a, d), __dmul_rn(b, c));
}

__device__ __forceinline__ double2 c_mul(double2 a, double2 b) {
    return make_double2(c_re(a.x, a.y, b.x, b.y), c_im(a.x, a.y, b.x, b.y));
}
__device__ __forceinline__ double2 c_msub(double2 t, double2 u, double2 l) {
    return make_double2(__dsub_rn(t.x, c_re(u.x, u.y, l.x, l.y)),
                        __dsub_rn(t.y, c_im(u.x, u.y, l.x, l.y)));
}
__device__ __forceinline__ double2 c_shfl(double2 v, int lane) {
    return make_double2(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane));
}
__device__ __forceinline__ bool c_zero(double2 v) { return v.x == 0.0 && v.y == 0.0; }

// The dataflow refactor of lu_cta.cuh (refactor_column, run_step) on complex
// values: a warp's column stays in a shared buffer, runs of kRun entries of
// equal structure are applied together, other entries load their operands
// kGroup at a time, and completion is published before anything else waits on
// the warp.  In place in global memory, an entry and a flag at a time, 150
// frequency points of a 1026-unknown mesh took 1.14 ms, here 0.51 ms.
template <int kThreads, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks)
complex_flow_refactor_kernel(const PlanDesc* __restrict__ plans, const int32_t* __restrict__ pool,
                             const InstDesc* __restrict__ insts, const double* __restrict__ A,
                             double* LU, int32_t* status, int colbuf) {
    extern __shared__ __align__(16) double2 cols[];
    __shared__ int32_t s_next, s_fail, s_timeout;
    const InstDesc id = insts[blockIdx.x];
    const PlanDesc& pd = plans[id.plan];
    const int32_t n = pd.n;
    const int32_t* col_ptr = pool + pd.off[PA_col_ptr];
    const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
    const int32_t* lu_src = pool + pd.off[PA_lu_src];
    const int32_t* upd_dst = pool + pd.off[PA_upd_dst];
    const int32_t map16 = pd.map16;
    const double* a = A + 2 * id.a_off;
    double2* lu = reinterpret_cast<double2*>(LU) + id.lu_off;
    const int lane = threadIdx.x & 31;
    double2* buf = cols + (threadIdx.x >> 5) * colbuf;
    volatile int32_t* done = reinterpret_cast<volatile int32_t*>(cols + (kThreads / 32) * colbuf);
    for (int32_t j = threadIdx.x; j < n; j += blockDim.x) done[j] = 0;
    if (threadIdx.x == 0) {
        s_next = 0;
        s_fail = 0x7fffffff;
        s_timeout = 0;
    }
    __syncthreads();
    const int limit = c_wait_limit;
    const double2 zero = make_double2(0.0, 0.0);
    for (;;) {
        int32_t j = 0;
        if (lane == 0) j = atomicAdd(&s_next, 1);
        j = __shfl_sync(0xffffffffu, j, 0);
        if (j >= n) break;
        const int32_t c0 = col_ptr[j];
        const int32_t len = col_ptr[j + 1] - c0;
        const int32_t dj = diag_pos[j] - c0;
        for (int32_t t = lane; t < len; t += 32) {
            const int32_t src = lu_src[c0 + t];
            buf[t] = src >= 0 ? make_double2(a[2 * src], a[2 * src + 1]) : zero;
        }
        __syncwarp();
        auto dest = [&](int32_t us, int32_t t) { return upd_at(upd_dst, map16, us + t); };
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
            if (q - base > 32 - kRunLanes && base + 32 < dj) window(q);
            const int32_t k0 = q - base;
            const int32_t ahead = min(min(kRunLanes, dj - q), 32 - k0);
            const int32_t src = __shfl_sync(0xffffffffu, meta.x, k0 + (lane & (kRunLanes - 1)));
            int32_t ready = 0;
            for (int spins = 0;;) {
                const bool open = lane < ahead && flag_acquire(done + src) == 0;
                const unsigned mask = __ballot_sync(0xffffffffu, open);
                ready = mask ? __ffs(mask) - 1 : ahead;
                if (ready > 0) break;
                if (++spins > limit) {
                    timed_out = true;
                    break;
                }
                __nanosleep(64);
            }
            if (timed_out) break;
            __syncwarp();
            const int32_t run = __ffs(~(chain >> k0));
            if (min(run, ready) >= kRun) {
                int32_t at[kRun];
#pragma unroll
                for (int i = 0; i < kRun; ++i) at[i] = __shfl_sync(0xffffffffu, meta.y, k0 + i);
                const int32_t cnt =
                    __shfl_sync(0xffffffffu, meta.z, k0 + kRun - 1) & 0x7fffffff;
                const int32_t us = __shfl_sync(0xffffffffu, meta.w, k0 + kRun - 1);
                const int32_t dp = __shfl_sync(0xffffffffu, meta.y, k0 + (lane & (kRun - 1)));
                double2 x = lane < kRun ? buf[q + lane] : zero;
                const double2 rd = lane < kRun ? lu[dp] : zero;
                double2 tri[kRun], l[kRun], u[kRun];
                int32_t d;
#pragma unroll
                for (int i = 0; i < kRun - 1; ++i)
                    tri[i] = (lane > i && lane < kRun) ? lu[at[i] + lane - i] : zero;
                auto load = [&](int32_t t) {
                    d = t < cnt ? dest(us, t) : 0;
#pragma unroll
                    for (int i = 0; i < kRun; ++i) l[i] = t < cnt ? lu[at[i] + (kRun - i) + t] : zero;
                };
                load(lane);
#pragma unroll
                for (int i = 0; i < kRun; ++i) {
                    const double2 v = c_mul(x, rd);
                    u[i] = c_shfl(v, i);
                    if (lane == i) x = v;
                    if (i < kRun - 1 && lane > i) x = c_msub(x, u[i], tri[i]);
                }
                if (lane < kRun) buf[q + lane] = x;
                for (int32_t t = lane; t < cnt + lane; t += 32) {
                    if (t >= 32) load(t);
                    if (t < cnt) {
                        double2 v = buf[d];
#pragma unroll
                        for (int i = 0; i < kRun; ++i) v = c_msub(v, u[i], l[i]);
                        buf[d] = v;
                    }
                }
                __syncwarp();
                q += kRun;
            } else {
                const int32_t count = min(kGroup, ready);
                int32_t l0[kGroup], cnt[kGroup], us[kGroup], dd[kGroup];
                double2 rd[kGroup], ll[kGroup];
#pragma unroll
                for (int g = 0; g < kGroup; ++g) {
                    const int32_t k = k0 + min(g, count - 1);
                    const int32_t dp = __shfl_sync(0xffffffffu, meta.y, k);
                    l0[g] = dp + 1;
                    cnt[g] = __shfl_sync(0xffffffffu, meta.z, k) & 0x7fffffff;
                    if (g >= count) cnt[g] = 0;
                    us[g] = __shfl_sync(0xffffffffu, meta.w, k);
                    rd[g] = lu[dp];
                    ll[g] = lane < cnt[g] ? lu[l0[g] + lane] : zero;
                    dd[g] = lane < cnt[g] ? dest(us[g], lane) : 0;
                }
#pragma unroll
                for (int g = 0; g < kGroup; ++g) {
                    if (g < count) {
                        const double2 u = c_mul(buf[q + g], rd[g]);
                        __syncwarp();
                        if (lane == 0) buf[q + g] = u;
                        if (lane < cnt[g]) buf[dd[g]] = c_msub(buf[dd[g]], u, ll[g]);
                        for (int32_t t = lane + 32; t < cnt[g]; t += 32) {
                            const int32_t d = dest(us[g], t);
                            buf[d] = c_msub(buf[d], u, lu[l0[g] + t]);
                        }
                        __syncwarp();
                    }
                }
                q += count;
            }
        }
        const double2 piv = buf[dj];
        const bool singular = __dadd_rn(fabs(piv.x), fabs(piv.y)) == 0.0;
        double2 inv = piv;
        if (!timed_out && !singular) c_recip(piv.x, piv.y, inv.x, inv.y);
        for (int32_t t = lane; t < len; t += 32) lu[c0 + t] = t == dj ? inv : buf[t];
        __syncwarp();
        if (lane == 0) {
            if (timed_out) s_timeout = 1;
            else if (singular) atomicMin(&s_fail, j);
            flag_release(done + j, 1);
        }
        __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x == 0)
        status[id.index] = s_timeout ? kStatusTimeout
                                     : (s_fail != 0x7fffffff ? kStatusSingular : kStatusOk);
}

// The row sweeps of lu_cta.cuh (sweep_rows) on complex values: a warp per row,
// 32 entries and flags at once, products in parallel, subtractions in order.
// kForward: L, entries with a zero operand left out, then the reciprocal pivot
// unless the row is zero; else U.  The factor is read through the plan's row
// positions (pos), the vector and the flags are in shared memory.  False if a
// bounded wait gave up.
template <bool kForward>
__device__ __forceinline__ bool c_sweep_rows(const int32_t* order, const int32_t* ptr,
                                             const int32_t* idx, const int32_t* pos,
                                             const int32_t* diag_pos, const double2* lu, int32_t n,
                                             double2* w, volatile int32_t* done, int32_t target) {
    const int lane = threadIdx.x & 31;
    const int32_t warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int limit = c_wait_limit;
    const double2 zero = make_double2(0.0, 0.0);
    bool ok = true;
    for (int32_t base = warp; base < n; base += 32 * nwarps) {
        const int32_t at = base + lane * nwarps;
        int32_t row = 0, beg = 0, end = 0;
        double2 piv = zero;
        if (at < n) {
            row = order[at];
            beg = ptr[row];
            end = ptr[row + 1];
            if (kForward) piv = lu[diag_pos[row]];
        }
        const int32_t rows = min(32, (n - base + nwarps - 1) / nwarps);
        auto load = [&](int32_t e, int32_t e1, int32_t& c, double2& v) {
            c = e < e1 ? idx[e] : 0;
            v = e < e1 ? lu[pos[e]] : zero;
        };
        int32_t e0 = __shfl_sync(0xffffffffu, beg, 0), e1 = __shfl_sync(0xffffffffu, end, 0);
        int32_t c;
        double2 v;
        load(e0 + lane, e1, c, v);
        for (int32_t r = 0; r < rows; ++r) {
            const int32_t i = __shfl_sync(0xffffffffu, row, r);
            const int32_t ne0 = __shfl_sync(0xffffffffu, beg, (r + 1) & 31);
            const int32_t ne1 = __shfl_sync(0xffffffffu, end, (r + 1) & 31);
            int32_t nc = 0;
            double2 nv = zero;
            if (r + 1 < rows) load(ne0 + lane, ne1, nc, nv);
            const int32_t len = e1 - e0;
            double2 t = w[i];
            for (int32_t m0 = 0; m0 < len; m0 += 32) {
                const int32_t cc = c;
                const double2 vv = v;
                if (m0 + 32 < len) load(e0 + m0 + 32 + lane, e1, c, v);
                const int32_t m = min(32, len - m0);
                bool ready = lane >= m;
                double2 p = zero;
                int32_t k = 0;
                int spins = 0;
                while (k < m) {
                    if (!ready && (flag_acquire(done + cc) >= target || !ok)) {
                        ready = true;
                        const double2 x = w[cc];
                        p = (kForward && c_zero(x)) ? zero : c_mul(vv, x);
                    }
                    const unsigned open = __ballot_sync(0xffffffffu, !ready);
                    const int32_t stop = open ? min(m, __ffs(open) - 1) : m;
                    if (stop == k) {
                        if (++spins > limit) ok = false;
                        else if (spins > 4) __nanosleep(20);
                        continue;
                    }
                    for (; k + 2 <= stop; k += 2) {
                        const double2 p0 = c_shfl(p, k), p1 = c_shfl(p, k + 1);
                        t.x = __dsub_rn(__dsub_rn(t.x, p0.x), p1.x);
                        t.y = __dsub_rn(__dsub_rn(t.y, p0.y), p1.y);
                    }
                    if (k < stop) {
                        const double2 p0 = c_shfl(p, k++);
                        t.x = __dsub_rn(t.x, p0.x);
                        t.y = __dsub_rn(t.y, p0.y);
                    }
                }
            }
            if (kForward) {
                const double2 d = c_shfl(piv, r);
                if (!c_zero(t)) t = c_mul(t, d);
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

// Level after level, a thread per row (below).
__device__ void c_solve_levels(const PlanDesc& pd, const int32_t* pool, const double* lu, double* x,
                               double* w);

// x <- A^{-1} x for one instance per CTA with dataflow sweeps.  Level after
// level with a thread per row and the vector in global memory, 150 points of a
// 1026-unknown mesh took 1.81 ms, here 0.35 ms.  If a bounded wait gave up,
// x still holds the right-hand side and is solved level after level.
template <int kThreads, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks)
complex_flow_solve_kernel(const PlanDesc* __restrict__ plans, const int32_t* __restrict__ pool,
                          const InstDesc* __restrict__ insts, const double* __restrict__ LU,
                          double* X, bool any_wide) {
    extern __shared__ __align__(16) double2 cols[];
    const InstDesc id = insts[blockIdx.x];
    const PlanDesc& pd = plans[id.plan];
    const int32_t n = pd.n;
    const int32_t* perm_row = pool + pd.off[PA_perm_row];
    const int32_t* perm_col = pool + pd.off[PA_perm_col];
    const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
    const double2* lu = reinterpret_cast<const double2*>(LU) + id.lu_off;
    double* x = X + 2 * id.x_off;
    if (any_wide && wide_levels(pd)) {
        c_solve_levels(pd, pool, LU + 2 * id.lu_off, x, reinterpret_cast<double*>(cols));
        return;
    }
    volatile int32_t* done = reinterpret_cast<volatile int32_t*>(cols + n);
    __shared__ int32_t s_ok;
    if (threadIdx.x == 0) s_ok = 1;
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) {
        cols[i] = make_double2(x[2 * perm_row[i]], x[2 * perm_row[i] + 1]);
        done[i] = 0;
    }
    __syncthreads();
    bool ok = c_sweep_rows<true>(pool + pd.off[PA_fwd_lev], pool + pd.off[PA_lrow_ptr],
                                 pool + pd.off[PA_lrow_col], pool + pd.off[PA_lrow_pos], diag_pos,
                                 lu, n, cols, done, 1);
    __syncthreads();
    ok = c_sweep_rows<false>(pool + pd.off[PA_bwd_lev], pool + pd.off[PA_urow_ptr],
                             pool + pd.off[PA_urow_col], pool + pd.off[PA_urow_pos], diag_pos, lu,
                             n, cols, done, 2) && ok;
    if (!ok) s_ok = 0;
    __syncthreads();
    if (s_ok == 0) {
        c_solve_levels(pd, pool, LU + 2 * id.lu_off, x, reinterpret_cast<double*>(cols));
        return;
    }
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) {
        x[2 * perm_col[i]] = cols[i].x;
        x[2 * perm_col[i] + 1] = cols[i].y;
    }
}

// The general refactor: factors whose columns exceed shared memory, or a
// factor array that is not aligned for 16-byte loads.
// One CTA per instance; warps claim columns in pivot order and eliminate each
// in place in lu (interleaved complex), waiting (bounded) for the columns
// their U entries name.  Completion flags live in shared memory.
__global__ void __launch_bounds__(kCplxThreads)
complex_refactor_kernel(const PlanDesc* __restrict__ plans, const int32_t* __restrict__ pool,
                        const InstDesc* __restrict__ insts, const double* __restrict__ A,
                        double* LU, int32_t* status) {
    extern __shared__ int32_t s_done[];
    __shared__ int32_t s_next, s_fail, s_timeout;
    const InstDesc id = insts[blockIdx.x];
    const PlanDesc& pd = plans[id.plan];
    const int32_t n = pd.n;
    const int32_t* col_ptr = pool + pd.off[PA_col_ptr];
    const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
    const int32_t* lu_src = pool + pd.off[PA_lu_src];
    const int32_t* upd_dst = pool + pd.off[PA_upd_dst];
    const int32_t map16 = pd.map16;
    const int4* umeta = reinterpret_cast<const int4*>(pool + pd.off[PA_umeta]);
    const double* a = A + 2 * id.a_off;
    double* lu = LU + 2 * id.lu_off;
    const int lane = threadIdx.x & 31;
    for (int32_t j = threadIdx.x; j < n; j += blockDim.x) s_done[j] = 0;
    if (threadIdx.x == 0) {
        s_next = 0;
        s_fail = 0x7fffffff;
        s_timeout = 0;
    }
    __syncthreads();
    const int limit = c_wait_limit;
    for (;;) {
        int32_t j = 0;
        if (lane == 0) j = atomicAdd(&s_next, 1);
        j = __shfl_sync(0xffffffffu, j, 0);
        if (j >= n) break;
        const int32_t c0 = col_ptr[j];
        const int32_t len = col_ptr[j + 1] - c0;
        const int32_t dj = diag_pos[j] - c0;
        double* col = lu + 2 * static_cast<int64_t>(c0);
        for (int32_t t = lane; t < len; t += 32) {
            const int32_t src = lu_src[c0 + t];
            col[2 * t] = src >= 0 ? a[2 * src] : 0.0;
            col[2 * t + 1] = src >= 0 ? a[2 * src + 1] : 0.0;
        }
        __syncwarp();
        bool timed_out = false;
        for (int32_t q = 0; q < dj; ++q) {
            const int4 m = u_entry(umeta, c0 + q);  // {r, diag_pos[r], |L(:, r)|, upd_start}
            int ready = 0;
            if (lane == 0) {
                int spins = 0;
                while ((ready = flag_acquire(s_done + m.x)) == 0) {
                    if (++spins > limit) break;
                    __nanosleep(32);
                }
            }
            ready = __shfl_sync(0xffffffffu, ready, 0);
            if (!ready) {
                timed_out = true;
                break;
            }
            const double pr = lu[2 * static_cast<int64_t>(m.y)];
            const double pi = lu[2 * static_cast<int64_t>(m.y) + 1];
            const double xr = col[2 * q], xi = col[2 * q + 1];
            const double ur = c_re(xr, xi, pr, pi);
            const double ui = c_im(xr, xi, pr, pi);
            __syncwarp();
            if (lane == 0) {
                col[2 * q] = ur;
                col[2 * q + 1] = ui;
            }
            const double* lcol = lu + 2 * (static_cast<int64_t>(m.y) + 1);
            for (int32_t t = lane; t < m.z; t += 32) {
                const int32_t dst = upd_at(upd_dst, map16, m.w + t);
                const double lr = lcol[2 * t], li = lcol[2 * t + 1];
                col[2 * dst] = __dsub_rn(col[2 * dst], c_re(ur, ui, lr, li));
                col[2 * dst + 1] = __dsub_rn(col[2 * dst + 1], c_im(ur, ui, lr, li));
            }
            __syncwarp();
        }
        if (lane == 0) {
            if (timed_out) {
                s_timeout = 1;
            } else {
                const double vr = col[2 * dj], vi = col[2 * dj + 1];
                if (__dadd_rn(fabs(vr), fabs(vi)) == 0.0) {
                    atomicMin(&s_fail, j);
                } else {
                    double rr, ri;
                    c_recip(vr, vi, rr, ri);
                    col[2 * dj] = rr;
                    col[2 * dj + 1] = ri;
                }
            }
            __threadfence_block();
            flag_release(s_done + j, 1);
        }
        __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x == 0)
        status[id.index] = s_timeout ? kStatusTimeout
                                     : (s_fail != 0x7fffffff ? kStatusSingular : kStatusOk);
}

// x <- A^{-1} x by the whole CTA, level-synchronous: rows of a level in parallel,
// each accumulating its updates in the reference's order (forward: columns
// ascending, skipping zero x_c; backward: row dot in ascending column order).
// w: 2n doubles of scratch.
__device__ __forceinline__ void c_solve_rows(const PlanDesc& pd, const int32_t* pool,
                                             const double* lu, double* x, double* w) {
    const int32_t n = pd.n;
    const int32_t* perm_row = pool + pd.off[PA_perm_row];
    const int32_t* perm_col = pool + pd.off[PA_perm_col];
    const int32_t* diag_pos = pool + pd.off[PA_diag_pos];
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) {
        w[2 * i] = x[2 * perm_row[i]];
        w[2 * i + 1] = x[2 * perm_row[i] + 1];
    }
    __syncthreads();
    {
        const int32_t* lp = pool + pd.off[PA_lrow_ptr];
        const int32_t* lpos = pool + pd.off[PA_lrow_pos];
        const int32_t* lcol = pool + pd.off[PA_lrow_col];
        const int32_t* lev_ptr = pool + pd.off[PA_fwd_lev_ptr];
        const int32_t* lev = pool + pd.off[PA_fwd_lev];
        for (int32_t l = 0; l < pd.n_fwd_lev; ++l) {
            for (int32_t k = lev_ptr[l] + threadIdx.x; k < lev_ptr[l + 1]; k += blockDim.x) {
                const int32_t i = lev[k];
                double tr = w[2 * i], ti = w[2 * i + 1];
                for (int32_t e = lp[i]; e < lp[i + 1]; ++e) {
                    const int32_t c = lcol[e];
                    const double xr = w[2 * c], xi = w[2 * c + 1];
                    if (xr != 0.0 || xi != 0.0) {
                        const double lr = lu[2 * lpos[e]], li = lu[2 * lpos[e] + 1];
                        tr = __dsub_rn(tr, c_re(xr, xi, lr, li));
                        ti = __dsub_rn(ti, c_im(xr, xi, lr, li));
                    }
                }
                if (tr != 0.0 || ti != 0.0) {
                    const double pr = lu[2 * diag_pos[i]], pi = lu[2 * diag_pos[i] + 1];
                    const double nr = c_re(tr, ti, pr, pi);
                    ti = c_im(tr, ti, pr, pi);
                    tr = nr;
                }
                w[2 * i] = tr;
                w[2 * i + 1] = ti;
            }
            __syncthreads();
        }
    }
    {
        const int32_t* up = pool + pd.off[PA_urow_ptr];
        const int32_t* upos = pool + pd.off[PA_urow_pos];
        const int32_t* ucol = pool + pd.off[PA_urow_col];
        const int32_t* lev_ptr = pool + pd.off[PA_bwd_lev_ptr];
        const int32_t* lev = pool + pd.off[PA_bwd_lev];
        for (int32_t l = 0; l < pd.n_bwd_lev; ++l) {
            for (int32_t k = lev_ptr[l] + threadIdx.x; k < lev_ptr[l + 1]; k += blockDim.x) {
                const int32_t i = lev[k];
                double tr = w[2 * i], ti = w[2 * i + 1];
                for (int32_t e = up[i]; e < up[i + 1]; ++e) {
                    const int32_t c = ucol[e];
                    const double ur = lu[2 * upos[e]], ui = lu[2 * upos[e] + 1];
                    const double xr = w[2 * c], xi = w[2 * c + 1];
                    tr = __dsub_rn(tr, c_re(ur, ui, xr, xi));
                    ti = __dsub_rn(ti, __dadd_rn(__dmul_rn(ur, xi), __dmul_rn(ui, xr)));
                }
                w[2 * i] = tr;
                w[2 * i + 1] = ti;
            }
            __syncthreads();
        }
    }
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) {
        x[2 * perm_col[i]] = w[2 * i];
        x[2 * perm_col[i] + 1] = w[2 * i + 1];
    }
}

// The same out of line, for the kernel that reaches it only for wide levels or
// where a bounded wait gave up.
__device__ __noinline__ void c_solve_levels(const PlanDesc& pd, const int32_t* pool,
                                            const double* lu, double* x, double* w) {
    c_solve_rows(pd, pool, lu, x, w);
}

// The general solve (as the general refactor), one instance per CTA.
__global__ void __launch_bounds__(kCplxThreads)
complex_solve_kernel(const PlanDesc* __restrict__ plans, const int32_t* __restrict__ pool,
                     const InstDesc* __restrict__ insts, const double* __restrict__ LU,
                     double* X, double* W) {
    const InstDesc id = insts[blockIdx.x];
    c_solve_rows(plans[id.plan], pool, LU + 2 * id.lu_off, X + 2 * id.x_off, W + 2 * id.w_off);
}

}  // namespace

// Shared memory of the general complex refactor: the completion flags.
size_t complex_refactor_smem(int max_n) { return sizeof(int32_t) * static_cast<size_t>(max_n); }

namespace {

constexpr size_t kMaxCplxSmem = 200 * 1024;
constexpr int kWideThreads = 512;
constexpr int kRefactorNeed = 6, kSolveNeed = 4;  // flow_shape

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <class Kernel, class... Args>
cudaError_t launch_complex(Kernel kernel, int count, int threads, size_t smem, cudaStream_t stream,
                           Args... args) {
    if (smem > kUnaskedSmem) {
        const cudaError_t e = cudaFuncSetAttribute(
            kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMaxCplxSmem));
        if (e != cudaSuccess) return e;
    }
    kernel<<<count, threads, smem, stream>>>(args...);
    return cudaGetLastError();
}

size_t complex_flow_bytes(int colbuf, int max_n, int warps) {
    return sizeof(double2) * static_cast<size_t>(warps) * static_cast<size_t>(colbuf) +
           sizeof(int32_t) * static_cast<size_t>(max_n);
}
size_t complex_sweep_bytes(int max_n) {
    return (sizeof(double2) + sizeof(int32_t)) * static_cast<size_t>(max_n);
}

}  // namespace

cudaError_t launch_complex_refactor(const PlanDesc* plans, const int32_t* pool,
                                    const InstDesc* insts, const FlowBatch& b, const double* A,
                                    double* LU, int32_t* status, cudaStream_t stream) {
    const int colbuf = (b.max_col + 31) & ~31;
    if (complex_flow_bytes(colbuf, b.max_n, kWideThreads / 32) <= kMaxCplxSmem && aligned16(LU)) {
        // 8 warps take up to twice as long as 16 (the more entries, the closer to it), so
        // a last pass that is nearly empty costs more: 700 meshes of 577 unknowns 0.77
        // ms, on 16 warps 0.65; 592 0.50 and 0.51, 700 of 37 0.048 and 0.059
        const double slower = 1.0 + std::min(1.0, b.row_entries / 8);
        const int need = flow_waves(b, 4) * slower <= flow_waves(b, 2) ? kRefactorNeed : INT_MAX;
        const FlowShape shape =
            flow_shape(b, complex_flow_bytes(colbuf, b.max_n, kWideThreads / 64), need);
        const int threads = shape == kShapeMany ? kWideThreads / 2 : kWideThreads;
        auto launch = [&](auto kernel) {
            return launch_complex(kernel, b.count, threads,
                                  complex_flow_bytes(colbuf, b.max_n, threads / 32), stream, plans,
                                  pool, insts, A, LU, status, colbuf);
        };
        if (shape == kShapeAlone) return launch(complex_flow_refactor_kernel<kWideThreads, 1>);
        if (shape == kShapePair) return launch(complex_flow_refactor_kernel<kWideThreads, 2>);
        return launch(complex_flow_refactor_kernel<kWideThreads / 2, 4>);
    }
    const size_t smem = complex_refactor_smem(b.max_n);
    if (smem > kUnaskedSmem) {
        const cudaError_t e = cudaFuncSetAttribute(
            complex_refactor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
    }
    complex_refactor_kernel<<<b.count, kCplxThreads, smem, stream>>>(plans, pool, insts, A, LU,
                                                                      status);
    return cudaGetLastError();
}

// Whether launch_complex_solve can keep the vector in shared memory (and needs no
// workspace W).
bool complex_solve_in_smem(int max_n, const double* LU) {
    return complex_sweep_bytes(max_n) <= kMaxCplxSmem && aligned16(LU);
}

// Whether it had better run level after level in W (2 n doubles per instance) all
// the same.
bool complex_levels_pay(const FlowBatch& b, const double* LU) {
    const size_t smem = complex_sweep_bytes(b.max_n);
    return complex_solve_in_smem(b.max_n, LU) && levels_pay(b, flow_shape(b, smem, kSolveNeed), smem);
}

// W null: the dataflow sweeps although the other would pay.
cudaError_t launch_complex_solve(const PlanDesc* plans, const int32_t* pool, const InstDesc* insts,
                                 const FlowBatch& b, const double* LU, double* X, double* W,
                                 cudaStream_t stream) {
    if (complex_solve_in_smem(b.max_n, LU) && !(W && complex_levels_pay(b, LU))) {
        const size_t smem = complex_sweep_bytes(b.max_n);
        if (flow_shape(b, smem, kSolveNeed) == kShapeMany)
            return launch_complex(complex_flow_solve_kernel<kWideThreads / 2, 4>, b.count,
                                  kWideThreads / 2, smem, stream, plans, pool, insts, LU, X, b.wide);
        return launch_complex(complex_flow_solve_kernel<kWideThreads, 2>, b.count, kWideThreads, smem,
                              stream, plans, pool, insts, LU, X, b.wide);
    }
    complex_solve_kernel<<<b.count, kCplxThreads, 0, stream>>>(plans, pool, insts, LU, X, W);
    return cudaGetLastError();
}

}  // namespace nsg
