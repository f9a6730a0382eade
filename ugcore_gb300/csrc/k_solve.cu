// k_solve.cu -- SpMV-based multigrid and Krylov kernels (SELL-32 or diagonal).
//
// Every kernel is HBM-bound: one thread per row, matrix values streamed with
// evict-first loads (coalesced 32-wide), the gathered vector kept in L1/L2.
// Two operator layouts share the kernels through a "matrix view":
//   SELL-32   general sparsity: 32-row slices, column-major in the slice;
//   diagonal  <= 27 constant offsets (structured levels; 7, 9, 15, 27): values only, the
//             column of entry k is row + off[k]; no column stream and no
//             load that depends on another load.
// Row-local vector work is fused into the SpMV epilogue so each sweep reads
// the operator once:
//   Jacobi step     t = dinv*d ; d -= A t ; sc += t
//                   (Jacobi::step, lib_algebra/operator/preconditioner/
//                    jacobi.h:222; AssembledMultiGridCycle::
//                    presmooth_and_restriction / prolongation_and_postsmooth,
//                    mg_solver_impl.hpp:1687-1966) becomes one pass over the
//                   column-scaled operator At = A*diag(dinv): d_new = d - At x.
//   prolongation    t = P sc_c ; sc += t ; w = t / dinv (so that A t = At w)
//                   (StdTransfer::prolongate, std_transfer_impl.h:721)
//   restriction     d_c = R d (StdTransfer::do_restrict, std_transfer_impl.h:776)
//   CG              q = A z + beta q, p = z + beta p and lambda = (q,p) in one
//                   pass (CG::apply_return_defect, cg.h:163-226)
// Reductions are deterministic (grid_reduce: fixed-order tree per block,
// block partials summed in block order by the last block).
#include <algorithm>

#include "k_solve.cuh"

namespace ug4gb {

constexpr int NT = 256;

int row_grid(const Ctx &c, int nrows)
{
    int need = (int)div_up(nrows > 0 ? nrows : 1, NT);
    int cap = c.num_sms * 8;
    return need < cap ? need : cap;
}

// widening to FP64 of a level-precision value (identity for FP64)
__device__ __forceinline__ double f32_to_f64_t(double v) { return v; }
__device__ __forceinline__ double f32_to_f64_t(float v) { return f32_to_f64(v); }

// ------------------------------------------------------------ views ------
template <class V, int AHEAD = 8>
struct SellMV {
    static constexpr int kCache = AHEAD;   // entries of a row loaded ahead (the rest after the wait)
    SellView<V> s;
    struct Cache {
        int base, w;
        int col[kCache];
        V val[kCache];
    };
    __device__ __forceinline__ int rows() const { return s.nrows; }
    __device__ __forceinline__ void prefetch(int row, Cache &c) const
    {
        const int sl = row >> 5, lane = row & 31;
        c.base = __ldg(s.sptr + sl) + lane;
        c.w = __ldg(s.swidth + sl);
#pragma unroll
        for (int k = 0; k < kCache; ++k) {
            if (k < c.w) {
                c.col[k] = __ldg(s.col + c.base + k * kSliceH);
                c.val[k] = __ldg(s.val + c.base + k * kSliceH);
            }
        }
    }
    // dot with a prefetched row; same order of operations as dot.  FP64 leaves at the
    // row's end: a product that a predicate turns off still takes its turn on the
    // FP64 pipe (triangles, 7 of 8 slots, 2400 rows: a V(2,2) cycle 53.3 us, 50.0
    // with the branches; FP32 the other way round, 41.1 and 41.7).
    template <class ACC, class XT>
    __device__ __forceinline__ ACC dot_cached(const XT *__restrict__ x, int, const Cache &c) const
    {
        ACC xv[kCache];
#pragma unroll
        for (int k = 0; k < kCache; ++k)
            if (k < c.w) xv[k] = (ACC)x[c.col[k]];
        ACC acc = (ACC)0;
#pragma unroll
        for (int k = 0; k < kCache; ++k) {
            if constexpr (sizeof(ACC) == 8) {
                if (k >= c.w) return acc;
                acc = fma_rn((ACC)c.val[k], xv[k], acc);
            } else {
                if (k < c.w) acc = fma_rn((ACC)c.val[k], xv[k], acc);
            }
        }
        // the rest: the loads of kCache entries issued before their sum (one
        // entry after the other cost a level of 15000 rows 2 us per product)
#pragma unroll 1
        for (int k = kCache; k < c.w; k += kCache) {
            int col[kCache];
            V val[kCache];
#pragma unroll
            for (int q = 0; q < kCache; ++q)
                if (k + q < c.w) {
                    col[q] = ld_stream(s.col + c.base + (k + q) * kSliceH);
                    val[q] = ld_stream(s.val + c.base + (k + q) * kSliceH);
                }
#pragma unroll
            for (int q = 0; q < kCache; ++q)
                if (k + q < c.w) xv[q] = (ACC)x[col[q]];
#pragma unroll
            for (int q = 0; q < kCache; ++q) {
                if constexpr (sizeof(ACC) == 8) {
                    if (k + q >= c.w) return acc;
                    acc = fma_rn((ACC)val[q], xv[q], acc);
                } else {
                    if (k + q < c.w) acc = fma_rn((ACC)val[q], xv[q], acc);
                }
            }
        }
        return acc;
    }
    template <class ACC, class XT>
    __device__ __forceinline__ ACC dot(const XT *__restrict__ x, int row) const
    {
        const int sl = row >> 5, lane = row & 31;
        const int base = __ldg(s.sptr + sl) + lane;
        const int w = __ldg(s.swidth + sl);
        ACC acc = (ACC)0;
#pragma unroll 4
        for (int k = 0; k < w; ++k) {
            const int idx = base + k * kSliceH;
            acc += (ACC)ld_stream(s.val + idx) * (ACC)x[ld_stream(s.col + idx)];
        }
        return acc;
    }
};

// Products of few rows (up to a block per SM) of a SELL matrix load whole rows
// ahead of the launch wait, as an entry beyond takes another round of dependent
// loads; slots that a row does not fill cost instructions and registers.  So the
// slots follow the slices' mean width.  V(2,2) cycles with 8 / 12 / 16 / 24 slots
// (us; FP64, then FP32):
//   triangles, 7 entries, 37000 rows         73.3 / 71.9 / 72.4 / 74.0    57.5 / 58.0 / 59.0 / 59.6
//   the same, 148000 rows                   107.7 /101.6 /104.1 /107.3    73.7 / 74.0 / 74.7 / 75.4
//   quadrilaterals, 9 entries, 37000 rows    91.5 / 78.3 / 79.0 / 81.2    71.5 / 61.6 / 62.0 / 61.6
//   tetrahedra, 15 to 24, 36000 rows         88.5 / 78.5 / 79.9 / 71.4    63.1 / 66.0 / 56.5 / 46.7
//   hexahedra, 27, 36000 rows               113.9 /110.2 / 98.1 / 96.6    86.7 /121.9 / 66.5 / 78.0
// With more rows the registers cost more than the loads: a step of 117000 rows of
// tetrahedra FP32 11.1 -> 13.6 us with 24.
template <class V, class F>
void with_few_rows(const Sell<V> &m, const SellMV<V> &mv, F &&f)
{
    const int64_t slots = (int64_t)m.nslices * kSliceH;
    if (sizeof(V) == 4 && m.stored <= 8 * slots) f(mv);
    else if (m.stored <= 12 * slots) f(SellMV<V, 12>{mv.s});
    else if (m.stored <= 24 * slots) f(SellMV<V, 24>{mv.s});
    else f(SellMV<V, 16>{mv.s});
}

template <class V, int S>
struct DiaMV {
    static constexpr int kS = S;
    int n, ncols, ld;
    const V *__restrict__ val;
    Offs off;
    struct Cache {
        V a[S];
    };
    __device__ __forceinline__ int rows() const { return n; }
    __device__ __forceinline__ void prefetch(int i, Cache &c) const
    {
#pragma unroll
        for (int k = 0; k < S; ++k) c.a[k] = ld_stream(val + (size_t)k * ld + i);
    }
    // rows of a latency-bound level (row_sum)
    template <class ACC, class XT>
    __device__ __forceinline__ ACC dot_cached(const XT *__restrict__ x, int i, const Cache &c) const
    {
        ACC xv[S];
#pragma unroll
        for (int k = 0; k < S; ++k) {
            int j = i + off.o[k];
            j = j < 0 ? 0 : (j >= ncols ? ncols - 1 : j);
            xv[k] = (ACC)x[j];
        }
        return row_sum<ACC, S>(c.a, xv);
    }
    template <class ACC, class XT>
    __device__ __forceinline__ ACC dot(const XT *__restrict__ x, int i) const
    {
        ACC acc = (ACC)0;
#pragma unroll
        for (int k = 0; k < S; ++k) {
            int j = i + off.o[k];
            j = j < 0 ? 0 : (j >= ncols ? ncols - 1 : j);
            acc = fma_rn((ACC)ld_stream(val + (size_t)k * ld + i), (ACC)x[j], acc);
        }
        return acc;
    }
    // W consecutive rows i0..i0+W-1 (i0 % W == 0, all < n): one 16-byte
    // value load per diagonal instead of W scalar ones
    template <int W, class XT>
    __device__ __forceinline__ void dot_w(const XT *__restrict__ x, int i0, V (&acc)[W]) const
    {
#pragma unroll
        for (int e = 0; e < W; ++e) acc[e] = (V)0;
        // diagonals in three batches (all 7 at once): the packs in flight per
        // thread keep the register count low enough for a full SM
        constexpr int B = (S == 7) ? 7 : S / 3;
        static_assert(S % B == 0, "S must be a multiple of the batch");
#pragma unroll 1
        for (int kb = 0; kb < S; kb += B) {
            Pack<V, W> a[B];
#pragma unroll
            for (int k = 0; k < B; ++k) a[k] = ld_stream_pack<V, W>(val + (size_t)(kb + k) * ld + i0);
#pragma unroll
            for (int k = 0; k < B; ++k) {
                const int j = i0 + off.o[kb + k];
#pragma unroll
                for (int e = 0; e < W; ++e) {
                    int jj = j + e;
                    jj = jj < 0 ? 0 : (jj >= ncols ? ncols - 1 : jj);
                    acc[e] = fma_rn(a[k].v[e], (V)x[jj], acc[e]);
                }
            }
        }
    }
};

template <class MV>
struct is_dia : std::false_type {};
template <class V, int S>
struct is_dia<DiaMV<V, S>> : std::true_type {};

// Grid of a kernel with one row product per thread and iteration.  FP64
// products of 15 or 27 diagonals are bound by the FP64 issue rate, and the warps
// of an SM do not get equal shares of it: with one resident wave of blocks that
// stride over the rows, some finish early and the rest leave the pipe idle
// (129^3 hexes: 86% busy, 74% of the warps present).  More blocks than
// resident ones keep it fed: one row per thread (a smoothing step 126 -> 112
// us); with a reduction at each block's end one to four, about three waves
// of blocks (last step 140 -> 134 us, q = A z 130 -> 126 us at two rows, 125
// at four).  Products bound by memory (SELL, 7 or 9 diagonals, FP32) and
// levels of less than a wave keep the one wave.
template <class MV, class V>
static int spmv_grid(const Ctx &c, int nrows, bool reduces)
{
    constexpr bool fp64_bound = [] {
        if constexpr (is_dia<MV>::value) return sizeof(V) == 8 && MV::kS >= 15;
        else return false;
    }();
    const int wave = c.num_sms * 8 * NT;
    // FP32 levels of one to three waves: one row per thread too (97x65x65 hexes,
    // 1.3 waves: a flow gradient 16.4 -> 16.2 ms)
    if (is_dia<MV>::value && sizeof(V) == 4 && !reduces) return (int)div_up(nrows, NT);
    if (!fp64_bound || nrows <= wave) return row_grid(c, nrows);
    int per = 1;
    if (reduces) {
        per = nrows / (3 * wave);
        per = per < 1 ? 1 : (per > 4 ? 4 : per);
        while (div_up(nrows, (size_t)NT * per) > (unsigned)kRedMaxBlocks) ++per;
    }
    return (int)div_up(nrows, (size_t)NT * per);
}

// calls f(view) with the view type matching the operator's layout
template <class V, class F>
void with_mv(const OpMat<V> &m, F &&f)
{
    if (m.kind == 0) {
        f(SellMV<V>{view(m.sell)});
        return;
    }
    const Dia<V> &d = m.dia;
    switch (d.S) {
    case 7: f(DiaMV<V, 7>{d.nrows, d.ncols, d.ld, d.vals(), d.off}); break;
    case 9: f(DiaMV<V, 9>{d.nrows, d.ncols, d.ld, d.vals(), d.off}); break;
    case 15: f(DiaMV<V, 15>{d.nrows, d.ncols, d.ld, d.vals(), d.off}); break;
    case 27: f(DiaMV<V, 27>{d.nrows, d.ncols, d.ld, d.vals(), d.off}); break;
    default: throw Error{UG4GB_ERR_INVALID, "diagonal operator with unsupported width"};
    }
}

__device__ __forceinline__ bool conv_valid(double v)
{
    if (v == 0.0) return true;
    return v >= 2.2250738585072014e-308 && v <= 1.7976931348623157e308 && v == v && v >= 0.0;
}

__device__ __forceinline__ bool conv_ended(const KScal *ks)
{
    if (!conv_valid(ks->dcur)) return true;
    if (ks->step >= ks->maxit) return true;
    if (ks->dcur < ks->min_def) return true;
    if (ks->dcur / ks->d0 < ks->rel_red) return true;
    return false;
}

__device__ __forceinline__ void conv_update(KScal *ks, double d, int done_value)
{
    ks->dcur = d;
    ks->step += 1;
    if (ks->hist && ks->step < ks->hist_cap) ks->hist[ks->step] = d;
    if (conv_ended(ks)) ks->done = done_value;
}

// ------------------------------------------------------- smoothing step --
// PF (levels of at most one wave of rows, where latency rules): this
// thread's first row of the operator and its Jacobi factor are loaded
// before waiting for the predecessor (no solve kernel writes them).  Large
// levels skip it: the cached row would cost registers, hence occupancy.
template <class MV, class V, class XT, class DT, bool RHO, bool PF>
__global__ void __launch_bounds__(NT) k_smooth(MV A, const XT *__restrict__ x, const DT *__restrict__ dbase,
                                               const V *__restrict__ dinv, V *__restrict__ sc, V *__restrict__ dout,
                                               int sc_mode, const int *skip, const double *__restrict__ r_rho,
                                               RedArgs red, int rho_kind, double *__restrict__ z64)
{
    const int stride = gridDim.x * NT, n = A.rows(), row0 = blockIdx.x * NT + threadIdx.x;
    typename MV::Cache cache;
    V dinv0 = (V)0;
    if constexpr (PF) {
        pdl_trigger();
        if (row0 < n) {
            A.prefetch(row0, cache);
            dinv0 = dinv[row0];
        }
        pdl_wait();
    } else {
        PDL_ENTRY();
    }
    if (skip && *skip) return;
    double rsum = 0.0;
    for (int row = row0; row < n; row += stride) {
        const bool first = PF && (row == row0);
        V acc = first ? A.template dot_cached<V>(x, row, cache) : A.template dot<V>(x, row);
        V db = (V)dbase[row];
        V s;
        V dn = jacobi_row<V>(acc, db, first ? dinv0 : dinv[row], sc_mode,
                             sc_mode == SC_SET_FROM_BASE ? (V)0 : sc[row], s);
        if (dout) dout[row] = dn;
        sc[row] = s;
        if (RHO || z64) {
            const double s64 = f32_to_f64_t(s);   // one conversion per row, only where needed
            if (z64) z64[row] = s64;
            if (RHO) rsum += s64 * r_rho[row];
        }
    }
    if (RHO) {
        double v[1] = {rsum};
        KScal *ks = red.ks;
        grid_reduce<NT, 1>(v, red.partials, red.counter, [&](const double(&tot)[1]) {
            if (rho_kind == 0) {
                ks->rho_old = tot[0];
            } else {
                ks->rho = tot[0];
                ks->beta = tot[0] / ks->rho_old;
                ks->rho_old = tot[0];
            }
        });
    }
}

// The same step on the diagonal layout with W = 16/sizeof(V) consecutive rows
// per thread: every value and row-vector access is one 16-byte load or
// store (the gathered x stays scalar).  A tail of n % W rows is done by the
// thread that owns the last, partial group.  Per row the arithmetic is that
// of k_smooth.  32 registers (8 blocks of 256 threads per SM): the sweep is
// bound by memory latency, and the extra resident warps gave 2-4% per sweep.
// (The 7-diagonal step with the reduction spilled at 32: 40 registers, 6 blocks,
// 25.7 -> 22.0 us on the 129^3 tet level.)
constexpr int smooth_dia_blocks(int S, bool rho) { return S == 7 && rho ? 6 : 8; }   // resident per SM

template <class V, int S, bool RHO>
__global__ void __launch_bounds__(NT, smooth_dia_blocks(S, RHO))
    k_smooth_dia(DiaMV<V, S> A, const V *__restrict__ x, const V *__restrict__ dbase, const V *__restrict__ dinv,
                 V *__restrict__ sc, V *__restrict__ dout, int sc_mode, const int *skip,
                 const double *__restrict__ r_rho, RedArgs red, int rho_kind, double *__restrict__ z64)
{
    constexpr int W = 16 / sizeof(V);
    PDL_ENTRY();
    if (skip && *skip) return;
    double rsum = 0.0;
    const int n = A.rows(), ng = (n + W - 1) / W, stride = gridDim.x * NT;
    const bool wide64 = (((uintptr_t)z64 | (uintptr_t)r_rho) & 15u) == 0;
    for (int g = blockIdx.x * NT + threadIdx.x; g < ng; g += stride) {
        const int r0 = g * W;
        if (r0 + W <= n) {
            V acc[W];
            A.template dot_w<W>(x, r0, acc);
            Pack<V, W> db = ld_pack<V, W>(dbase + r0), di = ld_pack<V, W>(dinv + r0), s, dn;
            if (sc_mode != SC_SET_FROM_BASE) s = ld_pack<V, W>(sc + r0);
#pragma unroll
            for (int e = 0; e < W; ++e)
                dn.v[e] = jacobi_row<V>(acc[e], db.v[e], di.v[e], sc_mode,
                                        sc_mode == SC_SET_FROM_BASE ? (V)0 : s.v[e], s.v[e]);
            if (dout) st_pack<V, W>(dout + r0, dn);
            st_pack<V, W>(sc + r0, s);
            if (RHO || z64) {
                double s64[W];
#pragma unroll
                for (int e = 0; e < W; ++e) s64[e] = f32_to_f64_t(s.v[e]);
                if constexpr (W % 2 == 0) {
                    // FP64 side in 16-byte pairs when both arrays allow it
                    if (wide64) {
#pragma unroll
                        for (int e = 0; e < W; e += 2) {
                            if (z64) st_pack<double, 2>(z64 + r0 + e, Pack<double, 2>{{s64[e], s64[e + 1]}});
                            if (RHO) {
                                Pack<double, 2> rr = ld_pack<double, 2>(r_rho + r0 + e);
                                rsum += s64[e] * rr.v[0];
                                rsum += s64[e + 1] * rr.v[1];
                            }
                        }
                        continue;
                    }
                }
#pragma unroll
                for (int e = 0; e < W; ++e) {
                    if (z64) z64[r0 + e] = s64[e];
                    if (RHO) rsum += s64[e] * r_rho[r0 + e];
                }
            }
        } else {
            for (int row = r0; row < n; ++row) {
                V acc = A.template dot<V>(x, row);
                V s;
                V dn = jacobi_row<V>(acc, dbase[row], dinv[row], sc_mode,
                                     sc_mode == SC_SET_FROM_BASE ? (V)0 : sc[row], s);
                if (dout) dout[row] = dn;
                sc[row] = s;
                if (RHO || z64) {
                    const double s64 = f32_to_f64_t(s);
                    if (z64) z64[row] = s64;
                    if (RHO) rsum += s64 * r_rho[row];
                }
            }
        }
    }
    if (RHO) {
        double v[1] = {rsum};
        KScal *ks = red.ks;
        grid_reduce<NT, 1>(v, red.partials, red.counter, [&](const double(&tot)[1]) {
            if (rho_kind == 0) {
                ks->rho_old = tot[0];
            } else {
                ks->rho = tot[0];
                ks->beta = tot[0] / ks->rho_old;
                ks->rho_old = tot[0];
            }
        });
    }
}


inline bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

template <class V, class XT, class DT>
void smooth_step(Ctx &c, const OpMat<V> &At, const XT *x, const DT *dbase, const V *dinv, V *sc, V *dout, int sc_mode,
                 const int *skip, const double *r_rho, RedArgs *red, int rho_kind, double *z64)
{
    with_mv(At, [&](auto mv) {
        using MV = decltype(mv);
        const int g = spmv_grid<MV, V>(c, At.nrows, r_rho != nullptr);
        if constexpr (is_dia<MV>::value && std::is_same<XT, V>::value && std::is_same<DT, V>::value) {
            // FP32 levels of at least three full waves of one-row threads:
            // there the wider loads pay (8-9% per sweep on GB300).  FP64 sweeps
            // are bound by the FP64 FMA rate and smaller levels by latency;
            // there the one-row-per-thread kernel is as fast or faster.
            const bool wide = sizeof(V) == 4 && At.nrows >= c.num_sms * 2048 * 3;
            if (wide && aligned16(dbase) && aligned16(dinv) && aligned16(sc) && aligned16(dout)) {
                constexpr int W = 16 / sizeof(V);
                const int groups = (At.nrows + W - 1) / W;
                int gv = (int)div_up(groups > 0 ? groups : 1, NT);
                if (gv > kRedMaxBlocks) gv = kRedMaxBlocks;
                if (r_rho) {
                    // with the fused (z, r) reduction: one resident wave of blocks
                    // (8 per SM), so the blocks' reduction tails overlap and the
                    // last block sums fewer partials (-12% on the 129^3 tet level)
                    const int wave = c.num_sms * smooth_dia_blocks(MV::kS, true), gr = gv < wave ? gv : wave;
                    UG_LAUNCH_PDL(c, (k_smooth_dia<V, MV::kS, true>), gr, NT, 0, mv, x, dbase, dinv, sc, dout, sc_mode,
                                  skip, r_rho, *red, rho_kind, z64);
                } else {
                    RedArgs none{nullptr, nullptr, nullptr};
                    UG_LAUNCH_PDL(c, (k_smooth_dia<V, MV::kS, false>), gv, NT, 0, mv, x, dbase, dinv, sc, dout,
                                  sc_mode, skip, (const double *)nullptr, none, 0, z64);
                }
                return;
            }
        }
        // rows loaded ahead of the launch wait: FP64 levels of one row per thread
        // in a block per SM, FP32 ones of a whole wave (eight blocks per SM; 0.5 to
        // 3% of a solve over the smaller limit, where FP64 lost up to 7%)
        const bool pf = At.nrows <= c.num_sms * NT * (sizeof(V) == 4 ? 8 : 1);
        RedArgs none{nullptr, nullptr, nullptr};
        if constexpr (!is_dia<MV>::value) {
            if (pf && !r_rho && At.nrows <= c.num_sms * NT) {
                with_few_rows(At.sell, mv, [&](auto few) {
                    UG_LAUNCH_PDL(c, (k_smooth<decltype(few), V, XT, DT, false, true>), g, NT, 0, few, x, dbase, dinv,
                                  sc, dout, sc_mode, skip, (const double *)nullptr, none, 0, z64);
                });
                return;
            }
        }
        if (r_rho && pf) {
            UG_LAUNCH_PDL(c, (k_smooth<MV, V, XT, DT, true, true>), g, NT, 0, mv, x, dbase, dinv, sc, dout, sc_mode,
                          skip, r_rho, *red, rho_kind, z64);
        } else if (r_rho) {
            UG_LAUNCH_PDL(c, (k_smooth<MV, V, XT, DT, true, false>), g, NT, 0, mv, x, dbase, dinv, sc, dout, sc_mode,
                          skip, r_rho, *red, rho_kind, z64);
        } else if (pf) {
            UG_LAUNCH_PDL(c, (k_smooth<MV, V, XT, DT, false, true>), g, NT, 0, mv, x, dbase, dinv, sc, dout, sc_mode,
                          skip, (const double *)nullptr, none, 0, z64);
        } else {
            UG_LAUNCH_PDL(c, (k_smooth<MV, V, XT, DT, false, false>), g, NT, 0, mv, x, dbase, dinv, sc, dout, sc_mode,
                          skip, (const double *)nullptr, none, 0, z64);
        }
    });
}

#define INST_SMOOTH(V, XT, DT)                                                                              \
    template void smooth_step<V, XT, DT>(Ctx &, const OpMat<V> &, const XT *, const DT *, const V *, V *, V *, int, \
                                         const int *, const double *, RedArgs *, int, double *);
INST_SMOOTH(double, double, double)
INST_SMOOTH(float, float, float)

// --------------------------------------------------------- transfers -----
template <class MV, class V, bool PF>
__global__ void __launch_bounds__(NT) k_restrict(MV R, const V *__restrict__ d, V *__restrict__ dc, const int *skip)
{
    const int stride = gridDim.x * NT, n = R.rows(), row0 = blockIdx.x * NT + threadIdx.x;
    typename MV::Cache cache;
    if constexpr (PF) {
        pdl_trigger();
        if (row0 < n) R.prefetch(row0, cache);
        pdl_wait();
    } else {
        PDL_ENTRY();
    }
    if (skip && *skip) return;
    for (int row = row0; row < n; row += stride)
        dc[row] = (PF && row == row0) ? R.template dot_cached<V>(d, row, cache) : R.template dot<V>(d, row);
}

template <class V>
void restrict_apply(Ctx &c, const OpMat<V> &R, const V *d, V *dc, const int *skip)
{
    with_mv(R, [&](auto mv) {
        if constexpr (!is_dia<decltype(mv)>::value) {
            if (R.nrows <= c.num_sms * NT) {
                with_few_rows(R.sell, mv, [&](auto few) {
                    UG_LAUNCH_PDL(c, (k_restrict<decltype(few), V, true>), row_grid(c, R.nrows), NT, 0, few, d, dc,
                                  skip);
                });
                return;
            }
        }
        if (R.nrows <= c.num_sms * NT * (sizeof(V) == 4 ? 8 : 1))
            UG_LAUNCH_PDL(c, (k_restrict<decltype(mv), V, true>), row_grid(c, R.nrows), NT, 0, mv, d, dc, skip);
        else
            UG_LAUNCH_PDL(c, (k_restrict<decltype(mv), V, false>), row_grid(c, R.nrows), NT, 0, mv, d, dc, skip);
    });
}

template <class MV, class V, bool PF>
__global__ void __launch_bounds__(NT) k_prolong(MV P, const V *__restrict__ scc, V *__restrict__ sc,
                                                const V *__restrict__ dfac, V *__restrict__ w, const int *skip)
{
    const int stride = gridDim.x * NT, n = P.rows(), row0 = blockIdx.x * NT + threadIdx.x;
    typename MV::Cache cache;
    V dfac0 = (V)0;
    if constexpr (PF) {
        pdl_trigger();
        if (row0 < n) {
            P.prefetch(row0, cache);
            if (w) dfac0 = dfac[row0];
        }
        pdl_wait();
    } else {
        PDL_ENTRY();
    }
    if (skip && *skip) return;
    for (int row = row0; row < n; row += stride) {
        const bool first = PF && (row == row0);
        V t = first ? P.template dot_cached<V>(scc, row, cache) : P.template dot<V>(scc, row);
        sc[row] += t;
        if (w) w[row] = t * (first ? dfac0 : dfac[row]);
    }
}

template <class V>
void prolong_apply(Ctx &c, const OpMat<V> &P, const V *scc, V *sc, const V *dfac, V *w, const int *skip)
{
    with_mv(P, [&](auto mv) {
        if constexpr (!is_dia<decltype(mv)>::value) {
            // rows of one or two parents (triangles, tetrahedra: a V(2,2) cycle of
            // 148000 FP64 rows of triangles 108.0 -> 105.2 us)
            if (P.nrows <= c.num_sms * NT && P.sell.stored <= 2 * (int64_t)P.sell.nslices * kSliceH) {
                UG_LAUNCH_PDL(c, (k_prolong<SellMV<V, 2>, V, true>), row_grid(c, P.nrows), NT, 0, (SellMV<V, 2>{mv.s}),
                              scc, sc, dfac, w, skip);
                return;
            }
        }
        if (P.nrows <= c.num_sms * NT * (sizeof(V) == 4 ? 8 : 1))
            UG_LAUNCH_PDL(c, (k_prolong<decltype(mv), V, true>), row_grid(c, P.nrows), NT, 0, mv, scc, sc, dfac, w,
                          skip);
        else
            UG_LAUNCH_PDL(c, (k_prolong<decltype(mv), V, false>), row_grid(c, P.nrows), NT, 0, mv, scc, sc, dfac, w,
                          skip);
    });
}

// ------------------------------------------- grid-index transfers ---------

// Division by a run-time constant d >= 1 of 0 <= n < 2^31 as a multiplication
// and a shift (Granlund and Montgomery, "Division by invariant integers using
// multiplication", 1994): m = ceil(2^(31+s) / d) with s = ceil(log2 d).
struct FastDiv {
    unsigned d, m, s;
    explicit FastDiv(int n) : d((unsigned)n), m(0), s(0)
    {
        while ((1u << s) < d) ++s;
        m = (unsigned)((((unsigned long long)1 << (31 + s)) + d - 1) / d);
    }
    __device__ __forceinline__ int div(int n) const
    {
        return (int)(((unsigned long long)(unsigned)n * m) >> (31 + s));
    }
};

// t = P scc ; sc += t ; w = t * dfac (k_prolong on the assembled P), the
// parents and weights of prolong_value in its order.  A thread takes the two
// fine vertices 2I and 2I + 1 of a grid line: they share the coarse values
// of the lines around them, and the parities that choose the parents are those
// of the line, so a warp does not diverge; all loads of a pair are issued before
// its sums, the Jacobi factors of a thread's first pair (no solve kernel writes
// them) before the launch wait.  One vertex per thread, with loops over its 1
// to 8 parents, took 46 us on the 129^3 FP64 level and 54 us on the 193^3 FP32
// one.
template <class V>
__global__ void __launch_bounds__(NT) k_prolong_grid(GridPair g, FastDiv pairs, FastDiv lines, int npairs,
                                                     const V *__restrict__ scc, V *__restrict__ sc,
                                                     const V *__restrict__ dfac, V *__restrict__ w, const int *skip)
{
    const int stride = gridDim.x * NT;
    int q = blockIdx.x * NT + threadIdx.x;
    // fine vertices f and, if two, f + 1 of pair q; its line
    auto locate = [&](int qq, int &line, int &I, int &f, bool &two) {
        line = pairs.div(qq);
        I = qq - line * (int)pairs.d;
        f = 2 * I + g.nx * line;
        two = 2 * I + 1 < g.nx;
    };
    int line = 0, I = 0, f = 0;
    bool two = false;
    V df0 = (V)0, df1 = (V)0;
    pdl_trigger();
    if (q < npairs) {
        locate(q, line, I, f, two);
        if (w) {
            df0 = dfac[f];
            if (two) df1 = dfac[f + 1];
        }
    }
    pdl_wait();
    if (skip && *skip) return;
    for (bool first = true; q < npairs; q += stride, first = false) {
        if (!first) {
            locate(q, line, I, f, two);
            if (w) {
                df0 = dfac[f];
                if (two) df1 = dfac[f + 1];
            }
        }
        const int k = lines.div(line), j = line - k * (int)lines.d, i = 2 * I;
        const int p1 = j & 1, p2 = k & 1, J = j >> 1, K = k >> 1, I1 = two ? 1 : 0;
        V s0 = sc[f], s1 = two ? sc[f + 1] : (V)0;
        const bool edge = j == 0 || j == g.ny - 1 || (g.dim == 3 && (k == 0 || k == g.nz - 1));
        // on the boundary: only a coinciding coarse vertex, weight 1
        const bool b0 = edge || i == 0 || i == g.nx - 1, b1 = edge;
        const V *c = scc + I + g.cnx * (J + g.cny * K);
        V t0 = (V)0, t1 = (V)0;
        if (g.tet) {
            const V *e = c + g.cnx * (p1 + g.cny * p2);
            const bool odd = (p1 | p2) != 0;
            const V w0 = odd ? (b0 ? (V)0 : (V)0.5) : (V)1, w1 = b1 ? (V)0 : (V)0.5;
            const V c0 = c[0], e0 = e[0], e1 = e[I1];
            t0 = fma_rn(w0, c0, t0);
            if (odd) t0 = fma_rn(w0, e0, t0);
            t1 = fma_rn(w1, c0, t1);
            t1 = fma_rn(w1, e1, t1);
        } else {
            const V w0 = b0 ? ((p1 | p2) ? (V)0 : (V)1) : grid_weight<V>(p1 + p2);
            const V w1 = b1 ? (V)0 : grid_weight<V>(1 + p1 + p2);
            // the 1, 2 or 4 lines of coarse vertices around this line, in
            // increasing y, then z
            V a[4] = {}, b[4] = {};
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if ((m & 1) <= p1 && (m >> 1) <= p2) {
                    const V *e = c + g.cnx * ((m & 1) + g.cny * (m >> 1));
                    a[m] = e[0];
                    b[m] = e[I1];
                }
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if ((m & 1) <= p1 && (m >> 1) <= p2) {
                    t0 = fma_rn(w0, a[m], t0);
                    t1 = fma_rn(w1, a[m], t1);
                    t1 = fma_rn(w1, b[m], t1);
                }
        }
        if (g.dprol != 1.0) {
            t0 = mul_rn(t0, (V)g.dprol);
            t1 = mul_rn(t1, (V)g.dprol);
        }
        sc[f] = add_rn(s0, t0);
        if (w) w[f] = mul_rn(t0, df0);
        if (two) {
            sc[f + 1] = add_rn(s1, t1);
            if (w) w[f + 1] = mul_rn(t1, df1);
        }
    }
}

// The restriction runs in one of two thread layouts.  TILED: a 2D grid
// of 32 x 8 vertex tiles of the (x, y) plane, each thread walking z with the
// grid's z stride, so that a thread knows its grid indices without integer
// divisions by runtime extents (FP32 levels).
// Else one vertex per thread of a 1D grid-stride loop, every lane busy:
// FP64 levels are bound by the FP64 issue rate, where a partly filled warp
// costs as much as a full one.
template <class V, bool TILED>
__global__ void __launch_bounds__(NT) k_restrict_grid(GridPair g, const V *__restrict__ d, V *__restrict__ dc,
                                                      const int *skip)
{
    PDL_ENTRY();
    if (skip && *skip) return;
    if constexpr (TILED) {
        const int I = blockIdx.x * 32 + threadIdx.x, J = blockIdx.y * 8 + threadIdx.y;
        if (I >= g.cnx || J >= g.cny) return;
        for (int K = blockIdx.z; K < g.cnz; K += gridDim.z) restrict_row<V>(g, d, dc, I, J, K);
    } else {
        const int n = g.cnx * g.cny * g.cnz, stride = gridDim.x * NT;
        for (int c = blockIdx.x * NT + threadIdx.x; c < n; c += stride)
            restrict_row<V>(g, d, dc, c % g.cnx, (c / g.cnx) % g.cny, c / (g.cnx * g.cny));
    }
}

// grid of 32 x 8 tiles over (x, y) and enough z slices for about four
// resident waves of blocks
static dim3 transfer_grid(const Ctx &c, int nx, int ny, int nz)
{
    const unsigned gx = div_up(nx, 32), gy = div_up(ny, 8);
    int gz = (int)((size_t)c.num_sms * 8 * 4 / ((size_t)gx * gy));
    gz = gz < 1 ? 1 : (gz > nz ? nz : gz);
    return dim3(gx, gy, (unsigned)gz);
}

template <class V>
void prolong_grid(Ctx &c, const GridPair &g, const V *scc, V *sc, const V *dfac, V *w, const int *skip)
{
    const int per = (g.nx + 1) / 2, npairs = per * g.ny * g.nz;
    const int grid = sizeof(V) == 8 ? (int)div_up(npairs, NT) : row_grid(c, npairs);
    UG_LAUNCH_PDL(c, k_prolong_grid<V>, grid, NT, 0, g, FastDiv(per), FastDiv(g.ny), npairs, scc, sc,
                  dfac, w, skip);
}

template <class V>
void restrict_grid(Ctx &c, const GridPair &g, const V *d, V *dc, const int *skip)
{
    if constexpr (sizeof(V) == 4)
        UG_LAUNCH_PDL(c, (k_restrict_grid<V, true>), transfer_grid(c, g.cnx, g.cny, g.cnz), dim3(32, 8), 0, g, d, dc,
                      skip);
    else
        UG_LAUNCH_PDL(c, (k_restrict_grid<V, false>), row_grid(c, g.cnx * g.cny * g.cnz), NT, 0, g, d, dc, skip);
}
template void prolong_grid<double>(Ctx &, const GridPair &, const double *, double *, const double *, double *,
                                   const int *);
template void prolong_grid<float>(Ctx &, const GridPair &, const float *, float *, const float *, float *,
                                  const int *);
template void restrict_grid<double>(Ctx &, const GridPair &, const double *, double *, const int *);
template void restrict_grid<float>(Ctx &, const GridPair &, const float *, float *, const int *);

// dense base solve with the LU-factored inverse, FP64: one warp per row of
// Ainv, eight rows per block.  Each lane's first entries of its row are read
// before the launch wait (Ainv is set up once), the defect is staged in
// shared memory, and the row sum is a fixed-order warp reduction of the
// lanes' explicitly fused partial sums (the fused coarse cycle, k_coarse.cu,
// repeats them).
constexpr int kBaseRowsPerBlock = NT / 32;
constexpr int kBasePre = 8;   // entries per lane read before the wait (rows up to 256 wide)

template <class V>
__global__ void __launch_bounds__(NT) k_base_solve(const double *__restrict__ Ainv, int n, const V *__restrict__ d,
                                                   V *__restrict__ sc, const int *skip)
{
    extern __shared__ double dsh[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x * kBaseRowsPerBlock + warp;
    const double *arow = Ainv + (size_t)(row < n ? row : 0) * n;
    double a[kBasePre];
#pragma unroll
    for (int t = 0; t < kBasePre; ++t) {
        const int j = lane + 32 * t;
        a[t] = (row < n && j < n) ? __ldg(arow + j) : 0.0;
    }
    pdl_trigger();
    pdl_wait();
    if (skip && *skip) return;
    for (int j = threadIdx.x; j < n; j += blockDim.x) dsh[j] = (double)d[j];
    __syncthreads();
    if (row >= n) return;
    double s = 0.0;
#pragma unroll
    for (int t = 0; t < kBasePre; ++t) {
        const int j = lane + 32 * t;
        if (j < n) s = fma_rn(a[t], dsh[j], s);
    }
    for (int j = lane + 32 * kBasePre; j < n; j += 32) s = fma_rn(__ldg(arow + j), dsh[j], s);
    s = warp_sum(s);
    if (lane == 0) sc[row] = (V)s;
}

template <class V>
void base_solve(Ctx &c, const double *Ainv, int n, const V *d, V *sc, const int *skip)
{
    UG_LAUNCH_PDL(c, k_base_solve<V>, div_up(n, kBaseRowsPerBlock), NT, (size_t)n * sizeof(double), Ainv, n, d, sc,
                  skip);
}

// multicolour Gauss-Seidel: rows of one colour, t_i = relax (d_i - (A t)_i) / a_ii
// (t_i is still 0 when its colour is processed)
template <class MV, class V>
__global__ void __launch_bounds__(NT) k_mcgs(MV A, const int *__restrict__ rows, int nrows_c,
                                             const V *__restrict__ dr, const V *__restrict__ d, V *__restrict__ t,
                                             const int *skip)
{
    PDL_ENTRY();
    if (skip && *skip) return;
    const int stride = gridDim.x * NT;
    for (int q = blockIdx.x * NT + threadIdx.x; q < nrows_c; q += stride) {
        int row = rows[q];
        V acc = A.template dot<V>(t, row);
        // t_i += w/a_ii (d_i - (A t)_i): the forward sweep starts from t = 0,
        // the backward sweep of the symmetric smoother updates its result
        t[row] = t[row] + dr[row] * (d[row] - acc);
    }
}

template <class V>
void mcgs_colour(Ctx &c, const OpMat<V> &A, const int *rows, int nrows_c, const V *dinv_relax, const V *d, V *t,
                 const int *skip)
{
    with_mv(A, [&](auto mv) {
        UG_LAUNCH_PDL(c, (k_mcgs<decltype(mv), V>), row_grid(c, nrows_c), NT, 0, mv, rows, nrows_c, dinv_relax, d, t,
                  skip);
    });
}

// Two colours of a structured level in one launch: the lines (j, k) with the
// parities (b1, b2), whose vertices couple within a line and to lines of other
// parities only.  A block takes whole lines; a thread updates a vertex of
// the first colour (x parity first), then, behind a barrier, its neighbour of
// the second, so both halves of every sector of the operator are used while it
// is in the cache, and a sweep takes 4 launches (2D: 2) instead of 8.
// A sweep from t = 0 only reads the diagonals towards colours it has
// updated (mask_even / mask_odd: those of the two x parities): the others
// would multiply zeros, which leaves every sum as it is.
// The operator entries of the first colour are loaded before the launch wait.
// 97^3 hexes, FP32: eight launches of one colour each, with a pass that zeroed
// t, 54 us a sweep.
// Three blocks per SM: a wave then holds the whole level (461 us against 515 for
// the cycle; four blocks, 64 registers, spill: 551).
template <class V, int S>
__global__ void __launch_bounds__(NT, sizeof(V) == 4 ? 3 : 1)
    k_mcgs_lines(DiaMV<V, S> A, int nx, int ny, int b1, int b2, int nly, int nlines, int nz, int per, int per_block,
                 int first, unsigned mask_even, unsigned mask_odd, GsLines gs, bool from_zero,
                 const V *__restrict__ dr, const V *__restrict__ d, V *t, const int *skip)
{
    const int step = per < NT ? per : NT;   // vertices of a line (one x parity) that are in work at a time
    const int ln = threadIdx.x / step, q0 = threadIdx.x - ln * step;
    const int line = blockIdx.x * per_block + ln;
    const bool mine = ln < per_block && line < nlines;
    const int j = b1 + 2 * (line % nly), k = b2 + 2 * (line / nly), base = nx * (j + ny * k);
    unsigned off = 0u;   // the diagonals that leave the grid from this line
    if (j == 0) off |= gs.edge[2];
    if (j == ny - 1) off |= gs.edge[3];
    if (k == 0) off |= gs.edge[4];
    if (k == nz - 1) off |= gs.edge[5];
    auto inside = [&](int i, unsigned mask) {
        unsigned m = mask & ~off;
        if (i == 0) m &= ~gs.edge[0];
        if (i == nx - 1) m &= ~gs.edge[1];
        return m;
    };
    auto load = [&](int i, unsigned mask, V(&a)[S]) {
        mask = inside(i, mask);
#pragma unroll
        for (int e = 0; e < S; ++e)
            if ((mask >> e) & 1u) a[e] = __ldg(A.val + (size_t)e * A.ld + base + i);
    };
    auto update = [&](int i, unsigned mask, const V(&a)[S]) {
        const int row = base + i;
        mask = inside(i, mask);
        V x[S];
#pragma unroll
        for (int e = 0; e < S; ++e)
            if ((mask >> e) & 1u) x[e] = t[row + A.off.o[e]];
        V acc = (V)0;
#pragma unroll
        for (int e = 0; e < S; ++e)
            if ((mask >> e) & 1u) acc = fma_rn(a[e], x[e], acc);
        const V old = from_zero ? (V)0 : t[row];
        t[row] = fma_rn(dr[row], sub_rn(d[row], acc), old);
    };
    V a[S];
    const unsigned m0 = first ? mask_odd : mask_even, m1 = first ? mask_even : mask_odd;
    const int i0 = 2 * q0 + first;
    pdl_trigger();
    if (mine && i0 < nx) load(i0, m0, a);
    pdl_wait();
    if (skip && *skip) return;
    if (mine)
        for (int q = q0; q < per; q += step) {
            const int i = 2 * q + first;
            if (i >= nx) break;
            if (q != q0) load(i, m0, a);
            update(i, m0, a);
        }
    const int i1 = 2 * q0 + 1 - first;
    if (mine && i1 < nx) load(i1, m1, a);
    __syncthreads();
    if (mine)
        for (int q = q0; q < per; q += step) {
            const int i = 2 * q + 1 - first;
            if (i >= nx) break;
            if (q != q0) load(i, m1, a);
            update(i, m1, a);
        }
}

// vertices of one x parity in a line, lines per block
static int line_half(const GridPair &gp) { return (gp.nx + 1) / 2; }
static int lines_per_block(const GridPair &gp) { return line_half(gp) < NT ? NT / line_half(gp) : 1; }

// A block takes a line of more than 2 NT vertices in several rounds, one after the
// other; with few such lines most of the GPU is idle, where a launch per colour
// fills it.  Up to three rounds, or with 32 blocks per round, the lines are faster.
// Cycles with the top level by lines, against by colours (forward / symmetric sweeps):
// FP32 1025 x 257 quads, 3 rounds, 128 blocks 0.95 / 0.93; 2049 x 257, 5 rounds 0.99 /
// 1.01; 4097 x 257, 9 rounds - / 1.08; 12545 x 257, 25 rounds - / 1.26; 2049 x 33 x 33
// hexes, 5 rounds, 256 blocks 0.87 / 0.91; 2049 x 17 x 17, 64 blocks - / 1.07; 4097^2
// quads, 9 rounds, 2048 blocks 0.78 / 0.82 (FP64 0.87 / 0.93).
// FP64 rounds of 15 and 27 diagonals take 2 us of an SM's FP64 pipe and hold a row's
// entries in registers, at one or two blocks per SM.  With fewer than four blocks one
// round is the limit (1025 x 3 x 3 hexes below 4097 x 9 x 9: a cycle 895 us with three
// rounds, 833 with one, 816 by colours), and on large levels the colours' full
// occupancy is faster: 65^3 hexes 0.84 / 0.81, 513 x 33 x 33 0.97 / 0.97, 769 x 33 x 33
// 1.03 / 1.03, 97^3 1.00 / 1.02, 129^3 1.07 / 1.14.
static bool lines_fill(const GridPair &gp, bool fp64_bound)
{
    constexpr int64_t kFp64Rows = 700000;
    if (fp64_bound && (int64_t)gp.nx * gp.ny * gp.nz > kFp64Rows) return false;
    const int rounds = (int)div_up(line_half(gp), NT);
    const int lines = (gp.ny / 2) * (gp.dim == 3 ? gp.nz / 2 : 1);   // of the smallest set
    const int blocks = (int)div_up(lines, lines_per_block(gp));
    if (rounds <= 1) return true;
    if (rounds <= 3) return !fp64_bound || blocks >= 4;
    return blocks >= 32 * rounds;
}

GsLines gs_lines(bool fp64, const Offs &offs, int S, const std::vector<int> &entries, const GridPair &gp)
{
    GsLines g;
    if (gp.nx < 3 || gp.ny < 3 || S > 32 || !lines_fill(gp, fp64 && S >= 15)) return g;
    for (int k = 0; k < S; ++k) {
        const int o = offs.o[k];
        if (!std::binary_search(entries.begin(), entries.end(), o)) continue;
        int pm = -1;   // parity bits that differ along this offset
        for (int z = gp.dim == 3 ? -1 : 0; z <= (gp.dim == 3 ? 1 : 0); ++z)
            for (int y = -1; y <= 1; ++y)
                for (int x = -1; x <= 1; ++x)
                    if (x + gp.nx * (y + gp.ny * z) == o) {
                        pm = (x & 1) | ((y & 1) << 1) | ((z & 1) << 2);
                        if (x) g.edge[x > 0 ? 1 : 0] |= 1u << k;
                        if (y) g.edge[y > 0 ? 3 : 2] |= 1u << k;
                        if (z) g.edge[z > 0 ? 5 : 4] |= 1u << k;
                    }
        if (pm < 0) return g;
        g.all |= 1u << k;
        for (int c = 0; c < 8; ++c) {
            if ((c ^ pm) < c) g.below[c] |= 1u << k;
            if ((c ^ pm) > c) g.above[c] |= 1u << k;
        }
    }
    g.usable = true;
    return g;
}

template <class V>
void mcgs_sweep_lines(Ctx &c, const OpMat<V> &A, const GsLines &gs, const GridPair &gp, bool backward, bool from_zero,
                      const V *dinv_relax, const V *d, V *t, const int *skip)
{
    with_mv(A, [&](auto mv) {
        using MV = decltype(mv);
        if constexpr (is_dia<MV>::value) {
            const int np = gp.dim == 3 ? 4 : 2, per = line_half(gp), per_block = lines_per_block(gp);
            for (int s = 0; s < np; ++s) {
                const int p = backward ? np - 1 - s : s, b1 = p & 1, b2 = p >> 1;
                const int nly = (gp.ny - b1 + 1) / 2, nlz = gp.dim == 3 ? (gp.nz - b2 + 1) / 2 : 1;
                const int nlines = nly * nlz;
                if (nlines <= 0) continue;
                const unsigned *m = backward ? gs.above : gs.below;
                const unsigned even = from_zero ? m[2 * p] : gs.all, odd = from_zero ? m[2 * p + 1] : gs.all;
                UG_LAUNCH_PDL(c, (k_mcgs_lines<V, MV::kS>), div_up(nlines, per_block), NT, 0, mv, gp.nx, gp.ny, b1, b2,
                              nly, nlines, gp.nz, per, per_block, backward ? 1 : 0, even, odd, gs, from_zero,
                              dinv_relax, d, t, skip);
            }
        } else {
            throw Error{UG4GB_ERR_INVALID, "Gauss-Seidel by lines: not a diagonal layout"};
        }
    });
}
template void mcgs_sweep_lines<double>(Ctx &, const OpMat<double> &, const GsLines &, const GridPair &, bool, bool,
                                       const double *, const double *, double *, const int *);
template void mcgs_sweep_lines<float>(Ctx &, const OpMat<float> &, const GsLines &, const GridPair &, bool, bool,
                                      const float *, const float *, float *, const int *);

template <class MV, class V, class DT>
__global__ void __launch_bounds__(NT) k_resupd(MV A, const V *__restrict__ t, const DT *__restrict__ dbase,
                                               V *__restrict__ dout, V *__restrict__ sc, int sc_mode, const int *skip)
{
    PDL_ENTRY();
    if (skip && *skip) return;
    const int stride = gridDim.x * NT, n = A.rows();
    for (int row = blockIdx.x * NT + threadIdx.x; row < n; row += stride) {
        V acc = A.template dot<V>(t, row);
        dout[row] = (V)dbase[row] - acc;
        if (sc_mode == 1) sc[row] = t[row];
        else if (sc_mode == 0) sc[row] += t[row];
    }
}

template <class V, class DT>
void residual_update(Ctx &c, const OpMat<V> &A, const V *t, const DT *dbase, V *dout, V *sc, int sc_mode,
                     const int *skip)
{
    with_mv(A, [&](auto mv) {
        UG_LAUNCH_PDL(c, (k_resupd<decltype(mv), V, DT>), row_grid(c, A.nrows), NT, 0, mv, t, dbase, dout, sc, sc_mode,
                  skip);
    });
}

template void restrict_apply<double>(Ctx &, const OpMat<double> &, const double *, double *, const int *);
template void restrict_apply<float>(Ctx &, const OpMat<float> &, const float *, float *, const int *);
template void prolong_apply<double>(Ctx &, const OpMat<double> &, const double *, double *, const double *, double *,
                                    const int *);
template void prolong_apply<float>(Ctx &, const OpMat<float> &, const float *, float *, const float *, float *,
                                   const int *);
template void base_solve<double>(Ctx &, const double *, int, const double *, double *, const int *);
template void base_solve<float>(Ctx &, const double *, int, const float *, float *, const int *);
template void mcgs_colour<double>(Ctx &, const OpMat<double> &, const int *, int, const double *, const double *,
                                  double *, const int *);
template void mcgs_colour<float>(Ctx &, const OpMat<float> &, const int *, int, const float *, const float *, float *,
                                 const int *);
template void residual_update<double, double>(Ctx &, const OpMat<double> &, const double *, const double *, double *,
                                              double *, int, const int *);
template void residual_update<float, float>(Ctx &, const OpMat<float> &, const float *, const float *, float *,
                                            float *, int, const int *);
template void residual_update<float, double>(Ctx &, const OpMat<float> &, const float *, const double *, float *,
                                             float *, int, const int *);

// ------------------------------------------------------------ Krylov -----
// (BiCGStab::apply_return_defect, bicgstab.h:158-390).  A restart at the top
// of an iteration comes from the previous iteration's orthogonality test
// (ks->restart) or from the fixed restart period (step % num_restarts == 0,
// bicgstab.h:161-170; the check counts half steps).
__device__ __forceinline__ bool bicg_restarting(const KScal *ks)
{
    return ks->restart || (ks->num_restarts > 0 && ks->step % ks->num_restarts == 0);
}

// The scalars at the top of an iteration from r0r = (r0, r) and rr = (r, r),
// called by the kernel that wrote r (there is no pass of its own over r0 and
// r for them): rho, beta, whether this iteration restarts (k_bicg_p then
// sets r0 = p = r, so (r0, r) is (r, r)).
__device__ __forceinline__ void bicg_top(KScal *ks, double r0r, double rr)
{
    if (ks->done) return;
    const bool again = bicg_restarting(ks);
    ks->restarted = again ? 1 : 0;
    if (again) {
        ks->alpha = 0.0;
        ks->omega = 1.0;
        ks->rho = 1.0;
        ks->norm_r0 = ks->dcur;
        ks->restart = 0;
    }
    const double tot = again ? rr : r0r;
    const double rho_old = ks->rho;
    ks->rho_old = rho_old;
    ks->rho = tot;
    // restart in the next iteration when (r, r0) <= minOrtho |r| |r0|
    // (bicgstab.h:206-215)
    if (fabs(tot) / (ks->dcur * ks->norm_r0) <= ks->min_ortho) ks->restart = 1;
    if (rho_old == 0.0) {
        ks->fail = 1;
        ks->done = 1;
    }
    ks->beta = (tot / rho_old) * (ks->alpha / ks->omega);
}

// r = b - A x (r holds b on entry); start the convergence check with |r|;
// bicg: and BiCGStab's first iteration, which restarts
template <class MV>
__global__ void __launch_bounds__(NT) k_krylov_start(MV A, const double *__restrict__ x, double *__restrict__ r,
                                                     float *__restrict__ r32, bool bicg, RedArgs red)
{
    PDL_ENTRY();
    double sum = 0.0;
    const int stride = gridDim.x * NT, n = A.rows();
    for (int row = blockIdx.x * NT + threadIdx.x; row < n; row += stride) {
        double ax = A.template dot<double>(x, row);
        double rv = r[row] - ax;
        r[row] = rv;
        if (r32) r32[row] = f64_to_f32(rv);
        sum += rv * rv;
    }
    double v[1] = {sum};
    KScal *ks = red.ks;
    grid_reduce<NT, 1>(v, red.partials, red.counter, [&](const double(&tot)[1]) {
        double d = sqrt(tot[0]);
        ks->d0 = d;
        ks->dcur = d;
        ks->step = 0;
        ks->done = 0;
        ks->fail = 0;
        ks->restart = 1;
        if (ks->hist && ks->hist_cap > 0) ks->hist[0] = d;
        if (conv_ended(ks)) ks->done = 1;
        if (bicg) bicg_top(ks, tot[0], tot[0]);
    });
}

void krylov_start(Ctx &c, const OpMat<double> &A, const double *x, double *r, RedArgs red, float *r32, bool bicg)
{
    with_mv(A, [&](auto mv) {
        const int g = spmv_grid<decltype(mv), double>(c, A.nrows, true);
        UG_LAUNCH_PDL(c, k_krylov_start<decltype(mv)>, g, NT, 0, mv, x, r, r32, bicg, red);
    });
}

// first: p = z, q = A z ; else p = z + beta p, q = A z + beta q ; lambda = (q,p)
template <class MV, class ZT>
__global__ void __launch_bounds__(NT) k_cg_spmv_dot(MV A, const ZT *__restrict__ z, double *__restrict__ p,
                                                    double *__restrict__ q, int first, RedArgs red)
{
    PDL_ENTRY();
    KScal *ks = red.ks;
    if (ks->done) return;
    const double beta = first ? 0.0 : ks->beta;
    double sum = 0.0;
    const int stride = gridDim.x * NT, n = A.rows();
    for (int row = blockIdx.x * NT + threadIdx.x; row < n; row += stride) {
        double az = A.template dot<double>(z, row);
        double pn = first ? (double)z[row] : (double)z[row] + beta * p[row];
        double qn = first ? az : az + beta * q[row];
        p[row] = pn;
        q[row] = qn;
        sum += qn * pn;
    }
    double v[1] = {sum};
    grid_reduce<NT, 1>(v, red.partials, red.counter, [&](const double(&tot)[1]) {
        ks->lambda = tot[0];
        if (tot[0] == 0.0) {
            ks->fail = 1;
            ks->done = 1;
        }
        ks->alpha = ks->rho_old / tot[0];
    });
}

template <class ZT>
void cg_spmv_dot_t(Ctx &c, const OpMat<double> &A, const ZT *z, double *p, double *q, int first, RedArgs red)
{
    with_mv(A, [&](auto mv) {
        const int g = spmv_grid<decltype(mv), double>(c, A.nrows, true);
        UG_LAUNCH_PDL(c, (k_cg_spmv_dot<decltype(mv), ZT>), g, NT, 0, mv, z, p, q, first, red);
    });
}
template void cg_spmv_dot_t<double>(Ctx &, const OpMat<double> &, const double *, double *, double *, int, RedArgs);
template void cg_spmv_dot_t<float>(Ctx &, const OpMat<double> &, const float *, double *, double *, int, RedArgs);

// x += alpha p ; r -= alpha q ; |r| -> convergence check; optionally
// r32 = (float) r, the FP32 defect the mixed-precision multigrid starts from.
// Two entries per thread with 16-byte accesses (all pointers 16-byte
// aligned; the odd last entry alone).
__global__ void __launch_bounds__(NT) k_cg_update(int n, double *__restrict__ x, double *__restrict__ r,
                                                  const double *__restrict__ p, const double *__restrict__ q,
                                                  float *__restrict__ r32, RedArgs red)
{
    PDL_ENTRY();
    KScal *ks = red.ks;
    if (ks->done) return;
    const double alpha = ks->alpha;
    double sum = 0.0;
    const int stride = gridDim.x * NT, npair = (n + 1) / 2;
    for (int k = blockIdx.x * NT + threadIdx.x; k < npair; k += stride) {
        const int i = 2 * k;
        if (i + 1 < n) {
            Pack<double, 2> xv = ld_pack<double, 2>(x + i), pv = ld_pack<double, 2>(p + i);
            Pack<double, 2> rv = ld_pack<double, 2>(r + i), qv = ld_pack<double, 2>(q + i);
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                xv.v[e] = xv.v[e] + alpha * pv.v[e];
                rv.v[e] = rv.v[e] + (-alpha) * qv.v[e];
                sum += rv.v[e] * rv.v[e];
            }
            st_pack<double, 2>(x + i, xv);
            st_pack<double, 2>(r + i, rv);
            if (r32) {
                float2 f = make_float2(f64_to_f32(rv.v[0]), f64_to_f32(rv.v[1]));
                *reinterpret_cast<float2 *>(r32 + i) = f;
            }
        } else {
            x[i] = x[i] + alpha * p[i];
            double rv = r[i] + (-alpha) * q[i];
            r[i] = rv;
            sum += rv * rv;
            if (r32) r32[i] = f64_to_f32(rv);
        }
    }
    double v[1] = {sum};
    grid_reduce<NT, 1>(v, red.partials, red.counter, [&](const double(&tot)[1]) { conv_update(ks, sqrt(tot[0]), 1); });
}

// the same one entry per thread (pointers not 16-byte aligned)
__global__ void __launch_bounds__(NT) k_cg_update1(int n, double *__restrict__ x, double *__restrict__ r,
                                                   const double *__restrict__ p, const double *__restrict__ q,
                                                   float *__restrict__ r32, RedArgs red)
{
    PDL_ENTRY();
    KScal *ks = red.ks;
    if (ks->done) return;
    const double alpha = ks->alpha;
    double sum = 0.0;
    const int stride = gridDim.x * NT;
    for (int i = blockIdx.x * NT + threadIdx.x; i < n; i += stride) {
        x[i] = x[i] + alpha * p[i];
        double rv = r[i] + (-alpha) * q[i];
        r[i] = rv;
        sum += rv * rv;
        if (r32) r32[i] = f64_to_f32(rv);
    }
    double v[1] = {sum};
    grid_reduce<NT, 1>(v, red.partials, red.counter, [&](const double(&tot)[1]) { conv_update(ks, sqrt(tot[0]), 1); });
}

static inline bool al16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

void cg_update(Ctx &c, int n, double *x, double *r, const double *p, const double *q, RedArgs red, float *r32)
{
    if (al16(x) && al16(r) && al16(p) && al16(q) && (!r32 || ((uintptr_t)r32 & 7u) == 0))
        UG_LAUNCH_PDL(c, k_cg_update, row_grid(c, (n + 1) / 2), NT, 0, n, x, r, p, q, r32, red);
    else
        UG_LAUNCH_PDL(c, k_cg_update1, row_grid(c, n), NT, 0, n, x, r, p, q, r32, red);
}

// rho = (z, r) when the preconditioner could not fuse it (kind 0: first, 1: loop)
template <class ZT>
__global__ void __launch_bounds__(NT) k_rho(int n, const ZT *__restrict__ z, const double *__restrict__ r, int kind,
                                            RedArgs red)
{
    PDL_ENTRY();
    KScal *ks = red.ks;
    if (ks->done) return;
    double sum = 0.0;
    const int stride = gridDim.x * NT;
    for (int i = blockIdx.x * NT + threadIdx.x; i < n; i += stride) sum += (double)z[i] * r[i];
    double v[1] = {sum};
    grid_reduce<NT, 1>(v, red.partials, red.counter, [&](const double(&tot)[1]) {
        if (kind == 0) {
            ks->rho_old = tot[0];
        } else {
            ks->rho = tot[0];
            ks->beta = tot[0] / ks->rho_old;
            ks->rho_old = tot[0];
        }
    });
}

template <class ZT>
void rho_dot(Ctx &c, int n, const ZT *z, const double *r, int kind, RedArgs red)
{
    UG_LAUNCH_PDL(c, k_rho<ZT>, row_grid(c, n), NT, 0, n, z, r, kind, red);
}
template void rho_dot<double>(Ctx &, int, const double *, const double *, int, RedArgs);
template void rho_dot<float>(Ctx &, int, const float *, const double *, int, RedArgs);

template <class ZT>
__global__ void k_copy_z(int n, const ZT *__restrict__ z, double *__restrict__ out, const int *skip)
{
    PDL_ENTRY();
    if (skip && *skip) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = f32_to_f64_t(z[i]);
}

template <class ZT>
void copy_z(Ctx &c, int n, const ZT *z, double *out, const int *skip)
{
    UG_LAUNCH_PDL(c, k_copy_z<ZT>, div_up(n, NT), NT, 0, n, z, out, skip);
}
template void copy_z<double>(Ctx &, int, const double *, double *, const int *);
template void copy_z<float>(Ctx &, int, const float *, double *, const int *);

// ------------------------------------------------------------ BiCGStab ---
// p = r + beta p - beta omega v; a restart: r0 = p = r.  Optionally p32 =
// (float) p, the FP32 defect the mixed-precision multigrid starts from.
__global__ void __launch_bounds__(NT) k_bicg_p(int n, const double *__restrict__ r, double *__restrict__ p,
                                               const double *__restrict__ v, double *__restrict__ r0,
                                               float *__restrict__ p32, const KScal *ks)
{
    PDL_ENTRY();
    if (ks->done) return;
    const bool again = ks->restarted != 0;
    const double beta = ks->beta, bo = -ks->beta * ks->omega;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double rv = r[i];
    const double pv = again ? rv : 1.0 * rv + beta * p[i] + bo * v[i];
    p[i] = pv;
    if (again) r0[i] = rv;
    if (p32) p32[i] = f64_to_f32(pv);
}

void bicg_p(Ctx &c, int n, const double *r, double *p, const double *v, double *r0, float *p32, RedArgs red)
{
    UG_LAUNCH_PDL(c, k_bicg_p, div_up(n, NT), NT, 0, n, r, p, v, r0, p32, red.ks);
}

template <class MV, class ZT>
__global__ void __launch_bounds__(NT) k_bicg_spmv_dot(MV A, const ZT *__restrict__ q, double *__restrict__ v,
                                                      const double *__restrict__ r0, RedArgs red)
{
    PDL_ENTRY();
    KScal *ks = red.ks;
    if (ks->done) return;
    double sum = 0.0;
    const int stride = gridDim.x * NT, n = A.rows();
    for (int row = blockIdx.x * NT + threadIdx.x; row < n; row += stride) {
        double av = A.template dot<double>(q, row);
        v[row] = av;
        sum += av * r0[row];
    }
    double vv[1] = {sum};
    grid_reduce<NT, 1>(vv, red.partials, red.counter, [&](const double(&tot)[1]) {
        if (tot[0] == 0.0) {
            ks->fail = 1;
            ks->done = 1;
        }
        ks->alpha = ks->rho / tot[0];
    });
}

template <class ZT>
void bicg_spmv_dot_t(Ctx &c, const OpMat<double> &A, const ZT *q, double *v, const double *r0, RedArgs red)
{
    with_mv(A, [&](auto mv) {
        const int g = spmv_grid<decltype(mv), double>(c, A.nrows, true);
        UG_LAUNCH_PDL(c, (k_bicg_spmv_dot<decltype(mv), ZT>), g, NT, 0, mv, q, v, r0, red);
    });
}
template void bicg_spmv_dot_t<double>(Ctx &, const OpMat<double> &, const double *, double *, const double *, RedArgs);
template void bicg_spmv_dot_t<float>(Ctx &, const OpMat<double> &, const float *, double *, const double *, RedArgs);

// x += alpha q ; s = r - alpha v ; |s| -> check; optionally s32 = (float) s
template <class ZT>
__global__ void __launch_bounds__(NT) k_bicg_x_s(int n, double *__restrict__ x, const ZT *__restrict__ q,
                                                 const double *__restrict__ r, const double *__restrict__ v,
                                                 double *__restrict__ s, float *__restrict__ s32, RedArgs red)
{
    PDL_ENTRY();
    KScal *ks = red.ks;
    if (ks->done) return;
    const double alpha = ks->alpha;
    double sum = 0.0;
    const int stride = gridDim.x * NT;
    for (int i = blockIdx.x * NT + threadIdx.x; i < n; i += stride) {
        x[i] = 1.0 * x[i] + alpha * (double)q[i];
        double sv = 1.0 * r[i] + (-alpha) * v[i];
        s[i] = sv;
        if (s32) s32[i] = f64_to_f32(sv);
        sum += sv * sv;
    }
    double vv[1] = {sum};
    grid_reduce<NT, 1>(vv, red.partials, red.counter, [&](const double(&tot)[1]) { conv_update(ks, sqrt(tot[0]), 2); });
}

template <class ZT>
void bicg_x_s(Ctx &c, int n, double *x, const ZT *q, const double *r, const double *v, double *s, float *s32,
              RedArgs red)
{
    UG_LAUNCH_PDL(c, k_bicg_x_s<ZT>, row_grid(c, n), NT, 0, n, x, q, r, v, s, s32, red);
}
template void bicg_x_s<double>(Ctx &, int, double *, const double *, const double *, const double *, double *, float *,
                               RedArgs);
template void bicg_x_s<float>(Ctx &, int, double *, const float *, const double *, const double *, double *, float *,
                              RedArgs);

// after the loop: a solve that ended at a half step returns s as the defect
__global__ void k_bicg_s_to_r(int n, const double *__restrict__ s, double *__restrict__ r, const KScal *ks)
{
    PDL_ENTRY();
    if (ks->done != 2) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) r[i] = s[i];
}

void bicg_s_to_r(Ctx &c, int n, const double *s, double *r, RedArgs red)
{
    UG_LAUNCH(c, k_bicg_s_to_r, div_up(n, NT), NT, 0, n, s, r, red.ks);
}

template <class MV, class ZT>
__global__ void __launch_bounds__(NT) k_bicg_spmv_2dot(MV A, const ZT *__restrict__ q, double *__restrict__ t,
                                                       const double *__restrict__ s, RedArgs red)
{
    PDL_ENTRY();
    KScal *ks = red.ks;
    if (ks->done) return;
    double tt = 0.0, st = 0.0;
    const int stride = gridDim.x * NT, n = A.rows();
    for (int row = blockIdx.x * NT + threadIdx.x; row < n; row += stride) {
        double av = A.template dot<double>(q, row);
        t[row] = av;
        tt += av * av;
        st += s[row] * av;
    }
    double vv[2] = {tt, st};
    grid_reduce<NT, 2>(vv, red.partials, red.counter, [&](const double(&tot)[2]) {
        if (tot[0] == 0.0) {
            ks->fail = 1;
            ks->done = 1;
        }
        ks->omega = tot[1] / tot[0];
    });
}

template <class ZT>
void bicg_spmv_2dot_t(Ctx &c, const OpMat<double> &A, const ZT *q, double *t, const double *s, RedArgs red)
{
    with_mv(A, [&](auto mv) {
        const int g = spmv_grid<decltype(mv), double>(c, A.nrows, true);
        UG_LAUNCH_PDL(c, (k_bicg_spmv_2dot<decltype(mv), ZT>), g, NT, 0, mv, q, t, s, red);
    });
}
template void bicg_spmv_2dot_t<double>(Ctx &, const OpMat<double> &, const double *, double *, const double *,
                                       RedArgs);
template void bicg_spmv_2dot_t<float>(Ctx &, const OpMat<double> &, const float *, double *, const double *, RedArgs);

// x += omega q ; r = s - omega t ; |r| -> check, and (r0, r) for the next
// iteration (bicg_top)
template <class ZT>
__global__ void __launch_bounds__(NT) k_bicg_x_r(int n, double *__restrict__ x, const ZT *__restrict__ q,
                                                 const double *__restrict__ s, const double *__restrict__ t,
                                                 double *__restrict__ r, const double *__restrict__ r0, RedArgs red)
{
    PDL_ENTRY();
    KScal *ks = red.ks;
    if (ks->done) return;
    const double omega = ks->omega;
    double sum = 0.0, r0r = 0.0;
    const int stride = gridDim.x * NT;
    for (int i = blockIdx.x * NT + threadIdx.x; i < n; i += stride) {
        x[i] = 1.0 * x[i] + omega * (double)q[i];
        double rv = 1.0 * s[i] + (-omega) * t[i];
        r[i] = rv;
        sum += rv * rv;
        r0r += r0[i] * rv;
    }
    double vv[2] = {sum, r0r};
    grid_reduce<NT, 2>(vv, red.partials, red.counter, [&](const double(&tot)[2]) {
        conv_update(ks, sqrt(tot[0]), 1);
        if (ks->omega == 0.0) {
            ks->fail = 1;
            ks->done = 1;
        }
        bicg_top(ks, tot[1], tot[0]);
    });
}

template <class ZT>
void bicg_x_r(Ctx &c, int n, double *x, const ZT *q, const double *s, const double *t, double *r, const double *r0,
              RedArgs red)
{
    UG_LAUNCH_PDL(c, k_bicg_x_r<ZT>, row_grid(c, n), NT, 0, n, x, q, s, t, r, r0, red);
}
template void bicg_x_r<double>(Ctx &, int, double *, const double *, const double *, const double *, double *,
                               const double *, RedArgs);
template void bicg_x_r<float>(Ctx &, int, double *, const float *, const double *, const double *, double *,
                              const double *, RedArgs);

// ------------------------------------------------------ vector/matrix API --
__global__ void __launch_bounds__(NT) k_vec_dot(int n, const double *__restrict__ a, const double *__restrict__ b,
                                                RedArgs red)
{
    PDL_ENTRY();
    double sum = 0.0;
    const int stride = gridDim.x * NT;
    for (int i = blockIdx.x * NT + threadIdx.x; i < n; i += stride) sum += a[i] * b[i];
    double v[1] = {sum};
    KScal *ks = red.ks;
    grid_reduce<NT, 1>(v, red.partials, red.counter, [&](const double(&tot)[1]) { ks->dot_out[0] = tot[0]; });
}

void vec_dot(Ctx &c, int n, const double *a, const double *b, RedArgs red)
{
    UG_LAUNCH_PDL(c, k_vec_dot, row_grid(c, n), NT, 0, n, a, b, red);
}

__global__ void k_vec_scale_add(int n, double *dest, double alpha, const double *a, double beta, const double *b)
{
    PDL_ENTRY();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dest[i] = alpha * a[i] + beta * b[i];
}

void vec_scale_add(Ctx &c, int n, double *dest, double alpha, const double *a, double beta, const double *b)
{
    UG_LAUNCH_PDL(c, k_vec_scale_add, div_up(n, NT), NT, 0, n, dest, alpha, a, beta, b);
}

// dest = alpha*v1 + beta*A*w1 (SparseMatrix::axpy, sparsematrix_impl.h:294-342)
template <class MV>
__global__ void __launch_bounds__(NT) k_op_axpy(MV A, double *dest, double alpha, const double *v1, double beta,
                                                const double *__restrict__ w1)
{
    PDL_ENTRY();
    const int stride = gridDim.x * NT, n = A.rows();
    for (int row = blockIdx.x * NT + threadIdx.x; row < n; row += stride) {
        double aw = A.template dot<double>(w1, row);
        dest[row] = (alpha == 0.0 ? 0.0 : alpha * v1[row]) + beta * aw;
    }
}

void op_axpy(Ctx &c, const OpMat<double> &A, double *dest, double alpha, const double *v1, double beta,
             const double *w1)
{
    with_mv(A, [&](auto mv) {
        const int g = spmv_grid<decltype(mv), double>(c, A.nrows, false);
        UG_LAUNCH_PDL(c, k_op_axpy<decltype(mv)>, g, NT, 0, mv, dest, alpha, v1, beta, w1);
    });
}

// dest += beta * A^T w1 (atomics; API path only)
__global__ void k_csr_axpy_t(int nrows, const int *rowptr, const int *col, const double *val, double *dest,
                             double beta, const double *w1)
{
    PDL_ENTRY();
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrows) return;
    double wr = beta * w1[r];
    for (int a = rowptr[r]; a < rowptr[r + 1]; ++a)
        if (val[a] != 0.0) atomicAdd(dest + col[a], val[a] * wr);
}

void csr_axpy_transposed(Ctx &c, const Csr &A, double *dest, double beta, const double *w1)
{
    UG_LAUNCH_PDL(c, k_csr_axpy_t, div_up(A.nrows, NT), NT, 0, A.nrows, A.rowptr.p, A.col.p, A.val.p, dest, beta, w1);
}

template <class TO, class TI>
__global__ void k_convert(int n, const TI *in, TO *out)
{
    PDL_ENTRY();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (TO)in[i];
}

template <class TO, class TI>
void convert(Ctx &c, int n, const TI *in, TO *out)
{
    UG_LAUNCH_PDL(c, (k_convert<TO, TI>), div_up(n, NT), NT, 0, n, in, out);
}
template void convert<float, double>(Ctx &, int, const double *, float *);
template void convert<double, float>(Ctx &, int, const float *, double *);
template void convert<double, double>(Ctx &, int, const double *, double *);

}  // namespace ug4gb
