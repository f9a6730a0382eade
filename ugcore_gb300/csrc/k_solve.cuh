// k_solve.cuh -- device-side state of the Krylov solvers and the launch
// wrappers of the multigrid / Krylov kernels (implemented in k_solve.cu).
// Every operator argument is an OpMat (SELL-32 or diagonal layout); the
// wrappers dispatch to the kernel instantiated for that layout.
#pragma once

#include <memory>

#include "common.cuh"

namespace ug4gb {

// Scalars of one Krylov solve, resident in device memory.  The finishing
// block of each reduction updates them, so no host round trip is needed
// between kernels.  Convergence follows StdConvCheck
// (lib_algebra/operator/convergence_check_impl.h:85-172).
struct KScal {
    int step, done, fail, restart;
    int restarted;                              // BiCGStab: this iteration set r0 = r
    int maxit, hist_cap;
    double min_def, rel_red;
    double d0, dcur;
    double rho, rho_old, alpha, beta, lambda;   // CG
    double omega, norm_r0;                      // BiCGStab
    int num_restarts;                           // BiCGStab::set_restart (0: off)
    double min_ortho;                           // BiCGStab::set_min_orthogonality
    double dot_out[2];                          // plain reductions
    double *hist;                               // hist_cap entries
};

enum ScMode { SC_SET_FROM_BASE = 0, SC_ADD_FROM_BASE = 1, SC_ADD_FROM_NEW = 2 };

// Explicitly rounded arithmetic of the smoothing and transfer row updates.
// Every kernel that applies a damped-Jacobi step (one step per launch, or two
// fused) or the prolongation goes through these, so the compiler cannot
// contract them differently in different kernels: the results of all
// variants are bit-identical.
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }

// One damped-Jacobi row update after the row's SpMV value acc = (At x)_i:
// dn = db - acc; t = dinv * (dn or db); sc (=|+=) t.  Returns dn; sc is
// updated in place (sc_in is only read when the mode adds).
template <class V>
__device__ __forceinline__ V jacobi_row(V acc, V db, V dinv, int mode, V sc_in, V &sc_out)
{
    const V dn = sub_rn(db, acc);
    const V t = mul_rn(dinv, mode == SC_ADD_FROM_NEW ? dn : db);
    sc_out = (mode == SC_SET_FROM_BASE) ? t : add_rn(sc_in, t);
    return dn;
}

// Sum of a row's S products on a level small enough that latency rules
// (k_smooth with its row loaded ahead, the coarse cycle).  FP32: the one FMA
// chain of the other kernels.  A dependent FP64 FMA takes some 130 cycles on
// GB300, twice what its issue does: FP64 rows go in two chains, the lower
// offsets and the rest (so that symmetric layouts of one matrix, with and
// without its zero diagonals, sum the same terms), added at the end.
template <class V, int S>
__device__ __forceinline__ V row_sum(const V (&a)[S], const V (&x)[S])
{
    if constexpr (sizeof(V) == 4) {
        V acc = (V)0;
#pragma unroll
        for (int k = 0; k < S; ++k) acc = fma_rn(a[k], x[k], acc);
        return acc;
    } else {
        V lo = (V)0, hi = (V)0;
#pragma unroll
        for (int k = 0; k < S / 2; ++k) lo = fma_rn(a[k], x[k], lo);
#pragma unroll
        for (int k = S / 2; k < S; ++k) hi = fma_rn(a[k], x[k], hi);
        return add_rn(lo, hi);
    }
}

struct RedArgs {
    double *partials;
    unsigned int *counter;
    KScal *ks;
};

// grid size used by every row-parallel kernel (grid-stride loops)
int row_grid(const Ctx &c, int nrows);

// ---- multigrid level kernels (V = level precision) ----
// dnew = dbase - At*x ; sc (=|+=) dinv*(dbase|dnew) ; optional dout = dnew;
// optional rho = sum sc_i * r_i (final top-level step inside a Krylov solve);
// optional z64 = (double) sc (mixed precision: FP64 correction for the Krylov loop)
template <class V, class XT, class DT>
void smooth_step(Ctx &c, const OpMat<V> &At, const XT *x, const DT *dbase, const V *dinv, V *sc, V *dout,
                 int sc_mode, const int *skip, const double *r_rho, RedArgs *red, int rho_kind,
                 double *z64 = nullptr);
struct GridPair;
// The operator of a structured 3D FP32 level prepared for smooth_pair: a copy
// with 16-byte aligned grid lines and its TMA tensor descriptor (k_sweep2.cu).
struct Sweep2Op;
// Set-up (may synchronise): null unless At is a 15- or 27-diagonal FP32
// operator of the structured level gp (nx, ny, nz) with the stencil of that
// level's element type and no nonzero entry towards a vertex outside it.
template <class V>
std::shared_ptr<Sweep2Op> sweep2_prepare(Ctx &c, const OpMat<V> &At, const GridPair &gp);
// Two consecutive damped-Jacobi steps of a structured 3D FP32 level in one
// pass over the operator (k_sweep2.cu):
//   step A: d1 = dbA - At xA,  sc (=|+=) dinv*(dbA|d1)   (modeA)
//   step B: d2 = d1 - At d1,   sc += dinv*(d1|d2)        (modeB)
// dbA == nullptr: dbA = xA.  dout (nullable) receives d2; r_rho / z64 as in
// smooth_step.  Returns false (and launches nothing) when op is null or the
// level does not qualify (see Ctx::sweep_fusion); the caller then applies the
// steps one by one.  Results are bit-identical to two smooth_step calls; only
// the summation order of the optional rho reduction differs.
template <class V>
bool smooth_pair(Ctx &c, const Sweep2Op *op, const GridPair &gp, const V *xA, const V *dbA, const V *dinv, V *sc,
                 V *dout, int modeA, int modeB, const int *skip, const double *r_rho, RedArgs *red, int rho_kind,
                 double *z64);
template <class V>
void restrict_apply(Ctx &c, const OpMat<V> &R, const V *d, V *dc, const int *skip);
template <class V>
void prolong_apply(Ctx &c, const OpMat<V> &P, const V *scc, V *sc, const V *dfac, V *w, const int *skip);
// StdTransfer on a structured hierarchy without a stored matrix: the
// parents of a fine vertex and the weights (1, 1/2, 1/4, 1/8; Dirichlet rows
// adjusted as in the assembled P and R) follow from its grid indices.  Same
// entries, same order of summation as the assembled P and R = P^T.
struct GridPair {
    int nx, ny, nz;      // fine level vertices per direction (nz = 1 in 2D)
    int cnx, cny, cnz;   // coarse level
    int dim, tet;        // tet: Kuhn split (two parents per edge midpoint)
    // StdTransfer::set_prolongation_damping / set_restriction_damping: factors
    // of the applied transfers (std_transfer_impl.h:740,792), 1 = none
    double dprol = 1.0, dres = 1.0;
};
__device__ __forceinline__ bool on_box_boundary(int i, int j, int k, int nx, int ny, int nz, int dim)
{
    return i == 0 || i == nx - 1 || j == 0 || j == ny - 1 || (dim == 3 && (k == 0 || k == nz - 1));
}

// StdTransfer weight of a parent along `nodd` odd directions: 1, 1/2, 1/4, 1/8
template <class V>
__device__ __forceinline__ V grid_weight(int nodd)
{
    return nodd == 0 ? (V)1 : (nodd == 1 ? (V)0.5 : (nodd == 2 ? (V)0.25 : (V)0.125));
}

// t = (P scc)_f for the fine vertex f = (i, j, k): parents in increasing
// coarse index, as the rows of the assembled P (StdTransfer::
// assemble_prolongation_p1, std_transfer_impl.h:47-168, with
// DirichletBoundary::adjust_prolongation: a Dirichlet fine vertex keeps only
// a coinciding coarse parent, weight 1).
// at(c): the coarse value of vertex c; the loads are issued before the sum.
template <class V, class F>
__device__ __forceinline__ V prolong_value(const GridPair &g, F &&at, int i, int j, int k)
{
    const int p0 = i & 1, p1 = j & 1, p2 = k & 1;
    const int c = (i >> 1) + g.cnx * ((j >> 1) + g.cny * (k >> 1));
    const bool bnd = on_box_boundary(i, j, k, g.nx, g.ny, g.nz, g.dim);
    V t = (V)0;
    if (g.tet) {
        const bool odd = (p0 | p1 | p2) != 0;
        const V wt = odd ? (bnd ? (V)0 : (V)0.5) : (V)1;
        const V v0 = at(c), v1 = at(c + p0 + g.cnx * (p1 + g.cny * p2));
        t = fma_rn(wt, v0, t);
        if (odd) t = fma_rn(wt, v1, t);
    } else {
        const int np = 1 << (p0 + p1 + p2);
        const V wt = bnd ? (np == 1 ? (V)1 : (V)0) : grid_weight<V>(p0 + p1 + p2);
        V v[8] = {};
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if ((q & 1) <= p0 && ((q >> 1) & 1) <= p1 && (q >> 2) <= p2)
                v[q] = at(c + (q & 1) + g.cnx * (((q >> 1) & 1) + g.cny * (q >> 2)));
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if ((q & 1) <= p0 && ((q >> 1) & 1) <= p1 && (q >> 2) <= p2) t = fma_rn(wt, v[q], t);
    }
    return t;
}

// (R d) for coarse vertex (I, J, K): R = P^T, Dirichlet coarse rows =
// injection (k_restrict on the assembled R); children in increasing fine
// index.  at(f): the fine value of vertex f.  The loads of a plane of
// children are issued before their sum.
template <class V, class F>
__device__ __forceinline__ V restrict_value(const GridPair &g, F &&at, int I, int J, int K)
{
    const int fv = 2 * I + g.nx * (2 * J + g.ny * 2 * K);
    if (on_box_boundary(I, J, K, g.cnx, g.cny, g.cnz, g.dim)) {
        const V v = (V)0 + (V)1 * at(fv);
        return (g.dres != 1.0) ? mul_rn(v, (V)g.dres) : v;
    }
    const int kr = (g.dim == 3) ? 1 : 0;
    V acc = (V)0;
#pragma unroll 1
    for (int dk = -kr; dk <= kr; ++dk) {
        V v[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) v[q] = at(fv + (q % 3 - 1) + g.nx * ((q / 3 - 1) + g.ny * dk));
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            const int di = q % 3 - 1, dj = q / 3 - 1;
            const int nodd = (di != 0) + (dj != 0) + (dk != 0);
            V wt;
            if (g.tet) {
                const bool pos = di > 0 || dj > 0 || dk > 0, neg = di < 0 || dj < 0 || dk < 0;
                if (pos && neg) continue;   // not a Kuhn edge through this vertex
                wt = nodd ? (V)0.5 : (V)1;
            } else {
                wt = grid_weight<V>(nodd);
            }
            acc = fma_rn(wt, v[q], acc);
        }
    }
    return (g.dres != 1.0) ? mul_rn(acc, (V)g.dres) : acc;
}

template <class V>
__device__ __forceinline__ void restrict_row(const GridPair &g, const V *__restrict__ d, V *__restrict__ dc, int I,
                                             int J, int K)
{
    dc[I + g.cnx * (J + g.cny * K)] = restrict_value<V>(g, [&](int f) { return d[f]; }, I, J, K);
}

template <class V>
void prolong_grid(Ctx &c, const GridPair &g, const V *scc, V *sc, const V *dfac, V *w, const int *skip);
template <class V>
void restrict_grid(Ctx &c, const GridPair &g, const V *d, V *dc, const int *skip);
template <class V>
void base_solve(Ctx &c, const double *Ainv, int n, const V *d, V *sc, const int *skip);

// ---- the coarse end of a V-cycle in one launch (k_coarse.cu) ----
// Levels [0] (the base, dense LU inverse) .. [m-1] (the entry level) of a
// structured hierarchy with damped-Jacobi smoothing on diagonal-layout
// operators and grid transfers; the entry level's defect arrives in d_in
// (its dA) and its correction leaves in sc_out (its sc), bit-identical to
// the separate launches of lmgc.  A cluster of `ctas` blocks keeps everything
// in shared memory: block q holds rows [q * per, (q + 1) * per) of a level, of
// a solo level block 0 holds all.  The layout is the same in every block:
// its rows of Ainv (per x nbase doubles) at byte 0, the base defect in FP64
// (nbase doubles), then the level-precision region at byte vbase with, per
// level, its part of the operator (S x per), the Jacobi factors and the
// vectors, at the element offsets below (the operator and the factors 16-byte
// aligned; per is a multiple of 4).
constexpr int kCoarseMaxLevels = 8;
template <class V>
struct alignas(16) CoarseLevel {
    const V *val;           // column-scaled operator At, diagonal layout (Dia::vals(), S x ld)
    const V *dinv, *dfac;   // Jacobi factors (unused on the base level)
    int n, ncols, ld, S;
    int solo;               // block 0 alone works on it
    int per;                // rows per block
    unsigned mul;           // j / per == (j * mul) >> 32 for j < n
    int off[kMaxDiag];
    GridPair gp;            // this level and the next coarser one (unused on the base level)
    int aofs;               // operator values (S * per elements)
    int iofs, fofs;         // dinv, dfac (per elements each)
    int vofs;               // vectors sc, dA[, dB, w] (per elements each)
};
template <class V>
struct alignas(16) CoarsePlan {
    int m, nu1, nu2, nbase;
    int ctas;
    const double *Ainv;     // nbase x nbase, row-major
    const V *d_in;
    V *sc_out;
    int vbase;              // byte offset of the level-precision region
    CoarseLevel<V> lev[kCoarseMaxLevels];
};
// plan_dev: the plan in device memory (written at set-up); S: the stencil
// width of every level above the base (coarse_width_ok); smem_bytes: the
// extent of the layout above
template <class V>
void coarse_cycle(Ctx &c, const CoarsePlan<V> *plan_dev, int ctas, int S, size_t smem_bytes, const int *skip);
bool coarse_width_ok(int S);
// set-up: allows launches for width S with up to smem_bytes of dynamic shared
// memory; returns the blocks per cluster that the device runs with that much: 16,
// 8, 4, 2 or 1, at most most_blocks; 0 where it runs none
template <class V>
int coarse_prepare(Ctx &c, int S, int most_blocks, size_t smem_bytes);

// ---- a 2D level of the V-cycle in two launches (k_level2d.cu) ----
template <class V>
struct DiaRows {
    const V *val;   // diagonal layout, S x ld
    int ld;
};
// FP64 levels of up to this many vertices: above, the repeated vertices of the
// tiles cost more FP64 time than the launches they save (solves in FP64: 257^2 751
// -> 738 us, 385^2 986 either way, 513^2 1237 -> 1318 us).  FP32 levels gain at
// more (257^2 617 -> 493 us, 513^2 862 -> 690 us; from the size of the wide steps of
// k_smooth_dia on not: 1025^2 1279 -> 1368 us): the operator is read 1.6
// and 1.4 times instead of four times.
template <class V>
constexpr int64_t kLevel2dRows = sizeof(V) == 8 ? 100000 : 900000;
// At holds the nine-point stencil of the structured 2D level gp, quadrilaterals
template <class V>
bool level2d_ok(const OpMat<V> &At, const GridPair &gp);
// two damped-Jacobi steps from sc = 0 and the defect d (sc, and the defect in
// dout, which d is not), dc = R dout
template <class V>
void level2d_pre(Ctx &c, const OpMat<V> &At, const GridPair &gp, const V *dinv, const V *d, V *sc, V *dout, V *dc,
                 const int *skip);
// sc += P scc and two damped-Jacobi steps from the defect d; r_rho, z64 as in
// smooth_step
template <class V>
void level2d_post(Ctx &c, const OpMat<V> &At, const GridPair &gp, const V *dinv, const V *dfac, const V *scc,
                  const V *d, V *sc, const int *skip, const double *r_rho, RedArgs *red, int rho_kind, double *z64);

// ---- a small 3D level of the V-cycle with its smoothing in two launches (k_level3d.cu) ----
// FP32 levels of up to this many vertices: above, the repeated vertices of the
// tiles (2.8 times the first step) cost more than the launches they save (49^3
// beside 25^3: 97^3 time step 2262 -> 2296 us; 49 x 33 x 33 beside 25 x 17 x 17:
// 97 x 65 x 65 gradient 15.19 -> 15.13 ms).  FP64 lost at every size (129^3 solve
// 6805 -> 6843 us with 17^3, 7005 with 33^3), and the seven-point levels of
// tetrahedra gained less than 1 %.
constexpr int kLevel3dRows = 60000;
// At holds the 27-point stencil of the structured 3D level gp
bool level3d_ok(const OpMat<float> &At, const GridPair &gp);
// as level2d_pre without the restriction
void level3d_pre(Ctx &c, const OpMat<float> &At, const GridPair &gp, const float *dinv, const float *d, float *sc,
                 float *dout, const int *skip);
// as level2d_post, below the top level
void level3d_post(Ctx &c, const OpMat<float> &At, const GridPair &gp, const float *dinv, const float *dfac,
                  const float *scc, const float *d, float *sc, const int *skip);

// Multicolour Gauss-Seidel sweeps of a structured level line by line
// (k_mcgs_lines): per colour (parity bits of the vertex), which diagonals lead
// to vertices of lower colours, of higher ones, and which are entries at all.
// (An entry beyond the grid's edge would multiply 0 with another line's value,
// which a sweep from zero may not have written.)
struct GsLines {
    bool usable = false;
    unsigned below[8] = {}, above[8] = {};
    unsigned all = 0;
    unsigned edge[6] = {};   // the diagonals that leave the grid at x = 0, x = max, y = 0, ...
};
// offs: the layout's offsets, entries: those of them that the CRS holds (the
// rest is padding); unusable where an entry is no neighbour in the grid or
// couples vertices of one colour, and where few long lines would leave the GPU idle
GsLines gs_lines(bool fp64, const Offs &offs, int S, const std::vector<int> &entries, const GridPair &gp);
// one sweep over all colours: t_i = t_i + dinv_relax_i (d_i - (A t)_i), colours
// increasing or (backward) decreasing; from_zero: t is 0 before the sweep and
// need not be written
template <class V>
void mcgs_sweep_lines(Ctx &c, const OpMat<V> &A, const GsLines &gs, const GridPair &gp, bool backward, bool from_zero,
                      const V *dinv_relax, const V *d, V *t, const int *skip);
template <class V>
void mcgs_colour(Ctx &c, const OpMat<V> &A, const int *rows, int nrows_c, const V *dinv_relax, const V *d, V *t,
                 const int *skip);
// d_out = d_base - A t ; sc_mode 1: sc = t, 0: sc += t, 2: sc untouched
template <class V, class DT>
void residual_update(Ctx &c, const OpMat<V> &A, const V *t, const DT *dbase, V *dout, V *sc, int sc_mode,
                     const int *skip);

// ILU(0) in multicolour order (k_ilu.cu): level CRS rows re-ordered by
// (colour, column), L multipliers before the diagonal, U from the diagonal on
template <class V>
struct IluFactors {
    int n = 0;
    DevBuf<int> rowptr, col, nlow;   // nlow[i]: position of the diagonal in row i
    DevBuf<V> val, uinv;
};
// factorise the level operator A (FP64) with the vertex colours `color` and the
// rows of each colour; throws UG4GB_ERR_SINGULAR on a zero pivot
template <class V>
void ilu_setup(Ctx &c, const Csr &A, const int *color, const std::vector<DevBuf<int>> &crow,
               const std::vector<int> &ncrow, IluFactors<V> &F);
// t = damp (L U)^{-1} d (y: scratch of the forward substitution)
template <class V>
void ilu_apply(Ctx &c, const IluFactors<V> &F, const std::vector<DevBuf<int>> &crow, const std::vector<int> &ncrow,
               const V *d, V *y, V *t, double damp, const int *skip);

// ---- Krylov kernels (FP64 outer vectors; z may be FP32 in mixed mode) ----
// r -= A x, |r| starts the check; optionally r32 = (float) r; bicg: the scalars
// of BiCGStab's first iteration too
void krylov_start(Ctx &c, const OpMat<double> &A, const double *x, double *r, RedArgs red, float *r32, bool bicg);
// first: p = z, q = A z; else p = z + beta p, q = A z + beta q; lambda = (q,p), alpha = rho_old/lambda
template <class ZT>
void cg_spmv_dot_t(Ctx &c, const OpMat<double> &A, const ZT *z, double *p, double *q, int first, RedArgs red);
// x += alpha p, r -= alpha q, |r| -> check; optionally r32 = (float) r
void cg_update(Ctx &c, int n, double *x, double *r, const double *p, const double *q, RedArgs red,
               float *r32 = nullptr);
// rho = (z, r); kind 0: rho_old = rho (first), 1: beta = rho/rho_old, rho_old = rho
template <class ZT>
void rho_dot(Ctx &c, int n, const ZT *z, const double *r, int kind, RedArgs red);
template <class ZT>
void copy_z(Ctx &c, int n, const ZT *z, double *out, const int *skip);

// p32, s32: FP32 copies for the mixed-precision multigrid, or null
void bicg_p(Ctx &c, int n, const double *r, double *p, const double *v, double *r0, float *p32, RedArgs red);
template <class ZT>
void bicg_spmv_dot_t(Ctx &c, const OpMat<double> &A, const ZT *q, double *v, const double *r0, RedArgs red);
template <class ZT>
void bicg_x_s(Ctx &c, int n, double *x, const ZT *q, const double *r, const double *v, double *s, float *s32,
              RedArgs red);
void bicg_s_to_r(Ctx &c, int n, const double *s, double *r, RedArgs red);
template <class ZT>
void bicg_spmv_2dot_t(Ctx &c, const OpMat<double> &A, const ZT *q, double *t, const double *s, RedArgs red);
template <class ZT>
void bicg_x_r(Ctx &c, int n, double *x, const ZT *q, const double *s, const double *t, double *r, const double *r0,
              RedArgs red);

// ---- BLAS-1 / SpMV for the public vector and matrix API ----
void vec_dot(Ctx &c, int n, const double *a, const double *b, RedArgs red);
void vec_scale_add(Ctx &c, int n, double *dest, double alpha, const double *a, double beta, const double *b);
void op_axpy(Ctx &c, const OpMat<double> &A, double *dest, double alpha, const double *v1, double beta,
             const double *w1);
void csr_axpy_transposed(Ctx &c, const Csr &A, double *dest, double beta, const double *w1);
template <class TO, class TI>
void convert(Ctx &c, int n, const TI *in, TO *out);

}  // namespace ug4gb
