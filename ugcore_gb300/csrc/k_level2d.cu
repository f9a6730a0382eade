// k_level2d.cu -- a 2D level of the V-cycle in two launches.
//
// On 2D levels of up to some 10^5 vertices a Jacobi step or a transfer is a
// launch of about 3 us, most of it the launch and chains of dependent loads and
// FP64 operations, and a level takes six.  Two kernels replace them for
// nu1 = nu2 = 2, with the row arithmetic of the separate kernels in their order.
// (FP32 corrections are the same bits.  FP64 rows are summed in two chains,
// row_sum, which the separate kernels do on levels of up to a block of rows per SM
// only, 38912 rows: above them the rounding differs.)
//   k_pre2d    two pre-smoothing steps and the restriction
//   k_post2d   the prolongation and two post-smoothing steps (on the top level
//              with the fused (z, r) and the FP64 copy of the correction)
// A block owns a tile of 16 x 8 vertices (8 x 4 coarse ones) and computes the
// vertices around it that it needs from other tiles itself: the first step on
// 19 x 11 vertices, the second on 17 x 9 (after the prolongation 20 x 12 and 18 x
// 10), one vertex per thread, the vectors in shared memory, each thread's
// operator row in registers for both steps, loaded before the launch wait.
// 129^2 solve, FP64: 632 -> 526 us; 257^2 adjoint gradient 3.86 -> 3.59 ms.
#include "k_solve.cuh"

namespace ug4gb {

namespace {

constexpr int kT = 256;                    // threads per block
constexpr int kOX = 16, kOY = 8;           // vertices of a tile
constexpr int kCX = kOX / 2, kCY = kOY / 2;

// The operator row and Jacobi factor of vertex (i, j); 0 outside the level.
template <class V>
__device__ __forceinline__ void load_row(const DiaRows<V> &A, const V *__restrict__ dinv, int row, bool in, V (&a)[9],
                                         V &di)
{
#pragma unroll
    for (int k = 0; k < 9; ++k) a[k] = in ? ld_stream(A.val + (size_t)k * A.ld + row) : (V)0;
    di = in ? __ldg(dinv + row) : (V)0;
}

// (At x) of the vertex at (x, y) of a tile of width W held in shared memory
template <class V, int W>
__device__ __forceinline__ V tile_row(const V (&a)[9], const V *t, int x, int y)
{
    V v[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) v[k] = t[(x + k % 3 - 1) + W * (y + k / 3 - 1)];
    return row_sum<V, 9>(a, v);
}

// d1 = d - At d, sc = dinv d; d2 = d1 - At d1, sc += dinv d1; dc = R d2
template <class V>
__global__ void __launch_bounds__(kT) k_pre2d(DiaRows<V> A, GridPair g, const V *__restrict__ dinv,
                                              const V *__restrict__ d, V *__restrict__ sc, V *__restrict__ dout,
                                              V *__restrict__ dc, const int *skip)
{
    constexpr int AX = kOX + 3, AY = kOY + 3;   // first step, from (-2, -2) of the tile on
    constexpr int DX = AX + 2, DY = AY + 2;     // the defect, from (-3, -3)
    static_assert(AX * AY <= kT, "one vertex per thread");
    __shared__ V s0[DX * DY], s1[AX * AY], s2[AX * AY];
    const int t = threadIdx.x, ox = blockIdx.x * kOX, oy = blockIdx.y * kOY;
    const int ax = t % AX, ay = t / AX, i = ox - 2 + ax, j = oy - 2 + ay;
    const bool in = t < AX * AY && i >= 0 && i < g.nx && j >= 0 && j < g.ny;
    const int row = i + g.nx * j;
    V a[9], di;
    pdl_trigger();
    load_row<V>(A, dinv, row, in, a, di);
    pdl_wait();
    if (skip && *skip) return;
    for (int q = t; q < DX * DY; q += kT) {
        const int x = ox - 3 + q % DX, y = oy - 3 + q / DX;
        s0[q] = (x >= 0 && x < g.nx && y >= 0 && y < g.ny) ? d[x + g.nx * y] : (V)0;
    }
    __syncthreads();
    V db = (V)0, d1 = (V)0, s = (V)0;
    if (t < AX * AY) {
        if (in) {
            db = s0[(ax + 1) + DX * (ay + 1)];
            d1 = jacobi_row<V>(tile_row<V, DX>(a, s0, ax + 1, ay + 1), db, di, SC_SET_FROM_BASE, (V)0, s);
        }
        s1[t] = d1;
    }
    __syncthreads();
    // the second step: all but the rim
    if (t < AX * AY && ax > 0 && ax < AX - 1 && ay > 0 && ay < AY - 1) {
        V d2 = (V)0;
        if (in) {
            V sn;
            d2 = jacobi_row<V>(tile_row<V, AX>(a, s1, ax, ay), d1, di, SC_ADD_FROM_BASE, s, sn);
            if (ax >= 2 && ax < 2 + kOX && ay >= 2 && ay < 2 + kOY) {
                sc[row] = sn;
                dout[row] = d2;
            }
        }
        s2[t] = d2;
    }
    __syncthreads();
    if (t < kCX * kCY) {
        const int cx = t % kCX, cy = t / kCX, I = blockIdx.x * kCX + cx, J = blockIdx.y * kCY + cy;
        if (I < g.cnx && J < g.cny) {
            // fine vertex f = x + nx y at (x - ox + 2, y - oy + 2) of s2
            const int f0 = 2 * I + g.nx * 2 * J, p0 = (2 * cx + 2) + AX * (2 * cy + 2);
            auto at = [&](int f) {
                // f - f0 = dx + nx dy with dx, dy in {-1, 0, 1}
                const int o = f - f0 + g.nx + 1, dy = o / g.nx - 1, dx = o - (dy + 1) * g.nx - 1;
                return s2[p0 + dx + AX * dy];
            };
            dc[I + g.cnx * J] = restrict_value<V>(g, at, I, J, 0);
        }
    }
}

// t = P scc, sc += t, w = t dfac; d3 = d - At w, sc += dinv d3; d4 = d3 - At d3,
// sc += dinv d4
template <class V, bool RHO>
__global__ void __launch_bounds__(kT) k_post2d(DiaRows<V> A, GridPair g, const V *__restrict__ dinv,
                                               const V *__restrict__ dfac, const V *__restrict__ scc,
                                               const V *__restrict__ d, V *__restrict__ sc, const int *skip,
                                               const double *__restrict__ r_rho, RedArgs red, int rho_kind,
                                               double *__restrict__ z64)
{
    constexpr int WX = kOX + 4, WY = kOY + 4;   // the prolongation, from (-2, -2) of the tile on
    static_assert(WX * WY <= kT, "one vertex per thread");
    __shared__ V sw[WX * WY], s3[WX * WY];
    const int t = threadIdx.x, ox = blockIdx.x * kOX, oy = blockIdx.y * kOY;
    const int wx = t % WX, wy = t / WX, i = ox - 2 + wx, j = oy - 2 + wy;
    const bool in = t < WX * WY && i >= 0 && i < g.nx && j >= 0 && j < g.ny;
    const bool step1 = in && wx > 0 && wx < WX - 1 && wy > 0 && wy < WY - 1;
    const bool own = in && wx >= 2 && wx < 2 + kOX && wy >= 2 && wy < 2 + kOY;
    const int row = i + g.nx * j;
    V a[9], di, df = (V)0;
    pdl_trigger();
    load_row<V>(A, dinv, row, step1, a, di);
    if (in) df = __ldg(dfac + row);
    pdl_wait();
    if (skip && *skip) return;
    V tv = (V)0, s = (V)0, db = (V)0;
    if (own) s = sc[row];
    if (step1) db = d[row];
    if (in) {
        tv = prolong_value<V>(g, [&](int c) { return scc[c]; }, i, j, 0);
        if (g.dprol != 1.0) tv = mul_rn(tv, (V)g.dprol);
    }
    if (t < WX * WY) {
        sw[t] = mul_rn(tv, df);
        s3[t] = (V)0;
    }
    s = add_rn(s, tv);
    __syncthreads();
    V d3 = (V)0;
    if (step1) {
        V sn;
        d3 = jacobi_row<V>(tile_row<V, WX>(a, sw, wx, wy), db, di, SC_ADD_FROM_NEW, s, sn);
        s = sn;
        s3[t] = d3;
    }
    __syncthreads();
    double rsum = 0.0;
    if (own) {
        V sn;
        jacobi_row<V>(tile_row<V, WX>(a, s3, wx, wy), d3, di, SC_ADD_FROM_NEW, s, sn);
        sc[row] = sn;
        if (RHO || z64) {
            double s64;
            if constexpr (sizeof(V) == 8) s64 = sn;
            else s64 = f32_to_f64(sn);
            if (z64) z64[row] = s64;
            if (RHO) rsum = s64 * r_rho[row];
        }
    }
    if (RHO) {
        double v[1] = {rsum};
        KScal *ks = red.ks;
        grid_reduce<kT, 1>(v, red.partials, red.counter, [&](const double(&tot)[1]) {
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

template <class V>
DiaRows<V> rows_of(const OpMat<V> &At)
{
    return DiaRows<V>{At.dia.vals(), At.dia.ld};
}
dim3 tiles(const GridPair &g) { return dim3(div_up(g.nx, kOX), div_up(g.ny, kOY)); }

}  // namespace

template <class V>
bool level2d_ok(const OpMat<V> &At, const GridPair &g)
{
    if (At.kind != 1 || At.dia.S != 9 || g.dim != 2 || g.tet || g.nx < 3 || g.ny < 3) return false;
    if (At.nrows != g.nx * g.ny || At.ncols != At.nrows) return false;
    for (int k = 0; k < 9; ++k)
        if (At.dia.off.o[k] != (k % 3 - 1) + g.nx * (k / 3 - 1)) return false;
    const dim3 b = tiles(g);
    return (int64_t)At.nrows <= kLevel2dRows<V> && b.x * b.y <= (unsigned)kRedMaxBlocks;
}

template <class V>
void level2d_pre(Ctx &c, const OpMat<V> &At, const GridPair &g, const V *dinv, const V *d, V *sc, V *dout, V *dc,
                 const int *skip)
{
    UG_LAUNCH_PDL(c, k_pre2d<V>, tiles(g), kT, 0, rows_of(At), g, dinv, d, sc, dout, dc, skip);
}

template <class V>
void level2d_post(Ctx &c, const OpMat<V> &At, const GridPair &g, const V *dinv, const V *dfac, const V *scc, const V *d,
                  V *sc, const int *skip, const double *r_rho, RedArgs *red, int rho_kind, double *z64)
{
    RedArgs none{nullptr, nullptr, nullptr};
    if (r_rho)
        UG_LAUNCH_PDL(c, (k_post2d<V, true>), tiles(g), kT, 0, rows_of(At), g, dinv, dfac, scc, d, sc, skip, r_rho,
                      *red, rho_kind, z64);
    else
        UG_LAUNCH_PDL(c, (k_post2d<V, false>), tiles(g), kT, 0, rows_of(At), g, dinv, dfac, scc, d, sc, skip,
                      (const double *)nullptr, none, 0, z64);
}

#define INST_LEVEL2D(V)                                                                                            \
    template bool level2d_ok<V>(const OpMat<V> &, const GridPair &);                                               \
    template void level2d_pre<V>(Ctx &, const OpMat<V> &, const GridPair &, const V *, const V *, V *, V *, V *,   \
                                 const int *);                                                                     \
    template void level2d_post<V>(Ctx &, const OpMat<V> &, const GridPair &, const V *, const V *, const V *,      \
                                  const V *, V *, const int *, const double *, RedArgs *, int, double *);
INST_LEVEL2D(double)
INST_LEVEL2D(float)

}  // namespace ug4gb
