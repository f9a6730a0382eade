// k_level3d.cu -- the smoothing of a small 3D FP32 level of the V-cycle in two
// launches, for nu1 = nu2 = 2 and 27-point stencils.
//
// On 3D levels of some 10^4 vertices a Jacobi step is a launch of 2.5 to 4 us,
// most of it the launch and the latency of its loads.  Two kernels replace five
// launches (the row arithmetic is that of the separate kernels, in their order,
// so corrections are the same bits):
//   k_pre3d    two pre-smoothing steps
//   k_post3d   the prolongation and two post-smoothing steps
// A block owns a tile of 8 x 4 x 4 vertices and computes the first step on the
// layer of vertices around it too (and the prolongation on two layers): one
// vertex per thread, the vectors in shared memory, each thread's operator row in
// registers for both steps, loaded before the launch wait.  The restriction stays
// a launch of its own: it would need a third layer.
// 97 x 65 x 65 convection gradient 15.78 -> 15.13 ms, 97^3 time step 2300 -> 2255
// us, 193^3 convection solve 66.1 -> 65.8 ms.  (Tiles of 8 x 8 x 4: 15.22 ms;
// 4 x 4 x 4: 15.31; 8 x 4 x 2 and 16 x 4 x 2: 15.62 and 15.42.)
#include "k_solve.cuh"

namespace ug4gb {

namespace {

constexpr int kOX = 8, kOY = 4, kOZ = 4;                         // vertices of a tile
constexpr int kAX = kOX + 2, kAY = kOY + 2, kAZ = kOZ + 2;       // of the first step, from (-1, -1, -1) on
constexpr int kWX = kOX + 4, kWY = kOY + 4, kWZ = kOZ + 4;       // what that reads, from (-2, -2, -2)
constexpr int kA = kAX * kAY * kAZ, kW = kWX * kWY * kWZ;
constexpr int kT = (kA + 31) / 32 * 32;                          // threads: one per vertex of the first step

// (At x) of the vertex at *t of a region of lines of sx and planes of sxy values
__device__ __forceinline__ float tile_row(const float (&a)[27], const float *t, int sx, int sxy)
{
    float v[27];
#pragma unroll
    for (int k = 0; k < 27; ++k) v[k] = t[k % 3 - 1 + sx * (k / 3 % 3 - 1) + sxy * (k / 9 - 1)];
    return row_sum<float, 27>(a, v);
}

// this thread's vertex of the first step
struct Place {
    int ax, ay, az, i, j, k, row;
    bool in, own;
    __device__ __forceinline__ Place(const GridPair &g)
    {
        const int t = threadIdx.x;
        ax = t % kAX;
        ay = t / kAX % kAY;
        az = t / (kAX * kAY);
        i = (int)blockIdx.x * kOX - 1 + ax;
        j = (int)blockIdx.y * kOY - 1 + ay;
        k = (int)blockIdx.z * kOZ - 1 + az;
        in = t < kA && i >= 0 && i < g.nx && j >= 0 && j < g.ny && k >= 0 && k < g.nz;
        own = in && ax > 0 && ax <= kOX && ay > 0 && ay <= kOY && az > 0 && az <= kOZ;
        row = i + g.nx * (j + g.ny * k);
    }
    __device__ __forceinline__ int in_a() const { return threadIdx.x; }
    __device__ __forceinline__ int in_w() const { return ax + 1 + kWX * (ay + 1 + kWY * (az + 1)); }
};

// the operator row and Jacobi factor; 0 outside the level
__device__ __forceinline__ void load_row(const DiaRows<float> &A, const float *__restrict__ dinv, const Place &p,
                                         float (&a)[27], float &di)
{
#pragma unroll
    for (int k = 0; k < 27; ++k) a[k] = p.in ? ld_stream(A.val + (size_t)k * A.ld + p.row) : 0.0f;
    di = p.in ? __ldg(dinv + p.row) : 0.0f;
}

// f(vertex, its place in the region read by the first step) for all of it; the
// value outside the level is 0
template <class F>
__device__ __forceinline__ void fill_region(const GridPair &g, float *s, F &&f)
{
    for (int q = threadIdx.x; q < kW; q += kT) {
        const int x = q % kWX, y = q / kWX % kWY, z = q / (kWX * kWY);
        const int i = (int)blockIdx.x * kOX - 2 + x, j = (int)blockIdx.y * kOY - 2 + y,
                  k = (int)blockIdx.z * kOZ - 2 + z;
        const bool in = i >= 0 && i < g.nx && j >= 0 && j < g.ny && k >= 0 && k < g.nz;
        s[q] = in ? f(i, j, k, q) : 0.0f;
    }
}

// d1 = d - At d, sc = dinv d; d2 = d1 - At d1, sc += dinv d1
__global__ void __launch_bounds__(kT, 2)
    k_pre3d(DiaRows<float> A, GridPair g, const float *__restrict__ dinv, const float *__restrict__ d,
            float *__restrict__ sc, float *__restrict__ dout, const int *skip)
{
    __shared__ float s0[kW], s1[kA];
    const Place p(g);
    float a[27], di;
    pdl_trigger();
    load_row(A, dinv, p, a, di);
    pdl_wait();
    if (skip && *skip) return;
    fill_region(g, s0, [&](int i, int j, int k, int) { return d[i + g.nx * (j + g.ny * k)]; });
    __syncthreads();
    float d1 = 0.0f, s = 0.0f;
    if (p.in) d1 = jacobi_row<float>(tile_row(a, s0 + p.in_w(), kWX, kWX * kWY), s0[p.in_w()], di, SC_SET_FROM_BASE,
                                     0.0f, s);
    if (threadIdx.x < kA) s1[p.in_a()] = d1;
    __syncthreads();
    if (p.own) {
        float sn;
        const float d2 = jacobi_row<float>(tile_row(a, s1 + p.in_a(), kAX, kAX * kAY), d1, di, SC_ADD_FROM_BASE, s, sn);
        sc[p.row] = sn;
        dout[p.row] = d2;
    }
}

// t = P scc, sc += t, w = t dfac; d3 = d - At w, sc += dinv d3; d4 = d3 - At d3,
// sc += dinv d4
__global__ void __launch_bounds__(kT, 2)
    k_post3d(DiaRows<float> A, GridPair g, const float *__restrict__ dinv, const float *__restrict__ dfac,
             const float *__restrict__ scc, const float *__restrict__ d, float *__restrict__ sc, const int *skip)
{
    __shared__ float sw[kW], st[kW], s3[kA];
    const Place p(g);
    float a[27], di;
    pdl_trigger();
    load_row(A, dinv, p, a, di);
    pdl_wait();
    if (skip && *skip) return;
    const float db = p.in ? d[p.row] : 0.0f;
    float s = p.own ? sc[p.row] : 0.0f;
    fill_region(g, sw, [&](int i, int j, int k, int q) {
        const float df = __ldg(dfac + (i + g.nx * (j + g.ny * k)));
        float t = prolong_value<float>(g, [&](int c) { return scc[c]; }, i, j, k);
        if (g.dprol != 1.0) t = mul_rn(t, (float)g.dprol);
        st[q] = t;
        return mul_rn(t, df);
    });
    __syncthreads();
    float d3 = 0.0f;
    if (p.in) {
        float sn;
        s = add_rn(s, st[p.in_w()]);
        d3 = jacobi_row<float>(tile_row(a, sw + p.in_w(), kWX, kWX * kWY), db, di, SC_ADD_FROM_NEW, s, sn);
        s = sn;
    }
    if (threadIdx.x < kA) s3[p.in_a()] = d3;
    __syncthreads();
    if (p.own) {
        float sn;
        jacobi_row<float>(tile_row(a, s3 + p.in_a(), kAX, kAX * kAY), d3, di, SC_ADD_FROM_NEW, s, sn);
        sc[p.row] = sn;
    }
}

DiaRows<float> rows_of(const OpMat<float> &At) { return DiaRows<float>{At.dia.vals(), At.dia.ld}; }
dim3 tiles(const GridPair &g) { return dim3(div_up(g.nx, kOX), div_up(g.ny, kOY), div_up(g.nz, kOZ)); }

}  // namespace

bool level3d_ok(const OpMat<float> &At, const GridPair &g)
{
    if (At.kind != 1 || g.dim != 3 || g.nx < 3 || g.ny < 3 || g.nz < 3) return false;
    if (At.nrows != g.nx * g.ny * g.nz || At.ncols != At.nrows) return false;
    if (At.dia.S != 27 || At.nrows > kLevel3dRows) return false;
    for (int k = 0; k < 27; ++k)
        if (At.dia.off.o[k] != k % 3 - 1 + g.nx * (k / 3 % 3 - 1) + g.nx * g.ny * (k / 9 - 1)) return false;
    return true;
}

void level3d_pre(Ctx &c, const OpMat<float> &At, const GridPair &g, const float *dinv, const float *d, float *sc,
                 float *dout, const int *skip)
{
    UG_LAUNCH_PDL(c, k_pre3d, tiles(g), kT, 0, rows_of(At), g, dinv, d, sc, dout, skip);
}

void level3d_post(Ctx &c, const OpMat<float> &At, const GridPair &g, const float *dinv, const float *dfac,
                  const float *scc, const float *d, float *sc, const int *skip)
{
    UG_LAUNCH_PDL(c, k_post3d, tiles(g), kT, 0, rows_of(At), g, dinv, dfac, scc, d, sc, skip);
}

}  // namespace ug4gb
