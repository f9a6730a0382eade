// k_fv1_gather.cu -- FV1 diffusion assembly of unstructured simplex levels row
// by row.
//
// On a simplex the box method's diffusion matrix is K |T| grad phi_i . grad
// phi_j and every SCV has |T| / K of the volume (the element kernel of
// k_fv1.cu sums the same numbers over the SCVFs).  Two launches replace one
// per element colour:
//   k_simplex_terms  one thread per element: the off-diagonal entries and the
//                    SCV volume to a workspace of 4 (triangles) or 8
//                    (tetrahedra) doubles per element;
//   k_gather_rows    four threads per row, one per corner, add the row's
//                    elements in increasing element order and write every
//                    value of the row and its right-hand side once.  The values
//                    of a block's rows are one contiguous range of the CRS,
//                    accumulated in shared memory and written by consecutive
//                    threads.
// The vertex -> element lists and the position of every corner in its row
// depend on the mesh only and are built with the first assembly of a level.
// No atomics, fixed order: the same bits in every run.
//
// 1.57 million tetrahedra (FP64, about 76 FP64 instructions per element):
// k_simplex_terms 0.21 ms, at the FP64 issue rate; k_gather_rows 0.10 ms.  The
// element kernel scattered each element matrix with a binary search per entry
// in 43 colour launches: 5.4 ms.
//
// Convection, quadrilaterals and hexahedra stay with the element kernel.
#include <type_traits>

#include "common.cuh"
#include "disc.cuh"

namespace ug4gb {

namespace {

template <int K>
struct Simplex {
    static constexpr int DIM = K - 1;
    static constexpr int NOFF = K * (K - 1) / 2;    // off-diagonal entries
    static constexpr int WS = (K == 4) ? 8 : 4;     // workspace doubles per element: NOFF entries, SCV volume
    // position of entry (i, j), i != j: (0,1), (0,2), [(0,3),] (1,2), ...
    __host__ __device__ static constexpr int pos(int i, int j)
    {
        const int a = i < j ? i : j, b = i < j ? j : i;
        return a * (2 * K - a - 1) / 2 + (b - a - 1);
    }
};

// ------------------------------------------------- lists of the mesh ------
__global__ void k_count_corner(const int *__restrict__ elems, int nek, int *deg)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nek) atomicAdd(deg + elems[t], 1);
}

// entry: 4 * element + corner
__global__ void k_fill_corner(const int *__restrict__ elems, int nek, int k, const int *__restrict__ vptr, int *cursor,
                              unsigned *adj)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nek) return;
    const int v = elems[t];
    adj[vptr[v] + atomicAdd(cursor + v, 1)] = 4u * (unsigned)(t / k) + (unsigned)(t % k);
}

// a vertex's entries in increasing order, and for each the positions of the
// element's corners in the vertex's row, one byte per corner (csr_from_elements
// admits at most 256 candidates for a row)
__global__ void k_sort_slots(const int *__restrict__ elems, int nv, int k, const int *__restrict__ vptr, unsigned *adj,
                             const int *__restrict__ rowptr, const int *__restrict__ col, unsigned *slots)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nv) return;
    const int s0 = vptr[v], s1 = vptr[v + 1];
    for (int a = s0 + 1; a < s1; ++a) {
        const unsigned x = adj[a];
        int b = a - 1;
        while (b >= s0 && adj[b] > x) {
            adj[b + 1] = adj[b];
            --b;
        }
        adj[b + 1] = x;
    }
    const int q0 = rowptr[v], q1 = rowptr[v + 1];
    for (int a = s0; a < s1; ++a) {
        const size_t e = adj[a] >> 2;
        unsigned packed = 0u;
        for (int j = 0; j < k; ++j) {
            const int c = elems[e * k + j];
            int lo = q0, hi = q1 - 1;   // the row holds every corner of its elements
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (col[mid] < c) lo = mid + 1; else hi = mid;
            }
            packed |= (unsigned)(lo - q0) << (8 * j);
        }
        slots[a] = packed;
    }
}

// ------------------------------------------------------------- elements ---
template <int K>
__global__ void __launch_bounds__(256) k_simplex_terms(const double *__restrict__ coords, const int *__restrict__ elems,
                                                       int ne, const double *__restrict__ coef, double *__restrict__ ws)
{
    using S = Simplex<K>;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    int v[K];
    if constexpr (K == 4) {
        const int4 q = __ldg(reinterpret_cast<const int4 *>(elems) + e);
        v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
    } else {
#pragma unroll
        for (int j = 0; j < K; ++j) v[j] = __ldg(elems + (size_t)e * K + j);
    }
    double x[K][S::DIM];
#pragma unroll
    for (int j = 0; j < K; ++j)
#pragma unroll
        for (int d = 0; d < S::DIM; ++d) x[j][d] = __ldg(coords + (size_t)v[j] * S::DIM + d);
    // n[i] = det * grad phi_i, det = DIM! |T|
    double n[K][S::DIM], det;
    if constexpr (K == 4) {
        double a[3], b[3], c[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            a[d] = x[1][d] - x[0][d];
            b[d] = x[2][d] - x[0][d];
            c[d] = x[3][d] - x[0][d];
        }
        auto cross = [](const double(&p)[3], const double(&q)[3], double(&r)[3]) {
            r[0] = p[1] * q[2] - p[2] * q[1];
            r[1] = p[2] * q[0] - p[0] * q[2];
            r[2] = p[0] * q[1] - p[1] * q[0];
        };
        cross(b, c, n[1]);
        cross(c, a, n[2]);
        cross(a, b, n[3]);
        det = a[0] * n[1][0] + a[1] * n[1][1] + a[2] * n[1][2];
    } else {
        const double ax = x[1][0] - x[0][0], ay = x[1][1] - x[0][1], bx = x[2][0] - x[0][0], by = x[2][1] - x[0][1];
        n[1][0] = by, n[1][1] = -bx;
        n[2][0] = -ay, n[2][1] = ax;
        det = ax * by - ay * bx;
    }
#pragma unroll
    for (int d = 0; d < S::DIM; ++d) {
        double s = 0.0;
#pragma unroll
        for (int j = 1; j < K; ++j) s += n[j][d];
        n[0][d] = -s;
    }
    constexpr double kFact = (K == 4) ? 6.0 : 2.0;
    const double w = coef[e] / (kFact * det);
    double out[S::WS] = {};
#pragma unroll
    for (int i = 0; i < K; ++i)
#pragma unroll
        for (int j = i + 1; j < K; ++j) {
            double s = 0.0;
#pragma unroll
            for (int d = 0; d < S::DIM; ++d) s += n[i][d] * n[j][d];
            out[S::pos(i, j)] = w * s;
        }
    out[S::NOFF] = det * (1.0 / (kFact * K));
#pragma unroll
    for (int q = 0; q < S::WS; q += 2)
        *reinterpret_cast<double2 *>(ws + (size_t)e * S::WS + q) = make_double2(out[q], out[q + 1]);
}

// ----------------------------------------------------------------- rows ---
constexpr int kGatherRows = 64;   // rows of a block of 256 threads

// the most values the rows of a block hold
__global__ void k_block_values(const int *__restrict__ rowptr, int nv, int *most)
{
    const int r0 = (blockIdx.x * blockDim.x + threadIdx.x) * kGatherRows;
    if (r0 < nv) atomicMax(most, rowptr[min(r0 + kGatherRows, nv)] - rowptr[r0]);
}

// INST: rows of sm0 M + sa0 A, right-hand side sa0 f V - sm1 V u_old
// - sa1 A u_old + sa1 f V (AsmArgs)
template <int K, bool INST>
__global__ void __launch_bounds__(256) k_gather_rows(AsmArgs a, int nv, const int *__restrict__ vptr,
                                                     const unsigned *__restrict__ adj,
                                                     const unsigned *__restrict__ slots,
                                                     const double *__restrict__ ws,
                                                     const unsigned char *__restrict__ bnd)
{
    using S = Simplex<K>;
    extern __shared__ double acc[];   // the values of the block's rows
    const int r0 = blockIdx.x * kGatherRows, r1 = min(r0 + kGatherRows, nv);
    const int q0 = __ldg(a.rowptr + r0), nq = __ldg(a.rowptr + r1) - q0;
    for (int i = threadIdx.x; i < nq; i += blockDim.x) acc[i] = 0.0;
    __syncthreads();
    const int r = r0 + (int)(threadIdx.x >> 2), j = threadIdx.x & 3;
    const unsigned group = 0xfu << (threadIdx.x & 28);
    if (r < r1) {
        const int off = __ldg(a.rowptr + r) - q0, s0 = __ldg(vptr + r), s1 = __ldg(vptr + r + 1);
        auto slot = [&](unsigned packed, int c) { return off + (int)((packed >> (8 * c)) & 255u); };
        const bool dir = bnd[r];
        if (dir || s0 == s1) {
            // a Dirichlet row is the identity row with b = 0; a vertex without
            // elements has an empty row
            if (j == 0) {
                if (dir && s1 > s0) acc[slot(slots[s0], (int)(adj[s0] & 3u))] = 1.0;
                if (a.b) a.b[r] = 0.0;
            }
        } else {
            // lane j adds the entry towards corner j; the lane of the vertex
            // itself gathers the volume in the diagonal's place
            for (int t = s0; t < s1; ++t) {
                const unsigned ea = __ldg(adj + t), packed = __ldg(slots + t);
                const int li = (int)(ea & 3u);
                if (j < K)
                    acc[slot(packed, j)] += __ldg(ws + (size_t)(ea >> 2) * S::WS + (j == li ? S::NOFF : S::pos(li, j)));
                __syncwarp(group);   // another lane may add to this slot next
            }
            const int diag = slot(__ldg(slots + s0), (int)(__ldg(adj + s0) & 3u));
            const double vol = acc[diag];
            // the diagonal entry: minus the sum of the others
            const int len = __ldg(a.rowptr + r + 1) - q0 - off;
            double sum = 0.0;
            for (int i = j; i < len; i += 4) sum += (off + i == diag) ? 0.0 : acc[off + i];
            sum += __shfl_xor_sync(group, sum, 1);
            sum += __shfl_xor_sync(group, sum, 2);
            if (j == 0) acc[diag] = -sum;
            __syncwarp(group);
            double au = 0.0;
            if constexpr (INST) {
                if (a.b && a.sa1 != 0.0) {
                    for (int i = j; i < len; i += 4) au += acc[off + i] * a.u_old[__ldg(a.col + q0 + off + i)];
                    au += __shfl_xor_sync(group, au, 1);
                    au += __shfl_xor_sync(group, au, 2);
                }
                __syncwarp(group);
                for (int i = j; i < len; i += 4) acc[off + i] *= a.sa0;
                __syncwarp(group);
                if (j == 0) acc[diag] += a.sm0 * vol;
            }
            if (a.b && j == 0) {
                const double f =
                    a.f ? a.f[r] : (a.use_seed ? 2.0 * hash_uniform(a.f_seed, (uint64_t)r) - 1.0 : 0.0);
                const double fv = f * vol;
                double b = fv;
                if constexpr (INST) {
                    b = a.sa0 != 0.0 ? a.sa0 * fv : 0.0;
                    b -= a.sm1 * (vol * a.u_old[r]);
                    if (a.sa1 != 0.0) {
                        b -= a.sa1 * au;
                        b += a.sa1 * fv;
                    }
                }
                a.b[r] = b;
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nq; i += blockDim.x) a.val[q0 + i] = acc[i];
}

// b with room for n values; false where the device has no memory for them
template <class T>
bool reserve(const Ctx &c, DevBuf<T> &b, size_t n)
{
    if (b.n >= n && !c.scratch_test) return true;
    try {
        b.alloc(c.scratch_test ? (size_t)1 << 48 : n);
    } catch (const Error &e) {
        if (e.code != UG4GB_ERR_NOMEM) throw;
        (void)cudaGetLastError();
        return false;
    }
    return true;
}

template <int K>
bool assemble_gather(Ctx &c, const Level &L, const AsmArgs &a, GatherCache &g, DevBuf<double> &ws)
{
    using S = Simplex<K>;
    // (the element kernel needs none of this)
    if (!reserve(c, ws, (size_t)L.ne * S::WS)) return false;
    if (!g.ready) {
        const int nek = L.ne * K;
        DevBuf<int> deg, most;
        if (!reserve(c, deg, L.nv + 1) || !reserve(c, most, 1) || !reserve(c, g.vptr, L.nv + 1) ||
            !reserve(c, g.adj, nek) || !reserve(c, g.slots, nek)) {
            g = GatherCache();
            return false;
        }
        UG_CUDA(cudaMemsetAsync(deg.p, 0, deg.bytes(), c.stream));
        UG_CUDA(cudaMemsetAsync(most.p, 0, sizeof(int), c.stream));
        UG_LAUNCH(c, k_count_corner, div_up(nek, 256), 256, 0, L.elems.p, nek, deg.p);
        exclusive_scan_int(c, deg.p, g.vptr.p, L.nv + 1, nullptr);
        UG_CUDA(cudaMemsetAsync(deg.p, 0, deg.bytes(), c.stream));
        UG_LAUNCH(c, k_fill_corner, div_up(nek, 256), 256, 0, L.elems.p, nek, K, g.vptr.p, deg.p, g.adj.p);
        UG_LAUNCH(c, k_sort_slots, div_up(L.nv, 128), 128, 0, L.elems.p, L.nv, K, g.vptr.p, g.adj.p, a.rowptr, a.col,
                  g.slots.p);
        UG_LAUNCH(c, k_block_values, div_up(div_up(L.nv, kGatherRows), 256), 256, 0, a.rowptr, L.nv, most.p);
        int h = 0;
        copy_out(c, &h, most.p, sizeof(int));
        g.smem = sizeof(double) * (size_t)h;   // at most 64 x 256 values, 128 KB
        g.ready = true;
    }
    // (the most that any level asks for, as another thread may launch with less or more)
    if (g.smem > 48 * 1024)
        UG_CUDA(cudaFuncSetAttribute(a.inst ? k_gather_rows<K, true> : k_gather_rows<K, false>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(double) * kGatherRows * 256));
    UG_LAUNCH(c, k_simplex_terms<K>, div_up(L.ne, 256), 256, 0, L.coords.p, L.elems.p, L.ne, a.K, ws.p);
    const unsigned blocks = div_up(L.nv, kGatherRows);
    if (a.inst)
        UG_LAUNCH(c, (k_gather_rows<K, true>), blocks, 256, g.smem, a, L.nv, g.vptr.p, g.adj.p, g.slots.p, ws.p,
                  L.bnd.p);
    else
        UG_LAUNCH(c, (k_gather_rows<K, false>), blocks, 256, g.smem, a, L.nv, g.vptr.p, g.adj.p, g.slots.p, ws.p,
                  L.bnd.p);
    return true;
}

}  // namespace

bool launch_assemble_gather(Ctx &c, const Level &L, const AsmArgs &a, GatherCache &g, DevBuf<double> &ws)
{
    if (L.structured || a.vmodes > 0 || L.ne == 0) return false;
    if (L.elem_type == UG4GB_TET) return assemble_gather<4>(c, L, a, g, ws);
    if (L.elem_type == UG4GB_TRI) return assemble_gather<3>(c, L, a, g, ws);
    return false;
}

}  // namespace ug4gb
