// k_coarse.cu -- the coarse end of a multigrid V-cycle in one launch.
//
// Below some thousand rows a level's smoothing steps, transfers and the base
// solve are latency work: every one of them is a separate launch of about
// 3 us (in the solve's graph) in which a few blocks touch a few KB.  The coarse
// levels of the hierarchy are therefore cycled by one cluster of up to 16
// blocks with every such level (operator, Jacobi factors, vectors) and the
// base inverse spread over the blocks' shared memory, a cluster barrier
// between the phases that the separate launches would order:
//   per level, from the entry level down:   nu1 damped-Jacobi steps, then
//                                           restriction to the level below
//   base level:                             sc = Ainv d (dense inverse)
//   per level, back up:                     prolongation (sc += t, w = t*dfac),
//                                           nu2 damped-Jacobi steps
// (AssembledMultiGridCycle::lmgc, mg_solver_impl.hpp:2091-2134, for
// gamma = 1 below the entry level).  A block reads its neighbours' vector
// entries through distributed shared memory.  On the smallest (solo) levels a
// barrier of the cluster would cost more than the work: block 0 runs them with
// its own barrier while the others wait.  Every row is computed with the
// arithmetic of the separate kernels (diagonal-layout row product with the
// same clamped columns and FMA order, jacobi_row, prolong_value,
// restrict_value, the base solve's per-lane partial sums and warp reduction),
// so corrections are bit-identical to those of the separate launches.
#include "k_solve.cuh"

namespace ug4gb {

constexpr int kCoarseThreads = 512;

// Asynchronous copies global -> shared (cp.async): every thread issues all
// of its copies before waiting, so the staging of a few hundred KB is bound
// by bandwidth, not by one load's latency per thread and iteration.
__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// bytes from src to dst, both 16-byte aligned: 16-byte copies, the tail
// (bytes % 16, a multiple of 4) in 4-byte copies
__device__ __forceinline__ void stage(void *dst, const void *src, size_t bytes)
{
    const size_t n16 = bytes / 16;
    for (size_t i = threadIdx.x; i < n16; i += blockDim.x)
        cp_async16((char *)dst + 16 * i, (const char *)src + 16 * i);
    for (size_t i = 16 * n16 + 4 * threadIdx.x; i < bytes; i += 4 * blockDim.x)
        cp_async4((char *)dst + i, (const char *)src + i);
}

// every block of the cluster has arrived, their shared-memory writes visible
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// the shared-memory word at `addr` of this block's layout, in block `rank`
__device__ __forceinline__ float ld_cluster(unsigned addr, unsigned rank, float)
{
    float v;
    asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}"
                 : "=f"(v)
                 : "r"(addr), "r"(rank));
    return v;
}
__device__ __forceinline__ double ld_cluster(unsigned addr, unsigned rank, double)
{
    double v;
    asm volatile("{\n\t.reg .u32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f64 %0, [a];\n\t}"
                 : "=d"(v)
                 : "r"(addr), "r"(rank));
    return v;
}

// read access to a level's vector from any block (p: this block's part)
template <class V>
struct ClusterVec {
    unsigned addr;
    unsigned mul;
    int per;
    __device__ __forceinline__ ClusterVec(const CoarseLevel<V> &L, const V *p)
        : addr((unsigned)__cvta_generic_to_shared(p)), mul(L.solo ? 0u : L.mul), per(L.per)
    {
    }
    __device__ __forceinline__ V operator()(int j) const
    {
        const int q = (int)__umulhi((unsigned)j, mul);
        return ld_cluster(addr + (unsigned)(j - q * per) * (unsigned)sizeof(V), (unsigned)q, (V)0);
    }
};
template <class V>
struct LocalVec {
    const V *p;
    __device__ __forceinline__ V operator()(int j) const { return p[j]; }
};

// (At x)_i of the diagonal layout, i = r0 + q: DiaMV::dot_cached's order of
// operations (the same clamped columns, row_sum), with this block's part of
// the operator a (S x per); S fixed at compile time, so every load of the row
// is issued before the sum starts
template <class V, int S, class X>
__device__ __forceinline__ V coarse_dot(const CoarseLevel<V> &L, const V *a, const X &x, int r0, int q)
{
    V av[S], xv[S];
#pragma unroll
    for (int k = 0; k < S; ++k) {
        int j = r0 + q + L.off[k];
        j = j < 0 ? 0 : (j >= L.ncols ? L.ncols - 1 : j);
        xv[k] = x(j);
    }
#pragma unroll
    for (int k = 0; k < S; ++k) av[k] = a[k * L.per + q];
    return row_sum<V, S>(av, xv);
}

// The phases on this block's rows r0 .. r0 + nr - 1 of a level; one copy of
// their code each (not inlined at their several places: a launch runs every
// phase a few times, so its instructions come from a cold cache).
// One damped-Jacobi step: dn = db - At x; sc (=|+=) dinv*(db|dn); dout
// (nullable) = dn.  x: this block's part of the vector, db, sc, dout likewise.
template <class V, int S>
__device__ __noinline__ void coarse_step(const CoarseLevel<V> &L, const V *a, const V *dinv, const V *x, const V *db,
                                         V *sc, V *dout, int mode, int r0, int nr)
{
    for (int q = threadIdx.x; q < nr; q += blockDim.x) {
        const V acc = L.solo ? coarse_dot<V, S>(L, a, LocalVec<V>{x}, r0, q)
                             : coarse_dot<V, S>(L, a, ClusterVec<V>(L, x), r0, q);
        V s;
        const V dn = jacobi_row<V>(acc, db[q], dinv[q], mode, mode == SC_SET_FROM_BASE ? (V)0 : sc[q], s);
        if (dout) dout[q] = dn;
        sc[q] = s;
    }
}

// dc = R d, rows c0 .. c0 + nc - 1 of the level below L
template <class V>
__device__ __noinline__ void coarse_restrict(const CoarseLevel<V> &L, const V *d, V *dc, int c0, int nc)
{
    const GridPair &g = L.gp;
    const ClusterVec<V> at(L, d);
    for (int q = threadIdx.x; q < nc; q += blockDim.x) {
        const int c = c0 + q;
        dc[q] = restrict_value<V>(g, at, c % g.cnx, (c / g.cnx) % g.cny, c / (g.cnx * g.cny));
    }
}

// sc += P scc, w = t * dfac (w nullable); C: the level below
template <class V>
__device__ __noinline__ void coarse_prolong(const CoarseLevel<V> &L, const CoarseLevel<V> &C, const V *scc, V *sc,
                                            const V *dfac, V *w, int r0, int nr)
{
    const GridPair &g = L.gp;
    const ClusterVec<V> at(C, scc);
    for (int q = threadIdx.x; q < nr; q += blockDim.x) {
        const int f = r0 + q;
        V t = prolong_value<V>(g, at, f % g.nx, (f / g.nx) % g.ny, f / (g.nx * g.ny));
        if (g.dprol != 1.0) t = mul_rn(t, (V)g.dprol);
        sc[q] = add_rn(sc[q], t);
        if (w) w[q] = mul_rn(t, dfac[q]);
    }
}

template <class V, int S>
__global__ void __launch_bounds__(kCoarseThreads, 1)
    k_coarse_cycle(const CoarsePlan<V> *__restrict__ plan, const int *skip)
{
    __shared__ CoarsePlan<V> P;
    extern __shared__ __align__(16) unsigned char coarse_smem[];
    const int tid = threadIdx.x, nt = blockDim.x, rank = (int)cluster_rank();
    {
        // the plan, the operators, the Jacobi factors and the base inverse
        // are written at set-up, never by a solve kernel: staged before the
        // wait for the predecessor, so the copies overlap its tail
        static_assert(sizeof(CoarsePlan<V>) % 16 == 0, "plan copied in 16-byte words");
        const int4 *src = reinterpret_cast<const int4 *>(plan);
        int4 *dst = reinterpret_cast<int4 *>(&P);
        for (int i = tid; i < (int)(sizeof(CoarsePlan<V>) / 16); i += nt) dst[i] = __ldg(src + i);
    }
    __syncthreads();
    double *ainv = reinterpret_cast<double *>(coarse_smem);
    double *dwide = ainv + (size_t)P.lev[0].per * P.nbase;
    V *vr = reinterpret_cast<V *>(coarse_smem + P.vbase);
    // this block's rows of level l: first row, number of rows
    auto first = [&](int l) { return P.lev[l].solo ? 0 : rank * P.lev[l].per; };
    auto rows = [&](int l) {
        const CoarseLevel<V> &L = P.lev[l];
        if (L.solo) return rank == 0 ? L.n : 0;
        const int left = L.n - rank * L.per;
        return left < 0 ? 0 : (left < L.per ? left : L.per);
    };
    stage(ainv, P.Ainv + (size_t)first(0) * P.nbase, (size_t)rows(0) * P.nbase * sizeof(double));
    for (int l = 1; l < P.m; ++l) {
        const CoarseLevel<V> &L = P.lev[l];
        const int r0 = first(l), nr = rows(l);
        // whole 16-byte words of each diagonal: its padding rows are zero
        int na = (nr + 3) / 4 * 4;
        if (r0 + na > L.ld) na = L.ld - r0;
        if (nr > 0) {
            constexpr int W = 16 / (int)sizeof(V);
            const int words = na / W;   // per diagonal
            for (int i = tid; i < S * words; i += nt) {
                const int k = i / words, q = (i - k * words) * W;
                cp_async16(vr + L.aofs + k * L.per + q, L.val + (size_t)k * L.ld + r0 + q);
            }
            stage(vr + L.iofs, L.dinv + r0, (size_t)nr * sizeof(V));
            stage(vr + L.fofs, L.dfac + r0, (size_t)nr * sizeof(V));
        }
    }
    pdl_trigger();
    pdl_wait();
    if (skip && *skip) {
        cp_async_wait_all();   // no copy outlives the block
        return;
    }
    const int top = P.m - 1;
    // this block's parts of the vectors of level l: sc, dA, dB, w (the base
    // level: sc, dA)
    auto vsc = [&](int l) { return vr + P.lev[l].vofs; };
    auto vdA = [&](int l) { return vr + P.lev[l].vofs + P.lev[l].per; };
    auto vdB = [&](int l) { return vr + P.lev[l].vofs + 2 * P.lev[l].per; };
    auto vw = [&](int l) { return vr + P.lev[l].vofs + 3 * P.lev[l].per; };
    // a phase has ended whose results the next one reads on other blocks, or,
    // between phases of solo levels, on block 0 only
    auto sync = [&](bool solo) {
        if (solo) __syncthreads();
        else cluster_sync();
    };
    {
        V *d = vdA(top);
        const int r0 = first(top), nr = rows(top);
        for (int i = tid; i < nr; i += nt) d[i] = P.d_in[r0 + i];
    }
    cp_async_wait_all();
    cluster_sync();
    // ---- down: pre-smoothing and restriction (the defect of a level
    // arrives in its dA; the steps alternate dA -> dB -> dA ...)
    for (int l = top; l >= 1; --l) {
        const CoarseLevel<V> &L = P.lev[l];
        const bool solo = L.solo != 0;
        if (solo && rank != 0) continue;   // block 0 runs the levels below alone
        const int r0 = first(l), nr = rows(l);
        const V *a = vr + L.aofs, *dinv = vr + L.iofs;
        V *sc = vsc(l), *dA = vdA(l), *dB = vdB(l);
        if (P.nu1 == 0) {
            for (int i = tid; i < nr; i += nt) sc[i] = (V)0;
            sync(solo);
        }
        V *cur = dA;
        for (int k = 0; k < P.nu1; ++k) {
            V *out = (cur == dA) ? dB : dA;
            const int mode = k == 0 ? SC_SET_FROM_BASE : SC_ADD_FROM_BASE;
            coarse_step<V, S>(L, a, dinv, cur, cur, sc, out, mode, r0, nr);
            sync(solo);
            cur = out;
        }
        coarse_restrict<V>(L, cur, vdA(l - 1), first(l - 1), rows(l - 1));
        sync(P.lev[l - 1].solo != 0);
    }
    // ---- base: sc = Ainv d, one warp per row (k_base_solve's partial sums);
    // the defect is collected and widened once per entry first (conversions
    // issue on the FP64 pipe)
    {
        const CoarseLevel<V> &L = P.lev[0];
        const bool solo = L.solo != 0;
        if (!solo || rank == 0) {
            const int n0 = P.nbase, warp = tid >> 5, lane = tid & 31, nr = rows(0);
            const ClusterVec<V> dv(L, vdA(0));
            for (int j = tid; j < n0; j += nt) dwide[j] = (double)(solo ? vdA(0)[j] : dv(j));
            __syncthreads();
            V *sc = vsc(0);
            for (int row = warp; row < nr; row += nt >> 5) {
                const double *arow = ainv + (size_t)row * n0;
                double s = 0.0;
                for (int j = lane; j < n0; j += 32) s = fma_rn(arow[j], dwide[j], s);
                s = warp_sum(s);
                if (lane == 0) sc[row] = (V)s;
            }
        }
    }
    // ---- up: prolongation and post-smoothing
    for (int l = 1; l <= top; ++l) {
        const CoarseLevel<V> &L = P.lev[l];
        const bool solo = L.solo != 0;
        if (solo && rank != 0) continue;
        sync(solo);   // the level below is complete (the cluster waits for block 0's solo levels here)
        const int r0 = first(l), nr = rows(l);
        const V *a = vr + L.aofs, *dinv = vr + L.iofs, *dfac = vr + L.fofs;
        V *sc = vsc(l), *dA = vdA(l), *dB = vdB(l), *w = vw(l);
        coarse_prolong<V>(L, P.lev[l - 1], vsc(l - 1), sc, dfac, P.nu2 > 0 ? w : (V *)nullptr, r0, nr);
        V *dbase = (P.nu1 & 1) ? dB : dA;   // the defect after pre-smoothing
        for (int k = 0; k < P.nu2; ++k) {
            sync(solo);
            const V *x = (k == 0) ? w : dbase;
            V *out = (k < P.nu2 - 1) ? ((dbase == dA) ? dB : dA) : nullptr;
            coarse_step<V, S>(L, a, dinv, x, dbase, sc, out, SC_ADD_FROM_NEW, r0, nr);
            if (out) dbase = out;
        }
    }
    __syncthreads();
    {
        const V *sc = vsc(top);
        const int r0 = first(top), nr = rows(top);
        for (int i = tid; i < nr; i += nt) P.sc_out[r0 + i] = sc[i];
    }
    cluster_sync();   // no block leaves while another reads its shared memory
}

namespace {

// one cluster of ctas blocks, with programmatic dependent launch as
// UG_LAUNCH_PDL
template <class V>
cudaLaunchConfig_t coarse_config(Ctx &c, int ctas, size_t smem, cudaLaunchAttribute (&at)[2], bool pdl)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kCoarseThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c.stream;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 2 : 1;
    return cfg;
}

template <class V>
using CoarseKernel = void (*)(const CoarsePlan<V> *, const int *);

template <class V>
CoarseKernel<V> coarse_kernel(int S)
{
    switch (S) {
    case 7: return k_coarse_cycle<V, 7>;
    case 9: return k_coarse_cycle<V, 9>;
    case 15: return k_coarse_cycle<V, 15>;
    case 27: return k_coarse_cycle<V, 27>;
    default: throw Error{UG4GB_ERR_INVALID, "coarse cycle: unsupported stencil width"};
    }
}

}  // namespace

template <class V>
void coarse_cycle(Ctx &c, const CoarsePlan<V> *plan_dev, int ctas, int S, size_t smem_bytes, const int *skip)
{
    cudaLaunchAttribute at[2];
    const cudaLaunchConfig_t cfg = coarse_config<V>(c, ctas, smem_bytes, at, c.pdl && !c.profiling);
    cudaEvent_t ev_a = nullptr;
    if (c.profiling) {
        ev_a = prof_event(c);
        UG_CUDA(cudaEventRecord(ev_a, c.stream));
    }
    UG_CUDA(cudaLaunchKernelEx(&cfg, coarse_kernel<V>(S), plan_dev, skip));
    c.launches++;
    if (c.profiling) {
        cudaEvent_t ev_b = prof_event(c);
        UG_CUDA(cudaEventRecord(ev_b, c.stream));
        c.prof.push_back(ProfRec{c.prof_tag + "|k_coarse_cycle<" + std::to_string(S) + ">", ev_a, ev_b});
    }
}

bool coarse_width_ok(int S) { return S == 7 || S == 9 || S == 15 || S == 27; }

template <class V>
int coarse_prepare(Ctx &c, int S, int most_blocks, size_t smem_bytes)
{
    const CoarseKernel<V> kernel = coarse_kernel<V>(S);
    UG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes));
    UG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    // a cluster needs a processing cluster of the GPU (or of the partition of it
    // that is visible) with that many free SMs
    for (int ctas = 16; ctas >= 1; ctas /= 2) {
        if (ctas > most_blocks) continue;
        cudaLaunchAttribute at[2];
        const cudaLaunchConfig_t cfg = coarse_config<V>(c, ctas, smem_bytes, at, false);
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) == cudaSuccess && clusters > 0) return ctas;
        (void)cudaGetLastError();
    }
    return 0;
}

template void coarse_cycle<double>(Ctx &, const CoarsePlan<double> *, int, int, size_t, const int *);
template void coarse_cycle<float>(Ctx &, const CoarsePlan<float> *, int, int, size_t, const int *);
template int coarse_prepare<double>(Ctx &, int, int, size_t);
template int coarse_prepare<float>(Ctx &, int, int, size_t);

}  // namespace ug4gb
