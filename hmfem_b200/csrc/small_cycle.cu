// small_cycle.cu -- the coarse end of the V-cycle in one launch.
//
// The Chebyshev levels of a few thousand rows and the coarse solve are ten
// kernels a level that each wait for a chain of dependent loads and hold a
// handful of warps: 4.2 us a kernel inside the captured iteration whatever
// the level's size.  Here one cluster of CTAs runs them all.  Each CTA owns a
// contiguous block of every level's rows and holds their matrix entries,
// transfers and vectors in shared memory, loaded before the kernel waits for
// its predecessor (nothing in them changes during a solve); the vectors that
// rows gather from have a place for every row in every CTA, each row's new
// value is written through distributed shared memory to the CTAs whose rows
// read it (sets found at setup: a few neighbours of sixteen), and a cluster
// barrier separates the phases.  The matrix is read once per V-cycle instead of once
// per sweep, and a phase costs a shared-memory row sum and a barrier.
//
// Row by row the operations are those of the level kernels (cycle.cu:
// pre_row, cheb0_row, cheb_step_row, k_restrict, k_prolong_add,
// k_dense_solve), in the same order: same bits.
//
// Bound by the phases' latency: ~1000 cycles for the cluster barrier, as much
// for a row (its loads and the stores to the readers), twelve phases for one
// level and the coarse solve.  Measured, one CG iteration in the captured
// graph (us), level kernels -> this: 32^3 FP64 91 -> 67 (levels of 2176 and
// 320 rows), 87x61x75 FP64 220 -> 180 (3490, 482), 160x96x64 reduced 248 ->
// 197 (8200, 1068, 147), 210x42x20 reduced 124 -> 103 (1590, 239), 128^3
// reduced 331 -> 299, 256^3 reduced 1360 -> 1311.
//
// Which levels: as many as fit.  A level of n rows needs two whole vectors
// per CTA beside its share of the entries, so with 16 CTAs the shared memory
// ends near 9000 FP32 or 4000 FP64 rows; keeping only the rows a CTA reads
// let a level of 11550 rows in, but its phases (2.6 us) were no faster than
// its kernels and the window checks cost the small levels more.  16 CTAs
// against 8: 182 against 193 us at 87x61x75, 197 against 218 at 160x96x64.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "cycle.cuh"

namespace hm {

namespace {

namespace cg = cooperative_groups;

constexpr int kScThreads = 1024;
constexpr size_t kScSmem = 220 * 1024;
constexpr int kScRows = 16384;
constexpr int kScDegree = 10;
constexpr unsigned kScNone = 0xffffffffu;

// One Chebyshev level; the offsets are into each CTA's shared memory.
struct ScLevel {
    const long long *sptr;
    const int *col;
    const void *val, *dinv;
    const int *prow, *pcol, *rrow, *rcol;
    int n, nc;
    int own, cown;  // rows and coarse rows per CTA (the last CTAs may have fewer)
    unsigned o_val, o_col, o_slice, o_prow, o_pcol, o_rrow, o_rcol;
    unsigned o_f, o_u, o_r, o_dv;  // own rows
    unsigned o_b[2];               // vectors of all rows
    int at[kScCtas + 1][3];        // entries, P and R entries before each CTA's rows
};

struct ScArgs {
    ScLevel lv[kScLevels];
    int levels, degree;
    int dn, down;               // coarse solve: rows, rows per CTA
    unsigned o_df, o_du;        // its right-hand side and solution (all rows)
    const double *dense;        // explicit inverse; o_dense: the CTA's rows of it,
    unsigned o_dense;           // kScNone: read through L2
    const void *f, *d0;         // of the first level
    void *u;
    double ith, c1[kScDegree], c2[kScDegree];
    const unsigned *masks;      // [level][CTA][ScMask], the coarse solve's last
    const Ctl *ctl;
};

// The CTAs that read a CTA's rows: through the matrix, through R (rs), and
// through the finer level's P (u).
enum ScMask { SC_A, SC_R, SC_P, SC_MASKS };

// t -/+ sum of a row's entries in stored order; o: the row's first entry, 32
// apart; eight (FP64: four) at a time so that the gathers overlap
template <class T, class M, bool SUB, class X>
__device__ __forceinline__ T sc_row(T t, const M *val, const int *col, int o, int wd, int row, X x)
{
    constexpr int CH = sizeof(T) == 8 ? 4 : 8;
    for (int k0 = 0; k0 < wd; k0 += CH, o += 32 * CH) {
        T a[CH], xv[CH];
#pragma unroll
        for (int q = 0; q < CH; q++) {
            const bool ok = k0 + q < wd;
            if constexpr (std::is_same<M, unsigned>::value) {  // Sell::pk
                const unsigned e = ok ? val[o + 32 * q] : 0u;
                a[q] = (T)__uint_as_float(e << 16);
                xv[q] = ok ? x(row + ((int)e >> 16)) : (T)0;
            } else {
                a[q] = ok ? (T)val[o + 32 * q] : (T)0;
                xv[q] = ok ? x(col[o + 32 * q]) : (T)0;
            }
        }
#pragma unroll
        for (int q = 0; q < CH; q++)
            if (k0 + q < wd) t = SUB ? nmul_add(t, a[q], xv[q]) : pmul_add(t, a[q], xv[q]);
    }
    return t;
}

template <class T, class M>
__global__ void __launch_bounds__(kScThreads, 1)
k_small_cycle(const __grid_constant__ ScArgs a)
{
    using A = Ar<T>;
    constexpr bool kCol = !std::is_same<M, unsigned>::value;
    extern __shared__ __align__(16) unsigned char sm[];
    cg::cluster_group cl = cg::this_cluster();
    const int me = (int)cl.block_rank();
    const int tid = threadIdx.x;
    auto at = [&](unsigned o) { return sm + o; };
    // this CTA's rows of a level: [r0, r1)
    auto first = [&](int own, int n) { const int r = me * own; return r < n ? r : n; };
    // writes entry i of the vector at o in the CTAs of a set
    const unsigned base = (unsigned)__cvta_generic_to_shared(sm);
    auto share = [&](unsigned cs, unsigned o, int i, T v) {
        const unsigned p = base + o + (unsigned)(i * sizeof(T));
        for (; cs; cs &= cs - 1) {
            unsigned q;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(q) : "r"(p), "r"(__ffs(cs) - 1));
            if constexpr (sizeof(T) == 8)
                asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(q), "d"(v) : "memory");
            else
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(q), "f"(v) : "memory");
        }
    };
    __shared__ unsigned masks[kScLevels + 1][SC_MASKS];
    if (tid < (a.levels + 1) * SC_MASKS)
        (&masks[0][0])[tid] = a.masks[(tid / SC_MASKS * kScCtas + me) * SC_MASKS + tid % SC_MASKS];
    auto vec = [&](int l, int k) { return (T *)at(a.lv[l].o_b[k]); };
    // ---- what does not change during a solve
    for (int l = 0; l < a.levels; l++) {
        const ScLevel &L = a.lv[l];
        const int r0 = first(L.own, L.n), r1 = min(r0 + L.own, L.n);
        const int q0 = r0 / 32, q1 = (r1 + 31) / 32;  // own is a multiple of 32
        const int e0 = L.at[me][0], ne = L.at[me + 1][0] - e0;
        int *slice = (int *)at(L.o_slice);
        for (int q = tid; q <= q1 - q0; q += kScThreads) slice[q] = (int)L.sptr[q0 + q] - e0;
        // entries: multiples of 32 on 128-byte boundaries
        const uint4 *sv = (const uint4 *)((const M *)L.val + e0);
        uint4 *dv4 = (uint4 *)at(L.o_val);
        for (int k = tid; k < (int)(ne * sizeof(M) / 16); k += kScThreads) dv4[k] = sv[k];
        if (kCol) {
            const uint4 *sc = (const uint4 *)(L.col + e0);
            uint4 *dc = (uint4 *)at(L.o_col);
            for (int k = tid; k < ne / 4; k += kScThreads) dc[k] = sc[k];
        }
        T *dv = (T *)at(L.o_dv);
        for (int i = tid; i < r1 - r0; i += kScThreads) dv[i] = ((const T *)L.dinv)[r0 + i];
        // transfers: P of the own rows, R of the own coarse rows
        int *pr = (int *)at(L.o_prow), *pc = (int *)at(L.o_pcol);
        const int p0 = L.at[me][1], p1 = L.at[me + 1][1];
        for (int i = tid; i <= r1 - r0; i += kScThreads) pr[i] = L.prow[r0 + i] - p0;
        for (int k = tid; k < p1 - p0; k += kScThreads) pc[k] = L.pcol[p0 + k];
        const int c0 = first(L.cown, L.nc), c1 = min(c0 + L.cown, L.nc);
        int *rr = (int *)at(L.o_rrow), *rc = (int *)at(L.o_rcol);
        const int s0 = L.at[me][2], s1 = L.at[me + 1][2];
        for (int i = tid; i <= c1 - c0; i += kScThreads) rr[i] = L.rrow[c0 + i] - s0;
        for (int k = tid; k < s1 - s0; k += kScThreads) rc[k] = L.rcol[s0 + k];
    }
    if (a.o_dense != kScNone) {
        const int r0 = first(a.down, a.dn), r1 = min(r0 + a.down, a.dn);
        const double *src = a.dense + r0 * (long)a.dn;
        double *dst = (double *)at(a.o_dense);
        for (int k = tid; k < (r1 - r0) * a.dn; k += kScThreads) dst[k] = src[k];
    }
    cl.sync();  // every CTA runs: its shared memory may be written to
    PDL_ENTRY();
    {
        const ScLevel &L = a.lv[0];
        T *b0 = vec(0, 0), *f = (T *)at(L.o_f);
        const bool over = finished(a.ctl);  // the same in every CTA
        for (int i = tid; i < L.n; i += kScThreads) b0[i] = ((const T *)a.d0)[i];
        const int r0 = first(L.own, L.n), r1 = min(r0 + L.own, L.n);
        for (int i = tid; i < r1 - r0; i += kScThreads) f[i] = ((const T *)a.f)[r0 + i];
        if (over) return;
    }
    __syncthreads();
    const int K = a.degree;
    // ---- down: smoothing from zero, residual, restriction
    for (int l = 0; l < a.levels; l++) {
        const ScLevel &L = a.lv[l];
        const int r0 = first(L.own, L.n), rows = min(r0 + L.own, L.n) - r0;
        const M *val = (const M *)at(L.o_val);
        const int *col = (const int *)at(L.o_col), *slice = (const int *)at(L.o_slice);
        T *f = (T *)at(L.o_f), *u = (T *)at(L.o_u), *r = (T *)at(L.o_r);
        const T *dv = (const T *)at(L.o_dv);
        for (int k = 1; k < K; k++) {
            const T *din = vec(l, (k - 1) & 1);
            const T c1 = (T)a.c1[k], c2 = (T)a.c2[k];
            for (int i = tid; i < rows; i += kScThreads) {
                const int o = slice[i >> 5], wd = (slice[(i >> 5) + 1] - o) >> 5;
                const T ad = sc_row<T, M, false>((T)0, val, col, o + (i & 31), wd, r0 + i,
                                                 [&](int c) { return din[c]; });
                const T di = dv[i], dold = din[r0 + i];
                const T rn = k == 1 ? mul_sub(di, f[i], di, ad) : nmul_add(r[i], di, ad);
                const T dn = mul_add(c1, dold, c2, rn);
                const T un = k == 1 ? A::add(dold, dn) : A::add(u[i], dn);
                u[i] = un;
                r[i] = rn;
                // after the last step the residual gathers u
                share(masks[l][SC_A], L.o_b[k & 1], r0 + i, k == K - 1 ? un : dn);
            }
            cl.sync();
        }
        {
            const T *ub = vec(l, (K - 1) & 1);
            const int *pr = (const int *)at(L.o_prow);
            for (int i = tid; i < rows; i += kScThreads) {
                const int o = slice[i >> 5], wd = (slice[(i >> 5) + 1] - o) >> 5;
                const T t = sc_row<T, M, true>(f[i], val, col, o + (i & 31), wd, r0 + i,
                                               [&](int c) { return ub[c]; });
                const int pc = pr[i + 1] - pr[i];
                share(masks[l][SC_R], L.o_b[K & 1], r0 + i, pc == 1 ? t : A::div(t, (T)pc));
            }
            cl.sync();
        }
        {
            const T *rs = vec(l, K & 1);
            const int *rr = (const int *)at(L.o_rrow), *rc = (const int *)at(L.o_rcol);
            const int c0 = first(L.cown, L.nc), crows = min(c0 + L.cown, L.nc) - c0;
            for (int e = tid; e < crows; e += kScThreads) {
                T acc = (T)0;
                for (int k = rr[e]; k < rr[e + 1]; k++) acc = A::add(acc, rs[rc[k]]);
                if (l + 1 < a.levels) {
                    const ScLevel &N = a.lv[l + 1];
                    ((T *)at(N.o_f))[e] = acc;
                    share(masks[l + 1][SC_A], N.o_b[0], c0 + e,
                          A::mul(A::mul((T)a.ith, acc), ((const T *)at(N.o_dv))[e]));
                } else {
                    share(masks[l + 1][SC_A], a.o_df, c0 + e, acc);
                }
            }
            cl.sync();
        }
    }
    // ---- coarse solve: a warp per row of the inverse
    {
        const T *f = (const T *)at(a.o_df);
        const int lane = tid & 31, r0 = first(a.down, a.dn), r1 = min(r0 + a.down, a.dn);
        for (int i = r0 + (tid >> 5); i < r1; i += kScThreads / 32) {
            const double *row = a.o_dense != kScNone
                                    ? (const double *)at(a.o_dense) + (i - r0) * a.dn
                                    : a.dense + i * (long)a.dn;
            double acc = 0.0;
#pragma unroll 8
            for (int j = lane; j < a.dn; j += 32) acc += row[j] * (double)f[j];
            acc = warp_sum(acc);
            // a lane per reader
            share(masks[a.levels][SC_P] & (1u << lane), a.o_du, i, (T)acc);
        }
        cl.sync();
    }
    // ---- up: prolongation, smoothing
    for (int l = a.levels - 1; l >= 0; l--) {
        const ScLevel &L = a.lv[l];
        const int r0 = first(L.own, L.n), rows = min(r0 + L.own, L.n) - r0;
        const M *val = (const M *)at(L.o_val);
        const int *col = (const int *)at(L.o_col), *slice = (const int *)at(L.o_slice);
        T *f = (T *)at(L.o_f), *u = (T *)at(L.o_u), *r = (T *)at(L.o_r);
        const T *dv = (const T *)at(L.o_dv);
        const T *uc = l + 1 < a.levels ? vec(l + 1, K & 1)
                                       : (const T *)at(a.o_du);
        const int *pr = (const int *)at(L.o_prow), *pc = (const int *)at(L.o_pcol);
        for (int i = tid; i < rows; i += kScThreads) {
            const int b = pr[i], c = pr[i + 1] - b;
            T un = u[i];
            if (c > 0) {
                T t = uc[pc[b]];
                for (int k = 1; k < c; k++) t = A::add(t, uc[pc[b + k]]);
                un = A::add(un, c == 1 ? t : A::div(t, (T)c));
            }
            u[i] = un;
            share(masks[l][SC_A], L.o_b[0], r0 + i, un);
        }
        cl.sync();
        {
            const T *ub = vec(l, 0);
            for (int i = tid; i < rows; i += kScThreads) {
                const int o = slice[i >> 5], wd = (slice[(i >> 5) + 1] - o) >> 5;
                const T t = sc_row<T, M, true>(f[i], val, col, o + (i & 31), wd, r0 + i,
                                               [&](int c) { return ub[c]; });
                const T di = dv[i];
                r[i] = A::mul(di, t);
                share(masks[l][SC_A], L.o_b[1], r0 + i,
                      A::mul(A::mul((T)a.ith, t), di));
            }
            cl.sync();
        }
        for (int k = 1; k < K; k++) {
            const T *din = vec(l, k & 1);
            const T c1 = (T)a.c1[k], c2 = (T)a.c2[k];
            const bool last = k == K - 1;
            for (int i = tid; i < rows; i += kScThreads) {
                const int o = slice[i >> 5], wd = (slice[(i >> 5) + 1] - o) >> 5;
                const T ad = sc_row<T, M, false>((T)0, val, col, o + (i & 31), wd, r0 + i,
                                                 [&](int c) { return din[c]; });
                const T di = dv[i], dold = din[r0 + i];
                const T rn = nmul_add(r[i], di, ad);
                const T dn = mul_add(c1, dold, c2, rn);
                const T un = k == 1 ? A::add(A::add(u[i], dold), dn) : A::add(u[i], dn);
                u[i] = un;
                r[i] = rn;
                if (last && l == 0) ((T *)a.u)[r0 + i] = un;
                else share(masks[l][last ? SC_P : SC_A], L.o_b[(k - 1) & 1], r0 + i,
                           last ? un : dn);
            }
            if (!(last && l == 0)) cl.sync();
        }
    }
}

// What the layout needs of a candidate level and a CTA count: entry, P and R
// counts at the CTAs' row boundaries, and the readers of every CTA's rows
// (masks zeroed before).
struct ScScan {
    const long long *sptr;
    const int *col, *prow, *pcol, *rrow, *rcol;
    int n, nc, own, cown;
};
struct ScScans {
    ScScan lv[kScLevels];
    int levels, ctas;
};
struct ScFound {
    int at[3];
};

// a block per level and CTA
__global__ void k_sc_scan(const __grid_constant__ ScScans a, ScFound *found, unsigned *masks)
{
    const int l = blockIdx.x, c = blockIdx.y;
    const ScScan &L = a.lv[l];
    __shared__ unsigned s_m[3];   // owners read through A, R, P
    if (threadIdx.x < 3) s_m[threadIdx.x] = 0u;
    __syncthreads();
    unsigned m[3] = {0u, 0u, 0u};
    const int r0 = min(c * L.own, L.n), r1 = min(r0 + L.own, L.n);
    for (int i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
        m[0] |= 1u << c;  // a row reads its own entries too
        const long long o = L.sptr[i >> 5];
        const int wd = (int)((L.sptr[(i >> 5) + 1] - o) >> 5);
        for (int k = 0; k < wd; k++) m[0] |= 1u << (L.col[o + 32 * k + (i & 31)] / L.own);
        for (int k = L.prow[i]; k < L.prow[i + 1]; k++) m[2] |= 1u << (L.pcol[k] / L.cown);
    }
    const int e0 = min(c * L.cown, L.nc), e1 = min(e0 + L.cown, L.nc);
    for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x)
        for (int k = L.rrow[e]; k < L.rrow[e + 1]; k++) m[1] |= 1u << (L.rcol[k] / L.own);
    for (int k = 0; k < 3; k++)
        if (m[k]) atomicOr(&s_m[k], m[k]);
    __syncthreads();
    if (threadIdx.x != 0) return;
    ScFound f;
    f.at[0] = (int)L.sptr[(r0 + 31) / 32];
    f.at[1] = L.prow[r0];
    f.at[2] = L.rrow[e0];
    found[l * (kScCtas + 1) + c] = f;
    if (c == a.ctas) return;  // only the end of the counts
    for (int k = 0; k < 3; k++)
        for (unsigned b = s_m[k]; b; b &= b - 1)
            atomicOr(masks + (((k == 2 ? l + 1 : l) * kScCtas + __ffs(b) - 1) * SC_MASKS +
                              (k == 0 ? SC_A : k == 1 ? SC_R : SC_P)),
                     1u << c);
    // the coarse solve's right-hand side is read by every CTA
    if (l == a.levels - 1 && threadIdx.x == 0)
        for (int o = 0; o < a.ctas; o++)
            atomicOr(masks + (((l + 1) * kScCtas + o) * SC_MASKS + SC_A), 1u << c);
}

template <class T, class M>
cudaError_t sc_launch(const ScArgs &a, int ctas, size_t smem, bool pdl, cudaStream_t st,
                      int *active)
{
    // (the attributes are the process's: the same values from every thread)
    cudaError_t e = cudaFuncSetAttribute(
        k_small_cycle<T, M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_small_cycle<T, M>,
                                 cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kScThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    if (active) {  // only asked whether such a cluster fits on the device
        cfg.numAttrs = 1;
        return cudaOccupancyMaxActiveClusters(active, k_small_cycle<T, M>, &cfg);
    }
    cfg.numAttrs = pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k_small_cycle<T, M>, a);
}

template <class F>
cudaError_t sc_typed(int kind, F fn)
{
    switch (kind) {
    case 0: return fn((double *)nullptr, (double *)nullptr);
    case 1: return fn((float *)nullptr, (float *)nullptr);
    default: return fn((float *)nullptr, (unsigned *)nullptr);
    }
}

// the launch's arguments but for the smoother's coefficients
ScArgs sc_args(const Solver &s)
{
    const SmallCycle &S = s.small;
    const int lo = S.first, d = s.direct_level;
    ScArgs a{};
    a.levels = d - lo;
    a.degree = s.opt.cheb_degree;
    for (int l = lo; l < d; l++) {
        const Level &L = s.lv[l];
        const SmallLayout::Lv &o = S.layout.lv[l - lo];
        ScLevel &A = a.lv[l - lo];
        A.sptr = L.S.sptr;
        A.col = L.S.col;
        A.val = S.kind == 0 ? (const void *)L.S.val : S.kind == 1 ? (const void *)L.S.val32
                                                                  : (const void *)L.S.pk;
        A.dinv = S.kind == 0 ? (const void *)L.dsm : (const void *)L.dsm32;
        A.prow = L.P.rowptr;
        A.pcol = L.P.col;
        A.rrow = L.R.rowptr;
        A.rcol = L.R.col;
        A.n = L.A.n;
        A.nc = L.nc;
        A.own = o.own;
        A.cown = o.cown;
        A.o_val = o.o_val; A.o_col = o.o_col; A.o_slice = o.o_slice;
        A.o_prow = o.o_prow; A.o_pcol = o.o_pcol; A.o_rrow = o.o_rrow; A.o_rcol = o.o_rcol;
        A.o_f = o.o_f; A.o_u = o.o_u; A.o_r = o.o_r; A.o_dv = o.o_dv;
        A.o_b[0] = o.o_b[0]; A.o_b[1] = o.o_b[1];
        for (int c = 0; c <= S.ctas; c++)
            for (int k = 0; k < 3; k++) A.at[c][k] = o.at[c][k];
    }
    a.dn = s.lv[d].A.n;
    a.down = (int)ceil_div(a.dn, S.ctas);
    a.o_df = S.layout.o_df;
    a.o_du = S.layout.o_du;
    a.dense = s.dense_L;
    a.o_dense = S.layout.o_dense;
    const Level &F = s.lv[lo];
    if (S.kind == 0) { a.f = F.f; a.d0 = F.ub; a.u = F.ua; }
    else { a.f = F.f32; a.d0 = F.ub32; a.u = F.ua32; }
    a.masks = S.masks + S.mask0;
    return a;
}

}  // namespace

// Lays the launch out: which levels and how many CTAs.  Leaves S.first = -1
// where the form does not apply (no coarse solve above a Chebyshev level,
// values stored in another form, or nothing fits).
int small_cycle_build(Solver &s, cudaStream_t st)
{
    SmallCycle &S = s.small;
    S.first = -1;
    const int d = s.direct_level;
    // HMFEM_SMALL_CYCLE=0 keeps the level kernels (a check of this form)
    const char *on = getenv("HMFEM_SMALL_CYCLE");
    if (d < 1 || s.opt.cheb_degree >= kScDegree || (on && atoi(on) == 0)) return HMFEM_OK;
    // 0 FP64, 1 FP32, 2 packed BF16 entries
    auto kind_of = [&](const Level &L, int l) {
        if (s.opt.precision == 0) return 0;
        return s.use_bf16(l) ? (L.S.pk ? 2 : -1) : 1;
    };
    int lo = d;
    const int kind = kind_of(s.lv[d - 1], d - 1);
    while (lo > 1 && d - lo < kScLevels && s.lv[lo - 1].cheb && !s.lv[lo - 1].gs &&
           !s.lv[lo - 1].g19.v && kind_of(s.lv[lo - 1], lo - 1) == kind &&
           s.lv[lo - 1].A.n <= kScRows)
        lo--;
    if (lo == d || kind < 0) return HMFEM_OK;
    const size_t T = kind == 0 ? 8 : 4, M = kind == 0 ? 8 : 4;
    const bool has_col = kind != 2;
    const size_t mask_bytes = sizeof(unsigned) * (kScLevels + 1) * kScCtas * SC_MASKS;
    if (!S.masks) S.masks = (unsigned *)dalloc(mask_bytes);
    ScFound *dev = (ScFound *)dalloc(sizeof(ScFound) * kScLevels * (kScCtas + 1));
    if (!S.masks || !dev) return HMFEM_E_CUDA;
    struct Free { void *p; ~Free() { dfree(p); } } free_dev{dev};
    for (int ctas = kScCtas; ctas >= 8; ctas /= 2) {
        ScScans q{};
        q.levels = d - lo;
        q.ctas = ctas;
        const int down = (int)ceil_div(s.lv[d].A.n, ctas);
        auto own_of = [&](int l) {
            return l == d ? down : 32 * (int)ceil_div(ceil_div(s.lv[l].A.n, 32), ctas);
        };
        for (int l = lo; l < d; l++) {
            const Level &L = s.lv[l];
            q.lv[l - lo] = {L.S.sptr, L.S.col, L.P.rowptr, L.P.col, L.R.rowptr, L.R.col,
                            L.A.n,    L.nc,    own_of(l),  own_of(l + 1)};
        }
        HM_CUDA(cudaMemsetAsync(S.masks, 0, mask_bytes, st));
        k_sc_scan<<<dim3(q.levels, ctas + 1), 256, 0, st>>>(q, dev, S.masks);
        HM_LAUNCHED();
        ScFound h[kScLevels][kScCtas + 1];
        static_assert(sizeof(h) <= sizeof(int) * (PIN_WORDS - PIN_BLOCK), "pinned words");
        HM_CHECK(read_back(PIN_BLOCK, dev, (int)(sizeof(h) / sizeof(int)), st));
        HM_CUDA(cudaStreamSynchronize(st));
        memcpy(h, pinned_words() + PIN_BLOCK, sizeof(h));
        auto most = [&](int l, int k) {
            int m = 0;
            for (int c = 0; c < ctas; c++) m = std::max(m, h[l - lo][c + 1].at[k] - h[l - lo][c].at[k]);
            return (size_t)m;
        };
        // from the coarse solve upwards while the shared memory lasts
        SmallLayout P{};
        unsigned top = 0;
        auto take = [&](size_t bytes) {
            const unsigned o = top;
            top += (unsigned)((bytes + 127) & ~(size_t)127);
            return o;
        };
        P.o_df = take(T * s.lv[d].A.n);
        P.o_du = take(T * s.lv[d].A.n);
        int from = d;
        for (int l = d - 1; l >= lo; l--) {
            const unsigned before = top;
            SmallLayout::Lv &o = P.lv[l - lo];
            const int own = own_of(l), cown = own_of(l + 1);
            o.own = own;
            o.cown = cown;
            for (int c = 0; c <= ctas; c++)
                for (int k = 0; k < 3; k++) o.at[c][k] = h[l - lo][c].at[k];

            o.o_val = take(M * most(l, 0));
            o.o_col = take(has_col ? 4 * most(l, 0) : 0);
            o.o_slice = take(4 * (own / 32 + 1));
            o.o_prow = take(4 * (own + 1));
            o.o_pcol = take(4 * most(l, 1));
            o.o_rrow = take(4 * (cown + 1));
            o.o_rcol = take(4 * most(l, 2));
            o.o_f = take(T * own);
            o.o_u = take(T * own);
            o.o_r = take(T * own);
            o.o_dv = take(T * own);
            o.o_b[0] = take(T * s.lv[l].A.n);
            o.o_b[1] = take(T * s.lv[l].A.n);
            if (top > kScSmem) {
                top = before;
                break;
            }
            from = l;
        }
        if (from == d) continue;
        P.o_dense = top;
        if (top + 8 * (size_t)down * s.lv[d].A.n <= kScSmem) take(8 * (size_t)down * s.lv[d].A.n);
        else P.o_dense = kScNone;
        int active = 0;
        const cudaError_t e = sc_typed(kind, [&](auto *t, auto *m) {
            using TT = typename std::remove_pointer<decltype(t)>::type;
            using MM = typename std::remove_pointer<decltype(m)>::type;
            return sc_launch<TT, MM>(ScArgs{}, ctas, top, false, st, &active);
        });
        if (e != cudaSuccess || active < 1) {
            cudaGetLastError();
            continue;
        }
        for (int l = from; l < d; l++) P.lv[l - from] = P.lv[l - lo];
        S.layout = P;
        S.first = from;
        S.ctas = ctas;
        S.kind = kind;
        S.smem = top;
        S.mask0 = (from - lo) * kScCtas * SC_MASKS;
        return HMFEM_OK;
    }
    return HMFEM_OK;
}

// The V-cycle from level s.small.first down and back (f and the seeded first
// direction of that level in, its u out).
int small_cycle(Solver &s, const double *c1, const double *c2, double ith, const Ctl *ctl,
                cudaStream_t st)
{
    const SmallCycle &S = s.small;
    ScArgs a = sc_args(s);
    a.ith = ith;
    for (int k = 1; k < a.degree; k++) {
        a.c1[k] = c1[k];
        a.c2[k] = c2[k];
    }
    a.ctl = ctl;
    KRec rec{nullptr, t_klevel, nullptr, nullptr};
    if (t_kprof) {
        cudaEventCreate(&rec.e0);
        cudaEventCreate(&rec.e1);
        cudaEventRecord(rec.e0, st);
    }
    HM_CUDA(sc_typed(S.kind, [&](auto *t, auto *m) {
        using TT = typename std::remove_pointer<decltype(t)>::type;
        using MM = typename std::remove_pointer<decltype(m)>::type;
        rec.fn = (const void *)k_small_cycle<TT, MM>;
        return sc_launch<TT, MM>(a, S.ctas, S.smem, g_pdl, st, nullptr);
    }));
    if (t_kprof) {
        cudaEventRecord(rec.e1, st);
        t_kprof->push_back(rec);
    }
    HM_COUNT();
    return HMFEM_OK;
}

}  // namespace hm
