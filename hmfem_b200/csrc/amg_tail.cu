// amg_tail.cu -- the small end of the AMG hierarchy in one launch.
//
// Below a few hundred rows a coarsening step is all launches, allocations and
// size read-backs (0.6 ms a level for microseconds of work, and a hierarchy
// has four to six such levels).  Here one CTA coarsens a level of at most
// kTailRows rows, then the one it made, and so on to the end of the
// hierarchy; the host reads the sizes back once.  Same split, numbering, P,
// R and Galerkin values as amg_coarsen's general path (amg.h:1-32, 326-403,
// 408-582), bit for bit: every sum takes its terms in the same order and
// starts from -0.0, which leaves the first term as it is.
//
// With at most 512 rows a set of rows is 16 words, so the steps work on bit
// sets: the greedy split tests a row's lower neighbours against the C rows
// with one vote per row; the bit row of a coarse unknown's fine rows is R in
// ascending order without a sort; the bit row of A P's columns is its
// pattern, its values a dense row.  Bound by the latency of the rows' serial
// chains on one SM.  Measured (host time of the steps): 320 -> 1 rows, four
// steps, 2.1 -> 0.26 ms; 482 -> 1, five steps, 2.2 -> 0.40 ms.  Above 512 rows
// the bit sets no longer fit, and one SM would soon take longer than the
// general path's launches.
#include <stdlib.h>
#include <string.h>

#include <algorithm>

#include "hm.cuh"

namespace hm {

namespace {

constexpr int kTailRows = 512;
constexpr int kTailWords = kTailRows / 32;
constexpr int kTailThreads = 1024;
constexpr int kTailWarps = kTailThreads / 32;
constexpr int kTailLevels = 64;
// accumulator rows in shared memory: eight lanes per row of A P while 128
// rows of nc entries fit, a warp per row otherwise
constexpr int kTailAcc = kTailWarps * kTailRows;  // doubles
constexpr size_t kTailArena = 2u << 20;

struct TailLevel {
    int n, nc, pnnz, nnz;  // rows, coarse rows, P entries, coarse entries
    // arena offsets: transfer of this level, then the coarse level
    unsigned sel, cid, prow, pcol, pw, pw32, rrow, rcol, arow, acol, aval, dinv, dinv32;
};

struct TailOut {
    int levels;    // levels coarsened
    unsigned top;  // arena bytes in use after them
    TailLevel lv[kTailLevels];
};

// The arena's size; a smaller one when the environment sets
// HMFEM_TEST_TAIL_ARENA (a test makes the levels run out of room and checks
// that the general path goes on from there to the same hierarchy).
size_t tail_arena_bytes()
{
    const char *e = getenv("HMFEM_TEST_TAIL_ARENA");
    if (!e || !*e) return kTailArena;
    const long long v = atoll(e);
    return v < 0 ? 0 : std::min((size_t)v, kTailArena);
}

struct TailShared {
    double acc[kTailAcc];
    unsigned bits[kTailRows][kTailWords];   // lower neighbours; then the fine rows of a coarse row
    unsigned apb[kTailRows][kTailWords];    // columns of A P
    double w[kTailRows];
    int prow[kTailRows + 1], rrow[kTailRows + 1], cid[kTailRows + 1];
    unsigned cset[kTailWords];
    int wsum[kTailWarps];
};

// exclusive scan of v[0..n] (v[n] = 0 on entry, the total on exit), n < blockDim.x
__device__ void block_scan(int *v, int n, int *wsum)
{
    const int i = threadIdx.x, lane = i & 31, w = i >> 5;
    const int x = i < n ? v[i] : 0;
    int s = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += y;
    }
    if (lane == 31) wsum[w] = s;
    __syncthreads();
    if (w == 0) {
        int t = wsum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        wsum[lane] = t;
    }
    __syncthreads();
    if (i <= n) v[i] = s - x + (w > 0 ? wsum[w - 1] : 0);
    __syncthreads();
}

__device__ __forceinline__ bool bit_of(const unsigned *b, int i) { return (b[i >> 5] >> (i & 31)) & 1u; }

// Rows of A P by groups of G lanes: row i's accumulators in shared memory,
// the entries a_ij in stored order, the columns of P(j) side by side.
template <int G>
__device__ void tail_ap(TailShared &S, int n, int nc, const int *rowptr, const int *col,
                        const double *val, const int *pcol, double *ap)
{
    const int gl = threadIdx.x % G, grp = threadIdx.x / G, groups = kTailThreads / G;
    const unsigned mask = G == 32 ? 0xffffffffu
                                  : ((1u << (G & 31)) - 1u) << ((threadIdx.x & 31) / G * G);
    double *acc = S.acc + grp * nc;
    for (int i = grp; i < n; i += groups) {
        for (int d = gl; d < nc; d += G) acc[d] = -0.0;
        for (int q = gl; q < kTailWords; q += G) S.apb[i][q] = 0u;
        __syncwarp(mask);
        const int a = rowptr[i], e = rowptr[i + 1];
        for (int k0 = a; k0 < e; k0 += G) {
            const bool on = k0 + gl < e;
            const int jl = on ? col[k0 + gl] : 0;
            const double sl = on ? dmul(val[k0 + gl], S.w[jl]) : 0.0;
            const int m = e - k0 < G ? e - k0 : G;
            for (int t = 0; t < m; t++) {
                const int j = __shfl_sync(mask, jl, t, G);
                const double s = __shfl_sync(mask, sl, t, G);
                const int pb = S.prow[j], pe = S.prow[j + 1];
                for (int q = pb + gl; q < pe; q += G) {
                    const int d = pcol[q];
                    acc[d] = dadd(acc[d], s);
                    atomicOr(&S.apb[i][d >> 5], 1u << (d & 31));
                }
                __syncwarp(mask);
            }
        }
        for (int d = gl; d < nc; d += G) ap[(long)i * nc + d] = acc[d];
        __syncwarp(mask);
    }
}

__global__ void __launch_bounds__(kTailThreads)
k_tail(int n, const int *rowptr, const int *col, const double *val, int level, int max_levels,
       int min_coarse, unsigned char *arena, unsigned top0, unsigned cap, double *ap, TailOut *out)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    TailShared &S = *(TailShared *)s_raw;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned top = top0;  // arena bytes in use (the same in every thread)
    int done = 0;
    auto take = [&](size_t bytes) {
        const unsigned o = top;
        top += (unsigned)((bytes + 15) & ~(size_t)15);
        return o;
    };
    while (done < kTailLevels) {
        // ---- lower neighbours of every row
        for (int q = tid; q < n * kTailWords; q += kTailThreads) (&S.bits[0][0])[q] = 0u;
        __syncthreads();
        for (int i = tid; i < n; i += kTailThreads)
            for (int k = rowptr[i]; k < rowptr[i + 1]; k++) {
                const int u = col[k];
                if (u < i) S.bits[i][u >> 5] |= 1u << (u & 31);
            }
        __syncthreads();
        // ---- greedy split: C when no lower neighbour is C
        if (warp == 0) {
            unsigned c = 0;
            unsigned nxt = lane < kTailWords ? S.bits[0][lane] : 0u;
            for (int i = 0; i < n; i++) {
                const unsigned b = nxt;
                if (i + 1 < n) nxt = lane < kTailWords ? S.bits[i + 1][lane] : 0u;
                if (!__any_sync(0xffffffffu, b & c) && lane == (i >> 5)) c |= 1u << (i & 31);
            }
            if (lane < kTailWords) S.cset[lane] = c;
        }
        __syncthreads();
        // ---- P row counts, coarse ids, weights
        if (tid < n) {
            S.cid[tid] = bit_of(S.cset, tid);
            int c = 0;
            if (S.cid[tid]) c = 1;
            else
                for (int k = rowptr[tid]; k < rowptr[tid + 1]; k++) c += bit_of(S.cset, col[k]);
            S.prow[tid] = c;
            S.w[tid] = 1.0 / (double)c;
        }
        __syncthreads();
        block_scan(S.cid, n, S.wsum);
        block_scan(S.prow, n, S.wsum);
        const int nc = S.cid[n], pnnz = S.prow[n];
        // room for the transfer arrays, and the coarse level at its largest
        const unsigned start = top;
        TailLevel t{};
        t.n = n;
        t.nc = nc;
        t.pnnz = pnnz;
        t.sel = take(n);
        t.cid = take(4 * (n + 1));
        t.prow = take(4 * (n + 1));
        t.pcol = take(4 * (size_t)pnnz);
        t.pw = take(8 * n);
        t.pw32 = take(4 * n);
        t.rrow = take(4 * (nc + 1));
        t.rcol = take(4 * (size_t)pnnz);
        t.arow = take(4 * (nc + 1));
        t.dinv = take(8 * nc);
        t.dinv32 = take(4 * nc);
        if (top > cap) {
            top = start;
            break;
        }
        signed char *sel = (signed char *)(arena + t.sel);
        int *cid = (int *)(arena + t.cid), *prow = (int *)(arena + t.prow),
            *pcol = (int *)(arena + t.pcol), *rrow = (int *)(arena + t.rrow),
            *rcol = (int *)(arena + t.rcol), *arow = (int *)(arena + t.arow);
        double *pw = (double *)(arena + t.pw), *dinv = (double *)(arena + t.dinv);
        float *pw32 = (float *)(arena + t.pw32), *dinv32 = (float *)(arena + t.dinv32);
        // ---- P rows; the fine rows of every coarse row as bit rows
        for (int q = tid; q < nc * kTailWords; q += kTailThreads) (&S.bits[0][0])[q] = 0u;
        __syncthreads();
        if (tid < n) {
            const bool c = bit_of(S.cset, tid);
            sel[tid] = c ? 1 : 2;
            pw[tid] = S.w[tid];
            pw32[tid] = (float)S.w[tid];
            int q = S.prow[tid];
            if (c) {
                pcol[q] = S.cid[tid];
                atomicOr(&S.bits[S.cid[tid]][tid >> 5], 1u << (tid & 31));
            } else {
                for (int k = rowptr[tid]; k < rowptr[tid + 1]; k++) {
                    const int j = col[k];
                    if (!bit_of(S.cset, j)) continue;
                    pcol[q++] = S.cid[j];
                    atomicOr(&S.bits[S.cid[j]][tid >> 5], 1u << (tid & 31));
                }
            }
        }
        if (tid <= n) {
            cid[tid] = S.cid[tid];
            prow[tid] = S.prow[tid];
        }
        __syncthreads();
        // ---- R = P^T: fine rows ascending
        if (tid < nc) {
            int c = 0;
            for (int q = 0; q < kTailWords; q++) c += __popc(S.bits[tid][q]);
            S.rrow[tid] = c;
        }
        __syncthreads();
        block_scan(S.rrow, nc, S.wsum);
        if (tid <= nc) rrow[tid] = S.rrow[tid];
        if (tid < nc) {
            int o = S.rrow[tid];
            for (int q = 0; q < kTailWords; q++)
                for (unsigned b = S.bits[tid][q]; b; b &= b - 1) rcol[o++] = 32 * q + __ffs(b) - 1;
        }
        // ---- A P, dense rows of nc
        if (128 * nc <= kTailAcc) tail_ap<8>(S, n, nc, rowptr, col, val, pcol, ap);
        else tail_ap<32>(S, n, nc, rowptr, col, val, pcol, ap);
        __syncthreads();
        // ---- P^T (A P): the pattern, then the values
        const int words = (nc + 31) / 32;
        for (int e = warp; e < nc; e += kTailWarps) {
            // lane q < 16: the row's columns in word q
            unsigned b = 0;
            for (int q = 0; q < kTailWords; q++)
                for (unsigned f = S.bits[e][q]; f; f &= f - 1)
                    if (lane < words) b |= S.apb[32 * q + __ffs(f) - 1][lane];
            int c = __popc(b);
            c = __reduce_add_sync(0xffffffffu, c);
            if (lane == 0) S.rrow[e] = c;
        }
        __syncthreads();
        block_scan(S.rrow, nc, S.wsum);
        const int nnz = S.rrow[nc];
        t.nnz = nnz;
        t.acol = take(4 * (size_t)nnz);
        t.aval = take(8 * (size_t)nnz);
        if (top > cap) {
            top = start;
            break;
        }
        int *acol = (int *)(arena + t.acol);
        double *aval = (double *)(arena + t.aval);
        if (tid <= nc) arow[tid] = S.rrow[tid];
        for (int e = warp; e < nc; e += kTailWarps) {
            int o = S.rrow[e];
            for (int q = 0; q < words; q++) {
                const int d = 32 * q + lane;
                double acc = -0.0;
                unsigned pat = 0;
                for (int f = 0; f < kTailWords; f++)
                    for (unsigned m = S.bits[e][f]; m; m &= m - 1) {
                        const int i = 32 * f + __ffs(m) - 1;
                        const unsigned b = S.apb[i][q];
                        pat |= b;
                        if ((b >> lane) & 1u) acc = dadd(acc, dmul(ap[(long)i * nc + d], S.w[i]));
                    }
                if ((pat >> lane) & 1u) {
                    const int p = o + __popc(pat & ((1u << lane) - 1u));
                    acol[p] = d;
                    aval[p] = acc;
                }
                if (d == e) {
                    const double v = 1.0 / ((pat >> lane) & 1u ? acc : 0.0);
                    dinv[e] = v;
                    dinv32[e] = (float)v;
                }
                o += __popc(pat);
            }
        }
        __syncthreads();
        if (tid == 0) out->lv[done] = t;
        done++;
        level++;
        // the level loop's test (amg.h:1186-1213)
        const bool more = level < max_levels - 1 && nc > min_coarse && nc < n;
        rowptr = arow;
        col = acol;
        val = aval;
        n = nc;
        __syncthreads();
        if (!more) break;
    }
    if (tid == 0) {
        out->levels = done;
        out->top = top;
    }
}

}  // namespace

bool tail_applies(const Level &L, int l)
{
    // level 0 may hold a caller's unsorted or repeated columns; the levels
    // with a structure of their own have their own kernels
    return l >= 1 && L.A.n <= kTailRows && L.A.n > 0 && L.g19.nx == 0 && !L.sel_split;
}

int amg_tail(std::vector<Level> &lv, int l, int max_levels, int min_coarse, TailArena &T,
             cudaStream_t st, int *levels)
{
    *levels = 0;
    // A hierarchy may come here more than once (the arena was full, the general
    // path made the next level): its earlier levels keep their place.
    const size_t cap = tail_arena_bytes();
    if (T.used >= cap) return HMFEM_OK;
    if (!T.mem) T.mem = (unsigned char *)dalloc(kTailArena);
    const Level &L0 = lv[l];
    double *ap = (double *)dalloc(sizeof(double) * (size_t)L0.A.n * L0.A.n);
    TailOut *out = (TailOut *)dalloc(sizeof(TailOut));
    if (!T.mem || !ap || !out) {
        set_last_error("out of device memory (coarse levels)", __FILE__, __LINE__);
        return HMFEM_E_CUDA;
    }
    HM_CUDA(cudaFuncSetAttribute(k_tail, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(TailShared)));
    k_tail<<<1, kTailThreads, sizeof(TailShared), st>>>(
        L0.A.n, L0.A.rowptr, L0.A.col, L0.A.val, l, max_levels, min_coarse, T.mem, T.used,
        (unsigned)cap, ap, out);
    HM_LAUNCHED();
    static_assert(sizeof(TailOut) <= sizeof(int) * (PIN_WORDS - PIN_BLOCK), "pinned words");
    HM_CHECK(read_back(PIN_BLOCK, out, (int)(sizeof(TailOut) / sizeof(int)), st));
    HM_CUDA(cudaStreamSynchronize(st));
    TailOut h;
    memcpy(&h, pinned_words() + PIN_BLOCK, sizeof(h));
    dfree(ap);
    dfree(out);
    for (int k = 0; k < h.levels; k++) {
        const TailLevel &t = h.lv[k];
        lv.emplace_back();
        Level &L = lv[l + k], &C = lv[l + k + 1];
        L.tail_transfer = true;
        L.sel = (signed char *)(T.mem + t.sel);
        L.cid = (int *)(T.mem + t.cid);
        L.nc = t.nc;
        L.P.n = t.n;
        L.P.nnz = t.pnnz;
        L.P.rowptr = (int *)(T.mem + t.prow);
        L.P.col = (int *)(T.mem + t.pcol);
        L.pw = (double *)(T.mem + t.pw);
        L.pw32 = (float *)(T.mem + t.pw32);
        L.R.n = t.nc;
        L.R.nnz = t.pnnz;
        L.R.rowptr = (int *)(T.mem + t.rrow);
        L.R.col = (int *)(T.mem + t.rcol);
        C.tail_matrix = true;
        C.A.n = t.nc;
        C.A.nnz = t.nnz;
        C.A.rowptr = (int *)(T.mem + t.arow);
        C.A.col = (int *)(T.mem + t.acol);
        C.A.val = (double *)(T.mem + t.aval);
        C.dinv = (double *)(T.mem + t.dinv);
        C.dinv32 = (float *)(T.mem + t.dinv32);
    }
    T.used = h.top;
    *levels = h.levels;
    return HMFEM_OK;
}

}  // namespace hm
