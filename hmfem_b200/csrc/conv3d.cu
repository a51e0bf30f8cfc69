// conv3d.cu -- 3x3x3 convolutions of the learned initial guess on the
// 5th-generation tensor cores (tcgen05, sm_100a): BF16 operands, FP32
// accumulation in tensor memory.  No counterpart in the reference.
//
// Activations are channel-blocked: C/8 slabs, each holding the grid's cells
// (s = x + nx (y + ny z)) with 8 consecutive BF16 channels per cell, i.e.
// channel c of cell s at (c/8) n + s) * 8 + c % 8; weights are
// [27 taps][Cout][Cin] with tap t = 9 (dz+1) + 3 (dy+1) + (dx+1); zero
// padding outside the grid.
//
// Forward (and, with flipped / transposed weights, the data gradient) is an
// implicit GEMM: D[m][n] = sum_tap sum_ci A_tap[m][ci] B_tap[n][ci] with m a
// run of 128 cells, n the output channel, A_tap the input at cell m shifted
// by the tap.  The input of a tile of cells, with its halo, is brought into
// shared memory once per 16 input channels by bulk copies and every tap's A operand
// is a shifted view of it (the layout and the roles are described at
// k_conv3d); tcgen05.mma (M = 128, N = Cout, K = 16) accumulates in tensor
// memory and the epilogue reads it with tcgen05.ld, adds the bias, applies
// ReLU and stores BF16.
//
// Weight gradient: the cells are the K dimension, and in the channel-blocked
// layout 8 consecutive cells x 8 channels of a slab already form a core
// matrix of a channel-major (MN-major) operand, so nothing is transposed: one
// operand holds three copies shifted by the x taps, the other the y taps'
// rows of three z planes, and every MMA forms a block of all 27 taps (the
// layout and the roles are described at k_wgrad).
//
// Every mbarrier wait is bounded: on a timeout the kernel flags err, waits
// (bounded again) for its MMAs in flight, frees its TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <mutex>

#include "common.cuh"

namespace hm {

namespace {

constexpr unsigned kWaitPolls = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor, K-major without swizzle: start address,
// leading-dimension byte offset (between the two 8-element K halves of one
// MMA), stride byte offset (between 8-row groups), version 1 (sm_100).
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, M x N.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ bool mbar_test(uint64_t *m, unsigned parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(m)), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait for the phase with this parity to complete
__device__ __forceinline__ bool mbar_wait(uint64_t *m, unsigned parity)
{
    for (unsigned i = 0; i < kWaitPolls; i++) {
        if (mbar_test(m, parity)) return true;
        if (i > 64) __nanosleep(64);
    }
    return false;
}

__device__ __forceinline__ void fence_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_before_sync()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_after_sync()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// TMEM allocation by warp 0 (whole warp), address left in *slot
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(slot)),
                 "r"(ncols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}

__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr),
                 "r"(ncols));
}

// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
          "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// 16 columns of this thread's TMEM lane into registers, without waiting:
// the registers are valid after tmem_wait_ld()
__device__ __forceinline__ void tmem_ld16_nw(uint32_t taddr, float v[16])
{
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
          "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
          "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld()
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- forward / data gradient ----------------------------------------------
//
// A tile is bx x by x bz output cells.  Its input with a one-cell halo,
// (bx+2) x (by+2) x (bz+2) cells, is copied into shared memory once per
// 16-channel chunk of the input: halo cell q = xi + W (yi + H zi) (W = bx+2,
// H = by+2) at byte q*16 of each 8-channel slab, the chunk's two slabs SB
// bytes apart -- the K-major no-swizzle layout with rows 16 bytes apart, so
// any 128 consecutive halo cells form an MMA operand (LBO = SB, SBO = 128).
// An MMA run is 128 consecutive halo positions q0 .. q0+127; the operand of
// tap (dx, dy, dz) for the run is the same rows shifted by dx + W dy + W H dz,
// i.e. the run's descriptor with another start address: the 27 taps read the
// tile that was copied once.  Row mode (bx = 128): a run is one x row of the
// tile.  Plane mode (bx = nx, any width): the runs of a z plane cover its interior
// rows in steps of 128 positions; positions on halo columns or beyond the
// plane are computed and dropped by the epilogue.  The copy of a tile reads
// (bx+2)(by+2)(bz+2) / (bx by bz) times its cells from L2.
//
// Roles (one CTA per SM, persistent over the tiles): warp 4 loads each halo
// chunk into a ring of `ns` stages with one bulk copy per halo row and slab
// (a halo row of a slab is contiguous in the channel-blocked input); the
// cells and rows outside the grid (the convolution's zero padding) are
// stored by the warp itself and fenced for the tensor cores;
// lane 0 of warp 5 issues, per chunk, 27 taps x runs MMAs of M = 128,
// N = COUT, K = 16 into the tile's accumulator (runs x COUT FP32 columns of
// tensor memory, `nb` = 2 buffers when they fit) and commits the stage back
// to the producer; warps 0-3 read a finished accumulator (tcgen05.ld, warp w
// lanes 32w..32w+31), add the bias, apply ReLU, store BF16 and release the
// buffer -- loads, MMAs and the epilogue of different tiles overlap.  The
// weights of a chunk come as two TMA copies of box {8, COUT, 27} (the two
// 8-channel halves, each [tap][COUT][8]); all chunks stay resident when they
// fit in kWResMax bytes, otherwise each stage carries its chunk's weights.
// No multicast.
// Grouped x taps (XG, when 3 COUT <= 256 and the tile spans the whole x
// extent): an MMA's cost is set by its A operand (128 rows from shared
// memory) up to N ~ 90, so the three taps dx = -1, 0, +1 of a (dy, dz) pair
// share one A operand -- the run's rows shifted by W dy + W H dz only -- and
// one MMA with N = 3 COUT (B = the three taps' weights, consecutive rows of
// the weight tile) accumulates D_dx for all three: 9 MMAs per run and chunk
// instead of 27.  The output of row m is D_-1[m-1] + D_0[m] + D_+1[m+1]: the
// epilogue shifts by one TMEM lane (warp shuffles; shared memory across the
// warps' lane quarters and, in plane mode, between consecutive runs of a z
// plane).  Any other neighbour of a stored cell is a halo column, i.e. zero
// padding, because the tile covers the whole x extent.
// Grouped z taps (ZG, when 3 COUT <= 256 and a tile has at least 4 planes):
// the three taps dz = -1, 0, +1 of a (dx, dy) pair share the operand of one
// input plane zi and feed three output planes zi+1, zi, zi-1 at the same x
// and y.  A run column's planes lie next to each other in tensor memory,
// highest plane first, so one MMA with N = 3 COUT adds into all three at
// once, and nothing has to be shifted afterwards.  The tile's first and last
// planes take N = COUT and 2 COUT; a plane's first MMA (not accumulating) is
// issued by itself.  9 (bz + 2) MMAs per run column and chunk instead of
// 27 bz; each output still adds its taps in the order of the ungrouped form,
// so its bits are the same.  Bound by the operands' shared-memory reads (44
// cycles per MMA at COUT = 16).  Measured against the ungrouped and x-grouped
// forms: see plan_conv.
struct ConvPlan {
    int bx, by, bz;          // tile (interior cells)
    int W, H;                // halo row pitch bx+2, halo rows per plane by+2
    int hc, hcp;             // halo cells; cells per slab with the run overrun (x8)
    int runs, rp;            // MMA runs per tile; runs per z plane
    int row_mode;            // 1: bx == 128, one run per x row
    int ntx, nty, ntz;       // tiles per axis
    int ns, nb;              // input stages, accumulator buffers
    int wres;                // weights of every chunk resident
    int xg;                  // x taps grouped: N = 3 COUT per MMA (see k_conv3d)
    int zg;                  // z taps grouped
    int tmem_cols;
    unsigned stage_bytes, wbytes, smem_bytes;
};

constexpr int kConvThreads = 192;  // warps 0-3 epilogue, 4 TMA producer, 5 MMA
constexpr int kEpilogue = 128;
constexpr int kMaxSmem = 227 * 1024;  // dynamic shared memory a block may have
constexpr unsigned kWResMax = 64 * 1024;  // resident weights (all chunks) up to this size
constexpr unsigned kBarBytes = 128;       // mbarriers (ns, nb <= 4), TMEM slot, abort flag
constexpr int kMaxPlaneX = 1024;          // widest grid a plane-mode tile spans

// shared memory after the stages: barriers, then (grouped x taps) three
// exchange buffers of 4 + 4 + 1 boundary rows of COUT floats, then the bias
__host__ __device__ constexpr unsigned conv_tail_bytes(int cout, bool xg)
{
    return kBarBytes + (xg ? 3u * 9u * 4u * (unsigned)cout : 0u) + 4u * (unsigned)cout;
}

// The MMA warp runs its loop with all lanes (descriptor arithmetic stays
// warp-uniform); one elected lane issues.  Every MMA and commit of the
// kernel goes through the same election, so a commit tracks the MMAs it
// follows (both are per issuing thread).
__device__ __forceinline__ void umma_bf16_elect(uint32_t tmem, uint64_t da, uint64_t db,
                                                uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred e, p;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
}

// Eight accumulating MMAs into one accumulator, elected once: operand A at
// da + off[i], operand B at db + (i + 1) BSTEP (16-byte units).
template <int BSTEP>
__device__ __forceinline__ void umma_bf16_elect8(uint32_t tmem, uint64_t da, const int off[8],
                                                 uint64_t db, uint32_t idesc)
{
#define HM_MMA8_ONE(i, k)                                                               \
    "add.s64 a, %1, %" #i ";\n\t"                                                       \
    "add.s64 b, %2, %" #k ";\n\t"                                                       \
    "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t"
    asm volatile(
        "{\n\t.reg .pred e, p;\n\t.reg .b64 a, b;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.eq.u32 p, %3, %3;\n\t" HM_MMA8_ONE(4, 12) HM_MMA8_ONE(5, 13) HM_MMA8_ONE(6, 14)
            HM_MMA8_ONE(7, 15) HM_MMA8_ONE(8, 16) HM_MMA8_ONE(9, 17) HM_MMA8_ONE(10, 18)
                HM_MMA8_ONE(11, 19) "}\n" ::"r"(tmem),
        "l"(da), "l"(db), "r"(idesc), "l"((int64_t)off[0]), "l"((int64_t)off[1]),
        "l"((int64_t)off[2]), "l"((int64_t)off[3]), "l"((int64_t)off[4]), "l"((int64_t)off[5]),
        "l"((int64_t)off[6]), "l"((int64_t)off[7]), "n"(BSTEP), "n"(2 * BSTEP), "n"(3 * BSTEP),
        "n"(4 * BSTEP), "n"(5 * BSTEP), "n"(6 * BSTEP), "n"(7 * BSTEP), "n"(8 * BSTEP));
#undef HM_MMA8_ONE
}

__device__ __forceinline__ void umma_commit_elect(uint64_t *mbar)
{
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n"
        ::"r"(smem_u32(mbar))
        : "memory");
}

__device__ __forceinline__ void mbar_init_n(uint64_t *m, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(count));
}

__device__ __forceinline__ void mbar_arrive(uint64_t *m)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(m)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx_only(uint64_t *m, uint32_t bytes)
{
    asm volatile("mbarrier.expect_tx.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(m)), "r"(bytes)
                 : "memory");
}

// bulk copy global -> this CTA's shared memory (16-byte aligned, multiple of 16)
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes,
                                          uint64_t *m)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_u32(m))
        : "memory");
}

// TMA tensor copies into this CTA's shared memory, completion on an mbarrier
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, int c0, int c1,
                                            int c2, uint64_t *m)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(m))
        : "memory");
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, int c0, int c1,
                                            int c2, int c3, uint64_t *m)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
        "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(m))
        : "memory");
}

// A position in a ring of barriers and the phase parity of its current use.
struct Ring {
    int i;
    unsigned ph;
    __device__ __forceinline__ void next(int n)
    {
        if (++i == n) {
            i = 0;
            ph ^= 1u;
        }
    }
};

// named barrier 1 among the epilogue warps; the reduction form returns the
// AND of every thread's predicate (all threads agree on leaving)
__device__ __forceinline__ void epi_sync()
{
    asm volatile("bar.sync 1, %0;" ::"n"(kEpilogue) : "memory");
}

__device__ __forceinline__ bool epi_all(bool v)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, 1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(r)
        : "r"((uint32_t)v), "n"(kEpilogue)
        : "memory");
    return r != 0;
}

// bounded wait that also leaves when another role gave up (abort flag)
__device__ __forceinline__ bool role_wait(uint64_t *m, unsigned parity, volatile int *abort_flag,
                                          int *err)
{
    for (unsigned i = 0; i < kWaitPolls; i++) {
        if (mbar_test(m, parity)) return true;
        if (*abort_flag) return false;
        if (i > 64) __nanosleep(64);
    }
    *abort_flag = 1;
    atomicExch(err, 1);
    return false;
}

// first halo position of run r; its plane (0..bz-1) and, in row mode, row
__device__ __forceinline__ int run_start(const ConvPlan &p, int r, int &plane, int &row)
{
    if (p.row_mode) {
        plane = r / p.by;
        row = r - plane * p.by;
        return 1 + p.W * (row + 1) + p.W * p.H * (plane + 1);
    }
    plane = r / p.rp;
    row = -1;
    return 1 + p.W + p.W * p.H * (plane + 1) + 128 * (r - plane * p.rp);
}

template <int CIN, int COUT, bool XG, bool ZG>
__global__ void __launch_bounds__(kConvThreads, 1)
k_conv3d(const __nv_bfloat16 *__restrict__ in, const __grid_constant__ CUtensorMap tm_w,
         const float *__restrict__ bias, __nv_bfloat16 *__restrict__ out, int nx, int ny,
         int nz, int relu, const ConvPlan p, int *err)
{
    static_assert(CIN % 16 == 0 && COUT % 16 == 0 && COUT <= 256, "channel counts");
    static_assert(!(XG || ZG) || 3 * COUT <= 256, "grouped taps: N = 3 COUT <= 256");
    static_assert(!(XG && ZG), "one grouping at a time");
    constexpr int KC = CIN / 16;
    constexpr int NACC = XG ? 3 * COUT : COUT;  // accumulator columns per run
    constexpr uint32_t IDESC = idesc_bf16(128, NACC);
    constexpr int WTAP = COUT * 16;       // one tap's rows of one 8-channel half
    constexpr int WHALF = 27 * WTAP;      // the second half follows all 27 taps of the first
    extern __shared__ __align__(128) unsigned char smem[];
    const unsigned SB = (unsigned)p.hcp * 16u, SA = 2u * SB;
    unsigned char *wres = smem;                    // resident weights (p.wres)
    unsigned char *stages = smem + p.wbytes;
    uint64_t *bar = (uint64_t *)(stages + (size_t)p.ns * p.stage_bytes);
    uint64_t *full = bar, *empty = bar + p.ns, *tfull = bar + 2 * p.ns, *tempty = tfull + p.nb,
             *drain = tempty + p.nb;
    uint32_t *tslot = (uint32_t *)(drain + 1);
    volatile int *abort_flag = (volatile int *)(tslot + 1);
    // grouped x taps: boundary rows exchanged between warps / runs, three
    // buffers (by a running run count): lane 31's D_-1 of each warp, lane
    // 0's D_+1 of each warp, row 0's D_+1 of the next run
    float *xlo = (float *)(stages + (size_t)p.ns * p.stage_bytes + kBarBytes);
    float *xhi = xlo + 3 * 4 * COUT;
    float *xnx = xhi + 3 * 4 * COUT;
    float *sbias = (float *)(stages + (size_t)p.ns * p.stage_bytes + kBarBytes) +
                   (XG ? 27 * COUT : 0);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long ntiles = (long)p.ntx * p.nty * p.ntz;
    const int WH = p.W * p.H;
    if (tid == 0) {
        for (int s = 0; s < p.ns; s++) {
            mbar_init_n(&full[s], 1);
            mbar_init_n(&empty[s], 1);
        }
        for (int b = 0; b < p.nb; b++) {
            mbar_init_n(&tfull[b], 1);
            mbar_init_n(&tempty[b], kEpilogue);
        }
        mbar_init_n(drain, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) tmem_alloc(tslot, p.tmem_cols);
    for (int i = tid; i < COUT; i += kConvThreads) sbias[i] = bias ? bias[i] : 0.f;
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = *tslot;

    if (warp == 4) {
        // ---- producer (whole warp): bulk copies of the halo rows
        const long n = (long)nx * ny * nz;
        const int D = p.bz + 2, rows = p.H * D;
        unsigned wkc = 0xffffffffu;  // per stage (8 bits each): chunk of its weights
        long item = 0;
        Ring ring{0, 0u};
        bool ok = true;
        // row / H as a product: exact for row * H < 2^32
        const unsigned inv_h = 0xffffffffu / (unsigned)p.H + 1u;
        for (long tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
            const int tx = (int)(tile % p.ntx), ty = (int)((tile / p.ntx) % p.nty),
                      tz = (int)(tile / ((long)p.ntx * p.nty));
            const int x0 = tx * p.bx - 1, y0 = ty * p.by - 1, z0 = tz * p.bz - 1;
            // the part [xa, xb) of every halo row inside the grid, and the
            // number of halo rows (of one slab) inside it
            const int xa = x0 < 0 ? 0 : x0, xb = x0 + p.W < nx ? x0 + p.W : nx;
            const int ya = y0 < 0 ? 0 : y0, yb = y0 + p.H < ny ? y0 + p.H : ny;
            const int za = z0 < 0 ? 0 : z0, zb = z0 + D < nz ? z0 + D : nz;
            const int rows_in = (yb - ya) * (zb - za);
            for (int kc = 0; kc < KC; kc++, item++, ring.next(p.ns)) {
                const int s = ring.i;
                if (!__all_sync(0xffffffffu,
                                role_wait(&empty[s], ring.ph ^ 1u, abort_flag, err))) {
                    ok = false;
                    break;
                }
                const uint32_t a = smem_u32(stages + (size_t)s * p.stage_bytes);
                const bool need_w = p.wres ? item == 0
                                           : ((wkc >> (8 * s)) & 0xffu) != (unsigned)kc;
                if (lane == 0)
                    mbar_expect_tx_only(&full[s], 32u * (unsigned)(rows_in * (xb - xa)) +
                                                      (need_w ? (p.wres ? KC : 1) * 2u * WHALF
                                                              : 0u));
                __syncwarp();
                const uint4 zero = make_uint4(0, 0, 0, 0);
                for (int i = lane; i < 2 * rows; i += 32) {
                    const int sl = i >= rows, rr = i - sl * rows,
                              zi = (int)__umulhi((unsigned)rr, inv_h), yi = rr - zi * p.H;
                    const int gy = y0 + yi, gz = z0 + zi;
                    unsigned char *drow_p = stages + (size_t)s * p.stage_bytes + (size_t)sl * SB +
                                            (size_t)(rr * p.W) * 16u;
                    if (gy < 0 || gy >= ny || gz < 0 || gz >= nz) {
                        for (int c = 0; c < p.W; c++) ((uint4 *)drow_p)[c] = zero;
                        continue;
                    }
                    const __nv_bfloat16 *src =
                        in + ((long)(2 * kc + sl) * n + xa + (long)nx * (gy + (long)ny * gz)) * 8;
                    bulk_load(smem_u32(drow_p) + (uint32_t)(xa - x0) * 16u, src,
                              (uint32_t)(xb - xa) * 16u, &full[s]);
                    for (int c = 0; c < xa - x0; c++) ((uint4 *)drow_p)[c] = zero;
                    for (int c = xb - x0; c < p.W; c++) ((uint4 *)drow_p)[c] = zero;
                }
                fence_async_smem();  // the zeros, written by this warp, for the MMAs
                if (need_w && lane == 0) {
                    for (int c = p.wres ? 0 : kc; c < (p.wres ? KC : kc + 1); c++) {
                        const uint32_t wb = p.wres ? smem_u32(wres) + (uint32_t)c * 2u * WHALF
                                                   : a + SA;
                        if (ZG) {  // [dx, dy][dz][COUT][8]
                            tma_load_4d(wb, &tm_w, 16 * c, 0, 0, 0, &full[s]);
                            tma_load_4d(wb + WHALF, &tm_w, 16 * c + 8, 0, 0, 0, &full[s]);
                        } else {
                            tma_load_3d(wb, &tm_w, 16 * c, 0, 0, &full[s]);
                            tma_load_3d(wb + WHALF, &tm_w, 16 * c + 8, 0, 0, &full[s]);
                        }
                    }
                }
                if (need_w) wkc = (wkc & ~(0xffu << (8 * s))) | ((unsigned)kc << (8 * s));
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[s]);
            }
        }
        // copies still in flight land before the CTA leaves: wait for the
        // last use of every stage (already complete unless a role gave up)
        if (lane == 0)
            for (int j = 0; j < p.ns && j < item; j++) {
                const long it = item - 1 - j;
                if (!mbar_wait(&full[it % p.ns], (unsigned)(it / p.ns) & 1u)) atomicExch(err, 1);
            }
        __syncwarp();
    } else if (warp == 5) {
        // ---- MMA issue (the whole warp, one elected lane issuing).  Per run
        // the 27 taps are unrolled: the A descriptor is the run's base plus a
        // per-tap offset held in a register, the B descriptor the stage's
        // base plus an immediate.
        {
            constexpr int NT = XG || ZG ? 9 : 27;  // taps or groups of an operand run
            int offs[NT];
#pragma unroll
            for (int t = 0; t < NT; t++)
                offs[t] = ZG   ? (t % 3 - 1) + p.W * (t / 3 - 1)
                          : XG ? p.W * (t % 3 - 1) + WH * (t / 3 - 1)
                             : (t % 3 - 1) + p.W * ((t / 3) % 3 - 1) + WH * (t / 9 - 1);
            Ring ring{0, 0u}, acc_ring{0, 0u};
            bool ok = true;
            for (long tile = blockIdx.x; tile < ntiles && ok;
                 tile += gridDim.x, acc_ring.next(p.nb)) {
                const int b = acc_ring.i;
                if (!__all_sync(0xffffffffu,
                                role_wait(&tempty[b], acc_ring.ph ^ 1u, abort_flag, err)))
                    break;
                tc_after_sync();
                const uint32_t acc0 = tmem + (uint32_t)(b * p.runs * NACC);
                for (int kc = 0; kc < KC; kc++, ring.next(p.ns)) {
                    const int s = ring.i;
                    if (!__all_sync(0xffffffffu, role_wait(&full[s], ring.ph, abort_flag, err))) {
                        ok = false;
                        break;
                    }
                    tc_after_sync();
                    const uint32_t a = smem_u32(stages + (size_t)s * p.stage_bytes);
                    const uint32_t wb =
                        p.wres ? smem_u32(wres) + (uint32_t)kc * 2u * WHALF : a + SA;
                    // descriptor start addresses count 16-byte units: a run's
                    // operand row q is one unit per position
                    const uint64_t da0 = kmajor_desc(a, SB, 128);
                    const uint64_t db0 = kmajor_desc(wb, WHALF, 128);
                    const uint32_t first = kc == 0 ? 0u : 1u;
                    if (ZG) {
                        for (int j = 0; j < p.rp; j++) {
                            const uint64_t daj =
                                da0 + (uint64_t)(1 + p.W * (p.row_mode ? j + 1 : 1) +
                                                 (p.row_mode ? 0 : 128 * j));
                            for (int zi = 0; zi < p.bz + 2; zi++) {
                                // output planes zi - d, d = dz + 1 in [lo, hi]
                                const int lo = zi < p.bz ? 0 : zi - p.bz + 1,
                                          hi = zi < 2 ? zi : 2;
                                const uint64_t dar = daj + (uint64_t)(WH * zi);
                                const uint32_t acc =
                                    acc0 + (uint32_t)((j * p.bz + p.bz - 1 - zi + lo) * COUT);
                                const uint64_t db = db0 + (uint64_t)(lo * (WTAP / 16));
                                const uint32_t idn = idesc_bf16(128, (hi - lo + 1) * COUT);
                                // the plane that starts here (d = 0)
                                const bool fresh = kc == 0 && zi < p.bz;
                                if (fresh) {
                                    umma_bf16_elect(acc, dar + (uint64_t)offs[0], db,
                                                    idesc_bf16(128, COUT), 0u);
                                    if (hi > 0)
                                        umma_bf16_elect(acc + COUT, dar + (uint64_t)offs[0],
                                                        db + (uint64_t)(WTAP / 16),
                                                        idesc_bf16(128, hi * COUT), 1u);
                                } else {
                                    umma_bf16_elect(acc, dar + (uint64_t)offs[0], db, idn, 1u);
                                }
                                umma_bf16_elect8<3 * (WTAP / 16)>(acc, dar, offs + 1, db, idn);
                            }
                        }
                        umma_commit_elect(&empty[s]);
                        continue;
                    }
                    // run starts without divisions (the order of run_start)
                    int plane = 0, j = 0;
                    for (int r = 0; r < p.runs; r++) {
                        const int q0 = p.row_mode
                                           ? 1 + p.W * (j + 1) + WH * (plane + 1)
                                           : 1 + p.W + WH * (plane + 1) + 128 * j;
                        if (++j == p.rp) {
                            j = 0;
                            plane++;
                        }
                        const uint64_t dar = da0 + (uint64_t)q0;
                        const uint32_t acc = acc0 + (uint32_t)(r * NACC);
                        // tap t (or group g: taps 3g .. 3g+2) starts at row t (3g) x COUT
                        // of the weight tile
#pragma unroll
                        for (int t = 0; t < NT; t++)
                            umma_bf16_elect(acc, dar + (uint64_t)offs[t],
                                            db0 + (uint64_t)(t * (XG ? 3 : 1) * (WTAP / 16)),
                                            IDESC, t == 0 ? first : 1u);
                    }
                    umma_commit_elect(&empty[s]);
                }
                if (ok) umma_commit_elect(&tfull[b]);
            }
        }
        __syncwarp();
    } else {
        // ---- epilogue: warp w reads TMEM lanes 32w .. 32w+31 (rows of a run)
        const int m = 32 * warp + lane;
        const long nc = (long)nx * ny * nz;
        long jt = 0, gr = 0;  // tiles, runs (running count: exchange buffers)
        for (long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, jt++) {
            const int b = (int)(jt % p.nb);
            const unsigned u = (unsigned)(jt / p.nb);
            bool okw = role_wait(&tfull[b], u & 1u, abort_flag, err);
            if (XG) okw = epi_all(okw);  // named barriers below: leave together
            if (!okw) break;
            tc_after_sync();
            const int tx = (int)(tile % p.ntx), ty = (int)((tile / p.ntx) % p.nty),
                      tz = (int)(tile / ((long)p.ntx * p.nty));
            const int X0 = tx * p.bx - 1, Y0 = ty * p.by - 1, Z0 = tz * p.bz - 1;
            for (int r = 0; r < p.runs; r++, gr++) {
                int plane, row;
                const int q = run_start(p, r, plane, row) + m;
                const int zi = q / WH, rem = q - zi * WH, yi = rem / p.W, xi = rem - yi * p.W;
                const int gx = X0 + xi, gy = Y0 + yi, gz = Z0 + zi;
                const bool v = zi == plane + 1 && yi >= 1 && yi <= p.by && xi >= 1 &&
                               xi <= p.bx && (row < 0 || yi == row + 1) && gx < nx && gy < ny &&
                               gz < nz;
                // run r's columns: by run, or (grouped z taps) by run column,
                // the highest plane first
                const int rc = ZG ? (r - plane * p.rp) * p.bz + p.bz - 1 - plane : r;
                const uint32_t ta = tmem + ((uint32_t)(32 * warp) << 16) +
                                    (uint32_t)((b * p.runs + rc) * NACC);
                const long cell = gx + (long)nx * (gy + (long)ny * gz);
                // runs r-1 and r+1 of the same z plane (plane mode only)
                const bool same_prev = !p.row_mode && r > 0 && r % p.rp != 0;
                const bool same_next = !p.row_mode && r + 1 < p.runs && (r + 1) % p.rp != 0;
                const int xb = (int)(gr % 3), xbp = (int)((gr + 2) % 3);
#pragma unroll
                for (int c0 = 0; c0 < COUT; c0 += 16) {
                    float f[16];
                    if (XG) {
                        float dm[16], dp[16], dn1[16];
                        tmem_ld16_nw(ta + c0, dm);              // D_-1
                        tmem_ld16_nw(ta + COUT + c0, f);        // D_0
                        tmem_ld16_nw(ta + 2 * COUT + c0, dp);   // D_+1
                        if (warp == 0 && same_next)
                            tmem_ld16_nw(ta + NACC + 2 * COUT + c0, dn1);  // next run's D_+1
                        tmem_wait_ld();
                        // publish the rows other warps (and the next run) need
                        float4 *lo = (float4 *)(xlo + (xb * 4 + warp) * COUT + c0);
                        float4 *hi = (float4 *)(xhi + (xb * 4 + warp) * COUT + c0);
                        if (lane == 31)
#pragma unroll
                            for (int i = 0; i < 4; i++)
                                lo[i] = make_float4(dm[4 * i], dm[4 * i + 1], dm[4 * i + 2],
                                                    dm[4 * i + 3]);
                        if (lane == 0) {
#pragma unroll
                            for (int i = 0; i < 4; i++)
                                hi[i] = make_float4(dp[4 * i], dp[4 * i + 1], dp[4 * i + 2],
                                                    dp[4 * i + 3]);
                            if (warp == 0 && same_next) {
                                float4 *nx4 = (float4 *)(xnx + xb * COUT + c0);
#pragma unroll
                                for (int i = 0; i < 4; i++)
                                    nx4[i] = make_float4(dn1[4 * i], dn1[4 * i + 1],
                                                         dn1[4 * i + 2], dn1[4 * i + 3]);
                            }
                        }
                        epi_sync();
                        // row m-1's D_-1 and row m+1's D_+1
                        float up[16], dn[16];
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            up[i] = __shfl_up_sync(0xffffffffu, dm[i], 1);
                            dn[i] = __shfl_down_sync(0xffffffffu, dp[i], 1);
                        }
                        if (lane == 0) {
                            const float *src = warp > 0 ? xlo + (xb * 4 + warp - 1) * COUT + c0
                                             : same_prev ? xlo + (xbp * 4 + 3) * COUT + c0
                                                         : nullptr;
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                const float4 t4 = src ? ((const float4 *)src)[i]
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
                                up[4 * i] = t4.x, up[4 * i + 1] = t4.y, up[4 * i + 2] = t4.z,
                                up[4 * i + 3] = t4.w;
                            }
                        }
                        if (lane == 31) {
                            const float *src = warp < 3 ? xhi + (xb * 4 + warp + 1) * COUT + c0
                                             : same_next ? xnx + xb * COUT + c0
                                                         : nullptr;
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                const float4 t4 = src ? ((const float4 *)src)[i]
                                                      : make_float4(0.f, 0.f, 0.f, 0.f);
                                dn[4 * i] = t4.x, dn[4 * i + 1] = t4.y, dn[4 * i + 2] = t4.z,
                                dn[4 * i + 3] = t4.w;
                            }
                        }
#pragma unroll
                        for (int i = 0; i < 16; i++) f[i] += up[i] + dn[i];
                    } else {
                        tmem_ld16_nw(ta + c0, f);
                        tmem_wait_ld();
                    }
                    if (v) {
                        __nv_bfloat16 o[16];
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            float t = f[i] + sbias[c0 + i];
                            if (relu) t = fmaxf(t, 0.f);
                            o[i] = __float2bfloat16(t);
                        }
                        *(uint4 *)(out + ((long)(c0 / 8) * nc + cell) * 8) = *(uint4 *)&o[0];
                        *(uint4 *)(out + ((long)(c0 / 8 + 1) * nc + cell) * 8) = *(uint4 *)&o[8];
                    }
                }
            }
            tc_before_sync();
            mbar_arrive(&tempty[b]);
        }
    }
    // teardown: every MMA this CTA issued has completed before TMEM is freed
    if (warp == 5) {
        umma_commit_elect(drain);
        if (lane == 0 && !mbar_wait(drain, 0)) atomicExch(err, 1);
        __syncwarp();
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    if (warp == 5) tmem_free(tmem, p.tmem_cols);
}

// ---- weight gradient --------------------------------------------------------
//
// dW[tap][co][ci] = sum_c dY[c][co] X[c + tap][ci].  Writing the tap as a sum
// of an x shift on one side and a (y, z) shift on the other,
//     D[(dx, m)][(z plane, y row, n)] = sum_p M[p + dx][m] N[p + (y, z)][n],
// with M and N the two tensors in the order that wastes less (WgPlan::flip:
// M = dY, N = X), one MMA has all three x taps in its rows and the y and z
// taps in its columns: with 16 -> 16 channels 48 x 144 useful entries of
// 128 x 144 for 16 cells, against 16 x 16 of 128 x 16 for one tap per MMA
// (one tap per CTA, both operands transposed through registers).  Measured
// against that form: 16 -> 16 at 128^3 2707 -> 110 us, 48 -> 16 3814 -> 204,
// 96 -> 32 at 64^3 1335 -> 80, 64 -> 64 at 32^3 125 -> 26.  Bound by the
// operands' shared-memory reads (16 -> 16) or the copies (96 -> 32): a copy
// brings all slabs of one shift (one per group took 104 us at 96 -> 32), and
// bulk copies by row with zeros stored around them were slower (162).
//
// A step is 32 x BY cells of one z plane.  A group is one slab (8 channels)
// of a step, BY rows of 32 cells, 16 bytes a cell: an MN-major operand
// without swizzle whose K groups (8 cells) lie 128 bytes and whose 8-channel
// groups SP = 512 BY bytes apart.  Tensor copies bring the groups in and
// fill what lies outside the grid (x, y or z) with zeros, so no tile edge
// has a case of its own: the M side as 3 x slabs groups at x - 1, x, x + 1,
// the N side per z plane as 3 x NS groups at y - 1, y, y + 1.  A CTA walks
// z, so each N plane is loaded once for its three z taps (a ring of RN
// planes); M planes go through a ring of RM stages.  Groups of the A operand
// beyond the tensor's (M = 128 is 16 groups) read whatever shared memory
// follows: their rows of D are never looked at.
//
// A part is one block of 16 M groups and NS slabs of N; a CTA keeps one
// part's D in tensor memory over all its cells and adds it into dw at the
// end.  Roles: warp 4 loads (a lane per group), warp 5 issues, warps 0-3
// read D.
//
// The zeros outside the grid are multiplied like cells, and zero times a
// non-finite cell is NaN: entries of D that come out NaN where the CTA meets
// the grid's edge are summed again over its pairs of cells that both lie in
// the grid (wgrad_nan_entries), so only those pairs count whatever the cells
// hold.
struct WgPlan {
    int nx, ny, nz;
    int flip;              // 0: M = x, N = dy; 1: M = dy, N = x
    int ms, gm, gmax;      // M side: slabs, groups (3 ms), groups per stage
    int mb;                // groups per copy: divides ms and 16
    int mblk, parts;       // M blocks; parts = mblk x (N slabs / NS)
    int cin, cout;
    int nxc, nyb, zl, nzc; // 32-cell columns, BY-row blocks, z planes per item, items along z
    int per;               // CTAs per part
    int vec;               // dw is 16-byte aligned
};

template <int NS, int BY>
struct WgCfg {
    static constexpr int SP = BY * 512;        // bytes of a group
    static constexpr int KS = BY * 2;          // MMAs (16 cells) along K per step
    static constexpr int GN = 3 * NS;          // groups of an N plane
    static constexpr int COLS = 72 * NS;       // columns of D: 3 planes x GN x 8
    static constexpr int TCOLS = COLS <= 256 ? 256 : 512;
    static constexpr int RM = BY == 4 ? 3 : 4;
    static constexpr int RN = BY == 4 ? 10 : NS == 4 ? 8 : 7;
    static constexpr int kBytes(int gmax) { return (RM * gmax + RN * GN) * SP + 256; }
};

// kind::f16 with both operands MN-major (bits 15 and 16)
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int m, int n)
{
    return idesc_bf16(m, n) | (1u << 15) | (1u << 16);
}

// Whether any step of CTA idx multiplies, in the entries of shift (i, j, k), a
// cell of the grid with a place outside it.
template <int BY>
__device__ __noinline__ bool wgrad_meets_edge(const WgPlan &p, int idx, int i, int j, int k)
{
    for (long it = idx; it < (long)p.nxc * p.nyb * p.nzc; it += p.per) {
        const int xc = (int)(it % p.nxc), yb = (int)((it / p.nxc) % p.nyb),
                  zc = (int)(it / ((long)p.nxc * p.nyb));
        const bool xe = xc == p.nxc - 1, ye = yb == p.nyb - 1;
        if (i == 0 ? xc == 0 || (xe && p.nx % 32) : i == 2 && xe) return true;
        if (j == 0 ? yb == 0 || (ye && p.ny % BY) : j == 2 && ye) return true;
        if (k == 0 ? zc == 0 : k == 2 && zc == p.nzc - 1) return true;
    }
    return false;
}

// Eight entries of CTA idx's D, sum_p M[p + (i-1)][cm] N[p + (j-1, k-1)][8 slab
// + 0..7] over its steps without the pairs of which a cell lies outside the
// grid: a warp, a lane per cell of a row.  Left as soon as all eight are NaN.
struct Entries {
    float v[8];
};
template <int BY>
__device__ __noinline__ Entries wgrad_nan_entries(const __nv_bfloat16 *__restrict__ m,
                                                  const __nv_bfloat16 *__restrict__ nn,
                                                  const WgPlan &p, int idx, int cm, int slab,
                                                  int i, int j, int k)
{
    const int lane = threadIdx.x & 31;
    const long nx = p.nx, nxy = nx * p.ny, cells = nxy * p.nz;
    double t[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    bool nan = false;
    for (long it = idx; it < (long)p.nxc * p.nyb * p.nzc && !nan; it += p.per) {
        const int xc = (int)(it % p.nxc), yb = (int)((it / p.nxc) % p.nyb),
                  zc = (int)(it / ((long)p.nxc * p.nyb));
        const int x = 32 * xc + lane;
        const bool on = x >= (i == 0) && x < p.nx - (i == 2);
        const int y0 = max(BY * yb, j == 0), y1 = min(BY * yb + BY, p.ny - (j == 2));
        const int z0 = max(p.zl * zc, k == 0), z1 = min(p.zl * zc + p.zl, p.nz - (k == 2));
        for (int z = z0; z < z1 && !nan; z++) {
#pragma unroll
            for (int r = 0; r < BY; r++) {
                const int y = BY * yb + r;
                if (!on || y < y0 || y >= y1) continue;
                const long c = x + y * nx + z * nxy;
                const double a = (double)__bfloat162float(
                    m[((cm / 8) * cells + c + i - 1) * 8 + cm % 8]);
                const uint4 q = ((const uint4 *)nn)[slab * cells + c + (j - 1) * nx +
                                                    (k - 1) * nxy];
                const __nv_bfloat16 *e = (const __nv_bfloat16 *)&q;
#pragma unroll
                for (int w = 0; w < 8; w++) t[w] += a * (double)__bfloat162float(e[w]);
            }
            nan = true;
#pragma unroll
            for (int w = 0; w < 8; w++) nan = __any_sync(0xffffffffu, t[w] != t[w]) && nan;
        }
    }
    Entries f;
#pragma unroll
    for (int w = 0; w < 8; w++) f.v[w] = (float)__shfl_sync(0xffffffffu, warp_sum(t[w]), 0);
    return f;
}

template <int NS, int BY>
__global__ void __launch_bounds__(kConvThreads, 1)
k_wgrad(const __grid_constant__ CUtensorMap tm_m, const __grid_constant__ CUtensorMap tm_n,
        const __nv_bfloat16 *__restrict__ gm, const __nv_bfloat16 *__restrict__ gn,
        float *__restrict__ dw, const __grid_constant__ WgPlan p, int *err)
{
    using C = WgCfg<NS, BY>;
    const int nz = p.nz;
    constexpr int SP = C::SP, GN = C::GN, RM = C::RM, RN = C::RN;
    extern __shared__ __align__(128) unsigned char smem[];
    const int mstage = p.gmax * SP;
    unsigned char *mring = smem, *nring = smem + RM * mstage;
    uint64_t *bar = (uint64_t *)(nring + RN * GN * SP);
    uint64_t *full_m = bar, *empty_m = bar + RM, *full_n = bar + 2 * RM, *empty_n = full_n + RN,
             *done = empty_n + RN;
    uint32_t *tslot = (uint32_t *)(done + 1);
    volatile int *abort_flag = (volatile int *)(tslot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int part = blockIdx.x % p.parts, idx = blockIdx.x / p.parts;
    const int g0 = 16 * (part % p.mblk), s0 = NS * (part / p.mblk);
    const int gmc = p.gm - g0 < 16 ? p.gm - g0 : 16;
    const long items = (long)p.nxc * p.nyb * p.nzc;
    if (tid == 0) {
        for (int i = 0; i < 2 * RM + 2 * RN + 1; i++) mbar_init_n(&bar[i], 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) tmem_alloc(tslot, C::TCOLS);
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    const uint32_t tmem = *tslot;

    if (warp == 4) {
        Ring rm{0, 0u}, rn{0, 0u};
        long mseq = 0, nseq = 0;
        // a lane's copy: mb groups (slabs of one x shift) of the M side, the NS
        // slabs of one y shift of an N plane
        const int gl = lane * p.mb;
        const int gi = (g0 + gl) / p.ms, gs = (g0 + gl) % p.ms;
        bool ok = true;
        for (long it = idx; it < items && ok; it += p.per) {
            const int xc = (int)(it % p.nxc), yb = (int)((it / p.nxc) % p.nyb),
                      zc = (int)(it / ((long)p.nxc * p.nyb));
            const int z0 = zc * p.zl, z1 = z0 + p.zl < nz ? z0 + p.zl : nz;
            for (int z = z0 - 1; z <= z1; z++) {  // N plane z, then M plane z - 1
                if (!__all_sync(0xffffffffu,
                                role_wait(&empty_n[rn.i], rn.ph ^ 1u, abort_flag, err))) {
                    ok = false;
                    break;
                }
                if (lane == 0) mbar_expect_tx_only(&full_n[rn.i], GN * SP);
                __syncwarp();
                if (lane < 3)
                    tma_load_4d(smem_u32(nring + (rn.i * GN + lane * NS) * SP), &tm_n, 256 * xc,
                                BY * yb + lane - 1, z, s0, &full_n[rn.i]);
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_n[rn.i]);
                rn.next(RN);
                nseq++;
                if (z <= z0) continue;
                if (!__all_sync(0xffffffffu,
                                role_wait(&empty_m[rm.i], rm.ph ^ 1u, abort_flag, err))) {
                    ok = false;
                    break;
                }
                if (lane == 0) mbar_expect_tx_only(&full_m[rm.i], (uint32_t)(gmc * SP));
                __syncwarp();
                if (gl < gmc)
                    tma_load_4d(smem_u32(mring + rm.i * mstage + gl * SP), &tm_m,
                                256 * xc + 8 * (gi - 1), BY * yb, z - 1, gs, &full_m[rm.i]);
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_m[rm.i]);
                rm.next(RM);
                mseq++;
            }
        }
        // copies still in flight land before the CTA leaves
        if (lane == 0) {
            for (int j = 0; j < RN && j < nseq; j++) {
                const long q = nseq - 1 - j;
                if (!mbar_wait(&full_n[q % RN], (unsigned)(q / RN) & 1u)) atomicExch(err, 1);
            }
            for (int j = 0; j < RM && j < mseq; j++) {
                const long q = mseq - 1 - j;
                if (!mbar_wait(&full_m[q % RM], (unsigned)(q / RM) & 1u)) atomicExch(err, 1);
            }
        }
        __syncwarp();
    } else if (warp == 5) {
        // ring positions kept incrementally: the scalar work between two
        // steps' MMAs is this one warp's (positions from 64-bit remainders
        // cost ~950 cycles a step)
        Ring rm{0, 0u}, rn[3];  // planes z - 1, z, z + 1
        for (int k = 0; k < 3; k++) rn[k] = Ring{k, 0u};
        bool ok = true;
        uint32_t acc = 0;  // nothing in D yet
        const uint64_t nbase = kmajor_desc(smem_u32(nring), 128, SP),
                       mbase = kmajor_desc(smem_u32(mring), 128, SP);
        for (long it = idx; it < items && ok; it += p.per) {
            const int zc = (int)(it / ((long)p.nxc * p.nyb));
            const int z0 = zc * p.zl, z1 = z0 + p.zl < nz ? z0 + p.zl : nz;
            for (int z = z0; z < z1 && ok; z++) {
                for (int k = z == z0 ? 0 : 2; k < 3; k++)
                    ok = ok && __all_sync(0xffffffffu, role_wait(&full_n[rn[k].i], rn[k].ph,
                                                                 abort_flag, err));
                ok = ok && __all_sync(0xffffffffu,
                                      role_wait(&full_m[rm.i], rm.ph, abort_flag, err));
                if (!ok) break;
                tc_after_sync();
                const uint64_t da = mbase + (uint64_t)((rm.i * mstage) >> 4);
                uint64_t db[3];
#pragma unroll
                for (int k = 0; k < 3; k++)
                    db[k] = nbase + (uint64_t)(rn[k].i * (GN * SP / 16));
                // one MMA over the three planes where they are consecutive
                // in the ring and N = 3 GN 8 <= 256, otherwise one per plane
                if (C::COLS <= 256 && rn[0].i + 2 < RN) {
#pragma unroll
                    for (int ks = 0; ks < C::KS; ks++) {  // 256 bytes further each
                        umma_bf16_elect(tmem, da + (uint64_t)(16 * ks),
                                        db[0] + (uint64_t)(16 * ks),
                                        idesc_bf16_mn(128, C::COLS <= 256 ? C::COLS : 256), acc);
                        acc = 1;
                    }
                } else {
#pragma unroll
                    for (int ks = 0; ks < C::KS; ks++) {
#pragma unroll
                        for (int k = 0; k < 3; k++)
                            umma_bf16_elect(tmem + (uint32_t)(k * GN * 8),
                                            da + (uint64_t)(16 * ks), db[k] + (uint64_t)(16 * ks),
                                            idesc_bf16_mn(128, GN * 8), acc);
                        acc = 1;
                    }
                }
                umma_commit_elect(&empty_m[rm.i]);
                umma_commit_elect(&empty_n[rn[0].i]);
                if (z == z1 - 1) {  // the walk's last two planes
                    umma_commit_elect(&empty_n[rn[1].i]);
                    umma_commit_elect(&empty_n[rn[2].i]);
                }
                rm.next(RM);
                // one plane on, or three at the end of the walk
                for (int q = 0; q < (z == z1 - 1 ? 3 : 1); q++) {
                    rn[0] = rn[1];
                    rn[1] = rn[2];
                    rn[2].next(RN);
                }
            }
        }
        umma_commit_elect(done);
        if (lane == 0 && !mbar_wait(done, 0)) {
            *abort_flag = 1;
            atomicExch(err, 1);
        }
        __syncwarp();
    } else if (__all_sync(0xffffffffu, role_wait(done, 0, abort_flag, err) && !*abort_flag)) {
        tc_after_sync();
        const int g = g0 + 4 * warp + (lane >> 3);  // row 32 warp + lane: group, channel
        const bool v = g < p.gm;
        const int i = v ? g / p.ms : 0, cm = v ? 8 * (g % p.ms) + (lane & 7) : 0;
#pragma unroll 1
        for (int c = 0; c < C::COLS; c += 16) {
            float f[16];
            __syncwarp();  // (rows beyond the tensor's skip the stores; the read is the warp's)
            tmem_ld16(tmem + ((uint32_t)(32 * warp) << 16) + c, f);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int q = c / 8 + h, k = q / GN, j = (q / NS) % 3, sn = s0 + q % NS;
                const int cn = 8 * sn;
                const float t = ((f[8 * h] + f[8 * h + 1]) + (f[8 * h + 2] + f[8 * h + 3])) +
                                ((f[8 * h + 4] + f[8 * h + 5]) + (f[8 * h + 6] + f[8 * h + 7]));
                if (__any_sync(0xffffffffu, t != t)) {
                    // a row at a time, by the warp
                    unsigned rows = __ballot_sync(
                        0xffffffffu, v && t != t && wgrad_meets_edge<BY>(p, idx, i, j, k));
                    for (; rows; rows &= rows - 1) {
                        const int r = __ffs(rows) - 1;
                        const Entries n = wgrad_nan_entries<BY>(
                            gm, gn, p, idx, __shfl_sync(0xffffffffu, cm, r), sn,
                            __shfl_sync(0xffffffffu, i, r), j, k);
#pragma unroll
                        for (int e = 0; e < 8; e++)
                            if (lane == r) f[8 * h + e] = n.v[e];
                    }
                }
                if (!v) continue;
                if (!p.flip) {
                    // X at p + (i-1), dY at p + (j-1, k-1): tap (i-1, 1-j, 1-k)
                    const int tap = 9 * (2 - k) + 3 * (2 - j) + i;
                    float *o = dw + ((long)tap * p.cout + cn) * p.cin + cm;
#pragma unroll
                    for (int e = 0; e < 8; e++) atomicAdd(o + (long)e * p.cin, f[8 * h + e]);
                } else {
                    // dY at p + (i-1), X at p + (j-1, k-1): tap (1-i, j-1, k-1)
                    const int tap = 9 * k + 3 * j + (2 - i);
                    float *o = dw + ((long)tap * p.cout + cm) * p.cin + cn;
                    if (p.vec) {
                        atomicAdd((float4 *)o, make_float4(f[8 * h], f[8 * h + 1], f[8 * h + 2],
                                                           f[8 * h + 3]));
                        atomicAdd((float4 *)o + 1, make_float4(f[8 * h + 4], f[8 * h + 5],
                                                               f[8 * h + 6], f[8 * h + 7]));
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; e++) atomicAdd(o + e, f[8 * h + e]);
                    }
                }
            }
        }
    }
    tc_before_sync();
    __syncthreads();
    tc_after_sync();
    if (warp == 5) tmem_free(tmem, C::TCOLS);
}

// Tile choice for a forward launch: row mode (bx = 128) or plane mode (bx =
// nx, the whole x extent); the mode, the form (x taps grouped or not) and (by, bz)
// minimise an estimate of the makespan -- per tile the largest of the MMA
// issue (~42 cycles per MMA up to N = 84, N/2 above: the A operand read),
// the halo copy (a bulk copy per row and slab plus its bytes) and the
// epilogue (added instead with one accumulator buffer), times the tile
// waves over the SMs -- subject to the tensor-memory columns (runs x COUT,
// x3 grouped, doubled when two accumulators fit in 512) and the shared
// memory.  Grouping pays where the MMAs dominate: many input chunks and
// few output columns, and the tile is too flat to group the z taps instead.
// Grouping the z taps needs no work in the epilogue but two more input planes
// per tile: from 4 planes on it halves the MMAs (at 2 planes it would save a
// third of them and load twice the cells).  It adds an output's taps in the
// order of the ungrouped form, the x grouping in another one: so z grouping
// takes over from the ungrouped form only, and a shape's results keep their
// bits.  Against the ungrouped form: 16 -> 16 at 128^3 95 -> 80 us, 32 -> 16
// at 64^3 47 -> 36, 96 -> 32 100 -> 78; the copies of the halo rows (~55 us
// alone at 16 -> 16) and the MMAs (~65 us) now bound it about equally.
ConvPlan plan_conv(int nx, int ny, int nz, int cin, int cout, int nsm, int smem_max)
{
    ConvPlan best{};
    double best_cost = 1e300;
    const int kc = cin / 16;
    const unsigned wchunk = 27u * (unsigned)cout * 32u;
    // row mode (bx = 128, x tiles) when nx >= 128; plane mode (bx = nx, the
    // whole x extent) for any width up to kMaxPlaneX
    for (int g = 0; g < 3 && !(g == 2 && best.xg); g++)
    for (int pm = 0; pm < 2; pm++)
        for (int bz = 1; bz <= (nz < 16 ? nz : 16); bz++)
            for (int by = 1; by <= (ny < 64 ? ny : 64); by++) {
                const bool row_mode = pm == 0;
                const int xg = g == 1, zg = g == 2;
                if (row_mode ? nx < 128 : nx > kMaxPlaneX) continue;
                const int bx = row_mode ? 128 : nx;
                const int W = bx + 2;
                // grouped x taps need N = 3 COUT <= 256 and tiles spanning
                // the x extent (their x neighbours outside the tile are zero)
                if (xg && (3 * cout > 256 || (row_mode && nx != 128))) continue;
                if (zg && (3 * cout > 256 || bz < 4)) continue;
                ConvPlan p{};
                p.bx = bx;
                p.by = by;
                p.bz = bz;
                p.W = W;
                p.H = by + 2;
                p.hc = W * p.H * (bz + 2);
                p.hcp = (p.hc + 128 + 7) / 8 * 8;
                p.row_mode = row_mode;
                p.xg = xg;
                p.zg = zg;
                p.rp = row_mode ? by : (W * (by - 1) + bx + 127) / 128;
                p.runs = bz * p.rp;
                const int nacc = (xg ? 3 : 1) * cout;
                if (p.runs * nacc > 512) continue;
                p.nb = 2 * p.runs * nacc <= 512 ? 2 : 1;
                p.wres = (unsigned)kc * wchunk <= kWResMax;
                p.wbytes = p.wres ? (unsigned)kc * wchunk : 0;
                p.stage_bytes = 32u * (unsigned)p.hcp + (p.wres ? 0 : wchunk);
                const unsigned fixed = conv_tail_bytes(cout, xg);
                if ((unsigned)smem_max < fixed + p.wbytes + p.stage_bytes) continue;
                int ns = (int)(((unsigned)smem_max - fixed - p.wbytes) / p.stage_bytes);
                p.ns = ns > 4 ? 4 : ns;
                p.ntx = (nx + bx - 1) / bx;
                p.nty = (ny + by - 1) / by;
                p.ntz = (nz + bz - 1) / bz;
                const long tiles = (long)p.ntx * p.nty * p.ntz;
                const double mma_c = nacc / 2.0 > 42.0 ? nacc / 2.0 : 42.0;
                double mma = (double)p.runs * (xg ? 9 : 27) * kc * mma_c;
                if (zg) {  // per plane N = 1, 2, 3 .. 3, 2, 1 times COUT, and the first MMAs
                    double c[4];
                    for (int q = 1; q < 4; q++) {
                        c[q] = q * cout / 2.0;                      // tensor pipe
                        const double rd = (4096 + 32.0 * q * cout) / 128;  // operand reads
                        if (c[q] < rd) c[q] = rd;
                        if (c[q] < 42) c[q] = 42;
                    }
                    mma = p.rp * (kc * 9.0 * ((bz - 2) * c[3] + 2 * c[2] + 2 * c[1]) + bz * c[1]);
                }
                const double load = kc * (2.0 * p.H * (bz + 2) * 30.0 + 32.0 * p.hc / 48.0) +
                                    (p.wres ? 0.0 : 27.0 * cout * kc);
                // epilogue per run and 16 columns (measured): ~300 cycles, ~2000
                // grouped (three TMEM reads, the boundary exchange, a barrier)
                const double epi = (double)p.runs * (cout / 16) * (xg ? 2000.0 : 300.0);
                double tile_t = mma > load ? mma : load;
                if (p.ns < 2) tile_t = mma + load;
                tile_t = p.nb == 2 ? (tile_t > epi ? tile_t : epi) : tile_t + epi;
                const double cost = (double)((tiles + nsm - 1) / nsm) * (tile_t + 300.0);
                if (cost < best_cost) {
                    best_cost = cost;
                    best = p;
                }
            }
    const int nacc = (best.xg ? 3 : 1) * cout;
    best.tmem_cols = 32;
    while (best.tmem_cols < best.nb * best.runs * nacc) best.tmem_cols *= 2;
    best.smem_bytes = best.wbytes + (unsigned)best.ns * best.stage_bytes +
                      conv_tail_bytes(cout, best.xg);
    // one CTA per SM: its tensor-memory allocation may take all 512 columns
    if (best.smem_bytes < (unsigned)smem_max / 2 + 1024) best.smem_bytes = smem_max / 2 + 1024;
    return best;
}

// cuTensorMapEncodeTiled from the driver (no link against libcuda)
using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                                 const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                 const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// A BF16 tensor map without swizzle: 16-byte aligned base and strides, boxes
// of box[] elements, zeros outside the tensor.
int encode_bf16_map(CUtensorMap *map, const void *base, int rank, const cuuint64_t *dims,
                    const cuuint64_t *strides, const cuuint32_t *box)
{
    static EncodeTiled fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiled)f;
    });
    if (!fn) {
        set_last_error("conv3d: cuTensorMapEncodeTiled unavailable", __FILE__, __LINE__);
        return HMFEM_E_CUDA;
    }
    if (((uintptr_t)base & 15u) != 0) {
        set_last_error("conv3d: tensors must be 16-byte aligned", __FILE__, __LINE__);
        return HMFEM_E_ARG;
    }
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank,
                          const_cast<void *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_last_error("conv3d: tensor map rejected", __FILE__, __LINE__);
        return HMFEM_E_ARG;
    }
    return HMFEM_OK;
}

template <int CIN, int COUT>
int launch_fwd(const void *in, const void *w, const float *bias, void *out, int nx, int ny,
               int nz, int relu, int *err, cudaStream_t st)
{
    int dev = 0, nsm = 0, smem_max = 0;
    HM_CUDA(cudaGetDevice(&dev));
    HM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    HM_CUDA(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    // the last plan this thread made for these channels: a network runs the
    // same grid again and again, and the search takes some 50 us
    struct Key { int nx, ny, nz, nsm, smem; };
    static thread_local Key key{};
    static thread_local ConvPlan plan;
    if (key.nx != nx || key.ny != ny || key.nz != nz || key.nsm != nsm || key.smem != smem_max) {
        plan = plan_conv(nx, ny, nz, CIN, COUT, nsm, smem_max);
        key = {nx, ny, nz, nsm, smem_max};
    }
    const ConvPlan &p = plan;
    auto k = k_conv3d<CIN, COUT, false, false>;
    if constexpr (3 * COUT <= 256) {
        if (p.xg) k = k_conv3d<CIN, COUT, true, false>;
        if (p.zg) k = k_conv3d<CIN, COUT, false, true>;
    }
    if (p.ns < 1) {
        set_last_error("conv3d: no tile fits in shared memory", __FILE__, __LINE__);
        return HMFEM_E_ARG;
    }
    if (((uintptr_t)in & 15u) || ((uintptr_t)out & 15u)) {
        set_last_error("conv3d: tensors must be 16-byte aligned", __FILE__, __LINE__);
        return HMFEM_E_ARG;
    }
    CUtensorMap tm_w;
    if (p.zg) {  // the taps as (dz, dx dy): dz inside
        const cuuint64_t dims[4] = {(cuuint64_t)CIN, (cuuint64_t)COUT, 3, 9};
        const cuuint64_t tap = (cuuint64_t)COUT * CIN * 2;
        const cuuint64_t strides[3] = {(cuuint64_t)CIN * 2, 9 * tap, tap};
        const cuuint32_t box[4] = {8, (cuuint32_t)COUT, 3, 9};
        const int rc = encode_bf16_map(&tm_w, w, 4, dims, strides, box);
        if (rc != HMFEM_OK) return rc;
    } else {
        const cuuint64_t dims[3] = {(cuuint64_t)CIN, (cuuint64_t)COUT, 27};
        const cuuint64_t strides[2] = {(cuuint64_t)CIN * 2, (cuuint64_t)COUT * CIN * 2};
        const cuuint32_t box[3] = {8, (cuuint32_t)COUT, 27};
        const int rc = encode_bf16_map(&tm_w, w, 3, dims, strides, box);
        if (rc != HMFEM_OK) return rc;
    }
    // (the attribute is the process's: the same value from every thread)
    HM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
    const long tiles = (long)p.ntx * p.nty * p.ntz;
    const int grid = (int)(tiles < nsm ? tiles : nsm);
    k<<<grid, kConvThreads, p.smem_bytes, st>>>((const __nv_bfloat16 *)in, tm_w, bias,
                                                (__nv_bfloat16 *)out, nx, ny, nz, relu, p, err);
    HM_LAUNCHED();
    return HMFEM_OK;
}

// N slabs per part: all of them where 9 x 8 NS columns fit in tensor memory
constexpr int wgrad_ns(int cn) { return cn == 16 ? 2 : cn == 32 || cn == 64 ? 4 : 6; }

// Estimated cycles per 16 cells of every part with these M and N channels:
// N / 2 per MMA (M = 128 rows are the array's full height), or the shared
// memory's 128 bytes a cycle where operands and incoming groups need longer.
double wgrad_cost(int cm, int cn)
{
    const int ns = wgrad_ns(cn), mblk = (3 * cm / 8 + 15) / 16, nblk = cn / 8 / ns;
    const double mma = 36.0 * ns;
    const int gmax = 3 * cm / 8 < 16 ? 3 * cm / 8 : 16;
    const double smem = ((ns == 2 ? 1 : 3) * 4096.0 + 72.0 * ns * 32 + (gmax + 3 * ns) * 256.0) / 128;
    return mblk * nblk * (mma > smem ? mma : smem);
}

template <int NS, int BY>
int launch_wgrad_cfg(const void *m, const void *nn, int cm, int cn, float *dw, int nx, int ny,
                     int nz, WgPlan p, int nsm, int *err, cudaStream_t st)
{
    using C = WgCfg<NS, BY>;
    p.nx = nx;
    p.ny = ny;
    p.nz = nz;
    p.ms = cm / 8;
    p.gm = 3 * p.ms;
    p.gmax = p.gm < 16 ? p.gm : 16;
    p.mb = p.ms % 8 == 0 ? 8 : p.ms % 4 == 0 ? 4 : 2;
    p.mblk = (p.gm + 15) / 16;
    p.parts = p.mblk * (cn / 8 / NS);
    p.nxc = (nx + 31) / 32;
    p.nyb = (ny + BY - 1) / BY;
    // CTAs per part: the SMs' share, but no fewer than ~16 steps each (every
    // CTA adds its whole D into dw at the end)
    const long cols = (long)p.nxc * p.nyb;
    long per = nsm / p.parts < 1 ? 1 : nsm / p.parts;
    const long by_work = (cols * nz + 15) / 16;
    if (per > by_work) per = by_work;
    // z planes per item: an item of zl planes loads zl + 2 N planes; the
    // makespan is the items of the fullest CTA
    double best = 1e300;
    p.zl = nz;
    for (int c = 1; c <= nz; c++) {
        const int zl = (nz + c - 1) / c, zc = (nz + zl - 1) / zl;
        const double t = (double)((cols * zc + per - 1) / per) * (zl + 1.5);
        if (t < best) {
            best = t;
            p.zl = zl;
        }
    }
    p.nzc = (nz + p.zl - 1) / p.zl;
    if (per > cols * p.nzc) per = cols * p.nzc;
    p.per = (int)per;
    p.vec = ((uintptr_t)dw & 15u) == 0;
    CUtensorMap tm[2];
    const void *base[2] = {m, nn};
    const int ch[2] = {cm, cn};
    for (int i = 0; i < 2; i++) {
        const cuuint64_t dims[4] = {(cuuint64_t)nx * 8, (cuuint64_t)ny, (cuuint64_t)nz,
                                    (cuuint64_t)ch[i] / 8};
        const cuuint64_t strides[3] = {(cuuint64_t)nx * 16, (cuuint64_t)nx * ny * 16,
                                       (cuuint64_t)nx * ny * nz * 16};
        const cuuint32_t box[4] = {256, (cuuint32_t)BY, 1, (cuuint32_t)(i == 0 ? p.mb : NS)};
        const int rc = encode_bf16_map(&tm[i], base[i], 4, dims, strides, box);
        if (rc != HMFEM_OK) return rc;
    }
    const int bytes = C::kBytes(p.gmax);
    // the A operand's 16 groups from the last M stage stay inside the buffer
    static_assert(16 * C::SP <= C::RN * C::GN * C::SP, "operand overrun");
    auto k = k_wgrad<NS, BY>;
    HM_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem));
    k<<<(unsigned)(per * p.parts), kConvThreads, bytes, st>>>(
        tm[0], tm[1], (const __nv_bfloat16 *)m, (const __nv_bfloat16 *)nn, dw, p, err);
    HM_LAUNCHED();
    return HMFEM_OK;
}

int launch_wgrad(const void *x, const void *dy, float *dw, int nx, int ny, int nz, int cin,
                 int cout, int *err, cudaStream_t st)
{
    int dev = 0, nsm = 0;
    HM_CUDA(cudaGetDevice(&dev));
    HM_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    WgPlan p{};
    p.cin = cin;
    p.cout = cout;
    p.flip = wgrad_cost(cout, cin) < wgrad_cost(cin, cout);
    const void *m = p.flip ? dy : x, *nn = p.flip ? x : dy;
    const int cm = p.flip ? cout : cin, cn = p.flip ? cin : cout;
    switch (wgrad_ns(cn)) {
    case 2: return launch_wgrad_cfg<2, 4>(m, nn, cm, cn, dw, nx, ny, nz, p, nsm, err, st);
    case 4: return launch_wgrad_cfg<4, 2>(m, nn, cm, cn, dw, nx, ny, nz, p, nsm, err, st);
    default: return launch_wgrad_cfg<6, 2>(m, nn, cm, cn, dw, nx, ny, nz, p, nsm, err, st);
    }
}

#define HM_CONV_SHAPES(X)                                                                \
    X(16, 16) X(16, 32) X(32, 16) X(32, 32) X(32, 64) X(64, 32) X(64, 64) X(96, 32)     \
    X(32, 96) X(48, 16) X(16, 48)

}  // namespace

}  // namespace hm

extern "C" {

int hmfem_conv3d_fwd(const void *in, const void *w, const float *bias, void *out, int nx,
                     int ny, int nz, int cin, int cout, int relu, int *err, void *stream)
{
    if (!in || !w || !out || !err || nx < 1 || ny < 1 || nz < 1) return HMFEM_E_ARG;
    cudaStream_t st = (cudaStream_t)stream;
#define X(a, b)                                                                               \
    if (cin == a && cout == b)                                                                \
        return hm::launch_fwd<a, b>(in, w, bias, out, nx, ny, nz, relu, err, st);
    HM_CONV_SHAPES(X)
#undef X
    hm::set_last_error("conv3d: unsupported channel counts", __FILE__, __LINE__);
    return HMFEM_E_ARG;
}

int hmfem_conv3d_plan(int nx, int ny, int nz, int cin, int cout, int nsm, int smem_max,
                      int *plan)
{
    if (!plan || nx < 1 || ny < 1 || nz < 1 || cin < 16 || cin % 16 || cout < 16 ||
        cout % 16 || cout > 256 || nsm < 1 || smem_max < 1024)
        return HMFEM_E_ARG;
    const hm::ConvPlan p = hm::plan_conv(nx, ny, nz, cin, cout, nsm, smem_max);
    const int v[21] = {p.bx, p.by, p.bz, p.W, p.H, p.hc, p.hcp, p.runs, p.rp, p.row_mode,
                       p.ntx, p.nty, p.ntz, p.ns, p.nb, p.wres, p.tmem_cols,
                       (int)p.stage_bytes, (int)p.wbytes, (int)p.smem_bytes, p.xg};
    for (int i = 0; i < 21; i++) plan[i] = v[i];
    return p.ns >= 1 ? HMFEM_OK : HMFEM_E_ARG;
}

int hmfem_conv3d_plan_zg(int nx, int ny, int nz, int cin, int cout, int nsm, int smem_max, int *zg)
{
    if (!zg || nx < 1 || ny < 1 || nz < 1 || cin < 16 || cin % 16 || cout < 16 ||
        cout % 16 || cout > 256 || nsm < 1 || smem_max < 1024)
        return HMFEM_E_ARG;
    const hm::ConvPlan p = hm::plan_conv(nx, ny, nz, cin, cout, nsm, smem_max);
    *zg = p.zg;
    return p.ns >= 1 ? HMFEM_OK : HMFEM_E_ARG;
}

int hmfem_conv3d_wgrad(const void *x, const void *dy, float *dw, int nx, int ny, int nz,
                       int cin, int cout, int *err, void *stream)
{
    if (!x || !dy || !dw || !err || nx < 1 || ny < 1 || nz < 1) return HMFEM_E_ARG;
    cudaStream_t st = (cudaStream_t)stream;
#define X(a, b)                                                                               \
    if (cin == a && cout == b) return hm::launch_wgrad(x, dy, dw, nx, ny, nz, a, b, err, st);
    HM_CONV_SHAPES(X)
#undef X
    hm::set_last_error("conv3d: unsupported channel counts", __FILE__, __LINE__);
    return HMFEM_E_ARG;
}

}  // extern "C"
