// k_blktri.cu -- POT3's mode solves in the reference's own algorithm and
// order: FISHPACK BLKTRI generalized cyclic reduction (pot/blktri.f:60-260),
// FP64, replayed from the schedule recorded on the host (blk.h).
//
// Work items are (solve, mode) pairs, 32 to a group: one lane of a warp per
// item.  Every item of a group runs the same stage/task/program sequence
// (the schedule does not depend on the mode), so a warp's lanes never
// diverge; only BM, the radial diagonal, differs between lanes.  Each item's
// vectors (Y(:,1..N) and the intermediate products, M doubles each) are
// stored lane-interleaved, [group][vector][j][lane], so every access of a
// warp is one contiguous 256-byte run.
//
// A CTA, or a cluster of CTAs, owns a group at a time and walks the stages; the
// tasks of a stage are independent PRDCT calls (or element-wise combinations)
// spread over its warps, with a barrier between stages.  k_blk_solve_tab reads
// the plan's table of pivots; k_blk_solve divides, keeps its elimination
// multipliers D and partial solution W in per-warp scratch in global memory, and
// serves plans without a table (fewer than 17 or more than 408 rows, no memory for
// one, or the caller's limit).
//
// This file is compiled with --fmad=false and its quotients are the IEEE ones:
// every product, sum and quotient rounds as the reference's, so the modes equal
// the reference's BLKTRI output bit for bit.
#include "devplan.h"
#include "pdl.h"

#include <type_traits>

namespace chy {

constexpr int kBlkLanes = 32;
constexpr int kBlkUnroll = 8;   // rows whose loads are issued ahead of the recurrence

// Y(j,k) = 4 pi G Xhat(j,k) - boundary folds (pot/pot3.f:212-224), in that
// order of operations.
__device__ __forceinline__ double blk_rhs(const DevTables &t, const double *Xl, int j, int k)
{
    double y = t.pig4 * Xl[(size_t)k * t.J + j];
    if (k == t.NZ - 1) y = y - t.cnmax * Xl[(size_t)t.NZ * t.J + j];
    if (j == t.M - 1) y = y - t.cmmax * Xl[(size_t)k * t.J + t.M];
    return y;
}

// X (mode-major) -> lane-interleaved right-hand sides Y(:,k+1) of every item
// of group g.  Grid (groups, NZ, row tiles of 32).
__global__ void __launch_bounds__(256) k_blk_gather(DevTables t, Work w, int nb)
{
    __shared__ double tile[kBlkLanes][kBlkLanes + 1];
    const int g = blockIdx.x, k = blockIdx.y, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int M = t.M, L = t.L;
    const BlkDev &d = t.blk;
    double *out = w.bvec + ((size_t)g * d.nvec + k) * (size_t)M * kBlkLanes;
    pdl_go();
    pdl_wait();
    const int j0 = blockIdx.z * kBlkLanes;
    for (int r = ty; r < kBlkLanes; r += 8) {
        const int item = g * kBlkLanes + r, b = item / L, l = item % L, j = j0 + tx;
        double v = 0.0;
        if (b < nb && j < M) v = blk_rhs(t, w.X + (size_t)b * w.sX + (size_t)l * t.K * t.J, j, k);
        tile[r][tx] = v;
    }
    __syncthreads();
    for (int jj = ty; jj < kBlkLanes; jj += 8) {
        const int j = j0 + jj;
        if (j < M) out[(size_t)j * kBlkLanes + tx] = tile[tx][jj];
    }
}

// Solved Y(:,k+1) of every item of group g -> interior of X.
__global__ void __launch_bounds__(256) k_blk_scatter(DevTables t, Work w, int nb)
{
    __shared__ double tile[kBlkLanes][kBlkLanes + 1];
    const int g = blockIdx.x, k = blockIdx.y, tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int M = t.M, L = t.L;
    const BlkDev &d = t.blk;
    const double *in = w.bvec + ((size_t)g * d.nvec + k) * (size_t)M * kBlkLanes;
    pdl_go();
    pdl_wait();
    const int j0 = blockIdx.z * kBlkLanes;
    for (int jj = ty; jj < kBlkLanes; jj += 8) {
        const int j = j0 + jj;
        tile[tx][jj] = (j < M) ? in[(size_t)j * kBlkLanes + tx] : 0.0;
    }
    __syncthreads();
    for (int r = ty; r < kBlkLanes; r += 8) {
        const int item = g * kBlkLanes + r, b = item / L, l = item % L, j = j0 + tx;
        if (b < nb && j < M) w.X[(size_t)b * w.sX + (size_t)l * t.K * t.J + (size_t)k * t.J + j] = tile[r][tx];
    }
}

// One PRDCT call (pot/blktri.f:177-260) for the 32 items of a warp.  Vector
// pointers are already offset to the lane; consecutive rows are 32 apart.
__device__ __forceinline__ void blk_prdct(const BlkProg &pg, const BlkStep *__restrict__ steps,
                                          const double *__restrict__ X, double *__restrict__ Y,
                                          double *__restrict__ Wv, double *__restrict__ Dv,
                                          const double *__restrict__ bm, const double *am, const double *cm, int m)
{
    constexpr int S = kBlkLanes, U = kBlkUnroll;
    // entry: W = X or -X, Y = W, and Y = AA(NA) W when NA > 0 (:183-208)
#pragma unroll 8
    for (int j = 0; j < m; j++) {
        double v = X[(size_t)j * S];
        if (pg.neg) v = -v;
        Y[(size_t)j * S] = pg.pre ? pg.pre_coef * v : v;
    }
    for (int q = 0; q < pg.nsteps; q++) {
        const BlkStep sp = steps[pg.first + q];
        const double rt = sp.rt;
        // elimination from row M (:214-221)
        const double bl = bm[(size_t)(m - 1) * S] - rt;
        double dn = am[m - 1] / bl;
        double wn = Y[(size_t)(m - 1) * S] / bl;
        Dv[(size_t)(m - 1) * S] = dn;
        Wv[(size_t)(m - 1) * S] = wn;
        // rows m-2 .. 1 in chunks of U; the next chunk's loads are issued
        // before this chunk's recurrence runs
        double yv[U], bv[U], yn[U], bn[U];
        auto load_e = [&](int i0, double *ya, double *ba) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 - u;
                ya[u] = (i >= 1) ? Y[(size_t)i * S] : 0.0;
                ba[u] = (i >= 1) ? bm[(size_t)i * S] : 0.0;
            }
        };
        load_e(m - 2, yv, bv);
        for (int i0 = m - 2; i0 >= 1; i0 -= U) {
            load_e(i0 - U, yn, bn);
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = i0 - u;
                if (i >= 1) {
                    const double den = bv[u] - rt - cm[i] * dn;
                    dn = am[i] / den;
                    wn = (yv[u] - cm[i] * wn) / den;
                    Dv[(size_t)i * S] = dn;
                    Wv[(size_t)i * S] = wn;
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                yv[u] = yn[u];
                bv[u] = bn[u];
            }
        }
        // row 1 (:222-228)
        const double den = bm[0] - rt - cm[0] * dn;
        double w = (den == 0) ? 1. : (Y[0] - cm[0] * wn) / den;
        // substitution (:229-231) fused with the right-hand-side update that
        // follows the pass: Y = W (:234-238), Y = Y + c W (:254-257),
        // Y = c W (:201-208)
        const int post = sp.post;
        const double c = sp.coef;
        const bool rd = post == BLK_AXPY;   // the update reads the pass's right-hand side
        auto put = [&](int j, double v, double y) {
            if (post == BLK_COPY) Y[(size_t)j * S] = v;
            else if (post == BLK_AXPY) Y[(size_t)j * S] = y + c * v;
            else if (post == BLK_SCALE) Y[(size_t)j * S] = c * v;
        };
        put(0, w, rd ? Y[0] : 0.0);
        double wv[U], dv[U], yw[U], wx[U], dx[U], yx[U];
        auto load_f = [&](int j0, double *wa, double *da, double *ya) {
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int j = j0 + u;
                wa[u] = (j < m) ? Wv[(size_t)j * S] : 0.0;
                da[u] = (j < m) ? Dv[(size_t)j * S] : 0.0;
                ya[u] = (rd && j < m) ? Y[(size_t)j * S] : 0.0;
            }
        };
        load_f(1, wv, dv, yw);
        for (int j0 = 1; j0 < m; j0 += U) {
            load_f(j0 + U, wx, dx, yx);
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int j = j0 + u;
                if (j < m) {
                    w = wv[u] - dv[u] * w;
                    put(j, w, yw[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                wv[u] = wx[u];
                dv[u] = dx[u];
                yw[u] = yx[u];
            }
        }
    }
}

// Persistent CTAs over groups; NW warps per CTA.  Dynamic shared memory
// holds AM and CM (2 M doubles).
template <int NW>
__global__ void __launch_bounds__(NW * 32) k_blk_solve(DevTables t, Work w, int ngroups)
{
    extern __shared__ double sm[];
    const BlkDev &d = t.blk;
    const int m = t.M, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *am = sm, *cm = sm + m;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        am[i] = t.am[i];
        cm[i] = t.cm[i];
    }
    __syncthreads();
    const size_t vlen = (size_t)m * kBlkLanes;
    double *Wv = w.bscr + ((size_t)blockIdx.x * NW + warp) * 2 * vlen + lane;
    double *Dv = Wv + vlen;
    for (int g = blockIdx.x; g < ngroups; g += gridDim.x) {
        double *base = w.bvec + (size_t)g * d.nvec * vlen;
        const double *bm = d.bmt + (size_t)(g % d.nblk) * vlen + lane;
        for (int s = 0; s < d.nstage; s++) {
            const BlkStage st = d.stages[s];
            if (st.kind == BLK_TASK_PRDCT) {
                for (int i = warp; i < st.ntasks; i += NW) {
                    const BlkTask tk = d.tasks[st.first + i];
                    const BlkProg pg = d.progs[tk.prog];
                    blk_prdct(pg, d.steps, base + (size_t)tk.a * vlen + lane, base + (size_t)tk.out * vlen + lane,
                              Wv, Dv, bm, am, cm, m);
                }
            } else {
                const long long total = (long long)st.ntasks * (long long)vlen;
                for (long long e = threadIdx.x; e < total; e += blockDim.x) {
                    const BlkTask tk = d.tasks[st.first + (int)(e / (long long)vlen)];
                    const size_t r = (size_t)(e % (long long)vlen);
                    const double a = base[(size_t)tk.a * vlen + r];
                    const double b = tk.b < 0 ? 0.0 : base[(size_t)tk.b * vlen + r];
                    const double c = tk.c < 0 ? 0.0 : base[(size_t)tk.c * vlen + r];
                    // Y = W1 + W2 - Y (:106-108); W1 = Y - W1 - W2 (:157-159)
                    base[(size_t)tk.out * vlen + r] = (st.kind == BLK_TASK_SUMSUB) ? (a + b) - c : (a - b) - c;
                }
            }
            __syncthreads();
        }
    }
}


// ---------------------------------------------------------------------------
// Cyclic reduction with tabulated pivots.
//
// PRDCT's elimination (pot/blktri.f:214-227) divides twice per row, for the
// multiplier D and for W.  The pivots den_i = BM_i - rt - CM_i D_(i+1) and D
// depend on the shift and the mode only, so the plan holds, for every distinct
// shift and lane-interleaved like the vectors, 1/den as the unevaluated sum
// z + l (z = 1/den rounded towards zero, l = RN(z (1 - den z)), together good to
// 2^-104), and D.
// A pass is left with one recurrence a row, W_i = (Y_i - CM_i W_(i+1)) / den_i.
//
// That quotient stays the IEEE one.  For a dividend a,
//     p = RN(a l),  q = RN(a z + p),  s = RN(RN(a z - q) + p)
// leaves a/den - q = s + e with |e| < 2^-100 |q| (2^-100 <= |den| <= 2^100 and
// |a| >= 2^-860 keep every underflow below that), and RN(q + s (1 + 2^-40)) = q
// then says that |s| is below half an ulp of q by more than |e|, so q is a/den
// rounded to nearest.  A zero a gives a z, the quotient's zero: l has z's sign.
// The recurrence goes on with q, two operations after a; a pass in which the
// test fails in any lane, or in which a dividend is tiny or not finite, is
// formed again with divisions.  (Solutions of columns without density decay over
// the rows, to 1e-155 at JMAX = 256: a threshold of 2^-500 redid one pass in ten.)
// One solve of 64x32x64 / 256x128x256: 2.29 / 50.5 ms with two divisions a row
// and the vectors in L2, 0.563 / 8.8 ms now, 112 cycles a row of both sweeps
// (clock64 around the sweeps: elimination 64, substitution 48; their dependent chains
// are 32 and 16); a batch of 32 of the latter 74.3 -> 59.2 ms.
// ---------------------------------------------------------------------------
constexpr double kBlkDenMin = 0x1p-100, kBlkDenMax = 0x1p100, kBlkNumMin = 0x1p-860;

constexpr int kBlkSlots = 4;                               // ring depth, chunks
constexpr int kBlkSlotBytes = 8 * kBlkLanes * 16;          // eight rows of (z, l) pairs

// Rows of a column as the tabulated kernel holds it: M rounded up to whole
// chunks of eight.  The rows past M are made harmless: z = l = D = CM = 0 and a
// right-hand side of one, so they solve to zero and pass the test.
__host__ __device__ inline int blk_rows(int m) { return (m + 7) & ~7; }

// Table of shift `root` and mode block blk, Mp = blk_rows(M):
// [Mp][32][z, l], then D as [Mp / 2][32][row 2r, row 2r + 1] with D_1 = 0 (the
// substitution starts from W_1 like any row).  *bad is set where a pivot is not
// a negative number of moderate size.
__global__ void __launch_bounds__(32) k_blk_table(DevTables t, double *tab, int *bad)
{
    const BlkDev &d = t.blk;
    const int m = t.M, mp = blk_rows(m), lane = threadIdx.x;
    const double *bm = d.bmt + (size_t)blockIdx.y * m * kBlkLanes + lane;
    double *zl = tab + ((size_t)blockIdx.x * d.ntab + blockIdx.y) * 3 * mp * kBlkLanes, *dd = zl + (size_t)2 * mp * kBlkLanes;
    const double rt = d.roots[blockIdx.x];
    auto put_d = [&](int i, double v) { dd[((size_t)(i >> 1) * kBlkLanes + lane) * 2 + (i & 1)] = v; };
    for (int i = m; i < mp; ++i) {
        zl[((size_t)i * kBlkLanes + lane) * 2] = zl[((size_t)i * kBlkLanes + lane) * 2 + 1] = 0.0;
        put_d(i, 0.0);
    }
    double dn = 0.0;
    bool ok = true;
    for (int i = m - 1; i >= 0; --i) {
        double den = bm[(size_t)i * kBlkLanes] - rt;
        if (i < m - 1) den = den - t.cm[i] * dn;
        dn = t.am[i] / den;
        ok = ok && den <= -kBlkDenMin && den >= -kBlkDenMax;
        const double z = __drcp_rz(den);
        zl[((size_t)i * kBlkLanes + lane) * 2] = z;
        const double e = __fma_rn(-den, z, 1.0);   // >= 0
        zl[((size_t)i * kBlkLanes + lane) * 2 + 1] = e == 0.0 ? -0.0 : __dmul_rn(e, z);
        put_d(i, i ? dn : 0.0);
    }
    if (!ok) *bad = 1;
}

__device__ __forceinline__ uint32_t blk_s32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// Eight doubles of the thread's tensor-memory lane, columns col .. col + 15.
__device__ __forceinline__ void blk_tm_st(uint32_t addr, const double (&v)[8])
{
    uint32_t r[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        r[2 * i] = (uint32_t)__double2loint(v[i]);
        r[2 * i + 1] = (uint32_t)__double2hiint(v[i]);
    }
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void blk_tm_ld(uint32_t addr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr)
        : "memory");
}
// The loads above have landed (the registers are operands, so that no use moves
// ahead of the wait).
__device__ __forceinline__ void blk_tm_wait_ld(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}
__device__ __forceinline__ void blk_tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 16-byte shared-memory accesses at a 32-bit address plus a constant.
template <int OFS>
__device__ __forceinline__ double2 blk_lds(uint32_t a)
{
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2 + %3];" : "=d"(v.x), "=d"(v.y) : "r"(a), "n"(OFS) : "memory");
    return v;
}
template <int OFS>
__device__ __forceinline__ void blk_sts(uint32_t a, double x, double y)
{
    asm volatile("st.shared.v2.f64 [%0 + %1], {%2, %3};" ::"r"(a), "n"(OFS), "d"(x), "d"(y) : "memory");
}
// f(std::integral_constant<int, 0>) .. f(std::integral_constant<int, N - 1>)
template <int N, int I = 0, class F>
__device__ __forceinline__ void blk_unroll(F f)
{
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        blk_unroll<N, I + 1>(f);
    }
}

// A lane's place in shared memory (32-bit addresses) and tensor memory.  Every
// address is the lane's own, so nothing here needs a barrier.  Columns are
// [Mp / 2][32][row 2r, row 2r + 1], 512 bytes a row pair.
struct BlkWarp {
    uint32_t y;       // right-hand side column
    uint32_t ring;    // [kBlkSlots][kBlkSlotBytes]
    uint32_t w;       // partial solutions, in shared memory or
    uint32_t tm;      // the tensor-memory address of the warp's lanes
    uint32_t cm;      // CM, [Mp] doubles, the same for every lane
};

// Passes formed again with divisions on this device so far, for the tests (as a
// plan's word it would take a register of every pass: 1% of a solve).
__device__ unsigned g_blk_redone;

// The chunk of rows i0 .. i0-7 again, with IEEE divisions: one whose quotients
// the tabulated reciprocals did not settle.  dd: the table's D.
__device__ __noinline__ double blk_elim_div(uint32_t y, uint32_t cm, const double *bm, const double *dd, double rt, int m,
                                            int i0, double wn, double *o)
{
    if (i0 < 8 && (threadIdx.x & 31) == 0) atomicAdd(&g_blk_redone, 1u);   // the pass's last chunk
#pragma unroll 1
    for (int u = 0; u < 8; ++u) {
        const int i = i0 - u;
        o[u] = 0.0;
        if (i >= m) continue;
        double yi, c;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(yi) : "r"(y + (i >> 1) * 512 + (i & 1) * 8) : "memory");
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(c) : "r"(cm + i * 8) : "memory");
        const double a = yi - c * wn;
        wn = -a;   // 0 / negative
        if (a != 0.0) {
            double den = bm[(size_t)i * kBlkLanes] - rt;
            if (i < m - 1) den = den - c * dd[((size_t)((i + 1) >> 1) * kBlkLanes) * 2 + ((i + 1) & 1)];
            wn = __ddiv_rn(a, den);
        }
        o[u] = wn;
    }
    return wn;
}

// One PRDCT call (pot/blktri.f:177-260) for the 32 items of a warp, X -> Y;
// X is read as (X - X1) - X2 where X1, X2 are given (:157-159, the combination
// that back-substitution's centre products start from).
// The right-hand side stays in shared memory between the passes and the
// partial solutions W in tensor memory (TM) or shared memory; the table comes
// through a ring of cp.async chunks of eight rows, three ahead of the
// recurrence across sweeps and passes, since loads into registers one chunk
// ahead stalled on L2.  With one warp on its scheduler every instruction of
// the two sweeps counts: two rows to a shared-memory access, constant offsets,
// no copies between register sets.
template <bool TM>
__device__ __noinline__ void blk_prdct_tab(const BlkProg &pg, const BlkStep *__restrict__ steps, const double *X,
                                              const double *X1, const double *X2, double *Y, const BlkWarp bw, const double *__restrict__ tab,
                                              size_t rstride, const double *bm, int m)
{
    constexpr int S = kBlkLanes;
    const int mp = blk_rows(m), nc = mp / 8, lane = threadIdx.x & 31, nsteps = pg.nsteps;
    // entry: Y = +-X, times AA(NA) when NA > 0 (:183-208)
    {
        // exact for +-1, and c (-v) = (-c) v
        const double f = pg.neg ? -(pg.pre ? pg.pre_coef : 1.0) : pg.pre ? pg.pre_coef : 1.0;
        auto rhs = [&](double v) { return f * v; };
        for (int j = 0; j < m; j += 32) {
            double v[32];
#pragma unroll
            for (int u = 0; u < 32; ++u) v[u] = j + u < m ? __ldcg(X + (size_t)(j + u) * S) : 0.0;
            if (X1 || X2) {   // an edge's missing neighbour product is zero
#pragma unroll
                for (int u = 0; u < 32; ++u) v[u] = v[u] - (X1 && j + u < m ? __ldcg(X1 + (size_t)(j + u) * S) : 0.0);
#pragma unroll
                for (int u = 0; u < 32; ++u) v[u] = v[u] - (X2 && j + u < m ? __ldcg(X2 + (size_t)(j + u) * S) : 0.0);
            }
            if (nsteps == 0) {
#pragma unroll
                for (int u = 0; u < 32; ++u)
                    if (j + u < m) Y[(size_t)(j + u) * S] = rhs(v[u]);
            } else {
                // rows past M hold one
                blk_unroll<16>([&](auto r) {
                    constexpr int R = decltype(r)::value;
                    if (j + 2 * R < mp)
                        blk_sts<R * 512>(bw.y + (j >> 1) * 512, j + 2 * R < m ? rhs(v[2 * R]) : 1.0,
                                         j + 2 * R + 1 < m ? rhs(v[2 * R + 1]) : 1.0);
                });
            }
        }
    }
    if (nsteps == 0) return;
    // ring: chunk n of the task is slot n % kBlkSlots; 2 nc chunks a pass, the
    // elimination's (z, l) rows from the last down, then D's rows from the first
    const BlkStep *st = steps + pg.first;
    const ptrdiff_t dofs = (ptrdiff_t)2 * mp * S;   // D within a table, doubles
    const double *tl = tab + 2 * lane;
    // a pass's table on its way into L2 while the pass before it runs: the
    // ring's lead covers L2's latency, not HBM's
    auto prefetch = [&](int q) {
        if (lane == 0 && q < nsteps)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(tab + (size_t)st[q].pad * rstride),
                         "r"((unsigned)(3 * mp * S * sizeof(double)))
                         : "memory");
    };
    prefetch(1);   // the first pass's: the stage before it
    constexpr uint32_t kRing = kBlkSlots * kBlkSlotBytes;
    uint32_t wslot = 0, rslot = 0;
    auto copy = [&](const double *src, auto rows) {
        const uint32_t dst = bw.ring + wslot;
        blk_unroll<decltype(rows)::value>([&](auto u) {
            constexpr int U = decltype(u)::value;
            asm volatile("cp.async.cg.shared.global [%0 + %2], [%1 + %2], 16;" ::"r"(dst), "l"(src), "n"(U * S * 16) : "memory");
        });
        asm volatile("cp.async.commit_group;" ::: "memory");
        wslot = wslot + kBlkSlotBytes == kRing ? 0 : wslot + kBlkSlotBytes;
    };
    auto copy_zl = [&](const double *t, int c) { copy(t + (ptrdiff_t)(mp - 8 - 8 * c) * S * 2, std::integral_constant<int, 8>{}); };
    auto copy_d = [&](const double *t, int c) { copy(t + dofs + (ptrdiff_t)(4 * c) * S * 2, std::integral_constant<int, 4>{}); };
    // the next chunk's slot, once it has landed
    auto next_slot = [&]() {
        asm volatile("cp.async.wait_group %0;" ::"n"(kBlkSlots - 2) : "memory");
        const uint32_t a = bw.ring + rslot;
        rslot = rslot + kBlkSlotBytes == kRing ? 0 : rslot + kBlkSlotBytes;
        return a;
    };
    constexpr int LEAD = kBlkSlots - 1;
    BlkStep sp = st[0];
    const double *tq = tl + (size_t)sp.pad * rstride;
#pragma unroll
    for (int c = 0; c < LEAD; ++c) copy_zl(tq, c);   // nc >= LEAD
#pragma unroll 1
    for (int q = 0; q < nsteps; ++q) {
        const bool last = q + 1 == nsteps;
        const BlkStep nx = st[last ? q : q + 1];
        const double *tn = tl + (size_t)nx.pad * rstride;
        prefetch(q + 2);
        double wn = 0.0;
        bool bad = false;
        // elimination from row M (:214-228); rows M and 1 are ordinary rows
        // (W_(M+1) = 0, and den is never zero here)
        auto keep = [&](int c, const double (&v)[8]) {   // rows ascending
            const int j0 = mp - 8 - 8 * c;
            if constexpr (TM) {
                blk_tm_st(bw.tm + 2 * j0, v);
            } else {
                const uint32_t ws = bw.w + (j0 >> 1) * 512;
                blk_unroll<4>([&](auto r) {
                    constexpr int R = decltype(r)::value;
                    blk_sts<R * 512>(ws, v[2 * R], v[2 * R + 1]);
                });
            }
        };
        // a chunk's dividends, quotients and what their tests need; a chunk is
        // tested in the gaps of the next one's recurrence
#pragma unroll 1
        for (int c = 0; c < nc; ++c) {
            const int j0 = mp - 8 - 8 * c;
            const uint32_t zs = next_slot(), ys = bw.y + (j0 >> 1) * 512, cs = bw.cm + j0 * 8;
            double2 zl[8], y[4], cr[4];
            blk_unroll<4>([&](auto r) {   // rows descending
                constexpr int R = decltype(r)::value;
                cr[R] = blk_lds<(3 - R) * 16>(cs);
                y[R] = blk_lds<(3 - R) * 512>(ys);
                zl[2 * R] = blk_lds<(7 - 2 * R) * 512>(zs);
                zl[2 * R + 1] = blk_lds<(6 - 2 * R) * 512>(zs);
            });
            if (c + LEAD < nc) copy_zl(tq, c + LEAD);
            else copy_d(tq, c + LEAD - nc);
            double a[8], pl[8], o[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                a[u] = (u & 1 ? y[u / 2].x : y[u / 2].y) - (u & 1 ? cr[u / 2].x : cr[u / 2].y) * wn;
                pl[u] = __dmul_rn(a[u], zl[u].y);
                o[7 - u] = wn = __fma_rn(a[u], zl[u].x, pl[u]);
            }
            keep(c, o);
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const double qt = o[7 - u], r = __dadd_rn(__fma_rn(a[u], zl[u].x, -qt), pl[u]);
                bad = bad | (__fma_rn(r, 1.0 + 0x1p-40, qt) != qt) | ((fabs(a[u]) < kBlkNumMin) & (a[u] != 0.0));
            }
        }
        if (__any_sync(0xffffffffu, bad)) {
            // the rows stored above go to the same columns as these: no order among
            // stores in flight
            if constexpr (TM) blk_tm_wait_st();
            wn = 0.0;
#pragma unroll 1
            for (int c = 0; c < nc; ++c) {
                double div[8], up[8];
                wn = blk_elim_div(bw.y, bw.cm, bm, tq + dofs, sp.rt, m, mp - 1 - 8 * c, wn, div);
#pragma unroll
                for (int u = 0; u < 8; ++u) up[u] = div[7 - u];
                __syncwarp();   // the store is the warp's
                keep(c, up);
            }
        }
        if constexpr (TM) blk_tm_wait_st();
        // substitution (:229-231) fused with the right-hand-side update that
        // follows the pass: Y = W (:234-238), Y = Y + c W (:254-257),
        // Y = c W (:201-208)
        const double cf = sp.coef;
        auto sweep_up = [&](auto kind) {
            constexpr int POST = decltype(kind)::value;
            double w = 0.0;
            uint32_t wr[2][16];
            if constexpr (TM) blk_tm_ld(bw.tm, wr[0]);
            auto chunk = [&](int c, uint32_t (&cur)[16], uint32_t (&nxt)[16]) {
                const uint32_t ds = next_slot(), ys = bw.y + c * 2048;
                double2 d[4], y[4], ww[4];
                blk_unroll<4>([&](auto r) {
                    constexpr int R = decltype(r)::value;
                    d[R] = blk_lds<R * 512>(ds);
                    if constexpr (!TM) ww[R] = blk_lds<R * 512>(bw.w + c * 2048);
                    if constexpr (POST == BLK_AXPY) y[R] = blk_lds<R * 512>(ys);
                });
                if constexpr (TM) {
                    blk_tm_wait_ld(cur);
                    if (c + 1 < nc) blk_tm_ld(bw.tm + 16 * (c + 1), nxt);
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        ww[r] = make_double2(__hiloint2double((int)cur[4 * r + 1], (int)cur[4 * r]),
                                             __hiloint2double((int)cur[4 * r + 3], (int)cur[4 * r + 2]));
                }
                if (c + LEAD < nc) copy_d(tq, c + LEAD);
                else if (!last) copy_zl(tn, c + LEAD - nc);
                else asm volatile("cp.async.commit_group;" ::: "memory");
                double x[8], v[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    x[u] = w = (u & 1 ? ww[u / 2].y : ww[u / 2].x) - (u & 1 ? d[u / 2].y : d[u / 2].x) * w;
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    v[u] = POST == BLK_AXPY ? (u & 1 ? y[u / 2].y : y[u / 2].x) + cf * x[u] : POST == BLK_SCALE ? cf * x[u] : x[u];
                if (last) {
                    double *out = Y + (size_t)(8 * c) * S;
                    const int n = m - 8 * c;
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        if (u < n) out[u * S] = v[u];
                } else {
                    if (c + 1 == nc) {   // the padding rows keep their ones
                        const int n = m - 8 * c;
#pragma unroll
                        for (int u = 1; u < 8; ++u)
                            if (u >= n) v[u] = 1.0;
                    }
                    blk_unroll<4>([&](auto r) {
                        constexpr int R = decltype(r)::value;
                        blk_sts<R * 512>(ys, v[2 * R], v[2 * R + 1]);
                    });
                }
            };
#pragma unroll 1
            for (int c = 0; c < nc; c += 2) {
                chunk(c, wr[0], wr[1]);
                if (c + 1 < nc) chunk(c + 1, wr[1], wr[0]);
            }
        };
        if (sp.post == BLK_AXPY) sweep_up(std::integral_constant<int, BLK_AXPY>{});
        else if (sp.post == BLK_SCALE) sweep_up(std::integral_constant<int, BLK_SCALE>{});
        else sweep_up(std::integral_constant<int, BLK_COPY>{});
        sp = nx;
        tq = tn;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

__device__ __forceinline__ void blk_group_sync(int ctas)
{
    if (ctas > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
}

// A cluster of `ctas` CTAs (1: no cluster) owns a group of 32 items at a time:
// a stage's tasks are spread over the CTAs first, then over their warps (at
// most four: a warp reaches a quarter of tensor memory's lanes).  Vectors
// another CTA may have written are read past L1.  Dynamic shared memory: CM
// (Mp doubles), then per warp ring, right-hand side column and, without TM, the
// column of partial solutions.  One CTA per SM (the launch asks for over half of
// the shared memory), so tensor memory is never waited for.  Hands over at its end:
// the next solve's clusters, resident and waiting through this one, held the SMs
// that a second stream's solve needs (two plans on two streams, 128x64x128 4.04 ->
// 2.07 ms a pair, 256x128x256 17.5 -> 12.4; one solve of 64x32x64 567 -> 561 us).
template <bool TM>
__global__ void __launch_bounds__(128, 1) k_blk_solve_tab(DevTables t, Work w, int ngroups, int ctas)
{
    extern __shared__ __align__(16) char smraw[];
    __shared__ uint32_t tm_base;
    const BlkDev &d = t.blk;
    const int m = t.M, mp = blk_rows(m), lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int rank = blockIdx.x % ctas, slot = blockIdx.x / ctas, slots = gridDim.x / ctas;
    const size_t vlen = (size_t)m * kBlkLanes, col = (size_t)mp * kBlkLanes;
    double *cm = reinterpret_cast<double *>(smraw);
    for (int i = threadIdx.x; i < mp; i += blockDim.x) cm[i] = i < m ? t.cm[i] : 0.0;
    char *mine = smraw + (size_t)mp * 8 + (size_t)warp * (kBlkSlots * kBlkSlotBytes + col * 8 * (TM ? 1 : 2));
    BlkWarp bw;
    bw.ring = blk_s32(mine) + 16 * lane;
    bw.y = bw.ring + kBlkSlots * kBlkSlotBytes;
    bw.w = bw.y + (uint32_t)(col * 8);
    bw.tm = 0;
    bw.cm = blk_s32(cm);
    uint32_t ncols = 32;
    while ((int)ncols < 2 * mp) ncols *= 2;
    if constexpr (TM) {
        if (warp == 0)
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(blk_s32(&tm_base)), "r"(ncols)
                         : "memory");
    }
    __syncthreads();
    if constexpr (TM) bw.tm = tm_base + ((uint32_t)(warp * 32) << 16);
    pdl_wait();
    const size_t rstride = (size_t)d.ntab * 3 * col;
    const int worker = rank + ctas * warp, workers = ctas * nw;
    for (int g = slot; g < ngroups; g += slots) {
        double *base = w.bvec + (size_t)g * d.nvec * vlen;
        const int mb = g % d.nblk, half = t.N / kBlkLanes, tb = mb <= half ? mb : mb - half;
        const double *tab = d.tab + (size_t)tb * 3 * col, *bm = d.bmt + (size_t)mb * vlen + lane;
        // the first passes' tables of this worker's tasks of a stage, on their way
        // into L2 a stage ahead
        auto prefetch = [&](int s) {
            if (s < d.nstage && d.stages[s].kind == BLK_TASK_SUBSUB) ++s;
            if (s >= d.nstage || d.stages[s].kind != BLK_TASK_PRDCT) return;
            const BlkStage st = d.stages[s];
            for (int i = worker + workers * lane; i < st.ntasks; i += workers * 32) {
                const BlkProg &pg = d.progs[d.tasks[st.first + i].prog];
                if (pg.nsteps > 0)
                    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(tab + (size_t)d.steps[pg.first].pad * rstride),
                                 "r"((unsigned)(3 * col * sizeof(double)))
                                 : "memory");
            }
            __syncwarp();
        };
        prefetch(0);
        for (int s = 0; s < d.nstage; ++s) {
            // back-substitution's combination W1 = Y - W1 - W2 (:157-159) feeds
            // the centre product of the same index in the stage after it, and
            // nothing else: that product forms it as it reads
            const bool sub = d.stages[s].kind == BLK_TASK_SUBSUB;
            const BlkTask *cmb = d.tasks + d.stages[s].first;
            if (sub) ++s;
            const BlkStage st = d.stages[s];
            prefetch(s + 1);
            if (s + 2 < d.nstage && d.stages[s + 1].kind == BLK_TASK_SUMSUB) prefetch(s + 2);
            auto at = [&](int v) { return v < 0 ? nullptr : base + (size_t)v * vlen + lane; };
            if (st.kind == BLK_TASK_PRDCT) {
                for (int i = worker; i < st.ntasks; i += workers) {
                    const BlkTask tk = d.tasks[st.first + i];
                    blk_prdct_tab<TM>(d.progs[tk.prog], d.steps, at(sub ? cmb[i].a : tk.a), sub ? at(cmb[i].b) : nullptr,
                                      sub ? at(cmb[i].c) : nullptr, at(tk.out), bw, tab, rstride, bm, m);
                }
            } else {
                // Y(:,I) = W1 + W2 - Y(:,I) (:106-108), sixteen rows at a time
                const int nch = (m + 15) / 16;
                for (int e = worker; e < st.ntasks * nch; e += workers) {
                    const BlkTask tk = d.tasks[st.first + e / nch];
                    const int j0 = 16 * (e % nch);
                    const size_t r = (size_t)j0 * kBlkLanes + lane;
                    const double *pa = base + (size_t)tk.a * vlen + r, *pb = base + (size_t)tk.b * vlen + r,
                                 *pc = base + (size_t)tk.c * vlen + r;
                    double a[16], b[16], c[16];
#pragma unroll
                    for (int u = 0; u < 16; ++u)
                        if (j0 + u < m) {
                            a[u] = __ldcg(pa + u * kBlkLanes);
                            b[u] = __ldcg(pb + u * kBlkLanes);
                            c[u] = __ldcg(pc + u * kBlkLanes);
                        }
                    double *o = base + (size_t)tk.out * vlen + r;
#pragma unroll
                    for (int u = 0; u < 16; ++u)
                        if (j0 + u < m) o[u * kBlkLanes] = (a[u] + b[u]) - c[u];
                }
            }
            blk_group_sync(ctas);
        }
    }
    pdl_go();
    if constexpr (TM) {
        __syncthreads();
        if (warp == 0) {
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm_base), "r"(ncols));
        }
    }
}

static int blk_groups(const DevTables &t, int nb) { return (nb * t.L + kBlkLanes - 1) / kBlkLanes; }

// Scratch holds two vectors per warp for any stage schedule the launch accepts:
// NW warps per CTA and up to ctas_per_sm CTAs per SM with NW * ctas_per_sm <= 16
// (at most 16 warps per SM, at most one CTA per group).
size_t blk_scratch_doubles(const DevTables &t, int max_batch, int num_sms)
{
    const int g = blk_groups(t, max_batch);
    return (size_t)16 * (g < num_sms ? g : num_sms) * 2 * (size_t)t.M * kBlkLanes;
}

size_t blk_vector_doubles(const DevTables &t, int nb)
{
    return (size_t)blk_groups(t, nb) * t.blk.nvec * (size_t)t.M * kBlkLanes;
}

bool blk_schedule_valid(int nw, int ctas_per_sm)
{
    return (nw == 4 || nw == 8 || nw == 16) && ctas_per_sm >= 1 && nw * ctas_per_sm <= 16;
}

template <int NW>
static cudaError_t blk_launch(const DevTables &t, const Work &w, int ngroups, int ctas, cudaStream_t s)
{
    const size_t smem = (size_t)2 * t.M * sizeof(double);
    cudaError_t e = ensure_smem((const void *)k_blk_solve<NW>, smem);
    if (e != cudaSuccess) return e;
    k_blk_solve<NW><<<ctas, NW * 32, smem, s>>>(t, w, ngroups);
    return cudaGetLastError();
}

// Shared memory a CTA of the tabulated kernel may use, and how much keeps a
// second one off its SM.
constexpr size_t kBlkSmem = 227 * 1024, kBlkSmemHalf = 116 * 1024;
static bool blk_tab_tm(int m) { return blk_rows(m) <= 256; }   // W fits tensor memory's 512 columns
static size_t blk_tab_smem(int m, int nw)
{
    const size_t col = (size_t)blk_rows(m) * kBlkLanes * 8;
    return (size_t)blk_rows(m) * 8 + nw * (kBlkSlots * kBlkSlotBytes + col * (blk_tab_tm(m) ? 1 : 2));
}
static int blk_tab_warps(int m)
{
    int nw = 4;
    while (nw > 0 && blk_tab_smem(m, nw) > kBlkSmem) --nw;
    return nw;
}

int blk_table_blocks(int L) { return L >= 64 ? L / 64 + 1 : 1; }

size_t blk_table_doubles(int M, int L, int nroots)
{
    // the ring's lead crosses no more than one sweep's end
    if (blk_tab_warps(M) == 0 || blk_rows(M) < 8 * (kBlkSlots - 1)) return 0;
    return (size_t)nroots * blk_table_blocks(L) * 3 * blk_rows(M) * kBlkLanes;
}

cudaError_t launch_blk_table(const DevTables &t, int nroots, double *tab, int *bad, cudaStream_t s)
{
    k_blk_table<<<dim3(nroots, t.blk.ntab), 32, 0, s>>>(t, tab, bad);
    return cudaGetLastError();
}

template <bool TM>
static cudaError_t blk_solve_tab(const DevTables &t, const Work &w, int ngroups, int num_sms, int nw, cudaStream_t s)
{
    const int fit = blk_tab_warps(t.M);
    if (nw > fit) nw = fit;
    size_t smem = blk_tab_smem(t.M, nw);
    if (smem < kBlkSmemHalf) smem = kBlkSmemHalf;
    cudaError_t e = ensure_smem((const void *)k_blk_solve_tab<TM>, smem);
    if (e != cudaSuccess) return e;
    // idle SMs join a group as a cluster
    int ctas = 1;
    while (ctas < 8 && 2 * ctas * ngroups <= num_sms) ctas *= 2;
    const int slots = ngroups < num_sms / ctas ? ngroups : num_sms / ctas;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(slots * ctas);
    cfg.blockDim = dim3(nw * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2] = {};
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = w.pdl ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k_blk_solve_tab<TM>, t, w, ngroups, ctas);
}

cudaError_t launch_solve_blk(const DevTables &t, const Work &w, int nb, int num_sms, int nw, int ctas_per_sm,
                             cudaStream_t s, int *launches)
{
    if (!blk_schedule_valid(nw, ctas_per_sm)) return cudaErrorInvalidValue;
    const int ngroups = blk_groups(t, nb);
    // one CTA per group at most; nw * ctas_per_sm <= 16 keeps the warps within
    // the scratch (16 per SM, no more than 16 per group)
    const int cap = ctas_per_sm * num_sms, ctas = ngroups < cap ? ngroups : cap;
    const int rtiles = (t.M + kBlkLanes - 1) / kBlkLanes;
    cudaError_t e = launch_pdl(w.pdl, k_blk_gather, dim3(ngroups, t.NZ, rtiles), dim3(256), 0, s, t, w, nb);
    if (e != cudaSuccess) return e;
    if (t.blk.tab)
        e = blk_tab_tm(t.M) ? blk_solve_tab<true>(t, w, ngroups, num_sms, nw, s)
                            : blk_solve_tab<false>(t, w, ngroups, num_sms, nw, s);
    else if (nw == 4) e = blk_launch<4>(t, w, ngroups, ctas, s);
    else if (nw == 8) e = blk_launch<8>(t, w, ngroups, ctas, s);
    else e = blk_launch<16>(t, w, ngroups, ctas, s);
    if (e != cudaSuccess) return e;
    if (launches) *launches = 3;
    return launch_pdl(w.pdl, k_blk_scatter, dim3(ngroups, t.NZ, rtiles), dim3(256), 0, s, t, w, nb);
}

cudaError_t blk_redone(unsigned *n) { return cudaMemcpyFromSymbol(n, g_blk_redone, sizeof *n); }

}  // namespace chy
