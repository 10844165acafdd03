// k_solve.cu -- the per-mode (R,Z) solves of POT3 (pot/pot3.f:201-248).
//
// For every azimuthal mode l (m = l for the cosine half, l - N for the sine
// half) POT3 solves the block-tridiagonal system
//     AN(k) x(j,k-1) + BN(k) x(j,k) + CN(k) x(j,k+1)
//   + AM(j) x(j-1,k) + BM_m(j) x(j,k) + CM(j) x(j+1,k) = Y(j,k)
// with FISHPACK BLKTRI.  The vertical operator T_z = (AN, BN, CN) does not
// depend on m, so this library diagonalises it once per grid,
// T_z = V diag(lam) U, and solves each mode as
//     W = U Y              (vertical transform, a GEMM over all modes)
//     (T_r(m) + lam_p) w_p = W_p  for each p   (radial tridiagonal sweeps)
//     x = V W              (inverse vertical transform)
// This file holds the plain FP64 version of that pipeline.
//
// W layout: [l][j][p] (p fastest, leading dimension K) so the radial sweeps
// of 32 consecutive p's read and write coalesced rows.  Column p = K-1 holds
// zero.
//
// The vertical transforms run on the FP64 tensor pipe (mma.sync m8n8k4, IEEE
// fused multiply-adds like the scalar pipe's).  A CTA of sixteen warps keeps
// the eigenbasis matrix in registers as mma fragments, eight of its rows per
// warp, and walks (solve, l, j-tile) items through three shared-memory
// buffers filled by asynchronous copies two tiles ahead, one barrier a tile.
// At 8 solves of 256x128x256 (17.2 GFLOP each way, padded): forward 2.33 ->
// 0.605 ms, inverse 2.43 -> 0.591 ms, 29 TFLOP/s, 78% of the FP64 tensor pipe
// (ncu).  Before, scalar 4 x 4 register tiles read eight shared-memory values
// per 16 multiply-adds (7.2 TFLOP/s).  Measured on the way: eight warps with 16
// rows each 0.835 / 0.697 ms; m16n8k8 products in place of m8n8k4 the same as
// these (0.665 / 0.659 ms against 0.661 / 0.642); 64-bit item divisions in
// every warp cost 0.02-0.05 ms.
#include "devplan.h"
#include "pdl.h"

namespace chy {

constexpr int kZThreads = 512;

// Tile shape for KP = max(KMAX, 16): NWP warps along the 8-row blocks of the
// eigenbasis, NWJ warps along j, 8 MT columns each.  Shared-memory rows are
// padded so that the 16 lanes of a fragment load's half warp (4 x 4 elements)
// fall on 16 different 8-byte banks: leading dimensions are 4 or 12 mod 16.
template <int KP, int MT>
struct ZTile {
    static constexpr int NWP = KP / 8, NWJ = 16 / NWP, JT = 8 * MT * NWJ, KS = KP / 4;
    static constexpr int LDY = JT + 4, LDW = KP + 4;
    static constexpr int kFwdBuf = KP * LDY, kInvBuf = JT * LDW;   // doubles
    static constexpr size_t kFwdBytes = (size_t)3 * kFwdBuf * 8, kInvBytes = (size_t)3 * kInvBuf * 8;
};

__device__ __forceinline__ void z_cp16(double *dst, const double *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void z_cp8(double *dst, const double *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void z_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void z_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ int mode_m(int l, int n) { return l <= n ? l : l - n; }

// c += a b, the warp-wide 8 x 8 x 4 FP64 product: a holds A[lane/4][lane%4],
// b holds B[lane%4][lane/4], c holds C[lane/4][2 (lane%4) + {0, 1}].
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// W[l][j][p] = sum_k U(p,k) Y_l(j,k), Y(j,k) = 4 pi G Xhat(j,k) with the
// Dirichlet boundary folded in (pot/pot3.f:212-224).  The tile holds X as it
// lies in memory, the boundary row k = NZ with it: 4 pi G is a factor of the
// fragments, and row NZ's fragment -CN(NZ) U(p, NZ-1) folds the top boundary.
// The outer boundary column is folded into column M-1 in shared memory.
template <int KP, int MT>
__global__ void __launch_bounds__(kZThreads, 1) k_zfwd_f64(DevTables t, Work w, int nb)
{
    using Z = ZTile<KP, MT>;
    extern __shared__ __align__(16) double smem[];   // [3][KP][LDY]
    const int NZ = t.NZ, M = t.M, J = t.J, K = t.K, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wp = warp % Z::NWP, wj = warp / Z::NWP;
    double u[Z::KS];
#pragma unroll
    for (int s = 0; s < Z::KS; ++s) {
        const int k = 4 * s + lane % 4, p = wp * 8 + lane / 4;
        u[s] = (k < NZ && p < NZ) ? t.pig4 * t.U[(size_t)p * NZ + k]
               : (k == NZ && p < NZ) ? -(t.cnmax * t.U[(size_t)p * NZ + NZ - 1]) : 0.0;
    }
    // rows k >= K and columns no copy reaches start as zeros
    for (int i = tid; i < 3 * Z::kFwdBuf; i += kZThreads) smem[i] = 0.0;
    __syncthreads();
    pdl_wait();
    const int njt = (M + Z::JT - 1) / Z::JT;
    const int items = nb * t.L * njt;   // item = (solve * L + mode) * njt + tile
    const bool even = (J & 1) == 0;
    // GRAV = 0: the boundary is zero like the sources, and so is its fold
    const double edge = t.pig4 != 0.0 ? t.cmmax / t.pig4 : 0.0;
    auto load = [&](int it, double *Y) {
        if (it < items) {
            const int q = it / njt, j0 = (it - q * njt) * Z::JT;
            const double *Xl = w.X + (size_t)q * K * J;
            const int nj = J - j0 < Z::JT ? J - j0 : Z::JT;
            if (even) {
                constexpr int H = Z::JT / 2;
                for (int i = tid; i < K * H; i += kZThreads) {
                    const int k = i / H, c = 2 * (i % H);
                    if (c < nj) z_cp16(Y + k * Z::LDY + c, Xl + (size_t)k * J + j0 + c);
                }
            } else {
                for (int i = tid; i < K * Z::JT; i += kZThreads) {
                    const int k = i / Z::JT, c = i % Z::JT;
                    if (c < nj) z_cp8(Y + k * Z::LDY + c, Xl + (size_t)k * J + j0 + c);
                }
            }
        }
        z_commit();
    };
    int it = blockIdx.x;
    load(it, smem);
    load(it + (int)gridDim.x, smem + Z::kFwdBuf);
    for (int buf = 0; it < items; it += gridDim.x, buf = buf == 2 ? 0 : buf + 1) {
        if (it + (int)gridDim.x >= items) pdl_go();
        double *Yt = smem + buf * Z::kFwdBuf;
        z_wait<1>();
        __syncthreads();
        // every warp is past the previous tile: its buffer takes the tile after next
        load(it + 2 * (int)gridDim.x, smem + (buf == 0 ? 2 : buf - 1) * Z::kFwdBuf);
        const int q = it / njt, jt = it - q * njt;
        if (jt == njt - 1) {
            // Y(k, M-1) -= CM(M) X(k, M) for the tile's last column
            const double *Xl = w.X + (size_t)q * K * J;
            const int c = M - 1 - jt * Z::JT;
            if (tid < NZ)
                Yt[tid * Z::LDY + c] -= edge * (c + 1 < Z::JT ? Yt[tid * Z::LDY + c + 1] : Xl[(size_t)tid * J + M]);
            __syncthreads();
        }
        const double *Y = Yt + (lane % 4) * Z::LDY + wj * 8 * MT + lane / 4;
        double acc[MT][2] = {};
#pragma unroll
        for (int s = 0; s < Z::KS; ++s) {
            double a[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) a[m] = Y[4 * s * Z::LDY + 8 * m];
#pragma unroll
            for (int m = 0; m < MT; ++m) dmma(acc[m], a[m], u[s]);
        }
        double *Wl = w.W + (size_t)q * J * K;
        const int p = wp * 8 + 2 * (lane % 4);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const int j = jt * Z::JT + wj * 8 * MT + 8 * m + lane / 4;
            if (j < M && p < K) *reinterpret_cast<double2 *>(Wl + (size_t)j * K + p) = make_double2(acc[m][0], acc[m][1]);
        }
    }
}

// Elimination table of the radial systems (T_r(m) + lam_p): per (m, j, p) the
// pivot reciprocal 1/d_j and the multiplier c_j/d_j, BM_m(j) as
// pot/pot3.f:226-230 builds it.  They depend on the grid only, so a plan forms
// them once; each of the L modes reads the slice of its m = mode_m(l).
__global__ void __launch_bounds__(128) k_thomas_table(DevTables t, double *rec, double *mul)
{
    const int p = threadIdx.x, m = blockIdx.x, M = t.M, K = t.K;
    if (p >= t.NZ) return;
    const double xl2 = 2.0 * (t.xlamm[m] - 1.0);
    const double axis = ((m % 2 == 0) ? 1.0 : -1.0) - 1.0;
    const double lam = t.lam[p];
    size_t o = (size_t)m * M * K + p;
    double r = 1.0 / (t.bm0[0] + axis * t.ammin + xl2 * t.cc[0] + lam);
    double c = t.cm[0] * r;
    rec[o] = r;
    mul[o] = c;
    for (int j = 1; j < M; ++j) {
        o += K;
        r = 1.0 / ((t.bm0[j] + xl2 * t.cc[j]) + lam - t.am[j] * c);
        c = t.cm[j] * r;
        rec[o] = r;
        mul[o] = c;
    }
}

// Radial sweeps (T_r(m) + lam_p) w = W_p with the plan's table, one thread per
// (l, p), 128 / K modes per CTA: elimination down W, then back substitution,
// both in place.  The table takes the division (and the multiplier's store and
// reload) out of the recurrence, whose chain is then two dependent operations
// a row.  A lone warp is bound by its instruction count and its loads' latency,
// so the sweeps run over whole eight-row chunks, loaded one chunk ahead into a
// second register set at constant offsets (KC = KMAX; 0: KMAX known at run time
// only); AM is staged in shared memory (the streaming loads evict it from L1).
// At 8 solves of 256x128x256: 0.53 ms with the divisions, 0.345 ms now, about
// the time of its 330 MB per solve (W read and written twice); with an eight-byte cp.async ring three
// chunks deep instead of the registers 0.54 ms (bound by the copies' issue).
template <int KC>
__global__ void __launch_bounds__(128) k_thomas_f64(DevTables t, Work w)
{
    constexpr int U = 8;
    const int M = t.M, K = KC ? KC : t.K, p = threadIdx.x % K, b = blockIdx.y;
    const int l = blockIdx.x * (blockDim.x / K) + threadIdx.x / K;
    extern __shared__ double am[];
    for (int j = threadIdx.x; j < M; j += blockDim.x) am[j] = t.am[j];
    __syncthreads();
    pdl_wait();
    if (p >= t.NZ || l >= t.L) return;
    double *Wp = w.W + (size_t)b * w.sW + (size_t)l * t.J * K + p;
    const size_t tab = (size_t)mode_m(l, t.N) * M * K + p;
    const double *rec = t.th_rec + tab, *mul = t.th_mul + tab;
    double ya[U], ta[U], yb[U], tb[U];
    const double *lw = Wp, *lt = rec;   // next rows to load
    double prev = 0.0;
    int j = 0;
    auto load_down = [&](double (&y)[U], double (&r)[U]) {
#pragma unroll
        for (int i = 0; i < U; ++i) {
            y[i] = lw[i * K];
            r[i] = __ldg(lt + i * K);
        }
        lw += U * K;
        lt += U * K;
    };
    auto down = [&](const double (&y)[U], const double (&r)[U]) {
        double *o = Wp + (size_t)j * K;
#pragma unroll
        for (int i = 0; i < U; ++i) {
            prev = (y[i] - am[j + i] * prev) * r[i];
            o[i * K] = prev;
        }
        j += U;
    };
    int nf = M / U;
    if (nf > 0) load_down(ya, ta);
    for (int c = 0; c < nf; c += 2) {
        if (c + 1 < nf) load_down(yb, tb);
        down(ya, ta);
        if (c + 2 < nf) load_down(ya, ta);
        if (c + 1 < nf) down(yb, tb);
    }
    for (; j < M; ++j) {
        prev = (Wp[(size_t)j * K] - am[j] * prev) * __ldg(rec + (size_t)j * K);
        Wp[(size_t)j * K] = prev;
    }
    // rows M-2 .. 0, the odd ones first
    double x = prev;
    j = M - 2;
    for (int n = (M - 1) % U; n > 0; --n, --j) {
        x = Wp[(size_t)j * K] - __ldg(mul + (size_t)j * K) * x;
        Wp[(size_t)j * K] = x;
    }
    lw = Wp + (ptrdiff_t)j * K;
    lt = mul + (ptrdiff_t)j * K;
    auto load_up = [&](double (&y)[U], double (&c)[U]) {
#pragma unroll
        for (int i = 0; i < U; ++i) {
            y[i] = lw[-i * K];
            c[i] = __ldg(lt - i * K);
        }
        lw -= U * K;
        lt -= U * K;
    };
    auto up = [&](const double (&y)[U], const double (&c)[U]) {
        double *o = Wp + (ptrdiff_t)j * K;
#pragma unroll
        for (int i = 0; i < U; ++i) {
            x = y[i] - c[i] * x;
            o[-i * K] = x;
        }
        j -= U;
    };
    nf = (M - 1) / U;
    if (nf > 0) load_up(ya, ta);
    for (int c = 0; c < nf; c += 2) {
        if (c + 1 < nf) load_up(yb, tb);
        up(ya, ta);
        if (c + 2 < nf) load_up(ya, ta);
        if (c + 1 < nf) up(yb, tb);
    }
    pdl_go();
}

// The same sweeps with the eliminated rows on chip, for grids of at most 256 rows
// and KMAX >= 32: the 128 threads of a CTA own the 128 lanes of tensor memory,
// whose 512 columns hold a lane's M <= 256 FP64 values, so W is read once and
// written once.  One persistent CTA per SM walks the groups of 128 / K modes; W
// and the table rows arrive as bulk copies, sixteen rows (32 KB) a slot, kTmSlots
// slots ahead, also across groups: the next group's rows are on their way while
// this one substitutes back and stores.  Bound by HBM and the table's L2 reads.
// The recurrences, and so the bits, are k_thomas_f64's.  Eight solves of
// 256x128x256: 0.352 -> 0.228 ms (4.7 TB/s of W alone), 0.286 with the groups
// solve by solve (each solve's pass over the 67 MB of table evicts it).
constexpr int kTmSlots = 6, kTmRows = 16;
constexpr size_t kTmSlotDoubles = 2 * kTmRows * 128;
constexpr size_t kTmBytes = kTmSlots * kTmSlotDoubles * 8 + 256 * 8 + kTmSlots * 8 + 16;

__device__ __forceinline__ uint32_t tm_sm32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// bounded wait on phase `parity`: false after `limit` polls
__device__ __forceinline__ bool tm_bar_wait(uint64_t *bar, uint32_t parity, int limit)
{
    for (int i = 0; i < limit; ++i) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(tm_sm32(bar)), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tm_bulk(double *dst, const double *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(tm_sm32(dst)),
                 "l"(src), "r"(bytes), "r"(tm_sm32(bar))
                 : "memory");
}

// eight FP64 values (sixteen columns) of this thread's lane
__device__ __forceinline__ void tm_put8(uint32_t ta, const double *v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(ta),
                 "r"(__double2loint(v[0])), "r"(__double2hiint(v[0])), "r"(__double2loint(v[1])), "r"(__double2hiint(v[1])),
                 "r"(__double2loint(v[2])), "r"(__double2hiint(v[2])), "r"(__double2loint(v[3])), "r"(__double2hiint(v[3])),
                 "r"(__double2loint(v[4])), "r"(__double2hiint(v[4])), "r"(__double2loint(v[5])), "r"(__double2hiint(v[5])),
                 "r"(__double2loint(v[6])), "r"(__double2hiint(v[6])), "r"(__double2loint(v[7])), "r"(__double2hiint(v[7]))
                 : "memory");
}
__device__ __forceinline__ void tm_get8(uint32_t ta, double *v)
{
    int r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(ta)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __hiloint2double(r[2 * i + 1], r[2 * i]);
}

template <int K>
__global__ void __launch_bounds__(128, 1) k_thomas_tm(DevTables t, Work w, int groups)
{
    constexpr int R = kTmRows, G = 128 / K;   // rows of a slot, modes of a group
    extern __shared__ __align__(128) double tsm[];
    double *am = tsm + kTmSlots * kTmSlotDoubles;
    uint64_t *bar = reinterpret_cast<uint64_t *>(am + 256);
    uint32_t *slot = reinterpret_cast<uint32_t *>(bar + kTmSlots);
    const int tid = threadIdx.x, p = tid % K, g = tid / K, M = t.M, nc = (M + R - 1) / R, gl = t.L / G;
    pdl_go();
    if (tid == 0) {
        for (int i = 0; i < kTmSlots; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tm_sm32(bar + i)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int j = tid; j < M; j += 128) am[j] = t.am[j];
    pdl_wait();
    // tensor memory only once nothing is waited for that another kernel does
    if (tid < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tm_sm32(slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tm = *slot + ((uint32_t)(tid & 96) << 16);

    // group i is solve b's modes l0 ..: all solves' groups of the same table rows, of
    // both halves of the modes (m = l and l - N), one after the other, so that the
    // table comes from memory once
    const int per = 2 * (groups / gl);
    auto place = [&](int i, int &b, int &l0) {
        const int q = i / per, r = i - q * per;
        b = r >> 1;
        l0 = (q + (r & 1) * (gl / 2)) * G;
    };

    // the copies, in the order of their use: per group the chunks of W and the
    // pivot reciprocals upwards, then the multipliers' downwards (thread 0)
    int pg = blockIdx.x, ps = 0, pslot = 0, fills = 0;
    auto issue = [&]() {
        if (pg >= groups) return;
        const int c = ps < nc ? ps : 2 * nc - 1 - ps, rows = min(R, M - c * R);
        int b, l0;
        place(pg, b, l0);
        const uint32_t bytes = (uint32_t)(rows * K * 8);
        double *d = tsm + pslot * kTmSlotDoubles;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tm_sm32(bar + pslot)),
                     "r"(bytes * G * (ps < nc ? 2u : 1u))
                     : "memory");
        for (int q = 0; q < G; ++q) {
            const size_t tab = ((size_t)mode_m(l0 + q, t.N) * M + c * R) * K;
            if (ps < nc) {
                tm_bulk(d + q * R * K, w.W + (size_t)b * w.sW + ((size_t)(l0 + q) * t.J + c * R) * K, bytes, bar + pslot);
                tm_bulk(d + R * 128 + q * R * K, t.th_rec + tab, bytes, bar + pslot);
            } else {
                tm_bulk(d + R * 128 + q * R * K, t.th_mul + tab, bytes, bar + pslot);
            }
        }
        ++fills;
        pslot = pslot + 1 == kTmSlots ? 0 : pslot + 1;
        if (++ps == 2 * nc) {
            ps = 0;
            pg += gridDim.x;
        }
    };
    int cs = 0;
    uint32_t ph = 0;
    bool ok = true;
    // test hook: no copy is issued, and the first wait runs out after `probe` polls
    const int polls = w.probe > 0 ? w.probe : 1 << 26;
    if (tid == 0 && w.probe == 0)
        for (int i = 0; i < kTmSlots; ++i) issue();

    auto next = [&]() {   // this chunk's slot has been read: refill it
        __syncthreads();
        if (tid == 0 && ok) issue();
        if (++cs == kTmSlots) {
            cs = 0;
            ph ^= 1u;
        }
    };
    for (int gr = blockIdx.x; gr < groups; gr += gridDim.x) {
        int b, l;
        place(gr, b, l);
        l += g;
        double *Wp = w.W + (size_t)b * w.sW + (size_t)l * t.J * K + p;
        double prev = 0.0;
        for (int c = 0; c < nc; ++c) {
            ok = ok && tm_bar_wait(bar + cs, ph, polls);
            __syncwarp();   // the warp's tensor-memory accesses are collective
            const double *y = tsm + cs * kTmSlotDoubles + g * R * K + p, *r = y + R * 128;
            double v[R];
            const int rows = M - c * R;
            if (rows >= R) {
#pragma unroll
                for (int i = 0; i < R; ++i) v[i] = prev = (y[i * K] - am[c * R + i] * prev) * r[i * K];
            } else {
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    if (i < rows) prev = (y[i * K] - am[c * R + i] * prev) * r[i * K];
                    v[i] = prev;
                }
            }
            tm_put8(tm + c * 2 * R, v);
            tm_put8(tm + c * 2 * R + 16, v + 8);
            next();
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        double x = ok ? prev : __longlong_as_double(0x7ff8000000000000ll);   // a copy that never came
        for (int c = nc - 1; c >= 0; --c) {
            double v[R];
            tm_get8(tm + c * 2 * R, v);
            tm_get8(tm + c * 2 * R + 16, v + 8);
            ok = ok && tm_bar_wait(bar + cs, ph, polls);
            __syncwarp();
            const double *m = tsm + cs * kTmSlotDoubles + R * 128 + g * R * K + p;
            double *o = Wp + (size_t)c * R * K;
            const int last = M - 1 - c * R;   // the last row's place in its chunk: x as it is
            if (!ok) x = __longlong_as_double(0x7ff8000000000000ll);
            if (last >= R) {
#pragma unroll
                for (int i = R - 1; i >= 0; --i) {
                    x = v[i] - m[i * K] * x;
                    if (p < t.NZ) o[i * K] = x;
                }
            } else {
#pragma unroll
                for (int i = R - 1; i >= 0; --i) {
                    if (i < last) x = v[i] - m[i * K] * x;
                    if (i <= last && p < t.NZ) o[i * K] = x;
                }
            }
            next();
        }
    }
    if (!ok) {   // a wait that ran out: every slot's last copy (bounded) before the memory goes
        atomicExch(w.stat, 1);
        if (tid == 0)
            for (int i = 0; i < kTmSlots; ++i) {
                const int f = fills / kTmSlots + (i < fills % kTmSlots ? 1 : 0);
                if (f > 0) tm_bar_wait(bar + i, (uint32_t)(f - 1) & 1u, polls);
            }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(*slot));
}

// X_l(j,k) = sum_p V(k,p) W[l][j][p] for the interior (k < NZ, j < M).  A tile
// of W is one contiguous run of rows.
template <int KP, int MT>
__global__ void __launch_bounds__(kZThreads, 1) k_zinv_f64(DevTables t, Work w, int nb)
{
    using Z = ZTile<KP, MT>;
    extern __shared__ __align__(16) double smem[];   // [3][JT][LDW]
    const int NZ = t.NZ, M = t.M, J = t.J, K = t.K, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wk = warp % Z::NWP, wj = warp / Z::NWP;
    const int k = wk * 8 + lane / 4;
    pdl_go();
    double va[Z::KS];
#pragma unroll
    for (int s = 0; s < Z::KS; ++s) {
        const int p = 4 * s + lane % 4;
        va[s] = (k < NZ && p < NZ) ? t.V[(size_t)k * NZ + p] : 0.0;
    }
    // columns p >= K of narrow grids and rows no copy reaches start as zeros
    for (int i = tid; i < 3 * Z::kInvBuf; i += kZThreads) smem[i] = 0.0;
    __syncthreads();
    pdl_wait();
    const int njt = (M + Z::JT - 1) / Z::JT;
    const int items = nb * t.L * njt;
    const int h = K / 2, hs = __ffs(h) - 1;   // KMAX is a power of two
    auto load = [&](int it, double *T) {
        if (it < items) {
            const int q = it / njt, j0 = (it - q * njt) * Z::JT, rows = M - j0 < Z::JT ? M - j0 : Z::JT;
            const double *Wl = w.W + ((size_t)q * J + j0) * K;
            for (int i = tid; i < rows * h; i += kZThreads) {
                const int r = i >> hs, c = 2 * (i & (h - 1));
                z_cp16(T + r * Z::LDW + c, Wl + (size_t)r * K + c);
            }
        }
        z_commit();
    };
    int it = blockIdx.x;
    load(it, smem);
    load(it + (int)gridDim.x, smem + Z::kInvBuf);
    const bool pairs = (J & 1) == 0;
    for (int buf = 0; it < items; it += gridDim.x, buf = buf == 2 ? 0 : buf + 1) {
        z_wait<1>();
        __syncthreads();
        load(it + 2 * (int)gridDim.x, smem + (buf == 0 ? 2 : buf - 1) * Z::kInvBuf);
        const double *T = smem + buf * Z::kInvBuf + (wj * 8 * MT + lane / 4) * Z::LDW + lane % 4;
        double acc[MT][2] = {};
#pragma unroll
        for (int s = 0; s < Z::KS; ++s) {
            double x[MT];
#pragma unroll
            for (int n = 0; n < MT; ++n) x[n] = T[8 * n * Z::LDW + 4 * s];
#pragma unroll
            for (int n = 0; n < MT; ++n) dmma(acc[n], va[s], x[n]);
        }
        const int q = it / njt, jt = it - q * njt;
        double *Xl = w.X + (size_t)q * K * J;
#pragma unroll
        for (int n = 0; n < MT; ++n) {
            const int j = jt * Z::JT + wj * 8 * MT + 8 * n + 2 * (lane % 4);
            double *o = Xl + (size_t)k * J + j;
            if (k < NZ && j + 1 < M && pairs) {
                *reinterpret_cast<double2 *>(o) = make_double2(acc[n][0], acc[n][1]);
            } else if (k < NZ) {
                if (j < M) o[0] = acc[n][0];
                if (j + 1 < M) o[1] = acc[n][1];
            }
        }
    }
}

size_t thomas_table_doubles(int J, int K, int L) { return (size_t)(L / 2 + 1) * (J - 1) * K; }

cudaError_t launch_thomas_table(const DevTables &t, double *rec, double *mul, cudaStream_t s)
{
    k_thomas_table<<<t.N + 1, 128, 0, s>>>(t, rec, mul);
    return cudaGetLastError();
}

template <int KP, int MT>
static cudaError_t solve_fp64(const DevTables &t, const Work &w, int nb, int num_sms, cudaStream_t s, bool *tm)
{
    using Z = ZTile<KP, MT>;
    const int items = nb * t.L * ((t.M + Z::JT - 1) / Z::JT);   // at most 64 x 1024 x 512
    // narrower tiles while the items do not fill the SMs twice
    if constexpr (MT > 1)
        if (items < 2 * num_sms) return solve_fp64<KP, MT / 2>(t, w, nb, num_sms, s, tm);
    cudaError_t e = ensure_smem((const void *)k_zfwd_f64<KP, MT>, Z::kFwdBytes);
    if (e == cudaSuccess) e = ensure_smem((const void *)k_zinv_f64<KP, MT>, Z::kInvBytes);
    auto sweep = KP == 16 && t.K < 16 ? k_thomas_f64<0> : k_thomas_f64<KP>;
    if (e == cudaSuccess) e = ensure_smem((const void *)sweep, (size_t)t.M * sizeof(double));
    if (e != cudaSuccess) return e;
    const int grid = items < num_sms ? items : num_sms;
    e = launch_pdl(w.pdl, k_zfwd_f64<KP, MT>, dim3(grid), dim3(kZThreads), Z::kFwdBytes, s, t, w, nb);
    if (e != cudaSuccess) return e;
    const int mpb = 128 / t.K;   // modes per CTA
    const int groups = t.L / mpb * nb;
    // k_thomas_tm holds an SM with four warps.  While the groups do not outnumber
    // the SMs its chain is the shorter one (us, k_thomas_tm / k_thomas_f64): one
    // solve of 64x32x64 11.0 / 15.8, 128x64x128 14.0 / 24.8, 256x64x64 22.9 / 39.7,
    // 128x128x128 14.0 / 25.9.  Beyond that it wins by the traffic that it saves
    // where W and the table outgrow L2: 256x128x256 37 / 56, eight 228 / 352; but
    // 256x64x128 x4 43.1 / 43.7, 128x64x128 x8 42 / 37, 64x32x64 x32 31 / 21,
    // 200x32x128 x8 48 / 33 (short chains want more warps, narrow groups more copies).
    bool on_chip = false;
    if constexpr (KP >= 32) on_chip = t.K == KP && t.M <= 256 && t.L % (2 * mpb) == 0 && (groups <= num_sms || (KP == 128 && t.M > 128));
    if constexpr (KP >= 32)
        if (on_chip) {
            e = ensure_smem((const void *)k_thomas_tm<KP>, kTmBytes);
            if (e == cudaSuccess)
                e = launch_pdl(w.pdl, k_thomas_tm<KP>, dim3(groups < num_sms ? groups : num_sms), dim3(128), kTmBytes, s, t, w, groups);
        }
    *tm = on_chip;
    // k_thomas_f64 hands over at its end and starts early in up to sixteen CTAs only:
    // beside a product's 200 KB of shared memory its streaming loads have next to no
    // L1.  Queued solves, both kernels overlapped from their start / so (us): 512x32x64
    // 202 / 104, 300x128x64 221 / 181, 512x64x128 322 / 205, 512x128x128 490 / 380,
    // 129x16x64 57 / 52.  Early start against none: 4 CTAs (257x16x32) 61 / 64, 8
    // (512x16x64) 94 / 95, 16 (257x16x128) 81 / 82, 32 (300x32x128) 98 / 94, 64
    // (300x64x128) 171 / 144, 128 (512x128x128) 530 / 380.
    if (!on_chip) {
        const dim3 g((t.L + mpb - 1) / mpb, nb);
        e = launch_pdl(w.pdl && g.x * g.y <= 16, sweep, g, dim3(128), (size_t)t.M * sizeof(double), s, t, w);
    }
    if (e != cudaSuccess) return e;
    return launch_pdl(w.pdl, k_zinv_f64<KP, MT>, dim3(grid), dim3(kZThreads), Z::kInvBytes, s, t, w, nb);
}

cudaError_t launch_solve_fp64(const DevTables &t, const Work &w, int nb, int num_sms, cudaStream_t s, bool *on_chip)
{
    if (t.K <= 16) return solve_fp64<16, 4>(t, w, nb, num_sms, s, on_chip);
    if (t.K <= 32) return solve_fp64<32, 8>(t, w, nb, num_sms, s, on_chip);
    if (t.K <= 64) return solve_fp64<64, 8>(t, w, nb, num_sms, s, on_chip);
    if (t.K <= 128) return solve_fp64<128, 8>(t, w, nb, num_sms, s, on_chip);
    return cudaErrorInvalidValue;
}

}  // namespace chy
