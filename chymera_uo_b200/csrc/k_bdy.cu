// k_bdy.cu -- BDYGEN's mass integrals without the O(rings x boundary points)
// masked accumulation.
//
// The reference adds every ring's multipole contribution MRING into
// MASSIN(JK) for each boundary point JK with RSPHER <= RBDY(JK), and its
// r^-(2l+1)-scaled contribution into MASSOUT(JK) for RSPHER > RBDY(JK)
// (pot/boundary.f:558-604): ~1.6 G adds at 256x128.  With the rings sorted by
// spherical radius, MASSIN(JK) is a prefix sum and MASSOUT(JK) a suffix sum
// of the same sequence, cut at the number of rings inside RBDY(JK).  The
// sorted sequence is split into sub-chunks that never straddle a cut; one CTA
// sums each sub-chunk, and each column's sub-chunk sums are scanned in
// in-order runs.  Every sum has a fixed order, so results are bit-reproducible
// alone or in a batch.
// The outside sums are accumulated from the outermost ring inward, so the
// huge r^-(2l+1) factors of inner rings never enter a difference.
//
// Compiled with --fmad=false: each product and sum rounds separately, in a
// fixed order.
#include "devplan.h"
#include "pdl.h"

namespace chy {

// Grid: (nsub, 1, ceil(batch / kSubBatch)), four threads per column.  The
// ring-table slice of a sub-chunk is loaded once and serves up to kSubBatch
// solves, two solves per pass.  Every column sum keeps its order, whatever
// the pairing.
// Latency-bound when few solves share the launch: the table slice arrives by
// asynchronous copies while a thread's moments are in flight together (one solve
// of 256x128x256 28 -> 16.4 us, of 64x32x64 14.5 -> 6.6 us, 32 solves 236 -> 225
// us against loads one after another behind the slice).
constexpr int kSubBatch = 8;
constexpr int kSubThreads = 512;
__global__ void __launch_bounds__(kSubThreads) k_bdy_sub(DevTables t, Work w, int nb, int spp)
{
    extern __shared__ double smem[];
    const int RL = t.srow, NT_ = t.ntrm;
    double *s_row = smem;                                      // [ns][RL]: TERM, r^-(2l+1), DV
    double *s_mom = smem + kSubChunk * RL;                     // [spp][ns][21]
    const int sc = blockIdx.x;
    const int s0 = t.sub_start[sc], s1 = t.sub_start[sc + 1], ns = s1 - s0;

    pdl_go();
    // per ring, geometry from the plan (TERM(I) of pot/boundary.f:385-502,
    // r^-(2l+1) of :587, DV of :516): asynchronous copies, under way while the
    // moments are gathered into registers
    const double *row = t.sterm + (size_t)s0 * RL;
    if ((RL & 1) == 0) {
        for (int i = threadIdx.x; i < ns * RL / 2; i += blockDim.x)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(s_row + 2 * i)),
                         "l"(row + 2 * i)
                         : "memory");
    } else {
        for (int i = threadIdx.x; i < ns * RL; i += blockDim.x)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(s_row + i)),
                         "l"(row + i)
                         : "memory");
    }
    pdl_wait();
    const int b0 = blockIdx.z * kSubBatch, b1 = min(nb, b0 + kSubBatch);
    for (int b = b0; b < b1; b += spp) {
        const int nsl = min(spp, b1 - b);
        // the moments of these solves, kGather of a thread's in flight at once;
        // consecutive threads take consecutive rings of one moment
        constexpr int kGather = 10;
        const int total = nsl * 21 * kSubChunk;   // rings ns .. 63 of each moment are skipped
        for (int g0 = 0; g0 < total; g0 += kGather * blockDim.x) {
            double v[kGather];
#pragma unroll
            for (int u = 0; u < kGather; ++u) {
                const int it = g0 + u * blockDim.x + threadIdx.x;
                const int r = it % kSubChunk, sl = it / (21 * kSubChunk), q = it / kSubChunk - 21 * sl;
                v[u] = 0.0;
                if (it < total && r < ns) {
                    v[u] = w.mom[(size_t)(b + sl) * w.smom + (size_t)q * t.nring + __ldg(t.ring_sorted + s0 + r)];
                }
            }
            if (g0 == 0) {
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();   // s_row landed / s_mom of the previous solves consumed
            }
            // DV * moments
#pragma unroll
            for (int u = 0; u < kGather; ++u) {
                const int it = g0 + u * blockDim.x + threadIdx.x;
                const int r = it % kSubChunk, sl = it / (21 * kSubChunk), q = it / kSubChunk - 21 * sl;
                if (it < total && r < ns) {
                    s_mom[((size_t)sl * kSubChunk + r) * 21 + q] = s_row[r * RL + NT_ + 11] * v[u];
                }
            }
        }
        __syncthreads();
        // Column col's inside and outside sums of these solves, each as four
        // partial sums (rings 4i .. 4i+3 into a0 .. a3, a remainder into a0)
        // added as (a0 + a1) + (a2 + a3): a fixed order with a quarter of the
        // dependent chain.  Lane 4 c + i of a warp holds partial sum a_i of
        // its column for both sums and both solves, so a ring's TERM and
        // r^-(2l+1) are read once for four accumulations and the product
        // TERM * DV * MRING once for the inside and the outside sum.
        {
            const int col = threadIdx.x >> 2, ph = threadIdx.x & 3;
            const bool live = col < t.ncol;
            int term = 0, l = 0, mq = 0;
            if (live) {
                term = t.col_term[col];
                l = t.col_l[col];
                mq = t.col_part[col] == 0 ? t.col_m[col] : 10 + t.col_m[col];
            }
            const double *sm0 = s_mom, *sm1 = s_mom + (size_t)kSubChunk * 21;
            double ai0 = 0.0, ao0 = 0.0, ai1 = 0.0, ao1 = 0.0;
            auto ring = [&](int r) {
                const double tt = s_row[r * RL + term], qh = s_row[r * RL + NT_ + l];
                const double p0 = tt * sm0[r * 21 + mq];
                ai0 = ai0 + p0;
                ao0 = ao0 + p0 * qh;
                if (nsl > 1) {
                    const double p1 = tt * sm1[r * 21 + mq];
                    ai1 = ai1 + p1;
                    ao1 = ao1 + p1 * qh;
                }
            };
            const int q4 = ns & ~3;
            if (live) {
                for (int r = ph; r < q4; r += 4) ring(r);
                if (ph == 0)
                    for (int r = q4; r < ns; ++r) ring(r);
            }
            // (a0 + a1) + (a2 + a3); IEEE addition commutes, so every lane of
            // the four ends with the same bits
            auto tree = [&](double v) {
                v = v + __shfl_xor_sync(0xffffffffu, v, 1);
                return v + __shfl_xor_sync(0xffffffffu, v, 2);
            };
            ai0 = tree(ai0);
            ao0 = tree(ao0);
            ai1 = tree(ai1);
            ao1 = tree(ao1);
            if (live && ph == 0) {
                double *sub = w.sub + (size_t)b * w.ssub + (size_t)sc * 2 * t.ncol + col;
                sub[0] = ai0;
                sub[t.ncol] = ao0;
                if (nsl > 1) {
                    sub[w.ssub] = ai1;
                    sub[w.ssub + t.ncol] = ao1;
                }
            }
        }
    }
}

// Grid: (ceil(2*ncol / kScanCols), 1, batch): half a warp takes kScanCols
// consecutive columns of the [2][ncol] row (inside sums, then outside sums), so
// each row is read and written in one 128-byte piece, and half-warp s the s-th of
// kScanRuns consecutive runs of sub-chunks in scan order.  Latency-bound: with
// 16 runs, each read twice eight loads at a time, one solve of 256x128x256 (872
// sub-chunks) took 17.2 us, now 7.8 us.
// scan[i][0][col] = sum of inside sums of sub-chunks < i (prefix from the
// innermost ring); scan[i][1][col] = sum of outside sums of sub-chunks >= i
// (suffix from the outermost ring).  Each run is summed in order, the run
// totals are added in order, and every prefix is that base plus the run's
// running sum: a fixed order, so the result is bit-reproducible.
constexpr int kScanCols = 16, kScanRuns = 64, kScanRegs = 16;
__global__ void __launch_bounds__(kScanCols *kScanRuns) k_bdy_scan(DevTables t, Work w)
{
    __shared__ double run_tot[kScanRuns][kScanCols];
    pdl_go();
    pdl_wait();
    const int lane = threadIdx.x % kScanCols, seg = threadIdx.x / kScanCols, b = blockIdx.z;
    const int cc = blockIdx.x * kScanCols + lane, ld = 2 * t.ncol;
    const bool live = cc < ld, out = cc >= t.ncol;
    const double *__restrict__ sub = w.sub + (size_t)b * w.ssub;
    double *__restrict__ scan = w.scan + (size_t)b * w.sscan;
    const int ns = t.nsub, per = (ns + kScanRuns - 1) / kScanRuns;
    const int lo = min(seg * per, ns), hi = min(lo + per, ns);
    // position p in scan order -> sub-chunk index
    auto idx = [&](int p) { return out ? ns - 1 - p : p; };
    // a run's loads go kU at a time, so that their latencies overlap; runs of
    // up to kScanRegs sub-chunks stay in registers for the second pass.  The
    // sums stay in order.
    constexpr int kU = 8;
    const bool held = per <= kScanRegs;
    double v[kScanRegs];
    double local = 0.0;
    if (live) {
        if (held) {
#pragma unroll
            for (int u = 0; u < kScanRegs; ++u) v[u] = lo + u < hi ? sub[(size_t)idx(lo + u) * ld + cc] : 0.0;
#pragma unroll
            for (int u = 0; u < kScanRegs; ++u)
                if (lo + u < hi) local = local + v[u];
        } else {
            for (int p0 = lo; p0 < hi; p0 += kU) {
#pragma unroll
                for (int u = 0; u < kU; ++u) v[u] = p0 + u < hi ? sub[(size_t)idx(p0 + u) * ld + cc] : 0.0;
#pragma unroll
                for (int u = 0; u < kU; ++u)
                    if (p0 + u < hi) local = local + v[u];
            }
        }
    }
    run_tot[seg][lane] = local;
    __syncthreads();
    double base = 0.0;
    for (int i = 0; i < seg; ++i) base = base + run_tot[i][lane];
    if (!live) return;
    double run = base;
    auto put = [&](int p, double x) {
        const size_t at = (size_t)idx(p) * ld + cc;
        if (!out) {
            scan[at] = run;
            run = run + x;
        } else {
            run = run + x;
            scan[at] = run;
        }
    };
    if (held) {
#pragma unroll
        for (int u = 0; u < kScanRegs; ++u)
            if (lo + u < hi) put(lo + u, v[u]);
    } else {
        for (int p0 = lo; p0 < hi; p0 += kU) {
#pragma unroll
            for (int u = 0; u < kU; ++u) v[u] = p0 + u < hi ? sub[(size_t)idx(p0 + u) * ld + cc] : 0.0;
#pragma unroll
            for (int u = 0; u < kU; ++u)
                if (p0 + u < hi) put(p0 + u, v[u]);
        }
    }
    if (seg == kScanRuns - 1) scan[(size_t)ns * ld + cc] = out ? 0.0 : run;   // the inside total
}

cudaError_t launch_bdy_sums(const DevTables &t, const Work &w, int nb, cudaStream_t s)
{
    // four lanes per column (one per partial sum), two solves per pass
    // when there are two
    if (4 * t.ncol > kSubThreads) return cudaErrorInvalidConfiguration;
    const int spp = nb >= 2 ? 2 : 1;
    const int threads = ((4 * t.ncol + 31) / 32) * 32;
    const size_t sm = (size_t)kSubChunk * (t.srow + 21 * spp) * sizeof(double);
    cudaError_t e = ensure_smem((const void *)k_bdy_sub, sm);
    if (e != cudaSuccess) return e;
    e = launch_pdl(w.pdl, k_bdy_sub, dim3(t.nsub, 1, (nb + kSubBatch - 1) / kSubBatch), dim3(threads), sm, s, t, w, nb, spp);
    if (e != cudaSuccess) return e;
    return launch_pdl(w.pdl, k_bdy_scan, dim3((2 * t.ncol + kScanCols - 1) / kScanCols, 1, nb), dim3(kScanCols * kScanRuns), 0, s, t, w);
}

}  // namespace chy
