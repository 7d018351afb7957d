// Finite-volume relaxation kernels: coloured Gauss-Seidel sweeps (the
// reference's computePotential update), FP64 residual and norm reductions,
// and the FP32 conjugate-gradient iterations used inside the FP64
// defect-correction solve.
//
// Update rule restated from Grid_3d::Table::computePotential
// (tapsim/grid_3d.cpp:1317-1371):
//   Dirichlet row: unchanged
//   Neumann row:   phi_i = (sum_j c_ij phi_j - q_i) / sum_j c_ij      (all j)
//   other rows:    the same sums skipping Neumann neighbours
// The skip is folded into ceff (0 for a Neumann neighbour of a non-Neumann
// row), so every free row is phi_i = (sum_j ceff_ij phi_j - q_i) / diag_i.
#include <cooperative_groups.h>

#include <atomic>

#include "kernels.cuh"

namespace tgd {
namespace {

constexpr int kBlock = 256;

// One row's update: phi_i = (sum_j ceff_ij phi_j - q_i) / diag_i, the sum in
// CSR order; returns |delta|, 0 with S_NAN for a NaN.  Row holds what no
// sweep writes, the first kAhead couplings among it, so that a thread has it
// in registers before the sweep before its own has ended, and the row costs
// one round of gathers.
struct SweepRow {
    static constexpr int kAhead = 16;
    int i, q0, q1;
    double d, qi;
    int c[kAhead];
    double a[kAhead];
};
__device__ __forceinline__ void sweep_load(const DevMesh& m, int i, SweepRow& r) {
    r.i = i;
    r.q0 = m.row_ptr[i];
    r.q1 = m.row_ptr[i + 1];
    r.d = m.diag64[i];
    r.qi = m.q64[i];
#pragma unroll
    for (int k = 0; k < SweepRow::kAhead; k++) {
        const bool in = r.q0 + k < r.q1;
        r.c[k] = in ? m.col[r.q0 + k] : i;
        r.a[k] = in ? m.ceff64[r.q0 + k] : 0.0;
    }
}
__device__ __forceinline__ double sweep_row(const DevMesh& m, const SweepRow& r) {
    double p[SweepRow::kAhead];
#pragma unroll
    for (int k = 0; k < SweepRow::kAhead; k++) p[k] = m.phi64[r.c[k]];
    const double old = m.phi64[r.i];
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < SweepRow::kAhead; k++)
        if (r.q0 + k < r.q1) s = fma(r.a[k], p[k], s);
    for (int q = r.q0 + SweepRow::kAhead; q < r.q1; q++) s = fma(m.ceff64[q], m.phi64[m.col[q]], s);
    const double v = (s - r.qi) / r.d;
    if (!(v == v)) {
        atomicOr(m.status, S_NAN);
        return 0.0;
    }
    m.phi64[r.i] = v;
    return fabs(v - old);
}

// One colour of a sweep over all free cells, the non-Neumann and the Neumann
// rows together (cells of one colour are never neighbours, so their order
// does not matter).  A colour of a 307k-cell tip is 15k rows, a microsecond's
// work: small blocks put it on every SM, and as links of a chain
// (launch_chain) the colours follow one another without a launch's gap.
// 25 sweeps and the copy of the potentials took 4.8 ms there with a launch per
// row list and colour and a thread loading its row as it went, 1.8 so; with
// the rows staged through shared memory by sixteen lanes each the sweeps
// alone went from 1.58 to 1.77 ms (835k cells: 2.03 to 3.36).
constexpr int kSweepBlock = 64;
__global__ void __launch_bounds__(kSweepBlock) k_sweep64(DevMesh m, const int32_t* __restrict__ rowsV, int countV,
                                                         const int32_t* __restrict__ rowsN, int countN,
                                                         double* maxdev) {
    const int t = blockIdx.x * kSweepBlock + threadIdx.x;
    const bool live = t < countV + countN;
    SweepRow r;
    if (live) sweep_load(m, t < countV ? rowsV[t] : rowsN[t - countV], r);
    chain_wait();
    double dev = live ? sweep_row(m, r) : 0.0;
    if (maxdev) {
        dev = warp_max_d(dev);
        if ((threadIdx.x & 31) == 0 && dev > 0.0) atomic_max_double_nonneg(maxdev, dev);
    }
}

// `sweeps` sweeps over the rows that k_local_set has grouped by colour, one
// block; max |delta| of the last sweep into *maxdev (cleared first).  A shell
// is a few hundred cells: a barrier per colour in one block costs less than
// a launch per colour.
constexpr int kLocalThreads = 512;
__global__ void __launch_bounds__(kLocalThreads) k_local_sweeps(DevMesh m, const int32_t* __restrict__ rows,
                                                                const int32_t* __restrict__ counts, int ncolours,
                                                                int sweeps, double* maxdev) {
    if (threadIdx.x == 0) *maxdev = 0.0;
    double dev = 0.0;
    for (int it = 0; it < sweeps; it++) {
        dev = 0.0;
        int first = 0;
        for (int c = 0; c < ncolours; c++) {
            const int n = counts[c];
            if (n == 0) continue;
            for (int t = threadIdx.x; t < n; t += kLocalThreads) {
                SweepRow r;
                sweep_load(m, rows[first + t], r);
                dev = fmax(dev, sweep_row(m, r));
            }
            first += n;
            __syncthreads();
        }
    }
    __syncthreads();
    dev = warp_max_d(dev);
    if ((threadIdx.x & 31) == 0 && dev > 0.0) atomic_max_double_nonneg(maxdev, dev);
}

// FP64 residual r_i = sum_j ceff_ij phi_j - diag_i phi_i - q_i of a row
// list, sum r^2 into *acc; one thread per row, the row's entries in CSR
// order with unfused products and sums (resid_row in cg.cu repeats them for
// the incremental residuals, bit for bit).  One thread per row keeps a
// row's whole chain of loads in flight per thread; groups of lanes per row,
// or a warp staging its rows' span in shared memory first, measured slower
// on the 7.3M-cell tip (2.4 and 3.0 TB/s against 4.1).
// r32 (may be null) gets r as float, at slotOf[i] when slotOf is given (the
// V system's slot) and at i otherwise; r64 and b64 (may be null) keep r and
// the Dirichlet part by node.  With bacc, also the squared norm of the rows'
// Dirichlet part b_i = sum over Dirichlet neighbours ceff_ij phi_j - q_i
// from the same pass.
__global__ void k_residual(DevMesh m, const int32_t* __restrict__ rows, int count, float* r32,
                           const int32_t* __restrict__ slotOf, double* acc, double* bacc, double* r64, double* b64) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const bool withB = bacc != nullptr;  // uniform over the grid
    double r2 = 0.0, b2 = 0.0;
    if (t < count) {
        const int i = rows[t];
        const int q0 = m.row_ptr[i], q1 = m.row_ptr[i + 1];
        double s = 0.0, sb = 0.0;
        for (int q = q0; q < q1; q++) {
            const int j = m.col[q];
            const double c = __dmul_rn(m.ceff64[q], m.phi64[j]);
            s = __dadd_rn(s, c);
            if (withB && (m.flags[j] & F_DIRICHLET)) sb = __dadd_rn(sb, c);
        }
        const double qi = m.q64[i];
        const double r = __dsub_rn(__dsub_rn(s, __dmul_rn(m.diag64[i], m.phi64[i])), qi);
        const double b = __dsub_rn(sb, qi);
        if (r32) r32[slotOf ? slotOf[i] : i] = (float)r;
        if (r64) r64[i] = r;
        if (b64) b64[i] = b;
        r2 = r * r;
        b2 = b * b;
    }
    if (withB) block_sum2_atomic<kBlock>(r2, b2, acc, bacc);
    else block_sum_atomic<kBlock>(r2, acc);
}

// z = r / diag, p = z, rz -> scal[0]
__global__ void k_cg_init(DevMesh m, const int32_t* __restrict__ rows, int count, CGVectors v) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double rz = 0.0, rr = 0.0;
    if (t < count) {
        const int i = rows[t];
        const float r = v.r[i];
        const float z = r / m.diag32[i];
        v.z[i] = z;
        v.p[i] = z;
        v.x[i] = 0.0f;
        rz = (double)r * (double)z;
        rr = (double)r * (double)r;
    }
    block_sum_atomic<kBlock>(rz, &v.scal[0]);
    block_sum_atomic<kBlock>(rr, &v.scal[2]);
}

// The target of r.r: rel2 times its start value (scal[2]), and at least
// abs2; an iteration whose r.r (scal[3it+2]) meets it is done.  Formed on
// the device, so that iterations queue before the host has read r.r.
__device__ __forceinline__ bool cg_met(const double* scal, int it, double rel2, double abs2) {
    return scal[3 * it + 2] <= fmax(rel2 * scal[2], abs2);
}

// an iteration replayed from a CUDA graph takes its index and targets from
// device memory (CGVectors::iter, tgt)
__device__ __forceinline__ void cg_replayed(const CGVectors& v, int& it, double& rel2, double& abs2) {
    if (v.iter) {
        it += *v.iter;
        rel2 = v.tgt[0];
        abs2 = v.tgt[1];
    }
}

// ap = A p on the rows (A = diag - offdiag), pAp -> scal[3it+1]; all three
// kernels of an iteration are skipped once it is done (cg_met)
__global__ void k_cg_spmv(DevMesh m, const int32_t* __restrict__ rows, int count, CGVectors v, int it, double rel2,
                          double abs2) {
    cg_replayed(v, it, rel2, abs2);
    if (cg_met(v.scal, it, rel2, abs2)) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double pap = 0.0;
    if (t < count) {
        const int i = rows[t];
        const int q0 = m.row_ptr[i], q1 = m.row_ptr[i + 1];
        float s = 0.0f;
        for (int q = q0; q < q1; q++) s += m.ceff32[q] * v.p[m.col[q]];
        const float pi = v.p[i];
        const float ap = m.diag32[i] * pi - s;
        v.ap[i] = ap;
        pap = (double)pi * (double)ap;
    }
    block_sum_atomic<kBlock>(pap, &v.scal[3 * it + 1]);
}

// x += a p, r -= a ap, z = r/diag, rz_next -> scal[3(it+1)], r.r -> scal[3(it+1)+2]
__global__ void k_cg_update(DevMesh m, const int32_t* __restrict__ rows, int count, CGVectors v, int it, double rel2,
                            double abs2) {
    cg_replayed(v, it, rel2, abs2);
    const double rz = v.scal[3 * it];
    if (cg_met(v.scal, it, rel2, abs2)) return;
    const double pap = v.scal[3 * it + 1];
    const float alpha = pap > 0.0 ? (float)(rz / pap) : 0.0f;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    double rzn = 0.0, rrn = 0.0;
    if (t < count) {
        const int i = rows[t];
        v.x[i] += alpha * v.p[i];
        const float r = v.r[i] - alpha * v.ap[i];
        v.r[i] = r;
        const float z = r / m.diag32[i];
        v.z[i] = z;
        rzn = (double)r * (double)z;
        rrn = (double)r * (double)r;
    }
    block_sum_atomic<kBlock>(rzn, &v.scal[3 * (it + 1)]);
    block_sum_atomic<kBlock>(rrn, &v.scal[3 * (it + 1) + 2]);
}

// p = z + beta p
__global__ void k_cg_pupdate(const int32_t* __restrict__ rows, int count, CGVectors v, int it, double rel2,
                             double abs2) {
    cg_replayed(v, it, rel2, abs2);
    const double rz = v.scal[3 * it];
    if (cg_met(v.scal, it, rel2, abs2)) return;
    const double rzn = v.scal[3 * (it + 1)];
    const float beta = (float)(rzn / rz);
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < count) {
        const int i = rows[t];
        v.p[i] = v.z[i] + beta * v.p[i];
    }
}

__global__ void k_cg_replay_begin(int32_t* iter, double* tgt, double rel2, double abs2) {
    *iter = 0;
    tgt[0] = rel2;
    tgt[1] = abs2;
}
__global__ void k_cg_replay_step(int32_t* iter) { *iter += 1; }

// The whole node-space CG solve of the Neumann rows in one launch of one
// cluster: the V rows' correction taken into the right-hand side (as
// k_vcg_couple_neumann takes it), the iterations of k_cg_spmv, k_cg_update
// and k_cg_pupdate with the same arithmetic per row, their sums through
// distributed shared memory and three cluster barriers in place of the
// kernel boundaries, and the correction applied (as k_apply_correction);
// *iters gets the iterations taken (as cg_met ends them).  The rows are a
// few thousand (6,103 of the 307k-cell tip, 11,845 of the 835k-cell one): a
// grid of them is a few blocks, and an iteration from replayed graphs was
// launches and host reads, 34 us each.  Here every block keeps the whole of p
// in shared memory, each thread its rows' couplings (to rows of the list; p
// is zero elsewhere, and there are six on average) and the rest of their
// state in registers.  What bounds an iteration is the barriers and each
// warp's share of the reductions, so 512 threads a block with up to four
// rows each beat 1024 with up to two (11,845 rows: 24 us an iteration).
// Measured: the Neumann part of a 307k-cell tip's event (15 iterations, three
// solves) 510 -> 150 us, of an 835k-cell tip's 370 -> 115 us.
constexpr int kCgThreads = 512;
constexpr int kCgCluster = 8;
constexpr int kCgWarps = kCgCluster * kCgThreads / 32;
// couplings per row kept in shared memory; a longer row reads its last ones
// from global memory
constexpr int kCgWidth = 12;
constexpr size_t cg_solve_smem(int rowsPerThread) {
    return rowsPerThread * (sizeof(float) * kCgCluster * kCgThreads +
                            (sizeof(float) + sizeof(uint16_t)) * kCgWidth * kCgThreads);
}

// Sums over the cluster of one or two values per thread: every warp's sums
// go to every block, and each warp adds them all in the same order.
// parts[turn] is written again only after another barrier.
template <bool kTwo>
__device__ __forceinline__ void cluster_sum(cooperative_groups::cluster_group& cl, double (*parts)[2][kCgWarps],
                                            int& turn, double& a, double& b) {
    const int lane = threadIdx.x & 31;
    const int warp = (int)cl.block_rank() * (kCgThreads / 32) + (threadIdx.x >> 5);
    a = warp_sum(a);
    if (kTwo) b = warp_sum(b);
    if (lane < kCgCluster) {
        *cl.map_shared_rank(&parts[turn][0][warp], lane) = a;
        if (kTwo) *cl.map_shared_rank(&parts[turn][1][warp], lane) = b;
    }
    cl.sync();
    a = b = 0.0;
#pragma unroll
    for (int k = 0; k < kCgWarps / 32; k++) {
        a += parts[turn][0][k * 32 + lane];
        if (kTwo) b += parts[turn][1][k * 32 + lane];
    }
    a = warp_sum(a);
    if (kTwo) b = warp_sum(b);
    turn ^= 1;
}

template <int kRows>
__global__ void __launch_bounds__(kCgThreads) k_cg_solve(DevMesh m, const int32_t* __restrict__ rows, int count,
                                                         CGVectors v, const int32_t* __restrict__ slotOf,
                                                         const float* __restrict__ xV, const double* __restrict__ xV64,
                                                         double rel2, double abs2, int maxIter, int32_t* iters) {
    constexpr int W = kCgWidth;
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    extern __shared__ float p[];  // the whole of p, by position in the list
    float* const val = p + kRows * kCgCluster * kCgThreads;
    uint16_t* const idx = reinterpret_cast<uint16_t*>(val + W * kRows * kCgThreads);
    __shared__ double parts[2][2][kCgWarps];
    const int tid = threadIdx.x;
    // position + 1 in the list by node (0: not in it), in the words of the
    // vector A p, which is zero outside a solve
    int32_t* const pos = reinterpret_cast<int32_t*>(v.ap);
    int row[kRows], groups[kRows], more[kRows], end[kRows];
    float x[kRows], r[kRows], z[kRows], pi[kRows], d[kRows];
#pragma unroll
    for (int k = 0; k < kRows; k++) {
        const int t = (k * kCgCluster + (int)cl.block_rank()) * kCgThreads + tid;
        row[k] = t < count ? rows[t] : -1;
        if (row[k] >= 0) __stcg(pos + row[k], t + 1);
    }
    cl.sync();  // every block has started, and pos is complete
    int turn = 0;
    double rz = 0.0, rr = 0.0;
#pragma unroll
    for (int k = 0; k < kRows; k++) {
        x[k] = r[k] = z[k] = pi[k] = 0.0f;
        d[k] = 1.0f;
        groups[k] = more[k] = end[k] = 0;
        if (row[k] < 0) continue;
        int q = m.row_ptr[row[k]], len = 0;
        end[k] = m.row_ptr[row[k] + 1];
        more[k] = end[k];
        float s = 0.0f;
        for (; q < end[k]; q += 4) {
            int c[4], j[4], sl[4];
            float a[4];
            double xv[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const bool in = q + u < end[k];
                c[u] = in ? m.col[q + u] : -1;
                a[u] = in ? m.ceff32[q + u] : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                j[u] = c[u] >= 0 ? __ldcg(pos + c[u]) : 0;
                sl[u] = c[u] >= 0 ? slotOf[c[u]] : -1;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) xv[u] = sl[u] < 0 ? 0.0 : (xV64 ? xV64[sl[u]] : (double)xV[sl[u]]);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (sl[u] >= 0) s = fmaf(a[u], (float)xv[u], s);
                if (j[u] == 0) continue;
                if (len < W) {
                    val[(k * W + len) * kCgThreads + tid] = a[u];
                    idx[(k * W + len) * kCgThreads + tid] = (uint16_t)(j[u] - 1);
                } else if (len == W) {
                    more[k] = q + u;  // the couplings from here on stay in global memory
                }
                len++;
            }
        }
        len = min(len, W);
        groups[k] = (len + 3) / 4;
        for (; len < 4 * groups[k]; len++) {  // padding: zero times the first row's p
            val[(k * W + len) * kCgThreads + tid] = 0.0f;
            idx[(k * W + len) * kCgThreads + tid] = 0;
        }
        r[k] = v.r[row[k]] + s;
        d[k] = m.diag32[row[k]];
        z[k] = pi[k] = r[k] / d[k];
        rz += (double)r[k] * (double)z[k];
        rr += (double)r[k] * (double)r[k];
        const int t = (k * kCgCluster + (int)cl.block_rank()) * kCgThreads + tid;
#pragma unroll
        for (int b = 0; b < kCgCluster; b++) cl.map_shared_rank(p, b)[t] = pi[k];
    }
    cluster_sum<true>(cl, parts, turn, rz, rr);
    const double target = fmax(rel2 * rr, abs2);
    int it = 0;
    while (it < maxIter && rr > target) {  // a NaN ends the solve
        double pap = 0.0, none = 0.0;
        float ap[kRows];
#pragma unroll
        for (int k = 0; k < kRows; k++) {
            float s = 0.0f;
            for (int g = 0; g < groups[k]; g++) {
                float a[4], pj[4];
                int at[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    a[u] = val[(k * W + 4 * g + u) * kCgThreads + tid];
                    at[u] = idx[(k * W + 4 * g + u) * kCgThreads + tid];
                }
#pragma unroll
                for (int u = 0; u < 4; u++) pj[u] = p[at[u]];
#pragma unroll
                for (int u = 0; u < 4; u++) s = fmaf(a[u], pj[u], s);
            }
            for (int q = more[k]; q < end[k]; q++) {
                const int j = __ldcg(pos + m.col[q]);
                if (j > 0) s = fmaf(m.ceff32[q], p[j - 1], s);
            }
            ap[k] = fmaf(d[k], pi[k], -s);
            pap += (double)pi[k] * (double)ap[k];
        }
        cluster_sum<false>(cl, parts, turn, pap, none);
        const float alpha = pap > 0.0 ? (float)(rz / pap) : 0.0f;
        double rzn = 0.0, rrn = 0.0;
#pragma unroll
        for (int k = 0; k < kRows; k++) {
            x[k] = fmaf(alpha, pi[k], x[k]);
            r[k] = fmaf(-alpha, ap[k], r[k]);
            z[k] = r[k] / d[k];
            rzn += (double)r[k] * (double)z[k];
            rrn += (double)r[k] * (double)r[k];
        }
        cluster_sum<true>(cl, parts, turn, rzn, rrn);
        const float beta = (float)(rzn / rz);
        rz = rzn;
        rr = rrn;
        it++;
        if (!(rr > target)) break;
        // no block still reads the old p: all have passed pap's barrier
#pragma unroll
        for (int k = 0; k < kRows; k++) {
            if (row[k] < 0) continue;
            pi[k] = fmaf(beta, pi[k], z[k]);
            const int t = (k * kCgCluster + (int)cl.block_rank()) * kCgThreads + tid;
#pragma unroll
            for (int b = 0; b < kCgCluster; b++) cl.map_shared_rank(p, b)[t] = pi[k];
        }
        cl.sync();
    }
    cl.sync();  // no block reads pos, or writes into another, any more
#pragma unroll
    for (int k = 0; k < kRows; k++)
        if (row[k] >= 0) {
            m.phi64[row[k]] += (double)x[k];
            v.r[row[k]] = 0.0f;
            __stcg(pos + row[k], 0);
        }
    if (cl.block_rank() == 0 && tid == 0) *iters = it;
}

__global__ void k_apply_correction(DevMesh m, const int32_t* __restrict__ rows, int count, CGVectors v) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    const int i = rows[t];
    m.phi64[i] += (double)v.x[i];
    v.x[i] = 0.0f;
    v.r[i] = 0.0f;
    v.z[i] = 0.0f;
    v.p[i] = 0.0f;
    v.ap[i] = 0.0f;
}

__global__ void k_rebuild_rows(DevMesh m) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m.n) return;
    const bool neuI = (m.flags[i] & F_NEUMANN) != 0;
    double d = 0.0;
    for (int q = m.row_ptr[i]; q < m.row_ptr[i + 1]; q++) {
        const bool neuJ = (m.flags[m.col[q]] & F_NEUMANN) != 0;
        const double c = (!neuI && neuJ) ? 0.0 : m.c64[q];
        m.ceff64[q] = c;
        m.ceff32[q] = (float)c;
        d += c;
    }
    m.diag64[i] = d;
    m.diag32[i] = (float)d;
}

// Breadth-first k-hop neighbourhood of one node, one block.  The visited set
// is an open-addressing hash in shared memory; frontiers live in global
// scratch.  Non-Dirichlet members are written grouped by colour.
constexpr int kHashSize = 8192;

__global__ void k_local_set(DevMesh m, int node, int hops, int32_t* out, int32_t* outCount, int cap, int32_t* scratch,
                            int scratchCap, int ncolours) {
    __shared__ int32_t hashKeys[kHashSize];
    __shared__ int frontierStart, frontierEnd, tail, overflow;
    __shared__ int colourCount[64], colourOffset[64];
    for (int k = threadIdx.x; k < kHashSize; k += blockDim.x) hashKeys[k] = -1;
    if (threadIdx.x < 64) colourCount[threadIdx.x] = 0;
    if (threadIdx.x == 0) {
        scratch[0] = node;
        frontierStart = 0;
        frontierEnd = 1;
        tail = 1;
        overflow = 0;
    }
    __syncthreads();
    // the start node is only recorded when reached again (find_localNodes)
    for (int h = 0; h < hops; h++) {
        const int fs = frontierStart, fe = frontierEnd;
        for (int f = fs + threadIdx.x; f < fe; f += blockDim.x) {
            const int u = scratch[f];
            for (int q = m.row_ptr[u]; q < m.row_ptr[u + 1]; q++) {
                const int v = m.col[q];
                uint32_t hsh = ((uint32_t)v * 2654435761u) & (kHashSize - 1);
                bool inserted = false;
                for (int probe = 0; probe < kHashSize; probe++) {
                    const int prev = atomicCAS(&hashKeys[hsh], -1, v);
                    if (prev == -1) { inserted = true; break; }
                    if (prev == v) break;
                    hsh = (hsh + 1) & (kHashSize - 1);
                }
                if (inserted) {
                    const int pos = atomicAdd(&tail, 1);
                    if (pos < scratchCap) scratch[pos] = v;
                    else overflow = 1;
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            frontierStart = fe;
            frontierEnd = min(tail, scratchCap);
        }
        __syncthreads();
    }
    // members: scratch[1 .. tail) plus the start node if it was reached again
    const int members = min(tail, scratchCap);
    for (int f = 1 + threadIdx.x; f < members; f += blockDim.x) {
        const int v = scratch[f];
        if (!(m.flags[v] & F_DIRICHLET)) atomicAdd(&colourCount[m.colour[v]], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int c = 0; c < ncolours; c++) {
            colourOffset[c] = s;
            outCount[c] = colourCount[c];
            s += colourCount[c];
            colourCount[c] = 0;
        }
        outCount[ncolours] = s;
        outCount[ncolours + 1] = overflow;
    }
    __syncthreads();
    for (int f = 1 + threadIdx.x; f < members; f += blockDim.x) {
        const int v = scratch[f];
        if (!(m.flags[v] & F_DIRICHLET)) {
            const int c = m.colour[v];
            const int pos = colourOffset[c] + atomicAdd(&colourCount[c], 1);
            if (pos < cap) out[pos] = v;
        }
    }
}

inline int blocks(int n) { return (n + kBlock - 1) / kBlock; }

}  // namespace

void launch_sweep64(const DevMesh& m, const int32_t* rowsV, int countV, const int32_t* rowsN, int countN,
                    double* maxdev, cudaStream_t s) {
    const int rows = countV + countN;
    if (rows <= 0) return;
    count_launch();
    launch_chain(k_sweep64, (unsigned)((rows + kSweepBlock - 1) / kSweepBlock), kSweepBlock, s, m, rowsV, countV, rowsN,
                 countN, maxdev);
}
void launch_local_sweeps(const DevMesh& m, const int32_t* rows, const int32_t* counts, int ncolours, int sweeps,
                         double* maxdev, cudaStream_t s) {
    count_launch();
    k_local_sweeps<<<1, kLocalThreads, 0, s>>>(m, rows, counts, ncolours, sweeps, maxdev);
}
void launch_residual(const DevMesh& m, const int32_t* rows, int count, float* r32, double* acc, cudaStream_t s,
                     double* bacc, double* r64, double* b64, const int32_t* slotOf) {
    if (count <= 0) return;
    count_launch();
    b64 = bacc ? b64 : nullptr;
    k_residual<<<blocks(count), kBlock, 0, s>>>(m, rows, count, r32, slotOf, acc, bacc, r64, b64);
}
void launch_cg_init(const DevMesh& m, const int32_t* rows, int count, CGVectors v, cudaStream_t s) {
    if (count > 0) { count_launch(); k_cg_init<<<blocks(count), kBlock, 0, s>>>(m, rows, count, v); }
}
void launch_cg_iter(const DevMesh& m, const int32_t* rows, int count, CGVectors v, int it, double rel2, double abs2,
                    cudaStream_t s) {
    if (count <= 0) return;
    { count_launch(); k_cg_spmv<<<blocks(count), kBlock, 0, s>>>(m, rows, count, v, it, rel2, abs2); }
    { count_launch(); k_cg_update<<<blocks(count), kBlock, 0, s>>>(m, rows, count, v, it, rel2, abs2); }
    { count_launch(); k_cg_pupdate<<<blocks(count), kBlock, 0, s>>>(rows, count, v, it, rel2, abs2); }
}
cudaError_t launch_cg_solve(const DevMesh& m, const int32_t* rows, int count, CGVectors v, const VSys& vs, bool fromX64,
                            double rel2, double abs2, int maxIter, int32_t* iters, cudaStream_t s) {
    static_assert(kCgSolveRows == 4 * kCgCluster * kCgThreads, "four rows per thread at most");
    auto go = [&](auto kernel, int rowsPerThread, std::atomic<uint64_t>& done) -> cudaError_t {
        const size_t smem = cg_solve_smem(rowsPerThread);
        const cudaError_t e = once_per_device(done, [&] {
            return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        });
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kCgCluster);
        cfg.blockDim = dim3(kCgThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kCgCluster;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        count_launch();
        return cudaLaunchKernelEx(&cfg, kernel, m, rows, count, v, (const int32_t*)vs.slot_of, (const float*)vs.x,
                                  (const double*)(fromX64 ? vs.x64 : nullptr), rel2, abs2, maxIter, iters);
    };
    static std::atomic<uint64_t> done[4];
    const int per = (count + kCgCluster * kCgThreads - 1) / (kCgCluster * kCgThreads);
    if (per <= 1) return go(k_cg_solve<1>, 1, done[0]);
    if (per == 2) return go(k_cg_solve<2>, 2, done[1]);
    if (per == 3) return go(k_cg_solve<3>, 3, done[2]);
    return go(k_cg_solve<4>, 4, done[3]);
}
void launch_cg_replay_begin(int32_t* iter, double* tgt, double rel2, double abs2, cudaStream_t s) {
    count_launch();
    k_cg_replay_begin<<<1, 1, 0, s>>>(iter, tgt, rel2, abs2);
}
void launch_cg_replay_step(int32_t* iter, cudaStream_t s) {
    count_launch();
    k_cg_replay_step<<<1, 1, 0, s>>>(iter);
}
void launch_apply_correction(const DevMesh& m, const int32_t* rows, int count, CGVectors v, cudaStream_t s) {
    if (count > 0) { count_launch(); k_apply_correction<<<blocks(count), kBlock, 0, s>>>(m, rows, count, v); }
}
void launch_rebuild_rows(const DevMesh& m, cudaStream_t s) {
    if (m.n > 0) { count_launch(); k_rebuild_rows<<<blocks(m.n), kBlock, 0, s>>>(m); }
}
void launch_local_set(const DevMesh& m, int node, int hops, int32_t* out, int32_t* outCount, int cap, int32_t* scratch,
                      int scratchCap, int ncolours, cudaStream_t s) {
    { count_launch(); k_local_set<<<1, 512, 0, s>>>(m, node, hops, out, outCount, cap, scratch, scratchCap, ncolours); }
}

}  // namespace tgd
