// Kernels of the learned warm start (sm_100a).
//
// Tensor-core GEMM (tcgen05):
// C[M x N] (FP32) = A[M x K] (BF16, row-major) * B[N x K]^T (BF16, row-major),
// M a multiple of 128, N 64 or 128, K a multiple of 64.  One CTA of four
// warps computes a 128 x N tile: K is staged in chunks of 64 into shared
// memory in the canonical K-major layout without swizzle (core matrices of
// 8 rows x 16 bytes; the two core matrices of one K = 16 step 128 bytes
// apart, 8-row groups 1024 bytes apart), one thread issues four
// tcgen05.mma.kind::f16 per chunk into a TMEM accumulator of N columns and
// commits them to an mbarrier, and after the last chunk each warp reads its
// 32 TMEM lanes (rows) with tcgen05.ld.  Every wait on the mbarrier is
// bounded: on timeout the kernel sets S_TIMEOUT, waits once more (bounded)
// for the MMAs in flight, frees its TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>

#include "kernels.cuh"

namespace tgd {
namespace {

constexpr int kGemmThreads = 128;
// dynamic shared memory per CTA: tiles (16 KB + 16 KB) plus slack, sized so
// that at most four CTAs share an SM and their TMEM (4 x 128 columns) fits
constexpr int kGemmSmem = 56 * 1024;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// shared-memory matrix descriptor: start, leading (K) and stride (8-row
// group) byte offsets, descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
    d |= static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16;
    d |= static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    return d;
}

// instruction descriptor: D FP32, A and B BF16, both K-major, M = 128
__host__ __device__ constexpr uint32_t idesc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(128 >> 4) << 24);
}

// bounded wait for the mbarrier phase of the given parity
__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t parity) {
    for (int i = 0; i < (1 << 22); i++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// The 16-byte piece i of a chunk as (row, K group): a warp takes eight rows
// by four groups, 512 contiguous bytes of the staged layout (eight groups of
// four rows put a warp's pieces on the same banks eightfold) and 64 of each
// row in global memory
__device__ __forceinline__ int piece_row(int i) { return (i >> 6) * 8 + (i & 7); }
__device__ __forceinline__ int piece_group(int i) { return ((i >> 5) & 1) * 4 + ((i >> 3) & 3); }

// byte offset of the 16-byte piece (row r, K group k8) of a staged chunk
__device__ __forceinline__ int tile_off(int r, int k8) { return (r >> 3) * 1024 + k8 * 128 + (r & 7) * 16; }

template <int N>
__global__ void __launch_bounds__(kGemmThreads) k_gemm_bf16(const __nv_bfloat16* __restrict__ A,
                                                            const __nv_bfloat16* __restrict__ B, float* __restrict__ C,
                                                            int M, int K, int* status) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* sA = smem;
    unsigned char* sB = smem + 16384;
    __shared__ uint64_t mbar;
    __shared__ uint32_t tmemSlot;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int row0 = blockIdx.x * 128;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmemSlot)),
                     "r"(N));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&mbar)), "r"(1));
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmemSlot;
    const uint32_t mb = smem_u32(&mbar);

    bool ok = true;
    int issued = 0;  // chunks committed to the mbarrier
    const int nk = K / 64;
    for (int kc = 0; kc < nk; kc++) {
        for (int i = tid; i < 128 * 8; i += kGemmThreads) {
            const int r = piece_row(i), c = piece_group(i);
            const uint4 v = *reinterpret_cast<const uint4*>(A + (size_t)(row0 + r) * K + kc * 64 + c * 8);
            *reinterpret_cast<uint4*>(sA + tile_off(r, c)) = v;
        }
        for (int i = tid; i < N * 8; i += kGemmThreads) {
            const int r = piece_row(i), c = piece_group(i);
            const uint4 v = *reinterpret_cast<const uint4*>(B + (size_t)r * K + kc * 64 + c * 8);
            *reinterpret_cast<uint4*>(sB + tile_off(r, c)) = v;
        }
        // the tensor core reads shared memory through the async proxy
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
            for (int ks = 0; ks < 4; ks++) {
                const uint64_t ad = umma_desc(smem_u32(sA) + ks * 256, 128, 1024);
                const uint64_t bd = umma_desc(smem_u32(sB) + ks * 256, 128, 1024);
                const uint32_t accumulate = (kc > 0 || ks > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(idesc_bf16(N)), "r"(accumulate));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mb)
                         : "memory");
        }
        issued++;
        ok = mbar_wait(mb, kc & 1);
        ok = __syncthreads_and(ok);
        if (!ok) break;
    }
    if (!ok) {
        // let the MMAs in flight finish (bounded) before the TMEM is freed
        if (tid == 0) atomicOr(status, S_TIMEOUT);
        mbar_wait(mb, (issued - 1) & 1);
    }
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (ok) {
        const int r = row0 + warp * 32 + (tid & 31);
#pragma unroll
        for (int c0 = 0; c0 < N; c0 += 16) {
            uint32_t v[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15])
                : "r"(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(c0)));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (r < M) {
                float4* out = reinterpret_cast<float4*>(C + (size_t)r * N + c0);
#pragma unroll
                for (int j = 0; j < 4; j++)
                    out[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                         __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(N));
}

// The same product for a long K and few rows (a weight gradient: 128 x 64
// with thousands of rows for its K).  One CTA per 128 x 16 tile, its chunks
// in a ring of kLongStages slots that TMA fills (128-byte swizzle): one
// thread waits for a slot, issues its MMAs, commits them to the slot's
// mbarrier and refills the slot of the step before once its MMAs are done.
// The products are added in the order of k_gemm_bf16, so the result is the
// same to the bit.  There each chunk's load, MMAs and wait followed one
// another: 343 us on 4736 rows, most of a training step, against 33
// here; with cp.async in place of TMA 75, the copies' issue the bound.
// Sharing K out over CTAs adds in another order, and Adam's first steps carry
// the last digit of a gradient near zero into the weights.
constexpr int kLongN = 16, kLongStages = 5, kLongSub = 2;  // chunks of 64 per slot
constexpr int kLongSubBytes = 16384 + kLongN * 128;
constexpr int kLongStageBytes = kLongSub * kLongSubBytes;
constexpr int kLongSmem = kLongStages * kLongStageBytes + 1024;  // slots start on 1024 bytes

// shared-memory matrix descriptor of a K-major tile with the 128-byte
// swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>((1024u >> 4) & 0x3FFFu) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}

__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t mbar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
            "r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(mbar)
        : "memory");
}

__global__ void __launch_bounds__(kGemmThreads) k_gemm_bf16_long(const __grid_constant__ CUtensorMap mapA,
                                                                 const __grid_constant__ CUtensorMap mapB,
                                                                 float* __restrict__ C, int N, int K, int* status) {
    extern __shared__ unsigned char smemRaw[];
    __shared__ uint64_t full[kLongStages], done[kLongStages];
    __shared__ uint32_t tmemSlot;
    __shared__ int good;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int row0 = blockIdx.x * 128, col0 = blockIdx.y * kLongN;
    const uint32_t smem = (smem_u32(smemRaw) + 1023u) & ~1023u;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmemSlot)),
                     "r"(32));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int k = 0; k < kLongStages; k++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&full[k])), "r"(1));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&done[k])), "r"(1));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmemSlot;
    const int chunks = K / 64, steps = (chunks + kLongSub - 1) / kLongSub;
    if (tid == 0) {
        int loaded = 0;  // steps whose copies have been issued
        auto load = [&] {
            if (loaded >= steps) return;
            const int slot = loaded % kLongStages;
            const int subs = min(kLongSub, chunks - loaded * kLongSub);
            const uint32_t mb = smem_u32(&full[slot]);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(subs * kLongSubBytes)
                         : "memory");
            for (int sub = 0; sub < subs; sub++) {
                const uint32_t at = smem + (uint32_t)(slot * kLongStageBytes + sub * kLongSubBytes);
                const int x = (loaded * kLongSub + sub) * 64;
                tma_load(at, &mapA, x, row0, mb);
                tma_load(at + 16384, &mapB, x, col0, mb);
            }
            loaded++;
        };
        for (int k = 0; k < kLongStages - 1; k++) load();
        bool ok = true;
        int issued = 0;
        for (int kc = 0; kc < steps; kc++) {
            const int slot = kc % kLongStages;
            ok = mbar_wait(smem_u32(&full[slot]), (kc / kLongStages) & 1);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            const int mmas = 4 * min(kLongSub, chunks - kc * kLongSub);
            for (int ks = 0; ks < mmas; ks++) {
                const uint32_t at = smem + (uint32_t)(slot * kLongStageBytes + (ks >> 2) * kLongSubBytes + (ks & 3) * 32);
                const uint64_t ad = umma_desc_sw128(at), bd = umma_desc_sw128(at + 16384);
                const uint32_t accumulate = (kc > 0 || ks > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(idesc_bf16(kLongN)), "r"(accumulate));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&done[slot]))
                         : "memory");
            issued++;
            if (kc > 0) {
                ok = mbar_wait(smem_u32(&done[(kc - 1) % kLongStages]), ((kc - 1) / kLongStages) & 1);
                if (!ok) break;
            }
            load();
        }
        // the last MMAs (they complete in order), and after a time-out the
        // copies still in flight
        if (issued > 0)
            ok = mbar_wait(smem_u32(&done[(issued - 1) % kLongStages]), ((issued - 1) / kLongStages) & 1) && ok;
        for (int k = issued; k < loaded; k++) mbar_wait(smem_u32(&full[k % kLongStages]), (k / kLongStages) & 1);
        if (!ok) atomicOr(status, S_TIMEOUT);
        good = ok ? 1 : 0;
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (good) {
        const int r = row0 + warp * 32 + (tid & 31);
        uint32_t v[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(tmem + (static_cast<uint32_t>(warp * 32) << 16)));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        float4* out = reinterpret_cast<float4*>(C + (size_t)r * N + col0);
#pragma unroll
        for (int j = 0; j < 4; j++)
            out[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                 __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(32));
}

// Tensor map of a row-major BF16 matrix of `rows` rows of K values: boxes of
// 64 values by boxRows rows, 128-byte swizzle (K a multiple of 64, so a box
// starts on 128 bytes and never leaves its rows)
cudaError_t bf16_map(CUtensorMap* map, const void* p, int rows, int K, int boxRows) {
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {  // initialised once, also under concurrent host threads
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult found{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            fn = nullptr;
        return reinterpret_cast<Encode>(fn);
    }();
    if (!encode) return cudaErrorNotSupported;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)boxRows}, step[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, step,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------
// Message-passing network on the free cells around a removed atom.
//
// Graph: the free cells within `hops` steps of the removed cell (a BFS over
// the coupling graph that does not enter Dirichlet cells), edges weighted
// a_ij = c_ij / d_i (the Jacobi weights of the relaxation), stored ELL
// (width D, -1 padding).  Per node 16 input features (below); an input
// layer and four message layers of width 64:
//   h0 = relu(x W0 + b0);  h_l = h_{l-1} + relu([h_{l-1}, A h_{l-1}] W_l + b_l)
//   y  = h4 . w_out + b_out,   predicted correction = sigma * y
// with sigma = |r_site| / d_site, the Jacobi step of the removed cell.  The
// GEMMs run on the tensor cores (BF16 operands, FP32 accumulate); the rest
// is FP32 on the CUDA cores.  Inputs are padded to 128 columns so that every
// GEMM has M % 128 == 0 and K % 64 == 0.
// ---------------------------------------------------------------------------
constexpr int kFeat = 16, kHid = 64, kCat = 128;

// Breadth-first search from `site` over the free cells, `hops` levels, one
// CTA: each warp takes a frontier cell and its lanes its neighbours, which
// claim their cell with an atomic on localOf (-1 -> -2), so a level costs
// one round of loads instead of one per neighbour.  The list order follows
// the claims (it varies from run to run; nothing downstream depends on it).
__global__ void k_ball_bfs(DevMesh m, int site, int hops, int cap, int32_t* nodes, int8_t* level, int32_t* count,
                           int32_t* localOf) {
    __shared__ int lvlStart, lvlEnd, total;
    if (threadIdx.x == 0) {
        nodes[0] = site;
        level[0] = 0;
        localOf[site] = 0;
        lvlStart = 0;
        lvlEnd = 1;
        total = 1;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int L = 0; L < hops; L++) {
        const int s0 = lvlStart, s1 = lvlEnd;
        for (int t = s0 + warp; t < s1; t += nwarps) {
            const int u = nodes[t];
            const int q1 = m.row_ptr[u + 1];
            for (int q = m.row_ptr[u] + lane; q < q1; q += 32) {
                const int j = m.col[q];
                if (m.flags[j] & F_DIRICHLET) continue;
                if (atomicCAS(&localOf[j], -1, -2) != -1) continue;
                const int idx = atomicAdd(&total, 1);
                if (idx < cap) {
                    nodes[idx] = j;
                    level[idx] = (int8_t)(L + 1);
                    localOf[j] = idx;
                } else {
                    localOf[j] = -1;
                }
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            lvlStart = s1;
            lvlEnd = min(total, cap);
        }
        __syncthreads();
    }
    // a neighbourhood larger than `cap` is cut at cap cells (a smaller
    // prediction region, not an error: the solve still converges)
    if (threadIdx.x == 0) *count = min(total, cap);
}

__global__ void k_ball_reset(const int32_t* nodes, const int32_t* count, int32_t* localOf) {
    const int n = *count;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) localOf[nodes[t]] = -1;
}

// scale[0] = sigma = |r_site| / d_site, scale[1] = mean distance from the
// site to its neighbours
__global__ void k_site_scale(DevMesh m, int site, float* scale) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double sum = 0.0, dist = 0.0;
    int nbs = 0;
    const double xs = m.xyz[3 * site], ys = m.xyz[3 * site + 1], zs = m.xyz[3 * site + 2];
    for (int q = m.row_ptr[site]; q < m.row_ptr[site + 1]; q++) {
        const int j = m.col[q];
        sum += m.ceff64[q] * m.phi64[j];
        const double dx = m.xyz[3 * j] - xs, dy = m.xyz[3 * j + 1] - ys, dz = m.xyz[3 * j + 2] - zs;
        dist += sqrt(dx * dx + dy * dy + dz * dz);
        nbs++;
    }
    const double r = sum - m.diag64[site] * m.phi64[site] - m.q64[site];
    const double d = m.diag64[site];
    double sigma = d > 0.0 ? fabs(r) / d : 0.0;
    if (!(sigma > 1e-30)) sigma = 1e-30;
    scale[0] = (float)sigma;
    scale[1] = nbs > 0 ? (float)(dist / nbs) : 1.0f;
}

// features, ELL rows and (for sample collection) the start potentials; one
// warp per cell, its lanes over the cell's neighbours (warp sums, and the
// ELL row compacted in CSR order by ballots)
__global__ void k_ball_features(DevMesh m, int site, int hops, int D, const int32_t* nodes, const int8_t* level,
                                const int32_t* count, const int32_t* localOf, const float* scale, float* X,
                                int32_t* ellCol, float* ellW, double* phiStart) {
    const int n = *count;
    const int lane = threadIdx.x & 31;
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= n) return;
    const int g = nodes[t];
    const double sigma = scale[0], ell = scale[1];
    const double xs = m.xyz[3 * site], ys = m.xyz[3 * site + 1], zs = m.xyz[3 * site + 2];
    const double dx = m.xyz[3 * g] - xs, dy = m.xyz[3 * g + 1] - ys, dz = m.xyz[3 * g + 2] - zs;
    const double dist = sqrt(dx * dx + dy * dy + dz * dz);
    double sum = 0.0, fixedC = 0.0, allC = 0.0;
    int k = 0;  // ELL entries written so far (the same in every lane)
    const double dg = m.diag64[g];
    const int q0 = m.row_ptr[g], q1 = m.row_ptr[g + 1];
    for (int base = q0; base < q1; base += 32) {
        const int q = base + lane;
        int lj = -1;
        double c = 0.0;
        if (q < q1) {
            const int j = m.col[q];
            c = m.ceff64[q];
            sum += c * m.phi64[j];
            const double c64 = m.c64[q];
            allC += c64;
            if (m.flags[j] & F_DIRICHLET) fixedC += c64;
            lj = localOf[j];
        }
        const bool take = q < q1 && lj >= 0 && lj < n && c != 0.0;
        const unsigned mask = __ballot_sync(0xffffffffu, take);
        const int at = k + __popc(mask & ((1u << lane) - 1u));
        if (take && at < D) {
            ellCol[(size_t)t * D + at] = lj;
            ellW[(size_t)t * D + at] = dg > 0.0 ? (float)(c / dg) : 0.0f;
        }
        k = min(D, k + __popc(mask));
    }
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        allC += __shfl_xor_sync(0xffffffffu, allC, o);
        fixedC += __shfl_xor_sync(0xffffffffu, fixedC, o);
    }
    for (int e = k + lane; e < D; e += 32) {
        ellCol[(size_t)t * D + e] = -1;
        ellW[(size_t)t * D + e] = 0.0f;
    }
    if (lane != 0) return;
    const double r = sum - dg * m.phi64[g] - m.q64[g];
    float* x = X + (size_t)t * kFeat;
    x[0] = (float)(dx / ell);
    x[1] = (float)(dy / ell);
    x[2] = (float)(dz / ell);
    x[3] = (float)(dist / ell);
    x[4] = (float)level[t] / (float)hops;
    x[5] = g == site ? 1.0f : 0.0f;
    x[6] = (m.flags[g] & F_NEUMANN) ? 1.0f : 0.0f;
    x[7] = allC > 0.0 ? (float)(fixedC / allC) : 0.0f;
    x[8] = dg > 0.0 ? (float)(r / (dg * sigma)) : 0.0f;
    x[9] = (float)(m.phi64[g] - m.phi64[site]);
    x[10] = (dg > 0.0 && m.diag64[site] > 0.0) ? (float)log(dg / m.diag64[site]) : 0.0f;
    x[11] = (float)(log10(sigma) / 10.0);
    x[12] = x[13] = x[14] = x[15] = 0.0f;
    if (phiStart) phiStart[t] = m.phi64[g];
}

// A tile of kTileRows rows, kept by column so that its transposed copy goes
// out in runs of rows: the kernels that write an activation both ways are a
// block per tile, a thread per feature of every eighth or sixteenth row
// (written straight to a column-major array, each value went to a sector of
// its own).
constexpr int kTileRows = 32, kTileThreads = 512, kConcatThreads = 1024;
template <int kCols>
struct RowTile {
    __nv_bfloat16 v[kCols][kTileRows + 2];
    // out[f * npad + row0 ..] for every column f; npad is a multiple of 128
    __device__ __forceinline__ void store_transposed(__nv_bfloat16* out, int npad, int row0) const {
        for (int e = threadIdx.x; e < kCols * (kTileRows / 8); e += blockDim.x) {
            const int f = e / (kTileRows / 8), r = (e % (kTileRows / 8)) * 8;
            uint4 w;
            uint32_t* p = reinterpret_cast<uint32_t*>(&w);
#pragma unroll
            for (int k = 0; k < 4; k++) p[k] = *reinterpret_cast<const uint32_t*>(&v[f][r + 2 * k]);
            *reinterpret_cast<uint4*>(out + (size_t)f * npad + row0 + r) = w;
        }
    }
};
// Sum over the block's rows of a thread's value for feature threadIdx.x % 64
// into out[feature], one atomic per feature
__device__ __forceinline__ void feature_sum(float s, float* out) {
    __shared__ float part[kTileThreads];
    part[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x < 64) {
        float sum = 0.0f;
#pragma unroll
        for (int k = 0; k < kTileThreads / 64; k++) sum += part[threadIdx.x + 64 * k];
        if (sum != 0.0f) atomicAdd(&out[threadIdx.x], sum);
    }
    __syncthreads();
}

// BF16 input block: features in columns 0..15, zeros to 128; also the
// transposed copy (column-major) for the weight gradient
// nDev (may be null): the graph's row count on the device, which caps n
__global__ void __launch_bounds__(kTileThreads) k_input_bf16(const float* X, int n, const int32_t* nDev, int npad,
                                                             __nv_bfloat16* Z, __nv_bfloat16* ZT) {
    __shared__ RowTile<kCat> tile;
    const int row0 = blockIdx.x * kTileRows;
    if (nDev && *nDev < n) n = *nDev;
    for (int e = threadIdx.x; e < kTileRows * kCat; e += kTileThreads) {
        const int r = e / kCat, f = e % kCat, i = row0 + r;
        const __nv_bfloat16 b = __float2bfloat16_rn((i < n && f < kFeat) ? X[(size_t)i * kFeat + f] : 0.0f);
        Z[(size_t)i * kCat + f] = b;
        tile.v[f][r] = b;
    }
    __syncthreads();
    tile.store_transposed(ZT, npad, row0);
}

// u = C + b; h = hPrev + relu(u) (hPrev may be null)
__global__ void k_bias_act(const float* C, const float* b, const float* hPrev, float* u, float* h, int npad) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= npad * kHid) return;
    const float v = C[t] + b[t % kHid];
    u[t] = v;
    h[t] = (hPrev ? hPrev[t] : 0.0f) + fmaxf(v, 0.0f);
}

// z = [h, A h] in BF16 (row-major and transposed)
__global__ void __launch_bounds__(kConcatThreads) k_message_concat(const float* h, const int32_t* ellCol,
                                                                   const float* ellW, int D, int n,
                                                                   const int32_t* nDev, int npad, __nv_bfloat16* Z,
                                                                   __nv_bfloat16* ZT) {
    __shared__ RowTile<kCat> tile;
    const int row0 = blockIdx.x * kTileRows;
    const int f = threadIdx.x % kHid;
    if (nDev && *nDev < n) n = *nDev;
    for (int r = threadIdx.x / kHid; r < kTileRows; r += kConcatThreads / kHid) {
        const int i = row0 + r;
        float hv = 0.0f, mv = 0.0f;
        if (i < n) {
            hv = h[(size_t)i * kHid + f];
            // four neighbours' loads in flight (D is a multiple of 4 or its
            // last ones are taken singly; a row ends at its first -1)
            int k = 0;
            bool more = true;
            for (; more && k + 4 <= D; k += 4) {
                int j[4];
                float w[4], v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    j[u] = ellCol[(size_t)i * D + k + u];
                    w[u] = ellW[(size_t)i * D + k + u];
                }
#pragma unroll
                for (int u = 0; u < 4; u++) v[u] = j[u] >= 0 ? h[(size_t)j[u] * kHid + f] : 0.0f;
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    more = more && j[u] >= 0;
                    if (more) mv = fmaf(w[u], v[u], mv);
                }
            }
            for (; more && k < D; k++) {
                const int j = ellCol[(size_t)i * D + k];
                if (j < 0) break;
                mv = fmaf(ellW[(size_t)i * D + k], h[(size_t)j * kHid + f], mv);
            }
        }
        const __nv_bfloat16 hb = __float2bfloat16_rn(hv), mbv = __float2bfloat16_rn(mv);
        Z[(size_t)i * kCat + f] = hb;
        Z[(size_t)i * kCat + kHid + f] = mbv;
        tile.v[f][r] = hb;
        tile.v[kHid + f][r] = mbv;
    }
    __syncthreads();
    tile.store_transposed(ZT, npad, row0);
}

__global__ void k_readout(const float* h, const float* w, const float* b, int n, const int32_t* nDev, float* y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (nDev && *nDev < n) n = *nDev;
    if (i >= n) return;
    float s = b[0];
    for (int f = 0; f < kHid; f++) s += h[(size_t)i * kHid + f] * w[f];
    y[i] = s;
}

// loss = sum (y - t)^2 / count over the nodes; dy = 2 (y - t) / count
__global__ void k_loss(const float* y, const float* tgt, int n, float invCount, float* dy, float* loss) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.0f;
    if (i < n) {
        const float e = y[i] - tgt[i];
        dy[i] = 2.0f * e * invCount;
        l = e * e * invCount;
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0 && l != 0.0f) atomicAdd(loss, l);
}

// gradients of the readout; dh = dy w (zero on padding rows)
__global__ void __launch_bounds__(kTileThreads) k_readout_back(const float* h, const float* dy, const float* w, int n,
                                                               float* gw, float* gb, float* dh) {
    const int row0 = blockIdx.x * kTileRows;
    const int f = threadIdx.x % kHid;
    float sw = 0.0f, sb = 0.0f;
    for (int r = threadIdx.x / kHid; r < kTileRows; r += kTileThreads / kHid) {
        const size_t t = (size_t)(row0 + r) * kHid + f;
        const float d = row0 + r < n ? dy[row0 + r] : 0.0f;
        dh[t] = d * w[f];
        if (d != 0.0f) sw += d * h[t];
        sb += d;
    }
    feature_sum(sw, gw);
    __shared__ float bias[kHid];  // every feature's thread has summed the same rows
    if (f == 0) bias[threadIdx.x / kHid] = sb;
    __syncthreads();
    if (threadIdx.x == 0) {
        float sum = 0.0f;
        for (int k = 0; k < kTileThreads / kHid; k++) sum += bias[k];
        if (sum != 0.0f) atomicAdd(gb, sum);
    }
}

// du = dh * [u > 0] (BF16, row-major and transposed); gb += sum du
__global__ void __launch_bounds__(kTileThreads) k_act_back(const float* dh, const float* u, int npad,
                                                           __nv_bfloat16* DU, __nv_bfloat16* DUT, float* gb) {
    __shared__ RowTile<kHid> tile;
    const int row0 = blockIdx.x * kTileRows;
    const int f = threadIdx.x % kHid;
    float s = 0.0f;
    for (int r = threadIdx.x / kHid; r < kTileRows; r += kTileThreads / kHid) {
        const size_t t = (size_t)(row0 + r) * kHid + f;
        const float d = u[t] > 0.0f ? dh[t] : 0.0f;
        const __nv_bfloat16 b = __float2bfloat16_rn(d);
        DU[t] = b;
        tile.v[f][r] = b;
        s += d;
    }
    feature_sum(s, gb);
    tile.store_transposed(DUT, npad, row0);
}

// dhPrev = dh + dz[:, :64]; the message half flows back along the edges:
// dhPrev[j] += a_ij dz[i, 64 + f]
__global__ void k_message_back(const float* dh, const float* dz, const int32_t* ellCol, const float* ellW, int D, int n,
                               int npad, float* dhPrev) {
    // four features a thread, added as one vector
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= npad * (kHid / 4)) return;
    const int i = t / (kHid / 4), f = (t % (kHid / 4)) * 4;
    const float4 a = *reinterpret_cast<const float4*>(dh + (size_t)i * kHid + f);
    const float4 z = *reinterpret_cast<const float4*>(dz + (size_t)i * kCat + f);
    atomicAdd(reinterpret_cast<float4*>(dhPrev + (size_t)i * kHid + f),
              make_float4(a.x + z.x, a.y + z.y, a.z + z.z, a.w + z.w));
    if (i >= n) return;
    const float4 d = *reinterpret_cast<const float4*>(dz + (size_t)i * kCat + kHid + f);
    if (d.x == 0.0f && d.y == 0.0f && d.z == 0.0f && d.w == 0.0f) return;
    for (int k = 0; k < D; k++) {
        const int j = ellCol[(size_t)i * D + k];
        if (j < 0) break;
        const float w = ellW[(size_t)i * D + k];
        atomicAdd(reinterpret_cast<float4*>(dhPrev + (size_t)j * kHid + f),
                  make_float4(w * d.x, w * d.y, w * d.z, w * d.w));
    }
}

// Adam on the FP32 parameters
__global__ void k_adam(float* p, const float* g, float* m1, float* m2, int count, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    const float gt = g[t];
    const float a = b1 * m1[t] + (1.0f - b1) * gt;
    const float v = b2 * m2[t] + (1.0f - b2) * gt * gt;
    m1[t] = a;
    m2[t] = v;
    p[t] -= lr * (a / c1) / (sqrtf(v / c2) + eps);
}

// BF16 copies of one layer's weights: W (in x out) and W^T (out x in)
__global__ void k_weights_bf16(const float* W, __nv_bfloat16* Wb, __nv_bfloat16* WTb) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= kCat * kHid) return;
    const int i = t / kHid, o = t % kHid;
    const __nv_bfloat16 b = __float2bfloat16_rn(W[t]);
    Wb[t] = b;
    WTb[(size_t)o * kCat + i] = b;
}

// phi += sigma y on the graph's cells (and on the recorded correction of the
// V rows, so that the next event recycles the whole correction)
__global__ void k_apply_prediction(DevMesh m, const int32_t* nodes, const int32_t* count, const float* y,
                                   const float* scale, float gain, const int32_t* slotOf, float* hist) {
    const int n = *count;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int g = nodes[t];
    const float d = gain * scale[0] * y[t];
    m.phi64[g] += (double)d;
    if (hist) {
        const int s = slotOf[g];
        if (s >= 0) hist[s] += d;
    }
}

// Damped Jacobi sweeps over the graph's cells after the prediction, every
// other cell held: phi_i += omega ((sum_j ceff_ij phi_j - q_i) / diag_i -
// phi_i) (computePotential's update, grid_3d.cpp:1317-1371).  One CTA: each
// sweep computes every cell's new value from the old ones, then writes them
// (the same result for any thread count).  The change joins the recorded
// correction of the cells' V slots when hist is given.  The graph has at
// most cap <= kRefineMax cells.
constexpr int kRefineMax = 4096;
__global__ void __launch_bounds__(1024) k_local_refine(DevMesh m, const int32_t* nodes, const int32_t* count,
                                                       int cap, int sweeps, float omega, const int32_t* slotOf,
                                                       float* hist) {
    extern __shared__ double refineShared[];  // start[cap], next[cap]
    double* start = refineShared;
    double* next = refineShared + cap;
    const int n = min(*count, cap);
    for (int t = threadIdx.x; t < n; t += blockDim.x) start[t] = m.phi64[nodes[t]];
    __syncthreads();
    for (int sw = 0; sw < sweeps; sw++) {
        for (int t = threadIdx.x; t < n; t += blockDim.x) {
            const int i = nodes[t];
            const double d = m.diag64[i];
            double sum = 0.0;
            for (int q = m.row_ptr[i]; q < m.row_ptr[i + 1]; q++) sum += m.ceff64[q] * m.phi64[m.col[q]];
            const double pi = m.phi64[i];
            next[t] = d > 0.0 ? pi + (double)omega * ((sum - m.q64[i]) / d - pi) : pi;
        }
        __syncthreads();
        for (int t = threadIdx.x; t < n; t += blockDim.x) m.phi64[nodes[t]] = next[t];
        __syncthreads();
    }
    if (hist)
        for (int t = threadIdx.x; t < n; t += blockDim.x) {
            const int sl = slotOf[nodes[t]];
            if (sl >= 0) hist[sl] += (float)(m.phi64[nodes[t]] - start[t]);
        }
}

// training target: (phi_final - phi_start) / sigma
__global__ void k_collect_target(DevMesh m, const int32_t* nodes, const int32_t* count, const double* phiStart,
                                 const float* scale, float* tgt) {
    const int n = *count;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    tgt[t] = (float)((m.phi64[nodes[t]] - phiStart[t]) / (double)scale[0]);
}

// A batch gathered from the samples: sample b of the batch is the rows
// table[b] .. of the sample store and the rows start[b] .. start[b + 1] of the
// batch (table: batch offsets, then batch + 1 starts), its ELL columns
// shifted by its start.  One warp per row.
__global__ void k_stage_batch(const int64_t* __restrict__ table, int batch, int D, const float* __restrict__ sX,
                              const float* __restrict__ sW, const int32_t* __restrict__ sCol,
                              const float* __restrict__ sT, float* bX, float* bW, int32_t* bCol, float* bT) {
    const int64_t* start = table + batch;
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= start[batch]) return;
    int lo = 0, hi = batch - 1;  // the last sample that starts at or before row i
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (start[mid] <= i) lo = mid;
        else hi = mid - 1;
    }
    const int64_t o = table[lo] + (i - start[lo]);
    const int shift = (int)start[lo];
    if (lane < kFeat) bX[i * kFeat + lane] = sX[o * kFeat + lane];
    for (int k = lane; k < D; k += 32) {
        const int c = sCol[o * D + k];
        bCol[i * D + k] = c >= 0 ? c + shift : c;
        bW[i * D + k] = sW[o * D + k];
    }
    if (lane == 0) bT[i] = sT[o];
}

inline unsigned nblk(long long n, int b = 256) { return (unsigned)((n + b - 1) / b); }

}  // namespace

bool gemm_shape_ok(int M, int N, int K) { return M > 0 && M % 128 == 0 && (N == 64 || N == 128) && K > 0 && K % 64 == 0; }

cudaError_t launch_gemm_bf16(const void* A, const void* B, float* C, int M, int N, int K, int* status,
                             cudaStream_t s) {
    static std::atomic<uint64_t> attrSet{0};
    cudaError_t e = once_per_device(attrSet, [] {
        cudaError_t r = cudaFuncSetAttribute(k_gemm_bf16<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem);
        if (r == cudaSuccess)
            r = cudaFuncSetAttribute(k_gemm_bf16<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem);
        if (r == cudaSuccess)
            r = cudaFuncSetAttribute(k_gemm_bf16_long, cudaFuncAttributeMaxDynamicSharedMemorySize, kLongSmem);
        return r;
    });
    if (e != cudaSuccess) return e;
    const auto* a = static_cast<const __nv_bfloat16*>(A);
    const auto* b = static_cast<const __nv_bfloat16*>(B);
    count_launch();
    // a K of more chunks than the ring holds, on few row tiles: the ring pays
    if (K / 64 > kLongStages * kLongSub && M / 128 <= 8) {
        CUtensorMap mapA, mapB;
        if ((e = bf16_map(&mapA, A, M, K, 128)) != cudaSuccess) return e;
        if ((e = bf16_map(&mapB, B, N, K, kLongN)) != cudaSuccess) return e;
        k_gemm_bf16_long<<<dim3(M / 128, N / kLongN), kGemmThreads, kLongSmem, s>>>(mapA, mapB, C, N, K, status);
    } else if (N == 64)
        k_gemm_bf16<64><<<M / 128, kGemmThreads, kGemmSmem, s>>>(a, b, C, M, K, status);
    else
        k_gemm_bf16<128><<<M / 128, kGemmThreads, kGemmSmem, s>>>(a, b, C, M, K, status);
    return cudaGetLastError();
}

void launch_ball_bfs(const DevMesh& m, int site, int hops, int cap, int32_t* nodes, int8_t* level, int32_t* count,
                     int32_t* localOf, cudaStream_t s) {
    count_launch();
    k_ball_bfs<<<1, 512, 0, s>>>(m, site, hops, cap, nodes, level, count, localOf);
}
void launch_ball_reset(const int32_t* nodes, const int32_t* count, int32_t* localOf, int cap, cudaStream_t s) {
    count_launch();
    k_ball_reset<<<nblk(cap), 256, 0, s>>>(nodes, count, localOf);
}
void launch_ball_features(const DevMesh& m, int site, int hops, int D, const int32_t* nodes, const int8_t* level,
                          const int32_t* count, const int32_t* localOf, float* scale, float* X, int32_t* ellCol,
                          float* ellW, double* phiStart, int cap, cudaStream_t s) {
    count_launch();
    k_site_scale<<<1, 32, 0, s>>>(m, site, scale);
    count_launch();
    k_ball_features<<<nblk((long long)cap * 32), 256, 0, s>>>(m, site, hops, D, nodes, level, count, localOf, scale, X,
                                                               ellCol, ellW,
                                               phiStart);
}
void launch_input_bf16(const float* X, int n, int npad, void* Z, void* ZT, cudaStream_t s, const int32_t* nDev) {
    count_launch();
    k_input_bf16<<<npad / kTileRows, kTileThreads, 0, s>>>(X, n, nDev, npad, static_cast<__nv_bfloat16*>(Z),
                                                            static_cast<__nv_bfloat16*>(ZT));
}
void launch_bias_act(const float* C, const float* b, const float* hPrev, float* u, float* h, int npad,
                     cudaStream_t s) {
    count_launch();
    k_bias_act<<<nblk((long long)npad * kHid), 256, 0, s>>>(C, b, hPrev, u, h, npad);
}
void launch_message_concat(const float* h, const int32_t* ellCol, const float* ellW, int D, int n, int npad, void* Z,
                           void* ZT, cudaStream_t s, const int32_t* nDev) {
    count_launch();
    k_message_concat<<<npad / kTileRows, kConcatThreads, 0, s>>>(h, ellCol, ellW, D, n, nDev, npad,
                                                                static_cast<__nv_bfloat16*>(Z),
                                                                static_cast<__nv_bfloat16*>(ZT));
}
void launch_readout(const float* h, const float* w, const float* b, int n, float* y, cudaStream_t s,
                    const int32_t* nDev) {
    count_launch();
    k_readout<<<nblk(n), 256, 0, s>>>(h, w, b, n, nDev, y);
}
void launch_loss(const float* y, const float* tgt, int n, float invCount, float* dy, float* loss, cudaStream_t s) {
    count_launch();
    k_loss<<<nblk(n), 256, 0, s>>>(y, tgt, n, invCount, dy, loss);
}
void launch_readout_back(const float* h, const float* dy, const float* w, int n, int npad, float* gw, float* gb,
                         float* dh, cudaStream_t s) {
    count_launch();
    k_readout_back<<<npad / kTileRows, kTileThreads, 0, s>>>(h, dy, w, n, gw, gb, dh);
}
void launch_act_back(const float* dh, const float* u, int npad, void* DU, void* DUT, float* gb, cudaStream_t s) {
    count_launch();
    k_act_back<<<npad / kTileRows, kTileThreads, 0, s>>>(dh, u, npad, static_cast<__nv_bfloat16*>(DU),
                                                          static_cast<__nv_bfloat16*>(DUT), gb);
}
void launch_message_back(const float* dh, const float* dz, const int32_t* ellCol, const float* ellW, int D, int n,
                         int npad, float* dhPrev, cudaStream_t s) {
    count_launch();
    k_message_back<<<nblk((long long)npad * (kHid / 4)), 256, 0, s>>>(dh, dz, ellCol, ellW, D, n, npad, dhPrev);
}
void launch_adam(float* p, const float* g, float* m1, float* m2, int count, float lr, float b1, float b2, float eps,
                 float c1, float c2, cudaStream_t s) {
    count_launch();
    k_adam<<<nblk(count), 256, 0, s>>>(p, g, m1, m2, count, lr, b1, b2, eps, c1, c2);
}
void launch_weights_bf16(const float* W, void* Wb, void* WTb, cudaStream_t s) {
    count_launch();
    k_weights_bf16<<<nblk(kCat * kHid), 256, 0, s>>>(W, static_cast<__nv_bfloat16*>(Wb),
                                                     static_cast<__nv_bfloat16*>(WTb));
}
void launch_apply_prediction(const DevMesh& m, const int32_t* nodes, const int32_t* count, const float* y,
                             const float* scale, float gain, const int32_t* slotOf, float* hist, int cap,
                             cudaStream_t s) {
    count_launch();
    k_apply_prediction<<<nblk(cap), 256, 0, s>>>(m, nodes, count, y, scale, gain, slotOf, hist);
}
void launch_local_refine(const DevMesh& m, const int32_t* nodes, const int32_t* count, int cap, int sweeps,
                         float omega, const int32_t* slotOf, float* hist, cudaStream_t s) {
    if (sweeps <= 0 || cap <= 0 || cap > kRefineMax) return;
    static std::atomic<uint64_t> opted{0};
    once_per_device(opted, [] {
        return cudaFuncSetAttribute(k_local_refine, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(2 * sizeof(double) * kRefineMax));
    });
    count_launch();
    k_local_refine<<<1, 1024, 2 * sizeof(double) * (size_t)cap, s>>>(m, nodes, count, cap, sweeps, omega, slotOf,
                                                                     hist);
}
void launch_collect_target(const DevMesh& m, const int32_t* nodes, const int32_t* count, const double* phiStart,
                           const float* scale, float* tgt, int cap, cudaStream_t s) {
    count_launch();
    k_collect_target<<<nblk(cap), 256, 0, s>>>(m, nodes, count, phiStart, scale, tgt);
}
void launch_stage_batch(const int64_t* table, int batch, int rows, int D, const float* sX, const float* sW,
                        const int32_t* sCol, const float* sT, float* bX, float* bW, int32_t* bCol, float* bT,
                        cudaStream_t s) {
    if (rows <= 0) return;
    count_launch();
    k_stage_batch<<<nblk((long long)rows * 32), 256, 0, s>>>(table, batch, D, sX, sW, sCol, sT, bX, bW, bCol, bT);
}

}  // namespace tgd
