// Dense row-major linear for 16-bit weights on the tensor cores (tcgen05, sm_100a), at size:
//
//   out[r, o] = cast( sum_k x[r, k] * w[o, k] )        x [rows, k], w [out, k] (both k-inner), bf16 or f16, f32 sums
//
// What bounds it: with up to a few hundred rows the weights' bytes (each is used once per row), from there on the tensor
// pipe. The WEIGHT rows are the M = 128 side of the MMA and the activation rows the N side (16..256 columns, as many as the
// call has), so that a handful of rows wastes no tensor work on padding and every weight byte is loaded once per 256 rows.
// A tile is 128 outputs x BN rows; 14336 outputs are 112 tiles and 4096 only 32, so the k range of a tile is split over a
// thread-block cluster of up to 8 CTAs (whatever brings the grid to about two CTAs per SM), each leaves its f32 partial tile
// in its own shared memory and the cluster adds them in rank order over distributed shared memory (deterministic, no
// workspace, no second launch). Per CTA: one TMA warp (128-byte swizzled boxes, 64 k a stage), one MMA warp, four epilogue
// warps. Two CTAs share an SM up to 32 rows (about 100 KB of weight loads in flight each).
// Measured (one B200, ncu, cold caches): 16 rows, 14336 x 4096 bf16: the one-thread-per-output kernel of ref_ops.cu, whose
// neighbouring lanes read weights a row apart, took 3528 us; this one 27 us (4.4 TB/s, 0.67 of the measured copy peak); the
// 14336 -> 4096 projection, 32 tiles x 8 parts: 3564 -> 26 us.
//
// The products of 16-bit operands are exact in f32; the sums run in another order than the reference's (sequential k), so
// results agree with it within f32 rounding before the cast. Small shapes stay on the reference-order kernel, and the
// payload records which of the two a program got.
//
// Every wait is bounded; on expiry a status word is raised, the CTA waits for what it has started and frees its TMEM. No multicast.
//
// Replaces, at size, the generated kernel of vyre-libs/src/nn/linear/inner/linear_rows.rs (typed, [out, in] weights).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <atomic>

#include "kernels.h"
#include "tcgen05_common.cuh"

namespace vybk {
namespace {

using namespace tc;

constexpr int BM = 128, BK = 64, UMMA_K = 16;
constexpr int MAX_BN = 256, MAX_STAGES = 8, MAX_SPLIT = 8;
constexpr int A_BYTES = BM * BK * 2;
constexpr int THREADS = 192;  // TMA, MMA, 4 epilogue warps
constexpr int CTRL_BYTES = 256, ALIGN_SLACK = 1024;
constexpr int HALF_SM = 112 * 1024, FULL_SM = 224 * 1024;

struct Bars {
    unsigned long long full[MAX_STAGES], empty[MAX_STAGES], acc_full, drained;
    uint32_t tmem_base;
    unsigned int abort_flag;
    uint32_t issued;  // copies of the TMA role
};

struct Params {
    void* out;
    uint32_t* status;
    uint32_t rows, n, k;
    uint32_t bn;      // activation rows per tile: a multiple of 16
    uint32_t split;   // CTAs of the cluster that share a tile
    uint32_t stages, tmem_cols;
    uint32_t f16;
};

// grid: x = weight tiles * split (a cluster spans the k parts of one tile), y = tiles of bn rows
__global__ void __launch_bounds__(THREADS, 2)
dense_rows_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Params p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t b_bytes = p.bn * BK * 2, stage_bytes = A_BYTES + b_bytes;
    Bars* bars = reinterpret_cast<Bars*>(tiles + p.stages * stage_bytes);
    volatile unsigned int* abort_flag = &bars->abort_flag;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t part = blockIdx.x % p.split, n0 = (blockIdx.x / p.split) * BM, r0 = blockIdx.y * p.bn;
    const uint32_t k_blocks = (p.k + BK - 1) / BK;
    // this CTA's run of k blocks; the first k_blocks % split parts take one more
    const uint32_t base = k_blocks / p.split, rem = k_blocks % p.split;
    const uint32_t kb0 = part * base + min(part, rem), kbs = base + (part < rem ? 1u : 0u);

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(&bars->full[s]), 1);
            mbar_init(smem_u32(&bars->empty[s]), 1);
        }
        mbar_init(smem_u32(&bars->acc_full), 1);
        mbar_init(smem_u32(&bars->drained), 1);
        bars->abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&map_w);
        tma_prefetch_desc(&map_x);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&bars->tmem_base), p.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;

    bool ok = true;
    if (warp == 0) {
        if (elect_one()) {
            uint32_t i = 0;
            for (; i < kbs; ++i) {
                const uint32_t s = i % p.stages, bar = smem_u32(&bars->full[s]), dst = smem_u32(tiles + s * stage_bytes);
                if (i >= p.stages && !mbar_wait(smem_u32(&bars->empty[s]), ((i / p.stages) - 1) & 1, abort_flag)) break;
                mbar_arrive_expect_tx(bar, stage_bytes);
                tma_load_2d(dst, &map_w, int((kb0 + i) * BK), int(n0), bar);
                tma_load_2d(dst + A_BYTES, &map_x, int((kb0 + i) * BK), int(r0), bar);
            }
            bars->issued = i;
        }
        __syncwarp();
    } else if (warp == 1) {
        // M = 128 weight rows, N = bn activation rows; c f32, a / b both bf16 or both f16
        const uint32_t idesc = (1u << 4) | (p.f16 ? 0u : (1u << 7) | (1u << 10)) | ((p.bn >> 3) << 17) | (uint32_t(BM >> 4) << 24);
        if (elect_one()) {
            for (uint32_t i = 0; i < kbs; ++i) {
                const uint32_t s = i % p.stages, src = smem_u32(tiles + s * stage_bytes);
                if (!mbar_wait(smem_u32(&bars->full[s]), (i / p.stages) & 1, abort_flag)) break;
                tc_fence_after();
                const uint64_t da = smem_desc_sw128(src), db = smem_desc_sw128(src + A_BYTES);
#pragma unroll
                for (int k = 0; k < BK / UMMA_K; ++k)
                    mma_f16(tmem, smem_desc_advance(da, k * UMMA_K * 2), smem_desc_advance(db, k * UMMA_K * 2), idesc, (i | uint32_t(k)) != 0);
                tc_commit(smem_u32(&bars->empty[s]));
                if (i + 1 == kbs) tc_commit(smem_u32(&bars->acc_full));
            }
            if (*abort_flag != 0) settle_mma(smem_u32(&bars->drained));
        }
        __syncwarp();
    }
    auto store = [&](uint32_t row, uint32_t col, float v) {
        // the reference flushes subnormal f32 results before it rounds to the storage type
        v = fabsf(v) < 1.17549435e-38f ? copysignf(0.0f, v) : v;
        const size_t at = size_t(row) * p.n + col;
        if (p.f16) static_cast<__half*>(p.out)[at] = __float2half_rn(v);
        else static_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16_rn(v);
    };
    float* partial = reinterpret_cast<float*>(tiles);  // [bn][128]; the stages are free once the last MMA has completed
    if (warp >= 2) {
        ok = mbar_wait(smem_u32(&bars->acc_full), 0, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            tc_fence_after();
            const uint32_t quad = warp & 3, o = quad * 32 + lane;  // TMEM lane = weight row of the tile
            const uint32_t taddr = tmem + ((quad * 32) << 16);
            for (uint32_t c = 0; c < p.bn; c += 16) {
                uint32_t r[16];
                tmem_ld_32x16(taddr + c, r);
                tmem_ld_wait();
                if (p.split == 1) {
#pragma unroll
                    for (uint32_t j = 0; j < 16; ++j)
                        if (r0 + c + j < p.rows && n0 + o < p.n) store(r0 + c + j, n0 + o, __uint_as_float(r[j]));
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < 16; ++j) partial[(c + j) * BM + o] = __uint_as_float(r[j]);
                }
            }
        }
    }
    tc_fence_before();
    if (p.split > 1) {
        cluster_sync();  // every part's partial tile is in its shared memory
        // rank r adds the columns c % split == r, in rank order; neighbouring threads take neighbouring outputs
        for (uint32_t idx = threadIdx.x; idx < ((p.bn + p.split - 1 - part) / p.split) * BM; idx += THREADS) {
            const uint32_t c = (idx / BM) * p.split + part, o = idx % BM;
            if (r0 + c >= p.rows || n0 + o >= p.n) continue;
            const uint32_t addr = smem_u32(partial + c * BM + o);
            float v[MAX_SPLIT];
#pragma unroll
            for (uint32_t q = 0; q < MAX_SPLIT; ++q)
                if (q < p.split) v[q] = ld_cluster_f32(mapa(addr, q));
            float sum = v[0];
#pragma unroll
            for (uint32_t q = 1; q < MAX_SPLIT; ++q)
                if (q < p.split) sum += v[q];
            store(r0 + c, n0 + o, sum);
        }
        cluster_sync();  // no CTA leaves while another still reads its shared memory
    } else {
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, p.tmem_cols);
    }
    if (threadIdx.x == 0 && bars->abort_flag != 0) {
        settle_copies(bars->full, p.stages, bars->issued);
        if (p.status) atomicOr(p.status, 32u);
    }
}

}  // namespace

// The target compiler chooses this kernel from the op spec (variant 10, at most 65535 row tiles). Tensor-map strides are multiples of
// 16 bytes and bases 16-byte aligned, which resident and temporary buffers of the contract always are.
bool dense_rows_supported(const void* x, const void* w, uint32_t in_dim) {
    return in_dim % 8 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15u) == 0;
}

cudaError_t launch_dense_rows(const void* x, const void* w, void* out, uint32_t rows, uint32_t in_dim, uint32_t out_dim, bool f16,
                              int sm_count, cudaStream_t stream, uint32_t* status) {
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        e = cudaFuncSetAttribute(dense_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FULL_SM);
        if (e != cudaSuccess) return e;
        configured.fetch_or(bit, std::memory_order_release);
    }
    Params p = {};
    p.out = out;
    p.status = status;
    p.rows = rows;
    p.n = out_dim;
    p.k = in_dim;
    p.f16 = f16 ? 1u : 0u;
    const uint32_t row_tiles = (rows + MAX_BN - 1) / MAX_BN;
    p.bn = ((rows + row_tiles - 1) / row_tiles + 15) / 16 * 16;
    const uint32_t stage_bytes = A_BYTES + p.bn * BK * 2;
    const uint32_t budget = p.bn <= 32 ? HALF_SM : FULL_SM, fixed = ALIGN_SLACK + CTRL_BYTES;
    p.stages = (budget - fixed) / stage_bytes;
    if (p.stages > uint32_t(MAX_STAGES)) p.stages = MAX_STAGES;
    p.tmem_cols = 32;
    while (p.tmem_cols < p.bn) p.tmem_cols *= 2;
    const uint32_t n_tiles = (out_dim + BM - 1) / BM, k_blocks = (in_dim + BK - 1) / BK;
    // two CTAs per SM when they fit, at least four k blocks each
    const uint32_t slots = uint32_t(sm_count) * (p.bn <= 32 ? 2u : 1u), tiles = n_tiles * row_tiles;
    p.split = slots / tiles;
    if (p.split > k_blocks / 4) p.split = k_blocks / 4;
    if (p.split > uint32_t(MAX_SPLIT)) p.split = MAX_SPLIT;
    if (p.split < 1) p.split = 1;
    CUtensorMap mw, mx;
    if (!encode_tensor_map_2d(&mw, w, out_dim, in_dim, 2, BM, BK, true) || !encode_tensor_map_2d(&mx, x, rows, in_dim, 2, p.bn, BK, true))
        return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_tiles * p.split, row_tiles);
    cfg.blockDim = dim3(THREADS);
    // the partial tile (bn x 512 bytes) reuses the stages: at four stages and more they always hold it
    cfg.dynamicSmemBytes = p.stages * stage_bytes + fixed;
    cfg.stream = stream;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = p.split;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, dense_rows_kernel, mw, mx, p);
}

}  // namespace vybk
