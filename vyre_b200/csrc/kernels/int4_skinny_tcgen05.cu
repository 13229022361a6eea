// Group-quantized int4 linear for up to 64 activation rows on the tensor cores (tcgen05, sm_100a), weights exact:
//
//   y[m, n] = cast( sum_g s[n, g] * sum_{k in g} x[m, k] * (q[n, k] - 8) )        group 128
//
// What bounds it: the packed weights' bytes (each is read once for all rows) and, close behind, the instructions that turn
// nibbles into tensor-core operands. So the WEIGHT rows are the M = 128 side of the MMA and the activation rows its N side
// (16, 48 or 64 columns), and the unpacked weights never touch shared memory: a thread owns a weight row, reads 64 packed
// bytes (one group), makes 64 registers of bf16 pairs (q - 8 is exact in bf16; thirteen instructions per eight weights, in
// natural k order, so that the activations are TMA boxes of x as it lies in memory) and stores them to TENSOR MEMORY, which
// the MMA reads as its A operand. Through shared memory the same bytes would be written and read once more, 4 bytes per
// weight at 128 bytes a cycle, 6 us at 14336 x 4096 against 4.6 us of HBM time.
//
// bf16 x bf16 products are exact in f32; every 128-k group gets an accumulator of its own (two alternate), and the epilogue
// warps add s * group sum in f32 registers while the next group's MMAs run. Weights are not rounded (the prefill kernel
// rounds (q - 8) * s to bf16), activations are not converted.
//
// Per CTA: warp 0 TMA (256 k a stage: 128 x 128 packed bytes, 4 boxes of x), warp 1 MMA, warps 4-7 / 8-11 unpack the first /
// second group of a stage, warps 12-15 epilogue. Up to 16 rows two CTAs share an SM (each holds less than half of its shared
// memory, and half of its registers and tensor memory), so that under programmatic dependent launch the next launch's CTA already streams
// its weights while this one drains. Few weight tiles: the k range of a tile is split over a cluster, the partial sums are
// added in rank order over distributed shared memory (deterministic, no workspace).
//
// f32 outputs run here only where the kernel they had sums in f32 as well (beyond eight rows of 2048 and 4096 k); the others keep the
// integer kernels, whose group sums are exact (launch_int4_gemv). Next to the rounding to bf16 the difference does not show (relative
// error 1.65e-3 on both).
//
// Measured (64-launch graphs over rotating weights): 14336 x 4096 at 48 rows 15.1 us (six launches of the 8-row kernel: 91 us),
// at 64 rows 17.2 us, at 16 rows 14.4 us; 4096 x 14336 at 8 rows 13.7 us (two launches of the four-row k-block form: 26.6 us).
// At 3 to 8 rows of 4096 k the 8-row kernel (10.8 us) is the faster one and stays.
//
// Every wait is bounded; on expiry a status word is raised, the CTA waits for what it has started and frees its TMEM. No multicast.
//
// Replaces the generated scalar kernel of vyre-libs/src/nn/linear/inner/linear_4bit.rs:399-775 for the row-major layout of
// vyre-primitives/src/math/quantized/programs.rs:186-300 at decode batches.
#include <cuda_bf16.h>

#include <atomic>

#include "dependent_launch.cuh"
#include "kernels.h"
#include "tcgen05_common.cuh"

namespace vybk {
namespace {

using namespace tc;

constexpr int BM = 128, UMMA_K = 16, GROUP = 128;
constexpr int KB = 256;                  // k per stage: two groups
constexpr int RAW_BYTES = BM * KB / 2;   // 16 KB
constexpr int MAX_SPLIT = 8;
constexpr int THREADS = 512;
constexpr int CTRL_BYTES = 512, ALIGN_SLACK = 1024;

template <int BN>
struct Cfg {
    static constexpr int B_BYTES = BN * KB * 2;
    static constexpr int STAGE_BYTES = RAW_BYTES + B_BYTES;
    static constexpr bool HALF = BN <= 16;  // two CTAs per SM
    static constexpr int STAGES = BN == 48 ? 5 : 4;
    // Groups that one pass of the MMA loop takes (its waits and commits cost more than its MMAs): both of a stage where a CTA has
    // all of an SM's tensor memory (64 rows: 14336 x 4096 19.1 -> 17.2 us, 4096 x 14336 21.8 -> 16.0, 28672 x 8192 85 -> 58). A_SLOTS passes' unpacked weights and two passes' accumulators are held.
    static constexpr int PASS = HALF ? 1 : 2;
    static constexpr int A_SLOTS = HALF ? 3 : 2;
    static constexpr int TMEM_COLS = HALF ? 256 : 512;
    static constexpr int A_COL = 2 * PASS * BN;   // the accumulators come first
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + CTRL_BYTES + ALIGN_SLACK;
    static_assert(A_COL + A_SLOTS * PASS * 64 <= TMEM_COLS, "tensor memory");
    static_assert(SMEM_BYTES <= (HALF ? 113 * 1024 : 227 * 1024), "shared memory");
    static_assert(BN * BM * 4 <= STAGES * STAGE_BYTES, "the partial tile reuses the stages");
};

struct Bars {
    unsigned long long full[8], empty[8], a_full[4], a_empty[4], d_full[2], d_empty[2], drained;
    uint32_t tmem_base;
    unsigned int abort_flag;
    uint32_t issued;  // copies of the TMA role
};
static_assert(sizeof(Bars) <= CTRL_BYTES, "control block");

struct Params {
    const uint16_t* scales;  // bf16 [n][k / 128]
    void* y;
    uint32_t* status;
    uint32_t m, n, k, split;
    uint32_t tile0;          // first weight tile of this launch
    uint32_t constant;       // weights and scales may be read before the launches before this one are complete
    uint32_t early;          // the next launch may start beside this one
};

template <int BN, bool OUT_F32>
__global__ void __launch_bounds__(THREADS, Cfg<BN>::HALF ? 2 : 1)
int4_skinny_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Params p) {
    using C = Cfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    Bars* bars = reinterpret_cast<Bars*>(tiles + C::STAGES * C::STAGE_BYTES);
    volatile unsigned int* abort_flag = &bars->abort_flag;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t part = blockIdx.x % p.split, n0 = (p.tile0 + blockIdx.x / p.split) * BM;
    const uint32_t blocks = p.k / KB, base = blocks / p.split, rem = blocks % p.split;
    auto store = [&](size_t at, float v) {
        if constexpr (OUT_F32) static_cast<float*>(p.y)[at] = v;
        else static_cast<__nv_bfloat16*>(p.y)[at] = __float2bfloat16_rn(v);
    };
    const uint32_t kb0 = part * base + min(part, rem), kbs = base + (part < rem ? 1u : 0u);

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(smem_u32(&bars->full[s]), 1);
            mbar_init(smem_u32(&bars->empty[s]), 9);  // eight unpack warps and the MMAs
        }
        for (int s = 0; s < C::A_SLOTS; ++s) {
            mbar_init(smem_u32(&bars->a_full[s]), 4 * C::PASS);
            mbar_init(smem_u32(&bars->a_empty[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(smem_u32(&bars->d_full[s]), 1);
            mbar_init(smem_u32(&bars->d_empty[s]), 4);
        }
        mbar_init(smem_u32(&bars->drained), 1);
        bars->abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&map_w);
        tma_prefetch_desc(&map_x);
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&bars->tmem_base), C::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    // only now, with this CTA's tensor memory in hand, may the next launch's CTA take the rest of it
    if (p.early) lets_next_start();
    // Before any wait with a limit: the time that the launches before this one still take is not this one's. Only constant weights (warp 0) and
    // scales (from warp 12 on) are read before.
    if (warp != 0 && !(p.constant && warp >= 12)) waits_for_previous();

    bool ok = true;
    if (warp == 0) {
        // ---- TMA: weights are constants and are fetched before the previous launch is known to be complete, x is not ----
        auto load_raw = [&](uint32_t i) {
            const uint32_t s = i % C::STAGES, bar = smem_u32(&bars->full[s]);
            mbar_arrive_expect_tx(bar, C::STAGE_BYTES);
            tma_load_2d(smem_u32(tiles + s * C::STAGE_BYTES), &map_w, int((kb0 + i) * (KB / 2)), int(n0), bar);
        };
        auto load_x = [&](uint32_t i) {
            const uint32_t s = i % C::STAGES, bar = smem_u32(&bars->full[s]);
            const uint32_t dst = smem_u32(tiles + s * C::STAGE_BYTES + RAW_BYTES);
#pragma unroll
            for (int j = 0; j < KB / 64; ++j) tma_load_2d(dst + j * BN * 128, &map_x, int((kb0 + i) * KB + j * 64), 0, bar);
        };
        const uint32_t ahead = min(kbs, uint32_t(C::STAGES));
        if (elect_one()) {
            if (!p.constant) {
                for (uint32_t i = 0; i < ahead; ++i) tma_prefetch_2d(&map_w, int((kb0 + i) * (KB / 2)), int(n0));
                waits_for_previous();
            }
            for (uint32_t i = 0; i < ahead; ++i) load_raw(i);
            waits_for_previous();
            for (uint32_t i = 0; i < ahead; ++i) load_x(i);
            uint32_t i = ahead;
            for (; i < kbs; ++i) {
                if (!mbar_wait(smem_u32(&bars->empty[i % C::STAGES]), ((i / C::STAGES) - 1) & 1, abort_flag)) break;
                load_raw(i);
                load_x(i);
            }
            bars->issued = i;
        }
        __syncwarp();
    } else if (warp == 1) {
        // ---- MMA: eight k steps per group, D of its own per group ----
        constexpr uint32_t idesc = idesc_bf16_f32(BM, BN);
        if (elect_one()) {
            uint32_t s = 0, slot = 0, a_parity = 0;
            for (uint32_t it = 0; it < 2 / C::PASS * kbs; ++it) {
                const uint32_t set = it & 1;
                // the unpack warps saw the whole stage land before they arrived here: no wait of its own for x
                if (!(it < 2 ? mbar_wait(smem_u32(&bars->a_full[slot]), a_parity, abort_flag)
                             : mbar_wait2(smem_u32(&bars->a_full[slot]), a_parity, smem_u32(&bars->d_empty[set]), ((it >> 1) - 1) & 1, abort_flag))) break;
                tc_fence_after();
#pragma unroll
                for (int h = 0; h < C::PASS; ++h) {
                    const uint32_t half = C::PASS == 2 ? uint32_t(h) : set;  // which group of the stage
                    const uint32_t b = smem_u32(tiles + s * C::STAGE_BYTES + RAW_BYTES) + half * 2 * BN * 128;
                    const uint64_t db0 = smem_desc_sw128(b), db1 = smem_desc_sw128(b + BN * 128);
#pragma unroll
                    for (int k = 0; k < GROUP / UMMA_K; ++k)
                        mma_f16_ts(tmem + (set * C::PASS + h) * BN, tmem + C::A_COL + (slot * C::PASS + h) * 64 + k * (UMMA_K / 2),
                                   smem_desc_advance(k < 4 ? db0 : db1, (k & 3) * UMMA_K * 2), idesc, k != 0);
                }
                tc_commit(smem_u32(&bars->a_empty[slot]));
                tc_commit(smem_u32(&bars->d_full[set]));
                if (C::PASS == 2 || set == 1) {
                    tc_commit(smem_u32(&bars->empty[s]));
                    s = s + 1 == uint32_t(C::STAGES) ? 0u : s + 1;
                }
                if (++slot == uint32_t(C::A_SLOTS)) {
                    slot = 0;
                    a_parity ^= 1;
                }
            }
            if (*abort_flag != 0) settle_mma(smem_u32(&bars->drained));
        }
        __syncwarp();
    } else if (warp >= 4 && warp < 12) {
        // ---- unpack: a thread per weight row; warps 4-7 the even groups, 8-11 the odd ones ----
        const uint32_t half = (warp >> 2) - 1, quad = warp & 3, r = quad * 32 + lane;
        for (uint32_t i = 0; i < kbs && ok; ++i) {
            const uint32_t s = i % C::STAGES, it = C::PASS == 2 ? i : 2 * i + half, slot = it % C::A_SLOTS;
            ok = mbar_wait(smem_u32(&bars->full[s]), (i / C::STAGES) & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const uint8_t* row = tiles + s * C::STAGE_BYTES + r * 128;
            uint4 raw[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) raw[j] = *reinterpret_cast<const uint4*>(row + (((half * 4 + j) ^ (r & 7u)) << 4));
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->empty[s]));  // the packed bytes are in registers
            if (it >= uint32_t(C::A_SLOTS)) ok = mbar_wait(smem_u32(&bars->a_empty[slot]), ((it / C::A_SLOTS) - 1) & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t dst = tmem + ((quad * 32) << 16) + C::A_COL + (slot * C::PASS + (C::PASS == 2 ? half : 0)) * 64;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t a[32];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const uint32_t words[4] = {raw[2 * h + j].x, raw[2 * h + j].y, raw[2 * h + j].z, raw[2 * h + j].w};
#pragma unroll
                    for (int u = 0; u < 4; ++u) unpack_int4_bf16(words[u], &a[16 * j + 4 * u]);
                }
                tmem_st_32x32(dst + h * 32, a);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->a_full[slot]));
        }
    } else if (warp >= 12) {
        // ---- epilogue: acc += scale * group sum ----
        const uint32_t quad = warp & 3, o = quad * 32 + lane, row = n0 + o;
        const uint32_t groups = p.k / GROUP;
        const uint32_t* sp = reinterpret_cast<const uint32_t*>(p.scales + size_t(min(row, p.n - 1)) * groups) + kb0;  // a pair per stage
        float acc[BN];
#pragma unroll
        for (int c = 0; c < BN; ++c) acc[c] = 0.0f;
        constexpr uint32_t AHEAD = 4;  // scale pairs in flight: an L2 round trip is several stages long
        uint32_t queue[AHEAD];
#pragma unroll
        for (uint32_t d = 0; d < AHEAD; ++d) queue[d] = d < kbs ? sp[d] : 0u;
        waits_for_previous();
        for (uint32_t i0 = 0; i0 < kbs && ok; i0 += AHEAD) {
#pragma unroll
            for (uint32_t d = 0; d < AHEAD; ++d) {
                const uint32_t i = i0 + d;
                if (i >= kbs || !ok) break;
                const uint32_t pair = queue[d];
                if (i + AHEAD < kbs) queue[d] = sp[i + AHEAD];
#pragma unroll
                for (uint32_t buf = 0; buf < 2; ++buf) {
                    // PASS = 1: one accumulator per group, set = group parity; PASS = 2: both groups' accumulators, set = stage parity
                    const uint32_t set = C::PASS == 2 ? i & 1 : buf;
                    if (C::PASS == 1 || buf == 0) {
                        ok = ok && mbar_wait(smem_u32(&bars->d_full[set]), (C::PASS == 2 ? i >> 1 : i) & 1, abort_flag);
                        ok = __all_sync(0xffffffffu, ok);
                        if (!ok) break;
                        tc_fence_after();
                    }
                    const float s = __uint_as_float(buf ? pair & 0xFFFF0000u : pair << 16);
                    uint32_t v[BN / 16][16];
#pragma unroll
                    for (int c = 0; c < BN / 16; ++c)
                        tmem_ld_32x16(tmem + ((quad * 32) << 16) + (C::PASS == 2 ? set * 2 + buf : set) * BN + c * 16, v[c]);
                    tmem_ld_wait();
                    if (C::PASS == 1 || buf == 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(smem_u32(&bars->d_empty[set]));
                    }
#pragma unroll
                    for (int c = 0; c < BN; ++c) acc[c] = fmaf(s, __uint_as_float(v[c / 16][c % 16]), acc[c]);
                }
            }
        }
        if (ok) {
            if (p.split == 1) {
#pragma unroll
                for (int c = 0; c < BN; ++c)
                    if (uint32_t(c) < p.m && row < p.n) store(size_t(c) * p.n + row, acc[c]);
            } else {
                // the last group sum is complete, so every load and MMA of this CTA is: the stages are free
                float* partial = reinterpret_cast<float*>(tiles);  // [BN][128]
#pragma unroll
                for (int c = 0; c < BN; ++c) partial[c * BM + o] = acc[c];
            }
        }
    }
    tc_fence_before();
    if (p.split > 1) {
        cluster_sync();  // every part's partial tile is in its shared memory
        for (uint32_t idx = threadIdx.x; idx < ((BN + p.split - 1 - part) / p.split) * BM; idx += THREADS) {
            const uint32_t c = (idx / BM) * p.split + part, o = idx % BM;
            if (c >= p.m || n0 + o >= p.n) continue;
            const uint32_t addr = smem_u32(reinterpret_cast<float*>(tiles) + c * BM + o);
            float v[MAX_SPLIT];
#pragma unroll
            for (uint32_t q = 0; q < MAX_SPLIT; ++q)
                if (q < p.split) v[q] = ld_cluster_f32(mapa(addr, q));
            float sum = v[0];
#pragma unroll
            for (uint32_t q = 1; q < MAX_SPLIT; ++q)
                if (q < p.split) sum += v[q];
            store(size_t(c) * p.n + n0 + o, sum);
        }
        cluster_sync();  // no CTA leaves while another still reads its shared memory
    } else {
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, C::TMEM_COLS);
    }
    if (threadIdx.x == 0 && bars->abort_flag != 0) {
        settle_copies(bars->full, C::STAGES, bars->issued);
        if (p.status) atomicOr(p.status, 64u);
    }
}

template <int BN>
cudaError_t launch_bn(const void* x, const void* w, const Params& p0, uint32_t out_f32, int sm_count, cudaStream_t stream, bool constant_weights) {
    using C = Cfg<BN>;
    using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const Params);
    static const Kernel kernels[2] = {int4_skinny_kernel<BN, false>, int4_skinny_kernel<BN, BN != 16>};  // sixteen columns: bf16 outputs alone
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        for (const Kernel f : kernels) {
            e = cudaFuncSetAttribute((const void*)f, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute((const void*)f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
            if (e != cudaSuccess) return e;
        }
        configured.fetch_or(bit, std::memory_order_release);
    }
    Params p = p0;
    const uint32_t tiles = (p.n + BM - 1) / BM, blocks = p.k / KB;
    // as many parts as fit at once, two stages each at least (14336 x 4096 at 16 columns: 16.6 / 14.1 / 17.5 us with 1 / 2 / 4
    // parts of 112 tiles on 296 slots; 4096 x 14336: 24.1 / 14.8 / 13.7 us with 2 / 4 / 8 parts of 32 tiles)
    const uint32_t slots = uint32_t(sm_count) * (C::HALF ? 2u : 1u);
    p.split = slots / tiles;
    if (p.split > blocks / 2) p.split = blocks / 2;
    if (p.split > uint32_t(MAX_SPLIT)) p.split = MAX_SPLIT;
    if (p.split < 1) p.split = 1;
    const bool all_sms = whole_device(dev, sm_count);
    CUtensorMap mw, mx;
    if (!encode_tensor_map_2d(&mw, w, p.n, p.k / 2, 1, BM, KB / 2, true) || !encode_tensor_map_2d(&mx, x, p.m, p.k, 2, BN, 64, true))
        return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = C::SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.split;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    dependent(attr[1]);
    cfg.attrs = attr;
    p.constant = constant_weights;
    p.early = constant_weights || all_sms;
    cfg.numAttrs = p.early ? 2 : 1;
    // A caller that wants an SM left free (sm_count below the device's, VYB_LAUNCH_LEAVE_ONE_SM) gets launches that fit the other SMs at once:
    // a second wave of one launch would fill every SM as the first one drains. Anybody else: one launch for all tiles.
    const uint32_t step = all_sms ? tiles : slots;
    for (p.tile0 = 0; p.tile0 < tiles; p.tile0 += step) {
        cfg.gridDim = dim3((tiles - p.tile0 < step ? tiles - p.tile0 : step) * p.split);
        e = cudaLaunchKernelEx(&cfg, kernels[out_f32 ? 1 : 0], mw, mx, p);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

bool int4_skinny_supported(const void* x, const void* w, const void* scale, uint32_t m, uint32_t n, uint32_t k, uint32_t group) {
    return m >= 1 && m <= 64 && n >= 1 && group == uint32_t(GROUP) && k >= uint32_t(KB) && k % KB == 0 &&
           ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15u) == 0 && (reinterpret_cast<uintptr_t>(scale) & 3u) == 0;
}

cudaError_t launch_int4_skinny(const void* x_bf16, const void* w_packed, const void* scale_bf16, void* y, uint32_t m, uint32_t n,
                               uint32_t k, uint32_t out_f32, int sm_count, cudaStream_t stream, uint32_t* status, bool constant_weights) {
    Params p = {};
    p.scales = static_cast<const uint16_t*>(scale_bf16);
    p.y = y;
    p.status = status;
    p.m = m;
    p.n = n;
    p.k = k;
    // 17..32 rows take the 48-column form: a 32-column form with two CTAs per SM measured 18.7 us at 14336 x 4096, 48 columns 15.7
    // f32 outputs of up to 16 rows come from other kernels (run_int4_linear, launch_int4_gemv); called for here, they take 48 columns too
    if (m <= 16 && !out_f32) return launch_bn<16>(x_bf16, w_packed, p, out_f32, sm_count, stream, constant_weights);
    if (m <= 48) return launch_bn<48>(x_bf16, w_packed, p, out_f32, sm_count, stream, constant_weights);
    return launch_bn<64>(x_bf16, w_packed, p, out_f32, sm_count, stream, constant_weights);
}

}  // namespace vybk
