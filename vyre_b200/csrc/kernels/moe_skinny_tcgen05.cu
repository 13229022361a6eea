// Grouped expert GEMMs of the MoE FFN layer when the experts have few rows each (tcgen05, sm_100a):
//
//   glu:    h[r, j] = bf16( g * (u * sigmoid(g)) ),  g = bf16(x[r, :] . W1[e, j, :]),  u = bf16(x[r, :] . W3[e, j, :])
//   plain:  y[r, j] = bf16( x[r, :] . W2[e, j, :] )                weights bf16((q - 8) * s), f32 sums over the whole k
//
// What bounds it: the experts' packed weights (all of them are read, whatever the token count) and the instructions that
// unpack them. The pair GEMM (int4_gemm_pair_tcgen05.cu) puts 256 activation rows on the M side of its tiles; with sixteen
// rows per expert it does the same unpacking into shared memory and sixteen times the tensor work for padding. Here the
// WEIGHT rows are the M side, the activation rows the N side (BN = 32 or 64 columns), and the unpacked weights go to tensor
// memory, from where the MMA reads them as its A operand. An item is 256 weight rows (glu: 128 gate and the same 128 up rows)
// x BN rows of one expert x the whole k; one persistent CTA per SM walks the items. Per stage of 256 k: two packed boxes and
// four activation boxes by TMA; sixteen warps unpack (four for each 128 weight rows x 128 k of a stage: eight warps took 219 us
// where sixteen took 180, latency is half of a stage); one thread issues the MMAs; warps 20-23 drain the accumulators of the
// previous item (two sets).
// Measured (8 experts, 4096 / 14336, 64 tokens x 2, cold): gate / up GEMM 399 -> 150 us, down GEMM 377 -> 76 us; the layer
// 774 -> 267 us at 64 tokens, 268 -> 160 us at one. The unpacking still issues 27 instructions a word (15 of them the
// conversion) and keeps the logic pipe 70 % busy; the packed bytes alone would take 108 us.
// Inside every eight k the activations lie in the order 0 4 1 5 2 6 3 7 (the gather and the glu epilogue write them so): that
// is the order in which a shift and a mask unpack a word, 15 instructions per eight weights instead of 17, 7 of them on the
// half-rate logic pipe instead of 9. Values and rounding points are the pair GEMM's.
//
// Every wait is bounded; on expiry a status word is raised, the CTA waits for what it has started and frees its TMEM. No multicast.
//
// Replaces the per-token expert_mlp of vyre-libs/src/nn/moe/expert_mlp.rs:18-150 for decode batches.
#include <cuda_bf16.h>

#include <atomic>

#include "dependent_launch.cuh"
#include "kernels.h"
#include "tcgen05_common.cuh"

namespace vybk {
namespace {

using namespace tc;

constexpr int BM = 128, UMMA_K = 16, STEP = 128;  // k per unpack step
constexpr int KB = 256;                           // k per stage
constexpr int RAW_BYTES = BM * KB / 2;            // 16 KB per 128 weight rows
constexpr int UNPACK_WARPS = 16, EPI_WARP = 4 + UNPACK_WARPS;
constexpr int THREADS = (EPI_WARP + 4) * 32, TMEM_COLS = 512;
constexpr uint32_t MAX_EXPERTS = 64;
constexpr uint32_t ROW_TILE = 256;                // rows that an expert's segment is padded to

struct Bars {
    unsigned long long full[4], empty[4], a_full[4], a_empty[4], d_full[2], d_empty[2], drained;
    uint32_t tmem_base;
    unsigned int abort_flag;
    uint32_t issued;  // copies of the TMA role
    uint32_t seg_row[MAX_EXPERTS], seg_count[MAX_EXPERTS];
};

template <int BN>
struct Cfg {
    static constexpr int B_BYTES = BN * KB * 2;
    static constexpr int STAGE_BYTES = 2 * RAW_BYTES + B_BYTES;
    static constexpr int STAGES = BN == 32 ? 4 : 3;
    static constexpr int SLOTS = BN == 32 ? 3 : 2;  // unpacked steps, 64 columns for each 128 weight rows
    static constexpr int A_COL = 4 * BN;            // two sets of two accumulators come first
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 2048 /*control*/ + 1024 /*alignment*/;
    static_assert(A_COL + SLOTS * 128 <= TMEM_COLS, "tensor memory");
    static_assert(SMEM_BYTES <= 227 * 1024 && sizeof(Bars) <= 2048, "shared memory");
};

struct Params {
    const uint16_t* scales;   // bf16 [weight rows][k / group]
    __nv_bfloat16* y;         // [rows][ldy]
    const uint32_t* plan;     // moe_plan_kernel's words: [1 + e] = first row of expert e's segment | padding rows at its end
    uint32_t* status;
    uint32_t experts, n_tiles, k, group, ldy;
    uint32_t expert_rows;     // weight rows per expert
    uint32_t second;          // weight rows between the two halves of an item (glu: W1 -> W3; plain: 128)
    uint32_t tile_rows;       // weight rows between two items of an expert (glu 128, plain 256)
    uint32_t group_inv;       // group / 64 > 1: (i * group_inv) >> 32 = i / (group / 64) for the 64-k blocks i of a row; else 0
};

struct Item {
    uint32_t expert, chunk, tile;
};

// a packed word of eight nibbles -> bf16 pairs (k, k + 4) = bf16((q - 8) * s); the subtraction is exact
__device__ __forceinline__ void dequant_word(uint32_t w, uint32_t s2, uint32_t* out) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t t = and_or(w >> (4 * i), 0x000F000Fu, 0x43004300u);  // 0x43nn is 128 + nn in bf16
        asm("{\n\t.reg .b32 d;\n\tsub.bf16x2 d, %1, %2;\n\tmul.bf16x2 %0, d, %3;\n\t}" : "=r"(out[i]) : "r"(t), "r"(0x43084308u), "r"(s2));
    }
}
__device__ __forceinline__ float bf16_round(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

template <int BN, bool GLU>
__global__ void __launch_bounds__(THREADS, 1)
moe_skinny_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Params p) {
    using C = Cfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    Bars* bars = reinterpret_cast<Bars*>(tiles + C::STAGES * C::STAGE_BYTES);
    volatile unsigned int* abort_flag = &bars->abort_flag;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t stages_per_item = p.k / KB;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(smem_u32(&bars->full[s]), 1);
            mbar_init(smem_u32(&bars->empty[s]), UNPACK_WARPS + 1);  // the unpack warps and the MMAs
        }
        for (int s = 0; s < C::SLOTS; ++s) {
            mbar_init(smem_u32(&bars->a_full[s]), 8);
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
        tmem_alloc(smem_u32(&bars->tmem_base), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    lets_next_start();
    waits_for_previous();
    for (uint32_t e = threadIdx.x; e < p.experts; e += THREADS) {
        const uint32_t here = p.plan[1 + e], next = p.plan[2 + e];
        const uint32_t row = here & ~(ROW_TILE - 1);
        bars->seg_row[e] = row;
        bars->seg_count[e] = (next & ~(ROW_TILE - 1)) - row - (here & (ROW_TILE - 1));
    }
    __syncthreads();

    uint32_t total = 0;
    for (uint32_t e = 0; e < p.experts; ++e) total += (bars->seg_count[e] + BN - 1) / BN * p.n_tiles;
    // items expert by expert; the row chunks of a weight tile are neighbours, so that they find its bytes in L2
    auto decode = [&](uint32_t i) {
        Item it{0, 0, 0};
        for (; it.expert < p.experts; ++it.expert) {
            const uint32_t chunks = (bars->seg_count[it.expert] + BN - 1) / BN, n = chunks * p.n_tiles;
            if (i < n) {
                it.tile = i / chunks;
                it.chunk = i % chunks;
                break;
            }
            i -= n;
        }
        return it;
    };

    bool ok = true;
    if (warp == 0) {
        if (elect_one()) {
            uint32_t s = 0, parity = 1, issued = 0;
            bool first = true;
            for (uint32_t i = blockIdx.x; i < total && ok; i += gridDim.x) {
                const Item it = decode(i);
                const int row0 = int(it.expert * p.expert_rows + it.tile * p.tile_rows), row1 = row0 + int(p.second);
                const int x_row = int(bars->seg_row[it.expert] + it.chunk * BN);
                for (uint32_t kb = 0; kb < stages_per_item; ++kb) {
                    if (!first && !mbar_wait(smem_u32(&bars->empty[s]), parity, abort_flag)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = smem_u32(&bars->full[s]), dst = smem_u32(tiles + s * C::STAGE_BYTES);
                    mbar_arrive_expect_tx(bar, C::STAGE_BYTES);
                    tma_load_2d(dst, &map_w, int(kb * (KB / 2)), row0, bar);
                    tma_load_2d(dst + RAW_BYTES, &map_w, int(kb * (KB / 2)), row1, bar);
#pragma unroll
                    for (int j = 0; j < KB / 64; ++j)
                        tma_load_2d(dst + 2 * RAW_BYTES + j * BN * 128, &map_x, int(kb * KB + j * 64), x_row, bar);
                    ++issued;
                    if (++s == uint32_t(C::STAGES)) {
                        s = 0;
                        first = false;
                        parity ^= 1;
                    }
                }
            }
            bars->issued = issued;
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc = idesc_bf16_f32(BM, BN);
            uint32_t s = 0, slot = 0, a_parity = 0, local = 0;
            for (uint32_t i = blockIdx.x; i < total && ok; i += gridDim.x, ++local) {
                const uint32_t set = local & 1, d = tmem + set * 2 * BN;
                if (local >= 2 && !mbar_wait(smem_u32(&bars->d_empty[set]), ((local >> 1) - 1) & 1, abort_flag)) break;
                for (uint32_t step = 0; step < 2 * stages_per_item; ++step) {
                    // the unpack warps saw the whole stage land before they arrived here: no wait of its own for x
                    if (!mbar_wait(smem_u32(&bars->a_full[slot]), a_parity, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t b = smem_u32(tiles + s * C::STAGE_BYTES + 2 * RAW_BYTES) + (step & 1) * 2 * BN * 128;
                    const uint64_t db0 = smem_desc_sw128(b), db1 = smem_desc_sw128(b + BN * 128);
                    const uint32_t a = tmem + C::A_COL + slot * 128;
#pragma unroll
                    for (int k = 0; k < STEP / UMMA_K; ++k) {
                        const uint64_t db = smem_desc_advance(k < 4 ? db0 : db1, (k & 3) * UMMA_K * 2);
                        mma_f16_ts(d, a + k * (UMMA_K / 2), db, idesc, (step | uint32_t(k)) != 0);
                        mma_f16_ts(d + BN, a + 64 + k * (UMMA_K / 2), db, idesc, (step | uint32_t(k)) != 0);
                    }
                    tc_commit(smem_u32(&bars->a_empty[slot]));
                    if (step & 1) {
                        tc_commit(smem_u32(&bars->empty[s]));
                        s = s + 1 == uint32_t(C::STAGES) ? 0u : s + 1;
                    }
                    if (++slot == uint32_t(C::SLOTS)) {
                        slot = 0;
                        a_parity ^= 1;
                    }
                }
                if (ok) tc_commit(smem_u32(&bars->d_full[set]));
            }
            if (*abort_flag != 0) settle_mma(smem_u32(&bars->drained));
        }
        __syncwarp();
    } else if (warp >= 4 && warp < uint32_t(EPI_WARP)) {
        // ---- unpack: a thread per weight row, one of the two steps of every stage ----
        const uint32_t unit = (warp >> 2) - 1, half = unit & 1, part = unit >> 1, quad = warp & 3, r = quad * 32 + lane;
        const uint32_t groups = p.k / p.group, dst0 = tmem + ((quad * 32) << 16) + C::A_COL + half * 64;
        uint32_t s = 0, parity = 0, slot = part, a_parity = 1;
        bool a_first = true;
        for (uint32_t i = blockIdx.x; i < total && ok; i += gridDim.x) {
            const Item it = decode(i);
            const uint16_t* srow = p.scales + size_t(it.expert * p.expert_rows + it.tile * p.tile_rows + half * p.second + r) * groups;
            // the scales of the step's two 64-k blocks, two stages ahead
            auto fetch = [&](uint32_t kb) {
                const uint32_t b0 = kb * 4 + part * 2, b1 = b0 + 1;
                return kb < stages_per_item ? make_uint2(srow[p.group_inv ? __umulhi(b0, p.group_inv) : b0],
                                                         srow[p.group_inv ? __umulhi(b1, p.group_inv) : b1])
                                            : make_uint2(0, 0);
            };
            uint2 sc = fetch(0), sc1 = fetch(1);
#pragma unroll 1
            for (uint32_t kb = 0; kb < stages_per_item; ++kb) {
                const uint2 sc2 = fetch(kb + 2);
                ok = mbar_wait(smem_u32(&bars->full[s]), parity, abort_flag);
                if (!a_first) ok = ok && mbar_wait(smem_u32(&bars->a_empty[slot]), a_parity, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
                const uint8_t* row = tiles + s * C::STAGE_BYTES + half * RAW_BYTES + r * 128;
#pragma unroll 1
                for (uint32_t j = 0; j < 4; ++j) {
                    const uint4 v = *reinterpret_cast<const uint4*>(row + (((part * 4 + j) ^ (r & 7u)) << 4));
                    const uint32_t s2 = (j < 2 ? sc.x : sc.y) * 0x10001u;
                    uint32_t a[16];
                    dequant_word(v.x, s2, a);
                    dequant_word(v.y, s2, a + 4);
                    dequant_word(v.z, s2, a + 8);
                    dequant_word(v.w, s2, a + 12);
                    tmem_st_32x16(dst0 + slot * 128 + j * 16, a);
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(smem_u32(&bars->empty[s]));
                    mbar_arrive(smem_u32(&bars->a_full[slot]));
                }
                sc = sc1;
                sc1 = sc2;
                if (++s == uint32_t(C::STAGES)) {
                    s = 0;
                    parity ^= 1;
                }
                slot += 2;
                if (slot >= uint32_t(C::SLOTS)) {
                    slot -= C::SLOTS;
                    a_first = false;
                    a_parity ^= 1;
                }
            }
        }
    } else if (warp >= uint32_t(EPI_WARP)) {
        const uint32_t quad = warp & 3, o = quad * 32 + lane;
        uint32_t local = 0;
        for (uint32_t i = blockIdx.x; i < total && ok; i += gridDim.x, ++local) {
            const Item it = decode(i);
            const uint32_t set = local & 1, taddr = tmem + ((quad * 32) << 16) + set * 2 * BN;
            ok = mbar_wait(smem_u32(&bars->d_full[set]), (local >> 1) & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t rows = min(uint32_t(BN), bars->seg_count[it.expert] - it.chunk * BN);
            const uint32_t at = GLU ? (o & ~7u) + (o & 3u) * 2 + ((o >> 2) & 1u) : o;  // glu: in the next GEMM's k order
            __nv_bfloat16* y = p.y + size_t(bars->seg_row[it.expert] + it.chunk * BN) * p.ldy + it.tile * p.tile_rows + at;
#pragma unroll 1
            for (uint32_t c = 0; c < BN; c += 16) {
                if (c >= rows) break;  // warp-uniform
                uint32_t v0[16], v1[16];
                tmem_ld_32x16(taddr + c, v0);
                tmem_ld_32x16(taddr + BN + c, v1);
                tmem_ld_wait();
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) {
                    if (c + j >= rows) break;
                    __nv_bfloat16* dst = y + size_t(c + j) * p.ldy;
                    if constexpr (GLU) {
                        // the single-token ops' rounding points: g and u are bf16 values, the activation is evaluated in f32
                        const float g = bf16_round(__uint_as_float(v0[j])), uu = bf16_round(__uint_as_float(v1[j]));
                        const float sig = 1.0f / (1.0f + expf(-g));
                        dst[0] = __float2bfloat16_rn(g * (uu * sig));
                    } else {
                        dst[0] = __float2bfloat16_rn(__uint_as_float(v0[j]));
                        dst[BM] = __float2bfloat16_rn(__uint_as_float(v1[j]));
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->d_empty[set]));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
    if (threadIdx.x == 0 && bars->abort_flag != 0) {
        settle_copies(bars->full, C::STAGES, bars->issued);
        if (p.status) atomicOr(p.status, 512u);
    }
}

template <int BN, bool GLU>
cudaError_t launch_cfg(const CUtensorMap& mw, const void* x, uint32_t max_rows, const Params& p, int sm_count, cudaStream_t stream) {
    using C = Cfg<BN>;
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        e = cudaFuncSetAttribute(moe_skinny_kernel<BN, GLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
        if (e != cudaSuccess) return e;
        configured.fetch_or(bit, std::memory_order_release);
    }
    CUtensorMap mx;
    if (!encode_tensor_map_2d(&mx, x, max_rows, p.k, 2, BN, 64, true)) return cudaErrorInvalidValue;
    return launch_dependent(moe_skinny_kernel<BN, GLU>, dim3(sm_count), dim3(THREADS), C::SMEM_BYTES, stream, mw, mx, p);
}

}  // namespace

cudaError_t launch_moe_skinny(const void* x_sorted, const void* w, const void* scales, void* y, const uint32_t* plan, uint32_t max_rows,
                              uint32_t n, uint32_t k, uint32_t group, uint32_t experts, bool glu, bool wide, int sm_count, cudaStream_t stream,
                              uint32_t* status) {
    if (n % 256 || k % 256 || group % 64 || experts > MAX_EXPERTS) return cudaErrorNotSupported;
    Params p = {};
    p.scales = static_cast<const uint16_t*>(scales);
    p.y = static_cast<__nv_bfloat16*>(y);
    p.plan = plan;
    p.status = status;
    p.experts = experts;
    p.k = k;
    p.group = group;
    p.ldy = n;
    p.tile_rows = glu ? 128 : 256;
    p.group_inv = group == 64 ? 0u : 0xFFFFFFFFu / (group / 64) + 1u;
    p.second = glu ? n : 128;
    p.expert_rows = glu ? 2 * n : n;
    p.n_tiles = n / p.tile_rows;
    CUtensorMap mw;
    if (!encode_tensor_map_2d(&mw, w, uint64_t(experts) * p.expert_rows, k / 2, 1, BM, KB / 2, true)) return cudaErrorInvalidValue;
    if (glu) return wide ? launch_cfg<64, true>(mw, x_sorted, max_rows, p, sm_count, stream) : launch_cfg<32, true>(mw, x_sorted, max_rows, p, sm_count, stream);
    return wide ? launch_cfg<64, false>(mw, x_sorted, max_rows, p, sm_count, stream) : launch_cfg<32, false>(mw, x_sorted, max_rows, p, sm_count, stream);
}

}  // namespace vybk
