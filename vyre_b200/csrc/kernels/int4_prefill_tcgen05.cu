// Group-quantized int4 linear with the weights in tensor memory on single CTAs (tcgen05, sm_100a): prefill batches of up to 128 rows or of few or
// short tiles (launch_int4_prefill; the CTA-pair GEMM has the rest), and few rows of any row length.
//
//   rounded (prefill):  y[m, n] = cast( sum_k x[m, k] * bf16((q[n, k] - 8) * s[n, g(k)]) )          any group of whole 64 k, f32 sums
//   exact (few rows):   y[m, n] = cast( sum_g s[n, g] * sum_{k in g} x[m, k] * (q[n, k] - 8) )      groups of 64 or 128, up to 16 rows
//
// The WEIGHT rows are the M = 128 side of the MMA and the activation rows its N side (16 to 128 columns); a thread unpacks a weight row's
// nibbles in registers and stores them to tensor memory, where the MMA reads its A operand: no unpacked byte goes through shared memory.
// A CTA per 128 x BN tile; k is split over a cluster where tiles leave SMs idle (partial tiles meet in distributed shared memory, added
// in rank order). Per CTA: warp 0 packed weights by TMA (256 k a stage), warp 2 activations, warp 1 MMAs, warp 3 prefetches scales, sixteen
// warps unpack (two sets of eight take the stages in turn), the last warps drain the sums: exact weights have an accumulator per
// group (up to eight rows: per 64 k), which meets its scale in f32 registers; rounded ones one accumulator for the whole row.
//
// What bounds it: a chain per stage (unpack 700 to 1500 cycles, MMA thread 400 + 430, waits of about 150 each), 1100 cycles with three unpacked
// stages in flight, where the logic pipe needs 512 and, at 128 columns, the MMAs 1024. Packed bytes at HBM speed would take 5 us of the
// 14 at 16 x 4096 -> 14336. Measured (nothing promised about the weights, HBM-cold, us, before / now): prefill kernels 16 x 4096 -> 14336 49 / 14,
// 64 x 3072 -> 2658 52 / 7.5, 128 x 7168 -> 1024 81 / 11; generic kernel at groups of 64 8 x 6400 -> 14336 371 / 21, 1 x 4096 -> 8192 58 / 10; the other
// tensor-memory kernel (int4_skinny_tcgen05.cu) 8 x 4096 -> 14336 15.8 / 13.5, 8 x 1024 -> 14336 7.1 / 5.4: that one keeps the decode launches,
// since two of its CTAs share an SM and with constant weights the next launch's are on their way under this one's (four decode blocks of
// 2048 / 6144 at 6 rows 92 us with it, 109 with this).
//
// Every wait is bounded; on expiry a status word is raised, the CTA waits for what it has started and frees its TMEM. No multicast.
//
// Replaces the generated scalar kernel of vyre-libs/src/nn/linear/inner/linear_4bit.rs:399-775 for the row-major layout of
// vyre-primitives/src/math/quantized/programs.rs:186-300 at prefill batches.
#include <cuda_bf16.h>

#include <atomic>

#include "dependent_launch.cuh"
#include "kernels.h"
#include "tcgen05_common.cuh"

namespace vybk {
namespace {

using namespace tc;

constexpr int BM = 128, UMMA_K = 16;
constexpr int KB = 256;                           // k per stage
constexpr int RAW_BYTES = BM * KB / 2;            // 16 KB of packed weights
constexpr int MAX_SPLIT = 8;
constexpr int UNPACK_WARPS = 16, EPI_WARP = 4 + UNPACK_WARPS;
constexpr int READY = 4, DONE = 8;                // barriers of stages that are ready and that are done: who follows them is never further behind
constexpr int TMEM_COLS = 512;
constexpr int CTRL_BYTES = 512, ALIGN_SLACK = 1024;
constexpr uint32_t PREFETCH_STAGES = 24;

// BN: activation rows of a tile. G: exact weights, an accumulator per 128 k (1) or per 64 k (2; HALVES: a group is two of them); 0: rounded
// weights, one accumulator for the whole row.
template <int BN, int G>
struct Cfg {
    static constexpr int X_BYTES = BN * KB * 2;
    // Weights and activations have rings of their own: a stage of weights is free as soon as it is unpacked, one of activations when its MMAs
    // are complete.
    static constexpr int STAGES = BN == 16 ? 10 : BN == 32 ? 9 : BN == 64 ? 6 : 5, X_STAGES = BN == 16 ? 6 : BN <= 64 ? 4 : 2;
    static constexpr int RING_BYTES = STAGES * RAW_BYTES + X_STAGES * X_BYTES;
    static constexpr int SMEM_BYTES = RING_BYTES + CTRL_BYTES + ALIGN_SLACK;
    static constexpr int SETS = G == 0 ? 1 : 2 * G;            // accumulators of a stage
    static constexpr int A_COL = G == 0 ? BN : 2 * SETS * BN;  // accumulators (of two stages) come first
    static constexpr int A_SLOTS = 3;                          // unpacked stages (8 x 4096 -> 14336: 13.4 us with two, 12.1 with three)
    static_assert(A_COL + A_SLOTS * 128 <= TMEM_COLS && X_STAGES <= DONE && STAGES <= 10, "tensor memory, barriers");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
    static_assert(BN * BM * 4 <= RING_BYTES, "the partial tile reuses the stages");
};
constexpr int EPI_WARPS = 4, THREADS = (EPI_WARP + EPI_WARPS) * 32;

struct Bars {
    unsigned long long full[10], empty[10], x_full[6], b_full[READY], done[DONE], acc_full, drained;
    uint32_t tmem_base;
    unsigned int abort_flag;
    uint32_t issued, x_issued;  // copies of the TMA roles
    uint32_t redo;              // an output of this tile is not finite
};
static_assert(sizeof(Bars) <= CTRL_BYTES, "control block");

// The bytes of a row's scales that `stages` stages from `stage` on need
struct Range {
    uint32_t first, last;
};
__host__ __device__ constexpr Range scale_bytes(uint32_t stage, uint32_t stages, uint32_t group, uint32_t groups) {
    const uint32_t end = uint32_t((uint64_t(stage + stages) * KB + group - 1) / group);
    return {uint32_t(uint64_t(stage) * KB / group) * 2, (end < groups ? end : groups) * 2};
}
constexpr bool same(Range a, uint32_t first, uint32_t last) { return a.first == first && a.last == last; }
// two parts of 4096 k: each half of the row's scales, whatever the group; a group that spans both; a last stage past the row's end
static_assert(same(scale_bytes(0, 8, 64, 64), 0, 64) && same(scale_bytes(8, 8, 64, 64), 64, 128), "groups of 64");
static_assert(same(scale_bytes(0, 8, 128, 32), 0, 32) && same(scale_bytes(8, 8, 128, 32), 32, 64), "groups of 128");
static_assert(same(scale_bytes(8, 8, 512, 8), 8, 16) && same(scale_bytes(8, 8, 4096, 1), 0, 2), "long groups");
static_assert(same(scale_bytes(2, 2, 192, 5), 4, 10) && same(scale_bytes(6, 1, 64, 25), 48, 50), "a group on a part's border, ends");

struct Params {
    const uint16_t* x;       // bf16 [m][k] and packed weights [n][k / 8], for by_definition
    const uint32_t* w;
    const uint16_t* scales;  // bf16 [n][k / group]
    void* y;
    uint32_t* status;
    uint32_t m, n, k, split;
    uint32_t group_inv;      // G = 0: group / 64 > 1: (i * group_inv) >> 32 = i / (group / 64) for the 64-k blocks i of a row; else 0
    uint32_t group, groups;  // k of a group, groups of a row
    uint32_t halves;         // HALVES: 1, read from here, as a constant shift makes an instance that spills 108 bytes
    uint32_t tile0;          // first weight tile of this launch
    uint32_t early;          // the next launch may start beside this one
    // unpack_word's, from here so that they stay in registers: an instruction takes one immediate, and the compiler makes a second one
    // anew before every use (three instructions a word)
    uint32_t mask, mul, add;
};

// A packed word of eight nibbles -> four bf16 pairs (k, k + 1) = (q - 8) / 64. A byte in both halves of a register, masked to its low nibble
// below and to its high one above, is a pair of subnormal bf16 numbers n 2^-133 and 16 n 2^-133; one exact fused multiply-add makes n / 64 - 1 / 8.
__device__ __forceinline__ void unpack_word(uint32_t w, uint32_t* out, uint32_t mask, uint32_t mul, uint32_t add) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t t = __byte_perm(w, 0u, 0x4040 | i | i << 8) & mask;
        asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(out[i]) : "r"(t), "r"(mul), "r"(add));
    }
}

__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.40282347e38f; }  // false for NaN

// One output of exact weights by the definition, as int4_linear_generic_kernel computes it (a lane's words in ascending order, then the lanes
// as the shuffles add them): a group's sum, or a scale times 64, can leave f32's range where no term does. An output that does not come out
// finite is computed anew, so that an infinity or NaN stands only where the definition has one.
__device__ float by_definition(const Params& p, uint32_t m, uint32_t n) {
    const uint16_t* x = p.x + size_t(m) * p.k;
    const uint32_t* w = p.w + size_t(n) * (p.k / 8);
    const uint16_t* scales = p.scales + size_t(n) * p.groups;
    const uint32_t k = p.k, group = p.group;
    float part[32];
#pragma unroll 1
    for (uint32_t lane = 0; lane < 32; ++lane) {
        float acc = 0.0f;
#pragma unroll 1
        for (uint32_t wi = lane; wi < k / 8; wi += 32) {
            const float s = __uint_as_float(uint32_t(scales[wi * 8 / group]) << 16);
            for (uint32_t i = 0; i < 8; ++i)
                acc = fmaf(__uint_as_float(uint32_t(x[wi * 8 + i]) << 16), float(int(w[wi] >> (4 * i) & 15u) - 8) * s, acc);
        }
        part[lane] = acc;
    }
#pragma unroll 1
    for (uint32_t o = 16; o > 0; o >>= 1)
        for (uint32_t lane = 0; lane < o; ++lane) part[lane] += part[lane + o];
    return part[0];
}

// Those of a tile that are not finite: columns `part`, `part` + `split` and so on are this block's. Out of line, since next to nothing takes it, and its
// parameters by value: a reference would need the kernel's in memory (16 x 4096 -> 14336 with f32 outputs 14.7 / 15.4 us).
template <int BN, bool OUT_F32>
__device__ __noinline__ void redo_tile(const Params p, uint32_t m0, uint32_t n0, uint32_t part) {
    for (uint32_t idx = threadIdx.x; idx < BN * BM; idx += THREADS) {
        const uint32_t m = m0 + idx / BM * p.split + part, n = n0 + idx % BM;
        if (idx / BM * p.split + part >= BN || m >= p.m || n >= p.n) continue;
        const size_t at = size_t(m) * p.n + n;
        if constexpr (OUT_F32) {
            float* y = static_cast<float*>(p.y) + at;
            if (!finite(*y)) *y = by_definition(p, m, n);
        } else {
            __nv_bfloat16* y = static_cast<__nv_bfloat16*>(p.y) + at;
            if (!finite(__bfloat162float(*y))) *y = __float2bfloat16_rn(by_definition(p, m, n));
        }
    }
}

template <int BN, int G, bool HALVES, bool OUT_F32>
__global__ void __launch_bounds__(THREADS, 1)
int4_tmem_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Params p) {
    using C = Cfg<BN, G>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* x_tiles = tiles + C::STAGES * RAW_BYTES;
    Bars* bars = reinterpret_cast<Bars*>(tiles + C::RING_BYTES);
    volatile unsigned int* abort_flag = &bars->abort_flag;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t part = blockIdx.x % p.split, n0 = (p.tile0 + blockIdx.x / p.split) * BM, m0 = blockIdx.y * BN;
    const uint32_t blocks = (p.k + KB - 1) / KB, base = blocks / p.split, rem = blocks % p.split;
    const uint32_t kb0 = part * base + min(part, rem), kbs = base + (part < rem ? 1u : 0u);  // stages of this part
    auto store = [&](uint32_t c, uint32_t row, float v) {
        if (m0 + c >= p.m || row >= p.n) return;
        const size_t at = size_t(m0 + c) * p.n + row;
        if constexpr (OUT_F32) static_cast<float*>(p.y)[at] = v;
        else static_cast<__nv_bfloat16*>(p.y)[at] = __float2bfloat16_rn(v);
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) {
            mbar_init(smem_u32(&bars->full[s]), 1);
            mbar_init(smem_u32(&bars->empty[s]), UNPACK_WARPS / 2);
        }
        for (int s = 0; s < C::X_STAGES; ++s) mbar_init(smem_u32(&bars->x_full[s]), 1);
        for (int s = 0; s < READY; ++s) mbar_init(smem_u32(&bars->b_full[s]), UNPACK_WARPS / 2 + (G == 0 ? 0 : EPI_WARPS));  // unpacked, and its accumulators free
        for (int s = 0; s < DONE; ++s) mbar_init(smem_u32(&bars->done[s]), 1);
        mbar_init(smem_u32(&bars->acc_full), 1);
        mbar_init(smem_u32(&bars->drained), 1);
        bars->abort_flag = 0;
        bars->redo = 0;
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
    if (p.early) lets_next_start();
    // Every role waits for the launches before this one before it waits for anything with a limit: their time is not this launch's. (One wait
    // here for all roles but the prefetching ones costs the exact forms 72 bytes of spilled registers: 8 x 6400 -> 14336 20.7 / 28 us.)
    auto done_wait = [&](uint32_t i) { return mbar_wait(smem_u32(&bars->done[i % DONE]), (i / DONE) & 1, abort_flag); };

    bool ok = true;
    if (warp == 0) {
        // ---- packed weights: into L2 while the launches before this one run, from there when they are complete ----
        if (elect_one())
            for (uint32_t i = 0; i < min(kbs, PREFETCH_STAGES); ++i) tma_prefetch_2d(&map_w, int((kb0 + i) * (KB / 2)), int(n0));
        __syncwarp();
        waits_for_previous();
        if (elect_one()) {
            uint32_t i = 0;
            for (; i < kbs; ++i) {
                const uint32_t s = i % C::STAGES, bar = smem_u32(&bars->full[s]);
                if (i >= uint32_t(C::STAGES) && !mbar_wait(smem_u32(&bars->empty[s]), ((i / C::STAGES) - 1) & 1, abort_flag)) break;
                mbar_arrive_expect_tx(bar, RAW_BYTES);
                tma_load_2d(smem_u32(tiles + s * RAW_BYTES), &map_w, int((kb0 + i) * (KB / 2)), int(n0), bar);
            }
            bars->issued = i;
        }
        __syncwarp();
    } else if (warp == 2) {
        // ---- activations ----
        waits_for_previous();
        if (elect_one()) {
            uint32_t i = 0;
            for (; i < kbs; ++i) {
                const uint32_t s = i % C::X_STAGES, bar = smem_u32(&bars->x_full[s]), dst = smem_u32(x_tiles + s * C::X_BYTES);
                if (i >= uint32_t(C::X_STAGES) && !done_wait(i - C::X_STAGES)) break;
                mbar_arrive_expect_tx(bar, C::X_BYTES);
#pragma unroll
                for (int j = 0; j < KB / 64; ++j) tma_load_2d(dst + j * BN * 128, &map_x, int((kb0 + i) * KB + j * 64), int(m0), bar);
            }
            bars->x_issued = i;
        }
        __syncwarp();
    } else if (warp == 3) {
        // ---- scales into L2: a row's share is a few sectors, read two bytes at a time ----
        const uint32_t row_bytes = p.groups * 2;
        const Range range = scale_bytes(kb0, kbs, p.group, p.groups);
        for (uint32_t r = lane; r < BM && n0 + r < p.n; r += 32)
            for (uint32_t at = range.first; at < range.last; at += 32)
                prefetch_l2(reinterpret_cast<const uint8_t*>(p.scales) + size_t(n0 + r) * row_bytes + at);
        waits_for_previous();
    } else if (warp == 1) {
        // ---- MMA: one commit per stage frees the unpacked weights and the activations and hands the sums on ----
        constexpr uint32_t idesc = idesc_bf16_f32(BM, BN);
        waits_for_previous();
        if (elect_one()) {
            uint32_t xs = 0, x_parity = 0, slot = 0;
#pragma unroll 1
            for (uint32_t i = 0; i < kbs; ++i) {
                // One round trip for all that a stage waits for: a wait takes this thread 150 cycles although the barrier is complete, a commit
                // 60 to 100, an MMA 20 (with waits and commits of their own for activations, accumulators and slots 830 cycles per 128 k).
                if (!mbar_wait2(smem_u32(&bars->x_full[xs]), x_parity, smem_u32(&bars->b_full[i % READY]), (i / READY) & 1, abort_flag)) break;
                tc_fence_after();
                const uint32_t b = smem_u32(x_tiles + xs * C::X_BYTES), d = G == 0 ? tmem : tmem + (i & 1) * C::SETS * BN, a = tmem + C::A_COL + slot * 128;
                const uint64_t db = smem_desc_sw128(b);
#pragma unroll
                for (int k = 0; k < KB / UMMA_K; ++k)
                    mma_f16_ts(d + k / (16 / C::SETS) * BN, a + k * (UMMA_K / 2), smem_desc_advance(db, k / 4 * BN * 128 + (k & 3) * UMMA_K * 2), idesc,
                               k % (16 / C::SETS) != 0 || (G == 0 && i != 0));
                tc_commit(smem_u32(&bars->done[i % DONE]));
                slot = slot + 1 == uint32_t(C::A_SLOTS) ? 0u : slot + 1;
                if (++xs == uint32_t(C::X_STAGES)) {
                    xs = 0;
                    x_parity ^= 1;
                }
            }
            if (G == 0 && *abort_flag == 0) tc_commit(smem_u32(&bars->acc_full));
            if (*abort_flag != 0) settle_mma(smem_u32(&bars->drained));
        }
        __syncwarp();
    } else if (warp < uint32_t(EPI_WARP)) {
        // ---- unpack: a thread per weight row, eight warps a stage, two sets of eight in turn: what one set waits for lies under the work of the other ----
        const uint32_t unit = (warp >> 2) - 1, half = unit & 1, quad = warp & 3, r = quad * 32 + lane;
        const uint32_t mask = p.mask, mul = p.mul, add = p.add;
        uint32_t s = unit >> 1, parity = 0;
        waits_for_previous();
        // G = 0: the scales of this thread's two 64-k blocks, a stage of its own ahead
        const uint16_t* sp = p.scales + size_t(min(n0 + r, p.n - 1)) * p.groups;
        auto scale = [&](uint32_t i, uint32_t b) {
            const uint32_t at = (kb0 + i) * 4 + half * 2 + b, g = p.group_inv ? __umulhi(at, p.group_inv) : at;
            return g < p.groups ? uint32_t(sp[g]) * 0x10001u : 0u;  // past the row's last group the activations are zeros
        };
        uint32_t next0 = G == 0 ? scale(s, 0) : 0, next1 = G == 0 ? scale(s, 1) : 0;
#pragma unroll 1
        for (uint32_t i = s; i < kbs; i += 2) {
            const uint32_t s0 = next0, s1 = next1;
            if constexpr (G == 0) {
                next0 = scale(i + 2, 0);
                next1 = scale(i + 2, 1);
            }
            ok = mbar_wait(smem_u32(&bars->full[s]), parity, abort_flag);
            if (i >= uint32_t(C::A_SLOTS)) ok = ok && done_wait(i - C::A_SLOTS);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint8_t* row = tiles + s * RAW_BYTES + r * 128;
            const uint32_t dst = tmem + ((quad * 32) << 16) + C::A_COL + i % C::A_SLOTS * 128 + half * 64;
            uint4 v[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) v[j] = *reinterpret_cast<const uint4*>(row + (((half * 4 + j) ^ (r & 7u)) << 4));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t a[16];
                const uint32_t words[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if constexpr (G != 0) {
                        unpack_word(words[u], a + 4 * u, mask, mul, add);
                    } else {
                        uint32_t q[4];
                        unpack_int4_bf16(words[u], q);
#pragma unroll
                        for (int e = 0; e < 4; ++e) asm("mul.bf16x2 %0, %1, %2;" : "=r"(a[4 * u + e]) : "r"(q[e]), "r"(j < 2 ? s0 : s1));
                    }
                }
                tmem_st_32x16(dst + j * 16, a);
            }
            // The packed bytes have been used, not only loaded: the compiler may move loads below an arrival that only follows them in the
            // source, and the next copy then lands under them (wrong rows in half of a few hundred launches).
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->empty[s]));
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->b_full[i % READY]));
            s += 2;
            if (s >= uint32_t(C::STAGES)) {
                s -= C::STAGES;
                parity ^= 1;
            }
        }
    } else if constexpr (G == 0) {
        // ---- epilogue: the sums as they are ----
        waits_for_previous();
        const uint32_t quad = warp & 3, o = quad * 32 + lane, row = n0 + o;
        ok = mbar_wait(smem_u32(&bars->acc_full), 0, abort_flag);  // of its own: this role does not follow `done` stage by stage
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            tc_fence_after();
            float* partial = reinterpret_cast<float*>(tiles);  // every load and MMA of this CTA is complete: the stages are free
#pragma unroll 1
            for (uint32_t c = 0; c < BN && m0 + c < p.m; c += 16) {
                uint32_t v[16];
                tmem_ld_32x16(tmem + ((quad * 32) << 16) + c, v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (p.split == 1) store(c + j, row, __uint_as_float(v[j]));
                    else partial[(c + j) * BM + o] = __uint_as_float(v[j]);
                }
            }
        }
    } else {
        // ---- epilogue: acc += scale * group sum ----
        waits_for_previous();
        const uint32_t quad = warp & 3, o = quad * 32 + lane, row = n0 + o;
        const uint32_t groups = p.groups, g0 = kb0 * 2 * G;
        const uint16_t* sp = p.scales + size_t(min(row, p.n - 1)) * groups;
        float acc[BN];
#pragma unroll
        for (int c = 0; c < BN; ++c) acc[c] = 0.0f;
        if (lane == 0) {  // both stages' accumulators are free
            mbar_arrive(smem_u32(&bars->b_full[0]));
            mbar_arrive(smem_u32(&bars->b_full[1]));
        }
        constexpr uint32_t AHEAD = 2;  // stages whose scales are in flight
        uint32_t queue[AHEAD][G];
        auto load_scales = [&](uint32_t i, uint32_t (&q)[G]) {
#pragma unroll
            for (int h = 0; h < G; ++h) {  // past the row's last group the activations are zeros
                const uint32_t set = g0 + (i * G + h) * 2, g = HALVES ? set >> p.halves : set, g1 = HALVES ? (set + 1) >> p.halves : set + 1;
                q[h] = (g < groups ? uint32_t(sp[g]) : 0u) | (g1 < groups ? uint32_t(sp[g1]) << 16 : 0u);
            }
        };
#pragma unroll
        for (uint32_t d = 0; d < AHEAD; ++d) load_scales(d, queue[d]);
#pragma unroll 1
        for (uint32_t i0 = 0; i0 < kbs && ok; i0 += AHEAD) {
#pragma unroll
            for (uint32_t d = 0; d < AHEAD; ++d) {
                const uint32_t i = i0 + d;
                if (i >= kbs || !ok) break;
                uint32_t bits[G];
#pragma unroll
                for (int h = 0; h < G; ++h) bits[h] = queue[d][h];
                load_scales(i + AHEAD, queue[d]);
                ok = done_wait(i);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int h = 0; h < C::SETS; ++h) {
                    const float s = __uint_as_float(h & 1 ? bits[h / 2] & 0xFFFF0000u : bits[h / 2] << 16) * 64.0f;  // tensor memory holds (q - 8) / 64
                    uint32_t v[BN];
                    tmem_ld_32x16(tmem + ((quad * 32) << 16) + (d * C::SETS + h) * BN, v);
                    tmem_ld_wait();
                    if (h == C::SETS - 1) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(smem_u32(&bars->b_full[(i + 2) % READY]));  // for the stage after the next
                    }
#pragma unroll
                    for (int c = 0; c < BN; ++c) acc[c] = fmaf(s, __uint_as_float(v[c]), acc[c]);
                }
            }
        }
        if (ok) {
            if (p.split == 1) {
                bool good = true;
#pragma unroll
                for (int c = 0; c < BN; ++c) {
                    store(c, row, acc[c]);
                    good = good && finite(acc[c]);
                }
                if (!good) bars->redo = 1;
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
            if (m0 + c >= p.m || n0 + o >= p.n) continue;
            const uint32_t addr = smem_u32(reinterpret_cast<float*>(tiles) + c * BM + o);
            float v[MAX_SPLIT];
#pragma unroll
            for (uint32_t q = 0; q < MAX_SPLIT; ++q)
                if (q < p.split) v[q] = ld_cluster_f32(mapa(addr, q));
            float sum = v[0];
#pragma unroll
            for (uint32_t q = 1; q < MAX_SPLIT; ++q)
                if (q < p.split) sum += v[q];
            store(c, n0 + o, sum);
            if (G != 0 && !finite(sum)) bars->redo = 1;
        }
        cluster_sync();  // no CTA leaves while another still reads its shared memory
    } else {
        __syncthreads();
    }
    if (G != 0 && bars->redo) redo_tile<BN, OUT_F32>(p, m0, n0, part);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
    if (threadIdx.x == 0 && bars->abort_flag != 0) {
        settle_copies(bars->full, C::STAGES, bars->issued);
        settle_copies(bars->x_full, C::X_STAGES, bars->x_issued);
        if (p.status) atomicOr(p.status, 8u);
    }
}

template <int BN, int G, bool OUT_F32, bool HALVES = false>
cudaError_t launch_cfg(const void* x, const void* w, Params p, int sm_count, cudaStream_t stream) {
    using C = Cfg<BN, G>;
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        const void* f = (const void*)int4_tmem_kernel<BN, G, HALVES, OUT_F32>;
        e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
        configured.fetch_or(bit, std::memory_order_release);
    }
    const uint32_t tiles = (p.n + BM - 1) / BM, rows = (p.m + BN - 1) / BN, slots = uint32_t(sm_count) / rows > 0 ? uint32_t(sm_count) / rows : 1u;
    // as many parts of the k range as fit at once, two stages each at least
    const uint32_t blocks = (p.k + KB - 1) / KB;
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
    p.early = all_sms;
    cfg.numAttrs = p.early ? 2 : 1;
    // A caller that wants an SM left free (sm_count below the device's) gets launches that fit the other SMs at once: a second wave of one
    // launch would fill every SM as the first one drains. Anybody else: one launch for all tiles.
    const uint32_t step = all_sms ? tiles : slots;
    for (p.tile0 = 0; p.tile0 < tiles; p.tile0 += step) {
        cfg.gridDim = dim3((tiles - p.tile0 < step ? tiles - p.tile0 : step) * p.split, rows);
        e = cudaLaunchKernelEx(&cfg, int4_tmem_kernel<BN, G, HALVES, OUT_F32>, mw, mx, p);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

Params make_params(const void* x, const void* w, const void* scale, void* y, uint32_t m, uint32_t n, uint32_t k, uint32_t group, uint32_t* status) {
    Params p = {};
    p.x = static_cast<const uint16_t*>(x);
    p.w = static_cast<const uint32_t*>(w);
    p.scales = static_cast<const uint16_t*>(scale);
    p.y = y;
    p.status = status;
    p.m = m;
    p.n = n;
    p.k = k;
    p.group = group;
    p.groups = k / group;
    p.mask = 0x00F0000Fu;
    p.mul = 0x7D007F00u;  // 2^123 | 2^127
    p.add = 0xBE00BE00u;  // -1/8
    return p;
}

}  // namespace

bool int4_prefill_supported(uint32_t m, uint32_t n, uint32_t k, uint32_t group) {
    // 64-k blocks must not straddle a scale group; tensor-map strides need 16-byte multiples
    return m >= 1 && n >= 1 && k >= 64 && k % 64 == 0 && group >= 64 && group % 64 == 0 && k % group == 0;
}
bool int4_few_rows_supported(const void* x, const void* w, const void* scale, uint32_t m, uint32_t n, uint32_t k, uint32_t group) {
    return m >= 1 && m <= 16 && n >= 1 && (group == 128 || group == 64) && k >= 64 && k % group == 0 &&
           ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15u) == 0 && (reinterpret_cast<uintptr_t>(scale) & 1u) == 0;
}

cudaError_t launch_int4_few_rows(const void* x_bf16, const void* w_packed, const void* scale_bf16, void* y, uint32_t m, uint32_t n, uint32_t k,
                                 uint32_t group, uint32_t out_f32, int sm_count, cudaStream_t stream, uint32_t* status) {
    Params p = make_params(x_bf16, w_packed, scale_bf16, y, m, n, k, group, status);
    p.halves = group == 128;
    const auto launch = [&](auto f32, auto bf16) { return out_f32 ? f32(x_bf16, w_packed, p, sm_count, stream) : bf16(x_bf16, w_packed, p, sm_count, stream); };
    // Up to eight rows: sums in the tensor core over 64 k (run_int4_linear has the errors). More: over a whole group, as the kernel has them that
    // takes 17 rows on.
    if (group == 64) return launch(launch_cfg<16, 2, true>, launch_cfg<16, 2, false>);
    return m <= 8 ? launch(launch_cfg<16, 2, true, true>, launch_cfg<16, 2, false, true>) : launch(launch_cfg<16, 1, true>, launch_cfg<16, 1, false>);
}

cudaError_t launch_int4_prefill(const void* x_bf16, const void* w_packed, const void* scale_bf16, void* y, uint32_t m, uint32_t n, uint32_t k,
                                uint32_t group, uint32_t out_f32, int sm_count, cudaStream_t stream, uint32_t* status) {
    // The CTA-pair GEMM from 129 rows on, except where this kernel splits the k range over SMs that few tiles leave idle, and in short rows whose tiles
    // all run at once: one tile's way through the pair's pipeline is longer (pair / this, us: 256 x 4096 -> 4096 18.1 / 16.0, 256 x 3072 -> 2658 14.7 /
    // 11.9, 200 x 512 -> 8192 11.7 / 10.6, 512 x 1024 -> 4096 12.7 / 12.5, 384 x 1536 -> 6272 18.8 / 14.7; 512 x 3072 -> 4096 18.8 / 19.0, f32
    // 1024 x 2048 -> 2048 14.7 / 15.4, 256 x 3072 -> 8192 16.1 / 18.6).
    const uint64_t items = uint64_t((n + 127) / 128) * ((m + 127) / 128), sms = uint64_t(sm_count);
    if (int4_gemm_pair_supported(m, n, k, group) && sm_count >= 2 && items > (k <= 1536 ? sms : sms / 2))
        return launch_int4_gemm_pair(x_bf16, w_packed, scale_bf16, y, m, n, k, group, out_f32, 0, 1, nullptr, nullptr, n, sm_count, stream, status);
    Params p = make_params(x_bf16, w_packed, scale_bf16, y, m, n, k, group, status);
    const uint32_t per = group / 64;
    if (per > 1) p.group_inv = uint32_t((0x100000000ull + per - 1) / per);
    const auto launch = [&](auto f32, auto bf16) { return out_f32 ? f32(x_bf16, w_packed, p, sm_count, stream) : bf16(x_bf16, w_packed, p, sm_count, stream); };
    if (m <= 16) return launch(launch_cfg<16, 0, true>, launch_cfg<16, 0, false>);
    if (m <= 32) return launch(launch_cfg<32, 0, true>, launch_cfg<32, 0, false>);
    return m <= 64 ? launch(launch_cfg<64, 0, true>, launch_cfg<64, 0, false>) : launch(launch_cfg<128, 0, true>, launch_cfg<128, 0, false>);
}

}  // namespace vybk
