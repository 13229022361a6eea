// int4 group-quantized GEMM on CTA pairs (tcgen05 cta_group::2, sm_100a): dense prefill, grouped (per-expert) and
// grouped with a fused SwiGLU epilogue.
//
//   plain:  y[m, n]  = bf16|f32( sum_k x[m, k] * bf16((q[e(m), n, k] - 8) * s[e(m), n, k / group]) )
//   glu:    h[m, j]  = bf16( g * (u * sigmoid(g)) ),  g = bf16(x[m,:] . W1[e(m), j, :]),  u = bf16(x[m,:] . W3[e(m), j, :])
//
// Two CTAs of a cluster (one TPC) share every MMA: M = 256 WEIGHT rows, 128 in each CTA's tensor memory, N = up to 256 activation rows, half
// of them in each CTA's shared memory. The unpacked weights go from registers to tensor memory, where the MMA reads its A operand, so that
// shared memory carries the activations alone (with weights unpacked into shared memory its writes and operand reads bound this kernel).
//
// Roles per CTA (28 warps): warp 0 packed weights by TMA (256 k a stage), warp 2 activations (128 k a pass, completion counted on the LEADER's
// barrier), warp 1 tensor memory and, in the leader, the MMAs (one commit a pass to each CTA); four sets of four warps unpack, a thread per
// weight row, each set a pass in four; eight warps drain the one accumulator, half of its columns each (the unpacking of the next tile's first
// four passes lies under it).
// bf16 results pass through 64 KB of shared memory, so that the accumulator is free as soon as it is read (about 1200 cycles): with SwiGLU and 2-byte
// stores between its read and its release 4096 tokens of eight experts took 3220 us a layer, now 2700 to 2810 (2990 with the weights through shared memory).
// In glu mode lanes 0-63 of a CTA hold gate rows and lanes 64-127 the same up rows; they meet where the results pass through shared memory.
// The activation rows of a plain tile are chosen so that the tiles fill whole waves of pairs (choose_bn).
//
// What bounds it: at 2048 and more rows of wide projections the power cap (2048 x 4096 -> 14336 takes 171 us in a burst of a dozen, at 1.965 GHz, and
// 204 in a stream of sixty or more, at 1.40 to 1.45 GHz); below, the MMAs (1024 cycles a pass; unpacking takes 830 to 1500, four passes at once) and how full the
// waves of tiles are; in short rows the one accumulator, whose read and release take about as long as three passes. Measured, us in a burst, with the
// weights unpacked into shared memory / into tensor memory: 2048 x 4096 -> 14336 187 / 171, 1024 x 4096 -> 14336 152 / 94, 512 x 4096 -> 14336 90 / 51, 2048 x
// 4096 -> 4096 89 / 53, 2048 x 3072 -> 2658 118 / 30, 4096 x 4096 -> 14336 394 / 340, 4096 x 1024 -> 14336 114 / 103, 8192 x 1088 -> 14336 437 / 285 (before, a
// single-CTA kernel); 4096 x 256 -> 14336 64 / 68 and 8192 x 320 -> 14336 170 / 188 are what the one accumulator costs.
//
// Every wait is clock-bounded; on expiry the CTA raises a status word, drains and frees its TMEM. No multicast.
//
// Replaces, for large batches, the generated scalar kernel of
// vyre-libs/src/nn/linear/inner/linear_4bit.rs:399-775 and, in grouped form, the per-token expert_mlp of
// vyre-libs/src/nn/moe/expert_mlp.rs:18-150 (SwiGLU order of vyre-libs/src/nn/activation/unary.rs:79-100).
#include <cuda_bf16.h>

#include <atomic>

#include "kernels.h"
#include "tcgen05_common.cuh"

namespace vybk {
namespace {

using namespace tc;

constexpr int BM = 128;        // weight rows per CTA (256 per pair)
constexpr int MAX_BN = 256;    // activation rows per pair
constexpr int PASS = 128, KB = 256, UMMA_K = 16;
constexpr int RAW_STAGES = 4, X_STAGES = 3, SLOTS = 4, DONE = 8;
constexpr int RAW_BYTES = BM * KB / 2;               // 16 KB: two boxes of 64 rows, 128-byte swizzle
constexpr int X_BYTES = (MAX_BN / 2) * PASS * 2;     // 32 KB: this CTA's half, two boxes of 64 k
constexpr int X_RING = RAW_STAGES * RAW_BYTES, OUT = X_RING + X_STAGES * X_BYTES;
constexpr int OUT_BYTES = MAX_BN * BM * 2;           // 64 KB: a tile's sums as bf16 [activation row][weight row]
constexpr int RING_BYTES = OUT + OUT_BYTES;
constexpr int UNPACK_WARP = 4, EPI_WARP = 20, EPI_WARPS = 8, THREADS = (EPI_WARP + EPI_WARPS) * 32, MMA_WARP = 1;
constexpr int TMEM_COLS = 512, A_COL = MAX_BN;       // the accumulator, then four slots of 64 columns
constexpr int SMEM_BYTES = RING_BYTES + 1024 + 1024;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");

struct Bars {
    unsigned long long raw_full[RAW_STAGES], raw_empty[RAW_STAGES], a_full[X_STAGES], b_full[SLOTS], done[DONE];
    unsigned long long acc_full, acc_empty, dumped, stored, drained;
    uint32_t tmem_base;
    unsigned int abort_flag;
    uint32_t a_issued, raw_issued;  // copies of the TMA roles
};
static_assert(sizeof(Bars) <= 1024, "control block");

struct Params {
    const uint16_t* scales;     // bf16 [weight rows][K / group]
    void* y;                    // [rows][ldy] bf16 or f32
    const uint32_t* m_tiles_dev;  // optional: number of 256-row tiles decided on the device (grouped launches)
    const uint32_t* tile_expert;  // optional: expert of each 256-row tile
    uint32_t* status;
    uint32_t M, N, K, group;    // M: activation/output rows; N: output columns
    uint32_t bn;                // activation rows per tile
    uint32_t m_tiles, n_tiles;
    uint32_t expert_rows;       // weight rows per expert in the stacked weight tensor
    uint32_t glu_stride;        // glu: rows between W1[j] and W3[j] of one expert
    uint32_t ldy;               // output row stride in elements
    uint32_t out_f32;           // plain mode only: store f32 instead of bf16
    uint32_t group_inv;         // group / 64 > 1: (i * group_inv) >> 32 = i / (group / 64) for the 64-k blocks i of a row; else 0
};

__device__ __forceinline__ uint32_t bf16x2_mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

struct TileCoord {
    uint32_t mt, nt, expert;
};

template <bool GLU>
__global__ void __launch_bounds__(THREADS, 1)
int4_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const Params p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    Bars* bars = reinterpret_cast<Bars*>(tiles + RING_BYTES);
    volatile unsigned int* abort_flag = &bars->abort_flag;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();  // 0 = leader
    const uint32_t pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const uint32_t m_tiles = p.m_tiles_dev ? min(*p.m_tiles_dev, p.m_tiles) : p.m_tiles;
    const uint32_t total_tiles = m_tiles * p.n_tiles, stages = (p.K + KB - 1) / KB, passes = stages * (KB / PASS);
    const uint32_t half_bn = p.bn >> 1;          // activation rows in this CTA's shared memory

    auto coord = [&](uint32_t tile) {
        TileCoord c;
        c.mt = tile % m_tiles;
        c.nt = tile / m_tiles;
        c.expert = p.tile_expert ? p.tile_expert[c.mt] : 0u;
        return c;
    };
    // first output column of this CTA's weight rows (glu: of its 64 gate and 64 up rows)
    auto column0 = [&](const TileCoord& c) { return GLU ? c.nt * BM + rank * (BM / 2) : c.nt * 2 * BM + rank * BM; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < RAW_STAGES; ++s) {
            mbar_init(smem_u32(&bars->raw_full[s]), 1);
            mbar_init(smem_u32(&bars->raw_empty[s]), 8);  // the warps of a stage's two passes
        }
        for (int s = 0; s < X_STAGES; ++s) mbar_init(smem_u32(&bars->a_full[s]), 1);  // leader: one expect_tx arrival, bytes from both CTAs
        for (int s = 0; s < SLOTS; ++s) mbar_init(smem_u32(&bars->b_full[s]), 8);     // leader: four warps of each CTA
        for (int s = 0; s < DONE; ++s) mbar_init(smem_u32(&bars->done[s]), 1);        // a commit to each CTA
        mbar_init(smem_u32(&bars->acc_full), 1);
        mbar_init(smem_u32(&bars->acc_empty), 2 * EPI_WARPS);  // leader: both CTAs' epilogue warps
        mbar_init(smem_u32(&bars->dumped), EPI_WARPS);
        mbar_init(smem_u32(&bars->stored), EPI_WARPS);
        mbar_init(smem_u32(&bars->drained), 1);
        bars->abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&map_x);
        tma_prefetch_desc(&map_w);
    }
    if (warp == uint32_t(MMA_WARP)) {
        tmem_alloc_pair(smem_u32(&bars->tmem_base), TMEM_COLS);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs' barriers exist before any remote arrive, commit or TMA completion can target them
    tc_fence_after();
    const uint32_t tmem_base = bars->tmem_base;
    // passes are numbered through all tiles; nobody is further behind than the eight barriers of completed ones
    auto done_wait = [&](uint32_t gp) { return mbar_wait(smem_u32(&bars->done[gp % DONE]), (gp / DONE) & 1, abort_flag); };

    bool ok = true;
    if (warp == 0) {
        // ---- packed weights ----
        if (elect_one()) {
            uint32_t gi = 0;
            for (uint32_t tile = pair; tile < total_tiles && ok; tile += pairs) {
                const TileCoord c = coord(tile);
                const int row0 = int(c.expert * p.expert_rows + column0(c)), row1 = row0 + int(GLU ? p.glu_stride : BM / 2);
                for (uint32_t i = 0; i < stages; ++i, ++gi) {
                    const uint32_t s = gi % RAW_STAGES, bar = smem_u32(&bars->raw_full[s]), dst = smem_u32(tiles + s * RAW_BYTES);
                    if (gi >= uint32_t(RAW_STAGES) && !mbar_wait(smem_u32(&bars->raw_empty[s]), ((gi / RAW_STAGES) - 1) & 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(bar, RAW_BYTES);
                    tma_load_2d(dst, &map_w, int(i * (KB / 2)), row0, bar);
                    tma_load_2d(dst + RAW_BYTES / 2, &map_w, int(i * (KB / 2)), row1, bar);
                }
            }
            bars->raw_issued = gi;
        }
        __syncwarp();
    } else if (warp == 2) {
        // ---- activations: both CTAs' boxes count on the leader's barrier; the leader posts the expectation ----
        if (elect_one()) {
            uint32_t gp = 0;
            for (uint32_t tile = pair; tile < total_tiles && ok; tile += pairs) {
                const int m0 = int((tile % m_tiles) * p.bn + rank * half_bn);
                for (uint32_t i = 0; i < passes; ++i, ++gp) {
                    const uint32_t s = gp % X_STAGES, dst = smem_u32(tiles + X_RING + s * X_BYTES);
                    if (gp >= uint32_t(X_STAGES) && !done_wait(gp - X_STAGES)) {
                        ok = false;
                        break;
                    }
                    const uint32_t leader_bar = mapa(smem_u32(&bars->a_full[s]), 0);
                    if (rank == 0) mbar_arrive_expect_tx(smem_u32(&bars->a_full[s]), 2 * half_bn * PASS * 2);
#pragma unroll
                    for (int j = 0; j < PASS / 64; ++j) tma_load_2d_pair(dst + j * half_bn * 128, &map_x, int(i * PASS + j * 64), m0, leader_bar);
                }
            }
            bars->a_issued = gp;
        }
        __syncwarp();
    } else if (warp == uint32_t(MMA_WARP)) {
        // ---- MMA issuer (leader CTA only) ----
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = idesc_bf16_f32(2 * BM, p.bn);
            uint32_t gp = 0, local = 0, xs = 0, x_parity = 0;
            for (uint32_t tile = pair; tile < total_tiles && ok; tile += pairs, ++local) {
                if (local >= 1 && !mbar_wait(smem_u32(&bars->acc_empty), (local - 1) & 1, abort_flag)) break;
                for (uint32_t i = 0; i < passes; ++i, ++gp) {
                    const uint32_t s = gp % SLOTS, parity = (gp / SLOTS) & 1;
                    if (!mbar_wait2(smem_u32(&bars->a_full[xs]), x_parity, smem_u32(&bars->b_full[s]), parity, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a = tmem_base + A_COL + s * 64, b = smem_u32(tiles + X_RING + xs * X_BYTES);
                    const uint64_t db0 = smem_desc_sw128(b), db1 = smem_desc_sw128(b + half_bn * 128);
#pragma unroll
                    for (int k = 0; k < PASS / UMMA_K; ++k)
                        mma_f16_ts_pair(tmem_base, a + k * (UMMA_K / 2), smem_desc_advance(k < 4 ? db0 : db1, (k & 3) * UMMA_K * 2), idesc,
                                        (i | uint32_t(k)) != 0);
                    const uint32_t dn = smem_u32(&bars->done[gp % DONE]);
                    tc_commit_pair(dn);
                    tc_commit_pair(mapa(dn, 1));
                    if (++xs == uint32_t(X_STAGES)) {
                        xs = 0;
                        x_parity ^= 1;
                    }
                }
                if (ok) {
                    const uint32_t af = smem_u32(&bars->acc_full);
                    tc_commit_pair(af);
                    tc_commit_pair(mapa(af, 1));
                }
            }
            if (*abort_flag != 0) {
                tc_commit_pair(smem_u32(&bars->drained));
                mbar_settle(smem_u32(&bars->drained), 0);
            }
        }
        __syncwarp();
    } else if (warp >= uint32_t(UNPACK_WARP) && warp < uint32_t(EPI_WARP)) {
        // ---- unpack: a thread per weight row, every fourth pass ----
        const uint32_t unit = (warp - UNPACK_WARP) >> 2, quad = warp & 3, r = quad * 32 + lane, half = unit & 1;
        const uint32_t groups = p.K / p.group, dst = tmem_base + ((quad * 32) << 16) + A_COL + unit * 64;
        const uint32_t ready = mapa(smem_u32(&bars->b_full[unit]), 0);
        uint32_t tile = pair, pass = unit;
        const uint16_t* srow = nullptr;
        bool valid = false;
        auto settle_tile = [&]() {  // the tile that `pass` falls into, and this row's scales
            bool moved = srow == nullptr;
            while (pass >= passes && tile < total_tiles) {
                pass -= passes;
                tile += pairs;
                moved = true;
            }
            if (!moved || tile >= total_tiles) return;
            const TileCoord c = coord(tile);
            const uint32_t col = column0(c) + (GLU ? r % (BM / 2) : r);
            valid = col < p.N;
            srow = p.scales + size_t(c.expert * p.expert_rows + (valid ? col : 0u) + (GLU && r >= BM / 2 ? p.glu_stride : 0u)) * groups;
        };
        auto scale = [&](uint32_t b) {
            const uint32_t at = pass * 2 + b;
            return valid && at < p.K / 64 ? uint32_t(__ldg(srow + (p.group_inv ? __umulhi(at, p.group_inv) : at))) * 0x10001u : 0u;
        };
        settle_tile();
        bool more = tile < total_tiles;
        uint32_t s0 = more ? scale(0) : 0, s1 = more ? scale(1) : 0;
#pragma unroll 1
        for (uint32_t gp = unit; more; gp += 4) {
            const uint32_t c0 = s0, c1 = s1, gi = gp >> 1, s = gi % RAW_STAGES;
            pass += 4;
            settle_tile();
            more = tile < total_tiles;
            if (more) {
                s0 = scale(0);
                s1 = scale(1);
            }
            ok = mbar_wait(smem_u32(&bars->raw_full[s]), (gi / RAW_STAGES) & 1, abort_flag);
            if (gp >= uint32_t(SLOTS)) ok = ok && done_wait(gp - SLOTS);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint8_t* row = tiles + s * RAW_BYTES + r * 128;
            uint4 v[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) v[j] = lds_128(row + (((half * 4 + j) ^ (r & 7u)) << 4));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t a[16];
                const uint32_t words[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    uint32_t q[4];
                    unpack_int4_bf16(words[u], q);  // exact q - 8, natural order; one rounding of the product
#pragma unroll
                    for (int e = 0; e < 4; ++e) a[4 * u + e] = bf16x2_mul(q[e], j < 2 ? c0 : c1);
                }
                tmem_st_32x16(dst + j * 16, a);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&bars->raw_empty[s]));  // the packed bytes have been used
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(ready);
        }
    } else if (warp >= uint32_t(EPI_WARP)) {
        // ---- epilogue: a thread per weight row (output column), 16 activation rows at a time. bf16 results go to shared memory first: the accumulator
        // is free after 1200 cycles, and rounding points, SwiGLU and 128- or 256-byte stores lie under the next tile's MMAs ----
        const uint32_t quad = warp & 3, ew = warp - EPI_WARP, set = ew >> 2, taddr = tmem_base + ((quad * 32) << 16);
        const uint32_t chunks = p.bn / 16, first = set * (chunks / 2), last = first + chunks / 2;
        const uint32_t empty = mapa(smem_u32(&bars->acc_empty), 0), dumped = smem_u32(&bars->dumped), stored = smem_u32(&bars->stored);
        const bool staged = GLU || p.out_f32 == 0;
        __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(tiles + OUT);
        uint32_t local = 0;
        for (uint32_t tile = pair; tile < total_tiles && ok; tile += pairs, ++local) {
            const uint32_t mt = tile % m_tiles, m0 = mt * p.bn;
            const TileCoord c{mt, tile / m_tiles, 0};
            ok = mbar_wait(smem_u32(&bars->acc_full), local & 1, abort_flag);
            if (staged && local >= 1) ok = ok && mbar_wait(stored, (local - 1) & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t col = column0(c) + quad * 32 + lane;
            for (uint32_t cc = first; cc < last; ++cc) {
                uint32_t v[16];
                tmem_ld_32x16(taddr + cc * 16, v);
                tmem_ld_wait();
                if (staged) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) out[(cc * 16 + j) * BM + quad * 32 + lane] = __float2bfloat16_rn(__uint_as_float(v[j]));
                } else if (col < p.N) {
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (m0 + cc * 16 + j < p.M) static_cast<float*>(p.y)[size_t(m0 + cc * 16 + j) * p.ldy + col] = __uint_as_float(v[j]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(empty);
            if (!staged) continue;
            if (lane == 0) mbar_arrive(dumped);
            ok = mbar_wait(dumped, local & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            // Two activation rows a warp, eight of them read before the first is stored: a row at a time, each store behind its own read and address, took
            // 240 cycles a row (4096 x 256 -> 14336 101 us, of which the stores 50; now 68).
            __nv_bfloat16* y = static_cast<__nv_bfloat16*>(p.y);
            const uint32_t rows = min(p.bn, p.M - m0);
            constexpr uint32_t AHEAD = 4;
            if constexpr (GLU) {  // a lane: four neighbouring outputs
                const uint32_t l = lane & 15u, j = column0(c) + 4 * l;
                const bool whole = j + 3 < p.N && (p.ldy & 3u) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 7u) == 0;
                for (uint32_t t0 = 2 * ew + (lane >> 4); t0 < rows; t0 += 2 * EPI_WARPS * AHEAD) {
                    uint2 g[AHEAD], u[AHEAD];
#pragma unroll
                    for (uint32_t a = 0; a < AHEAD; ++a) {
                        const __nv_bfloat16* from = out + (t0 + 2 * EPI_WARPS * a) % MAX_BN * BM + 4 * l;  // past the rows: some row, not stored
                        g[a] = *reinterpret_cast<const uint2*>(from);
                        u[a] = *reinterpret_cast<const uint2*>(from + BM / 2);
                    }
#pragma unroll
                    for (uint32_t a = 0; a < AHEAD; ++a) {
                        const uint32_t t = t0 + 2 * EPI_WARPS * a;
                        if (t >= rows) break;
                        // same rounding points as the single-token reference ops: g and u are bf16 values, the
                        // activation is evaluated in f32 as g * (u * (1 / (1 + exp(-g)))) and stored as bf16
                        const uint32_t gw[2] = {g[a].x, g[a].y}, uw[2] = {u[a].x, u[a].y};
                        uint32_t h[2];
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const float g0 = __uint_as_float(gw[q] << 16), g1 = __uint_as_float(gw[q] & 0xFFFF0000u);
                            const float u0 = __uint_as_float(uw[q] << 16), u1 = __uint_as_float(uw[q] & 0xFFFF0000u);
                            const __nv_bfloat162 h2 = __floats2bfloat162_rn(g0 * (u0 * (1.0f / (1.0f + expf(-g0)))), g1 * (u1 * (1.0f / (1.0f + expf(-g1)))));
                            h[q] = *reinterpret_cast<const uint32_t*>(&h2);
                        }
                        __nv_bfloat16* to = y + size_t(m0 + t) * p.ldy + j;
                        if (whole) {
                            *reinterpret_cast<uint2*>(to) = make_uint2(h[0], h[1]);
                        } else {
#pragma unroll
                            for (uint32_t q = 0; q < 4; ++q)
                                if (j + q < p.N) reinterpret_cast<uint16_t*>(to)[q] = uint16_t(h[q / 2] >> (16 * (q & 1)));
                        }
                    }
                }
            } else if ((p.ldy & 7u) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15u) == 0) {  // eight
                const uint32_t l = lane & 15u, j = column0(c) + 8 * l;
                for (uint32_t t0 = 2 * ew + (lane >> 4); t0 < rows; t0 += 2 * EPI_WARPS * AHEAD) {
                    uint4 v[AHEAD];
#pragma unroll
                    for (uint32_t a = 0; a < AHEAD; ++a) v[a] = *reinterpret_cast<const uint4*>(out + (t0 + 2 * EPI_WARPS * a) % MAX_BN * BM + 8 * l);
#pragma unroll
                    for (uint32_t a = 0; a < AHEAD; ++a) {
                        const uint32_t t = t0 + 2 * EPI_WARPS * a;
                        if (t >= rows) break;
                        __nv_bfloat16* to = y + size_t(m0 + t) * p.ldy + j;
                        const uint32_t e[4] = {v[a].x, v[a].y, v[a].z, v[a].w};
                        if (j + 7 < p.N) {
                            *reinterpret_cast<uint4*>(to) = v[a];
                        } else {
#pragma unroll
                            for (uint32_t q = 0; q < 8; ++q)
                                if (j + q < p.N) reinterpret_cast<uint16_t*>(to)[q] = uint16_t(e[q / 2] >> (16 * (q & 1)));
                        }
                    }
                }
            } else {  // rows that start anywhere: a row a warp, neighbouring lanes two neighbouring outputs, and once more 64 outputs on
                const bool pairs_whole = (p.ldy & 1u) == 0 && (reinterpret_cast<uintptr_t>(p.y) & 3u) == 0;
                for (uint32_t t0 = ew; t0 < rows; t0 += EPI_WARPS * AHEAD) {
                    uint32_t v[AHEAD][2];
#pragma unroll
                    for (uint32_t a = 0; a < AHEAD; ++a) {
                        const uint32_t* from = reinterpret_cast<const uint32_t*>(out + (t0 + EPI_WARPS * a) % MAX_BN * BM) + lane;
                        v[a][0] = from[0];
                        v[a][1] = from[32];
                    }
#pragma unroll
                    for (uint32_t a = 0; a < AHEAD; ++a) {
                        const uint32_t t = t0 + EPI_WARPS * a;
                        if (t >= rows) break;
#pragma unroll
                        for (uint32_t h = 0; h < 2; ++h) {
                            const uint32_t j = column0(c) + 64 * h + 2 * lane;
                            __nv_bfloat16* to = y + size_t(m0 + t) * p.ldy + j;
                            if (pairs_whole && j + 1 < p.N) {
                                *reinterpret_cast<uint32_t*>(to) = v[a][h];
                            } else {
                                if (j < p.N) reinterpret_cast<uint16_t*>(to)[0] = uint16_t(v[a][h]);
                                if (j + 1 < p.N) reinterpret_cast<uint16_t*>(to)[1] = uint16_t(v[a][h] >> 16);
                            }
                        }
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(stored);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && bars->abort_flag != 0) {
        settle_copies(bars->raw_full, RAW_STAGES, bars->raw_issued);
        if (rank == 0) settle_copies(bars->a_full, X_STAGES, bars->a_issued);  // the leader's count both CTAs' boxes; the pair leaves together
    }
    __syncwarp();
    cluster_sync();  // the peer may still be reading this CTA's shared memory / TMEM through the pair MMA until here
    if (warp == uint32_t(MMA_WARP)) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, TMEM_COLS);
    }
    if (threadIdx.x == 0 && bars->abort_flag != 0 && p.status) atomicOr(p.status, 16u);
}

}  // namespace

bool int4_gemm_pair_supported(uint32_t m, uint32_t n, uint32_t k, uint32_t group) {
    // 64-k blocks must not straddle a scale group. Weights are fetched 256 k at a time; past the row's end copies and scales are zeros.
    return m > 128 && n >= 1 && k >= 64 && k % 64 == 0 && group >= 64 && group % 64 == 0 && k % group == 0;
}

namespace {

// Activation rows of a plain tile: what makes the waves of pairs shortest, a tile's time being its rows and about 24 rows' worth of epilogue (us at 128,
// 160, 192, 224 and 256 rows, * what is taken: 2048 x 4096 -> 14336 187 / 171* / 173 / 175 / 169, 1024 x 4096 -> 14336 110 / 119 / 112 / 99* / 113, 512 x 4096 -> 14336
// 73 / 82 / 74 / 84 / 62*, 2048 x 4096 -> 4096 74 / 69* / 78 / 91 / 68, 2048 x 3072 -> 2658 53 / 49* / 53 / 60 / 63, 300 x 4096 -> 8192 39 / 30* / 35 / 37 / 37, 1400 x 7168 -> 10000
// 151* / 143 / 155 / 148 / 162, 2048 x 1024 -> 14336 71 / 68* / 72 / 65 / 64)
uint32_t choose_bn(uint32_t m, uint32_t n_tiles, uint32_t pairs) {
    uint32_t best = MAX_BN;
    uint64_t cost = ~0ull;
    for (uint32_t bn = MAX_BN; bn >= 128; bn -= 32) {
        const uint64_t t = uint64_t((m + bn - 1) / bn) * n_tiles, c = (t + pairs - 1) / pairs * (bn + 24);
        if (c < cost) {
            cost = c;
            best = bn;
        }
    }
    return best;
}

}  // namespace

cudaError_t launch_int4_gemm_pair(const void* x_bf16, const void* w_packed, const void* scale_bf16, void* y, uint32_t m,
                                  uint32_t n, uint32_t k, uint32_t group, uint32_t out_f32, uint32_t glu, uint32_t experts,
                                  const uint32_t* tile_expert, const uint32_t* m_tiles_dev, uint32_t ldy, int sm_count,
                                  cudaStream_t stream, uint32_t* status) {
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load() & bit)) {
        e = cudaFuncSetAttribute(int4_gemm_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(int4_gemm_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return e;
        configured.fetch_or(bit);
    }
    if (experts == 0) experts = 1;
    const uint32_t pairs_avail = uint32_t(sm_count) / 2;
    if (pairs_avail == 0) return cudaErrorInvalidConfiguration;
    Params p{};
    const uint32_t cols = glu ? BM : 2 * BM;
    p.n_tiles = (n + cols - 1) / cols;
    p.bn = tile_expert || glu ? uint32_t(MAX_BN) : choose_bn(m, p.n_tiles, pairs_avail);  // grouped: the segments' 256-row tiles
    p.m_tiles = (m + p.bn - 1) / p.bn;
    p.scales = static_cast<const uint16_t*>(scale_bf16);
    p.y = y;
    p.m_tiles_dev = m_tiles_dev;
    p.tile_expert = tile_expert;
    p.status = status;
    p.M = m;
    p.N = n;
    p.K = k;
    p.group = group;
    p.expert_rows = glu ? 2 * n : n;
    p.glu_stride = n;
    p.ldy = ldy;
    p.out_f32 = out_f32;
    const uint32_t per = group / 64;
    p.group_inv = per > 1 ? uint32_t((0x100000000ull + per - 1) / per) : 0u;
    const uint64_t weight_rows = uint64_t(experts) * p.expert_rows;
    CUtensorMap mx, mw;
    if (!encode_tensor_map_2d(&mx, x_bf16, m, k, 2, p.bn / 2, 64, true) ||
        !encode_tensor_map_2d(&mw, w_packed, weight_rows, k / 2, 1, BM / 2, KB / 2, true))
        return cudaErrorInvalidValue;
    const uint64_t tiles = uint64_t(p.m_tiles) * p.n_tiles;
    const uint32_t pairs = tiles < pairs_avail ? uint32_t(tiles) : pairs_avail;

    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (glu)
        e = cudaLaunchKernelEx(&cfg, int4_gemm_pair_kernel<true>, mx, mw, p);
    else
        e = cudaLaunchKernelEx(&cfg, int4_gemm_pair_kernel<false>, mx, mw, p);
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace vybk
