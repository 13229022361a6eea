// vyre-libs::nn::linear_4bit_affine_grouped at size on the tensor cores, in the reference's own layout
// (vyre-libs/src/nn/linear/inner/linear_4bit.rs:357-775):
//
//   out[b, i] = bias[i] + sum_g s[g, i] * ( sum_{k in g} x[b, k] * (q[k, i] - 8)  -  (zp[g, i] - 8) * sum_{k in g} x[b, k] )
//
// words w[(k / 8) * N + i] (nibble k % 8 at bit 4 (k % 8)), f32 scales and u32 zero points [group][N], f32 activations and output.
//
// What bounds it: at decode batches the weights' bytes, then the instructions per weight. The f32 kernels of dropin_fast.cu
// spend an extraction, a subtraction and an FMA on every weight and batch row. Here a weight is unpacked once into a bf16 pair
// (q - 8 is exact) for mma.sync.m16n8k16, and the f32 activation is three bf16 numbers (24 significant bits), each a B column of
// its own. The split is exact from 2^-110 on and leaves less than 2^-133 below (its residuals keep their subnormals).
// Products are exact, sums are f32 per group; scale and zero point are applied once per group and column.
// The fragments need no shuffles: k labels inside an MMA are a dummy index, so a lane's word (8 k of one output) IS its A
// fragment of two MMAs, and the activations are staged in the matching order (one 16-byte shared load per lane and word).
// A lane loads 4 (2) neighbouring outputs of a word row, a warp four rows of 128 (64) bytes, four steps ahead.
// Measured: see launch_affine_grouped_mma.
//
// An output that does not come out below 2^64 is computed again by the definition in f32: a group sum meets its scale late, so that it
// can overflow (activations from about 1e35 on, or not finite) where the definition, which scales every weight first, does not;
// and where the definition's own product of scale and zero point overflows, the sum here is at least that large.
// Replaces, at size, the generated kernel of vyre-libs/src/nn/linear/inner/linear_4bit.rs:399-775.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "dependent_launch.cuh"
#include "kernels.h"
#include "tcgen05_common.cuh"

namespace vybk {
namespace {

constexpr int WARPS = 8, THREADS = WARPS * 32;
constexpr uint32_t XS_BYTES = 64 * 1024;  // staged activations of one k chunk

// nibbles i and i + 4 of a word -> bf16 pair q - 8 (0x43nn is 128 + nn, the subtraction is exact)
__device__ __forceinline__ uint32_t unpack_pair(uint32_t w, int i) {
    uint32_t d;
    asm("sub.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(tc::and_or(w >> (4 * i), 0x000F000Fu, 0x43004300u)), "r"(0x43084308u));
    return d;
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t bf16_bits(float v) { return uint32_t(__bfloat16_as_ushort(__float2bfloat16_rn(v))); }
__device__ __forceinline__ float from_bits(uint32_t b) { return __uint_as_float(b << 16); }
// subnormal operands and results kept (this file's own arithmetic flushes them)
__device__ __forceinline__ float sub_keep(float a, float b) {
    float d;
    asm("sub.rn.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float add_keep(float a, float b) {
    float d;
    asm("add.rn.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float fma_keep(float a, float b, float c) {
    float d;
    asm("fma.rn.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ bool ordinary(float v) { return fabsf(v) < 0x1p64f; }  // false for NaN

// One output by the definition, without its bias. Out of line: next to nothing takes it, and its loop stays off the main path's registers.
__device__ __noinline__ float by_definition(const float* x, const uint32_t* w, const float* scale,
                                            const uint32_t* zp, uint32_t in_dim, uint32_t out_dim, uint32_t group, uint32_t row, uint32_t n) {
    float v = 0.0f;
    for (uint32_t k = 0; k < in_dim; ++k) {
        const size_t at = size_t(k / group) * out_dim + n;
        const float q = float((w[size_t(k / 8) * out_dim + n] >> (4 * (k % 8))) & 15u), s = scale[at];
        v = fmaf(x[size_t(row) * in_dim + k], fmaf(q, s, -__fmul_rn(float(zp[at]), s)), v);
    }
    return v;
}

// R: 16-output MMA tiles per warp (4: a lane loads 16 bytes of a word row, 2: 8 bytes).
// NB: blocks of eight batch rows; the three parts of a block are an 8-column tile each, so a lane holds all parts of its rows.
//     NB = 0: up to two rows, row r part q in column 3 r + q of one 8-column tile.
// WK: warps of the block that share a tile of outputs and split its groups; the other WARPS / WK factors are further outputs.
template <int R, int NB, int WK>
__global__ void __launch_bounds__(THREADS, 2)
affine_grouped_mma_kernel(const float* x, const uint32_t* w, const float* scale,
                          const uint32_t* zp, const float* bias, float* out, uint32_t in_dim,
                          uint32_t out_dim, uint32_t group, uint32_t batch, uint32_t chunk) {
    constexpr uint32_t NT = NB == 0 ? 1 : 3 * NB, COLS = 8 * NT, ROWS = NB == 0 ? 2 : 8 * NB;
    constexpr uint32_t AC = NB == 0 ? 1 : NB, SUMS = 8 * AC;  // accumulators per output: columns (NB = 0) or rows
    constexpr uint32_t WN = WARPS / WK, TILE = 16 * R;        // outputs per warp tile
    constexpr uint32_t PITCH = SUMS + 1;
    constexpr int AHEAD = NB == 2 ? 2 : 4;                    // steps of weights in flight (registers: sixteen rows leave room for two)
    extern __shared__ __align__(16) uint8_t smem[];
    lets_next_start();
    waits_for_previous();
    uint4* xs = reinterpret_cast<uint4*>(smem);               // [chunk / 8][COLS]: (k0,k4) (k1,k5) (k2,k6) (k3,k7) of a column
    float* xsum = reinterpret_cast<float*>(smem + XS_BYTES);  // [groups of the chunk][SUMS]
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint32_t wk = warp % WK, wn = warp / WK;
    const uint32_t b0 = blockIdx.y * ROWS, nb = min(ROWS, batch - b0);
    const uint32_t tiles = (out_dim + TILE * WN - 1) / (TILE * WN);
    const uint32_t spg = group / 32;                          // 32-k steps per group
    const bool one_chunk = chunk >= in_dim;
    auto column = [](uint32_t r, uint32_t q) { return NB == 0 ? 3 * r + q : (r / 8) * 24 + q * 8 + r % 8; };
    // columns of a word row are permuted with it: a quarter warp reads two columns of four word rows
    auto slot = [](uint32_t kw, uint32_t col) { return kw * COLS + (col & ~7u) + ((col & 7u) ^ ((kw & 3u) << 1)); };

    // a word row of 8 k of one batch row -> its three bf16 parts in the staged order
    auto stage = [&](uint32_t k0, uint32_t kc) {
        const uint32_t kws = kc / 8;
        for (uint32_t e = threadIdx.x; e < kws * (NB == 0 ? 3 : ROWS); e += THREADS) {
            const uint32_t kw = e % kws, r = e / kws;
            uint32_t part[3][4] = {};
            if (r < nb) {
                const float4* src = reinterpret_cast<const float4*>(x + size_t(b0 + r) * in_dim + k0 + kw * 8);
                const float4 lo = src[0], hi = src[1];
                const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t p0 = bf16_bits(v[i]);
                    const float r1 = sub_keep(v[i], from_bits(p0));
                    const uint32_t p1 = bf16_bits(r1), p2 = bf16_bits(sub_keep(r1, from_bits(p1)));
                    part[0][i & 3] |= p0 << ((i >> 2) * 16);
                    part[1][i & 3] |= p1 << ((i >> 2) * 16);
                    part[2][i & 3] |= p2 << ((i >> 2) * 16);
                }
            }
#pragma unroll
            for (uint32_t q = 0; q < 3; ++q)  // rows past the batch (and the two spare columns of NB = 0) are zero
                if (column(r, q) < COLS) xs[slot(kw, column(r, q))] = make_uint4(part[q][0], part[q][1], part[q][2], part[q][3]);
        }
        __syncthreads();
        for (uint32_t e = threadIdx.x; e < (kc / group) * SUMS; e += THREADS) {
            const uint32_t c = e % SUMS, kw0 = (e / SUMS) * (group / 8);
            float sum = 0.0f;
            for (uint32_t j = 0; j < group / 8; ++j)
#pragma unroll
                for (uint32_t q = 0; q < (NB == 0 ? 1u : 3u); ++q) {
                    const uint4 v = xs[slot(kw0 + j, NB == 0 ? c : column(c, q))];
                    const uint32_t r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum = add_keep(sum, add_keep(__uint_as_float(r[i] << 16), __uint_as_float(r[i] & 0xFFFF0000u)));
                }
            xsum[e] = sum;
        }
        __syncthreads();
    };

    // where this warp reads: its outputs (MMA tile i has na + i in row g and nz + i in row g + 8) and its run of groups
    uint32_t na, nz, kw_first, steps, g_begin, kbase;
    bool in_a, in_z;
    const uint32_t* wp;
    uint32_t wa[AHEAD][R], wz[AHEAD][R];
    auto load = [&](uint32_t st, uint32_t (&a)[R], uint32_t (&z)[R]) {
        const uint32_t* row = wp + size_t(st) * 4 * out_dim;
        if constexpr (R == 4) {
            const uint4 va = st < steps && in_a ? *reinterpret_cast<const uint4*>(row + na) : make_uint4(0, 0, 0, 0);
            const uint4 vz = st < steps && in_z ? *reinterpret_cast<const uint4*>(row + nz) : make_uint4(0, 0, 0, 0);
            a[0] = va.x; a[1] = va.y; a[2] = va.z; a[3] = va.w;
            z[0] = vz.x; z[1] = vz.y; z[2] = vz.z; z[3] = vz.w;
        } else {
            const uint2 va = st < steps && in_a ? *reinterpret_cast<const uint2*>(row + na) : make_uint2(0, 0);
            const uint2 vz = st < steps && in_z ? *reinterpret_cast<const uint2*>(row + nz) : make_uint2(0, 0);
            a[0] = va.x; a[1] = va.y;
            z[0] = vz.x; z[1] = vz.y;
        }
    };
    auto aim = [&](uint32_t tile, uint32_t k0) {
        na = (tile * WN + wn) * TILE + R * g;
        nz = na + 8 * R;
        in_a = na < out_dim;  // out_dim is a multiple of 4: all of a lane's outputs or none
        in_z = nz < out_dim;
        const uint32_t gc = min(chunk, in_dim - k0) / group, per = (gc + WK - 1) / WK;
        g_begin = min(gc, wk * per);
        steps = (min(gc, g_begin + per) - g_begin) * spg;
        kw_first = g_begin * (group / 8) + t;  // inside the chunk
        kbase = k0;
        wp = w + size_t(k0 / 8 + kw_first) * out_dim;
#pragma unroll
        for (int d = 0; d < AHEAD; ++d) load(d, wa[d], wz[d]);
    };
    auto columns4 = [&](const auto* p, auto (&v)[R]) {  // R neighbouring words of a sidecar row
        if constexpr (R == 4) {
            const uint4 q = *reinterpret_cast<const uint4*>(p);
            *reinterpret_cast<uint4*>(&v) = q;
        } else {
            *reinterpret_cast<uint2*>(&v) = *reinterpret_cast<const uint2*>(p);
        }
    };
    if (one_chunk && blockIdx.x < tiles) {
        aim(blockIdx.x, 0);  // the first weights are under way while the activations are staged
        stage(0, in_dim);
    }
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        float acc[R][AC][4];
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int c = 0; c < int(AC); ++c) acc[i][c][0] = acc[i][c][1] = acc[i][c][2] = acc[i][c][3] = 0.0f;
        for (uint32_t k0 = 0; k0 < in_dim; k0 += chunk) {
            if (!one_chunk) {
                aim(tile, k0);
                __syncthreads();
                stage(k0, min(chunk, in_dim - k0));
            }
            __align__(16) float sa[R], sz[R];
            __align__(16) uint32_t za[R], zz[R];
            float d[R][NT][4];
            uint32_t in_group = 0, grp = g_begin;
            for (uint32_t st0 = 0; st0 < steps; st0 += AHEAD) {
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) {
                    const uint32_t st = st0 + u;
                    if (st >= steps) break;
                    if (in_group == 0) {
                        const size_t at = size_t(kbase / group + grp) * out_dim;
#pragma unroll
                        for (int i = 0; i < R; ++i) {
                            sa[i] = sz[i] = 0.0f;
                            za[i] = zz[i] = 0u;
#pragma unroll
                            for (int c = 0; c < int(NT); ++c) d[i][c][0] = d[i][c][1] = d[i][c][2] = d[i][c][3] = 0.0f;
                        }
                        if (in_a) {
                            columns4(scale + at + na, sa);
                            columns4(zp + at + na, za);
                        }
                        if (in_z) {
                            columns4(scale + at + nz, sz);
                            columns4(zp + at + nz, zz);
                        }
                    }
                    const uint32_t kw = kw_first + st * 4;
                    uint4 xb[NT];
#pragma unroll
                    for (int c = 0; c < int(NT); ++c) xb[c] = xs[kw * COLS + c * 8 + (g ^ ((kw & 3u) << 1))];
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        const uint32_t a = wa[u][i], z = wz[u][i];
                        const uint32_t a0 = unpack_pair(a, 0), a1 = unpack_pair(z, 0), a2 = unpack_pair(a, 1), a3 = unpack_pair(z, 1);
#pragma unroll
                        for (int c = 0; c < int(NT); ++c) mma_bf16(d[i][c], a0, a1, a2, a3, xb[c].x, xb[c].y);
                        const uint32_t e0 = unpack_pair(a, 2), e1 = unpack_pair(z, 2), e2 = unpack_pair(a, 3), e3 = unpack_pair(z, 3);
#pragma unroll
                        for (int c = 0; c < int(NT); ++c) mma_bf16(d[i][c], e0, e1, e2, e3, xb[c].z, xb[c].w);
                    }
                    load(st + AHEAD, wa[u], wz[u]);
                    if (++in_group == spg) {
                        in_group = 0;
#pragma unroll
                        for (int c = 0; c < int(AC); ++c) {
                            const float* xq = xsum + grp * SUMS + c * 8 + 2 * t;
                            const float x0 = xq[0], x1 = xq[1];
#pragma unroll
                            for (int i = 0; i < R; ++i) {
                                const float fa = 8.0f - float(za[i]), fz = 8.0f - float(zz[i]);
                                float s4[4];
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                    s4[j] = NB == 0 ? d[i][0][j] : add_keep(add_keep(d[i][(3 * c) % NT][j], d[i][(3 * c + 1) % NT][j]), d[i][(3 * c + 2) % NT][j]);
                                acc[i][c][0] = fma_keep(sa[i], fma_keep(fa, x0, s4[0]), acc[i][c][0]);
                                acc[i][c][1] = fma_keep(sa[i], fma_keep(fa, x1, s4[1]), acc[i][c][1]);
                                acc[i][c][2] = fma_keep(sz[i], fma_keep(fz, x0, s4[2]), acc[i][c][2]);
                                acc[i][c][3] = fma_keep(sz[i], fma_keep(fz, x1, s4[3]), acc[i][c][3]);
                            }
                        }
                        ++grp;
                    }
                }
            }
        }
        const uint32_t oa = na, oz = nz;
        const bool have_a = in_a, have_z = in_z;
        if (one_chunk && tile + gridDim.x < tiles) aim(tile + gridDim.x, 0);  // the next tile's first weights, under this one's stores
        if constexpr (WK == 1 && NB > 0) {
            // a lane holds whole sums: outputs oa + i and oz + i of rows 2 t, 2 t + 1 of every block of eight
            bool good = true;
            float ba[R], bz[R];  // before the stores, past which no load may move
#pragma unroll
            for (int i = 0; i < R; ++i) {
                ba[i] = have_a ? bias[oa + i] : 0.0f;
                bz[i] = have_z ? bias[oz + i] : 0.0f;
            }
#pragma unroll
            for (int c = 0; c < int(AC); ++c)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t r = c * 8 + 2 * t + (j & 1), n = j < 2 ? oa : oz;
                    if (r >= nb || !(j < 2 ? have_a : have_z)) continue;
#pragma unroll
                    for (int i = 0; i < R; ++i) {
                        out[size_t(b0 + r) * out_dim + n + i] = (j < 2 ? ba[i] : bz[i]) + acc[i][c][j];
                        good = good && ordinary(acc[i][c][j]);
                    }
                }
            if (!good)  // this lane's outputs once more
                for (uint32_t e = 0; e < 4 * R * AC; ++e) {
                    const uint32_t r = e / (4 * R) * 8 + 2 * t + (e & 1), n = (e & 2 ? oz : oa) + e / 4 % R;
                    if (r < nb && (e & 2 ? have_z : have_a))
                        out[size_t(b0 + r) * out_dim + n] = bias[n] + by_definition(x, w, scale, zp, in_dim, out_dim, group, b0 + r, n);
                }
        } else {
            // sum the k slices (and, with NB = 0, the parts) in a fixed order
            float* red = xsum + (one_chunk ? in_dim / group : chunk / group) * SUMS;  // [WARPS][TILE][PITCH]
#pragma unroll
            for (int i = 0; i < R; ++i)
#pragma unroll
                for (int c = 0; c < int(AC); ++c) {
                    float* ra = red + (warp * TILE + R * g + i) * PITCH + c * 8 + 2 * t;
                    float* rz = ra + 8 * R * PITCH;
                    ra[0] = acc[i][c][0];
                    ra[1] = acc[i][c][1];
                    rz[0] = acc[i][c][2];
                    rz[1] = acc[i][c][3];
                }
            __syncthreads();
            auto bias_of = [&](uint32_t e) {
                const uint32_t n = tile * WN * TILE + e % (WN * TILE);
                return e < WN * TILE * nb && n < out_dim ? bias[n] : 0.0f;
            };
            float next = bias_of(threadIdx.x);  // one ahead: no load moves up past a store
            for (uint32_t e = threadIdx.x; e < WN * TILE * nb; e += THREADS) {
                const uint32_t j = e % (WN * TILE), r = e / (WN * TILE), n = tile * WN * TILE + j;
                const float bn = next;
                next = bias_of(e + THREADS);
                if (n >= out_dim) continue;
                float v = 0.0f;
#pragma unroll
                for (int q = 0; q < WK; ++q) {
                    const float* p = red + (((j / TILE) * WK + q) * TILE + j % TILE) * PITCH;
                    v += NB == 0 ? (p[3 * r] + p[3 * r + 1]) + p[3 * r + 2] : p[r];
                }
                if (!ordinary(v)) v = by_definition(x, w, scale, zp, in_dim, out_dim, group, b0 + r, n);
                out[size_t(b0 + r) * out_dim + n] = bn + v;
            }
            __syncthreads();
        }
    }
}

template <int R, int NB, int WK>
cudaError_t launch_cfg(const float* x, const uint32_t* w, const float* scale, const uint32_t* zp, const float* b, float* out, uint32_t in_dim,
                       uint32_t out_dim, uint32_t group, uint32_t batch, int sm_count, cudaStream_t s) {
    constexpr uint32_t COLS = NB == 0 ? 8 : 24 * NB, ROWS = NB == 0 ? 2 : 8 * NB, SUMS = NB == 0 ? 8 : 8 * NB, OUTS = 16 * R * (WARPS / WK);
    uint32_t chunk = XS_BYTES / (2 * COLS) / group * group;  // 2 bytes a column and k
    if (chunk > in_dim) chunk = in_dim;
    const size_t smem = XS_BYTES + (size_t(chunk / group) * SUMS + (WK == 1 ? 0 : size_t(WARPS) * 16 * R * (SUMS + 1))) * 4;
    static std::atomic<uint64_t> configured{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = 1ull << (dev & 63);
    if (!(configured.load(std::memory_order_acquire) & bit)) {
        e = cudaFuncSetAttribute(affine_grouped_mma_kernel<R, NB, WK>, cudaFuncAttributeMaxDynamicSharedMemorySize, 113 * 1024);
        if (e != cudaSuccess) return e;
        configured.fetch_or(bit, std::memory_order_release);
    }
    const uint32_t tiles = (out_dim + OUTS - 1) / OUTS, rows = (batch + ROWS - 1) / ROWS;
    if (rows > 65535u) return cudaErrorInvalidValue;
    // two blocks per SM walk the tiles, so that activations are staged once
    const uint32_t fit = (2u * uint32_t(sm_count) + rows - 1) / rows, grid = tiles < fit ? tiles : fit;
    return launch_dependent(affine_grouped_mma_kernel<R, NB, WK>, dim3(grid, rows), dim3(THREADS), smem, s, x, w, scale, zp, b, out, in_dim, out_dim,
                            group, batch, chunk);
}

}  // namespace

bool affine_grouped_mma_supported(const void* x, const void* w, const void* scale, const void* zp, uint32_t in_dim, uint32_t out_dim,
                                  uint32_t group) {
    // whole 32-k steps per group, 16-byte loads along the outputs; a group's activations fit a chunk of sixteen-row blocks
    return group % 32 == 0 && group <= 512 && in_dim % group == 0 && out_dim % 4 == 0 &&
           ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(scale) | reinterpret_cast<uintptr_t>(zp)) & 15u) == 0;
}

cudaError_t launch_affine_grouped_mma(const float* x, const uint32_t* w, const float* scale, const uint32_t* zp, const float* b, float* out,
                                      uint32_t in_dim, uint32_t out_dim, uint32_t group, uint32_t batch, int sm_count, cudaStream_t s) {
    // Device time of a submission, before (f32 kernels of dropin_fast.cu) and now, group 128 (64 at k = 256 and 2048), us:
    //   1 x 4096 x 14336  31 / 23    1 x 4096 x 28672  52 / 35    2 x 4096 x 14336  39 / 25    4 x 4096 x 14336  68 / 43
    //   8 x 4096 x 14336  82 / 46   16 x 2048 x 4096   29 / 21   64 x 4096 x 4096  123 / 56  256 x 256 x 4096    29 / 19
    //   256 x 4096 x 4096 322 / 129; 1 x 512 x 40000 with group 32: 52 / 15
    // One row: 32 outputs a warp instead of 64 (27 us at 14336) and four k slices instead of eight (29 us) are slower.
    if (batch <= 2) return launch_cfg<4, 0, 8>(x, w, scale, zp, b, out, in_dim, out_dim, group, batch, sm_count, s);
    // Whole sums in one warp for sixteen rows when that gives every SM a block; else blocks of eight rows whose warps split k
    // as far as it takes to fill the SMs (a block stages its rows' activations for all of its outputs: wide blocks stage less).
    const uint64_t sms = uint64_t(sm_count), r16 = (batch + 15) / 16, r8 = (batch + 7) / 8;
    if ((out_dim + 255) / 256 * r16 >= sms) return launch_cfg<2, 2, 1>(x, w, scale, zp, b, out, in_dim, out_dim, group, batch, sm_count, s);
    if ((out_dim + 127) / 128 * r8 >= sms) return launch_cfg<2, 1, 2>(x, w, scale, zp, b, out, in_dim, out_dim, group, batch, sm_count, s);
    if ((out_dim + 63) / 64 * r8 >= sms) return launch_cfg<2, 1, 4>(x, w, scale, zp, b, out, in_dim, out_dim, group, batch, sm_count, s);
    return launch_cfg<2, 1, 8>(x, w, scale, zp, b, out, in_dim, out_dim, group, batch, sm_count, s);
}

}  // namespace vybk
