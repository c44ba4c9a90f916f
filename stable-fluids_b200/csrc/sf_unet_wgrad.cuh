// sf_unet_wgrad.cuh -- weight gradient of a 3x3x3 convolution of the warm-start
// network, all 27 taps from one pass over the activations.
//
//   dw[tap][co][ci] += sum_v dout[v][co] * in[v + off(tap)][ci],   db[co] += sum_v dout[v][co]
//
// A CTA owns 16 input channels and walks tiles of TX x TY x TZ voxels. The TMA
// brings a tile's dout and the halo of `in` into shared memory as 8-channel
// chunks of 16-byte rows, one row a voxel (out-of-grid voxels as zeros: the
// convolution's padding), two tiles in flight. What a tile has past the grid is
// left out, or meets zeros on both sides where a block of 16 reaches past it:
// dout's zeros alone would make NaN of an infinity in the halo. Per tap the tile is a GEMM with M = 16 output channels,
// N = 16 input channels and K = its voxels, 16 consecutive x at a time; the
// tap's shift is an offset of whole rows. Both operands lie K-major in rows of
// channels, which is what ldmatrix.trans turns into mma.sync fragments.
// Warp w owns the taps of one dz (w % 3) and either a tile of 16 output
// channels or, where there are fewer tiles than warps, a share of the voxels;
// its 9 taps x 16 x 16 accumulators stay in registers over all its tiles, and
// a CTA adds its sums to dw once, at the end.
//
// Why mma.sync and not tcgen05: the GEMM is 16 x 16 (up to 64 x 96) and its
// depth is the voxels. tcgen05.mma has M = 64 at least, so a 16-channel layer
// fills a quarter of it, and it reads its operands from shared memory for
// every instruction: a tap's 16 voxels cost at least 2.5 KB of operand reads
// for 8 KFLOP, against 0.5 KB here, where the dout fragment is loaded once for
// nine taps. What it replaces (one tap a CTA, tcgen05 with M = 128, each
// activation read 27 times from L2) ran at 7 TFLOP/s.
//
// What bounds it: shared memory reads (10 ldmatrix.x4 for 18 MMAs; the tensor
// pipe is busy half the time in a 64-channel layer at 32^3, 33 us). The bias is
// summed from the dout fragments on the FP32 units, to nearest: as MMAs with
// ones a 64-channel sum over 64 x 32 x 64 voxels was short by 5.2e-6, now 2.6e-7.
//
// The layers of 16 output channels (the full grid) take k_conv3d_wgrad_chain
// instead. The tensor cores add their products to an FP32 accumulator rounded
// towards zero, so a sum over many voxels is short of the exact one by an
// amount that grows with the number of MMAs in the chain, at 128^3 by 6e-4 of
// the sum; shorter chains, as above, would give these layers other sums than
// they have given so far, by that much (the smaller layers' change by 5e-5 at
// most). The chain kernel keeps the order of the sums: K runs over the voxels
// in memory order in blocks of 16, in as many segments as before (one wave of
// one CTA a tap: five), and mma.sync accumulates with the bits of tcgen05.mma.
// The work is split by taps (a CTA owns the three dx taps of one (dz, dy), 16
// input channels and one segment), and the layers, which do not depend on each
// other, share one launch: 0.93 ms a layer one after the other, 1.8 ms for all
// five together. What bounds it is filling shared memory: each of the nine CTAs
// of a group brings its whole dout and in again, 8.5 GB from L2 at 128^3, 4.7
// TB/s. The chains of 26,215 dependent MMAs leave room (70 cycles a block of 16
// voxels, 20 of them the MMA's latency; the tensor pipe is busy 0.32 of the time).
//
// The whole gradient of a 128^3 pair: 26.0 -> 4.0 ms (2.8 with short chains
// everywhere, which changes the sums).
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "sf_types.h"
#include "sf_unet_tc.cuh"

namespace sfb::net::wg {

constexpr int TX = 32, TY = 8;
constexpr int kThreads = 384;  // 12 warps: 3 dz x (output channel tiles x shares of the voxels)

template <int COUT>
struct Cfg {
    static constexpr int MT = COUT / 16;                 // tiles of 16 output channels
    static constexpr int SPLIT = 4 / MT;                 // shares of a tile's voxels
    static constexpr int TZ = 2;
    static constexpr int IN_CHUNK = (TX + 2) * (TY + 2) * (TZ + 2) * 16;
    static constexpr int OUT_CHUNK = TX * TY * TZ * 16;
    static constexpr int STAGE = 2 * IN_CHUNK + COUT / 8 * OUT_CHUNK;
    static constexpr int ZERO = 2 * STAGE;               // rows of zeros, as far as the taps of one row reach
    static constexpr int BAR_OFF = ZERO + (2 * (TX + 2) + 2 + 1) * 16;  // full[2], abort flag
    static constexpr int BYTES = BAR_OFF + 32;
    static_assert(COUT == 32 || COUT == 64, "output channels");
    static_assert(IN_CHUNK % 128 == 0 && OUT_CHUNK % 128 == 0 && BYTES <= 232448, "shared memory");
    static_assert(SPLIT == 1 || 3 * MT * (SPLIT - 1) * 32 * 74 * 4 <= 2 * STAGE, "the reduction over the shares reuses the stages");
};

struct Args {
    float* dw;      // [27][COUT][cin]
    float* db;      // COUT
    int cin;        // input channels of the layer (16 a CTA: blockIdx.y)
    int tiles_x, tiles_y, tiles;
    Dims d;
    unsigned* error;
};

__device__ __forceinline__ void ldmatrix4_trans(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// map_in: (channel, x, y, z) boxes of 8 x (TX + 2) x (TY + 2) x (TZ + 2);
// map_out: boxes of 8 x TX x TY x TZ.
template <int COUT>
__global__ void __launch_bounds__(kThreads, 1) k_conv3d_wgrad(const __grid_constant__ CUtensorMap map_in, const __grid_constant__ CUtensorMap map_out, Args a) {
    using C = Cfg<COUT>;
    constexpr int TZ = C::TZ, SPLIT = C::SPLIT, PX = TX + 2, PY = TY + 2;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31;
    const uint32_t base = tc::smem_u32(smem);
    const auto full = [&](int s) { return base + static_cast<uint32_t>(C::BAR_OFF + 8 * s); };
    volatile int* abort = reinterpret_cast<volatile int*>(smem + C::BAR_OFF + 16);
    if (tid == 0) {
        tc::mbar_init(full(0), 1);
        tc::mbar_init(full(1), 1);
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < (C::BAR_OFF - C::ZERO) / 16; i += kThreads) *reinterpret_cast<uint4*>(smem + C::ZERO + 16 * i) = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const int c0 = 16 * static_cast<int>(blockIdx.y);
    const int mine = a.tiles > static_cast<int>(blockIdx.x) ? (a.tiles - 1 - static_cast<int>(blockIdx.x)) / static_cast<int>(gridDim.x) + 1 : 0;
    const auto corner = [&](int k) {  // of tile k of this CTA
        const int tile = static_cast<int>(blockIdx.x) + k * static_cast<int>(gridDim.x);
        return make_int3(tile % a.tiles_x * TX, tile / a.tiles_x % a.tiles_y * TY, tile / (a.tiles_x * a.tiles_y) * TZ);
    };
    const auto load = [&](int k) {  // tile k into stage k & 1 (one thread)
        const auto [x, y, z] = corner(k);
        const uint32_t st = base + static_cast<uint32_t>((k & 1) * C::STAGE), bar = full(k & 1);
        tc::mbar_expect_tx(bar, static_cast<uint32_t>(C::STAGE));
        for (int c = 0; c < 2; ++c) tc::tma_load_4d(st + static_cast<uint32_t>(c * C::IN_CHUNK), &map_in, c0 + 8 * c, x - 1, y - 1, z - 1, bar);
        for (int c = 0; c < COUT / 8; ++c) tc::tma_load_4d(st + static_cast<uint32_t>(2 * C::IN_CHUNK + c * C::OUT_CHUNK), &map_out, 8 * c, x, y, z, bar);
    };
    if (tid == 0) {
        if (mine > 0) load(0);
        if (mine > 1) load(1);
    }
    const int dz = warp % 3, mt = warp / 3 % C::MT, share = warp / (3 * C::MT);
    const bool bias = dz == 1 && blockIdx.y == 0;  // these warps sum dout itself, too
    float acc[9][2][4], sum[2];  // sum: of dout, rows lane / 4 and lane / 4 + 8 of the tile's 16 channels
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[t][n][i] = 0.0f;
    sum[0] = sum[1] = 0.0f;
    // lane l gives ldmatrix the address of row l % 8 of matrix l / 8: for A
    // (dout) the matrices are (chunk 0, k 0-7), (chunk 1, k 0-7), (chunk 0,
    // k 8-15), (chunk 1, k 8-15); for B (in) chunk and k change places
    const uint32_t lane_a = static_cast<uint32_t>(((lane >> 3) & 1) * C::OUT_CHUNK + (((lane >> 4) & 1) * 8 + (lane & 7)) * 16);
    const int voxel = ((lane >> 3) & 1) * 8 + (lane & 7);  // of a block of 16: the row whose address this lane gives for B
    const uint32_t lane_b = static_cast<uint32_t>(((lane >> 4) & 1) * C::IN_CHUNK + voxel * 16);
    for (int k = 0; k < mine; ++k) {
        const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(full(k & 1), static_cast<uint32_t>((k >> 1) & 1), abort, a.error));
        const uint32_t st = base + static_cast<uint32_t>((k & 1) * C::STAGE);
        const uint32_t out = st + static_cast<uint32_t>(2 * C::IN_CHUNK + 2 * mt * C::OUT_CHUNK) + lane_a;
        const uint32_t in = st + static_cast<uint32_t>(dz * PY * PX * 16) + lane_b;
        const int3 at = corner(k);
        const int x_end = a.d.nx - at.x, y_end = a.d.ny - at.y, z_end = a.d.nz - at.z;  // of the grid, seen from the tile
        // rows (z, y) of the tile, this warp's share of them
#pragma unroll 1
        for (int r = share * (TY * TZ / SPLIT); ok && r < (share + 1) * (TY * TZ / SPLIT); ++r) {
            if (r % TY >= y_end || r / TY >= z_end) continue;
            const uint32_t row_out = out + static_cast<uint32_t>(r * TX * 16);
            const uint32_t row_in = in + static_cast<uint32_t>((r / TY * PY + r % TY) * PX * 16);
#pragma unroll
            for (int h = 0; h < TX / 16; ++h) {
                if (16 * h >= x_end) break;
                const uint32_t in_h = 16 * h + voxel < x_end ? row_in + static_cast<uint32_t>(h * 256) : base + static_cast<uint32_t>(C::ZERO);
                uint32_t fa[4];
                ldmatrix4_trans(row_out + static_cast<uint32_t>(h * 256), fa);
                if (bias) {  // FP32 sums: the tensor cores would round theirs towards zero
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum[i & 1] += __uint_as_float(fa[i] << 16) + __uint_as_float(fa[i] & 0xffff0000u);
                }
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    uint32_t fb[4];
                    ldmatrix4_trans(in_h + static_cast<uint32_t>((t / 3 * PX + t % 3) * 16), fb);
                    mma_16816(acc[t][0], fa, fb[0], fb[1]);
                    mma_16816(acc[t][1], fa, fb[2], fb[3]);
                }
            }
        }
        __syncthreads();  // the stage is free
        if (tid == 0 && k + 2 < mine && !*abort) load(k + 2);
    }
    if (*abort) {  // a wait gave up: nothing is added, and copies still under way land before the CTA leaves
        __nanosleep(1000000);
        return;
    }
    // the shares' sums into the first share's registers, through shared memory
    if constexpr (SPLIT > 1) {
        float* const part = reinterpret_cast<float*>(smem);
        __syncthreads();
        if (share > 0) {
            float* const p = part + (((share - 1) * 3 * C::MT + mt * 3 + dz) * 74) * 32 + lane;
#pragma unroll
            for (int t = 0; t < 9; ++t)
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) p[(t * 8 + n * 4 + i) * 32] = acc[t][n][i];
            p[72 * 32] = sum[0];
            p[73 * 32] = sum[1];
        }
        __syncthreads();
        if (share > 0) return;
        for (int s = 0; s < SPLIT - 1; ++s) {
            const float* const p = part + ((s * 3 * C::MT + mt * 3 + dz) * 74) * 32 + lane;
#pragma unroll
            for (int t = 0; t < 9; ++t)
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[t][n][i] += p[(t * 8 + n * 4 + i) * 32];
            sum[0] += p[72 * 32];
            sum[1] += p[73 * 32];
        }
    }
    if (mine == 0) return;
    const int co = 16 * mt + (lane >> 2), ci = c0 + 2 * (lane & 3);
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            float* const w = a.dw + (static_cast<size_t>(dz * 9 + t) * COUT + co) * a.cin + ci + 8 * n;
            atomicAdd(w, acc[t][n][0]);
            atomicAdd(w + 1, acc[t][n][1]);
            atomicAdd(w + 8 * a.cin, acc[t][n][2]);
            atomicAdd(w + 8 * a.cin + 1, acc[t][n][3]);
        }
    if (bias) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {  // over the four lanes of a row
            sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 1);
            sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 2);
            if ((lane & 3) == 0) atomicAdd(a.db + co + 8 * i, sum[i]);
        }
    }
}

// ---- the chain kernel (16 output channels) ---------------------------------
constexpr int kSegmentUnit = 128;   // segments are whole multiples of this many voxels
constexpr int kChunk = 512;         // voxels a stage
constexpr int kChainStages = 2;  // 68 KB: three CTAs fit an SM, so that the layers' 315 CTAs are one wave
constexpr int kHelpers = 160;       // threads that write the voxels' flags (the first of them starts the copies)
constexpr int kChainThreads = 3 * 32 + kHelpers + 32;  // a warp a tap, the helpers, the bias

struct ChainCfg {
    static constexpr int BOX = 256;                      // voxels of a TMA box: rows of 16 channels, 32 bytes
    static constexpr int OUT = kChunk * 32;
    static constexpr int IN = (kChunk + 8) * 32;         // one voxel more on each side, for the dx taps
    static constexpr int FLAGS = OUT + IN;
    static constexpr int STAGE = FLAGS + kChunk;         // a byte a voxel, [voxel % 16][voxel / 16]: bit dx + 1 set where the tap's voxel is in the grid
    static constexpr int ZERO = kChainStages * STAGE;    // a row of zeros, for the voxels outside
    static constexpr int BAR_OFF = ZERO + 16;            // full[], abort flag
    static constexpr int BYTES = BAR_OFF + 8 * kChainStages + 8;
    static_assert(OUT % 256 == 0 && IN % 256 == 0 && STAGE % 256 == 0 && kChunk == 2 * BOX, "the swizzle repeats every 256 bytes");
};

// 16 input channels of one layer. The maps view a tensor as (channel, voxel);
// boxes of 16 channels x 256 (in, out) or 8 (rest, the end of a chunk's `in`)
// voxels, 32-byte swizzle: the 16 bytes of channels 0-7 and 8-15 change places
// in rows 4-7 of every 8, so that the 8 rows of an ldmatrix lie in 8 different
// bank groups whichever row is the first.
struct ChainGroup {
    CUtensorMap in, rest, out;
    float* dw;                  // [27][16][cin]
    float* db;                  // null: another group of the layer sums the bias
    int cin, c0;
};

constexpr int kChainGroups = 7;  // all layers of 16 output channels

struct ChainArgs {
    ChainGroup group[kChainGroups];
    Dims d;
    int nvox, segment;          // voxels in all and a segment
    unsigned* error;
};

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar) : "memory");
}

// blockIdx: x the segment, y (dz + 1) * 3 + dy + 1, z the group.
__global__ void __launch_bounds__(kChainThreads) k_conv3d_wgrad_chain(const __grid_constant__ ChainArgs a) {
    using C = ChainCfg;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31;
    const uint32_t base = tc::smem_u32(smem);
    const auto full = [&](int i) { return base + static_cast<uint32_t>(C::BAR_OFF + 8 * (i % kChainStages)); };
    volatile int* abort = reinterpret_cast<volatile int*>(smem + C::BAR_OFF + 8 * kChainStages);
    const int dz = static_cast<int>(blockIdx.y) / 3 - 1, dy = static_cast<int>(blockIdx.y) % 3 - 1;
    const ChainGroup& g = a.group[blockIdx.z];
    const bool bias = dz == 0 && dy == 0 && g.db != nullptr;
    const int v_first = static_cast<int>(blockIdx.x) * a.segment, v_end = min(v_first + a.segment, a.nvox);
    const int n = (v_end - v_first + kChunk - 1) / kChunk;
    if (tid == 0) {
        for (int s = 0; s < kChainStages; ++s) tc::mbar_init(full(s), 1);
        *abort = 0;
        *reinterpret_cast<uint4*>(smem + C::ZERO) = make_uint4(0, 0, 0, 0);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    // chunk i: its copies (voxels outside the tensor as zeros), its flags
    const int shift = (dz * a.d.ny + dy) * a.d.nx - 1;
    const auto load = [&](int i) {
        const int t = tid - 96, v0 = v_first + i * kChunk;
        const uint32_t stage = static_cast<uint32_t>(i % kChainStages * C::STAGE), st = base + stage;
        if (t == 0) {
            tc::mbar_expect_tx(full(i), static_cast<uint32_t>(C::OUT + C::IN));
            for (int h = 0; h < 2; ++h) {
                tma_load_2d(st + static_cast<uint32_t>(h * C::BOX * 32), &g.out, 0, v0 + h * C::BOX, full(i));
                tma_load_2d(st + static_cast<uint32_t>(C::OUT + h * C::BOX * 32), &g.in, g.c0, v0 + shift + h * C::BOX, full(i));
            }
            tma_load_2d(st + static_cast<uint32_t>(C::OUT + kChunk * 32), &g.rest, g.c0, v0 + shift + kChunk, full(i));
        }
        for (int q = t; q < kChunk; q += kHelpers) {
            const unsigned v = static_cast<unsigned>(v0 + q), r = v / static_cast<unsigned>(a.d.nx);
            const int x = static_cast<int>(v - r * static_cast<unsigned>(a.d.nx)), z = static_cast<int>(r / static_cast<unsigned>(a.d.ny)), y = static_cast<int>(r) - z * a.d.ny;
            const bool row = static_cast<int>(v) < v_end && static_cast<unsigned>(y + dy) < static_cast<unsigned>(a.d.ny) && static_cast<unsigned>(z + dz) < static_cast<unsigned>(a.d.nz);
            smem[stage + C::FLAGS + (q & 15) * (kChunk / 16) + (q >> 4)] = static_cast<unsigned char>(row ? (x > 0 ? 1 : 0) | 2 | (x < a.d.nx - 1 ? 4 : 0) : 0);
        }
    };
    const bool helps = warp >= 3 && warp < 3 + kHelpers / 32;
    if (helps) load(0);
    __syncthreads();

    float acc[2][4], sum[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j >> 2][j & 3] = sum[j] = 0.0f;
    // lane l points at row l % 8 of ldmatrix's matrix l / 8: for A (dout) the
    // matrices are (channels 0-7, voxels 0-7), (8-15, 0-7), (0-7, 8-15), (8-15,
    // 8-15) of a block of 16 voxels; for B (in) channels and voxels change
    // places. A block is 512 bytes: the swizzle is the same in every block.
    const auto at = [](int row, int half) { return static_cast<uint32_t>(row * 32 + ((half ^ (row >> 2)) & 1) * 16); };
    const uint32_t lane_a = at(((lane >> 4) & 1) * 8 + (lane & 7), (lane >> 3) & 1);
    const int voxel = ((lane >> 3) & 1) * 8 + (lane & 7);
    const uint32_t lane_b = static_cast<uint32_t>(C::OUT) + at(voxel + warp, lane >> 4);
    const uint32_t zero = base + C::ZERO;
    bool ok = true;
    for (int i = 0; i < n; ++i) {
        const unsigned char* const stage = smem + i % kChainStages * C::STAGE;
        const uint32_t st = base + static_cast<uint32_t>(i % kChainStages * C::STAGE);
        if (helps) {
            if (i + 1 < n && !*abort) load(i + 1);  // into the stage of chunk i - 1
        } else if (warp < 3) {
            // the tap (dz, dy, warp - 1): one chain of MMAs per accumulator,
            // each block's operands fetched before the MMAs of the one before
            ok = ok && tc::mbar_wait(full(i), static_cast<uint32_t>((i / kChainStages) & 1), abort, a.error);
            const uint4* const f = reinterpret_cast<const uint4*>(stage + C::FLAGS + voxel * (kChunk / 16));
            const uint4 f0 = f[0], f1 = f[1];
            const uint32_t flags[8] = {f0.x >> warp, f0.y >> warp, f0.z >> warp, f0.w >> warp, f1.x >> warp, f1.y >> warp, f1.z >> warp, f1.w >> warp};
            uint32_t fa[2][4], fb[2][4];
            const auto fetch = [&](int k) {
                ldmatrix4_trans(st + lane_a + static_cast<uint32_t>(k * 512), fa[k & 1]);
                ldmatrix4_trans(flags[k >> 2] & (1u << (8 * (k & 3))) ? st + lane_b + static_cast<uint32_t>(k * 512) : zero, fb[k & 1]);
            };
            const int blocks = (v_end - v_first - i * kChunk + 15) / 16;  // of this segment; past it lies another's dout
            if (blocks >= kChunk / 16) {
                fetch(0);
#pragma unroll
                for (int k = 0; k < kChunk / 16; ++k) {
                    if (k + 1 < kChunk / 16) fetch(k + 1);
                    mma_16816(acc[0], fa[k & 1], fb[k & 1][0], fb[k & 1][1]);
                    mma_16816(acc[1], fa[k & 1], fb[k & 1][2], fb[k & 1][3]);
                }
            } else {
#pragma unroll 1
                for (int k = 0; k < blocks; ++k) {
                    const unsigned flag = stage[C::FLAGS + voxel * (kChunk / 16) + k];
                    ldmatrix4_trans(st + lane_a + static_cast<uint32_t>(k * 512), fa[0]);
                    ldmatrix4_trans((flag >> warp) & 1u ? st + lane_b + static_cast<uint32_t>(k * 512) : zero, fb[0]);
                    mma_16816(acc[0], fa[0], fb[0][0], fb[0][1]);
                    mma_16816(acc[1], fa[0], fb[0][2], fb[0][3]);
                }
            }
        } else if (bias) {
            // FP32 sums of dout, 8 channels of every 16th voxel a lane
            ok = ok && tc::mbar_wait(full(i), static_cast<uint32_t>((i / kChainStages) & 1), abort, a.error);
            const int rows = v_end - v_first - i * kChunk - (lane & 15);  // of this lane's, to the segment's end
            const unsigned char* const row = stage + at(lane & 15, lane >> 4);
#pragma unroll 8
            for (int k = 0; k < kChunk / 16; ++k) {
                const uint4 q = 16 * k < rows ? *reinterpret_cast<const uint4*>(row + 512 * k) : make_uint4(0, 0, 0, 0);
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    sum[2 * j] += __uint_as_float(w[j] << 16);
                    sum[2 * j + 1] += __uint_as_float(w[j] & 0xffff0000u);
                }
            }
        }
        __syncthreads();
    }
    if (*abort) {  // as in k_conv3d_wgrad
        __nanosleep(1000000);
        return;
    }
    if (warp < 3) {
        const int tap = static_cast<int>(blockIdx.y) * 3 + warp, co = lane >> 2, ci = g.c0 + 2 * (lane & 3);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            float* const w = g.dw + (static_cast<size_t>(tap) * 16 + co) * g.cin + ci + 8 * j;
            atomicAdd(w, acc[j][0]);
            atomicAdd(w + 1, acc[j][1]);
            atomicAdd(w + 8 * g.cin, acc[j][2]);
            atomicAdd(w + 8 * g.cin + 1, acc[j][3]);
        }
    } else if (!helps && bias) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum[j] += __shfl_down_sync(0xffffffffu, sum[j], o);
            if ((lane & 15) == 0) atomicAdd(g.db + (lane >> 4) * 8 + j, sum[j]);
        }
    }
}

}  // namespace sfb::net::wg
