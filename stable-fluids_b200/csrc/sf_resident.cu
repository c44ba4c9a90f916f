// sf_resident.cu -- whole 7-point solves of small grids in one launch, the
// iterate and the right-hand side resident in the shared memory of one thread
// block cluster.
//
// A small grid's solve is bound by launches: at 64^3 a colour launch moves
// 1.6 MB, a fraction of a microsecond of L2 traffic, but costs 4.3 us between
// the launches around it (1.5 us where three simulations share the device), and
// a step has some 250 of them. Here one cluster of up to 16 CTAs owns a solve
// from the first read of its right-hand side to the last write of the result:
// each CTA holds a block of rows (y, z) of the grid, boundary values travel to
// the neighbouring CTAs' shared memory by asynchronous stores that count their
// bytes on the receiver's mbarrier, and a CTA starts its next half-sweep when
// its neighbours' values are in (a cluster barrier per half-sweep instead cost
// 0.2 us more). The three velocity components are three clusters of one launch.
//
// A half-sweep takes 0.87 us at 32^3 (16 CTAs) and 1.87 us at 64^3. What bounds
// it is its chain (shared memory loads, the sums, the division, two CTA
// barriers, some 0.2 us until the neighbours' values are in) and, from 64^3 on,
// shared memory traffic, 58 % of the cycles. A step alone: 1.00 -> 0.19 ms at
// 32^3, 1.13 -> 0.38 ms at 64^3, 1.58 -> 0.51 ms at 181x47x29; three of them at
// once, each: 358 -> 64, 430 -> 138, 813 -> 181 us. Two rows a thread (fewer
// loads) lost to one (more warps): 98 against 88 us for the 64^3 diffusion.
//
// Layout. Both colours of the iterate are kept apart as in the colour-split
// solve (k_rb_half): row (y, z) of colour c holds the cells x = 2k + s,
// s = (y + z + c) & 1, at k = 0 .. count - 1, so an update reads whole float4s
// of the other colour. Rows carry one pad at each end, and the block one pad
// row on each side in y and z. A pad holds what the update beside it has to
// read: at a non-periodic face the ghost value of the face cell (a function of
// that cell, which is the only one to read it), elsewhere the neighbour's
// value. After a half-sweep a short pass over the block's edges writes the pads
// that depend on the new values, its own or the neighbours', so that the update
// itself has no branches for faces (with the pads written where the cells are
// updated a half-sweep at 64^3 took 2.6 us). A cell's ghost lives in
// the other colour's array, the one its update reads.
//
// Waits are bounded. A thread whose wait gives up sets the error word, tells the
// cluster, and sends and waits no more; the others give up at their next wait.
// Whether one did is known to all of them after the last cluster barrier, and
// then none writes its block of the result.
//
// Values, order of the sums, division and rounding are those of k_rb_half and
// k_jacobi_vec4 (BF16 storage: rounded to BF16 at every update), so the result
// has the same bits.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "sf_device.cuh"
#include "sf_divide.cuh"
#include "sf_f32x2.cuh"
#include "sf_launch.h"
#include "sf_per_device.h"
#include "sf_stencil_tb.cuh"
#include "sf_stencil_wave.cuh"

namespace sfb {

GhostRule make_ghost_rule(int kind, const FlowBC& fb, const ScalarBC& sb);

namespace {

constexpr int kResidentThreads = 512;
constexpr int kResidentShared = 232448;  // most shared memory of a CTA
// A cluster is doubled (up to 16 CTAs) until a CTA holds at most this many
// float4s of a colour: at 32^3 a pressure half-sweep takes 0.87 us with 256 a
// CTA (16 CTAs), 1.11 with 512 and 1.66 with 1024.
constexpr int kResidentItems = 256;
constexpr int kMaxSolves = 3;  // one launch: the three velocity components

struct ResidentArgs {
    void* x[kMaxSolves];        // result (and start, INIT_FROM_X)
    const void* b[kMaxSolves];  // right-hand side
    GhostRule g[kMaxSolves];
    Dims d;
    float coef, out_scale;
    int init, iterations;
    int py, pz;                 // CTAs of the cluster along y and z
    int rows_y, rows_z;         // most rows of one CTA along y and z
    int pitch;                  // floats of a padded row of one colour
    int lanes;                  // float4s of a row of one colour
    unsigned* error;            // set when a bounded wait gives up
};

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ uint32_t remote(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Stores 16 bytes into a CTA of the cluster and counts them on its mbarrier.
__device__ __forceinline__ void store_cluster(uint32_t addr, float4 v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar) : "memory");
}

// Sets a word of a CTA of the cluster.
__device__ __forceinline__ void set_remote(uint32_t addr, uint32_t rank, int v) { asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(remote(addr, rank)), "r"(v) : "memory"); }
// tb::mbar_wait that also gives up once *stop is set (by any CTA of the cluster).
__device__ __forceinline__ bool wait_neighbours(uint64_t* bar, unsigned parity, unsigned polls, const volatile int* stop) {
    const unsigned addr = tb::smem_addr(bar);
    if (tb::mbar_try_wait(addr, parity)) [[likely]] return true;
#pragma unroll 1
    for (unsigned it = 1; it < polls; ++it) {
        if (tb::mbar_try_wait(addr, parity)) return true;
        if ((it & 1023u) == 0 && *stop != 0) return false;
    }
    return false;
}

__device__ __forceinline__ float4 ghost_of(const GhostRule& g, int face, float4 v) {
    return make_float4(tb::ghost(g, face, v.x), tb::ghost(g, face, v.y), tb::ghost(g, face, v.z), tb::ghost(g, face, v.w));
}

// PRESSURE: the pressure update, else a diffusion. JACOBI: both colours from
// the previous sweep's values (two generations of the iterate), else red-black
// in place. RAGGED: rows are not a whole number of float4s of each colour.
template <bool PRESSURE, bool JACOBI, bool RAGGED, typename T>
__global__ void __launch_bounds__(kResidentThreads, 1) k_resident(const __grid_constant__ ResidentArgs a) {
    extern __shared__ __align__(16) float shared[];
    // two mbarriers, for the half-sweeps in turn: a neighbour may be one ahead
    uint64_t* const bar = reinterpret_cast<uint64_t*>(shared);
    float* const smem = shared + 4;
    // a word of the pad before the first array, zero with it: a CTA of the
    // cluster has given up a wait
    volatile int* const stop = reinterpret_cast<volatile int*>(smem);
    const int cs = a.py * a.pz;
    const int solve = static_cast<int>(blockIdx.x) / cs, rank = static_cast<int>(blockIdx.x) % cs;
    const int ry = rank % a.py, rz = rank / a.py;
    const Dims d = a.d;
    const int y0 = ry * d.ny / a.py, ny = (ry + 1) * d.ny / a.py - y0;
    const int z0 = rz * d.nz / a.pz, nz = (rz + 1) * d.nz / a.pz - z0;
    const GhostRule& g = a.g[solve];
    const bool px = g.periodic[0] != 0;
    const int P = a.pitch, PZ = P * (a.rows_y + 2);   // row and plane strides of an array
    const int array = PZ * (a.rows_z + 2);            // floats of one colour
    const int gen = 2 * array;                        // floats of one generation of the iterate
    const int H = 4 * a.lanes;                        // row stride of the right-hand side
    float* const field = smem + 4 + P + PZ;           // cell k = 0 of local row (0, 0), red, generation 0
    float* const rhs = smem + 4 + (JACOBI ? 2 : 1) * gen;  // [colour][z][y][H]
    const int rhs_colour = H * a.rows_y * a.rows_z;
    const uint32_t field_addr = static_cast<uint32_t>(__cvta_generic_to_shared(field));

    // neighbours: the rank that holds the rows beyond each side (-1: a face)
    const int y_lo = ry > 0 ? rank - 1 : (g.periodic[1] ? rank + a.py - 1 : -1);
    const int y_hi = ry + 1 < a.py ? rank + 1 : (g.periodic[1] ? rank - a.py + 1 : -1);
    const int z_lo = rz > 0 ? rank - a.py : (g.periodic[2] ? rank + a.py * (a.pz - 1) : -1);
    const int z_hi = rz + 1 < a.pz ? rank + a.py : (g.periodic[2] ? rank - a.py * (a.pz - 1) : -1);
    const auto rows_of = [&](int r, int parts, int n) { return (r + 1) * n / parts - r * n / parts; };
    // Each thread owns one float4 of every step-th row of the block.
    const int tid = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x);
    const int rows = ny * nz, step = nt / a.lanes;
    const int edges = 2 * (ny + nz);  // the rows on the block's edges
    const int k0 = 4 * (tid % a.lanes), first = tid / a.lanes < step ? tid / a.lanes : rows + edges;  // beyond both: no row
    int* const row_at = reinterpret_cast<int*>(rhs + 2 * rhs_colour);  // 2 x the row's offset in an array, + 1 where its red cells sit at odd x
    // The rows on the block's edges, {row, target, face, mbarrier}: a pad row
    // beside it is a ghost row of the other colour's array here (its offset;
    // mbarrier 0) or the neighbour's row of the same colour (its address in the
    // cluster, for the array at offset 0, and the neighbour's mbarrier).
    int4* const edge_at = reinterpret_cast<int4*>(row_at + (a.rows_y * a.rows_z + 3) / 4 * 4);
    const uint32_t bar_addr = static_cast<uint32_t>(__cvta_generic_to_shared(bar));

    // everything zero (pads that no cell sets are read by lanes past a row's end)
    const int used = 4 + (JACOBI ? 2 : 1) * gen + 2 * rhs_colour;
    for (int r = tid; r < rows; r += nt) row_at[r] = 2 * (r % ny * P + r / ny * PZ) + ((y0 + r % ny + z0 + r / ny) & 1);
    for (int e = tid; e < edges; e += nt) {
        // rows y = 0 and ny - 1 of every plane, then of planes z = 0 and nz - 1
        const bool on_y = e < 2 * nz;
        const int hi = e & 1, i = on_y ? e >> 1 : (e - 2 * nz) >> 1;
        const int across = on_y ? P : PZ, along = (on_y ? PZ : P) * i, count = on_y ? ny : nz;
        const int from = along + (hi ? (count - 1) * across : 0);
        const int to = on_y ? (hi ? y_hi : y_lo) : (hi ? z_hi : z_lo);
        int4 q = make_int4(from, from + (hi ? across : -across), (on_y ? YM : ZM) + hi, 0);
        if (to >= 0) {
            const int theirs = on_y ? rows_of(to % a.py, a.py, d.ny) : rows_of(to / a.py, a.pz, d.nz);  // the neighbour's rows across the side
            q.y = static_cast<int>(remote(field_addr, static_cast<uint32_t>(to)) + 4u * static_cast<uint32_t>(along + (hi ? -across : theirs * across)));
            q.w = static_cast<int>(remote(bar_addr, static_cast<uint32_t>(to)));
        }
        edge_at[e] = q;
    }
    // bytes the neighbours send this CTA a colour
    const int incoming = 16 * a.lanes * (nz * ((y_lo >= 0) + (y_hi >= 0)) + ny * ((z_lo >= 0) + (z_hi >= 0)));
    if (tid == 0) {
        tb::mbar_init(&bar[0], 1);
        tb::mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < used / 4; i += nt) reinterpret_cast<float4*>(smem)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    cluster_sync_all();  // before any neighbour writes its values here

    // the block's right-hand side by colour, cells taken in order of memory
    const T* const b = static_cast<const T*>(a.b[solve]);
    for (int r = tid / 32; r < rows; r += nt / 32) {
        const int y = r % ny, z = r / ny;
        const T* const src = b + lin(0, y0 + y, z0 + z, d);
        float* const dst = rhs + H * r;
        const int odd = (y0 + y + z0 + z) & 1;
        for (int x = tid % 32; x < d.nx; x += 32) dst[((x + odd) & 1) * rhs_colour + (x >> 1)] = to_f(src[x]);
    }
    __syncthreads();

    // the new values of the cells k0 .. of a row of colour array u (cells at x = 2k + s)
    const auto store_cells = [&](float* u, int s, float4 o) {
        const int count = (d.nx - s + 1) / 2 - k0;  // the row's cells from k0 on
        if (!RAGGED || count > 3) {
            *reinterpret_cast<float4*>(u) = o;
        } else {
            if (count > 0) u[0] = o.x;
            if (count > 1) u[1] = o.y;
            if (count > 2) u[2] = o.z;
        }
    };
    // A thread whose wait gives up writes no pads, arrives and waits no more (so
    // nothing is added to barriers that stay incomplete) and goes through the
    // remaining half-sweeps: the barriers of the CTA stay whole. The hot path has
    // no test for it, only other loop bounds (a flag looked at in every half-sweep
    // cost 1 to 2.5 % of a small grid's step).
    int pad_edge = first, pad_row = tid;
    unsigned polls = 1u << 26;
    bool arrives = tid == 0;
    // Writes the pads that depend on the new values of colour c, at offset
    // `at`; `other` is the other colour's array of the same generation, `turn`
    // the mbarrier of the half-sweep.
    const auto write_pads = [&](int c, int at, int other, int turn) {
#pragma unroll 1
        for (int e = pad_edge; e < edges; e += step) {
            const int4 q = edge_at[e];
            const float4 o = *reinterpret_cast<const float4*>(field + at + q.x + k0);
            if (q.w != 0) store_cluster(static_cast<uint32_t>(q.y) + 4u * static_cast<uint32_t>(at + k0), o, static_cast<uint32_t>(q.w + turn));
            else *reinterpret_cast<float4*>(field + other + q.y + k0) = ghost_of(g, q.z, o);
        }
#pragma unroll 1
        for (int r = pad_row; r < rows; r += nt) {
            const int row = row_at[r], s = (row ^ c) & 1;
            float* const u = field + at + (row >> 1);
            float* const v = field + other + (row >> 1);
            // even nx: the row's cells start at x = 0 (s = 0) or end at x = nx - 1; odd nx: both or neither
            if (s == 0) {
                const float o = u[0];
                *(px ? u + d.nx / 2 : v - 1) = px ? o : tb::ghost(g, XM, o);
            }
            if (RAGGED && (d.nx & 1) ? s == 0 : s == 1) {
                const float o = u[(d.nx - 1) / 2];
                *(px ? u - 1 : v + (d.nx + s) / 2) = px ? o : tb::ghost(g, XP, o);
            }
        }
    };
    // End of half-sweep `n` (each `colours` colours of rows): the CTA's own
    // values and its neighbours' are in place.
    const auto finish = [&](int n, int colours) {
        if (arrives) tb::mbar_expect_tx(&bar[n & 1], static_cast<unsigned>(colours * incoming));
        __syncthreads();
        if (!wait_neighbours(&bar[n & 1], static_cast<unsigned>((n >> 1) & 1), polls, stop) && polls != 0) {
            if (a.error != nullptr) atomicOr(a.error, 1u);
            for (int r = 0; r < cs; ++r) set_remote(static_cast<uint32_t>(__cvta_generic_to_shared(smem)), static_cast<uint32_t>(r), 1);
            pad_edge = edges;
            pad_row = rows;
            polls = 0;
            arrives = false;
        }
    };

    // the start
    const T* const start = static_cast<const T*>(a.x[solve]);
    for (int c = 0; c < 2; ++c)
        for (int r = first; r < rows; r += step) {
            const int s = (row_at[r] ^ c) & 1;
            float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (a.init == INIT_FROM_B) {
                o = *reinterpret_cast<const float4*>(rhs + c * rhs_colour + H * r + k0);
            } else if (a.init == INIT_FROM_X) {
                const T* const src = start + lin(0, y0 + r % ny, z0 + r / ny, d);
                const int x = 2 * k0 + s;
                o = make_float4(x < d.nx ? to_f(src[x]) : 0.0f, x + 2 < d.nx ? to_f(src[x + 2]) : 0.0f, x + 4 < d.nx ? to_f(src[x + 4]) : 0.0f, x + 6 < d.nx ? to_f(src[x + 6]) : 0.0f);
            }
            store_cells(field + c * array + (row_at[r] >> 1) + k0, s, o);
        }
    __syncthreads();
    write_pads(0, 0, array, 0);
    write_pads(1, array, 0, 0);
    finish(0, 2);
    cluster_sync_all();  // the first half-sweep writes pads that the start has written too

    const divide::Divisor div = divide::make_divisor(PRESSURE ? 6.0f : 1.0f + 6.0f * a.coef);
    constexpr int KIND = PRESSURE ? KIND_PRESSURE : KIND_VEL_X;
    const float inv = wave::jacobi_inverse(KIND, a.coef);
    // colour c of one sweep: from the other colour at offset `from` (and the
    // right-hand side) into offset `to`
    const auto half = [&](int c, int from, int to) {
        const float* w = rhs + c * rhs_colour + H * first + k0;
#pragma unroll 1
        for (int r = first; r < rows; r += step, w += H * step) {
            const int row = row_at[r], s = (row ^ c) & 1;
            const float* const v = field + from + (row >> 1) + k0;
            const float4 cur = *reinterpret_cast<const float4*>(v);
            const float ext = v[s ? 4 : -1];
            const float4 ym = *reinterpret_cast<const float4*>(v - P), yp = *reinterpret_cast<const float4*>(v + P);
            const float4 zm = *reinterpret_cast<const float4*>(v - PZ), zp = *reinterpret_cast<const float4*>(v + PZ);
            const float4 b4 = *reinterpret_cast<const float4*>(w);
            // x- + x+: the pairs of neighbouring cells of the other colour's row
            const float p0 = cur.x + cur.y, p1 = cur.y + cur.z, p2 = cur.z + cur.w, pe = ext + (s ? cur.w : cur.x);
            const F4 sum = F4{f2(s ? p0 : pe, s ? p1 : p0), f2(s ? p2 : p1, s ? pe : p2)} + f4(ym) + f4(yp) + f4(zm) + f4(zp);
            float4 o;
            if constexpr (JACOBI) {
                const float4 n = unpack(sum);
                o = make_float4(wave::jacobi_update<KIND>(n.x, b4.x, a.coef, inv), wave::jacobi_update<KIND>(n.y, b4.y, a.coef, inv), wave::jacobi_update<KIND>(n.z, b4.z, a.coef, inv), wave::jacobi_update<KIND>(n.w, b4.w, a.coef, inv));
            } else {
                // nb - h^2 div, or b + alpha nb, each in one rounding
                const F2 coef = PRESSURE ? f2(-a.coef, -a.coef) : f2(a.coef, a.coef);
                const F4 bb = f4(b4);
                float4 n = unpack(PRESSURE ? F4{fma2(coef, bb.lo, sum.lo), fma2(coef, bb.hi, sum.hi)} : F4{fma2(coef, sum.lo, bb.lo), fma2(coef, sum.hi, bb.hi)});
                if constexpr (RAGGED) {  // what lies past the row's end must not send the others down the slow division
                    const int count = (d.nx - s + 1) / 2 - k0;
                    n.y = count > 1 ? n.y : n.x;
                    n.z = count > 2 ? n.z : n.x;
                    n.w = count > 3 ? n.w : n.x;
                }
                o = divide::four<PRESSURE>(n, div);
            }
            if constexpr (sizeof(T) == 2) o = make_float4(to_f(from_f<T>(o.x)), to_f(from_f<T>(o.y)), to_f(from_f<T>(o.z)), to_f(from_f<T>(o.w)));
            store_cells(field + to + (row >> 1) + k0, s, o);
        }
    };
    int now = 0;  // generation that holds the iterate
    if constexpr (JACOBI) {
#pragma unroll 1
        for (int n = 1; n <= a.iterations; ++n) {
            const int next = gen - now;
#pragma unroll 1
            for (int c = 0; c < 2; ++c) half(c, now + (1 - c) * array, next + c * array);
            __syncthreads();
#pragma unroll 1
            for (int c = 0; c < 2; ++c) write_pads(c, next + c * array, next + (1 - c) * array, 8 * (n & 1));
            finish(n, 2);
            now = next;
        }
    } else {
#pragma unroll 1
        for (int n = 1; n <= 2 * a.iterations; ++n) {
            const int c = (n & 1) ^ 1;
            half(c, (1 - c) * array, c * array);
            __syncthreads();
            write_pads(c, c * array, (1 - c) * array, 8 * (n & 1));
            finish(n, 1);
        }
    }

    // no CTA reads another's shared memory, or leaves, while stores may be in flight
    cluster_sync_all();
    if (*stop != 0) {
        __nanosleep(1000000);  // stores of a half-sweep that was not waited for
        return;
    }
    T* const out = static_cast<T*>(a.x[solve]);
    for (int r = tid / 32; r < rows; r += nt / 32) {
        const int y = r % ny, z = r / ny;
        T* const dst = out + lin(0, y0 + y, z0 + z, d);
        const float* const row = field + now + y * P + z * PZ;
        const int odd = (y0 + y + z0 + z) & 1;
        for (int x = tid % 32; x < d.nx; x += 32) {
            const float q = row[((x + odd) & 1) * array + (x >> 1)];
            dst[x] = from_f<T>(a.out_scale != 1.0f ? __fmul_rn(q, a.out_scale) : q);
        }
    }
}

cudaLaunchConfig_t resident_config(int ctas, int cluster, int threads, size_t smem, cudaStream_t s, cudaLaunchAttribute& attr) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(ctas));
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(cluster);
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cfg;
}

struct ResidentKernel {
    void (*kernel)(const ResidentArgs);
    bool fits[5];  // clusters of 1, 2, 4, 8, 16 CTAs with all the shared memory can be resident
};

// The kernel with its attributes set, and the cluster sizes the device takes
// (looked up once a device: each query costs some 50 us of a context's creation).
template <bool PRESSURE, bool JACOBI, bool RAGGED, typename T>
const ResidentKernel& resident_kernel() {
    static PerDevice<ResidentKernel> kernels;
    return kernels.get([] {
        ResidentKernel k{k_resident<PRESSURE, JACOBI, RAGGED, T>, {}};
        if (cudaFuncSetAttribute(k.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kResidentShared) != cudaSuccess || cudaFuncSetAttribute(k.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            return k;
        }
        for (int i = 0; i < 5; ++i) {
            cudaLaunchAttribute attr{};
            cudaLaunchConfig_t cfg = resident_config(1 << i, 1 << i, kResidentThreads, kResidentShared, nullptr, attr);
            int clusters = 0;
            k.fits[i] = cudaOccupancyMaxActiveClusters(&clusters, k.kernel, &cfg) == cudaSuccess && clusters >= 1;
        }
        cudaGetLastError();
        return k;
    });
}

template <bool RAGGED>
const ResidentKernel& resident_kernel(bool pressure, bool jacobi, bool bf16) {
    if (pressure) return jacobi ? resident_kernel<true, true, RAGGED, float>() : resident_kernel<true, false, RAGGED, float>();
    if (bf16) return jacobi ? resident_kernel<false, true, RAGGED, __nv_bfloat16>() : resident_kernel<false, false, RAGGED, __nv_bfloat16>();
    return jacobi ? resident_kernel<false, true, RAGGED, float>() : resident_kernel<false, false, RAGGED, float>();
}

// The split of a grid over a cluster of py x pz CTAs, with the shared memory
// of one of them; false when it does not fit.
bool resident_shape(const Dims& d, int py, int pz, bool jacobi, ResidentArgs& a, size_t& smem) {
    if (py > d.ny || pz > d.nz) return false;
    a.py = py;
    a.pz = pz;
    a.rows_y = (d.ny + py - 1) / py;
    a.rows_z = (d.nz + pz - 1) / pz;
    const int hx = (d.nx + 1) / 2;  // cells of a row of one colour
    a.lanes = (hx + 3) / 4;
    a.pitch = (4 * a.lanes + 2 + 3) / 4 * 4;
    if (a.lanes > 128) return false;
    const size_t array = static_cast<size_t>(a.pitch) * (a.rows_y + 2) * (a.rows_z + 2);
    const size_t rows = static_cast<size_t>(a.rows_y) * a.rows_z;
    smem = 4 * (8 + (jacobi ? 4 : 2) * array + 8 * rows * a.lanes + (rows + 3) / 4 * 4) + 32 * static_cast<size_t>(a.rows_y + a.rows_z);
    return smem <= kResidentShared;
}

}  // namespace

// The solves of a[0 .. n - 1] (same grid, scheme, start, iterations and
// coefficient; n <= 3) in one launch; false (nothing launched) when they do
// not fit a cluster's shared memory or are asked for in another form, or when
// the device refuses the launch.
bool launch_resident(const StencilArgs* a, int n, cudaStream_t s) {
    const StencilArgs& f = a[0];
    if (n < 1 || n > kMaxSolves || f.per_pass != 0 || f.iterations < 1) return false;
    const size_t cells = static_cast<size_t>(f.dims.nx) * f.dims.ny * f.dims.nz;
    if (cells > (1u << 19)) return false;  // 16 CTAs hold at most 0.4 M cells
    const bool jacobi = f.scheme == SCHEME_JACOBI, pressure = f.kind == KIND_PRESSURE;
    ResidentArgs r{};
    r.d = f.dims;
    for (int k = 0; k < n; ++k) {
        r.x[k] = a[k].x;
        r.b[k] = a[k].b;
        r.g[k] = make_ghost_rule(a[k].kind, a[k].flow, a[k].scalar);
        for (int axis = 0; axis < 3; ++axis) {
            const int side = axis == 0 ? f.dims.nx : axis == 1 ? f.dims.ny : f.dims.nz;
            if (r.g[k].periodic[axis] && (side & 1)) return false;  // the colouring breaks across the wrap
        }
    }
    r.coef = f.coef;
    r.out_scale = f.out_scale;
    r.init = f.init;
    r.iterations = f.iterations;
    r.error = f.error_flag;
    const ResidentKernel& kern = f.dims.nx % 8 != 0 ? resident_kernel<true>(pressure, jacobi, f.bf16 != 0) : resident_kernel<false>(pressure, jacobi, f.bf16 != 0);
    // the smallest cluster whose CTAs hold few enough float4s, else the
    // largest that fits
    size_t smem = 0;
    ResidentArgs best{};
    size_t best_smem = 0;
    int best_size = 0;
    for (int i = 0; i < 5; ++i) {
        if (!kern.fits[i]) continue;
        const int size = 1 << i;
        long long cost = -1;
        for (int py = 1; py <= size; py *= 2) {
            if (!resident_shape(f.dims, py, size / py, jacobi, r, smem)) continue;
            const long long rows = static_cast<long long>(r.rows_y) * r.rows_z, edge = r.rows_y + r.rows_z;
            const long long c = 64 * rows + edge;
            if (cost >= 0 && c >= cost) continue;
            cost = c;
            best = r;
            best_smem = smem;
            best_size = size;
        }
        if (cost >= 0 && static_cast<long long>(best.rows_y) * best.rows_z * best.lanes <= kResidentItems) break;
    }
    if (best_size == 0) return false;
    // a float4 a thread, as far as the threads go
    const long long items = static_cast<long long>(best.rows_y) * best.rows_z * best.lanes;
    const int threads = static_cast<int>(std::min<long long>(kResidentThreads, std::max<long long>(128, (items + 31) / 32 * 32)));
    cudaLaunchAttribute attr{};
    const cudaLaunchConfig_t cfg = resident_config(n * best_size, best_size, threads, best_smem, s, attr);
    if (cudaLaunchKernelEx(&cfg, kern.kernel, static_cast<const ResidentArgs>(best)) != cudaSuccess) {
        cudaGetLastError();  // nothing was launched: the sweeps run instead
        return false;
    }
    if (f.launches) *f.launches += 1;
    return true;
}

}  // namespace sfb
