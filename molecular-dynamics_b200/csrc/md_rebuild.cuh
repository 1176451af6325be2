// One step's start in md_run's graphs, as one cooperative kernel: it closes the float modes' sums of the last step and,
// when the half-skin test of the step's drift flagged a particle (NeighbourList::update, src/NeighbourList.cpp:11-36),
// rebuilds the list: cell sort, reorder, frames, list, and what the precision keeps beside it (FP64's pair offsets,
// MD_PREC_FX32's near and far rows, the fixed-point frames). Without a flag it returns at once.
//
// Why one kernel: a graph node costs 1.1 us and a conditional node 7.2 us of every step, whether or not its body (14
// kernels) runs; a kernel that looks at the flag itself costs one node. The phases of a rebuild are separated by barriers
// over the whole grid, which is one resident wave (a cooperative launch). The barriers are bounded: one that gives up
// reports through state[1], and the chunk then reruns on the host path.
//
// The sort is the host path's (md_cells.cuh) with each particle's slot in its cell taken from the counting atomics, and
// the reorder writes each particle to its new place directly; the list build is build_cell, the rows are split by
// rows_split. Data written by other blocks is read with plain loads after a barrier (never through the read-only path).
#pragma once

#include "md_build.cuh"
#include "md_cells.cuh"
#include "md_common.cuh"
#include "md_fp32.cuh"
#include "md_fx32.cuh"

namespace md {

constexpr int kRebuildThreads = 128;
// 0.23 s (N = 4,000, B200), for a wait whose partners are resident and at most some ms behind
constexpr unsigned kBarrierPolls = 1u << 20;
constexpr int kDirectScan = 16384;            // cells up to which a block adds up the counts before its own

struct RebuildArgs {
    int n, ncells, ncps;
    double inv_cell, cell;
    Box box;
    // the system's arrays and their spares
    double4 *pos, *pos2;
    double *vel, *vel2, *force, *force2, *mass, *mass2;
    uint64_t *ids, *ids2;
    // the list
    double4* ref_pos;
    int *cell_of, *cell_sorted, *count, *start, *slot, *bucket, *block_sums;
    float4* frames;
    int4* iframes;  // nullptr: none kept
    CellBuild build;
    int *list, *listed;  // sparse systems: the cells left to blocks
    uint32_t* rows;
    int2* counts;
    int *stale, *max_count, *state;
    unsigned* barrier;  // [0] arrivals, [1] blocks done
    int report_always;
    unsigned missing;   // for tests: blocks that the barriers wait for in vain
    // FP64: pair offsets, the records' capacity, and this step's copy of the pair count
    long long* half_off;  // nullptr: none kept
    long long* offset_sums;
    long long rec_cap;
    long long* pair_count;
    unsigned long long* inside;  // FP64's inside count, cleared for this step
    // MD_PREC_FX32: the split rows (nullptr: none kept)
    uint32_t *near_rows, *far_rows;
    int2* counts_nf;
    float near2;
    CellOffsets offs;
    // the last step's float sums, closed here (k_finish_float_energy)
    unsigned long long* acc;  // nullptr: nothing to close
    FinishArgs finish;
};

// All blocks have arrived when the count passes the next multiple of the grid. False (in every thread) if it gave up.
__device__ __forceinline__ bool grid_barrier(const RebuildArgs& a) {
    __shared__ bool ok;
    unsigned* count = a.barrier;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned at = atomicAdd(count, 1u), target = (at / gridDim.x + 1u) * gridDim.x + a.missing;
        unsigned polls = 0, v;
        do {
            asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
        } while (v < target && ++polls < kBarrierPolls);
        ok = v >= target;
        if (!ok) atomicExch(a.state + 1, 1);
        __threadfence();
    }
    __syncthreads();
    return ok;
}

// Sum of v over the block (kRebuildThreads threads), in every thread
__device__ __forceinline__ long long block_sum(long long v) {
    __shared__ long long part[kRebuildThreads / 32];
    v = warp_sum_i64(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0;
#pragma unroll
    for (int w = 0; w < kRebuildThreads / 32; ++w) v += part[w];
    return v;
}

// Exclusive prefix of v over the block plus *total
__device__ __forceinline__ long long block_prefix(long long v, long long* total) {
    __shared__ long long part[kRebuildThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    __syncthreads();
    if (lane == 31) part[warp] = inc;
    __syncthreads();
    long long before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kRebuildThreads / 32; ++w) {
        if (w < warp) before += part[w];
        all += part[w];
    }
    *total = all;
    return before + inc - v;
}

// out[k] = sum of in(0 .. k-1) for this block's part of [0, n), out[n] the total; the sums of the parts before come from
// `before` (this block's exclusive sum)
template <typename Out, typename In>
__device__ __forceinline__ void write_prefix(int n, int part, long long before, Out* out, In in) {
    const int a = min(n, static_cast<int>(blockIdx.x) * part), b = min(n, a + part);
    for (int k0 = a; k0 < b; k0 += kRebuildThreads) {
        const int k = k0 + static_cast<int>(threadIdx.x);
        const long long v = k < b ? static_cast<long long>(in(k)) : 0;
        long long total;
        const long long p = block_prefix(v, &total);
        if (k < b) out[k] = static_cast<Out>(before + p);
        before += total;
    }
    if (a < n && b == n && threadIdx.x == 0) out[n] = static_cast<Out>(before);
}

template <int kHomes, int kRound, bool kSparse>
__global__ void __launch_bounds__(kRebuildThreads, 8) k_step_start(const __grid_constant__ RebuildArgs a) {
    extern __shared__ float4 sm_step[];
    __shared__ union Shared {
        CellItems items;
        float4 s_off[32];
        __device__ Shared() {}
    } sh;
    __shared__ int s_last;
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    const bool stale = *static_cast<volatile int*>(a.stale) != 0;
    if (first) {
        if (a.acc) finish_float_energy(a.acc, a.finish);
        if (a.inside) *a.inside = 0;
        if (!stale && a.pair_count) *a.pair_count = a.half_off[a.n];
    }
    // (after a report the chunk runs again anyway, and an abandoned rebuild leaves its counts behind)
    if (!stale || *static_cast<volatile int*>(a.state + 1) != 0) return;
    const int n = a.n, stride = static_cast<int>(gridDim.x) * kRebuildThreads;
    const int t0 = static_cast<int>(blockIdx.x) * kRebuildThreads + static_cast<int>(threadIdx.x);
    // cells and counts (src/CellList.cpp:25-40); the counts are zero between rebuilds
    for (int i = t0; i < n; i += stride) {
        const double4 p = a.pos[i];
        const int c = (cell_coord(p.x, a.inv_cell, a.ncps) * a.ncps + cell_coord(p.y, a.inv_cell, a.ncps)) * a.ncps +
                      cell_coord(p.z, a.inv_cell, a.ncps);
        a.cell_of[i] = c;
        a.slot[i] = atomicAdd(&a.count[c], 1);
    }
    if (!grid_barrier(a)) return;
    if (first) *a.stale = 0;  // every block has read it
    // the cells' first particles (src/CellList.cpp:42-46)
    {
        const int part = (a.ncells + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
        const int p0 = min(a.ncells, static_cast<int>(blockIdx.x) * part), p1 = min(a.ncells, p0 + part);
        long long before = 0;
        if (a.ncells <= kDirectScan) {  // few cells: each block adds up all those before its own
            for (int k = threadIdx.x; k < p0; k += kRebuildThreads) before += a.count[k];
            before = block_sum(before);
        } else {
            long long mine = 0;
            for (int k = p0 + static_cast<int>(threadIdx.x); k < p1; k += kRebuildThreads) mine += a.count[k];
            mine = block_sum(mine);
            if (threadIdx.x == 0) a.block_sums[blockIdx.x] = static_cast<int>(mine);
            if (!grid_barrier(a)) return;
            for (int k = threadIdx.x; k < static_cast<int>(blockIdx.x); k += kRebuildThreads) before += a.block_sums[k];
            before = block_sum(before);
        }
        write_prefix(a.ncells, part, before, a.start, [&](int k) { return a.count[k]; });
    }
    if (!grid_barrier(a)) return;
    for (int i = t0; i < n; i += stride) a.bucket[a.start[a.cell_of[i]] + a.slot[i]] = i;
    for (int c = t0; c < a.ncells; c += stride) a.count[c] = 0;
    if (kSparse && first) *a.listed = 0;
    if (!grid_barrier(a)) return;
    // the stable order: a particle's place in its cell is the number of smaller indices there (src/CellList.cpp:48-51);
    // the reorder (src/System.cpp:42-64) into the spare arrays, and the list's own copies
    if (first) a.frames[n] = make_float4(kSentinelCoord, kSentinelCoord, kSentinelCoord, 0.0f);
    for (int i = t0; i < n; i += stride) {
        const int c = a.cell_of[i], s = a.start[c], e = a.start[c + 1];
        int k = s;
        for (int f = s; f < e; ++f) k += a.bucket[f] < i;
        const double4 p = a.pos[i];
        a.pos2[k] = p;
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            a.vel2[static_cast<size_t>(v) * n + k] = a.vel[static_cast<size_t>(v) * n + i];
            a.force2[static_cast<size_t>(v) * n + k] = a.force[static_cast<size_t>(v) * n + i];
        }
        a.mass2[k] = a.mass[i];
        a.ids2[k] = a.ids[i];
        a.ref_pos[k] = p;
        a.cell_sorted[k] = c;
        a.frames[k] = list_frame_of(p, c, a.ncps, a.cell, a.box);
        if (a.iframes) a.iframes[k] = fixed_frame_of(p, c, a.ncps, a.cell, a.box);
    }
    if (!grid_barrier(a)) return;
    // the reordered arrays back into their places (the graph's kernels were recorded with those addresses)
    for (int k = t0; k < n; k += stride) {
        a.pos[k] = a.pos2[k];
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            a.vel[static_cast<size_t>(v) * n + k] = a.vel2[static_cast<size_t>(v) * n + k];
            a.force[static_cast<size_t>(v) * n + k] = a.force2[static_cast<size_t>(v) * n + k];
        }
        a.mass[k] = a.mass2[k];
        a.ids[k] = a.ids2[k];
    }
    int cells = a.ncells;
    if constexpr (kSparse) {  // a cell per warp, and then the cells too full for one by blocks (build_cells_sparse)
        const int per = kSparseWarps * a.build.group;
        const int first_cell = static_cast<int>(threadIdx.x >> 5) * a.build.group;
        block_turns((a.ncells + per - 1) / per, [&](int k) {
            build_cells_sparse(sm_step, a.frames, a.ref_pos, a.start, a.ncells, k * per + first_cell, static_cast<float>(a.cell),
                               a.build, a.rows, a.counts, a.max_count,
                               [&](int cell) { a.list[atomicAdd(a.listed, 1)] = cell; });
        });
        if (!grid_barrier(a)) return;
        cells = *static_cast<volatile int*>(a.listed);
    }
    block_turns(cells, [&](int k) {
        build_cell<kRebuildThreads / 32, kHomes, kRound>(sh.items, sm_step, a.frames, a.ref_pos, a.start,
                                                         kSparse ? a.list[k] : k, static_cast<float>(a.cell), a.build, a.rows,
                                                         a.counts, a.max_count);
        __syncthreads();
    });
    if (a.near_rows) {
        if (!grid_barrier(a)) return;
        if (threadIdx.x < 32) sh.s_off[threadIdx.x] = a.offs.off[threadIdx.x];
        __syncthreads();
        for (int i = t0; i < n; i += stride) {
            if (!rows_split(reinterpret_cast<uint32_t*>(sm_step), sh.s_off, a.frames, n, i, a.near2, a.rows, a.build.geom.cap,
                            a.counts, a.near_rows, a.far_rows, a.counts_nf))
                rows_split_fix(sh.s_off, a.frames, n, i, a.near2, a.rows, a.build.geom.cap, a.counts, a.near_rows,
                               a.far_rows, a.counts_nf);
        }
    }
    if (a.half_off) {  // the half-list offsets (src/NeighbourList.cpp:116-127)
        if (!grid_barrier(a)) return;
        const int part = (n + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
        const int p0 = min(n, static_cast<int>(blockIdx.x) * part), p1 = min(n, p0 + part);
        long long before = 0;
        long long mine = 0;
        for (int k = p0 + static_cast<int>(threadIdx.x); k < p1; k += kRebuildThreads) mine += a.counts[k].x;
        mine = block_sum(mine);
        if (threadIdx.x == 0) a.offset_sums[blockIdx.x] = mine;
        if (!grid_barrier(a)) return;
        for (int k = threadIdx.x; k < static_cast<int>(blockIdx.x); k += kRebuildThreads) before += a.offset_sums[k];
        before = block_sum(before);
        write_prefix(n, part, before, a.half_off, [&](int k) { return a.counts[k].x; });
    }
    // the last block to finish counts the rebuild and reports a row that outgrew the capacity, or records that outgrew
    // their buffer: the host reruns the chunk on its own path then
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(a.barrier + 1, 1u) % gridDim.x == gridDim.x - 1u;
        __threadfence();
        if (s_last) {
            a.state[0] += 1;
            if (*static_cast<volatile int*>(a.max_count) > a.build.geom.cap || a.report_always) a.state[1] = 1;
            *a.max_count = 0;
            if (a.half_off) {
                const long long pairs = *static_cast<volatile long long*>(a.half_off + n);
                if (pairs > a.rec_cap) a.state[1] = 1;
                if (a.pair_count) *a.pair_count = pairs;
            }
        }
    }
}

}  // namespace md
