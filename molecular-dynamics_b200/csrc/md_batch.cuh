// Batched replicas: many independent Lennard-Jones systems of uneven size, density and temperature advanced by
// the same kernel launches, each replica following the reference's single-system step (src/Integrator.cpp:18-30,
// src/NeighbourList.cpp:11-134, src/Forcefield.cpp:214-326, src/Thermostat.cpp:17-58) on its own box.
//
// Layout. Replica r owns the particle slots [off_r, off_r + n_r), off_r a multiple of kTile, so every tile of
// kTile slots (and every thread block over one) belongs to exactly one replica; tile_rep[t] names it. Positions,
// masses, ids, frames and neighbour rows are indexed by slot. Velocities and forces keep each replica's
// component-major arrays contiguous: component k of slot a sits at 3 off_r + k np_r + (a - off_r), np_r being n_r
// rounded up to kTile. The cell arrays are concatenated the same way (cell_off_r; the cell starts of replica r
// take ncells_r + 1 entries from cell_off_r + r).
//
// Rebuilds are decided on the device: the drift kernel flags a replica whose particle moved more than half the
// skin, k_b_stale_lists turns the flags into a list of stale replicas and of their tiles, and the rebuild kernels
// loop over those lists with a fixed grid, so a step needs no host decision and a run of steps can be one CUDA
// graph. Each replica's cell sort, reorder, list and sums repeat the single-system kernels' operation sequences,
// so a replica's trajectory is bit-identical to the same system run alone.
#pragma once

#include "md_build.cuh"
#include "md_cells.cuh"
#include "md_common.cuh"
#include "md_fp32.cuh"
#include "md_tiles.cuh"
#include "md_fp64.cuh"
#include "md_nlist.cuh"

namespace md {

constexpr int kTile = 128;          // slots per tile; replicas start on tile boundaries
constexpr int kListThreads = 1024;  // k_b_stale_lists block
constexpr int kRepScanThreads = 256;   // per-replica scans

struct BRep {
    Box box;
    double inv_cell;     // cells per side / L (src/CellList.cpp:18)
    double cell;         // L / cells per side
    double dof;          // 3 n - 3 (src/System.cpp:79-82)
    double temperature;  // thermostat target
    int off;             // first slot
    int n;               // particles
    int np;              // n rounded up to kTile: component stride of velocities and forces
    int ncps;            // cells per side
    int ncells;          // ncps^3
    int cell_off;        // first cell of the count/cursor arrays
    int use_cells;       // ncps >= 3 (src/NeighbourList.cpp:69); 2: so few particles a cell that threads build rows
    int tile_off;        // first tile
    int chunk_off;       // first 1024-particle block of the kinetic-energy sums
};

// Index of component k of slot a in the velocity and force arrays
__device__ __forceinline__ size_t bvec(const BRep& d, int k, int a) {
    return 3 * static_cast<size_t>(d.off) + static_cast<size_t>(k) * d.np + (a - d.off);
}

__device__ __forceinline__ int inclusive_warp_scan(int v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += x;
    }
    return v;
}

// Exclusive block scan of v with a running carry (kRepScanThreads threads); returns the exclusive prefix and adds
// the block's total to *carry after a barrier
__device__ __forceinline__ int block_scan_carry(int v, int* s_warp, int* carry) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x = inclusive_warp_scan(v);
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int y = lane < kRepScanThreads / 32 ? s_warp[lane] : 0;
        y = inclusive_warp_scan(y);
        if (lane < kRepScanThreads / 32) s_warp[lane] = y;
    }
    __syncthreads();
    const int excl = *carry + (warp ? s_warp[warp - 1] : 0) + x - v;
    __syncthreads();
    if (threadIdx.x == kRepScanThreads - 1) *carry = excl + v;
    __syncthreads();
    return excl;
}

// ---- integration --------------------------------------------------------------------------------------------

// One tile per block. A pending thermostat scale (scale[r].y != 0) is applied first, as scaleVelocities would
// have at the end of the previous step (src/Thermostat.cpp:7-14), then kickAndDrift (src/Integrator.cpp:32-53),
// the half-skin test (src/NeighbourList.cpp:24-30) that flags the replica stale, and with kFrames the float
// frame of the new position.
template <bool kFrames>
__global__ void __launch_bounds__(kTile)
    k_b_kick_drift(const BRep* __restrict__ reps, const int* __restrict__ tile_rep, double4* __restrict__ pos,
                   double* __restrict__ vel, const double* __restrict__ force, const double* __restrict__ mass,
                   double half_dt, double dt, const double4* __restrict__ ref_pos, double max_disp2,
                   int* __restrict__ stale, const double2* __restrict__ scale, const int* __restrict__ cell_sorted,
                   float4* __restrict__ frames) {
    const int r = tile_rep[blockIdx.x];
    const BRep d = reps[r];
    const int i = (blockIdx.x - d.tile_off) * kTile + threadIdx.x;
    if (i >= d.n) return;
    const int a = d.off + i;
    const double2 sc = scale[r];
    const double m = mass[a];
    double4 p = pos[a];
    double* pc[3] = {&p.x, &p.y, &p.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const size_t o = bvec(d, k, a);
        double v = vel[o];
        if (sc.y != 0.0) v = dmul(v, sc.x);
        v = dadd(v, ddiv(dmul(half_dt, force[o]), m));
        vel[o] = v;
        *pc[k] = wrap(dadd(*pc[k], dmul(dt, v)), d.box);
    }
    pos[a] = p;
    const double4 q = ref_pos[a];
    const double dx = min_image(dsub(p.x, q.x), d.box);
    const double dy = min_image(dsub(p.y, q.y), d.box);
    const double dz = min_image(dsub(p.z, q.z), d.box);
    if (norm2(dx, dy, dz) > max_disp2) stale[r] = 1;
    if (kFrames) frames[a] = frame_of(p, cell_sorted[a], d.ncps, d.cell, d.box);
}

// Applies and clears the pending thermostat scales (end of a run), one tile per block; k_b_clear_scale follows.
__global__ void __launch_bounds__(kTile) k_b_apply_scale(const BRep* __restrict__ reps, const int* __restrict__ tile_rep,
                                                         double* __restrict__ vel, const double2* __restrict__ scale) {
    const int r = tile_rep[blockIdx.x];
    const BRep d = reps[r];
    const int i = (blockIdx.x - d.tile_off) * kTile + threadIdx.x;
    const double2 sc = scale[r];
    if (i >= d.n || sc.y == 0.0) return;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const size_t o = bvec(d, k, d.off + i);
        vel[o] = dmul(vel[o], sc.x);
    }
}

__global__ void k_b_clear_scale(int R, double2* __restrict__ scale) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < R) scale[r] = make_double2(1.0, 0.0);
}

// ---- rebuild ------------------------------------------------------------------------------------------------

// Work items of a replica's list build: its cells, its tiles where threads build rows, or groups of kAllGroup slots in a box
// under 3 cells per side
constexpr int kAllGroup = 16;
__host__ __device__ __forceinline__ int build_items(const BRep& d) {
    return d.use_cells == 1 ? d.ncells : d.use_cells == 2 ? d.np / kTile : d.np / kAllGroup;
}

// One block. Reads and clears the stale flags, lists the stale replicas and their tiles in replica order
// (work[0] replicas, work[1] tiles, work[2] list-build items, those before stale replica w in stale_items[w]) and counts
// each replica's rebuild.
__global__ void __launch_bounds__(kListThreads)
    k_b_stale_lists(const BRep* __restrict__ reps, int R, int* __restrict__ stale, int* __restrict__ stale_reps,
                    int* __restrict__ stale_tiles, int* __restrict__ stale_items, int* __restrict__ work,
                    unsigned long long* __restrict__ rebuilds) {
    __shared__ int s_warp[3][32];
    __shared__ int s_base[3];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kWarps = kListThreads / 32;
    if (threadIdx.x == 0) s_base[0] = s_base[1] = s_base[2] = 0;
    __syncthreads();
    for (int r0 = 0; r0 < R; r0 += kListThreads) {
        const int r = r0 + threadIdx.x;
        int f = 0, nt = 0, t0 = 0, ni = 0;
        if (r < R && stale[r]) {
            stale[r] = 0;
            const BRep d = reps[r];
            f = 1;
            nt = d.np / kTile;
            t0 = d.tile_off;
            ni = build_items(d);
        }
        const int sf = inclusive_warp_scan(f), st = inclusive_warp_scan(nt), si = inclusive_warp_scan(ni);
        if (lane == 31) {
            s_warp[0][warp] = sf;
            s_warp[1][warp] = st;
            s_warp[2][warp] = si;
        }
        __syncthreads();
        if (warp == 0) {
            const int a = inclusive_warp_scan(s_warp[0][lane]);
            const int b = inclusive_warp_scan(s_warp[1][lane]);
            const int c = inclusive_warp_scan(s_warp[2][lane]);
            s_warp[0][lane] = a;
            s_warp[1][lane] = b;
            s_warp[2][lane] = c;
        }
        __syncthreads();
        if (f) {
            const int pf = s_base[0] + (warp ? s_warp[0][warp - 1] : 0) + sf - 1;
            const int pt = s_base[1] + (warp ? s_warp[1][warp - 1] : 0) + st - nt;
            stale_reps[pf] = r;
            stale_items[pf] = s_base[2] + (warp ? s_warp[2][warp - 1] : 0) + si - ni;
            for (int k = 0; k < nt; ++k) stale_tiles[pt + k] = t0 + k;
            rebuilds[r] += 1;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s_base[0] += s_warp[0][kWarps - 1];
            s_base[1] += s_warp[1][kWarps - 1];
            s_base[2] += s_warp[2][kWarps - 1];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        work[0] = s_base[0];
        work[1] = s_base[1];
        work[2] = s_base[2];
    }
}

// The particle of this thread in the w-th stale tile: returns false past the replica's end
__device__ __forceinline__ bool stale_slot(const BRep* __restrict__ reps, const int* __restrict__ tile_rep,
                                           const int* __restrict__ stale_tiles, int w, int& r, BRep& d, int& a) {
    const int t = stale_tiles[w];
    r = tile_rep[t];
    d = reps[r];
    const int i = (t - d.tile_off) * kTile + threadIdx.x;
    a = d.off + i;
    return i < d.n;
}

// CellList::build's cell index and histogram (src/CellList.cpp:25-40) for the stale replicas
__global__ void __launch_bounds__(kTile)
    k_b_cell_assign(const BRep* __restrict__ reps, const int* __restrict__ tile_rep, const int* __restrict__ stale_tiles,
                    const int* __restrict__ work, const double4* __restrict__ pos, int* __restrict__ cell_of,
                    int* __restrict__ count) {
    const int nw = work[1];
    for (int w = blockIdx.x; w < nw; w += gridDim.x) {
        int r, a;
        BRep d;
        if (!stale_slot(reps, tile_rep, stale_tiles, w, r, d, a)) continue;
        const double4 p = pos[a];
        const int c = (cell_coord(p.x, d.inv_cell, d.ncps) * d.ncps + cell_coord(p.y, d.inv_cell, d.ncps)) * d.ncps +
                      cell_coord(p.z, d.inv_cell, d.ncps);
        cell_of[a] = c;
        atomicAdd(&count[d.cell_off + c], 1);
    }
}

// Exclusive prefix sum of each stale replica's cell histogram into slot numbers (src/CellList.cpp:42-46); the
// histogram is cleared for the next rebuild. One block per stale replica.
__global__ void __launch_bounds__(kRepScanThreads)
    k_b_cell_scan(const BRep* __restrict__ reps, const int* __restrict__ stale_reps, const int* __restrict__ work,
                  int* __restrict__ count, int* __restrict__ start) {
    __shared__ int s_warp[32];
    __shared__ int s_carry;
    const int nr = work[0];
    for (int w = blockIdx.x; w < nr; w += gridDim.x) {
        const int r = stale_reps[w];
        const BRep d = reps[r];
        int* st = start + d.cell_off + r;
        if (threadIdx.x == 0) s_carry = d.off;
        __syncthreads();
        for (int c0 = 0; c0 < d.ncells; c0 += kRepScanThreads) {
            const int c = c0 + threadIdx.x;
            const int v = c < d.ncells ? count[d.cell_off + c] : 0;
            const int e = block_scan_carry(v, s_warp, &s_carry);
            if (c < d.ncells) {
                st[c] = e;
                count[d.cell_off + c] = 0;
            }
        }
        if (threadIdx.x == 0) st[d.ncells] = d.off + d.n;
        __syncthreads();
    }
}

// Scatter into the cell buckets in any order (k_cell_scatter)
__global__ void __launch_bounds__(kTile)
    k_b_cell_scatter(const BRep* __restrict__ reps, const int* __restrict__ tile_rep,
                     const int* __restrict__ stale_tiles, const int* __restrict__ work, const int* __restrict__ cell_of,
                     const int* __restrict__ start, int* __restrict__ cursor, uint32_t* __restrict__ bucket) {
    const int nw = work[1];
    for (int w = blockIdx.x; w < nw; w += gridDim.x) {
        int r, a;
        BRep d;
        if (!stale_slot(reps, tile_rep, stale_tiles, w, r, d, a)) continue;
        const int c = cell_of[a];
        bucket[start[d.cell_off + r + c] + atomicAdd(&cursor[d.cell_off + c], 1)] = static_cast<uint32_t>(a);
    }
}

// Stable order inside each cell: a particle's rank is the number of smaller slots in its bucket, as in the
// reference's serial scatter (src/CellList.cpp:48-51). Clears the scatter cursors for the next rebuild.
__global__ void __launch_bounds__(kTile)
    k_b_cell_rank(const BRep* __restrict__ reps, const int* __restrict__ tile_rep, const int* __restrict__ stale_tiles,
                  const int* __restrict__ work, const int* __restrict__ cell_of, const int* __restrict__ start,
                  int* __restrict__ cursor, const uint32_t* __restrict__ bucket, uint32_t* __restrict__ order) {
    const int nw = work[1];
    for (int w = blockIdx.x; w < nw; w += gridDim.x) {
        int r, a;
        BRep d;
        if (!stale_slot(reps, tile_rep, stale_tiles, w, r, d, a)) continue;
        const int c = cell_of[a];
        const int s = start[d.cell_off + r + c], e = start[d.cell_off + r + c + 1];
        int rank = 0;
        for (int f = s; f < e; ++f) rank += bucket[f] < static_cast<uint32_t>(a);
        order[s + rank] = static_cast<uint32_t>(a);
        cursor[d.cell_off + c] = 0;
    }
}

// new[a] = old[order[a]] inside each stale replica (src/System.cpp:42-64), into the scratch arrays; the sorted
// particles' cells go straight to cell_sorted
__global__ void __launch_bounds__(kTile)
    k_b_permute(const BRep* __restrict__ reps, const int* __restrict__ tile_rep, const int* __restrict__ stale_tiles,
                const int* __restrict__ work, const uint32_t* __restrict__ order, const int* __restrict__ cell_of,
                const double4* __restrict__ pos, const double* __restrict__ vel, const double* __restrict__ force,
                const double* __restrict__ mass, const uint64_t* __restrict__ ids, double4* __restrict__ pos2,
                double* __restrict__ vel2, double* __restrict__ force2, double* __restrict__ mass2,
                uint64_t* __restrict__ ids2, int* __restrict__ cell_sorted) {
    const int nw = work[1];
    for (int w = blockIdx.x; w < nw; w += gridDim.x) {
        int r, a;
        BRep d;
        if (!stale_slot(reps, tile_rep, stale_tiles, w, r, d, a)) continue;
        const int o = static_cast<int>(order[a]);
        pos2[a] = pos[o];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            vel2[bvec(d, k, a)] = vel[bvec(d, k, o)];
            force2[bvec(d, k, a)] = force[bvec(d, k, o)];
        }
        mass2[a] = mass[o];
        ids2[a] = ids[o];
        cell_sorted[a] = cell_of[o];
    }
}

// Copies the permuted arrays back and records the list's reference positions (src/NeighbourList.cpp:129-132)
// and the frames of the new order
__global__ void __launch_bounds__(kTile)
    k_b_commit(const BRep* __restrict__ reps, const int* __restrict__ tile_rep, const int* __restrict__ stale_tiles,
               const int* __restrict__ work, const double4* __restrict__ pos2, const double* __restrict__ vel2,
               const double* __restrict__ force2, const double* __restrict__ mass2, const uint64_t* __restrict__ ids2,
               const int* __restrict__ cell_sorted, double4* __restrict__ pos, double* __restrict__ vel,
               double* __restrict__ force, double* __restrict__ mass, uint64_t* __restrict__ ids,
               double4* __restrict__ ref_pos, float4* __restrict__ frames) {
    const int nw = work[1];
    for (int w = blockIdx.x; w < nw; w += gridDim.x) {
        int r, a;
        BRep d;
        if (!stale_slot(reps, tile_rep, stale_tiles, w, r, d, a)) continue;
        const double4 p = pos2[a];
        pos[a] = p;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            vel[bvec(d, k, a)] = vel2[bvec(d, k, a)];
            force[bvec(d, k, a)] = force2[bvec(d, k, a)];
        }
        mass[a] = mass2[a];
        ids[a] = ids2[a];
        ref_pos[a] = p;
        frames[a] = list_frame_of(p, cell_sorted[a], d.ncps, d.cell, d.box);
    }
}

// The six kernels above, cells to reordered particles, for a batch of small replicas: one block per stale replica, its
// cells, buckets and order in shared memory, the permuted arrays through the scratch arrays. The same integers and copies,
// so the same order. Either way latency bounds it, the launches and dependent loads of six kernels against the turns of one
// block: 128 replicas of 500 particles (B200, FP64, Bussi, 100 steps) 19.1 ms with six kernels, 17.9 with one; 33 of 2,048
// (FP32FX, 60 steps) 6.28 and 6.34; 100 of 500 to 6,912 15.3 and 17.2.
constexpr int kResortThreads = 1024;
constexpr int kResortMost = 1024;   // particles
constexpr int kResortCells = 4096;  // (39 KB of shared memory)
inline size_t resort_smem(int n, int cells) {
    return sizeof(int) * (2 * static_cast<size_t>(cells) + 1) + sizeof(uint16_t) * 3 * static_cast<size_t>(n);
}
__global__ void __launch_bounds__(kResortThreads)
    k_b_resort(const BRep* __restrict__ reps, const int* __restrict__ stale_reps, const int* __restrict__ work, int most_n,
               int most_cells, double4* pos, double* vel, double* force, double* mass, uint64_t* ids, double4* pos2,
               double* vel2, double* force2, double* mass2, uint64_t* ids2, int* __restrict__ start,
               int* __restrict__ cell_sorted, double4* __restrict__ ref_pos, float4* __restrict__ frames) {
    static_assert(kResortMost <= 65536 && kResortCells <= 65536, "cells and slots are kept in 16 bits");
    static_assert(sizeof(int) * (2 * kResortCells + 1) + 6 * kResortMost <= 48 * 1024, "no opt-in for shared memory");
    extern __shared__ float4 sm_cell[];
    __shared__ int s_warp[32];
    int* s_start = reinterpret_cast<int*>(sm_cell);          // [most_cells + 1]
    int* s_count = s_start + most_cells + 1;                 // [most_cells]: histogram, then scatter cursors
    uint16_t* s_cell = reinterpret_cast<uint16_t*>(s_count + most_cells);
    uint16_t* s_bucket = s_cell + most_n;
    uint16_t* s_order = s_bucket + most_n;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nr = work[0];
    for (int w = blockIdx.x; w < nr; w += gridDim.x) {
        const int r = stale_reps[w];
        const BRep d = reps[r];
        for (int c = t; c < d.ncells; c += kResortThreads) s_count[c] = 0;
        __syncthreads();
        for (int i = t; i < d.n; i += kResortThreads) {
            const double4 p = pos[d.off + i];
            const int c = (cell_coord(p.x, d.inv_cell, d.ncps) * d.ncps + cell_coord(p.y, d.inv_cell, d.ncps)) * d.ncps +
                          cell_coord(p.z, d.inv_cell, d.ncps);
            s_cell[i] = static_cast<uint16_t>(c);
            atomicAdd(&s_count[c], 1);
        }
        __syncthreads();
        int carry = 0;
        for (int c0 = 0; c0 < d.ncells; c0 += kResortThreads) {
            const int c = c0 + t;
            const int v = c < d.ncells ? s_count[c] : 0;
            const int x = inclusive_warp_scan(v);
            if (lane == 31) s_warp[warp] = x;
            __syncthreads();
            const int sums = inclusive_warp_scan(s_warp[lane]);  // (every warp scans the warps' sums)
            const int before = __shfl_sync(0xffffffffu, sums, warp ? warp - 1 : 0);
            const int e = carry + (warp ? before : 0) + x - v;
            if (c < d.ncells) {
                s_start[c] = e;
                s_count[c] = 0;
                start[d.cell_off + r + c] = d.off + e;
            }
            carry += __shfl_sync(0xffffffffu, sums, 31);
            __syncthreads();
        }
        if (t == 0) {
            s_start[d.ncells] = d.n;
            start[d.cell_off + r + d.ncells] = d.off + d.n;
        }
        __syncthreads();
        for (int i = t; i < d.n; i += kResortThreads) {
            const int c = s_cell[i];
            s_bucket[s_start[c] + atomicAdd(&s_count[c], 1)] = static_cast<uint16_t>(i);
        }
        __syncthreads();
        for (int i = t; i < d.n; i += kResortThreads) {
            const int c = s_cell[i], s = s_start[c], e = s_start[c + 1];
            int rank = 0;
            for (int f = s; f < e; ++f) rank += s_bucket[f] < i;
            s_order[s + rank] = static_cast<uint16_t>(i);
        }
        __syncthreads();
        for (int i = t; i < d.n; i += kResortThreads) {
            const int a = d.off + i, o = d.off + s_order[i];
            pos2[a] = pos[o];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                vel2[bvec(d, k, a)] = vel[bvec(d, k, o)];
                force2[bvec(d, k, a)] = force[bvec(d, k, o)];
            }
            mass2[a] = mass[o];
            ids2[a] = ids[o];
        }
        __syncthreads();
        for (int i = t; i < d.n; i += kResortThreads) {
            const int a = d.off + i, c = s_cell[s_order[i]];
            const double4 p = pos2[a];
            pos[a] = p;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                vel[bvec(d, k, a)] = vel2[bvec(d, k, a)];
                force[bvec(d, k, a)] = force2[bvec(d, k, a)];
            }
            mass[a] = mass2[a];
            ids[a] = ids2[a];
            ref_pos[a] = p;
            cell_sorted[a] = c;
            frames[a] = list_frame_of(p, c, d.ncps, d.cell, d.box);
        }
        __syncthreads();  // the next replica's cells go where this one's are read
    }
}

// The stale replica of a list-build item: the last w with stale_items[w] <= item
__device__ __forceinline__ int build_item_replica(const int* __restrict__ stale_items, int nr, int item) {
    int lo = 0, hi = nr;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (stale_items[mid] <= item) lo = mid; else hi = mid;
    }
    return lo;
}

// kAllGroup particles of a replica under 3 cells per side by the block's warps
template <int kWarps>
__device__ __forceinline__ void build_group_all(const BRep& d, int group, const double4* __restrict__ pos, const ListGeom& g,
                                                uint32_t* __restrict__ rows, int2* __restrict__ counts,
                                                int* __restrict__ max_count) {
    const int i0 = group * kAllGroup;
    for (int i = i0 + static_cast<int>(threadIdx.x >> 5); i < i0 + kAllGroup && i < d.n; i += kWarps)
        build_row_all(pos, d.off, d.off + d.n, g, d.off + i, rows, counts, max_count);
}

// The list build of the stale replicas (build_cell, with slots for indices): blocks take their cells in turn, and groups
// of particles of replicas under 3 cells per side, a warp per particle. In thin gases (kThinReplica) a block takes a tile, a
// thread per particle. bp.geom's box and cells per side are set per replica. max_count as in build_cell.
template <int kWarps, int kHomes, int kRound>
__global__ void __launch_bounds__(32 * kWarps)
    k_b_nlist_build(const BRep* __restrict__ reps, const int* __restrict__ stale_reps, const int* __restrict__ stale_items,
                    const int* __restrict__ work, const double4* __restrict__ pos, const float4* __restrict__ frames,
                    const int* __restrict__ start, const int* __restrict__ cell_sorted, CellBuild bp,
                    uint32_t* __restrict__ rows, int2* __restrict__ counts, int* __restrict__ max_count) {
    static_assert(kTile == 32 * kWarps, "a thread per particle of a tile");
    extern __shared__ float4 sm_cell[];
    __shared__ CellItems t;
    const int nr = work[0], total = work[2];
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
        const int w = build_item_replica(stale_items, nr, item), r = stale_reps[w];
        const BRep d = reps[r];
        bp.geom.box = d.box;
        bp.geom.ncps = d.ncps;
        bp.geom.use_cells = d.use_cells;
        const int* st = start + d.cell_off + r;
        const int part = item - stale_items[w];
        // an empty cell (the same for the whole block); replicas whose cells are hardly ever empty don't wait for the look
        if (d.use_cells == 1 && d.n < 8 * d.ncells && st[part] == st[part + 1]) continue;
        if (d.use_cells == 1) {
            build_cell<kWarps, kHomes, kRound>(t, sm_cell, frames, pos, st, part, static_cast<float>(d.cell), bp, rows, counts,
                                               max_count);
        } else if (d.use_cells == 2) {
            const int i = part * kTile + static_cast<int>(threadIdx.x);
            if (i < d.n) build_row(pos, bp.geom, d.off + i, cell_sorted[d.off + i], st, rows, counts, max_count);
        } else {
            build_group_all<kWarps>(d, part, pos, bp.geom, rows, counts, max_count);
        }
        __syncthreads();  // the shared memory goes to the next item
    }
}

// The same for a batch whose replicas are all under 3 cells per side, without build_cell's registers, stack and shared memory
__global__ void __launch_bounds__(kTile)
    k_b_nlist_build_all(const BRep* __restrict__ reps, const int* __restrict__ stale_reps, const int* __restrict__ stale_items,
                        const int* __restrict__ work, const double4* __restrict__ pos, ListGeom g, uint32_t* __restrict__ rows,
                        int2* __restrict__ counts, int* __restrict__ max_count) {
    const int nr = work[0], total = work[2];
    for (int item = blockIdx.x; item < total; item += gridDim.x) {
        const int w = build_item_replica(stale_items, nr, item);
        const BRep d = reps[stale_reps[w]];
        g.box = d.box;
        build_group_all<kTile / 32>(d, item - stale_items[w], pos, g, rows, counts, max_count);
    }
}

// ---- forces -------------------------------------------------------------------------------------------------

// First r^2 record of the replica in slot `off` on: rows name each pair from either end, so cap / 2 records a slot hold
// them (but for rows cut at the capacity, whose chunk is run again: records past the replica's end are dropped)
__device__ __forceinline__ long long brecords(int off, int cap) { return static_cast<long long>(off) * (cap >> 1); }

// computeForcesDeterministic's per-particle sums (fp64_row_quads, or Fp64Lanes with kLanes > 1 threads per particle and
// kLanes blocks per tile) per replica, with the closing half kick, the replica's inside-cutoff count into acc[4 r + 2] and,
// with pair_r2, the own pairs' r^2 records for the ordered energy sums at the replica's half-list offsets
template <int kLanes>
__global__ void __launch_bounds__(kTile)
    k_b_force_fp64(const BRep* __restrict__ reps, const int* __restrict__ tile_rep, const double4* __restrict__ pos,
                   LJ lj, const uint32_t* __restrict__ rows, int cap, const int2* __restrict__ counts,
                   double* __restrict__ force, unsigned long long* __restrict__ acc, double* __restrict__ kick_vel,
                   const double* __restrict__ mass, double half_dt, const int* __restrict__ half_off,
                   double* __restrict__ pair_r2) {
    const int t = blockIdx.x / kLanes, part = blockIdx.x % kLanes;
    const int r = tile_rep[t];
    const BRep d = reps[r];
    const int i = (t - d.tile_off) * kTile + part * (kTile / kLanes) + threadIdx.x / kLanes, u = threadIdx.x % kLanes;
    const bool real = i < d.n;
    const int a = real ? d.off + i : d.off;
    const int2 c = real ? counts[a] : make_int2(0, 0);
    const long long pb = pair_r2 ? brecords(d.off, cap) + half_off[a] : 0, end = brecords(d.off + d.np, cap);
    unsigned ins = 0;
    auto finish = [&](int k, double f) {
        const size_t o = bvec(d, k, a);
        force[o] = f;
        if (kick_vel) kick_vel[o] = dadd(kick_vel[o], ddiv(dmul(half_dt, f), mass[a]));
    };
    if constexpr (kLanes == 1) {
        const double3 f = fp64_row_quads(pos, a, d.box, lj, rows, cap, c, pair_r2, pb, end, ins);
        if (real) {
            finish(0, f.x);
            finish(1, f.y);
            finish(2, f.z);
        }
    } else {
        __shared__ double s_t[kTile / 32][Fp64Lanes<kLanes>::kTerms];
        const double f = Fp64Lanes<kLanes>::row(pos, a, d.box, lj, rows, cap, c, s_t[threadIdx.x >> 5], pair_r2, pb, end, ins);
        if (real && u < 3) finish(u, f);
    }
    count_inside(ins, &acc[4 * r + 2]);
}

// The float list forces per replica (k_force_fp32_rows and, for replicas under 3 cells per side,
// k_force_fp32_small), with the same pinned pair sequence and 8-entry groups (kPrefetch: rows one group ahead).
// Each block covers `apb`
// consecutive particles of one tile with kTPA threads per particle; thread u of a particle takes groups
// u, u + kTPA, ... and the threads' fixed-point sums are added as integers, so every (apb, kTPA) gives the same
// bits (kTPA > 1 only with fixed point). Per-replica sums go to acc[4 r .. 4 r + 3] (energy, virial, inside
// count, kinetic energy after the fused kick).
template <bool kFixed, bool kEnergy, int kTPA, bool kPrefetch = false>
__global__ void __launch_bounds__(256)
    k_b_force_fp32(const BRep* __restrict__ reps, const int* __restrict__ tile_rep, int apb,
                   const float4* __restrict__ frames, const double4* __restrict__ pos, FloatLJ lj,
                   const uint32_t* __restrict__ rows, int cap, const int2* __restrict__ counts,
                   double* __restrict__ force, unsigned long long* __restrict__ acc, double* __restrict__ kick_vel,
                   const double* __restrict__ mass, double half_dt) {
    static_assert(kFixed || kTPA == 1, "float accumulation keeps one thread per particle");
    // the replica's cell-code offsets as a table of (x, y) pairs and one of z: an 8- and a 4-byte shared load
    // per entry instead of one of 16 (fewer shared-memory wavefronts in the L1 data pipe)
    __shared__ __align__(16) float s_o[4][32];
    const int parts = kTile / apb;
    const int t = blockIdx.x / parts, part = blockIdx.x - t * parts;
    const int r = tile_rep[t];
    const BRep d = reps[r];
    if (threadIdx.x < 32) {
        const float4 o = code_offset(threadIdx.x, static_cast<float>(d.cell));
        reinterpret_cast<float2*>(s_o[0])[threadIdx.x] = make_float2(o.x, o.y);
        s_o[2][threadIdx.x] = o.z;
    }
    __syncthreads();
    const int sub = threadIdx.x % kTPA;
    const int i = (t - d.tile_off) * kTile + part * apb + threadIdx.x / kTPA;
    const bool active = i < d.n;
    const int a = d.off + i;
    long long e_fx = 0, w_fx = 0, k_fx = 0;
    unsigned ins = 0;
    FloatAcc<kFixed, kEnergy> acc_i;
    if (active) {
        const int2 c = counts[a];
        const int m = c.x + c.y;
        const int groups = (m + 7) >> 3;
        if (d.use_cells) {
            const float4 qi = frames[a];
            // with kPrefetch (one thread per particle) the next group's row quads are in flight while this
            // group's frames are gathered, as in k_force_fp32_rows
            uint4 n0 = make_uint4(0, 0, 0, 0), n1 = n0;
            if (kPrefetch && sub < groups) {
                n0 = row_quad_stream(rows, a, 2 * sub, cap);
                n1 = row_quad_stream(rows, a, 2 * sub + 1, cap);
            }
            for (int g = sub; g < groups; g += kTPA) {
                uint4 e0, e1;
                if (kPrefetch) {
                    e0 = n0;
                    e1 = n1;
                    if (g + kTPA < groups) {
                        n0 = row_quad_stream(rows, a, 2 * (g + kTPA), cap);
                        n1 = row_quad_stream(rows, a, 2 * (g + kTPA) + 1, cap);
                    }
                } else {
                    e0 = row_quad(rows, a, 2 * g, cap);
                    e1 = row_quad(rows, a, 2 * g + 1, cap);
                }
                const float2* s_xy = reinterpret_cast<const float2*>(s_o[0]);
                const float* s_z = s_o[2];
                const Box box = d.box;
                const GroupSums gs = float_group<kEnergy>(
                    e0, e1, lj,
                    [=](uint32_t e, float& dx, float& dy, float& dz) {
                        const uint32_t k = e >> kCodeShift;
                        const float2 oxy = s_xy[k];
                        return float_separation(qi, frames[e & kIndexMask], make_float4(oxy.x, oxy.y, s_z[k], 0.0f),
                                                dx, dy, dz);
                    },
                    [=](uint32_t e) { return exact_inside(pos[a], pos[e & kIndexMask], box, lj.rc2d); }, ins);
                acc_i.add_group(gs.x, gs.y, gs.z, gs.e, gs.w, e_fx, w_fx);
            }
        } else {
            const double4 pi = pos[a];
            for (int g = sub; g < groups; g += kTPA) {
                float gx = 0.f, gy = 0.f, gz = 0.f, ge = 0.f, gw = 0.f;
                for (int s = 8 * g; s < 8 * g + 8 && s < m; ++s) {
                    const double4 pj = pos[rows[row_index(a, s, cap)] & kIndexMask];
                    const double ddx = min_image(dsub(pi.x, pj.x), d.box);
                    const double ddy = min_image(dsub(pi.y, pj.y), d.box);
                    const double ddz = min_image(dsub(pi.z, pj.z), d.box);
                    const float dx = static_cast<float>(ddx), dy = static_cast<float>(ddy), dz = static_cast<float>(ddz);
                    const float r2 = fmaf(dx, dx, fmaf(dy, dy, __fmul_rn(dz, dz)));
                    const bool in = norm2(ddx, ddy, ddz) < lj.rc2d;
                    float_pair<kEnergy>(dx, dy, dz, in, r2, lj, gx, gy, gz, ge, gw, ins);
                }
                acc_i.add_group(gx, gy, gz, ge, gw, e_fx, w_fx);
            }
        }
    }
    if (kTPA > 1) {
#pragma unroll
        for (int o = 1; o < kTPA; o <<= 1) {
            acc_i.ax += __shfl_xor_sync(0xffffffffu, acc_i.ax, o);
            acc_i.ay += __shfl_xor_sync(0xffffffffu, acc_i.ay, o);
            acc_i.az += __shfl_xor_sync(0xffffffffu, acc_i.az, o);
        }
    }
    if (active && sub == 0) {
        const double F[3] = {kFixed ? static_cast<double>(acc_i.ax) * kForceUnit : static_cast<double>(acc_i.fx),
                             kFixed ? static_cast<double>(acc_i.ay) * kForceUnit : static_cast<double>(acc_i.fy),
                             kFixed ? static_cast<double>(acc_i.az) * kForceUnit : static_cast<double>(acc_i.fz)};
        double ke = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const size_t o = bvec(d, k, a);
            force[o] = F[k];
            if (kick_vel) {  // as FloatAcc::finish
                const double v = dadd(kick_vel[o], ddiv(dmul(half_dt, F[k]), mass[a]));
                kick_vel[o] = v;
                ke = dadd(ke, dmul(v, v));
            }
        }
        if (kick_vel) k_fx = __double2ll_rn(dmul(dmul(dmul(0.5, mass[a]), ke), kKineticScale));
    }
    if (kEnergy || kick_vel) flush_sums(e_fx, w_fx, ins, k_fx, acc + 4 * r);
}

// Per replica: the fixed-point sums of the float kernels as doubles (k_finish_float_energy's conversions), the
// kinetic energy into ke[r] when `kinetic`, energy and virial into pe_out/w_out when given; clears acc
__global__ void k_b_finish_float(int R, unsigned long long* __restrict__ acc, bool kinetic, double* __restrict__ ke,
                                 double* __restrict__ pe_out, double* __restrict__ w_out,
                                 unsigned long long* __restrict__ inside) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= R) return;
    unsigned long long* s = acc + 4 * r;
    if (pe_out) pe_out[r] = 0.5 * static_cast<double>(static_cast<long long>(s[0])) * kEnergyUnit;
    if (w_out) w_out[r] = 0.5 * static_cast<double>(static_cast<long long>(s[1])) * kEnergyUnit;
    if (inside) inside[r] = s[2] / 2;
    if (kinetic) ke[r] = static_cast<double>(static_cast<long long>(s[3])) * (1.0 / kKineticScale);
    s[0] = s[1] = s[2] = s[3] = 0;
}

// Inside-cutoff counts of the FP64 kernel (acc[4 r + 2]) into inside[r]; clears acc
__global__ void k_b_finish_fp64(int R, unsigned long long* __restrict__ acc, unsigned long long* __restrict__ inside,
                                double* __restrict__ record) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= R) return;
    unsigned long long* s = acc + 4 * r;
    if (inside) inside[r] = s[2];
    if (record) record[r] = static_cast<double>(s[2]);
    s[0] = s[1] = s[2] = s[3] = 0;
}

// The inside-cutoff count of every replica's last force evaluation into a record row (doubles)
__global__ void k_b_record_inside(int R, const unsigned long long* __restrict__ inside, double* __restrict__ out) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < R) out[r] = static_cast<double>(inside[r]);
}

// ---- kinetic energy and thermostats ---------------------------------------------------------------------------

// System::kineticEnergy's blocked sum (k_kinetic_blocks) per replica: one block per 1024-particle block of a
// replica; with `scale` the pending thermostat scale is applied to each velocity first (the kinetic energy
// after scaleVelocities).
__global__ void __launch_bounds__(kOrderedThreads)
    k_b_kinetic_blocks(const BRep* __restrict__ reps, const int* __restrict__ chunk_rep, const double* __restrict__ vel,
                       const double* __restrict__ mass, const double2* __restrict__ scale, double* __restrict__ chunk_sums) {
    __shared__ OrderedSmem<1, kChunk / kOrderedThreads> sm;
    const int r = chunk_rep[blockIdx.x];
    const BRep d = reps[r];
    const int i0 = (blockIdx.x - d.chunk_off) * kChunk;
    const int m = d.n - i0 < kChunk ? d.n - i0 : kChunk;
    const double2 sc = scale ? scale[r] : make_double2(1.0, 0.0);
    if (threadIdx.x == 0) sm.run[0] = 0.0;
    ordered_sum(sm, m, [&](long long q, double* v) {
        const int a = d.off + i0 + static_cast<int>(q);
        double c[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            c[k] = vel[bvec(d, k, a)];
            if (sc.y != 0.0) c[k] = dmul(c[k], sc.x);
        }
        v[0] = dmul(dmul(0.5, mass[a]), norm2(c[0], c[1], c[2]));
    });
    if (threadIdx.x == 0) chunk_sums[blockIdx.x] = sm.run[0];
}

// A step's thermostat: mode 0 none, 1 rescale, 2 Bussi (r1, chi2: the replicas' draws); the factors go to scale
struct BThermostat {
    int mode;
    double c;
    const double* r1;
    const double* chi2;
    double2* scale;
};
__device__ __forceinline__ void thermostat_scale(const BThermostat& t, const BRep& d, int r, double kinetic) {
    double2 out = make_double2(1.0, 0.0);
    if (t.mode == 1) {
        const double T = ddiv(dmul(2.0, kinetic), d.dof);
        if (T > 0.0) out = make_double2(__dsqrt_rn(ddiv(d.temperature, T)), 1.0);
    } else if (kinetic > 0.0) {
        out = make_double2(bussi_scale(kinetic, d.dof, d.temperature, t.c, t.r1[r], t.chi2[r]), 1.0);
    }
    t.scale[r] = out;
}

// deterministicSum's outer loop per replica: its block sums added in order; one warp per replica
__global__ void k_b_sum_chunks(const BRep* __restrict__ reps, int R, const double* __restrict__ chunk_sums,
                               double* __restrict__ out, BThermostat thermo) {
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= R) return;
    const BRep d = reps[r];
    const int nb = (d.n + kChunk - 1) / kChunk;
    double s = 0.0;
    for (int b0 = 0; b0 < nb; b0 += 32) {
        const double v = b0 + lane < nb ? chunk_sums[d.chunk_off + b0 + lane] : 0.0;
        const int m = nb - b0 < 32 ? nb - b0 : 32;
        for (int t = 0; t < m; ++t) {
            const double x = __shfl_sync(0xffffffffu, v, t);
            if (lane == 0) s = dadd(s, x);
        }
    }
    if (lane == 0) {
        out[r] = s;
        if (thermo.mode) thermostat_scale(thermo, d, r, s);
    }
}

// Fixed-point kinetic energy per replica (k_kinetic_fixed) with the pending scale applied, into acc[4 r + 3]
__global__ void __launch_bounds__(kTile)
    k_b_kinetic_fixed(const BRep* __restrict__ reps, const int* __restrict__ tile_rep, const double* __restrict__ vel,
                      const double* __restrict__ mass, const double2* __restrict__ scale,
                      unsigned long long* __restrict__ acc) {
    const int r = tile_rep[blockIdx.x];
    const BRep d = reps[r];
    const int i = (blockIdx.x - d.tile_off) * kTile + threadIdx.x;
    long long v = 0;
    if (i < d.n) {
        const int a = d.off + i;
        const double2 sc = scale[r];
        double ke = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            double x = vel[bvec(d, k, a)];
            if (sc.y != 0.0) x = dmul(x, sc.x);
            ke = dadd(ke, dmul(x, x));
        }
        v = __double2ll_rn(dmul(dmul(dmul(0.5, mass[a]), ke), kKineticScale));
    }
    v = warp_sum_i64(v);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&acc[4 * r + 3], static_cast<unsigned long long>(v));
}

// Thermostat factors per replica into scale[r] = (factor, 1), or (1, 0) to leave the replica alone.
// mode 1: rescaleVelocities to the replica's temperature (src/Thermostat.cpp:17-30); mode 2: Bussi with the
// step's draws r1[r], chi2[r] (src/Thermostat.cpp:36-58).
__global__ void k_b_thermostat(const BRep* __restrict__ reps, int R, const double* __restrict__ ke, BThermostat t) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r < R) thermostat_scale(t, reps[r], r, ke[r]);
}

// ---- FP64 energy and virial in the reference's pair order ----------------------------------------------------

// Exclusive prefix of each replica's own-pair counts (the half-list CSR offsets, src/NeighbourList.cpp:116-127)
// into half_off[slot] and the replica's pair count into pairs[r]; one block per replica
__global__ void __launch_bounds__(kRepScanThreads)
    k_b_half_offsets(const BRep* __restrict__ reps, int R, const int2* __restrict__ counts, int* __restrict__ half_off,
                     int* __restrict__ pairs) {
    __shared__ int s_warp[32];
    __shared__ int s_carry;
    for (int r = blockIdx.x; r < R; r += gridDim.x) {
        const BRep d = reps[r];
        if (threadIdx.x == 0) s_carry = 0;
        __syncthreads();
        for (int i0 = 0; i0 < d.n; i0 += kRepScanThreads) {
            const int i = i0 + threadIdx.x;
            const int v = i < d.n ? counts[d.off + i].x : 0;
            const int e = block_scan_carry(v, s_warp, &s_carry);
            if (i < d.n) half_off[d.off + i] = e;
        }
        if (threadIdx.x == 0) pairs[r] = s_carry;
        __syncthreads();
    }
}

// item_off[r] = number of 1024-pair blocks of the replicas before r; item_off[R] the total. One block.
__global__ void __launch_bounds__(kRepScanThreads) k_b_pair_items(int R, const int* __restrict__ pairs,
                                                               int* __restrict__ item_off) {
    __shared__ int s_warp[32];
    __shared__ int s_carry;
    if (threadIdx.x == 0) s_carry = 0;
    __syncthreads();
    for (int r0 = 0; r0 < R; r0 += kRepScanThreads) {
        const int r = r0 + threadIdx.x;
        const int v = r < R ? (pairs[r] + kChunk - 1) / kChunk : 0;
        const int e = block_scan_carry(v, s_warp, &s_carry);
        if (r < R) item_off[r] = e;
    }
    if (threadIdx.x == 0) item_off[R] = s_carry;
}

// Per replica: energy and virial of each 1024-pair block of the half list in the reference's pair order, summed
// from 0.0 one after another (deterministicSum's inner loop, include/Parallel.hpp:43-46; pairEnergy/pairVirial
// of src/Forcefield.cpp:288-296), from the force kernel's r^2 records (pair_block_sums). Each warp takes blocks (items)
// of all replicas in turn. (Evaluated from the positions, particle by particle, with one lane adding, the 3,900 blocks of
// 128 replicas of 500 particles took 120 us.)
__global__ void __launch_bounds__(32 * kSumWarps)
    k_b_energy_blocks(const BRep* __restrict__ reps, int R, const int* __restrict__ item_off,
                      const int* __restrict__ pairs, const double* __restrict__ pair_r2, LJ lj, int cap,
                      double2* __restrict__ item_sums) {
    __shared__ double2 s_term[kSumWarps][kSumStage + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total = item_off[R];
    for (int item = blockIdx.x * kSumWarps + warp; item < total; item += gridDim.x * kSumWarps) {
        int lo = 0, hi = R;  // the replica: last r with item_off[r] <= item
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (item_off[mid] <= item) lo = mid; else hi = mid;
        }
        const BRep d = reps[lo];
        const int k0 = (item - item_off[lo]) * kChunk;
        const long long all = pairs[lo], most = brecords(d.np, cap), left = (all < most ? all : most) - k0;
        const double* rec = pair_r2 + brecords(d.off, cap) + k0;
        const double sum = pair_block_sums<1>(s_term[warp], lj, [&](int, int k) { return k < left ? __ldcs(rec + k) : lj.rc2; });
        if (lane < 2) reinterpret_cast<double*>(item_sums + item)[lane] = sum;
    }
}

// The replica's block sums added in order (k_sum_blocks); one warp per replica
__global__ void k_b_sum_items(int R, const int* __restrict__ item_off, const double2* __restrict__ item_sums,
                              double* __restrict__ pe_out, double* __restrict__ w_out) {
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= R) return;
    const int b = item_off[r], nb = item_off[r + 1] - b;
    double se = 0.0, sw = 0.0;
    for (int b0 = 0; b0 < nb; b0 += 32) {
        const double2 v = b0 + lane < nb ? item_sums[b + b0 + lane] : make_double2(0.0, 0.0);
        const int m = nb - b0 < 32 ? nb - b0 : 32;
        for (int t = 0; t < m; ++t) {
            const double x = __shfl_sync(0xffffffffu, v.x, t);
            const double y = __shfl_sync(0xffffffffu, v.y, t);
            if (lane == 0) {
                se = dadd(se, x);
                sw = dadd(sw, y);
            }
        }
    }
    if (lane == 0) {
        pe_out[r] = se;
        w_out[r] = sw;
    }
}

// Moves row entries from a capacity-`cap0` buffer to a capacity-`cap1` one (cap1 > cap0), one thread per slot
__global__ void k_b_relayout_rows(int slots, const int2* __restrict__ counts, const uint32_t* __restrict__ src, int cap0,
                                  uint32_t* __restrict__ dst, int cap1) {
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= slots) return;
    const int2 c = counts[a];
    const int m = (c.x + c.y + 7) & ~7;
    for (int s = 0; s < m && s < cap0; ++s) dst[row_index(a, s, cap1)] = src[row_index(a, s, cap0)];
}

}  // namespace md
