// Double-precision kernels that reproduce the reference bit for bit: list forces in the deterministic
// summation order, the blocked energy/virial/kinetic sums, velocity Verlet, the half-skin check, thermostats
// and the g(r) histogram.
#pragma once

#include "md_common.cuh"
#include "md_ordered.cuh"

namespace md {

constexpr int kChainValues = 8;  // values per thread of a one-block ordered sum (45 KB of shared memory)

// ---- forces -----------------------------------------------------------------------------------------

// A block's inside-cutoff pairs into *inside by one atomic (every thread calls)
__device__ __forceinline__ void count_inside(unsigned ins, unsigned long long* __restrict__ inside) {
    __shared__ unsigned s_ins[32];
    ins = __reduce_add_sync(0xffffffffu, ins);
    if ((threadIdx.x & 31) == 0) s_ins[threadIdx.x >> 5] = ins;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (unsigned w = 0; w < (blockDim.x + 31) / 32; ++w) t += s_ins[w];
        if (t) atomicAdd(inside, t);
    }
}

// computeForcesDeterministic's per-particle sum (src/Forcefield.cpp:264-320): particle i adds F(i, j) over
// its own pairs in list order, then subtracts F(j, i) over the pairs where it is second, in increasing pair
// index. Pairs outside the cutoff contribute an exact zero in the reference and are skipped here. The
// inside-cutoff count is the number of own pairs with r^2 < r_c^2 (a sum of whole numbers, exact).
// With kick_vel set it also applies the closing half kick, v += (half_dt F) / m, with k_kick's sequence.
// With pair_r2 set, own pair s of particle i also stores its r^2, inside the cutoff or not, for the ordered energy sums
// at index half_off[i] + s; k_pair_block_sums recomputes the pair's E and (F/r) r^2 from it with the same pair_terms
// call (the same operations on the same r^2, so the same bits). Records past rec_cap, the buffer's size in records, are
// dropped: only a list rebuilt inside a CUDA graph can outgrow the buffer, and the graph's run then reports the overflow
// and repeats its steps on the host path.
__global__ void k_force_fp64(const double4* __restrict__ pos, int n, Box box, LJ lj, const uint32_t* __restrict__ rows,
                             int cap, const int2* __restrict__ counts, double* __restrict__ force,
                             unsigned long long* __restrict__ inside, double* __restrict__ kick_vel,
                             const double* __restrict__ mass, double half_dt, const long long* __restrict__ half_off,
                             double* __restrict__ pair_r2, long long rec_cap) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long ins = 0;
    if (i < n) {
        const double4 pi = pos[i];
        const int2 c = counts[i];
        const long long pb = pair_r2 ? half_off[i] : 0;
        double fx = 0.0, fy = 0.0, fz = 0.0;
        for (int s = 0; s < c.x; ++s) {
            const double4 pj = pos[rows[row_index(i, s, cap)] & kIndexMask];
            const double dx = min_image(dsub(pi.x, pj.x), box);
            const double dy = min_image(dsub(pi.y, pj.y), box);
            const double dz = min_image(dsub(pi.z, pj.z), box);
            const double r2 = norm2(dx, dy, dz);
            if (pair_r2 && pb + s < rec_cap) pair_r2[pb + s] = r2;
            if (!(r2 < lj.rc2)) continue;
            double f, e;
            pair_terms(r2, lj, f, e);
            fx = dadd(fx, dmul(f, dx));
            fy = dadd(fy, dmul(f, dy));
            fz = dadd(fz, dmul(f, dz));
            ++ins;
        }
        for (int s = c.x; s < c.x + c.y; ++s) {
            const double4 pj = pos[rows[row_index(i, s, cap)] & kIndexMask];
            const double dx = min_image(dsub(pj.x, pi.x), box);
            const double dy = min_image(dsub(pj.y, pi.y), box);
            const double dz = min_image(dsub(pj.z, pi.z), box);
            const double r2 = norm2(dx, dy, dz);
            if (!(r2 < lj.rc2)) continue;
            double f, e;
            pair_terms(r2, lj, f, e);
            fx = dsub(fx, dmul(f, dx));
            fy = dsub(fy, dmul(f, dy));
            fz = dsub(fz, dmul(f, dz));
        }
        const double F[3] = {fx, fy, fz};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const size_t o = static_cast<size_t>(k) * n + i;
            force[o] = F[k];
            if (kick_vel) kick_vel[o] = dadd(kick_vel[o], ddiv(dmul(half_dt, F[k]), mass[i]));
        }
    }
    ins = warp_sum_u64(ins);
    if ((threadIdx.x & 31) == 0 && ins) atomicAdd(inside, ins);
}

// Variant 2 of k_force_fp64, the same sums without a branch per entry: the row is read a quad (4 entries) at a
// time, one quad ahead with the streaming hint, the quad's four neighbour positions are gathered together, and
// every entry's terms are evaluated and masked (an exact 0.0 outside r_c and for the row's padding). Own and
// reverse entries take one form: the reverse pair's -F(j, i) dx(j, i) equals +F dx(i, j), since min_image is
// odd (round() and the |d| <= L/4 shortcut are symmetric) and IEEE subtraction antisymmetric, so each sum sees
// the reference's nonzero terms in the reference's order; a masked 0.0 leaves a sum unchanged because a sum
// that starts at +0.0 never becomes -0.0.
// Positions come in by one 32-byte load each (two of 16 bytes: 266 us at N = 864,000 without records, now 254), and
// the r^2 records go out by whole aligned quads of 32 bytes, shifted into place in registers (stored one by one: 493 us
// with records, now 352). What bounds it: gather and store latency at 40 % of the FP64 pipe's time.
// Particle i's sum and its count of own pairs inside the cutoff (added to ins), with rec its r^2 records from index pb on
__device__ __forceinline__ double3 fp64_row_quads(const double4* __restrict__ pos, int i, const Box& box, const LJ& lj,
                                                  const uint32_t* __restrict__ rows, int cap, const int2 c,
                                                  double* __restrict__ rec, long long pb, long long rec_cap,
                                                  unsigned& ins) {
    const double4 pi = load_pos(pos + i);
    const int m = c.x + c.y;
    const int quads = (m + 3) >> 2;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    const uint4* rq = reinterpret_cast<const uint4*>(rows) + static_cast<size_t>(i >> 5) * (cap >> 2) * 32 + (i & 31);
    uint4 nq = make_uint4(0, 0, 0, 0);
    if (quads > 0) nq = __ldcs(rq);
    // record k of the array belongs to the aligned quad k >> 2, which is written whole once its four are known; the quads
    // at either end of the particle's range are shared with its neighbours
    const int shift = static_cast<int>(pb & 3);
    double h0 = 0.0, h1 = 0.0, h2 = 0.0;  // the last records of the open aligned quad
    for (int q = 0; q < quads; ++q) {
        const uint4 eq = nq;
        if (q + 1 < quads) nq = __ldcs(rq + 32 * (q + 1));
        const uint32_t ent[4] = {eq.x, eq.y, eq.z, eq.w};
        double4 pj[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) pj[u] = load_pos(pos + (4 * q + u < m ? static_cast<int>(ent[u] & kIndexMask) : i));
        double r[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int sl = 4 * q + u;
            const double dx = min_image(dsub(pi.x, pj[u].x), box);
            const double dy = min_image(dsub(pi.y, pj[u].y), box);
            const double dz = min_image(dsub(pi.z, pj[u].z), box);
            const double r2 = norm2(dx, dy, dz);
            const bool in = sl < m && r2 < lj.rc2;
            double f, e;
            pair_terms(in ? r2 : 1.0, lj, f, e);
            fx = dadd(fx, in ? dmul(f, dx) : 0.0);
            fy = dadd(fy, in ? dmul(f, dy) : 0.0);
            fz = dadd(fz, in ? dmul(f, dz) : 0.0);
            r[u] = r2;
            ins += in && sl < c.x ? 1u : 0u;
        }
        if (rec && 4 * q < c.x) {
            // the aligned quad that ends inside this step's four: `shift` held back, 4 - shift new
            const double a0 = shift == 0 ? r[0] : shift == 1 ? h2 : shift == 2 ? h1 : h0;
            const double a1 = shift == 0 ? r[1] : shift == 1 ? r[0] : shift == 2 ? h2 : h1;
            const double a2 = shift == 0 ? r[2] : shift == 1 ? r[1] : shift == 2 ? r[0] : h2;
            const double a3 = shift == 0 ? r[3] : shift == 1 ? r[2] : shift == 2 ? r[1] : r[0];
            const long long k = pb - shift + 4 * q;
            const int s0 = 4 * q - shift;  // row entry of a0
            if (s0 >= 0 && s0 + 4 <= c.x && k + 4 <= rec_cap) {
                store_4(rec + k, a0, a1, a2, a3);
            } else {
                if (s0 >= 0 && s0 < c.x && k < rec_cap) rec[k] = a0;
                if (s0 >= -1 && s0 + 1 < c.x && k + 1 < rec_cap) rec[k + 1] = a1;
                if (s0 >= -2 && s0 + 2 < c.x && k + 2 < rec_cap) rec[k + 2] = a2;
                if (s0 + 3 < c.x && k + 3 < rec_cap) rec[k + 3] = a3;
            }
            if (4 * q + 4 >= c.x) {  // the last step with own pairs: the records still held back
                const int s1 = s0 + 4;
                const double b0 = shift == 1 ? r[3] : shift == 2 ? r[2] : r[1];
                const double b1 = shift == 2 ? r[3] : r[2];
                if (shift >= 1 && s1 < c.x && k + 4 < rec_cap) rec[k + 4] = b0;
                if (shift >= 2 && s1 + 1 < c.x && k + 5 < rec_cap) rec[k + 5] = b1;
                if (shift >= 3 && s1 + 2 < c.x && k + 6 < rec_cap) rec[k + 6] = r[3];
            }
            h0 = r[1];
            h1 = r[2];
            h2 = r[3];
        }
    }
    return make_double3(fx, fy, fz);
}

__global__ void __launch_bounds__(128) k_force_fp64_quads(const double4* __restrict__ pos, int n, Box box, LJ lj,
                                                          const uint32_t* __restrict__ rows, int cap,
                                                          const int2* __restrict__ counts, double* __restrict__ force,
                                                          unsigned long long* __restrict__ inside,
                                                          double* __restrict__ kick_vel, const double* __restrict__ mass,
                                                          double half_dt, const long long* __restrict__ half_off,
                                                          double* __restrict__ pair_r2, long long rec_cap) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned ins = 0;
    if (i < n) {
        const double3 f = fp64_row_quads(pos, i, box, lj, rows, cap, counts[i], pair_r2, pair_r2 ? half_off[i] : 0, rec_cap,
                                         ins);
        const double F[3] = {f.x, f.y, f.z};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const size_t o = static_cast<size_t>(k) * n + i;
            force[o] = F[k];
            if (kick_vel) kick_vel[o] = dadd(kick_vel[o], ddiv(dmul(half_dt, F[k]), mass[i]));
        }
    }
    count_inside(ins, inside);
}

// The sums of k_force_fp64_quads with kLanes threads per particle: the lanes evaluate kLanes row entries at once and
// leave the terms in shared memory, where three of them add the x, y and z terms one after another in row order, so the
// sums are the same. Entries are read two steps and positions one step ahead. The energy records of consecutive row
// entries go out side by side.
// For small systems: a thread per particle leaves most of the GPU without a warp (2,048 particles are 64 of them) and
// walks its row in one long chain of gathers. Measured with records stored (B200, us; threads per particle 1 / 4 / 8 /
// 16): N = 500: 37 / 18 / 13 / 11; 2,048: 37 / 18 / 14 / 12; 10,976: 37 / 19 / 16 / 22; 32,000: 40 / 26 / 30 / 35;
// 108,000: 54 / 61 / 70 / 84; 65,536 slots of 128 replicas with rows of 124 entries: 55 / 61 (1 / 4). The lines between
// them follow: past about 50,000 particles the GPU is full either way and the shared-memory pass only costs.
constexpr int kFp64Lanes16 = 8192, kFp64Lanes8 = 24576, kFp64Lanes4 = 48000;
template <int kLanes>
struct Fp64Lanes {
    static constexpr int kGroups = 32 / kLanes, kPad = kLanes + 1, kRow = kGroups * kPad + 1;
    static constexpr int kTerms = 3 * kRow;  // doubles of shared memory a warp needs
    // Lane u of particle i's kLanes (a whole warp calls; c is (0, 0) where there is no particle): component u of the
    // force in lanes 0 to 2, the lane's count of own pairs inside the cutoff added to ins, and with rec the r^2 records
    // from index pb on
    static __device__ __forceinline__ double row(const double4* __restrict__ pos, int i, const Box& box, const LJ& lj,
                                                 const uint32_t* __restrict__ rows, int cap, const int2 c,
                                                 double* warp_terms, double* __restrict__ rec, long long pb,
                                                 long long rec_cap, unsigned& ins) {
        const int lane = threadIdx.x & 31, u = lane % kLanes;
        double* terms = warp_terms + (lane / kLanes) * kPad;  // component k of the group's entry t at terms[k * kRow + t]
        const int m = c.x + c.y;
        const double4 pi = load_pos(pos + i);
        // the longest row of the warp's particles: every lane takes part in the warp's steps
        int steps = (m + kLanes - 1) / kLanes;
#pragma unroll
        for (int o = kLanes; o < 32; o <<= 1) steps = max(steps, __shfl_xor_sync(0xffffffffu, steps, o));
        auto entry = [&](int s) { return s < m ? static_cast<int>(rows[row_index(i, s, cap)] & kIndexMask) : i; };
        double sum = 0.0;
        int j1 = entry(u + kLanes);
        double4 pj = load_pos(pos + entry(u));
        for (int q = 0; q < steps; ++q) {
            const int s = q * kLanes + u;
            const double dx = min_image(dsub(pi.x, pj.x), box);
            const double dy = min_image(dsub(pi.y, pj.y), box);
            const double dz = min_image(dsub(pi.z, pj.z), box);
            pj = load_pos(pos + j1);
            j1 = entry(s + 2 * kLanes);
            const double r2 = norm2(dx, dy, dz);
            const bool in = s < m && r2 < lj.rc2;
            double f, e;
            pair_terms(in ? r2 : 1.0, lj, f, e);
            terms[u] = in ? dmul(f, dx) : 0.0;
            terms[kRow + u] = in ? dmul(f, dy) : 0.0;
            terms[2 * kRow + u] = in ? dmul(f, dz) : 0.0;
            if (s < c.x) {
                ins += in ? 1u : 0u;
                if (rec && pb + s < rec_cap) rec[pb + s] = r2;
            }
            __syncwarp();
            if (u < 3) {
                const double* mine = terms + u * kRow;
                double t[kLanes];
#pragma unroll
                for (int k = 0; k < kLanes; ++k) t[k] = mine[k];
#pragma unroll
                for (int k = 0; k < kLanes; ++k) sum = dadd(sum, t[k]);
            }
            __syncwarp();
        }
        return sum;
    }
};

template <int kLanes>
__global__ void __launch_bounds__(128) k_force_fp64_lanes(const double4* __restrict__ pos, int n, Box box, LJ lj,
                                                          const uint32_t* __restrict__ rows, int cap,
                                                          const int2* __restrict__ counts, double* __restrict__ force,
                                                          unsigned long long* __restrict__ inside,
                                                          double* __restrict__ kick_vel, const double* __restrict__ mass,
                                                          double half_dt, const long long* __restrict__ half_off,
                                                          double* __restrict__ pair_r2, long long rec_cap) {
    __shared__ double s_t[4][Fp64Lanes<kLanes>::kTerms];
    const int i = static_cast<int>((blockIdx.x * 128 + threadIdx.x) / kLanes), u = threadIdx.x % kLanes;
    const bool real = i < n;
    unsigned ins = 0;
    const double f = Fp64Lanes<kLanes>::row(pos, real ? i : 0, box, lj, rows, cap, real ? counts[i] : make_int2(0, 0),
                                            s_t[threadIdx.x >> 5], pair_r2, pair_r2 && real ? half_off[i] : 0, rec_cap, ins);
    if (real && u < 3) {
        const size_t o = static_cast<size_t>(u) * n + i;
        force[o] = f;
        if (kick_vel) kick_vel[o] = dadd(kick_vel[o], ddiv(dmul(half_dt, f), mass[i]));
    }
    count_inside(ins, inside);
}

// Adds x[0], x[stride], ... x[(m - 1) stride] to s one after another. One thread's chain, bound by the latency of an
// addition (8 cycles): the next eight values are on their way from shared memory while the current ones are added.
__device__ __forceinline__ double add_in_order(const double* x, int stride, int m, double s) {
    double v[8];
    int k = 0;
    if (m >= 8) {
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = x[u * stride];
        for (; k + 16 <= m; k += 8) {
            double w[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) w[u] = x[(k + 8 + u) * stride];
#pragma unroll
            for (int u = 0; u < 8; ++u) s = dadd(s, v[u]);
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = w[u];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) s = dadd(s, v[u]);
        k += 8;
    }
    for (; k < m; ++k) s = dadd(s, x[k * stride]);
    return s;
}

// The inner loop of deterministicSum (include/Parallel.hpp:43-46) over the (pairEnergy, pairVirial) array, whose
// terms are recomputed here from the r^2 records the force kernel stored: block b sums pairs
// [1024 b, 1024 b + 1024) from 0.0 one after another, a pair outside the cutoff adding 0.0 as the reference's
// zero entries do (src/Forcefield.cpp:288-296).
// A warp advances kBlocks blocks together: its 32 lanes evaluate 256 / kBlocks records of each into shared memory (the
// next ones already loaded), then 2 kBlocks lanes, one per block and sum, add them in order. kBlocks = 1 finishes
// soonest, 4 spends the fewest instructions a block (the additions of 8 chains issue together).
constexpr int kSumWarps = 4;
constexpr int kSumStage = 256;  // records a warp holds
// The pair count is rec_cap, or, in a CUDA graph (where it is known only on the device), read from *pair_count
// (the step's copy of the list's count, so a rebuild for the next step cannot change it under the sums) and capped
// at rec_cap, the records' buffer size; the grid then covers rec_cap. The block count goes to *nblocks_out for
// k_sum_pair_blocks.
// The warp's part: r2_at(b, k) is record k of its block b (r_c^2 past the end, which adds 0.0); returns, in the lanes
// below 2 kBlocks, the sum of lane & 1 (energy, virial) of block lane >> 1. term: kSumStage + kBlocks records of shared
// memory.
template <int kBlocks, typename Load>
__device__ __forceinline__ double pair_block_sums(double2* term, const LJ& lj, Load r2_at) {
    constexpr int kEach = kSumStage / kBlocks;  // records of a block per step
    const int lane = threadIdx.x & 31;
    double r2[kSumStage / 32];  // record k of block b goes to term[b (kEach + 1) + k]
    auto fetch = [&](int step) {
#pragma unroll
        for (int q = 0; q < kSumStage / 32; ++q) r2[q] = r2_at(q * 32 / kEach, step * kEach + q * 32 % kEach + lane);
    };
    fetch(0);
    double sum = 0.0;
    for (int step = 0; step < kChunk / kEach; ++step) {
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kSumStage / 32; ++q) {
            const int b = q * 32 / kEach, k = q * 32 % kEach + lane;
            const bool in = r2[q] < lj.rc2;
            double f, e;
            pair_terms(in ? r2[q] : 1.0, lj, f, e);
            term[b * (kEach + 1) + k] = in ? make_double2(e, dmul(f, r2[q])) : make_double2(0.0, 0.0);
        }
        __syncwarp();
        if (step + 1 < kChunk / kEach) fetch(step + 1);
        if (lane < 2 * kBlocks)
            sum = add_in_order(reinterpret_cast<const double*>(term + (lane >> 1) * (kEach + 1)) + (lane & 1), 2, kEach, sum);
    }
    return sum;
}

template <int kBlocks>
__global__ void __launch_bounds__(32 * kSumWarps) k_pair_block_sums(const double* __restrict__ pair_r2,
                                                                    const long long* __restrict__ pair_count,
                                                                    long long rec_cap, LJ lj,
                                                                    double2* __restrict__ block_sums,
                                                                    int* __restrict__ nblocks_out) {
    __shared__ double2 s_term[kSumWarps][kSumStage + kBlocks];
    const long long count = pair_count ? *pair_count : rec_cap;
    const long long pairs = count < rec_cap ? count : rec_cap;
    const int nblocks = static_cast<int>((pairs + kChunk - 1) / kChunk);
    if (blockIdx.x == 0 && threadIdx.x == 0) *nblocks_out = nblocks;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b0 = (blockIdx.x * kSumWarps + warp) * kBlocks;
    if (b0 >= nblocks) return;
    const double sum = pair_block_sums<kBlocks>(s_term[warp], lj, [&](int b, int k) {
        const long long at = static_cast<long long>(b0 + b) * kChunk + k;
        return at < pairs ? __ldcs(pair_r2 + at) : lj.rc2;
    });
    const int b = b0 + (lane >> 1);
    if (lane < 2 * kBlocks && b < nblocks) reinterpret_cast<double*>(block_sums + b)[lane & 1] = sum;
}

// The outer loop of deterministicSum (include/Parallel.hpp:52-56): block sums added in order from 0.0. One block of
// kChainThreads. A short list is one chain a sum (8 cycles a value); a long one goes through ordered_sum, which
// gives the same bits: 31,600 block sums (N = 864,000) took 265 us as a chain.
constexpr int kChainThreads = 2 * kOrderedThreads;
constexpr int kChainSerial = 512;  // about where both take 4,500 cycles
union ChainSmem {
    OrderedSmem<2, kChainValues> ordered;
    double2 v[kChainSerial];
    __device__ ChainSmem() {}
};
__device__ __forceinline__ void sum_blocks(const double2* __restrict__ block_sums, int nblocks,
                                           double* __restrict__ out) {
    __shared__ ChainSmem sm;
    if (nblocks <= kChainSerial) {
        for (int k = threadIdx.x; k < nblocks; k += blockDim.x) sm.v[k] = block_sums[k];
        __syncthreads();
        if (threadIdx.x < 2)
            out[threadIdx.x] = add_in_order(reinterpret_cast<const double*>(sm.v) + threadIdx.x, 2, nblocks, 0.0);
        return;
    }
    if (threadIdx.x < 2) sm.ordered.run[threadIdx.x] = 0.0;
    ordered_sum(sm.ordered, nblocks, [&](long long k, double* v) {
        const double2 x = block_sums[k];
        v[0] = x.x;
        v[1] = x.y;
    });
    if (threadIdx.x < 2) out[threadIdx.x] = sm.ordered.run[threadIdx.x];
}

// record (a run's records; may be null) gets the kinetic energy too
__global__ void __launch_bounds__(kChainThreads) k_sum_blocks(const double2* __restrict__ block_sums, int nblocks,
                                                              double* __restrict__ out, double* __restrict__ record) {
    sum_blocks(block_sums, nblocks, out);
    if (record && threadIdx.x == 0) *record = out[0];
}

// sum_blocks over the 1024-pair blocks of k_pair_block_sums, as many as it reported; record (may be null) gets both sums
__global__ void __launch_bounds__(kChainThreads) k_sum_pair_blocks(const double2* __restrict__ block_sums,
                                                                   const int* __restrict__ nblocks,
                                                                   double* __restrict__ out, double* __restrict__ record) {
    sum_blocks(block_sums, *nblocks, out);
    if (record && threadIdx.x < 2) record[threadIdx.x] = out[threadIdx.x];
}

// ---- kinetic energy -----------------------------------------------------------------------------------

// 0.5 * m * (vx^2 + vy^2 + vz^2) over particles [1024 b, 1024 b + 1024) summed in order (src/System.cpp:67-76), one block
// of kOrderedThreads each: every load of the block in flight at once, then ordered_sum. The thermostats wait for this sum.
// (A warp per block, loading 32 at a time with one lane adding: 12.6 us at any N up to 864,000, 7 of them loads.)
__global__ void __launch_bounds__(kOrderedThreads) k_kinetic_blocks(const double* __restrict__ vel,
                                                                    const double* __restrict__ mass, int n,
                                                                    double2* __restrict__ block_sums) {
    __shared__ OrderedSmem<1, kChunk / kOrderedThreads> sm;
    const int i0 = blockIdx.x * kChunk;
    const int m = n - i0 < kChunk ? n - i0 : kChunk;
    if (threadIdx.x == 0) sm.run[0] = 0.0;
    ordered_sum(sm, m, [&](long long k, double* v) {
        const int i = i0 + static_cast<int>(k);
        const double vx = vel[i], vy = vel[static_cast<size_t>(n) + i], vz = vel[2 * static_cast<size_t>(n) + i];
        v[0] = dmul(dmul(0.5, mass[i]), norm2(vx, vy, vz));
    });
    if (threadIdx.x == 0) block_sums[blockIdx.x] = make_double2(sm.run[0], 0.0);
}

// ---- integration --------------------------------------------------------------------------------------

// VelocityVerletIntegrator::kickAndDrift (src/Integrator.cpp:32-53): v += (dt/2) f / m, then
// r = wrap(r + dt v). Fused with NeighbourList::update's staleness test (src/NeighbourList.cpp:24-30) against
// the reference positions of the last build, which sets *stale when any |d|^2 > skin^2 / 4.
__global__ void k_kick_drift(double4* __restrict__ pos, double* __restrict__ vel, const double* __restrict__ force,
                             const double* __restrict__ mass, int n, double half_dt, double dt, Box box,
                             const double4* __restrict__ ref_pos, double max_disp2, int* __restrict__ stale) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double m = mass[i];
    double4 p = pos[i];
    double* pc[3] = {&p.x, &p.y, &p.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const size_t o = static_cast<size_t>(k) * n + i;
        const double v = dadd(vel[o], ddiv(dmul(half_dt, force[o]), m));
        vel[o] = v;
        *pc[k] = wrap(dadd(*pc[k], dmul(dt, v)), box);
    }
    pos[i] = p;
    if (ref_pos) {
        const double4 r = ref_pos[i];
        const double dx = min_image(dsub(p.x, r.x), box);
        const double dy = min_image(dsub(p.y, r.y), box);
        const double dz = min_image(dsub(p.z, r.z), box);
        if (norm2(dx, dy, dz) > max_disp2) *stale = 1;
    }
}

// NeighbourList::update's test on its own (src/NeighbourList.cpp:24-30)
__global__ void k_skin_check(const double4* __restrict__ pos, int n, Box box, const double4* __restrict__ ref_pos,
                             double max_disp2, int* __restrict__ stale) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double4 p = pos[i], r = ref_pos[i];
    const double dx = min_image(dsub(p.x, r.x), box);
    const double dy = min_image(dsub(p.y, r.y), box);
    const double dz = min_image(dsub(p.z, r.z), box);
    if (norm2(dx, dy, dz) > max_disp2) *stale = 1;
}

// VelocityVerletIntegrator::kick (src/Integrator.cpp:55-71)
__global__ void k_kick(double* __restrict__ vel, const double* __restrict__ force, const double* __restrict__ mass,
                       int n, double half_dt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double m = mass[i];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const size_t o = static_cast<size_t>(k) * n + i;
        vel[o] = dadd(vel[o], ddiv(dmul(half_dt, force[o]), m));
    }
}

// ---- thermostats ----------------------------------------------------------------------------------------

// A thermostat's scale factor from the kinetic energy on the device, so no host round trip is needed: mode 1
// rescaleVelocities (src/Thermostat.cpp:17-30), 2 BussiThermostat::apply with the step's draws (src/Thermostat.cpp:36-58),
// 0 none. scale[0] = factor, scale[1] = 1 to apply or 0 to leave the velocities alone.
struct Thermostat {
    int mode;
    double dof;
    double temperature;
    double c;
    const double* r1;
    const double* chi2;
    double* scale;
};

// BussiThermostat::apply's velocity scale, equation A7 (src/Thermostat.cpp:40-57), for kinetic > 0
__device__ __forceinline__ double bussi_scale(double kinetic, double dof, double temperature, double c, double r1,
                                              double chi2) {
    const double target = dmul(dmul(0.5, dof), temperature);
    const double omc = dsub(1.0, c);
    const double t1 = dmul(omc, dsub(ddiv(dmul(target, dadd(chi2, dmul(r1, r1))), dof), kinetic));
    const double t2 = dmul(dmul(2.0, r1), __dsqrt_rn(dmul(dmul(dmul(ddiv(target, dof), kinetic), omc), c)));
    const double nk = dadd(dadd(kinetic, t1), t2);
    return __dsqrt_rn(ddiv(nk, kinetic));
}

__device__ __forceinline__ void thermostat_factor(const Thermostat& t, double kinetic) {
    double factor = 0.0;
    bool apply;
    if (t.mode == 1) {
        const double now = ddiv(dmul(2.0, kinetic), t.dof);  // System::temperature (src/System.cpp:79-82)
        apply = !(now <= 0.0);
        if (apply) factor = __dsqrt_rn(ddiv(t.temperature, now));
    } else {
        apply = !(kinetic <= 0.0);
        if (apply) factor = bussi_scale(kinetic, t.dof, t.temperature, t.c, *t.r1, *t.chi2);
    }
    if (apply) t.scale[0] = factor;
    t.scale[1] = apply ? 1.0 : 0.0;
}

__global__ void k_thermostat_factor(const double* __restrict__ ke, Thermostat t) { thermostat_factor(t, ke[0]); }

// k_kinetic_blocks, k_sum_blocks and what stands before and after them in one launch, for at most kChainSerial blocks:
// with `scale` the velocities are scaled first (k_scale_velocities), the last block to finish (counted in *done, which it
// leaves zero) adds the blocks' sums in order, and with a thermostat it makes its factor. A thermostat's step waits for
// all of it, and small systems spend that time in launches: N = 2,048 (B200) 3.2 + 3.4 us for the sum and the factor and
// 3.5 for the scaling, each after a launch of its own, around the 6.1 of k_kinetic_blocks.
__global__ void __launch_bounds__(kOrderedThreads)
    k_kinetic_sum(double* vel, const double* __restrict__ mass, int n, const double* __restrict__ scale,
                  double* __restrict__ block_sums, unsigned* __restrict__ done, double* __restrict__ out,
                  double* __restrict__ record, Thermostat thermostat) {
    __shared__ OrderedSmem<1, kChunk / kOrderedThreads> sm;
    __shared__ double s_sums[kChainSerial];
    __shared__ bool s_last;
    const int i0 = blockIdx.x * kChunk;
    const int m = n - i0 < kChunk ? n - i0 : kChunk;
    const bool scaled = scale && scale[1] != 0.0;
    const double factor = scaled ? scale[0] : 1.0;
    if (threadIdx.x == 0) sm.run[0] = 0.0;
    ordered_sum(sm, m, [&](long long k, double* v) {
        const int i = i0 + static_cast<int>(k);
        double c[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) c[q] = vel[q * static_cast<size_t>(n) + i];
        if (scaled) {
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                c[q] = dmul(c[q], factor);
                vel[q * static_cast<size_t>(n) + i] = c[q];
            }
        }
        v[0] = dmul(dmul(0.5, mass[i]), norm2(c[0], c[1], c[2]));
    });
    if (threadIdx.x == 0) {
        block_sums[blockIdx.x] = sm.run[0];
        __threadfence();
        s_last = gridDim.x == 1 || atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (unsigned k = threadIdx.x; k < gridDim.x; k += kOrderedThreads) s_sums[k] = __ldcg(block_sums + k);
    __syncthreads();
    if (threadIdx.x == 0) {
        const double kinetic = add_in_order(s_sums, 1, static_cast<int>(gridDim.x), 0.0);
        *out = kinetic;
        if (record) *record = kinetic;
        if (thermostat.mode) thermostat_factor(thermostat, kinetic);
        if (gridDim.x > 1) *done = 0u;
    }
}

__global__ void k_scale_velocities(double* __restrict__ vel, long long count, const double* __restrict__ scale) {
    if (scale[1] == 0.0) return;
    const double s = scale[0];
    for (long long t = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; t < count;
         t += static_cast<long long>(gridDim.x) * blockDim.x)
        vel[t] = dmul(vel[t], s);
}

// ---- g(r) -------------------------------------------------------------------------------------------------

// RadialDistribution::sample (src/RadialDistribution.cpp:11-30): every half-list pair with r^2 < r_max^2
// adds one to bin (size_t)(sqrt(r^2) / binWidth). Counts are integers, so atomics keep the result exact.
// A bin index of `bins` or more (possible only through rounding at r just under r_max) is dropped: the
// reference would write past its histogram there.
// kRdfLanes threads per particle, lane u taking the row's quads u, u + kRdfLanes, ...: four positions are on their way at
// once. One thread per particle, entry by entry, was a chain of dependent loads (B200, md_rdf_sample with its copies:
// N = 2,048: 56 us, now 22; 500,000: 166, now 147).
constexpr int kRdfLanes = 4;
__global__ void k_rdf_sample(const double4* __restrict__ pos, int n, Box box, const uint32_t* __restrict__ rows,
                             int cap, const int2* __restrict__ counts, double rmax2, double bin_width, int bins,
                             unsigned long long* __restrict__ hist) {
    extern __shared__ unsigned int sm_hist[];
    for (int b = threadIdx.x; b < bins; b += blockDim.x) sm_hist[b] = 0;
    __syncthreads();
    const int u = threadIdx.x % kRdfLanes, i = static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) / kRdfLanes);
    if (i < n) {
        const double4 pi = load_pos(pos + i);
        const int own = counts[i].x;
        for (int s = 4 * u; s < own; s += 4 * kRdfLanes) {
            const uint4 q = row_quad(rows, i, s >> 2, cap);
            const uint32_t e[4] = {q.x, q.y, q.z, q.w};
            double4 pj[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) pj[k] = load_pos(pos + (s + k < own ? e[k] & kIndexMask : static_cast<uint32_t>(i)));
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const double dx = min_image(dsub(pi.x, pj[k].x), box);
                const double dy = min_image(dsub(pi.y, pj[k].y), box);
                const double dz = min_image(dsub(pi.z, pj[k].z), box);
                const double r2 = norm2(dx, dy, dz);
                if (s + k < own && r2 < rmax2) {
                    const unsigned long long b = __double2ull_rz(ddiv(__dsqrt_rn(r2), bin_width));
                    if (b < static_cast<unsigned long long>(bins)) atomicAdd(&sm_hist[b], 1u);
                }
            }
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < bins; b += blockDim.x)
        if (sm_hist[b]) atomicAdd(&hist[b], static_cast<unsigned long long>(sm_hist[b]));
}

// ---- O(N^2) forces ----------------------------------------------------------------------------------------

// computeForces(System&) (src/Forcefield.cpp:39-78). Particle p receives, in the reference's loop order,
// -F(i, p) for i = 0 .. p-1 and then +F(p, j) for j = p+1 .. n-1; pairs at or beyond the cutoff are skipped. The
// potential and virial are one sequential sum over the pairs (i, j > i) inside the cutoff in loop order, from 0.0.
//
// One warp per particle: the lanes test 32 partners at a time and the few inside the cutoff are then added one after
// another in partner order, from shuffled terms, by every lane alike. Both signs take the one form +F dx(p, i), which
// is the same double (min_image is odd, IEEE subtraction antisymmetric). Bound by the FP64 pipe: about 40 double
// operations a pair tested (three minimum images; their rounding is skipped within a quarter box).
// own[p] = pairs (p, j > p) inside the cutoff. With `rec` (kRecords), the (E, W) of those pairs are written instead,
// in order, at rec[off[p] - off0] for the particles [p0, p1); ordered_sum adds them with the serial sum's bits.
template <bool kRecords>
__global__ void __launch_bounds__(128) k_all_pairs(const double4* __restrict__ pos, int n, Box box, LJ lj, int p0,
                                                   int p1, double* __restrict__ force, int* __restrict__ own,
                                                   const long long* __restrict__ off, long long off0,
                                                   double2* __restrict__ rec) {
    const int p = p0 + static_cast<int>((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (p >= p1) return;
    const double4 pp = pos[p];
    double fx = 0.0, fy = 0.0, fz = 0.0;
    int hits = 0;
    double2* out = kRecords ? rec + (off[p] - off0) : nullptr;
    for (int i0 = kRecords ? (p + 1) & ~31 : 0; i0 < n; i0 += 32) {
        const int i = i0 + lane;
        bool in = i < n && (kRecords ? i > p : i != p);
        double dx = 0.0, dy = 0.0, dz = 0.0, r2 = 0.0;
        if (in) {
            const double4 q = pos[i];
            dx = min_image(dsub(pp.x, q.x), box);
            dy = min_image(dsub(pp.y, q.y), box);
            dz = min_image(dsub(pp.z, q.z), box);
            r2 = norm2(dx, dy, dz);
            in = kRecords ? r2 < lj.rc2 : !(r2 >= lj.rc2);  // (a NaN separation enters the forces, not the sums)
        }
        unsigned mask = __ballot_sync(0xffffffffu, in);
        if (!mask) continue;
        double fr = 0.0, e = 0.0;
        if (in) pair_terms(r2, lj, fr, e);
        if (kRecords) {
            if (in) out[hits + __popc(mask & ((1u << lane) - 1u))] = make_double2(e, dmul(fr, r2));
            hits += __popc(mask);
        } else {
            hits += __popc(__ballot_sync(0xffffffffu, in && i > p && r2 < lj.rc2));
            dx = dmul(fr, dx);
            dy = dmul(fr, dy);
            dz = dmul(fr, dz);
            while (mask) {
                const int t = __ffs(mask) - 1;
                mask &= mask - 1;
                fx = dadd(fx, __shfl_sync(0xffffffffu, dx, t));
                fy = dadd(fy, __shfl_sync(0xffffffffu, dy, t));
                fz = dadd(fz, __shfl_sync(0xffffffffu, dz, t));
            }
        }
    }
    if (!kRecords && lane == 0) {
        force[p] = fx;
        force[static_cast<size_t>(n) + p] = fy;
        force[2 * static_cast<size_t>(n) + p] = fz;
        own[p] = hits;
    }
}

// The same for n <= 32 in one launch: warp p takes particle p, one thread adds the pairs' (E, W) in order; out = potential,
// virial, inside pairs. (Through k_all_pairs, the offsets' scan and k_sum_pairs, with the pair count read back in between, a
// call on 2 particles takes 62 us, with this kernel 22.)
constexpr int kFewParticles = 32;
__global__ void __launch_bounds__(32 * kFewParticles) k_all_pairs_few(const double4* __restrict__ pos, int n, Box box, LJ lj,
                                                                      double* __restrict__ force, double* __restrict__ out) {
    __shared__ double2 s_rec[kFewParticles][kFewParticles];
    __shared__ int s_own[kFewParticles];
    const int p = threadIdx.x >> 5, i = threadIdx.x & 31;
    if (p < n) {
        bool in = i < n && i != p;
        double dx = 0.0, dy = 0.0, dz = 0.0, r2 = 0.0, fr = 0.0, e = 0.0;
        if (in) {
            const double4 pp = pos[p], q = pos[i];
            dx = min_image(dsub(pp.x, q.x), box);
            dy = min_image(dsub(pp.y, q.y), box);
            dz = min_image(dsub(pp.z, q.z), box);
            r2 = norm2(dx, dy, dz);
            in = !(r2 >= lj.rc2);
        }
        if (in) pair_terms(r2, lj, fr, e);
        const bool mine = in && i > p && r2 < lj.rc2;
        const unsigned own = __ballot_sync(0xffffffffu, mine);
        if (mine) s_rec[p][__popc(own & ((1u << i) - 1u))] = make_double2(e, dmul(fr, r2));
        if (i == 0) s_own[p] = __popc(own);
        dx = dmul(fr, dx);
        dy = dmul(fr, dy);
        dz = dmul(fr, dz);
        double fx = 0.0, fy = 0.0, fz = 0.0;
        for (unsigned mask = __ballot_sync(0xffffffffu, in); mask; mask &= mask - 1) {
            const int t = __ffs(mask) - 1;
            fx = dadd(fx, __shfl_sync(0xffffffffu, dx, t));
            fy = dadd(fy, __shfl_sync(0xffffffffu, dy, t));
            fz = dadd(fz, __shfl_sync(0xffffffffu, dz, t));
        }
        if (i < 3) force[static_cast<size_t>(i) * n + p] = i == 0 ? fx : i == 1 ? fy : fz;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double pe = 0.0, w = 0.0;
        int inside = 0;
        for (int k = 0; k < n; ++k) {
            for (int t = 0; t < s_own[k]; ++t) {
                pe = dadd(pe, s_rec[k][t].x);
                w = dadd(w, s_rec[k][t].y);
            }
            inside += s_own[k];
        }
        out[0] = pe;
        out[1] = w;
        out[2] = static_cast<double>(inside);
    }
}

// The all-pairs records added to the running (potential, virial) in out[0..1]; out[2] = inside pairs so far. One block.
__global__ void __launch_bounds__(2 * kOrderedThreads) k_sum_pairs(const double2* __restrict__ rec, long long m,
                                                                   double* __restrict__ out, double inside) {
    __shared__ OrderedSmem<2, kChainValues> sm;
    if (threadIdx.x < 2) sm.run[threadIdx.x] = out[threadIdx.x];
    ordered_sum(sm, m, [&](long long k, double* v) {
        const double2 r = rec[k];
        v[0] = r.x;
        v[1] = r.y;
    });
    if (threadIdx.x < 2) out[threadIdx.x] = sm.run[threadIdx.x];
    if (threadIdx.x == 0) out[2] = inside;
}

}  // namespace md
