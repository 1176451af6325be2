// Adjoint of the FP64 velocity-Verlet trajectory (md_adjoint_* in include/md_b200.h): gradients of the
// trajectory averages of the potential energy and the virial pressure with respect to epsilon, sigma and the
// initial positions and velocities.
//
// The trajectory is the reference's NVE step (src/Integrator.cpp:18-71) with the truncated and shifted pair
// terms (src/Forcefield.cpp:25-36), minimum image and wrap (include/System.hpp:86-112) and blocked sums
// (include/Parallel.hpp:32-57), with two choices that make forward runs, recomputations and the CPU adjoint give
// the same bits: particles are never reordered (the list is built from a stable cell sort of indices), and each
// particle's row holds all its partners within r_c + skin in the reference's candidate order, so every
// per-particle sum runs over that whole row in that order. Every double operation is an explicit
// round-to-nearest intrinsic (no contraction).
//
// For a pair with separation d, r2 = |d|^2, s6 = (sigma^2 / r2)^3, s12 = s6^2:
//   F/r  = fr  = 24 eps (2 s12 - s6) / r2          d fr / d r2  = frp = 24 eps (4 s6 - 14 s12) / r2^2
//   e    = 4 eps (s12 - s6) - shift                 d fr / d sig = frs = 24 eps (24 s12 - 6 s6) / (r2 sig)
//   d e / d sig = es = 4 eps (12 s12 - 6 s6) / sig - d shift / d sig
// The force Jacobian block of a pair is B = fr I + 2 frp d d^T, so (H w)_i = sum_j B_ij (w_i - w_j).
#pragma once

#include "md_common.cuh"
#include "md_fp64.cuh"

namespace md {

struct AdjConsts {
    Box box;
    double sig2, eps24, eps4, shift, rc2;
    double eps, inv_sigma, shift_sigma;
};

struct AdjPair {
    double dx, dy, dz, r2, fr, e, frp, frs, es;
};

// The pair (i, j) at positions a, b; false at or beyond the cutoff. kDeriv adds frp, frs, es.
template <bool kDeriv>
__device__ __forceinline__ bool adj_pair(const double4& a, const double4& b, const AdjConsts& c, AdjPair& q) {
    q.dx = min_image(dsub(a.x, b.x), c.box);
    q.dy = min_image(dsub(a.y, b.y), c.box);
    q.dz = min_image(dsub(a.z, b.z), c.box);
    q.r2 = norm2(q.dx, q.dy, q.dz);
    if (!(q.r2 < c.rc2)) return false;
    const double inv = ddiv(1.0, q.r2);
    const double s2 = dmul(c.sig2, inv);
    const double s6 = dmul(dmul(s2, s2), s2);
    const double s12 = dmul(s6, s6);
    q.fr = dmul(dmul(c.eps24, dsub(dmul(2.0, s12), s6)), inv);
    q.e = dsub(dmul(c.eps4, dsub(s12, s6)), c.shift);
    if (kDeriv) {
        const double inv2 = dmul(inv, inv);
        q.frp = dmul(dmul(c.eps24, dsub(dmul(4.0, s6), dmul(14.0, s12))), inv2);
        q.frs = dmul(dmul(c.eps24, dsub(dmul(24.0, s12), dmul(6.0, s6))), dmul(inv, c.inv_sigma));
        q.es = dsub(dmul(dmul(c.eps4, dsub(dmul(12.0, s12), dmul(6.0, s6))), c.inv_sigma), c.shift_sigma);
    }
    return true;
}

// Full rows (every partner within r_c + skin, the particle itself excluded) in the reference's candidate
// order from a stable cell sort (order[start[c] .. start[c + 1]) lists cell c's particles by index); under 3
// cells per side, every particle by index. counts[i] is kept within cap; max_count gets the true longest row.
// A warp per particle tests 32 candidates at once and places the accepted by the ballot. (A thread per particle, one
// candidate at a time, took 311 us at N = 32,000.)
__global__ void __launch_bounds__(128) k_adj_rows(const double4* __restrict__ pos, int n, Box box, double rl2, int ncps,
                                                  const int* __restrict__ cell_of, const int* __restrict__ start,
                                                  const uint32_t* __restrict__ order, int cap, uint32_t* __restrict__ rows,
                                                  int* __restrict__ counts, int* __restrict__ max_count) {
    const int i = static_cast<int>((blockIdx.x * 128 + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (i >= n) return;
    const unsigned below = (1u << lane) - 1u;
    const double4 pi = load_pos(pos + i);
    int cnt = 0;
    auto take = [&](int j) {  // j < 0: no candidate in this lane
        const double4 pj = load_pos(pos + (j < 0 ? i : j));
        const double dx = min_image(dsub(pi.x, pj.x), box);
        const double dy = min_image(dsub(pi.y, pj.y), box);
        const double dz = min_image(dsub(pi.z, pj.z), box);
        const bool in = j >= 0 && j != i && norm2(dx, dy, dz) < rl2;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        const int at = cnt + __popc(m & below);
        if (in && at < cap) rows[row_index(i, at, cap)] = static_cast<uint32_t>(j);
        cnt += __popc(m);
    };
    if (ncps < 3) {
        for (int j0 = 0; j0 < n; j0 += 32) take(j0 + lane < n ? j0 + lane : -1);
    } else {
        // lane c holds the range of the cell of code c
        const int c = cell_of[i];
        int s = 0, e = 0;
        if (lane < 27) {
            int x = c / (ncps * ncps) + lane / 9 - 1, y = (c / ncps) % ncps + (lane / 3) % 3 - 1, z = c % ncps + lane % 3 - 1;
            x += x < 0 ? ncps : x >= ncps ? -ncps : 0;
            y += y < 0 ? ncps : y >= ncps ? -ncps : 0;
            z += z < 0 ? ncps : z >= ncps ? -ncps : 0;
            const int nb = (x * ncps + y) * ncps + z;
            s = start[nb];
            e = start[nb + 1];
        }
        auto fetch = [&](int code) {  // the first 32 particles of a cell
            const int a = __shfl_sync(0xffffffffu, s, code), b = __shfl_sync(0xffffffffu, e, code);
            return a + lane < b ? static_cast<int>(order[a + lane]) : -1;
        };
        int next = fetch(0);
        for (int code = 0; code < 27; ++code) {
            const int j = next;
            if (code < 26) next = fetch(code + 1);
            take(j);
            const int a = __shfl_sync(0xffffffffu, s, code), b = __shfl_sync(0xffffffffu, e, code);
            for (int t = a + 32; t < b; t += 32) take(t + lane < b ? static_cast<int>(order[t + lane]) : -1);
        }
    }
    if (lane == 0) {
        counts[i] = cnt < cap ? cnt : cap;
        if (cnt > *static_cast<volatile int*>(max_count)) atomicMax(max_count, cnt);
    }
}

// A particle's ordered sums by kLanes threads: the lanes evaluate kLanes row entries at once (term(j, t) fills the kSums
// terms of partner j, zeros outside the cutoff, which leave a sum as it is) and lane v < kSums adds sum v's terms in row
// order; returned in the lanes below kSums (kSums <= kLanes). A whole warp calls, with m = 0 where there is no particle;
// stage holds kStage doubles per warp. (A thread per particle took 53 us for the forces and 74 us for a backward pass at
// N = 32,000, 250 blocks of chained gathers.)
template <int kLanes, int kSums>
struct AdjLanes {
    static_assert(kSums <= kLanes, "a lane per sum");
    static constexpr int kGroups = 32 / kLanes, kPad = kLanes + 1, kRow = kGroups * kPad + 1;
    static constexpr int kStage = kSums * kRow;
    template <typename Term>
    static __device__ __forceinline__ double sums(const uint32_t* __restrict__ rows, int i, int m, int cap, double* stage,
                                                  Term term) {
        const int lane = threadIdx.x & 31, u = lane % kLanes;
        double* mine = stage + (lane / kLanes) * kPad;
        int steps = (m + kLanes - 1) / kLanes;
#pragma unroll
        for (int o = kLanes; o < 32; o <<= 1) steps = max(steps, __shfl_xor_sync(0xffffffffu, steps, o));
        auto entry = [&](int s) { return s < m ? static_cast<int>(rows[row_index(i, s, cap)]) : -1; };
        int next = entry(u);
        double sum = 0.0;
        for (int q = 0; q < steps; ++q) {
            const int j = next;
            next = entry((q + 1) * kLanes + u);
            double t[kSums];
#pragma unroll
            for (int v = 0; v < kSums; ++v) t[v] = 0.0;
            if (j >= 0) term(j, t);
#pragma unroll
            for (int v = 0; v < kSums; ++v) mine[v * kRow + u] = t[v];
            __syncwarp();
            if (u < kSums) {
                double x[kLanes];
#pragma unroll
                for (int k = 0; k < kLanes; ++k) x[k] = mine[u * kRow + k];
#pragma unroll
                for (int k = 0; k < kLanes; ++k) sum = dadd(sum, x[k]);
            }
            __syncwarp();
        }
        return sum;
    }
};

// Forces (3 x n, component-major) and the row sums of pair energy and virial
constexpr int kAdjForceLanes = 8;
__global__ void __launch_bounds__(128) k_adj_forces(const double4* __restrict__ pos, int n, AdjConsts c,
                                                    const uint32_t* __restrict__ rows, int cap,
                                                    const int* __restrict__ counts, double* __restrict__ force,
                                                    double* __restrict__ u, double* __restrict__ w) {
    using Lanes = AdjLanes<kAdjForceLanes, 5>;
    __shared__ double stage[4][Lanes::kStage];
    const int i = static_cast<int>((blockIdx.x * 128 + threadIdx.x) / kAdjForceLanes), l = threadIdx.x % kAdjForceLanes;
    const bool real = i < n;
    const double4 pi = pos[real ? i : 0];
    const double sum = Lanes::sums(rows, i, real ? counts[i] : 0, cap, stage[threadIdx.x >> 5], [&](int j, double* t) {
        AdjPair q;
        if (!adj_pair<false>(pi, load_pos(pos + j), c, q)) return;
        t[0] = dmul(q.fr, q.dx);
        t[1] = dmul(q.fr, q.dy);
        t[2] = dmul(q.fr, q.dz);
        t[3] = q.e;
        t[4] = dmul(q.fr, q.r2);
    });
    if (!real) return;
    if (l < 3) force[static_cast<size_t>(l) * n + i] = sum;
    else if (l == 3) u[i] = sum;
    else if (l == 4) w[i] = sum;
}

// Blocked sums in order of pairs of per-particle arrays (k_kinetic_blocks' blocks): pair p = blockIdx.y of `in` into
// block_sums[p * gridDim.x + block]
struct AdjArrays {
    const double* a[3];
    const double* b[3];
};
__global__ void __launch_bounds__(kChainThreads) k_adj_blocks2(AdjArrays in, int n, double2* __restrict__ block_sums) {
    __shared__ OrderedSmem<2, kChunk / kOrderedThreads> sm;
    const double *x = in.a[blockIdx.y], *y = in.b[blockIdx.y];
    const int i0 = blockIdx.x * kChunk, m = n - i0 < kChunk ? n - i0 : kChunk;
    if (threadIdx.x < 2) sm.run[threadIdx.x] = 0.0;
    ordered_sum(sm, m, [&](long long k, double* v) {
        v[0] = x[i0 + k];
        v[1] = y[i0 + k];
    });
    if (threadIdx.x == 0) block_sums[blockIdx.y * gridDim.x + blockIdx.x] = make_double2(sm.run[0], sm.run[1]);
}

// After step k of the forward pass, from the block sums of (u, w) and of the kinetic energy: U_k = 0.5 sum u,
// W_k = 0.5 sum w, KE_k, and the running sums of U and P = (2 KE + W) / 3V in run[0], run[1]. One block; uw and ke hold
// the outer sums.
__global__ void __launch_bounds__(kChainThreads) k_adj_record(const double2* __restrict__ uw_blocks,
                                                              const double2* __restrict__ ke_blocks, int nblocks,
                                                              double* __restrict__ uw, double* __restrict__ ke,
                                                              double volume, int k, double* __restrict__ U,
                                                              double* __restrict__ W, double* __restrict__ KE,
                                                              double* __restrict__ run) {
    sum_blocks(uw_blocks, nblocks, uw);
    __syncthreads();
    sum_blocks(ke_blocks, nblocks, ke);
    __syncthreads();
    if (threadIdx.x != 0) return;
    const double u = dmul(0.5, uw[0]), w = dmul(0.5, uw[1]), kin = ke[0];
    U[k] = u;
    W[k] = w;
    KE[k] = kin;
    run[0] = dadd(run[0], u);
    run[1] = dadd(run[1], ddiv(dadd(dmul(2.0, kin), w), dmul(3.0, volume)));
}

// The backward of a half kick's velocities and the weights of its pass, wv = (half_dt av) / m (a particle's three in
// one 32-byte record, gathered whole by the pass). Before the second half kick (vel set): av += (aK m) v, the objective's
// kinetic-energy term at the state; before the first (ar set): av += dt ar, the drift's backward.
__global__ void k_adj_weights(double* __restrict__ av, const double* __restrict__ vel, const double* __restrict__ ar,
                              const double* __restrict__ mass, int n, double aK, double dt, double half_dt,
                              double4* __restrict__ wv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double m = mass[i];
    double w[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const size_t o = static_cast<size_t>(k) * n + i;
        double v = av[o];
        if (vel) v = dadd(v, dmul(dmul(aK, m), vel[o]));
        if (ar) v = dadd(v, dmul(dt, ar[o]));
        av[o] = v;
        w[k] = ddiv(dmul(half_dt, v), m);
    }
    wv[i] = make_double4(w[0], w[1], w[2], 0.0);
}

// One backward pass at positions pos with weights wv: ar_i += -aU F_i + aW dW/dr_i + (H w)_i, and per particle
// the parameter-gradient terms: pe = w_i . F_i, ps = w_i . dF_i/dsig, us = sum es, ws = sum frs r2,
// ue = sum e, we = sum fr r2 (the last four for the objective's own parameter derivatives). Without the objective
// (aU = aW = 0) its sums are left out: their terms would add zeros.
template <bool kObjective>
__global__ void __launch_bounds__(128) k_adj_pass(const double4* __restrict__ pos, int n, AdjConsts c,
                                                  const uint32_t* __restrict__ rows, int cap,
                                                  const int* __restrict__ counts, const double4* __restrict__ wv,
                                                  double aU, double aW, double* __restrict__ ar, double* __restrict__ pe,
                                                  double* __restrict__ ps, double* __restrict__ us,
                                                  double* __restrict__ ws, double* __restrict__ ue,
                                                  double* __restrict__ we) {
    constexpr int kLanes = kObjective ? 16 : 8, kSums = kObjective ? 14 : 7;
    using Lanes = AdjLanes<kLanes, kSums>;
    __shared__ double stage[4][Lanes::kStage];
    const int i = static_cast<int>((blockIdx.x * 128 + threadIdx.x) / kLanes), l = threadIdx.x % kLanes;
    const bool real = i < n;
    const int at = real ? i : 0;
    const size_t N = static_cast<size_t>(n);
    const double4 pi = pos[at];
    const double4 wi = wv[at];
    const double wix = wi.x, wiy = wi.y, wiz = wi.z;
    const double sum = Lanes::sums(rows, i, real ? counts[i] : 0, cap, stage[threadIdx.x >> 5], [&](int j, double* t) {
        AdjPair q;
        const double4 wj = load_pos(wv + j);
        if (!adj_pair<true>(pi, load_pos(pos + j), c, q)) return;
        t[0] = dmul(q.fr, q.dx);  // F
        t[1] = dmul(q.fr, q.dy);
        t[2] = dmul(q.fr, q.dz);
        const double dwx = dsub(wix, wj.x), dwy = dsub(wiy, wj.y), dwz = dsub(wiz, wj.z);
        const double h = dmul(dmul(2.0, q.frp), norm2p(q.dx, dwx, q.dy, dwy, q.dz, dwz));
        t[3] = dadd(dmul(q.fr, dwx), dmul(h, q.dx));  // H w
        t[4] = dadd(dmul(q.fr, dwy), dmul(h, q.dy));
        t[5] = dadd(dmul(q.fr, dwz), dmul(h, q.dz));
        t[6] = dmul(q.frs, norm2p(q.dx, wix, q.dy, wiy, q.dz, wiz));
        if constexpr (kObjective) {
            const double g = dmul(2.0, dadd(q.fr, dmul(q.r2, q.frp)));
            t[7] = dmul(g, q.dx);  // dW/dr
            t[8] = dmul(g, q.dy);
            t[9] = dmul(g, q.dz);
            t[10] = q.es;
            t[11] = dmul(q.frs, q.r2);
            t[12] = q.e;
            t[13] = dmul(q.fr, q.r2);
        }
    });
    // component k's lane gathers F_k, H_k and G_k
    const double h = __shfl_down_sync(0xffffffffu, sum, 3), g = kObjective ? __shfl_down_sync(0xffffffffu, sum, 7) : 0.0;
    const double fy = __shfl_down_sync(0xffffffffu, sum, 1), fz = __shfl_down_sync(0xffffffffu, sum, 2);
    if (!real) return;
    if (l < 3) {
        const size_t o = l * N + i;
        if (kObjective) ar[o] = dadd(dadd(dadd(ar[o], dmul(-aU, sum)), dmul(aW, g)), h);
        else ar[o] = dadd(ar[o], h);
    }
    if (l == 0) pe[i] = norm2p(wix, sum, wiy, fy, wiz, fz);
    if (l == 6) ps[i] = sum;
    if (kObjective && l >= 10 && l < 14) (l == 10 ? us : l == 11 ? ws : l == 12 ? ue : we)[i] = sum;
}

// The pass's parameter gradients from the outer sums of k_adj_blocks2's pairs ((pe, ps), and with the objective (us, ws)
// and (ue, we)), a block for each pair added in turn by one block: theta[0] += sum pe / eps (+ (aU U + aW W) / eps),
// theta[1] += sum ps (+ aU dU/dsig + aW dW/dsig)
__global__ void __launch_bounds__(kChainThreads) k_adj_theta(const double2* __restrict__ block_sums, int nblocks, double eps,
                                                             double aU, double aW, bool objective,
                                                             double* __restrict__ sums, double* __restrict__ theta) {
    for (int p = 0; p < (objective ? 3 : 1); ++p) {
        sum_blocks(block_sums + static_cast<size_t>(p) * nblocks, nblocks, sums + 2 * p);
        __syncthreads();
    }
    if (threadIdx.x != 0) return;
    double geps = ddiv(sums[0], eps);
    double gsig = sums[1];
    if (objective) {
        const double Uk = dmul(0.5, sums[4]), Wk = dmul(0.5, sums[5]);
        geps = dadd(geps, ddiv(dadd(dmul(aU, Uk), dmul(aW, Wk)), eps));
        gsig = dadd(dadd(gsig, dmul(aU, dmul(0.5, sums[2]))), dmul(aW, dmul(0.5, sums[3])));
    }
    theta[0] = dadd(theta[0], geps);
    theta[1] = dadd(theta[1], gsig);
}

}  // namespace md
