// Sums of doubles added one after another, computed by a thread block with the serial sum's bits.
//
// The reference's energies are serial sums (include/Parallel.hpp:43-56, src/Forcefield.cpp:60-70): each value is
// added to the running sum and rounded before the next one, so no other order of addition gives the same double.
// What makes them parallel all the same: while the running sum s stays inside one binade, 2^e <= |s| < 2^(e+1), it is
// a whole multiple of u = 2^(e-52), and adding x changes it by x rounded to a multiple of u, whatever s is, unless x
// lies exactly halfway between two multiples (then the parity of s / u decides). That rounded change is
// d = (B + x) - B for any B of the binade, and sums of such d are exact, so a stretch of the array that stays in
// one binade and holds no halfway value is a sum of whole numbers, in any order.
//
// One tile of 256 C values at a time, C consecutive values a thread:
//   1. a plain scan gives each thread the running sum at its first value to about 1e-15, hence its binade;
//   2. a thread whose stretch may leave the binade (with a margin for the scan's rounding), touches zero, holds a
//      halfway value or a value too large for the shortcut is marked; the others sum their d;
//   3. a scan of the d, restarted at every marked thread (so that each scan stays in one binade and is exact);
//   4. one thread walks the marked ones in order: the exact sum up to each, then its C values by plain additions;
//   5. every other thread now knows its exact first running sum and checks that its stretch did stay inside the
//      binade. If one did not, the tile is added again serially, so the result never rests on step 1.
// A serial sum crosses a binade about log2 of its length times, and halfway values become rare as s outgrows x, so a
// 1024-value block that starts at zero marks some 20 threads and later tiles few or none.
//
// What bounds it: latency (six barriers, two scans and the walk a tile), not bandwidth. Measured on the B200 for two
// sums side by side: 2,048 values each take 4,850 cycles (2.6 us) in the middle of a long sum, against 16 cycles a value
// for one thread adding both (8.3 ns, 17 us for 2,048); a first tile, which starts at zero and marks more threads, takes
// 7,000 to 14,000 cycles. So it is for long sums: the serial loop is as good for a single 1,024-value block.
#pragma once

#include "md_common.cuh"

namespace md {

constexpr int kOrderedThreads = 256;  // threads per stream of values
constexpr int kOrderedWarps = kOrderedThreads / 32;

// Shared memory of ordered_sum: kStreams independent sums side by side (a block of kStreams * 256 threads)
template <int kStreams, int C>
struct OrderedSmem {
    // value k of a tile at k + k / C: a thread's C values start an odd number of doubles apart (no bank conflicts)
    double x[kStreams][kOrderedThreads * C + kOrderedThreads];
    double before[kStreams][kOrderedThreads];  // exact sum since the previous marked thread, at each marked thread
    double after[kStreams][kOrderedThreads];   // running sum after each marked thread
    double scan[kStreams][kOrderedWarps], seg[kStreams][kOrderedWarps];
    unsigned marked[kStreams][kOrderedWarps];
    double run[kStreams];                      // the running sums
};

__device__ __forceinline__ unsigned sign_exponent(double x) { return static_cast<unsigned>(__double2hiint(x)) >> 20; }

// Adds values [0, m) to the running sums sm.run[0 .. kStreams), which the caller has set (any thread; a barrier
// follows here). load(k, out) writes the kStreams values of record k. Every thread of the block calls it, with the same
// m; on return (after a barrier) sm.run holds the results.
template <int kStreams, int C, typename Load>
__device__ __forceinline__ void ordered_sum(OrderedSmem<kStreams, C>& sm, long long m, Load load) {
    static_assert(C % kStreams == 0, "each thread stages C / kStreams records");
    constexpr int T = kOrderedThreads * C, kRecs = C / kStreams, kLogValues = 5;
    static_assert(C <= (1 << kLogValues), "C half units fit the check's allowance");
    const int stream = kStreams == 1 ? 0 : threadIdx.x / kOrderedThreads;
    const int t = threadIdx.x % kOrderedThreads, lane = t & 31, warp = t >> 5;
    double rec[kRecs][kStreams];
    auto fetch = [&](long long base) {
#pragma unroll
        for (int q = 0; q < kRecs; ++q) {
            const long long k = base + q * (kOrderedThreads * kStreams) + threadIdx.x;
#pragma unroll
            for (int v = 0; v < kStreams; ++v) rec[q][v] = 0.0;
            if (k < m) load(k, rec[q]);
        }
    };
    if (m > 0) fetch(0);
    for (long long base = 0; base < m; base += T) {
        __syncthreads();  // the previous tile's values and sums have been read
#pragma unroll
        for (int q = 0; q < kRecs; ++q) {
            const int k = q * (kOrderedThreads * kStreams) + threadIdx.x;
#pragma unroll
            for (int v = 0; v < kStreams; ++v) sm.x[v][k + k / C] = rec[q][v];
        }
        __syncthreads();
        if (base + T < m) fetch(base + T);
        const double s0 = sm.run[stream];
        const double* x = sm.x[stream] + t * (C + 1);
        double v[C], sum = 0.0, size = 0.0;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            v[c] = x[c];
            sum = dadd(sum, v[c]);
            size = dadd(size, fabs(v[c]));
        }
        const bool zero = size == 0.0;
        // 1. the approximate running sum at this thread's first value
        double inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc = dadd(inc, y);
        }
        if (lane == 31) sm.scan[stream][warp] = inc;
        __syncthreads();
        double p = s0, part[kOrderedWarps - 1];
#pragma unroll
        for (int w = 0; w + 1 < kOrderedWarps; ++w) part[w] = w < warp ? sm.scan[stream][w] : 0.0;
#pragma unroll
        for (int w = 0; w + 1 < kOrderedWarps; ++w) p = dadd(p, part[w]);
        p = dadd(p, dsub(inc, sum));
        // 2. the stretch stays within p -+ size, widened, which must keep one sign and exponent
        const double reach = __fma_rn(1e-11, fabs(p), dmul(1.0 + 1e-11, size));
        const unsigned key = sign_exponent(dsub(p, reach));
        const int e = static_cast<int>(key & 0x7ffu);
        bool ok = key == sign_exponent(dadd(p, reach)) && e > 64 && e < 2000;
        double d = 0.0;
        if (ok) {
            const double mid = __hiloint2double(static_cast<int>((key << 20) | 0x80000u), 0);  // 1.5 * 2^e, signed
            const double half_unit = __hiloint2double((e - 53) << 20, 0);
            ok = size < __hiloint2double((e - 2) << 20, 0);  // mid + v stays in the binade
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const double step = dsub(dadd(mid, v[c]), mid);
                ok = ok && fabs(dsub(v[c], step)) != half_unit;
                d = dadd(d, step);
            }
        }
        const bool mark = !ok && !zero;  // adding zeros changes no sum
        if (mark || zero) d = 0.0;
        const unsigned marks = __ballot_sync(0xffffffffu, mark);
        // 3. exact sums since the last marked thread: `ex` before this thread
        const unsigned upto = marks & (0xffffffffu >> (31 - lane));
        const int first = upto ? 31 - __clz(upto) : 0;
        double seg = d;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, seg, o);
            if (lane - o >= first) seg = dadd(seg, y);
        }
        double ex = __shfl_up_sync(0xffffffffu, seg, 1);
        if (lane == 0) ex = 0.0;
        if (lane == 31) sm.seg[stream][warp] = seg;
        if (lane == 0) sm.marked[stream][warp] = marks;
        __syncthreads();
        const unsigned below = marks & ((1u << lane) - 1u);
        int last = below ? warp * 32 + 31 - __clz(below) : -1;  // the marked thread before this one
        {
            double carry = 0.0;
            int prev = -1;
#pragma unroll
            for (int w = 0; w + 1 < kOrderedWarps; ++w) part[w] = sm.seg[stream][w];
#pragma unroll
            for (int w = 0; w + 1 < kOrderedWarps; ++w) {
                const unsigned mw = sm.marked[stream][w];
                if (w < warp) {
                    carry = mw ? part[w] : dadd(carry, part[w]);
                    if (mw) prev = w * 32 + 31 - __clz(mw);
                }
            }
            if (!below) {
                ex = dadd(carry, ex);
                last = prev;
            }
        }
        if (mark) sm.before[stream][t] = ex;
        __syncthreads();
        // 4. the walk over the marked threads
        if (t == 0) {
            double s = s0, tail = 0.0, seg_of[kOrderedWarps];
            unsigned marks_of[kOrderedWarps];
#pragma unroll
            for (int w = 0; w < kOrderedWarps; ++w) {
                seg_of[w] = sm.seg[stream][w];
                marks_of[w] = sm.marked[stream][w];
            }
#pragma unroll
            for (int w = 0; w < kOrderedWarps; ++w) {
                unsigned mw = marks_of[w];
                tail = mw ? seg_of[w] : dadd(tail, seg_of[w]);
                while (mw) {
                    const int f = w * 32 + __ffs(mw) - 1;
                    mw &= mw - 1;
                    const double* xf = sm.x[stream] + f * (C + 1);
                    s = dadd(s, sm.before[stream][f]);
#pragma unroll
                    for (int c = 0; c < C; ++c) s = dadd(s, xf[c]);
                    sm.after[stream][f] = s;
                }
            }
            sm.run[stream] = dadd(s, tail);
        }
        __syncthreads();
        // 5. the check, and the serial sum if it fails: the steps of a stretch add up to at most size + C half units
        // (checked with 32 units), and a partial sum of exactly 2^e may hide an exact sum just below it, where the
        // spacing halves
        bool bad = false;
        if (!mark && !zero) {
            const double start = dadd(last >= 0 ? sm.after[stream][last] : s0, ex);
            const double most = dadd(size, __hiloint2double((e - 52 + kLogValues) << 20, 0));
            const double bottom = __hiloint2double(e << 20, 0);
            auto inside = [&](double z) { return sign_exponent(z) == key && fabs(z) > bottom; };
            bad = !inside(start) || !inside(dsub(start, most)) || !inside(dadd(start, most));
        }
        if (__syncthreads_or(bad)) {
            if (t == 0) {
                double s = s0;
                const int valid = static_cast<int>(m - base < T ? m - base : T);
                for (int k = 0; k < valid; ++k) s = dadd(s, sm.x[stream][k + k / C]);
                sm.run[stream] = s;
            }
        }
    }
    __syncthreads();
}

}  // namespace md
