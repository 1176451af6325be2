// Verlet list build by cells (boxes of at least 3 cells per side): NeighbourList::build pass 1
// (src/NeighbourList.cpp:75-111), the rows of md_nlist.cuh.
//
// One home cell at a time. Its candidates, the particles of the 27 cells around it that are within r_l of the home cell's
// cube (three quarters of them), are laid out in shared memory in the home cell's frame, in the order in which a row
// lists them: the cells after the home cell (all their particles j > i) in the reference's candidate order, the home cell
// in its place among them, then the cells before it (all j < i) in increasing cell id, then the home cell again. Then, for
// kHomes home particles at a time:
//   - test: 32 candidates at once, a lane each; ballots give each home particle a mask of the accepted;
//   - rows: half a warp per home particle, a mask word per lane; in the words of the two copies of the home cell a mask
//     keeps the j > i and the j < i; a scan of the words' counts gives each lane its place in the row, where it writes the
//     entries of its word's bits, into shared memory; whole rows go out as 16-byte quads.
//
// The test: r^2 - r_l^2 = (|h|^2 - r_l^2) + |c|^2 - 2 h.c, three FMAs from sums kept per home h and candidate c, for two
// homes at a time in packed instructions. Exactness: a candidate is accepted when that is below -margin. With
// coordinates of at most 1.5 cell sides (c) and 0.5 (h) and sides under 4/3 r_l, all roundings together stay below
// 7e-6 r_l^2, and the margin is 1e-5 r_l^2 + 1e-4. Every lane keeps the smallest |r^2 - r_l^2| it has met; when it falls
// inside the margin (about one group of homes in fifty) the group is tested again with the reference's double test
// deciding those candidates. So the rows are the reference's, bit for bit. A cell that has a position outside the box among
// its candidates (list_frame_of marks them: such a particle lies outside its cell, and with 3 cells a side the frames may
// then name another image than the nearest), or more candidates than the shared memory holds, goes through build_row.
//
// What bounds it: instruction issue (71 % of the slots; 482 warp instructions a particle: a third in laying out the candidates,
// a seventh in the tests, the rest in the rows). A thread per particle walking its candidates one by one (k_nlist_build_tile)
// takes 630 and scattered 4-byte stores, and leaves small systems to a few long chains. Measured (B200, kernel alone, liquid,
// tiles / cells): N = 4,000,000: 2.59 / 2.28 ms; 864,000: 0.60 / 0.53; 2,048: 36 / 15 us.
#pragma once

#include "md_common.cuh"
#include "md_fp32.cuh"
#include "md_nlist.cuh"

namespace md {

struct CellBuild {
    ListGeom geom;  // for build_row
    float rl2;      // r_l^2
    float margin;   // |float r^2 - r_l^2| up to this: decided in double
    float prune;    // candidates farther than this from the home cube (squared) are left out
    int stage;      // candidates the shared memory holds (multiple of 32; 0: rows too long, every cell through build_row)
    int warp_stage; // sparse systems: candidates that a warp lays out by itself (multiple of 32); 0: blocks build every cell
    int group;      // cells that a warp looks at together then (at most 32)
};

constexpr int kCellItems = 28;  // 27 cells, the home cell twice
constexpr float kCellFar = 1.0e30f;  // |c|^2 of an empty candidate

__host__ __device__ inline int cell_row_pitch(int cap) { return cap + 4; }
inline size_t cell_build_smem(int stage, int cap, int warps, int homes) {
    return (sizeof(float4) + sizeof(uint32_t)) * stage +
           sizeof(uint32_t) * warps * homes * (static_cast<size_t>(cell_row_pitch(cap)) + stage / 32);
}

// Bits x and up of a 32-bit mask (PTX shifts give 0 from 32 on)
__device__ __forceinline__ uint32_t bits_from(int x) {
    uint32_t m;
    asm("shl.b32 %0, %1, %2;" : "=r"(m) : "r"(0xffffffffu), "r"(max(x, 0)));
    return m;
}

// The candidates of one home cell: item r (in row order) is particles [first, first + count) of the cell of `code`, shifted
// by (x, y, z) into the home cell's frame, candidates [off[r], off[r + 1])
struct CellItems {
    int4 cell[kCellItems];  // first, count, code
    float4 shift[kCellItems];
    int off[kCellItems + 1];
    int own_items;  // the items before this one are j > i
    int home;       // item of the home cell's first copy (the second is the last item)
    int odd;        // a position outside the box
};

// Fills t for home cell `cell` (one warp)
__device__ __forceinline__ void cell_items(const int* __restrict__ cell_start, int nc, int cell, float side, CellItems& t) {
    const int lane = threadIdx.x & 31;
    const int cx = cell / (nc * nc), cy = (cell / nc) % nc, cz = cell % nc;
    const int dx = lane / 9 - 1, dy = (lane / 3) % 3 - 1, dz = lane % 3 - 1;
    int id = -1, first = 0, count = 0;
    if (lane < 27) {
        int x = cx + dx, y = cy + dy, z = cz + dz;
        x += x < 0 ? nc : x >= nc ? -nc : 0;
        y += y < 0 ? nc : y >= nc ? -nc : 0;
        z += z < 0 ? nc : z >= nc ? -nc : 0;
        id = (x * nc + y) * nc + z;
        first = cell_start[id];
        count = cell_start[id + 1] - first;
    }
    const unsigned below = (1u << lane) - 1u;
    const unsigned after = __ballot_sync(0xffffffffu, id > cell);
    const unsigned before = __ballot_sync(0xffffffffu, id >= 0 && id < cell);
    // the home cell and the cells after it in candidate order, then the cells before it in increasing id
    int rank = __popc((after | (1u << 13)) & below);
    if (id < cell) rank = __popc(before & below);
    if (cx == 0 || cy == 0 || cz == 0 || cx == nc - 1 || cy == nc - 1 || cz == nc - 1) {  // cells wrap: ids out of order
        int r = 0;
        for (int k = 0; k < 27; ++k) {
            const int other = __shfl_sync(0xffffffffu, id, k);
            r += ((before >> k) & 1u) && other < id;
        }
        if (id < cell) rank = r;
    }
    if (id < cell) rank += __popc(after) + 1;
    if (lane < 27) {
        t.cell[rank] = make_int4(first, count, lane, 0);
        t.shift[rank] = make_float4(dx * side, dy * side, dz * side, 0.0f);
        if (lane == 13) {
            t.cell[27] = make_int4(first, count, 13, 0);
            t.shift[27] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    if (lane == 0) {
        t.odd = 0;
        t.own_items = __popc(after) + 1;
        t.home = __popc(after & ((1u << 13) - 1u));
    }
}

// A candidate: its position c in the home cell's frame, and |c|^2
__device__ __forceinline__ float4 cell_candidate(const float4& f, const float4& shift) {
    const float x = __fadd_rn(f.x, shift.x), y = __fadd_rn(f.y, shift.y), z = __fadd_rn(f.z, shift.z);
    return make_float4(x, y, z, __fmaf_rn(x, x, __fmaf_rn(y, y, __fmul_rn(z, z))));
}

// Is a candidate within reach of the home cube [-half, half]^3? Candidates are counted and then laid out by the same test, so
// its roundings are spelled out: a product that the compiler fused with the difference in one of the two places only would
// leave a slot that nothing writes.
__device__ __forceinline__ float cell_half(float side) { return __fmul_rn(0.501f, side); }
__device__ __forceinline__ bool cell_reachable(const float4& c, float half, float prune) {
    const float x = fmaxf(__fsub_rn(fabsf(c.x), half), 0.0f), y = fmaxf(__fsub_rn(fabsf(c.y), half), 0.0f),
                z = fmaxf(__fsub_rn(fabsf(c.z), half), 0.0f);
    return __fmaf_rn(x, x, __fmaf_rn(y, y, __fmul_rn(z, z))) <= prune;
}

// r^2 - r_l^2 of a candidate and two home particles: (-2 h, |h|^2 - r_l^2) in (hx, hy, hz, hk)
__device__ __forceinline__ float2 cell_gap(const float4& q, const float2& hx, const float2& hy, const float2& hz,
                                           const float2& hk) {
    return __ffma2_rn(make_float2(q.x, q.x), hx,
                      __ffma2_rn(make_float2(q.y, q.y), hy,
                                 __ffma2_rn(make_float2(q.z, q.z), hz, __fadd2_rn(make_float2(q.w, q.w), hk))));
}

// The masks of a group of home particles (home[k] their frames, i their first index, `left` of them real) with the
// reference's double test on the candidates inside the margin. Out of line: one group in fifty comes here.
template <int kHomes>
__device__ __noinline__ void cell_masks_exact(const float4* cand, const uint32_t* entries, int words, const float4* home,
                                              int left, int i, const double4* __restrict__ pos, const ListGeom geom,
                                              float rl2, float margin, uint32_t* masks) {
    const int lane = threadIdx.x & 31;
    for (int k = 0; k < kHomes && k < left; ++k) {
        const float4 f = home[k];
        const float2 hx = make_float2(-2.0f * f.x, 0.0f), hy = make_float2(-2.0f * f.y, 0.0f),
                     hz = make_float2(-2.0f * f.z, 0.0f), hk = make_float2(f.w - rl2, 0.0f);
        for (int w = 0; w < words; ++w) {
            const float gap = cell_gap(cand[32 * w + lane], hx, hy, hz, hk).x;
            bool take = gap < -margin;
            if (fabsf(gap) <= margin)
                take = within_list(pos[i + k], pos[entries[32 * w + lane] & kIndexMask], geom);
            const unsigned m = __ballot_sync(0xffffffffu, take);
            if (lane == 0) masks[w * kHomes + k] = m;
        }
    }
}

// Mask words (32 candidates each) that build_cell's rows are written from at a time, for cells of per_cell particles on
// average: 16 hold the candidates of a liquid's list of r_l = 2.8; where about that many take a second round nearly
// empty, 24 (4 homes a warp, kernel alone with the same code otherwise, 16 / 24: N = 500,000, density 0.85, r_l = 3.2, 20
// words: 438 / 406 us; N = 864,000, density 0.8442, r_l = 2.8, 15 words: 545 / 560).
inline int cell_round(double per_cell) {
    const double words = 0.8 * kCellItems * per_cell / 32.0;
    return words > 18.0 && words <= 24.0 ? 24 : 16;
}

// kHomes home particles for the test: (-2 h, |h|^2 - r_l^2) in pairs
template <int kHomes>
struct CellHomes {
    float2 x[kHomes / 2], y[kHomes / 2], z[kHomes / 2], k[kHomes / 2];
};
// home[k]: the candidate of the group's particle k < left
template <int kHomes>
__device__ __forceinline__ CellHomes<kHomes> cell_homes(const float4* home, int left, float rl2) {
    CellHomes<kHomes> hm;
#pragma unroll
    for (int k = 0; k < kHomes; ++k) {
        float4 f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float sq = kCellFar;
        if (k < left) {
            f = home[k];
            sq = f.w - rl2;
        }
        (k & 1 ? hm.x[k / 2].y : hm.x[k / 2].x) = -2.0f * f.x;
        (k & 1 ? hm.y[k / 2].y : hm.y[k / 2].x) = -2.0f * f.y;
        (k & 1 ? hm.z[k / 2].y : hm.z[k / 2].x) = -2.0f * f.z;
        (k & 1 ? hm.k[k / 2].y : hm.k[k / 2].x) = sq;
    }
    return hm;
}

// The masks of a group of homes over `words` words of candidates (one warp): masks[w * kHomes + k]. home: the group's
// candidates, i: its first particle, left: its real ones.
template <int kHomes>
__device__ __forceinline__ void cell_masks(const float4* cand, const uint32_t* entries, int words, const float4* home, int left,
                                           int i, const double4* __restrict__ pos, const CellBuild& bp, uint32_t* masks) {
    static_assert(kHomes == 2 || kHomes == 4, "masks are stored as 8 or 16 bytes");
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const CellHomes<kHomes> hm = cell_homes<kHomes>(home, left, bp.rl2);
    float nearest = kCellFar;
    for (int w = 0; w < words; ++w) {
        const float4 q = cand[32 * w + lane];
        unsigned m[kHomes];
#pragma unroll
        for (int p = 0; p < kHomes / 2; ++p) {
            const float2 gap = cell_gap(q, hm.x[p], hm.y[p], hm.z[p], hm.k[p]);
            nearest = fminf(nearest, fminf(fabsf(gap.x), fabsf(gap.y)));
            m[2 * p] = __ballot_sync(kAll, gap.x < -bp.margin);
            m[2 * p + 1] = __ballot_sync(kAll, gap.y < -bp.margin);
        }
        if (lane == 0) {
            if constexpr (kHomes == 4) reinterpret_cast<uint4*>(masks)[w] = make_uint4(m[0], m[1], m[2], m[3]);
            else reinterpret_cast<uint2*>(masks)[w] = make_uint2(m[0], m[1]);
        }
    }
    if (__any_sync(kAll, nearest <= bp.margin))
        cell_masks_exact<kHomes>(cand, entries, words, home, left, i, pos, bp.geom, bp.rl2, bp.margin, masks);
    __syncwarp();
}

// Where the home cell's two copies and the items before a row's j < i lie among a cell's candidates
struct CellOrder {
    int home0, home1, own_end;
};

// Adds the accepted candidates of `words` words to the rows of a group of homes (one warp): kLanes lanes per home particle,
// kWords adjacent mask words a lane, kRound words at a time. h: this lane's home particle in the cell (real: there is one),
// mine: its row in shared memory, len and own: its entries so far.
template <int kHomes, int kRound>
__device__ __forceinline__ void cell_append(const uint32_t* entries, const uint32_t* masks, int words, const CellOrder& order,
                                            int h, bool real, int cap, uint32_t* mine, int& len, int& own) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int kLanes = 32 / kHomes, kWords = kRound / kLanes;
    const int lane = threadIdx.x & 31, k = lane / kLanes, l = lane % kLanes;
    for (int w0 = 0; w0 < words; w0 += kRound) {
        uint32_t bits[kWords];
        int c = 0, c_own = 0;
#pragma unroll
        for (int u = 0; u < kWords; ++u) {
            const int w = w0 + l * kWords + u, v = 32 * w;
            bits[u] = real && w < words ? masks[w * kHomes + k] : 0u;
            // in the home cell's first copy j > i, in the second j < i
            bits[u] &= (~bits_from(order.home0 - v) | bits_from(order.home0 + h + 1 - v)) & ~bits_from(order.home1 + h - v);
            c += __popc(bits[u]);
            c_own += __popc(bits[u] & ~bits_from(order.own_end - v));
        }
        int inc = c | (c_own << 16);  // both counts in one scan (kRound words hold far fewer than 65,536)
#pragma unroll
        for (int o = 1; o < kLanes; o <<= 1) {
            const int y = __shfl_up_sync(kAll, inc, o, kLanes);
            inc += l >= o ? y : 0;
        }
        int at = len + (inc & 0xffff) - c;
        const int sums = __shfl_sync(kAll, inc, kLanes - 1, kLanes);
        len += sums & 0xffff;
        own += sums >> 16;
        const bool fits = __all_sync(kAll, len <= cap);
#pragma unroll
        for (int u = 0; u < kWords; ++u) {
            uint32_t left = __brev(bits[u]);  // the first candidate in the highest bit
            const uint32_t* in = entries + 32 * (w0 + l * kWords + u);
            if (fits) {
                uint32_t* out = mine + at;
                at += __popc(left);
                while (left) {
                    const int b = __clz(left);
                    left ^= 0x80000000u >> b;
                    *out++ = in[b];
                }
            } else {
                for (; left; ++at) {
                    const int b = __clz(left);
                    left ^= 0x80000000u >> b;
                    if (at < cap) mine[at] = in[b];
                }
            }
        }
    }
}

// Pads the rows of a group of homes and writes them and their counts out (one warp). row: the group's rows in shared memory;
// i: its first particle, the others as in cell_append. Returns this lane's padded length, within the capacity or not.
template <int kHomes>
__device__ __forceinline__ int cell_write(uint32_t* row, int i, bool real, int len, int own, const CellBuild& bp,
                                          uint32_t* __restrict__ rows, int2* __restrict__ counts) {
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int kLanes = 32 / kHomes;
    const int lane = threadIdx.x & 31, k = lane / kLanes, l = lane % kLanes, cap = bp.geom.cap, pitch = cell_row_pitch(cap);
    const int padded = real ? (len + 7) & ~7 : 0;
    if (real) {
        if (l < 8 && len + l < padded && len + l < cap) row[k * pitch + len + l] = bp.geom.sentinel;
        // a row past the capacity keeps counts within it, so every reader stays in bounds until the host has seen
        // max_count, which reports the full length
        const int own_c = min(own, cap);
        if (l == 0) counts[i + k] = make_int2(own_c, min(len, cap) - own_c);
    }
    const int my_quads = __shfl_sync(kAll, min(padded, cap) >> 2, (lane % kHomes) * kLanes);
    __syncwarp();
    // quad q of home particle o by lane (q, o): neighbouring lanes write neighbouring particles' quads
    const int o = lane % kHomes, io = i + o;
    uint4* out = reinterpret_cast<uint4*>(rows) + static_cast<size_t>(io >> 5) * (cap >> 2) * 32 + (io & 31);
    for (int q = lane / kHomes; q < my_quads; q += kLanes)
        out[32 * q] = *reinterpret_cast<const uint4*>(row + o * pitch + 4 * q);
    __syncwarp();
    return padded;
}

__device__ __forceinline__ void report_longest(int longest, int* max_count) {
    longest = __reduce_max_sync(0xffffffffu, longest);
    if ((threadIdx.x & 31) == 0 && longest > *static_cast<volatile int*>(max_count)) atomicMax(max_count, longest);
}

// The rows of one home cell's particles, by the kWarps warps of a block; cell_start is the system's (values are particle
// indices). `shared` is the block's dynamic shared memory (cell_build_smem). max_count[0] gets the longest padded row,
// max_count[1] the candidates of a cell that goes through build_row for having too many.
template <int kWarps, int kHomes, int kRound>
__device__ __forceinline__ void build_cell(CellItems& t, float4* shared, const float4* __restrict__ frames,
                                           const double4* __restrict__ pos, const int* __restrict__ cell_start, int cell,
                                           float side, const CellBuild& bp, uint32_t* __restrict__ rows,
                                           int2* __restrict__ counts, int* __restrict__ max_count) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int cap = bp.geom.cap, max_words = bp.stage >> 5;
    float4* cand = shared;
    uint32_t* entries = reinterpret_cast<uint32_t*>(cand + bp.stage);
    uint32_t* masks = entries + bp.stage + warp * kHomes * max_words;  // masks[w * kHomes + k]
    uint32_t* row = entries + bp.stage + kWarps * kHomes * max_words + warp * kHomes * cell_row_pitch(cap);

    if (warp == 0) cell_items(cell_start, bp.geom.ncps, cell, side, t);
    __syncthreads();
    const int i0 = t.cell[kCellItems - 1].x, homes = t.cell[kCellItems - 1].y;
    if (homes == 0) return;
    const unsigned below = (1u << lane) - 1u;
    const float half = cell_half(side);
    {
        // Each warp takes kItems of the items, a particle per lane, all their loads in flight at once; the kept ones are
        // counted, then laid out. (A cell of more than 32 particles goes through the rest in a loop.)
        constexpr int kItems = (kCellItems + kWarps - 1) / kWarps;
        float4 c[kItems];
        unsigned kept[kItems];
        bool odd = false;
        auto keep = [&](const float4& q, int code) { return code == 13 || cell_reachable(q, half, bp.prune); };
#pragma unroll
        for (int q = 0; q < kItems; ++q) {
            const int r = warp * kItems + q;
            c[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (r < kCellItems && lane < t.cell[r].y) c[q] = frames[t.cell[r].x + lane];
        }
#pragma unroll
        for (int q = 0; q < kItems; ++q) {
            const int r = warp * kItems + q;
            if (r < kCellItems) {
                const int4 item = t.cell[r];
                const float4 shift = t.shift[r];
                odd |= c[q].w != 0.0f;
                c[q] = cell_candidate(c[q], shift);
                kept[q] = __ballot_sync(kAll, lane < item.y && keep(c[q], item.z));
                int more = 0;
                for (int u = 32; u < item.y; u += 32) {
                    const float4 f = frames[min(item.x + u + lane, item.x + item.y - 1)];
                    odd |= f.w != 0.0f;
                    more += __popc(__ballot_sync(kAll, u + lane < item.y && keep(cell_candidate(f, shift), item.z)));
                }
                if (lane == 0) t.off[r + 1] = __popc(kept[q]) + more;
            }
        }
        if (odd) t.odd = 1;
        __syncthreads();
        if (warp == 0) {
            int inc = lane > 0 && lane <= kCellItems ? t.off[lane] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kAll, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane <= kCellItems) t.off[lane] = inc;
        }
        __syncthreads();
        if (t.odd || t.off[kCellItems] > bp.stage) {
            if (threadIdx.x == 0) atomicMax(max_count + 1, t.off[kCellItems]);
            for (int h = threadIdx.x; h < homes; h += 32 * kWarps)
                build_row(pos, bp.geom, i0 + h, cell, cell_start, rows, counts, max_count);
            return;
        }
        auto put = [&](int at, unsigned mask, const float4& q, uint32_t entry) {
            if ((mask >> lane) & 1u) {
                const int v = at + __popc(mask & below);
                cand[v] = q;
                entries[v] = entry;
            }
        };
#pragma unroll
        for (int q = 0; q < kItems; ++q) {
            const int r = warp * kItems + q;
            if (r < kCellItems) {
                const int4 item = t.cell[r];
                const uint32_t entry = static_cast<uint32_t>(item.x + lane) | (static_cast<uint32_t>(item.z) << kCodeShift);
                int at = t.off[r];
                put(at, kept[q], c[q], entry);
                at += __popc(kept[q]);
                for (int u = 32; u < item.y; u += 32) {
                    const float4 more = cell_candidate(frames[min(item.x + u + lane, item.x + item.y - 1)], t.shift[r]);
                    const unsigned m = __ballot_sync(kAll, u + lane < item.y && keep(more, item.z));
                    put(at, m, more, entry + u);
                    at += __popc(m);
                }
            }
        }
        const int total = t.off[kCellItems];
        if (warp == 0 && total + lane < ((total + 31) & ~31)) cand[total + lane] = make_float4(0.0f, 0.0f, 0.0f, kCellFar);
    }
    __syncthreads();
    const int words = (t.off[kCellItems] + 31) >> 5;
    const CellOrder order{t.off[t.home], t.off[kCellItems - 1], t.off[t.own_items]};
    const int k = lane / (32 / kHomes);
    int longest = 0;
    for (int h0 = warp * kHomes; h0 < homes; h0 += kWarps * kHomes) {
        const bool real = h0 + k < homes;
        cell_masks<kHomes>(cand, entries, words, cand + order.home1 + h0, homes - h0, i0 + h0, pos, bp, masks);
        int len = 0, own = 0;
        cell_append<kHomes, kRound>(entries, masks, words, order, h0 + k, real, cap, row + k * cell_row_pitch(cap),
                                    len, own);
        longest = max(longest, cell_write<kHomes>(row, i0 + h0, real, len, own, bp, rows, counts));
    }
    report_longest(longest, max_count);
}

// Sparse systems: a cell's rows by one warp, all its candidates laid out one after another without regard to reach (a lane
// per item writes the item's entries, then a lane per candidate fetches it). `mem` is the warp's shared memory
// (sparse_smem). False, and nothing written, if there are more candidates than it holds.
template <int kHomes, int kRound>
__device__ __forceinline__ bool build_cell_warp(float4* mem, const float4* __restrict__ frames,
                                                const double4* __restrict__ pos, const int* __restrict__ cell_start,
                                                int cell, float side, const CellBuild& bp, uint32_t* __restrict__ rows,
                                                int2* __restrict__ counts, int* __restrict__ max_count) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, cap = bp.geom.cap;
    CellItems& t = *reinterpret_cast<CellItems*>(mem);
    float4* cand = mem + sizeof(CellItems) / sizeof(float4);
    uint32_t* entries = reinterpret_cast<uint32_t*>(cand + bp.warp_stage);
    uint32_t* masks = entries + bp.warp_stage;
    uint32_t* row = masks + kHomes * (bp.warp_stage >> 5);
    cell_items(cell_start, bp.geom.ncps, cell, side, t);
    __syncwarp();
    const int4 item = lane < kCellItems ? t.cell[lane] : make_int4(0, 0, 0, 0);
    int inc = item.y;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kAll, inc, o);
        if (lane >= o) inc += y;
    }
    const int total = __shfl_sync(kAll, inc, 31), words = (total + 31) >> 5;
    if (total > bp.warp_stage) return false;
    if (lane <= kCellItems) t.off[lane] = inc - item.y;
    for (int q = 0; q < item.y; ++q)
        entries[inc - item.y + q] = static_cast<uint32_t>(item.x + q) | (static_cast<uint32_t>(item.z) << kCodeShift);
    __syncwarp();
    bool odd = false;
    for (int v = lane; v < 32 * words; v += 32) {
        float4 q = make_float4(0.0f, 0.0f, 0.0f, kCellFar);
        if (v < total) {
            const uint32_t e = entries[v];
            const int code = static_cast<int>(e >> kCodeShift);
            const float4 f = frames[e & kIndexMask];
            odd |= f.w != 0.0f;
            q = cell_candidate(f, make_float4((code / 9 - 1) * side, (code / 3 % 3 - 1) * side, (code % 3 - 1) * side, 0.0f));
        }
        cand[v] = q;
    }
    const int i0 = t.cell[kCellItems - 1].x, homes = t.cell[kCellItems - 1].y;
    if (__any_sync(kAll, odd)) {
        for (int h = lane; h < homes; h += 32) build_row(pos, bp.geom, i0 + h, cell, cell_start, rows, counts, max_count);
        return true;
    }
    __syncwarp();
    const CellOrder order{t.off[t.home], t.off[kCellItems - 1], t.off[t.own_items]};
    const int k = lane / (32 / kHomes);
    int longest = 0;
    for (int h0 = 0; h0 < homes; h0 += kHomes) {
        const bool real = h0 + k < homes;
        cell_masks<kHomes>(cand, entries, words, cand + order.home1 + h0, homes - h0, i0 + h0, pos, bp, masks);
        int len = 0, own = 0;
        cell_append<kHomes, kRound>(entries, masks, words, order, h0 + k, real, cap, row + k * cell_row_pitch(cap), len,
                                    own);
        longest = max(longest, cell_write<kHomes>(row, i0 + h0, real, len, own, bp, rows, counts));
    }
    report_longest(longest, max_count);
    return true;
}

// Sparse systems: the warps of a block go through the cells [c0, c0 + bp.group) each, past the empty ones. The cells that are
// too full for a warp (a droplet's, in a box that is otherwise empty) go to a list, for blocks to build: full(cell) adds one.
constexpr int kSparseWarps = 4, kSparseHomes = 4;
constexpr int kMostWarpStage = 320;
__host__ __device__ inline size_t sparse_smem_warp(int warp_stage, int cap) {
    return sizeof(CellItems) + (sizeof(float4) + sizeof(uint32_t)) * warp_stage +
           sizeof(uint32_t) * kSparseHomes * (static_cast<size_t>(cell_row_pitch(cap)) + warp_stage / 32);
}
template <typename Full>
__device__ __forceinline__ void build_cells_sparse(float4* shared, const float4* __restrict__ frames,
                                                   const double4* __restrict__ pos, const int* __restrict__ cell_start,
                                                   int ncells, int c0, float side, const CellBuild& bp,
                                                   uint32_t* __restrict__ rows, int2* __restrict__ counts,
                                                   int* __restrict__ max_count, Full full) {
    static_assert(sizeof(CellItems) % 16 == 0, "the candidates behind it are 16-byte vectors");
    const int lane = threadIdx.x & 31, c = c0 + lane;
    float4* mem = shared + (threadIdx.x >> 5) * (sparse_smem_warp(bp.warp_stage, bp.geom.cap) / sizeof(float4));
    unsigned todo = __ballot_sync(0xffffffffu, lane < bp.group && c < ncells && cell_start[c] < cell_start[c + 1]);
    while (todo) {
        const int cell = c0 + __ffs(todo) - 1;
        todo &= todo - 1;
        const bool done = bp.warp_stage != 0 && build_cell_warp<kSparseHomes, 16>(mem, frames, pos, cell_start, cell, side, bp,
                                                                                  rows, counts, max_count);
        if (!done && lane == 0) full(cell);
        __syncwarp();
    }
}

// Calls f(k) for the k below n that fall to this block: one of every gridDim.x in a row, a place further in each row (with a
// fixed place a block would get cells of one z alone where the grid is a multiple of the cells per side, and a slab's cells
// would fall to a few of the blocks: slab of 300,000, 37 cells a side, 1,184 blocks: 134 us a step of md_run's graphs, in turns 105).
template <typename F>
__device__ __forceinline__ void block_turns(int n, F f) {
    const int blocks = static_cast<int>(gridDim.x);
    for (int k0 = 0, place = static_cast<int>(blockIdx.x); k0 < n; k0 += blocks, place = place + 1 < blocks ? place + 1 : 0)
        if (k0 + place < n) f(k0 + place);
}

// One home cell per block, or, with `list`, the `*listed` cells of the list in turn
template <int kWarps, int kHomes, int kRound, bool kList>
__global__ void __launch_bounds__(32 * kWarps)
    k_nlist_build_cells(const float4* __restrict__ frames, const double4* __restrict__ pos,
                        const int* __restrict__ cell_start, float side, CellBuild bp, uint32_t* __restrict__ rows,
                        int2* __restrict__ counts, int* __restrict__ max_count, const int* __restrict__ list,
                        const int* __restrict__ listed) {
    extern __shared__ float4 sm_cell[];
    __shared__ CellItems t;
    if constexpr (kList) {
        for (int k = blockIdx.x, n = *listed; k < n; k += gridDim.x) {
            build_cell<kWarps, kHomes, kRound>(t, sm_cell, frames, pos, cell_start, list[k], side, bp, rows, counts, max_count);
            __syncthreads();  // the shared memory goes to the next cell
        }
    } else {
        build_cell<kWarps, kHomes, kRound>(t, sm_cell, frames, pos, cell_start, blockIdx.x, side, bp, rows, counts, max_count);
    }
}

// Sparse systems: a cell per warp; list and *listed (zero before) get the cells left for k_nlist_build_cells
__global__ void __launch_bounds__(32 * kSparseWarps, 7)
    k_nlist_build_sparse(const float4* __restrict__ frames, const double4* __restrict__ pos,
                         const int* __restrict__ cell_start, int ncells, float side, CellBuild bp,
                         uint32_t* __restrict__ rows, int2* __restrict__ counts, int* __restrict__ max_count,
                         int* __restrict__ list, int* __restrict__ listed) {
    extern __shared__ float4 sm_cell[];
    build_cells_sparse(sm_cell, frames, pos, cell_start, ncells,
                       static_cast<int>(blockIdx.x * kSparseWarps + (threadIdx.x >> 5)) * bp.group, side, bp, rows, counts,
                       max_count, [&](int cell) { list[atomicAdd(listed, 1)] = cell; });
}

}  // namespace md
