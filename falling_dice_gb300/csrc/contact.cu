// contact.cu -- self-contact broad and narrow phase (the reference's MC/src/sim.cpp:144-165
// hash grid and closest-shape penalty), rebuilt as a Morton-ordered uniform grid.
//
// This translation unit is compiled with -fmad=false: the closest-point arithmetic must
// round exactly like the reference so that the set of pairs with dist < target is the
// reference's set bit for bit (positions are bit-identical, see k_state).
//
// Broad phase.  Every shape (N joint spheres, then B beam capsules, as sim.cpp:148-150)
// enters every grid cell its margin-inflated AABB touches (sim.cpp:153-157; the same floor() cell
// coordinates, the cell twice the reference's by default).  Cells are numbered by the Morton code of their
// coordinates relative to the grid origin (row-major when the Morton range does not fit),
// and each entry goes straight into a slot of its bin (bins of fixed capacity, the slot
// handed out by the bin's atomic counter).  The pair pass gives 128 shapes of a bin at
// a time to a warp, which meets them with those before them in the order the atomics handed out:
// the candidate list's order can vary from run to run, its content cannot, and nothing computed
// from it depends on the order (pair sets are reported sorted).  A pair is examined only in the cell that is the
// minimum corner of the intersection of the two shapes' cell ranges: every pair that
// shares a cell is examined exactly once -- the reference's `tested` set without a set.
// A conservative box test (32 levels per axis inside the bin), the local-shape exclusion
// (sim.cpp:24-39) and certified FP32 distance bounds run before the FP64 narrow phase.
//
// Sums without an order.  Candidates, kept candidates and contacts are appended to flat lists in
// whatever order the warps arrive; a contact's forces and energy are added to its nodes' records
// as fixed-point integers (NodeContact), whose sums are exact and the same in any order.  So no
// result depends on the lists' order, and no list is counted, scanned, filled or sorted per
// node.
//
// No host synchronisation: sizes that can overflow a buffer (a bin's slots, bins, candidates,
// contacts, a shape spanning too many cells) raise a flag instead of writing out of bounds, and
// the host repeats the evaluation with larger buffers (or coarser cells) when it sees one.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace mcg {

namespace {

constexpr long long kMaxCellsPerShape = 1 << 12;
constexpr uint32_t kBoxMax = 32767u;    // 15-bit box coordinates
constexpr int kPairThreads = 128;
constexpr int kPairWarps = kPairThreads / 32;
constexpr int kPairGroups = 4;           // groups of 32 shapes of a bin staged at a time
constexpr int kChunk = 32 * kPairGroups;  // shapes of a unit of pair work (ContactBufs::units)
constexpr int kLevelBits = 5;            // box levels inside a bin: 2^kLevelBits = 32 per axis
constexpr int kFilterBlocks = 4 * 152;   // 256 threads each, grid-stride
constexpr int kListThreads = 128;        // the contact kernel: a warp per FP64 unit and block
constexpr int kListWarps = kListThreads / 32;
constexpr int kListBlocks = 5 * 152;

__device__ __forceinline__ uint32_t spread3_10(uint32_t v) {  // 10 bits -> every third bit
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}
__device__ __forceinline__ uint32_t compact3_10(uint32_t v) {
    v &= 0x09249249u;
    v = (v ^ (v >> 2)) & 0x030c30c3u;
    v = (v ^ (v >> 4)) & 0x0300f00fu;
    v = (v ^ (v >> 8)) & 0x030000ffu;
    v = (v ^ (v >> 16)) & 0x000003ffu;
    return v;
}

// grid[]: 0-2 origin cell, 3-5 dims, 6 mode (0 Morton, 1 row-major), 7 valid,
//         8 number of bins
__device__ __forceinline__ uint32_t bin_of(const int* g, int i, int j, int k) {
    if (g[6] == 0) return spread3_10(uint32_t(i)) | (spread3_10(uint32_t(j)) << 1) | (spread3_10(uint32_t(k)) << 2);
    return uint32_t((k * g[4] + j) * g[3] + i);
}
__device__ __forceinline__ int3 cell_of(const int* g, uint32_t b) {
    if (g[6] == 0) return make_int3(int(compact3_10(b)), int(compact3_10(b >> 1)), int(compact3_10(b >> 2)));
    const int i = int(b % uint32_t(g[3]));
    const int j = int((b / uint32_t(g[3])) % uint32_t(g[4]));
    const int k = int(b / (uint32_t(g[3]) * uint32_t(g[4])));
    return make_int3(i, j, k);
}

// First cell of a shape packed for the pair test (10 bits per axis, relative to the grid
// origin).
__device__ __forceinline__ uint32_t pack_cell(int i, int j, int k) {
    return (uint32_t(i) & 1023u) | ((uint32_t(j) & 1023u) << 10) | ((uint32_t(k) & 1023u) << 20);
}

// ---- geometry (sim.cpp:9-22), rounding as the reference --------------------------------
__device__ __forceinline__ double sat(double x) { return clampd(x, 0.0, 1.0); }

struct Closest { double s, t; d3 pa, pb; };

struct ShapeRef {
    d3 a, b;
    double r;
    bool capsule;
};

__device__ __forceinline__ int2 shape_nodes(const DevTopo& t, uint32_t s) {
    if (s < uint32_t(t.N)) return make_int2(int(s), -1);
    return t.ab[s - uint32_t(t.N)];
}

__device__ __forceinline__ ShapeRef load_shape(const DevTopo& t, const double4_32a* x, double jr, uint32_t s) {
    ShapeRef sh;
    if (s < uint32_t(t.N)) {
        const double4_32a v = x[s];
        sh.a = sh.b = d3{v.x, v.y, v.z};
        sh.r = jr;
        sh.capsule = false;
    } else {
        const int bi = int(s) - t.N;
        const int2 ab = t.ab[bi];
        const double4_32a va = x[ab.x], vb = x[ab.y];
        sh.a = d3{va.x, va.y, va.z};
        sh.b = d3{vb.x, vb.y, vb.z};
        sh.r = t.radius[bi];
        sh.capsule = true;
    }
    return sh;
}

// Closest points of two shapes (sim.cpp:9-22: sphere or segment against sphere or segment), a the
// lower one, so never a segment against a sphere.  The lanes of a warp hold all three cases; they
// take one path, each case's quotients and clamps selected, as the reference rounds them.  Two
// divisions, and a third where a lane's t is clamped; comparisons on bit patterns.
__device__ __forceinline__ Closest shape_closest(const ShapeRef& A, const ShapeRef& B) {
    const d3 d1 = A.b - A.a, d2 = B.b - B.a, r = A.a - B.a;
    const double a = dot(d1, d1), e = dot(d2, d2), f = dot(d2, r), c = dot(d1, r), b = dot(d1, d2);
    // does the shape have a direction (a sphere against a segment has no threshold for the segment)
    const bool ga = A.capsule && less_bits(1e-20, a), gb = A.capsule ? less_bits(1e-20, e) : B.capsule;
    double s = 0, t = 0;
    if (ga && gb) {
        const double den = a * e - b * b;
        if (less_bits(1e-20, fabs(den))) s = sat((b * f - c * e) / den);
    }
    if (gb) t = (ga ? b * s + f : f) / (A.capsule ? e : fmax(1e-30, e));
    const bool low = ga && (!gb || t < 0), high = ga && gb && t > 1;
    if (low || high) s = sat((low ? -c : b - c) / a);
    t = low ? 0 : high ? 1 : ga ? t : sat(t);
    return {s, t, A.a + d1 * s, B.a + d2 * t};
}

// Membership of the node pair (u, v) in the connected set (sim.cpp:24-39 reads
// connected_.count(pairKey(u, v))): multiplicative hash, linear probing.
__device__ __forceinline__ bool is_connected(const DevTopo& t, int u, int v) {
    const unsigned long long key = u <= v ? ((unsigned long long)u << 32) | uint32_t(v)
                                          : ((unsigned long long)v << 32) | uint32_t(u);
    unsigned long long h = (key * 0x9E3779B97F4A7C15ull) >> t.conn_shift;
    for (unsigned long long probe = 0; probe <= t.conn_mask; probe++) {
        const unsigned long long k = t.conn_hash[h];
        if (k == key) return true;
        if (k == ~0ull) return false;
        h = (h + 1) & t.conn_mask;
    }
    return false;
}

// Local shapes (sim.cpp:24-39): a shared node, or a connected node pair.  Shapes are
// distinct here, so "same beam" cannot occur.  The shared-node half is cheap and decides
// most broad-phase candidates in a lattice; the connected half probes the hash set.
__device__ __forceinline__ bool any_connected(const DevTopo& t, int2 a, int2 b) {
    const int an[2] = {a.x, a.y}, bn[2] = {b.x, b.y};
    const int na = a.y >= 0 ? 2 : 1, nb = b.y >= 0 ? 2 : 1;
    for (int i = 0; i < na; ++i)
        for (int j = 0; j < nb; ++j)
            if (is_connected(t, an[i], bn[j])) return true;
    return false;
}

// Rest of the test of a candidate pair (sa < sb) that is not a local pair (shared or
// connected nodes, excluded by the pair pass and the filter): FP64 closest points,
// dist < target.  Out of line: few candidates get here, and keeping its registers out of the
// calling loops keeps their occupancy up.
struct PairHit {
    bool hit;
    double s, t, pen;
    d3 n;
};
__device__ __noinline__ PairHit narrow_phase(const DevTopo& t, const PhysParams& p, const double4_32a* x, uint32_t sa,
                                             uint32_t sb) {
    PairHit h;
    h.hit = false;
    const ShapeRef A = load_shape(t, x, p.joint_radius, sa);
    const ShapeRef B = load_shape(t, x, p.joint_radius, sb);
    const Closest cp = shape_closest(A, B);
    const d3 delta = cp.pb - cp.pa;
    const double dist = len(delta), target = A.r + B.r + p.contact_margin;
    if (!(dist < target)) return h;
    h.hit = true;
    h.s = cp.s;
    h.t = cp.t;
    h.pen = target - dist;
    h.n = dist > 1e-12 ? delta * (1.0 / dist) : unit(d3{.37 + .001 * double(int(sa)), .73, -.41 + .001 * double(int(sb))});
    return h;
}

// ---- kernels -------------------------------------------------------------------------------
// Boxes and bin entries of every shape, when the candidate list is rebuilt (flags[1], decided by
// the state and center kernels).
// The box is in single precision rounded outward: it contains the reference's double-precision
// box (sim.cpp:154), and cell indices are a monotone function of it, so two shapes whose
// reference boxes overlap share a cell.  The pair-test record holds the box quantized to 15 bits
// per axis (floor minus one quantum for the low side, ceil plus one for the high side, so the
// quantized box contains the FP32 box whatever the rounding of the scaling) and the first cell
// packed as three 10-bit fields.
// Entries: one per cell of the shape's range, written straight into the bin's slot that the bin
// counter hands out (all counters are zero here: the filter clears them at the end of a build), four
// returning atomics in flight per thread; the entry that begins a chunk of its bin lists the
// chunk as a unit of pair work.  A bin that fills up keeps counting (kOverEntries, and
// the largest count in counts[kLargestBin] so the host can size bin_slots).
__device__ __forceinline__ void emit_shape(const DevTopo& t, const PhysParams& p, const float4* __restrict__ xf_lo,
                                           const float4* __restrict__ xf_hi, float skin, const ContactBufs& c,
                                           const int* __restrict__ grid, int s) {
    const int2 nd = shape_nodes(t, uint32_t(s));
    const int n1 = nd.y >= 0 ? nd.y : nd.x;
    if (!t.active[t.node_inst[nd.x]]) return;  // inactive instances take no part
    const float4 al = xf_lo[nd.x], ah = xf_hi[nd.x], bl = xf_lo[n1], bh = xf_hi[n1];
    const float pad = __fadd_ru(s < t.N ? p.joint_padf : t.padf[s - t.N], skin);
    const float lo[3] = {__fsub_rd(fminf(al.x, bl.x), pad), __fsub_rd(fminf(al.y, bl.y), pad),
                         __fsub_rd(fminf(al.z, bl.z), pad)};
    const float hi[3] = {__fadd_ru(fmaxf(ah.x, bh.x), pad), __fadd_ru(fmaxf(ah.y, bh.y), pad),
                         __fadd_ru(fmaxf(ah.z, bh.z), pad)};
    if (!(isfinite(lo[0]) && isfinite(lo[1]) && isfinite(lo[2]) && isfinite(hi[0]) && isfinite(hi[1]) &&
          isfinite(hi[2]))) {
        atomicOr(c.flags, uint32_t(kNonFinite));
        return;
    }
    int c0[3], dim[3];
    uint32_t q0[3], q1[3];
    bool wide = false;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const float top = float(grid[3 + d] - 1);
        const float org = float(grid[d]);
        c0[d] = int(fminf(fmaxf(floorf(lo[d] * p.inv_cell_f) - org, 0.f), top));
        dim[d] = int(fminf(fmaxf(floorf(hi[d] * p.inv_cell_f) - org, 0.f), top)) - c0[d] + 1;
        wide |= dim[d] > 1024;
        const float qs = __int_as_float(grid[10 + d]), qo = __int_as_float(grid[13 + d]);
        q0[d] = uint32_t(fminf(fmaxf(floorf((lo[d] - qo) * qs) - 1.f, 0.f), float(kBoxMax)));
        q1[d] = uint32_t(fminf(fmaxf(ceilf((hi[d] - qo) * qs) + 1.f, 0.f), float(kBoxMax)));
    }
    if (wide || (long long)dim[0] * dim[1] * dim[2] > kMaxCellsPerShape) {
        atomicOr(c.flags, uint32_t(kOverSpan));  // the host coarsens the grid and evaluates again
        return;
    }
    c.rec[s] = make_uint4(q0[0] | (q0[1] << 16), q1[0] | (q1[1] << 16), q0[2] | (q1[2] << 16),
                          pack_cell(c0[0], c0[1], c0[2]));
    const int n = dim[0] * dim[1] * dim[2];
    int i = 0, j = 0, k = 0;  // the next cell of the range
    for (int e0 = 0; e0 < n; e0 += 4) {
        uint32_t bin[4], slot[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            if (e0 + e >= n) break;
            bin[e] = bin_of(grid, c0[0] + i, c0[1] + j, c0[2] + k);
            slot[e] = atomicAdd(&c.bin_count[bin[e]], 1u);
            if (++i == dim[0]) {
                i = 0;
                if (++j == dim[1]) {
                    j = 0;
                    k++;
                }
            }
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
            if (e0 + e >= n) break;
            if (slot[e] < uint32_t(c.bin_slots)) {
                c.bin_items[size_t(bin[e]) * size_t(c.bin_slots) + slot[e]] = uint32_t(s);
                if (slot[e] % kChunk == 0)  // the first shape of a chunk of the bin
                    c.units[atomicAdd(c.counts + kUnits, 1u)] = make_uint2(bin[e], slot[e] / kChunk);
            } else {
                atomicOr(c.flags, uint32_t(kOverEntries));
                atomicMax(c.counts + kLargestBin, slot[e] + 1);
            }
        }
    }
}

__global__ void __launch_bounds__(kBlock) k_shapes(DevTopo t, PhysParams p, const float4* __restrict__ xf_lo,
                                                   const float4* __restrict__ xf_hi, float skin, ContactBufs c) {
    const int S = t.N + t.B;
    const int* __restrict__ grid = c.grid;
    if (!c.flags[1] || !grid[7]) return;
    for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < unsigned(S); s += gridDim.x * blockDim.x)
        emit_shape(t, p, xf_lo, xf_hi, skin, c, grid, int(s));
}

// ---- pair enumeration inside a bin ---------------------------------------------------------
// 32 x 32 pairs at a time, one bit each.  Inside its bin a shape's box is reduced to 32 levels
// per axis, by one monotone map per axis, so overlapping boxes have overlapping level ranges.
// The low level is 0 exactly when the shape's first cell on that axis lies before the bin, so
// that "the bin is the pair's first common cell" (each pair is examined once, the reference's
// `tested` set without a set) reads: one of the two low levels is not 0.
// For a group of 32 shapes the warp makes, per axis, the tables
//   below[l] = the shapes whose low level is at most l, above[l] = those whose high level is at
//   least l,
// one bit per shape and one entry per level (32 entries: reads of different levels hit different
// banks).  A shape's box partners in the group are then below[its high] & above[its low] over
// the axes, without the below[0] (not starting here) where the shape does not start here either.
// The tables come from bit planes: a bit transpose across the warp turns the 32 shapes' levels
// into one word per level bit, and lane l compares its own number with all 32 levels by one
// three-input logic operation per bit.
struct PairRow {
    uint32_t id;
    int n0, n1;       // the shape's nodes (a joint's node twice)
    uint32_t levels;  // low levels in bits 5 d, high levels in bits 15 + 5 d
};

// The bin's frame: level of the quantized coordinate q on axis d is (q - base) scale + 1, clamped
// and rounded.
struct BinFrame {
    float base[3], scale[3];
    uint32_t cell;  // packed cell of the bin
};

__device__ __forceinline__ uint32_t level_of(const BinFrame& f, int d, uint32_t q) {
    // integer to float and back by adding powers of two: conversions run at a quarter of the rate
    const float v = (__int_as_float(int(0x4b000000u | q)) - 8388608.f - f.base[d]) * f.scale[d] + 1.f;
    return uint32_t(__float_as_int(fminf(fmaxf(v, 1.f), float((1 << kLevelBits) - 1)) + 8388608.f)) & 31u;
}

__device__ __forceinline__ PairRow load_row(const DevTopo& t, uint32_t s, const uint4* __restrict__ rec, const BinFrame& f) {
    const uint4 r = rec[s];
    const int2 nd = s < uint32_t(t.N) ? make_int2(int(s), int(s)) : t.ab[s - uint32_t(t.N)];
    const uint32_t before = r.w ^ f.cell;  // cell spans are below 1024 per axis: a field is 0 where the first cell is the bin's
    PairRow row{s, nd.x, nd.y, 0};
    if (!(before & 0x3ffu)) row.levels |= level_of(f, 0, r.x & 0x7fffu);
    if (!(before & 0xffc00u)) row.levels |= level_of(f, 1, r.x >> 16) << 5;
    if (!(before & 0x3ff00000u)) row.levels |= level_of(f, 2, r.z & 0x7fffu) << 10;
    row.levels |= level_of(f, 0, r.y & 0x7fffu) << 15 | level_of(f, 1, r.y >> 16) << 20 | level_of(f, 2, r.z >> 16) << 25;
    return row;
}

// Transposes a 32 x 32 bit matrix held one row per lane: afterwards bit j of lane k is bit k of
// lane j's argument.
__device__ __forceinline__ uint32_t transpose_bits(uint32_t x, int lane) {
    uint32_t m = 0x0000ffffu;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x, s);
        x = (lane & s) ? (x & ~m) | ((y & ~m) >> s) : (x & m) | ((y & m) << s);
        m ^= m << (s >> 1);
    }
    return x;
}

// A warp's shared memory: the staged groups' tables, levels and shapes (the last place holds the
// shapes of a row group that is not staged), the queue of meeting boxes and the candidates on
// their way to the list.
constexpr int kPairOut = 64, kPairRound = 8;
struct PairShared {
    int4 shape[kPairGroups + 1][32];  // id, nodes
    uint32_t below[kPairGroups][3][32], above[kPairGroups][3][32];
    uint32_t levels[kPairGroups][32];
    uint2 out[kPairOut];
    uint16_t queue[32 * kPairRound + 32];  // row rank << 8 | column rank
};

// Pairs of meeting boxes come a few per lane and unevenly; queued, they are checked for a shared
// node (three quarters of them share one in a cubic+BCC lattice) 32 at a time.  Candidates go on
// to the flat list with one atomic and coalesced stores per flush; past cand_cap they are counted
// but not stored and kOverCandidates is raised.
// Every loop ends and every lane reaches every warp operation: nq, n and the claimed units are the
// same in all lanes; a pass of add takes at least one bit from each lane that has one, at most
// 32 kPairRound into a queue that holds less than 32 before; check takes min(32, nq) from it; a claim
// moves the cursor on, so a warp claims until the units are gone.  No warp waits for another.
struct PairQueue {
    PairShared& s;
    int nq, n;  // pairs queued, candidates held: the same in all lanes
    long long cand_cap;
    uint2* cand;
    uint32_t *ncand, *flags;
    __device__ __forceinline__ void flush(int lane) {
        __syncwarp();
        uint32_t base = 0;
        if (lane == 0 && n) {
            base = atomicAdd(ncand, uint32_t(n));
            if ((long long)base + n > cand_cap) atomicOr(flags, uint32_t(kOverCandidates));
        }
        base = __shfl_sync(0xffffffffu, base, 0);
        for (int i = lane; i < n; i += 32)
            if ((long long)base + i < cand_cap) cand[(long long)base + i] = s.out[i];
        n = 0;
        __syncwarp();
    }
    // Checks the last min(32, nq) queued pairs.
    __device__ __forceinline__ void check(int lane) {
        const int m = min(32, nq);
        nq -= m;
        bool keep = false;
        int4 p{}, q{};
        if (lane < m) {
            const uint32_t code = s.queue[nq + lane];
            p = (&s.shape[0][0])[code >> 8];
            q = (&s.shape[0][0])[code & 255u];
            keep = p.y != q.y && p.y != q.z && p.z != q.y && p.z != q.z;
        }
        const unsigned k = __ballot_sync(0xffffffffu, keep);
        if (keep) s.out[n + __popc(k & ((1u << lane) - 1u))] = make_uint2(min(uint32_t(p.x), uint32_t(q.x)), max(uint32_t(p.x), uint32_t(q.x)));
        n += __popc(k);
        if (n > kPairOut - 32) flush(lane);
    }
    // Bit j of `bits`: the row of rank `row` meets column 32 h + j.  All lanes call it.
    __device__ __forceinline__ void add(uint32_t bits, uint32_t row, uint32_t h, int lane) {
        const uint32_t code = row << 8 | h << 5;
        while (__any_sync(0xffffffffu, bits != 0)) {
            // up to kPairRound pairs per lane, placed by a warp scan
            const int cnt = min(__popc(bits), kPairRound);
            int incl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            uint16_t* at = s.queue + nq + (incl - cnt);
            nq += __shfl_sync(0xffffffffu, incl, 31);
            for (int k = 0; k < cnt; k++) {
                at[k] = uint16_t(code | uint32_t(__ffs(bits) - 1));
                bits &= bits - 1;
            }
            __syncwarp();
            while (nq >= 32) check(lane);
            __syncwarp();
        }
    }
};

// The row's box partners in group g whose first common cell is the bin.
__device__ __forceinline__ uint32_t meet(const PairShared& s, int g, uint32_t levels) {
    uint32_t hit = 0xffffffffu;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const uint32_t lo = levels >> (5 * d) & 31u, hi = levels >> (15 + 5 * d) & 31u;
        const uint32_t starts = lo ? 0xffffffffu : ~s.below[g][d][0];
        hit &= s.below[g][d][hi] & s.above[g][d][lo] & starts;
    }
    return hit;
}

// Candidate pairs of every bin holding two or more shapes.  A unit of work is a chunk of
// kPairGroups groups of 32 shapes of a bin: a warp stages the chunk's groups, and every group of
// the bin up to the staged ones (those of earlier chunks reread) meets them, one 32 x 32 block
// per step.  Warps claim units from a cursor (flags[3]), from the end of the list, where the later
// chunks of large bins are (they take longest), so units of uneven size balance over the grid;
// they count the build's cell entries and occupied bins on the way.
// An integer kernel, bound by instruction issue: its time follows the staged groups, the blocks
// and the meeting boxes.
__global__ void __launch_bounds__(kPairThreads, 7) k_bin_pairs(DevTopo t, const int* __restrict__ grid,
                                                               const uint32_t* __restrict__ bin_count, int bin_slots,
                                                               uint32_t* __restrict__ counts,
                                                               const uint2* __restrict__ unit_list,
                                                               const uint32_t* __restrict__ bin_items,
                                                               const uint4* __restrict__ rec, long long cand_cap,
                                                               uint2* __restrict__ cand, uint32_t* __restrict__ flags) {
    __shared__ PairShared shared[kPairWarps];
    if (!flags[1]) return;
    const int lane = threadIdx.x & 31;
    const uint32_t units = counts[kUnits];
    PairShared& s = shared[threadIdx.x >> 5];
    PairQueue out{s, 0, 0, cand_cap, cand, counts + kCand, flags};
    const float quanta[3] = {kBoxQuanta / float(grid[3]), kBoxQuanta / float(grid[4]), kBoxQuanta / float(grid[5])};
    BinFrame frame;
#pragma unroll
    for (int d = 0; d < 3; d++) frame.scale[d] = float((1 << kLevelBits) - 2) / quanta[d];
    uint32_t mine[kLevelBits];  // the bits of the lane's number, expanded
#pragma unroll
    for (int k = 0; k < kLevelBits; k++) mine[k] = (lane >> k & 1) ? 0xffffffffu : 0u;
    uint32_t entries = 0, occupied = 0;  // this lane's share of the build's counts
    // several units a claim while each warp of the grid still has many claims to come
    const uint32_t warps = kPairWarps * gridDim.x, grab = units > 16 * warps ? 4u : units > 8 * warps ? 2u : 1u;
    for (;;) {
        uint32_t u0 = 0;
        if (lane == 0) u0 = atomicAdd(flags + 3, grab);
        u0 = __shfl_sync(0xffffffffu, u0, 0);
        if (u0 >= units) break;
        uint2 unit = make_uint2(0, 0);
        uint32_t cnt = 0;
        if (uint32_t(lane) < grab && u0 + lane < units) {
            unit = unit_list[units - 1 - (u0 + lane)];
            cnt = bin_count[unit.x];
            if (unit.y == 0) {
                entries += cnt;
                occupied += cnt >= 2;
            }
        }
        // a full bin repeats the build (kOverEntries), so clamping only keeps reads in bounds
        cnt = min(cnt, uint32_t(bin_slots));
        unsigned todo = __ballot_sync(0xffffffffu, cnt >= 2);
        while (todo) {
            const int j = __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t b = __shfl_sync(0xffffffffu, unit.x, j);
            const int n = int(__shfl_sync(0xffffffffu, cnt, j));
            const int g0 = kPairGroups * int(__shfl_sync(0xffffffffu, unit.y, j));  // first staged group
            const uint32_t* items = bin_items + size_t(b) * size_t(bin_slots);
            const int3 cc = cell_of(grid, b);
            frame.cell = pack_cell(cc.x, cc.y, cc.z);
            frame.base[0] = float(cc.x) * quanta[0];
            frame.base[1] = float(cc.y) * quanta[1];
            frame.base[2] = float(cc.z) * quanta[2];
            const int left = n - 32 * g0;  // shapes from the first staged one on
            const int m = min((left + 31) >> 5, kPairGroups);
            __syncwarp();  // the last reads of the staged groups are done
            for (int g = 0; g < m; g++) {
                PairRow row{0, 0, 0, 0};
                if (32 * g + lane < left) row = load_row(t, items[32 * (g0 + g) + lane], rec, frame);
                s.shape[g][lane] = make_int4(int(row.id), row.n0, row.n1, 0);
                s.levels[g][lane] = row.levels;
                const uint32_t plane = transpose_bits(row.levels, lane);
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    uint32_t le = 0xffffffffu, ge = 0xffffffffu;
#pragma unroll
                    for (int k = 0; k < kLevelBits; k++) {
                        const uint32_t pl = __shfl_sync(0xffffffffu, plane, 5 * d + k);
                        const uint32_t ph = __shfl_sync(0xffffffffu, plane, 15 + 5 * d + k);
                        le = (mine[k] & ~pl) | (~(mine[k] ^ pl) & le);
                        ge = (ph & ~mine[k]) | (~(ph ^ mine[k]) & ge);
                    }
                    s.below[g][d][lane] = le;
                    s.above[g][d][lane] = ge;
                }
            }
            __syncwarp();
            for (int g = 0; g < m; g++) {
                const uint32_t levels = s.levels[g][lane];
                const bool valid = 32 * g + lane < left;
                for (int h = g; h < m; h++) {
                    uint32_t bits = meet(s, h, levels);
                    if (left - 32 * h < 32) bits &= (1u << (left - 32 * h)) - 1u;
                    if (h == g) bits &= ~1u << lane;  // each pair of a group once: j > lane
                    out.add(valid ? bits : 0u, uint32_t(32 * g + lane), uint32_t(h), lane);
                }
            }
            for (int g = 0; g < g0; g++) {  // groups (full) of earlier chunks
                const PairRow row = load_row(t, items[32 * g + lane], rec, frame);
                if (out.nq) out.check(lane);  // the queue refers to the row group replaced here
                __syncwarp();
                s.shape[kPairGroups][lane] = make_int4(int(row.id), row.n0, row.n1, 0);
                __syncwarp();
                for (int h = 0; h < m; h++) {
                    uint32_t bits = meet(s, h, row.levels);
                    if (left - 32 * h < 32) bits &= (1u << (left - 32 * h)) - 1u;
                    out.add(bits, uint32_t(32 * kPairGroups + lane), uint32_t(h), lane);
                }
            }
            if (out.nq) out.check(lane);  // the queue refers to the staged groups
        }
    }
    out.flush(lane);
    entries = __reduce_add_sync(0xffffffffu, entries);
    occupied = __reduce_add_sync(0xffffffffu, occupied);
    if (lane == 0) {
        if (entries) atomicAdd(counts + kEntries, entries);
        if (occupied) atomicAdd(counts + kOccupied, occupied);
    }
}

// Certified single-precision lower bound on the distance of a candidate pair.  A pair certainly
// farther apart than pad_a + pad_b (>= the reference's target ra + rb + margin) fails the
// reference's test dist < target; the others go to the exact test.
//
// For any unit vector n, the distance between segments p1 + s d1 and p2 + t d2 (s, t in
// [0, 1]) is at least  L(n) = n.(p1 - p2) + min(0, n.d1) - max(0, n.d2):  n.(P - Q) <= |P - Q|
// and the minimum of the linear form over the parameter square is at a corner.  n is the
// unit direction between approximate closest points (FP32, the clamped solution of
// sim.cpp:9-18), which makes the bound nearly tight.  L is evaluated from FP32 endpoints
// rounded down (|error| <= 2^-23 X per coordinate, X the largest endpoint coordinate); the
// rounding of the differences, the three dot products and the sums adds at most about
// 4e-6 X in total, bounded here by 3e-5 X + 1e-9 m, and |n| = 1 up to 1e-6.  Nothing is certified
// of touching segments and non-finite data.
struct DistBounds {
    bool far_ok;      // far is a valid lower bound (the closest points are not within 1e-7 m)
    float far;        // certified lower bound on the distance, already less its error
    float pad_sum;    // pad_a + pad_b >= the reference's target
};
__device__ __forceinline__ DistBounds dist_bounds(const DevTopo& t, const PhysParams& p, const float4* __restrict__ xf,
                                                  uint32_t sa, uint32_t sb) {
    const int2 na = sa < uint32_t(t.N) ? make_int2(int(sa), int(sa)) : t.ab[sa - uint32_t(t.N)];
    const int2 nb = sb < uint32_t(t.N) ? make_int2(int(sb), int(sb)) : t.ab[sb - uint32_t(t.N)];
    const float pa = sa < uint32_t(t.N) ? p.joint_padf : t.padf[sa - uint32_t(t.N)];
    const float pb = sb < uint32_t(t.N) ? p.joint_padf : t.padf[sb - uint32_t(t.N)];
    const float4 a0 = xf[na.x], a1 = xf[na.y], b0 = xf[nb.x], b1 = xf[nb.y];
    const float X = fmaxf(fmaxf(fmaxf(fabsf(a0.x), fabsf(a0.y)), fmaxf(fabsf(a0.z), fabsf(a1.x))),
                          fmaxf(fmaxf(fabsf(a1.y), fabsf(a1.z)), fmaxf(fmaxf(fabsf(b0.x), fabsf(b0.y)),
                                                                     fmaxf(fmaxf(fabsf(b0.z), fabsf(b1.x)),
                                                                           fmaxf(fabsf(b1.y), fabsf(b1.z))))));
    const float wx = a0.x - b0.x, wy = a0.y - b0.y, wz = a0.z - b0.z;
    const float ux = a1.x - a0.x, uy = a1.y - a0.y, uz = a1.z - a0.z;
    const float vx = b1.x - b0.x, vy = b1.y - b0.y, vz = b1.z - b0.z;
    // dot products by explicit FMAs (this unit is compiled without contraction, which only
    // the FP64 closest-point arithmetic needs; one rounding per FMA only tightens the bound)
    const float a = fmaf(ux, ux, fmaf(uy, uy, uz * uz)), e = fmaf(vx, vx, fmaf(vy, vy, vz * vz));
    const float f = fmaf(vx, wx, fmaf(vy, wy, vz * wz)), c = fmaf(ux, wx, fmaf(uy, wy, uz * wz));
    float s = 0.f, tt = 0.f;
    if (a > 1e-20f && e > 1e-20f) {
        const float b = fmaf(ux, vx, fmaf(uy, vy, uz * vz)), den = fmaf(a, e, -b * b);
        s = den > 1e-12f * a * e ? __saturatef(__fdividef(b * f - c * e, den)) : 0.f;
        tt = __fdividef(b * s + f, e);
        if (tt < 0.f) {
            tt = 0.f;
            s = __saturatef(__fdividef(-c, a));
        } else if (tt > 1.f) {
            tt = 1.f;
            s = __saturatef(__fdividef(b - c, a));
        }
    } else if (a > 1e-20f) {
        s = __saturatef(__fdividef(-c, a));
    } else if (e > 1e-20f) {
        tt = __saturatef(__fdividef(f, e));
    }
    const float nx = fmaf(-vx, tt, fmaf(ux, s, wx)), ny = fmaf(-vy, tt, fmaf(uy, s, wy)),
                nz = fmaf(-vz, tt, fmaf(uz, s, wz));
    const float nn = fmaf(nx, nx, fmaf(ny, ny, nz * nz));
    const float err = 3e-5f * X + 1e-9f;
    DistBounds r;
    r.pad_sum = (pa + pb) * 1.000001f;
    r.far_ok = nn > 1e-14f;  // false also when not finite
    r.far = 0.f;
    if (r.far_ok) {
        const float inv = rsqrtf(nn);
        const float mx = nx * inv, my = ny * inv, mz = nz * inv;
        const float nu = fmaf(mx, ux, fmaf(my, uy, mz * uz)), nv = fmaf(mx, vx, fmaf(my, vy, mz * vz));
        const float L = fmaf(mx, wx, fmaf(my, wy, mz * wz)) + fminf(0.f, nu) - fmaxf(0.f, nv);
        r.far = L * 0.999999f - err;
    }
    return r;
}

constexpr int kBatch = 4;  // candidates per lane behind one list atomic

// Appends the flagged candidates of a warp's batch to a list of capacity cap: bit u of `keep`
// stands for this lane's candidate u.  One atomic per warp and batch.  All lanes call it.
template <typename Put>
__device__ __forceinline__ void append_batch(uint32_t keep, uint32_t* __restrict__ count, long long cap, Put put) {
    const int lane = threadIdx.x & 31;
    const uint32_t below = (1u << lane) - 1u;
    uint32_t m[kBatch], total = 0;
#pragma unroll
    for (int u = 0; u < kBatch; u++) {
        m[u] = __ballot_sync(0xffffffffu, keep >> u & 1u);
        total += __popc(m[u]);
    }
    if (total == 0) return;  // warp-uniform
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(count, total);
    base = __shfl_sync(0xffffffffu, base, 0);
#pragma unroll
    for (int u = 0; u < kBatch; u++) {
        if (keep >> u & 1u) {
            const long long at = (long long)base + __popc(m[u] & below);
            if (at < cap) put(at, u);
        }
        base += __popc(m[u]);
    }
}

// Candidate filter, once per list build: keeps the candidates of one instance whose certified
// distance lower bound at the build does not exceed the pads plus `reach` (2 skin: every point
// of a segment whose endpoints move at most skin moves at most skin, so two segments close a gap
// by at most 2 skin) and whose nodes are not connected (sim.cpp:24-39; local pairs never make
// contact, so the narrow phase of every evaluation needs no hash lookups).
// The kernel also ends the build: it clears the bins, stores the positions that later evaluations
// measure their moves from, and the end of a forced rebuild.  A build that overflowed a buffer (bins, bin
// slots, cell span, candidates) left an incomplete list: the next evaluation must build again,
// whatever the skin says, so that the overflow is raised again there (the overflow bits are per
// evaluation; a caller that enqueues several evaluations before reading sees only the last one's).
__global__ void __launch_bounds__(kBlock) k_filter(DevTopo t, PhysParams p, const float4* __restrict__ xf, float reach,
                                                   ContactBufs c) {
    if (!c.flags[1]) return;
    const long long thread = (long long)blockIdx.x * blockDim.x + threadIdx.x, threads = (long long)gridDim.x * blockDim.x;
    for (long long i = thread; i < t.N; i += threads) c.xref[i] = xf[i];
    for (long long i = thread; i < c.grid[8]; i += threads) c.bin_count[i] = 0;  // for the next build
    if (thread == 0)
        c.flags[2] = (c.flags[0] & uint32_t(kOverEntries | kOverBins | kOverSpan | kOverCandidates)) ? 1u : 0u;
    const int lane = threadIdx.x & 31;
    const uint32_t total = uint32_t(min((long long)c.counts[kCand], c.cand_cap));
    for (long long b0 = thread / 32 * 32 * kBatch; b0 < total; b0 += threads * kBatch) {
        uint2 q[kBatch];
        uint32_t keep = 0;
#pragma unroll
        for (int u = 0; u < kBatch; u++)
            if (b0 + 32 * u + lane < total) q[u] = c.cand[b0 + 32 * u + lane];
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            if (b0 + 32 * u + lane >= total) continue;
            const int2 na = shape_nodes(t, q[u].x), nb = shape_nodes(t, q[u].y);
            if (t.I > 1 && t.node_inst[na.x] != t.node_inst[nb.x]) continue;
            const DistBounds d = dist_bounds(t, p, xf, q[u].x, q[u].y);
            if (!(d.far_ok && d.far > d.pad_sum + reach) && !any_connected(t, na, nb)) keep |= 1u << u;
        }
        append_batch(keep, c.counts + kKept, c.cand_cap, [&](long long at, int u) { c.cand2[at] = q[u]; });
    }
}

// Adds v to a fixed-point sum of quantum 2^e0 (kSumLimbs signed counters of 32 bits each, which
// hold 2^31 additions): the 53-bit mantissa lands in at most three limbs, added with v's sign.
// Bits below the quantum are dropped; false when v is not finite or beyond the top limb.
__device__ __forceinline__ bool add_fixed(long long* __restrict__ sum, double v, int e0) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const int e = int(b >> 52) & 0x7ff;
    if (e == 0) return true;       // zero (or subnormal, far below any quantum in use)
    if (e == 0x7ff) return false;
    unsigned long long m = (b & 0xfffffffffffffULL) | 0x10000000000000ULL;
    int at = e - 1023 - 52 - e0;   // bit position of the mantissa's lowest bit
    if (at < 0) {
        m = at <= -64 ? 0 : m >> -at;
        at = 0;
    }
    const int limb = at >> 5, sh = at & 31;
    const unsigned long long lo = m << sh;
    const unsigned parts[3] = {unsigned(lo), unsigned(lo >> 32), sh ? unsigned(m >> (64 - sh)) : 0u};
    const bool minus = b >> 63;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (!parts[k]) continue;
        if (limb + k >= kSumLimbs) {
            ok = false;
            continue;
        }
        const long long d = minus ? -(long long)parts[k] : (long long)parts[k];
        atomicAdd(reinterpret_cast<unsigned long long*>(sum + limb + k), (unsigned long long)d);
    }
    return ok;
}

// A pair too close to tell from FP32 bounds (valid: the lane has one): the exact FP64 test and a place
// in the contact list.  All lanes of a warp call it.
__device__ __forceinline__ PairHit find_contact(const DevTopo& t, const PhysParams& p, const double4_32a* __restrict__ x,
                                                const ContactBufs& c, bool valid, uint2 q) {
    const int lane = threadIdx.x & 31;
    PairHit h;
    h.hit = false;
    if (valid) h = narrow_phase(t, p, x, q.x, q.y);
    const unsigned m = __ballot_sync(0xffffffffu, h.hit);
    if (!m) return h;  // warp-uniform
    uint32_t base = 0;
    if (lane == 0) {
        base = atomicAdd(c.counts + kContacts, uint32_t(__popc(m)));
        if ((long long)base + __popc(m) > c.contact_cap) atomicOr(c.flags, uint32_t(kOverContacts));
    }
    const long long at = (long long)__shfl_sync(0xffffffffu, base, 0) + __popc(m & ((1u << lane) - 1u));
    if (h.hit && at < c.contact_cap) {
        c.c_a[at] = q.x;
        c.c_b[at] = q.y;
    }
    return h;
}

// One end of one side of a contact: the force of the penalty (sim.cpp:163-164, addShapeGradient
// sim.cpp:23: capsule ends split the force (1 - u, u); v the side's force, u its end's share) onto the
// node's fixed-point sums; with the first end of the lower shape go the contact's energy, count and
// penetration.
__device__ __forceinline__ void add_end(const DevTopo& t, const PhysParams& p, const ContactBufs& c, uint2 q, d3 v, double u,
                                        double pen, int side, int end) {
    const uint32_t shape = side ? q.y : q.x;
    const bool capsule = shape >= uint32_t(t.N);
    if (end && !capsule) return;
    const int2 nd = shape_nodes(t, shape);
    const int node = end ? nd.y : nd.x;
    const d3 f = !capsule ? v : end ? v * u : v * (1 - u);
    NodeContact& r = c.n_sum[node];
    bool ok = add_fixed(r.f[0], f.x, c.force_e0);
    ok &= add_fixed(r.f[1], f.y, c.force_e0);
    ok &= add_fixed(r.f[2], f.z, c.force_e0);
    if (side == 0 && end == 0) {
        ok &= add_fixed(r.energy, .5 * p.contact_k * pen * pen, c.energy_e0);
        atomicMax(&r.pen, (unsigned long long)__double_as_longlong(pen));  // pen > 0
        atomicAdd(c.n_count + node, 1ULL | (1ULL << 32));
    } else {
        atomicAdd(c.n_count + node, 1ULL);
    }
    // not finite: the evaluation's energy must be, too (the gather reads the flag)
    if (!ok) atomicOr(c.n_count + node, kContactNotFinite);
}

// The whole contact by one lane.
__device__ __forceinline__ void add_contact(const DevTopo& t, const PhysParams& p, const double4_32a* __restrict__ x,
                                            const ContactBufs& c, bool valid, uint2 q) {
    const PairHit h = find_contact(t, p, x, c, valid, q);
    if (!h.hit) return;
    const double mag = p.contact_k * h.pen;
#pragma unroll
    for (int side = 0; side < 2; side++)
#pragma unroll
        for (int end = 0; end < 2; end++) add_end(t, p, c, q, h.n * (side ? -mag : mag), side ? h.t : h.s, h.pen, side, end);
}

struct FoundContact {
    d3 force;  // on the lower shape
    double s, t, pen;
    uint2 q;
};
// The filtered list's pairs in contact and their forces, every evaluation.  A warp queues the pairs
// of the evaluated instances that are not certainly apart and takes them to FP64 as soon as it has
// one for every lane, a block's warps the rest together at the end, where the ends of the contacts
// found go over all threads (the sums of one contact by one lane are a chain of 13 additions: the
// compressed 32x32x16 lattice, mixed, 118 -> 112 us a call): the closest points run with
// full warps, and a short list spreads over the SMs.  The launch, the list between them and the
// second kernel's start bounded the two kernels this was (narrow phase, then contacts).  A whole
// evaluation of the 2x4x2 specimen 47.3 -> 43.0 us on the GPU, of the compressed 32x32x16 lattice in
// mixed precision 59.6 -> 51.5.  Filtering in this kernel too took 20 us longer on the 64x64x32 lattice
// (the closest points' registers halve the warps the filter has in flight).
__global__ void __launch_bounds__(kListThreads) k_contacts(DevTopo t, PhysParams p, const double4_32a* __restrict__ x,
                                                           const float4* __restrict__ xf, ContactBufs c) {
    __shared__ uint2 queue[kListWarps][64];
    __shared__ uint32_t left[kListWarps];
    __shared__ FoundContact found[kListThreads];
    __shared__ int hits;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long thread = (long long)blockIdx.x * kListThreads + threadIdx.x, threads = (long long)gridDim.x * kListThreads;
    const uint32_t total = uint32_t(min((long long)c.counts[kKept], c.cand_cap));
    uint32_t n = 0;  // pairs in the warp's queue
    for (long long b0 = thread / 32 * 32; b0 < total; b0 += threads) {  // warp-uniform
        uint2 q = make_uint2(0, 0);
        bool close = false;
        if (b0 + lane < total) {
            q = c.cand2[b0 + lane];  // not a local pair (k_filter)
            if (t.I == 1 || t.active[t.node_inst[shape_nodes(t, q.x).x]]) {
                const DistBounds d = dist_bounds(t, p, xf, q.x, q.y);
                close = !(d.far_ok && d.far > d.pad_sum);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, close);
        if (close) queue[warp][n + __popc(m & ((1u << lane) - 1u))] = q;
        n += __popc(m);
        __syncwarp();
        if (n >= 32) {
            n -= 32;
            add_contact(t, p, x, c, true, queue[warp][n + lane]);
            __syncwarp();
        }
    }
    if (lane == 0) left[warp] = n;
    if (threadIdx.x == 0) hits = 0;
    __syncthreads();
    // the rest of all warps' queues, dense; the ends of its contacts over all threads
    int from = threadIdx.x, w = 0, all = 0;
    for (int k = 0; k < kListWarps; k++) all += left[k];
    if (all == 0) return;  // block-uniform
    if (int(threadIdx.x & ~31u) < all) {
        const bool mine = from < all;
        while (mine && from >= int(left[w])) from -= left[w++];
        const uint2 q = mine ? queue[w][from] : make_uint2(0, 0);
        const PairHit h = find_contact(t, p, x, c, mine, q);
        if (h.hit) {
            const int k = atomicAdd(&hits, 1);
            const double mag = p.contact_k * h.pen;
            found[k] = FoundContact{h.n * mag, h.s, h.t, h.pen, q};
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 4 * hits; k += kListThreads) {
        const FoundContact& f = found[k >> 2];
        const int side = k >> 1 & 1;
        add_end(t, p, c, f.q, side ? -f.force : f.force, side ? f.t : f.s, f.pen, side, k & 1);
    }
}

}  // namespace


long long pair_units(long long bins, int slots) { return bins * ((slots + kChunk - 1) / kChunk); }

// One unit of pair work per warp or so (a bin at the default cell holds about 100 shapes, each in
// about three bins), and no more blocks than the GPU holds at a time: all of it, or four of eight
// per SM when it runs beside the FP64 beam kernel (shared).  That one lives on the FP64 pipe, this
// on the integer pipe, but whichever fills the SMs' registers runs alone.  A call of the largest
// lattice (2.95 million beams): 1980 us with eight blocks an SM, 1934 with five, 1915 with four, 1927
// with three; compressed 32x32x16, where the contacts take longer than the beams: 259, 247, 243, 260;
// where no list is built or the lattice is small, no difference (eight / four: 19x15x11 81.3 / 81.3, a
// batch of 48 lattices 455 / 456).
int contact_pair_blocks(long long shapes, bool shared) {
    const long long b = shapes / 128, most = shared ? 4 * 152 / (8 / kPairWarps) : 4 * 152;
    return int(b < 1 ? 1 : (b > most ? most : b));
}

void launch_contacts(const DevTopo& t, const PhysParams& p, const EvalBufs& e, ContactBufs& c, float skin,
                     cudaStream_t s, cudaEvent_t pairs_begin, cudaEvent_t pairs_end) {
    const float grow = skin > 0.f ? skin : 0.f;
    // candidate list (only when rebuilding)
    (k_shapes<<<std::min(grid_for((long long)t.N + t.B), unsigned(c.shape_blocks)), kBlock, 0, s>>>(t, p, e.xf_lo, e.xf_hi, grow, c), note_launches(1));
    if (pairs_begin) cudaEventRecord(pairs_begin, s);
    (k_bin_pairs<<<8 / kPairWarps * c.pair_blocks, kPairThreads, 0, s>>>(t, c.grid, c.bin_count, c.bin_slots, c.counts, c.units, c.bin_items,
                                                           c.rec,
                                                c.cand_cap, c.cand, c.flags),
     note_launches(1));
    if (pairs_end) cudaEventRecord(pairs_end, s);
    (k_filter<<<kFilterBlocks, kBlock, 0, s>>>(t, p, e.xf_lo, skin > 0.f ? 2.0001f * skin : 0.f, c),  // >= 2 skin
     note_launches(1));
    // every evaluation: the list's pairs in contact and their forces
    (k_contacts<<<kListBlocks, kListThreads, 0, s>>>(t, p, e.x, e.xf_lo, c), note_launches(1));
}

}  // namespace mcg
