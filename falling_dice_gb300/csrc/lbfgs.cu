// lbfgs.cu -- device vector kernels of the L-BFGS minimizer
// (the reference's Simulator::minimize and helpers, MC/src/sim.cpp:42-46, 174-211), for every
// instance of a context at once.
//
// Vectors hold 6 entries per node in the ABI layout; all instances' nodes are stored one
// after another and every kernel runs over the solver blocks of the context (DevTopo::sblk: runs
// of a few 64-node units of one instance, at most kSolveBlocks per instance, a partition that
// depends on the instance alone).  Each instance has its own solver state (history count, ring
// head, line-search step, which operations it takes part in) in a small control array.  Dot
// products are per-block partial sums (a fixed tree), summed in order by the last of the
// instance's blocks to finish: a batch reproduces the separate runs bit for bit.
//
// The two-loop recursion (sim.cpp:184-187) takes 2 m dependent dot products over the vectors,
// each a pass of its own.  Here each loop is one pass: with q = g - sum_j alpha_j y_j substituted
// into alpha_i = rho_i <s_i, q>, the alphas solve a triangular system whose matrix are the products
// <s_i, y_j> of the history, one column of which is new per accepted pair; likewise the second
// loop's coefficients.  Three passes make a direction:
//   k_dir_dots   <s_i, g> and the newest column <s_i, y_new>; then alpha (last block);
//   k_dir_first  q = g - sum alpha_i y_i and <y_i, q>; then the second loop's coefficients;
//   k_dir_second p = clamp(lock(-(H0 q + sum c_i s_i))) and <g, p>; then the descent check.
// The same products and sums as the recursion's; measured against extended precision over the
// histories of three specimens' minimizations the direction's error is the recursion's (ratio of
// geometric means 0.99, 1.14, 0.99).
//
// What bounds a pass: latency for a small lattice (the chain of loads, the block's reduction, the
// instance's counter, the last block's totals and solve: 8 us a pass at 343 nodes), the FP64 units
// from 10^4 nodes on (81 instructions per 32 half-nodes of the second pass; 17 us a pass at 17 500
// nodes, history 10).  So the nodes are spread one 64-node block per SM while they last (one warp
// per FP64 unit, few partials for the last block to sum), a thread keeps the loads of all its
// history in flight, and the scalar solves run in the last block instead of in launches of their
// own.  Whole minimizations against one pass per dot product: 6x6x6 cubic (18 rounds) 3.3 -> 1.6 ms,
// 32x32x16 cubic+BCC mixed (14 rounds) 3.4 -> 2.6 ms, a load/unload run of 6 lattices 6.4 -> 4.5 ms.
// With 64 blocks an instance 32x32x16 takes 98 us a direction, with 152 51; with 304 55 (the last
// block's totals).
#include "common.cuh"
#include "minimize.h"

namespace mcg {

namespace {

constexpr int kThreads = 256;            // one half-node (3 DOFs) per thread at a time
constexpr int kUnit = 64;                // nodes of a solver block of a small instance: a warp per FP64 unit
constexpr int kWarps = kThreads / 32;
constexpr int kDotPairs = 4;             // history pairs a block of the first pass takes
constexpr int kSmallHistory = 16;        // histories whose products are solved from shared memory
constexpr int kRegHistory = 12;          // histories whose vectors a thread holds in registers (the default is 10)

// An instance's control record with its history state (pairs held, oldest slot), which
// lives on the device: the solver kernels update it themselves.
__device__ __forceinline__ SolveCtl load_ctl(const SolveCtl* __restrict__ ctl, const int2* __restrict__ hist, int inst) {
    SolveCtl c = ctl[inst];
    const int2 h = hist[inst];
    c.m = h.x;
    c.head = h.y;
    return c;
}
// Slot of the h-th oldest history pair of an instance.
__device__ __forceinline__ int ring_slot(const SolveCtl& c, int H, int h) {
    const int s = c.head + h;
    return s < H ? s : s - H;
}

__device__ __forceinline__ d3 ld3(const double* v) { return d3{v[0], v[1], v[2]}; }
__device__ __forceinline__ void st3(double* v, d3 a) {
    v[0] = a.x;
    v[1] = a.y;
    v[2] = a.z;
}

// Block partial of up to four values into q[k * stride] (thread k writes value k).
template <int NV>
__device__ __forceinline__ void block_part(double a, double b, double c, double d, double* q, size_t stride,
                                           double (*sm)[kWarps]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (NV <= 2) {
        const double v = warp_sum2(a, b);
        if ((lane & 15) == 0) sm[lane >> 4][warp] = v;
    } else {
        const double v = warp_sum4(a, b, c, d);
        if ((lane & 7) == 0) sm[lane >> 3][warp] = v;
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        double s = sm[threadIdx.x][0];
        for (int w = 1; w < kWarps; w++) s += sm[threadIdx.x][w];
        q[threadIdx.x * stride] = s;
    }
    __syncthreads();
}

// Totals of nv values' partials over the instance's nb (<= kSolveBlocks) blocks, value k at
// part[k * stride + first ...], into out[k]; four values a warp at a time.
__device__ __forceinline__ void part_totals(const double* part, size_t stride, int first, int nb, int nv, double* out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k0 = 4 * warp; k0 < nv; k0 += 4 * kWarps) {
        double v[4] = {0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (k0 + j < nv) {
                const double* p = part + (k0 + j) * stride + first;
#pragma unroll
                for (int b = 0; b < kSolveBlocks; b += 32)
                    if (b + lane < nb) v[j] += __ldcg(p + b + lane);
            }
        const double s = warp_sum4(v[0], v[1], v[2], v[3]);
        if ((lane & 7) == 0 && k0 + (lane >> 3) < nv) out[k0 + (lane >> 3)] = s;
    }
    __syncthreads();
}

// ---- direction, first pass ------------------------------------------------------------------
// Block (b, k): the partials of <s, g> and <s, y_new> for history pairs 4 k ... 4 k + 3; the last
// block of the instance stores the newest column of the products and solves the first loop's
// alphas, newest to oldest: alpha_i = rho_i (<s_i, g> - sum_{j > i} alpha_j <s_i, y_j>).
__global__ void __launch_bounds__(kThreads) k_dir_dots(DevTopo t, const SolveCtl* __restrict__ ctl, LbfgsBufs v, MzStatus* st) {
    if (st && threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0) stage_mark(st, &st->t_post);
    __shared__ double sm[4][kWarps];
    __shared__ double val[2 * 64], R[kSmallHistory][kSmallHistory + 1];
    const int H = v.H;
    const int4 q = t.sblk[blockIdx.x];
    const int inst = q.z, h0 = kDotPairs * blockIdx.y;
    const SolveCtl c = load_ctl(ctl, v.hist, inst);
    const int m = c.m;
    if (!(c.flags & kOpDirection) || h0 >= m) return;  // block-uniform (none when m == 0)
    const int newest = ring_slot(c, H, m - 1);
    const double* s[kDotPairs];
#pragma unroll
    for (int k = 0; k < kDotPairs; k++) s[k] = v.S + v.stride * ring_slot(c, H, min(h0 + k, m - 1)) + 6 * size_t(q.x);
    const double* y = v.Y + v.stride * newest + 6 * size_t(q.x);
    const double* g = v.g + 6 * size_t(q.x);
    double d[2 * kDotPairs] = {};
    for (int i = threadIdx.x; i < 2 * q.y; i += kThreads) {
        const d3 b = ld3(g + 3 * i), e = ld3(y + 3 * i);
        d3 a[kDotPairs];
#pragma unroll
        for (int k = 0; k < kDotPairs; k++)
            if (h0 + k < m) a[k] = ld3(s[k] + 3 * i);
#pragma unroll
        for (int k = 0; k < kDotPairs; k++)
            if (h0 + k < m) {
                d[2 * k] = fma(a[k].z, b.z, fma(a[k].y, b.y, fma(a[k].x, b.x, d[2 * k])));
                d[2 * k + 1] = fma(a[k].z, e.z, fma(a[k].y, e.y, fma(a[k].x, e.x, d[2 * k + 1])));
            }
    }
#pragma unroll
    for (int k = 0; k < 2 * kDotPairs; k += 4)
        if (2 * h0 + k < 2 * m)
            block_part<4>(d[k], d[k + 1], d[k + 2], d[k + 3], v.part + size_t(2 * h0 + k) * t.n_sblk + blockIdx.x, t.n_sblk, sm);
    const int2 r = t.srange[inst];
    const int nb = r.y - r.x;
    if (!last_block(v.done + 4 * inst, unsigned(nb * ((m + kDotPairs - 1) / kDotPairs)))) return;
    part_totals(v.part, t.n_sblk, r.x, nb, 2 * m, val);
    double* gram = v.gram + size_t(inst) * H * H;  // <s_i, y_j> at [slot i][slot j], i not newer than j
    const bool small = m <= kSmallHistory;
    for (int i = threadIdx.x; i < m; i += kThreads) gram[ring_slot(c, H, i) * H + newest] = val[2 * i + 1];
    if (small)
        for (int k = threadIdx.x; k < m * m; k += kThreads) {
            const int i = k / m, j = k - i * m;
            if (i <= j) R[i][j] = j == m - 1 ? val[2 * i + 1] : gram[ring_slot(c, H, i) * H + ring_slot(c, H, j)];
        }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x, nu = m > 32 ? 2 : 1;
    const double* rho = v.rho + size_t(inst) * H;
    double a[2], rh[2];  // history pairs lane and lane + 32
    for (int u = 0; u < 2; u++) {
        const int i = lane + 32 * u;
        a[u] = i < m ? val[2 * i] : 0;
        rh[u] = i < m ? rho[ring_slot(c, H, i)] : 0;
    }
    for (int i = m - 1; i >= 0; i--) {
        const double al = __shfl_sync(0xffffffffu, i < 32 ? rh[0] * a[0] : rh[1] * a[1], i & 31);
        if (lane == (i & 31)) v.alpha[size_t(inst) * H + i] = al;
        for (int u = 0; u < nu; u++) {
            const int j = lane + 32 * u;
            if (j >= i) continue;
            const double rji = small ? R[j][i] : i == m - 1 ? val[2 * j + 1] : gram[ring_slot(c, H, j) * H + ring_slot(c, H, i)];
            a[u] = fma(-al, rji, a[u]);
        }
    }
}

// H0 of the direction: k_accept's for the newest pair, 0.1 without history (sim.cpp:186).
__device__ __forceinline__ double initial_scale(const LbfgsBufs& v, int inst, int m) { return m > 0 ? v.h0[inst] : .10; }

// ---- direction, second pass -----------------------------------------------------------------
// q = g - sum alpha_i y_i (newest first, into p) and the partials of <y_i, q>; the last block of
// the instance solves the second loop's coefficients, oldest to newest:
// c_i = alpha_i - rho_i (H0 <y_i, q> + sum_{j < i} c_j <s_j, y_i>).
__global__ void __launch_bounds__(kThreads) k_dir_first(DevTopo t, const SolveCtl* __restrict__ ctl, LbfgsBufs v) {
    __shared__ double sm[4][kWarps];
    __shared__ double al[64], val[64], R[kSmallHistory][kSmallHistory + 1];
    const int H = v.H;
    const int4 q = t.sblk[blockIdx.x];
    const int inst = q.z;
    const SolveCtl c = load_ctl(ctl, v.hist, inst);
    if (!(c.flags & kOpDirection)) return;
    const int m = c.m;
    for (int i = threadIdx.x; i < m; i += kThreads) al[i] = v.alpha[size_t(inst) * H + i];
    __syncthreads();
    double* p = v.p + 6 * size_t(q.x);
    const double* g = v.g + 6 * size_t(q.x);
    if (m <= kRegHistory) {
        // every load of the thread's half-node in flight at once, the y_i used for both sums
        const double* Y[kRegHistory];
#pragma unroll
        for (int h = 0; h < kRegHistory; h++) Y[h] = v.Y + v.stride * (h < m ? ring_slot(c, H, h) : 0) + 6 * size_t(q.x);
        double d[kRegHistory] = {};
        for (int i = threadIdx.x; i < 2 * q.y; i += kThreads) {
            d3 a = ld3(g + 3 * i), y[kRegHistory];
#pragma unroll
            for (int h = 0; h < kRegHistory; h++)
                if (h < m) y[h] = ld3(Y[h] + 3 * i);
#pragma unroll
            for (int h = kRegHistory - 1; h >= 0; h--)
                if (h < m) a = fmadd(y[h], -al[h], a);
            st3(p + 3 * i, a);
#pragma unroll
            for (int h = 0; h < kRegHistory; h++)
                if (h < m) d[h] = fma(a.z, y[h].z, fma(a.y, y[h].y, fma(a.x, y[h].x, d[h])));
        }
        if (m == 0) return;  // block-uniform: no history, p = g
        __shared__ double wsum[kRegHistory][kWarps];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int h = 0; h < kRegHistory; h += 4)
            if (h < m) {
                const double s4 = warp_sum4(d[h], d[h + 1], d[h + 2], d[h + 3]);
                if ((lane & 7) == 0) wsum[h + (lane >> 3)][warp] = s4;
            }
        __syncthreads();
        for (int h = threadIdx.x; h < m; h += kThreads) {
            double s = wsum[h][0];
            for (int w = 1; w < kWarps; w++) s += wsum[h][w];
            v.part[size_t(h) * t.n_sblk + blockIdx.x] = s;
        }
    } else {
        for (int i = threadIdx.x; i < 2 * q.y; i += kThreads) {
            d3 a = ld3(g + 3 * i);
            for (int h = m - 1; h >= 0; h--)
                a = fmadd(ld3(v.Y + v.stride * ring_slot(c, H, h) + 6 * size_t(q.x) + 3 * i), -al[h], a);
            st3(p + 3 * i, a);
        }
        for (int h = 0; h < m; h += 4) {
            double d[4] = {0, 0, 0, 0};
            for (int i = threadIdx.x; i < 2 * q.y; i += kThreads) {
                const d3 a = ld3(p + 3 * i);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (h + k >= m) break;
                    const d3 y = ld3(v.Y + v.stride * ring_slot(c, H, h + k) + 6 * size_t(q.x) + 3 * i);
                    d[k] = fma(a.z, y.z, fma(a.y, y.y, fma(a.x, y.x, d[k])));
                }
            }
            block_part<4>(d[0], d[1], d[2], d[3], v.part + size_t(h) * t.n_sblk + blockIdx.x, t.n_sblk, sm);
        }
    }
    const int2 r = t.srange[inst];
    const int nb = r.y - r.x;
    if (!last_block(v.done + 4 * inst + 1, unsigned(nb))) return;
    part_totals(v.part, t.n_sblk, r.x, nb, m, val);
    const double* gram = v.gram + size_t(inst) * H * H;
    const bool small = m <= kSmallHistory;
    if (small)
        for (int k = threadIdx.x; k < m * m; k += kThreads) {
            const int i = k / m, j = k - i * m;
            if (i < j) R[i][j] = gram[ring_slot(c, H, i) * H + ring_slot(c, H, j)];
        }
    __syncthreads();
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x, nu = m > 32 ? 2 : 1;
    const double* rho = v.rho + size_t(inst) * H;
    const double h0 = initial_scale(v, inst, m);
    double a[2], rh[2], u0[2];
    for (int u = 0; u < 2; u++) {
        const int i = lane + 32 * u;
        a[u] = i < m ? h0 * val[i] : 0;
        rh[u] = i < m ? rho[ring_slot(c, H, i)] : 0;
        u0[u] = i < m ? al[i] : 0;
    }
    for (int i = 0; i < m; i++) {
        const double co = __shfl_sync(0xffffffffu, i < 32 ? fma(-rh[0], a[0], u0[0]) : fma(-rh[1], a[1], u0[1]), i & 31);
        if (lane == (i & 31)) v.coef[size_t(inst) * H + i] = co;
        for (int u = 0; u < nu; u++) {
            const int j = lane + 32 * u;
            if (j <= i || j >= m) continue;
            const double rij = small ? R[i][j] : gram[ring_slot(c, H, i) * H + ring_slot(c, H, j)];
            a[u] = fma(co, rij, a[u]);
        }
    }
}

// p = clamp(lock(v)) of one half of a node (translations or rotations; sim.cpp:188-190, 46).
__device__ __forceinline__ d3 clamp_half(d3 a, const uint8_t* lk, double limit) {
    if (lk[0]) a.x = 0;
    if (lk[1]) a.y = 0;
    if (lk[2]) a.z = 0;
    const double l2 = fdot(a, a);
    // the length is taken only where its square can exceed the limit's
    if (!(limit >= 0 && l2 <= limit * limit * (1 - 0x1p-40))) {
        const double l = sqrt(l2);
        if (l > limit) a = a * (limit / l);
    }
    return a;
}

// p = clamp(lock(-src)) over the run of half-nodes and this thread's part of <g, p>.
__device__ __forceinline__ double steepest_part(const DevTopo& t, const double* g, double* p, int first, int halves,
                                                double mt, double mr) {
    double d = 0;
    for (int i = threadIdx.x; i < halves; i += kThreads) {
        const size_t o = 6 * size_t(first) + 3 * size_t(i);
        const d3 b = ld3(g + o), a = clamp_half(-b, t.locked + o, (i & 1) ? mr : mt);
        st3(p + o, a);
        d = fma(a.z, b.z, fma(a.y, b.y, fma(a.x, b.x, d)));
    }
    return d;
}

// ---- direction, third pass ------------------------------------------------------------------
// p = clamp(lock(-(H0 q + sum c_i s_i))) and the partial of <g, p>; the last block of the instance
// sums dg.  Not a descent direction (sim.cpp:191): that block takes steepest descent instead and
// clears the history.  Instances of the steepest-descent retry (kOpSteepest, sim.cpp:193-196) take
// p = clamp(lock(-g)) with the history cleared here as well.
__global__ void __launch_bounds__(kThreads) k_dir_second(DevTopo t, const SolveCtl* __restrict__ ctl, LbfgsBufs v) {
    __shared__ double sm[4][kWarps];
    __shared__ double co[64], total[1];
    const int H = v.H;
    const int4 q = t.sblk[blockIdx.x];
    const int inst = q.z;
    const SolveCtl c = load_ctl(ctl, v.hist, inst);
    if (!(c.flags & (kOpDirection | kOpSteepest))) return;
    const bool steepest = c.flags & kOpSteepest;
    const int m = c.m;
    for (int i = threadIdx.x; i < m; i += kThreads) co[i] = v.coef[size_t(inst) * H + i];
    const double h0 = initial_scale(v, inst, m);
    __syncthreads();
    double d = steepest ? steepest_part(t, v.g, v.p, q.x, 2 * q.y, v.mt, v.mr) : 0;
    for (int i = steepest ? 2 * q.y : threadIdx.x; i < 2 * q.y; i += kThreads) {
        const size_t o = 6 * size_t(q.x) + 3 * size_t(i);
        d3 a = ld3(v.p + o);
        if (m <= kRegHistory) {  // every load in flight at once
            d3 sv[kRegHistory];
#pragma unroll
            for (int h = 0; h < kRegHistory; h++)
                if (h < m) sv[h] = ld3(v.S + v.stride * ring_slot(c, H, h) + o);
            a = a * h0;
#pragma unroll
            for (int h = 0; h < kRegHistory; h++)
                if (h < m) a = fmadd(sv[h], co[h], a);
        } else {
            a = a * h0;
            for (int h = 0; h < m; h++) a = fmadd(ld3(v.S + v.stride * ring_slot(c, H, h) + o), co[h], a);
        }
        a = clamp_half(-a, t.locked + o, (i & 1) ? v.mr : v.mt);
        st3(v.p + o, a);
        const d3 b = ld3(v.g + o);
        d = fma(a.z, b.z, fma(a.y, b.y, fma(a.x, b.x, d)));
    }
    block_part<1>(d, 0, 0, 0, v.part + blockIdx.x, t.n_sblk, sm);
    const int2 r = t.srange[inst];
    const int nb = r.y - r.x;
    if (!last_block(v.done + 4 * inst + 2, unsigned(nb))) return;
    part_totals(v.part, t.n_sblk, r.x, nb, 1, total);
    const double dg = total[0];
    if (steepest || dg < 0) {
        if (threadIdx.x == 0) {
            v.dg[inst] = dg;
            if (steepest) v.hist[inst].x = 0;
        }
        return;
    }
    const double e = steepest_part(t, v.g, v.p, t.sblk[r.x].x, 2 * t.inst_n[inst], v.mt, v.mr);
    block_part<1>(e, 0, 0, 0, total, 1, sm);
    if (threadIdx.x == 0) {
        v.dg[inst] = total[0];
        v.hist[inst].x = 0;
    }
}

// ---- vectors around an evaluation ------------------------------------------------------------
// Per node, in this order for each instance's flags: z = 0 (kOpZero), z = best (kOpRestore),
// best = z (kOpKeepBest), zeval = z + step p with locked entries 0 (kOpCandidate, sim.cpp:179)
// or zeval = z (kOpEvalAtZ), zfinal = z (kOpFinal); a new minimization starts with an empty
// history (kOpResetHistory).
// In the device-resident loop (d.mins) the operations follow from the instance's minimizer, and
// its first block writes what the evaluation reads: active and trial masks, platen height, and the
// request for a new candidate list when the instance joins (its shapes have to be in it).
__global__ void __launch_bounds__(kEvalBlock) k_prepare(DevTopo t, const SolveCtl* __restrict__ ctl, LbfgsBufs v, MzDev d) {
    const MapPos mp = map_pos(t.eblk);
    const bool first = threadIdx.x == 0 && int(blockIdx.x) == t.erange[mp.inst].x;
    SolveCtl c{};
    if (d.mins) {
        if (threadIdx.x == 0 && blockIdx.x == 0) stage_mark(d.status, &d.status->t_dir);
        bool trials = false;
        c.flags = mz_stage_eval(d.mins[mp.inst], c.step, trials);
        if (first) {
            const uint8_t a = c.flags ? 1 : 0;
            if (a && !d.active[mp.inst] && d.contact_flags) d.contact_flags[2] = 1u;
            d.active[mp.inst] = a;
            d.trial_inst[mp.inst] = trials ? 1 : 0;
            if (a) d.tops[mp.inst] = d.mins[mp.inst].top;
        }
    } else {
        c = ctl[mp.inst];
    }
    if ((c.flags & kOpResetHistory) && first) v.hist[mp.inst] = make_int2(0, 0);
    if (!mp.valid || !(c.flags & (kOpZero | kOpRestore | kOpKeepBest | kOpCandidate | kOpEvalAtZ | kOpFinal))) return;
    const size_t o = 6 * size_t(mp.i);
    double a[6];
#pragma unroll
    for (int k = 0; k < 6; k++) {
        a[k] = (c.flags & kOpZero) ? 0.0 : v.z[o + k];
        if (c.flags & kOpRestore) a[k] = v.best[o + k];
    }
#pragma unroll
    for (int k = 0; k < 6; k++) {
        if (c.flags & (kOpZero | kOpRestore)) v.z[o + k] = a[k];
        if (c.flags & kOpKeepBest) v.best[o + k] = a[k];
        if (c.flags & kOpEvalAtZ) v.zeval[o + k] = a[k];
        if (c.flags & kOpFinal) v.zfinal[o + k] = a[k];
    }
    if (!(c.flags & kOpCandidate)) return;
    double p[6];
#pragma unroll
    for (int k = 0; k < 6; k++) p[k] = v.p[o + k];
#pragma unroll
    for (int k = 0; k < 6; k++) v.zeval[o + k] = t.locked[o + k] ? 0.0 : fma(c.step, p[k], a[k]);
}

// After an evaluation: g = geval for the instances that evaluated at z (kOpTakeGrad), and
// for accepted trials (kOpAccept, sim.cpp:205-206) s = zeval - z, y = geval - g into the
// next history slot (kOpPair), the partials of <s, y>, <s, s>, <y, y>, then z = zeval,
// g = geval; best = z afterwards when kOpKeepBestAfter.  The last block of the instance sums the
// products and keeps the pair when s.y > 1e-12 sqrt(max(1e-30, s.s y.y)) (rho = 1 / s.y in its
// slot), else clears the history.
__global__ void __launch_bounds__(kThreads) k_accept(DevTopo t, const SolveCtl* __restrict__ ctl, LbfgsBufs v) {
    __shared__ double sm[4][kWarps];
    __shared__ double total[4];
    const int H = v.H;
    const int4 q = t.sblk[blockIdx.x];
    const int inst = q.z;
    const SolveCtl c = load_ctl(ctl, v.hist, inst);
    if (!(c.flags & (kOpTakeGrad | kOpAccept))) return;
    if (c.flags & kOpTakeGrad) {
        for (int i = threadIdx.x; i < 6 * q.y; i += kThreads) v.g[6 * size_t(q.x) + i] = v.geval[6 * size_t(q.x) + i];
        return;
    }
    const int target = c.m < H ? (c.head + c.m) % H : c.head;
    double sy = 0, ss = 0, yy = 0;
    for (int i = threadIdx.x; i < 2 * q.y; i += kThreads) {
        const size_t o = 6 * size_t(q.x) + 3 * size_t(i);
        const d3 ze = ld3(v.zeval + o), ge = ld3(v.geval + o);
        const d3 a = ze - ld3(v.z + o), b = ge - ld3(v.g + o);
        if (c.flags & kOpPair) {
            st3(v.S + v.stride * target + o, a);
            st3(v.Y + v.stride * target + o, b);
        }
        sy = fma(a.z, b.z, fma(a.y, b.y, fma(a.x, b.x, sy)));
        ss = fma(a.z, a.z, fma(a.y, a.y, fma(a.x, a.x, ss)));
        yy = fma(b.z, b.z, fma(b.y, b.y, fma(b.x, b.x, yy)));
        st3(v.z + o, ze);
        st3(v.g + o, ge);
        if (c.flags & kOpKeepBestAfter) st3(v.best + o, ze);
    }
    block_part<3>(sy, ss, yy, 0, v.part + blockIdx.x, t.n_sblk, sm);
    const int2 r = t.srange[inst];
    if (!last_block(v.done + 4 * inst + 3, unsigned(r.y - r.x))) return;
    part_totals(v.part, t.n_sblk, r.x, r.y - r.x, 3, total);
    if (threadIdx.x == 32 && (c.flags & kOpPair))  // sim.cpp:186
        v.h0[inst] = total[0] > 1e-20 && total[2] > 1e-20 ? clampd(total[0] / total[2], 1e-7, 1e4) : .10;
    if (threadIdx.x != 0 || !(c.flags & kOpPair)) return;
    int2 h = v.hist[inst];
    if (total[0] > 1e-12 * sqrt(fmax(1e-30, total[1] * total[2]))) {
        v.rho[size_t(inst) * H + target] = 1 / total[0];
        if (h.x == H) h.y = (h.y + 1) % H;
        else h.x++;
    } else {
        h.x = 0;
    }
    v.hist[inst] = h;
}

}  // namespace

size_t lbfgs_part_doubles(int n_sblk, int H) { return size_t(2 * H + 4) * size_t(n_sblk) + 8; }

// Nodes per solver block of an instance of n nodes: one unit while that makes at most kSolveBlocks
// blocks, else runs that keep every thread busy.
int solve_block_nodes(int n) {
    if (n <= kUnit * kSolveBlocks) return kUnit;
    constexpr int step = kThreads / 2;
    const int steps = (n + step - 1) / step;
    return step * ((steps + kSolveBlocks - 1) / kSolveBlocks);
}

void bl_direction(const DevTopo& t, const SolveCtl* ctl, const LbfgsBufs& v, cudaStream_t s, MzStatus* st) {
    (k_dir_dots<<<dim3(unsigned(t.n_sblk), unsigned((v.H + kDotPairs - 1) / kDotPairs)), kThreads, 0, s>>>(t, ctl, v, st),
     note_launches(1));
    (k_dir_first<<<t.n_sblk, kThreads, 0, s>>>(t, ctl, v), note_launches(1));
    (k_dir_second<<<t.n_sblk, kThreads, 0, s>>>(t, ctl, v), note_launches(1));
}

void bl_prepare(const DevTopo& t, const SolveCtl* ctl, const LbfgsBufs& v, cudaStream_t s, const MzDev* d) {
    (k_prepare<<<t.n_eblk, kEvalBlock, 0, s>>>(t, ctl, v, d ? *d : MzDev{}), note_launches(1));
}

void bl_accept(const DevTopo& t, const SolveCtl* ctl, const LbfgsBufs& v, cudaStream_t s) {
    (k_accept<<<t.n_sblk, kThreads, 0, s>>>(t, ctl, v), note_launches(1));
}

}  // namespace mcg
