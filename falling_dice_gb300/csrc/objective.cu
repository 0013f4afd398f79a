// objective.cu -- FP64 kernels of the energy/gradient evaluation
// (the reference's Simulator::state + objective, MC/src/sim.cpp:136-172).
//
// Compiled without contraction: fused multiply-adds are written out where they are meant, so
// that a kernel's occupancy variants round identically.
//
//   k_state    per node: z -> current position; block partial sums of x
//   k_rotations per node: z -> current orientation
//   k_center   per instance: mean position for the centering term; the contact grid
//   k_beams    per beam: axial/shear/bending/torsion energy with return mapping,
//              the two end 6-vectors of its gradient, optional trial state
//   k_gather   per node: deterministic CSR sum of the incident beams' end vectors in
//              ascending beam order, gravity, centering, the node's self-contact sums,
//              platen contact; packs, scales and locks the 6-DOF gradient
//   k_finalize fixed-order totals, diagnostics, non-finite guard
#include "common.cuh"
#include "kernels.h"

namespace mcg {

static_assert(kMapBlock == kBlock, "the mixed form's beam blocks are launched with kBlock threads");

// ---- node state: MC/src/sim.cpp:136 -------------------------------------------------------
// Positions, their FP32 bounds and block partial sums and extrema: what the contact branch of an
// evaluation waits for.  Conversions and maxima on the integer pipe; 128-node blocks.
__global__ void __launch_bounds__(kEvalBlock) k_state(DevTopo t, PhysParams p, const double* __restrict__ z,
                                                      const double* __restrict__ bx, double4_32a* __restrict__ x4,
                                                      float4* __restrict__ xf_lo, float4* __restrict__ xf_hi,
                                                      double* __restrict__ part, BuildArgs build) {
    __shared__ StateParts sm;
    const MapPos mp = map_pos(t.eblk);
    if (!t.active[mp.inst]) return;  // block-uniform
    const int i = mp.i;
    double acc[3] = {0, 0, 0};
    StateBounds bounds;
    bool moved = false;
    if (mp.valid) {
        const double2* z2 = reinterpret_cast<const double2*>(z + 6 * size_t(i));
        const double2 za = z2[0], zb = z2[1];
        const uint8_t* li = t.locked + 6 * size_t(i);
        const double tr[3] = {li[0] ? 0.0 : za.x, li[1] ? 0.0 : za.y, li[2] ? 0.0 : zb.x};
        // x = base + s t, rounded exactly as the reference (no fused multiply-add), so that
        // positions -- and with them the contact pair set -- are bit-identical.
        const double ts = p.translation_scale;
        const double xx = __dadd_rn(bx[3 * size_t(i)], __dmul_rn(ts, tr[0]));
        const double xy = __dadd_rn(bx[3 * size_t(i) + 1], __dmul_rn(ts, tr[1]));
        const double xz = __dadd_rn(bx[3 * size_t(i) + 2], __dmul_rn(ts, tr[2]));
        x4[i] = make_double4_32a(xx, xy, xz, 0.0);
        float4 lo, hi;
        bounds.take(xx, xy, xz, t.off[mp.inst], lo, hi);
        xf_lo[i] = lo;
        xf_hi[i] = hi;
        if (build.flags && build.skin > 0.f) moved = moved_beyond(build.skin, lo, hi, build.xref[i]);
        acc[0] = xx; acc[1] = xy; acc[2] = xz;
    }
    if (build.flags) ask_build(build, moved);
    state_block_parts(acc, bounds, sm, part + 9 * size_t(blockIdx.x));
}

// Orientations R = exp(r) R_base and their fixed-point records, beside the contact branch.  Bound
// by the FP64 pipe like the beam kernel: rotations up to one radian by polynomials (larger ones by
// the general exponential), the quaternion normalized by one step when its norm is one but for
// rounding, the matrix on the integer pipe.  One kernel with the positions held the contact branch
// of a small lattice back (2x4x2 specimen: 68.5 us a call, split 63.7).
__global__ void __launch_bounds__(kEvalBlock) k_rotations(DevTopo t, const double* __restrict__ z, const double* __restrict__ br,
                                                          double4_32a* __restrict__ R4, double4_32a* __restrict__ M4) {
    const MapPos mp = map_pos(t.eblk);
    if (!t.active[mp.inst] || !mp.valid) return;
    const int i = mp.i;
    const double2* z2 = reinterpret_cast<const double2*>(z + 6 * size_t(i));
    const double2 zb = z2[1], zc = z2[2];
    const uint8_t* li = t.locked + 6 * size_t(i);
    const d3 rv{li[3] ? 0.0 : zb.y, li[4] ? 0.0 : zc.x, li[5] ? 0.0 : zc.y};
    const double4_32a b4 = reinterpret_cast<const double4_32a*>(br)[i];
    const double r2 = fdot(rv, rv);
    const q4 e = unsigned(__double2hiint(r2)) < 0x3ff00000u ? exp_map_small(rv, r2) : exp_map(rv);
    const q4 R = qnorm_near(fqmul(e, q4{b4.x, b4.y, b4.z, b4.w}));
    R4[i] = make_double4_32a(R.w, R.x, R.y, R.z);
    store_rotation(R, M4 + 4 * size_t(i));
}

// The grid of a rebuilt candidate list: origin, extent and bin numbering from the node bounding
// box ext = (min x, y, z, max x, y, z), by a whole block (thread d the axis d: the divisions are
// the cost).  grid[]: 0-2 origin cell, 3-5 dims, 6 mode (0 Morton, 1 row-major), 7 valid, 8 number
// of bins, 9 bins needed, 10-15 box quantization.
__device__ void grid_params(const BuildArgs& b, const double* ext) {
    __shared__ long long dims[3];
    __shared__ int good[3];
    const int d = threadIdx.x;
    if (d < 3) {
        const double lo = floor((ext[d] - b.pad) / b.cell) - 1.0;
        const double hi = floor((ext[3 + d] + b.pad) / b.cell) + 1.0;
        const bool ok = isfinite(lo) && isfinite(hi) && fabs(lo) <= 1e9 && fabs(hi) <= 1e9;
        const long long l = ok ? (long long)lo : 0, dim = ok ? (long long)hi - l + 1 : 1;
        good[d] = ok;
        dims[d] = dim;
        b.grid[d] = int(l);
        b.grid[3 + d] = int(dim);
        b.grid[10 + d] = __float_as_int(float(double(kBoxQuanta) / (double(dim) * b.cell)));
        b.grid[13 + d] = __float_as_int(float(double(l) * b.cell));
    }
    __syncthreads();
    if (d != 0) return;
    bool ok = good[0] && good[1] && good[2];
    int bits = 0;
    for (int k = 0; k < 3; k++)
        if (dims[k] > 1) bits = max(bits, 64 - __clzll(dims[k] - 1));
    const double dense = double(dims[0]) * double(dims[1]) * double(dims[2]);
    long long nb = dense < 1e18 ? dims[0] * dims[1] * dims[2] : 1LL << 60;
    int mode = 1;
    if (bits <= 10 && (1LL << (3 * bits)) <= b.bin_cap && (1LL << (3 * bits)) <= 4 * nb) {
        mode = 0;
        nb = 1LL << (3 * bits);
    }
    b.grid[9] = int(nb < (1LL << 30) ? nb : (1LL << 30));
    if (ok && nb > b.bin_cap) {  // the host enlarges the bins or coarsens the cells
        atomicOr(b.flags, uint32_t(kOverBins));
        ok = false;
    }
    b.grid[6] = mode;
    b.grid[7] = ok ? 1 : 0;
    b.grid[8] = ok ? int(nb) : 0;
}

// Mean position of each instance's nodes (MC/src/sim.cpp:143) and bounding boxes from the
// k_state partials: block i < I writes instance i's cen[9i..9i+8] (mean, minimum, maximum) and
// its centering force on each node (sim.cpp:143); block I the minimum and maximum over all
// instances at cen[9I + 3..8], and it decides whether this evaluation rebuilds the candidate
// list: every kernel of the build returns at once when it does not.
__global__ void __launch_bounds__(kBlock) k_center(DevTopo t, double centering, const double* __restrict__ part,
                                                   double* __restrict__ cen, double* __restrict__ cforce,
                                                   double* __restrict__ tops, const double* __restrict__ tops_host,
                                                   BuildArgs build) {
    __shared__ double sm[6 * kBlock];
    __shared__ double ext[6];
    __shared__ int rebuild;
    const int inst = blockIdx.x;
    int k0 = 0, k1 = t.n_eblk;
    if (inst < t.I) {
        const int2 r = t.erange[inst];
        k0 = r.x;
        k1 = r.y;
    }
    double acc[3] = {0, 0, 0};
    const long long lowest = (long long)0x8000000000000000ULL;
    long long mx[6] = {lowest, lowest, lowest, lowest, lowest, lowest};  // maxima on the integer pipe
#pragma unroll 4
    for (int k = k0 + int(threadIdx.x); k < k1; k += blockDim.x) {
        const double* q = part + 9 * size_t(k);
        if (inst < t.I) {
            acc[0] += q[0]; acc[1] += q[1]; acc[2] += q[2];
        }
#pragma unroll
        for (int j = 0; j < 6; j++) mx[j] = max(mx[j], order_key(q[3 + j]));
    }
    if (inst < t.I) block_sum_t<3>(acc, sm);
    long long* smx = reinterpret_cast<long long*>(sm);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < 6; j++) {
        const long long m = warp_max_key(mx[j]);
        if (lane == 0) smx[j * (kBlock / 32) + warp] = m;
    }
    __syncthreads();
    double* c = cen + 9 * size_t(inst);
    if (threadIdx.x < 6) {
        const int j = threadIdx.x;
        long long m = smx[j * (kBlock / 32)];
        for (int w = 1; w < kBlock / 32; w++) m = max(m, smx[j * (kBlock / 32) + w]);
        const double v = order_value(m);
        ext[j] = j < 3 ? -v : v;
        c[3 + j] = ext[j];
    }
    if (inst < t.I) {
        if (threadIdx.x == 32 && tops_host) tops[inst] = tops_host[inst];
        if (threadIdx.x == 0) {
            const double n = double(t.inst_n[inst]), inv = 1.0 / n;
            c[0] = acc[0] * inv; c[1] = acc[1] * inv; c[2] = acc[2] * inv;
            cforce[2 * inst] = centering * c[0] / n;
            cforce[2 * inst + 1] = centering * c[2] / n;
        }
        return;
    }
    if (!build.flags) return;
    if (threadIdx.x == 0) {
        rebuild = build.flags[1] || build.flags[2] || !(build.skin > 0.f);
        build.counts[kContacts] = 0;
        if (rebuild) {
            build.flags[1] = 1;
            build.flags[3] = 0;  // the pair pass's bin cursor
            build.flags[4]++;    // builds since the buffers were allocated
            for (int k : {int(kCand), int(kKept), int(kEntries), int(kLargestBin), int(kOccupied), int(kUnits)}) build.counts[k] = 0;
        }
    }
    __syncthreads();
    if (rebuild) grid_params(build, ext);
}

__device__ __forceinline__ d3 ldx(const double4_32a* x, int i) {
    const double4_32a v = x[i];
    return d3{v.x, v.y, v.z};
}
// ---- constitutive return maps: MC/src/sim.cpp:5-8 ------------------------------------------
// e: the trial elastic part (total - plastic), updated to the elastic part after the return;
// inv_kH = 1 / max(1e-20, k + H), precomputed per beam (the reference divides).  Elastic and
// hardening energies come as twice their value, k e^2 + H a^2: the factor 1/2 is applied once
// per block.
struct Ret1 { double force, p, a, dg, energy2; bool yielded; };
__device__ __forceinline__ Ret1 return1(double e, double pc, double ac, double k, double y, double H, double inv_kH) {
    Ret1 r{0, pc, ac, 0, 0, false};
    r.force = k * e;
    const double f = fabs(r.force) - fma(H, ac, y);
    if (positive(f)) {
        r.dg = f * inv_kH;
        const double s = xor_sign(r.dg, r.force);
        r.p = pc + s;
        r.a = ac + r.dg;
        e -= s;
        r.force = k * e;
        r.yielded = true;
    }
    r.energy2 = fma(r.force, e, (H * r.a) * r.a);
    return r;
}
// The vector form.  The yield test needs |trial| = k |e| only where it yields: whether it can
// is decided on the squares, k^2 |e|^2 > Y^2 (with a margin for their rounding), the square
// root is taken for those beams and the test as the reference writes it decides.
struct Ret3 { d3 force, p; double a, dg, energy2; bool yielded; };
__device__ __forceinline__ Ret3 return3(d3 e, d3 pc, double ac, double k, double y, double H, double inv_kH) {
    Ret3 r{{}, pc, ac, 0, 0, false};
    double e2 = fdot(e, e);
    const double Y = fma(H, ac, y);
    if (positive(fma((k * k) * (1.0 + 0x1p-48), e2, -Y * Y)) || negative_sign(Y)) {
        const double rs = rsqrt_any(e2), n = k * (e2 * rs), f = n - Y;
        if (positive(f) && less_bits(1e-20, n)) {
            r.dg = f * inv_kH;
            const double f1 = rs * r.dg;
            r.p = fmadd(e, f1, pc);
            r.a = ac + r.dg;
            e = fmadd(e, -f1, e);
            e2 = fdot(e, e);
            r.yielded = true;
        }
    }
    r.force = e * k;
    r.energy2 = fma(k, e2, (H * r.a) * r.a);
    return r;
}

// Length and inverse length of a chord from its square (from 2^-111 on by the estimate).  Both
// are rounded as the reference's sqrt and division, the inverse by one correction with the
// residual of 1 / sqrt(l2) as the start (Markstein, as sqrt_from): at rest the chord's tangent is
// then the stored director bit for bit, and the shear vanishes exactly.
__device__ __forceinline__ void chord_length(double l2, double& L, double& invL) {
    if (rsqrt_range(l2)) {
        const double y = rsqrt_est(l2);
        L = sqrt_from(l2, y);
        invL = fma(fma(-L, y, 1.0), y, y);
    } else {
        L = sqrt(l2);
        invL = 1.0 / L;
    }
}

// Polynomials in fixed point, coefficients c of units 2^-kBits, the argument x < 2^(64 - kArg) in
// units 2^-kArg: Horner's rule by the upper halves of 64 x 64-bit products.
template <int kBits>
__device__ constexpr unsigned long long poly_units(double c) {
    return (unsigned long long)(c * double(1ULL << (kBits - 32)) * 0x1p32);
}
template <int kArg>
__device__ __forceinline__ unsigned long long poly_step(unsigned long long acc, unsigned long long x, unsigned long long c) {
    return c + (__umul64hi(acc, x) >> (kArg - 64));
}

// Rotation vector of the relative rotation Q = Ra^* Rb (MC/include/core.hpp:52 quatLog of the
// normalized Q with w >= 0) in units times 2^e, Ra's and Rb's vector parts with exponents ea and eb.
// With s = |v| of the unit Q, the vector is 2 asin(s) / s v: a polynomial in s^2 up to s^2 = 0.1
// (angles up to 36.9 degrees; Chebyshev interpolation, error 2e-18), so that the usual beam takes no
// square root, division or arctangent; larger angles take atan2 as the reference does.  Q is a
// product of two quaternions of length one to 2^-56.  Its vector part a.w b - b.w a - a x b is summed
// at the larger exponent (it is below 2 there, the rotation vector below 4).
constexpr long long fx_limit(double v) { return (long long)(v * 0x1p58); }
__device__ __forceinline__ u3 relative_rotation(const fx4& a, int ea, const fx4& b, int eb, int& e) {
    e = max(ea, eb);
    const fx3 av{a.x, a.y, a.z}, bv{b.x, b.y, b.z};
    const u3 c = fx_cross(av, bv);
    const auto part = [&](fx p, fx q, long long r) {
        return fx_shr(fx_mul(a.w, q), e - eb) - fx_shr(fx_mul(b.w, p), e - ea) - fx_shr(r, e - ea - eb);
    };
    const u3 v{part(a.x, b.x, c.x), part(a.y, b.y, c.y), part(a.z, b.z, c.z)};
    const fx3 vf = fx_of(v);
    const long long s2 = fx_shr(fx_dot(vf, vf), -2 * e);
    if (s2 < fx_limit(0.1)) {
        constexpr int B = 62, X = 67;
        const unsigned long long u = (unsigned long long)s2 << (X - 58);
        unsigned long long g = poly_units<B>(0x1.c42a558b8b15bp-6);
        g = poly_step<X>(g, u, poly_units<B>(0x1.11d08867c9adep-6));
        g = poly_step<X>(g, u, poly_units<B>(0x1.80fd1940cecf2p-6));
        g = poly_step<X>(g, u, poly_units<B>(0x1.c90c2f25d23e5p-6));
        g = poly_step<X>(g, u, poly_units<B>(0x1.1c529e3ddf7c6p-5));
        g = poly_step<X>(g, u, poly_units<B>(0x1.6e8b80a6ac006p-5));
        g = poly_step<X>(g, u, poly_units<B>(0x1.f1c71d2f31c2ep-5));
        g = poly_step<X>(g, u, poly_units<B>(0x1.6db6db6c86271p-4));
        g = poly_step<X>(g, u, poly_units<B>(0x1.33333333342e1p-3));
        g = poly_step<X>(g, u, poly_units<B>(0x1.5555555555550p-2));
        g = poly_step<X>(g, u, poly_units<B>(2.0));
        // the sign of Q's real part, which is close to one
        const long long w = fx_hh(a.w, b.w) + fx_shr(fx_hh(a.x, b.x) + fx_hh(a.y, b.y) + fx_hh(a.z, b.z), -(ea + eb));
        const long long gu = (long long)(g >> (B - 58));
        const fx gf = fx_of(w < 0 ? -gu : gu);
        return u3{fx_mul(vf.x, gf), fx_mul(vf.y, gf), fx_mul(vf.z, gf)};
    }
    const d3 vd = fx_double(v, e - 58);
    q4 Q = qnorm(q4{fx_double(fx_mul(a.w, b.w) + fx_shr(fx_dot(av, bv), -(ea + eb))), vd.x, vd.y, vd.z});
    if (Q.w < 0) Q = q4{-Q.w, -Q.x, -Q.y, -Q.z};
    const double s = sqrt(Q.x * Q.x + Q.y * Q.y + Q.z * Q.z);
    d3 phi{2 * Q.x, 2 * Q.y, 2 * Q.z};
    if (!(s < 1e-12)) phi = d3{Q.x, Q.y, Q.z} * (2 * atan2(s, clampd(Q.w, -1, 1)) / s);
    e = 0;
    return fx_units(phi);
}

// R J_l^{-T}(phi) v (jl_inv_t): J^{-T} v = v + phi x v / 2 + A phi x (phi x v), the coefficient A a
// polynomial in |phi|^2 up to 0.42 (every angle of relative_rotation's polynomial; Chebyshev
// interpolation, error 4e-17 against 1/12, which enters multiplied by |phi|^2), in [1/12, 0.084].
__device__ __forceinline__ d3 transport_rotated(const FxRot& r, u3 phi, d3 v) {
    const fx3 pf = fx_of(phi);
    const long long phi2 = fx_dot(pf, pf);
    u3 n;
    int e;
    if (!block_units(v, n, e)) return fmrot(fx_matrix(r), jl_inv_t(fx_double(phi), v));
    if (phi2 < fx_limit(0.4199)) {
        constexpr int B = 66, X = 65;
        const unsigned long long u = (unsigned long long)phi2 << (X - 58);
        unsigned long long p = poly_units<B>(0x1.2bf59666dc69ep-31);
        p = poly_step<X>(p, u, poly_units<B>(0x1.6684f73f8bd8ep-26));
        p = poly_step<X>(p, u, poly_units<B>(0x1.bbd7b81461d47p-21));
        p = poly_step<X>(p, u, poly_units<B>(0x1.1566aba745146p-15));
        p = poly_step<X>(p, u, poly_units<B>(0x1.6c16c16c1de72p-10));
        p = poly_step<X>(p, u, poly_units<B>(0x1.5555555555553p-4));
        const fx A = fx_of((long long)(p >> (B - 58)));
        const u3 c1 = fx_cross(pf, fx_of(n));
        const fx3 c2 = fx_of(fx_cross(pf, fx_of(c1)));
        n = u3{n.x + (c1.x >> 1) + fx_mul(A, c2.x), n.y + (c1.y >> 1) + fx_mul(A, c2.y), n.z + (c1.z >> 1) + fx_mul(A, c2.z)};
    } else {
        if (!block_units(jl_inv_t(fx_double(phi), v), n, e)) return d3{0, 0, 0};  // v is in range, so this is a zero
    }
    return fx_rotate(r, n, e);
}

// The beam's axis in the material frame in units: unit(Ra^T t), t (units n) of length one but for
// rounding.
__device__ __forceinline__ u3 material_axis(const FxRot& m, u3 n, const fx3& t) {
    const int d = int(fx_dot(t, t) - kFxOne);
    const auto part = [&](long long k, fx a, fx b, fx c) { return fx_renorm(k + fx_shr(fx_dot(fx3{a, b, c}, t), -m.e), d); };
    return u3{part(n.x, m.r0.x, m.r1.x, m.r2.x), part(n.y, m.r0.y, m.r1.y, m.r2.y), part(n.z, m.r0.z, m.r1.z, m.r2.z)};
}
// R e0 - t = (R - I) e0 - (t - e0): a director's deviation from the chord, in units times 2^e, as te is
// of t - e0 (both small where the deviation is; below 8 with |e0| < 2 sqrt(3)).
__device__ __forceinline__ u3 deviation(const FxRot& r, const fx3& e0, u3 te, int e) {
    const int s = e - r.e;
    return u3{fx_shr(fx_dot(r.r0, e0), s) - te.x, fx_shr(fx_dot(r.r1, e0), s) - te.y, fx_shr(fx_dot(r.r2, e0), s) - te.z};
}

// ---- beam kernel: MC/src/sim.cpp:139-141 ---------------------------------------------------
// Bound by the FP64 pipe (one warp instruction per 19 cycles and SM, beside which loads and the
// other pipes are idle), so the formulas are written for few FP64 instructions: energies summed
// as twice their value, shear from the director-chord differences (2 t - da - db = -(ma + mb)),
// square roots from the FP32 estimate, comparisons on bit patterns, and everything that is a sum of
// products of unit vectors and rotation vectors (directors, relative rotation, material axis, trial
// twist and bending, the moment's transport and rotation) or a polynomial of one's coordinates in
// fixed point on the integer pipe.  A fixed-point sum rounds once: per beam against quadruple
// precision, rotations from 1e-15 to 1, the moment's median error is 0.7e-16 to 1.8e-16 (all in FP64:
// 0.9e-16 to 2.2e-16).
// FP64 instructions per 32 beams: 391 at first, 265 with all of it in FP64, 135 now (3430 in all;
// 132 and 3170 without the vectors' exponents, which cost 4 % of the kernel's time).
// The kernel alone: 184,400 beams 159 -> 98 -> 66 us, 2.95 million 1372 -> 835 us (one FP64
// instruction per 21 cycles and SM; nothing but FP64 reaches 19); a call at 2.95 million beams 2474 ->
// 1895 us, a batch of 762,000 beams 603 -> 455.
// Blocks of kBeamBlock = 128 beams: one warp on each of an SM's four FP64 units, so that a
// lattice of a few hundred beams spreads over several SMs.
// kMinBlocks: units of 256 threads per SM the register allocation must allow (an occupancy
// variant picked by mcg_autotune; the arithmetic, and so the result, is the same in every variant).
template <int kMinBlocks>
__global__ void __launch_bounds__(kBeamBlock, 2 * kMinBlocks) k_beams(DevTopo t, Material m,
                                                                      const double* __restrict__ plastic, int trials,
                                                                      EvalBufs e) {
    __shared__ double sm[2 * (kBeamBlock / 32)];
    const MapPos mp = map_pos(t.bblk);
    if (!t.active[mp.inst]) return;
    if (trials == 2) trials = t.trial_inst[mp.inst];  // per instance (device-resident solver)
    const int b = mp.i;
    const int B = t.B;
    double elastic2 = 0, diss = 0, penalty = 0;  // twice the elastic energy, plastic dissipation
    if (mp.valid) {
        const int2 ab = t.ab[b];
        const d3 xa = ldx(e.x, ab.x), xb = ldx(e.x, ab.y);
        // chord, its square and tangent rounded as the reference (no fused multiply-add), so
        // that a beam at its rest length has zero strain here too
        const d3 d{__dsub_rn(xb.x, xa.x), __dsub_rn(xb.y, xa.y), __dsub_rn(xb.z, xa.z)};
        double L, invL;
        chord_length(__dadd_rn(__dadd_rn(__dmul_rn(d.x, d.x), __dmul_rn(d.y, d.y)), __dmul_rn(d.z, d.z)), L, invL);
        double2* slot = reinterpret_cast<double2*>(e.slot) + 6 * size_t(b);
        if (less_bits(L, 1e-10)) {
            // Degenerate element: penalty energy only, no gradient and a default trial.
            penalty = 1e8 * sqr(1e-10 - L);
#pragma unroll
            for (int k = 0; k < 6; k++) slot[k] = make_double2(0, 0);
            if (trials) {
#pragma unroll
                for (int k = 0; k < 7; k++) { e.trial_next[k * size_t(B) + b] = 0; e.trial_aux[k * size_t(B) + b] = 0; }
#pragma unroll
                for (int k = 0; k < 3; k++) e.trial_flags[k * size_t(B) + b] = 0;
            }
        } else {
            const double pl_epsp = plastic[b], pl_alpha = plastic[size_t(B) + b];
            const d3 rotp{plastic[2 * size_t(B) + b], plastic[3 * size_t(B) + b], plastic[4 * size_t(B) + b]};
            const double pl_alphaB = plastic[5 * size_t(B) + b], pl_alphaT = plastic[6 * size_t(B) + b];
            const d3 tt{__dmul_rn(d.x, invL), __dmul_rn(d.y, invL), __dmul_rn(d.z, invL)};
            // axial
            const double eps = (L - t.L0[b]) * t.invL0[b];
            const Ret1 ax = return1(eps - pl_epsp, pl_epsp, pl_alpha, m.E, t.sy[b], m.H, m.inv_EH);
            const double uax2 = t.aL[b] * ax.energy2;
            if (ax.yielded) diss = t.aLsy[b] * ax.dg;
            // shear: the end directors against the chord (rotations by the nodes' matrices)
            const FxRot Ma = load_rotation(e.M + 4 * size_t(ab.x)), Mb = load_rotation(e.M + 4 * size_t(ab.y));
            const int2 e0x = t.e0fx[b], e0y = t.e0fy[b], e0z = t.e0fz[b];
            const double cs = t.cs[b];
            const u3 tu = fx_units(tt);
            const fx3 tf = fx_of(tu);
            const d3 e0{t.e0x[b], t.e0y[b], t.e0z[b]};
            d3 ma, mb, gm, Ga, Gb;  // deviations, their sum, and cs t x (R e0) = cs t x m
            if (e0x.y != kFxInvalid) {
                const fx3 e0f{fx{e0x.y, e0x.x}, fx{e0y.y, e0y.x}, fx{e0z.y, e0z.x}};
                const d3 te = tt - e0;
                const int e = max(fx_exponent(te), max(Ma.e, Mb.e));
                const u3 teu = fx_units(te, e), ua = deviation(Ma, e0f, teu, e), ub = deviation(Mb, e0f, teu, e);
                ma = fx_double(ua, e - 58);
                mb = fx_double(ub, e - 58);
                gm = ma + mb;
                Ga = fx_double(fx_cross(tf, fx_of(ua)), e - 58) * cs;
                Gb = fx_double(fx_cross(tf, fx_of(ub)), e - 58) * cs;
            } else {  // no direction
                ma = fmrot(fx_matrix(Ma), e0) - tt;
                mb = fmrot(fx_matrix(Mb), e0) - tt;
                gm = ma + mb;
                Ga = fcross(tt, ma) * cs;
                Gb = fcross(tt, mb) * cs;
            }
            const double us2 = fma(mb.z, mb.z, fma(mb.y, mb.y, fma(mb.x, mb.x, fdot(ma, ma))));  // times cs
            const double kt_ = cs * invL;
            const double kf = fma(kt_, fdot(gm, tt), t.area[b] * ax.force);
            // F = t N + ((I - t t^T) g) / L with g = -cs (ma + mb)
            const d3 F{fma(tt.x, kf, -(kt_ * gm.x)), fma(tt.y, kf, -(kt_ * gm.y)), fma(tt.z, kf, -(kt_ * gm.z))};
            // bending and torsion from the relative rotation Q = Ra^* Rb
            const fx4 qa = load_fx4(e.M + 4 * size_t(ab.x) + 3), qb = load_fx4(e.M + 4 * size_t(ab.y) + 3);
            int ep;  // exponent of phi
            const u3 phi = relative_rotation(qa, Ma.e, qb, Mb.e, ep), axis_u = material_axis(Ma, tu, tf);
            const d3 axis = fx_double(axis_u);
            // trial elastic parts: the twist and the bending of d = phi - rotp, at the larger exponent
            // (|phi| < 4 and |rotp| < sqrt(3)/2 there, so |d| < 5)
            double dtw = __longlong_as_double(0x7ff8000000000000LL);  // rotp not finite, or so large that
            d3 dbend{dtw, dtw, dtw};                                  // its square, an energy, is not
            const int ed = max(fx_exponent(rotp), ep);
            if (ed <= kFxMost) {
                const u3 rp = fx_units(rotp, ed), ph = fx_shr(phi, ed - ep), d{ph.x - rp.x, ph.y - rp.y, ph.z - rp.z};
                const fx3 af = fx_of(axis_u);
                const long long w = fx_dot(fx_of(d), af);
                const fx wf = fx_of(w);
                dtw = fx_double(w, ed - 58);
                dbend = fx_double(u3{d.x - fx_mul(af.x, wf), d.y - fx_mul(af.y, wf), d.z - fx_mul(af.z, wf)}, ed - 58);
            }
            double ptw = 0;  // the plastic parts enter the trial state only
            d3 pb{0, 0, 0};
            if (trials) {
                ptw = fdot(rotp, axis);
                pb = fmadd(axis, -ptw, rotp);
            }
            const double kb = t.kb[b], kt = t.kt[b];
            const Ret3 br = return3(dbend, pb, pl_alphaB, kb, t.my[b], t.hb[b], t.inv_kbh[b]);
            const Ret1 tor = return1(dtw, ptw, pl_alphaT, kt, t.ty[b], t.ht[b], t.inv_kth[b]);
            const d3 moment = fmadd(axis, tor.force, br.force);
            double dr = 0;
            if (br.yielded) dr = t.my[b] * br.dg;
            if (tor.yielded) dr = fma(t.ty[b], tor.dg, dr);
            const d3 world = transport_rotated(Ma, fx_shr(phi, -ep), moment);
            Ga = Ga - world;
            Gb = Gb + world;
            elastic2 = fma(cs, us2, uax2) + (br.energy2 + tor.energy2);
            if (qa.w.h == kFxInvalid || qb.w.h == kFxInvalid) elastic2 = __longlong_as_double(0x7ff8000000000000LL);
            slot[0] = make_double2(-F.x, -F.y);
            slot[1] = make_double2(-F.z, Ga.x);
            slot[2] = make_double2(Ga.y, Ga.z);
            slot[3] = make_double2(F.x, F.y);
            slot[4] = make_double2(F.z, Gb.x);
            slot[5] = make_double2(Gb.y, Gb.z);
            if (trials) {
                const size_t S = size_t(B);
                const d3 nrot = fmadd(axis, tor.p, br.p);
                e.trial_next[b] = ax.p;
                e.trial_next[S + b] = ax.a;
                e.trial_next[2 * S + b] = nrot.x;
                e.trial_next[3 * S + b] = nrot.y;
                e.trial_next[4 * S + b] = nrot.z;
                e.trial_next[5 * S + b] = br.a;
                e.trial_next[6 * S + b] = tor.a;
                e.trial_aux[b] = eps;
                e.trial_aux[S + b] = ax.force;
                e.trial_aux[2 * S + b] = moment.x;
                e.trial_aux[3 * S + b] = moment.y;
                e.trial_aux[4 * S + b] = moment.z;
                e.trial_aux[5 * S + b] = .5 * elastic2;
                e.trial_aux[6 * S + b] = diss + dr;
                e.trial_flags[b] = ax.yielded;
                e.trial_flags[S + b] = br.yielded;
                e.trial_flags[2 * S + b] = tor.yielded;
            }
            diss += dr;
        }
    }
    const double v = warp_sum2(elastic2, diss);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((lane & 15) == 0) sm[(lane >> 4) * (kBeamBlock / 32) + warp] = v;
    const bool degenerate = __syncthreads_or(__double_as_longlong(penalty) != 0);
    if (threadIdx.x == 0) {
        double el = 0, pl = 0;
#pragma unroll
        for (int w = 0; w < kBeamBlock / 32; w++) {
            el += sm[w];
            pl += sm[kBeamBlock / 32 + w];
        }
        el *= .5;
        e.part_beam[3 * blockIdx.x] = el + pl;
        e.part_beam[3 * blockIdx.x + 1] = el;
        e.part_beam[3 * blockIdx.x + 2] = pl;
    }
    if (degenerate) {  // block-uniform, rare
        __syncthreads();
        double acc[1] = {penalty};
        block_sum<1>(acc, sm);
        if (threadIdx.x == 0) e.part_beam[3 * blockIdx.x] += acc[0];
    }
}

// Value of a fixed-point sum (NodeContact): carries propagated, sign taken out, the magnitude's
// two halves converted and scaled by the quantum 2^e0.
__device__ __forceinline__ double fixed_value(const long long* l, int e0) {
    unsigned a[4];
    long long t = 0;
#pragma unroll
    for (int k = 0; k < kSumLimbs; k++) {
        t = l[k] + (t >> 32);
        a[k] = unsigned(t);
    }
    const bool minus = t < 0;
    unsigned long long lo = ((unsigned long long)a[1] << 32) | a[0], hi = ((unsigned long long)a[3] << 32) | a[2];
    if (minus) {
        lo = ~lo + 1;
        hi = ~hi + (lo == 0);
    }
    const double v = fma(double(hi), 0x1p64, double(lo)) * __hiloint2double((e0 + 1023) << 20, 0);
    return minus ? -v : v;
}

// ---- per-node gather: the scatter of MC/src/sim.cpp:139-172, as a deterministic CSR sum ---
// Sums one half (0 translations, 1 rotations) of the incident beams' end vectors of node i in
// ascending beam order: FP64 slots directly, FP32 slots (mixed form) with compensated FP32 sums.
template <bool F32>
__device__ __forceinline__ d3 sum_slots(const DevTopo& t, const EvalBufs& e, int i, int half) {
    const int k0 = t.inc_start[i], k1 = t.inc_start[i + 1];
    // unrolled so that the loads of several incident beams are in flight together; the
    // additions keep their order
    if (!F32) {
        d3 g{0, 0, 0};
#pragma unroll 4
        for (int k = k0; k < k1; k++) {
            const double* s = e.slot + 6 * size_t(t.inc[k]);  // 16-byte aligned, as are s + 2 and s + 4
            const double2 u = *reinterpret_cast<const double2*>(s + 4 * half);
            const double v = s[2 + half];
            g.x += half ? v : u.x;
            g.y += half ? u.x : u.y;
            g.z += half ? u.y : v;
        }
        return g;
    }
    float hi[3] = {0, 0, 0}, lo[3] = {0, 0, 0};
#pragma unroll 4
    for (int k = k0; k < k1; k++) {
        const float* s = e.slotf + 6 * size_t(t.inc[k]);  // 8-byte aligned, as are s + 2 and s + 4
        const float2 u = *reinterpret_cast<const float2*>(s + 4 * half);
        const float v = s[2 + half];
        const float x[3] = {half ? v : u.x, half ? u.x : u.y, half ? u.y : v};
#pragma unroll
        for (int j = 0; j < 3; j++) {  // two-sum
            const float a = x[j], sum = hi[j] + a, bp = sum - hi[j];
            lo[j] += (hi[j] - (sum - bp)) + (a - bp);
            hi[j] = sum;
        }
    }
    return d3{to_double(hi[0]) + to_double(lo[0]), to_double(hi[1]) + to_double(lo[1]), to_double(hi[2]) + to_double(lo[2])};
}

// Per-warp totals of the gather; then the evaluation's totals.
constexpr int kGatherNodes = kEvalBlock / 2;  // nodes of a gather block: two threads each
struct GatherParts {
    double g2[kGatherNodes];             // |g|^2 and max |g| of the rotations
    long long gbits[kGatherNodes];
    double sum[5][kGatherNodes / 32];    // gravity E, |g|^2, platen E, reaction, self-contact E
    int count[kGatherNodes / 32];
    long long m[2][kGatherNodes / 32];   // max penetration, max |g| (bits of non-negative doubles)
};

// ---- totals and the non-finite guard ---------------------------------------------------------
// An instance of few block partials (kFinSingle; a block reads six per thread in about the time of a
// launch) is summed by the last of its gather blocks to finish; a larger
// one by kFinFan blocks of k_finalize (block f takes the partials first + f + kFinFan j), the last
// of which to finish sums their results in order, so the FP64 additions spread over many SMs.
// Which way an instance goes depends on its own size only, so it sums alike alone and in a batch.
constexpr int kFinFan = 32;
constexpr int kFinVals = 11;  // beamE, elastic, plastic, gravityE, platenE, reaction, contactE,
                              // contacts, |g|^2, max penetration, max |g|
static_assert(kFinPartDoubles == kFinFan * kFinVals, "first-stage totals");

struct TotalParts {
    double sum[9][kEvalBlock / 32];
    long long m[2][kEvalBlock / 32];
    double tot[kFinVals];
    int nonfinite;
};
// Totals of the beam blocks r and gather blocks er (every fan-th from f on) into sm.tot.
__device__ __forceinline__ void sum_parts(const EvalBufs& e, int2 r, int2 er, int f, int fan, TotalParts& sm) {
    double all[9] = {};        // sums: beamE, elastic, plastic, gravityE, platenE, reaction, contactE, contacts, |g|^2
    long long m2[2] = {0, 0};  // max penetration, max |g| (bits of non-negative doubles)
    for (int k = r.x + f + fan * int(threadIdx.x); k < r.y; k += fan * kEvalBlock) {
        const double* q = e.part_beam + 3 * size_t(k);
        all[0] += q[0]; all[1] += q[1]; all[2] += q[2];
    }
#pragma unroll 2
    for (int k = er.x + f + fan * int(threadIdx.x); k < er.y; k += fan * kEvalBlock) {
        const double* q = e.part_node + kNodeParts * size_t(k);
        all[3] += __ldcg(q); all[4] += __ldcg(q + 1); all[5] += __ldcg(q + 2);
        m2[0] = max(m2[0], __double_as_longlong(__ldcg(q + 3)));
        all[7] += __ldcg(q + 4);
        all[6] += __ldcg(q + 5);
        all[8] += __ldcg(q + 6);
        m2[1] = max(m2[1], __double_as_longlong(__ldcg(q + 7)));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j = lane >> 3;
    const double a = warp_sum4(all[0], all[1], all[2], all[3]), b = warp_sum4(all[4], all[5], all[6], all[7]);
    const double c = warp_sum(all[8]);
    const long long pm = warp_max_key(m2[0]), gm = warp_max_key(m2[1]);
    if ((lane & 7) == 0) {
        sm.sum[j][warp] = a;
        sm.sum[4 + j][warp] = b;
    }
    if (lane == 0) {
        sm.sum[8][warp] = c;
        sm.m[0][warp] = pm;
        sm.m[1][warp] = gm;
    }
    __syncthreads();
    const int tid = threadIdx.x;
    constexpr int nw = kEvalBlock / 32;
    if (tid < 9) {
        double s = sm.sum[tid][0];
        for (int w = 1; w < nw; w++) s += sm.sum[tid][w];
        sm.tot[tid] = s;
    } else if (tid < kFinVals) {
        long long m = sm.m[tid - 9][0];
        for (int w = 1; w < nw; w++) m = max(m, sm.m[tid - 9][w]);
        sm.tot[tid] = __longlong_as_double(m);
    }
    __syncthreads();
}
// The instance's results from its totals sm.tot, by a whole block; clears the gradient of a
// non-finite evaluation (sim.cpp:172).
__device__ __forceinline__ void write_out(const DevTopo& t, const PhysParams& p, const EvalBufs& e, int inst, TotalParts& sm,
                                          double* __restrict__ grad) {
    const double* tot = sm.tot;
    if (threadIdx.x == 0 || threadIdx.x == 32) {  // one the energies, one the residual (a division and a root)
        const double* c = e.cen + 9 * size_t(inst);
        const double center = .5 * p.centering * (sqr(c[0]) + sqr(c[2]));
        // Group order of the reference's accumulation: beams, gravity, centering,
        // self-contact, platens (sim.cpp:139-171).
        double energy = tot[0];
        energy += tot[3];
        energy += center;
        energy += tot[6];
        energy += tot[4];
        const int nonfinite = isfinite(energy) ? 0 : 1;
        if (threadIdx.x == 32) {
            const long long nf = t.inst_free[inst];
            const double rms = nonfinite ? 0.0 : (nf ? sqrt(tot[8] / double(nf)) : 0.0);
            for (EvalOut* o : {e.out, e.out_host}) {
                if (!o) continue;
                o[inst].rms = rms;
                o[inst].gmax = nonfinite ? 0.0 : tot[10];
            }
        } else {
            for (EvalOut* o : {e.out, e.out_host}) {
                if (!o) continue;
                EvalOut* out = o + inst;
                out->energy = nonfinite ? __longlong_as_double(0x7ff0000000000000LL) : energy;
                out->elastic = tot[1];
                out->plastic = tot[2];
                out->contact = tot[6] + tot[4];
                out->reaction = tot[5];
                out->max_pen = tot[9];
                out->contacts = int(tot[7]);
                out->nonfinite = nonfinite;
                out->beam_energy = tot[0];
                out->node_energy = tot[3];
                out->center_energy = center;
                out->contact_energy = tot[6];
                out->platen_energy = tot[4];
            }
            sm.nonfinite = nonfinite;
        }
    }
    __syncthreads();
    if (sm.nonfinite) {  // non-finite energy: the instance's whole gradient is zero
        const size_t o = 6 * size_t(t.eblk[t.erange[inst].x].x);
        for (long long k = threadIdx.x; k < 6LL * t.inst_n[inst]; k += blockDim.x) {
            grad[o + k] = 0;
            if (e.grad_host) e.grad_host[o + k] = 0;
        }
    }
}
// Gather blocks of an instance: two per evaluation block.
__device__ __forceinline__ int2 gather_range(const DevTopo& t, int inst) {
    const int2 er = t.erange[inst];
    return make_int2(2 * er.x, 2 * er.y);
}

// One half-node per thread (warps 0 and 1 the translations of 64 nodes, 2 and 3 their rotations).
// Bound by the FP64 pipe (the incident vectors' additions) and, up to 10^4 nodes, the latency of
// their loads: a whole node per thread takes twice the additions in a row.
// Only what nearly every node has is reduced always (gravity energy and |g|^2, in five FP64
// additions a warp); platen and contact totals where a node of the warp touches something.
// 2x4x2 specimen 73.3 -> 66.5 us a call, 19x15x11 88.4 -> 82.4, a minimization of 6x6x6 1.04x, with
// the totals summed here; 64x64x32 and larger as before with whole nodes per thread.
// kMinBlocks: units of 256 threads per SM the register allocation must allow.
template <bool F32, int kMinBlocks>
__global__ void __launch_bounds__(kEvalBlock, 2 * kMinBlocks) k_gather(DevTopo t, PhysParams p, ContactBufs c,
                                                                       int use_contacts, EvalBufs e,
                                                                       double* __restrict__ grad, int first) {
    constexpr int kNodes = kGatherNodes;
    static_assert(kNodes == 64, "two warps of translations, two of rotations");
    __shared__ GatherParts sm;
    __shared__ TotalParts ts;
    const int block = int(blockIdx.x) + first;
    if (block == 0 && threadIdx.x == 0) {  // of the whole evaluation, whether instance 0 is active or not
        for (EvalOut* out : {e.out, e.out_host}) {
            if (!out) continue;
            out->overflow = use_contacts ? int(c.flags[0] & ~uint32_t(kNonFinite)) : 0;
            out->kernel_error = *e.err;
        }
        if (use_contacts) c.flags[0] = c.flags[1] = 0;  // for the next evaluation
    }
    const int4 blk = t.eblk[block >> 1];
    const int inst = blk.z;
    if (!t.active[inst]) return;  // block-uniform
    const int half = threadIdx.x / kNodes, at = kNodes * (block & 1) + threadIdx.x % kNodes;
    const int i = blk.x + at;
    double egrav = 0, g2 = 0, eplat = 0, reac = 0, econt = 0, pen_max = 0;
    int count = 0;
    unsigned long long gbits = 0;  // max |g| as the bits of a non-negative double (integer max)
    if (at < blk.y) {
        d3 g = sum_slots<F32>(t, e, i, half);
        if (half == 0) {
            const d3 xi = ldx(e.x, i);
            // gravity (sim.cpp:142)
            const double mg = t.mass[i] * p.gravity;
            egrav = mg * xi.y;
            g.y += mg;
            // centering (sim.cpp:143), the same force for all nodes of the instance
            g.x += e.cforce[2 * inst];
            g.z += e.cforce[2 * inst + 1];
            // self-contact: the node's fixed-point sums, cleared for the next evaluation
            const unsigned long long items = use_contacts ? c.n_count[i] : 0ULL;
            if (items) {
                NodeContact& r = c.n_sum[i];
                g.x += fixed_value(r.f[0], c.force_e0);
                g.y += fixed_value(r.f[1], c.force_e0);
                g.z += fixed_value(r.f[2], c.force_e0);
                if (items >> 32) {
                    econt = fixed_value(r.energy, c.energy_e0);
                    pen_max = __longlong_as_double((long long)r.pen);
                }
                if (items & kContactNotFinite) econt = __longlong_as_double(0x7ff8000000000000LL);
                count = int(items >> 32);
                r = NodeContact{};
                c.n_count[i] = 0;
            }
            // platens (sim.cpp:168-171)
            const double jr = p.joint_radius, kc = p.contact_k;
            const double pb = jr - xi.y;
            if (positive(pb)) {
                const double mm = kc * pb;
                eplat += .5 * kc * pb * pb;
                pen_max = fmax(pen_max, pb);
                count += 1;
                g.y -= mm;
            }
            const double pt = xi.y + jr - e.tops[inst];
            if (positive(pt)) {
                const double mm = kc * pt;
                eplat += .5 * kc * pt * pt;
                reac += mm;
                pen_max = fmax(pen_max, pt);
                count += 1;
                g.y += mm;
            }
            g = g * p.translation_scale;
        }
        // pack and lock (sim.cpp:172)
        const uint8_t* li = t.locked + 6 * size_t(i) + 3 * half;
        double gv[3] = {g.x, g.y, g.z};
        double* out = grad + 6 * size_t(i) + 3 * half;
        double* host = e.grad_host ? e.grad_host + 6 * size_t(i) + 3 * half : nullptr;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            if (li[k]) gv[k] = 0.0;
            // residual over free DOFs for the solver's convergence test (sim.cpp:44-45)
            g2 = fma(gv[k], gv[k], g2);
            // fmax(gmax, |g|) on the bit patterns; a NaN (above the infinity pattern) is
            // skipped as fmax skips it
            const unsigned long long b = (unsigned long long)__double_as_longlong(gv[k]) & 0x7fffffffffffffffULL;
            if (b <= 0x7ff0000000000000ULL && b > gbits) gbits = b;
            out[k] = gv[k];
            if (host) host[k] = gv[k];
        }
    }
    // the rotations' share of the residual goes to the translations' thread of the node
    if (half == 1) {
        sm.g2[threadIdx.x - kNodes] = g2;
        sm.gbits[threadIdx.x - kNodes] = (long long)gbits;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (half == 0) {
        const double v = warp_sum2(egrav, g2 + sm.g2[threadIdx.x]);
        const long long gm = warp_max_key(max((long long)gbits, sm.gbits[threadIdx.x]));
        double w = 0;
        long long pm = 0;
        int cn = 0;
        if (__any_sync(0xffffffffu, count != 0 || __double_as_longlong(econt) != 0)) {
            w = warp_sum4(eplat, reac, econt, 0.0);
            pm = warp_max_key(__double_as_longlong(pen_max));
            cn = __reduce_add_sync(0xffffffffu, count);
        }
        if (lane == 0) {
            sm.m[0][warp] = pm;
            sm.m[1][warp] = gm;
            sm.count[warp] = cn;
        }
        if ((lane & 15) == 0) sm.sum[lane >> 4][warp] = v;
        if ((lane & 7) == 0 && lane < 24) sm.sum[2 + (lane >> 3)][warp] = w;
    }
    __syncthreads();
    const int tid = threadIdx.x;
    double* q = e.part_node + kNodeParts * size_t(block);
    if (tid < 5) q[tid == 0 ? 0 : tid == 1 ? 6 : tid == 2 ? 1 : tid == 3 ? 2 : 5] = sm.sum[tid][0] + sm.sum[tid][1];
    else if (tid < 7) q[tid == 5 ? 3 : 7] = __longlong_as_double(max(sm.m[tid - 5][0], sm.m[tid - 5][1]));
    else if (tid == 7) q[4] = double(sm.count[0] + sm.count[1]);
    const int2 r = t.brange[inst], gr = gather_range(t, inst);
    if ((r.y - r.x) + (gr.y - gr.x) > kFinSingle) return;  // k_finalize's
    if (!last_block(e.done + inst, unsigned(gr.y - gr.x))) return;
    sum_parts(e, r, gr, 0, 1, ts);
    write_out(t, p, e, inst, ts, grad);
}

// Totals of the instances of more than kFinSingle block partials.
__global__ void __launch_bounds__(kEvalBlock) k_finalize(DevTopo t, PhysParams p, EvalBufs e, double* __restrict__ grad) {
    __shared__ TotalParts sm;
    const int inst = blockIdx.y, f = blockIdx.x;
    const int2 r = t.brange[inst], gr = gather_range(t, inst);
    if (!t.active[inst] || (r.y - r.x) + (gr.y - gr.x) <= kFinSingle) return;
    sum_parts(e, r, gr, f, kFinFan, sm);
    double* fp = e.part_fin + size_t(kFinPartDoubles) * inst;
    if (threadIdx.x < kFinVals) fp[kFinVals * f + threadIdx.x] = sm.tot[threadIdx.x];
    if (!last_block(e.done + inst, kFinFan)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = warp; k < kFinVals; k += kEvalBlock / 32) {
        const double v = __ldcg(fp + kFinVals * lane + k);
        const double s = k < 9 ? warp_sum(v) : warp_max(v);
        if (lane == 0) sm.tot[k] = s;
    }
    __syncthreads();
    write_out(t, p, e, inst, sm, grad);
}

// ---- commit (MC/src/sim.cpp:212): base state <- current state, plastic <- trial ----------
__global__ void __launch_bounds__(kEvalBlock) k_commit_nodes(DevTopo t, const uint8_t* __restrict__ mask,
                                                         const double4_32a* __restrict__ x4,
                                                         const double4_32a* __restrict__ R4, double* __restrict__ bx,
                                                         double* __restrict__ br) {
    const MapPos mp = map_pos(t.eblk);
    if (!mp.valid || (mask && !mask[mp.inst])) return;
    const int i = mp.i;
    const double4_32a x = x4[i], r = R4[i];
    bx[3 * size_t(i)] = x.x; bx[3 * size_t(i) + 1] = x.y; bx[3 * size_t(i) + 2] = x.z;
    br[4 * size_t(i)] = r.x; br[4 * size_t(i) + 1] = r.y; br[4 * size_t(i) + 2] = r.z; br[4 * size_t(i) + 3] = r.w;
}

// plastic <- trial.next for the beams of the committed instances (7 SoA arrays)
__global__ void __launch_bounds__(kBlock) k_commit_plastic(DevTopo t, const uint8_t* __restrict__ mask,
                                                           const double* __restrict__ next, double* __restrict__ pl) {
    const MapPos mp = map_pos(t.bblk);
    if (!mp.valid || (mask && !mask[mp.inst])) return;
#pragma unroll
    for (int k = 0; k < 7; k++) pl[k * size_t(t.B) + mp.i] = next[k * size_t(t.B) + mp.i];
}

// Plastic statistics of the committed state (MC/src/sim.cpp:339-362), one partial per beam
// block: sum and max of |epsp|, sum and max of |rotp|, counts above 1e-5 and 1e-4.
__global__ void __launch_bounds__(kBlock) k_plastic_part(DevTopo t, const double* __restrict__ pl,
                                                         double* __restrict__ part) {
    __shared__ double sm[4 * (kBlock / 32)];
    __shared__ double smx[kBlock / 32];
    const MapPos mp = map_pos(t.bblk);
    const int B = t.B;
    double acc[4] = {0, 0, 0, 0};
    double m0 = 0, m1 = 0;
    if (mp.valid) {
        const int b = mp.i;
        const double pa = fabs(pl[b]);
        const d3 r{pl[2 * size_t(B) + b], pl[3 * size_t(B) + b], pl[4 * size_t(B) + b]};
        const double pr = len(r);
        acc[0] += pa; acc[1] += pr;
        acc[2] += pa > 1e-5 ? 1.0 : 0.0;
        acc[3] += pr > 1e-4 ? 1.0 : 0.0;
        m0 = fmax(m0, pa); m1 = fmax(m1, pr);
    }
    block_sum<4>(acc, sm);
    m0 = block_max(m0, smx);
    m1 = block_max(m1, smx);
    if (threadIdx.x == 0) {
        double* q = part + 6 * size_t(blockIdx.x);
        q[0] = acc[0]; q[1] = m0; q[2] = acc[1]; q[3] = m1; q[4] = acc[2]; q[5] = acc[3];
    }
}
// One block per instance over its beam blocks.
__global__ void __launch_bounds__(kBlock) k_plastic_final(DevTopo t, const double* __restrict__ part,
                                                          double* __restrict__ out) {
    __shared__ double sm[4 * (kBlock / 32)];
    __shared__ double smx[kBlock / 32];
    const int2 r = t.brange[blockIdx.x];
    double acc[4] = {0, 0, 0, 0};
    double m0 = 0, m1 = 0;
    for (int k = r.x + int(threadIdx.x); k < r.y; k += blockDim.x) {
        const double* q = part + 6 * size_t(k);
        acc[0] += q[0]; acc[1] += q[2]; acc[2] += q[4]; acc[3] += q[5];
        m0 = fmax(m0, q[1]); m1 = fmax(m1, q[3]);
    }
    block_sum<4>(acc, sm);
    m0 = block_max(m0, smx);
    m1 = block_max(m1, smx);
    if (threadIdx.x == 0) {
        double* o = out + 6 * size_t(blockIdx.x);
        o[0] = acc[0]; o[1] = m0; o[2] = acc[1]; o[3] = m1; o[4] = acc[2]; o[5] = acc[3];
    }
}

// The trial states of an evaluation (next, aux and flags) in one launch.
template <typename In>
__global__ void __launch_bounds__(kBlock) k_trial_records(long long B, const In* __restrict__ next, const In* __restrict__ aux,
                                                          const uint8_t* __restrict__ flags, double* __restrict__ rnext,
                                                          double* __restrict__ raux, uint8_t* __restrict__ rflags) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < 7 * B; i += (long long)gridDim.x * blockDim.x) {
        const long long b = i / 7, from = (i - 7 * b) * B + b;
        rnext[i] = double(next[from]);
        raux[i] = double(aux[from]);
        if (i < 3 * B) rflags[i] = flags[(i - i / 3 * 3) * B + i / 3];
    }
}
// ---- per-beam records in the ABI's layout ----------------------------------------------------
// K values per beam: structure of arrays (device) <-> K consecutive values per beam (host), so
// that a host array is one copy.  Thread i handles the i-th value of the written layout.
template <int K, typename In, typename Out>
__global__ void __launch_bounds__(kBlock) k_to_records(long long B, const In* __restrict__ soa, Out* __restrict__ aos) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < K * B; i += (long long)gridDim.x * blockDim.x) {
        const long long b = i / K;
        aos[i] = Out(soa[(i - K * b) * B + b]);
    }
}
__global__ void __launch_bounds__(kBlock) k_from_records7(long long B, const double* __restrict__ aos, double* __restrict__ soa) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < 7 * B; i += (long long)gridDim.x * blockDim.x) {
        const long long k = i / B;
        soa[i] = aos[7 * (i - k * B) + k];
    }
}

// ---- launchers ------------------------------------------------------------------------------
void launch_state(const DevTopo& t, const PhysParams& p, const double* z, const double* base_x, const BuildArgs& b, EvalBufs& e,
                  cudaStream_t s) {
    k_state<<<t.n_eblk, kEvalBlock, 0, s>>>(t, p, z, base_x, e.x, e.xf_lo, e.xf_hi, e.part_state, b);
    note_launches(1);
}

void launch_rotations(const DevTopo& t, const double* z, const double* base_r, EvalBufs& e, cudaStream_t s) {
    k_rotations<<<t.n_eblk, kEvalBlock, 0, s>>>(t, z, base_r, e.R, e.M);
    note_launches(1);
}

void launch_center(const DevTopo& t, const PhysParams& p, const BuildArgs& b, EvalBufs& e, cudaStream_t s) {
    k_center<<<t.I + 1, kBlock, 0, s>>>(t, p.centering, e.part_state, e.cen, e.cforce, e.tops, e.tops_host, b);
    note_launches(1);
}

void launch_commit(const DevTopo& t, const uint8_t* mask, const EvalBufs& e, double* base_x, double* base_r,
                   double* plastic, cudaStream_t s) {
    k_commit_nodes<<<t.n_eblk, kEvalBlock, 0, s>>>(t, mask, e.x, e.R, base_x, base_r);
    note_launches(1);
    if (t.B > 0 && plastic) {
        k_commit_plastic<<<t.n_bblk, t.bdim, 0, s>>>(t, mask, e.trial_next, plastic);
        note_launches(1);
    }
}

void launch_plastic_stats(const DevTopo& t, const double* plastic, double* part, double* out6, cudaStream_t s) {
    if (t.B == 0) return;
    k_plastic_part<<<t.n_bblk, t.bdim, 0, s>>>(t, plastic, part);
    k_plastic_final<<<t.I, kBlock, 0, s>>>(t, part, out6);
    note_launches(2);
}

static unsigned record_grid(long long n) { return grid_for(n < 16 * 152 * kBlock ? n : 16 * 152 * kBlock); }

void launch_records7(long long B, const double* soa, double* aos, cudaStream_t s) {
    if (B) (k_to_records<7><<<record_grid(7 * B), kBlock, 0, s>>>(B, soa, aos), note_launches(1));
}
void launch_trial_records(long long B, const EvalBufs& e, bool mixed, const TrialRecords& r, cudaStream_t s) {
    if (!B) return;
    if (mixed) k_trial_records<<<record_grid(7 * B), kBlock, 0, s>>>(B, e.trial_nextf, e.trial_auxf, e.trial_flags, r.next, r.aux, r.flags);
    else k_trial_records<<<record_grid(7 * B), kBlock, 0, s>>>(B, e.trial_next, e.trial_aux, e.trial_flags, r.next, r.aux, r.flags);
    note_launches(1);
}
void launch_from_records7(long long B, const double* aos, double* soa, cudaStream_t s) {
    if (B) (k_from_records7<<<record_grid(7 * B), kBlock, 0, s>>>(B, aos, soa), note_launches(1));
}

// Occupancy variants of the FP64 beam kernel (256-thread units per SM) and of the gather.  The
// defaults first: four beam blocks of 128 threads an SM (two leave the integer pipe's latency
// uncovered: largest lattice 2165 us a call against 1930; six spill and gain nothing), eight of the
// gather's (64x64x32 480 us on the GPU against 499 with two).
constexpr int kBeamBlocks[] = {2, 1, 3};
constexpr int kGatherBlocks[] = {4, 2, 1};

int shape_variants(ShapeKernel k) {
    switch (k) {
        case ShapeKernel::kBeams: return 3;
        case ShapeKernel::kGather: return 3;
        default: return beams_mixed_variants();
    }
}
int shape_blocks(ShapeKernel k, int v) {
    switch (k) {
        case ShapeKernel::kBeams: return kBeamBlocks[v];
        case ShapeKernel::kGather: return kGatherBlocks[v];
        default: return beams_mixed_blocks(v);
    }
}

void launch_beams(const DevTopo& t, const Material& m, const double* plastic, int trials, EvalBufs& e,
                  cudaStream_t s, int variant) {
    if (t.B == 0) return;
    const int tr = trials;  // 0, 1, or 2: per instance (t.trial_inst)
    switch (variant) {
        case 1: k_beams<kBeamBlocks[1]><<<t.n_bblk, kBeamBlock, 0, s>>>(t, m, plastic, tr, e); break;
        case 2: k_beams<kBeamBlocks[2]><<<t.n_bblk, kBeamBlock, 0, s>>>(t, m, plastic, tr, e); break;
        default: k_beams<kBeamBlocks[0]><<<t.n_bblk, kBeamBlock, 0, s>>>(t, m, plastic, tr, e); break;
    }
    note_launches(1);
}

template <bool F32>
void gather_variant(const DevTopo& t, const PhysParams& p, const ContactBufs* c, double* grad, EvalBufs& e,
                    cudaStream_t s, int variant, int first, int blocks) {
    ContactBufs cc{};
    if (c) cc = *c;
    const int uc = c ? 1 : 0, n = blocks < 0 ? 2 * t.n_eblk : blocks;
    switch (variant) {
        case 1: k_gather<F32, kGatherBlocks[1]><<<n, kEvalBlock, 0, s>>>(t, p, cc, uc, e, grad, first); break;
        case 2: k_gather<F32, kGatherBlocks[2]><<<n, kEvalBlock, 0, s>>>(t, p, cc, uc, e, grad, first); break;
        default: k_gather<F32, kGatherBlocks[0]><<<n, kEvalBlock, 0, s>>>(t, p, cc, uc, e, grad, first); break;
    }
    note_launches(1);
}

void launch_gather(const DevTopo& t, const PhysParams& p, const ContactBufs* c, double* grad, EvalBufs& e,
                   cudaStream_t s, int variant, int first, int blocks) {
    gather_variant<false>(t, p, c, grad, e, s, variant, first, blocks);
}

void launch_gather_mixed(const DevTopo& t, const PhysParams& p, const ContactBufs* c, double* grad, EvalBufs& e,
                         cudaStream_t s, int variant, int first, int blocks) {
    gather_variant<true>(t, p, c, grad, e, s, variant, first, blocks);
}

void launch_finalize(const DevTopo& t, const PhysParams& p, double* grad, EvalBufs& e, cudaStream_t s) {
    if (!t.large_totals) return;
    k_finalize<<<dim3(kFinFan, t.I), kEvalBlock, 0, s>>>(t, p, e, grad);
    note_launches(1);
}

}  // namespace mcg
