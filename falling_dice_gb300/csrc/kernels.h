// kernels.h -- device data layout and the host-side launchers of the CUDA kernels.
//
// HBM layout (one context = one lattice):
//   per beam (SoA, FP64): L0, area, radius, e0[3 arrays], and the section constants the
//     reference recomputes on every call (E I/L0, G J/L0, yield moments, hardening
//     moduli, shear and axial energy scales), precomputed once with the reference's own
//     expressions so they are bit-identical; plastic state as 7 SoA arrays.
//   per node: base position (3 FP64, AoS), base orientation (4 FP64, AoS), current
//     position/orientation as 32-byte double4_32a records so each beam-end gather is one
//     sector; the 6-DOF z/grad vectors in the ABI layout.
//   incidence CSR: for every node the beams touching it in ascending beam order, as
//     (beam << 1 | role) -- the order the reference's scatter adds them in.
//   per-beam gradient slots: the beam kernel writes, for each end, the 6-vector it adds to
//     that end's node, and the gather sums them per node; no atomics anywhere on the
//     gradient path, so every evaluation is bitwise reproducible.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace mcg {

struct Material {
    double E, G, sy, H, bend_h, torsion_h;
    double inv_EH;  // 1 / max(1e-20, E + H)
    float Ef, Hf, bend_hf, torsion_hf;  // the same in single precision (mixed form)
};

struct DevTopo {
    int N, B;
    const int2* ab;
    const double *L0, *area, *radius;
    const double *e0x, *e0y, *e0z;
    const int2 *e0fx, *e0fy, *e0fz;  // the same in fixed point (fx: l, h); e0fx.y = kFxInvalid: no direction
    const double *kb, *kt, *my, *ty, *hb, *ht, *cs, *aL, *aLsy;
    const double *invL0, *inv_kbh, *inv_kth;  // 1/L0, 1/max(1e-20, kb+hb), 1/max(1e-20, kt+ht)
    const double* mass;
    const uint8_t* locked;    // [6N]
    const int* inc_start;     // [N+1]
    const int* inc;           // [2B]
    // connected node pairs (the reference's connected_ set) as an open-addressing hash set
    // of keys u << 32 | v, u <= v; empty slots hold ~0; at most half full
    const unsigned long long* conn_hash;
    unsigned long long conn_mask;  // slots - 1 (a power of two)
    int conn_shift;                // 64 - log2(slots)
    const float* padf;        // [B] radius + contact margin, rounded up to single precision
    const double* sy;         // [B] yield stress (the beam's instance)
    // Instances: a context holds I lattices stored one after another (I = 1 for a plain
    // context).  Node and beam kernels run over blocks that never straddle two instances,
    // so every block partial belongs to one instance and per-instance totals are sums over
    // an instance's own blocks, in the same order as for that lattice alone.
    int I;
    int n_bblk;               // beam blocks
    const int4* bblk;         // [n_bblk] first beam, beam count, instance, 0
    int bdim;                 // beams per beam block: kBeamBlock (FP64) or kMapBlock (mixed)
    const int2* brange;       // [I] beam blocks [x, y) of the instance
    int n_eblk;               // evaluation node blocks
    bool large_totals;        // an instance has more than kFinSingle beam and gather blocks
    const int4* eblk;         // [n_eblk] first node, node count, instance, 0
    const int2* erange;       // [I] evaluation node blocks [x, y) of the instance
    int n_sblk;               // solver blocks: at most kSolveBlocks runs of nodes per instance
    const int4* sblk;         // [n_sblk] first node, node count, instance, 0
    const int2* srange;       // [I] solver blocks [x, y) of the instance
    const int* inst_n;        // [I] nodes of the instance
    const long long* inst_free;  // [I] unlocked DOFs of the instance
    const float2* off;        // [I] (x, z) offset of the instance in the contact grid
    const int* node_inst;     // [N] instance of each node
    const uint8_t* active;    // [I] 0: the instance is not evaluated (its outputs keep old values)
    const uint8_t* trial_inst;  // [I] with trials == 2: 1 where the instance writes its trial states
};

// Elements per mapped block (the launch block size of the mapped kernels): the beam blocks of the
// mixed form; the FP64 form's beam blocks (one warp per FP64 unit of an SM).
constexpr int kMapBlock = 256;
constexpr int kBeamBlock = 128;
// Nodes per evaluation node block (state and gather).
constexpr int kEvalBlock = 128;
// Solver blocks an instance's vectors are divided into at most: one per SM.
constexpr int kSolveBlocks = 152;
constexpr int kFxInvalid = 0x7fffffff;  // the upper half of a fixed-point number that is none

#if defined(__CUDACC__)
// Position of a thread of a mapped block: element index, instance; valid == false past the
// block's element count.
struct MapPos {
    int i, inst;
    bool valid;
};
__device__ __forceinline__ MapPos map_pos(const int4* __restrict__ blk) {
    const int4 q = blk[blockIdx.x];
    return MapPos{q.x + int(threadIdx.x), q.z, int(threadIdx.x) < q.y};
}
#endif

struct PhysParams {
    double translation_scale, gravity, centering, contact_k, contact_margin, joint_radius;
    double broad_cell, top;
    float joint_padf;        // joint radius + margin, rounded up to single precision
    float inv_cell_f;        // 1 / broad_cell in single precision (broad-phase cell index)
    int self_contact;
};

// Totals of one evaluation: of an instance, by the last of its gather blocks or by k_finalize; the
// evaluation's flags (overflow, kernel_error), in the first instance's, by the first gather block.
struct EvalOut {
    double energy, elastic, plastic, contact, reaction, max_pen;
    int contacts, nonfinite;
    double beam_energy, node_energy, center_energy, contact_energy, platen_energy;
    int overflow;                    // ContactFlag bits that invalidate this evaluation
    unsigned kernel_error;           // a kernel's bounded wait gave up (EvalBufs::err)
    double rms, gmax;                // residual over free DOFs: sqrt(mean g^2), max |g| (sim.cpp:44-45)
};

// Device scratch of the contact pipeline (contact.cu).  Capacities are host-chosen and
// grown on demand: a kernel that would exceed one sets a bit in flags[0] instead.
enum ContactFlag : uint32_t {
    kOverEntries = 1,    // a bin holds more (cell, shape) entries than bin_slots
    kOverContacts = 2,   // more contacts than contact_cap
    kOverBins = 4,       // the grid needs more bins than bin_cap
    kNonFinite = 8,      // a shape has a non-finite bounding box (informational)
    kOverSpan = 16,      // a shape spans more cells than allowed: coarsen the grid
    kOverCandidates = 32 // more narrow-phase candidates than cand_cap
};

constexpr float kBoxQuanta = 32000.f;  // quantization steps of shape boxes across the contact grid's extent

// Counters of the contact pipeline (ContactBufs::counts).
enum ContactCount : int {
    kCand,        // candidates of the last build (may exceed cand_cap)
    kKept,        // candidates kept by its filter
    kEntries,     // its cell entries
    kLargestBin,  // its largest bin count above bin_slots (0 when every bin fitted)
    kOccupied,    // its bins holding two or more entries
    kUnits,       // its units of pair work
    kContacts,    // contacts of the last evaluation (may exceed contact_cap)
    kContactCounts
};

// Contact forces and energy of one node, summed as integers so that the sums are exact and do
// not depend on their order: a value is a signed multiple of a quantum (2^force_e0, 2^energy_e0),
// its bits spread over limbs of 32 bits with room for 2^31 additions each.  The gather reads the
// record of a node whose n_count is not zero and clears both.
constexpr int kSumLimbs = 4;
constexpr int kSumQuantumBits = 90;  // the quantum lies 2^-90 below stiffness times the reference length
struct NodeContact {
    long long f[3][kSumLimbs];
    long long energy[kSumLimbs];  // of the contacts whose lower shape's first node this is
    unsigned long long pen;       // their largest penetration (bits of a non-negative double)
    unsigned long long pad_;
};
// n_count: force items in the low 31 bits, contacts counted at this node from bit 32 on; this
// bit: a contact's force or energy was not finite.
constexpr unsigned long long kContactNotFinite = 1ULL << 31;

struct ContactBufs {
    // per shape (S = N + B)
    uint4* rec;             // [S] pair-test record: quantized AABB (3 words), packed first cell
    int* grid;              // [16]: origin i,j,k; dims i,j,k; mode; valid; bins; bins needed;
                            //       box quantization scale x,y,z and origin x,y,z (float bits)
    uint32_t* flags;        // [5]: [0] ContactFlag bits of this evaluation, [1] candidate list
                            //      rebuilt by this evaluation, [2] rebuild forced (by the host,
                            //      or by a build that overflowed), [3] the pair pass's
                            //      cursor, [4] builds since allocation.  [0] and
                            //      [1] are zero between evaluations (cleared by the gather)
    uint32_t* counts;       // [kContactCounts]
    float4* xref;           // [N] node positions (FP32, rounded down) when the list was built
    // bins of fixed capacity: the shapes of bin b at bin_items[b * bin_slots ...]
    long long bin_cap;
    int bin_slots;          // entries a bin holds, a power of two
    uint32_t* bin_count;    // [bin_cap+1] entries counted per bin (may exceed bin_slots); zero
                            //             between builds
    uint32_t* bin_items;    // [bin_cap * bin_slots]
    uint2* units;           // [pair_units()] (bin, chunk of the bin's shapes) with an entry
    // narrow-phase candidates: one flat list, appended by the pair grid's warps in chunks
    int pair_blocks;        // blocks of the pair grid (8 warps each)
    int shape_blocks;       // most blocks of the box kernel
    long long cand_cap;     // candidate slots, a multiple of 32
    uint2* cand;            // [cand_cap] (lower shape, higher shape)
    uint2* cand2;           // [cand_cap] the ones that can reach contact before the next build
    long long contact_cap;
    uint32_t* c_a;          // lower shape index
    uint32_t* c_b;          // higher shape index
    unsigned long long* n_count;  // [N] zero between evaluations
    NodeContact* n_sum;           // [N] zero between evaluations
    int force_e0, energy_e0;      // exponents of the sums' quanta
};

// The candidate-list decision of an evaluation, made by its state and center kernels: rebuild
// when some node has moved farther than the skin since the last build, or always with no skin,
// or when forced (flags[2]); then the grid of the build.
struct BuildArgs {
    const float4* xref;
    uint32_t* flags;   // null: no self-contact
    uint32_t* counts;
    int* grid;
    double pad, cell;  // shape boxes reach at most pad beyond the nodes; grid cell
    long long bin_cap;
    float skin;        // <= 0: rebuild at every evaluation
};

// per node block: gravity E, platen E, reaction, max penetration, contacts, self-contact E,
// sum of squared free gradient entries, max |free gradient entry|
constexpr int kNodeParts = 8;
constexpr int kFinPartDoubles = 32 * 11;  // per instance: 32 first-stage blocks x 11 totals
// Nodes up to which the gather writes the gradient to page-locked memory as well: a copy to the
// caller's array takes 8 us whatever its size, the stores and the host's copying 3 us at 1024 nodes
// (cubic+BCC 855 nodes 63 -> 58 us a call, 1241 65 -> 61, 1729 69 -> 66, 3059 even, 4941 73 -> 80).
constexpr int kHostGradNodes = 2048;
// Beams up to which trial states go the same way (three copies of 8 us): 6x6x6 cubic, 882 beams,
// 102 -> 75 us a call with both.
constexpr int kHostTrialBeams = 2048;
constexpr int kFinSingle = 768;  // block partials one block sums: six per thread

struct EvalBufs {
    double4_32a* x;             // [N]
    double4_32a* R;             // [N]
    double4_32a* M;             // [4N] R in fixed point: rows of R - I with their exponent, quaternion (FxRot)
    float4* xf_lo;              // [N] position rounded down to single precision
    float4* xf_hi;              // [N] position rounded up
    double* slot;           // [15B] per beam 12: (-F, Ga), added to node a, then (+F, Gb), added to
                            //   node b: entry 2 beam + role, the incidence list's numbering
    double* part_state;     // [9 * n_eblk] sum, -min, max of x per block
    double* part_beam;      // [3 * nb_beams]
    unsigned* err;          // [1] a kernel's bounded wait gave up (the host reports it)
    double* part_node;      // [kNodeParts * 2 n_eblk] per gather block
    unsigned* done;         // [I] blocks that have arrived; zero between kernels
    double* part_fin;       // [I * kFinPartDoubles] first-stage totals of the finalize
    double* cen;            // [9 (I + 1)] per instance mean, min, max of the node positions (min/max
                            //   in the contact grid's frame); then min/max over all instances
    double* cforce;         // [2 I] centering force of the instance on each node (x, z)
    double* tops;           // [I] platen height per instance
    EvalOut* out;           // [I]
    // the host's page-locked side of both, which the kernels read and write themselves: an
    // evaluation needs no copies for them (null: the device's only)
    const double* tops_host;
    EvalOut* out_host;
    double* grad_host;      // [6 N] the gradient too, for lattices of up to kHostGradNodes
    double* trial_next;     // [7B] SoA
    double* trial_aux;      // [7B] SoA
    uint8_t* trial_flags;   // [3B] SoA
    // mixed-precision form
    float* slotf;           // [12B] as slot
    float* trial_nextf;     // [7B] SoA
    float* trial_auxf;      // [7B] SoA
};

// Per-beam data of the mixed-precision form (objective_mixed.cu), float4 SoA.
struct MixedBeams {
    float4* B0;  // base chord d0 (FP32-rounded), c0 = |d0|^2 - L0^2
    float4* B1;  // base shear vector d_a0 - t0, L0
    float4* B2;  // base shear vector d_b0 - t0, |d0|
    float4* B5;  // base relative rotation Q0 as (w - 1, v)
    float4* P0;  // plastic: epsp, alpha, alphaB, alphaT
    float4* P1;  // plastic: rotp; radius
    // Section constants.  When every beam's area, I and J are the circular section's
    // (pi r^2, pi r^4 / 4, 2 I, MC/src/sim.cpp:115) they are formed in the kernel from r and
    // L0 with the factors below and C0/C1 stay null; otherwise they are streamed.
    float4* C0;  // kb, kt, my, ty (streamed form only)
    float4* C1;  // cs, area L0, area, area L0 yield (streamed form only)
    float4* ic;  // [I] per instance: yield, yield pi/4, yield pi/(2 sqrt 3), yield pi
    float4 kg;   // E pi/4, G pi/2, shear G pi/2, pi
};
// Per-node data of the mixed-precision form.
struct MixedNodes {
    float4* UE;   // [2 N] per node, one 32-byte sector: the increment displacement s t since
                  // the base state, then the increment rotation exp(r) as (w - 1, v)
    float4* R0f;  // base orientation (w, x, y, z)
};

// ---- launch accounting -------------------------------------------------------------------
extern std::atomic<long long> g_launch_count;
inline void note_launches(int k) { g_launch_count += k; }

// ---- launchers (objective.cu) ----------------------------------------------------------
void launch_state(const DevTopo& t, const PhysParams& p, const double* z, const double* base_x, const BuildArgs& b, EvalBufs& e,
                  cudaStream_t s);
void launch_rotations(const DevTopo& t, const double* z, const double* base_r, EvalBufs& e, cudaStream_t s);
// Occupancy variants of the beam kernels and the gather (CTAs per SM the register allocation
// allows; the arithmetic is the same in every variant).  Variant 0 is the default.
enum class ShapeKernel { kBeams, kBeamsMixed, kGather };
int shape_variants(ShapeKernel k);
int shape_blocks(ShapeKernel k, int variant);
int beams_mixed_variants();
// Once per context, outside any stream capture: the staged variants' shared-memory limit and
// the SM count that sizes their persistent grid.
void prepare_beams_mixed(int device);
int beams_mixed_blocks(int variant);
void launch_beams(const DevTopo& t, const Material& m, const double* plastic, int trials,
                  EvalBufs& e, cudaStream_t s, int variant = 0);
// Gather blocks [first, first + blocks) of the 2 n_eblk (all by default).
void launch_gather(const DevTopo& t, const PhysParams& p, const ContactBufs* c, double* grad,
                   EvalBufs& e, cudaStream_t s, int variant = 0, int first = 0, int blocks = -1);
void launch_finalize(const DevTopo& t, const PhysParams& p, double* grad, EvalBufs& e, cudaStream_t s);
// base state <- current state, plastic <- trial (plastic == nullptr skips it) for the
// instances with mask[i] != 0 (mask == nullptr: all)
void launch_commit(const DevTopo& t, const uint8_t* mask, const EvalBufs& e, double* base_x, double* base_r,
                   double* plastic, cudaStream_t s);
void launch_center(const DevTopo& t, const PhysParams& p, const BuildArgs& b, EvalBufs& e, cudaStream_t s);
// Per-beam arrays (7 values, 3 flags; structure of arrays) to and from consecutive values per beam.
void launch_records7(long long B, const double* soa, double* aos, cudaStream_t s);
// Trial states as records in 15 B doubles: the slots (which the gather has read by then) or
// page-locked memory.
struct TrialRecords {
    double *next, *aux;  // [7 B]
    uint8_t* flags;      // [3 B]
    TrialRecords(double* mem, long long B) : next(mem), aux(mem + 7 * B), flags(reinterpret_cast<uint8_t*>(mem + 14 * B)) {}
};
void launch_trial_records(long long B, const EvalBufs& e, bool mixed, const TrialRecords& r, cudaStream_t s);
void launch_from_records7(long long B, const double* aos, double* soa, cudaStream_t s);
void launch_gather_mixed(const DevTopo& t, const PhysParams& p, const ContactBufs* c, double* grad, EvalBufs& e,
                         cudaStream_t s, int variant = 0, int first = 0, int blocks = -1);

// ---- mixed-precision form (objective_mixed.cu) ------------------------------------------
void launch_state_mixed(const DevTopo& t, const PhysParams& p, const double* z, const double* base_x,
                        const MixedNodes& mn, const BuildArgs& b, EvalBufs& e, cudaStream_t s);
void launch_beams_mixed(const DevTopo& t, const Material& m, const MixedBeams& mb, const MixedNodes& mn, int trials,
                        EvalBufs& e, cudaStream_t s, int variant = 0);
void launch_rebase_mixed(const DevTopo& t, const double* base_x, const double* base_r, MixedBeams& mb,
                         MixedNodes& mn, cudaStream_t s);
// The streamed section constants (mb.C0/C1, when allocated), once per upload.
void launch_mixed_constants(const DevTopo& t, MixedBeams& mb, cudaStream_t s);
// plastic state of the mixed form from the FP64 SoA array (trial32 == nullptr, all beams) or
// from an FP32 trial (the beams of the instances with mask[i] != 0; mask == nullptr: all)
void launch_plastic_mixed(const DevTopo& t, const uint8_t* mask, const double* plastic64, const float* trial32,
                          MixedBeams& mb, cudaStream_t s);
void launch_plastic_mixed_to_f64(const DevTopo& t, const uint8_t* mask, const MixedBeams& mb, double* plastic64,
                                 cudaStream_t s);
// out6[6 i..]: per instance sum|epsp|, max|epsp|, sum|rotp|, max|rotp|, #|epsp|>1e-5, #|rotp|>1e-4
// (part: 6 doubles per beam block)
void launch_plastic_stats(const DevTopo& t, const double* plastic, double* part, double* out6, cudaStream_t s);

// ---- contact pipeline (contact.cu) ------------------------------------------------------
// Blocks of the pair grid for a model of `shapes` shapes (8 warps each); shared: beside the FP64 beam kernel.
int contact_pair_blocks(long long shapes, bool shared);
// Units of pair work that `bins` bins of `slots` entries can hold.
long long pair_units(long long bins, int slots);
// The whole broad/narrow phase after the state and center kernels: bins, pairs and filtered
// candidates (only when the list is rebuilt), contacts and their forces.
// pairs_begin / pairs_end (may be null) are recorded around the pair enumeration.
void launch_contacts(const DevTopo& t, const PhysParams& p, const EvalBufs& e, ContactBufs& c, float skin,
                     cudaStream_t s, cudaEvent_t pairs_begin = nullptr, cudaEvent_t pairs_end = nullptr);

// ---- L-BFGS vector kernels (lbfgs.cu), all instances of a context per launch --------------
// Operations an instance takes part in during one solver step (SolveCtl::flags).
enum SolveOp : int {
    kOpDirection = 1,      // two-loop direction from g, clamp, <g, p>
    kOpSteepest = 2,       // p = clamp(-g), <g, p>
    kOpZero = 4,           // z = 0
    kOpRestore = 8,        // z = best
    kOpKeepBest = 16,      // best = z
    kOpCandidate = 32,     // zeval = z + step p
    kOpEvalAtZ = 64,       // zeval = z
    kOpFinal = 128,        // zfinal = z
    kOpTakeGrad = 256,     // g = geval
    kOpAccept = 512,       // s, y, curvature dots, z = zeval, g = geval
    kOpPair = 1024,        // with kOpAccept: store (s, y) in history slot `target`
    kOpKeepBestAfter = 2048, // with kOpAccept: best = the accepted z
    kOpResetHistory = 4096   // the history starts empty (a new minimization)
};
// Per-instance solver control, written by the host before each step.  The history state
// (pairs held m, oldest slot head) lives on the device (int2 per instance) and is filled in
// by the kernels.
struct SolveCtl {
    double step;       // line-search step of the candidate
    int flags;         // SolveOp bits
    int m, head;       // (device history, loaded by the kernels)
    int pad_;
};
// The solver's vectors and scalars on the device: history H slots of `stride` doubles.
struct LbfgsBufs {
    double *z, *best, *zeval, *zfinal, *p, *g, *S, *Y;
    const double* geval;
    long long stride;
    int H;               // history slots (at least 1)
    int2* hist;          // [I] history pairs held, oldest slot
    double* rho;         // [I H] 1 / <s, y> per slot
    double* gram;        // [I H H] <s_i, y_j> at [slot i][slot j], pair i not newer than j
    double *alpha, *coef;  // [I H] the two loops' coefficients, oldest pair first
    double* h0;          // [I] initial scale of the newest pair: clamp(s.y / y.y, 1e-7, 1e4), else 0.1
    double* dg;          // [I] <g, p>
    double* part;        // [lbfgs_part_doubles] block partials
    unsigned* done;      // [4 I] blocks that have arrived, per pass; zero between passes
    double mt, mr;       // largest translation (in units of the scale) and rotation of a step
};
struct MzStatus;  // minimize.h
struct MzDev;
size_t lbfgs_part_doubles(int n_sblk, int H);
// Nodes per solver block of an instance of n nodes.
int solve_block_nodes(int n);
// Two-loop recursion (sim.cpp:184-187) into p for the kOpDirection instances, then
// p = clamp(lock(-p)) and dg = <g, p>; where not dg < 0, and for the kOpSteepest instances (the
// retry, sim.cpp:193-196), p = clamp(lock(-g)) with the history cleared (sim.cpp:191).
// st: the loop's status, for its stage times.
void bl_direction(const DevTopo& t, const SolveCtl* ctl, const LbfgsBufs& v, cudaStream_t s, MzStatus* st = nullptr);
// kOpResetHistory / kOpZero / kOpRestore / kOpKeepBest / kOpCandidate / kOpEvalAtZ / kOpFinal as ctl
// says, or as the device-resident minimizers of d say.
void bl_prepare(const DevTopo& t, const SolveCtl* ctl, const LbfgsBufs& v, cudaStream_t s, const MzDev* d = nullptr);
// kOpTakeGrad / kOpAccept (+kOpPair, kOpKeepBestAfter), h0 and the history
// update of the accepted instances (sim.cpp:205-206).
void bl_accept(const DevTopo& t, const SolveCtl* ctl, const LbfgsBufs& v, cudaStream_t s);

}  // namespace mcg
