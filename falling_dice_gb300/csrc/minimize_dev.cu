// minimize_dev.cu -- the stage kernels of the device-resident solver round.
//
// One round of Simulator::minimize (MC/src/sim.cpp:174-211) for every instance is the body of a
// CUDA-graph WHILE node: directions, vector preparation (what to evaluate), the evaluation, the
// decisions, accept steps.  Every kernel reads from the control records which instances it has
// work for; kernels without work return at once.  (IF nodes around the directions, the retry and
// the accept step cost more than that: a round of the 6x6x6 cubic specimen took 81 us with them and
// three more stage kernels, 70 us without.)  The decision functions are minimize.h's, the ones
// the host-stepped solver calls.  The loop runs while some instance is still minimizing and none
// has finished (the host commits finished instances and starts their next increment), up to a
// round cap.  No kernel waits on another: the graph orders them.
#include "minimize.h"

namespace mcg {

namespace {

constexpr int kMzThreads = 256;  // one block walks all instances

__global__ void __launch_bounds__(kMzThreads) k_mz_begin(MzDev d) {
    for (int i = threadIdx.x; i < d.I; i += blockDim.x) d.ctl[i] = SolveCtl{0.0, mz_stage_direction(d.mins[i]), 0, 0, 0};
    if (threadIdx.x == 0) *d.status = MzStatus{0, 0, 0, 0, 0, 0, 0, 0};
}

__global__ void __launch_bounds__(kMzThreads) k_mz_decide(MzDev d, MzParams p, cudaGraphConditionalHandle h_loop) {
    if (threadIdx.x == 0) stage_mark(d.status, &d.status->t_eval);
    // an evaluation that overflowed a contact buffer decided nothing: the host grows the buffers
    // and the next launch repeats the round's evaluation, its directions standing
    const bool overflow = d.out[0].overflow;
    int done = 0, running = 0;
    for (int i = threadIdx.x; i < d.I; i += blockDim.x) {
        Minimizer s = d.mins[i];
        int post = 0, dir = 0;
        if (overflow) {
            mz_directed(s);
        } else {
            post = mz_stage_decide(p, s, d.out[i], d.dg[i]);
            dir = mz_stage_direction(s);
        }
        d.mins[i] = s;
        d.ctl[i] = SolveCtl{0.0, dir, 0, 0, 0};
        d.ctl[d.I + i] = SolveCtl{0.0, post, 0, 0, 0};
        done |= s.phase == Minimizer::kDone;
        running |= s.phase != Minimizer::kDone && s.phase != Minimizer::kIdle;
    }
    done = __syncthreads_or(done);
    running = __syncthreads_or(running);
    if (threadIdx.x == 0) {
        if (overflow) {
            d.status->overflow = 1;
            cudaGraphSetConditional(h_loop, 0u);
            return;
        }
        const int rounds = ++d.status->rounds;
        if (done) d.status->done = 1;
        cudaGraphSetConditional(h_loop, (!done && running && rounds < d.round_cap) ? 1u : 0u);
    }
}

}  // namespace

void launch_mz_begin(const MzDev& d, cudaStream_t s) {
    k_mz_begin<<<1, kMzThreads, 0, s>>>(d);
    note_launches(1);
}

void launch_mz_decide(const MzDev& d, const MzParams& p, cudaGraphConditionalHandle h_loop, cudaStream_t s) {
    k_mz_decide<<<1, kMzThreads, 0, s>>>(d, p, h_loop);
    note_launches(1);
}

}  // namespace mcg
