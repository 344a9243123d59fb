// Prediction streaming of the simulation engine on the device: the re-simulation that
// SimulationEngine::sendState (src/engine.cpp:55-264) runs on the host after every closed-
// loop step to show where the controller's plan leads, for every controller of a batch in
// one launch.
//
//   mppi_predict   MPPI (engine.cpp:73-166): from the state after the step, under every
//                  hypothesis theta, the controller's plan (its chosen plan with the
//                  warm-start shift the next step will apply, the engine's h_nominal) is
//                  rolled out for the horizon with the belief update and branching on
//                  (environmentStep<true, true, false>), noise off: the initial branch, the
//                  positions of every agent at every step (repeated after a terminal step),
//                  the ego actions taken, the branch taken and when, why and when it
//                  stopped, and the discounted running + terminal cost (the engine prints
//                  it, engine.cpp:139-141).
//   pr_predict     PR-MPPI (engine.cpp:167-240): from the state before the step, the new
//                  nominal plan under every hypothesis and the robust plan under the last
//                  one (environmentStep<false, false, false>), noise off, with the running,
//                  safety and terminal cost of PRMPPIstateCost / PRMPPIsafetyCost /
//                  PRMPPIfinalCost evaluated on the predicted states (the engine evaluates
//                  them on the unchanged current state, engine.cpp:221-222, and only prints
//                  them).
// One CTA per controller stages the track grids in shared memory; thread r computes row r
// (a hypothesis, or the robust plan).
#include <cstdio>

#include "common.cuh"
#include "instance.cuh"
#include "launch.h"
#include "pair_model.cuh"

namespace dr
{

namespace
{

// The engine re-simulates with applyNoise = false: no draws, every noise term zero.
struct NoNoise
{
    __device__ __forceinline__ void begin_step(uint32_t)
    {
    }
    __device__ __forceinline__ float next()
    {
        return 0.0f;
    }
    __device__ __forceinline__ float2 next2()
    {
        return make_float2(0.0f, 0.0f);
    }
};

// EventType of the reference (include/protocol.h:17-23) for a terminal step (parseTerm,
// engine.cpp:365-380)
__device__ __forceinline__ int eventOf(int term)
{
    return term == TERM_LOSE ? 0 : term == TERM_WIN ? 1 : 2;
}
constexpr int EVT_TRUNCATED = 3;

__device__ __forceinline__ void stageTrack(float* sg, EnvParams& sE, const float* grids, const EnvParams& env)
{
    for (int i = threadIdx.x; i < GRID_FLOATS; i += blockDim.x)
        sg[i] = grids[i];
    for (int i = threadIdx.x; i < ENV_HOST_WORDS; i += blockDim.x)
        ((float*)&sE)[i] = ((const float*)&env)[i];
    envDeviceTerms(sE, env, threadIdx.x, blockDim.x);
}

template <int NA> __device__ __forceinline__ void loadPredState(DState<NA>& s, const dr_sim_state& st, float L)
{
#pragma unroll
    for (int a = 0; a < NA; a++)
    {
        s.pos[2 * a] = st.pos[2 * a];
        s.pos[2 * a + 1] = st.pos[2 * a + 1];
        s.vel[2 * a] = st.vel[2 * a];
        s.vel[2 * a + 1] = st.vel[2 * a + 1];
        s.S[a] = st.S[a];
        s.lat[a] = st.lat_dist[a];
        s.laps[a] = st.laps[a];
    }
    s.locate(L);
}

template <int NA> __device__ __forceinline__ void putPositions(float* out, const DState<NA>& s)
{
#pragma unroll
    for (int k = 0; k < 2 * NA; k++)
        out[k] = s.pos[k];
}

} // namespace

template <int NOPP, int NTH>
__global__ void __launch_bounds__(128) mppi_predict(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in,
                                                    const dr_sim_state* __restrict__ states, const float* __restrict__ beliefs, int beliefStride,
                                                    PredictOut out, int nInst)
{
    constexpr int NA = NOPP + 1;
    __shared__ __align__(16) float sg[GRID_FLOATS];
    __shared__ EnvParams sE;
    const int inst = blockIdx.x;
    if (inst >= nInst)
        return;
    const MppiDev& D = insts[inst];
    const MppiIn& I = in[inst];
    stageTrack(sg, sE, D.grids, D.env);
    __syncthreads();
    const int th = threadIdx.x;
    if (th >= NTH)
        return;
    const EnvParams& E = sE;
    const Track tr = trackIn(sg);
    const int T = D.cfg.T, nbp = NTH + 1;
    const size_t row = (size_t)inst * NTH + th;
    float* pos = out.pos + row * out.tStride * 2 * NA;
    float* act = out.act + row * out.tStride * 2;
    int* rec = out.rec + row * PREDICT_RECORD;
    // the controller's plan as the engine holds it: the chosen plan with the pending
    // warm-start shift of branch pendBranch (mppi_controller.cu:430-436)
    const float* plan = (I.pendBranch >= 0 && !I.pendUseNew) ? D.prevDense : D.dense;
    const int shiftB = (I.pendBranch >= 0 && I.pendBranch < nbp) ? I.pendBranch : -1;

    DState<NA> s;
    loadPredState<NA>(s, states[inst], E.trackLength);
    BState<NTH> bs;
    const float* belief = beliefs + (size_t)inst * beliefStride;
#pragma unroll
    for (int i = 0; i < NTH; i++)
        bs.belief[i] = belief[i];
    // initBranchState (state.h:154-163)
    bs.predTheta = findConfident<NTH>(bs.belief, D.cfg.minConf);
    bs.branchingTime = bs.predTheta == 0 ? -1 : 0;
    rec[0] = bs.predTheta;
    NoNoise rng;
    float cost = 0.0f, decay = 1.0f;
    int tOrigin = 0, stopTime = -1, stopReason = EVT_TRUNCATED;
    int t = 0;
    for (; t < T; t++)
    {
        const int b = bs.predTheta, local = t - tOrigin;
        float e0 = 0.0f, e1 = 0.0f;
        if (b == shiftB)
        {
            if (local + 1 < T)
            {
                e0 = plan[(b * T + local + 1) * 2];
                e1 = plan[(b * T + local + 1) * 2 + 1];
            }
        }
        else
        {
            e0 = plan[(b * T + local) * 2];
            e1 = plan[(b * T + local) * 2 + 1];
        }
        act[t * 2] = e0;
        act[t * 2 + 1] = e1;
        bool branched = false;
        StepOut o = envStep<NOPP, NTH, true, true, false, true>(t, th, tr, E, e0, e1, s, bs, branched, D.cfg.minConf, rng);
        if (branched)
            tOrigin = t + 1;
        putPositions<NA>(pos + (size_t)t * 2 * NA, s);
        cost += stateCost(o, E, D.cfg.w) * decay;
        decay *= DECAY;
        if (o.term != TERM_NONE)
        {
            stopTime = t;
            stopReason = eventOf(o.term);
            break;
        }
    }
    // after a terminal step the engine repeats the last state and leaves the actions zero
    for (int u = t + 1; u < T; u++)
    {
        putPositions<NA>(pos + (size_t)u * 2 * NA, s);
        act[u * 2] = 0.0f;
        act[u * 2 + 1] = 0.0f;
    }
    cost += finalCost<NOPP>(s, E, D.cfg.w.finalAdvWeight, D.cfg.w.finalOppAdvWeight);
    rec[1] = bs.branchingTime;
    rec[2] = bs.predTheta;
    rec[3] = stopReason;
    rec[4] = stopTime;
    out.cost[row] = cost;
}

// mppi_predict with one opponent: a pair of lanes per hypothesis (pair_model.cuh), one warp a
// controller, the track, the environment and the plan staged in shared memory. What bounds it is
// the latency of its T dependent steps; a lane per agent halves their instructions, and the
// plan no longer comes from global memory within them. Four controllers (B200, 1965 MHz): T 60, two
// hypotheses 227 -> 129 us, T 61, eight 525 -> 354; a whole host call of one, T 60: 269 -> 144.
// The staging is plain loads, by PREDICT_THREADS threads of which one warp goes on: it waits for
// nothing that could fail to arrive, and a prediction has no status to report that in. It takes the
// time that a bulk copy took (129 / 131 us); one warp's loads take 6 us more, and without the bound
// of one CTA an SM eight hypotheses get 105 registers a thread and take 373.
constexpr int PREDICT_THREADS = 256;

template <int NTH>
__global__ void __launch_bounds__(PREDICT_THREADS, 1) mppi_predict_pair(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in,
                                                        const dr_sim_state* __restrict__ states, const float* __restrict__ beliefs, int beliefStride,
                                                        PredictOut out, int nInst)
{
    static_assert(2 * NTH <= 32, "a warp holds the pairs");
    __shared__ __align__(16) float sg[GRID_FLOATS];
    __shared__ __align__(16) float plan[(NTH + 1) * DR_MAX_T * 2];
    __shared__ EnvParams sE;
    constexpr unsigned ALL = 0xffffffffu;
    const int inst = blockIdx.x;
    if (inst >= nInst)
        return;
    const MppiDev& D = insts[inst];
    const MppiIn& I = in[inst];
    const int T = D.cfg.T, nbp = NTH + 1;
    // the controller's plan as the engine holds it: the chosen plan with the pending
    // warm-start shift of branch pendBranch (mppi_controller.cu:430-436)
    const float4* planFrom = (const float4*)((I.pendBranch >= 0 && !I.pendUseNew) ? D.prevDense : D.dense);
    for (int i = threadIdx.x; i < GRID_FLOATS / 4; i += PREDICT_THREADS)
        ((float4*)sg)[i] = ((const float4*)D.grids)[i];
    for (int i = threadIdx.x; i < (nbp * T + 1) / 2; i += PREDICT_THREADS) // (the plans' storage is whole float4s)
        ((float4*)plan)[i] = planFrom[i];
    for (int i = threadIdx.x; i < ENV_HOST_WORDS; i += PREDICT_THREADS)
        ((float*)&sE)[i] = ((const float*)&D.env)[i];
    __syncthreads();
    envDeviceTerms(sE, sE, threadIdx.x, PREDICT_THREADS);
    __syncthreads();
    if (threadIdx.x >= 32)
        return;
    const int shiftB = (I.pendBranch >= 0 && I.pendBranch < nbp) ? I.pendBranch : -1;
    const int role = threadIdx.x & 1, th = (threadIdx.x >> 1) % NTH;
    const bool valid = threadIdx.x < 2 * NTH;
    const size_t row = (size_t)inst * NTH + th;
    float* pos = out.pos + row * out.tStride * 4 + 2 * role; // the caller's: aligned as floats are
    float* act = out.act + row * out.tStride * 2;
    int* rec = out.rec + row * PREDICT_RECORD;
    const EnvParams& E = sE;
    const Track tr = trackIn(sg);
    const dr_sim_state& st = states[inst];
    DState<1> s;
    s.pos[0] = st.pos[2 * role];
    s.pos[1] = st.pos[2 * role + 1];
    s.vel[0] = st.vel[2 * role];
    s.vel[1] = st.vel[2 * role + 1];
    s.S[0] = st.S[role];
    s.lat[0] = st.lat_dist[role];
    s.laps[0] = st.laps[role];
    s.locate(E.trackLength);
    BState<NTH> bs;
    const float* belief = beliefs + (size_t)inst * beliefStride;
#pragma unroll
    for (int i = 0; i < NTH; i++)
        bs.belief[i] = belief[i];
    // initBranchState (state.h:154-163)
    const int pred0 = findConfident<NTH>(bs.belief, D.cfg.minConf);
    bs.predTheta = pred0;
    bs.branchingTime = pred0 == 0 ? -1 : 0;
    float cost = 0.0f, decay = 1.0f;
    int tOrigin = 0, stopTime = -1, stopReason = EVT_TRUNCATED;
    bool active = valid;
    for (int t = 0; t < T; t++)
    {
        const unsigned mask = __ballot_sync(ALL, active);
        if (mask == 0u)
            break;
        if (!active)
            continue;
        const int b = bs.predTheta, local = t - tOrigin + (b == shiftB ? 1 : 0);
        const bool inside = local < T;
        const float e0 = inside ? plan[(b * T + local) * 2] : 0.0f, e1 = inside ? plan[(b * T + local) * 2 + 1] : 0.0f;
        bool branched = false;
        const StepOut o = pairStep<NTH, false, false>(mask, role, t, th, tr, E, e0, e1, 0.0f, 0.0f, s, bs, branched, D.cfg.minConf, PairNoise{});
        if (branched)
            tOrigin = t + 1;
        pos[4 * t] = s.pos[0];
        pos[4 * t + 1] = s.pos[1];
        act[2 * t + role] = role ? e1 : e0;
        cost += stateCost(o, E, D.cfg.w) * decay;
        decay *= DECAY;
        if (o.term != TERM_NONE)
        {
            stopTime = t;
            stopReason = eventOf(o.term);
            active = false;
        }
    }
    DState<2> both; // the final cost reads both agents' arc lengths and laps
    pairBoth(ALL, role, s.S[0], both.S[0], both.S[1]);
    pairBoth(ALL, role, s.laps[0], both.laps[0], both.laps[1]);
    if (!valid)
        return;
    // after a terminal step the engine repeats the last state and leaves the actions zero
    for (int u = stopTime < 0 ? T : stopTime + 1; u < T; u++)
    {
        pos[4 * u] = s.pos[0];
        pos[4 * u + 1] = s.pos[1];
        act[2 * u + role] = 0.0f;
    }
    if (role != 0)
        return;
    cost += finalCost<1>(both, E, D.cfg.w.finalAdvWeight, D.cfg.w.finalOppAdvWeight);
    rec[0] = pred0;
    rec[1] = bs.branchingTime;
    rec[2] = bs.predTheta;
    rec[3] = stopReason;
    rec[4] = stopTime;
    out.cost[row] = cost;
}

template <int NOPP, int NTH>
__global__ void __launch_bounds__(128) pr_predict(const PrDev* __restrict__ insts, const dr_sim_state* __restrict__ prevStates, PredictOut out, int nInst)
{
    constexpr int NA = NOPP + 1;
    constexpr int ROWS = NTH + 1;
    __shared__ __align__(16) float sg[GRID_FLOATS];
    __shared__ EnvParams sE;
    const int inst = blockIdx.x;
    if (inst >= nInst)
        return;
    const PrDev& D = insts[inst];
    stageTrack(sg, sE, D.grids, D.env);
    __syncthreads();
    const int j = threadIdx.x;
    if (j >= ROWS)
        return;
    const EnvParams& E = sE;
    const Track tr = trackIn(sg);
    const int T = D.cfg.T;
    const int theta = j < NTH ? j : NTH - 1;
    const float* plan = j < NTH ? D.nom : D.rob;
    const size_t row = (size_t)inst * ROWS + j;
    float* pos = out.pos + row * out.tStride * 2 * NA;
    float* act = out.act + row * out.tStride * 2;
    int* rec = out.rec + row * PREDICT_RECORD;

    DState<NA> s;
    loadPredState<NA>(s, prevStates[inst], E.trackLength);
    BState<NTH> bs{};
    NoNoise rng;
    const SafetyMargin margin = safetyMargin(E, D.cfg.collDistFactor);
    float cost = 0.0f, safe = -INFINITY, decay = 1.0f;
    int stopTime = -1, stopReason = EVT_TRUNCATED;
    int t = 0;
    for (; t < T; t++)
    {
        const float e0 = plan[t * 2], e1 = plan[t * 2 + 1];
        act[t * 2] = e0;
        act[t * 2 + 1] = e1;
        bool branched = false;
        StepOut o = envStep<NOPP, NTH, false, false, false, false>(t, theta, tr, E, e0, e1, s, bs, branched, 0.0f, rng);
        safe = fmaxf(safe, prSafetyCost(o, margin));
        cost += prStateCost(o, E, D.cfg.boundaryThresholdFactor, D.cfg.boundaryCost, D.cfg.winCost, D.cfg.oppWinCost) * decay;
        decay *= DECAY;
        putPositions<NA>(pos + (size_t)t * 2 * NA, s);
        if (o.term != TERM_NONE)
        {
            stopTime = t;
            stopReason = eventOf(o.term);
            break;
        }
    }
    for (int u = t + 1; u < T; u++)
    {
        putPositions<NA>(pos + (size_t)u * 2 * NA, s);
        act[u * 2] = 0.0f;
        act[u * 2 + 1] = 0.0f;
    }
    cost += finalCost<NOPP>(s, E, D.cfg.finalAdvWeight, D.cfg.finalOppAdvWeight);
    rec[0] = 0;
    rec[1] = -1;
    rec[2] = 0;
    rec[3] = stopReason;
    rec[4] = stopTime;
    out.cost[row] = cost + (safe > 0.0f ? D.cfg.safetyWeight : 0.0f);
}

#define DR_PRED_DISPATCH(NOPP_, NTH_, CALL)                                                                                                          \
    switch (NOPP_ * 16 + NTH_)                                                                                                                       \
    {                                                                                                                                                \
    case 1 * 16 + 1: CALL(1, 1); break;                                                                                                              \
    case 1 * 16 + 2: CALL(1, 2); break;                                                                                                              \
    case 1 * 16 + 4: CALL(1, 4); break;                                                                                                              \
    case 1 * 16 + 8: CALL(1, 8); break;                                                                                                              \
    case 2 * 16 + 2: CALL(2, 2); break;                                                                                                              \
    default: return cudaErrorInvalidValue;                                                                                                           \
    }

cudaError_t launchMppiPredict(cudaStream_t stream, int nopp, int nth, const MppiDev* insts, const MppiIn* in, const dr_sim_state* states,
                              const float* beliefs, int beliefStride, const PredictOut& out, int nInst)
{
    switch (nopp * 16 + nth)
    {
    case 1 * 16 + 1: mppi_predict_pair<1><<<nInst, PREDICT_THREADS, 0, stream>>>(insts, in, states, beliefs, beliefStride, out, nInst); break;
    case 1 * 16 + 2: mppi_predict_pair<2><<<nInst, PREDICT_THREADS, 0, stream>>>(insts, in, states, beliefs, beliefStride, out, nInst); break;
    case 1 * 16 + 4: mppi_predict_pair<4><<<nInst, PREDICT_THREADS, 0, stream>>>(insts, in, states, beliefs, beliefStride, out, nInst); break;
    case 1 * 16 + 8: mppi_predict_pair<8><<<nInst, PREDICT_THREADS, 0, stream>>>(insts, in, states, beliefs, beliefStride, out, nInst); break;
    case 2 * 16 + 2: mppi_predict<2, 2><<<nInst, 128, 0, stream>>>(insts, in, states, beliefs, beliefStride, out, nInst); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launchPrPredict(cudaStream_t stream, int nopp, int nth, const PrDev* insts, const dr_sim_state* prevStates, const PredictOut& out, int nInst)
{
#define CALL(P, Q) pr_predict<P, Q><<<nInst, 128, 0, stream>>>(insts, prevStates, out, nInst)
    DR_PRED_DISPATCH(nopp, nth, CALL)
#undef CALL
    return cudaGetLastError();
}

} // namespace dr
