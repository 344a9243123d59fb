// MPPI control-step kernels (reference: src/kernels.cu; host sequence
// src/mppi_controller.cu:250-466).
//
//   mppi_prologue   warm-start shift decided by the previous step (mppi_controller.cu:
//                   426-456 + shiftSplineKernel, kernels.cu:461-486), zeroes the
//                   verification histograms.
//   mppi_rollout    fused perturbation draw + rollout + running/terminal cost + branch
//                   bookkeeping (fullRolloutKernel, kernels.cu:34-171) + per-branch cost
//                   aggregation (aggregateBranchCostsKernel, kernels.cu:175-217). Two
//                   lanes (one opponent) or one thread (two) per (sample, hypothesis); the
//                   state stays in registers; the
//                   track, the control sequence and the spline basis are staged in shared
//                   memory by bulk copies; the perturbation is drawn from Philox instead of
//                   being read from a stored noise tensor.
//   mppi_update     per (branch plan, knot): masked minimum, exponential weights and the
//                   weighted average of the regenerated perturbations by one CTA or, with
//                   many samples and few knots, a cluster of up to eight
//                   (computeMaskedMinCostsKernel + weightedAverageKernelUnified,
//                   kernels.cu:221-408; the sums are accumulated in the reference's
//                   256-lane order); the last one of an instance to finish also does
//                   the spline interpolation and the clamp (kernels.cu:411-456).
//   mppi_ego_table  the ego's moves under a plan, which the verification's samples share,
//                   and its whereabouts (the clearance block).
//   mppi_verify     Monte-Carlo failure counts of the new and the previous plan
//                   (verifyNominalFailureKernel, kernels.cu:488-551), a launch a plan or
//                   both in one grid; samples that can no longer fail are not stepped on.
#include <cooperative_groups.h>

#include <cfloat>
#include <cstdio>
#include <type_traits>

#include "clear.cuh"
#include "common.cuh"
#include "instance.cuh"
#include "launch.h"
#include "pair_model.cuh"

namespace cg = cooperative_groups;

namespace dr
{

// Rollout block size. With one opponent a CTA is RB / 2 pairs of lanes, one per (sample,
// hypothesis) (rolloutTilePair); with two it is one thread per (sample, hypothesis).
#ifndef DR_ROLLOUT_BLOCK
#define DR_ROLLOUT_BLOCK 256
#endif
constexpr int RB = DR_ROLLOUT_BLOCK;
// CTAs per SM that the register allocation is sized for. A lane of a pair holds one
// agent's state: 64 registers a thread (4 CTAs) up to two hypotheses, 80 (3 CTAs) for four
// and eight, whose actions and beliefs spill 150 to 280 bytes at 64; 128 for two opponents.
// Measured (B200, 1965 MHz; the rollouts of the engine's front-end settings, K 65536 x 2 x T
// 80 spline controls / of two agents of K 3001 x 8 x T 61): 2 CTAs 1.48 / 0.94 ms, 3 CTAs
// 1.34 / 0.86, 4 CTAs 1.26 / 1.04.
template <int NOPP, int NTH> constexpr int rolloutMinBlocks()
{
    return NOPP == 1 ? (NTH <= 2 ? 4 : 3) : 512 / RB;
}
// Verification CTAs per SM that the register allocation is sized for (VERIFY_TILE = 512
// threads a CTA: 2 -> 64 registers a thread). Measured on the 4 x 2^17 x 40 verification
// of both plans (B200, 1965 MHz), exact arithmetic and a CTA barrier every step:
// 128-thread CTAs without the barrier 3.14 ms (72 registers); 128 with the barrier 3.05;
// 256 x 3 CTAs 2.90; 512 x 2 2.73; 1024 x 1 2.74. The barrier kept the warps of a CTA on
// the same step, where they fetched the same instructions of the then 55 KB kernel. The
// fast flavour with the ego tables is smaller and the barrier only held warps back: with
// it every 1 / 2 / 4 / 16 / 32 steps 1.292 / 1.272 / 1.200 / 1.180 / 1.174 ms, without it
// 1.171, so the warps now step on their own and leave the loop when their samples are done.
// The larger models (two opponents, or eight hypotheses) spill heavily at 64 registers
// and get one CTA per SM instead.
#ifndef VERIFY_MIN_BLOCKS
#define VERIFY_MIN_BLOCKS 2
#endif
template <int NOPP, int NTH> constexpr int verifyMinBlocks()
{
    return (NOPP == 1 && NTH <= 4) ? VERIFY_MIN_BLOCKS : 1;
}
constexpr int UB = 256; // update block size (the reference's reduction width)

__device__ __forceinline__ int infoPred(int v)
{
    return v >> 16;
}
__device__ __forceinline__ int infoTime(int v)
{
    return (int)(short)(v & 0xffff);
}

// Copies the host-filled part of EnvParams to shared memory and computes the
// device-filled part from there (from global memory its dependent reads were a chain of L2
// latencies at the start of every kernel); all threads of the CTA, and the caller's next
// __syncthreads publishes the terms.
__device__ __forceinline__ void copyEnv(EnvParams* dst, const EnvParams* src)
{
    for (int i = threadIdx.x; i < ENV_HOST_WORDS; i += blockDim.x)
        ((float*)dst)[i] = ((const float*)src)[i];
    __syncthreads();
    envDeviceTerms(*dst, *dst, threadIdx.x, blockDim.x);
}

__host__ __device__ __forceinline__ size_t align16(size_t x)
{
    return (x + 15) & ~(size_t)15;
}

// ---------------------------------------------------------------------------------------
// prologue: apply the previous step's warm-start shift
// ---------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) mppi_prologue(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in, int nInst)
{
    extern __shared__ float sh[];
    const int inst = blockIdx.x;
    if (inst >= nInst)
        return;
    const MppiDev& D = insts[inst];
    const MppiIn& I = in[inst];
    const int T = D.cfg.T, M = D.cfg.M, nbp = D.cfg.nth + 1;
    for (int i = threadIdx.x; i < 2 * T; i += blockDim.x)
        D.fail[i] = 0u;
    if (threadIdx.x < 4)
        D.stats[threadIdx.x] = 0;
    if (D.clear)
        for (int i = threadIdx.x; i < 2 * clearWords(D.cfg.H) / 4; i += blockDim.x)
            reinterpret_cast<float4*>(D.clear)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    const int b = I.pendBranch;
    if (b < 0 || b >= nbp)
        return;
    // prevDense := shift(chosen dense plan) on branch b (host shift, mppi_controller.cu:430-436)
    const float* src = I.pendUseNew ? D.dense : D.prevDense;
    const int n = nbp * T * 2;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        sh[i] = src[i];
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x)
    {
        int d = i & 1, t = (i >> 1) % T, bb = (i >> 1) / T;
        float v = sh[i];
        if (bb == b)
            v = (t < T - 1) ? sh[(bb * T + t + 1) * 2 + d] : 0.0f;
        D.prevDense[i] = v;
        D.dense[i] = v;
        if (!D.cfg.useSplines)
            D.knots[i] = v; // dense mode: the optimised sequence restarts from the shifted plan
    }
    if (D.cfg.useSplines)
    {
        // shiftSplineKernel on branch b (kernels.cu:461-486)
        float* old = sh + n;
        for (int i = threadIdx.x; i < M * 2; i += blockDim.x)
            old[i] = D.knots[(b * M) * 2 + i];
        __syncthreads();
        for (int i = threadIdx.x; i < M * 2; i += blockDim.x)
        {
            int dim = i & 1, newm = i >> 1;
            float sum = 0.0f;
            int tEval = D.cfg.knots[newm] + 1;
            if (tEval >= T)
                tEval = T - 1;
            for (int m = 0; m < M; m++)
                sum += D.B[tEval * M + m] * old[m * 2 + dim];
            D.knots[(b * M + newm) * 2 + dim] = sum;
        }
    }
}

// ---------------------------------------------------------------------------------------
// rollout + aggregation
// ---------------------------------------------------------------------------------------
struct RolloutSmem
{
    size_t env, grids, knots, B, vbuf, red, total;
};

// cols: columns of the spline buffer (a thread's, or a lane pair's, perturbed knots)
__host__ __device__ inline RolloutSmem rolloutLayout(int nbp, int T, int M, bool spl, int cols)
{
    auto a16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    RolloutSmem L;
    size_t off = 16; // mbarrier
    L.env = off;
    off = a16(off + sizeof(EnvParams));
    L.grids = off;
    off = a16(off + GRID_FLOATS * 4);
    L.knots = off;
    off = a16(off + (size_t)nbp * M * 2 * 4);
    L.B = off;
    if (spl)
        off = a16(off + (size_t)T * M * 4);
    L.vbuf = off;
    if (spl)
        off = a16(off + (size_t)((M + 3) & ~3) * 2 * cols * 4);
    L.red = off;
    off = a16(off + RB * 4);
    L.total = off;
    return L;
}

// One rollout tile: SPB samples x NTH hypotheses, a thread each, with the tile's
// instance already staged in shared memory; then the tile's aggregation.
template <int NOPP, int NTH, bool SPL, bool LOCK>
__device__ __forceinline__ void rolloutTile(const MppiDev& D, const MppiIn& I, const Tile& tile, int K, int T, int M, const EnvParams& E, const float* sGrid,
                                            const float* sKn, const float* sB, float* vbuf, float* red)
{
    constexpr int NA = NOPP + 1;
    const Track tr = trackIn(sGrid);

    const int th = threadIdx.x % NTH;
    const int sl = threadIdx.x / NTH;
    const int s = tile.s0 + sl;
    const bool valid = sl < tile.count;
    const float minConf = D.cfg.minConf;
    const uint32_t k0 = D.cfg.k0, k1 = D.cfg.k1, step = I.step;
    const float sig0 = D.cfg.sigma0, sig1 = D.cfg.sigma1;

    float belief0[NTH];
#pragma unroll
    for (int i = 0; i < NTH; i++)
        belief0[i] = I.belief[i];
    // initBranchState (state.h:154-163)
    const int pt0 = findConfident<NTH>(belief0, minConf);
    const int bt0 = pt0 == 0 ? -1 : 0;
    const bool compatible = (pt0 == 0 || pt0 == th + 1);

    float cost = INFINITY;
    int pt = pt0, bt = bt0;
    bool active = valid && compatible; // with LOCK, idle and incompatible lanes still take the barriers
    if (LOCK || active)
    {
        DState<NA> st;
#pragma unroll
        for (int a = 0; a < NA; a++)
        {
            st.pos[2 * a] = I.state.pos[2 * a];
            st.pos[2 * a + 1] = I.state.pos[2 * a + 1];
            st.vel[2 * a] = I.state.vel[2 * a];
            st.vel[2 * a + 1] = I.state.vel[2 * a + 1];
            st.S[a] = I.state.S[a];
            st.lat[a] = I.state.lat_dist[a];
            st.laps[a] = I.state.laps[a];
        }
        st.locate(E.trackLength);
        BState<NTH> bs;
#pragma unroll
        for (int i = 0; i < NTH; i++)
            bs.belief[i] = belief0[i];
        bs.predTheta = pt0;
        bs.branchingTime = bt0;
        if (active)
            cost = 0.0f;
        float decay = 1.0f;
        int tOrigin = 0;
        EnvNoise rng(k0, k1, (uint32_t)s, (uint32_t)th << 16, step, S_MPPI_ROLL_ENV);
        int curB = -1;
        for (int t = 0; t < T; t++)
        {
            if constexpr (LOCK)
            {
                // every thread of the CTA takes this barrier once per step (T is uniform),
                // keeping the warps on the same step
                if (!__syncthreads_or(active))
                    break;
                if (!active)
                    continue;
            }
            else if (!active)
                break; // the thread's rollout ended
            rng.begin_step((uint32_t)t);
            const int local = t - tOrigin;
            const int b = bs.predTheta;
            float ego0, ego1;
            if constexpr (SPL)
            {
                if (b != curB)
                {
                    // nominal + perturbation of this sample's knots for branch b
                    for (int m = 0; m < M; m++)
                    {
                        U4 r = draw(k0, k1, (uint32_t)s, (uint32_t)(b * M + m), step, S_MPPI_EPS, 0);
                        float e0 = scaled_normal(sig0, r.x);
                        float e1 = scaled_normal(sig1, r.y);
                        vbuf[(m * 2 + 0) * RB + threadIdx.x] = sKn[(b * M + m) * 2 + 0] + e0;
                        vbuf[(m * 2 + 1) * RB + threadIdx.x] = sKn[(b * M + m) * 2 + 1] + e1;
                    }
                    curB = b;
                }
                const float* Brow = sB + local * M;
                float sum = 0.0f;
                for (int m = 0; m < M; m++)
                    sum += Brow[m] * vbuf[(m * 2 + 0) * RB + threadIdx.x];
                ego0 = sum;
                sum = 0.0f;
                for (int m = 0; m < M; m++)
                    sum += Brow[m] * vbuf[(m * 2 + 1) * RB + threadIdx.x];
                ego1 = sum;
            }
            else
            {
                U4 r = draw(k0, k1, (uint32_t)s, (uint32_t)(b * T + local), step, S_MPPI_EPS, 0);
                float e0 = scaled_normal(sig0, r.x);
                float e1 = scaled_normal(sig1, r.y);
                ego0 = sKn[(b * T + local) * 2 + 0] + e0;
                ego1 = sKn[(b * T + local) * 2 + 1] + e1;
            }
            bool branched = false;
            StepOut o = envStep<NOPP, NTH, true, true, true, true>(t, th, tr, E, ego0, ego1, st, bs, branched, minConf, rng);
            if (branched)
                tOrigin = t + 1;
            if (o.term != TERM_NONE)
                active = false;
            cost += stateCost(o, E, D.cfg.w) * decay;
            decay *= DECAY;
        }
        if (valid && compatible)
        {
            cost += finalCost<NOPP>(st, E, D.cfg.w.finalAdvWeight, D.cfg.w.finalOppAdvWeight);
            pt = bs.predTheta;
            bt = bs.branchingTime;
        }
    }
    if (valid)
    {
        D.costsTrue[th * K + s] = cost;
        D.binfo[th * K + s] = packInfo(pt, bt);
        if (compatible && !isfinite(cost))
            atomicAdd(&D.stats[0], 1);
    }
    red[threadIdx.x] = cost;
    __syncthreads();
    // aggregateBranchCostsKernel (kernels.cu:175-217): costs[b][s] = E_belief[cost | b]
    if (valid)
    {
        const float* c = red + sl * NTH;
        if (th == 0)
        {
            float num = 0.0f, den = 0.0f;
#pragma unroll
            for (int m = 0; m < NTH; m++)
            {
                float cv = c[m];
                if (!isfinite(cv))
                    continue;
                float w = belief0[m];
                num += w * cv;
                den += w;
            }
            D.costs[s] = (den > 1e-30f) ? (num / den) : INFINITY;
        }
        {
            float num = 0.0f, den = 0.0f;
            float cv = c[th];
            if (isfinite(cv))
            {
                float w = belief0[th];
                num += w * cv;
                den += w;
            }
            D.costs[(size_t)(th + 1) * K + s] = (den > 1e-30f) ? (num / den) : INFINITY;
        }
    }
}

// One rollout tile with one opponent: a pair of lanes per (sample, hypothesis), the ego's
// lane and the opponent's (pair_model.cuh); RB / 2 pairs a CTA. The rollout is bound by the
// latency of its T dependent steps until the batch fills the device, and by instruction
// issue and divergence (samples that end early leave their lanes idle) from there. Against a
// thread per (sample, hypothesis), which moved both agents one after the other (B200, 1965
// MHz): one agent of K 1024 x 2 x T 50 0.23 -> 0.15 ms, four agents of K 4096 x 2 x T 64
// 0.32 -> 0.22 alone, one of K 65536 x 2 x T 80 with spline controls, the previous plan's
// verification beside it, 1.46 -> 1.09.
template <int NTH, bool SPL, bool LOCK>
__device__ __forceinline__ void rolloutTilePair(const MppiDev& D, const MppiIn& I, const Tile& tile, int K, int T, int M, const EnvParams& E,
                                                const float* sGrid, const float* sKn, const float* sB, float* vbuf, float* red)
{
    constexpr int PAIRS = RB / 2;
    const Track tr = trackIn(sGrid);
    const int role = threadIdx.x & 1, pair = threadIdx.x >> 1;
    const int th = pair % NTH;
    const int sl = pair / NTH;
    const int s = tile.s0 + sl;
    const bool valid = sl < tile.count;
    const float minConf = D.cfg.minConf;
    const uint32_t k0 = D.cfg.k0, k1 = D.cfg.k1, step = I.step;
    const float sig0 = D.cfg.sigma0, sig1 = D.cfg.sigma1;

    BState<NTH> bs;
#pragma unroll
    for (int i = 0; i < NTH; i++)
        bs.belief[i] = I.belief[i];
    // initBranchState (state.h:154-163)
    const int pt0 = findConfident<NTH>(bs.belief, minConf);
    bs.predTheta = pt0;
    bs.branchingTime = pt0 == 0 ? -1 : 0;
    const bool compatible = (pt0 == 0 || pt0 == th + 1);
    bool active = valid && compatible;
    float cost = active ? 0.0f : INFINITY;
    DState<1> st;
    st.pos[0] = I.state.pos[2 * role];
    st.pos[1] = I.state.pos[2 * role + 1];
    st.vel[0] = I.state.vel[2 * role];
    st.vel[1] = I.state.vel[2 * role + 1];
    st.S[0] = I.state.S[role];
    st.lat[0] = I.state.lat_dist[role];
    st.laps[0] = I.state.laps[role];
    st.locate(E.trackLength);
    float decay = 1.0f;
    int tOrigin = 0, curB = -1;
    for (int t = 0; t < T; t++)
    {
        if constexpr (LOCK)
        {
            // every thread of the CTA takes this barrier once per step (T is uniform),
            // keeping the warps on the same step
            if (!__syncthreads_or(active))
                break;
        }
        // the lanes still rolling out: whole pairs, since both lanes of one decide alike
        const unsigned mask = __ballot_sync(0xffffffffu, active);
        if (mask == 0u)
        {
            if constexpr (LOCK)
                continue;
            else
                break;
        }
        if (!active)
            continue;
        const int local = t - tOrigin;
        const int b = bs.predTheta;
        const bool oppNoise = E.actionNoise[th][0] != 0.0f;
        PairNoise noise{k0, k1, (uint32_t)s, ((uint32_t)th << 16) | (uint32_t)t, step, S_MPPI_ROLL_ENV};
        float ctl0, ctl1, opp0 = 0.0f, opp1 = 0.0f;
        if constexpr (SPL)
        {
            if (oppNoise)
            {
                const U4 r = draw(k0, k1, (uint32_t)s, noise.c1, step, S_MPPI_ROLL_ENV, 0);
                const float2 n = normal_pair_ool(r.x, r.y);
                opp0 = n.x;
                opp1 = n.y;
            }
            if (b != curB)
            {
                // nominal + perturbation of this sample's knots for branch b, the lanes
                // taking every other knot
                for (int m = role; m < M; m += 2)
                {
                    U4 r = draw(k0, k1, (uint32_t)s, (uint32_t)(b * M + m), step, S_MPPI_EPS, 0);
                    float e0 = scaled_normal(sig0, r.x);
                    float e1 = scaled_normal(sig1, r.y);
                    float* v = vbuf + ((m >> 2) * 2 * PAIRS + pair * 2) * 4 + (m & 3);
                    v[0] = sKn[(b * M + m) * 2 + 0] + e0;
                    v[4] = sKn[(b * M + m) * 2 + 1] + e1;
                }
                curB = b;
            }
            __syncwarp(mask);
            // a lane evaluates one axis of the control
            pairBoth(mask, role, splineSum(sB + local * M, vbuf, 2 * PAIRS, threadIdx.x, M), ctl0, ctl1);
        }
        else
        {
            // the ego's lane draws its perturbation, the opponent's lane its action noise
            const U4 r = draw(k0, k1, (uint32_t)s, role ? noise.c1 : (uint32_t)(b * T + local), step, role ? S_MPPI_ROLL_ENV : S_MPPI_EPS, 0);
            opp0 = normal_from_word(r.x);
            opp1 = normal_from_word(r.y);
            ctl0 = sKn[(b * T + local) * 2] + __fmul_rn(sig0, opp0);
            ctl1 = sKn[(b * T + local) * 2 + 1] + __fmul_rn(sig1, opp1);
        }
        bool branched = false;
        const StepOut o = pairStep<NTH>(mask, role, t, th, tr, E, ctl0, ctl1, opp0, opp1, st, bs, branched, minConf, noise);
        if (branched)
            tOrigin = t + 1;
        if (o.term != TERM_NONE)
            active = false;
        cost += stateCost(o, E, D.cfg.w) * decay;
        decay *= DECAY;
    }
    {
        DState<2> both; // the final cost reads both agents' arc lengths and laps
        pairBoth(0xffffffffu, role, st.S[0], both.S[0], both.S[1]);
        pairBoth(0xffffffffu, role, st.laps[0], both.laps[0], both.laps[1]);
        if (valid && compatible)
            cost += finalCost<1>(both, E, D.cfg.w.finalAdvWeight, D.cfg.w.finalOppAdvWeight);
    }
    if (valid && role == 0)
    {
        D.costsTrue[th * K + s] = cost;
        D.binfo[th * K + s] = packInfo(bs.predTheta, bs.branchingTime);
        if (compatible && !isfinite(cost))
            atomicAdd(&D.stats[0], 1);
    }
    if (role == 0)
        red[pair] = cost;
    __syncthreads();
    // aggregateBranchCostsKernel (kernels.cu:175-217): costs[b][s] = E_belief[cost | b]
    if (valid)
    {
        const float* c = red + sl * NTH;
        if (role == 0)
        {
            float num = 0.0f, den = 0.0f;
            float cv = c[th];
            if (isfinite(cv))
            {
                float w = I.belief[th];
                num += w * cv;
                den += w;
            }
            D.costs[(size_t)(th + 1) * K + s] = (den > 1e-30f) ? (num / den) : INFINITY;
        }
        else if (th == 0)
        {
            float num = 0.0f, den = 0.0f;
#pragma unroll
            for (int m = 0; m < NTH; m++)
            {
                float cv = c[m];
                if (!isfinite(cv))
                    continue;
                float w = I.belief[m];
                num += w * cv;
                den += w;
            }
            D.costs[s] = (den > 1e-30f) ? (num / den) : INFINITY;
        }
    }
}

// CTAs that share a tile of the table (rolloutSamplesPerBlock samples): a CTA of lane pairs
// takes half the samples that one of single threads does.
template <int NOPP> constexpr int rolloutParts()
{
    return NOPP == 1 ? 2 : 1;
}

template <int NOPP, int NTH, bool SPL, bool PQ, bool LOCK>
__global__ void __launch_bounds__(RB, (rolloutMinBlocks<NOPP, NTH>())) mppi_rollout(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in,
                                                                       const Tile* __restrict__ tiles, int nTiles, unsigned* __restrict__ queue)
{
    constexpr int NBP = NTH + 1;
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ int sTicket;
    pdl_trigger(); // the update may launch once every rollout CTA has started
    uint64_t* bar = (uint64_t*)smraw;
    if (threadIdx.x == 0)
        mbar_init(bar, 1);
    int staged = -1;     // instance whose track, knots and basis are in shared memory
    uint32_t phase = 0u; // parity of the staging barrier's next phase
    for (int iter = 0;; iter++)
    {
        const int ti = nextTile(PQ ? queue : nullptr, iter, &sTicket);
        constexpr int PARTS = rolloutParts<NOPP>();
        if (ti >= nTiles * PARTS)
            break;
        Tile tile = tiles[ti / PARTS];
        if constexpr (PARTS > 1)
        {
            constexpr int PER = RB / NTH / PARTS;
            const int part = ti % PARTS;
            tile.s0 += part * PER;
            tile.count = min(max(tile.count - part * PER, 0), PER);
        }
        const MppiDev& D = insts[tile.inst];
        const MppiIn& I = in[tile.inst];
        const int K = D.cfg.K, T = D.cfg.T, M = D.cfg.M;
        const RolloutSmem L = rolloutLayout(NBP, T, M, SPL, RB / PARTS);
        EnvParams* sE = (EnvParams*)(smraw + L.env);
        float* sGrid = (float*)(smraw + L.grids);
        float* sKn = (float*)(smraw + L.knots);
        float* sB = (float*)(smraw + L.B);
        float* vbuf = (float*)(smraw + L.vbuf);
        float* red = (float*)(smraw + L.red);
        if (tile.inst != staged)
        {
            const uint32_t knBytes = (uint32_t)align16((size_t)NBP * M * 2 * 4);
            const uint32_t bBytes = SPL ? (uint32_t)align16((size_t)T * M * 4) : 0u;
            if (threadIdx.x == 0)
            {
                mbar_expect_tx(bar, GRID_FLOATS * 4 + knBytes + bBytes);
                if (!D.cfg.dbgNoStage)
                {
                    bulk_g2s(sGrid, D.grids, GRID_FLOATS * 4, bar);
                    bulk_g2s(sKn, D.knots, knBytes, bar);
                    if (SPL)
                        bulk_g2s(sB, D.B, bBytes, bar);
                }
            }
            copyEnv(sE, &D.env);
            __syncthreads();
            if (!__syncthreads_and(mbar_wait(bar, phase, D.cfg.waitPolls)))
            {
                // The staging did not complete within the poll limit: write the tile's
                // defined timeout outputs, count the timeout for the host, return.
                rolloutTileTimedOut<NTH>(D, I, tile, K);
                if (threadIdx.x == 0)
                    atomicAdd(&D.stats[1], 1);
                return;
            }
            phase ^= 1u;
            staged = tile.inst;
        }
        if constexpr (NOPP == 1)
            rolloutTilePair<NTH, SPL, LOCK>(D, I, tile, K, T, M, *sE, sGrid, sKn, sB, vbuf, red);
        else
            rolloutTile<NOPP, NTH, SPL, LOCK>(D, I, tile, K, T, M, *sE, sGrid, sKn, sB, vbuf, red);
        if constexpr (PQ)
            fence_before_bulk();
        __syncthreads(); // the next tile's staging and reduction buffer reuse shared memory
    }
}

// aggregation alone (used by the update test hook, which takes costsTrue as input)
template <int NTH> __global__ void mppi_aggregate(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in)
{
    const MppiDev& D = insts[0];
    const MppiIn& I = in[0];
    const int K = D.cfg.K;
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= K)
        return;
    float num = 0.0f, den = 0.0f;
    for (int m = 0; m < NTH; m++)
    {
        float cv = D.costsTrue[m * K + s];
        if (!isfinite(cv))
            continue;
        float w = I.belief[m];
        num += w * cv;
        den += w;
    }
    D.costs[s] = (den > 1e-30f) ? (num / den) : INFINITY;
    for (int th = 0; th < NTH; th++)
    {
        float n2 = 0.0f, d2 = 0.0f;
        float cv = D.costsTrue[th * K + s];
        if (isfinite(cv))
        {
            float w = I.belief[th];
            n2 += w * cv;
            d2 += w;
        }
        D.costs[(size_t)(th + 1) * K + s] = (d2 > 1e-30f) ? (n2 / d2) : INFINITY;
    }
}

// ---------------------------------------------------------------------------------------
// update
// ---------------------------------------------------------------------------------------
// sampleContributed (state.h:203-219) for one factor.
__device__ __forceinline__ bool contributed(int b, int tLocal, int bt, int pt, int T)
{
    int origin = (b != 0 && bt > 0) ? bt : 0;
    int tGlobal = tLocal + origin;
    if (tGlobal >= T)
        return false;
    if ((b != 0 && b != pt) || (b == 0 && pt != 0 && tGlobal >= bt))
        return false;
    return true;
}

// The plan time whose contribution decides a knot's: a spline sample contributes to knot k when
// it does at one of the knots k - 1, k, k + 1 (splineSampleContributed, state.h:222-228), and
// what it contributes to (contributed) it contributes to at every earlier time too, so the
// first of the three decides; a dense knot is its own time. One test a hypothesis in place of
// three: update of 24 uneven agents up to K 16384, 107 -> 90 us; of K 65536, 93 -> 74.
__device__ __forceinline__ int knotTime(const MppiDev& D, int k, bool spl)
{
    return spl ? D.cfg.knots[k > 0 ? k - 1 : 0] : k;
}

// tk: knotTime of the knot
template <int NTH> __device__ __forceinline__ float sampleCoeff(const MppiDev& D, const float (&belief)[NTH], int b, int tk, int s, int T, int K)
{
    float coeff = 0.0f;
#pragma unroll
    for (int th = 0; th < NTH; th++)
    {
        if (belief[th] <= 0.0f)
            continue;
        if (!(b == 0 || b == th + 1))
            continue;
        const int v = D.binfo[th * K + s];
        if (contributed(b, tk, infoTime(v), infoPred(v), T))
            coeff += belief[th];
    }
    return coeff;
}

// One (branch plan, knot) per cluster of C CTAs. The sums keep the reference's order: lane l of
// its 256 adds samples l, l + 256, ... one after the other, then the lanes are added in a tree.
// The lanes are independent, so each CTA takes 256 / C of them, and within a CTA the terms
// (draw, normals, weight: some 300 instructions) are computed by all threads, C samples of a
// lane side by side, and only the additions (a fused multiply-add each) run in order, from
// shared memory. With C = 1 a thread is a lane. What bounds it: with few (branch, knot) blocks
// and many samples, too few threads for the device (60 blocks at 3 plans x 20 knots: 0.62 ms for
// 65536 samples with C = 1, see updateCluster); else instruction issue.
template <int NTH, int C>
__global__ void __launch_bounds__(UB) mppi_update(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in, const Tile* __restrict__ tiles)
{
    constexpr int NBP = NTH + 1;
    constexpr int W = UB / C;  // lanes of this CTA
    constexpr int R = 2;       // terms a thread computes between two barriers (C > 1)
    __shared__ float sNum0[UB], sNum1[UB], sDen[UB];
    __shared__ float sMin[UB / 32];
    __shared__ float sMinAll[C];
    __shared__ float4 sTerm[C > 1 ? 2 * R * UB : 1]; // (w, coeff, eps0, eps1) of C R samples a lane, twice
    __shared__ int sLast;
    if constexpr (C > 1)
        cg::this_cluster().barrier_arrive(); // this CTA runs: its shared memory may be written
    pdl_wait(); // the rollout's costs and branch records are complete and visible
    pdl_trigger();
    const Tile tile = tiles[blockIdx.x / C];
    const MppiDev& D = insts[tile.inst];
    const MppiIn& I = in[tile.inst];
    const int K = D.cfg.K, T = D.cfg.T, M = D.cfg.M;
    const bool spl = D.cfg.useSplines != 0;
    const int b = tile.s0 / M, k = tile.s0 % M;
    const int tk = knotTime(D, k, spl);
    const int tid = threadIdx.x;
    const int rank = C > 1 ? blockIdx.x % C : 0;
    const int first = (tid / W) * UB + rank * W + tid % W; // this thread's first sample; then every C UB
    float belief[NTH];
#pragma unroll
    for (int i = 0; i < NTH; i++)
        belief[i] = I.belief[i];
    const int initPred = findConfident<NTH>(belief, D.cfg.minConf);
    const float* costs = D.costs + (size_t)b * K;

    // masked minimum (computeMaskedMinCostsKernel, kernels.cu:221-301)
    float mn = INFINITY;
    if (initPred == 0 || initPred == b)
        for (int s = first; s < K; s += C * UB)
        {
            float coeff = sampleCoeff<NTH>(D, belief, b, tk, s, T, K);
            if (coeff > MIN_COEFF)
            {
                float c = costs[s];
                if (c < mn)
                    mn = c;
            }
        }
    mn = warp_min(mn);
    if ((tid & 31) == 0)
        sMin[tid >> 5] = mn;
    __syncthreads();
    float minC = sMin[0];
#pragma unroll
    for (int w = 1; w < UB / 32; w++)
        minC = fminf(minC, sMin[w]);
    if constexpr (C > 1)
    {
        // every CTA of the cluster gets every CTA's minimum
        cg::cluster_group cluster = cg::this_cluster();
        cluster.barrier_wait();
        if (tid < C)
            cluster.map_shared_rank(sMinAll, tid)[rank] = minC;
        cluster.sync();
#pragma unroll
        for (int q = 0; q < C; q++)
            minC = fminf(minC, sMinAll[q]);
    }

    // weighted average of the regenerated perturbation (weightedAverageKernelUnified,
    // kernels.cu:307-408); w = exp(-(c - min) / inv_temperature)
    const float lambda = I.lambda;
    const uint32_t k0 = D.cfg.k0, k1 = D.cfg.k1, step = I.step;
    float num0 = 0.0f, num1 = 0.0f, den = 0.0f;
    // sample s' term; all zero where it has none (adding it changes nothing)
    auto term = [&](int s) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (s < K)
        {
            const float coeff = sampleCoeff<NTH>(D, belief, b, tk, s, T, K);
            if (coeff > MIN_COEFF)
            {
                const float w = expf(-(costs[s] - minC) / lambda);
                if (w != 0.0f) // else the draw is multiplied by zero
                {
                    const U4 r = draw(k0, k1, (uint32_t)s, (uint32_t)(b * M + k), step, S_MPPI_EPS, 0);
                    v = make_float4(w, coeff, scaled_normal(D.cfg.sigma0, r.x), scaled_normal(D.cfg.sigma1, r.y));
                }
            }
        }
        return v;
    };
    auto add = [&](float4 v) {
        num0 += v.x * v.y * v.z;
        num1 += v.x * v.y * v.w;
        den += v.x * v.y;
    };
    if (!isinf(minC))
    {
        if constexpr (C == 1)
        {
            for (int s = tid; s < K; s += UB)
                add(term(s));
        }
        else
        {
            int buf = 0;
            for (int s0 = 0; s0 < K; s0 += R * C * UB, buf ^= 1)
            {
                float4* t = sTerm + buf * R * UB;
#pragma unroll
                for (int r = 0; r < R; r++)
                    t[r * UB + tid] = term(s0 + r * C * UB + first); // [(r, sample of the lane)][lane]
                __syncthreads();
                if (tid < W)
#pragma unroll 8
                    for (int i = 0; i < R * C; i++)
                        add(t[i * W + tid]);
            }
        }
    }
    if constexpr (C == 1)
    {
        sNum0[tid] = num0;
        sNum1[tid] = num1;
        sDen[tid] = den;
        __syncthreads();
    }
    else
    {
        // all lanes' sums to the cluster's first CTA, which goes on alone
        cg::cluster_group cluster = cg::this_cluster();
        if (tid < W)
        {
            cluster.map_shared_rank(sNum0, 0)[rank * W + tid] = num0;
            cluster.map_shared_rank(sNum1, 0)[rank * W + tid] = num1;
            cluster.map_shared_rank(sDen, 0)[rank * W + tid] = den;
        }
        cluster.sync();
        if (rank != 0)
            return;
    }
    // the reference's shared-memory tree: strides 128, 64, 32 across warps, then 16..1
#pragma unroll
    for (int stride = UB / 2; stride >= 32; stride >>= 1)
    {
        if (tid < stride)
        {
            sNum0[tid] += sNum0[tid + stride];
            sNum1[tid] += sNum1[tid + stride];
            sDen[tid] += sDen[tid + stride];
        }
        __syncthreads();
    }
    if (tid < 32)
    {
        float a0 = sNum0[tid], a1 = sNum1[tid], dd = sDen[tid];
#pragma unroll
        for (int stride = 16; stride > 0; stride >>= 1)
        {
            a0 += __shfl_down_sync(0xffffffffu, a0, stride);
            a1 += __shfl_down_sync(0xffffffffu, a1, stride);
            dd += __shfl_down_sync(0xffffffffu, dd, stride);
        }
        if (tid == 0)
        {
            float* kn = D.knots + (size_t)(b * M + k) * 2;
            if (dd > 1e-30f)
            {
                __stcg(kn + 0, __ldcg(kn + 0) + a0 / dd);
                __stcg(kn + 1, __ldcg(kn + 1) + a1 / dd);
            }
            if (k == 0)
                D.nu[b] = dd;
            D.minCosts[b * M + k] = minC;
            __threadfence();
            unsigned prev = atomicAdd(D.counter, 1u);
            sLast = (prev == (unsigned)(NBP * M - 1));
        }
    }
    __syncthreads();
    if (!sLast)
        return;
    __threadfence();
    // last block of this instance: interpolateSplineKernel + clampNominalKernel
    if (spl)
    {
        for (int idx = tid; idx < NBP * T * 2; idx += UB)
        {
            int dim = idx & 1, t = (idx >> 1) % T, br = (idx >> 1) / T;
            float sum = 0.0f;
            for (int m = 0; m < M; m++)
                sum += D.B[t * M + m] * __ldcg(D.knots + (br * M + m) * 2 + dim);
            D.dense[idx] = sum;
        }
        __syncthreads();
    }
    const float maxAccel = D.env.maxAccel[0];
    for (int v = tid; v < NBP * M; v += UB)
    {
        float x0 = __ldcg(D.knots + v * 2), x1 = __ldcg(D.knots + v * 2 + 1);
        float sq = 0.0f;
        sq += x0 * x0;
        sq += x1 * x1;
        float maxSq = maxAccel * maxAccel;
        if (sq > maxSq)
        {
            float scale = maxAccel / sqrtf(sq);
            x0 *= scale;
            x1 *= scale;
        }
        __stcg(D.knots + v * 2, x0);
        __stcg(D.knots + v * 2 + 1, x1);
        if (!spl)
        {
            D.dense[v * 2] = x0;
            D.dense[v * 2 + 1] = x1;
        }
    }
    if (tid == 0)
        *D.counter = 0u;
}

// ---------------------------------------------------------------------------------------
// sample-sharded update: one controller's samples split across processes (one per GPU),
// the processes' partial results exchanged once per step by the caller's all-gather
// ---------------------------------------------------------------------------------------
// One exchange per step for a sample-sharded controller: this process's masked minimum
// per (branch plan, knot) over its own samples and its weighted sums of the regenerated
// perturbations taken with that local minimum, partial[(b, k)] = (m_r, sum w coeff eps0,
// sum w coeff eps1, sum w coeff), w = exp(-(c - m_r) / lambda). The processes all-gather
// the partials; mppi_shard_merge brings them to the global minimum m with the factor
// exp(-(m_r - m) / lambda) (the weight of a sample relative to m is its weight relative to
// m_r times that factor), so no second exchange is needed for the sums.
template <int NTH> __global__ void __launch_bounds__(UB) mppi_shard_local(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in,
                                                                          const Tile* __restrict__ tiles, float* __restrict__ partial)
{
    __shared__ float sMin[UB / 32];
    __shared__ float sNum0[UB], sNum1[UB], sDen[UB];
    const Tile tile = tiles[blockIdx.x];
    const MppiDev& D = insts[tile.inst];
    const MppiIn& I = in[tile.inst];
    const int K = D.cfg.K, T = D.cfg.T, M = D.cfg.M, sLo = D.cfg.sLo, sHi = D.cfg.sHi;
    const bool spl = D.cfg.useSplines != 0;
    const int b = tile.s0 / M, k = tile.s0 % M;
    const int tk = knotTime(D, k, spl);
    const int tid = threadIdx.x;
    float belief[NTH];
#pragma unroll
    for (int i = 0; i < NTH; i++)
        belief[i] = I.belief[i];
    const int initPred = findConfident<NTH>(belief, D.cfg.minConf);
    const float* costs = D.costs + (size_t)b * K;
    float mn = INFINITY;
    if (initPred == 0 || initPred == b)
        for (int s = sLo + tid; s < sHi; s += UB)
        {
            float coeff = sampleCoeff<NTH>(D, belief, b, tk, s, T, K);
            if (coeff > MIN_COEFF)
            {
                float c = costs[s];
                if (c < mn)
                    mn = c;
            }
        }
    mn = warp_min(mn);
    if ((tid & 31) == 0)
        sMin[tid >> 5] = mn;
    __syncthreads();
    float minC = sMin[0];
#pragma unroll
    for (int w = 1; w < UB / 32; w++)
        minC = fminf(minC, sMin[w]);
    const float lambda = I.lambda;
    const uint32_t k0 = D.cfg.k0, k1 = D.cfg.k1, step = I.step;
    float num0 = 0.0f, num1 = 0.0f, den = 0.0f;
    if (!isinf(minC))
        for (int s = sLo + tid; s < sHi; s += UB)
        {
            float coeff = sampleCoeff<NTH>(D, belief, b, tk, s, T, K);
            if (coeff > MIN_COEFF)
            {
                float cost = costs[s];
                float w = expf(-(cost - minC) / lambda);
                U4 r = draw(k0, k1, (uint32_t)s, (uint32_t)(b * M + k), step, S_MPPI_EPS, 0);
                float eps0 = scaled_normal(D.cfg.sigma0, r.x);
                float eps1 = scaled_normal(D.cfg.sigma1, r.y);
                num0 += w * coeff * eps0;
                num1 += w * coeff * eps1;
                den += w * coeff;
            }
        }
    sNum0[tid] = num0;
    sNum1[tid] = num1;
    sDen[tid] = den;
    __syncthreads();
#pragma unroll
    for (int stride = UB / 2; stride >= 32; stride >>= 1)
    {
        if (tid < stride)
        {
            sNum0[tid] += sNum0[tid + stride];
            sNum1[tid] += sNum1[tid + stride];
            sDen[tid] += sDen[tid + stride];
        }
        __syncthreads();
    }
    if (tid < 32)
    {
        float a0 = sNum0[tid], a1 = sNum1[tid], dd = sDen[tid];
#pragma unroll
        for (int stride = 16; stride > 0; stride >>= 1)
        {
            a0 += __shfl_down_sync(0xffffffffu, a0, stride);
            a1 += __shfl_down_sync(0xffffffffu, a1, stride);
            dd += __shfl_down_sync(0xffffffffu, dd, stride);
        }
        if (tid == 0)
        {
            float* o = partial + (size_t)(b * M + k) * 4;
            o[0] = minC;
            o[1] = a0;
            o[2] = a1;
            o[3] = dd;
        }
    }
}

// The partials of all processes (gathered[r * words + ...], rank order), merged the same
// way on every process: the global minimum and the rescaled sums per (branch plan, knot)
// into mins / sums (the layout mppi_shard_apply reads), and the previous plan's failure
// histograms summed into the controller's fail[T .. 2T).
__global__ void __launch_bounds__(UB) mppi_shard_merge(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in, const float* __restrict__ gathered,
                                                       int words, int world, float* __restrict__ mins, float* __restrict__ sums)
{
    const MppiDev& D = insts[0];
    const int T = D.cfg.T, M = D.cfg.M, nbp = D.cfg.nth + 1;
    const float lambda = in[0].lambda;
    for (int v = threadIdx.x; v < nbp * M; v += blockDim.x)
    {
        float m = INFINITY;
        for (int r = 0; r < world; r++)
            m = fminf(m, gathered[(size_t)r * words + v * 4]);
        float a0 = 0.0f, a1 = 0.0f, dd = 0.0f;
        if (!isinf(m))
            for (int r = 0; r < world; r++)
            {
                const float* p = gathered + (size_t)r * words + v * 4;
                if (isinf(p[0]))
                    continue; // no sample of process r contributes
                const float f = expf(-(p[0] - m) / lambda);
                a0 += p[1] * f;
                a1 += p[2] * f;
                dd += p[3] * f;
            }
        mins[v] = m;
        sums[v * 3] = a0;
        sums[v * 3 + 1] = a1;
        sums[v * 3 + 2] = dd;
    }
    const int hOff = nbp * M * 4;
    for (int t = threadIdx.x; t < T; t += blockDim.x)
    {
        unsigned h = 0u;
        for (int r = 0; r < world; r++)
            h += __float_as_uint(gathered[(size_t)r * words + hOff + t]);
        D.fail[T + t] = h;
    }
}

// the update from the merged sums of all processes, then interpolateSplineKernel and
// clampNominalKernel (kernels.cu:411-456); one block per instance
__global__ void __launch_bounds__(UB) mppi_shard_apply(const MppiDev* __restrict__ insts, int nbp, const float* __restrict__ mins,
                                                       const float* __restrict__ sums)
{
    const MppiDev& D = insts[blockIdx.x];
    const int T = D.cfg.T, M = D.cfg.M;
    const bool spl = D.cfg.useSplines != 0;
    const int tid = threadIdx.x;
    for (int v = tid; v < nbp * M; v += UB)
    {
        const int b = v / M, k = v % M;
        const float a0 = sums[v * 3], a1 = sums[v * 3 + 1], dd = sums[v * 3 + 2];
        if (dd > 1e-30f)
        {
            D.knots[v * 2 + 0] += a0 / dd;
            D.knots[v * 2 + 1] += a1 / dd;
        }
        if (k == 0)
            D.nu[b] = dd;
        D.minCosts[v] = mins[v];
    }
    __syncthreads();
    if (spl)
    {
        for (int idx = tid; idx < nbp * T * 2; idx += UB)
        {
            int dim = idx & 1, t = (idx >> 1) % T, br = (idx >> 1) / T;
            float sum = 0.0f;
            for (int m = 0; m < M; m++)
                sum += D.B[t * M + m] * D.knots[(br * M + m) * 2 + dim];
            D.dense[idx] = sum;
        }
        __syncthreads();
    }
    const float maxAccel = D.env.maxAccel[0];
    for (int v = tid; v < nbp * M; v += UB)
    {
        float x0 = D.knots[v * 2], x1 = D.knots[v * 2 + 1];
        float sq = 0.0f;
        sq += x0 * x0;
        sq += x1 * x1;
        float maxSq = maxAccel * maxAccel;
        if (sq > maxSq)
        {
            float scale = maxAccel / sqrtf(sq);
            x0 *= scale;
            x1 *= scale;
        }
        D.knots[v * 2] = x0;
        D.knots[v * 2 + 1] = x1;
        if (!spl)
        {
            D.dense[v * 2] = x0;
            D.dense[v * 2 + 1] = x1;
        }
    }
}

// ---------------------------------------------------------------------------------------
// verification
// ---------------------------------------------------------------------------------------
// The ego tables of a plan (EgoRow; plan 0 the new one, 1 the previous one, 2 both): a row
// is the trajectory with no branch, or the one of a branch and a branching step, moved alone
// through the verification horizon with the fast arithmetic of the verification; each CTA of
// EGO_WARPS warps stages the track, the environment and the plan in shared memory. The
// kernel's time is one row's chain of H steps. Only position and velocity need that chain,
// and they do not need the track: so EGO_STEPS lanes take as many steps of a row, each lane
// runs the short chain up to its own step and then projects that position by itself, from the
// sample that the steps before ended at. The sample found is the one that the window scan of
// the step-by-step projection finds wherever the certificate holds there and the sample lies
// in that step's window, which the lane checks once its neighbour's arc length is known; where
// it does not, the steps are taken one by one (egoStep). The lane also runs the trajectory
// with no branch beside its own and puts its distance from it into the clearance block.
constexpr int EGO_WARPS = 4;

// 8 / 16 / 32 steps at a time: 18.5 / 17.0 / 16.6 us for a plan of four agents, H 40, two
// hypotheses (B200, 1965 MHz); more steps repeat more of the short chain, which large batches
// pay for. A warp per row, step by step, its lanes sharing the window scan: 31 us, without
// the clearance block.
#ifndef DR_EGO_STEPS
#define DR_EGO_STEPS 16
#endif
constexpr int EGO_STEPS = DR_EGO_STEPS;                  // steps of a row taken at a time, a lane each
constexpr int EGO_CTA_ROWS = EGO_WARPS * 32 / EGO_STEPS; // rows a CTA takes at a time

// The squared distance from (px, py) to track sample i (0 .. 511).
__device__ __forceinline__ float sampleSqDist(const Track& tr, int i, float px, float py)
{
    const float dx = tr.px[i] - px, dy = tr.py[i] - py;
    return dx * dx + dy * dy;
}

// egoStep's position, velocity and speed cap under a control already clamped
__device__ __forceinline__ void egoAdvance(const EnvParams& E, const float* ctl, float (&p)[2], float (&v)[2])
{
    p[0] += E.dt * v[0];
    p[1] += E.dt * v[1];
    v[0] += E.dt * ctl[0];
    v[1] += E.dt * ctl[1];
    float sqSpd = sqNorm(v[0], v[1]);
    if (sqSpd > E.maxSpeed[0] * E.maxSpeed[0])
    {
        float sc = mdivsqrt<true>(E.maxSpeed[0], sqSpd);
        v[0] *= sc;
        v[1] *= sc;
    }
}

// The bound of five CTAs an SM gives it 96 registers a thread and no spills. Without one the compiler may
// choose 80 with spills: beside the rollout the previous plan's table of four agents (H 40, two
// hypotheses) then took 160 us in place of 19, and the control step 657 in place of 632.
template <int NTH>
__global__ void __launch_bounds__(EGO_WARPS * 32, 5) mppi_ego_table(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in, int nInst, int plans)
{
    __shared__ __align__(16) float sg[GRID_FLOATS];
    __shared__ __align__(16) float sPlan[(NTH + 1) * DR_MAX_T * 2];
    __shared__ EnvParams sE;
    __shared__ __align__(8) uint64_t bar;
    const int inst = blockIdx.x;
    if (inst >= nInst)
        return;
    const MppiDev& D = insts[inst];
    const MppiIn& I = in[inst];
    if (!D.egoTab)
        return;
    const int H = D.cfg.H, T = D.cfg.T, rows = egoRows(NTH, H), nbp = NTH + 1;
    const int p0 = plans == 1 ? 1 : 0, p1 = plans == 0 ? 0 : 1;
    const uint32_t planBytes = (uint32_t)align16((size_t)nbp * T * 2 * 4);
    if (threadIdx.x == 0)
    {
        mbar_init(&bar, 1);
        mbar_expect_tx(&bar, GRID_FLOATS * 4 + planBytes);
        if (!D.cfg.dbgNoStage)
        {
            bulk_g2s(sg, D.grids, GRID_FLOATS * 4, &bar);
            bulk_g2s(sPlan, p0 == 0 ? D.dense : D.prevDense, planBytes, &bar);
        }
    }
    copyEnv(&sE, &D.env);
    const EnvParams& E = sE;
    const Track tr = trackIn(sg);
    float belief[NTH];
#pragma unroll
    for (int i = 0; i < NTH; i++)
        belief[i] = I.belief[i];
    const int pt0 = findConfident<NTH>(belief, D.cfg.minConf);
    const int sub = threadIdx.x % EGO_STEPS; // this lane's step
    constexpr unsigned ALL = 0xffffffffu;
    for (int plan = p0; plan <= p1; plan++)
    {
        if (plan != p0)
            fence_before_bulk(); // the clamp below wrote sPlan
        __syncthreads(); // the environment's terms, and the previous plan's rows are done with sPlan
        if (threadIdx.x == 0 && plan != p0)
        {
            mbar_expect_tx(&bar, planBytes);
            if (!D.cfg.dbgNoStage)
                bulk_g2s(sPlan, D.prevDense, planBytes, &bar);
        }
        if (!__syncthreads_and(mbar_wait(&bar, (uint32_t)(plan - p0), D.cfg.waitPolls)))
        {
            // uniform: the step reports the timeout, as for the other kernels' staging; a
            // clearance block without its rows leaves no sample out
            for (int q = plan + (int)threadIdx.x; q <= p1; q += blockDim.x)
                *ClearBlock<float>(D.clear + (size_t)q * clearWords(H), H).out = 1.0f;
            if (threadIdx.x == 0)
                atomicAdd(&D.stats[1], 1);
            return;
        }
        if (!egoNoiseFree(E))
            continue; // uniform: the verification moves the ego itself
        // egoStep's clamp of the controls
        for (int i = threadIdx.x; i < nbp * T; i += blockDim.x)
        {
            float ego0 = sPlan[2 * i], ego1 = sPlan[2 * i + 1];
            float sq = 0.0f;
            sq += ego0 * ego0;
            sq += ego1 * ego1;
            float factor = 1.0f;
            float maxSq = E.maxAccel[0] * E.maxAccel[0];
            if (sq > maxSq)
                factor = mdivsqrt<true>(E.maxAccel[0], sq);
            sPlan[2 * i] = ego0 * factor;
            sPlan[2 * i + 1] = ego1 * factor;
        }
        __syncthreads();
        EgoRow* tab = D.egoTab + (size_t)plan * rows * H;
        const ClearBlock<float> cb(D.clear + (size_t)plan * clearWords(H), H);
        const float L = E.trackLength, invL = E.invTrackLength;
        const int nRows = pt0 != 0 ? 1 : rows; // a confident initial belief never branches
        // whole warps take part as long as one of their rows exists; the others repeat row 0
        for (int base = blockIdx.y * EGO_CTA_ROWS; base + (int)(threadIdx.x & ~31u) / EGO_STEPS < nRows; base += gridDim.y * EGO_CTA_ROWS)
        {
            const int want = base + (int)threadIdx.x / EGO_STEPS;
            const bool mine = want < nRows;
            const int r = mine ? want : 0;
            const int bb = r > 0 ? 1 + (r - 1) / H : 0, tb = r > 0 ? (r - 1) % H : H;
            // the verification's plan index: branch pt0 before any branching, then the
            // branch taken, its clock restarting after the branching step
            auto control = [&](int t) { return sPlan + ((t <= tb ? pt0 : bb) * T + (t <= tb ? t : t - tb - 1)) * 2; };
            DState<1> s; // after the steps done, alike on the row's lanes
            s.pos[0] = I.state.pos[0];
            s.pos[1] = I.state.pos[1];
            s.vel[0] = I.state.vel[0];
            s.vel[1] = I.state.vel[1];
            s.S[0] = I.state.S[0];
            s.lat[0] = I.state.lat_dist[0];
            s.laps[0] = I.state.laps[0];
            s.locate(L);
            float bp[2] = {s.pos[0], s.pos[1]}, bv[2] = {s.vel[0], s.vel[1]}; // the trajectory with no branch
            AgentGeo<1> g; // of s
            agentGeometry<1, true>(tr, E, s, g);
            int near = wrapNts(s.tp[0].i0);
            for (int t0 = 0; t0 < H; t0 += EGO_STEPS)
            {
                const int t = t0 + sub;
                DState<1> m; // after step t
                float p[2] = {s.pos[0], s.pos[1]}, v[2] = {s.vel[0], s.vel[1]}, b0 = 0.0f, b1 = 0.0f;
#pragma unroll 4
                for (int u = 0; u < EGO_STEPS; u++)
                {
                    if (t0 + u < H)
                    {
                        egoAdvance(E, control(t0 + u), p, v);
                        egoAdvance(E, sPlan + (pt0 * T + t0 + u) * 2, bp, bv);
                    }
                    if (u <= sub)
                    {
                        m.pos[0] = p[0];
                        m.pos[1] = p[1];
                        m.vel[0] = v[0];
                        m.vel[1] = v[1];
                        b0 = bp[0];
                        b1 = bp[1];
                    }
                }
                // walk to a local minimum of the distances
                int c = near;
                float dc = sampleSqDist(tr, c, m.pos[0], m.pos[1]);
                const int dir = sampleSqDist(tr, wrapNts(c + 1), m.pos[0], m.pos[1]) < dc ? 1 : NTS - 1;
                for (int n = 0; n < NTS; n++)
                {
                    const int next = wrapNts(c + dir);
                    const float dn = sampleSqDist(tr, next, m.pos[0], m.pos[1]);
                    if (!(dn < dc))
                        break;
                    c = next;
                    dc = dn;
                }
                m.S[0] = projectSegments<true>(tr, L, invL, m.pos[0], m.pos[1], c, m.lat[0], m.tp[0]);
                AgentGeo<1> gm;
                agentGeometry<1, true>(tr, E, m, gm);
                // the state before step t: the neighbour's, or the one after the steps done
                EgoRow row;
                float pS = __shfl_up_sync(ALL, m.S[0], 1, EGO_STEPS);
                row.tn0 = __shfl_up_sync(ALL, gm.tn0[0], 1, EGO_STEPS);
                row.tn1 = __shfl_up_sync(ALL, gm.tn1[0], 1, EGO_STEPS);
                row.sdot = __shfl_up_sync(ALL, gm.sdot[0], 1, EGO_STEPS);
                if (sub == 0)
                {
                    pS = s.S[0];
                    row.tn0 = g.tn0[0];
                    row.tn1 = g.tn1[0];
                    row.sdot = g.sdot[0];
                }
                float q = pS;
                q += E.dt * row.sdot;
                q *= invL;
                q = q - floorf(q);
                const int j0 = (int)(q * NTS) - WIN;
                const bool found = dc <= tr.cert[c] && wrapNts(c - j0 + 2 * NTS) <= 2 * WIN;
                if (__all_sync(ALL, found || t >= H))
                {
                    int laps = (m.S[0] < pS - L * 0.5f ? 1 : 0) - (m.S[0] > pS + L * 0.5f ? 1 : 0);
#pragma unroll
                    for (int o = 1; o < EGO_STEPS; o *= 2)
                    {
                        const int x = __shfl_up_sync(ALL, laps, o, EGO_STEPS);
                        if (sub >= o)
                            laps += x;
                    }
                    row.pos0 = m.pos[0];
                    row.pos1 = m.pos[1];
                    row.vel0 = m.vel[0];
                    row.vel1 = m.vel[1];
                    row.S = m.S[0];
                    row.lat = m.lat[0];
                    row.w = m.tp[0].w;
                    row.laps = s.laps[0] + laps;
                    row.i0 = m.tp[0].i0;
                    constexpr int LAST = EGO_STEPS - 1;
                    s.pos[0] = p[0];
                    s.pos[1] = p[1];
                    s.vel[0] = v[0];
                    s.vel[1] = v[1];
                    s.S[0] = __shfl_sync(ALL, m.S[0], LAST, EGO_STEPS);
                    s.lat[0] = __shfl_sync(ALL, m.lat[0], LAST, EGO_STEPS);
                    s.laps[0] = __shfl_sync(ALL, row.laps, LAST, EGO_STEPS);
                    s.tp[0].i0 = __shfl_sync(ALL, m.tp[0].i0, LAST, EGO_STEPS);
                    s.tp[0].w = __shfl_sync(ALL, m.tp[0].w, LAST, EGO_STEPS);
                    g.tn0[0] = __shfl_sync(ALL, gm.tn0[0], LAST, EGO_STEPS);
                    g.tn1[0] = __shfl_sync(ALL, gm.tn1[0], LAST, EGO_STEPS);
                    g.sdot[0] = __shfl_sync(ALL, gm.sdot[0], LAST, EGO_STEPS);
                    near = __shfl_sync(ALL, c, LAST, EGO_STEPS);
                }
                else
                {
                    for (int u = 0; u < EGO_STEPS && t0 + u < H; u++)
                    {
                        const float* ctl = control(t0 + u);
                        EgoRow step;
                        egoStep<true, true>(tr, E, ctl[0], ctl[1], s, step);
                        if (sub == u)
                            row = step;
                    }
                    agentGeometry<1, true>(tr, E, s, g);
                    near = wrapNts(s.tp[0].i0);
                }
                if (mine && t < H)
                {
                    tab[(size_t)r * H + t] = row;
                    const bool off = !(E.trackWidth - fabsf(row.lat) >= E.droneRadius);
                    if (r == 0)
                    {
                        cb.xy[2 * t] = row.pos0;
                        cb.xy[2 * t + 1] = row.pos1;
                        if (off)
                            *cb.out = 1.0f;
                    }
                    else if (t > tb) // up to its branching step a row is the first one
                    {
                        // off the track, or a distance that is no number: infinitely far
                        const float dx = row.pos0 - b0, dy = row.pos1 - b1;
                        float d = sqrtf(dx * dx + dy * dy);
                        if (off || !(d <= FLT_MAX))
                            d = INFINITY;
                        // distances are not negative: they order as their words
                        atomicMax((unsigned*)&cb.all[t], __float_as_uint(d));
                        atomicMax((unsigned*)&cb.rho[tb / clearPer(H) * H + t], __float_as_uint(d));
                    }
                }
            }
        }
    }
}

// What bounds it: instruction issue, over the samples' steps. So a warp whose samples can no
// longer collide leaves (clearOfEgo), and a tile none of whose samples can ends at once.
// FAST: the fast arithmetic flavour and noise source (the default; the exact flavour
// reproduces the oracle's per-sample results and serves parity tests). EGO (with FAST):
// the ego's moves come from the instance's ego table of the plan (mppi_ego_table).
template <int NOPP, int NTH, bool PQ, bool FAST, bool EGO = false>
__global__ void __launch_bounds__(VERIFY_TILE, (verifyMinBlocks<NOPP, NTH>())) mppi_verify(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in, const Tile* __restrict__ tiles,
                                                  int nTiles, unsigned* __restrict__ queue, int* __restrict__ dbgFailTime, int* __restrict__ dbgTheta)
{
    constexpr int NA = NOPP + 1;
    constexpr int NBP = NTH + 1;
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ int sTicket;
    pdl_wait(); // the plan to verify is complete and visible
    uint64_t* bar = (uint64_t*)smraw;
    EnvParams* sE = (EnvParams*)(smraw + 16);
    const size_t offG = align16(16 + sizeof(EnvParams));
    float* sGrid = (float*)(smraw + offG);
    float* sPlan = (float*)(smraw + offG + GRID_FLOATS * 4);
    if (threadIdx.x == 0)
        mbar_init(bar, 1);
    int staged = -1;     // (instance, plan) whose track and plan are in shared memory
    uint32_t phase = 0u; // parity of the staging barrier's next phase
    for (int iter = 0;; iter++)
    {
        const int ti = nextTile(PQ ? queue : nullptr, iter, &sTicket);
        if (ti >= nTiles)
            break;
        const Tile tile = tiles[ti];
        const MppiDev& D = insts[tile.inst];
        const MppiIn& I = in[tile.inst];
        const int T = D.cfg.T, H = D.cfg.H;
        const int plan = tile.aux;
        const uint32_t planBytes = (uint32_t)align16((size_t)NBP * T * 2 * 4);
        const uint32_t clearBytes = EGO ? (uint32_t)clearWords(H) * 4u : 0u;
        float* sClear = (float*)(smraw + offG + GRID_FLOATS * 4 + planBytes);
        unsigned* hist = (unsigned*)((unsigned char*)sClear + clearBytes);
        const int key = tile.inst * 2 + plan;
        if constexpr (EGO)
        {
            // every sample starts from the same state: where it is clear of the ego over the
            // whole horizon, no sample of the tile can fail
            bool clear = !dbgTheta;
            const ClearBlock<const float> cb(D.clear + (size_t)plan * clearWords(H), H);
            clear = clear && *cb.out == 0.0f;
            for (int o = 1; o <= NOPP; o++)
            {
                int witness = -1;
                clear = clear && clearOfEgoCall(D.env.dt, D.env.droneRadius, cb.xy, cb.all, H, 0, true, I.state.pos[2 * o], I.state.pos[2 * o + 1], I.state.vel[2 * o],
                                            I.state.vel[2 * o + 1], D.env.maxSpeed[o], D.env.maxAccel[o], witness);
            }
            if (clear)
            {
                if constexpr (PQ)
                    __syncthreads(); // every thread has read its ticket
                continue;
            }
        }
        if (key != staged)
        {
            if (threadIdx.x == 0)
            {
                mbar_expect_tx(bar, GRID_FLOATS * 4 + planBytes + clearBytes);
                if (!D.cfg.dbgNoStage)
                {
                    bulk_g2s(sGrid, D.grids, GRID_FLOATS * 4, bar);
                    bulk_g2s(sPlan, plan == 0 ? D.dense : D.prevDense, planBytes, bar);
                    if (EGO)
                        bulk_g2s(sClear, D.clear + (size_t)plan * clearWords(H), clearBytes, bar);
                }
            }
            copyEnv(sE, &D.env);
        }
        for (int i = threadIdx.x; i < T; i += blockDim.x)
            hist[i] = 0u;
        __syncthreads();
        if (key != staged)
        {
            // on timeout the tile adds nothing to the histograms; the host reports it
            if (!__syncthreads_and(mbar_wait(bar, phase, D.cfg.waitPolls)))
            {
                if (threadIdx.x == 0)
                    atomicAdd(&D.stats[1], 1);
                return;
            }
            phase ^= 1u;
            staged = key;
            if constexpr (EGO)
            {
                clearSuffix(sClear, H);
                __syncthreads();
            }
        }
        const EnvParams& E = *sE;
        const Track tr = trackIn(sGrid);
        const int v = tile.s0 + threadIdx.x;
        bool active = threadIdx.x < tile.count; // idle lanes of a partial tile still take the barriers
        {
            const float minConf = D.cfg.minConf;
            DState<NA> st;
#pragma unroll
            for (int a = 0; a < NA; a++)
            {
                st.pos[2 * a] = I.state.pos[2 * a];
                st.pos[2 * a + 1] = I.state.pos[2 * a + 1];
                st.vel[2 * a] = I.state.vel[2 * a];
                st.vel[2 * a + 1] = I.state.vel[2 * a + 1];
                st.S[a] = I.state.S[a];
                st.lat[a] = I.state.lat_dist[a];
                st.laps[a] = I.state.laps[a];
            }
            st.locate(E.trackLength);
            BState<NTH> bs;
#pragma unroll
            for (int i = 0; i < NTH; i++)
                bs.belief[i] = I.belief[i];
            bs.predTheta = findConfident<NTH>(bs.belief, minConf);
            bs.branchingTime = bs.predTheta == 0 ? -1 : 0;
            const int pt0 = bs.predTheta;
            const EgoRow* egoTab = EGO ? D.egoTab + (size_t)plan * egoRows(NTH, H) * H : nullptr;
            // sampleModelFromBelief (state.h:118-131) on a Philox uniform
            const uint32_t k0 = D.cfg.k0, k1 = D.cfg.k1, step = I.step;
            float u = uniform_from_word(draw(k0, k1, (uint32_t)v, (uint32_t)plan, step, S_VERIF_THETA, 0).x);
            int theta = NTH - 1;
            {
                float cdf = 0.0f;
                bool found = false;
#pragma unroll
                for (int kk = 0; kk < NTH; kk++)
                {
                    cdf += bs.belief[kk];
                    if (!found && u <= cdf)
                    {
                        theta = kk;
                        found = true;
                    }
                }
            }
            using Noise = typename std::conditional<FAST, FastNoise, EnvNoise>::type;
            Noise rng(k0, k1, (uint32_t)v, (uint32_t)plan << 16, step, S_VERIF_ENV);
            int tOrigin = 0, t = 0, tEnd = H;
            int witness[NOPP];
#pragma unroll
            for (int o = 0; o < NOPP; o++)
                witness[o] = -1;
            bool failed = false;
            for (; t < H; t++)
            {
                // a warp leaves the loop once all its samples are done (no CTA barrier in
                // the loop: see VERIFY_MIN_BLOCKS)
                if (!__any_sync(0xffffffffu, active))
                    break;
                if constexpr (EGO)
                    if (clearTime(t))
                    {
                        // or once none of them can fail any more (see clearOfEgo)
                        // the group of the earliest branch that a sample has taken or can take
                        const int tau = bs.predTheta == 0 || pt0 != 0 ? t : tOrigin - 1;
                        const int gr = __reduce_min_sync(0xffffffffu, active ? (unsigned)tau : ~0u) / (unsigned)clearPer(H);
                        const ClearBlock<const float> cb(sClear, H);
                        bool clear = *cb.out == 0.0f;
#pragma unroll
                        for (int o = 1; o <= NOPP; o++)
                            clear = clear && clearOfEgoCall(E.dt, E.droneRadius, cb.xy, cb.rho + gr * H, H, t, active, st.pos[2 * o], st.pos[2 * o + 1], st.vel[2 * o],
                                                        st.vel[2 * o + 1], E.maxSpeed[o], E.maxAccel[o], witness[o - 1]);
                        if (clear)
                            break;
                    }
                if (!active)
                    continue;
                rng.begin_step((uint32_t)t);
                int local = t - tOrigin;
                int b = bs.predTheta;
                float e0 = sPlan[(b * T + local) * 2], e1 = sPlan[(b * T + local) * 2 + 1];
                bool branched = false;
                StepOut o;
                if constexpr (EGO)
                {
                    const int row = (bs.predTheta == 0 || pt0 != 0) ? 0 : 1 + (bs.predTheta - 1) * H + (tOrigin - 1);
                    const EgoRow er = egoTab[(size_t)row * H + t];
                    o = envStep<NOPP, NTH, true, true, false, true, FAST, Noise, true>(t, theta, tr, E, e0, e1, st, bs, branched, minConf, rng, &er);
                }
                else
                    o = envStep<NOPP, NTH, true, true, false, true, FAST>(t, theta, tr, E, e0, e1, st, bs, branched, minConf, rng);
                if (branched)
                    tOrigin = t + 1;
                if (o.term == TERM_LOSE)
                {
                    failed = true;
                    active = false;
                    tEnd = t;
                }
                else if (o.term == TERM_WIN || o.term == TERM_OPP_WIN)
                {
                    active = false;
                    tEnd = t;
                }
            }
            if (failed)
                atomicAdd(&hist[tEnd], 1u);
            if (threadIdx.x < tile.count)
            {
                if (dbgFailTime)
                    dbgFailTime[v] = failed ? tEnd : -1;
                if (dbgTheta)
                    dbgTheta[v] = theta;
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < T; i += blockDim.x)
            if (hist[i])
                atomicAdd(&D.fail[plan * T + i], hist[i]);
        if constexpr (PQ)
            fence_before_bulk();
        __syncthreads(); // the next tile's staging and histogram reuse shared memory
    }
}

// perturbation of the next step in the reference layout noise[nbp][M][K][2] (test hook)
__global__ void mppi_noise(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in, float* __restrict__ out)
{
    const MppiDev& D = insts[0];
    const int K = D.cfg.K, M = D.cfg.M, nbp = D.cfg.nth + 1;
    size_t n = (size_t)nbp * M * K;
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    int s = (int)(i % K);
    int bk = (int)(i / K);
    U4 r = draw(D.cfg.k0, D.cfg.k1, (uint32_t)s, (uint32_t)bk, in[0].step, S_MPPI_EPS, 0);
    out[i * 2] = scaled_normal(D.cfg.sigma0, r.x);
    out[i * 2 + 1] = scaled_normal(D.cfg.sigma1, r.y);
}

// ---------------------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------------------
size_t mppiRolloutSmem(int nopp, int nth, int T, int M, bool spl)
{
    return rolloutLayout(nth + 1, T, M, spl, nopp == 1 ? RB / rolloutParts<1>() : RB).total;
}

size_t mppiVerifySmem(int nth, int T)
{
    // the clearance block of the longest verification horizon, T
    return align16(16 + sizeof(EnvParams)) + GRID_FLOATS * 4 + ((((size_t)(nth + 1) * T * 2 * 4) + 15) & ~(size_t)15) +
           ((size_t)T * (3 + CLEAR_GROUPS) + 4) * 4 + (size_t)T * 4;
}

// Lockstep where the batch asks for it, and always by lane pairs with eight hypotheses: warps that
// drift apart fetch that long step's code again and again. Rollouts of two agents of K 3001 x T 61:
// 0.644 ms without the barrier, 0.605 with it; of 24 of K 2048: 3.43 and 3.24; of one of K 64:
// 0.424 and 0.425. With four it gains 4 % at K 65536 and loses up to 12 % at K 1000 with splines,
// with fewer it loses up to 5 %: there the batch chooses.
template <int NOPP, int NTH> constexpr bool rolloutLockstep()
{
    return NOPP == 1 && NTH >= 8;
}

template <int NOPP, int NTH, bool SPL> static cudaError_t launchRolloutS(const LaunchArgs& a, size_t smem)
{
    constexpr bool ALWAYS = rolloutLockstep<NOPP, NTH>();
    auto k = a.queue ? (a.lockstep ? mppi_rollout<NOPP, NTH, SPL, true, true> : mppi_rollout<NOPP, NTH, SPL, true, ALWAYS>)
                     : (a.lockstep ? mppi_rollout<NOPP, NTH, SPL, false, true> : mppi_rollout<NOPP, NTH, SPL, false, ALWAYS>);
    ensureSmem(k, smem);
    const int work = a.nTiles * rolloutParts<NOPP>();
    k<<<a.queue && a.grid < work ? a.grid : work, RB, smem, a.stream>>>(a.mppi, a.mppiIn, a.tiles, a.nTiles, a.queue);
    return cudaGetLastError();
}

template <int NOPP, int NTH> static cudaError_t launchRolloutT(const LaunchArgs& a, bool spl, size_t smem)
{
    return spl ? launchRolloutS<NOPP, NTH, true>(a, smem) : launchRolloutS<NOPP, NTH, false>(a, smem);
}

template <int NOPP, int NTH> static cudaError_t launchVerifyT(const LaunchArgs& a, size_t smem, int* ft, int* th)
{
    auto k = a.exactVerify ? (a.queue ? mppi_verify<NOPP, NTH, true, false> : mppi_verify<NOPP, NTH, false, false>)
             : a.egoTable  ? (a.queue ? mppi_verify<NOPP, NTH, true, true, true> : mppi_verify<NOPP, NTH, false, true, true>)
                           : (a.queue ? mppi_verify<NOPP, NTH, true, true> : mppi_verify<NOPP, NTH, false, true>);
    ensureSmem(k, smem);
    return launchMaybePdl(a.pdl != 0, k, dim3(launchGrid(a)), dim3(VERIFY_TILE), smem, a.stream, a.mppi, a.mppiIn, a.tiles, a.nTiles, a.queue, ft, th);
}

// CTAs of the persistent rollout / verification kernel that fit on one SM at once, for
// the given dynamic shared memory: the persistent grid is at most this times the SMs.
template <int NOPP, int NTH> static int residentT(bool verify, bool spl, size_t smem)
{
    int n = 0;
    if (verify)
    {
        ensureSmem(mppi_verify<NOPP, NTH, true, true>, smem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, mppi_verify<NOPP, NTH, true, true>, VERIFY_TILE, smem);
    }
    else if (spl)
    {
        ensureSmem(mppi_rollout<NOPP, NTH, true, true, rolloutLockstep<NOPP, NTH>()>, smem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, mppi_rollout<NOPP, NTH, true, true, rolloutLockstep<NOPP, NTH>()>, RB, smem);
    }
    else
    {
        ensureSmem(mppi_rollout<NOPP, NTH, false, true, rolloutLockstep<NOPP, NTH>()>, smem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, mppi_rollout<NOPP, NTH, false, true, rolloutLockstep<NOPP, NTH>()>, RB, smem);
    }
    return n;
}

#define DR_DISPATCH(NOPP_, NTH_, CALL)                                                                                                               \
    switch (NOPP_ * 16 + NTH_)                                                                                                                       \
    {                                                                                                                                                \
    case 1 * 16 + 1: return CALL(1, 1);                                                                                                             \
    case 1 * 16 + 2: return CALL(1, 2);                                                                                                             \
    case 1 * 16 + 4: return CALL(1, 4);                                                                                                             \
    case 1 * 16 + 8: return CALL(1, 8);                                                                                                             \
    case 2 * 16 + 2: return CALL(2, 2);                                                                                                             \
    default: return cudaErrorInvalidValue;                                                                                                           \
    }

#define DR_DISPATCH_INT(NOPP_, NTH_, CALL)                                                                                                           \
    switch (NOPP_ * 16 + NTH_)                                                                                                                       \
    {                                                                                                                                                \
    case 1 * 16 + 1: return CALL(1, 1);                                                                                                             \
    case 1 * 16 + 2: return CALL(1, 2);                                                                                                             \
    case 1 * 16 + 4: return CALL(1, 4);                                                                                                             \
    case 1 * 16 + 8: return CALL(1, 8);                                                                                                             \
    case 2 * 16 + 2: return CALL(2, 2);                                                                                                             \
    default: return 0;                                                                                                                               \
    }

bool mppiSupported(int nopp, int nth)
{
    int key = nopp * 16 + nth;
    return key == 17 || key == 18 || key == 20 || key == 24 || key == 34;
}

cudaError_t launchMppiPrologue(const LaunchArgs& a, int nInst, size_t smem)
{
    ensureSmem(mppi_prologue, smem);
    mppi_prologue<<<nInst, 256, smem, a.stream>>>(a.mppi, a.mppiIn, nInst);
    return cudaGetLastError();
}

cudaError_t launchMppiRollout(const LaunchArgs& a, int nopp, int nth, bool spl, size_t smem)
{
#define CALL(P, Q) launchRolloutT<P, Q>(a, spl, smem)
    DR_DISPATCH(nopp, nth, CALL)
#undef CALL
}

// CTAs per (branch plan, knot) of the update: as many as it takes to give every SM two (296
// CTAs of 256 threads), while a thread still has eight samples. One agent of K 65536, 3 plans
// x 20 knots (B200, 1965 MHz): 0.62 ms with one, 0.084 with eight; four agents of K 4096, 3 x 64: one
// either way.
static int updateCluster(int nTiles, int maxK)
{
    int c = 1;
    while (c < 8 && nTiles * c < 296 && maxK >= 2 * c * UB * 8)
        c *= 2;
    return c;
}

template <int NTH> static cudaError_t launchUpdateT(const LaunchArgs& a, int c)
{
    const bool pdl = a.pdl != 0;
    switch (c)
    {
    case 8: return launchCluster(pdl, 8, mppi_update<NTH, 8>, dim3(a.nTiles * 8), dim3(UB), 0, a.stream, a.mppi, a.mppiIn, a.tiles);
    case 4: return launchCluster(pdl, 4, mppi_update<NTH, 4>, dim3(a.nTiles * 4), dim3(UB), 0, a.stream, a.mppi, a.mppiIn, a.tiles);
    case 2: return launchCluster(pdl, 2, mppi_update<NTH, 2>, dim3(a.nTiles * 2), dim3(UB), 0, a.stream, a.mppi, a.mppiIn, a.tiles);
    default: return launchMaybePdl(pdl, mppi_update<NTH, 1>, dim3(a.nTiles), dim3(UB), 0, a.stream, a.mppi, a.mppiIn, a.tiles);
    }
}

cudaError_t launchMppiUpdate(const LaunchArgs& a, int nth, int maxK)
{
    const int c = updateCluster(a.nTiles, maxK);
    switch (nth)
    {
    case 1: return launchUpdateT<1>(a, c);
    case 2: return launchUpdateT<2>(a, c);
    case 4: return launchUpdateT<4>(a, c);
    case 8: return launchUpdateT<8>(a, c);
    default: return cudaErrorInvalidValue;
    }
}

cudaError_t launchShardLocal(const LaunchArgs& a, int nth, float* partial)
{
    switch (nth)
    {
    case 1: mppi_shard_local<1><<<a.nTiles, UB, 0, a.stream>>>(a.mppi, a.mppiIn, a.tiles, partial); break;
    case 2: mppi_shard_local<2><<<a.nTiles, UB, 0, a.stream>>>(a.mppi, a.mppiIn, a.tiles, partial); break;
    case 4: mppi_shard_local<4><<<a.nTiles, UB, 0, a.stream>>>(a.mppi, a.mppiIn, a.tiles, partial); break;
    case 8: mppi_shard_local<8><<<a.nTiles, UB, 0, a.stream>>>(a.mppi, a.mppiIn, a.tiles, partial); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launchShardMerge(cudaStream_t stream, const MppiDev* insts, const MppiIn* in, const float* gathered, int words, int world, float* mins,
                             float* sums)
{
    mppi_shard_merge<<<1, UB, 0, stream>>>(insts, in, gathered, words, world, mins, sums);
    return cudaGetLastError();
}

cudaError_t launchShardApply(cudaStream_t stream, const MppiDev* insts, int nInst, int nth, const float* mins, const float* sums)
{
    mppi_shard_apply<<<nInst, UB, 0, stream>>>(insts, nth + 1, mins, sums);
    return cudaGetLastError();
}

cudaError_t launchMppiAggregate(const LaunchArgs& a, int nth, int K)
{
    int grd = (K + 255) / 256;
    switch (nth)
    {
    case 1: mppi_aggregate<1><<<grd, 256, 0, a.stream>>>(a.mppi, a.mppiIn); break;
    case 2: mppi_aggregate<2><<<grd, 256, 0, a.stream>>>(a.mppi, a.mppiIn); break;
    case 4: mppi_aggregate<4><<<grd, 256, 0, a.stream>>>(a.mppi, a.mppiIn); break;
    case 8: mppi_aggregate<8><<<grd, 256, 0, a.stream>>>(a.mppi, a.mppiIn); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

int mppiResident(int nopp, int nth, bool verify, bool spl, size_t smem)
{
#define CALL(P, Q) residentT<P, Q>(verify, spl, smem)
    DR_DISPATCH_INT(nopp, nth, CALL)
#undef CALL
}

cudaError_t launchMppiVerify(const LaunchArgs& a, int nopp, int nth, size_t smem, int* dbgFailTime, int* dbgTheta)
{
#define CALL(P, Q) launchVerifyT<P, Q>(a, smem, dbgFailTime, dbgTheta)
    DR_DISPATCH(nopp, nth, CALL)
#undef CALL
}

cudaError_t launchEgoTable(cudaStream_t stream, int nopp, int nth, const MppiDev* insts, const MppiIn* in, int nInst, int plan, int maxH)
{
    (void)nopp; // the ego's moves do not depend on the opponents
    // blocks per instance: enough for the rows of the longest horizon of the batch
    const dim3 grid(nInst, (unsigned)((egoRows(nth, maxH) + EGO_CTA_ROWS - 1) / EGO_CTA_ROWS));
    switch (nth)
    {
    case 1: mppi_ego_table<1><<<grid, EGO_WARPS * 32, 0, stream>>>(insts, in, nInst, plan); break;
    case 2: mppi_ego_table<2><<<grid, EGO_WARPS * 32, 0, stream>>>(insts, in, nInst, plan); break;
    case 4: mppi_ego_table<4><<<grid, EGO_WARPS * 32, 0, stream>>>(insts, in, nInst, plan); break;
    case 8: mppi_ego_table<8><<<grid, EGO_WARPS * 32, 0, stream>>>(insts, in, nInst, plan); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launchMppiNoise(const LaunchArgs& a, size_t n, float* out)
{
    mppi_noise<<<(unsigned)((n + 255) / 256), 256, 0, a.stream>>>(a.mppi, a.mppiIn, out);
    return cudaGetLastError();
}

int rolloutSamplesPerBlock(int nth)
{
    return RB / nth;
}

} // namespace dr
