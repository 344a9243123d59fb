// MPPI kernels of the gate race (the reference's kernels.cu compiled with
// USE_ENV_DRONERACE): the rollout with per-branch cost aggregation and the plan
// verification, built like mppi_rollout / mppi_verify (a pair of lanes per (sample,
// hypothesis), resp. a thread per verification sample; state in registers; racelines in
// shared memory, staged by a bulk copy; gate parameters copied to shared memory;
// perturbations from Philox) on the model of gate_model.cuh and gate_pair.cuh. The prologue
// and the update kernels of
// mppi_kernels.cu serve both environments (they see only costs, bookkeeping and plans).
#include <cstdio>

#include <cfloat>
#include <type_traits>

#include "clear.cuh"
#include "common.cuh"
#include "gate_model.cuh"
#include "gate_pair.cuh"
#include "instance.cuh"
#include "launch.h"

namespace dr
{

namespace
{

constexpr int GRB = 256;          // rollout block size
constexpr int GPAIRS = GRB / 2;   // lane pairs of it

__host__ __device__ __forceinline__ size_t ga16(size_t x)
{
    return (x + 15) & ~(size_t)15;
}

__device__ __forceinline__ int gPackInfo(int pt, int bt)
{
    return (pt << 16) | (bt & 0xffff);
}

__device__ __forceinline__ void copyGate(GateParams* dst, const GateParams* src)
{
    for (int i = threadIdx.x; i < GATE_HOST_WORDS; i += blockDim.x)
        ((float*)dst)[i] = ((const float*)src)[i];
    gateDeviceTerms(*dst, *src, threadIdx.x, blockDim.x);
}

struct GateSmem
{
    size_t gp, track, knots, B, vbuf, red, total;
};

__host__ __device__ inline GateSmem gateRolloutLayout(int nbp, int T, int M, bool spl)
{
    GateSmem L;
    size_t off = 16; // mbarrier
    L.gp = off;
    off = ga16(off + sizeof(GateParams));
    L.track = off;
    off = ga16(off + GATE_TRACK_FLOATS * 4);
    L.knots = off;
    off = ga16(off + (size_t)nbp * M * 2 * 4);
    L.B = off;
    if (spl)
        off = ga16(off + (size_t)T * M * 4);
    L.vbuf = off;
    if (spl)
        off = ga16(off + (size_t)((M + 3) & ~3) * 2 * GPAIRS * 4);
    L.red = off;
    off = ga16(off + GRB * 4);
    L.total = off;
    return L;
}

} // namespace

// fullRolloutKernel (kernels.cu:34-171) + aggregateBranchCostsKernel (175-217) on the
// gate race: environmentStep<true, true, false> (kernels.cu:141-143). A pair of lanes per
// (sample, hypothesis), the ego's and the opponent's (gate_pair.cuh). What bounds it is the
// latency of its T dependent steps until the samples fill the device. Against a thread that
// moved both agents (B200, 1965 MHz): one agent of K 512 x 2 x T 40 0.126 -> 0.102 ms, four of
// K 4096 x 2 x T 64 0.33 -> 0.30 beside the verification.
template <int NTH, bool SPL, int ME>
__global__ void __launch_bounds__(GRB) gate_rollout(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in, const Tile* __restrict__ tiles)
{
    constexpr int NBP = NTH + 1;
    extern __shared__ __align__(128) unsigned char smraw[];
    const Tile tile = tiles[blockIdx.x];
    const MppiDev& D = insts[tile.inst];
    const MppiIn& I = in[tile.inst];
    const int K = D.cfg.K, T = D.cfg.T, M = D.cfg.M;
    const GateSmem L = gateRolloutLayout(NBP, T, M, SPL);
    uint64_t* bar = (uint64_t*)smraw;
    GateParams* sG = (GateParams*)(smraw + L.gp);
    float* sTrack = (float*)(smraw + L.track);
    float* sKn = (float*)(smraw + L.knots);
    float* sB = (float*)(smraw + L.B);
    float* vbuf = (float*)(smraw + L.vbuf);
    float* red = (float*)(smraw + L.red);
    const uint32_t knBytes = (uint32_t)ga16((size_t)NBP * M * 2 * 4);
    const uint32_t bBytes = SPL ? (uint32_t)ga16((size_t)T * M * 4) : 0u;
    if (threadIdx.x == 0)
    {
        mbar_init(bar, 1);
        mbar_expect_tx(bar, GATE_TRACK_FLOATS * 4 + knBytes + bBytes);
        if (!D.cfg.dbgNoStage)
        {
            bulk_g2s(sTrack, D.gtrack, GATE_TRACK_FLOATS * 4, bar);
            bulk_g2s(sKn, D.knots, knBytes, bar);
            if (SPL)
                bulk_g2s(sB, D.B, bBytes, bar);
        }
    }
    copyGate(sG, D.gate);
    __syncthreads();
    if (!__syncthreads_and(mbar_wait(bar, 0, D.cfg.waitPolls)))
    {
        rolloutTileTimedOut<NTH>(D, I, tile, K);
        if (threadIdx.x == 0)
            atomicAdd(&D.stats[1], 1);
        return;
    }
    const GateParams& G = *sG;
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
    const int pt0 = findConfident<NTH>(bs.belief, minConf);
    bs.predTheta = pt0;
    bs.branchingTime = pt0 == 0 ? -1 : 0;
    const bool compatible = (pt0 == 0 || pt0 == th + 1);
    bool active = valid && compatible;
    float cost = active ? 0.0f : INFINITY;
    GLane st;
    loadGLane(st, I.gstate, role ? 1 - ME : ME);
    float decay = 1.0f;
    int tOrigin = 0, curB = -1;
    for (int t = 0; t < T; t++)
    {
        // the lanes still rolling out: whole pairs, since both lanes of one decide alike
        const unsigned mask = __ballot_sync(0xffffffffu, active);
        if (mask == 0u)
            break;
        if (!active)
            continue;
        const int local = t - tOrigin;
        const int b = bs.predTheta;
        PairNoise noise{k0, k1, (uint32_t)s, ((uint32_t)th << 16) | (uint32_t)t, step, S_MPPI_ROLL_ENV};
        float ctl0, ctl1, opp0 = 0.0f, opp1 = 0.0f;
        if constexpr (SPL)
        {
            if (G.pidNoise[th] != 0.0f)
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
                    float* v = vbuf + ((m >> 2) * 2 * GPAIRS + pair * 2) * 4 + (m & 3);
                    v[0] = sKn[(b * M + m) * 2 + 0] + e0;
                    v[4] = sKn[(b * M + m) * 2 + 1] + e1;
                }
                curB = b;
            }
            __syncwarp(mask);
            // a lane evaluates one axis of the control
            pairBoth(mask, role, splineSum(sB + local * M, vbuf, 2 * GPAIRS, threadIdx.x, M), ctl0, ctl1);
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
        const StepOut o = gatePairStep<NTH, ME>(mask, role, t, th, sTrack, G, ctl0, ctl1, opp0, opp1, st, bs, branched, minConf, noise);
        if (branched)
            tOrigin = t + 1;
        if (o.term != TERM_NONE)
            active = false;
        cost += gateStateCost(o, G, D.cfg.w) * decay;
        decay *= DECAY;
    }
    {
        // gateFinalCost: the ego's advance and, where it is weighted, the opponent's
        float advE, advO;
        pairBoth(0xffffffffu, role, laneAdvance(st, G), advE, advO);
        if (valid && compatible)
        {
            float last = -D.cfg.w.finalAdvWeight * advE;
            if (D.cfg.w.finalOppAdvWeight != 0.0f)
                last += D.cfg.w.finalOppAdvWeight * advO;
            cost += last;
        }
    }
    if (valid && role == 0)
    {
        D.costsTrue[th * K + s] = cost;
        D.binfo[th * K + s] = gPackInfo(bs.predTheta, bs.branchingTime);
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

// The clearance block of a plan (ClearBlock; plan 0 the new one, 1 the previous one, 2 both)
// from the ego's trajectories (no branch, or a branch taken at a step: the rows of the
// strategic race's ego tables), which need the plan alone: the controls clamped, position,
// velocity and speed cap as gateStep takes them, up to rounding (clearOfEgo's slack). The time
// is one trajectory's chain of steps, so GCLEAR_STEPS lanes take as many steps of a row at a
// time: each runs the short chain, with the trajectory with no branch beside it, and then
// judges its own step (25 -> 12 us a plan of four agents, H 40, two hypotheses, against a
// lane per row; B200, 1965 MHz). Only for an ego that draws no noise.
constexpr int GCLEAR = 128, GCLEAR_STEPS = 8, GCLEAR_ROWS = GCLEAR / GCLEAR_STEPS;

template <int NTH, int ME>
__global__ void __launch_bounds__(GCLEAR) gate_clear(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in, int nInst, int plans)
{
    __shared__ GateParams sG; // without its belief terms
    __shared__ float2 ctl[(NTH + 1) * DR_MAX_T];
    const int inst = blockIdx.x;
    if (inst >= nInst)
        return;
    const MppiDev& D = insts[inst];
    const MppiIn& I = in[inst];
    if (!D.clear)
        return;
    const int H = D.cfg.H, T = D.cfg.T, rows = egoRows(NTH, H);
    for (int i = threadIdx.x; i < GATE_HOST_WORDS; i += GCLEAR)
        ((float*)&sG)[i] = ((const float*)D.gate)[i];
    const GateParams& G = sG;
    float belief[NTH];
#pragma unroll
    for (int i = 0; i < NTH; i++)
        belief[i] = I.belief[i];
    const int pt0 = findConfident<NTH>(belief, D.cfg.minConf);
    const int nRows = pt0 != 0 ? 1 : rows; // a confident initial belief never branches
    const int sub = threadIdx.x % GCLEAR_STEPS; // this lane's step
    for (int plan = plans == 1 ? 1 : 0; plan <= (plans == 0 ? 0 : 1); plan++)
    {
        __syncthreads(); // the parameters, and the previous plan's rows are done with ctl
        const float2* P = (const float2*)(plan == 0 ? D.dense : D.prevDense);
        const float maxAccel = G.maxAccel[ME], maxSpeed = G.maxSpeed[ME], dt = G.dt;
        for (int i = threadIdx.x; i < (NTH + 1) * T; i += GCLEAR)
        {
            const float2 u = P[i];
            const float sq = u.x * u.x + u.y * u.y;
            const float f = sq > maxAccel * maxAccel ? mdivsqrt<true>(maxAccel, sq) : 1.0f;
            ctl[i] = make_float2(u.x * f, u.y * f);
        }
        __syncthreads();
        const ClearBlock<float> cb(D.clear + (size_t)plan * clearWords(H), H);
        auto advance = [&](float2 u, float (&p)[2], float (&v)[2]) {
            p[0] += dt * v[0];
            p[1] += dt * v[1];
            v[0] += dt * u.x;
            v[1] += dt * u.y;
            const float sq = v[0] * v[0] + v[1] * v[1];
            if (sq > maxSpeed * maxSpeed)
            {
                const float sc = mdivsqrt<true>(maxSpeed, sq);
                v[0] *= sc;
                v[1] *= sc;
            }
        };
        for (int r = blockIdx.y * GCLEAR_ROWS + threadIdx.x / GCLEAR_STEPS; r < nRows; r += gridDim.y * GCLEAR_ROWS)
        {
            const int bb = r > 0 ? 1 + (r - 1) / H : 0, tb = r > 0 ? (r - 1) % H : H;
            float p[2] = {I.gstate.pos[2 * ME], I.gstate.pos[2 * ME + 1]}, v[2] = {I.gstate.vel[2 * ME], I.gstate.vel[2 * ME + 1]};
            float bp[2] = {p[0], p[1]}, bv[2] = {v[0], v[1]};
            for (int t0 = 0; t0 < H; t0 += GCLEAR_STEPS)
            {
                const int t = t0 + sub;
                float x = 0.0f, y = 0.0f, bx = 0.0f, by = 0.0f; // after step t
#pragma unroll
                for (int u = 0; u < GCLEAR_STEPS; u++)
                {
                    const int w = t0 + u;
                    if (w < H)
                    {
                        advance(ctl[(w <= tb ? pt0 : bb) * T + (w <= tb ? w : w - tb - 1)], p, v);
                        advance(ctl[pt0 * T + w], bp, bv);
                    }
                    if (u == sub)
                    {
                        x = p[0];
                        y = p[1];
                        bx = bp[0];
                        by = bp[1];
                    }
                }
                if (t >= H)
                    continue;
                // the ego's own boundary distance (the opponent far away), and some slack: the
                // verification moves the ego itself
                GState s;
                s.pos[2 * ME] = x;
                s.pos[2 * ME + 1] = y;
                s.pos[2 * (1 - ME)] = s.pos[2 * (1 - ME) + 1] = INFINITY;
                const bool off = !(gateBoundaryDist<ME, true>(s, G) >= G.droneRadius + 2e-3f + 4.8e-7f * (float)H * (fabsf(x) + fabsf(y)));
                if (r == 0)
                {
                    cb.xy[2 * t] = x;
                    cb.xy[2 * t + 1] = y;
                    if (off)
                        *cb.out = 1.0f;
                }
                else if (t > tb) // up to its branching step a row is the first one
                {
                    // off the arena, or a distance that is no number: infinitely far
                    float d = msqrt<true>((x - bx) * (x - bx) + (y - by) * (y - by));
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

// verifyNominalFailureKernel (kernels.cu:488-551) on the gate race:
// environmentStep<true, true, false, false>; one thread per sample, each plan's tiles in
// the grid, the CTA's warps in step (a barrier per step) in the exact flavour only.
// Two 512-thread CTAs per SM (64 registers a thread, ~20 bytes spilled) for up to four
// hypotheses: measured on the 4 x 2 x 2^17 x 40 gate verification (B200, 1965 MHz)
// 2.66 ms against 3.42 ms with one CTA per SM (128 registers, no spills).
#ifndef GATE_VERIFY_MIN_BLOCKS
#define GATE_VERIFY_MIN_BLOCKS 2
#endif
template <int NTH> constexpr int gateVerifyMinBlocks()
{
    return NTH <= 4 ? GATE_VERIFY_MIN_BLOCKS : 1;
}
// FAST: the verification's fast arithmetic flavour and noise source (the default; the
// exact flavour reproduces the oracle's per-sample results and serves parity tests), as
// in the strategic race's mppi_verify; its warps step without a CTA barrier.
// CLEAR (with FAST): warps whose samples can no longer collide leave, and tiles none of whose
// samples can end at once, by the plan's clearance block (gate_clear, clearOfEgo), as in
// mppi_verify; a sample fails at the first step with boundary distance below the drone radius,
// which the ego's own part of that distance, known with its trajectory, and the opponents'
// distance decide.
template <int NTH, int ME, bool FAST, bool CLEAR = false>
__global__ void __launch_bounds__(VERIFY_TILE, (gateVerifyMinBlocks<NTH>())) gate_verify(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in, const Tile* __restrict__ tiles,
                                                             int* __restrict__ dbgFailTime, int* __restrict__ dbgTheta)
{
    constexpr int NBP = NTH + 1;
    extern __shared__ __align__(128) unsigned char smraw[];
    const Tile tile = tiles[blockIdx.x];
    const MppiDev& D = insts[tile.inst];
    const MppiIn& I = in[tile.inst];
    const int T = D.cfg.T, H = D.cfg.H;
    const int plan = tile.aux;
    uint64_t* bar = (uint64_t*)smraw;
    GateParams* sG = (GateParams*)(smraw + 16);
    const size_t offT = ga16(16 + sizeof(GateParams));
    float* sTrack = (float*)(smraw + offT);
    float* sPlan = (float*)(smraw + offT + GATE_TRACK_FLOATS * 4);
    const uint32_t planBytes = (uint32_t)ga16((size_t)NBP * T * 2 * 4);
    const uint32_t clearBytes = CLEAR ? (uint32_t)clearWords(H) * 4u : 0u;
    float* sClear = (float*)(smraw + offT + GATE_TRACK_FLOATS * 4 + planBytes);
    unsigned* hist = (unsigned*)((unsigned char*)sClear + clearBytes);
    constexpr int opp = 1 - ME;
    if constexpr (CLEAR)
    {
        // every sample starts from the same state
        int witness = -1;
        const ClearBlock<const float> cb(D.clear + (size_t)plan * clearWords(H), H);
        if (!dbgTheta && *cb.out == 0.0f &&
            clearOfEgo(D.gate->dt, D.gate->droneRadius, cb.xy, cb.all, H, 0, true, I.gstate.pos[2 * opp], I.gstate.pos[2 * opp + 1], I.gstate.vel[2 * opp],
                       I.gstate.vel[2 * opp + 1], D.gate->maxSpeed[opp], D.gate->maxAccel[opp], witness))
            return;
    }
    if (threadIdx.x == 0)
    {
        mbar_init(bar, 1);
        mbar_expect_tx(bar, GATE_TRACK_FLOATS * 4 + planBytes + clearBytes);
        if (!D.cfg.dbgNoStage)
        {
            bulk_g2s(sTrack, D.gtrack, GATE_TRACK_FLOATS * 4, bar);
            bulk_g2s(sPlan, plan == 0 ? D.dense : D.prevDense, planBytes, bar);
            if (CLEAR)
                bulk_g2s(sClear, D.clear + (size_t)plan * clearWords(H), clearBytes, bar);
        }
    }
    copyGate(sG, D.gate);
    for (int i = threadIdx.x; i < T; i += blockDim.x)
        hist[i] = 0u;
    __syncthreads();
    if (!__syncthreads_and(mbar_wait(bar, 0, D.cfg.waitPolls)))
    {
        if (threadIdx.x == 0)
            atomicAdd(&D.stats[1], 1);
        return;
    }
    if constexpr (CLEAR)
    {
        clearSuffix(sClear, H);
        __syncthreads();
    }
    const GateParams& G = *sG;
    const int v = tile.s0 + threadIdx.x;
    bool active = threadIdx.x < tile.count; // idle lanes of a partial tile still take the barriers
    {
        const float minConf = D.cfg.minConf;
        const float gateMargin = D.cfg.gateMargin;
        GState st;
        loadGState(st, I.gstate);
        BState<NTH> bs;
#pragma unroll
        for (int i = 0; i < NTH; i++)
            bs.belief[i] = I.belief[i];
        bs.predTheta = findConfident<NTH>(bs.belief, minConf);
        bs.branchingTime = bs.predTheta == 0 ? -1 : 0;
        const int pt0 = bs.predTheta;
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
        int tOrigin = 0, tEnd = H, next = 2;
        bool failed = false;
        for (int t = 0; t < H; t++)
        {
            // exact flavour: every thread takes this barrier once per step (H is uniform),
            // which keeps the warps on the same step, where they fetch the same
            // instructions, and ends the loop once all samples of the CTA are done; fast
            // flavour: a warp leaves once its samples are done
            if constexpr (FAST)
            {
                if (!__any_sync(0xffffffffu, active))
                    break;
            }
            else if (!__syncthreads_or(active))
                break;
            if constexpr (CLEAR)
                if (t == next)
                {
                    int witness = -1, wait = 0;
                    // the group of the earliest branch that a sample has taken or can take
                    const int tau = bs.predTheta == 0 || pt0 != 0 ? t : tOrigin - 1;
                    const int gr = __reduce_min_sync(0xffffffffu, active ? (unsigned)tau : ~0u) / (unsigned)clearPer(H);
                    const ClearBlock<const float> cb(sClear, H);
                    if (*cb.out == 0.0f && clearOfEgo(G.dt, G.droneRadius, cb.xy, cb.rho + gr * H, H, t, active, st.pos[2 * opp], st.pos[2 * opp + 1],
                                                      st.vel[2 * opp], st.vel[2 * opp + 1], G.maxSpeed[opp], G.maxAccel[opp], witness, &wait))
                        break;
                    next = t + max(t == 2 ? 2 : 4, wait);
                }
            if (!active)
                continue;
            rng.begin_step((uint32_t)t);
            int local = t - tOrigin;
            int b = bs.predTheta;
            float e0 = sPlan[(b * T + local) * 2], e1 = sPlan[(b * T + local) * 2 + 1];
            bool branched = false;
            StepOut o = gateStep<NTH, true, true, false, false, ME, false, FAST, Noise>(t, theta, sTrack, G, e0, e1, st, bs, branched, minConf, rng, gateMargin);
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
}

// One true-dynamics step (environmentStep with noise, as the engine's dynStep).
template <int NTH, int ME>
__global__ void gate_env_step_kernel(const GateParams* __restrict__ gp, const float* __restrict__ track, int trueTheta, float a0, float a1,
                                     dr_gate_state* st, float* belief, int updateBelief, uint32_t k0, uint32_t k1, uint32_t step, int* term)
{
    __shared__ GateParams sG;
    if (threadIdx.x == 0)
    {
        sG = *gp;
        gateDeviceTerms(sG, *gp, 0, 1);
    }
    __syncthreads();
    if (threadIdx.x != 0)
        return;
    GState s;
    loadGState(s, *st);
    BState<NTH> bs;
    for (int i = 0; i < NTH; i++)
        bs.belief[i] = belief[i];
    bs.predTheta = 0;
    bs.branchingTime = -1;
    EnvNoise rng(k0, k1, 0u, 0u, step, S_ENV_STEP);
    rng.begin_step(0);
    bool branched = false;
    StepOut o;
    if (updateBelief)
        o = gateStep<NTH, true, false, false, true, ME>(0, trueTheta, track, sG, a0, a1, s, bs, branched, 2.0f, rng, 0.0f);
    else
        o = gateStep<NTH, false, false, false, true, ME>(0, trueTheta, track, sG, a0, a1, s, bs, branched, 2.0f, rng, 0.0f);
    storeGState(*st, s);
    for (int i = 0; i < NTH; i++)
        belief[i] = bs.belief[i];
    *term = o.term;
}

// The same for every controller of a batch (dr_mppi_batch_env_step_device): one CTA per
// controller, its gate parameters and racelines, the action it sent, the noise stream of
// its step counter.
template <int NTH, int ME>
__global__ void gate_batch_env_step(const MppiDev* __restrict__ insts, const MppiIn* __restrict__ in, const int* __restrict__ trueTheta,
                                    const float* __restrict__ actions, dr_gate_state* __restrict__ states, float* __restrict__ beliefs, int updateBelief,
                                    uint32_t k0, uint32_t k1, int* __restrict__ terms)
{
    __shared__ GateParams sG;
    const int inst = blockIdx.x;
    const MppiDev& D = insts[inst];
    if (threadIdx.x == 0)
    {
        sG = *D.gate;
        gateDeviceTerms(sG, *D.gate, 0, 1);
    }
    __syncthreads();
    if (threadIdx.x != 0)
        return;
    GState s;
    loadGState(s, states[inst]);
    float* belief = beliefs + (size_t)inst * DR_MAX_THETA;
    BState<NTH> bs;
    for (int i = 0; i < NTH; i++)
        bs.belief[i] = belief[i];
    bs.predTheta = 0;
    bs.branchingTime = -1;
    EnvNoise rng(k0, k1, 0u, 0u, in[inst].step, S_ENV_STEP);
    rng.begin_step(0);
    bool branched = false;
    const float a0 = actions[inst * 2], a1 = actions[inst * 2 + 1];
    StepOut o;
    if (updateBelief)
        o = gateStep<NTH, true, false, false, true, ME>(0, trueTheta[inst], D.gtrack, sG, a0, a1, s, bs, branched, 2.0f, rng, 0.0f);
    else
        o = gateStep<NTH, false, false, false, true, ME>(0, trueTheta[inst], D.gtrack, sG, a0, a1, s, bs, branched, 2.0f, rng, 0.0f);
    storeGState(states[inst], s);
    for (int i = 0; i < NTH; i++)
        belief[i] = bs.belief[i];
    terms[inst] = o.term;
}

// ---------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------
bool gateSupported(int nth)
{
    return nth == 1 || nth == 2 || nth == 4 || nth == 8;
}

size_t gateRolloutSmem(int nth, int T, int M, bool spl)
{
    return gateRolloutLayout(nth + 1, T, M, spl).total;
}

size_t gateVerifySmem(int nth, int T)
{
    // the clearance block of the longest verification horizon, T
    return ga16(16 + sizeof(GateParams)) + GATE_TRACK_FLOATS * 4 + ga16((size_t)(nth + 1) * T * 2 * 4) + ((size_t)T * (3 + CLEAR_GROUPS) + 4) * 4 +
           (size_t)T * 4;
}

int gateRolloutSamplesPerBlock(int nth)
{
    return GPAIRS / nth;
}

template <int NTH, int ME> static cudaError_t launchGateRolloutT(const LaunchArgs& a, bool spl, size_t smem)
{
    if (spl)
    {
        auto k = gate_rollout<NTH, true, ME>;
        ensureSmem(k, smem);
        k<<<a.nTiles, GRB, smem, a.stream>>>(a.mppi, a.mppiIn, a.tiles);
    }
    else
    {
        auto k = gate_rollout<NTH, false, ME>;
        ensureSmem(k, smem);
        k<<<a.nTiles, GRB, smem, a.stream>>>(a.mppi, a.mppiIn, a.tiles);
    }
    return cudaGetLastError();
}

template <int NTH, int ME> static cudaError_t launchGateVerifyT(const LaunchArgs& a, size_t smem, int* ft, int* th)
{
    auto k = a.exactVerify ? gate_verify<NTH, ME, false> : a.egoTable ? gate_verify<NTH, ME, true, true> : gate_verify<NTH, ME, true>;
    ensureSmem(k, smem);
    k<<<a.nTiles, VERIFY_TILE, smem, a.stream>>>(a.mppi, a.mppiIn, a.tiles, ft, th);
    return cudaGetLastError();
}

// (n_theta, ego index) -> instantiation
#define GATE_DISPATCH(NTH_, ME_, CALL)                                                                                                                \
    switch ((NTH_) * 2 + (ME_))                                                                                                                      \
    {                                                                                                                                                \
    case 1 * 2 + 0: return CALL(1, 0);                                                                                                              \
    case 1 * 2 + 1: return CALL(1, 1);                                                                                                              \
    case 2 * 2 + 0: return CALL(2, 0);                                                                                                              \
    case 2 * 2 + 1: return CALL(2, 1);                                                                                                              \
    case 4 * 2 + 0: return CALL(4, 0);                                                                                                              \
    case 4 * 2 + 1: return CALL(4, 1);                                                                                                              \
    case 8 * 2 + 0: return CALL(8, 0);                                                                                                              \
    case 8 * 2 + 1: return CALL(8, 1);                                                                                                              \
    default: return cudaErrorInvalidValue;                                                                                                           \
    }

cudaError_t launchGateRollout(const LaunchArgs& a, int nth, int me, bool spl, size_t smem)
{
#define CALL(P, Q) launchGateRolloutT<P, Q>(a, spl, smem)
    GATE_DISPATCH(nth, me, CALL)
#undef CALL
}

template <int NTH, int ME>
static cudaError_t launchGateClearT(cudaStream_t stream, const MppiDev* insts, const MppiIn* in, int nInst, int plans, int maxH)
{
    const dim3 grid(nInst, (unsigned)((egoRows(NTH, maxH) + GCLEAR_ROWS - 1) / GCLEAR_ROWS));
    gate_clear<NTH, ME><<<grid, GCLEAR, 0, stream>>>(insts, in, nInst, plans);
    return cudaGetLastError();
}

cudaError_t launchGateClear(cudaStream_t stream, int nth, int me, const MppiDev* insts, const MppiIn* in, int nInst, int plans, int maxH)
{
#define CALL(P, Q) launchGateClearT<P, Q>(stream, insts, in, nInst, plans, maxH)
    GATE_DISPATCH(nth, me, CALL)
#undef CALL
}

cudaError_t launchGateVerify(const LaunchArgs& a, int nth, int me, size_t smem, int* dbgFailTime, int* dbgTheta)
{
#define CALL(P, Q) launchGateVerifyT<P, Q>(a, smem, dbgFailTime, dbgTheta)
    GATE_DISPATCH(nth, me, CALL)
#undef CALL
}

template <int NTH, int ME>
static cudaError_t launchGateEnvStepT(cudaStream_t stream, const GateParams* gp, const float* track, int trueTheta, float a0, float a1, dr_gate_state* st,
                                      float* belief, int updateBelief, uint32_t k0, uint32_t k1, uint32_t step, int* term)
{
    gate_env_step_kernel<NTH, ME><<<1, 32, 0, stream>>>(gp, track, trueTheta, a0, a1, st, belief, updateBelief, k0, k1, step, term);
    return cudaGetLastError();
}

template <int NTH, int ME>
static cudaError_t launchGateBatchEnvStepT(cudaStream_t stream, const MppiDev* insts, const MppiIn* in, int nInst, const int* trueTheta, const float* actions,
                                           dr_gate_state* states, float* beliefs, int updateBelief, uint32_t k0, uint32_t k1, int* terms)
{
    gate_batch_env_step<NTH, ME><<<nInst, 32, 0, stream>>>(insts, in, trueTheta, actions, states, beliefs, updateBelief, k0, k1, terms);
    return cudaGetLastError();
}

cudaError_t launchGateBatchEnvStep(cudaStream_t stream, int nth, int me, const MppiDev* insts, const MppiIn* in, int nInst, const int* trueTheta,
                                   const float* actions, dr_gate_state* states, float* beliefs, int updateBelief, uint32_t k0, uint32_t k1, int* terms)
{
#define CALL(P, Q) launchGateBatchEnvStepT<P, Q>(stream, insts, in, nInst, trueTheta, actions, states, beliefs, updateBelief, k0, k1, terms)
    GATE_DISPATCH(nth, me, CALL)
#undef CALL
}

cudaError_t launchGateEnvStep(cudaStream_t stream, int nth, int me, const GateParams* gp, const float* track, int trueTheta, float a0, float a1,
                              dr_gate_state* st, float* belief, int updateBelief, uint32_t k0, uint32_t k1, uint32_t step, int* term)
{
#define CALL(P, Q) launchGateEnvStepT<P, Q>(stream, gp, track, trueTheta, a0, a1, st, belief, updateBelief, k0, k1, step, term)
    GATE_DISPATCH(nth, me, CALL)
#undef CALL
}

} // namespace dr
