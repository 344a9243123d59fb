// PR-MPPI on the gate race: the reference's PR-MPPI kernels (src/prmppi_kernels.cu)
// compiled with USE_ENV_DRONERACE, whose cost functions (include/costs.cuh:44-86) call the
// gate race's trackBoundaryDist / isWinner / isOppWinner / getAdvance
// (include/environments/env_dronerace.h:262-401). The step is the gate model's
// environment step (gate_model.cuh, gateStep<UPD = false, BR = false, ADDMARGIN = true,
// LOSE = true>), as PRMPPIfullRolloutKernel calls environmentStep<false, false, true>.
//
//   gate_pr_rollout      PRMPPIfullRolloutKernel (:55-130) with the per-sample average
//                        over hypotheses (PRMPPIcostAvgKernel, :134-166) in its epilogue;
//                        512-thread CTAs whose warps take a barrier every step, for an ego
//                        that draws noise; otherwise gate_pr_rollout_shared (and
//                        gate_pr_candidates_shared), one ego per sample
//   gate_pr_candidates   PRMPPIcomputeCandidateCostKernel (:285-347), the safety re-check
//                        (PRMPPIcomputeSafeCostKernel, :350-393) for both candidates, and
//                        the choice (prmppi_controller.cu:232-304)
// The prologue (shift, hypothesis draw) and the weighted averages do not depend on the
// environment and are the strategic race's kernels.
#include "common.cuh"
#include "gate_model.cuh"
#include "gate_pair.cuh"
#include "instance.cuh"
#include "launch.h"
#include "pr_split.cuh"

namespace dr
{

namespace
{
constexpr int GPR_TILE = 512;
constexpr int GPR_CAND = 128;

template <int NTH> constexpr int gatePrMinBlocks()
{
    return NTH <= 4 ? 2 : 1;
}

__host__ __device__ __forceinline__ size_t gp16(size_t x)
{
    return (x + 15) & ~(size_t)15;
}

__device__ __forceinline__ void copyGateP(GateParams* dst, const GateParams* src)
{
    for (int i = threadIdx.x; i < GATE_HOST_WORDS; i += blockDim.x)
        ((float*)dst)[i] = ((const float*)src)[i];
    gateDeviceTerms(*dst, *src, threadIdx.x, blockDim.x);
}

// PRMPPIstateCost (costs.cuh:44-63) on the gate race: trackBoundaryDist<true> is -1 once
// the opponent has won.
__device__ __forceinline__ float gatePrStateCost(const StepOut& o, const GateParams& G, const PrCfgDev& c)
{
    float cost = 0.0f;
    float bd = o.oppWon ? -1.0f : o.bdRaw;
    float danger = c.boundaryThresholdFactor * G.droneRadius;
    if (bd < danger)
        cost += c.boundaryCost * powf(bd / G.droneRadius, 2.0f);
    if (o.winner)
        cost -= c.winCost;
    if (o.oppWon)
        cost += c.oppWinCost;
    return cost;
}

// PRMPPIsafetyCost (costs.cuh:78-86): droneRadius * collDistFactor - trackBoundaryDist<false>,
// the product fused into the subtraction as in the strategic race's kernel
__device__ __forceinline__ float gatePrSafetyCost(const StepOut& o, const GateParams& G, float collDistFactor)
{
    return __fmaf_rn(G.droneRadius, collDistFactor, -o.bdRaw);
}

struct GatePrSmem
{
    size_t gp, track, nom, red, total;
};

__host__ __device__ inline GatePrSmem gatePrLayout(int T)
{
    GatePrSmem L;
    size_t off = 16; // mbarrier
    L.gp = off;
    off = gp16(off + sizeof(GateParams));
    L.track = off;
    off = gp16(off + GATE_TRACK_FLOATS * 4);
    L.nom = off;
    off = gp16(off + (size_t)T * 2 * 4);
    L.red = off;
    off = gp16(off + (size_t)GPR_TILE * 2 * 4);
    L.total = off;
    return L;
}
} // namespace

// tile: inst, s0 (first sample), count (samples), aux (0 nominal / 1 robust)
template <int NTH, int ME>
__global__ void __launch_bounds__(GPR_TILE, gatePrMinBlocks<NTH>()) gate_pr_rollout(const PrDev* __restrict__ insts, const PrIn* __restrict__ in,
                                                                                const Tile* __restrict__ tiles)
{
    extern __shared__ __align__(128) unsigned char smraw[];
    const Tile tile = tiles[blockIdx.x];
    const PrDev& D = insts[tile.inst];
    const PrIn& I = in[tile.inst];
    const int K = D.cfg.K, T = D.cfg.T, P = D.cfg.P;
    const int robust = tile.aux;
    const GatePrSmem L = gatePrLayout(T);
    uint64_t* bar = (uint64_t*)smraw;
    GateParams* sG = (GateParams*)(smraw + L.gp);
    float* sTrack = (float*)(smraw + L.track);
    float* sNom = (float*)(smraw + L.nom);
    float* red = (float*)(smraw + L.red);
    const uint32_t nomBytes = (uint32_t)gp16((size_t)T * 2 * 4);
    if (threadIdx.x == 0)
    {
        mbar_init(bar, 1);
        mbar_expect_tx(bar, GATE_TRACK_FLOATS * 4 + nomBytes);
        bulk_g2s(sTrack, D.gtrack, GATE_TRACK_FLOATS * 4, bar);
        bulk_g2s(sNom, robust ? D.rob : D.nom, nomBytes, bar);
    }
    copyGateP(sG, D.gate);
    __syncthreads();
    if (!__syncthreads_and(mbar_wait(bar, 0)))
    {
        if (threadIdx.x == 0)
            atomicAdd(&D.stats[1], 1);
        return;
    }
    const GateParams& G = *sG;
    const int spb = GPR_TILE / P;
    const int sl = threadIdx.x / P, p = threadIdx.x % P;
    const int s = tile.s0 + sl;
    const bool valid = sl < spb && sl < tile.count;
    float running = 0.0f, safe = -INFINITY;
    {
        const int theta = D.thetas[p];
        GState st;
        loadGState(st, I.gstate);
        BState<NTH> bs{};
        const uint32_t k0 = D.cfg.k0, k1 = D.cfg.k1, step = I.step;
        EnvNoise rng(k0, k1, (uint32_t)s, ((((uint32_t)robust << 8) | (uint32_t)p) << 16), step, S_PR_ROLL_ENV);
        float decay = 1.0f;
        bool active = valid;
        for (int t = 0; t < T; t++)
        {
            // every thread of the CTA takes this barrier once per step (T is uniform)
            if (!__syncthreads_or(active))
                break;
            if (!active)
                continue;
            rng.begin_step((uint32_t)t);
            U4 r = draw(k0, k1, (uint32_t)s, (uint32_t)t, step, S_PR_EPS, 0);
            float ego0 = sNom[t * 2] + scaled_normal(D.cfg.sigma0, r.x);
            float ego1 = sNom[t * 2 + 1] + scaled_normal(D.cfg.sigma1, r.y);
            bool branched = false;
            StepOut o = gateStep<NTH, false, false, true, true, ME, true>(t, theta, sTrack, G, ego0, ego1, st, bs, branched, 0.0f, rng, D.cfg.gateMargin);
            if (o.term != TERM_NONE)
                active = false;
            running += decay * gatePrStateCost(o, G, D.cfg);
            safe = fmaxf(safe, gatePrSafetyCost(o, G, D.cfg.collDistFactor));
            decay *= DECAY;
        }
        if (valid)
        {
            running += gateFinalCost<ME>(st, G, D.cfg.finalAdvWeight, D.cfg.finalOppAdvWeight);
            float* out = robust ? D.costRob : D.costNom;
            out[((size_t)p * K + s) * 2 + 0] = running;
            out[((size_t)p * K + s) * 2 + 1] = safe;
        }
    }
    red[threadIdx.x * 2] = running;
    red[threadIdx.x * 2 + 1] = safe;
    __syncthreads();
    // PRMPPIcostAvgKernel (prmppi_kernels.cu:134-166)
    if (valid && p == 0)
    {
        float avg = 0.0f, maxSafe = -INFINITY;
        for (int q = 0; q < P; q++)
        {
            avg += red[(sl * P + q) * 2];
            maxSafe = fmaxf(maxSafe, red[(sl * P + q) * 2 + 1]);
        }
        avg /= (float)P;
        float full = avg + ((maxSafe > 0.0f) ? D.cfg.safetyWeight : 0.0f);
        D.avg[((size_t)robust * K + s) * 2 + 0] = full;
        D.avg[((size_t)robust * K + s) * 2 + 1] = maxSafe;
        if (!isfinite(full))
            atomicAdd(&D.stats[0], 1);
    }
}

// The candidate choice (prmppi_controller.cu:236-256) and the safety decision (:264-275), by
// thread 0, then the new plans; all threads of the instance's CTA, the candidates' costs
// written and synchronised.
__device__ __forceinline__ void gatePrChoose(const PrDev& D, const float* sC1, const float* sC2, int T, int P, int* sChosen)
{
    if (threadIdx.x == 0)
    {
        float c1 = 0.0f, c2 = 0.0f;
        for (int p = 0; p < P; ++p)
        {
            c1 += D.candFull[p];
            c2 += D.candFull[P + p];
        }
        c1 /= (float)P;
        c2 /= (float)P;
        D.decision[0] = c2 < c1; // resetNom
        int chosen = (c1 <= c2) ? 0 : 1;
        int useNom = 1;
        for (int p = 0; p < P; p++)
            if (D.candSafe[chosen * P + p] > 0.0f)
            {
                useNom = 0;
                break;
            }
        D.decision[1] = useNom;
        D.decision[2] = chosen;
        *sChosen = chosen;
    }
    __syncthreads();
    const float* ch = *sChosen ? sC2 : sC1;
    for (int i = threadIdx.x; i < T * 2; i += blockDim.x)
    {
        D.nom[i] = ch[i];
        D.rob[i] = D.robWork[i];
    }
}

// one block per instance: threads (kind, cand, p), kind 0 = full cost, 1 = safety re-check
template <int NTH, int ME>
__global__ void __launch_bounds__(GPR_CAND) gate_pr_candidates(const PrDev* __restrict__ insts, const PrIn* __restrict__ in, int nInst)
{
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ int sChosen;
    const int inst = blockIdx.x;
    if (inst >= nInst)
        return;
    const PrDev& D = insts[inst];
    const PrIn& I = in[inst];
    const int T = D.cfg.T, P = D.cfg.P;
    uint64_t* bar = (uint64_t*)smraw;
    GateParams* sG = (GateParams*)(smraw + 16);
    const size_t offT = gp16(16 + sizeof(GateParams));
    float* sTrack = (float*)(smraw + offT);
    float* sC1 = (float*)(smraw + offT + GATE_TRACK_FLOATS * 4);
    const uint32_t cb = (uint32_t)gp16((size_t)T * 2 * 4);
    float* sC2 = (float*)((unsigned char*)sC1 + cb);
    if (threadIdx.x == 0)
    {
        mbar_init(bar, 1);
        mbar_expect_tx(bar, GATE_TRACK_FLOATS * 4 + 2 * cb);
        bulk_g2s(sTrack, D.gtrack, GATE_TRACK_FLOATS * 4, bar);
        bulk_g2s(sC1, D.cand1, cb, bar);
        bulk_g2s(sC2, D.cand2, cb, bar);
    }
    copyGateP(sG, D.gate);
    __syncthreads();
    if (!__syncthreads_and(mbar_wait(bar, 0)))
    {
        if (threadIdx.x == 0)
            atomicAdd(&D.stats[1], 1);
        return;
    }
    const GateParams& G = *sG;
    const uint32_t k0 = D.cfg.k0, k1 = D.cfg.k1, step = I.step;
    for (int task = threadIdx.x; task < 4 * P; task += blockDim.x)
    {
        const int kind = task / (2 * P);
        const int tid = task % (2 * P);
        const int second = tid >= P;
        const int p = second ? tid - P : tid;
        const float* nominal = second ? sC2 : sC1;
        const int theta = D.thetas[p];
        GState st;
        loadGState(st, I.gstate);
        BState<NTH> bs{};
        EnvNoise rng(k0, k1, (uint32_t)p, (uint32_t)second << 16, step, kind ? S_PR_SAFE_ENV : S_PR_CAND_ENV);
        float cost = 0.0f, safeCost = -INFINITY, decay = 1.0f;
        bool stop = false;
        for (int t = 0; t < T && !stop; ++t)
        {
            rng.begin_step((uint32_t)t);
            bool branched = false;
            StepOut o = gateStep<NTH, false, false, true, true, ME, true>(t, theta, sTrack, G, nominal[t * 2], nominal[t * 2 + 1], st, bs, branched, 0.0f,
                                                                          rng, D.cfg.gateMargin);
            stop = (o.term != TERM_NONE);
            cost += decay * gatePrStateCost(o, G, D.cfg);
            decay *= DECAY;
            safeCost = fmaxf(safeCost, gatePrSafetyCost(o, G, D.cfg.collDistFactor));
        }
        cost += gateFinalCost<ME>(st, G, D.cfg.finalAdvWeight, D.cfg.finalOppAdvWeight);
        if (safeCost > 0.0f)
            cost += D.cfg.safetyWeight;
        if (kind == 0)
            D.candFull[tid] = cost;
        else
            D.candSafe[tid] = safeCost;
    }
    __syncthreads();
    gatePrChoose(D, sC1, sC2, T, P, &sChosen);
}

// ---------------------------------------------------------------------------------------
// one ego per sample (egos that draw no noise), as in prmppi_kernels.cu
// ---------------------------------------------------------------------------------------
// One step of a shared ego: what the opponents' steps read of it ([field][ego]).
enum GateEgoField
{
    GEF_BX,   // position before
    GEF_BY,
    GEF_PX,   // position after
    GEF_PY,
    GEF_BOUND, // its own boundary distance after (arena, obstacles)
    GEF_LAPS, // laps and last gate after (integers' bits)
    GEF_GATES,
    GATE_EGO_FIELDS
};

template <int ME>
__device__ __forceinline__ void gateEgoStepShared(const float* __restrict__ track, const GateParams& G, float ego0, float ego1, GLane& s, float* row, int n,
                                                  float gateMargin)
{
    const float pp0 = s.pos[0], pp1 = s.pos[1];
    row[GEF_BX * n] = pp0;
    row[GEF_BY * n] = pp1;
    laneMove(G, ME, s, ego0, ego1, 0, [](int) { return 0.0f; });
    if (s.S[0] >= 0.0f)
#pragma unroll
        for (int r = 0; r < G_NR; r++)
            s.S[r] = projectRaceline(track, r, s.pos[0], s.pos[1], s.S[r]);
    laneGates<true>(G, s, pp0, pp1, gateMargin);
    row[GEF_PX * n] = s.pos[0];
    row[GEF_PY * n] = s.pos[1];
    row[GEF_BOUND * n] = laneBoundary(G, s.pos[0], s.pos[1]);
    row[GEF_LAPS * n] = __int_as_float(s.laps);
    row[GEF_GATES * n] = __int_as_float(s.gates);
}

// The opponent's part of gateStep<NTH, false, false, true, true, ME, true> under hypothesis th.
template <int ME>
__device__ __forceinline__ StepOut gateOppStepShared(int th, const float* __restrict__ track, const GateParams& G, GLane& s, const float* row, int n, float n0,
                                                     float n1, float gateMargin)
{
    constexpr int opp = 1 - ME;
    const float pp0 = s.pos[0], pp1 = s.pos[1];
    GState q; // what pidAction reads
    q.pos[2 * ME] = row[GEF_BX * n];
    q.pos[2 * ME + 1] = row[GEF_BY * n];
    q.pos[2 * opp] = pp0;
    q.pos[2 * opp + 1] = pp1;
    q.vel[2 * opp] = s.vel[0];
    q.vel[2 * opp + 1] = s.vel[1];
#pragma unroll
    for (int r = 0; r < G_NR; r++)
        q.S[opp * G_NR + r] = s.S[r];
    float u0, u1;
    pidAction<opp, true>(q, G, track, th, u0, u1);
    const float an = G.pidNoise[th];
    if (an != 0.0f)
    {
        u0 += an * n0;
        u1 += an * n1;
    }
    laneMove(G, opp, s, u0, u1, 0, [](int) { return 0.0f; });
    if (s.S[0] >= 0.0f)
#pragma unroll
        for (int r = 0; r < G_NR; r++)
            s.S[r] = projectRaceline(track, r, s.pos[0], s.pos[1], s.S[r]);
    laneGates<true>(G, s, pp0, pp1, gateMargin);
    StepOut r;
    r.oppWon = s.laps >= G.nWinLaps;
    const float e0 = row[GEF_PX * n], e1 = row[GEF_PY * n];
    float sqDist = 0.0f;
    float dx = ME == 0 ? e0 - s.pos[0] : s.pos[0] - e0;
    sqDist += dx * dx;
    dx = ME == 0 ? e1 - s.pos[1] : s.pos[1] - e1;
    sqDist += dx * dx;
    r.bdRaw = fminf(row[GEF_BOUND * n], sqrtf(sqDist) - G.droneRadius);
    r.winner = __float_as_int(row[GEF_LAPS * n]) >= G.nWinLaps || laneOut(G, s.pos[0], s.pos[1]);
    const float bdTerm = r.oppWon ? -1.0f : r.bdRaw;
    r.term = bdTerm < G.droneRadius ? TERM_LOSE : r.winner ? TERM_WIN : TERM_NONE;
    return r;
}

// The ego after its step `row`, as the final cost reads it.
__device__ __forceinline__ void gateEgoAfter(GLane& ego, const float* row, int n)
{
    ego.pos[0] = row[GEF_PX * n];
    ego.pos[1] = row[GEF_PY * n];
    ego.laps = __float_as_int(row[GEF_LAPS * n]);
    ego.gates = __float_as_int(row[GEF_GATES * n]);
}

__device__ __forceinline__ float gatePrFinalCost(const GLane& ego, const GLane& opp, const GateParams& G, const PrCfgDev& c)
{
    float cost = -c.finalAdvWeight * laneAdvance(ego, G);
    if (c.finalOppAdvWeight != 0.0f)
        cost += c.finalOppAdvWeight * laneAdvance(opp, G);
    return cost;
}

__host__ __device__ inline PrSplit gatePrSplit(int P, int threads)
{
    return prSplit(P, threads, GPR_TILE / P);
}

struct GatePrsSmem
{
    size_t gp, track, nom, rows, red, total;
};

__host__ __device__ inline GatePrsSmem gatePrsLayout(int T, int P, int n)
{
    GatePrsSmem L;
    size_t off = 16; // mbarrier
    L.gp = off;
    off = gp16(off + sizeof(GateParams));
    L.track = off;
    off = gp16(off + GATE_TRACK_FLOATS * 4);
    L.nom = off;
    off = gp16(off + (size_t)T * 2 * 4);
    L.rows = off;
    off = gp16(off + (size_t)2 * GATE_EGO_FIELDS * n * 4);
    L.red = off;
    off = gp16(off + (size_t)n * P * 2 * 4);
    L.total = off;
    return L;
}

// gate_pr_rollout with one ego per sample, stepped beside its opponents by warps of its own, a
// step ahead (pr_rollout_shared says why and how): one agent of 2 plans x 8 hypotheses x K 2048 x
// T 64 0.250 -> 0.171 ms, with CTAs of 256 threads 0.154 (B200, 1965 MHz). It is bound by the
// chain of its steps, whose barrier hands the egos' moves over.
template <int ME>
__global__ void __launch_bounds__(PRS_TILE, 2) gate_pr_rollout_shared(const PrDev* __restrict__ insts, const PrIn* __restrict__ in,
                                                                      const Tile* __restrict__ tiles)
{
    extern __shared__ __align__(128) unsigned char smraw[];
    const Tile tile = tiles[blockIdx.x];
    const PrDev& D = insts[tile.inst];
    const PrIn& I = in[tile.inst];
    const int K = D.cfg.K, T = D.cfg.T, P = D.cfg.P;
    const int robust = tile.aux;
    const PrSplit split = gatePrSplit(P, blockDim.x);
    const GatePrsSmem L = gatePrsLayout(T, P, split.samples);
    uint64_t* bar = (uint64_t*)smraw;
    GateParams* sG = (GateParams*)(smraw + L.gp);
    float* sTrack = (float*)(smraw + L.track);
    float* sNom = (float*)(smraw + L.nom);
    float* rows = (float*)(smraw + L.rows);
    float* red = (float*)(smraw + L.red);
    const uint32_t nomBytes = (uint32_t)gp16((size_t)T * 2 * 4);
    if (threadIdx.x == 0)
    {
        mbar_init(bar, 1);
        mbar_expect_tx(bar, GATE_TRACK_FLOATS * 4 + nomBytes);
        bulk_g2s(sTrack, D.gtrack, GATE_TRACK_FLOATS * 4, bar);
        bulk_g2s(sNom, robust ? D.rob : D.nom, nomBytes, bar);
    }
    copyGateP(sG, D.gate);
    __syncthreads();
    if (!__syncthreads_and(mbar_wait(bar, 0)))
    {
        if (threadIdx.x == 0)
            atomicAdd(&D.stats[1], 1);
        return;
    }
    const GateParams& G = *sG;
    const int n = split.samples, rowWords = GATE_EGO_FIELDS * n;
    const uint32_t k0 = D.cfg.k0, k1 = D.cfg.k1, step = I.step;
    const float gateMargin = D.cfg.gateMargin;
    const bool ego = (int)threadIdx.x >= split.opp; // whole warps
    GLane st;
    loadGLane(st, I.gstate, ego ? ME : 1 - ME);
    if (ego)
    {
        const int sl = threadIdx.x - split.opp;
        const bool valid = sl < n && sl < tile.count;
        const uint32_t s = (uint32_t)(tile.s0 + sl);
        // row t of the two is written while the opponents read row t - 1
        for (int t = 0;; t++)
        {
            if (valid && t < T)
            {
                const U4 r = draw(k0, k1, s, (uint32_t)t, step, S_PR_EPS, 0);
                const float ego0 = sNom[t * 2] + scaled_normal(D.cfg.sigma0, r.x);
                const float ego1 = sNom[t * 2 + 1] + scaled_normal(D.cfg.sigma1, r.y);
                gateEgoStepShared<ME>(sTrack, G, ego0, ego1, st, rows + (t & 1) * rowWords + sl, n, gateMargin);
            }
            // one barrier a step: T of them, or fewer once the opponents are all done
            if (t == T || !__syncthreads_or(0))
                break;
        }
    }
    else
    {
        const int sl = threadIdx.x / P, p = threadIdx.x % P;
        const int s = tile.s0 + sl;
        const bool valid = sl < n && sl < tile.count;
        const int theta = D.thetas[p];
        const uint32_t c1 = (((uint32_t)robust << 8) | (uint32_t)p) << 16;
        float running = 0.0f, safe = -INFINITY, decay = 1.0f;
        GLane last; // the ego, as the final cost reads it
        loadGLane(last, I.gstate, ME);
        bool active = valid;
        for (int t = 0; t < T; t++)
        {
            if (!__syncthreads_or(active))
                break;
            if (!active)
                continue;
            const float* row = rows + (t & 1) * rowWords + sl;
            float n0 = 0.0f, n1 = 0.0f;
            if (G.pidNoise[theta] != 0.0f)
            {
                const U4 r = draw(k0, k1, (uint32_t)s, c1 | (uint32_t)t, step, S_PR_ROLL_ENV, 0);
                const float2 nn = normal_pair_ool(r.x, r.y);
                n0 = nn.x;
                n1 = nn.y;
            }
            const StepOut o = gateOppStepShared<ME>(theta, sTrack, G, st, row, n, n0, n1, gateMargin);
            gateEgoAfter(last, row, n);
            if (o.term != TERM_NONE)
                active = false;
            running += decay * gatePrStateCost(o, G, D.cfg);
            safe = fmaxf(safe, gatePrSafetyCost(o, G, D.cfg.collDistFactor));
            decay *= DECAY;
        }
        if (valid)
        {
            running += gatePrFinalCost(last, st, G, D.cfg);
            float* out = robust ? D.costRob : D.costNom;
            out[((size_t)p * K + s) * 2 + 0] = running;
            out[((size_t)p * K + s) * 2 + 1] = safe;
            red[(sl * P + p) * 2] = running;
            red[(sl * P + p) * 2 + 1] = safe;
        }
    }
    __syncthreads();
    // PRMPPIcostAvgKernel (prmppi_kernels.cu:134-166)
    for (int sl = threadIdx.x; sl < n && sl < tile.count; sl += blockDim.x)
    {
        const int s = tile.s0 + sl;
        float avg = 0.0f, maxSafe = -INFINITY;
        for (int q = 0; q < P; q++)
        {
            avg += red[(sl * P + q) * 2];
            maxSafe = fmaxf(maxSafe, red[(sl * P + q) * 2 + 1]);
        }
        avg /= (float)P;
        float full = avg + ((maxSafe > 0.0f) ? D.cfg.safetyWeight : 0.0f);
        D.avg[((size_t)robust * K + s) * 2 + 0] = full;
        D.avg[((size_t)robust * K + s) * 2 + 1] = maxSafe;
        if (!isfinite(full))
            atomicAdd(&D.stats[0], 1);
    }
}

// gate_pr_candidates with the two candidates' egos shared by their opponents, as
// pr_candidates_shared: warps for the opponents, as many that draw their normals and one whose
// first two lanes move the egos, both a step ahead: 0.150 -> 0.100 ms at T 64 (B200, 1965 MHz).
template <int ME>
__global__ void __launch_bounds__(9 * 32) gate_pr_candidates_shared(const PrDev* __restrict__ insts, const PrIn* __restrict__ in, int nInst)
{
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ int sChosen;
    __shared__ float rows[2][GATE_EGO_FIELDS * 2];
    __shared__ float2 normals[2][4 * 32];
    const int inst = blockIdx.x;
    if (inst >= nInst)
        return;
    const PrDev& D = insts[inst];
    const PrIn& I = in[inst];
    const int T = D.cfg.T, P = D.cfg.P;
    uint64_t* bar = (uint64_t*)smraw;
    GateParams* sG = (GateParams*)(smraw + 16);
    const size_t offT = gp16(16 + sizeof(GateParams));
    float* sTrack = (float*)(smraw + offT);
    float* sC1 = (float*)(smraw + offT + GATE_TRACK_FLOATS * 4);
    const uint32_t cb = (uint32_t)gp16((size_t)T * 2 * 4);
    float* sC2 = (float*)((unsigned char*)sC1 + cb);
    if (threadIdx.x == 0)
    {
        mbar_init(bar, 1);
        mbar_expect_tx(bar, GATE_TRACK_FLOATS * 4 + 2 * cb);
        bulk_g2s(sTrack, D.gtrack, GATE_TRACK_FLOATS * 4, bar);
        bulk_g2s(sC1, D.cand1, cb, bar);
        bulk_g2s(sC2, D.cand2, cb, bar);
    }
    copyGateP(sG, D.gate);
    __syncthreads();
    if (!__syncthreads_and(mbar_wait(bar, 0)))
    {
        if (threadIdx.x == 0)
            atomicAdd(&D.stats[1], 1);
        return;
    }
    const GateParams& G = *sG;
    const uint32_t k0 = D.cfg.k0, k1 = D.cfg.k1, step = I.step;
    const float gateMargin = D.cfg.gateMargin;
    // the batch's widest controller sizes the block
    const int group = ((int)blockDim.x / 32 - 1) / 2 * 32, role = threadIdx.x / group; // 0 opponents, 1 draws, 2 egos
    const int task = threadIdx.x - role * group;
    const int kind = task / (2 * P), tid = task % (2 * P);
    const int second = role == 2 ? task : tid >= P;
    const int p = tid >= P ? tid - P : tid;
    const bool valid = role == 2 ? task < 2 : task < 4 * P;
    GLane st;
    loadGLane(st, I.gstate, role == 2 ? ME : 1 - ME);
    if (role != 0)
    {
        const float* nominal = second ? sC2 : sC1;
        const bool noisy = role == 1 && valid && G.pidNoise[D.thetas[valid ? p : 0]] != 0.0f;
        for (int t = 0;; t++)
        {
            if (t < T)
            {
                if (role == 2 && valid)
                    gateEgoStepShared<ME>(sTrack, G, nominal[t * 2], nominal[t * 2 + 1], st, rows[t & 1] + second, 2, gateMargin);
                else if (noisy)
                {
                    const U4 r = draw(k0, k1, (uint32_t)p, ((uint32_t)second << 16) | (uint32_t)t, step, kind ? S_PR_SAFE_ENV : S_PR_CAND_ENV, 0);
                    normals[t & 1][task] = make_float2(normal_from_word(r.x), normal_from_word(r.y));
                }
            }
            if (t == T || !__syncthreads_or(0))
                break;
        }
    }
    else
    {
        const int theta = D.thetas[valid ? p : 0];
        float cost = 0.0f, safeCost = -INFINITY, decay = 1.0f;
        GLane last; // the ego, as the final cost reads it
        loadGLane(last, I.gstate, ME);
        bool active = valid;
        for (int t = 0; t < T; ++t)
        {
            if (!__syncthreads_or(active))
                break;
            if (!active)
                continue;
            const float* row = rows[t & 1] + second;
            const float2 nn = normals[t & 1][task];
            const StepOut o = gateOppStepShared<ME>(theta, sTrack, G, st, row, 2, nn.x, nn.y, gateMargin);
            gateEgoAfter(last, row, 2);
            active = o.term == TERM_NONE;
            cost += decay * gatePrStateCost(o, G, D.cfg);
            decay *= DECAY;
            safeCost = fmaxf(safeCost, gatePrSafetyCost(o, G, D.cfg.collDistFactor));
        }
        if (valid)
        {
            cost += gatePrFinalCost(last, st, G, D.cfg);
            if (safeCost > 0.0f)
                cost += D.cfg.safetyWeight;
            if (kind == 0)
                D.candFull[tid] = cost;
            else
                D.candSafe[tid] = safeCost;
        }
    }
    __syncthreads();
    gatePrChoose(D, sC1, sC2, T, P, &sChosen);
}

size_t gatePrRolloutSmem(int T, int P)
{
    const size_t a = gatePrLayout(T).total, b = gatePrsLayout(T, P, gatePrSplit(P, PRS_TILE).samples).total;
    return a > b ? a : b;
}

int gatePrRolloutSamplesPerTile(bool shared, int P, int threads)
{
    return prTileSamples(shared, P, threads, GPR_TILE);
}

template <int NTH, int ME> static cudaError_t gatePrRollT(const LaunchArgs& a, size_t smem)
{
    if (a.prShared)
    {
        auto k = gate_pr_rollout_shared<ME>;
        ensureSmem(k, smem);
        k<<<a.nTiles, a.prThreads, smem, a.stream>>>(a.pr, a.prIn, a.tiles);
        return cudaGetLastError();
    }
    auto k = gate_pr_rollout<NTH, ME>;
    ensureSmem(k, smem);
    k<<<a.nTiles, GPR_TILE, smem, a.stream>>>(a.pr, a.prIn, a.tiles);
    return cudaGetLastError();
}

template <int NTH, int ME> static cudaError_t gatePrCandT(const LaunchArgs& a, int nInst, int maxT, int maxP)
{
    const size_t smem = gp16(16 + sizeof(GateParams)) + GATE_TRACK_FLOATS * 4 + 2 * gp16((size_t)maxT * 2 * 4);
    if (a.prShared)
    {
        auto k = gate_pr_candidates_shared<ME>;
        ensureSmem(k, smem);
        k<<<nInst, (2 * ((4 * maxP + 31) / 32) + 1) * 32, smem, a.stream>>>(a.pr, a.prIn, nInst);
        return cudaGetLastError();
    }
    auto k = gate_pr_candidates<NTH, ME>;
    ensureSmem(k, smem);
    k<<<nInst, GPR_CAND, smem, a.stream>>>(a.pr, a.prIn, nInst);
    return cudaGetLastError();
}

#define GPR_DISPATCH(NTH_, ME_, CALL)                                                                                                                 \
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

cudaError_t launchGatePrRollout(const LaunchArgs& a, int nth, int me, size_t smem)
{
#define CALL(P_, Q_) gatePrRollT<P_, Q_>(a, smem)
    GPR_DISPATCH(nth, me, CALL)
#undef CALL
}

cudaError_t launchGatePrCandidates(const LaunchArgs& a, int nth, int me, int nInst, int maxT, int maxP)
{
#define CALL(P_, Q_) gatePrCandT<P_, Q_>(a, nInst, maxT, maxP)
    GPR_DISPATCH(nth, me, CALL)
#undef CALL
}

} // namespace dr
