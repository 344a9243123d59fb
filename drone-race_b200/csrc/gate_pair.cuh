// The gate race's environment step taken by a pair of neighbouring lanes: lane 0 (role 0) moves
// the ego, lane 1 (role 1) the opponent, as pair_model.cuh does for the strategic race and for
// the same reason (a rollout is a chain of dependent steps). What both agents do (clamp,
// integration, speed cap, gate crossing) is one instruction stream over both lanes; the PID
// action is evaluated under two hypotheses at a time, and the opponent's two raceline
// projections side by side while the ego is untracked. The expressions are gateStep's, so the
// results agree with it bit for bit.
#pragma once

#include "gate_model.cuh"
#include "pair_model.cuh"

namespace dr
{

struct GLane // one agent
{
    float pos[2], vel[2], S[G_NR];
    int laps, gates;
};

__device__ __forceinline__ void loadGLane(GLane& l, const dr_gate_state& s, int a)
{
#pragma unroll
    for (int d = 0; d < 2; d++)
    {
        l.pos[d] = s.pos[2 * a + d];
        l.vel[d] = s.vel[2 * a + d];
    }
#pragma unroll
    for (int r = 0; r < G_NR; r++)
        l.S[r] = s.S[a * G_NR + r];
    l.laps = s.laps[a];
    l.gates = s.gates[a];
}

// updateGates' crossing test of one agent (env_dronerace.h:437-470), from its position before
// the step
template <bool ADDMARGIN>
__device__ __forceinline__ void laneGates(const GateParams& G, GLane& s, float pp0, float pp1, float margin)
{
    const float px = s.pos[0], py = s.pos[1];
    const int next = nextGateIndex(s.gates, G.nGates);
    const float gc0 = G.gateCenters[next * 2], gc1 = G.gateCenters[next * 2 + 1];
    const float gv0 = G.gateVectors[next * 2], gv1 = G.gateVectors[next * 2 + 1];
    float num = 0.f, denom = 0.f;
    num += gv0 * (gc0 - pp0);
    denom += gv0 * (px - pp0);
    num += gv1 * (gc1 - pp1);
    denom += gv1 * (py - pp1);
    if (fabsf(denom) < 1e-10f)
        return;
    float lambda = num / denom;
    if (lambda < 0.f || lambda > 1.f)
        return;
    float sqDist = 0.f;
    float dx = (1.f - lambda) * pp0 + lambda * px - gc0;
    sqDist += dx * dx;
    dx = (1.f - lambda) * pp1 + lambda * py - gc1;
    sqDist += dx * dx;
    float rad = G.gateRadius[next] * G.gateRadius[next];
    if constexpr (ADDMARGIN)
        rad *= margin * margin;
    if (sqDist <= rad)
    {
        s.gates++;
        if (s.gates == G.nGates)
        {
            s.gates = 0;
            s.laps++;
        }
    }
}

// Steps 3 to 6 of gateStep for one agent (index a) under the action (act0, act1); `normal`
// gives the j-th normal of the step's noise from its next unused one on.
template <class N>
__device__ __forceinline__ void laneMove(const GateParams& G, int a, GLane& s, float& act0, float& act1, int jn, N normal)
{
    float sqNorm = 0.0f;
    sqNorm += act0 * act0;
    sqNorm += act1 * act1;
    float factor = 1.0f;
    float maxSq = G.maxAccel[a] * G.maxAccel[a];
    if (sqNorm > maxSq)
        factor = mdivsqrt<false>(G.maxAccel[a], sqNorm);
    act0 *= factor;
    if (G.actionNoiseLevel != 0.0f)
        act0 += normal(jn + 2 * a) * G.actionNoiseLevel;
    act1 *= factor;
    if (G.actionNoiseLevel != 0.0f)
    {
        act1 += normal(jn + 2 * a + 1) * G.actionNoiseLevel;
        jn += 2 * G_NA;
    }
    s.pos[0] += G.dt * s.vel[0];
    s.pos[1] += G.dt * s.vel[1];
    s.vel[0] += G.dt * act0;
    s.vel[1] += G.dt * act1;
    float sq = 0.0f;
    sq += s.vel[0] * s.vel[0];
    sq += s.vel[1] * s.vel[1];
    float spd = sqrtf(sq);
    if (spd > G.maxSpeed[a])
    {
        float sc = G.maxSpeed[a] / spd;
        s.vel[0] *= sc;
        s.vel[1] *= sc;
    }
    if (G.posNoise != 0.0f || G.speedNoise != 0.0f)
    {
        const int per = (G.posNoise != 0.0f ? 1 : 0) + (G.speedNoise != 0.0f ? 1 : 0);
        int j = jn + a * 2 * per;
#pragma unroll
        for (int d = 0; d < 2; d++)
        {
            if (G.posNoise != 0.0f)
                s.pos[d] += normal(j++) * G.posNoise;
            if (G.speedNoise != 0.0f)
                s.vel[d] += normal(j++) * G.speedNoise;
        }
    }
}

// The ego's own part of gateBoundaryDist (arena and obstacles) and the opponent's of
// gateIsWinner (arena and obstacles), each from that agent's position.
__device__ __forceinline__ float laneBoundary(const GateParams& G, float c0, float c1)
{
    float minDist = INFINITY;
    minDist = fminf(minDist, fminf(c0 - G.arenaMin[0], G.arenaMax[0] - c0));
    minDist = fminf(minDist, fminf(c1 - G.arenaMin[1], G.arenaMax[1] - c1));
    for (int i = 0; i < G.nObs; i++)
    {
        float sqDist = 0.0f;
        float dist = fmaxf(0.0f, fmaxf(G.obstacles[i * 4 + 0] - c0, c0 - G.obstacles[(i * 2 + 1) * 2 + 0]));
        sqDist += dist * dist;
        dist = fmaxf(0.0f, fmaxf(G.obstacles[i * 4 + 1] - c1, c1 - G.obstacles[(i * 2 + 1) * 2 + 1]));
        sqDist += dist * dist;
        minDist = fminf(minDist, sqrtf(sqDist));
    }
    for (int i = 0; i < G.nRound; i++)
    {
        float sqDist = 0.0f;
        float dx = c0 - G.roundCenters[i * 2];
        sqDist += dx * dx;
        dx = c1 - G.roundCenters[i * 2 + 1];
        sqDist += dx * dx;
        minDist = fminf(minDist, sqrtf(sqDist) - G.roundRadius[i]);
    }
    return minDist;
}

__device__ __forceinline__ bool laneOut(const GateParams& G, float c0, float c1)
{
    const float radius = G.droneRadius;
    if (c0 < G.arenaMin[0] + radius || c0 > G.arenaMax[0] + radius)
        return true;
    if (c1 < G.arenaMin[1] + radius || c1 > G.arenaMax[1] + radius)
        return true;
    for (int i = 0; i < G.nObs; i++)
    {
        float sqDist = 0.0f;
        float dist = fmaxf(0.0f, fmaxf(G.obstacles[i * 4 + 0] - c0, c0 - G.obstacles[(i * 2 + 1) * 2 + 0]));
        sqDist += dist * dist;
        dist = fmaxf(0.0f, fmaxf(G.obstacles[i * 4 + 1] - c1, c1 - G.obstacles[(i * 2 + 1) * 2 + 1]));
        sqDist += dist * dist;
        if (sqDist < radius * radius)
            return true;
    }
    for (int i = 0; i < G.nRound; i++)
    {
        float sqDist = 0.0f;
        float dx = c0 - G.roundCenters[i * 2];
        sqDist += dx * dx;
        dx = c1 - G.roundCenters[i * 2 + 1];
        sqDist += dx * dx;
        if (sqDist < (radius + G.roundRadius[i]) * (radius + G.roundRadius[i]))
            return true;
    }
    return false;
}

__device__ __forceinline__ float projectRaceline(const float* __restrict__ track, int r, float px, float py, float prevS)
{
    return projectGreedy(track + r * NTS * 2, gateRowX(track, r), gateCert(track, r), px, py, prevS);
}

// One environment step (gateStep<NTH, true, true, false, true, ME>). `mask`: the lanes that
// take part, whole pairs. ctl0, ctl1: the ego's control (read on its lane), opp0, opp1: the
// normals of the opponent's action noise (read on its lane). Everything the two lanes return is
// the same on both, except `s`.
template <int NTH, int ME>
__device__ __forceinline__ StepOut gatePairStep(unsigned mask, int role, int t, int trueTheta, const float* __restrict__ track, const GateParams& G, float ctl0,
                                                float ctl1, float opp0, float opp1, GLane& s, BState<NTH>& bs, bool& branched, float minConf,
                                                const PairNoise& noise)
{
    static_assert(G_NR == 2, "two racelines");
    constexpr int opp = 1 - ME;
    const bool live = bs.predTheta == 0; // the belief is still read after this step
    const float pp0 = s.pos[0], pp1 = s.pos[1];
    // the agents as pidAction reads them: the opponent's state, the ego's position
    GState q;
    pairBoth(mask, role, s.pos[0], q.pos[2 * ME], q.pos[2 * opp]);
    pairBoth(mask, role, s.pos[1], q.pos[2 * ME + 1], q.pos[2 * opp + 1]);
    pairBoth(mask, role, s.vel[0], q.vel[2 * ME], q.vel[2 * opp]);
    pairBoth(mask, role, s.vel[1], q.vel[2 * ME + 1], q.vel[2 * opp + 1]);
#pragma unroll
    for (int r = 0; r < G_NR; r++)
        pairBoth(mask, role, s.S[r], q.S[ME * G_NR + r], q.S[opp * G_NR + r]);
    float nom0[NTH], nom1[NTH];
    float u0 = 0.f, u1 = 0.f;
#pragma unroll
    for (int r = 0; r < NTH; r += 2)
    {
        // the round's hypotheses, or in its first round a committed sample's own
        const int th = live ? (r + role < NTH ? r + role : r) : trueTheta;
        float a0 = 0.f, a1 = 0.f;
        if (live || r == 0)
            pidAction<opp>(q, G, track, th, a0, a1);
        pairBoth(mask, role, a0, nom0[r], nom0[r + 1 < NTH ? r + 1 : r]);
        pairBoth(mask, role, a1, nom1[r], nom1[r + 1 < NTH ? r + 1 : r]);
        if (!live && r == 0)
        {
            u0 = a0;
            u1 = a1;
        }
    }
    if (live)
    {
#pragma unroll
        for (int th = 0; th < NTH; th++)
            if (th == trueTheta)
            {
                u0 = nom0[th];
                u1 = nom1[th];
            }
    }
    int jn = 0; // normals of the step's stream taken before the next use
    {
        float an = G.pidNoise[trueTheta];
        if (an != 0.0f)
        {
            u0 += an * opp0;
            u1 += an * opp1;
            jn = 2;
        }
    }
    float act0 = role ? u0 : ctl0, act1 = role ? u1 : ctl1;
    laneMove(G, role ? opp : ME, s, act0, act1, jn, [&](int j) { return noise.at(j); });
    float pe0, pe1, po0, po1;
    pairBoth(mask, role, s.pos[0], pe0, po0);
    pairBoth(mask, role, s.pos[1], pe1, po1);
    // 8. projections of the tracked agents, then the gates
    if (q.S[ME * G_NR] >= 0.0f)
    {
        // both agents may be tracked: each lane its own
        if (s.S[0] >= 0.0f)
#pragma unroll
            for (int r = 0; r < G_NR; r++)
                s.S[r] = projectRaceline(track, r, s.pos[0], s.pos[1], s.S[r]);
    }
    else if (q.S[opp * G_NR] >= 0.0f)
    {
        // the opponent alone: a raceline a lane
        const float x = projectRaceline(track, role, po0, po1, role ? q.S[opp * G_NR + 1] : q.S[opp * G_NR]);
        float x0, x1;
        pairBoth(mask, role, x, x0, x1);
        if (role)
        {
            s.S[0] = x0;
            s.S[1] = x1;
        }
    }
    laneGates<false>(G, s, pp0, pp1, 0.0f);
    // 9. belief (updateBelief, :212-258): a hypothesis' likelihood on the lane that evaluated it
    {
        const float maxPIDaccel = G.maxAccel[opp];
        float unused, oa0, oa1;
        pairBoth(mask, role, act0, unused, oa0);
        pairBoth(mask, role, act1, unused, oa1);
        float w[NTH];
#pragma unroll
        for (int r = 0; r < NTH; r += 2)
        {
            constexpr int last = NTH - 1;
            const int th = r + role < NTH ? r + role : r;
            const int r1 = r + 1 < NTH ? r + 1 : last;
            const float n0 = role ? nom0[r1] : nom0[r], n1 = role ? nom1[r1] : nom1[r];
            float wr = role ? bs.belief[r1] : bs.belief[r];
            if (live)
            {
                float sqAccel = 0.f;
                sqAccel += n0 * n0;
                sqAccel += n1 * n1;
                float scale = 1.0f;
                if (sqAccel > maxPIDaccel * maxPIDaccel)
                    scale = mdivsqrt<false>(maxPIDaccel, sqAccel);
                float sqDist = 0.f;
                float dx = oa0 - n0 * scale;
                sqDist += dx * dx;
                dx = oa1 - n1 * scale;
                sqDist += dx * dx;
                wr *= expf((-0.5f * sqDist) / G.beliefSig2[th]) / G.beliefNorm[th];
            }
            pairBoth(mask, role, wr, w[r], w[r1]);
        }
        if (live)
        {
            float sum = 0.0f;
#pragma unroll
            for (int th = 0; th < NTH; th++)
                sum += w[th];
            if (sum < 1e-20f)
            {
                float uniform = 1.0f / NTH;
#pragma unroll
                for (int th = 0; th < NTH; ++th)
                    bs.belief[th] = uniform;
            }
            else
            {
#pragma unroll
                for (int th = 0; th < NTH; th++)
                    bs.belief[th] = w[th] / sum;
            }
        }
    }
    int np = findConfident<NTH>(bs.belief, minConf);
    if (bs.predTheta == 0 && np != 0)
    {
        bs.predTheta = np;
        bs.branchingTime = t + 1;
        branched = true;
    }
    // terminal checks (:672-679)
    int le, lo;
    pairBoth(mask, role, s.laps, le, lo);
    StepOut r;
    r.oppWon = lo >= G.nWinLaps;
    float sqDist = 0.0f;
    float dx = ME == 0 ? pe0 - po0 : po0 - pe0;
    sqDist += dx * dx;
    dx = ME == 0 ? pe1 - po1 : po1 - pe1;
    sqDist += dx * dx;
    r.bdRaw = fminf(laneBoundary(G, pe0, pe1), sqrtf(sqDist) - G.droneRadius);
    r.winner = le >= G.nWinLaps || laneOut(G, po0, po1);
    const float bdTerm = r.oppWon ? -1.0f : r.bdRaw;
    r.term = bdTerm < G.droneRadius ? TERM_LOSE : r.winner ? TERM_WIN : TERM_NONE;
    return r;
}

// gateAdvance of one agent (getAnyAdvance, env_dronerace.h:374-394)
__device__ __forceinline__ float laneAdvance(const GLane& s, const GateParams& G)
{
    float sqGateDist = 0.0f, sqConsGateDist = 0.0f;
    int nextGate = nextGateIndex(s.gates, G.nGates);
    float scale = 0.8f;
    const float* prevC = G.gateCenters + s.gates * 2;
    const float* nextC = G.gateCenters + nextGate * 2;
    const float p0 = s.pos[0], p1 = s.pos[1];
    sqGateDist += (nextC[0] - p0) * (nextC[0] - p0);
    sqConsGateDist += (nextC[0] - prevC[0]) * (nextC[0] - prevC[0]);
    sqGateDist += (nextC[1] - p1) * (nextC[1] - p1);
    sqConsGateDist += (nextC[1] - prevC[1]) * (nextC[1] - prevC[1]);
    return s.gates + G.nGates * s.laps + scale * (1.0f - sqrtf(sqGateDist / sqConsGateDist));
}

} // namespace dr
