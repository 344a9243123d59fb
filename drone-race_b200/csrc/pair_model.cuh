// The strategic race's environment step with one opponent, taken by a pair of neighbouring
// lanes: lane 0 (role 0) moves the ego, lane 1 (role 1) the opponent. What the two agents
// both do (geometry at the arc length, clamp, integration, speed cap, projection, laps) is
// one instruction stream over both lanes, the opponent's policy under two hypotheses at a
// time likewise, and the rest (boundary distance, terminal tests, costs) both lanes evaluate
// alike from exchanged values. The expressions are those of model.cuh's exact flavour, so
// the results agree with envStep's bit for bit.
//
// Why: a rollout is a chain of T dependent steps and small batches leave the device idle
// beside it, so the step's latency is the rollout's time. Two agents a thread is twice the
// instructions in that chain; a lane for each halves them at the same issue slots for the
// pair, and the state of one agent takes half the registers, which lets large batches keep
// more warps resident (figures at mppi_rollout).
#pragma once

#include "model.cuh"

namespace dr
{

__device__ __forceinline__ float pairSwap(unsigned mask, float v)
{
    return __shfl_xor_sync(mask, v, 1);
}

__device__ __forceinline__ int pairSwap(unsigned mask, int v)
{
    return __shfl_xor_sync(mask, v, 1);
}

// v of the ego's lane / of the opponent's lane, on both
template <class V> __device__ __forceinline__ void pairBoth(unsigned mask, int role, V v, V& ego, V& opp)
{
    const V o = pairSwap(mask, v);
    ego = role ? o : v;
    opp = role ? v : o;
}

// sum_m Brow[m] v[m] in knot order, v this column's knots: four at a time, [m / 4][column][4]
// (columns of `cols`). Brow is 16-byte aligned when M is a multiple of 4. A 4-byte read a knot
// and axis took a tenth of a spline rollout's issue slots: control step of 24 uneven agents
// 1483 -> 1457 us.
__device__ __forceinline__ float splineSum(const float* Brow, const float* vbuf, int cols, int col, int M)
{
    const float4* v = reinterpret_cast<const float4*>(vbuf) + col;
    float sum = 0.0f;
    if ((M & 3) == 0)
    {
        const float4* B = reinterpret_cast<const float4*>(Brow);
        for (int q = 0; q < M / 4; q++)
        {
            const float4 b = B[q], x = v[q * cols];
            sum += b.x * x.x;
            sum += b.y * x.y;
            sum += b.z * x.z;
            sum += b.w * x.w;
        }
    }
    else
        for (int m = 0; m < M; m += 4)
        {
            const float4 x = v[m / 4 * cols];
            sum += Brow[m] * x.x;
            if (m + 1 < M)
                sum += Brow[m + 1] * x.y;
            if (m + 2 < M)
                sum += Brow[m + 2] * x.z;
            if (m + 3 < M)
                sum += Brow[m + 3] * x.w;
        }
    return sum;
}

// Normal j of the step's environment noise (EnvNoise's stream, addressed by index: the two
// lanes of a pair take different normals of one stream).
struct PairNoise
{
    uint32_t k0, k1, c0, c1, step, stream;
    __device__ __forceinline__ float at(int j) const
    {
        const U4 b = draw_ool(k0, k1, c0, c1, step, stream, (uint32_t)(j >> 2));
        const int w = j & 3;
        return normal_from_word_ool(w == 0 ? b.x : w == 1 ? b.y : w == 2 ? b.z : b.w);
    }
};

// oppCommon<1> from the two agents' quantities at the start of the step.
struct PairGeo
{
    float S[2], lat[2], sdot[2]; // both agents
    float egoLong;               // the ego's speed along its tangent
    float tn0, tn1, kap;         // the opponent's tangent and curvature
    float e_n, v_t, v_n;         // the opponent's offset and velocity in its track frame
};

__device__ __forceinline__ void pairOppCommon(const EnvParams& E, const PairGeo& q, OppCommon& c)
{
    const float L = E.trackLength;
    float deltaSAhead = q.S[0] - q.S[1];
    if (deltaSAhead < 0.0f)
        deltaSAhead += L;
    float deltaSBehind = q.S[0] - q.S[1];
    if (deltaSBehind > 0.0f)
        deltaSBehind -= L;
    c.sdot_i = q.sdot[1];
    const float sdj = q.sdot[0];
    const float blockTol = __fmul_rn(E.maxSpeed[0], 0.3f);
#pragma unroll
    for (int k = 0; k <= 1; k++)
    {
        const float deltaS = k ? deltaSAhead : deltaSBehind;
        c.j[k] = 0;
        c.deltaS[k] = deltaS;
        c.deltaE[k] = q.lat[0] - q.lat[1];
        c.latJ[k] = q.lat[0];
        c.sdotJ[k] = sdj;
        c.blockTol[k] = blockTol;
        c.shouldBlock[k] = (deltaS < 0.0f) && (deltaS > -L * 0.25f) && (sdj + blockTol > c.sdot_i);
        c.fasterThanJ[k] = c.sdot_i > sdj;
        c.oppLong[k] = q.egoLong;
    }
    c.maxLatDis = E.trackWidth - E.droneRadius * E.maxOppLatDistFact;
    c.maxAccel = E.maxAccel[1];
    c.maxAccelSq = __fmul_rn(c.maxAccel, c.maxAccel);
    c.tang0 = q.tn0;
    c.tang1 = q.tn1;
    c.kappa = q.kap;
    c.norm0 = -c.tang1;
    c.norm1 = c.tang0;
    c.e_n = q.e_n;
    c.v_t = q.v_t;
    c.v_n = q.v_n;
    c.e_n_max = E.trackWidth - E.droneRadius * 1.2f;
    float metric_actual = 1.0f - c.kappa * c.e_n;
    if (fabsf(metric_actual) < 1e-6f)
        metric_actual = copysignf(1e-6f, metric_actual);
    c.metric_actual = metric_actual;
    c.a_centripetal = (c.v_t * c.v_t * c.kappa) / metric_actual;
    c.a_lat_max = fmaxf(c.maxAccel - fabsf(c.a_centripetal), c.maxAccel * 0.2f);
    c.distPos = fmaxf(c.e_n_max - c.e_n, 0.001f);
    c.distNeg = fmaxf(c.e_n_max + c.e_n, 0.001f);
    c.brakePos = c.v_n > 0.0f && c.v_n * c.v_n > 1.8f * c.a_lat_max * c.distPos;
    c.brakeNeg = c.v_n < 0.0f && c.v_n * c.v_n > 1.8f * c.a_lat_max * c.distNeg;
}

// One environment step (envStep<1, NTH, true, true, true, true>). `mask`: the lanes that take
// part, whole pairs. `s` is this lane's agent; ctl0, ctl1 the ego's control (read on its
// lane), opp0, opp1 the standard normals of the opponent's action noise (read on its lane).
// Everything the two lanes return is the same on both, except `s`. Hypotheses are evaluated
// two at a time, an even one on the ego's lane and the next on the opponent's; a round whose
// hypotheses all repeat an earlier one's action (EnvParams::dupAll / dupNoBlock) is skipped,
// and a committed sample evaluates the true hypothesis only. LOSE: an opponent's win ends the
// rollout as a loss (loseOnOppWin); NOISE: the environment's own noise, where it is on, is drawn.
template <int NTH, bool LOSE = true, bool NOISE = true>
__device__ __forceinline__ StepOut pairStep(unsigned mask, int role, int t, int trueTheta, const Track& tr, const EnvParams& E, float ctl0, float ctl1,
                                            float opp0, float opp1, DState<1>& s, BState<NTH>& bs, bool& branched, float minConf, const PairNoise& noise)
{
    const float prevS = s.S[0];
    const bool live = bs.predTheta == 0; // the belief is still read after this step
    AgentGeo<1> g;
    agentGeometry<1>(tr, E, s, g);
    OppCommon c;
    {
        float pc0, pc1;
        sampleAt2(tr.p, s.tp[0], pc0, pc1);
        const float norm0 = -g.tn1[0], norm1 = g.tn0[0];
        const float e_n = (s.pos[0] - pc0) * norm0 + (s.pos[1] - pc1) * norm1;
        const float v_t = s.vel[0] * g.tn0[0] + s.vel[1] * g.tn1[0];
        const float v_n = s.vel[0] * norm0 + s.vel[1] * norm1;
        PairGeo q;
        pairBoth(mask, role, s.S[0], q.S[0], q.S[1]);
        pairBoth(mask, role, s.lat[0], q.lat[0], q.lat[1]);
        pairBoth(mask, role, g.sdot[0], q.sdot[0], q.sdot[1]);
        pairBoth(mask, role, v_t, q.egoLong, q.v_t);
        float unused;
        pairBoth(mask, role, v_n, unused, q.v_n);
        pairBoth(mask, role, e_n, unused, q.e_n);
        pairBoth(mask, role, g.tn0[0], unused, q.tn0);
        pairBoth(mask, role, g.tn1[0], unused, q.tn1);
        pairBoth(mask, role, g.kap[0], unused, q.kap);
        pairOppCommon(E, q, c);
    }
    float nom0[NTH], nom1[NTH];
    float u0 = 0.f, u1 = 0.f;
    {
        const bool blocks = c.shouldBlock[0] || c.shouldBlock[1];
#pragma unroll
        for (int r = 0; r < NTH; r += 2)
        {
            float a0 = 0.f, a1 = 0.f;
            // the round's hypotheses, or in its first round a committed sample's own
            const int th = live ? (r + role < NTH ? r + role : r) : trueTheta;
            const bool need = live ? (r == 0 || (blocks ? E.dupAll[r][0] : E.dupNoBlock[r][0]) < 0 ||
                                      (r + 1 < NTH && (blocks ? E.dupAll[r + 1][0] : E.dupNoBlock[r + 1][0]) < 0))
                                   : r == 0;
            if (need)
                oppAction<false>(1, th, E, c, a0, a1);
            pairBoth(mask, role, a0, nom0[r], nom0[r + 1 < NTH ? r + 1 : r]);
            pairBoth(mask, role, a1, nom1[r], nom1[r + 1 < NTH ? r + 1 : r]);
            if (r > 0 && live && !need)
            {
#pragma unroll
                for (int th2 = r; th2 < (r + 2 < NTH ? r + 2 : NTH); th2++)
                {
                    const int src = blocks ? E.dupAll[th2][0] : E.dupNoBlock[th2][0];
#pragma unroll
                    for (int j = 0; j < r; j++)
                        if (src == j)
                        {
                            nom0[th2] = nom0[j];
                            nom1[th2] = nom1[j];
                        }
                }
            }
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
    }
    const float an = E.actionNoise[trueTheta][0];
    int jn = 0; // normals of the step's stream taken before the next use
    if (an != 0.0f)
    {
        u0 += an * opp0;
        u1 += an * opp1;
        jn = 2;
    }
    // 2. clamp + action noise
    const float maxAccel = E.maxAccel[role], maxSpeed = E.maxSpeed[role];
    float act0 = role ? u0 : ctl0, act1 = role ? u1 : ctl1;
    {
        float sq = 0.0f;
        sq += act0 * act0;
        sq += act1 * act1;
        float factor = 1.0f;
        float maxSq = maxAccel * maxAccel;
        if (sq > maxSq)
            factor = mdivsqrt<false>(maxAccel, sq);
        act0 *= factor;
        act1 *= factor;
        if (NOISE && E.actionNoiseLevel != 0.0f)
        {
            act0 += noise.at(jn + 2 * role) * E.actionNoiseLevel;
            act1 += noise.at(jn + 2 * role + 1) * E.actionNoiseLevel;
            jn += 4;
        }
    }
    // 3.-6. position, arc length, velocity, speed cap
    s.pos[0] += E.dt * s.vel[0];
    s.pos[1] += E.dt * s.vel[1];
    s.S[0] += E.dt * g.sdot[0];
    s.vel[0] += E.dt * act0;
    s.vel[1] += E.dt * act1;
    {
        float sqSpd = sqNorm(s.vel[0], s.vel[1]);
        if (sqSpd > maxSpeed * maxSpeed)
        {
            float sc = mdivsqrt<false>(maxSpeed, sqSpd);
            s.vel[0] *= sc;
            s.vel[1] *= sc;
        }
    }
    // 7. state noise: per agent and axis a position normal, then a speed normal
    if (NOISE && (E.posNoise != 0.0f || E.speedNoise != 0.0f))
    {
        const int per = (E.posNoise != 0.0f ? 1 : 0) + (E.speedNoise != 0.0f ? 1 : 0);
        int j = jn + role * 2 * per;
#pragma unroll
        for (int d = 0; d < 2; d++)
        {
            if (E.posNoise != 0.0f)
                s.pos[d] += noise.at(j++) * E.posNoise;
            if (E.speedNoise != 0.0f)
                s.vel[d] += noise.at(j++) * E.speedNoise;
        }
    }
    // 8. projection, 9. laps
    s.S[0] = projectOnTrack<false>(tr, E.trackLength, E.invTrackLength, s.pos[0], s.pos[1], s.S[0], s.lat[0], s.tp[0]);
    if (s.S[0] < prevS - E.trackLength * 0.5f)
        s.laps[0]++;
    if (s.S[0] > prevS + E.trackLength * 0.5f)
        s.laps[0]--;
    // 10. belief update: a hypothesis' likelihood on the lane that evaluated it
    {
        float unused, o0, o1;
        pairBoth(mask, role, act0, unused, o0);
        pairBoth(mask, role, act1, unused, o1);
        float w[NTH];
#pragma unroll
        for (int r = 0; r < NTH; r += 2)
        {
            const int th = r + role < NTH ? r + role : r;
            float n0 = nom0[r], n1 = nom1[r], bel = bs.belief[r];
            if (r + 1 < NTH && role)
            {
                n0 = nom0[r + 1 < NTH ? r + 1 : r];
                n1 = nom1[r + 1 < NTH ? r + 1 : r];
                bel = bs.belief[r + 1 < NTH ? r + 1 : r];
            }
            float wr = bel;
            if (live)
            {
                float logLikelihood = 0.0f;
                float sqAccel = 0.0f;
                sqAccel += n0 * n0;
                sqAccel += n1 * n1;
                float scale = 1.0f;
                if (sqAccel > E.maxAccel[1] * E.maxAccel[1])
                    scale = mdivsqrt<false>(E.maxAccel[1], sqAccel);
                float sqDist = 0.0f;
                float dx0 = o0 - n0 * scale;
                sqDist += dx0 * dx0;
                float dx1 = o1 - n1 * scale;
                sqDist += dx1 * dx1;
                float sqSigma = beliefSqSigma(E.actionNoise[th][0]);
                logLikelihood += (-0.5f * sqDist) / sqSigma - (float)2 * 0.5f * logf(2.0f * M_PIf32) - (float)2 * 0.5f * E.logSqSigma[th][0];
                wr *= expf(logLikelihood);
            }
            pairBoth(mask, role, wr, w[r], w[r + 1 < NTH ? r + 1 : r]);
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
    // terminal checks (trackBoundaryDist / isOutside / isWinner, env_stratrace.h:226-274)
    float pe0, pe1, po0, po1, le, lo;
    int he, ho;
    pairBoth(mask, role, s.pos[0], pe0, po0);
    pairBoth(mask, role, s.pos[1], pe1, po1);
    pairBoth(mask, role, s.lat[0], le, lo);
    pairBoth(mask, role, s.laps[0], he, ho);
    StepOut r;
    r.oppWon = ho >= E.nWinLaps;
    const float minSq = fminf(INFINITY, sqNorm(po0 - pe0, po1 - pe1));
    r.bdRaw = fminf(sqrtf(minSq) - E.droneRadius, E.trackWidth - fabsf(le));
    r.winner = he >= E.nWinLaps || fabsf(lo) > E.trackWidth - E.droneRadius;
    const float bdTerm = (LOSE && r.oppWon) ? -1.0f : r.bdRaw;
    r.term = bdTerm < E.droneRadius ? TERM_LOSE : r.winner ? TERM_WIN : !LOSE && r.oppWon ? TERM_OPP_WIN : TERM_NONE;
    return r;
}

// ---- the opponent beside an ego that several hypotheses share -------------------------

// One step of an ego that draws no noise, for the opponents of every hypothesis that meet it
// (the ego's moves depend on its own action only): what their policies read before the step,
// and the ego after it. Written by the ego's lane, read by its opponents' (shared memory,
// [field][ego], so that the lanes of a field are neighbours).
enum EgoField
{
    EF_S,     // before: arc length
    EF_LAT,   //         lateral offset
    EF_SDOT,  //         ds/dt
    EF_ALONG, //         speed along the tangent
    EF_PX,    // after: position
    EF_PY,
    EF_LAT1,  //        lateral offset
    EF_LAPS1, //        laps (as an integer's bits)
    EF_S1,    //        arc length
    EGO_FIELDS
};

// The ego's step (egoStep, exact flavour) into its column of `row` (stride n).
__device__ __forceinline__ void egoStepShared(const Track& tr, const EnvParams& E, float ego0, float ego1, DState<1>& s, float* row, int n)
{
    row[EF_S * n] = s.S[0];
    row[EF_LAT * n] = s.lat[0];
    const float v0 = s.vel[0], v1 = s.vel[1];
    EgoRow r;
    egoStep<false>(tr, E, ego0, ego1, s, r);
    row[EF_SDOT * n] = r.sdot;
    row[EF_ALONG * n] = v0 * r.tn0 + v1 * r.tn1;
    row[EF_PX * n] = r.pos0;
    row[EF_PY * n] = r.pos1;
    row[EF_LAT1 * n] = r.lat;
    row[EF_LAPS1 * n] = __int_as_float(r.laps);
    row[EF_S1 * n] = r.S;
}

// The opponent's part of envStep<1, NTH, false, false, true, false> (no belief update, an
// opponent's win ends the rollout) under hypothesis th, beside the ego's `row`; n0, n1 the
// standard normals of its action noise.
__device__ __forceinline__ StepOut oppStepShared(int th, const Track& tr, const EnvParams& E, DState<1>& s, const float* row, int n, float n0, float n1)
{
    const float prevS = s.S[0];
    AgentGeo<1> g;
    agentGeometry<1>(tr, E, s, g);
    OppCommon c;
    {
        float pc0, pc1;
        sampleAt2(tr.p, s.tp[0], pc0, pc1);
        const float norm0 = -g.tn1[0], norm1 = g.tn0[0];
        PairGeo q;
        q.S[0] = row[EF_S * n];
        q.S[1] = s.S[0];
        q.lat[0] = row[EF_LAT * n];
        q.lat[1] = s.lat[0];
        q.sdot[0] = row[EF_SDOT * n];
        q.sdot[1] = g.sdot[0];
        q.egoLong = row[EF_ALONG * n];
        q.tn0 = g.tn0[0];
        q.tn1 = g.tn1[0];
        q.kap = g.kap[0];
        q.e_n = (s.pos[0] - pc0) * norm0 + (s.pos[1] - pc1) * norm1;
        q.v_t = s.vel[0] * g.tn0[0] + s.vel[1] * g.tn1[0];
        q.v_n = s.vel[0] * norm0 + s.vel[1] * norm1;
        pairOppCommon(E, q, c);
    }
    float u0, u1;
    oppAction<false>(1, th, E, c, u0, u1);
    const float an = E.actionNoise[th][0];
    if (an != 0.0f)
    {
        u0 += an * n0;
        u1 += an * n1;
    }
    float sq = 0.0f;
    sq += u0 * u0;
    sq += u1 * u1;
    float factor = 1.0f;
    float maxSq = E.maxAccel[1] * E.maxAccel[1];
    if (sq > maxSq)
        factor = mdivsqrt<false>(E.maxAccel[1], sq);
    u0 *= factor;
    u1 *= factor;
    s.pos[0] += E.dt * s.vel[0];
    s.pos[1] += E.dt * s.vel[1];
    s.S[0] += E.dt * g.sdot[0];
    s.vel[0] += E.dt * u0;
    s.vel[1] += E.dt * u1;
    float sqSpd = sqNorm(s.vel[0], s.vel[1]);
    if (sqSpd > E.maxSpeed[1] * E.maxSpeed[1])
    {
        float sc = mdivsqrt<false>(E.maxSpeed[1], sqSpd);
        s.vel[0] *= sc;
        s.vel[1] *= sc;
    }
    s.S[0] = projectOnTrack<false>(tr, E.trackLength, E.invTrackLength, s.pos[0], s.pos[1], s.S[0], s.lat[0], s.tp[0]);
    if (s.S[0] < prevS - E.trackLength * 0.5f)
        s.laps[0]++;
    if (s.S[0] > prevS + E.trackLength * 0.5f)
        s.laps[0]--;
    StepOut r;
    r.oppWon = s.laps[0] >= E.nWinLaps;
    const float minSq = fminf(INFINITY, sqNorm(s.pos[0] - row[EF_PX * n], s.pos[1] - row[EF_PY * n]));
    r.bdRaw = fminf(sqrtf(minSq) - E.droneRadius, E.trackWidth - fabsf(row[EF_LAT1 * n]));
    r.winner = __float_as_int(row[EF_LAPS1 * n]) >= E.nWinLaps || fabsf(s.lat[0]) > E.trackWidth - E.droneRadius;
    const float bdTerm = r.oppWon ? -1.0f : r.bdRaw;
    r.term = bdTerm < E.droneRadius ? TERM_LOSE : r.winner ? TERM_WIN : TERM_NONE;
    return r;
}

} // namespace dr
