// The verification's clearance test: which samples can no longer collide with the ego, from
// where the ego can be under the plan (ClearBlock, instance.cuh).
#pragma once

#include "instance.cuh"

namespace dr
{

// Steps between two clearance tests of a verification warp: a test costs about 60
// instructions, a step about 700. Four agents of 2 x 2^17 x 40, three drawn mid-race states
// (B200, 1965 MHz; the verification of the new plan): without the test 0.52 / 0.45 / 0.55 ms,
// every step 0.36 / 0.27 / 0.08, every second 0.35 / 0.26 / 0.08, every fourth 0.35 / 0.25 /
// 0.10.
#ifndef DR_CLEAR_EVERY
#define DR_CLEAR_EVERY 2
#endif
constexpr int CLEAR_EVERY = DR_CLEAR_EVERY;

// The block's rho in shared memory, from each group's own distances to those of it and the
// later ones; all threads of the CTA, synchronised before and after by the caller.
__device__ __forceinline__ void clearSuffix(float* block, int H)
{
    const ClearBlock<float> cb(block, H);
    for (int j = threadIdx.x; j < H; j += blockDim.x)
        for (int g = clearGroups(H) - 2; g >= 0; g--)
            cb.rho[g * H + j] = fmaxf(cb.rho[g * H + j], cb.rho[(g + 1) * H + j]);
}

// Whether no remaining step (t .. H - 1) of the warp's active samples can bring an opponent
// within two drone radii of the ego, or the ego off the track: then none of them can fail any
// more (a sample fails at the first step with boundary distance below the drone radius) and
// their remaining steps decide nothing. px .. vy: this lane's opponent before step t; xy: the
// ego's trajectory with no branch (which stays on the track), rho: how far the samples' own may
// be from it, after each step.
//
// An opponent whose speed is within its limit vmax moves k dt v in k steps plus at most
// amax dt^2 k (k - 1) / 2: the step moves it by its velocity before the step and then adds an
// acceleration clamped to amax, and the cap to vmax, a projection onto a ball that holds the
// old velocity, never moves the new one farther from it. The warp's opponents lie within
// (dp, dv) of the first active lane's in position and velocity (1-norms, which bound the
// Euclidean ones). The ego is on a row of its table: within rho of the trajectory with no
// branch. So after step j the two are at least |ego_j - (p + k dt v)| - rho - dp - k dt dv -
// amax dt^2 k (k - 1) / 2 apart, k = j - t + 1. Slack for the arithmetic (the verification's
// approximate factors are within 1e-5, positions round to 2^-24 a step): two millimetres, 1e-4
// of the reach and of the speed limit's way, and a few H roundings of the coordinates.
__device__ __forceinline__ bool clearOfEgo(float dt, float radius, const float* xy, const float* rho, int H, int t, bool active, float px, float py,
                                           float vx, float vy, float vmax, float amax)
{
    vmax = fabsf(vmax);
    amax = fabsf(amax);
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int src = __ffs(__ballot_sync(ALL, active)) - 1;
    const float cx = __shfl_sync(ALL, px, src), cy = __shfl_sync(ALL, py, src), wx = __shfl_sync(ALL, vx, src), wy = __shfl_sync(ALL, vy, src);
    float dp = 0.0f, dv = 0.0f;
    bool ok = true;
    if (active)
    {
        dp = fabsf(px - cx) + fabsf(py - cy);
        dv = fabsf(vx - wx) + fabsf(vy - wy);
        ok = vx * vx + vy * vy <= vmax * vmax * 1.0001f;
    }
    // non-negative floats (and NaN, above them all) order as their words
    dp = __uint_as_float(__reduce_max_sync(ALL, __float_as_uint(dp)));
    dv = __uint_as_float(__reduce_max_sync(ALL, __float_as_uint(dv)));
    for (int j = t + lane; j < H; j += 32)
    {
        const float k = (float)(j - t + 1), kd = k * dt;
        const float ex = xy[2 * j] - (cx + kd * wx), ey = xy[2 * j + 1] - (cy + kd * wy);
        const float way = kd * vmax;
        const float reach = 2.0f * radius + rho[j] + dp + kd * dv + 0.5f * amax * dt * dt * (k * (k - 1.0f));
        const float slack = 2e-3f + 1e-4f * (reach + way) + 4.8e-7f * (float)H * (fabsf(cx) + fabsf(cy) + way);
        const float need = reach + slack;
        ok = ok && ex * ex + ey * ey > need * need;
    }
    return __all_sync(ALL, ok);
}

} // namespace dr
