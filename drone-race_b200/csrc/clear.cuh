// The verification's clearance test: which samples can no longer collide with the ego, from
// where the ego can be under the plan (ClearBlock, instance.cuh).
#pragma once

#include "instance.cuh"

namespace dr
{

// The steps before which a verification warp takes the clearance test (at the first one its
// tile has): a test costs up to 100 instructions, a step about 700. Control steps of four agents
// of 2 x 2^17 samples x 40, three drawn mid-race states (B200, 1965 MHz), every step / second /
// fourth: 680 673 670, 622 613 608, 401 400 412 us; the second besides the fourths gives the last
// row its 400. (The gate race's, whose steps cost less, wait longer after a test that failed by
// more: clearOfEgo's wait.)
__device__ __forceinline__ bool clearTime(int t)
{
    return t == 2 || (t > 0 && t % 4 == 0);
}

// The block's rho in shared memory, from each group's own distances to those of it and the
// later ones; all threads of the CTA, synchronised before and after by the caller.
__device__ __forceinline__ void clearSuffix(float* block, int H)
{
    const ClearBlock<float> cb(block, H);
    for (int j = threadIdx.x; j < H; j += blockDim.x)
        for (int g = clearGroups(H) - 2; g >= 0; g--)
            cb.rho[g * H + j] = fmaxf(cb.rho[g * H + j], cb.rho[(g + 1) * H + j]);
}

// Whether opponents within (dp, dv) of position c and velocity w before step t (1-norms, which
// bound the Euclidean ones) are out of reach of the ego after step j. The ego is within rho[j]
// of the trajectory with no branch, xy[j].
//
// An opponent moves by its velocity before the step; then an acceleration clamped to amax is
// added to that, and the result capped to vmax: a projection onto a ball that holds the old
// velocity, which moves the new one neither farther from the old one nor, along any direction,
// above vmax. So along the unit vector n its k = j - t + 1 steps take it at most
// sum_i dt min(w n + dv + amax dt i, vmax), and with the first m of the minima taken on the left
// and the others on the right, for any m, at most
//   k dt w n + m dt dv + amax dt^2 m (m - 1) / 2 + (k - m) dt (vmax - w n).
// n points to the ego from where the opponent gets at velocity w, m is about the steps that it
// takes to reach vmax along n: of an opponent that follows the ego near its speed limit, the
// limit bounds the way better than the acceleration does (control step of four agents with one
// such follower 764 -> 667 us). Slack for the arithmetic (the
// verification's approximate factors are within 1e-5, positions round to 2^-24 a step): two
// millimetres, 1e-4 of the reach and of the speed limit's way, and a few H roundings of the
// coordinates.
__device__ __forceinline__ bool clearAfter(float dt, float radius, const float* xy, const float* rho, int H, int t, int j, float cx, float cy, float wx,
                                           float wy, float dp, float dv, float vmax, float amax, float* margin = nullptr)
{
    const float k = (float)(j - t + 1), kd = k * dt;
    const float ex = xy[2 * j] - (cx + kd * wx), ey = xy[2 * j + 1] - (cy + kd * wy);
    const float sq = ex * ex + ey * ey;
    const float inv = rsqrtf(sq);
    const float room = fmaxf(vmax - (wx * ex + wy * ey) * inv, 0.0f);
    const float m = fmaxf(fminf(rintf(__fdividef(room - dv, amax * dt)), k), 0.0f);
    const float way = kd * vmax;
    const float reach = 2.0f * radius + rho[j] + dp + m * dt * dv + 0.5f * amax * dt * dt * (m * (m - 1.0f)) + (k - m) * dt * room;
    const float slack = 2e-3f + 1e-4f * (reach + way) + 4.8e-7f * (float)H * (fabsf(cx) + fabsf(cy) + way);
    const float need = reach + slack;
    if (margin) // negative: by how much it is missed
        *margin = sq * inv - need;
    return sq > need * need && sq < 1e30f;
}

// Whether no remaining step (t .. H - 1) of the warp's active samples can bring an opponent
// within two drone radii of the ego, or the ego off the track: then none of them can fail any
// more (a sample fails at the first step with boundary distance below the drone radius) and
// their remaining steps decide nothing. px .. vy: this lane's opponent before step t; xy, rho:
// the ego's trajectory with no branch (which stays on the track) and how far the samples' own
// may be from it, after each step. witness: the last step that was within reach, -1 at first.
// While a sample by itself can still be there, the others need no test: that takes 25
// instructions in place of up to 100.
// wait: after a test that failed, how many steps it takes until the reach to the witness is shorter
// by what was missing (each takes amax dt^2 k off it); 0 for 64 and more, since an infinite reach (a
// branch that leaves the track) ends with that branch's step. Tests before that seldom succeed. Gate
// race (B200, 1965 MHz), a test every fourth step / with the wait: control step of four agents in the
// benchmark's state, where nothing clears, 1.008 / 0.962 ms (0.958 without tests or tables), in three
// drawn mid-race states 627 588 525 / 616 574 513 us. Half the wait / 1.4 times / twice, against 0.964 ms
// and 617 577 513 us of a first form: 0.970 / 0.966 / 0.990, 622 579 515 / 635 593 513 / 710 641 533.
__device__ __forceinline__ bool clearOfEgo(float dt, float radius, const float* xy, const float* rho, int H, int t, bool active, float px, float py,
                                           float vx, float vy, float vmax, float amax, int& witness, int* wait = nullptr)
{
    vmax = fabsf(vmax);
    amax = fabsf(amax);
    constexpr unsigned ALL = 0xffffffffu;
    // the step that the last test found within reach: as long as a sample by itself can be there
    if (witness >= t && __any_sync(ALL, active && !clearAfter(dt, radius, xy, rho, H, t, witness, px, py, vx, vy, 0.0f, 0.0f, vmax, amax)))
        return false;
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
    if (!__all_sync(ALL, ok))
        return false;
    for (int j0 = H - 1 - (H - 1 - t) % 32; j0 >= t; j0 -= 32)
    {
        const int j = j0 + lane;
        float margin = 0.0f;
        const unsigned near = __ballot_sync(ALL, j < H && !clearAfter(dt, radius, xy, rho, H, t, j, cx, cy, wx, wy, dp, dv, vmax, amax, wait ? &margin : nullptr));
        if (near)
        {
            const int last = 31 - __clz(near);
            witness = j0 + last;
            if (wait)
            {
                const float miss = -__shfl_sync(ALL, margin, last);
                *wait = (int)fminf(__fdividef(miss, amax * dt * dt * (float)(witness - t + 1)), 64.0f) & 63;
            }
            return false;
        }
    }
    return true;
}

// The same out of line: in line it costs the race's verification, at its 64 registers a thread,
// 376 bytes of reloads against 82 (control steps of four agents 731 -> 677, 667 -> 613 us). The
// gate race's step has the registers and is 3 % faster with the test in line.
static __device__ __noinline__ bool clearOfEgoCall(float dt, float radius, const float* xy, const float* rho, int H, int t, bool active, float px, float py,
                                                   float vx, float vy, float vmax, float amax, int& witness)
{
    return clearOfEgo(dt, radius, xy, rho, H, t, active, px, py, vx, vy, vmax, amax, witness);
}

} // namespace dr
