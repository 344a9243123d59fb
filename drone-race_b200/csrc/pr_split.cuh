// How a PR-MPPI rollout CTA that shares one ego per sample splits its threads: whole warps that
// step an opponent each, one per (sample, hypothesis), then whole warps that step an ego each,
// one per sample (pr_rollout_shared, gate_pr_rollout_shared).
#pragma once

namespace dr
{

constexpr int PRS_TILE = 512;     // threads of a CTA, unless the launch is small (sharedThreads)
#ifndef DR_PRS_MIN_TILE
#define DR_PRS_MIN_TILE 128
#endif
constexpr int PRS_MIN_TILE = DR_PRS_MIN_TILE; // fewest

struct PrSplit
{
    int samples; // a tile's
    int opp;     // threads that step opponents: whole warps
};

__host__ __device__ inline int prWarps(int threads)
{
    return (threads + 31) & ~31;
}

// the most samples, up to `most`, whose opponents and egos fit `threads` threads
__host__ __device__ inline PrSplit prSplit(int P, int threads, int most)
{
    int n = threads / P < most ? threads / P : most;
    while (n > 1 && prWarps(n * P) + prWarps(n) > threads)
        n--;
    return PrSplit{n, prWarps(n * P)};
}

// The samples of a rollout tile: where the kernel shares egos, those whose opponents and egos fit
// `threads` threads, else those whose (sample, hypothesis) slots do; `most` slots a CTA.
__host__ __device__ inline int prTileSamples(bool shared, int P, int threads, int most)
{
    return shared ? prSplit(P, threads, most / P).samples : (threads < most ? threads : most) / P;
}

} // namespace dr
