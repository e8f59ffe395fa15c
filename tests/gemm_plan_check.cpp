// Draws routers that favour no expert and compares the tiles that their rows fill with wr_plan::likely_tiles, and the cut that is
// chosen for them with the best one for the tiles that there are (both by wr_plan::plan_cost).  The usual number may be off by
// its rounding, by four standard errors of the draws' mean and by 1 % (an approximation of the binomial numbers); the cost by 10 %
// on average over draws, as a tile more or less can make a round of its own.
#include <cmath>
#include <cstdio>
#include <numeric>
#include <random>
#include <vector>

#include "gemm_plan.h"

static uint64_t best_cost(uint32_t ranks, uint32_t tiles, uint32_t n, uint32_t workers)
{
    uint64_t best = ~0ull;
    for (uint32_t bn = wr_plan::kMapRows * ranks; bn <= wr_plan::kMaxN; bn += wr_plan::kMapRows * ranks)
        best = std::min(best, wr_plan::plan_cost(ranks, tiles, n, workers, 0, bn));
    return best;
}

int main()
{
    std::mt19937 rng(1);
    const uint32_t routers[][2] = {{32, 4}, {8, 2}, {64, 8}, {130, 1}, {5, 5}, {2, 1}};
    const uint32_t rows[] = {17, 18, 40, 64, 100, 129, 200, 300, 500, 682, 767, 768, 1024, 1501, 2048, 5000};
    double off = -1, slow = 0;
    for (const auto &r : routers)
        for (uint32_t n : rows)
            for (uint32_t tile : {128u, 256u}) {
                const uint32_t e = r[0], top = r[1], draws = 40;
                double mean = 0, squares = 0, cost = 0, best = 0;
                const wr_plan::Tiles likely = wr_plan::likely_tiles(n, e, top, tile);
                const uint32_t ranks = tile / 128, workers = 148 / ranks;
                for (uint32_t d = 0; d < draws; ++d) {
                    std::vector<uint32_t> count(e), all(e);
                    std::iota(all.begin(), all.end(), 0u);
                    for (uint32_t i = 0; i < n; ++i)
                        for (uint32_t k = 0; k < top; ++k) {
                            std::swap(all[k], all[k + rng() % (e - k)]);
                            ++count[all[k]];
                        }
                    uint32_t tiles = 0;
                    for (uint32_t c : count) tiles += (c + tile - 1) / tile;
                    mean += tiles;
                    squares += (double)tiles * tiles;
                    for (uint32_t cols : {1024u, 1536u, 2048u, 3072u, 4096u, 6144u}) {
                        const uint32_t bn = wr_plan::plan(ranks, likely, cols, cols, workers).bn1;
                        cost += wr_plan::plan_cost(ranks, tiles, cols, workers, 0, bn) / (double)best_cost(ranks, tiles, cols, workers);
                        best += 1;
                    }
                }
                mean /= draws;
                const double error = std::sqrt(std::max(0.0, squares / draws - mean * mean) / draws), room = 4 * error + 0.01 * mean;
                const double by = std::abs(mean - likely.usual) - 0.5 - room;
                off = std::max(off, by);
                slow = std::max(slow, cost / best);
                if (by > 0 || cost / best > 1.1 || likely.few > likely.usual || likely.many < likely.usual)
                    printf("experts %u top %u rows %u tile %u: %.1f tiles, taken for %u, cost %.2f\n", e, top, n, tile, mean, likely.usual, cost / best);
            }
    printf("off by %.2f, cost at most %.3f\n", off, slow);
    return off <= 0 && slow <= 1.1 ? 0 : 1;
}
