// gemm_plan.h — how a BF16 product of many rows is cut into tiles (gemm_bf16.cu).  Plain C++, so that it can be checked without a device.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>

namespace wr_plan {

constexpr uint32_t kBM = 128;                            // rows of one CTA
constexpr uint32_t kMaxN = 256;                          // columns of a tile, and of one accumulator of two
constexpr uint32_t kMapRows = 32;                        // a pair's rank takes a multiple of these of a tile's weight rows

struct Plan {
    uint64_t cost = ~0ull;
    uint32_t wide = 0, bn0 = kMaxN, bn1 = kMaxN;         // `wide` column tiles of bn0, the others of bn1
};

// A worker's clocks per 64 K-values of a tile: the products, or the operands on their way out of L2.  A pair takes 350 clocks
// or more, however narrow its tile (with 180 or 230 here narrower tiles are chosen: a prompt of 1501 rows with experts 1284 us
// -> 1295); a CTA by itself gets about 100 bytes a clock.
inline uint64_t tile_cost(uint32_t ranks, uint32_t bn) { return std::max(2u * bn, ranks == 2 ? 350u : 150u + (kBM + bn) * 5u / 4u) + 24u; }

// ... of the worker that has most: m_tiles x `wide` tiles of kMaxN columns, then m_tiles x the others (n columns in all) of bn.
inline uint64_t plan_cost(uint32_t ranks, uint32_t m_tiles, uint32_t n, uint32_t workers, uint32_t wide, uint32_t bn)
{
    const uint32_t left = n > wide * kMaxN ? (n - wide * kMaxN + bn - 1) / bn : 0u;
    const uint64_t t0 = (uint64_t)wide * m_tiles, tiles = t0 + (uint64_t)left * m_tiles;
    uint64_t cost = 0;                                   // tiles go round: the workers differ at two places only
    for (uint64_t w : {(uint64_t)0, t0 % workers}) {
        const uint64_t all = (tiles - std::min(w, tiles) + workers - 1) / workers, a = (t0 - std::min(w, t0) + workers - 1) / workers;
        cost = std::max(cost, a * tile_cost(ranks, kMaxN) + (all - a) * tile_cost(ranks, bn));
    }
    return cost;
}

// The cut of n columns into tiles that the workers finish first: tiles of 256 columns, and behind them (so that the last
// round is a full one) narrower tiles for the rest.  n_pad: n rounded up to whole blocks of the weight.
inline Plan plan(uint32_t ranks, uint32_t m_tiles, uint32_t n, uint32_t n_pad, uint32_t workers)
{
    Plan best;
    const uint32_t most = (n + kMaxN - 1) / kMaxN, rounds = (uint32_t)(((uint64_t)most * m_tiles + workers - 1) / workers);
    for (uint32_t k = 0; k < rounds && k < 9; ++k) {
        // wide tiles fill the first rounds but k (none at all: every tile has the narrow width)
        const uint64_t full = k + 1 == rounds || k == 8 ? 0 : (uint64_t)(rounds - 1 - k) * workers / m_tiles;
        const uint32_t wide = (uint32_t)std::min<uint64_t>(full, most);
        for (uint32_t bn = kMapRows * ranks; bn <= std::min(kMaxN, n_pad); bn += kMapRows * ranks) {
            const uint64_t cost = plan_cost(ranks, m_tiles, n, workers, wide, bn);
            if (cost < best.cost) {
                best.cost = cost;
                best.wide = wide;
                best.bn1 = bn;
            }
        }
    }
    return best;
}

// Tiles of experts' rows: how many there will be, one standard deviation less, and one more.
struct Tiles {
    uint32_t few = 0, usual = 0, many = 0;
};

// The same for tiles whose number only the device knows: one width, which finishes first on average.
inline Plan plan(uint32_t ranks, const Tiles &t, uint32_t n, uint32_t n_pad, uint32_t workers)
{
    Plan best;
    for (uint32_t bn = kMapRows * ranks; bn <= std::min(kMaxN, n_pad); bn += kMapRows * ranks) {
        const uint64_t cost = plan_cost(ranks, t.few, n, workers, 0, bn) + 2 * plan_cost(ranks, t.usual, n, workers, 0, bn) +
                              plan_cost(ranks, t.many, n, workers, 0, bn);
        if (cost < best.cost) {
            best.cost = cost;
            best.bn1 = bn;
        }
    }
    return best;
}

// Tiles of `tile` rows that `rows` rows with `top` of `experts` experts each fill, over routers that favour none: an expert's rows
// are a binomial number, which has ceil(number / tile) tiles, one for every k with number > k tile.  mean and dev: of all experts.
inline void expert_tiles(uint32_t rows, uint32_t experts, uint32_t top, uint32_t tile, double &mean, double &dev)
{
    const double p = std::min(1.0, (double)top / experts), middle = rows * p, spread = std::sqrt(middle * (1 - p));
    double one = 1 - std::pow(1 - p, (double)rows), squares = one;       // of one expert
    uint32_t k = 1;
    for (uint64_t at = tile; at < rows; at += tile, ++k) {
        const double d = at + 0.5 - middle, above = spread > 0 ? 0.5 * std::erfc(d / (spread * 1.4142135623730951)) : d < 0 ? 1.0 : 0.0;
        one += above;
        squares += (2 * k + 1) * above;
    }
    mean = experts * one;
    dev = std::sqrt(std::max(0.0, experts * (squares - one * one)));
}

// What counts is that the number is not too low: a cut for fewer tiles than there are has narrow columns, and rounds that its
// cost did not see.  (With rows * top / tile + half a tile per expert, 19 instead of 32 tiles for 100 rows of 32 experts, top 4,
// prompts of 17 to 200 rows took 1 to 3 % more: 4 layers of width 1024, 100 rows 452 -> 438 us, 129 rows 472 -> 457.)
inline Tiles likely_tiles(uint32_t rows, uint32_t experts, uint32_t top, uint32_t tile)
{
    double mean, dev;
    expert_tiles(rows, experts, top, tile, mean, dev);
    Tiles t;
    t.few = (uint32_t)std::max(1.0, std::round(mean - dev));
    t.usual = (uint32_t)std::max(1.0, std::round(mean));
    t.many = (uint32_t)std::max(1.0, std::round(mean + dev));
    return t;
}

// Rows of experts' tiles: 256, on pairs of CTAs, where nearly every tile of 256 stands for two of 128, else 128.  32 experts, top 4, us a
// prompt with tiles of 128 / 256 (4 layers of width 1024 and 2048, 2 of 4096), and how many of 128 one of 256 stands for:
//      768 rows 1.00   591 /  633   894 /  932   1033 / 1234        2048 rows 1.67  1017 / 1019  1514 / 1513   2211 / 2281
//     1024 rows 1.48   677 /  695  1009 / 1021   1315 / 1380        1152 rows 1.92   739 /  735  1113 / 1089   1631 / 1468
//     1280 rows 2.00   778 /  774  1171 / 1135   1733 / 1593        1501 rows 2.00   846 /  840  1251 / 1218   1772 / 1723
// and 2 layers   2560 rows 1.50  783 / 787  1160 / 1219    3584 rows 2.00  994 / 988  1518 / 1546    4096 rows 1.80  1097 / 1117  1714 / 1714
//     6000 rows 1.93  1676 / 1671  2609 / 2529    8192 rows 1.89  2157 / 2160  3561 / 3556
inline uint32_t expert_tile(uint32_t rows, uint32_t experts, uint32_t top)
{
    double one, two, dev;
    expert_tiles(rows, experts, top, kBM, one, dev);
    expert_tiles(rows, experts, top, 2 * kBM, two, dev);
    return one >= 1.9 * two ? 2 * kBM : kBM;
}

}  // namespace wr_plan
