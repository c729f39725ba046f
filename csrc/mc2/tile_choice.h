// Tile kernel of a plain bf16 product. Host arithmetic alone, so that the choice can be tested without a GPU.
#pragma once
#include <algorithm>
#include <cstdint>

namespace hccl {
namespace mc2 {

// Which tile kernel: waves of tiles times what a wave of that kernel takes, plus 40 for the launch of clusters. A part of the cost counts whole
// waves and the rest the fraction of the GPU that the tiles fill, since idle SMs leave power to the others. A wave per 4096 of K takes the tile's
// columns (pairs) or 0.9 of them (one CTA) plus what its loads of A and B hold it up, which is more where K is no multiple of 16: its rows then
// start inside 32-byte sectors. The constants were fitted to 130 random products on one B200. 122 others (513 to 8192 rows, N 512 to 28672, K 512 to 16384; every
// pair width in random order five times, 20 ms of its own before each; runs of one width differ by up to 8 %): the chosen pair width takes 1.010
// (K made of 64s), 1.005 (of 16s) and 1.002 (neither) of the best one on average, 1.12 at most; 192, 224 and 256 chosen by waves alone 1.019, 1.027
// and 1.108, 1.42 at most. With sectors and 128-byte lines taken for the same, K of 16s took 1.046 and up to 1.40: 5200 x 24872 x 864 274 us with 512
// columns, 195 with 256. Where rows start on sectors a width above 256 has to win by 2 %: 998 x 9128 x 5104 76.4 us with 512 columns and 68.2 with 256,
// 1358 x 12120 x 4480 129.5 and 113.9, 1000 x 6144 x 4096 42.1 with 352 columns and 43.0.
struct TileChoice { bool pair; uint32_t bn; };
inline TileChoice ChooseTile(uint64_t m, uint64_t n, uint64_t k, bool transposedB, uint64_t sms, bool pairsEnabled)
{
    const uint64_t pairs = sms / 2, rows = (m + 127) / 128, rowPairs = (rows + 1) / 2;
    const double k4 = (double)k / 4096;
    const bool straddle = k % 16 != 0;
    auto filled = [](uint64_t tiles, uint64_t slots) { return std::max(1.0, (double)tiles / (double)slots); };
    auto waves = [](uint64_t tiles, uint64_t slots) { return (double)((tiles + slots - 1) / slots); };
    auto one = [&](uint32_t bn) {
        const uint64_t tiles = rows * ((n + bn - 1) / bn);
        return (0.8 * waves(tiles, sms) + 0.2 * filled(tiles, sms)) * (20 + k4 * (0.9 * bn + (straddle ? 170 : 95)));
    };
    auto pair = [&](uint32_t bn) {
        const uint64_t tiles = rowPairs * ((n + bn - 1) / bn);
        const double whole = straddle ? 0.5 : 0.7, start = bn <= 256 ? 0 : straddle ? 20 : 45;
        return 40 + (whole * waves(tiles, pairs) + (1 - whole) * filled(tiles, pairs)) * (start + k4 * (bn + (straddle ? 200 : 45)));
    };
    TileChoice best{false, 64};
    double cost = one(64);
    auto offer = [&](bool isPair, uint32_t bn, double c) { if (c <= cost) { best = {isPair, bn}; cost = c; } };
    offer(false, 128, one(128));
    // 256-wide one-CTA tiles where N is made of them (another N was not measured)
    if (!transposedB && n % 256 == 0) offer(false, 256, one(256));
    if (!pairsEnabled) return best;
    offer(true, 256, pair(256));
    if (transposedB) {           // its tiles are whole 64-column boxes per CTA; 2048 x 4096 x 28672 377 / 359 us (256 / 512), 4096 x 4096 x 14336 389 / 368
        // from 8192 on: 4096 x 4096 x 8192 223 / 214, 2048 x 8192 x 8192 220 / 214, 8192 x 28672 x 8192 2790 / 2792; 2048 x 14336 x 4096 186 / 204
        if (k >= 8192) offer(true, 512, pair(512));
        return best;
    }
    offer(true, 224, pair(224));
    offer(true, 192, pair(192));
    const double limit = straddle ? cost : 0.98 * cost;
    for (uint32_t bn = 288; bn <= 512; bn += 32)
        if (pair(bn) <= limit) offer(true, bn, pair(bn));
    return best;
}

}  // namespace mc2
}  // namespace hccl
