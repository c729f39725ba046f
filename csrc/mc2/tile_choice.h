// Kernel of a plain product. Host arithmetic alone, so that the choice can be tested without a GPU.
#pragma once
#include <algorithm>
#include <cmath>
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
struct TileChoice { bool pair; uint32_t bn; double cost = 0; };          // cost: about 0.1 us
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
    TileChoice best{false, 64, one(64)};
    double &cost = best.cost;
    auto offer = [&](bool isPair, uint32_t bn, double c) { if (c <= cost) best = {isPair, bn, c}; };
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

// bt rows of A per tile (16, 32, 64, 128, 192, 256), split CTAs along K per tile (1 ... 8)
struct SplitKChoice { uint32_t bt = 0, split = 0; };

// The split-K rules below, their tables and their numbers of CTAs hold for the 148 SMs of a B200, whatever `sms` the tile rules are given: with fewer a choice is slower, not wrong.
// Clusters of 1 ... 8 CTAs that run at once with one CTA on an SM: SMs come in groups that a cluster does not cross. Read off the step in time over
// 967 products: with one cluster more than fit the product takes 1.4 times as long on average as with one CTA less along K.
constexpr uint32_t kClustersAtOnce[9] = {0, 148, 71, 44, 33, 26, 22, 15, 15};

// The same with two CTAs on an SM (16- to 64-row tiles), read off the step in time over 4900 products.
constexpr uint32_t kClustersOfTwoAtOnce[9] = {0, 296, 147, 91, 71, 55, 45, 37, 33};

// Time of a split-K product, in us up to `start`, as far as it depends on the tiles and the CTAs along K: a CTA's stream of B and A at its own rate (KB per us) and at the
// rate that all CTAs share, for each wave of clusters, and what a cluster and a further wave cost.
struct SplitKRates { double start, own, shared, cluster, wave; };
inline double SplitKCost(uint64_t tiles, uint32_t bt, uint64_t rowBytes, uint32_t s, const SplitKRates &r)
{
    const double kb = (double)(((rowBytes + 127) / 128 + s - 1) / s) * 0.128 * (128 + 0.7 * bt);
    auto wave = [&](uint64_t clusters) { return std::hypot(kb / r.own, (double)(clusters * s) * kb / r.shared); };
    const uint64_t cap = (bt <= 128 ? kClustersOfTwoAtOnce : kClustersAtOnce)[s], full = (tiles - 1) / cap;
    return r.start + (s > 1 ? r.cluster : 0.0) + 0.09 * s + (double)full * (wave(cap) + r.wave) + wave(tiles - full * cap);
}

// Whether the split-K form is the better one for this product, and its shape. narrowWave: the best tiles are 64 wide on one CTA and take one wave of at
// least 90 CTAs.
// Measured on one B200 with weights that rotate through more than L2, us per product in a graph of many (tile kernels / split-K):
//   rows <= 64: split-K wins or ties from K = 768 on with up to 32 rows (20 x 5016 x 1960: 18.6 / 8.2; 512 where N >= 2000: 24 x 9376 x 616 10.0 / 6.0), from 1024 on with up to
//     64 (44 x 584 x 1528 7.4 / 5.3, 55 x 5088 x 928 8.6 / 7.4; 39 x 2128 x 680 5.0 / 5.9), up to K = 2048 only where rows straddle sectors or N < 6000 (61 x 7224 x 1168 7.1 / 8.5);
//     block-scaled from 512 on (30 x 18280 x 1536 13.7 / 8.0). Long K: m x n x k = 4 x 4096 x 4096: 25.2 / 10.3; 16 x 4096 x 14336: 42.3 / 22.9; 1 x 512 x 16384:
//     47.8 / 11.1; 8 x 28672 x 4096: 50.5 / 40.6; 64 x 128256 x 4096: 195.8 / 171; 64 x 28672 x 8192: 81.3 / 79.8; 16 x 8192 x 1024: 9.8 / 7.1.
//   more rows: where the tile kernels leave the GPU partly empty (200 x 1024 x 8192: 26.1 / 13.4; 512 x 1024 x 4096: 15.4 / 12.2), not
//     where they have about as many CTAs as SMs (128 x 8192 x 1024: 8.1 / 10.3). One wave of 64-wide tiles is better up to K = 3700 (2400 where K straddles
//     sectors, which costs tiles more), and for every K where 257 to 384 rows leave the second 256-row tile half empty and two CTAs along
//     K: 193 x 4512 x 2624 11.0 / 12.7, 349 x 2216 x 2056 13.1 / 17.5, 365 x 3120 x 2880 11.7 / 16.6. Of 489 such products the choice takes 1.020 of the
//     best kernel's time on average; split-K for all of them 1.30.
//   more than 512 rows: where 256-row tiles with four or more CTAs along K run at once (683 x 624 x 16016: 49.4 / 21.8; 1191 x 528 x 3632: 13.7 / 13.1; 957 x 512 x 2176: 9.0 / 10.6),
//     with three where K straddles sectors or is long (1722 x 672 x 15048: 90.7 / 52.8; 1629 x 520 x 4112: 15.4 / 16.5), with two where it straddles (1.00 at K = 4700, 0.87 at
//     10000, aligned 1.02 at 9088). Over 276 products of 513 to 2048 rows with N up to 4096 and K from 2048 the best kernel is 1.15 times as fast as the tiles.
//   CTAs in all, rows <= 64: about one per SM while K is short (32 tiles, K 4096: split 4 10.3, 8 11.0; 64 tiles, K 1024: 2 7.1, 4 7.9), two per SM for a
//     long K (64 tiles, K 8192: 2 27.6, 4 25.9) or several row tiles (100 x 4096 x 4096: 3 14.2, 4 13.5). That rounds down: 92 tiles, K 3112 took one, 20.5, and with three 15.9. So
//     with up to 64 rows another number is taken where SplitKCost gives it less than 0.88 of that (0.75 below K = 2048): over 2739 bf16 and 2173 block-scaled products (1 to 64 rows, N 512 to 28672, K 512
//     to 16384, half of them held out of the fit) 1.014 and 1.010 of the best kernel's time on average, 1.058 and 1.044 before, these bounds on K included.
//   65 to 512 rows, bf16, us with 64-row tiles / chosen (split x rows): one tile of 128 rows in two CTAs per SM 88 x 10120 x 7160 74 / 39 (3 x 128),
//     122 x 10368 x 13952 91 / 56 (3 x 128), 69 x 4088 x 13504 30.7 / 24.3 (8 x 128); 256-row tiles, one CTA per SM, as many along K as run at once:
//     336 x 3704 x 15208 143 / 76 (3 x 256 although two would run at once, 91: K straddles sectors). 64-row tiles stay where six CTAs share one
//     (109 x 2088 x 15896 26.5 / 31.7 with 6 x 128) or three to five share a short K (229 x 1552 x 2464 9.1 / 10.0 with 8 x 256).
//   Over 967 random products of 65 to 512 rows the choice takes 1.030 of the best kernel's time on average; without 128- and 256-row tiles 1.075; with
//     four CTAs along K wherever 148 SMs have room for them, and tiles counted 128 wide, 1.041 and up to 1.95.
inline SplitKChoice ChooseSplitK(uint64_t m, uint64_t n, uint64_t k, bool mx, bool narrowWave)
{
    const uint64_t nt = (n + 127) / 128, tileCtas = (m + 127) / 128 * nt;       // tileCtas: CTAs that 128-wide tiles would use
    const bool straddle = !mx && k % 16 != 0;
    auto parts = [&](uint64_t s) { return (uint32_t)std::min<uint64_t>(8, std::min<uint64_t>(std::max<uint64_t>(1, s), k / 256)); };
    auto atOnce = [&](uint64_t tiles) { uint64_t s = 8; while (s > 1 && tiles > kClustersAtOnce[s]) --s; return s; };
    const uint64_t t256 = nt * ((m + 255) / 256);
    if (m > 512) {
        const uint64_t s = atOnce(t256), least = s >= 4 ? 3300 : s == 3 ? (straddle ? 3300 : 6000) : s == 2 && straddle ? 4600 : UINT64_MAX;
        return mx || k < least ? SplitKChoice{} : SplitKChoice{256, parts(s)};
    }
    if (m > 64 && (k < 2048 || tileCtas >= 90 || (narrowWave && k < (straddle ? 2400 : 3700)))) return {};
    if (m <= 64 && k < 512) return {};
    if (m > 16 && m <= 64 && !mx && k < 2048 && (m <= 32 ? k < 768 && n < 2000 : k < 1024 || (!straddle && n >= 6000))) return {};
    const uint32_t bt = m <= 16 ? 16 : m <= 32 ? 32 : 64;
    const uint64_t tiles = nt * ((m + bt - 1) / bt), ctas = k > 6144 || m > 64 ? 256 : 148;
    SplitKChoice narrow{bt, parts(ctas / tiles)};
    if (m <= 64) {
        const uint64_t rowBytes = mx ? k : 2 * k;
        const SplitKRates rates{0, rowBytes % 32 ? 25.0 : 78.0, 9700, 0.9, 2.4};          // a third where rows start inside 32-byte sectors
        double cost = (k < 2048 ? 0.75 : 0.88) * SplitKCost(nt, bt, rowBytes, narrow.split, rates);
        for (uint32_t s = 1; s <= parts(8); ++s)
            if (const double c = SplitKCost(nt, bt, rowBytes, s, rates); c < cost) { narrow.split = s; cost = c; }
    }
    if (m <= 64 || mx || narrow.split >= 6 || (k < 5000 && narrow.split >= 3)) return narrow;
    if (m <= 128) return k >= 4096 ? SplitKChoice{128, parts(256 / nt)} : SplitKChoice{};     // 72 x 7192 x 2576: 11.6, tiles 10.6
    const uint64_t s = atOnce(t256);
    if (s == 2 && narrowWave) return {};
    return {256, parts(s == 2 && straddle ? 3 : s)};
}

// The same for more than 64 rows, beside the tile that would be taken.
inline SplitKChoice ChooseSplitK(uint64_t m, uint64_t n, uint64_t k, const TileChoice &t, uint64_t sms)
{
    const uint64_t narrow = !t.pair && t.bn == 64 ? (m + 127) / 128 * ((n + 63) / 64) : 0;
    return ChooseSplitK(m, n, k, false, narrow >= 90 && narrow <= sms);
}

// Split-K with tiles of 192 or 256 rows, as many CTAs along K as run at once, where it beats the tiles (or ChooseSplitK's 256-row tiles) by its cost: 257 to 384 rows leave half of a second
// 256-row tile empty and three 128-row tiles of one CTA each wait for their operands, 384 x 4096 x 14336 76.9 us, now 41.5. Measured on one B200, 60 to 300 tiles of 128 x
// 128, us before / now: 367 x 3792 x 13504 55.0 / 40.5, 305 x 2528 x 14336 35.5 / 28.3, 671 x 2032 x 7920 38.0 / 30.1, 156 x 5736 x 15496 95.2 / 66.7. Over 426 products of 129 to 1100 rows and K from
// 4500 0.960 of the time before on average; two are 3 to 5 % slower. With a shorter K it is mixed: K = 3840 up to 17 % faster and up to 13 % slower, 273 x 4280 x 2048 11.4 / 13.2.
inline SplitKChoice ChooseWideSplit(uint64_t m, uint64_t n, uint64_t k, const TileChoice &t, SplitKChoice sk)
{
    if (m <= 128 || k < 4500 || (sk.split && sk.bt != 256)) return sk;
    auto cost = [&](uint32_t bt, uint64_t s) {
        const double part = (double)k / 4096 / (double)s;
        if (bt == 192) return k % 16 ? 6.9 + 0.1 * (double)s + 32.2 * part : 4.5 + 1.2 * (double)s + 18.9 * part;
        return k % 16 ? 7.7 + 37.6 * part : 6.1 + 0.7 * (double)s + 24.65 * part;
    };
    double least = sk.split ? 0.97 * cost(256, sk.split) : 0.9 * 0.084 * t.cost;
    for (uint32_t bt : {192u, 256u}) {
        const uint64_t tiles = (n + 127) / 128 * ((m + bt - 1) / bt);
        uint64_t s = 8;
        while (s > 1 && tiles > kClustersAtOnce[s]) --s;
        if (s > 1 && cost(bt, s) < least) { sk = {bt, (uint32_t)s}; least = cost(bt, s); }
    }
    return sk;
}

// The kernel of C = A * B^T in bf16: split-K where `split` is not 0, else the tile.
struct PlainChoice { SplitKChoice splitK; TileChoice tile; };
inline PlainChoice ChoosePlain(uint64_t m, uint64_t n, uint64_t k, uint64_t sms, bool pairsEnabled)
{
    if (m <= 64) {
        const SplitKChoice sk = ChooseSplitK(m, n, k, false, false);
        if (sk.split) return {sk, {false, 64}};
    }
    const TileChoice t = ChooseTile(m, n, k, false, sms, pairsEnabled);
    return {m <= 64 ? SplitKChoice{} : ChooseWideSplit(m, n, k, t, ChooseSplitK(m, n, k, t, sms)), t};
}

// The kernel of C = A * B with B stored [K, N] (the input gradient of a linear layer). It had no split-K form: few tiles each walked all of K. Measured on
// one B200, us tiles / split-K: 12 x 512 x 26784 74.5 / 13.8, 19 x 4456 x 2448 16.1 / 8.6, 94 x 312 x 21624 95.4 / 17.8, 109 x 9136 x 15336 76.5 / 60.3, 548 x 2528 x 12352 45.2 / 35.5.
// Up to 64 rows split-K from K = 512 on, 0.51 of the tiles' time on average over 384 products (1.015 of the best number of CTAs). More rows: the tile height whose one wave of
// clusters costs least, where that is below 0.85 of the tiles' cost: 0.70 on average over 570 products of 65 to 1100 rows, N 256 to 14336 and K 512 to 28672; 7 of them are more than 3 % slower.
inline PlainChoice ChooseNn(uint64_t m, uint64_t n, uint64_t k, uint64_t sms, bool pairsEnabled)
{
    PlainChoice best{{}, ChooseTile(m, n, k, true, sms, pairsEnabled)};
    if (k < 512) return best;
    const uint64_t nt = (n + 127) / 128;
    if (m <= 64) {
        const uint32_t bt = m <= 16 ? 16 : m <= 32 ? 32 : 64;
        double least = HUGE_VAL;
        for (uint32_t s = 1; s <= 8 && s * 256 <= k; ++s)
            if (const double c = SplitKCost(nt, bt, 2 * k, s, {0, 60, 9700, 0.9, 2.4}); c < least) { best.splitK = {bt, s}; least = c; }
        return best;
    }
    struct Rows { uint32_t bt; double start, perCta, along, straddling; };              // us, along 4096 of K in a CTA (rows of B inside 32-byte sectors)
    double least = 0.85 * 0.0917 * best.tile.cost;
    for (const Rows &r : {Rows{64, 4.5, 0.23, 23.8, 33.7}, Rows{128, 6.3, 0.27, 32.5, 41.4}, Rows{192, 6.0, 0.1, 22, 26.4}, Rows{256, 6.9, 0.05, 26.5, 30.6}}) {
        const uint64_t tiles = nt * ((m + r.bt - 1) / r.bt);
        uint64_t s = std::min<uint64_t>(8, k / 256);
        while (s > 1 && tiles > (r.bt <= 128 ? kClustersOfTwoAtOnce : kClustersAtOnce)[s]) --s;
        const double c = r.start + r.perCta * (double)s + (n % 16 ? r.straddling : r.along) * (double)k / 4096 / (double)s;
        if (s > 1 && c < least) { best.splitK = {r.bt, (uint32_t)s}; least = c; }
    }
    return best;
}

// The kernel of a block-scaled product: split-K where `split` is not 0, else tiles of CTA pairs (192 or 256 wide) or of one CTA (128, 192, 256).
// Up to 64 rows see ChooseSplitK. More: the rule by which products were split up to 512 rows and K from 2048, pair tiles taken where they about fill the GPU and 256-wide
// tiles where they do, kept most of the GPU idle just below each of its bounds. Another kernel is taken where its cost is below 0.92 of that rule's: a start, waves of
// tiles (a quarter of them by the fraction of the GPU that the tiles fill) of a fixed part and a part along K, or SplitKCost. Fitted on one B200 to 829 products of 65 to 8192
// rows, N 512 to 28672 and K 512 to 16384; over 828 others the choice takes 1.016 of the best kernel's time on average, the rule alone 1.080 and up to 1.72. us, rule / now:
// 125 x 520 x 1792 7.2 / 4.9, 197 x 10544 x 15104 64.9 / 41.3, 252 x 5432 x 11392 31.9 / 21.2, 620 x 4160 x 5120 23.1 / 15.4, 739 x 1176 x 16256 32.0 / 19.8.
struct MxChoice { SplitKChoice splitK; TileChoice tile; };
inline MxChoice ChooseMx(uint64_t m, uint64_t n, uint64_t k, uint64_t sms, bool pairsEnabled)
{
    const uint64_t rows = (m + 127) / 128, pairRows = (m + 255) / 256, pairs = sms / 2, t192 = pairRows * ((n + 191) / 192), t256 = pairRows * ((n + 255) / 256);
    const double k4 = (double)k / 4096;
    const SplitKChoice sk = ChooseSplitK(m, n, k, true, false);
    if (m <= 64 && sk.split) return {sk, {false, 128}};
    const bool canPair = pairsEnabled && n >= 256;
    auto tiles = [&](TileChoice t) {
        constexpr double kStart[5] = {3.2, 2.9, 2.9, 2.5, 2.1}, kWave[5] = {0.46, 1.2, 2.45, 1.75, 3.85}, kAlongK[5] = {7.9, 9.4, 11.8, 8.3, 10.2};
        const int i = t.pair ? (t.bn == 192 ? 3 : 4) : t.bn == 128 ? 0 : t.bn == 192 ? 1 : 2;
        const uint64_t count = (t.pair ? pairRows : rows) * ((n + t.bn - 1) / t.bn), slots = t.pair ? pairs : sms;
        const double waves = 0.75 * (double)((count + slots - 1) / slots) + 0.25 * std::max(1.0, (double)count / (double)slots);
        return kStart[i] + waves * (kWave[i] + kAlongK[i] * k4);
    };
    auto split = [&](SplitKChoice c) {
        const uint64_t count = (n + 127) / 128 * ((m + c.bt - 1) / c.bt);
        return SplitKCost(count, c.bt, k, c.split, c.bt == 64 ? SplitKRates{2.9, 98, 16300, 1.06, 2.8} : SplitKRates{6.0, 141, 17800, 0.94, 2.45});
    };
    MxChoice best{sk, {false, 128}};
    if (!sk.split) {
        if (canPair && (t192 >= pairs || t256 * 8 >= pairs * 7)) {
            const double c192 = (double)((t192 + pairs - 1) / pairs) * 11.2 * k4, c256 = (double)((t256 + pairs - 1) / pairs) * (14.0 * k4 + 4.5);
            best.tile = {true, c256 < c192 ? 256u : 192u};
        } else if (rows * ((n + 255) / 256) >= sms) best.tile = {false, 256};
    }
    if (m <= 64) return best;
    double cost = 0.92 * (sk.split ? split(sk) : tiles(best.tile));
    auto offer = [&](const MxChoice &c) {
        const double t = c.splitK.split ? split(c.splitK) : tiles(c.tile);
        if (t < cost) { best = c; cost = t; }
    };
    for (uint32_t bn : {128u, 192u, 256u}) {
        offer({{}, {false, bn}});
        if (canPair && bn > 128) offer({{}, {true, bn}});
    }
    for (uint32_t s = 1; s <= 8 && s * 256 <= k; ++s) {
        if (m <= 512) offer({{64, s}, {false, 128}});
        if (s > 1) offer({{256, s}, {false, 128}});
    }
    return best;
}

// Pair tile width of the product with SwiGLU in its epilogue (forward: half of it gate, half up; backward: columns of the intermediate gradient), 0 = the product and the
// element-wise kernel one after the other. Not where the product by itself splits K: the fused kernel has no such form, its tiles each walk all of K, and its sums would have another order. Us
// separate / fused there, one B200: forward 52 x 2 x 13152 x 1384 23.1 / 23.8, 35 x 2 x 3072 x 1144 9.3 / 11.7, 168 x 2 x 2952 x 8616 39.0 / 47.4, 781 x 2 x 184 x 16352 20.6 / 55.5; backward 1098 x 1400 x 10784
// 44.6 / 48.0, 620 x 128 x 13320 17.7 / 53.6. Of 340 such products fused would be faster for 26, by 17 % at most (two CTAs along K: 832 x 2 x 1040 x 5064 35.2 / 29.3), and takes 1.4 times as long on average. Elsewhere
// forward always: 60 x 2 x 512 x 256 5.5 / 5.2, 200 x 2 x 14336 x 4096 61.2 / 60.9, 300 x 2 x 3584 x 1024 11.5 / 12.2. Backward: above 512 rows (777 x 14336 x 4096 135 / 126, 513 x 2056 x 1032 14.1 / 13.7); up to there
// one-CTA tiles fill the GPU better: 300 x 7168 x 2048 22.8 / 24.2, 130 x 14336 x 4096 37.0 / 40.1, 256 x 512 x 256 6.3 / 8.5.
inline uint32_t ChooseSwiGlu(uint64_t m, uint64_t ffn, uint64_t k, bool backward, uint64_t sms, bool pairsEnabled)
{
    if (!pairsEnabled || (backward && m <= 512)) return 0;
    if ((backward ? ChooseNn(m, ffn, k, sms, pairsEnabled) : ChoosePlain(m, 2 * ffn, k, sms, pairsEnabled)).splitK.split) return 0;
    const uint64_t pairs = sms / 2, rowPairs = (m + 255) / 256;
    const double k4 = (double)k / 4096;
    uint32_t best = 0;
    double cost = 0;
    auto offer = [&](uint32_t bn) {
        const uint64_t cols = backward ? bn : bn / 2, tiles = rowPairs * ((ffn + cols - 1) / cols);
        const double whole = (double)((tiles + pairs - 1) / pairs), c = (0.7 * whole + 0.3 * std::max(1.0, (double)tiles / (double)pairs)) * (k4 * (bn + 45) + 20);
        if (!best || c <= cost) { best = bn; cost = c; }
    };
    offer(128);
    if (!backward) { offer(192); offer(224); }
    offer(256);
    return best;
}

}  // namespace mc2
}  // namespace hccl
