// Tile width, K split and stages a GEMM takes (csrc/gemm.cu). Host arithmetic
// only.
#pragma once

#include <cstdint>
#include <initializer_list>

namespace xg {
namespace ops {
namespace mm {

constexpr int BM = 128, BK = 64;

struct Shape {
    int bn, split, stages;
};
// A GEMM's time is, beside its start (2.5 us), waves x (k-blocks x T_KB + the tile's start and
// epilogue), in us. T_KB does not depend on the tile's width: 0.31 to 0.33 us a
// 64-deep k-block for 64, 128 and 256 columns alike (fits over 30 sizes of M and
// N, K 256 to 5,248, on one B200). What a k-block takes is the chain of waits and
// issues of the two threads that run the loop, then, and neither the operands'
// bytes, which double from 64 to 256 columns, nor the tensor core (0.07 to 0.27
// us); only transposed operands make wide tiles slower. So the widest tile wins
// until the SMs run out of tiles, and two CTAs an SM (128 columns, three stages)
// run their chains beside each other for a tenth more each. Against the same
// sizes' best shape the rule loses 0.1 % on average. A rule that took T_KB as
// proportional to the tile's bytes gave sizes of more than one wave one CTA an SM:
// 512 x 5,248 x 5,248 in 67 us against 37, 4,096 x 5,248 x 5,248 in 335 against 208.
constexpr double T_KB = 0.32, T_SPLIT = 2.2, T_PAIR = 1.6, PAIR_KB = 1.1;
constexpr double t_tile(int bn) { return bn == 256 ? 6.0 : bn == 128 ? 4.0 : 2.8; }
// more of a k-block where both operands are transposed
constexpr double t_kb_mn(int bn) { return bn == 256 ? 0.08 : bn == 128 ? 0.03 : 0.0; }

// One CTA an SM: 192 KB of operands in flight.
constexpr int stages_for(int bn) { return bn == 256 ? 4 : bn == 128 ? 6 : 8; }

// cluster_ctas(bn, split): CTAs of clusters of `split` that the GPU holds at
// once; 0 where it holds none, and then no shape has that split. mn: both operands
// are transposed.
template <class Ctas>
Shape shape_for(uint64_t M, uint64_t N, uint64_t K, int sms, bool may_split, bool mn,
                const Ctas &cluster_ctas) {
    const uint64_t KB = K / BK;
    Shape best{128, 1, 6};
    double cost = 1e300;
    auto consider = [&](int bn, int split, int stages, double c) {
        if (c < cost) {
            cost = c;
            best = Shape{bn, split, stages};
        }
    };
    auto waves = [&](uint64_t ctas, int slots) { return (double)((ctas + slots - 1) / slots); };
    for (int bn : {256, 128, 64}) {
        if (N % (uint64_t)bn) continue;
        const double kb = T_KB + (mn ? t_kb_mn(bn) : 0.0);
        for (int split : {1, 2, 4, 8}) {
            if (split > 1 && (!may_split || KB < 4ull * split)) break;
            const int slots = split > 1 ? cluster_ctas(bn, split) : sms;
            if (slots < split) continue;
            const uint64_t ctas = (M / BM) * (N / bn) * split;
            consider(bn, split, stages_for(bn),
                     waves(ctas, slots) * ((double)((KB + split - 1) / split) * kb + t_tile(bn) +
                                           (split > 1 ? T_SPLIT : 0.0)));
            if (bn == 128 && split == 1 && ctas > (uint64_t)sms)
                consider(bn, 1, 3, waves(ctas, 2 * sms) *
                                       ((double)KB * kb * PAIR_KB + t_tile(bn) + T_PAIR));
        }
    }
    return best;
}

}  // namespace mm
}  // namespace ops
}  // namespace xg
