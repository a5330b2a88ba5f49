// Token rows per tile that the expert kernels exist for, as the switches choose among them (plain C++: host tests include it).
#pragma once

namespace smoe {

// What a switch asked for: 0 (the built-in rule) for numbers below 1, else the next size there is, the largest beyond it.
template <int N>
inline int existing_tile(int asked, const int (&sizes)[N]) {
    if (asked <= 0) return 0;
    for (int s : sizes)
        if (asked <= s) return s;
    return sizes[N - 1];
}
// The tile list has room for tiles of 16 rows, not for smaller ones, and a tile of more rows than its kernel's stages hold
// would be copied past their end.
constexpr int kPairTileSizes[] = {16, 32, 64};
constexpr int kPlaneTileSizes[] = {16, 24};

}  // namespace smoe
