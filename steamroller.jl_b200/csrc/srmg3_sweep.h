// srmg3_sweep.h -- the cells of one colour of an octree level, as k3_gs_push counts them.
#pragma once
#include <cstdint>
#include <type_traits>

namespace srmg {

// MODE 0 red-black by rule, 1 red-black and 2 four colours from tables.  The tables exist only for
// fields of fewer than 2^31 values (so fewer than 2^30 cells a colour); the rule takes trees of
// any size, and a level of 2^20 blocks has 2^31 cells a colour.
template <int MODE>
struct Sweep3 {
  static constexpr int kCells = MODE == 2 ? 1024 : 2048;  // per block
  using Index = std::conditional_t<MODE == 0, int64_t, int>;
  static constexpr Index total(int nblk) { return (Index)nblk * kCells; }
};

}  // namespace srmg
