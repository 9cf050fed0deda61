// launch_shape.hpp -- launch shapes that depend on the size of a batch (host only, no CUDA).
#pragma once

#include <algorithm>
#include <cstdint>

namespace cmpmc_gpu {

// Launch shape of a thread-per-unit kernel (plain, inline, adjoint and charge kernels). A unit
// is one serial chain of thousands of steps, and the lanes of a warp that hold units wait for
// each other's branches, so a batch that cannot fill the chip runs fewer units per warp: as
// many lanes as it takes to give every resident warp work, never more warps than are resident.
// Against 32 lanes of fewer warps, per call with the steps as they were then: 2,000 plain phonon
// events 131 -> 84 ms, 203 plain mixed events 510 -> 234, 2,000 pairs 127 -> 101, adjoint of 200
// events 128 -> 112.
// `late` (percent) lets that share of the units beyond the resident warps start on a lane that
// came free, so that every warp still runs one unit alone. It pays for plain phonon events, at
// one lane only (kernel ms, one lane / two: 2,000 events of one phonon 62 / 72, 1,900 events of
// 100 phonons 5,930 / 6,410). From two lanes on every unit starts at once, since a late one adds
// its whole length at the end (all at once / a quarter late: 4,000 events of 100 phonons 10,450 /
// 12,080, 10,000 events 18,300 / 20,870), and events with carriers always do (1,400 mixed events
// 218 / 244, 4,000 360 / 550, 10,000 586 / 870).
struct Spread {
    uint64_t grid;   // blocks
    uint32_t lanes;  // lanes of each warp that take units
};
constexpr uint64_t kLatePhonons = 25, kLateNone = 0;
inline Spread spread_units(uint64_t units, uint64_t max_blocks, int tpb, uint64_t late) {
    const uint64_t wpb = static_cast<uint64_t>(tpb) / 32;
    const uint64_t warps = std::max<uint64_t>(1, max_blocks * wpb);
    units = std::max<uint64_t>(units, 1);
    Spread r;
    r.lanes = (units <= warps * (100 + late) / 100)
                  ? 1u
                  : static_cast<uint32_t>(std::min<uint64_t>(32, (units + warps - 1) / warps));
    r.grid = std::max<uint64_t>(1, std::min<uint64_t>(max_blocks, (units + r.lanes * wpb - 1) / (r.lanes * wpb)));
    return r;
}

}  // namespace cmpmc_gpu
