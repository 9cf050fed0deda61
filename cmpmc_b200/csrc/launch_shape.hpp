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

// Launch shape of the SM-phase pool: one block per SM (512 threads in FP32, 768 in FP64) from the
// first units on, since a unit's lineage runs on its block alone (a block per 512 units left 108
// of 148 SMs without work at 20,300 units: 45 against 26 ms; 100 units 10.8 against 8.5 ms).
// `ring` is the pending phonons that a block has room for. PoolRing::cap is for a block with one
// unit per thread or more; blocks that start with fewer units get twice the same room per unit (a
// power of two, at least PoolRing::low), so a small batch does not hold a gigabyte of rings.
struct PoolRing {
    uint32_t cap = 1u << 17;
    uint32_t low = 4096;
};
struct PoolShape {
    uint64_t grid;      // blocks
    uint32_t ring;      // ring entries per block (a power of two)
    uint64_t per_block;  // units per block
};
constexpr uint32_t kRingMax = 1u << 24;
// the fewest blocks that a batch is packed into: one unit per thread
inline uint64_t pool_packed_grid(uint64_t units, uint64_t sms, uint64_t threads) {
    return std::max<uint64_t>(1, std::min(sms, (units + threads - 1) / threads));
}
inline PoolShape pool_shape_of(const PoolRing& r, uint64_t units, uint64_t grid, uint64_t threads) {
    PoolShape s{grid, std::min(r.cap, r.low), (std::max<uint64_t>(units, 1) + grid - 1) / grid};
    while (s.ring < r.cap && s.ring / 2 * threads < r.cap * s.per_block) s.ring *= 2;
    return s;
}
// Rings that grew past 2^17 entries would take more memory on every SM than a full batch holds at
// first (1.6 GB in FP32): such a batch gets fewer blocks, down to the packed ones.
inline PoolShape pool_shape(const PoolRing& r, uint64_t units, uint64_t sms, uint64_t threads) {
    const uint64_t packed = pool_packed_grid(units, sms, threads), room = sms << 17;
    PoolShape s = pool_shape_of(r, units, std::max<uint64_t>(1, std::min(sms, units)), threads);
    while (s.grid > packed && s.grid * s.ring > room)
        s = pool_shape_of(r, units, std::max<uint64_t>(packed, room / s.ring), threads);
    return s;
}
// After a ring overflow of a launch of shape `used`: full rings if it had less, else four times as
// many entries. Where the units per block alone would not give them, they become the least size of
// a ring, so that the next call of its kind does not run twice; the blocks stay spread.
inline void pool_grow(PoolRing& r, const PoolShape& used, uint64_t threads) {
    const uint32_t want = used.ring < r.cap ? r.cap : std::min<uint32_t>(r.cap * 4, kRingMax);
    r.cap = std::max(r.cap, want);
    if (pool_shape_of(r, used.per_block, 1, threads).ring < want) r.low = want;
}

}  // namespace cmpmc_gpu
