// charge_shortcuts.cuh -- the two tests that spare the batched charge step its exit point and its
// kinetic energy (charge_kernel.inl), also compiled on the host to check them.
#pragma once

#include "phys.cuh"

namespace cmpmc_gpu {

// distance to the walls below which a step tests its exit point whatever its length, far above the
// FP32 rounding of that point
CMPMC_HD float wall_edge(float R, float H) { return 1e-4f * (R + H); }

// A carrier whose distance to every wall is over twice the step (plus the edge) cannot reach one;
// anything not finite takes the test.
CMPMC_HD bool clear_of_walls(float R, float H, float edge, float x, float y, float z, float d_step) {
    const float reach = 2.0f * d_step + edge;
    const float r_in = R - reach;
    return r_in > 0.0f && fabsf(z) < H - reach && x * x + y * y < r_in * r_in;
}

// |k| of an electron of mass m (eV) at the energies e_min (1 -+ 1e-3): far outside the rounding of
// either comparison, so |k| below lo or above hi decides as its kinetic energy against e_min would.
// A threshold that is not positive leaves every |k| between them.
struct KBand {
    float lo, hi;
};
inline KBand k_band(double e_min, double m) {
    if (!(e_min > 0.0)) return KBand{-1.0f, __builtin_huge_valf()};
    auto k_at = [&](double e) { return static_cast<float>(sqrt(e * e + 2.0 * e * m) / kHbarC); };
    return KBand{k_at(e_min * 0.999), k_at(e_min * 1.001)};
}

}  // namespace cmpmc_gpu
