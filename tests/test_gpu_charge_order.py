"""The order in which the waiting charge form starts its carriers is a permutation, also for carriers
whose drift distance lies on the edge of a bin of the order."""
import numpy as np
import pytest

from tests.test_gpu_spread import _same

pytestmark = pytest.mark.gpu


def test_carriers_on_bin_edges(ge_lattice):
    import cmpmc_b200 as cm
    det = cm.DetectorModel()
    det.e_field = cm.UniformElectricField.from_bias(4.0, 2.54 * cm.units.cm)
    det.luke_sample_fraction = 0.0
    n = 620  # nine carriers per warp of 148 blocks of 32 threads
    eng, dense = cm.SimulationEngine(ge_lattice, det), cm.SimulationEngine(ge_lattice, det)
    dense.configure(threads_per_block=32, blocks_per_sm=1)
    packed = eng.generate(cm.workloads.pair_drift, n, 19)
    # distances to both faces at multiples of a bin (2 max(R, H) / 64), one FP32 unit around them
    r, h = det.solid.radius, det.solid.half_z
    width = 2.0 * max(r, h) / 64.0
    k = np.arange(len(packed.charges))
    z = np.float32(h - width * (1 + k // 2 % int(2.0 * h / width - 1)))
    z = np.where(k % 3 == 0, z, np.where(k % 3 == 1, np.nextafter(z, np.float32(1)), np.nextafter(z, np.float32(-1))))
    packed.charges["pos"][:, 2] = z
    opt = cm.RunOptions(seed=19, form="batched_fp32", want_event_stats=True)
    a, b = eng.run_packed(packed, opt), dense.run_packed(packed, opt)
    assert a.stats.charges_collected == len(packed.charges)
    _same(a, b)
