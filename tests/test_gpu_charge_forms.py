"""The waiting form of the batched charge kernel against the other over what a carrier can meet: masks,
released energies, 2D and 3D field meshes, several valleys of fields, parked carriers. The two are one
text, but nothing makes a compiler round two copies alike: that they do is what this file shows."""
import numpy as np
import pytest

from tests.helpers import axisym_mesh, planar_mesh, recoil_mesh
from tests.test_gpu_spread import _same

pytestmark = pytest.mark.gpu


def _detector(case):
    import cmpmc_b200 as cm
    det = cm.DetectorModel()
    det.luke_sample_fraction = 0.0
    det.e_field = cm.UniformElectricField.from_bias(4.0, 2.54 * cm.units.cm)
    if case == "mask":  # bare crystal between the pads reflects
        for face in (0, 1):
            det.surfaces[face].electrode_mask = cm.ElectrodePatternMask.supercdms_qet_mask(det.solid.radius, 0.8)
    elif case == "debye":
        det.charge_release = 1
    elif case == "film":
        det.charge_release = 2
    elif case == "mesh3d":
        det.mesh_field_3d = recoil_mesh()
    elif case == "planar":
        det.mesh_field_2d = planar_mesh(det)
    elif case == "axisym_leman":
        det.mesh_field_2d = axisym_mesh(det)
        det.charge_stepping = 1
    elif case == "weak":
        det.e_field = cm.UniformElectricField.from_bias(0.3, 2.54 * cm.units.cm)
    elif case == "strong":
        det.e_field = cm.UniformElectricField.from_bias(60.0, 2.54 * cm.units.cm)
    return det


# 620 pairs: 1,240 carriers, one per warp as they are spread, nine per warp of 148 blocks of 32 threads
@pytest.mark.parametrize("case", ["plain", "mask", "debye", "film", "mesh3d", "planar", "axisym_leman", "weak", "strong"])
def test_forms_agree(ge_lattice, case):
    import cmpmc_b200 as cm
    det = _detector(case)
    eng, dense = cm.SimulationEngine(ge_lattice, det), cm.SimulationEngine(ge_lattice, det)
    dense.configure(threads_per_block=32, blocks_per_sm=1)
    ev = eng.generate(cm.workloads.pair_drift, 620, 29)
    opt = cm.RunOptions(seed=29, form="batched_fp32", want_event_stats=True)
    a, b = eng.run_packed(ev, opt), dense.run_packed(ev, opt)
    assert b.kernel_launches > a.kernel_launches  # the waiting form orders its carriers first
    assert a.stats.charges_collected > 0
    _same(a, b)


def test_parked_carriers(ge_lattice):
    """A queue of 8,192 phonons is less than the 32 that each of 1,240 carriers reserves: carriers park
    and resume over several rounds."""
    import cmpmc_b200 as cm
    det = _detector("plain")
    det.luke_sample_fraction = 0.002
    engines = [cm.SimulationEngine(ge_lattice, det) for _ in range(3)]
    engines[1].configure(threads_per_block=32, blocks_per_sm=1)
    engines[2].configure(threads_per_block=32, blocks_per_sm=1, queue_capacity=8192)
    ev = engines[0].generate(cm.workloads.pair_drift, 620, 29)
    opt = cm.RunOptions(seed=29, form="batched_fp32", want_event_stats=True)
    one, dense, parked = (e.run_packed(ev, opt) for e in engines)
    assert parked.kernel_launches > dense.kernel_launches
    assert np.array_equal(one.event_stats["charges_collected"], dense.event_stats["charges_collected"])
    _same(one, dense)
    _same(one, parked)
