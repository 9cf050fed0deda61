"""The rings of the SM-phase pool: a call whose rings do not overflow runs once."""
import pytest

pytestmark = pytest.mark.gpu


# A clean call without hits launches the unit map, the pool, the event offsets (two) and the totals;
# every rerun adds a pool launch. The phases near the end of a call claim from a nearly empty ring,
# where a floor read after other warps' claims lay past the tail and the next append counted as an
# overflow. 10,000 events in FP64 have more than 2^17 phonons pending in a block.
@pytest.mark.parametrize("form,n,ring", [(1, 1, 0), (1, 203, 0), (1, 2000, 0), (3, 203, 0), (3, 2000, 0),
                                         (3, 10000, 1 << 19)])
def test_no_rerun_without_overflow(ge_lattice, form, n, ring):
    import cmpmc_b200 as cm
    eng = cm.SimulationEngine(ge_lattice, cm.DetectorModel())
    eng.configure_pool(form, ring)
    packed = eng.generate(cm.workloads.mixed_energy, n, 31)
    opt = cm.RunOptions(seed=31, form="batched_fp32", keep_hits=False, want_event_stats=True)
    for _ in range(3):
        assert eng.run_packed(packed, opt).kernel_launches == 5


# Rings of 2,048 entries do not hold what 405 primaries of a block leave pending: the call reruns with
# larger ones (more than the five launches), the next has them from the start, and a call of a few
# units between them runs as it would have; a nearly full ring loses no phonon
@pytest.mark.parametrize("form", [1, 3])
def test_overflow_reruns_once_for_its_kind(ge_lattice, form):
    import cmpmc_b200 as cm
    from tests.test_gpu_spread import _same
    det = cm.DetectorModel()
    eng, ref = cm.SimulationEngine(ge_lattice, det), cm.SimulationEngine(ge_lattice, det)
    eng.configure_pool(form, 2048)
    ref.configure_pool(form, 1 << 17)
    opt = cm.RunOptions(seed=3, form="batched_fp32", keep_hits=False, want_event_stats=True)
    many = eng.generate(cm.workloads.mixed_energy, 600, 3)
    few = eng.generate(cm.workloads.mixed_energy, 2, 4)
    assert eng.run_packed(few, opt).kernel_launches == 5
    first = eng.run_packed(many, opt)
    assert first.kernel_launches > 5
    want = ref.run_packed(many, opt)
    assert want.kernel_launches == 5
    _same(first, want)
    assert eng.run_packed(few, opt).kernel_launches == 5
    again = eng.run_packed(many, opt)
    assert again.kernel_launches == 5
    _same(again, want)
