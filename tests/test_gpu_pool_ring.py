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
