"""Small batches spread over the chip: how many units a warp and a block take (and which lane,
warp or SM runs a unit) must not change any event. Each size is compared with the same batch
packed as densely as the launch allows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FLOAT_SUMS = ("total_luke_phonon_eV", "charge_recomb_edep_eV", "total_injected_eV", "total_deposited_eV",
              "escaped_or_killed_eV")


def _sorted_hits(res):
    """The hits with their event, in one fixed order: an event's hits are a set in no order."""
    ev = np.repeat(np.arange(len(res.hit_offsets) - 1), np.diff(res.hit_offsets.astype(np.int64)))
    order = np.lexsort((res.hits["edep"], res.hits["time"], ev))
    return ev[order], res.hits[order]


def _same(a, b):
    assert np.array_equal(a.hit_offsets, b.hit_offsets)
    for (ea, ha), (eb, hb) in [(_sorted_hits(a), _sorted_hits(b))]:
        assert np.array_equal(ea, eb)
        assert ha.tobytes() == hb.tobytes()
    for name in a.event_stats.dtype.names:
        x, y = a.event_stats[name], b.event_stats[name]
        if name in FLOAT_SUMS:  # FP64 atomic sums of an event's units: the order is free
            np.testing.assert_allclose(x, y, rtol=1e-12, atol=1e-18, err_msg=name)
        else:
            assert np.array_equal(x, y), name


def _engine(lattice, drift=False):
    import cmpmc_b200 as cm
    det = cm.DetectorModel()
    if drift:
        det.e_field = cm.UniformElectricField.from_bias(4.0, 2.54 * cm.units.cm)
        det.luke_sample_fraction = 0.0
        det.charge_max_dk_frac = 0.5
        det.charge_dt_cap_s = 1e-9
    return cm.SimulationEngine(lattice, det)


# 148 SMs: one unit per block below, two on one block above; 2,369 units: the first size at
# which a warp of a block claims two units (148 blocks of 16 warps)
@pytest.mark.parametrize("n", [1, 2, 147, 148, 149, 2368, 2369])
def test_pool_sizes(ge_lattice, n):
    import cmpmc_b200 as cm
    eng, dense = _engine(ge_lattice), _engine(ge_lattice)
    dense.configure_pool(2)  # the warp pool packs 128 units into a block
    packed = eng.generate(cm.workloads.single_l_volume, n, 31)
    opt = cm.RunOptions(seed=31, form="batched_fp32", want_event_stats=True)
    _same(eng.run_packed(packed, opt), dense.run_packed(packed, opt))


# a lineage that needs more ring than a spread block holds: the call reruns packed
def test_pool_overflow_falls_back_to_packed_blocks(ge_lattice):
    import cmpmc_b200 as cm
    det = cm.DetectorModel()
    eng, ref = cm.SimulationEngine(ge_lattice, det), cm.SimulationEngine(ge_lattice, det)
    ref.configure_pool(2)

    def generate(inp):  # one phonon of 2 eV: thousands of daughters are pending at once
        inp.phonons.append(eng.make_track((0.0, 0.0, 0.0), inp.rng.isotropic_dir(), 0, 2.0))
        inp.injected_eV = 2.0
    packed = eng.generate_python(generate, 2, 5)
    opt = cm.RunOptions(seed=5, form="batched_fp32", want_event_stats=True)
    first = eng.run_packed(packed, opt)
    _same(first, ref.run_packed(packed, opt))
    _same(first, eng.run_packed(packed, opt))


# one unit per warp up to the resident warps (1,776 at three 128-thread blocks per SM, a
# quarter more on freed lanes), then two; (threads_per_block 32, one block per SM) packs them
@pytest.mark.parametrize("form,n", [("plain_fp64", 1), ("plain_fp64", 149), ("plain_fp64", 2221),
                                    ("batched_fp32_inline", 1), ("batched_fp32_inline", 3553)])
def test_thread_per_unit_sizes(ge_lattice, form, n):
    import cmpmc_b200 as cm
    eng, dense = _engine(ge_lattice), _engine(ge_lattice)
    dense.configure(threads_per_block=32, blocks_per_sm=1)
    packed = eng.generate(cm.workloads.single_l_volume, n, 17)
    opt = cm.RunOptions(seed=17, form=form, want_event_stats=True)
    a, b = eng.run_packed(packed, opt), dense.run_packed(packed, opt)
    assert a.hits.tobytes() == b.hits.tobytes()  # a fixed order in these forms
    _same(a, b)


# 518 and 519 events: seven and eight carriers per packed warp, where event draws begin to wait
@pytest.mark.parametrize("n", [1, 75, 518, 519, 1481])
def test_carrier_sizes(ge_lattice, n):
    import cmpmc_b200 as cm
    eng, dense = _engine(ge_lattice, drift=True), _engine(ge_lattice, drift=True)
    dense.configure(threads_per_block=32, blocks_per_sm=1)
    packed = eng.generate(cm.workloads.pair_drift, n, 11)
    opt = cm.RunOptions(seed=11, form="batched_fp32", want_event_stats=True)
    _same(eng.run_packed(packed, opt), dense.run_packed(packed, opt))


# one deposit per warp up to 1,184 (two 128-thread blocks on each of 148 SMs), then two
@pytest.mark.parametrize("n", [1, 1184, 1185, 2369])
def test_partition_sizes(ge_lattice, n):
    """Deposits in one call and one by one groups of 37: the same records and final states."""
    import cmpmc_b200 as cm
    from cmpmc_b200 import _ffi
    rng = np.random.default_rng(n)
    dep = np.zeros(n, dtype=_ffi.DEPOSIT_DTYPE)
    dep["pos"] = rng.uniform(-0.01, 0.01, (n, 3))
    dep["edep_eV"] = 10.0 ** rng.uniform(1.0, 4.0, n)
    dep["is_nuclear_recoil"] = np.arange(n) % 2
    states = rng.integers(1, 1 << 63, size=(n, 4), dtype=np.uint64)
    eng = _engine(ge_lattice)
    opts = cm.PartitionOptions(max_sampled_pairs=16, max_sampled_phonons=8)
    coff, ch, poff, ph, st = cm.partition_deposits_on_device(eng, dep, states, opts)
    for lo in range(0, n, max(37, n // 3)):
        hi = min(n, lo + 37)
        c2, ch2, p2, ph2, st2 = cm.partition_deposits_on_device(eng, dep[lo:hi], states[lo:hi], opts)
        assert np.array_equal(coff[lo:hi + 1] - coff[lo], c2) and np.array_equal(poff[lo:hi + 1] - poff[lo], p2)
        assert ch[int(coff[lo]):int(coff[hi])].tobytes() == ch2.tobytes()
        assert ph[int(poff[lo]):int(poff[hi])].tobytes() == ph2.tobytes()
        assert np.array_equal(st[lo:hi], st2)


# the waiting form (packed: nine carriers per warp) against the other with Luke phonons tracked, a
# queue that parks carriers, reflecting walls, a mesh field (carriers ordered by type alone) and
# second-order stepping
@pytest.mark.parametrize("case", ["queue", "walls", "mesh", "leman"])
def test_waiting_charges(ge_lattice, case):
    import cmpmc_b200 as cm
    from tests.helpers import axisym_mesh
    det = cm.DetectorModel()
    det.e_field = cm.UniformElectricField.from_bias(2.0, 2.54 * cm.units.cm)
    det.luke_sample_fraction = 0.002 if case == "queue" else 0.0
    if case == "walls":
        for s in det.surfaces:
            s.prob_charge_abs, s.prob_charge_spec = 0.5, 0.5
    elif case == "mesh":
        det.mesh_field_2d = axisym_mesh(det)
    elif case == "leman":
        det.charge_stepping = 1
    eng, packed_eng = cm.SimulationEngine(ge_lattice, det), cm.SimulationEngine(ge_lattice, det)
    packed_eng.configure(threads_per_block=32, blocks_per_sm=1, queue_capacity=8192 if case == "queue" else 0)
    ev = eng.generate(cm.workloads.pair_drift, 620, 23)
    opt = cm.RunOptions(seed=23, form="batched_fp32", want_event_stats=True)
    _same(eng.run_packed(ev, opt), packed_eng.run_packed(ev, opt))
