"""GPU tests of the resident kernel (whole ion cycles of a small discharge in
one launch, kernels_resident.cu) against the driver's launch-per-kernel steps
and against the invariants the driver keeps between runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E_MASS = 9.10938356e-31
AR_MASS = 6.63352090e-26
E_CHARGE = 1.60217662e-19


def _state(e, i, capacity, seed=5, **kw):
    import cudapic_b200 as cp
    from cudapic_b200.sim import GpuSimState, ParticlesSoA
    st = GpuSimState(cp.default_params(capacity=capacity, **kw))
    st.upload_electrons(ParticlesSoA(*e))
    st.upload_ions(ParticlesSoA(*i))
    st.seed(e_master=(0x1234 + seed, 0x11112222, 0x22223333, 0x33334444),
            i_master=(0x4444 + seed, 0x55556666, 0x66667777, 0x77778888))
    return st


def _soa(p):
    from cudapic_b200.sim import ParticlesSoA
    return ParticlesSoA(*p)


def _bulk(n, seed):
    """Electrons of 0.1 to 2 eV in the middle half of the gap.  The vacuum
    field of 250 V and the shot noise of the charge (sqrt(n) W e / (eps0 A))
    are below 1e4 V/m each: 20 steps add at most 1.3e6 m/s to 0.84e6, 13 eV,
    so none ionizes (15.8 eV) or reaches an electrode."""
    r = np.random.default_rng(seed)
    v = r.normal(0.0, 1.0, (3, n))
    ev = r.uniform(0.1, 2.0, n)
    v *= np.sqrt(2.0 * ev * E_CHARGE / E_MASS) / np.linalg.norm(v, axis=0)
    x = 0.025 * r.uniform(0.25, 0.75, n)
    return tuple(a.astype(np.float32) for a in (x, *v))


def _ions(n, seed):
    r = np.random.default_rng(seed)
    v = r.normal(0.0, np.sqrt(0.03 * E_CHARGE / AR_MASS), (3, n))
    return tuple(a.astype(np.float32) for a in (0.025 * r.uniform(0.25, 0.75, n), *v))


# capacities up to 8 and 16 CTAs' worth (16 312 and 32 688), nearly full ones
# among them (the electrons are shared out again every ion cycle)
@pytest.mark.parametrize("n,n_g,cap", [(1, 3, 8), (3, 64, 40), (2049, 400, 4100), (5003, 1023, 16_312),
                                       (16_301, 400, 16_312), (16_303, 800, 16_316), (20_000, 1024, 32_688)])
def test_one_ion_cycle_matches_launched_steps(cudapic, cuda_device, oracle, n, n_g, cap):
    """The same start, 20 steps: every electron keeps its slot and stream until
    the compaction at the end, so both paths make the same decisions.  The
    launched steps add f32 partial densities (1e-6 relative at most), here the
    sums are exact: E differs by up to 1e-6 e n L / eps0 = 0.5 V/m, a velocity by
    20 x 1.6 m/s (scattering turns it, nothing amplifies it), a position by
    20 dt x 32 m/s = 1e-8 m beside its own rounding (20 x 1.5e-9)."""
    from gpu_util import device_array
    w = 7.0e4 * 120000 / max(n, 1000)
    e, i = _bulk(n, n), _ions(n, n + 1)
    out = []
    for launched in (False, True):
        st = _state(e, i, cap, n_g=n_g, weight=w)
        try:
            if launched:
                st.set_overlap(False)  # any default switched off: launched steps
            st.run_steps(20)
            assert st.counts() == (n, n) and st.device_error() == 0
            assert st.work() == 20 * n + n and st.steps_done() == 20
            p, _ = st.download_electrons()
            q, _ = st.download_ions()
            b = st.buffers()
            ph = oracle.phys_from_params(n_g=n_g, capacity=st.capacity, weight=w)
            dens = device_array(b.e_density, n_g, np.float32)
            ref = oracle.get_density_f64(p.x, ph)
            assert np.linalg.norm(dens - ref) <= 2e-5 * np.linalg.norm(ref)
            st.run_steps(1)  # an ion step: the density collected over the cycle becomes current
            st.synchronize()
            dens = device_array(st.buffers().i_density, n_g, np.float32)
            ref = oracle.get_density_f64(q.x, ph)
            assert np.linalg.norm(dens - ref) <= 2e-5 * np.linalg.norm(ref)
            out.append((p, q))
        finally:
            st.close()
    (p, q), (pl, ql) = out
    np.testing.assert_allclose(np.sort(p.x), np.sort(pl.x), rtol=0, atol=5e-8)
    np.testing.assert_allclose(np.sort(q.x), np.sort(ql.x), rtol=0, atol=5e-8)  # pushed before the collisions
    for c in ("vx", "vy", "vz"):
        np.testing.assert_allclose(np.sort(getattr(p, c)), np.sort(getattr(pl, c)), rtol=0, atol=100.0)


def test_discharge_statistics_and_invariants(cudapic, cuda_device, oracle):
    """A discharge of 20 000 + 20 000 particles over 2000 steps (absorption,
    ionization, compaction each cycle; launched steps before and between):
    the counts and the mean energies of six seeds agree with the launched
    steps within six standard errors, the planes hold no hole."""
    from cudapic_b200.workloads import steady_state
    import cudapic_b200 as cp
    n = 20_000
    g = cp.grid_from_params()
    res = {}
    for launched in (False, True):
        rows = []
        for seed in range(6):
            e = steady_state(n, E_MASS, 3.0, dt=g.dt_e, seed=10 * seed)
            i = steady_state(n, AR_MASS, 0.03, dt=g.dt_i, seed=10 * seed + 1)
            st = _state(e, i, 2 * n, seed=seed, weight=7.0e4 * 120000 / n)
            try:
                if launched:
                    st.set_overlap(False)
                for steps in (7, 13, 400, 1560, 20):  # an odd number of cycles in between
                    st.run_steps(steps)
                assert st.device_error() == 0 and st.steps_done() == 2000
                p, ne = st.download_electrons()
                q, ni = st.download_ions()
                for s in (p, q):
                    assert np.all((s.x >= 0) & (s.x <= np.float32(0.025)))
                rows.append((ne, ni, float(np.mean(p.vx ** 2 + p.vy ** 2 + p.vz ** 2)), float(np.mean(np.abs(q.vx)))))
            finally:
                st.close()
        res[launched] = np.array(rows, np.float64)
    a, b = res[False], res[True]
    se = np.sqrt(a.var(axis=0, ddof=1) / 6 + b.var(axis=0, ddof=1) / 6)
    assert np.all(np.abs(a.mean(axis=0) - b.mean(axis=0)) <= 6 * se), (a.mean(axis=0), b.mean(axis=0), se)


@pytest.mark.parametrize("n_e,n_i", [(0, 0), (0, 500), (500, 0)])
def test_empty_species(cudapic, cuda_device, n_e, n_i):
    e, i = _bulk(n_e, 1), _ions(n_i, 2)
    st = _state(e, i, 1024, weight=7.0e4)
    try:
        st.run_steps(60)
        assert st.counts() == (n_e, n_i) and st.device_error() == 0
    finally:
        st.close()


def test_capacity_overflow_is_flagged(cudapic, cuda_device):
    """Hot electrons ionizing into full planes: spawns that do not fit are
    dropped and flagged, nothing is written past the planes."""
    import cudapic_b200 as cp
    r = np.random.default_rng(3)
    n = 4000
    v = r.normal(0.0, 1.0, (3, n))
    v *= np.sqrt(2.0 * 60.0 * E_CHARGE / E_MASS) / np.linalg.norm(v, axis=0)
    e = tuple(a.astype(np.float32) for a in (0.025 * r.uniform(0.4, 0.6, n), *v))
    st = _state(e, _ions(n, 4), n + 4, pressure=50.0, weight=10.0)
    try:
        st.run_steps(200)
        ne, ni = st.counts()
        assert ne <= n + 4 and ni <= n + 4
        assert st.device_error() & (cp.DEVERR_SPAWN_E | cp.DEVERR_SPAWN_I)
        p, m = st.download_electrons()
        assert m == ne and np.all((p.x >= 0) & (p.x <= np.float32(0.025)))
    finally:
        st.close()


def test_uneven_growth_is_shared_out_again(cudapic, cuda_device):
    """The first CTA's share (1750 of at most 2047 entries) holds 500 electrons
    of 100 eV that ionize within a few steps, the rest is cold: the electrons
    are shared out again in the middle of an ion cycle.  Every spawn finds a
    place, and each ionization adds one electron and one ion (nothing gets
    from the middle fifth of the gap to an electrode in 40 steps)."""
    r = np.random.default_rng(8)
    n = 14_000
    v = r.normal(0.0, 1.0, (3, n))
    ev = np.where(np.arange(n) < 500, 100.0, 0.5)
    v *= np.sqrt(2.0 * ev * E_CHARGE / E_MASS) / np.linalg.norm(v, axis=0)
    e = tuple(a.astype(np.float32) for a in (0.025 * r.uniform(0.4, 0.6, n), *v))
    st = _state(e, _ions(n, 9), 16_312, pressure=500.0, weight=1.0)
    try:
        st.run_steps(40)
        ne, ni = st.counts()
        assert st.device_error() == 0
        assert ne == ni and n + 400 < ne < 16_312
        p, m = st.download_electrons()
        assert m == ne and np.all((p.x > 0) & (p.x < np.float32(0.025)))
    finally:
        st.close()


@pytest.mark.parametrize("launched", [False, True])
def test_growth_past_a_quarter_in_one_cycle_finds_every_free_slot(cudapic, cuda_device, launched):
    """A fifth of 5000 electrons are absorbed at once (their slots stay with the
    first CTAs), the rest have 200 eV and ionize about 0.04 times a step each
    (50 Pa): 3000 spawns or so per ion cycle, in CTAs without absorbed ones.
    After the first cycle 2000 to 3000 of the 10 800 slots have not been given
    out, fewer than the second cycle needs and more than a quarter of the
    electrons; with the thousand absorbed ones' they suffice.  Nothing gets
    from the middle fifth of the gap to an electrode in 40 steps, so each
    ionization leaves one electron and one ion more."""
    r = np.random.default_rng(21)
    n, gone = 5000, 1000
    v = r.normal(0.0, 1.0, (3, n))
    v *= np.sqrt(2.0 * 200.0 * E_CHARGE / E_MASS) / np.linalg.norm(v, axis=0)
    x = 0.025 * r.uniform(0.4, 0.6, n)
    x[:gone], v[0, :gone] = 1e-6, -np.abs(v[0, :gone]) - 1e6
    e = tuple(a.astype(np.float32) for a in (x, *v))
    st = _state(e, _ions(n - gone, 22), 10_800, pressure=50.0, weight=1e-6)
    try:
        if launched:
            st.set_overlap(False)
        first = []
        for k in (20, 40):  # what the first cycle leaves, then two cycles in one call
            if k == 40:
                st.upload_electrons(_soa(e))
                st.upload_ions(_soa(_ions(n - gone, 22)))
                st.seed(e_master=(0x1234, 5, 6, 7), i_master=(0x4444, 5, 6, 7))
            st.run_steps(k)
            first.append(st.counts())
        (c1, _), (c2, i2) = first
        print("\nelectrons after one cycle", c1, "after two", c2)
        free = 10_800 - (c1 + gone)
        assert (c1 + gone) // 4 < free < c2 - c1  # the case described
        assert c2 < 10_800
        assert st.device_error() == 0 and c2 == i2
    finally:
        st.close()


def _free(n, seed, n_sub=20, capacity=16_312, voltage=250.0, speed=2e5, **kw):
    """A state whose electrons and ions only fall through the vacuum field: no
    gas, no charge.  No draw and no slot then decides anything, so two paths
    give the same particles bit for bit whatever slots these end in."""
    r = np.random.default_rng(seed)
    x = (0.025 * r.uniform(0.1, 0.9, (2, n))).astype(np.float32)
    v = (r.normal(0.0, 1.0, (2, 3, n)) * np.array([[[speed]], [[300.0]]])).astype(np.float32)
    st = _state((x[0], *v[0]), (x[1], *v[1]), capacity, seed=seed, n_sub=n_sub, voltage=voltage, pressure=1e-9,
                weight=1e-20, **kw)
    return st


def _particles(st):
    """Rows of both species in the order of vy, vz, which nothing changes."""
    out = []
    for soa, n in (st.download_electrons(), st.download_ions()):
        rows = np.stack([soa.x, soa.vx, soa.vy, soa.vz])[:, :n]
        out.append(rows[:, np.lexsort((rows[3], rows[2]))])
    assert st.device_error() == 0
    return out


@pytest.mark.parametrize("n,capacity,n_sub,calls", [
    (2047, 4096, 2, (40, 1, 139)), (5003, 16_312, 8, (24, 3, 37, 64)), (5003, 16_312, 20, (7, 133)),
    (20_001, 32_688, 20, (20,) * 6), (9001, 9004, 50, (120, 30))])
def test_rows_match_launched_steps(cudapic, cuda_device, n, capacity, n_sub, calls):
    """Several N_SUB, calls that begin or end inside an ion cycle, many short
    ones: each electron's and ion's whole row as the launched steps give it,
    with the field's acceleration and absorption at the electrodes."""
    got = []
    for launched in (False, True):
        st = _free(n, 31, n_sub, capacity)
        try:
            if launched:
                st.set_overlap(False)
            for c in calls:
                st.run_steps(c)
            assert st.steps_done() == sum(calls)
            got.append(_particles(st))
        finally:
            st.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
    assert 0 < got[0][0].shape[1] < n  # some electrons reached an electrode


def test_two_states_on_two_streams(cudapic, cuda_device):
    """Two discharges enqueued in turn without waiting: each as when alone."""
    want = []
    for seed, n in ((41, 3001), (42, 15_001)):
        with _free(n, seed) as st:
            st.set_overlap(False)
            st.run_steps(200)
            want.append(_particles(st))
    both = [_free(3001, 41), _free(15_001, 42)]
    try:
        for _ in range(5):
            for st in both:
                st.run_steps(40)
        for st, w in zip(both, want):
            for a, b in zip(_particles(st), w):
                np.testing.assert_array_equal(a, b)
    finally:
        for st in both:
            st.close()


def test_checkpoint_of_a_resident_run(cudapic, cuda_device, tmp_path):
    """One RF cycle, saved, loaded into another state: the RNG planes are the
    same, and 40 more steps give the same particles and planes in both."""
    from gpu_util import device_array
    planes = lambda st: [device_array(p, st.capacity, np.uint32) for sp in (0, 1) for p in st.buffers().rng[sp]]  # noqa: E731
    a, b = (_free(4001, 51, voltage=0.0, speed=5e3) for _ in range(2))
    try:
        a.run_steps(4000)
        a.save(tmp_path / "picdata.bin")
        b.load(tmp_path / "picdata.bin")
        for steps in (0, 40):
            for st in (a, b):
                if steps:
                    st.run_steps(steps)
                st.synchronize()
            for p, q in zip(planes(a), planes(b)):
                np.testing.assert_array_equal(p, q)
        for p, q in zip(_particles(a), _particles(b)):
            np.testing.assert_array_equal(p, q)
    finally:
        a.close()
        b.close()


def test_overflow_leaves_counters_planes_and_densities_in_agreement(cudapic, cuda_device, oracle):
    """Spawns into full planes, as test_capacity_overflow_is_flagged, by what
    the device holds: both counters within the capacity, every slot below them
    a particle of its own in the gap, and the densities those of just these
    particles (2e-5, as the deposit elsewhere)."""
    from gpu_util import device_array
    r = np.random.default_rng(3)
    n, w = 4000, 10.0
    v = r.normal(0.0, 1.0, (3, n))
    v *= np.sqrt(2.0 * 60.0 * E_CHARGE / E_MASS) / np.linalg.norm(v, axis=0)
    e = tuple(a.astype(np.float32) for a in (0.025 * r.uniform(0.4, 0.6, n), *v))
    st = _state(e, _ions(n, 4), n + 4, pressure=50.0, weight=w)
    ph = oracle.phys_from_params(capacity=n + 4, weight=w)
    try:
        st.run_steps(200)
        st.synchronize()
        b = st.buffers()
        raw = [int(device_array(p, 1, np.uint32)[0]) for p in (b.n_electrons, b.n_ions)]
        assert max(raw) <= n + 4 and raw == list(st.counts()) and raw[1] == n + 4
        parts = []
        for sp, m in enumerate(raw):
            rows = np.stack([device_array(p[sp], m, np.float32) for p in (b.x, b.vx, b.vy, b.vz)])
            assert np.all(np.isfinite(rows)) and np.all((rows[0] >= 0) & (rows[0] <= np.float32(0.025)))
            assert np.unique(rows, axis=1).shape[1] == m
            parts.append(rows[0])
        dens = device_array(b.e_density, 400, np.float32)
        ref = oracle.get_density_f64(parts[0], ph)
        assert np.linalg.norm(dens - ref) <= 2e-5 * np.linalg.norm(ref)
        st.run_steps(1)  # an ion step: the density collected over the cycle becomes current
        st.synchronize()
        dens = device_array(st.buffers().i_density, 400, np.float32)
        ref = oracle.get_density_f64(parts[1], ph)
        assert np.linalg.norm(dens - ref) <= 2e-5 * np.linalg.norm(ref)
    finally:
        st.close()


_FEW_SMS = """
import sys
sys.path[:0] = [%r, %r]
from cuda.bindings import driver as d
import test_gpu_resident as T

def ok(r):
    assert r[0] == d.CUresult.CUDA_SUCCESS, r
    return r[1] if len(r) == 2 else r[1:]

ok(d.cuInit(0))
dev = ok(d.cuDeviceGet(0))
ok(d.cuCtxSetCurrent(ok(d.cuDevicePrimaryCtxRetain(dev))))
sms = ok(d.cuDeviceGetDevResource(dev, d.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
part = ok(d.cuDevSmResourceSplitByCount(1, sms, 0, 32))[0]
ctx = ok(d.cuGreenCtxCreate(ok(d.cuDevResourceGenerateDesc(part, 1)), dev,
                            d.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
few = ok(d.cuGreenCtxStreamCreate(ctx, d.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
whole = ok(d.cuStreamCreate(d.CUstream_flags.CU_STREAM_NON_BLOCKING))
n = 12_000
st = T._state(T._bulk(n, 1), T._ions(n, 2), 20_000, weight=1e-20, voltage=0.0, pressure=1e-9)  # free flight
for stream in (few, whole):
    st.set_stream(int(stream))
    st.run_steps(20)
    assert st.counts() == (n, n) and st.device_error() == 0
st.close()
print("done")
"""


def test_stream_with_few_sms(cudapic, cuda_device):
    """A stream of 32 SMs (a green context's) holds no cluster of 16 CTAs of
    one SM each: the steps run there as launched steps, and on a stream of
    the whole device as before.  In a process of its own, for the context."""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    r = subprocess.run([sys.executable, "-c", _FEW_SMS % (os.path.dirname(here), here)], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.endswith("done\n"), r.stderr[-2000:]
