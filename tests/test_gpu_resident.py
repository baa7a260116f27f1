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
