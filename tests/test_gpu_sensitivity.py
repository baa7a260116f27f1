"""GPU tests of the voltage-sensitivity path (cudapic_sens_*): the slot-form
forward run bit for bit against the oracle's f32 model, the adjoint against
the oracle's adjoint (double, Jacobians by central differences, Thomas
Poisson adjoint), checkpoint and horizon invariants, and the adjoint against
central differences with common random numbers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E_MASS = 9.10938356e-31
AR_MASS = 6.63352090e-26
V0 = 250.0


def _pair(oracle, n=3000, seed=1):
    """A GPU state and the oracle's copy of it: the same particles, the same
    RNG planes."""
    import cudapic_b200 as cp
    from cudapic_b200.sim import GpuSimState, ParticlesSoA
    from cudapic_b200.workloads import steady_state
    from gpu_util import device_array
    cap = 2 * n + 1000
    w = 7e4 * 120000 / n
    st = GpuSimState(cp.default_params(capacity=cap, weight=w))
    g = st.grid
    e = steady_state(n, E_MASS, 3.0, dt=g.dt_e, seed=seed)
    i = steady_state(n, AR_MASS, 0.03, dt=g.dt_i, seed=seed + 1)
    st.upload_electrons(ParticlesSoA(*e))
    st.upload_ions(ParticlesSoA(*i))
    st.seed(e_master=(0x1234 + seed, 0x11112222, 0x22223333, 0x33334444),
            i_master=(0x4444 + seed, 0x55556666, 0x66667777, 0x77778888))
    st.synchronize()
    b = st.buffers()
    rng = [[device_array(b.rng[sp][k], cap, np.uint32) for k in range(4)] for sp in (0, 1)]
    return st, oracle.SensState(cap, e, i, rng[0], rng[1]), oracle.phys_from_params(capacity=cap, weight=w)


def test_forward_bit_exact_against_oracle(cudapic, cuda_device, oracle, tables):
    """200 steps (10 ion steps, collisions, spawns, absorptions): every slot's
    position, velocity and RNG state, the slot counts and the observables
    equal the oracle's f32 model."""
    from cudapic_b200.sensitivity import VoltageSensitivity
    st, ost, ph = _pair(oracle)
    try:
        with VoltageSensitivity(st, 200, 40) as s:
            obs = s.forward(V0)
            info = s.info()
            got = [s.download(sp) for sp in (0, 1)]
    finally:
        st.close()
    oobs, _ = oracle.sens_run(ph, tables, V0, 200, ost, grad=False)
    assert info["device_error"] == 0 and ost.dev_err == 0
    assert list(info["slots"]) == list(ost.n)
    assert ost.n[0] > 3000 and ost.n[1] > 3000
    for sp in (0, 1):
        n = ost.n[sp]
        for k in range(4):
            np.testing.assert_array_equal(got[sp][k][:n], ost.p[sp][k][:n], err_msg="species %d plane %d" % (sp, k))
            np.testing.assert_array_equal(got[sp][4][k][:n], ost.rng[sp][k][:n], err_msg="species %d rng %d" % (sp, k))
        assert np.count_nonzero(got[sp][0][:n] < 0) > 0
    # observable sums: FP64 atomics on the GPU, sequential on the CPU
    assert obs["power_e"] == pytest.approx(oobs[0], rel=1e-9)
    assert obs["ion_flux_gnd"] == pytest.approx(oobs[1], rel=1e-9)


@pytest.mark.parametrize("n", [1, 255, 1025, 2_500_000])
def test_forward_sizes_bit_exact(cudapic, cuda_device, oracle, tables, n):
    """One ion cycle from a single particle to more rounds per CTA (17 of
    1024 slots) than a 32-bit deposit histogram takes without a drain (3).
    RNG states bit for bit.  Positions: the FP64 field sums run in another
    order than the oracle's, so a node's f32 field may round the other way:
    one ulp of at most 1e6 V/m in each of 20 steps moves a particle by at
    most 20 dt x 20 x |factor| x 1e6 x 2^-23 = 3e-9 m, and each step rounds
    x by 2^-24 of the gap (20 x 1.5e-9 m).  A drain that lost or doubled
    weights would change the charge by its own size."""
    from cudapic_b200.sensitivity import VoltageSensitivity
    st, ost, ph = _pair(oracle, n=n)
    try:
        with VoltageSensitivity(st, 20, 20) as s:
            s.forward(V0)
            info = s.info()
            got = [s.download(sp) for sp in (0, 1)]
    finally:
        st.close()
    oracle.sens_run(ph, tables, V0, 20, ost, grad=False)
    assert info["device_error"] == 0 and list(info["slots"]) == list(ost.n)
    for sp in (0, 1):
        m = ost.n[sp]
        np.testing.assert_allclose(got[sp][0][:m], ost.p[sp][0][:m], rtol=0, atol=3.3e-8)
        for k in range(4):
            np.testing.assert_array_equal(got[sp][4][k][:m], ost.rng[sp][k][:m])


@pytest.mark.parametrize("window,every", [(100, 100), (200, 40)])
def test_device_memory(cudapic, cuda_device, oracle, window, every):
    """Per slot: initial and present state 64 B each, spawn requests 28, a
    checkpoint of 64 per interval, the tape's 8 per step and per ion step,
    adjoints of one observable 32 (two are held: the first checkpoint is the
    initial state); the records of 36 and 40 B; nodes of the tape; 64 KB of
    small buffers."""
    from cudapic_b200.sensitivity import VoltageSensitivity
    st, _, _ = _pair(oracle, n=20_000)
    cap = st.capacity
    try:
        with VoltageSensitivity(st, window, every) as s:
            got = s.info()["device_bytes"]
            s.forward(V0)
            s.backward()
            assert s.info()["device_bytes"] == got
    finally:
        st.close()
    slot = 64 + 64 + 28 + 64 * (window // every) + 8 * every + 8 * (every // 20) + 32
    records = 36 * (cap * every // 32 + 65536) + 40 * (cap * (every // 20) // 8 + 65536)
    assert got <= slot * cap + records + 4 * 400 * every + 65536


@pytest.mark.parametrize("on", [True, False])
def test_launch_overlap_follows_the_state(cudapic, cuda_device, oracle, on):
    """set_overlap(False): no kernel of a forward and backward run begins
    before the one before it has ended (by the profiler's record); with it,
    some do (how many is the host's pace)."""
    from torch.autograd import DeviceType
    from torch.profiler import ProfilerActivity, profile
    from cudapic_b200.sensitivity import VoltageSensitivity
    st, _, _ = _pair(oracle)
    st.set_overlap(on)
    try:
        with VoltageSensitivity(st, 100, 100) as s:
            s.forward(V0)
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                s.forward(V0)
                s.backward()
    finally:
        st.close()
    spans = sorted((e.time_range.start, e.time_range.end) for e in prof.events()
                   if e.device_type == DeviceType.CUDA and "cudapic" in e.name)
    assert len(spans) > 1000
    early = sum(b[0] < a[1] for a, b in zip(spans, spans[1:]))
    assert early > 0 if on else early == 0, (early, len(spans))


def test_adjoint_against_oracle(cudapic, cuda_device, oracle, tables):
    """d obs / dV0 over 200 steps (checkpoints every 40): f32 tangents with
    FP64 field sums on the GPU against the oracle's double adjoint on the
    same trajectory."""
    from cudapic_b200.sensitivity import VoltageSensitivity
    st, ost, ph = _pair(oracle)
    try:
        with VoltageSensitivity(st, 200, 40) as s:
            s.forward(V0)
            g = s.backward()
    finally:
        st.close()
    _, og = oracle.sens_run(ph, tables, V0, 200, ost)
    print("\nadjoint GPU %s oracle %s" % (g, og))
    assert g["power_e"] == pytest.approx(og[0], rel=2e-3)
    assert g["ion_flux_gnd"] == pytest.approx(og[1], rel=2e-3)


def test_checkpoints_and_horizon(cudapic, cuda_device, oracle):
    """The recompute reproduces the forward run: the adjoint does not depend
    on the checkpoint interval; a horizon equal to the window is the full
    adjoint, a horizon of one checkpoint interval truncates it."""
    from cudapic_b200.sensitivity import VoltageSensitivity
    st, _, _ = _pair(oracle)
    res = {}
    try:
        for every, horizon in ((20, 0), (200, 0), (40, 200), (40, 40)):
            with VoltageSensitivity(st, 200, every, horizon) as s:
                s.forward(V0)
                res[(every, horizon)] = s.backward()
    finally:
        st.close()
    for key in ("power_e", "ion_flux_gnd"):
        a = res[(20, 0)][key]
        assert res[(200, 0)][key] == pytest.approx(a, rel=1e-9)
        assert res[(40, 200)][key] == pytest.approx(a, rel=1e-9)
        assert res[(40, 40)][key] != pytest.approx(a, rel=1e-6)


def test_adjoint_against_central_difference(cudapic, cuda_device):
    """The reference-case discharge with 2e5 electrons, relaxed one RF cycle
    (by the fused driver, whose compaction order varies from run to run, so
    the start differs between runs); a 200-step window: the pathwise adjoint
    against central differences with common random numbers.
    Measured over four starts: ion flux 0.4 - 4.5 % apart; electron power
    adjoint / difference 0.58 - 0.78, because the pathwise derivative omits
    what the difference also contains, the electrons whose collision
    decision or absorption at an electrode flips between V0 - dV and
    V0 + dV (the frozen events).  Such a flip can throw a single difference
    far off on an unlucky start (one start gave -3.1e15 for the flux at
    dV0 = 0.5 V against an adjoint of 1.9e14), and it depends on dV0: the
    difference taken is the median of those at dV0 = 0.5, 0.25 and 0.1 V.
    Asserted: the flux within 10 %, the power's sign and a factor 2.5.  The
    exact checks of the adjoint are the oracle's (central differences at
    1 mV, 1e-4) and the GPU against the oracle."""
    from cudapic_b200.sensitivity import VoltageSensitivity, steady_state
    st = steady_state(200_000, relax_cycles=1)
    try:
        with VoltageSensitivity(st, 200, 200) as s:
            s.forward(V0)
            g = s.backward()
            fds = [s.central_difference(V0, dv) for dv in (0.5, 0.25, 0.1)]
            assert s.info()["device_error"] == 0
    finally:
        st.close()
    fd = {k: float(np.median([f[k] for f in fds])) for k in g}
    print("\nadjoint %s\ncentral differences %s\nmedian %s" % (g, fds, fd))
    assert g["ion_flux_gnd"] == pytest.approx(fd["ion_flux_gnd"], rel=0.10)
    ratio = g["power_e"] / fd["power_e"]
    assert 0.4 < ratio < 2.5, ratio
