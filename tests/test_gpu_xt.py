"""GPU tests of the XT diagnostics and the <j E> power absorption (eduPIC's
measurement mode, C/eduPIC.cc:557-614, :705-715, :864-903, :1011-1026)
against the oracle's restatement of one step and of norm_all_xt."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

E_MASS = 9.10938356e-31
AR_MASS = 6.63352090e-26
E_CHARGE = 1.60217662e-19


def _state(n, n_g=400, seed=3, **kw):
    import cudapic_b200 as cp
    from cudapic_b200.sim import GpuSimState, ParticlesSoA
    from cudapic_b200.workloads import steady_state
    params = cp.default_params(n_g=n_g, capacity=2 * n, weight=7.0e4 * 120000 / n, **kw)
    st = GpuSimState(params)
    g = st.grid
    e = steady_state(n, E_MASS, 3.0, gap=params.gap, dt=g.dt_e, seed=seed)
    i = steady_state(n, AR_MASS, 0.03, gap=params.gap, dt=g.dt_i, seed=seed + 1)
    st.upload_electrons(ParticlesSoA(*e))
    st.upload_ions(ParticlesSoA(*i))
    st.seed()
    return st, e, i


def test_xt_first_step_matches_oracle(cudapic, cuda_device, oracle, tables):
    """Step 0 (an ion step) of a measurement window: column 0 of every XT
    quantity equals the oracle's accumulation of the particles before the
    push in the step's field, normalised as eduPIC does (f32 partial sums
    per CTA, hence the 2e-5 relative tolerance); the other columns are 0."""
    from gpu_util import device_array
    n = 60_000
    st, e, i = _state(n)
    try:
        st.set_measure(True)
        st.run_steps(1)
        st.synchronize()
        n_g, n_xt = st.xt_shape()
        assert (n_g, n_xt) == (400, 200)
        b = st.buffers()
        ef = device_array(b.efield, n_g, np.float32)
        pot = device_array(b.pot, n_g, np.float32)
        cumul_e, cumul_i, _ = st.download_measurements()
        ph = oracle.phys_from_params(capacity=2 * n, weight=7.0e4 * 120000 / n)
        cs_ion = tables[0].reshape(5, -1)[2]
        re = oracle.xt_accumulate(ef, *e, False, cs_ion, ph)
        ri = oracle.xt_accumulate(ef, *i, True, None, ph)
        raw = {"count_e": re[0], "ue": re[1], "meanee": re[2], "ioniz": re[3], "count_i": ri[0], "ui": ri[1],
               "meanei": ri[2], "pot": pot.astype(np.float64), "efield": ef.astype(np.float64),
               "ne": np.asarray(cumul_e), "ni": np.asarray(cumul_i)}
        raw = {k: np.stack([v] + [np.zeros_like(v)] * (n_xt - 1), axis=1) for k, v in raw.items()}
        p = st.params
        want = oracle.xt_normalise(raw, p.n_t, n_xt, 1, p.gap, p.n_g, p.frequency, p.weight, p.electrode_area)
        for name in ("pot", "efield", "ne", "ni"):
            np.testing.assert_array_equal(st.download_xt(name), want[name], err_msg=name)
        for name in ("je", "ji", "powere", "poweri", "meanee", "meanei", "ioniz"):
            got = st.download_xt(name)
            scale = float(np.abs(want[name]).max())
            assert scale > 0, name
            np.testing.assert_allclose(got, want[name], rtol=2e-5, atol=2e-5 * scale, err_msg=name)
            assert not np.any(got[:, 1:]), name
    finally:
        st.close()


def test_xt_batched_step_matches_each_discharge_alone(cudapic, cuda_device):
    """A measuring batch fills every discharge's XT columns like the
    discharges alone (same first step; f32 partial sums per CTA differ in
    partition, hence the tolerance)."""
    import cudapic_b200 as cp
    from cudapic_b200.sim import GpuBatch, GpuSimState, ParticlesSoA
    from cudapic_b200.workloads import steady_state
    cases = [(400, 1500, 250.0, 10.0, 0.025), (200, 997, 120.0, 30.0, 0.018), (800, 1789, 480.0, 6.0, 0.038)]

    def make(k, case):
        n_g, n, v, p, gap = case
        st = GpuSimState(cp.default_params(voltage=v, pressure=p, gap=gap, n_g=n_g, capacity=2048, weight=7.0e4))
        g = st.grid
        st.upload_electrons(ParticlesSoA(*steady_state(n, E_MASS, 3.0, gap=gap, dt=g.dt_e, seed=10 + k)))
        st.upload_ions(ParticlesSoA(*steady_state(n, AR_MASS, 0.03, gap=gap, dt=g.dt_i, seed=20 + k)))
        st.seed(e_master=(0x1234 + k, 1, 2, 3), i_master=(0x4444 + k, 5, 6, 7))
        st.set_measure(True)
        return st

    together = [make(k, c) for k, c in enumerate(cases)]
    alone = [make(k, c) for k, c in enumerate(cases)]
    try:
        with GpuBatch(together) as b:
            b.run_steps(1)
            b.synchronize()
        for st in alone:
            st.run_steps(1)
        for k, (x, y) in enumerate(zip(together, alone)):
            for name in ("pot", "efield", "ne", "ni"):
                np.testing.assert_array_equal(x.download_xt(name), y.download_xt(name), err_msg="%d %s" % (k, name))
            for name in ("je", "ji", "meanee", "meanei", "ioniz", "powere", "poweri"):
                gx, gy = x.download_xt(name), y.download_xt(name)
                scale = max(1e-300, float(np.abs(gy).max()))
                np.testing.assert_allclose(gx, gy, rtol=2e-5, atol=2e-5 * scale, err_msg="%d %s" % (k, name))
    finally:
        for st in together + alone:
            st.close()


def test_xt_files_and_power_over_periods(cudapic, cuda_device, tmp_path):
    """Two RF periods of measurement: every column filled, eduPIC's eleven
    *_xt.dat files of N_G rows and N_XT columns, and the report's <j E>
    power: the electrons absorb power on average, and the space-time mean
    of the power files is the report's figure."""
    st, _, _ = _state(200_000)
    try:
        st.run_steps(4000)
        st.set_measure(True)
        st.run_steps(8000)
        st.synchronize()
        n_g, n_xt = st.xt_shape()
        ne = st.download_xt("ne")
        assert np.all(ne[n_g // 2] > 0)                     # the centre is populated in every column
        st.write_xt(tmp_path)
        for name in ("pot", "efield", "ne", "ni", "je", "ji", "powere", "poweri", "meanee", "meanei", "ioniz"):
            a = np.loadtxt(tmp_path / ("%s_xt.dat" % name))
            assert a.shape == (n_g, n_xt), name
            np.testing.assert_allclose(a, st.download_xt(name), rtol=2e-6, atol=1e-300)
        r = st.report()
        assert r["power_e"] > 0 and np.isfinite(r["power_i"])
        assert r["power_e"] == pytest.approx(float(st.download_xt("powere").mean()), rel=1e-12)
        assert r["power_i"] == pytest.approx(float(st.download_xt("poweri").mean()), rel=1e-12)
        st.write_info(tmp_path / "info.txt")
        text = (tmp_path / "info.txt").read_text()
        if r["conditions_ok"]:
            assert "Absorbed power calculated as <j*E>:" in text
    finally:
        st.close()


@pytest.mark.parametrize("n_g", [3, 255, 800, 801, 1025, 4096])
def test_grid_quantities_over_several_columns(cudapic, cuda_device, oracle, n_g):
    """65 measured steps in a vacuum field of 250 V that changes every step:
    potential, field and densities summed per XT column equal, bit for bit, the
    FP64 sums of what each step leaves behind, in one call and in 65 (the same
    particles: three electrons and an ion without gas or charge)."""
    from cudapic_b200.sim import GpuSimState, ParticlesSoA
    from gpu_util import device_array
    steps, n_t = 65, 4000
    params = cudapic.default_params(capacity=64, n_g=n_g, pressure=1e-9, weight=1e-20, n_t=n_t)
    x = np.array([0.0070, 0.0125, 0.0190], np.float32)
    v = np.zeros((3, 3), np.float32)
    got, raw = [], None
    for calls in (1, steps):
        st = GpuSimState(params)
        st.upload_electrons(ParticlesSoA(x, *v))
        st.upload_ions(ParticlesSoA(x[:1], *v[:, :1]))
        st.seed()
        st.set_measure(True)
        n_xt = st.xt_shape()[1]
        if calls == 1:
            st.run_steps(steps)
        else:
            raw = {k: np.zeros((n_g, n_xt)) for k in ("pot", "efield", "ne", "ni", "count_e", "ue", "meanee", "ioniz",
                                                      "count_i", "ui", "meanei")}
            before, ion = (np.zeros(n_g), np.zeros(n_g)), None
            for t in range(steps):
                st.run_steps(1)
                st.synchronize()
                b = st.buffers()
                c = t // 20
                raw["pot"][:, c] += device_array(b.pot, n_g, np.float32).astype(np.float64)
                raw["efield"][:, c] += device_array(b.efield, n_g, np.float32).astype(np.float64)
                ce, ci, _ = st.download_measurements()
                if t % params.n_sub == 0:
                    ion = (ci - before[1]).astype(np.float32).astype(np.float64)
                raw["ne"][:, c] += (ce - before[0]).astype(np.float32).astype(np.float64)
                raw["ni"][:, c] += ion
                before = (ce.copy(), ci.copy())
        assert st.counts() == (3, 1) and st.device_error() == 0
        got.append({k: st.download_xt(k) for k in ("pot", "efield", "ne", "ni")} |
                   {"cumul": np.stack(st.download_measurements()[:2])})
        st.close()
    want = oracle.xt_normalise(raw, params.n_t, n_xt, steps, params.gap, n_g, params.frequency, params.weight,
                               params.electrode_area)
    for name in ("pot", "efield", "ne", "ni"):
        assert np.any(want[name])
        np.testing.assert_array_equal(got[1][name], want[name], err_msg=name)
        np.testing.assert_array_equal(got[0][name], got[1][name], err_msg=name)
    np.testing.assert_array_equal(got[0]["cumul"], got[1]["cumul"])


@pytest.mark.parametrize("over", [-3, 0, 1, 30_003])
def test_particle_sums_around_a_thread_per_particle(cudapic, cuda_device, oracle, tables, over):
    """The first measured step with as many particles as the grid's threads
    (1024 per SM: one per thread, beyond that four), and on both sides: the
    particle quantities of column 0 against the oracle (f32 partial sums per
    CTA of a few terms per node: 2e-5, as for smaller populations)."""
    import torch
    from gpu_util import device_array
    n = 1024 * torch.cuda.get_device_properties(0).multi_processor_count + over
    st, e, i = _state(n)
    try:
        st.set_measure(True)
        st.run_steps(1)
        st.synchronize()
        n_g, n_xt = st.xt_shape()
        ef = device_array(st.buffers().efield, n_g, np.float32)
        ph = oracle.phys_from_params(capacity=2 * n, weight=7.0e4 * 120000 / n)
        re = oracle.xt_accumulate(ef, *e, False, tables[0].reshape(5, -1)[2], ph)
        ri = oracle.xt_accumulate(ef, *i, True, None, ph)
        raw = dict(zip(("count_e", "ue", "meanee", "ioniz", "count_i", "ui", "meanei"), tuple(re) + tuple(ri)))
        cumul_e, cumul_i, _ = st.download_measurements()
        raw |= {"ne": np.asarray(cumul_e), "ni": np.asarray(cumul_i), "pot": np.zeros(n_g), "efield": np.zeros(n_g)}
        raw = {k: np.stack([v] + [np.zeros_like(v)] * (n_xt - 1), axis=1) for k, v in raw.items()}
        p = st.params
        want = oracle.xt_normalise(raw, p.n_t, n_xt, 1, p.gap, p.n_g, p.frequency, p.weight, p.electrode_area)
        for name in ("je", "ji", "meanee", "meanei", "ioniz"):
            got = st.download_xt(name)
            scale = float(np.abs(want[name]).max())
            assert scale > 0, name
            np.testing.assert_allclose(got, want[name], rtol=2e-5, atol=2e-5 * scale, err_msg=name)
    finally:
        st.close()
