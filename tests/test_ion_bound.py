"""The ion test's certain-rejection bound (mcc.cuh ion_collides, the
bounded ion MCC entry) checked on the CPU against the oracle's full test
(Rust-CUDA/src/main.rs:1180-1197): no ion whose test draw lies at or above
the bound collides, over populations from thermal to 20 eV ions and time
steps up to 200x the reference's.  The draws are xoshiro128+ steps restated
in numpy (the fifth output of each slot's stream: four for the target's
Box-Muller normals, then the test draw)."""
import numpy as np
import pytest

AR_MASS = 6.63352090e-26


def _next(s):
    """One xoshiro128+ step of every stream (four uint32 planes, updated in place)."""
    s0, s1, s2, s3 = s
    out = (s0 + s3).astype(np.uint32)
    t = (s1 << np.uint32(9)).astype(np.uint32)
    s2 ^= s0
    s3 ^= s1
    s1 ^= s2
    s0 ^= s3
    s2 ^= t
    s3[:] = ((s3 << np.uint32(11)) | (s3 >> np.uint32(21))).astype(np.uint32)
    return out


def _uniform(out):
    return ((out >> np.uint32(9)) | np.uint32(0x3F800000)).view(np.float32) - np.float32(1.0)


def _bound(k, vx, vy, vz, normal_range):
    """fmaf(k, |v| + 9.2 sigma, 6e-7) as the kernels compute it (f32 inputs,
    one rounding of the fused multiply-add)."""
    v2 = (vx * vx + vy * vy + vz * vz).astype(np.float32)
    vmag = np.sqrt(v2).astype(np.float32)
    s = (vmag + np.float32(9.2) * np.float32(normal_range)).astype(np.float32)
    return (np.float64(k) * s.astype(np.float64) + 6e-7).astype(np.float32)


@pytest.mark.parametrize("n_t,temp,seed", [(4000, 0.03, 1), (4000, 2.0, 2), (200, 0.03, 3), (200, 20.0, 4),
                                           (20, 2.0, 5), (20, 20.0, 6)])
def test_no_ion_above_the_bound_collides(cudapic, oracle, tables, n_t, temp, seed):
    from cudapic_b200.workloads import steady_state
    cs, _, si = tables
    n = 200_000
    g = cudapic.grid_from_params(n_t=n_t, capacity=n)
    ph = oracle.phys_from_params(n_t=n_t, capacity=n)
    k = np.nextafter(np.float32(float(si.max()) * float(g.dt_i) * (1.0 + 1e-5)), np.float32(np.inf))
    _, vx, vy, vz = steady_state(n, AR_MASS, temp, seed=seed, edge_fraction=0.0)
    rng = [np.asarray(p).copy() for p in oracle.seed_streams([seed, 7, 11, 13], n)]
    s = [p.copy() for p in rng]
    for _ in range(4):
        _next(s)
    u = _uniform(_next(s))
    b = _bound(k, vx, vy, vz, g.normal_range)
    events = oracle.check_collisions_i(si, cs, n, [vx.copy(), vy.copy(), vz.copy()], [p.copy() for p in rng], ph)
    skipped = u >= b
    assert not np.any(events[skipped]), "an ion above the bound collided"
    assert np.any(events > 0)
    if n_t == 4000:  # the reference's time step: nearly every ion skips the target's transcendentals
        assert skipped.mean() > 0.9, skipped.mean()


@pytest.mark.parametrize("n_t,temp,seed", [(4000, 0.03, 11), (4000, 2.0, 12), (200, 0.03, 13), (200, 20.0, 14),
                                           (20, 2.0, 15), (20, 20.0, 16)])
def test_bound_without_the_root_is_the_stricter_one(cudapic, oracle, tables, n_t, temp, seed):
    """kernels_mcc.cu's ion_surely_passes: the bound with the square root
    taken out.  Every draw it lets pass lies above the bound with the root, so
    no such ion collides, and it still decides nearly every thermal ion."""
    from cudapic_b200.workloads import steady_state
    f = np.float32
    cs, _, si = tables
    n = 200_000
    g = cudapic.grid_from_params(n_t=n_t, capacity=n)
    ph = oracle.phys_from_params(n_t=n_t, capacity=n)
    k = np.nextafter(f(float(si.max()) * float(g.dt_i) * (1.0 + 1e-5)), f(np.inf))
    k2 = (k * k).astype(f) * f(1.0001)
    c = f(np.float64(k) * np.float64(f(9.2) * f(g.normal_range)) + 6.5e-7) * f(1.000001)
    _, vx, vy, vz = steady_state(n, AR_MASS, temp, seed=seed, edge_fraction=0.0)
    v2 = (vx * vx + vy * vy + vz * vz).astype(f)

    def passes(u):
        y = (u - c).astype(f)
        return (y >= 0) & ((y * y).astype(f) >= (k2 * v2).astype(f))

    rng = [np.asarray(p).copy() for p in oracle.seed_streams([seed, 7, 11, 13], n)]
    s = [p.copy() for p in rng]
    for _ in range(4):
        _next(s)
    u = _uniform(_next(s))
    events = oracle.check_collisions_i(si, cs, n, [vx.copy(), vy.copy(), vz.copy()], [p.copy() for p in rng], ph)
    assert not np.any(events[passes(u)])
    b = _bound(k, vx, vy, vz, g.normal_range)
    assert np.all(u[passes(u)] >= b[passes(u)])
    # draws within a few ulp and within 1e-4 of the bound, where the two could differ
    for near in [b + f(d) for d in (-2e-7, -6e-8, 0.0, 6e-8, 1.2e-7, 1e-6, 1e-5)] + [(b * f(r)).astype(f) for r in (0.9999, 1.0001)]:
        near = near.astype(f)
        assert np.all(near[passes(near)] >= b[passes(near)])
    if n_t == 4000:
        assert passes(u).mean() > 0.9


@pytest.mark.parametrize("first", [None, 0, 1, 2, 11, 5001, 15801, 999_999])
def test_xt_ionization_bound_follows_the_table(cudapic, tables, first):
    """The energy below which the XT pass skips the ionization table
    (ionization_from) comes from the table itself: no entry that an electron
    below it meets (f32 index of common.cuh) has ionization in it, and the
    next two energies' may."""
    import ctypes
    lib = cudapic.lib
    fn = lib._ZN7cudapic15ionization_fromEPKf
    fn.restype, fn.argtypes = ctypes.c_float, [ctypes.c_void_p]
    cs = np.ascontiguousarray(tables[0]).reshape(5, -1).copy()
    if first is not None:
        cs[2, :first], cs[2, first:] = 0.0, 1e-20
    start = int(np.argmax(cs[2] != 0.0))
    assert first is None or start == first
    e = np.float32(fn(cs.ctypes.data))
    index = lambda v: int(np.float32(np.float32(v) / np.float32(0.001)) + np.float32(0.5))  # noqa: E731
    if e > 0:
        assert index(np.nextafter(e, np.float32(0))) < max(start, 1)
    assert start <= index(e) + 2
