"""The mixed SU(2)/SU(3) kernel over tiles of like sites (mixed_tiles.cuh) at the edges of its range: single sites,
kinds of different sizes or one kind alone, ragged tables with partners outside the lattice, one and two passes per
CTA, clusters of 1 to 16 CTAs.  Against the numpy restatement; tolerance as in test_gpu_mixed.py (states 1e-12)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mg(native):
    from classical_mcmc_spin_b200 import mixed_gpu_api
    return mixed_gpu_api


def _check(mg, arr, seed, method, steps, driven, save=3):
    import fixed_methods as fm
    import mixed_oracle as mo
    h, o = mg.create_from(arr), mo.MixedOracle(arr)
    rng = np.random.default_rng(seed)
    if driven:
        for sub, na, dim, set_pulse in ((2, arr["na2"], 3, mg.set_gpu_pulse_SU2), (3, arr["na3"], 8, mg.set_gpu_pulse_SU3)):
            fd = rng.normal(size=(2, na, dim))
            set_pulse(h, fd.ravel(), 0.5, 0.3, 1.1, 0.03, 0.1)
            o.set_pulse(sub, fd, 0.5, 0.3, 1.1, 0.03, 0.1)
    y0 = mg.random_mixed_state(arr, seed)
    mg.set_gpu_mixed_spins(h, y0)
    T1 = (steps - 0.5) * 0.02
    traj, times = mg.integrate_mixed_gpu(h, 0.0, T1, 0.02, save, method)
    rt, rs = fm.integrate(lambda y, t: o.rhs(y, t), y0, 0.0, T1, 0.02, save, method)
    np.testing.assert_array_equal(times, rt)
    assert np.abs(np.stack([s for _, s in traj]) - rs).max() <= 1e-12
    np.testing.assert_array_equal(mg.get_gpu_mixed_spins(h), traj[-1][1])


@pytest.mark.parametrize("L,na2,na3", [((1, 1, 1), 1, 1), ((1, 2, 3), 3, 1), ((2, 2, 7), 1, 3), ((7, 2, 1), 4, 4),
                                       ((3, 5, 8), 4, 3), ((7, 7, 7), 4, 4), ((8, 8, 8), 4, 4)])
@pytest.mark.parametrize("method,driven", [("ssprk53", True), ("rk4", False)])
def test_shapes(mg, L, na2, na3, method, driven):
    _check(mg, mg.synthetic_mixed_lattice(L, na2=na2, na3=na3, seed=sum(L) + na3), 50 + na2, method, 5, driven)


@pytest.mark.parametrize("method", ["euler", "rk2", "rk5", "dopri5", "rk78"])
def test_methods_over_several_ctas(mg, method):
    _check(mg, mg.synthetic_mixed_lattice((5, 4, 4), seed=60), 61, method, 4, True)


@pytest.mark.parametrize("L", [(2, 2, 2), (4, 4, 4)])
def test_ragged_tables(mg, L):
    arr = mg.synthetic_mixed_lattice(L, seed=70)
    rng = np.random.default_rng(71)
    for kp, kc, kv, z, n, limit, w in (("part2", "cnt2", "bil2", arr["z2"], arr["n2"], arr["n2"], 9),
                                       ("part3", "cnt3", "bil3", arr["z3"], arr["n3"], arr["n3"], 64),
                                       ("mpart2", "mcnt2", "mix2", arr["zm2"], arr["n2"], arr["n3"], 24),
                                       ("mpart3", "mcnt3", "mix3", arr["zm3"], arr["n3"], arr["n2"], 24)):
        cnt = rng.integers(0, z + 1, size=n)
        part = arr[kp].reshape(n, z).copy()
        part[rng.random((n, z)) < 0.2] = limit + rng.integers(0, 5)      # outside the lattice: skipped
        part[rng.random((n, z)) < 0.1] = -1
        val = arr[kv].reshape(n, z, w).copy()
        for s in range(n):
            val[s, cnt[s]:] = 1e300                                      # never read
        arr[kc], arr[kp], arr[kv] = cnt.astype(np.int64), part.ravel(), val.ravel()
    _check(mg, arr, 72, "ssprk53", 6, True)


@pytest.mark.parametrize("drop", [2, 3])
def test_one_kind_alone(mg, drop):
    arr = mg.synthetic_mixed_lattice((3, 4, 5), seed=80)
    keep = 5 - drop
    arr[f"n{drop}"] = 0
    arr[f"zm{keep}"] = 0
    for k in (f"field{drop}", f"onsite{drop}", f"bil{drop}", f"mix{drop}", f"mix{keep}"):
        arr[k] = np.zeros(0)
    for k in (f"part{drop}", f"cnt{drop}", f"mpart{drop}", f"mcnt{drop}", f"mpart{keep}"):
        arr[k] = np.zeros(0, np.int64)
    arr[f"mcnt{keep}"] = np.zeros(arr[f"n{keep}"], np.int64)
    _check(mg, arr, 81, "rk4", 6, False)
